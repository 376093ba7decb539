"""The C++ reference operators whose sweeps can run out of a bounded wait report
it themselves, once, and leave no status behind for another call.  The status
word is set from the host, as a sweep that gave up leaves it."""
import os
import subprocess

import pytest

from rochpcg_b200 import build as B

pytestmark = pytest.mark.gpu

PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include "hpcg_b200.h"
#include "internal.hpp"
#include "problem.hpp"
using namespace hpcg_b200;

int main()
{
    hpcgb200_problem* p = nullptr;
    if(hpcgb200_problem_create_ex(24, 16, 32, 2, HPCGB200_FLAG_KEEP_GENERATED, &p)) return 2;
    const int m = p->A.localNumberOfRows, one = 1;
    Vector r, z;
    CudaInitializeVector(r, m);
    CudaInitializeVector(z, m);
    CudaFillRandomVector(r);
    auto gave_up = [&] { cudaMemcpy(rt().ref_status, &one, sizeof one, cudaMemcpyHostToDevice); };
    auto symgs = [&] { return ComputeSYMGS_ref(p->A, r, z); };
    auto mg = [&] { return ComputeMG_ref(p->A, r, z); };
    auto cg = [&] {
        int n;
        double a, b;
        return CG_ref(p->A, p->data, r, z, 2, 0.0, n, a, b, nullptr, true, false);
    };
    auto twice = [&](auto op) {
        op();  // whatever the call before left
        gave_up();
        const int first = op();
        std::printf("%d %d\n", first, op());
    };
    twice(symgs);
    twice(mg);
    twice(cg);
    // in a capture the sweeps wait for nothing; same result
    if(mg() || cudaDeviceSynchronize()) return 3;
    std::vector<double> direct(m), replayed(m);
    cudaMemcpy(direct.data(), z.d_values, sizeof(double) * m, cudaMemcpyDeviceToHost);
    cudaMemset(z.d_values, 0, sizeof(double) * m);
    cudaDeviceSynchronize();
    cudaGraph_t graph;
    cudaGraphExec_t exec;
    if(cudaStreamBeginCapture(rt().stream, cudaStreamCaptureModeRelaxed) || mg()) return 4;
    if(cudaStreamEndCapture(rt().stream, &graph) || cudaGraphInstantiate(&exec, graph, 0)) return 5;
    if(cudaGraphLaunch(exec, rt().stream) || cudaStreamSynchronize(rt().stream)) return 6;
    cudaMemcpy(replayed.data(), z.d_values, sizeof(double) * m, cudaMemcpyDeviceToHost);
    std::printf("%d\n", std::memcmp(direct.data(), replayed.data(), sizeof(double) * m));
    CudaDeleteVector(r);
    CudaDeleteVector(z);
    return hpcgb200_problem_destroy(p);
}
"""


def test_operators_report_their_own_time_out(tmp_path):
    src, exe = tmp_path / "status.cu", tmp_path / "status"
    src.write_text(PROGRAM)
    subprocess.run([B.nvcc()] + B.NVCC_FLAGS + ["-I" + os.path.join(B.PKG, "host"), str(src), "-o", str(exe), B.LIB,
                                                "-Xlinker", "-rpath=" + B.PKG], check=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    # HPCGB200_ERR_DEVICE_STATUS (6) for the call that gave up, 0 for the next
    assert r.stdout.splitlines() == ["6 0"] * 3 + ["0"]
