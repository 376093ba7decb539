// Reference kernels in natural row order on the generated row-major arrays:
// the arithmetic of the benchmark's `_ref` routines (src/ComputeSPMV_ref.cpp,
// src/ComputeSYMGS_ref.cpp, src/ComputeRestriction_ref.cpp,
// src/ComputeProlongation_ref.cpp, src/ComputeWAXPBY_ref.cpp,
// src/ComputeDotProduct_ref.cpp) on the device.  The benchmark driver runs
// them before OptimizeProblem for the reference timing phase and for the
// 50-iteration reference residual (src/main.cpp:288-341).
#pragma once

#include "common.cuh"

namespace hb {

// One MG level as GenerateProblem leaves it: row i = (iz*ny + iy)*nx + ix,
// 27 slots per row in (dz, dy, dx) order, pads (column -1) at the end.
struct NaturalLevel
{
    int nx, ny, nz;
    const int* ind;           // [m][27] column ids
    const double* val;        // [m][27] values
    const int8_t* nnz;        // nonzeros per row
    const int* diag_slot;     // slot of a_ii in its row
    __host__ __device__ long long rows() const { return (long long)nx * ny * nz; }
};

// Wavefronts of the natural-order Gauss-Seidel sweep: t = ix + 2 iy + 4 iz.
// Every stencil neighbour that precedes a row in natural order has a smaller
// t and every one that follows has a larger t, so sweeping t upwards
// (forward) or downwards (backward), one launch per t, reads exactly the
// values the sequential sweep reads.
__host__ __device__ inline int natural_fronts(int nx, int ny, int nz) { return (nx - 1) + 2 * (ny - 1) + 4 * (nz - 1) + 1; }

// Rows of one front are indexed (iy, j), j < width (natural.cu).
__host__ __device__ inline int natural_front_width(int nx) { return (nx + 3) / 4 + 1; }

#ifdef __CUDACC__
// floor(a / 4) for any sign of a.
__device__ __forceinline__ int floor_div4(int a) { return a >= 0 ? a / 4 : -((3 - a) / 4); }

// Row idx of front t of the Gauss-Seidel sweep (src/ComputeSYMGS_ref.cpp:68-85
// for one row).  Index (iy, j) is iz = izmin + j, ix = t - 2 iy - 4 iz; at
// most ceil(nx/4) + 1 values of iz meet 0 <= ix < nx for one (t, iy).  x is
// read through L2: earlier fronts may have been written by other SMs in the
// same kernel.
__device__ __forceinline__ void natural_front_row(const NaturalLevel& L, int t, int width, int idx,
                                                  const double* __restrict__ r, double* x)
{
    const int iy = idx / width;
    const int j = idx - iy * width;
    if(iy >= L.ny) return;
    const int u = t - 2 * iy;  // ix + 4 iz
    if(u < 0) return;
    const int izmin = max(0, -floor_div4(L.nx - 1 - u));  // ceil((u - nx + 1) / 4)
    const int iz = izmin + j;
    if(iz >= L.nz || 4 * iz > u) return;
    const int ix = u - 4 * iz;
    const long long row = ((long long)iz * L.ny + iy) * L.nx + ix;
    const size_t base = (size_t)row * kWidth;
    const int n = L.nnz[row];
    double sum = r[row];
    for(int q = 0; q < n; ++q) sum = __dsub_rn(sum, __dmul_rn(L.val[base + q], __ldcg(x + L.ind[base + q])));
    const double d = L.val[base + L.diag_slot[row]];
    sum = __dadd_rn(sum, __dmul_rn(__ldcg(x + row), d));  // remove the diagonal term of the loop
    x[row] = __ddiv_rn(sum, d);
}
#endif

// y = A x (sum += a*x, products and sums rounded separately).
int launch_nat_spmv(const NaturalLevel& L, const double* x, double* y, cudaStream_t s);
// One symmetric Gauss-Seidel step in natural order (forward then backward).
int launch_nat_symgs(const NaturalLevel& L, const double* r, double* x, cudaStream_t s);
// The same step as one dataflow kernel per direction (natural_flow.cu), the
// same bits for any matrix launch_nat_symgs takes, on levels of at most 256
// lines (nat_flow_ok).  workspace: nat_flow_workspace_bytes(rows) bytes of
// device memory, 16-byte aligned.  prepared: the workspace holds this matrix
// and this r from the previous call.  *status (device) is set to 1 when a
// bounded wait ran out; x is then undefined.
bool nat_flow_ok(int nx, int ny, int nz);
size_t nat_flow_workspace_bytes(long long rows);
int launch_nat_symgs_flow(const NaturalLevel& L, const double* r, double* x, void* workspace, bool prepared,
                          int* status, cudaStream_t s);
// rc[i] = rf[f2c[i]] - Axf[f2c[i]].
int launch_nat_restrict(int nc, const int* f2c, const double* rf, const double* axf, double* rc, cudaStream_t s);
// xf[f2c[i]] += xc[i].
int launch_nat_prolong(int nc, const int* f2c, const double* xc, double* xf, cudaStream_t s);
// w = alpha x + beta y with the three forms of src/ComputeWAXPBY_ref.cpp:65-85.
int launch_nat_waxpby(int n, double alpha, const double* x, double beta, const double* y, double* w, cudaStream_t s);
// *result = sum x_i*y_i (products rounded, then summed in a fixed order).
int launch_nat_dot(int n, const double* x, const double* y, ReduceScratch* ws, double* result, cudaStream_t s);

// CheckProblem (src/CheckProblem.cpp:79-150) as a count instead of asserts:
// every row's columns, values, nonzero count and diagonal slot against the
// 27-point stencil on the global grid; b = 26 - (nnz - 1), x = 0 and
// xexact = 1 where given; local-to-global ids where given.  Adds the number
// of mismatching rows to *bad and the row nonzeros to *nnz_total.
int launch_nat_check(const NaturalLevel& L, long long gnx, long long gny, long long gnz, long long gix0,
                     long long giy0, long long giz0, const long long* l2g, const double* b, const double* x,
                     const double* xexact, unsigned long long* bad, unsigned long long* nnz_total, cudaStream_t s);

}  // namespace hb
