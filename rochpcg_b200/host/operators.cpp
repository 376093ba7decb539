// The reference's operator API on B200 kernels.  Each function keeps the
// signature and semantics of its rocHPCG counterpart (cited per function)
// and launches on the runtime stream; scalar-returning ones block for the
// result exactly like the reference (which syncs after every dot product).
#include <cstdlib>

#include "hpcg_b200.h"
#include "internal.hpp"

using namespace hpcg_b200;

namespace {

double read_scalar(int slot)
{
    Runtime& R = rt();
    HB_HOST_CUDA(cudaMemcpyAsync(R.h_scalar + slot, R.d_scalar + slot, sizeof(double), cudaMemcpyDeviceToHost,
                                 R.stream));
    HB_HOST_CUDA(cudaStreamSynchronize(R.stream));
    return R.h_scalar[slot];
}

}  // namespace

// src/ComputeSPMV.cpp:226-278.  (The reference computes only the rows the
// restriction needs when y is mgData->Axf; the full product is a superset.)
int ComputeSPMV(const SparseMatrix& A, Vector& x, Vector& y)
{
    return guarded([&] {
        ExchangeHalo(A, x);
        if(A.mgData && &y == A.mgData->Axf && !y.d_values) CudaInitializeVector(y, A.localNumberOfColumns);
        const LevelOpt* o = opt(A);
        return hb::launch_spmv(A.localNumberOfRows, o ? o->cc : hb::make_chunks(A.localNumberOfRows, 0, nullptr),
                               A.ell_col_ind, A.ell_val, x.d_values, y.d_values, rt().stream);
    });
}

namespace {

// The level runs its SymGS as one cluster kernel (small_level.cu): with T's
// arithmetic, ell: on the ELL values.
template <typename T>
bool small_level(const SparseMatrix& A, bool ell)
{
    const LevelOpt* o = opt(A);
    return o && o->stencil_ok && hb::small_level_ok<T>(o->st, ell);
}

hb::SmallEll small_ell(const SparseMatrix& A)
{
    const MGOpt* mo = mgopt(A);
    return hb::SmallEll{A.ell_col_ind, A.ell_val, A.diag_idx, mo ? mo->inj_f : nullptr,
                        mo ? A.Ac->localNumberOfRows : 0, opt(A)->ell_changed};
}

// A small level's zero-guess step (ell: on the ELL arrays) and, where rc is
// given, the restriction of its residual to rc, in one kernel.
int small_zero_restrict(const SparseMatrix& A, const double* r, double* x, bool ell, double* rc, cudaStream_t s,
                        hb::Prolong<double> pro = {})
{
    const LevelOpt* o = opt(A);
    const hb::SmallEll e = small_ell(A);
    return hb::launch_small_zero<double>(o->st, o->diag, A.inv_diag, nullptr, const_cast<double*>(r), x, ell ? &e : nullptr,
                                         rc ? mgopt(A)->inj_c : nullptr, rc, s, pro);
}

int small_zero_restrict(const SparseMatrix& A, const double* r64, float* r, float* x, cudaStream_t s,
                        hb::Prolong<float> pro = {})
{
    const LevelOpt* o = opt(A);
    const MGOpt* mo = mgopt(A);
    return hb::launch_small_zero<float>(o->st, o->diag32, o->inv_diag32, r64, r, x, nullptr, mo ? mo->inj_c : nullptr,
                                        mo ? mo->rc32 : nullptr, s, pro);
}

// One full / zero-guess SymGS step on the ELL matrix.
int symgs_ell(const SparseMatrix& A, const double* r, double* x, cudaStream_t s, hb::Prolong<double> pro = {})
{
    if(small_level<double>(A, true))
    {
        const hb::SmallEll e = small_ell(A);
        return hb::launch_small_symgs<double>(opt(A)->st, A.inv_diag, r, x, nullptr, &e, s, pro);
    }
    return hb::launch_symgs(A.localNumberOfRows, A.nblocks, A.ublocks, A.sizes, A.offsets, A.ell_col_ind, A.ell_val,
                            A.inv_diag, r, x, s, pro);
}

int symgs_zero_ell(const SparseMatrix& A, const double* r, double* x, cudaStream_t s, hb::Prolong<double> pro = {})
{
    const LevelOpt* o = opt(A);
    if(small_level<double>(A, true)) return small_zero_restrict(A, r, x, true, nullptr, s, pro);
    return hb::launch_symgs_zero(A.localNumberOfRows, A.nblocks, A.ublocks, A.sizes, A.offsets, A.ell_col_ind,
                                 A.ell_val, A.diag_idx, o->diag, A.inv_diag, r, x, s, pro, zg_of(A));
}

}  // namespace

// src/ComputeSYMGS.cpp:369-404.
int ComputeSYMGS(const SparseMatrix& A, const Vector& r, Vector& x)
{
    return guarded([&] {
        ExchangeHalo(A, x);
        return symgs_ell(A, r.d_values, x.d_values, rt().stream);
    });
}

// src/ComputeSYMGS.cpp:406-454.
int ComputeSYMGSZeroGuess(const SparseMatrix& A, const Vector& r, Vector& x)
{
    return guarded([&] { return symgs_zero_ell(A, r.d_values, x.d_values, rt().stream); });
}

// src/ComputeRestriction.cpp:199-237.
int ComputeFusedSpMVRestriction(const SparseMatrix& A, const Vector& rf, Vector& xf)
{
    return guarded([&] {
        ExchangeHalo(A, xf);
        const MGOpt* mo = mgopt(A);
        return hb::launch_restrict(A.mgData->rc->localLength, mo->inj_f, mo->inj_c, A.localNumberOfRows,
                                   A.ell_col_ind, A.ell_val, rf.d_values, xf.d_values, A.mgData->rc->d_values,
                                   rt().stream);
    });
}

// src/ComputeRestriction.cpp:182-197 (uses mgData->Axf = A xf from ComputeSPMV).
int ComputeRestriction(const SparseMatrix& A, const Vector& rf)
{
    return guarded([&] {
        const MGOpt* mo = mgopt(A);
        if(!A.mgData->Axf->d_values) return hb::record_error(HPCGB200_ERR_ARG, "ComputeRestriction: Axf not computed");
        return hb::launch_restrict_axf(A.mgData->rc->localLength, mo->inj_f, mo->inj_c, rf.d_values,
                                       A.mgData->Axf->d_values, A.mgData->rc->d_values, rt().stream);
    });
}

// src/ComputeProlongation.cpp:72-86.
int ComputeProlongation(const SparseMatrix& Af, Vector& xf)
{
    return guarded([&] {
        const MGOpt* mo = mgopt(Af);
        return hb::launch_prolong(Af.mgData->rc->localLength, mo->inj_f, mo->inj_c, Af.mgData->xc->d_values,
                                  xf.d_values, rt().stream);
    });
}

namespace hpcg_b200 {

bool fused_prolongation()
{
    static const bool on = [] {
        const char* e = std::getenv("HPCGB200_FUSED_PROLONG");
        return e && e[0] == '1';
    }();
    return on;
}

}  // namespace hpcg_b200

namespace {

// ComputeMG's recursion with the prolongation fused into the coarse level:
// `pro` (the finer level's x and the row map) rides on this level's last
// smoother passes -- the post-smoother's last step, or the zero-guess step of
// the coarsest level -- instead of a ComputeProlongation launch after it.
int mg64_ell(const SparseMatrix& A, const Vector& r, Vector& x, hb::Prolong<double> pro)
{
    cudaStream_t s = rt().stream;
    auto zero_guess = [&](hb::Prolong<double> p) { return symgs_zero_ell(A, r.d_values, x.d_values, s, p); };
    auto full = [&](hb::Prolong<double> p) {
        ExchangeHalo(A, x);
        return symgs_ell(A, r.d_values, x.d_values, s, p);
    };
    if(!A.mgData) return zero_guess(pro);
    const int pre = A.mgData->numberOfPresmootherSteps, post = A.mgData->numberOfPostsmootherSteps;
    if(pre == 1 && post > 0 && small_level<double>(A, true))
        HB_RETURN_IF(small_zero_restrict(A, r.d_values, x.d_values, true, A.mgData->rc->d_values, s));
    else
    {
        HB_RETURN_IF(zero_guess(post == 0 ? pro : hb::Prolong<double>{}));
        for(int i = 1; i < pre; ++i) HB_RETURN_IF(full({}));
        HB_RETURN_IF(ComputeFusedSpMVRestriction(A, r, x));
    }
    // src/ComputeMG.cpp:86-90: coarse solve, then ComputeProlongation -- here
    // carried out by the coarse level's final passes
    if(fused_prolongation())
        HB_RETURN_IF(mg64_ell(*A.Ac, *A.mgData->rc, *A.mgData->xc, hb::Prolong<double>{x.d_values, mgopt(A)->pro_f}));
    else
    {
        HB_RETURN_IF(mg64_ell(*A.Ac, *A.mgData->rc, *A.mgData->xc, {}));
        HB_RETURN_IF(ComputeProlongation(A, x));
    }
    for(int i = 0; i < post; ++i) HB_RETURN_IF(full(i == post - 1 ? pro : hb::Prolong<double>{}));
    return 0;
}

}  // namespace

// src/ComputeMG.cpp:64-102.
int ComputeMG(const SparseMatrix& A, const Vector& r, Vector& x)
{
    return guarded([&] { return mg64_ell(A, r, x, {}); });
}

namespace hpcg_b200 {

// FP32 V-cycle on level data, same recursion as ComputeMG (the prolongation
// into the finer level fused into this level's final passes).
int mg_fp32(const SparseMatrix& A, const float* r, float* x, cudaStream_t s, hb::Prolong<float> pro)
{
    const LevelOpt* o = opt(A);
    if(!A.mgData)
        return hb::launch32_symgs_zero(o->st, o->diag32, o->inv_diag32, nullptr, const_cast<float*>(r), x, s, pro);
    const MGOpt* mo = mgopt(A);
    const int nc = A.Ac->localNumberOfRows;
    if(small_level<float>(A, false)) HB_RETURN_IF(small_zero_restrict(A, nullptr, const_cast<float*>(r), x, s));
    else
    {
        HB_RETURN_IF(hb::launch32_symgs_zero(o->st, o->diag32, o->inv_diag32, nullptr, const_cast<float*>(r), x, s));
        HB_RETURN_IF(hb::launch32_restrict(o->st, nc, mo->inj_f, mo->inj_c, o->diag32, r, x, mo->rc32, s));
    }
    if(fused_prolongation()) HB_RETURN_IF(mg_fp32(*A.Ac, mo->rc32, mo->xc32, s, hb::Prolong<float>{x, mo->pro_f}));
    else
    {
        HB_RETURN_IF(mg_fp32(*A.Ac, mo->rc32, mo->xc32, s));
        HB_RETURN_IF(hb::launch32_prolong(o->st, nc, mo->inj_f, mo->inj_c, mo->xc32, x, s));
    }
    return hb::launch32_symgs(o->st, o->inv_diag32, r, x, nullptr, s, pro);
}

}  // namespace hpcg_b200

namespace hpcg_b200 {

// FP32 V-cycle preconditioner for FP64 vectors: the level-0 zero-guess sweep
// reads r in FP64 (storing its float copy); the result stays in the level's
// z32, and its post-smoother also writes the FP64 copy z64 when one is asked
// for (the CG iteration reads z32 itself).
int mg_mixed_to(const SparseMatrix& A, const double* r64, double* z64, cudaStream_t s)
{
    const LevelOpt* o = opt(A);
    for(const SparseMatrix* M = &A; M; M = M->Ac)
        if(!opt(*M) || !opt(*M)->stencil_ok)
            return hb::record_error(HPCGB200_ERR_NOT_STENCIL,
                                    "mixed V-cycle needs the 27-point stencil in parity colouring on every level");
    const int m = A.localNumberOfRows;
    const bool small = small_level<float>(A, false);
    if(small) HB_RETURN_IF(small_zero_restrict(A, r64, o->r32, o->z32, s));
    else HB_RETURN_IF(hb::launch32_symgs_zero(o->st, o->diag32, o->inv_diag32, r64, o->r32, o->z32, s));
    if(!A.mgData) return z64 ? hb::launch_cast_f2d(m, o->z32, z64, s) : 0;
    const MGOpt* mo = mgopt(A);
    const int nc = A.Ac->localNumberOfRows;
    if(!small)
        HB_RETURN_IF(hb::launch32_restrict(o->st, nc, mo->inj_f, mo->inj_c, o->diag32, o->r32, o->z32, mo->rc32, s));
    if(fused_prolongation()) HB_RETURN_IF(mg_fp32(*A.Ac, mo->rc32, mo->xc32, s, hb::Prolong<float>{o->z32, mo->pro_f}));
    else
    {
        HB_RETURN_IF(mg_fp32(*A.Ac, mo->rc32, mo->xc32, s));
        HB_RETURN_IF(hb::launch32_prolong(o->st, nc, mo->inj_f, mo->inj_c, mo->xc32, o->z32, s));
    }
    return hb::launch32_symgs(o->st, o->inv_diag32, o->r32, o->z32, z64, s);
}

}  // namespace hpcg_b200

int ComputeMG_Mixed(const SparseMatrix& A, const Vector& r, Vector& x)
{
    return guarded([&] { return mg_mixed_to(A, r.d_values, x.d_values, rt().stream); });
}

namespace {

bool stencil_vec_level(const SparseMatrix& A)
{
    const LevelOpt* o = opt(A);
    return o && o->stencil_ok && hb::stencil_vec4(o->st);
}

// ComputeMG's recursion (1 zero-guess pre-smoothing step, fused restriction,
// coarse solve, prolongation, 1 post-smoothing step) per level on the
// implicit-stencil kernels or, where the level is not the verified stencil
// or has too many planes for the one-row ones, the ELL ones.
int mg64_stencil(const SparseMatrix& A, const double* r, double* x, cudaStream_t s, hb::Prolong<double> pro)
{
    const LevelOpt* o = opt(A);
    const bool vec = stencil_vec_level(A), small = small_level<double>(A, false);
    // the one-row kernels have a colour's planes on their grid's z axis
    const bool stencil = vec || (o && o->stencil_ok && o->st.nz <= 2 * 65535);
    // the coarsest level's zero-guess step is its last: it carries `pro`
    const hb::Prolong<double> pz = A.mgData ? hb::Prolong<double>{} : pro;
    if(small)
        HB_RETURN_IF(small_zero_restrict(A, r, x, false, A.mgData ? A.mgData->rc->d_values : nullptr, s, pz));
    else if(stencil) HB_RETURN_IF(hb::launch64v_symgs_zero(o->st, o->diag, A.inv_diag, r, x, s, pz));
    else HB_RETURN_IF(symgs_zero_ell(A, r, x, s, pz));
    if(!A.mgData) return 0;
    const MGOpt* mo = mgopt(A);
    const int nc = A.Ac->localNumberOfRows;
    double* rc = A.mgData->rc->d_values;
    double* xc = A.mgData->xc->d_values;
    if(!small && stencil)
        HB_RETURN_IF(hb::launch64v_restrict(o->st, nc, mo->inj_f, mo->inj_c, o->diag, r, x, rc, s));
    else if(!small)
        HB_RETURN_IF(hb::launch_restrict(nc, mo->inj_f, mo->inj_c, A.localNumberOfRows, A.ell_col_ind, A.ell_val, r, x,
                                         rc, s));
    // coarse solve with the prolongation into x fused into its final passes
    if(fused_prolongation()) HB_RETURN_IF(mg64_stencil(*A.Ac, rc, xc, s, hb::Prolong<double>{x, mo->pro_f}));
    else
    {
        HB_RETURN_IF(mg64_stencil(*A.Ac, rc, xc, s, {}));
        if(vec) HB_RETURN_IF(hb::launch64v_prolong(o->st, nc, mo->inj_c, xc, x, s));
        else HB_RETURN_IF(hb::launch_prolong(nc, mo->inj_f, mo->inj_c, xc, x, s));
    }
    if(small) return hb::launch_small_symgs<double>(o->st, A.inv_diag, r, x, nullptr, nullptr, s, pro);
    if(stencil) return hb::launch64v_symgs(o->st, A.inv_diag, r, x, s, pro);
    return symgs_ell(A, r, x, s, pro);
}

}  // namespace

int ComputeMG_Stencil(const SparseMatrix& A, const Vector& r, Vector& x)
{
    return guarded([&] {
        for(const SparseMatrix* M = &A; M; M = M->Ac)
            if(M->mgData && (M->mgData->numberOfPresmootherSteps != 1 || M->mgData->numberOfPostsmootherSteps != 1))
                return hb::record_error(HPCGB200_ERR_ARG, "stencil V-cycle: 1 pre- and 1 post-smoothing step only");
        return mg64_stencil(A, r.d_values, x.d_values, rt().stream, {});
    });
}

// src/ComputeDotProduct.cpp:189-238 (blocking, like the reference).
int ComputeDotProduct(local_int_t n, const Vector& x, const Vector& y, double& result, double& time_allreduce,
                      bool& isOptimized)
{
    (void)time_allreduce;  // one rank: no allreduce
    (void)isOptimized;
    return guarded([&] {
        HB_RETURN_IF(hb::launch_dot(n, x.d_values, y.d_values, rt().ws, rt().d_scalar, rt().stream));
        result = read_scalar(0);
        return 0;
    });
}

// src/ComputeWAXPBY.cpp:111-135.
int ComputeWAXPBY(local_int_t n, double alpha, const Vector& x, double beta, const Vector& y, Vector& w,
                  bool& isOptimized)
{
    (void)isOptimized;
    return guarded([&] {
        if(n == 0) return 0;
        return hb::launch_waxpby(n, alpha, x.d_values, beta, y.d_values, w.d_values, rt().stream);
    });
}

// src/ComputeWAXPBY.cpp:198-240.
int ComputeFusedWAXPBYDot(local_int_t n, double alpha, const Vector& x, Vector& y, double& result,
                          double& time_allreduce)
{
    (void)time_allreduce;
    return guarded([&] {
        HB_RETURN_IF(hb::launch_waxpby_dot(n, alpha, x.d_values, y.d_values, rt().ws, rt().d_scalar, rt().stream));
        result = read_scalar(0);
        return 0;
    });
}

// src/ComputeResidual.cpp:121-152.
int ComputeResidual(local_int_t n, const Vector& v1, const Vector& v2, double& residual)
{
    return guarded([&] {
        HB_RETURN_IF(hb::launch_residual_inf(n, v1.d_values, v2.d_values, rt().ws, rt().d_scalar, rt().stream));
        residual = read_scalar(0);
        return 0;
    });
}
