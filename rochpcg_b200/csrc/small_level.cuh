// SymGS steps of a small multigrid level as one cluster kernel (see
// small_level.cu): the colour passes of launch32_symgs_zero / launch32_symgs
// (FP32), launch64v_* (FP64 on the implicit stencil) and launch_symgs_zero /
// launch_symgs (FP64 ELL values), bit for bit.
#pragma once

#include "mixed.cuh"
#include "ops64.cuh"

namespace hb {

// The level is small enough, canonically coloured and fits the cluster's
// shared memory.  T: float, or double (ell: with the ELL values).
template <typename T>
bool small_level_ok(const StencilLevel& L, bool ell);

// The ELL arrays of a level (launch_symgs, launch_symgs_zero, launch_restrict):
// the step is the one on their present contents, whatever was changed in them
// since set-up.
struct SmallEll
{
    const int* col;
    const double* val;
    const int* diag_idx;
    const int* inj_f;  // with nc: the restriction's
    int nc;
    int* changed;      // device word, 0 between steps
};

// One zero-guess step: x from r; r64 (float only, may be null): r comes in
// FP64 and its float copy is stored in r.  ell (double only): the level's ELL
// arrays; null: the verified stencil.  rc (may be null): also the residual
// at the injected rows, rc[inj_c[i]] for row i of the parity-0 colour.
template <typename T>
int launch_small_zero(const StencilLevel& L, const T* diag, const T* inv_diag, const double* r64, T* r, T* x,
                      const SmallEll* ell, const int* inj_c, T* rc, cudaStream_t s, Prolong<T> pro);
// One full step on x.  z64 (float only, may be null): also the FP64 copy.
template <typename T>
int launch_small_symgs(const StencilLevel& L, const T* inv_diag, const T* r, T* x, double* z64,
                       const SmallEll* ell, cudaStream_t s, Prolong<T> pro);

}  // namespace hb
