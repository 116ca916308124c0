// Left-looking triangular solves (the transposed and adjoint ones, whose
// reference order is an inner product per row) with a chain warp and producer
// warps per right-hand side (subst_left.cu), for lu.cu.
#pragma once

#include "subst_cols.h"
#include "tns_internal.h"

namespace tns {

// x (n x nrhs, ld ldx) solved in place; perm: row i of the solution goes to row
// perm[i] (the interchanges undone); null: to row i.
struct LeftSolve {
    const double* f;
    int ldf;
    double* x;
    int ldx, n, nrhs;
    const int* perm;
};

// lu.cu's staged kernels, a warp per two right-hand sides with the factor's
// columns in a ring of kStageSlots: the orders that fit their shared memory.
constexpr int kStageSlots = 6;
constexpr int kStagedRealMaxN = 3200;  // 6 slots + 2 columns of doubles: 200 KB
constexpr int kStagedCplxMaxN = 1280;  // 6 slots + 2 columns + 2 product rows of complex: 200 KB
inline size_t staged_left_smem(bool cplx, int n) { return (size_t)(cplx ? 16 * (kStageSlots + 4) : 8 * (kStageSlots + 2)) * n; }

// Whether the kernels take a solve: its order's products fit shared memory, and
// its right-hand sides, a CTA each, do not wait for one another so long that
// the kernels of lu.cu end first.
bool left_solve_takes(const Context& ctx, bool cplx, int n, int nrhs);
// Real: U^T forward (explicit diagonal) when asked, then L^T backward (kUnit, or
// kDivide for an explicit diagonal, or kNone).
void left_solve_real(Context& ctx, bool forward, LowerKind backward, const LeftSolve& s);
// Complex: L^H backward, unit diagonal.
void left_solve_cplx(Context& ctx, const LeftSolve& s);

}  // namespace tns
