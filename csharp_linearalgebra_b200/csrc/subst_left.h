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

// Whether the kernels take a solve: its order's products fit shared memory, and
// its right-hand sides, a CTA each, do not wait for one another so long that
// the staged kernels of lu.cu (a warp per two right-hand sides) end first.
bool left_solve_takes(const Context& ctx, bool cplx, int n, int nrhs);
// Real: U^T forward (explicit diagonal) when asked, then L^T backward (kUnit, or
// kDivide for an explicit diagonal, or kNone).
void left_solve_real(Context& ctx, bool forward, LowerKind backward, const LeftSolve& s);
// Complex: L^H backward, unit diagonal.
void left_solve_cplx(Context& ctx, const LeftSolve& s);

}  // namespace tns
