// Right-looking triangular solves with the right-hand sides in shared memory
// (subst_cols.cu), for lu.cu.
#pragma once

#include <vector>

#include "tns_internal.h"

namespace tns {

enum class LowerKind { kNone, kUnit, kDivide };

// One item: x (n x nrhs, ld ldx) := U^-1 L^-1 P x from the factors at f (ld
// ldf). perm: row i of P x is row perm[i] of x; null: no interchanges.
struct SubstCols {
    const double* f;
    int ldf;
    double* x;
    int ldx, n, nrhs;
    const int* perm;
};

// Largest order: one right-hand side's column fits a CTA's shared memory.
int subst_cols_max_order(bool cplx);
// Right-hand sides that a CTA takes (8, 4, 2 or 1) of one item of that order.
int subst_cols_per_cta(const Context& ctx, bool cplx, int n, long long nrhs);
// The lower solve (unit, or with an explicit diagonal, or none) and then the
// upper solve (when asked) of every item, in one launch.
void subst_cols(Context& ctx, bool cplx, LowerKind lower, bool upper, const std::vector<SubstCols>& items);

// One 32-row block of the blocked solves: rows and steps [k0, k0 + w) of the
// triangle at f, of every right-hand side of x (the whole matrices' origins).
constexpr int kDiagBlock = 32;
struct SubstDiagDesc {
    const double* f;
    int ldf;
    double* x;
    int ldx, nrhs;
    int k0, w;
};
// The blocks' own triangles in one launch, a thread per right-hand side.
void solve_diag_blocks(Context& ctx, bool cplx, LowerKind lower, bool upper, const std::vector<SubstDiagDesc>& v);

}  // namespace tns
