// The LU panel factorization with a panel's rows held in registers
// (lu_panel.cu), for lu.cu.
#pragma once

#include <vector>

#include "tns_internal.h"

namespace tns {

// Panel rows [r0, m) x columns [r0, r0 + w) of a (ld elements), factored in
// place with partial pivoting; pivots land as global 0-based rows in
// piv[r0 + j], the first exactly zero pivot's column in *singular (minimum).
// carry: the columns just left of the panel whose rows change places with the
// panel's (at most kRowPanelWidth; the register kernel only).
struct PanelFactorDesc {
    double* a;
    int ld, m, r0, w;
    int* piv;
    int* singular;
    int carry;
};

// Columns one launch of the register kernel factors.
constexpr int kRowPanelWidth = 32;
// Largest panel height it takes: a cluster of eight CTAs, one row per thread.
int row_panel_max_rows(bool cplx);
// One launch for a batch of panels of at most kRowPanelWidth columns and
// row_panel_max_rows() rows.
void launch_row_panels(Context& ctx, bool cplx, const std::vector<PanelFactorDesc>& v);

// A factored panel's effect on the columns [c0, c1) of its rows: the row
// interchanges k <-> piv[k], k = k0 .. k0 + w - 1 in turn (swap), and then rows
// k0 .. k0 + w - 1 := L11^-1 (those rows) with the unit lower L11 at (k0, k0)
// (solve), in the reference's order. a: the matrix's origin.
struct PanelRowsDesc {
    double* a;
    int ld, c0, c1;
    const int* piv;
    int k0, w;  // w <= kPanelRowsMaxWidth
    int swap, solve;
    int tile_begin;
};
constexpr int kPanelRowsMaxWidth = 64;
void launch_panel_rows(Context& ctx, bool cplx, std::vector<PanelRowsDesc>& v);

}  // namespace tns
