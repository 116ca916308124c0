// The LU panel factorization with a panel's rows held in registers
// (lu_panel.cu), for lu.cu.
#pragma once

#include <vector>

#include "tns_internal.h"

namespace tns {

// Panel rows [r0, m) x columns [r0, r0 + w) of a (ld elements), factored in
// place with partial pivoting; pivots land as global 0-based rows in
// piv[r0 + j], the first exactly zero pivot's column in *singular (minimum).
struct PanelFactorDesc {
    double* a;
    int ld, m, r0, w;
    int* piv;
    int* singular;
};

// Columns one launch of the register kernel factors.
constexpr int kRowPanelWidth = 32;
// Largest panel height it takes: a cluster of eight CTAs, one row per thread.
int row_panel_max_rows(bool cplx);
// One launch for a batch of panels of at most kRowPanelWidth columns and
// row_panel_max_rows() rows.
void launch_row_panels(Context& ctx, bool cplx, const std::vector<PanelFactorDesc>& v);

}  // namespace tns
