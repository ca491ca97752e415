// Device helpers of the cell expansions (csrc/fs_cells.cu, csrc/fs_treecells.cu).
#pragma once

#include "fs_device.cuh"

namespace fsb {

// Position in [0, L] (NaN stays NaN), its cell and its place in the cell.
__device__ __forceinline__ double cell_wrap(double x, double L) {
    const double w = x - L * floor(x / L);
    return w < 0.0 ? 0.0 : (w > L ? L : w);
}
__device__ __forceinline__ int cell_of(double w, const CellPlan& P) {
    return min(max((int)(w * P.inv_h), 0), P.M - 1);
}

// sum_l a[l] T_l(x) by Clenshaw's recurrence; a is 16-byte aligned.
__device__ __forceinline__ double cheb_sum(const double* __restrict__ a, double x) {
    const double2* a2 = reinterpret_cast<const double2*>(a);
    double b1 = 0.0, b2 = 0.0;
    const double x2 = x + x;
#pragma unroll
    for (int h = kCellTerms / 2 - 1; h > 0; --h) {
        const double2 c = __ldg(a2 + h);
        const double u = fma(x2, b1, c.y - b2);
        b2 = fma(x2, u, c.x - b1);
        b1 = b2;
        b2 = u;
    }
    const double2 c = __ldg(a2);
    const double u = fma(x2, b1, c.y - b2);
    return fma(x, u, c.x - b1);
}

}  // namespace fsb
