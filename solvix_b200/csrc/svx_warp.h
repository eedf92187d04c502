// svx_warp.h - warp sums on the FP64 tensor cores (device code of the
// chip-resident solvers).
#ifndef SVX_WARP_H
#define SVX_WARP_H
#ifdef __CUDACC__

namespace svx {

// D = A B with 8 x 4 by 4 x 8 FP64 operands: the lane's A element is (lane /
// 4, lane % 4), its B element (lane % 4, lane / 4), its two D elements
// (lane / 4, 2 (lane % 4) + {0, 1}).
__device__ __forceinline__ void mma(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%4,%4};"
                 : "=d"(d0), "=d"(d1) : "d"(a), "d"(b), "d"(0.0));
}
// Sum over the warp, the same bits in every lane (74 cycles against 187 by
// shuffles): ones x V gives the lane the sums of two quads of lanes, which
// add up to a quarter of the total per lane % 4; quarters x ones gives the
// total.
__device__ __forceinline__ double quarter_sum(double v) {
    double a, b;
    mma(a, b, 1.0, v);
    return a + b;
}
__device__ __forceinline__ double lane_sum(double v) {
    double a, b;
    mma(a, b, quarter_sum(v), 1.0);
    return a;
}
// Two sums at once: lanes 0-15 get x's, lanes 16-31 get y's.
__device__ __forceinline__ double lane_sum_pair(double x, double y, int lane) {
    const double qx = quarter_sum(x), qy = quarter_sum(y);
    double a, b;
    mma(a, b, lane < 16 ? qx : qy, 1.0);
    return a;
}

}  // namespace svx

#endif  // __CUDACC__
#endif  // SVX_WARP_H
