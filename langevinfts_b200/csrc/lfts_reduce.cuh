// Block sums in FP64: plain for FP64 data, compensated for FP32 data.
#pragma once
#include "lfts_step_kernels.cuh"

namespace lfts {

// warp + block sum of a double (block of NTHR threads); result valid in thread 0
__device__ __forceinline__ double block_sum(double v, double *sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) sh[w] = v;
    __syncthreads();
    v = 0;
    if (w == 0) {
        v = lane < NWARP ? sh[lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    return v;
}

// Compensated (error-free transform) summation for the FP32 propagator form:
// sums of FP32 products are accumulated in FP64 as a pair (s, c) where s is
// the running sum and c the running sum of the rounding errors of every
// addition (Knuth's two-sum; Neumaier's improvement of Kahan's method), and
// reduced across threads with the same transform.  The FP64 form keeps the
// plain FP64 sums.
__device__ __forceinline__ void comp_add(double &s, double &c, double x) {
    const double t = s + x;
    const double bp = t - s;
    c += (s - (t - bp)) + (x - bp);
    s = t;
}
// block sum of compensated pairs (block of NTHR threads, sh holds 2 * NWARP
// doubles); s + c of the block is valid in thread 0
__device__ __forceinline__ double block_sum_comp(double s, double c, double *sh) {
    for (int o = 16; o > 0; o >>= 1) {
        const double so = __shfl_down_sync(0xffffffffu, s, o), co = __shfl_down_sync(0xffffffffu, c, o);
        comp_add(s, c, so);
        c += co;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) { sh[w] = s; sh[NWARP + w] = c; }
    __syncthreads();
    s = 0.0;
    c = 0.0;
    if (w == 0) {
        s = lane < NWARP ? sh[lane] : 0.0;
        c = lane < NWARP ? sh[NWARP + lane] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            const double so = __shfl_down_sync(0xffffffffu, s, o), co = __shfl_down_sync(0xffffffffu, c, o);
            comp_add(s, c, so);
            c += co;
        }
    }
    return s + c;
}
template <typename T>
struct Acc {  // plain FP64 sum for T = double, compensated FP64 sum for T = float
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double x) {
        if (sizeof(T) == 4) comp_add(s, c, x);
        else s += x;
    }
    __device__ __forceinline__ double value() const { return s + c; }
    __device__ __forceinline__ double block(double *sh) const {
        return sizeof(T) == 4 ? block_sum_comp(s, c, sh) : block_sum(s, sh);
    }
};

}  // namespace lfts
