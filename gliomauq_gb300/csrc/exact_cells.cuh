// What the exact steps of the uniform grid (rd_exact.cu) and of the block grid
// (amr.cu) share: the classes of cells (rd_exact.cu says why), the offsets of
// their list, and the widening of a float. Both are compiled with
// -fmad=false.
#pragma once

namespace gbg {
namespace {

enum { kDead = 0, kPlain = 1, kSpecial = 2 };

__device__ __forceinline__ int cell_class(double b0, const double (&d)[6]) {
    bool nan = false, pos = b0 > 0.0;
    for (int f = 0; f < 6; ++f) {
        nan = nan || isnan(d[f]);
        pos = pos && d[f] > 0.0 && !isinf(d[f]);
    }
    return nan && b0 >= 0.0 ? kDead : (pos ? kPlain : kSpecial);
}

// counts -> exclusive offsets, the total behind them (one CTA)
__global__ void __launch_bounds__(1024) k_exact_offsets(int chunks, int *__restrict__ offset) {
    __shared__ int sums[32];
    __shared__ int total;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    for (int base = 0; base < chunks; base += 1024) {
        const int i = base + threadIdx.x;
        const int own = i < chunks ? offset[i] : 0;
        int v = own;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) sums[warp] = v;
        __syncthreads();
        int before = total;
        for (int k = 0; k < warp; ++k) before += sums[k];
        if (i < chunks) offset[i] = before + v - own;
        __syncthreads();
        if (threadIdx.x == 1023) total = before + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) offset[chunks] = total;
}

// a float widened with integer operations where it is a normal number (the
// conversion unit is as narrow as the FP64 pipe); a zero loses its sign
__device__ __forceinline__ double widen(double p) { return p; }
__device__ __forceinline__ double widen(float p) {
    const unsigned u = __float_as_uint(p), m = u & 0x7fffffffu;
    if (m - 0x00800000u < 0x7f000000u)
        return __hiloint2double((int)((u & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(u << 29));
    return m ? (double)p : 0.0;
}

}  // namespace
}  // namespace gbg
