// What the exact steps of the uniform grid (rd_exact.cu) and of the block grid
// (amr.cu) share: the classes of cells (rd_exact.cu says why), the offsets of
// their list, the faces' diffusivities and the reaction. Both are compiled
// with -fmad=false.
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

// What is known of a density before a step (Handle::exact_full):
//   kAnyState  nothing: set by the caller, or of other tables
//   kInRange   a step over every cell gave it: it is in [0, 1]
//   kDeadZero  and its dead cells are 0
//   kListed    and the other buffer is 0 where no listed cell is
enum { kAnyState = 0, kInRange = 1, kDeadZero = 2, kListed = 3 };
// The state after a step over every cell. From a density in [0, 1] the step
// leaves dead cells 0. From any finite one it does so too, but for p < 0 where
// cell and density together are no tissue: the faces count as 0 and p + dt rho p
// (1 - p) may be positive, if rho and dt are of unlike sign.
inline int after_full_step(int state, double rho, double dt) {
    return state == kAnyState && (rho < 0.0) != (dt < 0.0) ? kInRange : kDeadZero;
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

// The reciprocal conductivity of a cell and the diffusivity of the face between
// two, without the divisions (a dozen and more FP64 operations each) where the
// result is NaN: toward and between cells without tissue, two thirds of a grid.
__device__ __forceinline__ double as_nan() { return __hiloint2double(0x7ff80000, 0); }
template <typename Real>
__device__ __forceinline__ double inverse_k(Real a, Real b, Real Dw, Real Dg) {
    if (a == (Real)0 && b == (Real)0) return as_nan();
    const Real kk = (a * Dw + b * Dg) / (a + b);
    return 1.0 / (double)kk;
}
__device__ __forceinline__ double face_k(double inv0, double inv1) {
    const double s = inv0 + inv1;
    if (((unsigned)__double2hiint(s) & 0x7fffffffu) > 0x7ff00000u) return as_nan();
    return 2.0 * (1.0 / s);
}

__device__ __forceinline__ double reaction(double rho, double p) { return rho * p * (1. - p); }
__device__ __forceinline__ double reaction(float rho, float p) {
    const float rp = rho * p;
    return (double)rp * (1. - (double)p);
}

}  // namespace
}  // namespace gbg
