// Bit-faithful step kernels: the reference's operator arithmetic, rounded
// operation by operation as its source writes it.
//
// This translation unit is compiled with -fmad=false so that no a*b+c is
// contracted into a fused multiply-add: every + and * here rounds on its own,
// as it does in the reference (compiled without contraction). Division and
// the float<->double conversions are IEEE round-to-nearest.
//
// Real = double  : the reference built with -D_MRAG_REAL_=double
// Real = float   : the reference's default build, where the lab fields, Dw,
//                  Dg, rho and the brain sums are float and df[], the fluxes
//                  and the update are double
//                  (source/Glioma/Glioma_ReactionDiffusionOperator.h:40-42,155,174-216,258).
#include <algorithm>

#include "exact_cells.cuh"
#include "gbg_internal.cuh"

#include "arrivals.cuh"

namespace gbg {
namespace {

__device__ __forceinline__ int wrapm(int i, int n) { return i == 0 ? n - 1 : i - 1; }
__device__ __forceinline__ int wrapp(int i, int n) { return i == n - 1 ? 0 : i + 1; }

// Per-cell brain sum and the three "+" face diffusivities of the Case2 branch
// (Glioma_ReactionDiffusionOperator.h:174-188):
//   k_c  = (p_w Dw + p_g Dg) / (p_w + p_g)            in Real
//   df   = 2.0 * (1.0 / ((1.0/k_c) + (1.0/k_n)))      in double
// A face to a cell with p_w + p_g == 0 gives k_n = 0/0 = NaN, hence df = NaN:
// the reference's boundary-layer behaviour, reproduced as is. The face shared
// by cells c and c+e is the same value from either side (IEEE + commutes).
template <typename Real>
__global__ void k_build_tables(int n, const double *__restrict__ pw, const double *__restrict__ pg,
                               Real Dw, Real Dg, Real *__restrict__ b0, double *__restrict__ dfx,
                               double *__restrict__ dfy, double *__restrict__ dfz) {
    const size_t N = (size_t)n * n * n;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < N;
         c += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(c % n), y = (int)((c / n) % n), z = (int)(c / ((size_t)n * n));
        const size_t nb[4] = {c, (size_t)wrapp(x, n) + (size_t)n * (y + (size_t)n * z),
                              (size_t)x + (size_t)n * (wrapp(y, n) + (size_t)n * z),
                              (size_t)x + (size_t)n * (y + (size_t)n * wrapp(z, n))};
        double inv[4];
        Real bc = 0;
        for (int k = 0; k < 4; ++k) {
            const Real a = (Real)pw[nb[k]], b = (Real)pg[nb[k]];
            inv[k] = inverse_k(a, b, Dw, Dg);
            if (k == 0) bc = a + b;
        }
        b0[c] = bc;
        dfx[c] = face_k(inv[0], inv[1]);
        dfy[c] = face_k(inv[0], inv[2]);
        dfz[c] = face_k(inv[0], inv[3]);
    }
}

// rho * phi * (1. - phi): (rho*phi) in Real, times (1.0 - phi) in double.
// One step: RHS of Glioma_ReactionDiffusionOperator<3> (:148-218), the dphidt
// rounding to Real, and UpdateTumor<3> (:254-261) with std::max / std::min
// clamping (NaN -> 0).
template <typename Real>
__global__ void k_exact_step(int n, const Real *__restrict__ phi, Real *__restrict__ out,
                             const Real *__restrict__ b0, const double *__restrict__ dfx,
                             const double *__restrict__ dfy, const double *__restrict__ dfz,
                             Real rho, double dt, double ih2) {
    const size_t N = (size_t)n * n * n;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < N;
         c += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(c % n), y = (int)((c / n) % n), z = (int)(c / ((size_t)n * n));
        const size_t nn = (size_t)n, plane = nn * nn;
        const size_t cW = c - x + wrapm(x, n), cE = c - x + wrapp(x, n);
        const size_t cS = c + ((size_t)wrapm(y, n) - y) * nn, cN = c + ((size_t)wrapp(y, n) - y) * nn;
        const size_t cB = c + ((size_t)wrapm(z, n) - z) * plane, cF = c + ((size_t)wrapp(z, n) - z) * plane;
        const Real p0 = phi[c];
        const Real pW = phi[cW], pE = phi[cE], pS = phi[cS], pN = phi[cN], pB = phi[cB], pF = phi[cF];
        double df0 = 0.0, df1 = 0.0, df2 = 0.0, df3 = 0.0, df4 = 0.0, df5 = 0.0;
        const Real tissue = b0[c] + p0;
        if (tissue > 0.) {
            df0 = dfx[cW]; df1 = dfx[c];
            df2 = dfy[cS]; df3 = dfy[c];
            df4 = dfz[cB]; df5 = dfz[c];
        }
        // :198-203, in order
        if (df0 == 0 && pW > 0.) df1 *= 2.0;
        if (df1 == 0 && pE > 0.) df0 *= 2.0;
        if (df2 == 0 && pS > 0.) df3 *= 2.0;
        if (df3 == 0 && pN > 0.) df2 *= 2.0;
        if (df4 == 0 && pB > 0.) df5 *= 2.0;
        if (df5 == 0 && pF > 0.) df4 *= 2.0;
        const double fin = ih2 * (df0 * (double)pW + df1 * (double)pE + df2 * (double)pS +
                                  df3 * (double)pN + df4 * (double)pB + df5 * (double)pF);
        const double fout = -((df0 + df1 + df2 + df3 + df4 + df5) * (double)p0 * ih2);
        const double react = reaction(rho, p0);
        const Real dphidt = (Real)(fout + fin + react);
        Real v = (Real)((double)p0 + dt * (double)dphidt);
        v = ((Real)0 < v) ? v : (Real)0;
        v = (v < (Real)1) ? v : (Real)1;
        out[c] = v;
    }
}

// ---- the cells a step has to compute -----------------------------------------
// The FP64 pipe (2 lanes per clock and SM) bounds the exact step: 26 operations
// of a cell, and twelve FP64 comparisons for the doubling. Most cells need none:
//   dead     b0 >= 0 with a NaN among the six faces. If the cell is tissue, or
//            holds a positive density, the NaN reaches v and the clamp gives 0;
//            otherwise its faces count as 0 and so does its density: 0 again.
//   plain    b0 > 0 and all six faces positive: no doubling, and the sum of the
//            faces is a constant of the tables
//   special  anything else: the step as it is written
// (densities are finite and in [0, 1] from the first step on; a first step may
// leave dead cells a positive value, after_full_step). k_exact_list runs over
// the list of plain and special cells; a step over every cell leaves the dead
// ones' zeros in one buffer, and the other is filled with zeros. Measured on 64^3 (32 % plain),
// 237 steps with upload and download: 7.0 ms on every cell, 2.3 ms on the list
// with a launch per step, 1.6 in one launch (k_exact_resident).
struct Cell {
    size_t W, E, S, N, B, F;
};
__device__ __forceinline__ Cell neighbours_of(size_t c, int n) {
    const unsigned un = (unsigned)n, x = (unsigned)(c % un), r = (unsigned)(c / un), y = r % un, z = r / un;
    const size_t nn = un, plane = nn * nn;
    Cell q;
    q.W = x == 0 ? c + nn - 1 : c - 1;
    q.E = x == un - 1 ? c - (nn - 1) : c + 1;
    q.S = y == 0 ? c + plane - nn : c - nn;
    q.N = y == un - 1 ? c - (plane - nn) : c + nn;
    q.B = z == 0 ? c + plane * (nn - 1) : c - plane;
    q.F = z == un - 1 ? c - plane * (nn - 1) : c + plane;
    return q;
}

// chunks of 256 cells: the number of listed cells (FILL false), or their list
// from the chunk's offset: c, or ~c for special ones; and the plain cells' sums
// of faces in the same order
template <typename Real, bool FILL>
__global__ void __launch_bounds__(256) k_exact_collect(int n, const Real *__restrict__ b0, const double *__restrict__ dfx,
                                                       const double *__restrict__ dfy, const double *__restrict__ dfz,
                                                       int *__restrict__ offset, int *__restrict__ list, double *__restrict__ dsum) {
    const size_t N = (size_t)n * n * n, c = (size_t)blockIdx.x * 256 + threadIdx.x;
    int cls = kDead;
    double d[6];
    if (c < N) {
        const Cell q = neighbours_of(c, n);
        d[0] = dfx[q.W], d[1] = dfx[c], d[2] = dfy[q.S], d[3] = dfy[c], d[4] = dfz[q.B], d[5] = dfz[c];
        cls = cell_class((double)b0[c], d);
    }
    __shared__ int sums[8];
    const unsigned m = __ballot_sync(0xffffffffu, cls != kDead);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) sums[warp] = __popc(m);
    __syncthreads();
    if (!FILL) {
        if (threadIdx.x == 0) {
            int t = 0;
            for (int k = 0; k < 8; ++k) t += sums[k];
            offset[blockIdx.x] = t;
        }
        return;
    }
    if (cls == kDead) return;
    int at = offset[blockIdx.x] + __popc(m & ((1u << lane) - 1u));
    for (int k = 0; k < warp; ++k) at += sums[k];
    list[at] = cls == kPlain ? (int)c : ~(int)c;
    dsum[at] = d[0] + d[1] + d[2] + d[3] + d[4] + d[5];
}

// a value clamped to [0, 1], NaN to 0, in double on its bits: comparisons would
// go to the FP64 pipe
__device__ __forceinline__ float clamp01(float v) {
    v = 0.f < v ? v : 0.f;
    return v < 1.f ? v : 1.f;
}
__device__ __forceinline__ double clamp01(double v) {
    const unsigned hi = (unsigned)__double2hiint(v);
    if (hi < 0x3ff00000u) return v;
    const bool nan = (hi & 0x7fffffffu) > 0x7ff00000u || ((hi & 0x7fffffffu) == 0x7ff00000u && __double2loint(v) != 0);
    return (int)hi < 0 || nan ? 0.0 : 1.0;
}

// the step of listed cell e: d, the faces W E S N B F, and their sum; p, the
// densities of the cell and its neighbours in the same order
template <typename Real>
__device__ __forceinline__ Real listed_step(int e, const double (&t)[6], double sum, const Real (&p)[7], const Real *b0, Real rho, double dt,
                                            double ih2) {
    double d[6];
#pragma unroll
    for (int f = 0; f < 6; ++f) d[f] = t[f];
    if (e < 0) {
        const Real tissue = b0[~e] + p[0];
        if (!(tissue > 0.)) d[0] = d[1] = d[2] = d[3] = d[4] = d[5] = 0.0;
#pragma unroll
        for (int f = 0; f < 6; f += 2) {
            if (d[f] == 0 && p[1 + f] > 0.) d[f + 1] *= 2.0;
            if (d[f + 1] == 0 && p[2 + f] > 0.) d[f] *= 2.0;
        }
        sum = d[0] + d[1] + d[2] + d[3] + d[4] + d[5];
    }
    const double fin = ih2 * (d[0] * (double)p[1] + d[1] * (double)p[2] + d[2] * (double)p[3] + d[3] * (double)p[4] + d[4] * (double)p[5] +
                              d[5] * (double)p[6]);
    const double fout = -(sum * (double)p[0] * ih2);
    const double react = reaction(rho, p[0]);
    const Real dphidt = (Real)(fout + fin + react);
    return clamp01((Real)((double)p[0] + dt * (double)dphidt));
}

template <typename Real>
struct ExactArgs {
    int n, nsteps, cap;  // cap: cells with their faces in shared memory
    const int *count, *list;
    const double *dsum, *dfx, *dfy, *dfz;
    const Real *b0;
    Real *phi, *other;  // the density, and the buffer the first step writes
    Real rho;
    double dt, ih2;
    unsigned *arrived;  // arrivals at the barrier between steps
    int *status;
};
constexpr int kResidentSteps = 4;  // fewer do not repay the fill of shared memory (the faces, once: about a step)
constexpr int kResidentThreads = 1024;
constexpr size_t kCellBytes = 7 * sizeof(double) + sizeof(int);
// shared memory for cells; the limit set for the kernel, whatever a launch takes (it
// is the function's, shared by handles on other threads)
constexpr int kCellsBytes = 224 * 1024;

// All steps in one launch: a CTA keeps a stretch of the list, with the faces and
// their sums, in shared memory (what does not fit it reads again each step). The
// FP64 pipe's share of a step is 21 operations a cell at 16 cycles per warp and
// SM: 3.1 us on 64^3, 24 on 128^3. The rest of the 8.2 and 28.8 us that a launch
// per step took were the launch, the loads of the list and the faces and the
// last CTAs' tail; this takes 5.6 and 26.0 us. (Waiting for the CTAs that own
// cells within a plane, by flags of their own, instead of counting all: 5.7, and
// 2.8 against 2.7 us at 33^3.)
template <typename Real>
__global__ void __launch_bounds__(kResidentThreads, 1) k_exact_resident(ExactArgs<Real> a) {
    extern __shared__ double s_d[];  // faces and sum, [7][cap]; then the cells
    int *s_cell = (int *)(s_d + 7 * (size_t)a.cap);
    const int T = gridDim.x, rank = blockIdx.x, tid = threadIdx.x, m = *a.count;
    auto begin_of = [&](int r) { return (int)((long)m * r / T); };
    const int q0 = begin_of(rank), own = begin_of(rank + 1) - q0;
    auto faces = [&](int c, const Cell &q, double (&d)[6]) {
        d[0] = a.dfx[q.W];
        d[1] = a.dfx[c];
        d[2] = a.dfy[q.S];
        d[3] = a.dfy[c];
        d[4] = a.dfz[q.B];
        d[5] = a.dfz[c];
    };
    for (int i = tid; i < min(own, a.cap); i += kResidentThreads) {
        const int e = a.list[q0 + i], c = e < 0 ? ~e : e;
        double d[6];
        faces(c, neighbours_of((size_t)c, a.n), d);
#pragma unroll
        for (int f = 0; f < 6; ++f) s_d[(size_t)f * a.cap + i] = d[f];
        s_d[(size_t)6 * a.cap + i] = a.dsum[q0 + i];
        s_cell[i] = e;
    }
    Real *in = a.phi, *out = a.other;
    for (int s = 0; s < a.nsteps; ++s) {
        for (int i = tid; i < own; i += kResidentThreads) {
            const bool here = i < a.cap;
            const int e = here ? s_cell[i] : a.list[q0 + i], c = e < 0 ? ~e : e;
            const Cell q = neighbours_of((size_t)c, a.n);
            const Real p[7] = {in[c], in[q.W], in[q.E], in[q.S], in[q.N], in[q.B], in[q.F]};
            double d[6], sum;
            if (here) {
#pragma unroll
                for (int f = 0; f < 6; ++f) d[f] = s_d[(size_t)f * a.cap + i];
                sum = s_d[(size_t)6 * a.cap + i];
            } else {
                faces(c, q, d);
                sum = a.dsum[q0 + i];
            }
            out[c] = listed_step<Real>(e, d, sum, p, a.b0, a.rho, a.dt, a.ih2);
        }
        if (s == a.nsteps - 1) break;
        __syncthreads();
        int ok = 1;
        if (tid == 0) {
            arrive(a.arrived);
            ok = wait_for_arrivals(a.arrived, (unsigned)(s + 1) * T, a.status);
        }
        if (!__syncthreads_and(ok)) break;
        Real *const t = in;
        in = out;
        out = t;
    }
}

template <typename Real>
__global__ void __launch_bounds__(64) k_exact_list(int n, const int *__restrict__ count, const int *__restrict__ list,
                                                   const double *__restrict__ dsum, const Real *__restrict__ phi,
                                                   Real *__restrict__ out, const Real *__restrict__ b0, const double *__restrict__ dfx,
                                                   const double *__restrict__ dfy, const double *__restrict__ dfz, Real rho, double dt,
                                                   double ih2) {
    const int m = *count;
    for (int i = blockIdx.x * 64 + threadIdx.x; i < m; i += gridDim.x * 64) {
        const int e = list[i];
        const size_t c = (size_t)(e < 0 ? ~e : e);
        const Cell q = neighbours_of(c, n);
        const Real p[7] = {phi[c], phi[q.W], phi[q.E], phi[q.S], phi[q.N], phi[q.B], phi[q.F]};
        const double d[6] = {dfx[q.W], dfx[c], dfy[q.S], dfy[c], dfz[q.B], dfz[c]};
        out[c] = listed_step<Real>(e, d, dsum[i], p, b0, rho, dt, ih2);
    }
}

// Tissue tensor of the MALA slopes operator (Glioma_MALA_SlopesOperator.h:131-148):
// inside the tissue (p_w > 0 || p_g > 0), tt[f] = 2/(1/a_c + 1/a_f) with
// a = p_w + p_g * ratioD in double (1/0 = inf gives 0 toward a cell outside
// the tissue), then the Neumann doubling in order; zero outside. Fields are
// read as Real (the reference's cells store p_w, p_g in Real).
template <typename Real>
__global__ void k_mala_tables(int n, const double *__restrict__ pw, const double *__restrict__ pg, double ratio,
                              double *__restrict__ tt) {
    const size_t N = (size_t)n * n * n;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < N;
         c += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(c % n), y = (int)((c / n) % n), z = (int)(c / ((size_t)n * n));
        const size_t nn = (size_t)n, plane = nn * nn;
        const size_t nb[7] = {c,
                              c - x + wrapm(x, n),
                              c - x + wrapp(x, n),
                              c + ((size_t)wrapm(y, n) - y) * nn,
                              c + ((size_t)wrapp(y, n) - y) * nn,
                              c + ((size_t)wrapm(z, n) - z) * plane,
                              c + ((size_t)wrapp(z, n) - z) * plane};
        double t[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        const Real w0 = (Real)pw[c], g0 = (Real)pg[c];
        if (w0 > 0.0 || g0 > 0.0) {
            const double a0 = (double)w0 + (double)g0 * ratio;
            for (int f = 0; f < 6; ++f) {
                const double af = (double)(Real)pw[nb[f + 1]] + (double)(Real)pg[nb[f + 1]] * ratio;
                t[f] = 2.0 * (1.0 / ((1.0 / a0) + (1.0 / af)));
            }
            if (t[0] == 0) t[1] *= 2.0;
            if (t[1] == 0) t[0] *= 2.0;
            if (t[2] == 0) t[3] *= 2.0;
            if (t[3] == 0) t[2] *= 2.0;
            if (t[4] == 0) t[5] *= 2.0;
            if (t[5] == 0) t[4] *= 2.0;
        }
        for (int f = 0; f < 6; ++f) tt[(size_t)f * N + c] = t[f];
    }
}

// One step of the slopes (Glioma_MALAslopesRHS<3>, :152-182, then
// UpdateMALAslopes<3>, :215-223) from phi, sRho, sD before the step:
//   dsRho/dt = -ih2 Dw (sum tt) sRho_c + ih2 Dw sum tt_f sRho_f + phi (1 - phi)
//   dsD/dt   = -ih2 Dw (sum tt) sD_c + ih2 Dw sum tt_f sD_f
//              + ih2 sum tt_f phi_f - ih2 (sum tt) phi_c
// each sum and product in the reference's order, the rates rounded to Real,
// s += dt * rate in double.
template <typename Real>
__global__ void k_mala_slopes(int n, const Real *__restrict__ phi, const Real *__restrict__ sr,
                              const Real *__restrict__ sd, Real *__restrict__ sr_out, Real *__restrict__ sd_out,
                              const double *__restrict__ tt, Real Dw, double ih2, double dt) {
    const size_t N = (size_t)n * n * n;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < N;
         c += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(c % n), y = (int)((c / n) % n), z = (int)(c / ((size_t)n * n));
        const size_t nn = (size_t)n, plane = nn * nn;
        const size_t nb[6] = {c - x + wrapm(x, n),
                              c - x + wrapp(x, n),
                              c + ((size_t)wrapm(y, n) - y) * nn,
                              c + ((size_t)wrapp(y, n) - y) * nn,
                              c + ((size_t)wrapm(z, n) - z) * plane,
                              c + ((size_t)wrapp(z, n) - z) * plane};
        double t[6], s[6], d[6], p[6];
        for (int f = 0; f < 6; ++f) {
            t[f] = tt[(size_t)f * N + c];
            s[f] = (double)sr[nb[f]];
            d[f] = (double)sd[nb[f]];
            p[f] = (double)phi[nb[f]];
        }
        const double s0 = (double)sr[c], d0 = (double)sd[c], p0 = (double)phi[c];
        const double tsum = t[0] + t[1] + t[2] + t[3] + t[4] + t[5];
        const double ihD = ih2 * (double)Dw;
        const double inR = ihD * (t[0] * s[0] + t[1] * s[1] + t[2] * s[2] + t[3] * s[3] + t[4] * s[4] + t[5] * s[5]);
        const double outR = -ih2 * (double)Dw * tsum * s0;
        const double reR = p0 * (1. - p0);
        const Real rr = (Real)(outR + inR + reR);
        const double inD = ihD * (t[0] * d[0] + t[1] * d[1] + t[2] * d[2] + t[3] * d[3] + t[4] * d[4] + t[5] * d[5]);
        const double outD = -ih2 * (double)Dw * tsum * d0;
        const double rin = ih2 * (t[0] * p[0] + t[1] * p[1] + t[2] * p[2] + t[3] * p[3] + t[4] * p[4] + t[5] * p[5]);
        const double rout = -ih2 * tsum * p0;
        const Real rd = (Real)(outD + inD + rin + rout);
        sr_out[c] = (Real)(s0 + dt * (double)rr);
        sd_out[c] = (Real)(d0 + dt * (double)rd);
    }
}

int grid_for(const Handle &h) {
    const size_t blocks = (h.N + 255) / 256;
    const size_t cap = (size_t)h.num_sms * 8;
    return (int)(blocks < cap ? blocks : cap);
}

}  // namespace

int exact_build_tables(Handle &h, double Dw, double Dg) {
    if (h.tables_valid && h.tab_Dw == Dw && h.tab_Dg == Dg) return GBG_OK;
    const int g = grid_for(h);
    if (h.prec == GBG_PREC_F64) {
        k_build_tables<double><<<g, 256, 0, h.stream>>>(h.n, h.pw, h.pg, Dw, Dg, (double *)h.b0,
                                                        h.dfx, h.dfy, h.dfz);
    } else {
        k_build_tables<float><<<g, 256, 0, h.stream>>>(h.n, h.pw, h.pg, (float)Dw, (float)Dg,
                                                       (float *)h.b0, h.dfx, h.dfy, h.dfz);
    }
    h.launches++;
    GBG_CUDA_TRY(cudaGetLastError());
    h.tab_Dw = Dw;
    h.tab_Dg = Dg;
    h.tables_valid = true;
    h.exact_full = kAnyState;
    h.exact_listed = false;
    h.exact_fulls = 0;
    return GBG_OK;
}

void exact_alloc_list(Handle &h) {
    const size_t chunks = (h.N + 255) / 256;
    reserve_device({{(void **)&h.exact_list, (h.N + chunks + 2) * sizeof(int)}, {(void **)&h.exact_dsum, h.N * sizeof(double)}});
}

// nsteps steps over the list in one launch; GBG_ERR_UNSUPPORTED: not here
template <typename Real>
int resident_steps(Handle &h, double rho, double dt, double ih2, long nsteps, bool capturing) {
    const int T = h.num_sms, chunks = (int)((h.N + 255) / 256);
    ExactArgs<Real> a;
    a.n = h.n;
    a.nsteps = (int)nsteps;
    a.cap = (int)std::min<size_t>((h.N + T - 1) / T, kCellsBytes / kCellBytes);
    a.cap += a.cap & 1;
    const size_t smem = a.cap * kCellBytes;
    a.count = h.exact_list + h.N + chunks;
    a.list = h.exact_list;
    a.dsum = h.exact_dsum;
    a.dfx = h.dfx;
    a.dfy = h.dfy;
    a.dfz = h.dfz;
    a.b0 = (const Real *)h.b0;
    a.phi = (Real *)h.phi[h.cur];
    a.other = (Real *)h.phi[h.cur ^ 1];
    a.rho = (Real)rho;
    a.dt = dt;
    a.ih2 = ih2;
    a.arrived = (unsigned *)(h.exact_list + h.N + chunks + 1);
    a.status = h.dev_status;
    const void *fn = (const void *)k_exact_resident<Real>;
    GBG_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kCellsBytes));
    GBG_CUDA_TRY(cudaMemsetAsync(a.arrived, 0, sizeof(unsigned), h.stream));
    void *args[] = {&a};
    if (cudaLaunchCooperativeKernel(fn, dim3((unsigned)T), dim3(kResidentThreads), args, smem, h.stream) != cudaSuccess) {
        cudaGetLastError();
        return GBG_ERR_UNSUPPORTED;
    }
    h.exact_waited = true;
    h.exact_in_graph |= capturing;
    h.launches++;
    if (nsteps & 1) h.cur ^= 1;
    return GBG_OK;
}

int exact_steps(Handle &h, double Dw, double Dg, double rho, double dt, long nsteps) {
    int rc = exact_build_tables(h, Dw, Dg);
    if (rc) return rc;
    const double hh = 1.0 / h.n;
    const double ih2 = 1. / (hh * hh);
    const int g = grid_for(h), chunks = (int)((h.N + 255) / 256);
    const int gl = (int)std::min<size_t>((h.N + 63) / 64, (size_t)h.num_sms * 16);
    auto collect = [&](auto real) {
        using Real = decltype(real);
        int *offset = h.exact_list + h.N;
        const Real *b0 = (const Real *)h.b0;
        k_exact_collect<Real, false><<<chunks, 256, 0, h.stream>>>(h.n, b0, h.dfx, h.dfy, h.dfz, offset, nullptr, nullptr);
        k_exact_offsets<<<1, 1024, 0, h.stream>>>(chunks, offset);
        k_exact_collect<Real, true><<<chunks, 256, 0, h.stream>>>(h.n, b0, h.dfx, h.dfy, h.dfz, offset, h.exact_list, h.exact_dsum);
        h.launches += 3;
        h.exact_listed = true;
    };
    auto step = [&](auto real, const void *in, void *out) {
        using Real = decltype(real);
        if (h.exact_full == kListed && h.exact_list) {
            k_exact_list<Real><<<gl, 64, 0, h.stream>>>(h.n, h.exact_list + h.N + chunks, h.exact_list, h.exact_dsum, (const Real *)in,
                                                        (Real *)out, (const Real *)h.b0, h.dfx, h.dfy, h.dfz, (Real)rho, dt, ih2);
        } else {
            k_exact_step<Real><<<g, 256, 0, h.stream>>>(h.n, (const Real *)in, (Real *)out, (const Real *)h.b0, h.dfx, h.dfy, h.dfz,
                                                        (Real)rho, dt, ih2);
            h.exact_full = after_full_step(h.exact_full, rho, dt);
            ++h.exact_fulls;
        }
    };
    // Making the list costs 24 us, and a listed step saves 3 us of launch and 0.1
    // ns a cell: it pays from five steps on or 200,000 cell-steps. Counted are the
    // steps ahead in this call and the full ones taken with these tables, for
    // callers that step one by one. Coefficients that change with every call, of 2
    // steps at 32^3: 37 us, with the list 48; of 6: 70 and 65; of 3 at 48^3 85 and 79.
    auto list_pays = [&](long ahead) {
        const long due = ahead + h.exact_fulls - 1;
        return h.exact_listed || due >= 5 || due * (long)h.N >= 200000;
    };
    // What is known here does not hold when a captured graph runs: it takes its own
    // full step and makes its own list, and a call after it does so too.
    auto forget = [&] {
        h.exact_full = kAnyState;
        h.exact_listed = false;
        h.exact_fulls = 0;
    };
    bool capturing;
    if ((rc = stream_capturing(h, &capturing))) return rc;
    if (capturing) forget();
    for (long s = 0; s < nsteps; ++s) {
        if (h.exact_full == kDeadZero && h.exact_list && list_pays(nsteps - s)) {  // the other buffer's dead cells
            GBG_CUDA_TRY(cudaMemsetAsync(h.phi[h.cur ^ 1], 0, h.N * (h.prec == GBG_PREC_F64 ? sizeof(double) : sizeof(float)), h.stream));
            h.exact_full = kListed;
        }
        if (h.exact_full == kListed && h.exact_list) {
            if (!h.exact_listed) h.prec == GBG_PREC_F64 ? collect(double{}) : collect(float{});
            if (nsteps - s >= kResidentSteps && nsteps - s <= 0x7fffffffL) {
                const int rc = h.prec == GBG_PREC_F64 ? resident_steps<double>(h, rho, dt, ih2, nsteps - s, capturing)
                                                      : resident_steps<float>(h, rho, dt, ih2, nsteps - s, capturing);
                if (rc == GBG_OK) break;
                if (rc != GBG_ERR_UNSUPPORTED) return rc;
            }
        }
        if (h.prec == GBG_PREC_F64)
            step(double{}, h.phi[h.cur], h.phi[h.cur ^ 1]);
        else
            step(float{}, h.phi[h.cur], h.phi[h.cur ^ 1]);
        h.launches++;
        h.cur ^= 1;
    }
    if (capturing) forget();
    GBG_CUDA_TRY(cudaGetLastError());
    return GBG_OK;
}

int mala_steps(Handle &h, double Dw, double Dg, double rho, double dt, long nsteps) {
    // ratioD = Dg / Dw in Real, widened to double (Glioma_MALA_SlopesOperator.h:117)
    const double ratio = h.prec == GBG_PREC_F64 ? Dg / Dw : (double)((float)Dg / (float)Dw);
    const int g = grid_for(h);
    if (!h.mala_valid || h.mala_ratio != ratio) {
        if (h.prec == GBG_PREC_F64)
            k_mala_tables<double><<<g, 256, 0, h.stream>>>(h.n, h.pw, h.pg, ratio, h.mala_tt);
        else
            k_mala_tables<float><<<g, 256, 0, h.stream>>>(h.n, h.pw, h.pg, ratio, h.mala_tt);
        h.launches++;
        GBG_CUDA_TRY(cudaGetLastError());
        h.mala_ratio = ratio;
        h.mala_valid = true;
    }
    const double hh = 1.0 / h.n;
    const double ih2 = 1. / (hh * hh);
    for (long s = 0; s < nsteps; ++s) {
        const int c = h.cur;
        if (h.prec == GBG_PREC_F64) {
            k_mala_slopes<double><<<g, 256, 0, h.stream>>>(h.n, (const double *)h.phi[c], (const double *)h.sr[c],
                                                          (const double *)h.sd[c], (double *)h.sr[c ^ 1],
                                                          (double *)h.sd[c ^ 1], h.mala_tt, Dw, ih2, dt);
        } else {
            k_mala_slopes<float><<<g, 256, 0, h.stream>>>(h.n, (const float *)h.phi[c], (const float *)h.sr[c],
                                                         (const float *)h.sd[c], (float *)h.sr[c ^ 1],
                                                         (float *)h.sd[c ^ 1], h.mala_tt, (float)Dw, ih2, dt);
        }
        h.launches++;
        // the phi step reads the same phi[c] and toggles cur for phi and slopes
        if (int rc = exact_steps(h, Dw, Dg, rho, dt, 1)) return rc;
    }
    GBG_CUDA_TRY(cudaGetLastError());
    return GBG_OK;
}

}  // namespace gbg
