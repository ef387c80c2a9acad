// The first stage of delayed-acceptance MCMC on the GPU: `steps` Metropolis
// steps on the screening density
//   log pi*(v) = log L(phi(v)) + log prior(v),
//   phi(v) = m * clamp(phi0 + sum_p c_p(v - u_ref) J_p, 0, 1)
// (the affine model of affine.cu, evaluated at the observation lists' cells
// from the same gathered columns) for B chains at once, a cluster of CTAs per
// chain, so that a whole inner chain is one launch instead of one host round
// trip per step. The moves are those of the host sampler's inner chain
// (gliomauq_gb300/mcmc.py, da): with probability axis_prob a redraw of the
// symmetry coordinate from its prior conditional, accepted with the ratio of
// pi*'s likelihood factors; with probability ind_prob an independence
// proposal m + G xi for the other coordinates (a fixed Gaussian, accepted
// with the Metropolis-Hastings ratio of its density); otherwise a random
// walk v + step * C xi on the other coordinates. All three leave pi*
// invariant. Random numbers come from a
// counter-based hash (SplitMix64 finaliser, Steele, Lea & Flood 2014) of
// (seed, chain, step, draw), normals by the Box-Muller transform.
//
// Prior in the sampler's coordinates v: u = Ai v; theta_i = exp(u_i) where
// bit i of log_mask is set, else u_i; log prior = sum of those u_i (the
// log-Jacobian of the uniform prior on theta) inside the box lo <= theta <= hi
// with the seed voxel (rint of theta_2..4) inside the mask, -inf outside.
//
// Each observation point's model (phi0, the basis fields, the mask) and its
// observed values are one 16-float record (affine.cu builds them), read with
// four vector loads. The per-point likelihood terms are evaluated in float
// (this GPU's FP64 rate is a small fraction of its FP32 rate, and the screen
// only has to be one fixed function: the chain returns its own log pi* at the
// start and end points, which is what the second stage's ratio uses), summed
// in float per partial sum and in double over these. The Bernoulli terms of
// HGG_Likelihood (:136-153) in a form without cancellation: with
// q = (u - uc)^2 / slope, alpha = 1 - e^-q / 2 above uc and e^-q / 2 below,
// so log alpha and log(1 - alpha) are log1p(-e^-q / 2) and log(1/2) - q.
#include <math_constants.h>

#include <cmath>

#include "gbg_internal.cuh"
#include "lik_terms.cuh"

namespace gbg {
namespace {

constexpr int kChainThreads = 512;
constexpr int kChainWarps = kChainThreads / 32;

struct ChainArgs {
    int steps, P, quad_axis, axis, log_mask, n;
    double axis_prob, step, ind_prob;
    double u_ref[6], chol[36], Ai[36], lo[6], hi[6], ulo[6], uhi[6];
    double ind_mean[6], ind_chol[36], ind_inv[36];
    const unsigned char *mask;
    unsigned long long seed;
    const float4 *rec;  // 16 floats per observation point, PET list then T1/T2 list: four arrays of float4
    int n_pet, n_ti;
    double pet_scale, t1_uc, t2_uc, is2, pet_sigma2;
    double *v, *lp_start, *lp_end;
    int *counts;
};

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// uniform in (0, 1] from (seed, chain, step, draw)
__device__ __forceinline__ double uniform01(unsigned long long seed, int chain, int step, int k) {
    unsigned long long x = mix64(seed ^ mix64((unsigned long long)chain));
    x = mix64(x ^ ((unsigned long long)step << 8 | (unsigned long long)k));
    return (double)((x >> 11) + 1) * (1.0 / 9007199254740992.0);
}

// One proposal (or the start): the state it moves from, the proposed state, their
// log priors, the move and what its acceptance needs besides the likelihood.
struct Proposal {
    double v[6], y[6], lpv, lpy, lqd, logu;
    float c[12];   // the affine model's coefficients at y
    int eval, kind;  // inside the prior; 0 random walk, 2 axis redraw, 4 independence
};

struct Matrices {
    double chol[36], Ai[36], ind_chol[36], ind_inv[36];
};

// The functions below are a warp's: lane i < 6 holds coordinate i (the other
// lanes hold copies of coordinate 0 that nobody reads), and every sum runs in
// the order of the coordinates.
__device__ __forceinline__ double coord(double x, int i) { return __shfl_sync(0xffffffffu, x, i); }

__device__ __forceinline__ double row_times(const double *m, double x) {
    const int i = (threadIdx.x & 31) < 6 ? threadIdx.x & 31 : 0;
    double s = 0.0;
    for (int j = 0; j < 6; ++j) s += m[i * 6 + j] * coord(x, j);
    return s;
}

__device__ double prior_logp(const ChainArgs &a, const Matrices &m, double v) {
    const int lane = threadIdx.x & 31, i = lane < 6 ? lane : 0;
    const double u = row_times(m.Ai, v);
    const bool lg = (a.log_mask >> i) & 1;
    double th = u, jac = 0.0;
    if (lg) th = exp(u);
    for (int k = 0; k < 6; ++k) {
        const double uk = coord(u, k);
        if ((a.log_mask >> k) & 1) jac += uk;
    }
    if (!__all_sync(0xffffffffu, th >= a.lo[i] && th <= a.hi[i])) return -CUDART_INF;
    int c[3];
    for (int k = 0; k < 3; ++k) {
        const double r = rint(coord(th, 2 + k));
        if (!(r >= 0.0 && r < (double)a.n)) return -CUDART_INF;
        c[k] = (int)r;
    }
    if (!a.mask[((size_t)c[2] * a.n + c[1]) * a.n + c[0]]) return -CUDART_INF;
    return jac;
}

// coordinate `axis` of v redrawn from the prior conditional given the others:
// on the line v + t e_axis the prior density is exp(alpha t) on the interval
// the box allows; v is left unchanged when the line misses the box
__device__ double redraw_axis(const ChainArgs &a, const Matrices &m, double v, double q) {
    const int lane = threadIdx.x & 31, i = lane < 6 ? lane : 0, ax = a.axis;
    const double u = row_times(m.Ai, v), col = m.Ai[i * 6 + ax];
    const bool lg = (a.log_mask >> i) & 1;
    double b1 = 0.0, b2 = 0.0;
    if (lg && col != 0.0) {
        b1 = (a.ulo[i] - u) / col;
        b2 = (a.uhi[i] - u) / col;
    }
    double t_lo = -CUDART_INF, t_hi = CUDART_INF, alpha = 0.0;
    for (int k = 0; k < 6; ++k) {
        const double ck = coord(col, k), k1 = coord(b1, k), k2 = coord(b2, k);
        if (!((a.log_mask >> k) & 1)) continue;
        alpha += ck;
        if (ck == 0.0) continue;
        t_lo = fmax(t_lo, fmin(k1, k2));
        t_hi = fmin(t_hi, fmax(k1, k2));
    }
    if (!(isfinite(t_lo) && isfinite(t_hi) && t_hi > t_lo)) return v;
    double t;
    if (fabs(alpha) < 1e-12)
        t = t_lo + q * (t_hi - t_lo);
    else
        t = t_lo + log1p(q * expm1(alpha * (t_hi - t_lo))) / alpha;
    return lane == ax ? v + t : v;
}

// six normals from the step's draws 2 to 7, in float: their precision does not
// matter, the state they move stays double
__device__ double normals(const ChainArgs &a, int chain, int s) {
    const int lane = threadIdx.x & 31, i = lane < 6 ? lane : 0, k = i / 2;
    const float r = sqrtf(-2.0f * logf((float)uniform01(a.seed, chain, s, 2 + 2 * k)));
    float sn, cs;
    sincospif(2.0f * (float)uniform01(a.seed, chain, s, 3 + 2 * k), &sn, &cs);
    return (double)(i & 1 ? r * sn : r * cs);
}

// fills in what follows from y: the prior and the coefficients
__device__ void finish(const ChainArgs &a, const Matrices &m, double v, double y, double lpv, double lqd, int kind, double logu,
                       Proposal *o) {
    const int lane = threadIdx.x & 31;
    const double lpy = prior_logp(a, m, y);
    const double d = lane < 6 ? y - a.u_ref[lane] : 0.0;
    if (lane < 6) {
        o->v[lane] = v;
        o->y[lane] = y;
        o->c[lane] = (float)d;
    }
    if (a.quad_axis >= 0) {
        const int ax = a.quad_axis;
        const double da = coord(d, ax);
        if (lane < 6) {
            if (lane == ax)
                o->c[6] = (float)(0.5 * (da * da));
            else
                o->c[lane < ax ? 7 + lane : 6 + lane] = (float)(da * d);
        }
    }
    if (lane == 0) {
        o->lpv = lpv;
        o->lpy = lpy;
        o->lqd = lqd;
        o->logu = logu;
        o->eval = isfinite(lpy) ? 1 : 0;
        o->kind = kind;
    }
}

// the proposal of step s from v
__device__ void propose(const ChainArgs &a, const Matrices &m, int chain, int s, double v, double lpv, Proposal *o) {
    const int lane = threadIdx.x & 31, i = lane < 6 ? lane : 0;
    const double um = uniform01(a.seed, chain, s, 0);
    const bool jump = a.axis >= 0 && um <= a.axis_prob;
    const bool indep = !jump && um <= (a.axis >= 0 ? a.axis_prob : 0.0) + a.ind_prob;
    double y = v, lqd = 0.0;  // log proposal-density ratio of an independence move
    if (jump) {
        y = redraw_axis(a, m, v, uniform01(a.seed, chain, s, 1));
    } else if (indep) {
        // y = m + G xi on the coordinates other than the axis; the density
        // ratio q(v) / q(y) with z = G^-1 (x - m)
        double xi = normals(a, chain, s);
        if (i == a.axis) xi = 0.0;
        const double d = row_times(m.ind_chol, xi), z = row_times(m.ind_inv, v - a.ind_mean[i]);
        if (i != a.axis) y = a.ind_mean[i] + d;
        double qy = 0.0, qv = 0.0;
        for (int k = 0; k < 6; ++k) {
            const double xk = coord(xi, k), zk = coord(z, k);
            if (k == a.axis) continue;
            qy += xk * xk;
            qv += zk * zk;
        }
        lqd = 0.5 * (qy - qv);  // log q(v) - log q(y)
    } else {
        const double d = row_times(m.chol, normals(a, chain, s));
        if (i != a.axis) y = v + a.step * d;
    }
    finish(a, m, v, y, lpv, lqd, jump ? 2 : (indep ? 4 : 0), log(uniform01(a.seed, chain, s, 8)), o);
}

// log Bernoulli(alpha(u)) of observation y in float, without cancellation
__device__ __forceinline__ float log_bernoulli_f(float u, float y, float uc, float is2) {
    const float d = u - uc;
    const float q = d * d * is2;
    const float lhalf_q = -0.69314718f - q;          // log(e^-q / 2)
    const float l1m = log1pf(-0.5f * expf(-q));      // log(1 - e^-q / 2)
    float la, lna;                                   // log alpha, log(1 - alpha)
    if (d > 0.f) {
        la = l1m;
        lna = lhalf_q;
    } else if (d < 0.f) {
        la = lhalf_q;
        lna = l1m;
    } else {
        la = lna = -0.69314718f;
    }
    return y == 1.f ? la : lna;
}

__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// *p of CTA `rank` of the cluster = v, p in shared memory
__device__ __forceinline__ void store_to_rank(double *p, int rank, double v) {
    unsigned at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
}

__device__ __forceinline__ void load_record(const ChainArgs &a, int i, float4 (&r)[4]) {
    const int items = a.n_pet + a.n_ti;
    if (i < items) {
#pragma unroll
        for (int q = 0; q < 4; ++q) r[q] = __ldg(a.rec + (size_t)q * items + i);
    }
}

// rounds [q0, q1) of a lane's points first + q * kChainThreads * K, all PET
// points (kPet), all T1/T2 points (kTi) or some of both or of neither; next
// holds the record of round q0, and of round q1 afterwards
enum { kPet = 1, kTi = 2 };
template <int P, int K, int KIND>
__device__ __forceinline__ void rounds_of(const ChainArgs &a, int q0, int q1, int first, const float (&cf)[P], float4 (&next)[4],
                                          float &fp, float &f1, float &f2) {
    const float scale = (float)a.pet_scale, uc1 = (float)a.t1_uc, uc2 = (float)a.t2_uc, is2 = (float)a.is2;
#pragma unroll 2
    for (int q = q0; q < q1; ++q) {
        const int i = first + q * kChainThreads * K;
        float x[16];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[4 * k] = next[k].x;
            x[4 * k + 1] = next[k].y;
            x[4 * k + 2] = next[k].z;
            x[4 * k + 3] = next[k].w;
        }
        load_record(a, i + kChainThreads * K, next);
        float u = x[0];
#pragma unroll
        for (int p = 0; p < P; ++p) u = fmaf(cf[p], x[1 + p], u);
        u = fminf(fmaxf(u, 0.f), 1.f);
        if (x[P + 1] == 0.f) u = 0.f;
        // a sum without a term here adds +0, which changes no bit of it
        if (KIND & kPet) {
            const float r = u - scale * x[P + 2];
            const float term = KIND == kPet || i < a.n_pet ? r * r : 0.f;
#pragma unroll
            for (int e = 0; e < K; ++e) fp += K > 1 ? __shfl_sync(0xffffffffu, term, e, K) : term;
        }
        if (KIND & kTi) {
            float t1 = log_bernoulli_f(u, x[P + 2], uc1, is2), t2 = log_bernoulli_f(u, x[P + 3], uc2, is2);
            if (KIND != kTi && !(i >= a.n_pet && i < a.n_pet + a.n_ti)) t1 = t2 = 0.f;
#pragma unroll
            for (int e = 0; e < K; ++e) {
                f1 += K > 1 ? __shfl_sync(0xffffffffu, t1, e, K) : t1;
                f2 += K > 1 ? __shfl_sync(0xffffffffu, t2, e, K) : t2;
            }
        }
    }
}

// the sum of 32 floats f[0..31] in double, formed by 8 neighbouring lanes (l of
// them is this one) in the order of warp_sum; valid on their first
__device__ __forceinline__ double sum32(const float *f, int l) {
    const double a = (double)f[l] + (double)f[l + 16], b = (double)f[l + 8] + (double)f[l + 24];
    double v = a + b;
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// The chains are short of parallelism: 64 of them on one CTA each used 64 of
// the 152 SMs, and half of a step went by while one thread formed the proposal
// in double precision (44 us a step at 20632 points). So
//   * a cluster of K CTAs runs a chain, K the largest of 1, 2, 4, 8 for which
//     every CTA gets an SM of its own. The likelihood is the sum of 512 partial
//     sums, over every 512th point each, then by warps of partial sums, then
//     over these; it stays the same sum in the same order for every K: a CTA
//     has 512 / K partial sums, K neighbouring lanes form K consecutive terms
//     of one of them and all add them in order, and each warp's double goes to
//     the shared memory of every CTA of the cluster, which all take the same
//     decision: one cluster barrier a step.
//   * two more warps form the next step's proposals, one for each outcome of
//     the present step, while the others evaluate it.
//   * a point's record lies in four arrays of 16 bytes a point: as 64 bytes in
//     a row, its four loads took four times the passes through L1, which was
//     then 64 % busy.
// 64 chains of 64 steps: 2.81 ms before, 0.86 now.
constexpr int kBlock = kChainThreads + 64;

template <int P, int K>
__global__ void __launch_bounds__(kBlock, 1) k_affine_chain(ChainArgs a) {
    constexpr int kSums = kChainThreads / K, kSumWarps = kChainWarps / K;
    const int chain = blockIdx.x / K, rank = blockIdx.x % K;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    __shared__ Matrices m;
    __shared__ Proposal prop[2][2];  // by step, by the outcome of the step before
    __shared__ float s_f[3][kSums];
    __shared__ double s_red[2][3][kChainWarps];
    __shared__ int s_acc;
    if (t < 36) {
        m.chol[t] = a.chol[t];
        m.Ai[t] = a.Ai[t];
        m.ind_chol[t] = a.ind_chol[t];
        m.ind_inv[t] = a.ind_inv[t];
    }
    __syncthreads();
    if (warp == kChainWarps) {
        const double v = a.v[(size_t)chain * 6 + (lane < 6 ? lane : 0)];
        finish(a, m, v, v, 0.0, 0.0, 0, 0.0, &prop[0][0]);
    }
    if (K > 1)
        cluster_sync();  // every CTA of the cluster runs before its shared memory is written
    else
        __syncthreads();

    // rounds of PET points only, from there on of both, of T1/T2 points only, of
    // both or of the last few points
    const int per = kChainThreads * K, items = a.n_pet + a.n_ti, rounds = (items + per - 1) / per;
    const int pet_end = a.n_pet / per, ti_end = items / per, ti_begin = min((a.n_pet + per - 1) / per, ti_end);
    const int first = rank * kSums + t / K + kChainThreads * (t % K);
    double ly = 0.0, p1 = 0.0, ip = 0.0;  // warp 0
    int cnt[6] = {0, 0, 0, 0, 0, 0};
    if (warp == 0) {
        p1 = -0.5 * a.n_pet * log(2. * 3.14159265358979323846 * a.pet_sigma2);
        ip = -0.5 * (1. / a.pet_sigma2);
    }
    int branch = 0, buf = 0;
    for (int s = -1; s < a.steps; ++s) {  // -1: the start
        const Proposal &now = prop[(s + 1) & 1][branch];
        const bool eval = now.eval;
        if (warp >= kChainWarps) {
            if (s + 1 < a.steps) {
                const int accepted = warp - kChainWarps, l = lane < 6 ? lane : 0;
                propose(a, m, chain, s + 1, accepted || s < 0 ? now.y[l] : now.v[l], accepted || s < 0 ? now.lpy : now.lpv,
                        &prop[s & 1][accepted]);
            }
        } else if (eval) {
            float cf[P], fp = 0.f, f1 = 0.f, f2 = 0.f;
#pragma unroll
            for (int p = 0; p < P; ++p) cf[p] = now.c[p];
            float4 next[4] = {};
            load_record(a, first, next);
            rounds_of<P, K, kPet>(a, 0, pet_end, first, cf, next, fp, f1, f2);
            rounds_of<P, K, kPet | kTi>(a, pet_end, max(pet_end, ti_begin), first, cf, next, fp, f1, f2);
            rounds_of<P, K, kTi>(a, max(pet_end, ti_begin), ti_end, first, cf, next, fp, f1, f2);
            rounds_of<P, K, kPet | kTi>(a, max(max(pet_end, ti_begin), ti_end), rounds, first, cf, next, fp, f1, f2);
            if (t % K == 0) {
                s_f[0][t / K] = fp;
                s_f[1][t / K] = f1;
                s_f[2][t / K] = f2;
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kChainThreads) : "memory");
            // four sums of 32 partial sums to a warp
            for (int w = warp; 4 * w < 3 * kSumWarps; w += kChainWarps) {
                const int k = min(4 * w + lane / 8, 3 * kSumWarps - 1), kind = k / kSumWarps, part = k % kSumWarps;
                double sum = sum32(&s_f[kind][part * 32], lane & 7);
                double *dst = &s_red[buf][kind][rank * kSumWarps + part];
                if (K == 1) {
                    if ((lane & 7) == 0) *dst = sum;
                } else {
                    sum = __shfl_sync(0xffffffffu, sum, lane & ~7);
                    if ((lane & 7) < K) store_to_rank(dst, lane & 7, sum);
                }
            }
        }
        if (K > 1 && eval)
            cluster_sync();
        else
            __syncthreads();
        if (warp == 0) {
            double L = 0.0;
            if (eval) {
                double part = 0.0;
                if (lane < 3)
                    for (int j = 0; j < kChainWarps; ++j) part += s_red[buf][lane][j];
                const double p2 = ip * coord(part, 0);
                L = (p1 + p2) + coord(part, 1) + coord(part, 2);
            }
            const double lq = eval ? L + now.lpy : -CUDART_INF;
            bool acc = false;
            if (s < 0) {
                ly = lq;
                if (t == 0 && rank == 0) a.lp_start[chain] = lq;
            } else {
                // a prior-conditional redraw: its proposal density cancels the
                // prior; an independence move: the proposal density ratio
                const double corr = now.kind == 2 ? now.lpv - now.lpy : (now.kind == 4 ? now.lqd : 0.0);
                acc = isfinite(lq) && (now.logu < lq - ly + corr);
                if (acc) ly = lq;
#pragma unroll
                for (int k = 0; k < 6; k += 2) {
                    cnt[k] += now.kind == k && acc ? 1 : 0;
                    cnt[k + 1] += now.kind == k ? 1 : 0;
                }
                if (s == a.steps - 1 && rank == 0 && lane < 6) a.v[(size_t)chain * 6 + lane] = acc ? now.y[lane] : now.v[lane];
            }
            if (t == 0) s_acc = acc;
        }
        buf ^= eval ? 1 : 0;
        __syncthreads();
        branch = s_acc;
    }
    if (t == 0 && rank == 0) {
        a.lp_end[chain] = ly;
        for (int k = 0; k < 6; ++k) a.counts[(size_t)chain * 6 + k] = cnt[k];
    }
}

template <int P, int K>
cudaError_t launch_chain(int B, cudaStream_t stream, const ChainArgs &a) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)B * K);
    c.blockDim = dim3(kBlock);
    c.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = K;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    c.attrs = at;
    c.numAttrs = K > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&c, k_affine_chain<P, K>, a);
}

template <int P>
cudaError_t launch_chains(int B, int sms, cudaStream_t stream, const ChainArgs &a) {
    const int per = sms / B;
    if (per >= 8) return launch_chain<P, 8>(B, stream, a);
    if (per >= 4) return launch_chain<P, 4>(B, stream, a);
    if (per >= 2) return launch_chain<P, 2>(B, stream, a);
    return launch_chain<P, 1>(B, stream, a);
}

}  // namespace

int affine_set_prior_mask(Handle &h, const unsigned char *mask) {
    if (!h.aff_mask) GBG_CUDA_TRY(cudaMalloc((void **)&h.aff_mask, h.N));
    GBG_CUDA_TRY(cudaMemcpyAsync(h.aff_mask, mask, h.N, cudaMemcpyHostToDevice, h.stream));
    GBG_CUDA_TRY(cudaStreamSynchronize(h.stream));
    return GBG_OK;
}

int affine_chain(Handle &h, const gbg_affine_chain_opts &o, int B, int steps, unsigned long long seed,
                 double *v, double *lp_start, double *lp_end, int *counts) {
    const int P = o.quad_axis >= 0 ? 12 : 6;
    if (!h.aff_J || h.aff_P != P) {
        set_error("affine chain: the affine model must have 6 (no quad_axis) or 12 basis fields");
        return GBG_ERR_STATE;
    }
    if (!h.aff_mask) {
        set_error("affine chain: prior mask not set");
        return GBG_ERR_STATE;
    }
    if (!h.obs.valid) {
        set_error("observations not set");
        return GBG_ERR_STATE;
    }
    if (h.aff_cols_stale)
        if (int rc = affine_gather_columns(h)) return rc;
    // device scratch: v (B x 6), lp_start, lp_end (B), counts (B x 4)
    const size_t need = (size_t)B * (8 * sizeof(double) + 6 * sizeof(int));
    if (need > h.aff_chain_bytes) {
        if (h.aff_chain) cudaFree(h.aff_chain);
        h.aff_chain = nullptr;
        h.aff_chain_bytes = 0;
        GBG_CUDA_TRY(cudaMalloc(&h.aff_chain, need));
        h.aff_chain_bytes = need;
    }
    double *d_v = (double *)h.aff_chain, *d_l0 = d_v + (size_t)B * 6, *d_l1 = d_l0 + B;
    int *d_cnt = (int *)(d_l1 + B);
    ChainArgs a;
    a.steps = steps;
    a.P = P;
    a.quad_axis = o.quad_axis;
    a.axis = o.axis;
    a.log_mask = o.log_mask;
    a.n = h.n;
    a.axis_prob = o.axis_prob;
    a.ind_prob = o.ind_prob;
    for (int i = 0; i < 6; ++i) a.ind_mean[i] = o.ind_mean[i];
    for (int i = 0; i < 36; ++i) {
        a.ind_chol[i] = o.ind_chol[i];
        a.ind_inv[i] = o.ind_inv[i];
    }
    a.step = o.step;
    for (int i = 0; i < 6; ++i) {
        a.u_ref[i] = o.u_ref[i];
        a.lo[i] = o.lo[i];
        a.hi[i] = o.hi[i];
        const bool lg = (o.log_mask >> i) & 1;
        a.ulo[i] = lg ? std::log(o.lo[i]) : o.lo[i];
        a.uhi[i] = lg ? std::log(o.hi[i]) : o.hi[i];
    }
    for (int i = 0; i < 36; ++i) {
        a.chol[i] = o.chol[i];
        a.Ai[i] = o.Ai[i];
    }
    a.mask = h.aff_mask;
    a.seed = seed;
    a.rec = h.aff_rec;
    a.n_pet = h.obs.n_pet;
    a.n_ti = h.obs.n_ti;
    a.pet_scale = h.obs.pet_scale;
    a.t1_uc = h.obs.t1_uc;
    a.t2_uc = h.obs.t2_uc;
    a.is2 = 1. / h.obs.slope;
    a.pet_sigma2 = h.obs.pet_sigma2;
    a.v = d_v;
    a.lp_start = d_l0;
    a.lp_end = d_l1;
    a.counts = d_cnt;
    GBG_CUDA_TRY(cudaMemcpyAsync(d_v, v, (size_t)B * 6 * sizeof(double), cudaMemcpyHostToDevice, h.stream));
    GBG_CUDA_TRY(P == 12 ? launch_chains<12>(B, h.num_sms, h.stream, a) : launch_chains<6>(B, h.num_sms, h.stream, a));
    h.launches++;
    GBG_CUDA_TRY(cudaMemcpyAsync(v, d_v, (size_t)B * 6 * sizeof(double), cudaMemcpyDeviceToHost, h.stream));
    GBG_CUDA_TRY(cudaMemcpyAsync(lp_start, d_l0, (size_t)B * sizeof(double), cudaMemcpyDeviceToHost, h.stream));
    GBG_CUDA_TRY(cudaMemcpyAsync(lp_end, d_l1, (size_t)B * sizeof(double), cudaMemcpyDeviceToHost, h.stream));
    if (counts)
        GBG_CUDA_TRY(cudaMemcpyAsync(counts, d_cnt, (size_t)B * 6 * sizeof(int), cudaMemcpyDeviceToHost, h.stream));
    GBG_CUDA_TRY(cudaStreamSynchronize(h.stream));
    return GBG_OK;
}

}  // namespace gbg
