// Discrete adjoint of the tumour-growth solve for MALA gradients of the
// imaging log-likelihood with respect to (Dw, rho, x0, y0, z0, T).
//
// Forward model (its own discretisation, smooth in the parameters): the
// reference's time loop has dt = dt(Dw) and an integer step count, so its
// output is piecewise constant in Dw and T. Here every sample of a call uses
// one fixed step dt0, n = ceil(T/dt0) steps, the last of length
// T - (n-1) dt0. Each step is the fast-path operator
//   v   = phi + a_k sum_f c_f (phi_f - phi) + b_k phi (1 - phi)
//   phi'= m * clamp(v, 0, 1)
// with a_k = dt_k Dw / (L^2 h^2), b_k = dt_k rho, unit face coefficients c_f
// (Case2 harmonic means with Dg = 0.1 Dw) and the tissue mask m, from the
// Gaussian initial density peak * exp(-|x - x0|^2 / (2 sigma^2)) on tissue.
// With float states the forward pass is the batched solver's on its smooth
// time grid (gbg_batch_opts.dt0): the same coefficient tables, schedule,
// initial densities and operation order, so log L agrees bit for bit.
//
// Adjoint (L is symmetric, so L^T = L): with lambda = dlogL/dphi at step k+1,
//   mu_c     = m_c [0 <= v_c < 1] lambda_c
//   lambda_c'= mu_c (1 + b_k (1 - 2 phi_c)) + a_k sum_f c_f (mu_f - mu_c)
//   dlogL/da_k = sum_c mu_c L(phi)_c,  dlogL/db_k = sum_c mu_c phi_c (1 - phi_c)
// The clamp's derivative at v = 0 is taken from the right (cells at exactly 0
// respond to growth of their neighbours), at v = 1 from the left is dropped.
// The seed dlogL/dphi at the final state follows HGG_Likelihood's PET and
// T1/T2 terms (source/Likelihood/source/HGG_Likelihood.cpp:40-153):
//   PET: -(u - s PET) / sigma^2;  Ti: alpha'/alpha (y = 1) or -alpha'/(1 - alpha)
//   with alpha' = |d| / slope * exp(-d^2 / slope), d = u - uc.
// States are checkpointed every K steps and each segment is recomputed
// before its backward sweep. Templated on the state type: float (the
// production path) or double (used to check gradients against finite
// differences).
#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

#include "gbg_internal.cuh"

namespace gbg {
namespace {

// device memory the default checkpoint interval may take (checkpoints plus
// one segment's recomputed states)
constexpr double kAdjointBudget = 96e9;

__device__ __forceinline__ int wm(int i, int n) { return i == 0 ? n - 1 : i - 1; }
__device__ __forceinline__ int wp(int i, int n) { return i == n - 1 ? 0 : i + 1; }

template <typename Real>
__global__ void k_adj_tables(int n, const double *__restrict__ pw, const double *__restrict__ pg,
                             Real *__restrict__ cx, Real *__restrict__ cy, Real *__restrict__ cz,
                             Real *__restrict__ msk) {
    const size_t N = (size_t)n * n * n;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < N; c += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(c % n), y = (int)((c / n) % n), z = (int)(c / ((size_t)n * n));
        const size_t nn = n;
        const size_t nb[7] = {c, c - x + wp(x, n), c + ((size_t)wp(y, n) - y) * nn,
                              c + ((size_t)wp(z, n) - z) * nn * nn, c - x + wm(x, n),
                              c + ((size_t)wm(y, n) - y) * nn, c + ((size_t)wm(z, n) - z) * nn * nn};
        double k[4];
        bool all = true;
        for (int i = 0; i < 7; ++i) {
            const double b = pw[nb[i]] + pg[nb[i]];
            all = all && b > 0.0;
            if (i < 4) k[i] = b > 0.0 ? (pw[nb[i]] + (double)0.1f * pg[nb[i]]) / b : 0.0;
        }
        Real *dst[3] = {cx, cy, cz};
        for (int f = 0; f < 3; ++f) {
            const double s = k[0] + k[f + 1];
            dst[f][c] = (k[0] > 0.0 && k[f + 1] > 0.0 && s > 0.0) ? (Real)(2.0 * k[0] * k[f + 1] / s) : (Real)0;
        }
        msk[c] = all ? (Real)1 : (Real)0;
    }
}

struct Tabs {
    const void *cx, *cy, *cz, *msk;
};

// L(f)_c = sum_f c_f (f_nb - f_c)
// cell c of an n^3 field (n <= 1024, so every index fits 32 bits) -> x, y, z
__device__ __forceinline__ void decomp(int c, int n, int &x, int &y, int &z) {
    const int row = c / n;
    x = c - row * n;
    z = row / n;
    y = row - z * n;
}

template <typename Real>
__device__ __forceinline__ Real lap(const Real *f, const Real *cx, const Real *cy, const Real *cz, int n,
                                    int c, int x, int y, int z) {
    const int pl = n * n;
    const int cW = c - x + wm(x, n), cE = c - x + wp(x, n);
    const int cS = c + (wm(y, n) - y) * n, cN = c + (wp(y, n) - y) * n;
    const int cB = c + (wm(z, n) - z) * pl, cF = c + (wp(z, n) - z) * pl;
    const Real f0 = f[c];
    return cx[cW] * (f[cW] - f0) + cx[c] * (f[cE] - f0) + cy[cS] * (f[cS] - f0) + cy[c] * (f[cN] - f0) +
           cz[cB] * (f[cB] - f0) + cz[c] * (f[cF] - f0);
}

__device__ __forceinline__ float fma_r(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_r(double a, double b, double c) { return fma(a, b, c); }

// pre-clamp update v = phi + a L(phi) + b phi (1 - phi), in the batched
// solver's operation order (faces -x, +x, -y, +y, -z, +z)
template <typename Real>
__device__ __forceinline__ Real step_value(const Real *f, const Real *cx, const Real *cy, const Real *cz, int n,
                                           int c, int x, int y, int z, Real a, Real b) {
    const int pl = n * n;
    const int cW = c - x + wm(x, n), cE = c - x + wp(x, n);
    const int cS = c + (wm(y, n) - y) * n, cN = c + (wp(y, n) - y) * n;
    const int cB = c + (wm(z, n) - z) * pl, cF = c + (wp(z, n) - z) * pl;
    const Real f0 = f[c];
    Real lap = cx[cW] * (f[cW] - f0);
    lap = fma_r(cx[c], f[cE] - f0, lap);
    lap = fma_r(cy[cS], f[cS] - f0, lap);
    lap = fma_r(cy[c], f[cN] - f0, lap);
    lap = fma_r(cz[cB], f[cB] - f0, lap);
    lap = fma_r(cz[c], f[cF] - f0, lap);
    Real v = fma_r(a, lap, f0);
    return fma_r(b * f0, (Real)1 - f0, v);
}

template <typename Real>
__global__ void k_adj_ic(int n, int S, const gbg_sample *__restrict__ smp, double peak, double sigma,
                         const double *__restrict__ pw, const double *__restrict__ pg, Real *__restrict__ phi) {
    const int N = n * n * n;
    for (int s = blockIdx.y; s < S; s += gridDim.y)
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
        const size_t i = (size_t)s * N + c;
        int x, y, z;
        decomp(c, n, x, y, z);
        double v = 0.0;
        if (pw[c] + pg[c] > 0.0) {
            const double dx = x - smp[s].x0, dy = y - smp[s].y0, dz = z - smp[s].z0;
            const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
            v = __dmul_rn(peak, exp(__ddiv_rn(-d2, __dmul_rn(__dmul_rn(2.0, sigma), sigma))));
        }
        phi[i] = (Real)v;
    }
}

// one forward step for every active sample (a[s] < 0 marks a finished sample)
template <typename Real>
__global__ void k_adj_fwd(int n, int S, const Real *__restrict__ in, Real *__restrict__ out, Tabs t,
                          const double *__restrict__ a, const double *__restrict__ b) {
    const int N = n * n * n;
    const Real *cx = (const Real *)t.cx, *cy = (const Real *)t.cy, *cz = (const Real *)t.cz,
               *m = (const Real *)t.msk;
    for (int s = blockIdx.y; s < S; s += gridDim.y) {
        const Real *f = in + (size_t)s * N;
        Real *o = out + (size_t)s * N;
        const bool act = a[s] >= 0;
        const Real as = (Real)a[s], bs = (Real)b[s];
        for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
            if (!act) {
                o[c] = f[c];
                continue;
            }
            int x, y, z;
            decomp(c, n, x, y, z);
            Real v = step_value(f, cx, cy, cz, n, c, x, y, z, as, bs);
            v = v < (Real)0 ? (Real)0 : (v > (Real)1 ? (Real)1 : v);
            o[c] = m[c] != (Real)0 ? v : (Real)0;
        }
    }
}

template <typename Real>
__device__ __forceinline__ double block_sum(double v) {
    __shared__ double red[32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int j = 0; j < (int)(blockDim.x >> 5); ++j) t += red[j];
    return t;
}

// mu = m [0 <= v < 1] lambda, and this step's parameter sensitivities.
// grid: x over cells of one sample, y = sample
template <typename Real>
__global__ void k_adj_mu(int n, const Real *__restrict__ phi, const Real *__restrict__ lam, Real *__restrict__ mu,
                         Tabs t, const double *__restrict__ a, const double *__restrict__ b,
                         double *__restrict__ gA, double *__restrict__ gB) {
    const int N = n * n * n;
    const int s = blockIdx.y;
    const Real *cx = (const Real *)t.cx, *cy = (const Real *)t.cy, *cz = (const Real *)t.cz,
               *m = (const Real *)t.msk;
    const Real *f = phi + (size_t)s * N;
    // a thread's partial sums in Real (float: the FP64 pipe is narrow on this
    // GPU; a thread adds a few dozen terms), combined in double below
    Real sa = 0, sbb = 0;
    const bool act = a[s] >= 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
        const size_t i = (size_t)s * N + c;
        if (!act) {
            mu[i] = lam[i];
            continue;
        }
        int x, y, z;
        decomp(c, n, x, y, z);
        const Real p = f[c];
        const Real L = lap(f, cx, cy, cz, n, c, x, y, z);
        const Real v = step_value(f, cx, cy, cz, n, c, x, y, z, (Real)a[s], (Real)b[s]);
        const Real g = (m[c] != (Real)0 && v >= (Real)0 && v < (Real)1) ? (Real)1 : (Real)0;
        const Real u = g * lam[i];
        mu[i] = u;
        sa += u * L;
        sbb += u * p * ((Real)1 - p);
    }
    const double ta = block_sum<Real>((double)sa);
    const double tb = block_sum<Real>((double)sbb);
    if (threadIdx.x == 0 && act) {
        atomicAdd(gA + s, ta);
        atomicAdd(gB + s, tb);
    }
}

template <typename Real>
__global__ void k_adj_lam(int n, int S, const Real *__restrict__ phi, const Real *__restrict__ mu,
                          Real *__restrict__ lam, Tabs t, const double *__restrict__ a, const double *__restrict__ b) {
    const int N = n * n * n;
    const Real *cx = (const Real *)t.cx, *cy = (const Real *)t.cy, *cz = (const Real *)t.cz;
    for (int s = blockIdx.y; s < S; s += gridDim.y) {
        const Real *u = mu + (size_t)s * N;
        const Real *ps = phi + (size_t)s * N;
        Real *ls = lam + (size_t)s * N;
        const bool act = a[s] >= 0;
        const Real as = (Real)a[s], bs = (Real)b[s];
        for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
            if (!act) {
                ls[c] = u[c];
                continue;
            }
            int x, y, z;
            decomp(c, n, x, y, z);
            const Real p = ps[c];
            ls[c] = u[c] * ((Real)1 + bs * ((Real)1 - (Real)2 * p)) + as * lap(u, cx, cy, cz, n, c, x, y, z);
        }
    }
}

// dlogL/du at the final state: PET list, then the T list (two launches keep
// the order of additions fixed where a cell is in both lists)
template <typename Real>
__global__ void k_adj_seed_pet(int S, size_t N, int npet, const int *__restrict__ idx, const double *__restrict__ val,
                               double scale, double sigma2, const Real *__restrict__ phi, Real *__restrict__ lam) {
    const long total = (long)npet * S;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const size_t s = i / npet, c = idx[i % npet];
        const double u = phi[s * N + c];
        lam[s * N + c] = (Real)(-(u - scale * val[i % npet]) / sigma2);
    }
}

template <typename Real>
__global__ void k_adj_seed_ti(int S, size_t N, int nti, const int *__restrict__ idx, const double *__restrict__ y1,
                              const double *__restrict__ y2, double uc1, double uc2, double slope,
                              const Real *__restrict__ phi, Real *__restrict__ lam) {
    const long total = (long)nti * S;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const size_t s = i / nti;
        const int j = (int)(i % nti);
        const size_t c = idx[j];
        const double u = phi[s * N + c];
        double g = 0.0;
        for (int ti = 0; ti < 2; ++ti) {
            const double d = u - (ti == 0 ? uc1 : uc2);
            const double sg = d < 0 ? -1.0 : (d > 0 ? 1.0 : 0.0);
            const double e = exp(-d * d / slope);
            const double alpha = 0.5 + 0.5 * sg * (1. - e);
            const double dal = fabs(d) / slope * e;
            const double y = ti == 0 ? y1[j] : y2[j];
            g += (y == 1) ? dal / alpha : -dal / (1. - alpha);
        }
        lam[s * N + c] = (Real)((double)lam[s * N + c] + g);
    }
}

// lambda_0 off the live units, which adj_lanes_segment leaves out: from mu_0
struct RimLambda {
    const unsigned char *live;  // null: lambda_0 is stored everywhere
    int rows;                   // rows of a unit
    const float *mu, *cxs, *cy, *cz;
    const SampleRec *rec;
};
__device__ __forceinline__ float rim_lambda(const RimLambda &r, int n, int s, size_t i, float p, int c, int x, int y, int z) {
    const int pl = n * n;
    const size_t o = i - c;
    const float u0 = r.mu[i];
    const float *u = r.mu + o;
    const bool last = r.rec[s].nsteps == 1;
    const float a = last ? r.rec[s].a2 : r.rec[s].a, b = last ? r.rec[s].b2 : r.rec[s].b;
    const int cW = c - x + wm(x, n), cE = c - x + wp(x, n), cS = c + (wm(y, n) - y) * n, cN = c + (wp(y, n) - y) * n;
    const int cB = c + (wm(z, n) - z) * pl, cF = c + (wp(z, n) - z) * pl;
    float lu = fabsf(r.cxs[cW]) * (u[cW] - u0);
    lu = fmaf(fabsf(r.cxs[c]), u[cE] - u0, lu);
    lu = fmaf(r.cy[cS], u[cS] - u0, lu);
    lu = fmaf(r.cy[c], u[cN] - u0, lu);
    lu = fmaf(r.cz[cB], u[cB] - u0, lu);
    lu = fmaf(r.cz[c], u[cF] - u0, lu);
    return fmaf(a, lu, u0 * (1.0f + b * (1.0f - 2.0f * p)));
}

// dlogL/dx0 = sum_c lambda0_c * phi0_c * (x_c - x0) / sigma^2 (same for y0, z0)
template <typename Real>
__global__ void k_adj_ic_grad(int n, const gbg_sample *__restrict__ smp, double sigma, const Real *__restrict__ lam,
                              const Real *__restrict__ phi0,
                              double *__restrict__ gx, RimLambda rim, const int *__restrict__ box) {
    const size_t N = (size_t)n * n * n;
    const int s = blockIdx.y;
    double acc[3] = {0, 0, 0};
    // the rows of the initial support's box where one is given
    int y0 = 0, ny = n, z0 = 0, nz = n;
    if (box) {
        y0 = n - box[4 * s];
        ny = box[4 * s + 1] ? box[4 * s + 1] - y0 : 0;
        z0 = n - box[4 * s + 2];
        nz = box[4 * s + 3] ? box[4 * s + 3] - z0 : 0;
    }
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n * ny * nz; q += gridDim.x * blockDim.x) {
        const int c = q % n + n * (y0 + q / n % ny + n * (z0 + q / (n * ny)));
        const size_t i = (size_t)s * N + c;
        // a cell outside the initial support adds exactly zero: skip its FP64 work
        if (phi0[i] == (Real)0) continue;
        int x, y, z;
        decomp(c, n, x, y, z);
        const Real l0 = rim.live && rim.live[y / rim.rows * n + z] != 1 ? (Real)rim_lambda(rim, n, s, i, (float)phi0[i], c, x, y, z) : lam[i];
        const double w = (double)l0 * (double)phi0[i] / (sigma * sigma);
        acc[0] += w * (x - smp[s].x0);
        acc[1] += w * (y - smp[s].y0);
        acc[2] += w * (z - smp[s].z0);
    }
    for (int k = 0; k < 3; ++k) {
        const double t = block_sum<Real>(acc[k]);
        if (threadIdx.x == 0) atomicAdd(gx + 3 * s + k, t);
    }
}

// x over the cells of a sample, y over samples; about 16 CTAs per SM in all
dim3 grid_cells(const Handle &h, int S) {
    const size_t per = (h.N + 255) / 256;
    size_t gx = (size_t)h.num_sms * 16 / (size_t)std::max(S, 1);
    if (gx < 1) gx = 1;
    if (gx > per) gx = per;
    return dim3((unsigned)gx, (unsigned)std::min(S, 65535));
}

int grid_of(const Handle &h, size_t work) {
    const size_t blocks = (work + 255) / 256;
    const size_t cap = (size_t)h.num_sms * 16;
    return (int)(blocks < cap ? blocks : cap);
}

template <typename Real>
int run_adjoint(Handle &h, const gbg_sample *samples, int S, const gbg_adjoint_opts &o, double *loglik,
                double *grad) {
    const int n = h.n;
    const size_t N = h.N;
    const double hh = 1.0 / n, ih2 = 1.0 / (hh * hh), L2 = o.L * o.L;
    constexpr bool f32 = std::is_same<Real, float>::value;
    // per-sample schedule on the smooth time grid, from the batched solver's
    // schedule kernel (its float coefficients are the float path's a_k, b_k)
    std::vector<SampleRec> recs(S);
    {
        void *d = nullptr;
        const size_t bytes = S * (sizeof(gbg_sample) + sizeof(SampleRec)) + 256;
        GBG_CUDA_TRY(cudaMalloc(&d, bytes));
        gbg_sample *dsmp = (gbg_sample *)d;
        SampleRec *drec = (SampleRec *)((char *)d + bwork_align(S * sizeof(gbg_sample)));
        cudaError_t e = cudaMemcpyAsync(dsmp, samples, S * sizeof(gbg_sample), cudaMemcpyHostToDevice, h.stream);
        int rc = e == cudaSuccess ? launch_schedule_smooth(h, dsmp, S, o.L, o.dt0, drec) : GBG_ERR_CUDA;
        if (rc == GBG_OK &&
            (cudaMemcpyAsync(recs.data(), drec, S * sizeof(SampleRec), cudaMemcpyDeviceToHost, h.stream) != cudaSuccess ||
             cudaStreamSynchronize(h.stream) != cudaSuccess))
            rc = GBG_ERR_CUDA;
        cudaFree(d);
        if (rc) {
            set_error("adjoint: schedule failed");
            return rc;
        }
    }
    // samples ordered by step count, longest first, so that the samples still
    // running at step k are a prefix [0, A_k): every launch covers that prefix
    // only (a finished sample's state and adjoint are left where they are)
    {
        bool sorted = true;
        for (int s = 1; s < S; ++s) sorted = sorted && recs[s].nsteps <= recs[s - 1].nsteps;
        if (!sorted) {
            std::vector<int> perm(S);
            for (int s = 0; s < S; ++s) perm[s] = s;
            std::stable_sort(perm.begin(), perm.end(),
                             [&](int i, int j) { return recs[i].nsteps > recs[j].nsteps; });
            std::vector<gbg_sample> sp(S);
            for (int i = 0; i < S; ++i) sp[i] = samples[perm[i]];
            std::vector<double> ll(S), gg(grad ? 6 * (size_t)S : 0);
            const int rc = run_adjoint<Real>(h, sp.data(), S, o, ll.data(), grad ? gg.data() : nullptr);
            if (rc) return rc;
            for (int i = 0; i < S; ++i) {
                if (loglik) loglik[perm[i]] = ll[i];
                if (grad)
                    for (int j = 0; j < 6; ++j) grad[6 * (size_t)perm[i] + j] = gg[6 * (size_t)i + j];
            }
            return GBG_OK;
        }
    }
    std::vector<int> ns(S);
    std::vector<double> dtl(S);
    int nmax = 0;
    std::vector<double> dts(S);
    for (int s = 0; s < S; ++s) {
        const int k = recs[s].nsteps;
        ns[s] = k;
        dts[s] = recs[s].dt;
        dtl[s] = samples[s].tend - (k - 1) * dts[s];
        nmax = std::max(nmax, k);
    }
    // A[k] = samples still running at step k (ns[s] > k)
    std::vector<int> A(nmax + 1, 0);
    for (int k = 0; k <= nmax; ++k)
        while (A[k] < S && ns[A[k]] > k) ++A[k];
    if (f32) {
        if (int rc = fast_build_tables(h, (double)0.1f)) return rc;
    }
    // checkpoint interval: 50 steps by default (the MALA configuration's),
    // fewer when the checkpoints and a segment's states would pass
    // kAdjointBudget bytes, sqrt(steps) at the least memory
    int K = o.checkpoint_every;
    if (K <= 0) {
        K = 50;
        const double per = (double)S * N * sizeof(Real);
        if ((K + nmax / K + 1) * per > kAdjointBudget) K = std::max(1, (int)std::ceil(std::sqrt((double)nmax)));
    }
    // without a gradient only the forward pass runs: no checkpoints kept
    if (!grad) K = nmax + 1;
    const int nck = nmax / K + 1;
    const size_t segs = grad ? (size_t)std::max(K, 2) : 2;
    // the float forward sweep runs on the batched solver's population kernel,
    // one launch per checkpoint segment
    const bool pop_fwd = f32 && population_supported(n);
    // device working set: carved from the handle's grow-only workspace
    const size_t SN = (size_t)S * N;
    const size_t sizes[] = {f32 ? 0 : 4 * N * sizeof(Real), (size_t)nck * SN * sizeof(Real),
                            segs * SN * sizeof(Real), SN * sizeof(Real), SN * sizeof(Real), SN * sizeof(Real),
                            (size_t)nmax * S * sizeof(double), (size_t)nmax * S * sizeof(double),
                            (size_t)nmax * S * sizeof(double), (size_t)nmax * S * sizeof(double),
                            3 * S * sizeof(double), S * sizeof(gbg_sample), S * sizeof(gbg_lik_result),
                            2 * S * sizeof(SampleRec), S * sizeof(int), 4 * S * sizeof(int)};
    size_t total = 0;
    for (size_t b : sizes) total += bwork_align(b);
    if (h.adj_ws_bytes < total) {
        if (h.adj_ws) cudaFree(h.adj_ws);
        h.adj_ws = nullptr;
        h.adj_ws_bytes = 0;
        if (cudaMalloc(&h.adj_ws, total) != cudaSuccess) {
            cudaGetLastError();
            set_error("adjoint: device allocation failed");
            return GBG_ERR_NOMEM;
        }
        h.adj_ws_bytes = total;
    }
    void *parts[16];
    {
        char *q = (char *)h.adj_ws;
        for (int i = 0; i < 16; ++i) {
            parts[i] = q;
            q += bwork_align(sizes[i]);
        }
    }
    auto release = [] {};
    Real *tab = (Real *)parts[0];
    Real *ck = (Real *)parts[1];
    Real *seg = (Real *)parts[2];
    Real *lam = (Real *)parts[3];
    Real *mu = (Real *)parts[4];
    Real *fin = (Real *)parts[5];
    double *da = (double *)parts[6];
    double *db = (double *)parts[7];
    double *gA = (double *)parts[8];
    double *gB = (double *)parts[9];
    double *gX = (double *)parts[10];
    gbg_sample *dsm = (gbg_sample *)parts[11];
    gbg_lik_result *dlik = (gbg_lik_result *)parts[12];
    SampleRec *drec = (SampleRec *)parts[13], *dsorted = drec + S;
    int *drank = (int *)parts[14];
    int *dbox = (int *)parts[15];  // initial-support boxes (the skipping population kernel)
    // per-step coefficients; a < 0 marks a finished sample
    std::vector<double> ha((size_t)nmax * S), hb((size_t)nmax * S);
    for (int k = 0; k < nmax; ++k)
        for (int s = 0; s < S; ++s) {
            const bool last = k == ns[s] - 1;
            if (k >= ns[s]) {
                ha[(size_t)k * S + s] = -1.0;
                hb[(size_t)k * S + s] = 0.0;
            } else if (f32) {
                ha[(size_t)k * S + s] = last ? recs[s].a2 : recs[s].a;
                hb[(size_t)k * S + s] = last ? recs[s].b2 : recs[s].b;
            } else {
                const double dtk = last ? dtl[s] : dts[s];
                ha[(size_t)k * S + s] = dtk * (samples[s].Dw / L2) * ih2;
                hb[(size_t)k * S + s] = dtk * samples[s].rho;
            }
        }
    cudaStream_t st = h.stream;
    int rc = GBG_OK;
#define ADJ_TRY(expr)                                                        \
    do {                                                                     \
        cudaError_t _e = (expr);                                             \
        if (_e != cudaSuccess) {                                             \
            set_error(std::string(#expr) + ": " + cudaGetErrorString(_e));   \
            release();                                                       \
            return GBG_ERR_CUDA;                                             \
        }                                                                    \
    } while (0)
    ADJ_TRY(cudaMemcpyAsync(da, ha.data(), ha.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    ADJ_TRY(cudaMemcpyAsync(db, hb.data(), hb.size() * sizeof(double), cudaMemcpyHostToDevice, st));
    ADJ_TRY(cudaMemcpyAsync(dsm, samples, S * sizeof(gbg_sample), cudaMemcpyHostToDevice, st));
    ADJ_TRY(cudaMemsetAsync(gA, 0, (size_t)nmax * S * sizeof(double), st));
    ADJ_TRY(cudaMemsetAsync(gB, 0, (size_t)nmax * S * sizeof(double), st));
    ADJ_TRY(cudaMemsetAsync(gX, 0, 3 * S * sizeof(double), st));
    Tabs t{tab, tab + N, tab + 2 * N, tab + 3 * N};
    if (f32) {
        t = Tabs{h.cx, h.cy, h.cz, h.msk};
        ADJ_TRY(cudaMemsetAsync(dbox, 0, 4 * S * sizeof(int), st));
        rc = launch_gaussian_ic(h, dsm, S, o.ic_peak, o.ic_sigma, (float *)ck, dbox);
        if (rc) {
            release();
            return rc;
        }
    } else {
        k_adj_tables<Real><<<grid_of(h, N), 256, 0, st>>>(n, h.pw, h.pg, tab, tab + N, tab + 2 * N, tab + 3 * N);
        k_adj_ic<Real><<<grid_cells(h, S), 256, 0, st>>>(n, S, dsm, o.ic_peak, o.ic_sigma, h.pw, h.pg, ck);
        h.launches += 2;
    }
    // forward with checkpoints, each step over the samples still running; a
    // sample's final state is gathered into fin at the step it finishes
    auto finish = [&](const Real *from, int lo, int hi) -> cudaError_t {
        if (hi <= lo || from == fin) return cudaSuccess;
        return cudaMemcpyAsync(fin + (size_t)lo * N, from + (size_t)lo * N, (size_t)(hi - lo) * N * sizeof(Real),
                               cudaMemcpyDeviceToDevice, st);
    };
    ADJ_TRY(finish(ck, A[0], S));  // samples with no step keep the initial state
    if (pop_fwd) {
        // segment j: steps [jK, min(jK + K, nmax)) of the samples running at
        // jK, from checkpoint j in seg slot 0, seg slot 1 the second buffer
        Real *buf0 = seg, *buf1 = seg + SN;
        std::vector<SampleRec> srec(S);
        for (int j = 0; j * K < nmax; ++j) {
            const int k0 = j * K, k1 = std::min(nmax, k0 + K), act = A[k0];
            if (act <= 0) break;
            ADJ_TRY(cudaMemcpyAsync(buf0, ck + (size_t)j * SN, (size_t)act * N * sizeof(Real), cudaMemcpyDeviceToDevice,
                                    st));
            for (int s = 0; s < act; ++s) {
                SampleRec r = recs[s];
                r.nsteps = std::min(ns[s], k1) - k0;
                if (ns[s] > k1) {  // the segment ends before the sample's shortened last step
                    r.a2 = r.a;
                    r.b2 = r.b;
                }
                r.order = s;
                srec[s] = r;
            }
            ADJ_TRY(cudaMemcpyAsync(drec, srec.data(), (size_t)act * sizeof(SampleRec), cudaMemcpyHostToDevice, st));
            // the skipping kernel may run: checkpoint j's support lies within
            // the initial boxes grown by k0 cells, and it is zero on every
            // cell without the mask once a step has run; second buffer zeroed
            ADJ_TRY(cudaMemsetAsync(buf1, 0, (size_t)act * N * sizeof(Real), st));
            rc = population_steps(h, (float *)buf0, (float *)buf1, drec, dsorted, drank, act, 0, dbox, k0);
            if (rc) {
                release();
                return rc;
            }
            // samples that finish in this segment: their final states
            for (int s = A[k1]; s < act; ++s) {
                const Real *src = (((ns[s] - k0) & 1) ? buf1 : buf0) + (size_t)s * N;
                ADJ_TRY(cudaMemcpyAsync(fin + (size_t)s * N, src, N * sizeof(Real), cudaMemcpyDeviceToDevice, st));
            }
            // checkpoint j + 1: the samples still running took all K steps
            if (grad && k1 < nmax && A[k1] > 0)
                ADJ_TRY(cudaMemcpyAsync(ck + (size_t)(j + 1) * SN, ((K & 1) ? buf1 : buf0),
                                        (size_t)A[k1] * N * sizeof(Real), cudaMemcpyDeviceToDevice, st));
        }
    } else {
        Real *cur = ck;
        for (int k = 0; k < nmax; ++k) {
            Real *nxt;
            if (!grad)  // forward only: ping-pong through two segment slots
                nxt = (k + 1) == nmax ? fin : seg + (size_t)((k + 1) & 1) * S * N;
            else
                nxt = ((k + 1) % K == 0) ? ck + (size_t)((k + 1) / K) * S * N
                                         : ((k + 1) == nmax ? fin : seg + (size_t)((k + 1) % K) * S * N);
            k_adj_fwd<Real><<<grid_cells(h, A[k]), 256, 0, st>>>(n, A[k], cur, nxt, t, da + (size_t)k * S,
                                                                 db + (size_t)k * S);
            h.launches++;
            ADJ_TRY(finish(nxt, A[k + 1], A[k]));
            cur = nxt;
        }
    }
    // log-likelihood and its gradient at the final state
    {
        rc = std::is_same<Real, float>::value
                 ? lik_evaluate(h, (const float *)fin, nullptr, S, dlik)
                 : lik_evaluate(h, nullptr, (const double *)fin, S, dlik);
        if (rc) {
            release();
            return rc;
        }
        ADJ_TRY(cudaMemsetAsync(lam, 0, S * N * sizeof(Real), st));
        const ObsDevice &ob = h.obs;
        if (ob.n_pet > 0)
            k_adj_seed_pet<Real><<<grid_of(h, (size_t)ob.n_pet * S), 256, 0, st>>>(
                S, N, ob.n_pet, ob.pet_idx, ob.pet_val, ob.pet_scale, ob.pet_sigma2, fin, lam);
        if (ob.n_ti > 0)
            k_adj_seed_ti<Real><<<grid_of(h, (size_t)ob.n_ti * S), 256, 0, st>>>(
                S, N, ob.n_ti, ob.ti_idx, ob.t1_val, ob.t2_val, ob.t1_uc, ob.t2_uc, ob.slope, fin, lam);
        h.launches += 2;
    }
    if (!grad) {
        std::vector<gbg_lik_result> hl(S);
        ADJ_TRY(cudaMemcpyAsync(hl.data(), dlik, S * sizeof(gbg_lik_result), cudaMemcpyDeviceToHost, st));
        ADJ_TRY(cudaStreamSynchronize(st));
        release();
        for (int s = 0; s < S; ++s)
            if (loglik) loglik[s] = hl[s].total;
        return GBG_OK;
    }
    // backward, segment by segment, each step over the samples running at it
    const unsigned gcx = (unsigned)std::min<size_t>((N + 255) / 256, (size_t)h.num_sms * 4);
    // The float path at n = 128 on resident anatomy, where there are live units and
    // they fit the CTAs' shared memory (any do on a GB300): lambda in lam, mu in mu
    // and fin, whose final states the seed has read.
    const bool lanes = f32 && pop_fwd && adj_lanes_fit(h);
    if (lanes) {
        ADJ_TRY(cudaMemsetAsync(mu, 0, SN * sizeof(Real), st));
        ADJ_TRY(cudaMemsetAsync(fin, 0, SN * sizeof(Real), st));
    }
    std::vector<SampleRec> rrec(pop_fwd ? S : 0);
    for (int sgm = (nmax - 1) / K; sgm >= 0; --sgm) {
        const int k0 = sgm * K, k1 = std::min(nmax, k0 + K);
        // recompute states k0+1 .. k1-1 into seg[1..]
        ADJ_TRY(cudaMemcpyAsync(seg, ck + (size_t)sgm * S * N, (size_t)A[k0] * N * sizeof(Real),
                                cudaMemcpyDeviceToDevice, st));
        if (pop_fwd) {
            // one population launch keeping every state (slot mode): sample s
            // takes steps k0 .. min(ns[s] - 1, k1 - 1) - 1, all full steps (a
            // sample's shortened last step only feeds the likelihood); the
            // skipping kernel computes the tiles its rule keeps (the
            // checkpoint's support lies within the initial boxes grown by k0)
            // and writes zeros over the rest
            const int act = A[k0];
            int most = 0;
            for (int s = 0; s < act; ++s) {
                SampleRec r = recs[s];
                r.nsteps = std::min(ns[s] - 1, k1 - 1) - k0;
                r.a2 = r.a;
                r.b2 = r.b;
                r.order = s;
                rrec[s] = r;
                most = std::max(most, r.nsteps);
            }
            if (most > 0) {
                ADJ_TRY(cudaMemcpyAsync(drec, rrec.data(), (size_t)act * sizeof(SampleRec), cudaMemcpyHostToDevice,
                                        st));
                rc = population_steps(h, (float *)seg, (float *)seg, drec, dsorted, drank, act, SN, dbox, k0, !lanes);
                if (rc) {
                    release();
                    return rc;
                }
            }
        } else {
            for (int k = k0; k < k1 - 1; ++k) {
                k_adj_fwd<Real><<<grid_cells(h, A[k]), 256, 0, st>>>(n, A[k], seg + (size_t)(k - k0) * S * N,
                                                                     seg + (size_t)(k - k0 + 1) * S * N, t,
                                                                     da + (size_t)k * S, db + (size_t)k * S);
                h.launches++;
            }
        }
        if (lanes) {
            rc = adj_lanes_segment(h, A[k0], k0, k1, recs.data(), drec, (const float *)seg, SN, (float *)lam, (float *)mu, (float *)fin,
                                   S, gA, gB);
            if (rc) {
                release();
                return rc;
            }
        }
        for (int k = k1 - 1; k >= k0 && !lanes; --k) {
            const Real *phik = seg + (size_t)(k - k0) * S * N;
            const dim3 gC(gcx, (unsigned)A[k]);
            k_adj_mu<Real><<<gC, 256, 0, st>>>(n, phik, lam, mu, t, da + (size_t)k * S, db + (size_t)k * S,
                                               gA + (size_t)k * S, gB + (size_t)k * S);
            k_adj_lam<Real><<<grid_cells(h, A[k]), 256, 0, st>>>(n, A[k], phik, mu, lam, t,
                                                                 da + (size_t)k * S, db + (size_t)k * S);
            h.launches += 2;
        }
    }
    const RimLambda rim{lanes ? h.unit_live : nullptr, 2, (const float *)mu, h.cxs, h.cy, h.cz, drec};
    k_adj_ic_grad<Real><<<dim3(gcx, (unsigned)S), 256, 0, st>>>(n, dsm, o.ic_sigma, lam, ck, gX, rim, f32 ? dbox : nullptr);
    h.launches++;
    ADJ_TRY(cudaGetLastError());
    std::vector<double> hA((size_t)nmax * S), hB((size_t)nmax * S), hX(3 * S);
    std::vector<gbg_lik_result> hl(S);
    ADJ_TRY(cudaMemcpyAsync(hA.data(), gA, hA.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    ADJ_TRY(cudaMemcpyAsync(hB.data(), gB, hB.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    ADJ_TRY(cudaMemcpyAsync(hX.data(), gX, hX.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    ADJ_TRY(cudaMemcpyAsync(hl.data(), dlik, S * sizeof(gbg_lik_result), cudaMemcpyDeviceToHost, st));
    ADJ_TRY(cudaStreamSynchronize(st));
    release();
#undef ADJ_TRY
    // chain rule from the per-step sensitivities dlogL/da_k, dlogL/db_k,
    // a_k = dt_k Dw / (L^2 h^2), b_k = dt_k rho, with dt_k = dt for the full
    // steps and dt_l = tend - (k-1) dt for the last one (the step count is
    // piecewise constant). Fixed grid: dt does not depend on the parameters.
    // Scaled grid: dt = C h^2 / (6 Dw / L^2 + rho h^2 / 2), so
    // d dt / dDw = -dt (6 / L^2) / den and d dt / drho = -dt (h^2 / 2) / den.
    const bool scaled = o.dt0 < 0;
    for (int s = 0; s < S; ++s) {
        double gDw = 0.0, gRho = 0.0;
        const double Dw = samples[s].Dw, rho = samples[s].rho, dt = dts[s];
        double dtdDw = 0.0, dtdRho = 0.0;
        if (scaled) {
            const double den = 6.0 * Dw / L2 + 0.5 * rho / ih2;
            dtdDw = -dt * (6.0 / L2) / den;
            dtdRho = -dt * (0.5 / ih2) / den;
        }
        const double km1 = (double)(ns[s] - 1);
        for (int k = 0; k < ns[s]; ++k) {
            const bool last = k == ns[s] - 1;
            const double dtk = last ? dtl[s] : dt;
            const double dDw = last ? -km1 * dtdDw : dtdDw;   // d dt_k / dDw
            const double dRho = last ? -km1 * dtdRho : dtdRho;
            const double gA = hA[(size_t)k * S + s], gB = hB[(size_t)k * S + s];
            gDw += gA * (dDw * Dw + dtk) / L2 * ih2 + gB * dDw * rho;
            gRho += gA * dRho * Dw / L2 * ih2 + gB * (dRho * rho + dtk);
        }
        const int kl = ns[s] - 1;
        const double gT = hA[(size_t)kl * S + s] * samples[s].Dw / L2 * ih2 + hB[(size_t)kl * S + s] * samples[s].rho;
        double *g = grad + 6 * (size_t)s;
        g[0] = gDw;
        g[1] = gRho;
        g[2] = hX[3 * s];
        g[3] = hX[3 * s + 1];
        g[4] = hX[3 * s + 2];
        g[5] = gT;
        if (loglik) loglik[s] = hl[s].total;
    }
    return GBG_OK;
}

}  // namespace

int adjoint_grad(Handle &h, const gbg_sample *samples, int S, const gbg_adjoint_opts &o, double *loglik,
                 double *grad) {
    if (o.state_precision == GBG_PREC_F64) return run_adjoint<double>(h, samples, S, o, loglik, grad);
    return run_adjoint<float>(h, samples, S, o, loglik, grad);
}

}  // namespace gbg
