// Backward steps of the float adjoint at n = 128 with resident anatomy (see
// rd_lanes.cu): a lane takes a sample through all backward steps of a
// checkpoint segment, so that lambda and mu stay in L2 and only the recomputed
// states come from HBM. Step k, on the live units:
//   mu_k     = [m and 0 <= v < 1] lambda_{k+1},  v = the update before its clamp
//   lambda_k = mu_k (1 + b (1 - 2 phi_k)) + a L(mu_k)
// mu_k alternates between two buffers, so one barrier per step, between the
// two, is enough: a CTA that is past it has its neighbours' mu_k, and no one
// still reads the buffer mu_{k-1} goes to. lambda is read and written by the
// thread that owns the cell.
// A block is the part of a row pair's 16 planes 16 zb .. 16 zb + 15 that is
// live. A thread adds its row's sensitivity products over a block in float, in
// plane order, and widens them once. Blocks are dealt to the CTAs one by one, two
// per CTA on an ellipsoidal brain, one per warp with 4 lanes.
// 64 samples near the mode at 128^3: the backward kernels 34 ms, the whole call
// 52.4 ms, where a kernel that read halo tiles (8 rows x 16 planes, a block
// barrier per plane) took 56 and 86.3 ms.
#include <algorithm>
#include <vector>

#include "lanes.cuh"

namespace gbg {
namespace {
using namespace lanes;

constexpr int LR = 32, n = 128, plane = n * n, N = n * n * n;
constexpr int kBlockZ = 16, kBlocks = (n / 2) * (n / kBlockZ);
// Four lanes of two warps with 255 registers each, and two planes ahead. Eight
// lanes of two warps leave no registers for the second plane, and their
// samples' lambda, mu (twice) and states (the step's and the next one's) do not
// stay in L2 together: 59.6 ms for the call below (on other samples), against
// 56.5 with four; eight lanes of one warp 64, four lanes with three planes ahead
// (spilled) 65.
constexpr int kAdjWarps = 8, kAdjThreads = 32 * kAdjWarps, kAdjLanes = 4;
constexpr int kMaxBlocks = kMaxUnits / kBlockZ;  // per CTA

struct AdjArgs {
    int S, T, lanes, warps, k0, k1, nblocks, strideS;
    size_t slot;
    const float *seg;
    float *lam, *mu[2];
    const float *cxs, *cy, *cz;
    const SampleRec *rec;
    const int *list;
    unsigned *sync;
    int *status;
    double *gA, *gB;
};

// row y's y neighbours relative to the row pair y, y + 1
__device__ __forceinline__ int south(int y) { return y == 0 ? n * (n - 1) : -n; }
__device__ __forceinline__ int north2(int y) { return y + 2 == n ? -n * (n - 2) : 2 * n; }

// L of one row (the order of march_tile_s); r: its right-face fluxes' shuffles
__device__ __forceinline__ V4 lap_row(const V4 &P, const V4 &DS, float sS, const V4 &DT, const V4 &DB, const V4 &DF, const V4 &CX,
                                      const V4 &CYm, const V4 &CY, const V4 &CZp, const V4 &CZ, int li) {
    const float right = __shfl_sync(0xffffffffu, P.v[0], (li + 1) % LR, LR);
    const float d[4] = {P.v[1] - P.v[0], P.v[2] - P.v[1], P.v[3] - P.v[2], right - P.v[3]};
    const float flux = __shfl_sync(0xffffffffu, fabsf(CX.v[3]) * d[3], (li + LR - 1) % LR, LR);
    V4 o;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float lap = i ? -fabsf(CX.v[i - 1]) * d[i - 1] : -flux;
        lap = fmaf(fabsf(CX.v[i]), d[i], lap);
        lap = fmaf(sS * CYm.v[i], DS.v[i], lap);
        lap = fmaf(CY.v[i], DT.v[i], lap);
        lap = fmaf(-CZp.v[i], DB.v[i], lap);
        lap = fmaf(CZ.v[i], DF.v[i], lap);
        o.v[i] = lap;
    }
    return o;
}

// Planes z .. z + len - 1 of the row pair y, y + 1, f's stencil and the own
// cells' second operand g: MU: f = phi, g = lambda, out = mu, products added to
// acc; otherwise f = mu, g = phi, out = lambda. pre != 0: the cells pre floats
// from g's are brought to L2 (the next step's state).
template <bool MU>
__device__ __forceinline__ void sweep(const float4 *__restrict__ tab, int y, int z, int len, const float *__restrict__ f,
                                      const float *g, float *out, const float *__restrict__ cz, float a, float b, long pre, float (&acc)[4]) {
    const int li = threadIdx.x & 31;
    const int o0 = 4 * li + n * y + plane * z, below = z == 0 ? plane * (n - 1) : -plane, dS = south(y), dT = north2(y);
    const float *pN = f + o0;  // the plane last loaded
    out += o0;
    g += o0;
    int zn = z;
    // Registers in rings, as in the population kernel: the rows of planes j ..
    // j + 2, the rows beside them and the second operand of planes j and j + 1,
    // the difference and the face to the plane before.
    V4 X0[3], X1[3], S[2], T[2], G0[2], G1[2], B0[2], B1[2], C0[2], C1[2];
    auto load_st = [&](int d) {  // of the plane pN is on; then to the next plane
        S[d] = ldp(pN + dS);
        T[d] = ldp(pN + dT);
        pN += ++zn == n ? -plane * (n - 1) : plane;
    };
    X0[0] = ldp(pN);
    X1[0] = ldp(pN + n);
    B0[0] = ldp(pN + below);
    B1[0] = ldp(pN + below + n);
    C0[0] = ldg4(cz + o0 + below);
    C1[0] = ldg4(cz + o0 + below + n);
#pragma unroll
    for (int d = 0; d < 2; ++d)
        if (d < len) {
            load_st(d);
            X0[d + 1] = ldp(pN);
            X1[d + 1] = ldp(pN + n);
            G0[d] = ldp(g + d * plane);
            G1[d] = ldp(g + d * plane + n);
        }
    B0[0] = sub(X0[0], B0[0]);
    B1[0] = sub(X1[0], B1[0]);
    auto finish = [&](const V4 &P, const V4 &lap, const V4 &CX, const V4 &G, int r) {
        float o[4], pa = 0.0f, pb = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f0 = P.v[i];
            if (MU) {
                float v = fmaf(a, lap.v[i], f0);
                v = fmaf(b * f0, 1.0f - f0, v);
                const float gate = (!signbit(CX.v[i]) && v >= 0.0f && v < 1.0f) ? 1.0f : 0.0f;
                o[i] = gate * G.v[i];
                pa = fmaf(o[i], lap.v[i], pa);
                pb = fmaf(o[i] * f0, 1.0f - f0, pb);
            } else {
                o[i] = fmaf(a, lap.v[i], f0 * (1.0f + b * (1.0f - 2.0f * G.v[i])));
            }
        }
        if (MU) {
            acc[2 * r] += pa;
            acc[2 * r + 1] += pb;
        }
        *reinterpret_cast<float4 *>(out + r * n) = make_float4(o[0], o[1], o[2], o[3]);
    };
    for (int j = 0; j < len; j += 6) {
#pragma unroll
        for (int d = 0; d < 6; ++d) {
            if (j + d >= len) break;
            const V4 &P0 = X0[d % 3], &P1 = X1[d % 3], &N0 = X0[(d + 1) % 3], &N1 = X1[(d + 1) % 3];
            const int h = d & 1;
            const V4 DY = sub(P1, P0), Y1 = lds(tab + 3 * 32), CX0 = lds(tab);
            if (pre) {
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(g + pre));
                asm volatile("prefetch.global.L2 [%0];\n" ::"l"(g + pre + n));
            }
            B0[h ^ 1] = sub(N0, P0);
            C0[h ^ 1] = lds(tab + 5 * 32);
            finish(P0, lap_row(P0, sub(S[h], P0), 1.f, DY, B0[h], B0[h ^ 1], CX0, lds(tab + 2 * 32), Y1, C0[h], C0[h ^ 1], li), CX0, G0[h], 0);
            __syncwarp();
            const V4 CX1 = lds(tab + 32);
            B1[h ^ 1] = sub(N1, P1);
            C1[h ^ 1] = lds(tab + 6 * 32);
            finish(P1, lap_row(P1, DY, -1.f, sub(T[h], P1), B1[h], B1[h ^ 1], CX1, Y1, lds(tab + 4 * 32), C1[h], C1[h ^ 1], li), CX1, G1[h], 1);
            __syncwarp();
            if (j + d + 2 < len) {
                load_st(h);
                X0[d % 3] = ldp(pN);
                X1[d % 3] = ldp(pN + n);
                G0[h] = ldp(g + 2 * plane);
                G1[h] = ldp(g + 2 * plane + n);
            }
            g += plane;
            out += plane;
            tab += kSlots * 32;
        }
    }
}

struct Job {
    SampleRec rec;
    Lane lane;
};

__global__ void __launch_bounds__(kAdjThreads, 1) k_adj_lanes(AdjArgs p) {
    extern __shared__ __align__(16) float4 tab[];
    __shared__ Job s_job[kAdjLanes];
    __shared__ int s_blk[kMaxBlocks], s_at[kMaxBlocks + 1];  // rows | zb << 8 | planes << 16; first unit's table
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = blockIdx.x;
    const int nb = rank < p.nblocks ? (p.nblocks - rank - 1) / p.T + 1 : 0;  // blocks rank, rank + T, ...
    if (threadIdx.x == 0) {
        int at = 0;
        for (int i = 0; i < nb; ++i) {
            s_blk[i] = p.list[rank + i * p.T];
            s_at[i] = at;
            at += __popc((unsigned)s_blk[i] >> 16);
        }
        s_at[nb] = at;
    }
    __syncthreads();
    for (int i = 0; i < nb; ++i) {
        const int blk = s_blk[i], y0 = 2 * (blk & 255), z0 = kBlockZ * (blk >> 8 & 255);
        const unsigned mask = (unsigned)blk >> 16;
        for (int q = warp; q < kBlockZ * kSlots; q += kAdjThreads / 32) {
            const int j = q / kSlots, c = q % kSlots;
            if (!(mask >> j & 1u)) continue;
            int y = y0 + (c < 2 ? c : (c < 5 ? c - 3 : c - 5));
            y = y < 0 ? n - 1 : y;
            const float *src = c < 2 ? p.cxs : (c < 5 ? p.cy : p.cz);
            tab[((s_at[i] + __popc(mask & ((1u << j) - 1u))) * kSlots + c) * 32 + lane] =
                *reinterpret_cast<const float4 *>(src + 4 * lane + n * y + plane * (z0 + j));
        }
    }
    __syncthreads();
    const int g = warp / p.warps, w = warp % p.warps;
    if (g >= p.lanes) return;  // named barriers only from here on
    Job &jb = s_job[g];
    const bool lead = w == 0 && lane == 0;
    if (lead) jb.lane = Lane{g, 1, 0u, 0u};
    for (;;) {
        group_sync(1 + g, 32 * p.warps);
        const int s = jb.lane.next;
        if (s >= p.S || !jb.lane.ok) break;
        if (lead) jb.rec = p.rec[s];
        group_sync(1 + g, 32 * p.warps);
        const int ns = jb.rec.nsteps, top = min(ns, p.k1);
        if (top <= p.k0) break;  // sorted: so are all that follow
        float *lam = p.lam + (size_t)s * N;
        for (int k = top - 1; k >= p.k0; --k) {
            const bool last = k == ns - 1;
            const float a = last ? jb.rec.a2 : jb.rec.a, b = last ? jb.rec.b2 : jb.rec.b;
            const float *phi = p.seg + (size_t)(k - p.k0) * p.slot + (size_t)s * N;
            float *mu = p.mu[k & 1] + (size_t)s * N;
            for (int phase = 0; phase < 2; ++phase) {
                for (int i = w; i < nb; i += p.warps) {
                    const int blk = s_blk[i], y = 2 * (blk & 255), z0 = kBlockZ * (blk >> 8 & 255);
                    const float4 *t = tab + s_at[i] * kSlots * 32 + lane;
                    unsigned m = (unsigned)blk >> 16;
                    float acc[4] = {0.f, 0.f, 0.f, 0.f};
                    for (int z = z0; m;) {
                        const int skip = __ffs(m) - 1;
                        m >>= skip;
                        const int len = __ffs(~m) - 1;  // m is at most 16 bits
                        if (phase == 0)
                            sweep<true>(t, y, z + skip, len, phi, lam, mu, p.cz, a, b, 0, acc);
                        else
                            sweep<false>(t, y, z + skip, len, mu, phi, lam, p.cz, a, b, k > p.k0 ? -(long)p.slot : 0, acc);
                        t += len * kSlots * 32;
                        z += skip + len;
                        m >>= len;
                    }
                    if (phase == 0) {
                        double sa = (double)acc[0] + (double)acc[2], sb = (double)acc[1] + (double)acc[3];
                        for (int o = 16; o > 0; o >>= 1) {
                            sa += __shfl_down_sync(0xffffffffu, sa, o);
                            sb += __shfl_down_sync(0xffffffffu, sb, o);
                        }
                        if (lane == 0) {
                            atomicAdd(p.gA + (size_t)k * p.strideS + s, sa);
                            atomicAdd(p.gB + (size_t)k * p.strideS + s, sb);
                        }
                    }
                }
                if (phase) break;
                group_sync(1 + g, 32 * p.warps);
                if (lead)
                    lane_barrier(jb.lane, p.sync + (size_t)(g + 1) * kSyncStride, p.sync, p.T, rank, p.lanes, k == p.k0, p.status);
                group_sync(1 + g, 32 * p.warps);
                if (!jb.lane.ok) break;
            }
            if (!jb.lane.ok) break;
        }
    }
}

// blocks with a live unit: rows | zb << 8 | live planes << 16, in order, and their
// number (one CTA of kBlocks threads)
__global__ void __launch_bounds__(kBlocks) k_block_list(const unsigned char *__restrict__ live, int *__restrict__ list, int *__restrict__ count) {
    __shared__ int sums[kBlocks / 32];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, yp = t / (n / kBlockZ), zb = t % (n / kBlockZ);
    unsigned mask = 0;
    for (int j = 0; j < kBlockZ; ++j) mask |= (live[yp * n + zb * kBlockZ + j] == 1 ? 1u : 0u) << j;
    const unsigned m = __ballot_sync(0xffffffffu, mask != 0);
    if (lane == 0) sums[warp] = __popc(m);
    __syncthreads();
    int before = 0;
    for (int k = 0; k < warp; ++k) before += sums[k];
    if (mask) list[before + __popc(m & ((1u << lane) - 1u))] = yp | zb << 8 | (int)(mask << 16);
    if (t == kBlocks - 1) *count = before + __popc(m);
}

}  // namespace

bool adj_lanes_list(Handle &h, int *count) {
    if (h.n != n || !reserve_device({{(void **)&h.block_list, kBlocks * sizeof(int)}})) return false;
    k_block_list<<<1, kBlocks, 0, h.stream>>>(h.unit_live, h.block_list, count);
    h.launches++;
    return true;
}

bool adj_lanes_fit(const Handle &h) {
    return h.n == n && h.block_list && h.units[3] > 0 && (h.units[3] + h.num_sms - 1) / h.num_sms <= kMaxBlocks;
}

int adj_lanes_segment(Handle &h, int S, int k0, int k1, const SampleRec *recs, SampleRec *drec, const float *seg, size_t slot,
                      float *lam, float *mu0, float *mu1, int strideS, double *gA, double *gB) {
    AdjArgs a;
    a.S = S;
    a.T = std::min(h.num_sms, h.units[3]);
    a.lanes = std::min(kAdjLanes, S);
    a.warps = kAdjWarps / a.lanes;
    a.k0 = k0;
    a.k1 = k1;
    a.nblocks = h.units[3];
    a.strideS = strideS;
    a.slot = slot;
    a.seg = seg;
    a.lam = lam;
    a.mu[0] = mu0;
    a.mu[1] = mu1;
    a.cxs = h.cxs;
    a.cy = h.cy;
    a.cz = h.cz;
    a.rec = drec;
    a.list = h.block_list;
    a.sync = h.lane_sync;
    a.status = h.dev_status;
    a.gA = gA;
    a.gB = gB;
    const size_t smem = (size_t)((h.units[3] + a.T - 1) / a.T) * kBlockZ * kUnitBytes;
    GBG_CUDA_TRY(cudaMemcpyAsync(drec, recs, (size_t)S * sizeof(SampleRec), cudaMemcpyHostToDevice, h.stream));
    GBG_CUDA_TRY(cudaFuncSetAttribute(k_adj_lanes, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes));
    GBG_CUDA_TRY(cudaMemsetAsync(h.lane_sync, 0, (size_t)(a.lanes + 1) * kSyncStride * sizeof(unsigned), h.stream));
    void *args[] = {&a};
    GBG_CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_adj_lanes, dim3((unsigned)a.T), dim3(kAdjThreads), args, smem, h.stream));
    h.launches++;
    return GBG_OK;
}

}  // namespace gbg
