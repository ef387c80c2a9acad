// The skipping population kernel with resident anatomy (the batched solver's
// default). A step of the tumour model needs 4 bytes of density and 16 bytes
// of face coefficients per cell from the neighbourhood of that cell; the
// tile-march kernel of rd_fast.cu advances every sample of a population once
// per round and so streams both through L2 for each step (at 128^3 with 512
// samples it ran at 0.67 of the HBM copy rate, and neither deeper staging nor
// wider tiles moved it). Here nothing but the density moves:
//   * The grid's live units (a unit: 2 rows per lane segment of one z-plane,
//     full x-rows, holding at least one cell with the mask) are dealt once to
//     the CTAs of a team, one CTA per SM. A CTA keeps the face coefficients of
//     its units in shared memory for the whole launch (3.5 KB per unit: 93 KB
//     at 128^3 on an ellipsoidal brain, 194 KB if every unit is live).
//   * A team advances up to 8 samples side by side, one per "lane" of warps.
//     A lane takes its sample through all its steps before the next one, so
//     only the samples in flight are hot: 8 x 2 buffers of the live units fit
//     in L2, and HBM sees a sample's first and last state only.
//   * The lanes of a CTA are independent: each has its own barrier among the
//     team's CTAs, and while one lane waits for its barrier (2.5 us from the
//     last store to the release) the others have the SM.
//   * A warp marches its share of units up z, two rows in registers, with the
//     loads of the next planes in flight.
// What bounds it: a warp's latencies (16 warps an SM, of which a fifth waits at
// a barrier; L1's data path is 67 % busy, 28 of the 58 passes a unit takes
// through it are coefficients, and instructions issue in 47 % of the cycles),
// and, for one sample, the barrier.
// Per-cell operations and their order are those of march_tile_s (a difference
// taken the other way round is its exact negative), so every population
// kernel gives the same bits. Measured on a GB300, before (tile march) and
// now: 512 prior draws at 128^3 243 -> 150 ms; 64 draws near the mode, stable
// grid, 14.7 -> 9.5 ms; one of them 1.04 -> 0.62 ms; 512 at 64^3 51 -> 24.5 ms.
#include <algorithm>
#include <type_traits>

#include "lanes.cuh"

namespace gbg {
namespace {
using namespace lanes;

// At 32^3 a step is little but its barrier. While there are clusters of 16 SMs for
// all samples, a team is one and its barrier goes through shared memory: 0.33
// instead of 0.39 ms for 6 samples near the mode. Beyond that (7 on a GB300) waiting
// for a cluster costs more (16 samples 0.61 against 0.45), and clusters of 8 or 4
// gain nothing (0.38 and 0.43 for 6).
constexpr int kClusterTeam = 16;

struct LaneArgs {
    int S, T, teams, lanes, warps, cluster;
    int nlive, units, grow0;
    size_t stride, slot;  // slot: floats between kept states (kernels with KEEP)
    float *buf0, *buf1;
    const float *cxs, *cy, *cz;
    const SampleRec *rec;
    const int *list, *fill;  // live units; units KEEP writes zeros in (nfill of them)
    int nfill;
    const unsigned char *live;
    const int *box;
    unsigned *sync;   // queue counter, then per lane: arrivals, next sample (two slots)
    int *status;
    unsigned long long *visited;
};

// what a lane's warps share of the sample they are on
struct Sample {
    SampleRec rec;
    int ylo, yhi, zlo, zhi, any;  // the initial support, and whether there is one: without, the sample stays 0
    Lane lane;
};

// One row of four cells. DS = sS * (row(y-1) - P), DT = row(y+1) - P,
// DB = P - plane(z-1), DF = plane(z+1) - P.
template <int LR>
__device__ __forceinline__ float4 row_step(const V4 &P, const V4 &DS, float sS, const V4 &DT, const V4 &DB, const V4 &DF, const V4 &CX,
                                           const V4 &CYm, const V4 &CY, const V4 &CZp, const V4 &CZ, int li, float a, float b) {
    const float right = __shfl_sync(0xffffffffu, P.v[0], (li + 1) % LR, LR);
    const float d[4] = {P.v[1] - P.v[0], P.v[2] - P.v[1], P.v[3] - P.v[2], right - P.v[3]};
    // the left face of cell 0 is the right face of the lane before: the same
    // two cells' difference times the same coefficient
    const float flux = __shfl_sync(0xffffffffu, fabsf(CX.v[3]) * d[3], (li + LR - 1) % LR, LR);
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float f0 = P.v[i];
        float lap = i ? -fabsf(CX.v[i - 1]) * d[i - 1] : -flux;
        lap = fmaf(CX.v[i], d[i], lap);  // of either sign where the cell's result is dropped
        lap = fmaf(sS * CYm.v[i], DS.v[i], lap);
        lap = fmaf(CY.v[i], DT.v[i], lap);
        lap = fmaf(-CZp.v[i], DB.v[i], lap);
        lap = fmaf(CZ.v[i], DF.v[i], lap);
        const float v = fmaf(a, lap, f0);
        o[i] = __saturatef(fmaf(b * f0, 1.0f - f0, v));
        o[i] = signbit(CX.v[i]) ? 0.0f : o[i];
    }
    return make_float4(o[0], o[1], o[2], o[3]);
}

// Planes z .. z + len - 1 of the row pair y, y + 1. tab: the first unit's
// table at this lane.
template <int LR>
__device__ __forceinline__ void march(const float4 *__restrict__ tab, int y, int z, int len, const float *__restrict__ in,
                                      float *__restrict__ out, const float *__restrict__ cz, float a, float b) {
    constexpr int n = 4 * LR, plane = n * n;
    const int li = (threadIdx.x & 31) % LR;
    const int o0 = 4 * li + n * y + plane * z, below = z == 0 ? plane * (n - 1) : -plane;
    const float *pN = in + o0;  // the plane last loaded
    int dS = y == 0 ? n * (n - 1) : -n, dT = y + 2 == n ? -n * (n - 2) : 2 * n;
    out += o0;
    // Registers in rings, so that no plane's values are moved: the rows of
    // planes j .. j + 2, the rows below and above them of planes j and j + 1,
    // the difference and the face to the plane before. Unrolled by the rings'
    // common period. (Moving them plane by plane, and taking the coefficients'
    // magnitude in masked cells too: 232 instructions a unit instead of 204,
    // 164 ms instead of 150 on the population above.)
    V4 X0[kAhead + 1], X1[kAhead + 1], S[kAhead], T[kAhead], B0[2], B1[2], C0[2], C1[2];
    int zn = z;
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
    for (int d = 0; d < kAhead; ++d)
        if (d < len) {
            load_st(d);
            X0[d + 1] = ldp(pN);
            X1[d + 1] = ldp(pN + n);
        }
    B0[0] = sub(X0[0], B0[0]);
    B1[0] = sub(X1[0], B1[0]);
    constexpr int kPeriod = 2 * (kAhead + 1);
    static_assert(kAhead == 2, "the rings' common period");
    for (int j = 0; j < len; j += kPeriod) {
#pragma unroll
        for (int d = 0; d < kPeriod; ++d) {
            if (j + d >= len) break;
            constexpr int R = kAhead + 1;
            const V4 &P0 = X0[d % R], &P1 = X1[d % R], &N0 = X0[(d + 1) % R], &N1 = X1[(d + 1) % R];
            const int h = d & 1, q = d % kAhead;
            C0[h ^ 1] = lds(tab + 5 * 32);
            const V4 Y1 = lds(tab + 3 * 32);
            const V4 DY = sub(P1, P0);
            B0[h ^ 1] = sub(N0, P0);
            B1[h ^ 1] = sub(N1, P1);
            *reinterpret_cast<float4 *>(out) = row_step<LR>(P0, sub(S[q], P0), 1.f, DY, B0[h], B0[h ^ 1], lds(tab), lds(tab + 2 * 32), Y1,
                                                            C0[h], C0[h ^ 1], li, a, b);
            __syncwarp();
            C1[h ^ 1] = lds(tab + 6 * 32);
            *reinterpret_cast<float4 *>(out + n) = row_step<LR>(P1, DY, -1.f, sub(T[q], P1), B1[h], B1[h ^ 1], lds(tab + 32), Y1,
                                                                lds(tab + 4 * 32), C1[h], C1[h ^ 1], li, a, b);
            __syncwarp();
            out += plane;
            tab += kSlots * 32;
            if (j + d + kAhead < len) {
                load_st(q);
                X0[d % R] = ldp(pN);
                X1[d % R] = ldp(pN + n);
            }
        }
    }
}

// KEEP: every state is kept (step k reads buf0 + k * slot, writes buf0 + (k + 1)
// * slot) over arbitrary older contents, so the live units outside the grown
// support and the units of the fill list are written with zeros.
template <int LR, int WPS, bool KEEP, bool CLUSTER>
__global__ void __launch_bounds__(128 * WPS, 1) k_population10(LaneArgs p) {
    constexpr int n = 4 * LR, SUB = 32 / LR, ROWS = 2 * SUB;
    extern __shared__ __align__(16) float4 tab[];
    __shared__ int s_unit[kMaxUnits];  // y0 | z << 10 | length of the run of planes from here on << 20
    __shared__ Sample s_smp[kMaxLanes];
    __shared__ unsigned long long s_bar[kMaxLanes];  // CLUSTER: the lanes' barriers
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, li = lane % LR, sub_r = lane / LR;
    const int team = blockIdx.x / p.T, rank = blockIdx.x % p.T;
    // this CTA's units: two stretches of the list, half the list apart
    const int q0 = (int)((long)p.nlive * rank / (2 * p.T)), c0 = (int)((long)p.nlive * (rank + 1) / (2 * p.T)) - q0;
    const int q1 = (int)((long)p.nlive * (rank + p.T) / (2 * p.T)), c1 = (int)((long)p.nlive * (rank + p.T + 1) / (2 * p.T)) - q1;
    const int nu = c0 + c1;
    auto unit_at = [&](int i) { return p.list[i < c0 ? q0 + i : q1 + i - c0]; };  // yu * n + z
    for (int i = threadIdx.x; i < nu; i += 128 * WPS) {
        const int u = unit_at(i), end = i < c0 ? c0 : nu;
        int run = 1;
        while (i + run < end && unit_at(i + run) == u + run && (u + run) % n != 0) ++run;
        s_unit[i] = (u / n) * ROWS | (u % n) << 10 | run << 20;  // all below 1024
    }
    // the units' face coefficients, one float4 per lane and slot
    for (int q = warp; q < nu * kSlots; q += 4 * WPS) {
        const int u = unit_at(q / kSlots), c = q % kSlots, z = u % n;
        int y = (u / n) * ROWS + 2 * sub_r + (c < 2 ? c : (c < 5 ? c - 3 : c - 5));
        y = y < 0 ? n - 1 : y;
        const float *src = c < 2 ? p.cxs : (c < 5 ? p.cy : p.cz);
        tab[q * 32 + lane] = *reinterpret_cast<const float4 *>(src + 4 * li + (size_t)n * (y + (size_t)n * z));
    }
    if (CLUSTER) {
        if (threadIdx.x < kMaxLanes)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(s_bar + threadIdx.x)), "r"(p.T)
                         : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    __syncthreads();
    const int g = warp / p.warps, w = warp % p.warps;
    // named barriers only from here on, and the cluster's at the end
    if (g < p.lanes) {
        Sample &sm = s_smp[g];
        const int tl = g * p.teams + team;
        if (w == 0 && lane == 0) {
            sm.lane = Lane{tl, 1, 0u, 0u};
        }
        unsigned visited = 0;
        for (;;) {
            group_sync(1 + g, 32 * p.warps);
            const int r = sm.lane.next;
            if (r >= p.S || !sm.lane.ok) break;
            if (w == 0 && lane == 0) {
                sm.rec = p.rec[r];
                const int4 bx = reinterpret_cast<const int4 *>(p.box)[sm.rec.order];
                sm.ylo = n - bx.x;
                sm.yhi = bx.y - 1;
                sm.zlo = n - bx.z;
                sm.zhi = bx.w - 1;
                sm.any = bx.y != 0;
            }
            group_sync(1 + g, 32 * p.warps);
            const int nsteps = sm.rec.nsteps;
            if (nsteps <= 0) break;  // sorted: so are all that follow
            for (int k = 0; k < nsteps; ++k) {
                {
                    const size_t off = (size_t)sm.rec.order * p.stride;
                    const float *in = (KEEP ? p.buf0 + (size_t)k * p.slot : ((k & 1) ? p.buf1 : p.buf0)) + off;
                    float *out = (KEEP ? p.buf0 + (size_t)(k + 1) * p.slot : ((k & 1) ? p.buf0 : p.buf1)) + off;
                    auto zero = [&](int y0, int z) {  // unit (row group y0, plane z) of the output
                        float *o = out + 4 * li + (size_t)n * (y0 + 2 * sub_r + (size_t)n * z);
                        *reinterpret_cast<float4 *>(o) = make_float4(0.f, 0.f, 0.f, 0.f);
                        *reinterpret_cast<float4 *>(o + n) = make_float4(0.f, 0.f, 0.f, 0.f);
                    };
                    const bool lastk = k == nsteps - 1;
                    const float a = lastk ? sm.rec.a2 : sm.rec.a, b = lastk ? sm.rec.b2 : sm.rec.b;
                    const bool any = sm.any;
                    const int grow = p.grow0 + k + 1, u1 = nu * (w + 1) / p.warps;
                    for (int i = nu * w / p.warps; (KEEP || any) && i < u1;) {
                        const int un = s_unit[i], y0 = un & 1023, z = un >> 10 & 1023, len = min(un >> 20, u1 - i);
                        int za = z, zb = z + len;
                        if (sm.zlo >= grow && sm.zhi + grow < n) {
                            za = max(za, sm.zlo - grow);
                            zb = min(zb, sm.zhi + grow + 1);
                        }
                        if (!any || !span_hits(sm.ylo, sm.yhi, grow, y0, y0 + ROWS - 1, n)) zb = za;
                        if (za < zb) {
                            march<LR>(tab + (i + za - z) * kSlots * 32 + lane, y0 + 2 * sub_r, za, zb - za, in, out, p.cz, a, b);
                            visited += zb - za;
                        }
                        if (KEEP)
                            for (int q = z; q < z + len; ++q)
                                if (q < za || q >= zb) zero(y0, q);
                        i += len;
                    }
                    if (KEEP) {
                        for (int i = rank + p.T * w; i < p.nfill; i += p.T * p.warps) zero(p.fill[i] / n * ROWS, p.fill[i] % n);
                    } else if (k == 1 && any) {
                        // units without a live cell that the initial state may have
                        // left values in: zeros, as their step gives
                        for (int u = rank + p.T * w; u < p.units; u += p.T * p.warps) {
                            const int y0 = (u / n) * ROWS, z = u % n;
                            if (p.live[u] != 1 && span_hits(sm.ylo, sm.yhi, p.grow0, y0, y0 + ROWS - 1, n) &&
                                span_hits(sm.zlo, sm.zhi, p.grow0, z, z, n))
                                zero(y0, z);
                        }
                    }
                }
                // barrier of the team's CTAs on this lane
                group_sync(1 + g, 32 * p.warps);
                if (w == 0 && lane == 0) {
                    unsigned *sync = p.sync + (size_t)(tl + 1) * kSyncStride;
                    if (CLUSTER)
                        cluster_barrier(sm.lane, s_bar + g, sync, p.sync, p.T, rank, p.teams * p.lanes, k == nsteps - 1, p.status);
                    else
                        lane_barrier(sm.lane, sync, p.sync, p.T, rank, p.teams * p.lanes, k == nsteps - 1, p.status);
                }
                if (k == nsteps - 1) break;
                group_sync(1 + g, 32 * p.warps);
                if (!sm.lane.ok) break;
            }
        }
        if (lane == 0 && visited) atomicAdd(p.visited, (unsigned long long)visited);
    }
    if (CLUSTER) {  // no CTA leaves while others may arrive at its barriers
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// live[u] = unit u (2 rows per lane segment, one plane, full x-rows; u = row
// group * n + plane) has a cell that is tissue with six tissue neighbours (the
// fast tables' mask)
__global__ void k_unit_live(int n, int rows, const double *__restrict__ pw, const double *__restrict__ pg,
                            unsigned char *__restrict__ live) {
    const int y0 = (blockIdx.x / n) * rows, z = blockIdx.x % n;
    int any = 0;
    for (int i = threadIdx.x; i < n * rows; i += blockDim.x) {
        const int x = i % n, y = y0 + i / n;
        auto t = [&](int xx, int yy, int zz) {
            const size_t c = xx + (size_t)n * (yy + (size_t)n * zz);
            return pw[c] + pg[c] > 0.0;
        };
        any |= t(x, y, z) && t(wrapm(x, n), y, z) && t(wrapp(x, n), y, z) && t(x, wrapm(y, n), z) && t(x, wrapp(y, n), z) &&
               t(x, y, wrapm(z, n)) && t(x, y, wrapp(z, n));
    }
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) live[blockIdx.x] = (unsigned char)(any != 0);
}

// live[u] = 2 for units without a live cell next to a live one (rows or planes)
__global__ void k_unit_rim(int n, int units, unsigned char *__restrict__ live) {
    const int u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= units || live[u] == 1) return;
    const int z = u % n, y = u / n, ny = units / n;
    if (live[y * n + wrapm(z, n)] == 1 || live[y * n + wrapp(z, n)] == 1 || live[wrapm(y, ny) * n + z] == 1 ||
        live[wrapp(y, ny) * n + z] == 1)
        live[u] = 2;
}

// Three lists of units in increasing order, a CTA each, and their lengths behind
// them: the live ones, those without a live cell that a live unit's stencil reads,
// all without a live cell.
__global__ void __launch_bounds__(1024) k_unit_lists(int units, const unsigned char *__restrict__ live, int *__restrict__ lists) {
    const int which = blockIdx.x;
    int *list = lists + which * units;
    __shared__ int sums[32];
    __shared__ int total;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    for (int base = 0; base < units; base += 1024) {
        const int i = base + threadIdx.x;
        const int f = i < units && (which == 2 ? live[i] != 1 : live[i] == which + 1);
        const unsigned m = __ballot_sync(0xffffffffu, f);
        if (lane == 0) sums[warp] = __popc(m);
        __syncthreads();
        int before = total;
        for (int k = 0; k < warp; ++k) before += sums[k];
        if (f) list[before + __popc(m & ((1u << lane) - 1u))] = i;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int k = 0; k < 32; ++k) total += sums[k];
        __syncthreads();
    }
    if (threadIdx.x == 0) lists[3 * units + which] = total;
}

int unit_rows(int n) { return 2 * (32 / (n / 4)); }
int units_of(int n) { return (n / unit_rows(n)) * n; }
}  // namespace

int lanes_set_anatomy(Handle &h) {
    if (!population_supported(h.n)) return GBG_OK;
    const int nu = units_of(h.n);
    // without room for the lists every call takes the tile march (lanes_fit)
    if (!reserve_device({{(void **)&h.unit_live, (size_t)nu},
                         {(void **)&h.unit_list, (3 * nu + 4) * sizeof(int)},
                         {(void **)&h.lane_sync, (size_t)(h.num_sms * kMaxLanes + 1) * kSyncStride * sizeof(unsigned)}}))
        return GBG_OK;
    if (h.n == 32 && h.lane_clusters < 0) {
        // how many clusters run side by side, at the most units a CTA of one owns
        const void *fn = (const void *)k_population10<8, kWps, false, true>;
        cudaLaunchConfig_t c = {};
        cudaLaunchAttribute at[1];
        c.gridDim = dim3(kClusterTeam);
        c.blockDim = dim3(kThreads);
        c.dynamicSmemBytes = 2 * ((nu + 2 * kClusterTeam - 1) / (2 * kClusterTeam)) * kUnitBytes;
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kClusterTeam;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        c.attrs = at;
        c.numAttrs = 1;
        h.lane_clusters = 0;
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes) != cudaSuccess ||
            cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&h.lane_clusters, fn, &c) != cudaSuccess) {
            cudaGetLastError();
            h.lane_clusters = 0;
        }
    }
    k_unit_live<<<nu, 128, 0, h.stream>>>(h.n, unit_rows(h.n), h.pw, h.pg, h.unit_live);
    k_unit_rim<<<(nu + 127) / 128, 128, 0, h.stream>>>(h.n, nu, h.unit_live);
    k_unit_lists<<<3, 1024, 0, h.stream>>>(nu, h.unit_live, h.unit_list);
    h.launches += 3;
    GBG_CUDA_TRY(cudaGetLastError());
    const bool blocks = adj_lanes_list(h, h.unit_list + 3 * nu + 3);
    // one copy of the lengths: each waits for the stream
    GBG_CUDA_TRY(cudaMemcpyAsync(h.units, h.unit_list + 3 * nu, (blocks ? 4 : 3) * sizeof(int), cudaMemcpyDeviceToHost, h.stream));
    return GBG_OK;
}

// Teams and lanes for S samples. A CTA holds at most 28 units where the chip
// allows it (more: 30.1 against 26.3 ms at 52 units for 512 samples at 64^3,
// fewer: 32.2 ms at 14, the lanes then idle at their barriers). Where samples
// are few the teams grow until 8 lanes each cover them, down to 4 units per
// CTA, below which a step is all barrier (6 samples at 32^3: 1.71 ms at 28
// units, 1.42 ms at 4; 32 at 64^3: 4.9 ms at 28, 4.0 ms at 14). A lane has no
// more warps than its CTA units, and at most 8: a warp that comes to the
// barrier without work costs the others more than it helps (one sample at
// 32^3: 0.41 ms with 16 warps, 0.35 with 4; at 64^3 0.47 and 0.43; at 128^3
// 0.635 with 16, 0.62 with 8 warps, 0.70 with 4).
static void lane_shape(const Handle &h, int S, LaneArgs &a, int &units) {
    const int nl = std::max(1, h.units[0]), sms = h.num_sms;
    const int wide = sms / ((S + kMaxLanes - 1) / kMaxLanes), least = (nl + 27) / 28, most = (nl + 3) / 4;
    a.T = std::min(sms, std::max(least, std::min(wide, most)));
    a.teams = sms / a.T;
    a.T = sms / a.teams;
    a.cluster = h.n == 32 && S <= h.lane_clusters;
    if (a.cluster) {
        a.T = kClusterTeam;
        a.teams = S;
    }
    a.teams = std::min(a.teams, S);
    a.lanes = std::min(kMaxLanes, (S + a.teams - 1) / a.teams);
    units = 2 * ((nl + 2 * a.T - 1) / (2 * a.T));
    a.warps = std::min({4 * kWps / a.lanes, units, 8});
}

bool lanes_fit(const Handle &h, int S) {
    LaneArgs a;
    int units;
    if (!h.unit_list) return false;
    lane_shape(h, S, a, units);
    return units <= kMaxUnits;
}

int lanes_launch(Handle &h, float *buf0, float *buf1, const SampleRec *sorted, int S, const int *box, int grow0, size_t slot,
                 bool fill_all) {
    const int n = h.n;
    LaneArgs a;
    int units;
    lane_shape(h, S, a, units);
    a.S = S;
    a.nlive = h.units[0];
    a.units = units_of(n);
    a.grow0 = grow0;
    a.stride = h.N;
    a.buf0 = buf0;
    a.buf1 = buf1;
    a.cxs = h.cxs;
    a.cy = h.cy;
    a.cz = h.cz;
    a.rec = sorted;
    a.list = h.unit_list;
    a.fill = h.unit_list + (fill_all ? 2 : 1) * a.units;
    a.nfill = h.units[fill_all ? 2 : 1];
    a.slot = slot;
    a.live = h.unit_live;
    a.box = box;
    a.sync = h.lane_sync;
    a.status = h.dev_status;
    a.visited = reinterpret_cast<unsigned long long *>(h.barrier + 2);
    const size_t smem = units * kUnitBytes;
    auto kernel = [&](auto keep) {
        constexpr bool K = decltype(keep)::value;
        return n == 128    ? (const void *)k_population10<32, kWps, K, false>
               : n == 64   ? (const void *)k_population10<16, kWps, K, false>
               : a.cluster ? (const void *)k_population10<8, kWps, K, true>
                           : (const void *)k_population10<8, kWps, K, false>;
    };
    const void *fn = slot ? kernel(std::true_type{}) : kernel(std::false_type{});
    GBG_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kTableBytes));
    GBG_CUDA_TRY(cudaMemsetAsync(h.barrier, 0, 4 * sizeof(unsigned), h.stream));
    GBG_CUDA_TRY(
        cudaMemsetAsync(h.lane_sync, 0, (size_t)(a.teams * a.lanes + 1) * kSyncStride * sizeof(unsigned), h.stream));
    h.pop_tile_cells = (long long)unit_rows(n) * n;
    void *args[] = {&a};
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GBG_CUDA_TRY(cudaStreamIsCapturing(h.stream, &cap));
    const unsigned evf = cap == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : cudaEventRecordDefault;
    GBG_CUDA_TRY(cudaEventRecordWithFlags(h.ev_pop[0], h.stream, evf));
    if (a.cluster) {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3((unsigned)(a.teams * a.T));
        c.blockDim = dim3(kThreads);
        c.dynamicSmemBytes = smem;
        c.stream = h.stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = a.T;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        c.attrs = at;
        c.numAttrs = 1;
        GBG_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        GBG_CUDA_TRY(cudaLaunchKernelExC(&c, fn, args));
    } else {
        GBG_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3((unsigned)(a.teams * a.T)), dim3(kThreads), args, smem, h.stream));
    }
    GBG_CUDA_TRY(cudaEventRecordWithFlags(h.ev_pop[1], h.stream, evf));
    h.ev_pop_recorded = true;
    h.launches++;
    return GBG_OK;
}

}  // namespace gbg
