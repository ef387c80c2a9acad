// Posterior propagation statistics: per-cell mean and variance of S density
// fields, as the reference's propagation tool computes them over the
// samples' HGG_data.dat files (Glioma_HG_Propagation::_ic_PatientCasePropagation,
// source/Glioma/Glioma_HG_Propagation.cpp:346-440, then PropagationStatistics,
// Glioma_PropagationStatisticsOperator.h:24-50), in its default Real = float:
//   m = sum_s u_s                      (float, samples in order)
//   v = sum_s (u_s - m / S')^2         (float; m / S' = (1/S as float) * m)
//   mean = m * (1/S), var = v * (1/S)  (float)
// where a field value enters as the double it was written as, so each sum
// step is a double operation rounded to float. With reference_rules, cells
// with a zero x, y or z index keep mean = var = 0: the tool accumulates only
// mapped indices in (0, size] (:380-384, :432).
//
// The second sum needs the first one finished, so a CTA takes 32 to 256
// neighbouring cells, brings their values of all samples into shared memory
// and adds from there, a thread per cell in sample order. Reading every field
// twice took 1.30 ms for 512 fields of 128^3 (0.97 of the copy rate on twice
// the bytes), once takes 0.93 ms: the three CTAs an SM holds do not cover the
// copies of one with the serial sums of the others (16 cells per CTA, with
// 64-byte copies: 1.63 ms; 64 cells, one CTA per SM: 1.49 ms; a second read
// from L2 instead, of as many cells as it holds: 1.5 ms). Compiled with
// -fmad=false: every product and sum rounds on its own. The double sums
// rounded to float are float sums: 53 bits are more than 2 x 24 + 2, so the
// second rounding never changes the first one's result.
#include "gbg_internal.cuh"

namespace gbg {
namespace {

struct FieldSource {
    const float *f0, *f1;     // fields of sample s at s * N in f0, or in f1 when
    const SampleRec *recs;    // recs is non-null and recs[s].nsteps is odd
    __device__ __forceinline__ const float *field(int s, size_t N) const {
        const float *b = (recs && (recs[s].nsteps & 1)) ? f1 : f0;
        return b + (size_t)s * N;
    }
};

__global__ void k_field_stats(int n, int S, FieldSource src, int reference_rules, float *__restrict__ mean,
                              float *__restrict__ var) {
    const size_t N = (size_t)n * n * n;
    const float inv = (float)(1. / S);
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < N; c += (size_t)gridDim.x * blockDim.x) {
        const int x = (int)(c % n), y = (int)((c / n) % n), z = (int)(c / ((size_t)n * n));
        if (reference_rules && (x == 0 || y == 0 || z == 0)) {
            mean[c] = 0.0f;
            var[c] = 0.0f;
            continue;
        }
        float m = 0.0f;
        for (int s = 0; s < S; ++s) m = (float)((double)m + (double)src.field(s, N)[c]);
        const float p = __fmul_rn(inv, m);
        float v = 0.0f;
        for (int s = 0; s < S; ++s) {
            const float t = (float)((double)src.field(s, N)[c] - (double)p);
            v = __fadd_rn(v, __fmul_rn(t, t));
        }
        mean[c] = __fmul_rn(m, inv);
        var[c] = __fmul_rn(v, inv);
    }
}

constexpr int kStatThreads = 256;
constexpr size_t kStatBytes = 72 * 1024;  // values of a CTA: three CTAs per SM

// f(u[0]), f(u[C]), .. of S values in order, in batches whose loads go out
// together: the additions are a serial chain, and one that waits for a batch of
// 16 each time took 1.04 ms for 512 samples, of 96 0.94 (and the 64 cells of
// 250 samples 0.434 and 0.410).
template <int C, int N, class F>
__device__ __forceinline__ void batches(const float *u, int &s, int S, F f) {
    for (; s + N <= S; s += N) {
        float a[N];
#pragma unroll
        for (int k = 0; k < N; ++k) a[k] = u[(s + k) * C];
#pragma unroll
        for (int k = 0; k < N; ++k) f(a[k]);
    }
}
template <int C, class F>
__device__ __forceinline__ void in_order(const float *u, int S, F f) {
    int s = 0;
    batches<C, 96>(u, s, S, f);
    batches<C, 16>(u, s, S, f);
    batches<C, 4>(u, s, S, f);
    batches<C, 1>(u, s, S, f);
}

// C cells per CTA; W cells per copy: 4 where N is a multiple of 4 and the
// fields are 16-byte aligned, else 1
template <int C, int W>
__global__ void __launch_bounds__(kStatThreads) k_field_stats_once(int n, int S, FieldSource src, int reference_rules,
                                                                  float *__restrict__ mean, float *__restrict__ var) {
    extern __shared__ __align__(16) float s_val[];  // [sample][cell]
    constexpr int PER = C / W, ROWS = kStatThreads / PER;  // copies of a sample's cells, samples per sweep
    const size_t N = (size_t)n * n * n, c0 = (size_t)blockIdx.x * C;
    const int live = N - c0 < (size_t)C ? (int)(N - c0) : C, cc = threadIdx.x % PER * W;
    if (cc < live) {  // W divides N: a copy is inside or outside
        unsigned dst = (unsigned)__cvta_generic_to_shared(s_val + threadIdx.x / PER * C + cc);
#pragma unroll 4
        for (int s = threadIdx.x / PER; s < S; s += ROWS, dst += ROWS * C * sizeof(float))
            asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(src.field(s, N) + c0 + cc), "n"(4 * W)
                         : "memory");
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    if ((int)threadIdx.x >= live) return;
    const size_t c = c0 + threadIdx.x;
    const int x = (int)(c % n), y = (int)((c / n) % n), z = (int)(c / ((size_t)n * n));
    if (reference_rules && (x == 0 || y == 0 || z == 0)) {
        mean[c] = 0.0f;
        var[c] = 0.0f;
        return;
    }
    const float inv = (float)(1. / S), *u = s_val + threadIdx.x;
    float m = 0.0f;
    in_order<C>(u, S, [&](float x) { m = __fadd_rn(m, x); });
    const float p = __fmul_rn(inv, m);
    float v = 0.0f;
    in_order<C>(u, S, [&](float x) {
        const float t = __fsub_rn(x, p);
        v = __fadd_rn(v, __fmul_rn(t, t));
    });
    mean[c] = __fmul_rn(m, inv);
    var[c] = __fmul_rn(v, inv);
}

template <int C>
int launch_once(cudaStream_t st, int n, int S, const FieldSource &src, int reference_rules, float *mean, float *var) {
    const size_t N = (size_t)n * n * n, sm = (size_t)C * S * sizeof(float);
    const bool wide = N % 4 == 0 && ((uintptr_t)src.f0 | (uintptr_t)src.f1) % 16 == 0;
    auto *fn = wide ? k_field_stats_once<C, 4> : k_field_stats_once<C, 1>;
    if (sm > 48 * 1024) GBG_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStatBytes));
    fn<<<(unsigned)((N + C - 1) / C), kStatThreads, sm, st>>>(n, S, src, reference_rules, mean, var);
    GBG_CUDA_TRY(cudaGetLastError());
    return GBG_OK;
}

int launch_stats(int num_sms, cudaStream_t st, int n, int S, const FieldSource &src, int reference_rules,
                 float *mean, float *var) {
    const size_t N = (size_t)n * n * n;
    // Below 16 samples the second read is from L1 and the CTAs of the other form
    // have little to cover their copies with: 8 of 128^3 23.2 against 32.7 us, 12 31.4
    // and 34.4, 16 34.8 and 36.5, 24 49.2 and 47.1 (all 2 us more from HBM, where 16
    // take 43.0 and 38.9). Otherwise the most cells whose values fit; more samples
    // than fit with 32 cells (576) read the fields twice.
    const size_t fit = S < 16 ? 0 : kStatBytes / ((size_t)S * sizeof(float));
    if (fit >= 256) return launch_once<256>(st, n, S, src, reference_rules, mean, var);
    if (fit >= 128) return launch_once<128>(st, n, S, src, reference_rules, mean, var);
    if (fit >= 64) return launch_once<64>(st, n, S, src, reference_rules, mean, var);
    if (fit >= 32) return launch_once<32>(st, n, S, src, reference_rules, mean, var);
    size_t blocks = (N + 255) / 256;
    const size_t cap = (size_t)(num_sms > 0 ? num_sms : 132) * 8;
    if (blocks > cap) blocks = cap;
    k_field_stats<<<(unsigned)blocks, 256, 0, st>>>(n, S, src, reference_rules, mean, var);
    GBG_CUDA_TRY(cudaGetLastError());
    return GBG_OK;
}

}  // namespace

int batch_statistics(Handle &h, const gbg_sample *samples_device, int S, const gbg_batch_opts &o,
                     int reference_rules, float *mean_device, float *var_device) {
    if (int rc = batch_solve_device(h, samples_device, S, o, nullptr, nullptr)) return rc;
    FieldSource src{h.bphi[0], h.bphi[1], batch_unsorted(h)};
    h.launches++;
    return launch_stats(h.num_sms, h.stream, h.n, S, src, reference_rules, mean_device, var_device);
}

}  // namespace gbg

extern "C" int gbg_field_statistics(int n, const float *fields_device, int S, int reference_rules,
                                    float *mean_device, float *var_device, void *stream) {
    if (n < 1 || n > 1024 || S < 1 || !fields_device || !mean_device || !var_device) {
        gbg::set_error("gbg_field_statistics: bad argument");
        return GBG_ERR_ARG;
    }
    int dev = 0, sms = 0;
    GBG_CUDA_TRY(cudaGetDevice(&dev));
    GBG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    gbg::FieldSource src{fields_device, fields_device, nullptr};
    return gbg::launch_stats(sms, static_cast<cudaStream_t>(stream), n, S, src, reference_rules, mean_device,
                             var_device);
}
