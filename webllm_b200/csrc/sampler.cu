// Temperature / top-k / top-p sampling of one logits row where it lies, so that a decode loop reads back four bytes per token
// instead of the row (600 KB for a vocabulary of 151936). The rules and their rounding points are those of sampleToken
// (src/infer/sampler.ts:38-78): x / T in f32, weights exp(x / T - max) rounded to f32, candidates by descending weight and
// ascending index, the cut where the running share of the whole vocabulary's weight reaches top_p, then the first candidate at
// which the running sum reaches u times the kept sum.
//
// Three launches, 39 us for 151936 logits, 28 of them the last one's (the host's sort of the whole vocabulary took 38 ms): the maximum; the
// weights, their sum and a histogram of their leading bits, which bounds the k-th largest; one block that collects the few
// candidates above that bound, sorts them in shared memory and walks them in order.
#include "common.cuh"

namespace wb {

constexpr int kBlocks = 128, kHistShift = 18, kHistBins = (0x3f800000 >> kHistShift) + 1;  // weights are in [0, 1]
constexpr int kCandidates = 2048;  // what the last block can sort
constexpr int kTopKMax = 1024;

struct SampleScratch {
    float *w;          // [V] weights
    double *sums;      // [kBlocks]
    float *maxima;     // [kBlocks], NaN where a block saw one
    unsigned *hist;    // [kHistBins]
};

__device__ __forceinline__ float nan_max(float a, float b) { return (a != a || b != b) ? __int_as_float(0x7fc00000) : fmaxf(a, b); }

__global__ void __launch_bounds__(512) sample_max_kernel(const float *__restrict__ x, int V, SampleScratch s)
{
    pdl_sync();
    __shared__ float red[16];
    float m = -INFINITY;
    for (int i = blockIdx.x * 512 + threadIdx.x; i < V; i += kBlocks * 512) m = nan_max(m, x[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 16; i++) m = nan_max(m, red[i]);
        s.maxima[blockIdx.x] = m;
    }
    for (int i = blockIdx.x * 512 + threadIdx.x; i < kHistBins; i += kBlocks * 512) s.hist[i] = 0;
}

__device__ __forceinline__ float row_max(const SampleScratch &s)  // every thread of a block; a warp's worth of loads
{
    float m = -INFINITY;
    for (int i = threadIdx.x & 31; i < kBlocks; i += 32) m = nan_max(m, s.maxima[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = nan_max(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}

__global__ void __launch_bounds__(512) sample_weights_kernel(const float *__restrict__ x, int V, float T, SampleScratch s)
{
    pdl_sync();
    __shared__ double red[16];
    __shared__ unsigned hist[kHistBins];
    for (int i = threadIdx.x; i < kHistBins; i += 512) hist[i] = 0;
    const float m = __fdiv_rn(row_max(s), T);
    __syncthreads();
    double sum = 0.;
    for (int i = blockIdx.x * 512 + threadIdx.x; i < V; i += kBlocks * 512) {
        const float w = __double2float_rn(exp((double)__fsub_rn(__fdiv_rn(x[i], T), m)));
        s.w[i] = w;
        sum += (double)w;
        const unsigned bin = __float_as_uint(w) >> kHistShift;
        if (bin < (unsigned)kHistBins) atomicAdd(&hist[bin], 1u);  // (a NaN has no bin; the last kernel refuses the row)
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 16; i++) sum += red[i];
        s.sums[blockIdx.x] = sum;
    }
    for (int i = threadIdx.x; i < kHistBins; i += 512)
        if (hist[i]) atomicAdd(&s.hist[i], hist[i]);
}

// out[0] = the token, or -1 when the row is not for this kernel (NaN or infinite maximum, too many candidates of one weight)
__global__ void __launch_bounds__(1024) sample_pick_kernel(int V, int limit, double top_p, double u, SampleScratch s, volatile int *out)
{
    pdl_sync();
    __shared__ unsigned long long cand[kCandidates];
    __shared__ unsigned above[1024];
    __shared__ int bound, count, total_in;
    const int tid = threadIdx.x;
    const float m = row_max(s);
    // bins from the top: thread t holds the counts of bins [kHistBins - 4 t - 4, kHistBins - 4 t); an inclusive scan finds the
    // first bin at which at least `limit` weights are covered
    unsigned c[4], mine = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int b = kHistBins - 1 - (4 * tid + i);
        c[i] = b >= 0 ? s.hist[b] : 0;
        mine += c[i];
    }
    above[tid] = mine;
    if (tid == 0) bound = 0, count = 0, total_in = 0;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const unsigned v = tid >= o ? above[tid - o] : 0;
        __syncthreads();
        above[tid] += v;
        __syncthreads();
    }
    unsigned before = above[tid] - mine;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (before < (unsigned)limit && before + c[i] >= (unsigned)limit) bound = kHistBins - 1 - (4 * tid + i), total_in = (int)(before + c[i]);
        before += c[i];
    }
    __syncthreads();
    if (!(fabsf(m) < INFINITY) || total_in > kCandidates || total_in < limit) {
        if (tid == 0) *out = -1;
        return;
    }
    for (int i = tid; i < kCandidates; i += 1024) cand[i] = ~0ull;
    __syncthreads();
    const unsigned low = (unsigned)bound << kHistShift;
    const int V4 = V / 4;
    auto take = [&](float w, int i) {
        const unsigned bits = __float_as_uint(w);
        if (bits < low) return;
        const int at = atomicAdd(&count, 1);
        if (at < kCandidates) cand[at] = ((unsigned long long)(~bits) << 32) | (unsigned)i;  // ascending: weight down, index up
    };
#pragma unroll 4
    for (int i = tid; i < V4; i += 1024) {
        const float4 w = reinterpret_cast<const float4 *>(s.w)[i];
        take(w.x, 4 * i), take(w.y, 4 * i + 1), take(w.z, 4 * i + 2), take(w.w, 4 * i + 3);
    }
    for (int i = 4 * V4 + tid; i < V; i += 1024) take(s.w[i], i);
    __syncthreads();
    int size = 32;
    while (size < total_in) size <<= 1;
    for (int k = 2; k <= size; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < size; i += 1024) {
                const int p = i ^ j;
                if (p > i) {
                    const unsigned long long a = cand[i], b = cand[p];
                    if ((a > b) == ((i & k) == 0)) cand[i] = b, cand[p] = a;
                }
            }
            __syncthreads();
        }
    if (tid != 0) return;
    auto weight = [&](int i) { return (double)__uint_as_float(~(unsigned)(cand[i] >> 32)); };
    int kept = limit;
    if (top_p < 1.) {
        double total = 0., cum = 0.;
        for (int i = 0; i < kBlocks; i++) total += s.sums[i];
        for (int i = 0; i < limit; i++) {
            cum += weight(i) / total;
            if (cum >= top_p) {
                kept = i + 1;
                break;
            }
        }
    }
    double sum = 0., acc = 0.;
    for (int i = 0; i < kept; i++) sum += weight(i);
    const double r = u * sum;
    int pick = kept - 1;
    for (int i = 0; i < kept; i++) {
        acc += weight(i);
        if (acc >= r) {
            pick = i;
            break;
        }
    }
    *out = (int)(unsigned)cand[pick];
}

}  // namespace wb

using namespace wb;

extern "C" int wb_sample_token(wb_context *ctx, uint64_t logits_offset, int64_t vocab, float temperature, int64_t top_k, double top_p,
                               double u, int32_t *token)
{
    if (!ctx || !token) return fail(WB_ERR_BAD_ARG, "wb_sample_token: NULL argument");
    WB_CUDA(cudaSetDevice(ctx->device));
    WB_NOT_RECORDING(ctx, "wb_sample_token");
    if (vocab <= 0 || !(temperature > 0.f)) return fail(WB_ERR_BAD_ARG, "wb_sample_token: vocab and temperature must be positive");
    if (top_k < 1 || (top_k > kTopKMax && vocab > kTopKMax)) return fail(WB_ERR_UNSUPPORTED, "wb_sample_token: top_k must be 1 to %d", kTopKMax);
    if (logits_offset % 16) return fail(WB_ERR_BAD_ARG, "wb_sample_token: the logits must be 16-byte aligned");
    WB_CHECK(check_range(ctx, WB_ARENA_ACT, logits_offset, (uint64_t)vocab * 4, "wb_sample_token"));
    const uint64_t w_bytes = align_up((uint64_t)vocab * 4);
    if (w_bytes + 64 * 1024 > kWorkspaceBytes) return fail(WB_ERR_OOM, "wb_sample_token: vocabulary too large");
    SampleScratch s;
    s.w = (float *)ctx->workspace;
    s.sums = (double *)(ctx->workspace + w_bytes), s.maxima = (float *)(s.sums + kBlocks), s.hist = (unsigned *)(s.maxima + kBlocks);
    const float *x = (const float *)arena_ptr(ctx, WB_ARENA_ACT, logits_offset);
    const int V = (int)vocab, limit = (int)(top_k < vocab ? top_k : vocab);
    volatile int *out = ctx->status_host + 1;  // the word behind the status word, pinned and mapped
    WB_CUDA(launch_pdl(sample_max_kernel, dim3(kBlocks), dim3(512), 0, ctx->stream, x, V, s));
    WB_CUDA(launch_pdl(sample_weights_kernel, dim3(kBlocks), dim3(512), 0, ctx->stream, x, V, temperature, s));
    WB_CUDA(launch_pdl(sample_pick_kernel, dim3(1), dim3(1024), 0, ctx->stream, V, limit, top_p, u, s, (volatile int *)(ctx->status_word + 1)));
    ctx->launches += 3;
    WB_CHECK(wb_synchronize(ctx));
    *token = *out;
    return WB_OK;
}
