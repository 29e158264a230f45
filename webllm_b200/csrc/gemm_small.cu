// int4 GEMM of a small batch on a large matrix: up to 16 rows, whole 128-k chunks and 32-column tiles (the served batches between the GEMV and the
// tcgen05 GEMM). Same contract as gemm_tc.cu: fp16 operands, f32 accumulation, f32 activations rounded to fp16 when they are
// staged (gemm_nt_f16_from_f32.wgsl:58-62).
//
// At these row counts the work is to read the weights once (7B-class layer: 120 MB, 19 us of HBM time) and the tcgen05 kernel is
// bound by something else: every weight goes through shared memory twice on its way into the operand tile, after a launch that
// casts the activations and before one that adds K slices. Here, as in gemv_stream.cu, a packed word goes from global
// memory into a register and from there, as fp16 subnormals, into the warp-level MMA whose 16-row operand is the weight; the rows of
// the batch are the 8 columns of the other operand, two blocks of them, read from shared memory once for 32 columns of the weight.
//   * A CTA has 256 / WK columns (a warp 32) and one slice of K; two CTAs an SM. WK = 2 gives the halves of the slice to two
//     sets of warps, for matrices with few columns.
//   * The activations of the slice are staged once, in the order of the MMA's k-slots; the first chunks of the weight are
//     requested before that and before the wait on the previous kernel.
//   * All nibbles are shifted to the low position (7 instructions a word), so one set of accumulators does for the even and odd ones.
//   * The K slices of a column tile meet in the workspace: the last one to arrive adds them in slice order. No second launch.
// Measured, f32 activations, M = 16, tcgen05 kernel with its two extra launches -> this: 3584 -> 18944 24.4 -> 17.3 us, 18944 -> 3584
// 28.1 -> 24.4, 3584 -> 3584 11.6 -> 8.9; M = 9 alike. It is bound by its fixed parts (staging, the slices' meeting), not by
// HBM (5.2 us) or the MMAs. gemm_thin.cu is faster (16 fp16 rows: 16.1 and 12.0, 23.3 and 15.8, 8.3 and 6.5 us on the three), but these rows
// stay: here the nibbles are multiplied as they are and f32 sums are scaled, there each weight times its scale is rounded to fp16. Against
// 64 bits, with the same activations, 1.5e-6 and 1.8e-4 of the result (2-norm). A version for 24 and 32 rows was no faster than the tcgen05 kernel (three and four row blocks leave no
// registers for loads under way), nor were slices as clusters with one CTA of 16 warps an SM.
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"
#include "gemv_core.cuh"

namespace wb {

namespace {

constexpr int kMB = 2;  // blocks of 8 rows
constexpr int kCtasPerSm = 2;
constexpr size_t kSmallSmem = 104 * 1024;  // of a CTA

__device__ __forceinline__ void mma_first(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

struct Chunk {
    uint4 w[4];  // packed words: rows 4 st + t of the chunk, columns c .. c + 3
    uint2 s;     // four fp16 scales
    uint32_t z;  // the zero word of columns c .. c + 7 (or 0x77777777)
};

// grid (column groups, K slices), block 256. Dynamic shared memory: [16][xs_stride] activations, [chunks][16] their sums.
template <int WK>
__global__ void __launch_bounds__(256, kCtasPerSm) gptq_gemm_small_kernel(const GemvParams p)
{
    constexpr int MB = kMB, ROWS = 8 * MB, WN = 8 / WK, COLS = 32 * WN, NBUF = 3;
    extern __shared__ uint4 smem_u4[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int ch_begin = blockIdx.y * p.chunks_per_split, chunks_cta = min(p.chunks - ch_begin, p.chunks_per_split);
    const int wn = warp % WN, wk = warp / WN;
    const int n_warp = blockIdx.x * COLS + wn * 32, c = n_warp + 4 * g;
    const bool col_ok = n_warp < p.N;
    uint4 *xs = smem_u4;
    float *xsum = reinterpret_cast<float *>(smem_u4 + (size_t)ROWS * p.xs_stride);

    const uint32_t *wrow = p.qw + ((int64_t)ch_begin * 16 + t) * p.N + c;
    auto fetch = [&](int i, Chunk &r) {  // chunk i of the slice
        const uint32_t *src = wrow + (int64_t)i * 16 * p.N;
#pragma unroll
        for (int st = 0; st < 4; st++) r.w[st] = ldg_stream_v4(src + (int64_t)st * 4 * p.N);
        const int G = p.group_chunks == 1 ? ch_begin + i : (ch_begin + i) / p.group_chunks;
        r.s = *reinterpret_cast<const uint2 *>(p.sc + (int64_t)G * p.N + c);
        r.z = p.qz ? p.qz[(int64_t)G * p.zcols + (c >> 3)] : 0x77777777u;
    };
    Chunk buf[NBUF];
#pragma unroll
    for (int u = 0; u < NBUF; u++)
        if (col_ok && wk + u * WK < chunks_cta) fetch(wk + u * WK, buf[u]);
    pdl_sync();

    // ---- activations: a warp takes rows warp, warp + 8, ...; a lane 8 k's of every 32nd slot, four loads under way
    const int slots = chunks_cta * 16, k_begin = ch_begin * 128;
#pragma unroll 1
    for (int m = warp; m < ROWS; m += 8) {
        for (int s0 = 0; s0 < slots; s0 += 128) {
            uint4 raw[4][2];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int sl = s0 + u * 32 + lane;
                raw[u][0] = raw[u][1] = make_uint4(0, 0, 0, 0);
                if (m >= p.M || sl >= slots) continue;
                const int64_t at = (int64_t)m * p.K + k_begin + sl * 8;
                if (p.x_f16) {
                    raw[u][0] = *reinterpret_cast<const uint4 *>((const __half *)p.x + at);
                } else {
                    raw[u][0] = *reinterpret_cast<const uint4 *>((const float *)p.x + at);
                    raw[u][1] = *reinterpret_cast<const uint4 *>((const float *)p.x + at + 4);
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int sl = s0 + u * 32 + lane;
                if (s0 + u * 32 >= slots) break;
                __half h[8];
                if (p.x_f16) {
                    const __half2 *q = reinterpret_cast<const __half2 *>(&raw[u][0]);
#pragma unroll
                    for (int j = 0; j < 4; j++) h[2 * j] = __low2half(q[j]), h[2 * j + 1] = __high2half(q[j]);
                } else {
                    const uint32_t f[8] = {raw[u][0].x, raw[u][0].y, raw[u][0].z, raw[u][0].w, raw[u][1].x, raw[u][1].y, raw[u][1].z, raw[u][1].w};
#pragma unroll
                    for (int j = 0; j < 8; j++) h[j] = __float2half_rn(__uint_as_float(f[j]));
                }
                // k-slot order of the unpacked nibbles: (0, 4)(2, 6) and, from the word shifted by 4, (1, 5)(3, 7)
                uint4 o;
                o.x = h2_as_u32(__halves2half2(h[0], h[4])), o.y = h2_as_u32(__halves2half2(h[2], h[6]));
                o.z = h2_as_u32(__halves2half2(h[1], h[5])), o.w = h2_as_u32(__halves2half2(h[3], h[7]));
                if (sl < slots) xs[m * p.xs_stride + sl] = o;
                // the zero point multiplies the sum of a chunk's operands: 16 slots, half a warp
                float sx = ((__half2float(h[0]) + __half2float(h[4])) + (__half2float(h[2]) + __half2float(h[6]))) +
                           ((__half2float(h[1]) + __half2float(h[5])) + (__half2float(h[3]) + __half2float(h[7])));
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) sx += __shfl_xor_sync(0xffffffffu, sx, w);
                if ((lane & 15) == 0 && sl < slots) xsum[(sl >> 4) * ROWS + m] = sx;
            }
        }
    }
    __syncthreads();

    // ---- chunks wk, wk + WK, ... of the slice
    const uint4 *xrow = xs + (size_t)g * p.xs_stride + t;
    const int zshift = ((4 * g) & 7) * 4;
    float tot[2][MB][4];  // [tile][row block][(column c + 2 tile | + 1) x (row 2 t | + 1)]
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int b = 0; b < MB; b++)
#pragma unroll
            for (int e = 0; e < 4; e++) tot[s][b][e] = 0.f;
    auto step = [&](const Chunk &cur, int i) {
        float acc[2][MB][4];
#pragma unroll
        for (int st = 0; st < 4; st++) {
            const uint32_t wv[4] = {cur.w[st].x, cur.w[st].y, cur.w[st].z, cur.w[st].w};
            uint32_t e0[4], e1[4], o0[4], o1[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                e0[j] = wv[j] & 0x000f000fu, o0[j] = (wv[j] >> 4) & 0x000f000fu;
                e1[j] = (wv[j] >> 8) & 0x000f000fu, o1[j] = (wv[j] >> 12) & 0x000f000fu;
            }
#pragma unroll
            for (int b = 0; b < MB; b++) {
                const uint4 x = xrow[(size_t)b * 8 * p.xs_stride + i * 16 + st * 4];
                if (st == 0) {
                    mma_first(acc[0][b], e0[0], e0[1], e1[0], e1[1], x.x, x.y);
                    mma_first(acc[1][b], e0[2], e0[3], e1[2], e1[3], x.x, x.y);
                } else {
                    mma_16816(acc[0][b], e0[0], e0[1], e1[0], e1[1], x.x, x.y);
                    mma_16816(acc[1][b], e0[2], e0[3], e1[2], e1[3], x.x, x.y);
                }
                mma_16816(acc[0][b], o0[0], o0[1], o1[0], o1[1], x.z, x.w);
                mma_16816(acc[1][b], o0[2], o0[3], o1[2], o1[3], x.z, x.w);
            }
        }
        const float2 s01 = __half22float2(u32_as_h2(cur.s.x)), s23 = __half22float2(u32_as_h2(cur.s.y));
        const float scale[4] = {s01.x, s01.y, s23.x, s23.y};
        const uint32_t zw = cur.z >> zshift;
        float zp[4];
#pragma unroll
        for (int j = 0; j < 4; j++) zp[j] = -(float)(((zw >> (4 * j)) & 15u) + 1u);
#pragma unroll
        for (int b = 0; b < MB; b++) {
            const float2 sx = *reinterpret_cast<const float2 *>(xsum + i * ROWS + b * 8 + 2 * t);
#pragma unroll
            for (int s = 0; s < 2; s++)
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int j = 2 * s + (e >> 1);
                    tot[s][b][e] = fmaf(scale[j], fmaf(acc[s][b][e], 16777216.f, zp[j] * ((e & 1) ? sx.y : sx.x)), tot[s][b][e]);
                }
        }
    };
    if (col_ok) {
        for (int i = wk; i < chunks_cta;) {
#pragma unroll
            for (int u = 0; u < NBUF; u++) {
                if (i >= chunks_cta) break;
                step(buf[u], i);
                if (i + NBUF * WK < chunks_cta) fetch(i + NBUF * WK, buf[u]);
                i += WK;
            }
        }
    }

    // ---- the second set's sums, then the result or this slice's partial sums
    if constexpr (WK == 2) {
        __syncthreads();  // the activations have been read
        float4 *red = reinterpret_cast<float4 *>(smem_u4) + (wn * 32 + lane);
        if (wk == 1) {
#pragma unroll
            for (int s = 0; s < 2; s++)
#pragma unroll
                for (int b = 0; b < MB; b++) red[(s * MB + b) * (WN * 32)] = make_float4(tot[s][b][0], tot[s][b][1], tot[s][b][2], tot[s][b][3]);
        }
        __syncthreads();
        if (wk == 0) {
#pragma unroll
            for (int s = 0; s < 2; s++)
#pragma unroll
                for (int b = 0; b < MB; b++) {
                    const float4 o = red[(s * MB + b) * (WN * 32)];
                    tot[s][b][0] += o.x, tot[s][b][1] += o.y, tot[s][b][2] += o.z, tot[s][b][3] += o.w;
                }
        }
    }
    auto put = [&](int m, int n, float4 v) {
        if (p.bias) {
            const float4 b = make_float4(p.bias[n], p.bias[n + 1], p.bias[n + 2], p.bias[n + 3]);
            v.x += b.x, v.y += b.y, v.z += b.z, v.w += b.w;
        }
        if (p.out_f16) {
            uint2 o;
            o.x = h2_as_u32(__floats2half2_rn(v.x, v.y)), o.y = h2_as_u32(__floats2half2_rn(v.z, v.w));
            *reinterpret_cast<uint2 *>((__half *)p.out + (int64_t)m * p.N + n) = o;
        } else {
            *reinterpret_cast<float4 *>((float *)p.out + (int64_t)m * p.N + n) = v;
        }
    };
    if (col_ok && wk == 0) {
#pragma unroll
        for (int b = 0; b < MB; b++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int m = b * 8 + 2 * t + r;
                if (m >= p.M) continue;
                const float4 v = make_float4(tot[0][b][r], tot[0][b][2 + r], tot[1][b][r], tot[1][b][2 + r]);
                if (p.S == 1) put(m, c, v);
                else *reinterpret_cast<float4 *>(p.partial + ((int64_t)blockIdx.y * p.M + m) * p.N + c) = v;
            }
    }
    if (p.S > 1) {
        __shared__ int is_last;
        __threadfence();
        __syncthreads();
        if (tid == 0) is_last = atomicAdd(&p.counters[blockIdx.x], 1u) == (unsigned)(p.S - 1);
        __syncthreads();
        if (!is_last) return;
        __threadfence();
        for (int idx = tid; idx < p.M * (COLS / 4); idx += 256) {
            const int m = idx / (COLS / 4), n = blockIdx.x * COLS + (idx - m * (COLS / 4)) * 4;
            if (n >= p.N) continue;
            const float *src = p.partial + (int64_t)m * p.N + n;
            const int64_t slice = (int64_t)p.M * p.N;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
            for (int s = 0; s < p.S; s++) {
                const float4 a = __ldcg(reinterpret_cast<const float4 *>(src + s * slice));
                v.x += a.x, v.y += a.y, v.z += a.z, v.w += a.w;
            }
            put(m, n, v);
        }
        if (tid == 0) p.counters[blockIdx.x] = 0u;
    }
}

// (the second set of warps hands its sums over in the same memory)
size_t small_smem(int cps, int wk)
{
    const size_t act = (size_t)8 * kMB * (cps * 16 + 4) * 16 + (size_t)cps * 8 * kMB * 4, red = wk == 2 ? (size_t)2 * kMB * 4 * 32 * 16 : 0;
    return std::max(act, red);
}

}  // namespace

// Below this many weights the launch and the slices' meeting are all there is, and the tcgen05 kernel does them quicker (4864 -> 896,
// fp16, M = 9: 9.1 us here, 7.8 there; 3584 -> 512: 7.3 and 7.0).
constexpr int64_t kFromWeights = 8 << 20;

// WEBLLM_B200_GEMM_SMALL=0 leaves these calls to the tcgen05 kernel (for comparisons).
bool gemm_small_takes(wb_context *ctx, const Weight &w, int64_t M)
{
    static const bool on = [] { const char *e = getenv("WEBLLM_B200_GEMM_SMALL"); return !(e && e[0] == '0'); }();
    return on && w.kind == WeightKind::Gptq && M >= 1 && M <= 8 * kMB && w.K * w.N >= kFromWeights && w.K % 128 == 0 && w.N % 32 == 0 &&
           w.group % 128 == 0 && ctx->place.n_dst == 0;
}

// Slices and columns per CTA by a small cost model in microseconds: rounds of resident CTAs, each a fixed part (launch, staging,
// reduction) and a warp's chunks, and the traffic of the partial sums. False: not a shape for this kernel.
bool plan_gemm_small(wb_context *ctx, const Weight &w, int64_t M, wb_plan *plan)
{
    if (!gemm_small_takes(ctx, w, M)) return false;
    const int chunks = (int)(w.K / 128);
    double best = 0.;
    int best_s = 0, best_wk = 0;
    for (int wk = 1; wk <= 2; wk++) {
        const int cols = 256 / wk;
        const int64_t groups = (w.N + cols - 1) / cols;
        if (groups > kMaxCounters) continue;
        for (int S = 1; S <= 64 && S <= chunks; S++) {
            if (ctx->force_split > 0 && S != std::min(ctx->force_split, chunks)) continue;
            const int cps = (chunks + S - 1) / S;
            if ((chunks + cps - 1) / cps != S || small_smem(cps, wk) > kSmallSmem || (double)S * M * w.N * 4. > 32e6) continue;
            const int64_t ctas = groups * S, slots = (int64_t)ctx->sm_count * kCtasPerSm;
            const int64_t rounds = (ctas + slots - 1) / slots;
            const int resident = ctas > ctx->sm_count ? 2 : 1;
            double t = rounds * (2.0 + (cps + wk - 1) / wk * std::max(0.35, 0.29 * resident) + M * cps * 128. * 4. / 120e3 * resident);
            if (S > 1) t += 1.0 + 2. * S * M * w.N * 4. / 8e6;
            if (best_s == 0 || t < best) best = t, best_s = S, best_wk = wk;
        }
    }
    if (best_s == 0) return false;
    plan->kernel = WB_KERNEL_GEMM_TC;
    plan->tile_m = 8 * kMB, plan->tile_n = 256 / best_wk;
    plan->grid_x = (int)((w.N + plan->tile_n - 1) / plan->tile_n), plan->grid_y = best_s, plan->grid_z = 1;
    plan->split_k = best_s;
    plan->block = kSmallBlock;
    plan->launches = 1;
    plan->scratch_bytes = best_s > 1 ? (uint64_t)best_s * M * w.N * 4 : 0;
    return true;
}

int launch_gemm_small(wb_context *ctx, const Weight &w, const void *A, void *C, const float *bias, int64_t M, int act_dtype, int out_dtype,
                      const wb_plan &plan)
{
    const char *base = ctx->arena[WB_ARENA_WEIGHTS].base;
    GemvParams p = {};
    p.qw = (const uint32_t *)(base + w.off_main);
    p.qz = w.has_zeros ? (const uint32_t *)(base + w.off_zeros) : nullptr;
    p.sc = (const __half *)(base + w.off_scales);
    p.x = A, p.out = C, p.bias = bias;
    p.partial = (float *)ctx->workspace, p.counters = ctx->counters;
    p.M = (int)M, p.N = (int)w.N, p.K = (int)w.K;
    p.zcols = (int)w.zcols;
    p.chunks = (int)(w.K / 128), p.S = plan.split_k;
    p.chunks_per_split = (p.chunks + p.S - 1) / p.S;
    p.group_chunks = (int)(w.group / 128);
    p.x_f16 = act_dtype == WB_F16, p.out_f16 = out_dtype == WB_F16;
    p.xs_stride = p.chunks_per_split * 16 + 4;
    const dim3 grid((unsigned)plan.grid_x, (unsigned)plan.grid_y);
    const size_t smem = small_smem(p.chunks_per_split, 256 / plan.tile_n);
    auto go = [&](auto kern, cudaError_t limit) { return limit != cudaSuccess ? limit : launch_pdl(kern, grid, dim3(256), smem, ctx->stream, p); };
    const cudaError_t e = plan.tile_n == 256 ? go(gptq_gemm_small_kernel<1>, smem_limit_once<gptq_gemm_small_kernel<1>>((int)kSmallSmem))
                                             : go(gptq_gemm_small_kernel<2>, smem_limit_once<gptq_gemm_small_kernel<2>>((int)kSmallSmem));
    ctx->launches++;
    WB_CUDA(e);
    return WB_OK;
}

}  // namespace wb
