// Prefill attention on the 5th-generation tensor cores: causal GQA attention of many query rows against an fp16 KV cache, head
// size 64 (attention_gqa_cache.wgsl, attentionGqaRef, src/reference/qwen-ref.ts:67-116). Same operands and accumulation as the
// warp-level kernel of attention_prefill.cu (fp16 q, k, v and softmax weights, f32 sums), which keeps the other cases.
//
// One CTA = 128 query rows of one head, in four groups of four warps and a control warp each: group i takes every fourth block of 64
// keys from block i on, and the four states of a row are merged at the end. Per block the control thread of a group issues
//   S = Q K^T  (tcgen05.mma, both operands K-major tiles in shared memory, 128 x 64 f32 in tensor memory)
//   O += P V   (P from tensor memory, V as it lies in the cache: keys x dims, an MN-major operand; 128 x 64 f32)
// and in between a thread of the group owns one row: it reads its 64 scores, takes the maximum, the exponentials (ex2, 16 a cycle
// per SM) and writes P as fp16 over S. O stays in tensor memory; as in FlashAttention-4 it is rescaled only where a row's maximum has
// grown by more than 2^8 since the last time (the weights of the meantime are at most 2^8, and the final division takes the same maximum, so
// nothing is approximated). K and V boxes come by TMA, two stages each; rows past the last key read as zeros.
// Bound by the chain of a block, product - softmax - product, some 3000 cycles when four groups share the SM's exponentials, times
// the blocks of the longest CTA. So four groups of one row tile rather than two of each of two: half as many blocks in the
// chain for the same four at a time. CTAs are started longest first. 2048 tokens, 14 heads: 41.6 us (warp-level kernel) -> 31.9 (two
// groups) -> 29.9; exponentials 33 % of their rate.
#include "gemm_tc.cuh"
#include "qwen_ops.cuh"

namespace wb {

namespace {

using namespace tc;

constexpr int kD = 64, kRows = 128, kKeys = 64, kGroups = 4;
constexpr int kThreads = kGroups * 128 + kGroups * 32;
constexpr int kTile = kKeys * kD * 2;         // a K or V box: 64 rows of 128 bytes
constexpr int kGroupBytes = 2 * 2 * kTile;    // two stages of K, two of V
constexpr int kQBytes = kRows * kD * 2;
constexpr int kSmem = kQBytes + kGroups * kGroupBytes + kGroups * 2 * kRows * 4 + 256 + 1024 /*alignment slack*/;
constexpr uint32_t kGroupCols = 128;          // tensor-memory columns of a group: S (P over it) 64, O 64
static_assert(kRows * kD * 4 == kGroupBytes, "the merge hands O over in a group's stages");

__device__ __forceinline__ float ex2f(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A from tensor memory (fp16 pairs, two k per column)
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// An MN-major operand with 64 elements (one 128-byte swizzle atom) along MN: 8 rows of k make an atom of 1024 bytes, the next
// atom along K follows it. (One atom along MN: the leading offset is not used; both name the same 1024 bytes.)
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t saddr)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (64ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

__global__ void __launch_bounds__(kThreads, 1)
attention_tc_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const float *__restrict__ q,
                    const float *__restrict__ cs_table, float *__restrict__ out, __half *__restrict__ out16, int *status, int M, int H, int KVH, int past, int ldq,
                    float scale)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool control = warp >= kGroups * 4;
    const int grp = control ? warp - kGroups * 4 : warp >> 2;
    uint8_t *stages = smem + kQBytes + grp * kGroupBytes;  // K0 K1 V0 V1 of this group
    float *ml = (float *)(smem + kQBytes + kGroups * kGroupBytes);  // of each group [128] maxima, [128] sums
    uint64_t *bars = (uint64_t *)(ml + kGroups * 2 * kRows);
    uint64_t *kfull = bars + grp * 6, *vfull = kfull + 2, *s_full = kfull + 4, *p_ready = kfull + 5;
    uint32_t *tmem_slot = (uint32_t *)(bars + kGroups * 6);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    if (threadIdx.x == 0) {
        for (int i = 0; i < kGroups * 6; i++) mbar_init(bars + i, i % 6 == 5 ? 4 : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kGroups * 4) tmem_alloc(tmem_slot, kGroups * kGroupCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t t_s = *tmem_slot + (uint32_t)grp * kGroupCols, t_o = t_s + 64;

    const int h = blockIdx.x, kvh = h / (H / KVH);
    const int r0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * kRows;  // late (long) rows first
    const int n_blocks = (past + min(r0 + kRows, M) - 1) / kKeys + 1;
    const int nb = (n_blocks - grp + kGroups - 1) / kGroups;  // blocks of this group
    pdl_sync();

    auto load_k = [&](int j) {
        mbar_expect_tx(&kfull[j & 1], kTile);
        tma_load_2d(stages + (j & 1) * kTile, &map_k, kvh * kD, (kGroups * j + grp) * kKeys, &kfull[j & 1]);
    };
    auto load_v = [&](int j) {
        mbar_expect_tx(&vfull[j & 1], kTile);
        tma_load_2d(stages + (2 + (j & 1)) * kTile, &map_v, kvh * kD, (kGroups * j + grp) * kKeys, &vfull[j & 1]);
    };
    if (control) {
        if (lane == 0)
            for (int j = 0; j < 2 && j < nb; j++) load_k(j), load_v(j);
        __syncwarp();
    } else {
        // Q as fp16 rows of 128 bytes, 16-byte pieces swizzled as TMA would: a thread of each group per row, with dims 8 part to + 7
        // and the same of the upper half, which are what the rotary embedding turns together (ropeHalfRef,
        // src/reference/qwen-ref.ts:35-64; a pass over q by itself took 4 us at 2048 rows)
        static_assert(kGroups * 8 * 2 == kD, "two pieces per thread");
        const int r = threadIdx.x / kGroups, part = threadIdx.x % kGroups;
        const float4 *src = reinterpret_cast<const float4 *>(q + (int64_t)(r0 + r) * ldq + h * kD + part * 8);
        const float4 *cs = reinterpret_cast<const float4 *>(cs_table + ((int64_t)(past + r0 + r) * (kD / 2) + part * 8) * 2);
        uint32_t lo[4] = {}, hi[4] = {};
        if (r0 + r < M) {
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const float4 x = src[c], y = src[c + kD / 8];
                const float4 c0 = cs[2 * c], c1 = cs[2 * c + 1];  // cos, sin of a dim and the next
                const __half2 a0 = __floats2half2_rn(x.x * c0.x - y.x * c0.y, x.y * c0.z - y.y * c0.w);
                const __half2 a1 = __floats2half2_rn(x.z * c1.x - y.z * c1.y, x.w * c1.z - y.w * c1.w);
                const __half2 b0 = __floats2half2_rn(x.x * c0.y + y.x * c0.x, x.y * c0.w + y.y * c0.z);
                const __half2 b1 = __floats2half2_rn(x.z * c1.y + y.z * c1.x, x.w * c1.w + y.w * c1.z);
                lo[2 * c] = *reinterpret_cast<const uint32_t *>(&a0), lo[2 * c + 1] = *reinterpret_cast<const uint32_t *>(&a1);
                hi[2 * c] = *reinterpret_cast<const uint32_t *>(&b0), hi[2 * c + 1] = *reinterpret_cast<const uint32_t *>(&b1);
            }
        }
        *reinterpret_cast<uint4 *>(smem + r * 128 + ((part ^ (r & 7)) << 4)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<uint4 *>(smem + r * 128 + (((part + kGroups) ^ (r & 7)) << 4)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        fence_async_smem();
    }
    __syncthreads();

    float m = -INFINITY, l = 0.f;
    const int wq = warp & 3;
    const uint32_t lane_sel = (uint32_t)(wq * 32) << 16;
    const float sl2 = scale * 1.4426950408889634f;
    if (control) {
        if (lane == 0 && nb > 0) {
            constexpr uint32_t idesc_s = idesc_f16(kRows, kKeys), idesc_o = idesc_f16(kRows, kD) | (1u << 16);
            const uint64_t dq = smem_desc_sw128(smem_u32(smem));
            auto scores = [&](int j) {
                const uint64_t dk = smem_desc_sw128(smem_u32(stages + (j & 1) * kTile));
#pragma unroll
                for (int k = 0; k < kD / 16; k++) umma_f16(t_s, dq + 2 * k, dk + 2 * k, idesc_s, k != 0);
            };
            bool ok = mbar_wait(&kfull[0], 0, abort_flag, status, 21);
            if (ok) scores(0), umma_commit(s_full);
            for (int j = 0; j < nb && ok; j++) {
                // S_j is complete, and with it O of block j - 1: their K and V stages are free
                if (!(ok = mbar_wait(s_full, (uint32_t)j & 1u, abort_flag, status, 22))) break;
                if (j + 2 < nb) load_k(j + 2);
                if (j >= 1 && j + 1 < nb) load_v(j + 1);
                if (!(ok = mbar_wait(&vfull[j & 1], (uint32_t)(j >> 1) & 1u, abort_flag, status, 23))) break;
                if (j + 1 < nb && !(ok = mbar_wait(&kfull[(j + 1) & 1], (uint32_t)((j + 1) >> 1) & 1u, abort_flag, status, 24))) break;
                if (!(ok = mbar_wait(p_ready, (uint32_t)j & 1u, abort_flag, status, 25))) break;
                tc_fence_after();
                const uint64_t dv = smem_desc_mn_sw128(smem_u32(stages + (2 + (j & 1)) * kTile));
#pragma unroll
                for (int k = 0; k < kKeys / 16; k++) umma_f16_ts(t_o, t_s + 8 * k, dv + (uint64_t)(k * (2048 >> 4)), idesc_o, (j | k) != 0);
                if (j + 1 < nb) scores(j + 1);
                umma_commit(s_full);
            }
        }
        __syncwarp();
    } else {
        const int last_key = past + r0 + wq * 32 + lane;  // of this thread's row
        bool ok = true;
        for (int j = 0; j < nb; j++) {
            const int key0 = (kGroups * j + grp) * kKeys;
            ok = __all_sync(0xffffffffu, mbar_wait(s_full, (uint32_t)j & 1u, abort_flag, status, 26));
            if (!ok) break;
            tc_fence_after();
            uint32_t s[4][16];
#pragma unroll
            for (int c = 0; c < 4; c++) tmem_ld_32x32b_x16(t_s + lane_sel + c * 16, s[c]);
            tmem_ld_wait();
            if (key0 + kKeys - 1 > past + r0 + wq * 32) {  // the diagonal is in this block for some row of the warp
#pragma unroll
                for (int c = 0; c < 4; c++)
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (key0 + c * 16 + i > last_key) s[c][i] = 0xff800000u;  // -infinity
            }
            float mx[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                mx[c] = __uint_as_float(s[c][0]);
#pragma unroll
                for (int i = 1; i < 16; i++) mx[c] = fmaxf(mx[c], __uint_as_float(s[c][i]));
            }
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            if (j == 0) {
                m = top;
            } else {
                const bool grow = (top - m) * sl2 > 8.f;
                if (__any_sync(0xffffffffu, grow)) {
                    const float f = grow ? ex2f((m - top) * sl2) : 1.f;
                    if (grow) m = top, l *= f;
#pragma unroll 1
                    for (int c = 0; c < 4; c++) {
                        uint32_t o[16];
                        tmem_ld_32x32b_x16(t_o + lane_sel + c * 16, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                        tmem_st_32x32b_x16(t_o + lane_sel + c * 16, o);
                    }
                }
            }
            const float base = m == -INFINITY ? 0.f : m * sl2;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 2; c++) {
                uint32_t p[16];
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int e = c * 32 + i * 2;
                    const float a = ex2f(fmaf(__uint_as_float(s[e >> 4][e & 15]), sl2, -base));
                    const float b = ex2f(fmaf(__uint_as_float(s[e >> 4][(e & 15) + 1]), sl2, -base));
                    sum[(i & 1) * 2] += a, sum[(i & 1) * 2 + 1] += b;
                    const __half2 pr = __floats2half2_rn(a, b);
                    p[i] = *reinterpret_cast<const uint32_t *>(&pr);
                }
                tmem_st_32x32b_x16(t_s + lane_sel + c * 16, p);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
        }
        if (ok && nb > 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(s_full, (uint32_t)nb & 1u, abort_flag, status, 27));
            tc_fence_after();
        }
        // the states of a row meet in shared memory: every group's sums in its own stages, [64 dims][128 rows]
        float *po = (float *)stages;
        const int r = wq * 32 + lane;
#pragma unroll 1
        for (int c = 0; c < 4; c++) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(t_o + lane_sel + c * 16, o);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; i++) po[(c * 16 + i) * kRows + r] = nb > 0 ? __uint_as_float(o[i]) : 0.f;
        }
        ml[grp * 2 * kRows + r] = m, ml[(grp * 2 + 1) * kRows + r] = l;
    }
    __syncthreads();
    if (!control) {  // a group's thread takes 64 / kGroups dims of its row
        constexpr int DIMS = kD / kGroups;
        const int r = wq * 32 + lane;
        float mg[kGroups], w[kGroups], top = -INFINITY, sum = 0.f;
#pragma unroll
        for (int i = 0; i < kGroups; i++) mg[i] = ml[i * 2 * kRows + r], top = fmaxf(top, mg[i]);  // (key 0 is in group 0: finite)
#pragma unroll
        for (int i = 0; i < kGroups; i++) w[i] = ex2f((mg[i] - top) * sl2), sum += ml[(i * 2 + 1) * kRows + r] * w[i];
        float v[DIMS];
#pragma unroll
        for (int d = 0; d < DIMS; d++) v[d] = 0.f;
#pragma unroll
        for (int i = 0; i < kGroups; i++) {
            const float *po = (const float *)(smem + kQBytes + i * kGroupBytes) + grp * DIMS * kRows + r;
            const float wi = w[i] / sum;
#pragma unroll
            for (int d = 0; d < DIMS; d++) v[d] = fmaf(po[d * kRows], wi, v[d]);
        }
        const int64_t at = (int64_t)(r0 + r) * (H * kD) + h * kD + grp * DIMS;
        if (r0 + r < M) {
            if (out16) {  // the o projection takes the fp16 value it would round to itself
#pragma unroll
                for (int d = 0; d < DIMS; d += 8) {
                    uint32_t o[4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const __half2 pr = __floats2half2_rn(v[d + 2 * i], v[d + 2 * i + 1]);
                        o[i] = *reinterpret_cast<const uint32_t *>(&pr);
                    }
                    *reinterpret_cast<uint4 *>(out16 + at + d) = make_uint4(o[0], o[1], o[2], o[3]);
                }
            } else {
#pragma unroll
                for (int d = 0; d < DIMS; d += 4) *reinterpret_cast<float4 *>(out + at + d) = make_float4(v[d], v[d + 1], v[d + 2], v[d + 3]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == kGroups * 4) tmem_dealloc(*tmem_slot, kGroups * kGroupCols);
}

}  // namespace

// From 512 rows on. Below, the chain of a CTA is a block or two long, and its set-up (tensor memory, barriers, the merge of four groups)
// is more than the warp-level kernel's whole chain. Whole layers, us, warp-level and this: 14 heads, 64 rows 36.0, 37.9; 128 40.5,
// 43.2; 256 45.6, 47.7; 384 51.3, 51.9; 512 54.9, 54.3; 1024 75.1, 69.6; 2048 103, 92.2. 4 heads even at 576 rows (43.1, 43.7 at 512),
// 32 heads at about 350 (70.4, 69.1 at 384).
bool op_attention_tc_supported(int M, int D, int ldq, int kv_ld, int kv_f16, const void *q)
{
    return kv_f16 && D == kD && M >= 512 && ldq % 4 == 0 && kv_ld % 8 == 0 && ((uintptr_t)q & 15) == 0;
}

int op_attention_tc(wb_context *ctx, const float *q, const float *cs_table, const void *kmem, const void *vmem, float *out, __half *out16, int M, int H, int KVH,
                    int past, int ldq, int kv_ld)
{
    CUtensorMap maps[2];
    for (int i = 0; i < 2; i++) {
        cuuint64_t dims[2] = {(cuuint64_t)KVH * kD, (cuuint64_t)past + M}, strides[1] = {(cuuint64_t)kv_ld * 2};
        cuuint32_t box[2] = {kD, kKeys}, estr[2] = {1, 1};
        const CUresult r = ((EncodeTiledFn)ctx->tmap_encode)(&maps[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(i ? vmem : kmem), dims,
                                                             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(WB_ERR_CUDA, "cuTensorMapEncodeTiled (KV cache) failed with code %d", (int)r);
    }
    if (const cudaError_t e = smem_limit_once<attention_tc_kernel>(kSmem); e != cudaSuccess) WB_CUDA(e);
    const dim3 grid((unsigned)H, (unsigned)((M + kRows - 1) / kRows));
    const cudaError_t e = launch_pdl(attention_tc_kernel, grid, dim3(kThreads), (size_t)kSmem, ctx->stream, maps[0], maps[1], q, cs_table, out, out16,
                                     ctx->status_word, M, H, KVH, past, ldq, 1.0f / sqrtf((float)kD));
    ctx->launches++;
    WB_CUDA(e);
    return WB_OK;
}

}  // namespace wb
