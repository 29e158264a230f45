// int4 GEMM on the 5th-generation tensor cores with the weight operand taken from tensor memory, for products that are one round of tiles
// of 128 columns x up to 128 or 256 rows: served batches, short prompts, and the narrow projections of long ones. Same contract as
// gemm_tc.cu: fp16 operands, the weight rounded to fp16 once, f32 accumulation, f32 activations rounded to fp16
// (gemm_nt_f16_from_f32.wgsl:58-62).
//
// With few rows the weights have to be read once and unpacked once, and that is all there is to do. gemm_tc.cu takes 0.25 to
// 0.33 us for 64 k's of 128 columns whatever the rows: each unpacked weight goes through shared memory twice, and one thread waits,
// issues and commits for every 64 k's. Here a tile's 128 output columns are the 128 lanes of tensor memory, which is how the checkpoint
// already lies: thread = output column = lane, a packed word = eight consecutive k's of it.
//   * A chunk is 128 k's. 16 warps unpack, in four sets of 128 threads that take the chunks in turn: 16 words of a column from the TMA
//     box in shared memory, fp16 weights, tensor memory (tcgen05.st), from where tcgen05.mma takes them as its A operand. (SS form,
//     32 rows: 39 cycles an MMA, for reading A from shared memory; TS form 16.)
//   * The activations are the B operand, 128-byte swizzled tiles [rows][64 k], by TMA.
//   * Four threads issue MMAs, each for one set and into an accumulator of its own (two for more than 64 rows); the accumulators are
//     added up when they are read. One thread took 850 cycles a chunk of 64: waits of 200 cycles even on barriers that are over,
//     60 cycles an MMA; the order of the sum would not be fixed if they shared an accumulator.
//   * Words and scales have four warps that issue copies (one took as long as the unpack), and their first ones go out before
//     anything else is set up and before the wait on the kernel in front; everything arrives at barriers, no warp waits for its own loads.
//   * K slices of a tile are a cluster, which adds them through shared memory: every CTA a part of the rows, in the order of K.
// Bound by the integer pipe (8 or 5 of its instructions a word, at half rate) and the latencies of a set's turn, about 0.34 us a chunk
// with all SMs busy; HBM would need 0.19. f32 activations pass a launch that rounds them, which also puts the k's of a packed word in
// the order 0 4 1 5 2 6 3 7 that masks yield (13 instead of 16 instructions a word).
// Measured, gemm_tc.cu -> this, fp16 activations, us at 20 and 128 rows: 3584 -> 18944 20.4 -> 12.2, 23.2 -> 14.9; 18944 -> 3584 23.6 ->
// 16.1, 27.5 -> 19.2; 3584 -> 3584 9.2 -> 6.8, 11.5 -> 9.5; 3584 -> 512 6.9 -> 4.3, 8.4 -> 7.2; 896 -> 4864 6.9 -> 4.2, 8.6 -> 6.6; 4864 -> 896
// 7.6 -> 4.9, 9.2 -> 7.8; 896 -> 896 5.2 -> 4.1, 6.5 -> 6.4; at 512 and 2048 rows (against the CTA pairs where they were taken): 896 -> 1152
// 8.7 -> 6.6, 9.2 -> 7.9; 4864 -> 896 12.6 -> 10.5, 26.3 -> 18.2 (uncut, as a caller that adds slices itself has it; a layer of a prefill
// 125.9 -> 123.2, since the norm added the slices of the pair kernel at hardly any cost); 3584 -> 3584 at 512 and 1024 22.8 -> 14.3, 27.8 -> 22.6;
// 3584 -> 18944 at 256 29.7 -> 23.3. Built and slower: weights straight into registers (a use waits for the youngest load),
// cp.async for all of them (130 cycles each to issue), activations rounded by warps of this kernel, the next chunk's words read under
// this one's arithmetic, two CTAs of half the size per SM, and shares of several tiles per CTA (the code for that alone cost a
// fifth: the roles' code does not fit the instruction caches side by side).
#include <stdlib.h>

#include <algorithm>

#include "gemm_tc.cuh"

namespace wb {

namespace {

using namespace tc;

constexpr int kK = 128;                     // k of a chunk
constexpr int kSets = 4;                    // sets of unpack warps
constexpr int kUnpackWarps = 4 * kSets;
constexpr int kUnpackThreads = 32 * kUnpackWarps;
constexpr int kBufs = kSets;                // chunks in tensor memory, 64 columns each: one per set
constexpr int kWordBytes = kK / 8 * BN * 4;  // a packed chunk: a box of [16][128] words
constexpr int word_stages(bool big) { return big ? 4 : 8; }
constexpr int kHalfBytes = BN * 2 + BN / 2, kGroupBytes = 2 * kHalfBytes;  // of each half of a chunk: scales [128] fp16, zero words [16]
constexpr int kActStages = 8;               // at most
constexpr int act_warps(bool big) { return big ? 1 : 4; }
constexpr uint32_t kCols = 512, kABase = 256;  // tensor memory: the accumulators, then the weights
constexpr int kIssueWarp = kUnpackWarps, kIssuers = 4, kWordWarp = kIssueWarp + kIssuers, kWordWarps = 4;
constexpr int kActWarp = kWordWarp + kWordWarps, kActWarps = 4;
constexpr int kRows = 128, kRowsBig = 256;  // of a tile, in the two forms
static_assert(kThinBlock == 32 * (kActWarp + kActWarps), "the block size of a plan");
// A barrier is waited for by parity, so a warp that waits for a phase has to have seen the one before the last: the same warp comes round
// to the same buffer or stage.
static_assert(kBufs % kSets == 0 && kBufs % kIssuers == 0 && word_stages(true) % kSets == 0 && word_stages(true) % kWordWarps == 0 && kActStages % kActWarps == 0,
              "owners");

struct ThinParams {
    const uint32_t *qz;       // nullable
    const __half *sc;
    const float *bias;        // nullable
    void *out;
    int *status;
    int M, N, nt;             // nt: rows of an activation tile, a multiple of 16
    int accs;                 // accumulators, and threads that issue MMAs
    int zcols, chunks;        // chunks = K / 128 rounded up: what lies beyond K reads as zero activations
    int halves;               // K / 64
    uint32_t group_magic;     // h / (group / 64) = umulhi(h, group_magic); 0: group / 64 = 1
    int per, slices;          // chunks of a CTA; grid (column tiles, slices, row tiles), the slices of a tile a cluster
    int out_f16;
    int stages;               // of the activations
};

__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st_x16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
template <int BYTES>
__device__ __forceinline__ void copy_async(void *dst, const void *src, uint32_t there)  // bytes that are there (all or none), else zeros
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(BYTES), "r"(there) : "memory");
}
__device__ __forceinline__ uint32_t elect_one()
{
    uint32_t is;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(is));
    return is;
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }

// PERM: the activations' k's lie in the order 0 4 1 5 2 6 3 7 of every eight. BIG: tiles of 129 to 256 rows: one accumulator and one issuer
// (eight MMAs of a chunk take 1000 cycles there), and stages of 64 k's of the activations, of which as many as fit, walked in order.
template <bool PERM, bool BIG>
__global__ void __launch_bounds__(kThinBlock, 1)
gemm_thin_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const ThinParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int kWordStages = word_stages(BIG), kLoaders = act_warps(BIG), kPerChunk = BIG ? 2 : 1;  // stages of activations per chunk
    const int half_bytes = p.nt * 128, stage_bytes = 2 / kPerChunk * half_bytes;
    uint8_t *words = smem + p.stages * stage_bytes, *groups = words + kWordStages * kWordBytes;
    __shared__ uint64_t ready[kBufs], done[kBufs], full[kActStages], empty[kActStages], acc_full[kIssuers], word_full[kWordStages], word_empty[kWordStages];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int *abort_flag = &abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int set = warp >> 2, quarter = warp & 3, col = quarter * 32 + lane;  // an unpacking thread's column of the tile
    const int n0 = (int)blockIdx.x * BN, rank = (int)blockIdx.y, m0 = (int)blockIdx.z * p.nt, M = min(p.M - m0, p.nt);  // M: rows of this tile
    const int kb0 = rank * p.per, n_chunks = min(p.per, p.chunks - kb0);

    // Weights: a warp's every fourth chunk, a box of words and small copies that arrive at the same barrier. A lane copies four columns'
    // scales (N is a multiple of four, so they are there together), and every other one a zero word; what lies beyond K or N is
    // filled with zeros. They are constants: the first go out before anything else is done.
    int w_i = warp - kWordWarp, w_s = w_i;  // next chunk and its stage
    auto load_words = [&]() {
        if (lane == 0) {
            mbar_expect_tx(&word_full[w_s], (uint32_t)kWordBytes);
            tma_load_2d(words + w_s * kWordBytes, &map_w, n0, (kb0 + w_i) * (kK / 8), &word_full[w_s]);
        }
        const int n = n0 + lane * 4, n_in = min(n, p.N - 4);
        uint8_t *dst = groups + w_s * kGroupBytes;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int half = 2 * (kb0 + w_i) + h, at = min(half, p.halves - 1);
            const uint32_t there = half < p.halves && n < p.N;
            const int g = p.group_magic ? (int)__umulhi((uint32_t)at, p.group_magic) : at;
            copy_async<8>(dst + h * kHalfBytes + lane * 8, p.sc + (int64_t)g * p.N + n_in, there * 8);
            if (p.qz && (lane & 1) == 0) copy_async<4>(dst + h * kHalfBytes + BN * 2 + lane * 2, p.qz + (int64_t)g * p.zcols + (n_in >> 3), there * 4);
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&word_full[w_s])) : "memory");
        w_i += kWordWarps;
        if ((w_s += kWordWarps) >= kWordStages) w_s -= kWordStages;
    };
    if (warp >= kWordWarp && warp < kActWarp) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
            for (int i = w_s; i < kWordStages; i += kWordWarps) mbar_init(&word_full[i], 33), mbar_init(&word_empty[i], 4);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        for (int u = 0; u < kWordStages / kWordWarps; u++)
            if (w_i < n_chunks) load_words();
    } else if (threadIdx.x == 0) {
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
        for (int i = 0; i < kBufs; i++) mbar_init(&ready[i], 4), mbar_init(&done[i], 1);
        for (int i = 0; i < kActStages; i++) mbar_init(&full[i], 1), mbar_init(&empty[i], 1);
        for (int i = 0; i < kIssuers; i++) mbar_init(&acc_full[i], 1);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kIssueWarp) tmem_alloc(&tmem_slot, kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_trigger();

    bool ok = true;
    if (warp >= kIssueWarp && warp < kWordWarp) {
        // ------------------------------------------------------------------ MMA issuers: every accs-th chunk into an accumulator of its own
        // The whole warp walks the loop, so that its variables live in uniform registers, where the instructions want them.
        const int acc = __shfl_sync(0xffffffffu, warp, 0) - kIssueWarp, step = p.accs;
        if (acc < step) {
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint32_t idesc = idesc_f16(BN, p.nt), d = tm + (uint32_t)(acc * p.nt), elected = elect_one();
            const uint64_t bd0 = smem_desc_sw128(__shfl_sync(0xffffffffu, smem_u32(smem), 0));
            const uint32_t b_step = (uint32_t)stage_bytes >> 4, b_half = (uint32_t)half_bytes >> 4;
            uint32_t ph = 0;
            bool full_ok = false, ready_ok = false;
            int s = acc;  // (the number of stages is a multiple of the step)
#pragma unroll 1
            for (int i = acc; i < n_chunks; i += step) {
                const int b = i & (kBufs - 1);
                const uint32_t a = tm + kABase + b * 64;
                if constexpr (!BIG) {
                    ok = mbar_wait(&full[s], ph, abort_flag, p.status, 67);
                    if (!ok) break;
                    ok = mbar_wait(&ready[b], (uint32_t)(i / kBufs) & 1u, abort_flag, p.status, 61);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t bd = bd0 + (uint32_t)s * b_step;
                    if (elected) {
                        umma_ts(d, a, bd, idesc, i != acc);
#pragma unroll
                        for (int k = 1; k < 8; k++) umma_ts(d, a + 8 * k, bd + (k < 4 ? 2 * k : b_half + 2 * (k - 4)), idesc, 1);
                        umma_commit(&done[b]);
                        umma_commit(&empty[s]);
                        if (i + step >= n_chunks) umma_commit(&acc_full[acc]);
                    }
                    __syncwarp();
                    if ((s += step) >= p.stages) s -= p.stages, ph ^= 1;
                } else {
                    // a barrier is asked while the MMAs before it are issued: the answer alone takes 200 cycles
                    if (!ready_ok) ok = mbar_wait(&ready[b], (uint32_t)(i / kBufs) & 1u, abort_flag, p.status, 61);
#pragma unroll
                    for (int h = 0; h < 2 && ok; h++) {
                        if (!full_ok) ok = mbar_wait(&full[s], ph, abort_flag, p.status, 67);
                        if (!ok) break;
                        tc_fence_after();
                        const uint64_t bd = bd0 + (uint32_t)s * b_step;
                        uint64_t *emptied = &empty[s];
                        if (++s == p.stages) s = 0, ph ^= 1;
                        full_ok = mbar_try(&full[s], ph);
                        if (h == 1) ready_ok = mbar_try(&ready[(b + 1) & (kBufs - 1)], (uint32_t)((i + 1) / kBufs) & 1u);
                        if (elected) {
                            umma_ts(d, a + 32 * h, bd, idesc, (i | h) != 0);
#pragma unroll
                            for (int k = 1; k < 4; k++) umma_ts(d, a + 32 * h + 8 * k, bd + 2 * k, idesc, 1);
                            umma_commit(emptied);
                            if (h == 1) umma_commit(&done[b]);
                            if (h == 1 && i + 1 == n_chunks) umma_commit(&acc_full[0]);
                        }
                        __syncwarp();
                    }
                    if (!ok) break;
                }
            }
        }
    } else if (warp >= kWordWarp && warp < kActWarp) {
        // ------------------------------------------------------------------ packed weights, scales and zero points
        uint32_t ph = 0;
#pragma unroll 1
        while (w_i < n_chunks) {
            if (!mbar_wait_idle(&word_empty[w_s], ph, abort_flag, p.status, 68)) break;
            load_words();
            if (w_s == warp - kWordWarp) ph ^= 1;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (*abort_flag)  // a copy on its way has its time to arrive before the shared memory is given back
            for (int i = 0; i < 256; i++) __nanosleep(1000);
    } else if (warp >= kActWarp) {
        // ------------------------------------------------------------------ activations
        if (lane == 0 && warp < kActWarp + kLoaders) {
            pdl_wait();
            int s = warp - kActWarp;
            uint32_t ph = 1;
            for (int i = warp - kActWarp; i < n_chunks * kPerChunk; i += kLoaders) {
                if (!mbar_wait_idle(&empty[s], ph, abort_flag, p.status, 62)) break;
                mbar_expect_tx(&full[s], (uint32_t)stage_bytes);
                uint8_t *to = smem + s * stage_bytes;
                tma_load_2d(to, &map_x, kb0 * kK + i * (kK / kPerChunk), m0, &full[s]);
                if constexpr (!BIG) tma_load_2d(to + half_bytes, &map_x, kb0 * kK + i * kK + BK, m0, &full[s]);
                if ((s += kLoaders) >= p.stages) s -= p.stages, ph ^= 1;
            }
            if (*abort_flag)
                for (int i = 0; i < 256; i++) __nanosleep(1000);
        }
    } else {
        // ------------------------------------------------------------------ unpack
        const int zshift = (col & 7) * 4;
#pragma unroll 1
        for (int i = set; i < n_chunks; i += kSets) {
            const int ws = i & (kWordStages - 1), bi = i & (kBufs - 1);
            // the two waits as one where both are over, as they mostly are
            const uint32_t w_par = (uint32_t)(i / kWordStages) & 1u, d_par = ((uint32_t)(i / kBufs) & 1u) ^ 1u;
            const bool w_ok = mbar_try(&word_full[ws], w_par), d_ok = mbar_try(&done[bi], d_par);
            if (!w_ok) ok = mbar_wait(&word_full[ws], w_par, abort_flag, p.status, 69);
            if (!ok) break;
            const uint32_t *src = reinterpret_cast<const uint32_t *>(words + ws * kWordBytes) + col;
            uint32_t word[16], zw[2];
            __half sc[2];
#pragma unroll
            for (int r = 0; r < 16; r++) word[r] = src[r * BN];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint8_t *g = groups + ws * kGroupBytes + h * kHalfBytes;
                sc[h] = *reinterpret_cast<const __half *>(g + col * 2);
                zw[h] = p.qz ? *reinterpret_cast<const uint32_t *>(g + BN * 2 + (col >> 3) * 4) : 0x77777777u;
            }
            if (!d_ok) ok = mbar_wait(&done[bi], d_par, abort_flag, p.status, 65);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (int h = 0; h < 4; h++) {
                // -(1024 + zero) and -(64 + zero): the zero point in the low bits of a number whose last place is 1, and 1/16
                const uint32_t z = ((zw[h >> 1] >> zshift) & 15u) + 1u;
                const __half2 scale2 = __half2half2(sc[h >> 1]);
                const uint32_t m1024 = 0xe400u + z, m64 = 0xd400u + (z << 4);
                uint32_t o[16];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const uint32_t w = word[4 * h + r];
                    if constexpr (PERM) {
                        const uint32_t w8 = w >> 8;
                        const __half2 sub = as_h2(m1024 * 0x10001u), sub16 = as_h2(m64 * 0x10001u), sixteenth = as_h2(0x2c002c00u);
                        o[4 * r + 0] = as_u32(__hmul2(__hadd2(as_h2((w & 0x000f000fu) | 0x64006400u), sub), scale2));
                        o[4 * r + 1] = as_u32(__hmul2(__hfma2(as_h2((w & 0x00f000f0u) | 0x64006400u), sixteenth, sub16), scale2));
                        o[4 * r + 2] = as_u32(__hmul2(__hadd2(as_h2((w8 & 0x000f000fu) | 0x64006400u), sub), scale2));
                        o[4 * r + 3] = as_u32(__hmul2(__hfma2(as_h2((w8 & 0x00f000f0u) | 0x64006400u), sixteenth, sub16), scale2));
                    } else {  // byte j into both halves, then its low nibble in the lower and 16 times its high one in the upper
                        const __half2 one_sixteenth = as_h2(0x2c003c00u), sub = as_h2(m64 << 16 | m1024);
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const uint32_t x = __byte_perm(w, 0x64646464u, 0x4040u | (j * 0x0101u)) & 0x64f0640fu;
                            o[4 * r + j] = as_u32(__hmul2(__hfma2(as_h2(x), one_sixteenth, sub), scale2));
                        }
                    }
                }
                tmem_st_x16(tmem + kABase + bi * 64 + h * 16 + ((uint32_t)(quarter * 32) << 16), o);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready[bi]), mbar_arrive(&word_empty[ws]);
        }
        // the accumulators that have a chunk
        for (int a = 0; a < min(p.accs, n_chunks); a++)
            if (ok) ok = mbar_wait(&acc_full[a], 0, abort_flag, p.status, 66);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        pdl_wait();  // nothing is stored before the kernel in front is done
    }
    __syncwarp();

    // ---------------------------------------------------------------------- results: a warp has 32 columns and every fourth 16 rows
    const int n_accs = min(p.accs, n_chunks);
    auto result16 = [&](int c, uint32_t (&r)[16]) {  // rows c to c + 15 of this thread's column
#pragma unroll
        for (int j = 0; j < 16; j++) r[j] = 0u;
#pragma unroll 1
        for (int a = 0; a < n_accs; a++) {
            uint32_t o[16];
            tmem_ld_32x32b_x16(tmem + ((uint32_t)(quarter * 32) << 16) + a * p.nt + c, o);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; j++) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(o[j]));
        }
    };
    if (p.slices == 1) {
        if (warp < kUnpackWarps && ok) {
            StoreDst d;
            d.dst[0] = p.out, d.n_dst = 1, d.ld = p.N, d.col0 = 0;
            const int n_warp = n0 + quarter * 32, n = n_warp + lane;
            const float bias = p.bias && n < p.N ? p.bias[n] : 0.f;
#pragma unroll 1
            for (int c = set * 16; c < p.nt; c += 16 * kSets) {
                uint32_t r[16];
                result16(c, r);
                store_block16<false>(d, p.out_f16 != 0, (p.N & 7) == 0, r, bias, m0 + c, p.M, n_warp, p.N, lane);
            }
        }
    } else {
        // Every CTA of the cluster adds up its part of the rows, which all of them write into its shared memory in the place of what has
        // been read there (every copy has arrived: the last chunk's results are there).
        const int rows = (M + p.slices - 1) / p.slices;
        float *sums = reinterpret_cast<float *>(smem);  // [slices][rows][128 columns]
        cluster_barrier();
        if (warp < kUnpackWarps && ok) {
#pragma unroll 1
            for (int c = set * 16; c < p.nt; c += 16 * kSets) {
                uint32_t r[16];
                result16(c, r);
                int to = c / rows, row = c - to * rows;
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    if (c + j < M) cluster_store_f32(cluster_map_shared(sums + (rank * rows + row) * BN + col, (uint32_t)to), __uint_as_float(r[j]));
                    if (++row == rows) row = 0, to++;
                }
            }
        }
        __syncwarp();
        cluster_barrier();
        if (warp < kUnpackWarps) {
            const int here = min(rows, M - rank * rows);
            for (int i = threadIdx.x; i < here * (BN / 4); i += kUnpackThreads) {
                const int m = m0 + rank * rows + (i >> 5), n4 = n0 + (i & 31) * 4;
                if (n4 >= p.N) continue;
                const float4 *src = reinterpret_cast<const float4 *>(sums) + i;
                float4 v = src[0];
                for (int k = 1; k < p.slices; k++) {
                    const float4 a = src[k * rows * (BN / 4)];
                    v.x += a.x, v.y += a.y, v.z += a.z, v.w += a.w;
                }
                if (p.bias) v.x += p.bias[n4], v.y += p.bias[n4 + 1], v.z += p.bias[n4 + 2], v.w += p.bias[n4 + 3];
                if (p.out_f16) {
                    uint2 o;
                    o.x = as_u32(__floats2half2_rn(v.x, v.y)), o.y = as_u32(__floats2half2_rn(v.z, v.w));
                    *reinterpret_cast<uint2 *>((__half *)p.out + (int64_t)m * p.N + n4) = o;
                } else {
                    *reinterpret_cast<float4 *>((float *)p.out + (int64_t)m * p.N + n4) = v;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kIssueWarp) tmem_dealloc(tmem, kCols);
}

// Row tiles of at most `most` rows, and the rows of one.
int64_t thin_tiles(int64_t M, int most) { return (M + most - 1) / most; }
int thin_rows(int64_t M, int most) { return (int)(((M + thin_tiles(M, most) - 1) / thin_tiles(M, most) + 15) / 16 * 16); }
constexpr size_t kSmemMost = 227 * 1024 - 512;  // (the barriers are outside)
constexpr size_t word_bytes(bool big) { return 1024 + (size_t)word_stages(big) * (kWordBytes + kGroupBytes); }
int thin_stages(int nt)
{
    if (nt <= kRows) return nt > 64 ? 4 : kActStages;
    return (int)std::min<size_t>(kActStages, (kSmemMost - word_bytes(true)) / ((size_t)nt * 128));
}
size_t thin_smem(int nt) { return word_bytes(nt > kRows) + (size_t)thin_stages(nt) * nt * (nt > kRows ? 128 : 256); }
constexpr size_t kSmemThin = word_bytes(false) + kActStages * 64 * 256;  // the most that the form for up to 128 rows takes
static_assert(kSmemThin <= kSmemMost && 4 * kRows == kActStages * 64, "shared memory");
// (the slices meet in at most (rows + 8) * 512 bytes, which is less than the stages take)
static_assert((kRows + 8) * BN * 4 <= word_bytes(false) - 1024 + 4 * 16 * 256 && (kRowsBig + 8) * BN * 4 <= word_bytes(true) - 1024 + 5 * kRowsBig * 128, "the slices' meeting");

// Clusters of S CTAs that are resident at once, as the driver counts them for this device (a cluster stays inside a GPC, and these
// differ in size). 0: not known, so not taken.
int thin_clusters(int S, int sms)
{
    if (S == 1) return sms;
    static std::atomic<int> known[16][9] = {};  // count + 1
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 16 && known[dev][S].load(std::memory_order_relaxed)) return known[dev][S].load(std::memory_order_relaxed) - 1;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1, attr.val.clusterDim.y = (unsigned)S, attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(1, (unsigned)S), cfg.blockDim = dim3(kThinBlock), cfg.dynamicSmemBytes = kSmemThin, cfg.attrs = &attr, cfg.numAttrs = 1;
    int n = 0;
    if (smem_limit_once<gemm_thin_kernel<false, false>>((int)kSmemThin) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, gemm_thin_kernel<false, false>, &cfg) != cudaSuccess)
        return cudaGetLastError(), 0;
    if (dev < 16) known[dev][S].store(n + 1, std::memory_order_relaxed);
    return n;
}

}  // namespace

// WEBLLM_B200_GEMM_THIN=0 leaves these calls to the kernel of gemm_tc.cu (for comparisons).
bool gemm_thin_takes(wb_context *ctx, const Weight &w, int64_t M)
{
    static const bool on = [] { const char *e = getenv("WEBLLM_B200_GEMM_THIN"); return !(e && e[0] == '0'); }();
    return on && w.kind == WeightKind::Gptq && M >= 1 && w.K % 64 == 0 && w.N % 4 == 0 && w.group % 64 == 0 && ctx->place.n_dst == 0 &&
           w.K * (w.group / BK) < (int64_t)1 << 37;  // (group_magic)
}

// Slices by a small cost model in microseconds (measured; see the rule in plan_gemm_tc). False: not a shape, or forced split, for this kernel.
bool plan_gemm_thin(wb_context *ctx, const Weight &w, int64_t M, int act_dtype, wb_plan *plan, double *t_out)
{
    if (!gemm_thin_takes(ctx, w, M)) return false;
    const int chunks = (int)((w.K + kK - 1) / kK), sms = ctx->sm_count;
    const int64_t cols = (w.N + BN - 1) / BN;
    double best = -1.;
    int best_s = 0, best_rows = 0;
    for (int most : {kRows, kRowsBig}) {
        if (M <= kRows && most != kRows) continue;
        const int nt = thin_rows(M, most);
        const int64_t rows = thin_tiles(M, most), tiles = cols * rows;
        if (rows > 1 && tiles > sms) continue;  // every CTA sets itself up and drains: larger products go to persistent ones
        for (int S = 1; S <= 8 && S <= chunks; S++) {
            if (ctx->force_split > 0 && S != std::min(ctx->force_split, chunks)) continue;
            const int per = (chunks + S - 1) / S, at_once = thin_clusters(S, sms);
            if ((chunks + per - 1) / per != S || (S > 1 && tiles > at_once)) continue;
            // A long K of nine row tiles or more is cut while a fifth of the SMs would have no tile: of a call by itself a plan
            // promises that, and here it is the slower choice, by a third. Uncut and cut, us: 4864 -> 896 at 1500 rows 18.2, 21.1 (three
            // slices of 256-row tiles), 2048 rows 18.2, 24.5 (two); 6144 -> 1200 at 1280 21.0, 27.5; 18944 -> 512 at 2048 63, 42.
            // With fewer SMs idle, or cut in slices of 128-row tiles, nothing holds it back: 4864 -> 896 at 2500 rows 30.4 -> 19.5, at
            // 1100 19.8 -> 14.2; 11008 -> 2048 at 1100 54 -> 41. A caller that adds the slices itself has the uncut one everywhere.
            if (S == 1 && rows > 8 && chunks > 32 && tiles * 5 < sms * 4 && !ctx->keep_slices) continue;
            const int64_t rounds = S > 1 ? 1 : (tiles + sms - 1) / sms;
            const double chunk = nt > kRows ? 0.66 : 0.27 + 0.07 * std::min<double>(1., (double)tiles * S / sms);
            const double t = 1.6 + 0.022 * nt + rounds * per * chunk + (S > 1 ? 1.3 : 0.);
            if (best < 0. || t < best) best = t, best_s = S, best_rows = most;
        }
    }
    if (best_s == 0) return false;
    const bool cast = act_dtype == WB_F32;
    plan->kernel = WB_KERNEL_GEMM_TC;
    plan->tile_m = thin_rows(M, best_rows), plan->tile_n = BN;
    plan->grid_x = (int)thin_tiles(M, best_rows), plan->grid_y = (int)cols, plan->grid_z = best_s;  // (the launch has the slices in y, for the clusters)
    plan->split_k = best_s;
    plan->block = kThinBlock;
    plan->launches = cast ? 2 : 1;
    plan->scratch_bytes = cast ? align_up((uint64_t)M * w.K * 2) : 0;
    *t_out = best + (cast ? 1.2 : 0.);  // (the cast has no room beside this kernel's CTAs, as it has in gemm_tc.cu)
    return plan->scratch_bytes <= kWorkspaceBytes;
}

// `perm`: a launch in front has rounded the activations, in the order of the kernel's PERM.
int launch_gemm_thin(wb_context *ctx, const Weight &w, const void *x, bool perm, void *C, const float *bias, int64_t M, int out_dtype, const wb_plan &plan)
{
    const char *base = ctx->arena[WB_ARENA_WEIGHTS].base;
    const int nt = plan.tile_m;
    CallMap &cx = w.tmap_x;
    CUtensorMap &mx = *reinterpret_cast<CUtensorMap *>(cx.map.bytes);
    if (cx.base != x || cx.M != M || cx.a != nt) {
        cx.base = nullptr;
        WB_CHECK(make_map_2d(ctx, &mx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, x, (uint64_t)w.K, (uint64_t)M, BK, (uint32_t)nt, true));
        cx.base = x, cx.M = M, cx.a = nt;
    }
    TmapSlot &ws = w.tmap_tc[3];
    CUtensorMap &mw = *reinterpret_cast<CUtensorMap *>(ws.bytes);
    if (!ws.ok) WB_CHECK(make_map_2d(ctx, &mw, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, base + w.off_main, (uint64_t)w.N, (uint64_t)w.pack_rows, BN, kK / 8, false));
    ws.ok = true;
    ThinParams p;
    p.qz = w.has_zeros ? (const uint32_t *)(base + w.off_zeros) : nullptr;
    p.sc = (const __half *)(base + w.off_scales);
    p.bias = bias, p.out = C, p.status = ctx->status_word;
    p.M = (int)M, p.N = (int)w.N, p.nt = nt, p.accs = nt <= 64 ? kIssuers : nt <= kRows ? kIssuers / 2 : 1;
    p.zcols = (int)w.zcols, p.chunks = (int)((w.K + kK - 1) / kK), p.halves = (int)(w.K / BK);
    const uint32_t gb = (uint32_t)(w.group / BK);
    p.group_magic = gb == 1 ? 0u : (uint32_t)((0x100000000ull + gb - 1) / gb);  // exact while halves * gb < 2^32
    p.slices = plan.split_k, p.per = (p.chunks + p.slices - 1) / p.slices;
    p.out_f16 = out_dtype == WB_F16;
    p.stages = thin_stages(nt);
    auto go = [&](auto kern, cudaError_t limit) {
        return limit != cudaSuccess ? limit : launch_pdl_cluster(kern, dim3((unsigned)plan.grid_y, (unsigned)plan.grid_z, (unsigned)plan.grid_x), dim3(kThinBlock), thin_smem(nt),
                                                                 ctx->stream, (unsigned)plan.grid_z, mx, mw, p);
    };
    const cudaError_t e = nt > kRows ? (perm ? go(gemm_thin_kernel<true, true>, smem_limit_once<gemm_thin_kernel<true, true>>((int)kSmemMost))
                                             : go(gemm_thin_kernel<false, true>, smem_limit_once<gemm_thin_kernel<false, true>>((int)kSmemMost)))
                                     : (perm ? go(gemm_thin_kernel<true, false>, smem_limit_once<gemm_thin_kernel<true, false>>((int)kSmemThin))
                                             : go(gemm_thin_kernel<false, false>, smem_limit_once<gemm_thin_kernel<false, false>>((int)kSmemThin)));
    ctx->launches++;
    WB_CUDA(e);
    return WB_OK;
}

}  // namespace wb
