// Causal attention of prompt portions over the paged cache on the fifth-generation tensor
// cores: tiles of 128 queries against blocks of 64 keys in four streams, head size 64, bfloat16.
//
// A CTA takes one tile of up to 128 consecutive new tokens of one request and one head.  Its keys, in blocks of 64, are dealt
// to four streams that know nothing of each other until the end: block b (positions [64 b, 64 b + 64)) belongs to stream b % 4.
// A stream has 64 columns of tensor memory for its scores and 64 for its sums, and
//  * a producer warp that brings its key and value pages with TMA (cp.async.bulk.tensor, 128-byte swizzle; a page of one head is
//    a box of page_size rows x 64 values; pages that no row of the tile can see are fetched from beyond the pool, i.e. zeros);
//  * an issuing warp: S = Q.K^T (tcgen05.mma 128 x 64 x 16), and O += P.V with P as the MMA's tensor-memory operand and V as it
//    lies in the pages, an MN-major operand;
//  * four softmax warps, a thread per query row: read 64 scores, write the weights p = hi + lo, two bfloat16 terms (the product
//    then keeps about 16 bits of them), over the scores, and keep the row's maximum and sum in 32-bit
//      m' = max(m, s), p = exp(s - m'), O = O*exp(m - m') + p.v, l = l*exp(m - m') + sum p
//    (the reference's recurrence, src/kernels/prefill/flashattention.cu:129-168, with base-2 exponentials and the scale
//    folded in).  The sums stay in tensor memory; m and O move only where a score exceeds m by more than 2^8 (until then p
//    grows beyond 1, in 32-bit and in both terms alike), which after the first blocks is rare.  What that costs in precision lies far
//    below the rounding of the results (relative error against 64 bits 1.60 to 1.66e-3 with it and with the rounding alone, to 6 digits;
//    results that are not the correctly rounded ones, 1,024 tokens behind 1,000: 2.4e-3 of them with flat scores, 1.4e-3 with sharp
//    ones; with m always exact 2.2e-3 and 0.8e-3, and 22.9 instead of 20.1 us a launch for 2 x 1,024 tokens back to back).
// At the end a row's four streams meet: out = sum_g O_g 2^(m_g - m) / sum_g l_g 2^(m_g - m), in the order of g.
//
// What bounds it: the softmax, about 11 instructions per score on 4 x 32 lanes, 1,400 cycles per 128 x 128 scores; the MMAs
// take a fifth of that.  A stream's own chain (scores, weights, product and the hand-overs between, some 900 cycles a block
// beside its arithmetic) is hidden by the other three.  With all sixteen warps on one block of 128 keys, maxima exchanged, P
// through shared memory and O added in registers, every hand-over stood in the way of all of them: 4,200 cycles per 128 x 128.
// 2 x 1,024 tokens, 12 heads: 17 us a launch, 22 us so; 512 tokens behind 450, 16 heads: 17 and 25 us.
//
// A block's place and stream follow from positions, so the order of the additions for a query does not depend on how the
// prompt was cut or what else is in the batch.  Every wait on an mbarrier is bounded; after the limit the kernel records an
// error code that the host reads, lets its copies land, frees its tensor memory and returns.
//
// The reference's prefill attention handles one score at a time with block-wide reductions
// (src/kernels/prefill/flashattention.cu:7-32) and reads the step's own Q|K|V buffer.
#include "split_f32.cuh"

namespace {

using namespace tc;

constexpr int BQ = 128, BKV = 64, DH = 64, STREAMS = 4;
constexpr int SOFTMAX_WARPS = 4 * STREAMS, ISSUE_WARP = SOFTMAX_WARPS, LOAD_WARP = ISSUE_WARP + STREAMS;   // 16, 4 and 4 warps
constexpr int THREADS = (LOAD_WARP + STREAMS) * 32;
constexpr int Q_BYTES = BQ * DH * 2;                 // 16 KB
constexpr int KV_BYTES = BKV * DH * 2;               // 8 KB each for K and V of a block
constexpr int STAGES = 2;
constexpr int ML_BYTES = 2 * STREAMS * BQ * 4;       // every stream's row maxima and sums
constexpr size_t SMEM = 1024 + Q_BYTES + STREAMS * STAGES * 2 * KV_BYTES + ML_BYTES + 512;
constexpr uint32_t TMEM_COLS = 512, TMEM_O = STREAMS * BKV;      // scores (then weights: 32 columns hi, 32 lo), then sums
constexpr float LOG2E = 1.4426950408889634f;
constexpr float LAZY = 8.f;                          // how far (in powers of two) a score may exceed the maximum in use

__device__ int g_attn_error = 0;                     // first error code seen by this kernel

// Instruction descriptor with the B operand MN-major (bit 16): D=F32, A=B=BF16.
__host__ __device__ constexpr uint32_t make_idesc_bmn(int m, int n) { return make_idesc(m, n) | (1u << 16); }

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// A stream's barriers: a stage's keys and values have arrived, its MMAs have read both; a block's scores, weights and sums are there.
struct Stream {
    uint64_t k_full[STAGES], v_full[STAGES], empty[STAGES], s_full, p_full, o_full;
};

__global__ void __launch_bounds__(THREADS, 1)
attention_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const int* __restrict__ block_table,
                         int bt_stride, const int* __restrict__ tiles, const int* __restrict__ positions,
                         __nv_bfloat16* __restrict__ out, long long out_stride, int H, int Hkv, int page_size,
                         int pool_rows, float scale, int window) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = base;
    uint8_t* sKV = sQ + Q_BYTES;                                  // [STREAMS][STAGES][K 8 KB | V 8 KB]
    float* sm_m = reinterpret_cast<float*>(sKV + STREAMS * STAGES * 2 * KV_BYTES);     // [STREAMS][BQ]
    float* sm_l = sm_m + STREAMS * BQ;
    Stream* streams = reinterpret_cast<Stream*>(sm_l + STREAMS * BQ);
    uint64_t* q_full = (uint64_t*)(streams + STREAMS);
    uint32_t* tmem_slot = (uint32_t*)(q_full + 1);
    volatile int* failed = (volatile int*)(tmem_slot + 1);

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int h = blockIdx.x, tile = blockIdx.y;

    if (threadIdx.x == 32) {
        prefetch_map(&map_q);
        prefetch_map(&map_k);
        prefetch_map(&map_v);
    }
    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int g = 0; g < STREAMS; ++g) {
            Stream& st = streams[g];
            for (int s = 0; s < STAGES; ++s) { mbar_init(&st.k_full[s], 1); mbar_init(&st.v_full[s], 1); mbar_init(&st.empty[s], 1); }
            mbar_init(&st.s_full, 1);
            mbar_init(&st.p_full, 4);
            mbar_init(&st.o_full, 1);
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == ISSUE_WARP) tmem_alloc(tmem_slot, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // tiles, positions and block tables are written by the host before the step
    const int seq = __ldcg(tiles + tile * 3), tok0 = __ldcg(tiles + tile * 3 + 1), rows = __ldcg(tiles + tile * 3 + 2);
    const int pos0 = __ldcg(positions + tok0), pos_max = pos0 + rows - 1;
    const int hk = h / (H / Hkv);
    const int first_key = window > 0 && pos0 - window + 1 > 0 ? pos0 - window + 1 : 0;
    const int b_lo = first_key / BKV, b_hi = pos_max / BKV;
    const int g = warp < SOFTMAX_WARPS ? warp >> 2 : (warp - SOFTMAX_WARPS) % STREAMS;       // this warp's stream
    // blocks of stream x: first_block(x), first_block(x) + 4, ... up to b_hi
    auto first_block = [&](int x) { return b_lo + ((x - b_lo) & (STREAMS - 1)); };
    auto blocks_of = [&](int x) { const int b = first_block(x); return b > b_hi ? 0 : (b_hi - b) / STREAMS + 1; };
    const int steps = blocks_of(g);
    Stream& st = streams[g];
    const uint32_t t_s = tmem + (uint32_t)(g * BKV), t_o = tmem + TMEM_O + (uint32_t)(g * DH);

    if (warp >= LOAD_WARP) {
        // ---------------------------------------------------------------- the stream's pages; lane p brings page p of a block
        const int box = page_size < BKV ? page_size : BKV, boxes = BKV / box;
        const int* bt = block_table + (size_t)seq * bt_stride;
        auto row_of = [&](int b) {                                // the pool row at which this lane's box of block b starts
            const int k0 = b * BKV + lane * box;
            if (lane >= boxes || b > b_hi || k0 > pos_max || k0 + box <= first_key) return pool_rows;     // beyond the pool: zeros
            const int page = __ldcg(bt + k0 / page_size);
            return page < 0 ? pool_rows : (page * Hkv + hk) * page_size + k0 % page_size;
        };
        int b = first_block(g), row = row_of(b);
        pdl_wait();
        pdl_launch();
        if (g == 0 && lane == 0) {
            mbar_expect_tx(q_full, Q_BYTES);
            tma_load_2d(sQ, &map_q, h * DH, tok0, q_full);
        }
        for (int i = 0; i < steps; ++i, b += STREAMS) {
            const int s = i % STAGES;
            const int next = row_of(b + STREAMS);
            bool ok = i < STAGES || mbar_wait(&st.empty[s], ((i / STAGES) - 1) & 1);
            if (!ok) *failed = 1;
            if (!__all_sync(0xffffffffu, ok && !*failed)) break;
            if (lane == 0) {
                mbar_expect_tx(&st.k_full[s], KV_BYTES);
                mbar_expect_tx(&st.v_full[s], KV_BYTES);
            }
            __syncwarp();
            if (lane < boxes) {
                uint8_t* dst = sKV + (size_t)(g * STAGES + s) * 2 * KV_BYTES + (size_t)lane * box * (DH * 2);
                tma_load_2d(dst, &map_k, 0, row, &st.k_full[s]);
                tma_load_2d(dst + KV_BYTES, &map_v, 0, row, &st.v_full[s]);
            }
            row = next;
        }
    } else if (warp >= ISSUE_WARP) {
        // ---------------------------------------------------------------- the stream's MMAs
        // (the warp as a whole runs the loop, one elected lane issues: tcgen05.cuh says why)
        pdl_wait();
        pdl_launch();
        constexpr uint32_t idesc_s = make_idesc(BQ, BKV), idesc_o = make_idesc_bmn(BQ, DH);
        const uint64_t q_desc = make_smem_desc(smem_u32(sQ)),
                       kv_desc = make_smem_desc(smem_u32(sKV + (size_t)g * STAGES * 2 * KV_BYTES));
        auto all_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity) && !*failed); };
        bool ok = steps == 0 || all_wait(q_full, 0);
        if (!ok && !*failed) *failed = 2;
        for (int i = 0; i < steps && ok; ++i) {
            const int s = i % STAGES;
            const uint64_t k_desc = kv_desc + (uint64_t)(s * (2 * KV_BYTES >> 4)), v_desc = k_desc + (uint64_t)(KV_BYTES >> 4);
            // the scores' columns are free once the product that read the last block's weights there is complete
            if (i > 0 && !all_wait(&st.o_full, (i - 1) & 1)) { if (!*failed) *failed = 3; break; }
            if (!all_wait(&st.k_full[s], (i / STAGES) & 1)) { if (!*failed) *failed = 4; break; }
            tc_fence_after();
#pragma unroll
            for (int k = 0; k < DH / 16; ++k) umma_f16_warp(t_s, q_desc + 2 * k, k_desc + 2 * k, idesc_s, k != 0);
            umma_commit_warp(&st.s_full);
            if (!all_wait(&st.v_full[s], (i / STAGES) & 1)) { if (!*failed) *failed = 5; break; }
            if (!all_wait(&st.p_full, i & 1)) { if (!*failed) *failed = 6; break; }
            tc_fence_after();
#pragma unroll
            for (int term = 0; term < 2; ++term)                  // hi, then lo
#pragma unroll
                for (int kk = 0; kk < BKV / 16; ++kk)
                    umma_f16_ts_warp(t_o, t_s + (uint32_t)(term * (BKV / 2) + kk * 8), v_desc + (uint64_t)(kk * (2048 >> 4)), idesc_o,
                                     (i | term | kk) != 0);
            umma_commit_warp(&st.o_full);
            umma_commit_warp(&st.empty[s]);
        }
    } else {
        pdl_wait();
        pdl_launch();
        // ---------------------------------------------------------------- softmax: one query row per thread
        const int q4 = warp & 3;                              // the quarter of the tensor-memory lanes this warp may read
        const int r = q4 * 32 + lane;                         // row of the tile
        const int qp = pos0 + r;                              // its absolute position (rows beyond the tile are not stored)
        const uint32_t t_lane = (uint32_t)(q4 * 32) << 16;
        const float sl2 = scale * LOG2E;
        float m_run = -INFINITY, l_run = 0.f;
        bool alive = true;
        for (int i = 0; i < steps; ++i) {
            const int k0 = (first_block(g) + i * STREAMS) * BKV;
            bool got = mbar_wait(&st.s_full, i & 1);
            if (!got) *failed = 7;
            alive = __all_sync(0xffffffffu, got && !*failed);
            if (!alive) break;
            tc_fence_after();
            uint32_t v[2][32];
            tmem_ld32_issue(t_s + t_lane, v[0]);
            tmem_ld32_issue(t_s + t_lane + 32, v[1]);
            tmem_ld_wait();
            if (k0 + BKV - 1 > pos0 + q4 * 32 || window > 0) {        // some row of the warp does not see all keys
#pragma unroll
                for (int e = 0; e < 64; ++e)
                    if (k0 + e > qp || (window > 0 && k0 + e <= qp - window)) v[e >> 5][e & 31] = __float_as_uint(-INFINITY);
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < 64; ++e) mx[e & 3] = fmaxf(mx[e & 3], __uint_as_float(v[e >> 5][e & 31]));
            const float mb = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * sl2;
            const bool moves = mb > m_run + LAZY;             // (from -inf on: any visible key)
            if (__any_sync(0xffffffffu, moves)) {
                // rows that keep their maximum are multiplied by one
                const float alpha = moves ? fast_exp2(m_run - mb) : 1.f;
                if (moves) m_run = mb;
                l_run *= alpha;
                if (i > 0) {
#pragma unroll
                    for (int c = 0; c < DH; c += 16) {
                        uint32_t w[16];
                        tmem_ld16_issue(t_o + t_lane + c, w);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; ++e) w[e] = __float_as_uint(__uint_as_float(w[e]) * alpha);
                        tmem_st8(t_o + t_lane + c, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
                        tmem_st8(t_o + t_lane + c + 8, make_uint4(w[8], w[9], w[10], w[11]), make_uint4(w[12], w[13], w[14], w[15]));
                    }
                }
            }
            const float muse = m_run == -INFINITY ? 0.f : m_run;
            float rs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c = 0; c < 4; ++c) {                         // 16 keys: 8 columns of each term
                uint32_t hi[8], lo[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const int k = c * 16 + 2 * e;
                    const float p0 = fast_exp2(fmaf(__uint_as_float(v[k >> 5][k & 31]), sl2, -muse)),
                                p1 = fast_exp2(fmaf(__uint_as_float(v[k >> 5][(k & 31) + 1]), sl2, -muse));
                    rs[e & 3] += p0 + p1;
                    hi[e] = bf16x2_rn(p0, p1);
                    lo[e] = bf16x2_rn(p0 - __uint_as_float(hi[e] << 16), p1 - __uint_as_float(hi[e] & 0xffff0000u));
                }
                tmem_st8(t_s + t_lane + c * 8, make_uint4(hi[0], hi[1], hi[2], hi[3]), make_uint4(hi[4], hi[5], hi[6], hi[7]));
                tmem_st8(t_s + t_lane + 32 + c * 8, make_uint4(lo[0], lo[1], lo[2], lo[3]), make_uint4(lo[4], lo[5], lo[6], lo[7]));
            }
            l_run += (rs[0] + rs[1]) + (rs[2] + rs[3]);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&st.p_full);
        }
        if (alive && steps > 0) {
            bool got = mbar_wait(&st.o_full, (steps - 1) & 1);
            if (!got) *failed = 8;
        }
        // the four streams of a row meet; thread (g, r) writes the columns 16 g ..
        sm_m[g * BQ + r] = m_run;
        sm_l[g * BQ + r] = l_run;
        asm volatile("bar.sync %0, %1;" ::"r"(1 + q4), "n"(STREAMS * 32) : "memory");
        tc_fence_after();
        float m = -INFINITY, l = 0.f, o[16];
#pragma unroll
        for (int x = 0; x < STREAMS; ++x) m = fmaxf(m, sm_m[x * BQ + r]);
#pragma unroll
        for (int e = 0; e < 16; ++e) o[e] = 0.f;
#pragma unroll
        for (int x = 0; x < STREAMS; ++x) {
            if (blocks_of(x) == 0) continue;                      // uniform: the stream's columns were never written
            const float mx = sm_m[x * BQ + r], f = mx == -INFINITY ? 0.f : fast_exp2(mx - m);
            uint32_t w[16];
            tmem_ld16_issue(tmem + TMEM_O + t_lane + (uint32_t)(x * DH + g * 16), w);
            tmem_ld_wait();
            l = fmaf(f, sm_l[x * BQ + r], l);
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = fmaf(f, __uint_as_float(w[e]), o[e]);
        }
        if (r < rows && !*failed) {
            const float inv = 1.f / l;
            __nv_bfloat16* orow = out + (size_t)(tok0 + r) * out_stride + (size_t)h * DH + g * 16;
#pragma unroll
            for (int c = 0; c < 2; ++c)
                *reinterpret_cast<uint4*>(orow + c * 8) =
                    make_uint4(bf16x2_rn(o[c * 8] * inv, o[c * 8 + 1] * inv), bf16x2_rn(o[c * 8 + 2] * inv, o[c * 8 + 3] * inv),
                               bf16x2_rn(o[c * 8 + 4] * inv, o[c * 8 + 5] * inv), bf16x2_rn(o[c * 8 + 6] * inv, o[c * 8 + 7] * inv));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*failed) {
        if (threadIdx.x == 0) { atomicCAS(&g_attn_error, 0, *failed); report_to_host(200 + *failed); }
        for (int i = 0; i < 2000; ++i) __nanosleep(100);          // copies and MMAs already issued may still be running
        __syncthreads();
    }
    if (warp == ISSUE_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

}  // namespace

MLLM_EXPORT int mllm_attention_tcgen05_tile() { return BQ; }

// The pinned host word that this file's kernels write when they give up on a wait.
MLLM_EXPORT int mllm_attention_tcgen05_bind_error(int* word) { return bind_host_error(word); }

// The first error recorded by the kernel since the last call (0 = none); resets it.
MLLM_EXPORT int mllm_attention_tcgen05_error(int* code) {
    int zero = 0;
    MLLM_CUDA(cudaMemcpyFromSymbol(code, g_attn_error, sizeof(int)));
    if (*code) MLLM_CUDA(cudaMemcpyToSymbol(g_attn_error, &zero, sizeof(int)));
    return 0;
}

// tiles: n_tiles x (request index in the batch, flat index of the tile's first token, rows <= 128).
// bfloat16, head size 64, pages of 8, 16, 32, 64 or 128 tokens; q [T, *] with row stride q_stride
// (elements), 16-byte aligned; k_pages / v_pages [num_pages, Hkv, page_size, 64] contiguous.
MLLM_EXPORT int mllm_attention_tcgen05(const void* q, long long q_stride, int T, const void* k_pages,
                                       const void* v_pages, int num_pages, const int* block_table, int bt_stride,
                                       const int* tiles, int n_tiles, const int* positions, void* out,
                                       long long out_stride, int H, int Hkv, int dh, int page_size, float scale,
                                       int window, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (dh != DH) return mllm_fail(1, "attention_tcgen05: head size %d is not 64", dh);
    if (Hkv <= 0 || H % Hkv != 0) return mllm_fail(1, "attention_tcgen05: %d heads over %d key/value heads", H, Hkv);
    if (page_size < 8 || page_size > 128 || (page_size & (page_size - 1)))
        return mllm_fail(1, "attention_tcgen05: page size %d is not a power of two in 8..128", page_size);
    if (n_tiles > 65535) return mllm_fail(1, "attention_tcgen05: %d query tiles are more than one launch takes", n_tiles);
    if (!(scale > 0.f)) return mllm_fail(1, "attention_tcgen05: the score scale must be positive, got %g", (double)scale);
    if (q_stride % 8 || (uintptr_t)q % 16 || out_stride % 8 || (uintptr_t)out % 16)
        return mllm_fail(1, "attention_tcgen05: queries and outputs must be 16-byte aligned");
    if ((uintptr_t)k_pages % 16 || (uintptr_t)v_pages % 16)
        return mllm_fail(1, "attention_tcgen05: the page pools must be 16-byte aligned");
    const long long pool_rows = (long long)num_pages * Hkv * page_size;
    if (pool_rows + page_size > 2147483647LL) return mllm_fail(1, "attention_tcgen05: the page pool is too large");
    CUtensorMap mq, mk, mv;
    int rc = get_map(q, q_stride, T, H * DH, DH, BQ, MAP_BF16_SW128, &mq);
    if (rc) return rc;
    const int box = page_size < BKV ? page_size : BKV;
    rc = get_map(k_pages, DH, (int)pool_rows, DH, DH, box, MAP_BF16_SW128, &mk);
    if (rc) return rc;
    rc = get_map(v_pages, DH, (int)pool_rows, DH, DH, box, MAP_BF16_SW128, &mv);
    if (rc) return rc;
    auto kern = attention_tcgen05_kernel;
    static bool set = false;
    if (!set) {
        MLLM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
        set = true;
    }
    using bf = __nv_bfloat16;
    MLLM_CUDA(mllm_launch(kern, dim3(H, n_tiles), dim3(THREADS), SMEM, stream, true, mq, mk, mv, block_table, bt_stride,
                          tiles, positions, (bf*)out, out_stride, H, Hkv, page_size, (int)pool_rows, scale, window));
    return 0;
}
