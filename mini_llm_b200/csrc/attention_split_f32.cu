// Causal attention of prompt portions over the paged cache with 32-bit queries, keys and values, heads of 64, on the
// fifth-generation tensor cores: the prefill attention of the 32-bit path.
//
// As in linear_split_f32.cu every 32-bit operand is cut exactly into three bfloat16 pieces and the six largest of the
// nine products of pieces are formed, smallest first; that holds for queries, keys, values and for the softmax weights
// p, which keep their 24 bits.  Scores, softmax (expf) and the sums over blocks of 128 keys are 32-bit as before.
// Against float64 the result is at least as close as the CUDA-core kernels' (tests/test_kernels_gpu.py compares).
//
// A CTA takes one tile of up to 128 consecutive new tokens of a request (the wide tile list) and one head and walks over
// blocks of 128 keys, counted from position 0 whatever the cut of the prompt:
//  * warps 16-19 and 20-23 fetch the keys and the values of a block row by row from their pages (any page size), cut them
//    and write the pieces into swizzled shared memory;
//  * warp 24 issues S = Q K^T (24 MMAs of 128 x 128 x 16, two S buffers in tensor memory) one block ahead, then
//    O_blk = P V (48 MMAs of 128 x 64 x 16, P's pieces from tensor memory, V read MN-major as it lies);
//  * warps 0-15, four threads per query row, keep the online softmax in registers and write P's pieces to tensor memory.
// What bounds a block is the softmax warps' instructions (32 expf and the cutting of 32 weights per thread).
//
// Measured (us, this kernel / 128 x 128 tiles on CUDA cores / 64 x 32 tiles there): 2 x 1,024 tokens and 12 heads
// 53 / 190 / 489; 512 tokens after 450 and 16 heads 50 / 187 / 299; 200 tokens and 12 heads 19 / 51 / 71 (19 us is what an
// isolated launch costs the host; 16 tokens: 19 / 27 / 18).
//
// A tile whose queries, keys or values do not all have pieces (infinities, NaN, values above the largest bfloat16) is
// computed again by plain_rows() with fmaf, one key after the other, so that infinities and NaN come out as they should.
//
// Every wait is bounded: after the limit the kernel records an error code, frees its tensor memory and returns.
#include "tcgen05.cuh"
#include "split_f32.cuh"

namespace {

using namespace tc;

constexpr int BQ = 128, BKV = 128, DH = 64;
constexpr int PARTS = 4;                             // threads per query row: each takes 32 keys of a block and 16 of the 64 output values
constexpr int SOFTMAX_WARPS = 4 * PARTS, CUT_WARPS = 8, K_WARP = SOFTMAX_WARPS, V_WARP = K_WARP + 4, MMA_WARP = V_WARP + 4;
constexpr int THREADS = (SOFTMAX_WARPS + CUT_WARPS + 4) * 32;
// Registers: 896 threads x 72 = 64,512 at launch; 512 x 88 + 256 x 64 + 128 x 24 = 64,512 after the split.  The compiler keeps
// all of the code to the 72 (12 bytes spill, and 124 in plain_rows).
constexpr int PLANE = 128 * DH * 2;                  // 16 KB: a piece of the tile's queries, of a block's keys or values
constexpr int XCH_BYTES = 2 * PARTS * BQ * 4;        // partial row maxima, double-buffered; reused for the row sums at the end
constexpr size_t SMEM = 1024 + 9 * PLANE + XCH_BYTES + 256;
constexpr uint32_t TMEM_O = 256, TMEM_P = 320;       // S of even blocks in columns 0..127, of odd ones in 128..255, O_blk, P's pieces

__device__ int g_attn_split_error = 0;

__host__ __device__ constexpr uint32_t make_idesc_bmn(int m, int n) { return make_idesc(m, n) | (1u << 16); }

// Whether the values have pieces (infinities, NaN and the largest finite values have not).
__device__ __forceinline__ bool has_pieces(const float4& v) {
    return fabsf(v.x) <= SPLIT_MAX && fabsf(v.y) <= SPLIT_MAX && fabsf(v.z) <= SPLIT_MAX && fabsf(v.w) <= SPLIT_MAX;
}

// 8 consecutive values of row `row` (piece g of 8) into the three swizzled planes at `plane0`
__device__ __forceinline__ void put_row8(uint8_t* plane0, int row, int g, const float4& x, const float4& y) {
    uint4 h, m, l;
    cut8(x, y, h, m, l);
    uint8_t* dst = plane0 + row * 128 + ((g ^ (row & 7)) << 4);
    *reinterpret_cast<uint4*>(dst) = h;
    *reinterpret_cast<uint4*>(dst + PLANE) = m;
    *reinterpret_cast<uint4*>(dst + 2 * PLANE) = l;
}

// The rows of a tile, a warp per row in turn: lane l holds the values 2l and 2l + 1 of the head.
__device__ __noinline__ void plain_rows(const float* q, long long q_stride, const float* k_pages, const float* v_pages,
                                        const int* bt, float* out, long long out_stride, int h, int Hkv, int hk,
                                        int page_size, float scale, int window, int tok0, int rows, int pos0) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int r = warp; r < rows; r += SOFTMAX_WARPS) {
        const float2 qv = *reinterpret_cast<const float2*>(q + (size_t)(tok0 + r) * q_stride + (size_t)h * DH + 2 * lane);
        const int qp = pos0 + r;
        float m = -INFINITY, l = 0.f, o0 = 0.f, o1 = 0.f;
        for (int kp = window > 0 && qp - window + 1 > 0 ? qp - window + 1 : 0; kp <= qp; ++kp) {
            const size_t off = (((size_t)bt[kp / page_size] * Hkv + hk) * page_size + kp % page_size) * DH + 2 * lane;
            const float2 kv = *reinterpret_cast<const float2*>(k_pages + off);
            const float2 vv = *reinterpret_cast<const float2*>(v_pages + off);
            const float s = warp_sum(fmaf(qv.y, kv.y, qv.x * kv.x)) * scale;
            const float mn = fmaxf(m, s), muse = mn == -INFINITY ? 0.f : mn;
            const float alpha = expf(m - muse), p = expf(s - muse);
            l = fmaf(l, alpha, p);
            o0 = fmaf(p, vv.x, o0 * alpha);
            o1 = fmaf(p, vv.y, o1 * alpha);
            m = mn;
        }
        *reinterpret_cast<float2*>(out + (size_t)(tok0 + r) * out_stride + (size_t)h * DH + 2 * lane) = make_float2(o0 / l, o1 / l);
    }
}

__global__ void __launch_bounds__(THREADS, 1)
attention_split_f32_kernel(const float* q, long long q_stride, const float* k_pages,        // written by kernels of this step:
                           const float* v_pages, const int* __restrict__ block_table,       // no __restrict__
                           int bt_stride, const int* __restrict__ tiles, const int* __restrict__ positions, float* out,
                           long long out_stride, int H, int Hkv, int page_size, float scale, int window) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sQ = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sK = sQ + 3 * PLANE;
    uint8_t* sV = sK + 3 * PLANE;
    float* xch = reinterpret_cast<float*>(sV + 3 * PLANE);        // [2][PARTS][BQ]
    uint64_t* q_full = (uint64_t*)((uint8_t*)xch + XCH_BYTES);
    uint64_t* k_full = q_full + 1;
    uint64_t* k_empty = k_full + 1;
    uint64_t* v_full = k_empty + 1;
    uint64_t* v_empty = v_full + 1;
    uint64_t* s_full = v_empty + 1;                               // [2]: one per S buffer
    uint64_t* p_full = s_full + 2;
    uint64_t* o_full = p_full + 1;
    uint32_t* tmem_slot = (uint32_t*)(o_full + 1);
    volatile int* failed = (volatile int*)(tmem_slot + 1);
    volatile int* odd = failed + 1;                               // some operand has no pieces

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int h = blockIdx.x, tile = blockIdx.y;
    if (threadIdx.x == 0) {
        mbar_init(q_full, SOFTMAX_WARPS);
        mbar_init(k_full, 4);
        mbar_init(k_empty, 1);
        mbar_init(v_full, 4);
        mbar_init(v_empty, 1);
        mbar_init(&s_full[0], 1);
        mbar_init(&s_full[1], 1);
        mbar_init(p_full, SOFTMAX_WARPS);
        mbar_init(o_full, 1);
        *failed = 0;
        *odd = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int seq = tiles[tile * 3], tok0 = tiles[tile * 3 + 1], rows = tiles[tile * 3 + 2];
    const int pos0 = positions[tok0], pos_max = pos0 + rows - 1;
    const int hk = h / (H / Hkv);
    const int* bt = block_table + (size_t)seq * bt_stride;
    const int first_key = window > 0 && pos0 - window + 1 > 0 ? pos0 - window + 1 : 0;
    const int j_lo = first_key / BKV, nblk = pos_max / BKV - j_lo + 1;
    pdl_wait();
    pdl_launch();

    if (warp >= MMA_WARP) {
        fewer_registers<24>();
        if (warp == MMA_WARP) {
            constexpr uint32_t idesc_s = make_idesc(BQ, BKV), idesc_o = make_idesc_bmn(BQ, DH);
            constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};       // the six products, smallest first
            const uint64_t q_desc = make_smem_desc(smem_u32(sQ)), k_desc = make_smem_desc(smem_u32(sK)),
                           v_desc = make_smem_desc(smem_u32(sV));
            auto all_wait = [&](uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); };
            auto issue_s = [&](int i) {
#pragma unroll
                for (int t = 0; t < 6; ++t)
#pragma unroll
                    for (int k = 0; k < DH / 16; ++k)
                        umma_f16_warp(tmem + (uint32_t)(i & 1) * 128, q_desc + (uint64_t)(PA[t] * (PLANE >> 4) + 2 * k),
                                      k_desc + (uint64_t)(PB[t] * (PLANE >> 4) + 2 * k), idesc_s, (t | k) != 0);
                umma_commit_warp(&s_full[i & 1]);
                umma_commit_warp(k_empty);
            };
            bool ok = all_wait(q_full, 0) && all_wait(k_full, 0);
            if (!ok) *failed = 2;
            if (ok) {
                tc_fence_after();
                issue_s(0);
            }
            for (int i = 0; i < nblk && ok; ++i) {
                if (i + 1 < nblk) {
                    // S of the next block goes ahead of this block's P V: its buffer was read two blocks ago
                    if (!all_wait(k_full, (i + 1) & 1)) { *failed = 3; break; }
                    tc_fence_after();
                    issue_s(i + 1);
                }
                // P(i) is written, and O_blk of block i - 1 was read before it was
                if (!all_wait(p_full, i & 1)) { *failed = 4; break; }
                if (!all_wait(v_full, i & 1)) { *failed = 5; break; }
                tc_fence_after();
#pragma unroll
                for (int t = 0; t < 6; ++t)
#pragma unroll
                    for (int kk = 0; kk < BKV / 16; ++kk)
                        umma_f16_ts_warp(tmem + TMEM_O, tmem + TMEM_P + (uint32_t)(PA[t] * 64 + kk * 8),
                                         v_desc + (uint64_t)(PB[t] * (PLANE >> 4) + kk * (2048 >> 4)), idesc_o, (t | kk) != 0);
                umma_commit_warp(o_full);
                umma_commit_warp(v_empty);
            }
        }
    } else if (warp >= K_WARP) {
        fewer_registers<64>();
        // ------------------------------------------------------------ keys (warps 16-19) and values (20-23): a thread
        // takes 8 values of the rows r0, r0 + 16, ...; the pages of the next half block are looked up ahead of time
        const bool keys = warp < V_WARP;
        const float* pages = keys ? k_pages : v_pages;
        uint64_t* full = keys ? k_full : v_full;
        uint64_t* empty = keys ? k_empty : v_empty;
        uint8_t* dst = keys ? sK : sV;
        const int t = (threadIdx.x - K_WARP * 32) & 127, r0 = t >> 3, g = t & 7;
        int page[4];
        float4 x[4][2];
        auto look_up = [&](int half) {                            // half blocks counted over the tile
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int kp = j_lo * BKV + half * 64 + u * 16 + r0;
                page[u] = half < 2 * nblk && kp <= pos_max && kp >= first_key ? __ldcg(bt + kp / page_size) : -1;
            }
        };
        auto fetch = [&](int half) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int kp = j_lo * BKV + half * 64 + u * 16 + r0;
                x[u][0] = x[u][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (page[u] >= 0) {
                    const float* p = pages + (((size_t)page[u] * Hkv + hk) * page_size + kp % page_size) * DH + g * 8;
                    x[u][0] = *reinterpret_cast<const float4*>(p);
                    x[u][1] = *reinterpret_cast<const float4*>(p + 4);
                }
            }
        };
        bool ok = true, fine = true;
        look_up(0);
        fetch(0);
        look_up(1);
        for (int half = 0; half < 2 * nblk; ++half) {
            if (!(half & 1)) {                                    // the planes are free once the MMAs of the block before have read them
                ok = half == 0 || mbar_wait(empty, ((half >> 1) - 1) & 1);
                if (!ok) *failed = 1;
                ok = __all_sync(0xffffffffu, ok && !*failed);
                if (!ok) break;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                fine &= has_pieces(x[u][0]) && has_pieces(x[u][1]);
                put_row8(dst, (half & 1) * 64 + u * 16 + r0, g, x[u][0], x[u][1]);
            }
            if (half & 1) {
                fence_async_smem();
                __syncwarp();
                if (lane == 0) mbar_arrive(full);
            }
            fetch(half + 1);                                      // (nothing beyond the last: its pages are -1)
            look_up(half + 2);
        }
        if (!fine) *odd = 1;
    } else {
        more_registers<88>();
        // ------------------------------------------------------------ softmax: one query row per thread
        const int q4 = warp & 3, part = warp >> 2;                // quarter of the lanes; which 32 keys and which 16 outputs
        const int r = q4 * 32 + lane, qp = pos0 + r;
        const uint32_t t_lane = tmem + ((uint32_t)(q4 * 32) << 16);
        // the tile's queries in pieces: 16 values of a row per thread
        {
            const int row = threadIdx.x >> 2, g = (threadIdx.x & 3) * 2;
            float4 x[4];
            const float* p = q + (size_t)(tok0 + row) * q_stride + (size_t)h * DH + g * 8;
            bool fine = true;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                x[e] = row < rows ? *reinterpret_cast<const float4*>(p + 4 * e) : make_float4(0.f, 0.f, 0.f, 0.f);
                fine &= has_pieces(x[e]);
            }
            put_row8(sQ, row, g, x[0], x[1]);
            put_row8(sQ, row, g + 1, x[2], x[3]);
            if (!fine) *odd = 1;
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(q_full);
        }
        float o[16];
#pragma unroll
        for (int d = 0; d < 16; ++d) o[d] = 0.f;
        float m_run = -INFINITY, l_part = 0.f, alpha_prev = 1.f;
        // A warp that gave up on a wait stays in step with the three that share its rows: it skips the work but still
        // arrives at their barriers, which also carry whether all of them are still running.
        bool alive = true;
        auto row_barrier = [&](bool fine) -> bool {
            uint32_t all;
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t"
                "setp.ne.b32 p, %1, 0;\n\t"
                "bar.red.and.pred q, %2, %3, p;\n\t"
                "selp.u32 %0, 1, 0, q;\n\t}"
                : "=r"(all) : "r"((uint32_t)fine), "r"(1 + q4), "n"(PARTS * 32) : "memory");
            return all != 0;
        };
        // o = o * alpha + O_blk for the block whose P V was issued last
        auto add_block = [&](int i, float alpha) -> bool {
            bool fine = mbar_wait(o_full, i & 1);
            if (!fine) *failed = 8;
            fine = __all_sync(0xffffffffu, fine && !*failed);
            if (!fine) return false;
            tc_fence_after();
            uint32_t w[16];
            tmem_ld16_issue(t_lane + TMEM_O + part * 16, w);
            tmem_ld_wait();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = fmaf(o[e], alpha, __uint_as_float(w[e]));
            return true;
        };
        for (int i = 0; i < nblk; ++i) {
            const int j = j_lo + i, k0 = j * BKV + part * 32;     // first key of this thread's 32
            if (alive) {
                bool got = mbar_wait(&s_full[i & 1], (i >> 1) & 1);
                if (!got) *failed = 7;
                alive = __all_sync(0xffffffffu, got && !*failed);
            }
            const bool need_mask = (j * BKV + BKV - 1 > pos0) || (window > 0);     // uniform over the CTA
            uint32_t v[32];
            float mx = -INFINITY;
            if (alive) {
                tc_fence_after();
                tmem_ld32_issue(t_lane + (uint32_t)(i & 1) * 128 + part * 32, v);
                tmem_ld_wait();
#pragma unroll
                for (int e = 0; e < 32; ++e) {
                    float sv = __uint_as_float(v[e]) * scale;
                    if (need_mask && (k0 + e > qp || (window > 0 && k0 + e <= qp - window))) sv = -INFINITY;
                    v[e] = __float_as_uint(sv);
                    mx = fmaxf(mx, sv);
                }
            }
            // the row's maximum over the block: the four threads of the row meet in shared memory
            float* xb = xch + (i & 1) * PARTS * BQ;
            xb[part * BQ + r] = mx;
            alive = row_barrier(alive);
            if (!alive) continue;                                 // all four warps of the quarter take this branch together
#pragma unroll
            for (int p = 0; p < PARTS; ++p) mx = fmaxf(mx, xb[p * BQ + r]);
            const float m_new = fmaxf(m_run, mx);
            const float muse = m_new == -INFINITY ? 0.f : m_new;
            const float alpha = expf(m_run - muse);
            m_run = m_new;
            float rs = 0.f;
#pragma unroll
            for (int e = 0; e < 32; ++e) {
                const float p = expf(__uint_as_float(v[e]) - muse);
                rs += p;
                v[e] = __float_as_uint(p);
            }
            l_part = l_part * alpha + rs;
            // the block before this one: its P V has had the time of this block's exponentials; P's place is free after it
            if (i > 0) alive = add_block(i - 1, alpha_prev);
            alpha_prev = alpha;
            if (alive) {
                const uint32_t tp = t_lane + TMEM_P + part * 16;
#pragma unroll
                for (int c = 0; c < 2; ++c) {                     // 16 keys = 8 columns of each piece
                    uint4 h4[2], m4[2], l4[2];
#pragma unroll
                    for (int d = 0; d < 2; ++d) {
                        const uint32_t* s = v + c * 16 + d * 8;
                        cut8(make_float4(__uint_as_float(s[0]), __uint_as_float(s[1]), __uint_as_float(s[2]), __uint_as_float(s[3])),
                             make_float4(__uint_as_float(s[4]), __uint_as_float(s[5]), __uint_as_float(s[6]), __uint_as_float(s[7])),
                             h4[d], m4[d], l4[d]);
                    }
                    tmem_st8(tp + c * 8, h4[0], h4[1]);
                    tmem_st8(tp + 64 + c * 8, m4[0], m4[1]);
                    tmem_st8(tp + 128 + c * 8, l4[0], l4[1]);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full);
            }
        }
        if (alive) alive = add_block(nblk - 1, alpha_prev);
        // the row's sum: the four partial sums added in a fixed order
        alive = row_barrier(alive);                               // the last maxima have been read
        xch[part * BQ + r] = l_part;
        alive = row_barrier(alive);
        if (alive && r < rows) {
            float l = 0.f;
#pragma unroll
            for (int p = 0; p < PARTS; ++p) l += xch[p * BQ + r];
            float* orow = out + (size_t)(tok0 + r) * out_stride + (size_t)h * DH + part * 16;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *reinterpret_cast<float4*>(orow + c * 4) = make_float4(o[c * 4] / l, o[c * 4 + 1] / l, o[c * 4 + 2] / l, o[c * 4 + 3] / l);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*failed) {
        if (threadIdx.x == 0) { atomicCAS(&g_attn_split_error, 0, *failed); report_to_host(700 + *failed); }
        for (int i = 0; i < 2000; ++i) __nanosleep(100);          // MMAs already issued may still be running
        __syncthreads();
    } else if (*odd && warp < SOFTMAX_WARPS) {
        plain_rows(q, q_stride, k_pages, v_pages, bt, out, out_stride, h, Hkv, hk, page_size, scale, window, tok0, rows, pos0);
    }
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace

// The pinned host word that this file's kernel writes when it gives up on a wait.
MLLM_EXPORT int mllm_attention_split_f32_bind_error(int* word) { return bind_host_error(word); }

// The first error recorded since the last call (0 = none); resets it.
MLLM_EXPORT int mllm_attention_split_f32_error(int* code) {
    int zero = 0;
    MLLM_CUDA(cudaMemcpyFromSymbol(code, g_attn_split_error, sizeof(int)));
    if (*code) MLLM_CUDA(cudaMemcpyToSymbol(g_attn_split_error, &zero, sizeof(int)));
    return 0;
}

// 32-bit q [T, H*64] (row stride q_stride), pages [pages, Hkv, page_size, 64], out [T, H*64]; tiles: (request, first flat
// token, rows <= 128) triples.  Row strides multiples of 4 and everything 16-byte aligned.
MLLM_EXPORT int mllm_attention_split_f32(const float* q, long long q_stride, const float* k_pages, const float* v_pages,
                                         const int* block_table, int bt_stride, const int* tiles, int n_tiles,
                                         const int* positions, float* out, long long out_stride, int H, int Hkv, int dh,
                                         int page_size, float scale, int window, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (dh != DH) return mllm_fail(1, "attention_split_f32: head size %d, this kernel takes %d", dh, DH);
    if (H <= 0 || Hkv <= 0 || H % Hkv || page_size <= 0 || n_tiles > 65535)
        return mllm_fail(1, "attention_split_f32: %d heads over %d, page size %d, %d tiles", H, Hkv, page_size, n_tiles);
    if (((uintptr_t)q | (uintptr_t)k_pages | (uintptr_t)v_pages | (uintptr_t)out) % 16 || q_stride % 4 || out_stride % 4)
        return mllm_fail(1, "attention_split_f32: rows must be 16-byte aligned");
    static bool set = false;
    if (!set) {
        MLLM_CUDA(cudaFuncSetAttribute(attention_split_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
        set = true;
    }
    MLLM_CUDA(mllm_launch(attention_split_f32_kernel, dim3(H, n_tiles), dim3(THREADS), SMEM, stream, true, q, q_stride, k_pages,
                          v_pages, block_table, bt_stride, tiles, positions, out, out_stride, H, Hkv, page_size, scale, window));
    return 0;
}
