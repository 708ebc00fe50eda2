// out = act(A[M,K] . W[N,K]^T + bias) (+ out) with 32-bit operands and more than 64 rows, on the fifth-generation
// tensor cores: the product of prefill and mixed steps on the 32-bit path.
//
// A 32-bit value x is cut exactly into three bfloat16 pieces, x = h + m + l, by rounding to nearest twice (split_f32.cuh).
// Of the nine products of pieces the six largest are formed: hh, hm, mh, mm, hl, lh; the rest is at most 2^-24 of |a w|
// and has either sign.  A product of two bfloat16 is exact in the tensor core.
// The tensor memory holds the sum over 64 of K only: every 64 wide block is read out and added to a sum in registers
// by plain 32-bit additions, and within a block the small terms come first, so that the accumulator's own rounding
// (which drops bits instead of rounding to nearest) meets only 4 additions of full-size terms.  Against float64 the
// result is closer than a chain of fmaf over K (see tests/test_kernels_gpu.py for the comparison).
//
// Work of a (persistent) CTA on a 128 x BN tile, 64 of K at a time:
//  * warp 17 brings 32-bit boxes of A and W, 32 of K each, into a ring of shared-memory slots with TMA;
//  * warps 0-7 cut them: A's pieces go to tensor memory (a thread owns a row, as the MMA's A operand wants it), W's
//    pieces to swizzled shared memory, two stages of each.  A in tensor memory halves what the MMAs read from shared
//    memory, whose bandwidth is the bound: copies in, cutting and MMAs pass 272 KB of it per block of BN = 128, 2,125
//    cycles against the MMAs' 1,400; a block takes 2,600 to 2,800 (sixteen cutting warps: the same);
//  * warp 16 issues 24 tcgen05.mma (128 x BN x 16) per block into one of two accumulators;
//  * warps 8-15 drain the accumulators and run the epilogue.
// The sum over K of an element runs in an order that depends on K alone.
//
// An element whose sum is not finite (an operand is infinite, NaN or above the largest bfloat16, or the sum overflows:
// inf - inf appears in the pieces) is computed again as a chain of fmaf over the 32-bit operands, so infinities come out as they should.
//
// Every wait is bounded: after the limit the kernel records an error code, frees its tensor memory and returns.
#include "tcgen05.cuh"
#include "split_f32.cuh"

namespace {

using namespace tc;

constexpr int BM = 128, BK = 64, HK = 32;                  // a block of K, and the half of it that a ring slot holds
constexpr int CUT_WARPS = 8, EPI_WARPS = 8;
constexpr int MMA_WARP = CUT_WARPS + EPI_WARPS, TMA_WARP = MMA_WARP + 1;
constexpr int THREADS = (CUT_WARPS + EPI_WARPS + 4) * 32;      // five warpgroups; of the last one two warps work
// Registers: 640 threads x 96 = 61,440 at launch; 256 x 80 + 256 x 120 + 128 x 40 = 56,320 after the split.
__device__ int g_split_error = 0;

template <int BN> struct Cfg {
    static constexpr int W_PLANE = BN * BK * 2;                             // one piece of a block of W
    static constexpr int W_STAGE = 3 * W_PLANE;
    static constexpr int A_SLOT = BM * HK * 4, SLOT = A_SLOT + BN * HK * 4; // 32-bit boxes of a half block
    static constexpr int SLOTS = 98304 / SLOT + (BN == 64 ? 2 : 0);         // 3 (BN = 128), 6 (BN = 64)
    static constexpr int EPI_BYTES = EPI_WARPS * 4096;                      // 32 x 32 floats per warp
    static constexpr size_t SMEM = 2 * (size_t)W_STAGE + (size_t)SLOTS * SLOT + EPI_BYTES + 1024 /*alignment*/ + 256 /*barriers*/;
    static constexpr int HALF = BN / 2;                                     // columns per epilogue warp
    static constexpr int A_COLS = 3 * BK / 2;                               // tensor-memory columns of a stage of A
};

// Where the key and value columns of a Q|K|V projection go (k_pages null: a plain product); see linear_tcgen05.cu.
struct KvOut32 {
    float* k_pages;
    float* v_pages;
    const int* slots;
    int q_size, kv_heads, head_dim, page_size;
};

template <int BN>
__global__ void __launch_bounds__(THREADS, 1)
linear_split_f32_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                        const __grid_constant__ CUtensorMap map_o, const float* A, long long lda,
                        const float* __restrict__ W, const float* __restrict__ bias, float* out, long long ldo, int M,
                        int N, int K, int act, int accumulate, int tma_out, int tiles_n, int num_items, int slices, KvOut32 kv) {
    using C = Cfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* w_stages = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = w_stages + 2 * (size_t)C::W_STAGE;
    uint8_t* epi = ring + (size_t)C::SLOTS * C::SLOT;
    uint64_t* full = (uint64_t*)(epi + C::EPI_BYTES);      // [2] a stage's pieces are written
    uint64_t* empty = full + 2;                            // [2] its MMAs have read them
    uint64_t* acc_full = empty + 2;                        // [2] a block's sums are complete
    uint64_t* acc_empty = acc_full + 2;                    // [2] they have been read out
    uint64_t* raw_full = acc_empty + 2;                    // [SLOTS] the 32-bit boxes have arrived
    uint64_t* raw_empty = raw_full + C::SLOTS;             // [SLOTS] they have been cut
    uint32_t* tmem_slot = (uint32_t*)(raw_empty + C::SLOTS);
    volatile int* failed = (volatile int*)(tmem_slot + 1);

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    // An item is a K slice of a tile (slices of whole blocks, all equally long: blocks beyond K are zeros).
    const int nk = ((K + BK - 1) / BK + slices - 1) / slices;
    const int my_items = (num_items - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;       // the grid has no more CTAs than items
    const int steps = my_items * nk;
    if (threadIdx.x == 32) {
        prefetch_map(&map_a);
        if (tma_out) prefetch_map(&map_o);
    }
    if (threadIdx.x == 0) {
        prefetch_map(&map_w);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full[s], CUT_WARPS);
            mbar_init(&empty[s], 1);
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], EPI_WARPS);
        }
        for (int s = 0; s < C::SLOTS; ++s) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], CUT_WARPS);
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) tmem_alloc(tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a = tmem_base + 2 * BN;            // [2] stages of A's pieces behind the two accumulators

    if (warp < CUT_WARPS) {
        fewer_registers<80>();
        pdl_wait();
        pdl_launch();
        // A: this thread's row and half (16 values) of a half block.  W: row and run of 8 values; rows are dealt to the
        // lanes so that 8 neighbouring lanes hit all banks in the reads (with the two 16-byte pieces taken in turn) and
        // in the writes.
        const int row_a = (warp & 3) * 32 + lane, part = warp >> 2;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const int li = lane >> 2, g = lane & 3, swap = li & 1;
        const int row_w = warp * 8 + (li >> 1) + (swap << 2);          // + 64 per round
        int slot = 0;
        uint32_t parity = 0;
        bool ok = true;
        for (int it = 0; it < steps && ok; ++it) {
            const int s = it & 1;
            ok = it < 2 || mbar_wait(&empty[s], ((it >> 1) - 1) & 1);
            if (!ok) *failed = 1;
            tc_fence_after();
            uint8_t* st = w_stages + (size_t)s * C::W_STAGE;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (ok && !mbar_wait(&raw_full[slot], parity)) { *failed = 5; ok = false; }
                ok = __all_sync(0xffffffffu, ok && !*failed);
                if (!ok) break;
                // every value is read before the first is cut, so that the reads' latency is met once
                const uint8_t* raw = ring + (size_t)slot * C::SLOT;
                float4 x[4], y[BN / 64][2];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    x[j] = *reinterpret_cast<const float4*>(raw + row_a * 128 + (((part * 4 + j) ^ (row_a & 7)) << 4));
#pragma unroll
                for (int i = 0; i < BN / 64; ++i) {
                    const int row = row_w + i * 64;
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        y[i][j] = *reinterpret_cast<const float4*>(raw + C::A_SLOT + row * 128 + (((2 * g + (j ^ swap)) ^ (row & 7)) << 4));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[slot]);
                if (++slot == C::SLOTS) { slot = 0; parity ^= 1; }
                const uint32_t ta = tmem_a + lane_off + (uint32_t)(s * C::A_COLS + half * 16 + part * 8);
                uint4 h[2], m[2], l[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) cut8(x[2 * j], x[2 * j + 1], h[j], m[j], l[j]);
                tmem_st8(ta, h[0], h[1]);
                tmem_st8(ta + BK / 2, m[0], m[1]);
                tmem_st8(ta + BK, l[0], l[1]);
#pragma unroll
                for (int i = 0; i < BN / 64; ++i) {
                    const int row = row_w + i * 64;
                    uint8_t* dst = st + row * 128 + (((half * 4 + g) ^ (row & 7)) << 4);
                    cut8(swap ? y[i][1] : y[i][0], swap ? y[i][0] : y[i][1], h[0], m[0], l[0]);
                    *reinterpret_cast<uint4*>(dst) = h[0];
                    *reinterpret_cast<uint4*>(dst + C::W_PLANE) = m[0];
                    *reinterpret_cast<uint4*>(dst + 2 * C::W_PLANE) = l[0];
                }
            }
            if (!ok) break;
            tmem_st_wait();
            tc_fence_before();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    } else if (warp >= MMA_WARP) {
        fewer_registers<40>();
        if (warp == TMA_WARP) {
            const int total = 2 * steps, pre = total < C::SLOTS ? total : C::SLOTS;
            // the half block that is brought next, counted up (a division per box would cost as much as its copy)
            struct Next { int item, m0, n0, k, k_end, slot; } w{(int)blockIdx.x, 0, 0, 0, 0, 0};
            auto place = [&](Next& x) {
                const int tile = x.item / slices;
                x.m0 = (tile / tiles_n) * BM;
                x.n0 = (tile % tiles_n) * BN;
                x.k = (x.item % slices) * nk * BK;
                x.k_end = x.k + nk * BK;
            };
            auto step = [&](Next& x) {
                if (++x.slot == C::SLOTS) x.slot = 0;
                x.k += HK;
                if (x.k == x.k_end) { x.item += gridDim.x; place(x); }
            };
            place(w);
            Next a = w;
            for (int hb = 0; hb < pre; ++hb) {             // weights: written by no kernel of the step
                mbar_expect_tx_warp(&raw_full[w.slot], C::SLOT);
                tma_load_2d_warp(ring + (size_t)w.slot * C::SLOT + C::A_SLOT, &map_w, w.k, w.n0, &raw_full[w.slot]);
                step(w);
            }
            pdl_wait();
            pdl_launch();
            for (int hb = 0; hb < pre; ++hb) {
                tma_load_2d_warp(ring + (size_t)a.slot * C::SLOT, &map_a, a.k, a.m0, &raw_full[a.slot]);
                step(a);
            }
            uint32_t parity = 0;
            for (int hb = pre; hb < total; ++hb) {
                if (!__all_sync(0xffffffffu, mbar_wait(&raw_empty[w.slot], parity) && !*failed)) {
                    if (!*failed) *failed = 6;
                    break;
                }
                mbar_expect_tx_warp(&raw_full[w.slot], C::SLOT);
                tma_load_2d_warp(ring + (size_t)w.slot * C::SLOT + C::A_SLOT, &map_w, w.k, w.n0, &raw_full[w.slot]);
                tma_load_2d_warp(ring + (size_t)w.slot * C::SLOT, &map_a, w.k, w.m0, &raw_full[w.slot]);
                step(w);
                if (w.slot == 0) parity ^= 1;
            }
        } else {
            pdl_wait();
            pdl_launch();
        }
        if (warp == MMA_WARP) {
            constexpr uint32_t idesc = make_idesc(BM, BN);
            // (piece of A, piece of W) of the six products, smallest first
            constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};
            const uint64_t desc0 = make_smem_desc(smem_u32(w_stages));
            for (int it = 0; it < steps; ++it) {
                const int s = it & 1;
                if (it >= 2 && !__all_sync(0xffffffffu, mbar_wait(&acc_empty[s], ((it >> 1) - 1) & 1))) { *failed = 2; break; }
                if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (it >> 1) & 1))) { *failed = 3; break; }
                tc_fence_after();
                const uint64_t dw = desc0 + (uint64_t)(s * (C::W_STAGE >> 4));
                const uint32_t d = tmem_base + (uint32_t)(s * BN), ta = tmem_a + (uint32_t)(s * C::A_COLS);
#pragma unroll
                for (int t = 0; t < 6; ++t)
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k)
                        umma_f16_ts_warp(d, ta + (uint32_t)(PA[t] * (BK / 2) + k * 8), dw + (uint64_t)(PW[t] * (C::W_PLANE >> 4) + 2 * k),
                                         idesc, (t | k) != 0);
                umma_commit_warp(&empty[s]);
                umma_commit_warp(&acc_full[s]);
            }
        }
    } else {
        more_registers<120>();
        pdl_wait();
        pdl_launch();
        const int q = warp & 3, half = (warp - CUT_WARPS) >> 2;
        uint8_t* blk = epi + (size_t)(warp - CUT_WARPS) * 4096;
        int it = 0;
        bool ok = true;
        const int slice_rows = (M + BM - 1) / BM * BM;     // slice z of the partial sums: rows z * slice_rows ... of `out`
        for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
            const int tile = item / slices, slice = item % slices, k0 = slice * nk * BK;
            float acc[C::HALF];
#pragma unroll
            for (int j = 0; j < C::HALF; ++j) acc[j] = 0.f;
            for (int kb = 0; kb < nk; ++kb, ++it) {
                const int s = it & 1;
                ok = mbar_wait(&acc_full[s], (it >> 1) & 1);
                if (!ok) *failed = 4;
                ok = __all_sync(0xffffffffu, ok && !*failed);
                if (!ok) break;
                tc_fence_after();
                const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * BN + half * C::HALF);
#pragma unroll
                for (int c = 0; c < C::HALF / 16; ++c) {
                    uint32_t r[16];
                    tmem_ld16_issue(t_addr + c * 16, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c * 16 + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[s]);
            }
            if (!ok) break;
            const int row0 = (tile / tiles_n) * BM + q * 32, row = row0 + lane;
#pragma unroll
            for (int c = 0; c < C::HALF / 32; ++c) {
                const int n0 = (tile % tiles_n) * BN + half * C::HALF + c * 32;
                if (n0 >= N || row0 >= M) continue;        // the whole warp alike
                float* v = acc + c * 32;
                bool odd = false;
#pragma unroll
                for (int j = 0; j < 32; ++j) odd |= !(fabsf(v[j]) <= 3.402823466e38f);
                if (odd && row < M) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (!(fabsf(v[j]) <= 3.402823466e38f) && n0 + j < N)
                            v[j] = plain_dot(A + (size_t)row * lda + k0, W + (size_t)(n0 + j) * K + k0, min(K - k0, nk * BK));
                }
                __syncwarp();
                if (bias) {
                    const float mine = n0 + lane < N ? __ldg(bias + n0 + lane) : 0.f;
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] += __shfl_sync(0xffffffffu, mine, j);
                }
                if (act == MLLM_ACT_GELU_TANH) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = gelu_tanh_f(v[j]);
                } else if (act == MLLM_ACT_GELU_ERF) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = gelu_erf_f(v[j]);
                }
                if (kv.k_pages && n0 >= kv.q_size) {       // 32 columns lie inside one head: head_dim is a multiple of 32
                    const int slot = row < M ? kv.slots[row] : -1;
                    if (slot >= 0) {
                        const int cc = n0 - kv.q_size, kvs = kv.kv_heads * kv.head_dim;
                        const int c2 = cc % kvs, head = c2 / kv.head_dim, d0 = c2 % kv.head_dim;
                        float* dst = (cc < kvs ? kv.k_pages : kv.v_pages) +
                            (((size_t)(slot / kv.page_size) * kv.kv_heads + head) * kv.page_size + slot % kv.page_size) *
                                kv.head_dim + d0;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            *reinterpret_cast<float4*>(dst + 4 * j) =
                                make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    }
                    continue;
                }
                if (tma_out && lane == 0) bulk_wait_read();     // the copy engine has read the block before
                __syncwarp();
                uint8_t* rowp = blk + lane * 128;               // lane = row, 16-byte pieces swizzled by the row
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    *reinterpret_cast<float4*>(rowp + ((j ^ (lane & 7)) << 4)) =
                        make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                if (tma_out) {
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        if (accumulate) tma_reduce_add_2d(&map_o, n0, row0, blk);
                        else tma_store_2d(&map_o, n0, slice * slice_rows + row0, blk);
                        bulk_commit();
                    }
                } else {                                        // rows that are not 16-byte aligned: lane = column
                    __syncwarp();
                    const int n = n0 + lane;
#pragma unroll 4
                    for (int rr = 0; rr < 32; ++rr) {
                        if (row0 + rr >= M || n >= N) continue;
                        float x = *reinterpret_cast<const float*>(blk + rr * 128 + (((lane >> 2) ^ (rr & 7)) << 4) + (lane & 3) * 4);
                        float* o = out + (size_t)(row0 + rr) * ldo + n;
                        if (accumulate) x += *o;
                        *o = x;
                    }
                }
            }
        }
        if (lane == 0 && tma_out) bulk_wait_all();
    }
    tc_fence_before();
    __syncthreads();
    if (*failed) {
        if (threadIdx.x == 0) { atomicCAS(&g_split_error, 0, *failed); report_to_host(500 + *failed); }
        for (int i = 0; i < 2000; ++i) __nanosleep(100);       // copies and MMAs already issued may still be running
        __syncthreads();
    }
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

// out = act(ws[0] + ws[1] + ... + bias) (+ out): the K slices of the kernel above, added in slice order, four columns per
// thread.
__global__ void __launch_bounds__(256)
linear_split_f32_finish_kernel(const float* ws, int slices, size_t slice_floats, const float* __restrict__ bias, float* out,
                               long long ldo, int M, int N, int act, int accumulate, int vec) {
    const int n4 = N / 4, total = M * n4;
    pdl_wait();
    pdl_launch();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const int m = i / n4, n = (i - m * n4) * 4;
        float* o = out + (size_t)m * ldo + n;
        float4 old = make_float4(0.f, 0.f, 0.f, 0.f);
        if (accumulate) old = vec ? *reinterpret_cast<const float4*>(o) : make_float4(o[0], o[1], o[2], o[3]);
        const float4 b = bias ? make_float4(__ldg(bias + n), __ldg(bias + n + 1), __ldg(bias + n + 2), __ldg(bias + n + 3))
                              : make_float4(0.f, 0.f, 0.f, 0.f);
        const float* p = ws + (size_t)m * N + n;
        float4 v = __ldcg(reinterpret_cast<const float4*>(p));
#pragma unroll 3
        for (int z = 1; z < slices; ++z) {
            const float4 x = __ldcg(reinterpret_cast<const float4*>(p + (size_t)z * slice_floats));
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        v.x = apply_act(v.x + b.x, act) + old.x;
        v.y = apply_act(v.y + b.y, act) + old.y;
        v.z = apply_act(v.z + b.z, act) + old.z;
        v.w = apply_act(v.w + b.w, act) + old.w;
        if (vec) *reinterpret_cast<float4*>(o) = v;
        else { o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w; }
    }
}

int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    }
    return n;
}

// K slices, from N and K alone (a row's sum must not depend on the rows beside it): a narrow result has few tiles, each of
// which walks all of K on its SM.  Three slices give most where rows are few and take an extra write and read of the sums
// where the tiles fill the GPU without them.  us with one / three slices:
//     rows              77          552         2,048        8,192
//      768 x  768    19 / 14     21 / 18      27 / 27      64 / 79
//      768 x 3072    56 / 27     58 / 36      78 / 63     216 / 219
//     1024 x 1024    23 / 16     25 / 21      34 / 42     104 / 136
//     1024 x 4096    72 / 33     78 / 46     103 / 111    380 / 391
//      768 x  512    15 / 13     16 / 16      21 / 24      47 / 65     shorter rows gain less than they lose (384: 13 / 12,
//      768 x  256    11 / 12     12 / 14      14 / 20      29 / 51     14 / 14, 18 / 20, 38 / 52)
//     1600 x 1024    23 / 16     26 / 30      57 / 63     152 / 204    wider results lose from 552 rows on, 1,280 as well
//     1600 x 4096    76 / 38     82 / 81     193 / 180    570 / 619    (4096: 77 / 38, 85 / 79, 194 / 144, 478 / 472)
// 768 x 3072 with two / three / four slices: 34 / 27 / 23 at 77 rows, 36 / 36 / 30 at 552, 47 / 37 / 48 at 1,024, 83 / 63 /
// 68 at 2,048.
int slices_for(int N, int K) { return N <= 1024 && N % 4 == 0 && K >= 512 ? 3 : 1; }

template <int BN>
int launch(const float* A, long long lda, const float* W, const float* bias, float* out, long long ldo, int M, int N,
           int K, int act, int accumulate, float* ws, int slices, const KvOut32& kv, cudaStream_t stream) {
    using C = Cfg<BN>;
    CUtensorMap ma, mw, mo = {};
    int rc = get_map(A, lda, M, K, HK, BM, MAP_F32_SW128, &ma);
    if (rc) return rc;
    rc = get_map(W, K, N, K, HK, BN, MAP_F32_SW128, &mw);
    if (rc) return rc;
    const int tiles_n = (N + BN - 1) / BN, tiles_m = (M + BM - 1) / BM;
    const int vec = (uintptr_t)out % 16 == 0 && ldo % 4 == 0, tma_out = slices > 1 || vec;
    if (slices > 1) rc = get_map(ws, N, slices * tiles_m * BM, N, 32, 32, MAP_F32_SW128, &mo);
    else if (tma_out) rc = get_map(out, ldo, M, kv.k_pages ? kv.q_size : N, 32, 32, MAP_F32_SW128, &mo);
    if (rc) return rc;
    auto kern = linear_split_f32_kernel<BN>;
    static bool set = false;
    if (!set) {
        MLLM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
        set = true;
    }
    const int items = tiles_n * tiles_m * slices, grid = items < sm_count() ? items : sm_count();
    if (slices == 1) {
        MLLM_CUDA(mllm_launch(kern, dim3(grid), dim3(THREADS), C::SMEM, stream, true, ma, mw, mo, A, lda, W, bias, out, ldo, M, N,
                              K, act, accumulate, tma_out, tiles_n, items, 1, kv));
        return 0;
    }
    MLLM_CUDA(mllm_launch(kern, dim3(grid), dim3(THREADS), C::SMEM, stream, true, ma, mw, mo, A, lda, W, (const float*)nullptr, ws,
                          (long long)N, M, N, K, (int)MLLM_ACT_NONE, 0, tma_out, tiles_n, items, slices, kv));
    const long long quads = (long long)M * N / 4;
    MLLM_CUDA(mllm_launch(linear_split_f32_finish_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, stream, true,
                          (const float*)ws, slices, (size_t)tiles_m * BM * N, bias, out, ldo, M, N, act, accumulate, vec));
    return 0;
}

int go(const float* A, long long lda, const float* W, const float* bias, float* out, long long ldo, int M, int N, int K,
       int act, int accumulate, float* ws, long long ws_floats, const KvOut32& kv, cudaStream_t stream) {
    if (K <= 0 || K % 4 != 0 || lda % 4 != 0)
        return mllm_fail(1, "linear_split_f32: K=%d and the row stride %lld must be multiples of 4", K, lda);
    if ((uintptr_t)A % 16 != 0 || (uintptr_t)W % 16 != 0)
        return mllm_fail(1, "linear_split_f32: operands must be 16-byte aligned");
    const long long tiles_m = (M + BM - 1) / BM;
    if (tiles_m * ((N + 63) / 64) > 0x7fffffffLL) return mllm_fail(1, "linear_split_f32: M=%d, N=%d exceed the grid limit", M, N);
    int slices = ws && !kv.k_pages ? slices_for(N, K) : 1;
    if (slices > 1 && (slices * tiles_m * BM * N > ws_floats || (uintptr_t)ws % 16 != 0 || (long long)M * N > 0x3fffffffLL))
        return mllm_fail(1, "linear_split_f32: %lld floats of scratch for %d slices of %d x %d", ws_floats, slices, M, N);
    // A 64-wide tile takes about three quarters of a 128-wide one's time (1.08 against 1.45 us per block of 64: what
    // W costs halves, the cutting of A stays).
    const long long r128 = (tiles_m * ((N + 127) / 128) * slices + sm_count() - 1) / sm_count();
    const long long r64 = (tiles_m * ((N + 63) / 64) * slices + sm_count() - 1) / sm_count();
    if (r64 * 3 < r128 * 4) return launch<64>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, ws, slices, kv, stream);
    return launch<128>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, ws, slices, kv, stream);
}

}  // namespace

// The pinned host word that this file's kernel writes when it gives up on a wait.
MLLM_EXPORT int mllm_linear_split_f32_bind_error(int* word) { return bind_host_error(word); }

// The first error recorded since the last call (0 = none); resets it.
MLLM_EXPORT int mllm_linear_split_f32_error(int* code) {
    int zero = 0;
    MLLM_CUDA(cudaMemcpyFromSymbol(code, g_split_error, sizeof(int)));
    if (*code) MLLM_CUDA(cudaMemcpyToSymbol(g_split_error, &zero, sizeof(int)));
    return 0;
}

// K slices that mllm_linear_split_f32 uses (1: no scratch needed, no second kernel).
MLLM_EXPORT int mllm_linear_split_f32_slices(int N, int K) { return slices_for(N, K); }

// 32-bit A [M,K] (row stride lda), W [N,K] and out; K and lda multiples of 4, A and W 16-byte aligned.  ws: room for the
// partial sums, slices * (M rounded up to 128) * N floats, 16-byte aligned (null: no slices).
MLLM_EXPORT int mllm_linear_split_f32(const float* A, long long lda, const float* W, const float* bias, float* out,
                                      long long ldo, int M, int N, int K, int act, int accumulate, float* ws,
                                      long long ws_floats, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    return go(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, ws, ws_floats, KvOut32{}, stream);
}

// The Q|K|V projection with the cache write fused in: out [M, q_size] receives the query columns, keys and values go
// to their page slots (slots[m] = page * page_size + offset, negative: not stored); q_size and head_dim multiples of 32.
// It never cuts K, so where mllm_linear_split_f32 would, the sums of the two run in different orders.
MLLM_EXPORT int mllm_linear_split_f32_qkv(const float* A, long long lda, const float* W, const float* bias, float* out,
                                          long long ldo, int M, int N, int K, float* k_pages, float* v_pages,
                                          const int* slots, int q_size, int kv_heads, int head_dim, int page_size,
                                          cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (q_size <= 0 || q_size % 32 || head_dim <= 0 || head_dim % 32 || kv_heads <= 0 || page_size <= 0 ||
        N != q_size + 2 * kv_heads * head_dim)
        return mllm_fail(1, "linear_split_f32: %d output columns do not split into %d query and 2 x %d x %d cache columns "
                            "in blocks of 32", N, q_size, kv_heads, head_dim);
    if ((uintptr_t)k_pages % 16 || (uintptr_t)v_pages % 16) return mllm_fail(1, "linear_split_f32: the pages must be 16-byte aligned");
    KvOut32 kv{k_pages, v_pages, slots, q_size, kv_heads, head_dim, page_size};
    return go(A, lda, W, bias, out, ldo, M, N, K, MLLM_ACT_NONE, 0, nullptr, 0, kv, stream);
}
