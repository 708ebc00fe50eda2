// out = act(A[M,K] . W[N,K]^T + bias) (+ out) with 32-bit operands and up to 64 rows, on the fifth-generation tensor
// cores: the products of decode batches of more than 16 tokens on the 32-bit path, and their vocabulary.
//
// The arithmetic is that of linear_split_f32.cu: operands cut exactly into three bfloat16 pieces (split_f32.cuh), the six
// largest of the nine products of pieces on tcgen05.mma, smallest first, the accumulator holding 64 of K, every block of 64
// added to 32-bit registers.  The roles are swapped as in linear_cluster.cu: 128 rows of W are the M side (their pieces lie
// in tensor memory), the 32 or 64 rows of A (zeros beyond M) the N side, and K is cut over the CTAs of a cluster.
//
// What bounds it: on CUDA cores a weight costs one fmaf per row of A, 64 of them per 4 bytes, so 64 rows ran at the rate
// of the cores' operands (7 MB of weights: 16 us against 1.1 us from HBM).  Here a block of 128 x 64 weights costs 1.1 to 1.3 us
// whatever the rows: the eight cutting warps' reads, arithmetic and stores, about 2,000 cycles (sixteen of them, half blocks as the
// unit of hand-over and a deeper ring changed nothing).  Layer matrices are bound by the chain of latencies (weights, cut, MMAs,
// exchange of the sums), a vocabulary by the cutting.  Chains of matrices that are not in L2, us here / in the kernel of
// linear_stream_f32.cu that took them before, at 24, 40 and 64 rows:
//   2304 x  768   8.0 /  11.4    9.2 / 15.6    9.7 /  16.0       3072 x  768   9.4 /  9.9   11.0 / 14.3   11.5 /  21.1
//    768 x  768   6.7 /   6.9    7.8 /  9.5    8.2 /   9.5        768 x 3072  11.4 /  9.8   13.1 / 13.2   13.3 /  19.6
//   4096 x 1024  10.4 /  12.0   12.0 / 17.0   12.4 /  33.3       1024 x 4096  13.7 / 14.0   15.6 / 19.4   15.7 /  28.9
//   4800 x 1600  15.5 /  34.0   17.7 / 55.0   18.3 /  57.3       1600 x 6400  19.2 / 33.5   21.7 / 49.2   21.9 /  76.5
//  50257 x  768  45   /  70     54   / 106    55   / 162        50257 x 1024  57   / 83     67   / 128    67   / 289
//
// Work of a CTA, 64 of K at a time:
//  * warp 17 brings 32-bit boxes of 32 of K into four slots with TMA, the weights' before the wait on the previous kernel;
//  * warps 0-7 cut them: W's pieces to tensor memory (a thread owns a row; also before the wait), A's to swizzled shared
//    memory, two stages of each;
//  * warp 16 issues 24 tcgen05.mma (128 x 32|64 x 16) per block into one of two accumulators;
//  * warps 8-15 drain the accumulators.
// The CTAs of a cluster then share the rows of A among them: each writes its sums of a row into the shared memory of the
// row's owner, and after one cluster barrier the owner adds them in rank order and runs the epilogue.  A matrix with more
// tiles than SMs is not cut along K; its CTAs stay and walk the tiles.
// Slices follow from N and K alone and the sums' order from K and the slices: a row's bits do not depend on its neighbours.
//
// An element whose sum is not finite is computed again as a chain of fmaf, as in linear_split_f32.cu.
// Every wait is bounded: after the limit the kernel records an error code, frees its tensor memory and returns.
#include "split_f32.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

using namespace tc;

constexpr int WM = 128, BK = 64, HK = 32;                  // rows of W per tile, a block of K and the half that a slot holds
constexpr int CUT_WARPS = 8, SUM_WARPS = 8, MMA_WARP = CUT_WARPS + SUM_WARPS, TMA_WARP = MMA_WARP + 1;
constexpr int THREADS = (TMA_WARP + 1) * 32, MAX_SLICES = 8, SLOTS = 4;
constexpr int W_SLOT = WM * HK * 4, W_COLS = 3 * BK / 2;   // a slot's weights; tensor-memory columns of a stage of W's pieces

__device__ int g_batch_error = 0;

template <int TN> struct Cfg {
    static constexpr int A_SLOT = TN * HK * 4, SLOT = W_SLOT + A_SLOT;
    static constexpr int PLANE = TN * BK * 2, STAGE = 3 * PLANE;            // A's pieces of a block
    static constexpr int SUMS = (TN + MAX_SLICES - 1) * WM * 4;             // [slice][row that this CTA owns][column]
    static constexpr size_t SMEM = 1024 /*alignment*/ + 2 * STAGE + SLOTS * SLOT + SUMS + 256 /*barriers*/;
    static constexpr int HALF = TN / 2;                                     // rows of A per draining warp
    static constexpr uint32_t TMEM = 2 * TN + 2 * W_COLS <= 256 ? 256 : 512;
};

// Where the key and value columns of a Q|K|V projection go (k_pages null: a plain product).
struct KvOut32 {
    float* k_pages;
    float* v_pages;
    const int* slots;
    int q_size, kv_heads, head_dim, page_size;
};

// What a column of the result needs: its bias and, for keys and values, where in a page it lies.
struct Column {
    float* pages;
    size_t off;
    float bias;
    __device__ Column(int col, const float* __restrict__ b, const KvOut32& kv) : pages(nullptr), off(0), bias(b ? __ldg(b + col) : 0.f) {
        if (kv.k_pages && col >= kv.q_size) {
            const int cc = col - kv.q_size, kvs = kv.kv_heads * kv.head_dim, c2 = cc % kvs;
            pages = cc < kvs ? kv.k_pages : kv.v_pages;
            off = (size_t)(c2 / kv.head_dim) * kv.page_size * kv.head_dim + c2 % kv.head_dim;
        }
    }
    __device__ void store(float v, float old, int m, int col, float* out, long long ldo, int act, const KvOut32& kv) const {
        v = apply_act(v + bias, act);
        if (pages) {
            const int slot = kv.slots[m];
            if (slot >= 0)
                pages[((size_t)(slot / kv.page_size) * kv.kv_heads * kv.page_size + slot % kv.page_size) * kv.head_dim + off] = v;
        } else {
            out[(size_t)m * ldo + col] = v + old;
        }
    }
};

template <int TN>
__global__ void __launch_bounds__(THREADS, 1)
linear_batch_f32_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const float* A,
                        long long lda, const float* __restrict__ W, const float* __restrict__ bias, float* out, long long ldo,
                        int M, int N, int K, int act, int accumulate, int slices, int tiles, KvOut32 kv) {
    using C = Cfg<TN>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* stages = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = stages + 2 * C::STAGE;
    float* sums = reinterpret_cast<float*>(ring + SLOTS * C::SLOT);
    uint64_t* full = (uint64_t*)((uint8_t*)sums + C::SUMS);     // [2] a stage's pieces are written
    uint64_t* empty = full + 2;                                 // [2] its MMAs have read them
    uint64_t* acc_full = empty + 2;                             // [2] a block's sums are complete
    uint64_t* acc_empty = acc_full + 2;                         // [2] they have been read out
    uint64_t* w_full = acc_empty + 2;                           // [SLOTS] the weights have arrived
    uint64_t* a_full = w_full + SLOTS;                          // [SLOTS] so have the rows of A
    uint64_t* raw_empty = a_full + SLOTS;                       // [SLOTS] both have been cut
    uint32_t* tmem_slot = (uint32_t*)(raw_empty + SLOTS);
    volatile int* failed = (volatile int*)(tmem_slot + 1);

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int rank = slices > 1 ? blockIdx.x : 0;
    const int nb = (K + BK - 1) / BK;
    const int b_lo = rank * nb / slices, nk = (rank + 1) * nb / slices - b_lo;         // this slice's blocks: at least one
    const int my_tiles = (tiles - 1 - (int)blockIdx.y) / (int)gridDim.y + 1;           // one, where K is cut
    const int steps = my_tiles * nk;
    // first barrier, arrival only: once it completes every CTA of the cluster runs and its shared memory may be written
    if (slices > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (threadIdx.x == 32) prefetch_map(&map_a);
    if (threadIdx.x == 0) {
        prefetch_map(&map_w);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full[s], CUT_WARPS);
            mbar_init(&empty[s], 1);
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], SUM_WARPS);
        }
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(&w_full[s], 1);
            mbar_init(&a_full[s], 1);
            mbar_init(&raw_empty[s], CUT_WARPS);
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) tmem_alloc(tmem_slot, C::TMEM);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot, tmem_w = tmem + 2 * TN;   // [2] stages of W's pieces behind the two accumulators

    if (warp < CUT_WARPS) {
        // W: this thread's row and half (16 values) of a half block.  A: row and run of 8 values, dealt to the lanes so that 8
        // neighbouring lanes hit all banks in the reads (with the two 16-byte pieces taken in turn) and in the writes.
        const int row_w = (warp & 3) * 32 + lane, part = warp >> 2;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const int li = lane >> 2, g = lane & 3, swap = li & 1;
        const int row_a = warp * 8 + (li >> 1) + (swap << 2);
        const bool cuts_a = warp * 8 < TN;
        bool ok = true;
        for (int it = 0; it < steps && ok; ++it) {
            const int s = it & 1;
            const uint32_t parity = (it >> 1) & 1;
            ok = it < 2 || mbar_wait(&empty[s], parity ^ 1);
            if (!ok) *failed = 1;
            tc_fence_after();
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int slot = s * 2 + half;
                if (ok && !mbar_wait(&w_full[slot], parity)) { *failed = 5; ok = false; }
                ok = __all_sync(0xffffffffu, ok && !*failed);
                if (!ok) break;
                const uint8_t* raw = ring + slot * C::SLOT;
                float4 x[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    x[j] = *reinterpret_cast<const float4*>(raw + row_w * 128 + (((part * 4 + j) ^ (row_w & 7)) << 4));
                const uint32_t tw = tmem_w + lane_off + (uint32_t)(s * W_COLS + half * 16 + part * 8);
                uint4 h[2], m[2], l[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) cut8(x[2 * j], x[2 * j + 1], h[j], m[j], l[j]);
                tmem_st8(tw, h[0], h[1]);
                tmem_st8(tw + BK / 2, m[0], m[1]);
                tmem_st8(tw + BK, l[0], l[1]);
            }
            if (!ok) break;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int slot = s * 2 + half;
                if (ok && !mbar_wait(&a_full[slot], parity)) { *failed = 6; ok = false; }
                ok = __all_sync(0xffffffffu, ok && !*failed);
                if (!ok) break;
                float4 y[2];
                const uint8_t* raw = ring + slot * C::SLOT + W_SLOT + row_a * 128;
                if (cuts_a) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        y[j] = *reinterpret_cast<const float4*>(raw + (((2 * g + (j ^ swap)) ^ (row_a & 7)) << 4));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[slot]);
                if (cuts_a) {
                    uint8_t* dst = stages + s * C::STAGE + row_a * 128 + (((half * 4 + g) ^ (row_a & 7)) << 4);
                    uint4 h, m, l;
                    cut8(swap ? y[1] : y[0], swap ? y[0] : y[1], h, m, l);
                    *reinterpret_cast<uint4*>(dst) = h;
                    *reinterpret_cast<uint4*>(dst + C::PLANE) = m;
                    *reinterpret_cast<uint4*>(dst + 2 * C::PLANE) = l;
                }
            }
            if (!ok) break;
            tmem_st_wait();
            tc_fence_before();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
        pdl_wait();
        pdl_launch();
    } else if (warp == TMA_WARP) {
        const int total = 2 * steps, pre = total < SLOTS ? total : SLOTS;
        struct Next { int tile, k, slot; } w{(int)blockIdx.y, b_lo * BK, 0};
        auto step = [&](Next& x) {
            x.slot = (x.slot + 1) & (SLOTS - 1);
            x.k += HK;
            if (x.k == (b_lo + nk) * BK) { x.k = b_lo * BK; x.tile += gridDim.y; }
        };
        auto weights = [&] {
            mbar_expect_tx_warp(&w_full[w.slot], W_SLOT);
            tma_load_2d_warp(ring + w.slot * C::SLOT, &map_w, w.k, w.tile * WM, &w_full[w.slot]);
        };
        auto rows = [&](const Next& x) {
            mbar_expect_tx_warp(&a_full[x.slot], C::A_SLOT);
            tma_load_2d_warp(ring + x.slot * C::SLOT + W_SLOT, &map_a, x.k, 0, &a_full[x.slot]);
        };
        Next a = w;
        for (int hb = 0; hb < pre; ++hb) { weights(); step(w); }          // written by no kernel of the step
        pdl_wait();
        pdl_launch();
        for (int hb = 0; hb < pre; ++hb) { rows(a); step(a); }
        uint32_t parity = 0;
        for (int hb = pre; hb < total; ++hb) {
            if (!__all_sync(0xffffffffu, mbar_wait(&raw_empty[w.slot], parity) && !*failed)) {
                if (!*failed) *failed = 7;
                break;
            }
            weights();
            rows(w);
            step(w);
            if (w.slot == 0) parity ^= 1;
        }
    } else if (warp == MMA_WARP) {
        pdl_wait();
        pdl_launch();
        constexpr uint32_t idesc = make_idesc(WM, TN);
        // (piece of W, piece of A) of the six products, smallest first
        constexpr int PW[6] = {2, 0, 1, 1, 0, 0}, PA[6] = {0, 2, 1, 0, 1, 0};
        const uint64_t desc0 = make_smem_desc(smem_u32(stages));
        for (int it = 0; it < steps; ++it) {
            const int s = it & 1;
            if (it >= 2 && !__all_sync(0xffffffffu, mbar_wait(&acc_empty[s], ((it >> 1) - 1) & 1))) { *failed = 2; break; }
            if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (it >> 1) & 1))) { *failed = 3; break; }
            tc_fence_after();
            const uint64_t da = desc0 + (uint64_t)(s * (C::STAGE >> 4));
            const uint32_t d = tmem + (uint32_t)(s * TN), tw = tmem_w + (uint32_t)(s * W_COLS);
#pragma unroll
            for (int t = 0; t < 6; ++t)
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_f16_ts_warp(d, tw + (uint32_t)(PW[t] * (BK / 2) + k * 8), da + (uint64_t)(PA[t] * (C::PLANE >> 4) + 2 * k),
                                     idesc, (t | k) != 0);
            umma_commit_warp(&empty[s]);
            umma_commit_warp(&acc_full[s]);
        }
    } else {
        pdl_wait();
        pdl_launch();
        const int q = warp & 3, m0 = ((warp - CUT_WARPS) >> 2) * C::HALF;      // rows m0 .. of A, lane = row of W
        bool ok = true;
        int it = 0;
        for (int tile = blockIdx.y; tile < tiles && ok; tile += gridDim.y) {
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
                const uint32_t t_addr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * TN + m0);
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
            const int col = tile * WM + q * 32 + lane;
            bool odd = false;
#pragma unroll
            for (int j = 0; j < C::HALF; ++j) odd |= !(fabsf(acc[j]) <= 3.402823466e38f);
            if (odd && col < N) {
                const int k0 = b_lo * BK, len = min(K - k0, nk * BK);
#pragma unroll
                for (int j = 0; j < C::HALF; ++j)
                    if (!(fabsf(acc[j]) <= 3.402823466e38f) && m0 + j < M)
                        acc[j] = plain_dot(A + (size_t)(m0 + j) * lda + k0, W + (size_t)col * K + k0, len);
            }
            if (slices > 1) {
                __syncwarp();
                asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
                cg::cluster_group cluster = cg::this_cluster();
                const int own = (M + slices - 1) / slices;         // rows per owner: row m belongs to CTA m % slices
                int owner = m0 % slices, at = m0 / slices;
#pragma unroll
                for (int j = 0; j < C::HALF; ++j) {
                    if (m0 + j < M) cluster.map_shared_rank(sums, owner)[(rank * own + at) * WM + q * 32 + lane] = acc[j];
                    if (++owner == slices) { owner = 0; ++at; }
                }
            } else if (col < N) {
                const Column c(col, bias, kv);
#pragma unroll
                for (int j0 = 0; j0 < C::HALF; j0 += 8) {
                    float old[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) old[j] = accumulate && m0 + j0 + j < M ? out[(size_t)(m0 + j0 + j) * ldo + col] : 0.f;
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (m0 + j0 + j < M) c.store(acc[j0 + j], old[j], m0 + j0 + j, col, out, ldo, act, kv);
                }
            }
        }
        if (!ok && slices > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    __syncwarp();
    tc_fence_before();
    if (slices > 1) {
        if (warp < CUT_WARPS || warp >= MMA_WARP) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        cg::this_cluster().sync();                             // every slice's sums have arrived
        const int own = (M + slices - 1) / slices, n = threadIdx.x & (WM - 1), col = blockIdx.y * WM + n;
        constexpr int GROUPS = THREADS / WM;
        if (threadIdx.x < GROUPS * WM && col < N) {
            const Column c(col, bias, kv);
#pragma unroll 4
            for (int i = threadIdx.x / WM; i < own; i += GROUPS) {
                const int m = i * slices + rank;
                if (m >= M) break;
                float part[MAX_SLICES], old = 0.f;
                if (accumulate) old = out[(size_t)m * ldo + col];
#pragma unroll
                for (int z = 0; z < MAX_SLICES; ++z)
                    if (z < slices) part[z] = sums[(z * own + i) * WM + n];
                float v = part[0];
#pragma unroll
                for (int z = 1; z < MAX_SLICES; ++z)
                    if (z < slices) v += part[z];
                c.store(v, old, m, col, out, ldo, act, kv);
            }
        }
    } else {
        __syncthreads();
    }
    if (*failed) {
        if (threadIdx.x == 0) { atomicCAS(&g_batch_error, 0, *failed); report_to_host(800 + *failed); }
        for (int i = 0; i < 2000; ++i) __nanosleep(100);       // copies and MMAs already issued may still be running
        __syncthreads();
    }
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem, C::TMEM);
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

// K slices, from N and K alone: as many CTAs as run at once (a CTA fills an SM; FIT: how many clusters of a size then run at
// once, by cudaOccupancyMaxActiveClusters on 148 SMs), of at least two blocks each.
int slices_for(int N, int K) {
    constexpr int FIT[MAX_SLICES + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
    const int tiles = (N + WM - 1) / WM, nb = (K + BK - 1) / BK;
    for (int s = MAX_SLICES; s > 1; --s)
        if (s <= nb / 2 && tiles <= FIT[s]) return s;
    return 1;
}

template <int TN>
int launch(const float* A, long long lda, const float* W, const float* bias, float* out, long long ldo, int M, int N, int K,
           int act, int accumulate, const KvOut32& kv, cudaStream_t stream) {
    using C = Cfg<TN>;
    CUtensorMap ma, mw;
    int rc = get_map(A, lda, M, K, HK, TN, MAP_F32_SW128, &ma);
    if (rc) return rc;
    rc = get_map(W, K, N, K, HK, WM, MAP_F32_SW128, &mw);
    if (rc) return rc;
    auto kern = linear_batch_f32_kernel<TN>;
    static bool set = false;
    if (!set) {
        MLLM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
        set = true;
    }
    const int slices = slices_for(N, K), tiles = (N + WM - 1) / WM;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(slices, slices > 1 || tiles < sm_count() ? tiles : sm_count());
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = slices;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_mllm_pdl ? 2 : 1;
    MLLM_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mw, A, lda, W, bias, out, ldo, M, N, K, act, accumulate, slices, tiles, kv));
    return 0;
}

}  // namespace

// The pinned host word that this file's kernel writes when it gives up on a wait.
MLLM_EXPORT int mllm_linear_batch_f32_bind_error(int* word) { return bind_host_error(word); }

// The first error recorded since the last call (0 = none); resets it.
MLLM_EXPORT int mllm_linear_batch_f32_error(int* code) {
    int zero = 0;
    MLLM_CUDA(cudaMemcpyFromSymbol(code, g_batch_error, sizeof(int)));
    if (*code) MLLM_CUDA(cudaMemcpyToSymbol(g_batch_error, &zero, sizeof(int)));
    return 0;
}

// 32-bit A [M,K] (M up to 64, row stride lda), W [N,K] and out; K and lda multiples of 4, A and W 16-byte aligned.  With
// k_pages the columns from q_size on are keys, then values, and go to the page slots `slots[m]` (negative: not stored).
MLLM_EXPORT int mllm_linear_batch_f32(const float* A, long long lda, const float* W, const float* bias, float* out,
                                      long long ldo, int M, int N, int K, int act, int accumulate, float* k_pages,
                                      float* v_pages, const int* slots, int q_size, int kv_heads, int head_dim, int page_size,
                                      cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 64 || K <= 0 || K % 4 != 0 || lda % 4 != 0)
        return mllm_fail(1, "linear_batch_f32: %d rows of %d (stride %lld): at most 64, multiples of 4", M, K, lda);
    if ((uintptr_t)A % 16 != 0 || (uintptr_t)W % 16 != 0) return mllm_fail(1, "linear_batch_f32: operands must be 16-byte aligned");
    if (k_pages && (!v_pages || !slots || q_size < 0 || kv_heads <= 0 || head_dim <= 0 || page_size <= 0 ||
                    N != q_size + 2 * kv_heads * head_dim || accumulate))
        return mllm_fail(1, "linear_batch_f32: cache write arguments do not fit N=%d", N);
    const KvOut32 kv{k_pages, v_pages, slots, q_size, kv_heads, head_dim, page_size};
    return M <= 32 ? launch<32>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, kv, stream)
                   : launch<64>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, kv, stream);
}
