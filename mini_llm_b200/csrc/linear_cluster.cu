// out = act(A[M,K] . W[N,K]^T + bias) (+ out) for up to 128 rows of bfloat16: the products of decode batches and of
// short prompts, and the vocabulary for a few rows.
//
// What bounds these is how fast a matrix of a few MB comes out of HBM, and the chain of latencies around it; the
// arithmetic is nothing.  The persistent kernel (linear_tcgen05.cu) gives a narrow matrix to few SMs (12 for 768
// columns) and walks K on each, the weight-streaming kernel (linear_smallm.cu) reads its rows of A again for every 16
// rows of W.  Here the roles are swapped: 128 rows of W are the M side of a tcgen05.mma, all rows of A (32, 64 or 128 of
// them, zeros beyond M) its N side, and K is cut into up to 8 slices, one per CTA of a thread-block cluster, so that
// more SMs stream weights (36 to 144 of 148: 36 for 768 x 768, 48 for 768 x 3072, 104 for 1600 x 6400, 108 for 2304 x 768)
// and A passes once per 128 rows of W.  The CTAs of a cluster share the rows of A among
// them: a CTA writes its sums of a row straight from tensor memory into the shared memory of the row's owner, and after
// one cluster barrier the owner adds the slices in rank order and runs the epilogue (bias, GELU, residual sum, cache
// write).
//
// Ring and sums take about 100 KB with up to 64 rows, so that the next kernel's CTA fits beside this one and its weights,
// which are asked for before the wait on the previous kernel, arrive while this kernel works.
// Slices are chosen from N and K alone: a row's result does not depend on the rows beside it.
//
// Measured in a replayed chain over 16 matrices (us; this kernel / persistent / weight-streaming, see ops._cluster_wins
// for the rule made from it): 768 x 3072 at 24 rows 4.9 / 11.1 / 7.2, at 64 rows 6.4 / 11.4, at 128 rows 9.0 / 11.8;
// 1600 x 6400 at 24 rows 8.6 / 21.9 / 14.9 (20 MB: 0.37 of the copy rate); 6400 x 1600 at 24 rows 9.1 / 14.8 / 15.9;
// 2304 x 768 at 24 rows 3.7 / 5.4 / 4.4.  What grows with the rows is the exchange of the sums (about 0.03 us a row).
//
// Every wait is bounded: after the limit the kernel records an error code, lets its copies land and returns.
#include "tcgen05.cuh"
#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace {

using namespace tc;

constexpr int WM = 128, BK = 64, THREADS = 256, MAX_SLICES = 8;

__device__ int g_cluster_error = 0;

// Where the key and value columns of a Q|K|V projection go (k_pages null: a plain product); see linear_tcgen05.cu.
struct KvOut {
    __nv_bfloat16* k_pages;
    __nv_bfloat16* v_pages;
    const int* slots;
    int q_size, kv_heads, head_dim, page_size;
};

template <int TN> struct Cfg {
    static constexpr int W_BYTES = WM * BK * 2, A_BYTES = TN * BK * 2, STAGE = W_BYTES + A_BYTES;
    static constexpr int STAGES = TN == 32 ? 4 : 3;
    static constexpr int RING = STAGES * STAGE;
    // [slice][row of A that this CTA owns][column of the tile]: at most TN + slices - 1 rows
    static constexpr int SUMS = (TN + MAX_SLICES - 1) * WM * 4;
    static constexpr size_t SMEM = RING + SUMS + 1024 /*alignment*/ + 256 /*barriers*/;
};

template <int TN, typename TO>
__global__ void __launch_bounds__(THREADS)
linear_cluster_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                      const float* __restrict__ bias, TO* out, long long ldo, int M, int N, int K, int act, int accumulate,
                      int slices, KvOut kv) {
    using C = Cfg<TN>;
    constexpr int STAGES = C::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    float* sums = reinterpret_cast<float*>(ring + C::RING);
    uint64_t* full = (uint64_t*)(ring + C::RING + C::SUMS);
    uint64_t* empty = full + STAGES;
    uint64_t* acc_full = empty + STAGES;
    uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
    volatile int* failed = (volatile int*)(tmem_slot + 1);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int rank = blockIdx.x, n0 = blockIdx.y * WM;
    const int nb = (K + BK - 1) / BK;
    // first barrier, arrival only: once it completes every CTA of the cluster runs and its shared memory may be written
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    const int b_lo = rank * nb / slices, blocks = (rank + 1) * nb / slices - b_lo;       // at least one: slices <= nb
    if (threadIdx.x == 32) { prefetch_map(&map_a); }
    if (threadIdx.x == 0) {
        prefetch_map(&map_w);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(tmem_slot, TN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        const int pre = min(blocks, STAGES);
        for (int b = 0; b < pre; ++b) {                    // weights: written by no kernel of the step
            mbar_expect_tx_warp(&full[b], C::STAGE);
            tma_load_2d_warp(ring + b * C::STAGE, &map_w, (b_lo + b) * BK, n0, &full[b]);
        }
        pdl_wait();
        pdl_launch();
        for (int b = 0; b < pre; ++b) tma_load_2d_warp(ring + b * C::STAGE + C::W_BYTES, &map_a, (b_lo + b) * BK, 0, &full[b]);
        for (int b = pre; b < blocks; ++b) {
            const int s = b % STAGES;
            if (!__all_sync(0xffffffffu, mbar_wait(&empty[s], (b / STAGES - 1) & 1))) { *failed = 1; break; }
            mbar_expect_tx_warp(&full[s], C::STAGE);
            tma_load_2d_warp(ring + s * C::STAGE, &map_w, (b_lo + b) * BK, n0, &full[s]);
            tma_load_2d_warp(ring + s * C::STAGE + C::W_BYTES, &map_a, (b_lo + b) * BK, 0, &full[s]);
        }
    } else {
        pdl_wait();
        pdl_launch();
        if (warp == 1) {
            constexpr uint32_t idesc = make_idesc(WM, TN);
            const uint64_t desc0 = make_smem_desc(smem_u32(ring));
            for (int b = 0; b < blocks; ++b) {
                const int s = b % STAGES;
                if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (b / STAGES) & 1))) { *failed = 2; break; }
                tc_fence_after();
                const uint64_t dw = desc0 + (uint64_t)(s * (C::STAGE >> 4));
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_f16_warp(tmem, dw + 2 * k, dw + (uint64_t)((C::W_BYTES >> 4) + 2 * k), idesc, (b | k) != 0);
                umma_commit_warp(&empty[s]);
            }
            umma_commit_warp(acc_full);
        }
    }
    __syncwarp();
    if (!__all_sync(0xffffffffu, mbar_wait(acc_full, 0))) *failed = 3;
    tc_fence_after();
    const int q = warp & 3, rows_half = warp >> 2;         // two warps per quarter of the lanes take the rows in turn
    const int own = (M + slices - 1) / slices;             // rows per owner: row m belongs to CTA m % slices
    cg::cluster_group cluster = cg::this_cluster();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll
    for (int c = 0; c < TN / 16; ++c) {
        if ((c & 1) != rows_half || c * 16 >= M) continue;
        uint32_t r[16];
        tmem_ld16_issue(tmem + ((uint32_t)(q * 32) << 16) + c * 16, r);
        tmem_ld_wait();
        int owner = (c * 16) % slices, at = (c * 16) / slices;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            if (c * 16 + j < M)
                cluster.map_shared_rank(sums, owner)[(rank * own + at) * WM + q * 32 + lane] = __uint_as_float(r[j]);
            if (++owner == slices) { owner = 0; ++at; }
        }
    }
    tc_fence_before();
    cluster.sync();                                        // every slice's sums have arrived
    const int n = threadIdx.x & (WM - 1), col = n0 + n;
    if (col < N) {
        const float bv = bias ? __ldg(bias + col) : 0.f;
        const bool to_cache = kv.k_pages && col >= kv.q_size;
        __nv_bfloat16* pages = nullptr;
        size_t cache_off = 0;
        if (to_cache) {
            const int cc = col - kv.q_size, kvs = kv.kv_heads * kv.head_dim, c2 = cc % kvs;
            pages = cc < kvs ? kv.k_pages : kv.v_pages;
            cache_off = (size_t)(c2 / kv.head_dim) * kv.page_size * kv.head_dim + c2 % kv.head_dim;
        }
#pragma unroll 4
        for (int i = threadIdx.x / WM; i < own; i += THREADS / WM) {
            const int m = i * slices + rank;
            if (m >= M) break;
            float part[MAX_SLICES], old = 0.f;
            if (accumulate) old = to_f32(out[(size_t)m * ldo + col]);
#pragma unroll
            for (int z = 0; z < MAX_SLICES; ++z)
                if (z < slices) part[z] = sums[(z * own + i) * WM + n];
            float v = part[0];
#pragma unroll
            for (int z = 1; z < MAX_SLICES; ++z)
                if (z < slices) v += part[z];
            v += bv;
            if (act == MLLM_ACT_GELU_TANH) v = sizeof(TO) == 2 ? gelu_tanh_fast(v) : gelu_tanh_f(v);
            else if (act == MLLM_ACT_GELU_ERF) v = gelu_erf_f(v);
            if (to_cache) {
                const int slot = kv.slots[m];
                if (slot >= 0)
                    pages[((size_t)(slot / kv.page_size) * kv.kv_heads * kv.page_size + slot % kv.page_size) * kv.head_dim + cache_off] =
                        __float2bfloat16_rn(v);
            } else {
                out[(size_t)m * ldo + col] = from_f32<TO>(v + old);
            }
        }
    }
    if (*failed) {
        if (threadIdx.x == 0) { atomicCAS(&g_cluster_error, 0, *failed); report_to_host(600 + *failed); }
        for (int i = 0; i < 2000; ++i) __nanosleep(100);   // copies already issued may still be landing
        __syncthreads();
    }
    if (warp == 1) {                                       // every warp's reads ended before the cluster barrier
        tc_fence_after();
        tmem_dealloc(tmem, TN);
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

// K slices: as many as keep the grid within one CTA per SM, of at least two blocks of 64 each.  (At most 4 instead of 8
// slices: 9.2 against 6.9 us for 768 columns inside a decode step of 64 rows; at least four blocks: 8.6.)
int slices_for(int N, int K) {
    const int tiles = (N + WM - 1) / WM, nb = (K + BK - 1) / BK;
    int s = sm_count() / tiles;
    s = s < MAX_SLICES ? s : MAX_SLICES;
    s = s < nb / 2 ? s : nb / 2;
    return s < 1 ? 1 : s;
}

template <int TN, typename TO>
int launch(const void* A, long long lda, const void* W, const float* bias, void* out, long long ldo, int M, int N, int K,
           int act, int accumulate, const KvOut& kv, cudaStream_t stream) {
    using C = Cfg<TN>;
    CUtensorMap ma, mw;
    int rc = get_map(A, lda, M, K, BK, TN, MAP_BF16_SW128, &ma);
    if (rc) return rc;
    rc = get_map(W, K, N, K, BK, WM, MAP_BF16_SW128, &mw);
    if (rc) return rc;
    auto kern = linear_cluster_kernel<TN, TO>;
    static bool set = false;
    if (!set) {
        MLLM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
        set = true;
    }
    const int slices = slices_for(N, K);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(slices, (N + WM - 1) / WM);
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
    MLLM_CUDA(cudaLaunchKernelEx(&cfg, kern, ma, mw, bias, (TO*)out, ldo, M, N, K, act, accumulate, slices, kv));
    return 0;
}

template <typename TO>
int go(const void* A, long long lda, const void* W, const float* bias, void* out, long long ldo, int M, int N, int K,
       int act, int accumulate, const KvOut& kv, cudaStream_t stream) {
    if (K <= 0 || K % 8 != 0 || lda % 8 != 0)
        return mllm_fail(1, "linear_cluster: K=%d and the row stride %lld must be multiples of 8", K, lda);
    if ((uintptr_t)A % 16 != 0 || (uintptr_t)W % 16 != 0) return mllm_fail(1, "linear_cluster: operands must be 16-byte aligned");
    if (M > 128) return mllm_fail(1, "linear_cluster: %d rows, at most 128", M);
    if ((N + WM - 1) / WM > 65535) return mllm_fail(1, "linear_cluster: N=%d exceeds the grid limit", N);
    if (M <= 32) return launch<32, TO>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, kv, stream);
    if (M <= 64) return launch<64, TO>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, kv, stream);
    return launch<128, TO>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, kv, stream);
}

}  // namespace

// The pinned host word that this file's kernel writes when it gives up on a wait.
MLLM_EXPORT int mllm_linear_cluster_bind_error(int* word) { return bind_host_error(word); }

// The first error recorded since the last call (0 = none); resets it.
MLLM_EXPORT int mllm_linear_cluster_error(int* code) {
    int zero = 0;
    MLLM_CUDA(cudaMemcpyFromSymbol(code, g_cluster_error, sizeof(int)));
    if (*code) MLLM_CUDA(cudaMemcpyToSymbol(g_cluster_error, &zero, sizeof(int)));
    return 0;
}

// bfloat16 A [M,K] (M up to 128, row stride lda) and W [N,K]; out bfloat16 or 32-bit.  K and lda multiples of 8,
// operands 16-byte aligned.
MLLM_EXPORT int mllm_linear_cluster(const void* A, long long lda, const void* W, const float* bias, void* out, long long ldo,
                                    int M, int N, int K, int act, int accumulate, int out_dtype, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (out_dtype == MLLM_BF16)
        return go<__nv_bfloat16>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, KvOut{}, stream);
    if (out_dtype == MLLM_F32) return go<float>(A, lda, W, bias, out, ldo, M, N, K, act, accumulate, KvOut{}, stream);
    return mllm_fail(1, "linear_cluster: unknown dtype code %d", out_dtype);
}

// The Q|K|V projection with the cache write fused in, bfloat16 throughout: out [M, q_size] receives the query columns,
// keys and values go to their page slots (slots[m] = page * page_size + offset, negative: not stored).
MLLM_EXPORT int mllm_linear_cluster_qkv(const void* A, long long lda, const void* W, const float* bias, void* out,
                                        long long ldo, int M, int N, int K, void* k_pages, void* v_pages,
                                        const int* slots, int q_size, int kv_heads, int head_dim, int page_size,
                                        cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (q_size <= 0 || head_dim <= 0 || kv_heads <= 0 || page_size <= 0 || N != q_size + 2 * kv_heads * head_dim)
        return mllm_fail(1, "linear_cluster: %d output columns do not split into %d query and 2 x %d x %d cache columns", N,
                         q_size, kv_heads, head_dim);
    KvOut kv{(__nv_bfloat16*)k_pages, (__nv_bfloat16*)v_pages, slots, q_size, kv_heads, head_dim, page_size};
    return go<__nv_bfloat16>(A, lda, W, bias, out, ldo, M, N, K, MLLM_ACT_NONE, 0, kv, stream);
}
