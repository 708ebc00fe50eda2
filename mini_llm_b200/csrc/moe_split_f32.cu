// The products of a routed feed-forward over many (token, choice) pairs in 32-bit, on the tensor cores: prompt portions of
// models with routed experts on the 32-bit path (moe.cu has the routing, the order of the pairs and the kernels for few pairs).
//
// The arithmetic and the roles of the warps are those of linear_split_f32.cu: operands cut exactly into three bfloat16 pieces,
// six products of pieces, 64 of K in the accumulator, sums over blocks in 32-bit registers, non-finite elements again as a
// chain of fmaf.  What differs: a tile is 128 consecutive pairs of one expert, which its CTA finds from the offsets on the
// device; A's rows lie in the order of the pairs (the first product's input is gathered so by a kernel before it); with a gate
// the 128 rows of W are 32 gate rows, the 32 up rows beside them, and 32 of each once more, so that a draining warp holds gate
// and up of the same columns; results go to the rows of the pairs.
// On CUDA cores a tile of 32 pairs and 64 columns read every operand element from shared memory for each multiply-add or two.
// Both products of a layer, us here / there, top 2:   34 pairs       256         1,500       4,000
//    8 experts of   512 x  768 (gated)              53 / 132     55 / 153     61 / 256   108 /   521
//    8 experts of 1,024 x  768                      66 / 204     68 / 296    102 / 564   188 / 1,124
//   64 experts of   256 x 1,024                     77 / 277    129 / 330    133 / 367   142 /   686
// Few pairs are bound by one tile's chain (12 blocks of 64, 1.5 us each, and what stands around them), many by the cutting.
//
// Every wait is bounded: after the limit the kernel records an error code, frees its tensor memory and returns.
#include "split_f32.cuh"

namespace {

using namespace tc;

constexpr int BM = 128, BN = 128, BK = 64, HK = 32, MAX_E = 512;
constexpr int CUT_WARPS = 8, EPI_WARPS = 8, MMA_WARP = CUT_WARPS + EPI_WARPS, TMA_WARP = MMA_WARP + 1;
constexpr int THREADS = (TMA_WARP + 1) * 32, SLOTS = 3;
constexpr int W_PLANE = BN * BK * 2, W_STAGE = 3 * W_PLANE, A_SLOT = BM * HK * 4, SLOT = A_SLOT + BN * HK * 4;
constexpr int HALF = BN / 2, A_COLS = 3 * BK / 2, WBOX = 32;
constexpr size_t SMEM = 1024 /*alignment*/ + 2 * W_STAGE + SLOTS * SLOT + (MAX_E + 1) * 4 + 12 + 256 /*barriers*/;

__device__ int g_moe_error = 0;

// xs[i] = A[sorted[i] / a_div]: a block per pair, 16 bytes per thread and trip.
__global__ void __launch_bounds__(128)
moe_gather_kernel(const float* A, long long lda, const int* sorted, float* xs, int K4, int a_div) {
    pdl_wait();
    pdl_launch();
    const float4* src = reinterpret_cast<const float4*>(A + (size_t)(sorted[blockIdx.x] / a_div) * lda);
    float4* dst = reinterpret_cast<float4*>(xs) + (size_t)blockIdx.x * K4;
#pragma unroll 4
    for (int k = threadIdx.x; k < K4; k += 128) dst[k] = src[k];
}

__global__ void __launch_bounds__(THREADS, 1)
moe_split_f32_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const float* A,
                     const float* __restrict__ W, float* out, long long ldo, const int* offsets, const int* sorted, int E, int N,
                     int K, int out_by_pair, int gated, float limit, float alpha, int uact, int tiles_n) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* w_stages = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = w_stages + 2 * (size_t)W_STAGE;
    uint64_t* full = (uint64_t*)(ring + (size_t)SLOTS * SLOT);     // [2] a stage's pieces are written
    uint64_t* empty = full + 2;                            // [2] its MMAs have read them
    uint64_t* acc_full = empty + 2;                        // [2] a block's sums are complete
    uint64_t* acc_empty = acc_full + 2;                    // [2] they have been read out
    uint64_t* raw_full = acc_empty + 2;                    // [SLOTS] the 32-bit boxes have arrived
    uint64_t* raw_empty = raw_full + SLOTS;                // [SLOTS] they have been cut
    uint32_t* tmem_slot = (uint32_t*)(raw_empty + SLOTS);
    volatile int* failed = (volatile int*)(tmem_slot + 1);
    int* s_tiles = (int*)(tmem_slot + 2);
    int* s_off = s_tiles + 1;                              // [E + 1]

    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int nk = (K + BK - 1) / BK;
    if (threadIdx.x == 32) { prefetch_map(&map_a); prefetch_map(&map_w); }
    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full[s], CUT_WARPS);
            mbar_init(&empty[s], 1);
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], EPI_WARPS);
        }
        for (int s = 0; s < SLOTS; ++s) {
            mbar_init(&raw_full[s], 1);
            mbar_init(&raw_empty[s], CUT_WARPS);
        }
        *failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) tmem_alloc(tmem_slot, 512);
    pdl_wait();                                            // offsets and rows are written by kernels of this step
    pdl_launch();
    for (int e = threadIdx.x; e <= E; e += THREADS) s_off[e] = offsets[e];
    __syncthreads();
    if (threadIdx.x == 0) {
        int n = 0;
        for (int e = 0; e < E; ++e) n += (s_off[e + 1] - s_off[e] + BM - 1) / BM;
        *s_tiles = n;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tmem_a = tmem_base + 2 * BN;            // [2] stages of A's pieces behind the two accumulators
    const int num_items = *s_tiles * tiles_n;
    const int my_items = num_items > (int)blockIdx.x ? (num_items - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int steps = my_items * nk;
    // the expert, first pair and number of pairs of a row tile
    auto tile_of = [&](int tile, int& e, int& r0, int& cnt) {
        for (e = 0; e < E - 1; ++e) {
            const int t = (s_off[e + 1] - s_off[e] + BM - 1) / BM;
            if (tile < t) break;
            tile -= t;
        }
        r0 = s_off[e] + tile * BM;
        cnt = min(BM, s_off[e + 1] - r0);
    };
    const int cols = gated ? BN / 2 : BN;                  // columns of the result per tile

    if (warp < CUT_WARPS) {
        // A: this thread's row and half (16 values) of a half block.  W: row and run of 8 values; see linear_split_f32.cu
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
            uint8_t* st = w_stages + (size_t)s * W_STAGE;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                if (ok && !mbar_wait(&raw_full[slot], parity)) { *failed = 5; ok = false; }
                ok = __all_sync(0xffffffffu, ok && !*failed);
                if (!ok) break;
                const uint8_t* raw = ring + (size_t)slot * SLOT;
                float4 x[4], y[BN / 64][2];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    x[j] = *reinterpret_cast<const float4*>(raw + row_a * 128 + (((part * 4 + j) ^ (row_a & 7)) << 4));
#pragma unroll
                for (int i = 0; i < BN / 64; ++i) {
                    const int row = row_w + i * 64;
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        y[i][j] = *reinterpret_cast<const float4*>(raw + A_SLOT + row * 128 + (((2 * g + (j ^ swap)) ^ (row & 7)) << 4));
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[slot]);
                if (++slot == SLOTS) { slot = 0; parity ^= 1; }
                const uint32_t ta = tmem_a + lane_off + (uint32_t)(s * A_COLS + half * 16 + part * 8);
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
                    *reinterpret_cast<uint4*>(dst + W_PLANE) = m[0];
                    *reinterpret_cast<uint4*>(dst + 2 * W_PLANE) = l[0];
                }
            }
            if (!ok) break;
            tmem_st_wait();
            tc_fence_before();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
        }
    } else if (warp == TMA_WARP) {
        int slot = 0, hb = 0;
        uint32_t parity = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
            int e, r0, cnt;
            tile_of(item / tiles_n, e, r0, cnt);
            const int n0 = item % tiles_n * cols, w0 = e * (gated ? 2 * N : N) + n0;
            for (int k = 0; k < nk * BK; k += HK, ++hb) {
                if (hb >= SLOTS && !__all_sync(0xffffffffu, mbar_wait(&raw_empty[slot], parity) && !*failed)) {
                    if (!*failed) *failed = 6;
                    ok = false;
                    break;
                }
                mbar_expect_tx_warp(&raw_full[slot], SLOT);
                uint8_t* dst = ring + (size_t)slot * SLOT;
                tma_load_2d_warp(dst, &map_a, k, r0, &raw_full[slot]);
#pragma unroll
                for (int j = 0; j < BN / WBOX; ++j)        // gated: gate rows, up rows, gate rows, up rows
                    tma_load_2d_warp(dst + A_SLOT + j * WBOX * HK * 4, &map_w, k,
                                     gated ? w0 + (j & 1) * N + (j >> 1) * WBOX : w0 + j * WBOX, &raw_full[slot]);
                if (++slot == SLOTS) {
                    slot = 0;
                    if (hb >= SLOTS) parity ^= 1;
                }
            }
        }
    } else if (warp == MMA_WARP) {
        constexpr uint32_t idesc = make_idesc(BM, BN);
        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};      // smallest products first
        const uint64_t desc0 = make_smem_desc(smem_u32(w_stages));
        for (int it = 0; it < steps; ++it) {
            const int s = it & 1;
            if (it >= 2 && !__all_sync(0xffffffffu, mbar_wait(&acc_empty[s], ((it >> 1) - 1) & 1))) { *failed = 2; break; }
            if (!__all_sync(0xffffffffu, mbar_wait(&full[s], (it >> 1) & 1))) { *failed = 3; break; }
            tc_fence_after();
            const uint64_t dw = desc0 + (uint64_t)(s * (W_STAGE >> 4));
            const uint32_t d = tmem_base + (uint32_t)(s * BN), ta = tmem_a + (uint32_t)(s * A_COLS);
#pragma unroll
            for (int t = 0; t < 6; ++t)
#pragma unroll
                for (int k = 0; k < BK / 16; ++k)
                    umma_f16_ts_warp(d, ta + (uint32_t)(PA[t] * (BK / 2) + k * 8), dw + (uint64_t)(PW[t] * (W_PLANE >> 4) + 2 * k),
                                     idesc, (t | k) != 0);
            umma_commit_warp(&empty[s]);
            umma_commit_warp(&acc_full[s]);
        }
    } else {
        const int q = warp & 3, half = (warp - CUT_WARPS) >> 2;
        int it = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < num_items && ok; item += gridDim.x) {
            float acc[HALF];
#pragma unroll
            for (int j = 0; j < HALF; ++j) acc[j] = 0.f;
            for (int kb = 0; kb < nk; ++kb, ++it) {
                const int s = it & 1;
                ok = mbar_wait(&acc_full[s], (it >> 1) & 1);
                if (!ok) *failed = 4;
                ok = __all_sync(0xffffffffu, ok && !*failed);
                if (!ok) break;
                tc_fence_after();
                const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(s * BN + half * HALF);
#pragma unroll
                for (int c = 0; c < HALF / 16; ++c) {
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
            int e, r0, cnt;
            tile_of(item / tiles_n, e, r0, cnt);
            if (q * 32 + lane < cnt) {
                const int i = r0 + q * 32 + lane, n0 = item % tiles_n * cols + half * (cols / 2);
                float* o = out + (size_t)(out_by_pair ? sorted[i] : i) * ldo + n0;
                bool odd = false;
#pragma unroll
                for (int j = 0; j < HALF; ++j) odd |= !(fabsf(acc[j]) <= 3.402823466e38f);
                if (odd) {
                    const float* a = A + (size_t)i * K;
#pragma unroll
                    for (int j = 0; j < HALF; ++j) {
                        const int n = n0 + (gated ? j & 31 : j);
                        if (n < N && !(fabsf(acc[j]) <= 3.402823466e38f))
                            acc[j] = plain_dot(a, W + ((size_t)e * (gated ? 2 * N : N) + (gated && j >= 32 ? N : 0) + n) * K, K);
                    }
                }
                const int width = min(N - n0, cols / 2);       // columns of this warp that exist
                const bool vec = width == cols / 2 && (uintptr_t)o % 16 == 0;
                if (gated) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) acc[j] = gate_mul(acc[j], acc[32 + j], gated, limit, alpha);
                } else if (uact) {
#pragma unroll
                    for (int j = 0; j < HALF; ++j) acc[j] = unary_act(acc[j], uact);
                }
#pragma unroll
                for (int j = 0; j < HALF; j += 4) {
                    if (gated && j >= 32) break;
                    if (vec) {
                        *reinterpret_cast<float4*>(o + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
                    } else {
#pragma unroll
                        for (int b = 0; b < 4; ++b)
                            if (j + b < width) o[j + b] = acc[j + b];
                    }
                }
            }
            __syncwarp();
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*failed) {
        if (threadIdx.x == 0) { atomicCAS(&g_moe_error, 0, *failed); report_to_host(900 + *failed); }
        for (int i = 0; i < 2000; ++i) __nanosleep(100);       // copies and MMAs already issued may still be running
        __syncthreads();
    }
    if (warp == MMA_WARP) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace

// The pinned host word that this file's kernel writes when it gives up on a wait.
MLLM_EXPORT int mllm_moe_split_f32_bind_error(int* word) { return bind_host_error(word); }

// The first error recorded since the last call (0 = none); resets it.
MLLM_EXPORT int mllm_moe_split_f32_error(int* code) {
    int zero = 0;
    MLLM_CUDA(cudaMemcpyFromSymbol(code, g_moe_error, sizeof(int)));
    if (*code) MLLM_CUDA(cudaMemcpyToSymbol(g_moe_error, &zero, sizeof(int)));
    return 0;
}

// mllm_moe_grouped (moe.cu) for 32-bit operands and no identity experts: kinds 0 (gated), 1 and 2 as there.  K a multiple of
// 4, A and W 16-byte aligned, lda a multiple of 4.  a_div > 0: row i of the product is A[sorted[i] / a_div], which a first kernel
// gathers into xs [n_pairs, K] (16-byte aligned); else A's rows stand in the order of the pairs, lda = K.
MLLM_EXPORT int mllm_moe_split_f32(const float* A, long long lda, const float* W, float* out, long long ldo, const int* offsets,
                                   const int* sorted, int n_pairs, int E, int N, int K, int a_div, int out_by_pair, int kind, int act,
                                   float limit, float alpha, float* xs, cudaStream_t stream) {
    if (n_pairs <= 0 || N <= 0) return 0;
    if (E < 1 || E > MAX_E) return mllm_fail(1, "moe_split_f32: %d experts (at most %d)", E, MAX_E);
    if (K <= 0 || K % 4 || lda % 4 || ((uintptr_t)A | (uintptr_t)W | (uintptr_t)xs) % 16)
        return mllm_fail(1, "moe_split_f32: rows of %d (stride %lld) must be multiples of 4, operands 16-byte aligned", K, lda);
    if (a_div > 0 ? !xs : lda != K) return mllm_fail(1, "moe_split_f32: no place for the gathered rows, or rows in order with a stride of %lld", lda);
    if (kind < 0 || kind > 2) return mllm_fail(1, "moe_split_f32: kind %d", kind);
    if (kind == 0 && act != MLLM_ACT_SILU && act != MLLM_ACT_SWIGLU_CLAMP) return mllm_fail(1, "moe_split_f32: activation code %d", act);
    if (kind == 2 && act != MLLM_ACT_RELU_SQ && act != MLLM_ACT_RELU && act != MLLM_ACT_GELU_TANH)
        return mllm_fail(1, "moe_split_f32: activation code %d of an expert without a gate", act);
    if ((long long)E * N * 2 > 0x7fffffffLL) return mllm_fail(1, "moe_split_f32: %d experts of %d columns", E, N);
    static int sms = 0;
    if (!sms) {
        int dev = 0, n = 0;
        MLLM_CUDA(cudaGetDevice(&dev));
        MLLM_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
        MLLM_CUDA(cudaFuncSetAttribute(moe_split_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
        sms = n;                    // last: another thread that finds it set launches at once
    }
    if (a_div > 0) {
        MLLM_CUDA(mllm_launch(moe_gather_kernel, dim3(n_pairs), dim3(128), 0, stream, true, A, lda, sorted, xs, K / 4, a_div));
        A = xs;
    }
    CUtensorMap ma, mw;
    int rc = get_map(A, K, n_pairs, K, HK, BM, MAP_F32_SW128, &ma);
    if (rc) return rc;
    rc = get_map(W, K, E * (kind == 0 ? 2 * N : N), K, HK, WBOX, MAP_F32_SW128, &mw);
    if (rc) return rc;
    const int cols = kind == 0 ? BN / 2 : BN, tiles_n = (N + cols - 1) / cols;
    const long long most = ((long long)n_pairs / BM + E) * tiles_n;        // every expert may have a tile that is not full
    MLLM_CUDA(mllm_launch(moe_split_f32_kernel, dim3((unsigned)(most < sms ? most : sms)), dim3(THREADS), SMEM, stream, true, ma, mw, A, W,
                          out, ldo, offsets, sorted, E, N, K, out_by_pair, kind == 0 ? act : 0, limit, alpha, kind == 2 ? act : 0,
                          tiles_n));
    return 0;
}
