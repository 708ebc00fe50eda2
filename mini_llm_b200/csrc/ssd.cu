// Mamba-2 (state-space duality) as three kernels around the projections:
//
//   conv_silu          the causal short convolution per channel over the step's tokens, with bias and silu; the taps - 1
//                      inputs before a portion come from the request's state (zero for a new request), so a prompt can
//                      be cut anywhere.  conv_state_update then stores the last taps - 1 inputs of every request.
//   ssd_scan           per request and head: dt = softplus(raw + bias), S <- exp(-exp(A_log) dt) S + dt B x^T,
//                      y = S^T C + D x, token by token.  A CTA owns 32 columns of a head's state S [N, P]; a warp owns 4
//                      columns, its lanes 8 row groups of consecutive rows, so a thread keeps N / 8 state elements
//                      in registers and the sum over rows ends in three shuffles.  Tokens are staged 16 at a time.
//                      Every state element is a recurrence of its own, so the state after n tokens is the same bits
//                      however the n tokens were cut into steps.
//   gated_group_norm   out = rms_norm_in_groups(y * silu(z)) * w.
// Everything here is 32-bit: the state, dt, the decay, the products; inputs come in the activation dtype.
#include "common.cuh"

namespace {

constexpr int MAX_TAPS = 16;
constexpr int CHUNK = 16;

__device__ __forceinline__ float silu_f(float v) { return v / (1.0f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return fmaxf(v, 0.f) + log1pf(expf(-fabsf(v))); }
// A cp.async of 4 bytes goes through L1, whatever the compiler's flag says: a kernel that uses it lets its lines go (an acquiring
// fence) after the wait, since an earlier kernel may have left some at the addresses that the last one has written anew.
__device__ __forceinline__ void cp4(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

__device__ __forceinline__ void cp16(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// grid (channel blocks of 256, tokens).  u = proj[:, off : off + C]; state [slots][stride], the conv part at conv_off:
// [taps - 1][C], oldest first.
template <typename T, typename TO>
__global__ void __launch_bounds__(256)
conv_silu_kernel(const T* proj, long long ld, int off, const float* __restrict__ w, const float* __restrict__ bias,
                 const float* state, long long state_stride, int conv_off, const int* token_seq, const int* cu_q,
                 const int* slots, TO* out, long long ldo, int Tn, int C, int taps) {
    pdl_wait();
    pdl_launch();
    const int t = blockIdx.y, ch = blockIdx.x * 256 + threadIdx.x;
    if (ch >= C) return;
    const int s = token_seq[t];
    const int qi = t - cu_q[s];
    float acc = bias[ch];
    if (qi >= taps - 1) {                   // every input lies in this step
        for (int j = 0; j < taps; ++j)
            acc = fmaf(w[(size_t)ch * taps + j], to_f32(proj[(size_t)(t - (taps - 1) + j) * ld + off + ch]), acc);
    } else {
        const float* st = state + (size_t)slots[s] * state_stride + conv_off;
        for (int j = 0; j < taps; ++j) {
            const int src = qi - (taps - 1) + j;
            const float u = src >= 0 ? to_f32(proj[(size_t)(t - (taps - 1) + j) * ld + off + ch])
                                     : st[(size_t)(taps - 1 + src) * C + ch];
            acc = fmaf(w[(size_t)ch * taps + j], u, acc);
        }
    }
    out[(size_t)t * ldo + ch] = from_f32<TO>(silu_f(acc));
}

// Steps in which every request brings one token: grid (channel blocks, requests); a thread computes its channel's output
// from the state and the token, and shifts the token into the state (one launch instead of two).
template <typename T, typename TO>
__global__ void __launch_bounds__(256)
conv_step_kernel(const T* proj, long long ld, int off, const float* __restrict__ w, const float* __restrict__ bias,
                 float* state, long long state_stride, int conv_off, const int* cu_q, const int* slots, TO* out,
                 long long ldo, int C, int taps, int write_state) {
    pdl_wait();
    pdl_launch();
    const int ch = blockIdx.x * 256 + threadIdx.x, s = blockIdx.y;
    if (ch >= C) return;
    const int t = cu_q[s];
    float* st = state + (size_t)slots[s] * state_stride + conv_off;
    const float u = to_f32(proj[(size_t)t * ld + off + ch]);
    float acc = bias[ch];
    float keep[MAX_TAPS];
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
        if (k < taps - 1) {
            keep[k] = st[(size_t)k * C + ch];
            acc = fmaf(w[(size_t)ch * taps + k], keep[k], acc);
        }
    }
    acc = fmaf(w[(size_t)ch * taps + taps - 1], u, acc);
    out[(size_t)t * ldo + ch] = from_f32<TO>(silu_f(acc));
    if (write_state) {
#pragma unroll
        for (int k = 0; k < MAX_TAPS; ++k) {
            if (k + 1 < taps - 1) st[(size_t)k * C + ch] = keep[k + 1];
            else if (k + 1 == taps - 1) st[(size_t)k * C + ch] = u;
        }
    }
}

// grid (channel blocks, requests): the state's conv part becomes the last taps - 1 inputs of the request.
template <typename T>
__global__ void __launch_bounds__(256)
conv_state_update_kernel(const T* proj, long long ld, int off, float* state, long long state_stride, int conv_off,
                         const int* cu_q, const int* slots, int C, int taps) {
    pdl_wait();
    pdl_launch();
    const int ch = blockIdx.x * blockDim.x + threadIdx.x, s = blockIdx.y;
    if (ch >= C) return;
    const int t0 = cu_q[s], n = cu_q[s + 1] - t0;
    float* st = state + (size_t)slots[s] * state_stride + conv_off;
    float keep[MAX_TAPS];
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k) {
        if (k < taps - 1) {
            const int idx = n - (taps - 1) + k;
            keep[k] = idx >= 0 ? to_f32(proj[(size_t)(t0 + idx) * ld + off + ch]) : st[(size_t)(k + n) * C + ch];
        }
    }
#pragma unroll
    for (int k = 0; k < MAX_TAPS; ++k)
        if (k < taps - 1) st[(size_t)k * C + ch] = keep[k];
}

// grid (column blocks of 32, heads, requests), 256 threads.  xbc [T][C] 32-bit (x at 0, B at b_off, C at c_off);
// dt_raw = proj[:, dt_off + head] in the activation dtype; state [slots][stride] with S of head h at h * N * P, [N][P].
// Thread (column, rg) owns the ROWS consecutive state rows rg * ROWS ..: it reads its part of B_t and C_t with 16-byte
// loads (a token's B and C are staged with 4 floats of padding after every ROWS rows, so the eight row groups fall on
// different banks; rows beyond N are staged as zeros and stay zero in the state).
template <typename T, int ROWS, bool VEC>
__global__ void __launch_bounds__(256)
ssd_scan_kernel(const float* xbc, int Cw, int b_off, int c_off, const T* proj, long long ld, int dt_off,
                const float* __restrict__ dt_bias, const float* __restrict__ A_log, const float* __restrict__ Dh,
                float* state, long long state_stride, const int* cu_q, const int* slots, float* y, int Hm, int N, int P,
                int G, int write_state) {
    constexpr int PAD = ROWS == 4 ? 0 : 4;
    constexpr int NP = 8 * (ROWS + PAD);    // floats of a token's B (or C) in shared memory
    extern __shared__ __align__(16) float sm[];
    // two buffers of: B [CHUNK][NP], C [CHUNK][NP], x [CHUNK][32], dt [CHUNK], decay [CHUNK]
    const int h = blockIdx.y, s = blockIdx.z, j0 = blockIdx.x * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = j0 + warp * 4 + (lane >> 3), rg = lane & 7;
    const int g = h / (Hm / G);
    // before the wait: the integers that the host wrote before the step, the parameters, and the state asked into L2
    const int t0 = __ldcg(cu_q + s), n = __ldcg(cu_q + s + 1) - t0;
    float* S = state + (size_t)__ldcg(slots + s) * state_stride + (size_t)h * N * P;
    for (int r = threadIdx.x; r < N; r += 256) asm volatile("prefetch.global.L2 [%0];" ::"l"(S + (size_t)r * P + j0));
    const float a = -expf(A_log[h]), dskip = Dh[h], dtb = dt_bias[h];
    pdl_wait();
    pdl_launch();
    if (!VEC) __threadfence();
    const bool live = col < P;
    float st[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const int r = rg * ROWS + i;
        st[i] = (live && r < N) ? S[(size_t)r * P + col] : 0.f;
    }
    constexpr int BUF = 2 * CHUNK * NP + CHUNK * 32 + 2 * CHUNK;     // floats of one chunk's buffer
    // a chunk's B, C and x come in by cp.async, 16 bytes at a time where the sizes allow (VEC; 24 heads of 64, us a launch so / 4 bytes
    // at a time: 3 x 250 tokens, 128 state rows 80 / 83, 256 rows 118 / 134; 1 x 1,000, 64 rows 210 / 219; steps of single tokens
    // level), while the chunk before it is walked; its step sizes are read into a register at the same time and turned into dt and
    // the decay after the walk
    float raw_dt = 0.f;
    auto stage = [&](int c0, int buf) {
        const int nc = min(CHUNK, n - c0);
        float* B2 = sm + buf * BUF;
        float* C2 = B2 + CHUNK * NP;
        float* x2 = C2 + CHUNK * NP;
        constexpr int E = VEC ? 4 : 1;                        // floats per copy
        auto copy = [](float* dst, const float* src) { if constexpr (VEC) cp16(dst, src); else cp4(dst, src); };
        auto clear = [](float* dst) { if constexpr (VEC) *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f); else *dst = 0.f; };
        for (int i = threadIdx.x; i < nc * 8 * ROWS / E; i += 256) {
            const int tt = i / (8 * ROWS / E), r = (i - tt * (8 * ROWS / E)) * E;
            const float* rowp = xbc + (size_t)(t0 + c0 + tt) * Cw;
            const int at = tt * NP + r + (r / ROWS) * PAD;
            if (r < N) {
                copy(B2 + at, rowp + b_off + g * N + r);
                copy(C2 + at, rowp + c_off + g * N + r);
            } else {
                clear(B2 + at);
                clear(C2 + at);
            }
        }
        for (int i = threadIdx.x; i < nc * (32 / E); i += 256) {
            const int tt = i / (32 / E), c = i % (32 / E) * E;
            if (j0 + c < P) copy(x2 + tt * 32 + c, xbc + (size_t)(t0 + c0 + tt) * Cw + (size_t)h * P + j0 + c);
            else clear(x2 + tt * 32 + c);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (threadIdx.x < nc) raw_dt = to_f32(proj[(size_t)(t0 + c0 + threadIdx.x) * ld + dt_off + h]);
    };
    auto steps = [&](int c0, int buf) {
        if (threadIdx.x < min(CHUNK, n - c0)) {
            float* d2 = sm + buf * BUF + 2 * CHUNK * NP + CHUNK * 32;
            const float dt = softplus_f(raw_dt + dtb);
            d2[threadIdx.x] = dt;
            d2[CHUNK + threadIdx.x] = expf(a * dt);
        }
    };
    if (n > 0) {
        stage(0, 0);
        steps(0, 0);
    }
    for (int c0 = 0, buf = 0; c0 < n; c0 += CHUNK, buf ^= 1) {
        const int nc = min(CHUNK, n - c0);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                    // this chunk is in; the other buffer has been walked
        const bool more = c0 + CHUNK < n;
        if (more) stage(c0 + CHUNK, buf ^ 1);
        const float* Bs = sm + buf * BUF;
        const float* Cs = Bs + CHUNK * NP;
        const float* xs = Cs + CHUNK * NP;
        const float* dts = xs + CHUNK * 32;
        const float* das = dts + CHUNK;
        for (int tt = 0; tt < nc; ++tt) {
            const float dt = dts[tt], da = das[tt], xv = xs[tt * 32 + warp * 4 + (lane >> 3)];
            const float dx = dt * xv;
            const float4* Bt = reinterpret_cast<const float4*>(Bs + tt * NP + rg * (ROWS + PAD));
            const float4* Ct = reinterpret_cast<const float4*>(Cs + tt * NP + rg * (ROWS + PAD));
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;        // four partial sums: the order is fixed, the chain short
#pragma unroll
            for (int i = 0; i < ROWS / 4; ++i) {
                const float4 b = Bt[i], c = Ct[i];
                st[4 * i] = fmaf(da, st[4 * i], b.x * dx);
                a0 = fmaf(st[4 * i], c.x, a0);
                st[4 * i + 1] = fmaf(da, st[4 * i + 1], b.y * dx);
                a1 = fmaf(st[4 * i + 1], c.y, a1);
                st[4 * i + 2] = fmaf(da, st[4 * i + 2], b.z * dx);
                a2 = fmaf(st[4 * i + 2], c.z, a2);
                st[4 * i + 3] = fmaf(da, st[4 * i + 3], b.w * dx);
                a3 = fmaf(st[4 * i + 3], c.w, a3);
            }
            float acc = (a0 + a1) + (a2 + a3);
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
            if (rg == 0 && live) y[(size_t)(t0 + c0 + tt) * ((size_t)Hm * P) + (size_t)h * P + col] = fmaf(dskip, xv, acc);
        }
        if (more) steps(c0 + CHUNK, buf ^ 1);
    }
    if (write_state && live) {
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const int r = rg * ROWS + i;
            if (r < N) S[(size_t)r * P + col] = st[i];
        }
    }
}

// grid (groups, tokens): out[t][g] = v / sqrt(mean(v^2) + eps) * w with v = y * silu(z) over the group's columns.
// Blocks up to which the next kernel may start early: letting it costs every block about 50 ns of its SM, which many small blocks
// feel (512 columns in 8 groups, us a launch with / without: 512 tokens 5.0 / 4.0, 2,048 tokens 18.0 / 10.7; 8 groups of 256 and 2,048
// tokens 18.1 / 11.8).
constexpr unsigned EARLY_BLOCKS = 2048;
template <typename T>
__global__ void __launch_bounds__(128)
gated_group_norm_kernel(const float* y, const T* z, long long ldz, const float* __restrict__ w, T* out, long long ldo,
                        int width, int gw, float eps) {
    __shared__ float scratch[33];
    pdl_wait();
    if (gridDim.x * gridDim.y <= EARLY_BLOCKS) pdl_launch();
    const int t = blockIdx.y, c0 = blockIdx.x * gw;
    const float* yr = y + (size_t)t * width + c0;
    const T* zr = z + (size_t)t * ldz + c0;
    float ss = 0.f;
    for (int i = threadIdx.x; i < gw; i += blockDim.x) {
        const float v = yr[i] * silu_f(to_f32(zr[i]));
        ss = fmaf(v, v, ss);
    }
    const float r = sqrtf(block_sum(ss, scratch) / (float)gw + eps);
    for (int i = threadIdx.x; i < gw; i += blockDim.x) {
        const float v = yr[i] * silu_f(to_f32(zr[i]));
        out[(size_t)t * ldo + c0 + i] = from_f32<T>(v / r * w[c0 + i]);
    }
}

__device__ __forceinline__ float4 four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 four(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16),
                       __uint_as_float(u.y & 0xffff0000u));
}

// The same for groups of up to 4,096 columns that can be read four at a time: a thread keeps its four columns, so a token costs
// one round of loads (the weights' before the wait) instead of one per trip of the loops above, twice.  3 tokens of one group
// of 1,536 in a decode step: 2.2 us, with the loops 12.2 us.
template <typename T>
__global__ void __launch_bounds__(1024)
gated_group_norm_wide_kernel(const float* y, const T* z, long long ldz, const float* __restrict__ w, T* out, long long ldo,
                             int width, int gw, float eps) {
    __shared__ float scratch[33];
    const int t = blockIdx.y, c0 = blockIdx.x * gw, i = threadIdx.x * 4;
    const bool in = i < gw;
    const float4 wv = in ? __ldg(reinterpret_cast<const float4*>(w + c0 + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
    pdl_wait();
    if (gridDim.x * gridDim.y <= EARLY_BLOCKS) pdl_launch();
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (in) {
        const float4 a = four(y + (size_t)t * width + c0 + i), b = four(z + (size_t)t * ldz + c0 + i);
        v = make_float4(a.x * silu_f(b.x), a.y * silu_f(b.y), a.z * silu_f(b.z), a.w * silu_f(b.w));
    }
    const float ss = fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x)));
    const float r = sqrtf(block_sum(ss, scratch) / (float)gw + eps);
    if (!in) return;
    T* o = out + (size_t)t * ldo + c0 + i;
    const float f[4] = {v.x / r * wv.x, v.y / r * wv.y, v.z / r * wv.z, v.w / r * wv.w};
    if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(o) = make_float4(f[0], f[1], f[2], f[3]);
    } else {
        uint2 pk;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
        h[0] = __floats2bfloat162_rn(f[0], f[1]);
        h[1] = __floats2bfloat162_rn(f[2], f[3]);
        *reinterpret_cast<uint2*>(o) = pk;
    }
}

template <typename T>
int group_norm_launch(const float* y, const T* z, long long ldz, const float* w, T* out, long long ldo, int Tn, int width,
                      int groups, float eps, cudaStream_t stream) {
    const int gw = width / groups;
    constexpr uintptr_t A = 4 * sizeof(T);
    if (gw % 4 == 0 && gw <= 4096 && width % 4 == 0 && ldz % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)y | (uintptr_t)w) % 16 == 0 &&
        ((uintptr_t)z | (uintptr_t)out) % A == 0)
        MLLM_CUDA(mllm_launch(gated_group_norm_wide_kernel<T>, dim3(groups, Tn), dim3((gw / 4 + 31) / 32 * 32), 0, stream, true, y, z,
                              ldz, w, out, ldo, width, gw, eps));
    else
        MLLM_CUDA(mllm_launch(gated_group_norm_kernel<T>, dim3(groups, Tn), dim3(128), 0, stream, true, y, z, ldz, w, out, ldo, width,
                              gw, eps));
    return 0;
}

template <typename T>
int scan_launch(int rows, dim3 grid, size_t smem, cudaStream_t stream, const float* xbc, int Cw, int b_off, int c_off,
                const void* proj, long long ld, int dt_off, const float* dt_bias, const float* A_log, const float* Dh,
                float* state, long long state_stride, const int* cu_q, const int* slots, float* y, int Hm, int N, int P, int G,
                int write_state) {
    // rows that can be read 16 bytes at a time
    const bool vec = ((N | P | Cw | b_off | c_off) & 3) == 0 && (uintptr_t)xbc % 16 == 0;
#define MLLM_SCAN(R, V)                                                                                                  \
    do {                                                                                                                 \
        static bool raised = false;                                                                                      \
        if (smem > 48 * 1024 && !raised) {                                                                               \
            MLLM_CUDA(cudaFuncSetAttribute(ssd_scan_kernel<T, R, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024)); \
            raised = true;                                                                                               \
        }                                                                                                                \
        MLLM_CUDA(mllm_launch(ssd_scan_kernel<T, R, V>, grid, dim3(256), smem, stream, true, xbc, Cw, b_off, c_off,      \
                              (const T*)proj, ld, dt_off, dt_bias, A_log, Dh, state, state_stride, cu_q, slots, y, Hm, N, P, \
                              G, write_state));                                                                          \
    } while (0)
    if (rows <= 4 && vec) MLLM_SCAN(4, true);
    else if (rows <= 4) MLLM_SCAN(4, false);
    else if (rows <= 8 && vec) MLLM_SCAN(8, true);
    else if (rows <= 8) MLLM_SCAN(8, false);
    else if (rows <= 16 && vec) MLLM_SCAN(16, true);
    else if (rows <= 16) MLLM_SCAN(16, false);
    else if (vec) MLLM_SCAN(32, true);
    else MLLM_SCAN(32, false);
#undef MLLM_SCAN
    return 0;
}

}  // namespace

MLLM_EXPORT int mllm_ssd_max_state_rows() { return 256; }
MLLM_EXPORT int mllm_ssd_max_taps() { return MAX_TAPS; }

// The convolution of the step's tokens (out [T][ldo] 32-bit, or in `dtype` when out_act is 1), then the update of the requests'
// conv states.
namespace {
template <typename T, typename TO>
int conv_launch(const void* proj, long long ld, int off, const float* w, const float* bias, float* state, long long state_stride,
                int conv_off, const int* token_seq, const int* cu_q, const int* slots, void* out, long long ldo, int Tn, int S, int C,
                int taps, int write_state, cudaStream_t stream) {
    const dim3 grid((C + 255) / 256, Tn);
    const dim3 ugrid((C + 255) / 256, S);
    if (Tn == S) {                          // one token per request: output and state update in one launch
        MLLM_CUDA(mllm_launch(conv_step_kernel<T, TO>, ugrid, dim3(256), 0, stream, true, (const T*)proj, ld, off, w, bias, state,
                              state_stride, conv_off, cu_q, slots, (TO*)out, ldo, C, taps, write_state));
        return 0;
    }
    MLLM_CUDA(mllm_launch(conv_silu_kernel<T, TO>, grid, dim3(256), 0, stream, true, (const T*)proj, ld, off, w, bias,
                          (const float*)state, state_stride, conv_off, token_seq, cu_q, slots, (TO*)out, ldo, Tn, C, taps));
    if (write_state && taps > 1)
        MLLM_CUDA(mllm_launch(conv_state_update_kernel<T>, ugrid, dim3(256), 0, stream, true, (const T*)proj, ld, off, state,
                              state_stride, conv_off, cu_q, slots, C, taps));
    return 0;
}
}  // namespace

MLLM_EXPORT int mllm_ssd_conv(const void* proj, long long ld, int off, const float* w, const float* bias, float* state,
                              long long state_stride, int conv_off, const int* token_seq, const int* cu_q, const int* slots,
                              void* out, long long ldo, int out_act, int Tn, int S, int C, int taps, int write_state, int dtype,
                              cudaStream_t stream) {
    if (Tn <= 0 || C <= 0) return 0;
    if (taps < 1 || taps > MAX_TAPS) return mllm_fail(1, "ssd_conv: %d taps (1 to %d)", taps, MAX_TAPS);
    if (Tn > 65535 || S > 65535) return mllm_fail(1, "ssd_conv: more than 65535 tokens in a step");
    using bf = __nv_bfloat16;
    if (dtype == MLLM_F32)
        return conv_launch<float, float>(proj, ld, off, w, bias, state, state_stride, conv_off, token_seq, cu_q, slots, out, ldo, Tn, S, C,
                                         taps, write_state, stream);
    if (dtype == MLLM_BF16 && out_act)
        return conv_launch<bf, bf>(proj, ld, off, w, bias, state, state_stride, conv_off, token_seq, cu_q, slots, out, ldo, Tn, S, C, taps,
                                   write_state, stream);
    if (dtype == MLLM_BF16)
        return conv_launch<bf, float>(proj, ld, off, w, bias, state, state_stride, conv_off, token_seq, cu_q, slots, out, ldo, Tn, S, C,
                                      taps, write_state, stream);
    return mllm_fail(1, "ssd_conv: unknown dtype code %d", dtype);
}

MLLM_EXPORT int mllm_ssd_scan(const float* xbc, int Cw, int b_off, int c_off, const void* proj, long long ld, int dt_off,
                              const float* dt_bias, const float* A_log, const float* Dh, float* state, long long state_stride,
                              const int* cu_q, const int* slots, float* y, int S, int Hm, int N, int P, int G, int write_state,
                              int dtype, cudaStream_t stream) {
    if (S <= 0) return 0;
    if (N < 1 || N > 256) return mllm_fail(1, "ssd_scan: a state of %d rows (1 to 256)", N);
    if (G < 1 || Hm % G) return mllm_fail(1, "ssd_scan: %d heads in %d groups", Hm, G);
    if (S > 65535 || Hm > 65535) return mllm_fail(1, "ssd_scan: grid too large");
    const dim3 grid((P + 31) / 32, Hm, S);
    const int rows = (N + 7) / 8;
    const int rpt = rows <= 4 ? 4 : rows <= 8 ? 8 : rows <= 16 ? 16 : 32;            // the instantiation's rows per thread
    const size_t smem = 2 * ((size_t)2 * CHUNK * 8 * (rpt + (rpt == 4 ? 0 : 4)) + CHUNK * 32 + 2 * CHUNK) * sizeof(float);
    if (dtype == MLLM_F32)
        return scan_launch<float>(rows, grid, smem, stream, xbc, Cw, b_off, c_off, proj, ld, dt_off, dt_bias, A_log, Dh, state,
                                  state_stride, cu_q, slots, y, Hm, N, P, G, write_state);
    if (dtype == MLLM_BF16)
        return scan_launch<__nv_bfloat16>(rows, grid, smem, stream, xbc, Cw, b_off, c_off, proj, ld, dt_off, dt_bias, A_log, Dh,
                                          state, state_stride, cu_q, slots, y, Hm, N, P, G, write_state);
    return mllm_fail(1, "ssd_scan: unknown dtype code %d", dtype);
}

MLLM_EXPORT int mllm_gated_group_norm(const float* y, const void* z, long long ldz, const float* w, void* out, long long ldo,
                                      int Tn, int width, int groups, float eps, int dtype, cudaStream_t stream) {
    if (Tn <= 0) return 0;
    if (groups < 1 || width % groups) return mllm_fail(1, "gated_group_norm: %d columns in %d groups", width, groups);
    if (Tn > 65535) return mllm_fail(1, "gated_group_norm: more than 65535 tokens in a step");
    if (dtype == MLLM_F32)
        return group_norm_launch(y, (const float*)z, ldz, w, (float*)out, ldo, Tn, width, groups, eps, stream);
    if (dtype == MLLM_BF16)
        return group_norm_launch(y, (const __nv_bfloat16*)z, ldz, w, (__nv_bfloat16*)out, ldo, Tn, width, groups, eps, stream);
    return mllm_fail(1, "gated_group_norm: unknown dtype code %d", dtype);
}
