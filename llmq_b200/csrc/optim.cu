// Optimiser-side kernels: AdamW with stochastic rounding (bf16 / fp32 / block-scaled e4m3 moments),
// global gradient norm with a deterministic reduction, and the stochastic-rounding vector add / reduce
// used for sharded gradient accumulation.
// Behavioural counterparts of src/kernels/{adamw,global_norm,vector_add}.cu of the reference.
#include <cstring>
#include "api.h"
#include "common.cuh"

namespace {

int grid_for(long long work_items, int threads, int num_sms) {
    long long blocks = ceil_div_ll(work_items, threads);
    long long cap = static_cast<long long>(num_sms) * 8;
    return static_cast<int>(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

template <typename T> __device__ __forceinline__ void load8(float (&f)[8], const T* p);
template <> __device__ __forceinline__ void load8<bf16>(float (&f)[8], const bf16* p) {
    Vec16<bf16> v = Vec16<bf16>::load(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = __bfloat162float(v.v[i]);
}
template <> __device__ __forceinline__ void load8<float>(float (&f)[8], const float* p) {
    float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
template <> __device__ __forceinline__ void load8<e4m3>(float (&f)[8], const e4m3* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) {                       // two values per conversion
        const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>((i < 2 ? raw.x : raw.y) >> (16 * (i & 1))), __NV_E4M3);
        const float2 v = __half22float2(__half2(h));
        f[2 * i] = v.x; f[2 * i + 1] = v.y;
    }
}
template <typename T> __device__ __forceinline__ void store8_sr(T* p, const float (&f)[8], uint64_t ctr, uint32_t seed);
template <> __device__ __forceinline__ void store8_sr<bf16>(bf16* p, const float (&f)[8], uint64_t ctr, uint32_t seed) {
    Vec16<bf16> v;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
        uint32_t r = rng_u32(ctr + i / 2, seed);         // 16 random bits per element
        v.v[i] = sr_bf16(f[i], r);
        v.v[i + 1] = sr_bf16(f[i + 1], r >> 16);
    }
    v.store(p);
}
template <> __device__ __forceinline__ void store8_sr<float>(float* p, const float (&f)[8], uint64_t, uint32_t) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
}

// Random words for one thread-iteration (8 elements x {param, m, v}): one full hash of the element counter,
// then cheap multiply / xor-shift steps.  Depends only on (element index, seed), never on launch geometry.
struct SrWords {
    static constexpr uint32_t kMul = 0x85ebca6bu;
    uint32_t h;                          // (hash + j * 0x9e3779b9) * kMul = hash * kMul + a constant: one multiplication for all words
    __device__ __forceinline__ SrWords(uint64_t ctr, uint32_t seed) : h(rng_u32(ctr, seed) * kMul) {}
    __device__ __forceinline__ uint32_t get(uint32_t j) const {
        uint32_t x = h + j * (0x9e3779b9u * kMul);
        x ^= x >> 15;
        x *= 0xc2b2ae35u;
        return x ^ (x >> 16);
    }
};
__device__ __forceinline__ float sqrt_approx(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float div_approx(float a, float b) {
    float r;
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
// The scale of a block whose largest value is `am` (at least 1e-30), am / 448, and its reciprocal: approximations and one correction each with the remainder in an
// fma (Markstein's method), which gives the rounded quotients without the range checks of a general division.  An infinity is its own scale, of reciprocal 0.
__device__ __forceinline__ float e4m3_scale(float am, float& inv) {
    constexpr float kR = 1.f / 448.f;
    const float q = am * kR, sc = fmaf(fmaf(-448.f, q, am), kR, q);
    const float y = div_approx(1.f, sc);
    inv = fmaf(y, fmaf(-sc, y, 1.f), y);
    if (isinf(am)) { inv = 0.f; return am; }                // the remainders are NaN
    return sc;
}
template <typename T> __device__ __forceinline__ void store8_srw(T* p, const float (&f)[8], const SrWords& w, uint32_t j0);
template <> __device__ __forceinline__ void store8_srw<bf16>(bf16* p, const float (&f)[8], const SrWords& w, uint32_t j0) {
    uint32_t v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = sr_bf16x2(f[2 * i], f[2 * i + 1], w.get(j0 + i));
    *reinterpret_cast<uint4*>(p) = make_uint4(v[0], v[1], v[2], v[3]);
}
template <> __device__ __forceinline__ void store8_srw<float>(float* p, const float (&f)[8], const SrWords&, uint32_t) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(p + 4) = make_float4(f[4], f[5], f[6], f[7]);
}

// One thread updates 8 consecutive parameters.  Bound by memory and by instruction issue at once: the 12 random words, 24 roundings
// and conversions of a thread took longer than its loads and stores.  Roundings in pairs (sr_bf16x2) bring 67.9 M parameters with
// bf16 state (950 MB) from 193 to 166-182 us.  For e4m3 first moments 16 consecutive threads share one
// fp32 scale (128 elements); the scale is recomputed from the new values every step.  They are converted and rounded in pairs too (sr_e4m3x2), and the
// division by the scale checks no range: 67.9 M parameters with e4m3 and bf16 state 193.2 / 179.9 us, same bits.
template <typename P, typename G, typename M, typename Vv>
__device__ __forceinline__ void adamw_vec(long long i, bool active, P* __restrict__ param, const G* __restrict__ grad, M* __restrict__ m_state,
                                          Vv* __restrict__ v_state, float* __restrict__ m_scales, float lr, float beta1, float beta2, float bc1,
                                          float bc2, float eps, float wd, float gs, uint32_t seed, long long elem_offset, float& tmax) {
    const long long e = i * 8;
    float p[8], g[8], m[8], v[8];
    if (active) {
        load8<P>(p, param + e);
        load8<G>(g, grad + e);
        load8<Vv>(v, v_state + e);
        load8<M>(m, m_state + e);
        if constexpr (sizeof(M) == 1) {
            float sc = m_scales[e / 128];
#pragma unroll
            for (int k = 0; k < 8; ++k) m[k] *= sc;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) { p[k] = g[k] = m[k] = v[k] = 0.f; }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        float gk = g[k] * gs;
        m[k] = beta1 * m[k] + (1.f - beta1) * gk;
        v[k] = beta2 * v[k] + (1.f - beta2) * gk * gk;
        float mh = m[k] * bc1, vh = v[k] * bc2;
        // not div.approx.ftz (1 to 2 % faster): it takes a subnormal moment for 0, and this quotient is 1 / eps times as large
        p[k] -= lr * (__fdividef(mh, sqrt_approx(vh) + eps) + wd * p[k]);
    }
    const uint64_t ctr = static_cast<uint64_t>(e + elem_offset);
    const SrWords words(ctr, seed);
    if constexpr (sizeof(M) == 1) {
        float am = 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) am = fmaxf(am, fabsf(m[k]));
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
        float inv;
        const float sc = e4m3_scale(fmaxf(am, 1e-30f), inv);
        if (active) {
            uint32_t q[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = sr_e4m3x2(m[2 * k] * inv, m[2 * k + 1] * inv, words.get(4 + 2 * k), words.get(5 + 2 * k));
            *reinterpret_cast<uint2*>(m_state + e) = make_uint2(q[0] | q[1] << 16, q[2] | q[3] << 16);
            if ((i & 15) == 0) m_scales[e / 128] = sc;
        }
    } else {
        if (active) store8_srw<M>(m_state + e, m, words, 4);
    }
    if (active) {
        store8_srw<Vv>(v_state + e, v, words, 12);
        if constexpr (sizeof(P) == 2) {
            uint32_t o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                o[k] = sr_bf16x2(p[2 * k], p[2 * k + 1], words.get(k));
                tmax = fmaxf(tmax, fmaxf(fabsf(__uint_as_float(o[k] << 16)), fabsf(__uint_as_float(o[k] & 0xFFFF0000u))));
            }
            *reinterpret_cast<uint4*>(reinterpret_cast<bf16*>(param) + e) = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
            store8_srw<float>(reinterpret_cast<float*>(param) + e, p, words, 0);
#pragma unroll
            for (int k = 0; k < 8; ++k) tmax = fmaxf(tmax, fabsf(p[k]));
        }
    }
}

template <typename P, typename G, typename M, typename Vv>
__global__ void __launch_bounds__(256)
adamw_kernel(P* __restrict__ param, const G* __restrict__ grad, M* __restrict__ m_state, Vv* __restrict__ v_state,
             float* __restrict__ m_scales, long long n, float lr, float beta1, float beta2, float bc1, float bc2, float eps,
             float wd, const float* __restrict__ grad_scale, float* __restrict__ absmax_out, uint32_t seed, long long elem_offset,
             const float* __restrict__ hyper) {
    grid_wait(grad_scale, hyper);
    const int bx = after_wait(blockIdx.x), tx = after_wait(threadIdx.x);
    __shared__ float scratch[32];
    if (hyper) {
        // Step-dependent scalars from device memory: {lr, beta1, beta2, 1/(1-beta1^t), 1/(1-beta2^t), eps, weight decay,
        // seed bits}.  The launch itself is then the same every step and can be replayed from a CUDA graph; `wd` of the
        // launch selects (non-zero) or masks (zero) the weight decay, `seed` is added to the step's seed.
        lr = hyper[0]; beta1 = hyper[1]; beta2 = hyper[2]; bc1 = hyper[3]; bc2 = hyper[4]; eps = hyper[5];
        wd = wd != 0.f ? hyper[6] : 0.f;
        seed += __float_as_uint(hyper[7]);
    }
    const float gs = grad_scale ? *grad_scale : 1.f;
    float tmax = 0.f;
    const long long nvec = n / 8;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    // all threads of a 16-lane group must iterate together for the e4m3 path: round the loop bound up
    const long long nvec_pad = (nvec + 31) / 32 * 32;       // whole warps take part in the shuffles
    for (long long i = bx * static_cast<long long>(blockDim.x) + tx; i < nvec_pad; i += stride)
        adamw_vec(i, i < nvec, param, grad, m_state, v_state, m_scales, lr, beta1, beta2, bc1, bc2, eps, wd, gs, seed, elem_offset, tmax);
    block_absmax_commit(absmax_out, tmax, scratch);
}

// All tensors of an optimizer step in one launch.  A model has a handful of large tensors and hundreds of small ones; one launch per
// tensor left the GPU waiting for the host (about 10 us a call) and for the last CTAs of every launch.  A CTA takes chunks of
// kAdamChunk elements and finds the tensor of a chunk by bisection.  Same arithmetic and random words as adamw_kernel.
// The table and the step's scalars are found through a zero that comes out of the wait, so that they can be loaded again instead of kept in registers
// (64, four blocks per SM; 80 and three with their pointers out of the wait: 24 layers of 0.5B shapes, bf16, 960 us, 770 now).  One chunk per block: as
// many blocks as reside stride through the same few megabytes of every stream in step (as in llmq_adamw_hyper); 8 blocks per SM / this, us:
// 24 layers of 0.5B shapes, bf16 801 / 773, bf16 and fp32 moments, 6 of 1.5B shapes 935 / 811, all fp32 1178 / 1026, e4m3 and bf16 moments, 12 layers 1701 /
// 1596, 24 layers of 256 channels, bf16 73.7 / 74.7.
struct AdamTensor {                              // 11 x 8 bytes, filled by the host
    void* param; const void* grad; void* m; void* v;
    float* m_scales; float* absmax;              // optional
    long long n, elem_offset, first_chunk;
    long long seed;                              // added to the step's seed
    long long decay;                             // 1: weight decay applies
};
constexpr int kAdamChunk = 16384;

template <typename P, typename G, typename M, typename Vv>
__global__ void __launch_bounds__(256)
adamw_multi_kernel(const AdamTensor* __restrict__ tensors, int n_tensors, long long n_chunks, float lr, float beta1, float beta2, float bc1,
                   float bc2, float eps, float wd, const float* __restrict__ grad_scale, uint32_t seed, const float* __restrict__ hyper) {
    grid_wait(grad_scale);
    const int bx = after_wait(blockIdx.x), tx = after_wait(threadIdx.x), zero = after_wait(0u);
    __shared__ float scratch[32];
    if (hyper) {
        const float* h = hyper + zero;
        lr = h[0]; beta1 = h[1]; beta2 = h[2]; bc1 = h[3]; bc2 = h[4]; eps = h[5]; wd = h[6];
        seed += __float_as_uint(h[7]);
    }
    const float gs = grad_scale ? *grad_scale : 1.f;
    for (long long chunk = bx; chunk < n_chunks; chunk += gridDim.x) {
        int lo = zero, hi = n_tensors - 1;          // last tensor whose first chunk is not behind this one
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (tensors[mid].first_chunk <= chunk) lo = mid; else hi = mid - 1;
        }
        const AdamTensor t = tensors[lo];
        const long long nvec = t.n / 8, v0 = (chunk - t.first_chunk) * (kAdamChunk / 8);
        const long long v1 = min((nvec + 31) / 32 * 32, v0 + kAdamChunk / 8);
        float tmax = 0.f;
        for (long long i = v0 + tx; i < v1; i += blockDim.x)
            adamw_vec(i, i < nvec, static_cast<P*>(t.param), static_cast<const G*>(t.grad), static_cast<M*>(t.m), static_cast<Vv*>(t.v), t.m_scales,
                      lr, beta1, beta2, bc1, bc2, eps, t.decay ? wd : 0.f, gs, seed + static_cast<uint32_t>(t.seed), t.elem_offset, tmax);
        block_absmax_commit(t.absmax, tmax, scratch);
    }
}

// Sum of squares; block b adds its partial to out[b], so several tensors accumulate into the same
// partial vector in stream order and the result does not depend on atomics.
// FLIGHT loads of a thread in flight, added up in order; STREAM: read once, first to leave the L2.
template <typename T, int FLIGHT, bool STREAM>
__device__ __forceinline__ float thread_sum_squares(const T* __restrict__ x, long long n) {
    using V = Vec16<T>;
    const long long nvec = n / V::N, stride = static_cast<long long>(gridDim.x) * blockDim.x;
    long long i0 = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    float s = 0.f;
    if constexpr (FLIGHT > 1) {
        for (; i0 + (FLIGHT - 1) * stride < nvec; i0 += FLIGHT * stride) {
            V v[FLIGHT];
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j) v[j] = STREAM ? V::load_stream(x + (i0 + j * stride) * V::N) : V::load(x + (i0 + j * stride) * V::N);
#pragma unroll
            for (int j = 0; j < FLIGHT; ++j)
#pragma unroll
                for (int k = 0; k < V::N; ++k) { const float f = to_float(v[j].v[k]); s += f * f; }
        }
    }
    for (; i0 < nvec; i0 += stride) {
        V v = STREAM ? V::load_stream(x + i0 * V::N) : V::load(x + i0 * V::N);
#pragma unroll
        for (int k = 0; k < V::N; ++k) { const float f = to_float(v.v[k]); s += f * f; }
    }
    if (blockIdx.x == 0)
        for (long long i = nvec * V::N + threadIdx.x; i < n; i += blockDim.x) { float f = to_float(x[i]); s += f * f; }
    return s;
}

// One load in flight for tensors that give a thread fewer than four vectors (128 to 3 M bf16 values: 2.0-3.6 us, 2.1-4.3 with the longer
// code), else four.  Four blocks on an SM: at the 34 registers that the compiler would take, three fit and the last 68 of 512 blocks
// run alone.  us after an L2 flush / right after the gradient was written, for 1 load / 4 loads and three blocks / 4 loads and four
// blocks: 67.9 M bf16 values 32.1, 36.8, 31.5 / 35.6, 33.9, 28.7;  268 M 95, 111, 96 (5.6 TB/s) / 104, 110, 88.  fp32 values within the L2
// the same without streaming, which spills at 32 registers: 16.8 M 19.3, 20.0, 19.0 / 18.4, 16.8, 16.4;  beyond it streaming
// loads with the registers they want (BLOCKS 0: no bound): 67.9 M 49.6, 50.5, 50.9 / 60.0, 49.4, 57.8.
template <typename T, int FLIGHT, bool STREAM, int BLOCKS>
__global__ void __launch_bounds__(512, BLOCKS) norm_squared_kernel(float* __restrict__ out, const T* __restrict__ x, long long n) {
    grid_wait(x);                        // thread_sum_squares() finds its loads through plain indices
    const int bx = after_wait(blockIdx.x), tx = after_wait(threadIdx.x);
    __shared__ float scratch[32];
    const float s = block_reduce_sum(thread_sum_squares<T, FLIGHT, STREAM>(x, n), scratch);
    if (tx == 0) out[bx] += s;
}

// The gradients of all tensors in one launch.  Bit for bit what norm_squared_kernel adds up launch by launch: the same sums per thread
// and per tensor, and the tensors' block sums added to out[b] in their order.  Tensors are reduced 16 at a time (one per warp), so
// that a block waits at one pair of barriers per 16 tensors instead of two barriers per tensor.
template <typename T>
__global__ void __launch_bounds__(512) norm_squared_multi_kernel(float* __restrict__ out, const AdamTensor* __restrict__ tensors, int n_tensors) {
    grid_wait();
    const int bx = after_wait(blockIdx.x), tx = after_wait(threadIdx.x), zero = after_wait(0u);
    __shared__ float warp_sums[16][16], sums[16];
    const int warp = tx >> 5, lane = tx & 31;
    float total = tx == 0 ? out[bx] : 0.f;
    for (int t0 = zero; t0 < n_tensors; t0 += 16) {
        const int n = min(16, n_tensors - t0);
        for (int t = 0; t < n; ++t) {
            const float s = warp_reduce_sum(thread_sum_squares<T, 4, true>(static_cast<const T*>(tensors[t0 + t].grad), tensors[t0 + t].n));
            if (lane == 0) warp_sums[t][warp] = s;
        }
        __syncthreads();
        if (warp < n) {
            const float s = warp_reduce_sum(lane < 16 ? warp_sums[warp][lane] : 0.f);
            if (lane == 0) sums[warp] = s;
        }
        __syncthreads();
        if (tx == 0) for (int t = 0; t < n; ++t) total += sums[t];
    }
    if (tx == 0) out[bx] = total;
}

__global__ void __launch_bounds__(512) deterministic_sum_kernel(float* __restrict__ out, const float* __restrict__ in, int n) {
    grid_wait(out, in);
    __shared__ float scratch[32];
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += in[i];
    s = block_reduce_sum(s, scratch);
    if (threadIdx.x == 0) *out = s;
}

// io[0]: squared norm in -> norm out;  io[1]: multiplier that clips the gradient to `clip` (1 if no clipping)
__device__ __forceinline__ void finish_norm(float* io, float nsq, float clip, float* host_norm) {
    float norm = sqrtf(nsq);
    float scale = 1.f;
    if (clip > 0.f && norm > clip) scale = clip / norm;
    if (!isfinite(norm)) scale = 0.f;          // a non-finite gradient must not reach the weights
    io[0] = norm;
    io[1] = scale;
    if (host_norm) *host_norm = norm;
}
__global__ void norm_finish_kernel(float* io, float clip, float* host_norm) {
    grid_wait(io, host_norm);
    finish_norm(io, io[0], clip, host_norm);
}
// deterministic_sum_kernel and norm_finish_kernel in one launch, for callers that have nothing to do in between (2 us a launch)
__global__ void __launch_bounds__(512) norm_sum_finish_kernel(float* __restrict__ io, const float* __restrict__ in, int n, float clip, float* __restrict__ host_norm) {
    grid_wait(io, in, host_norm);
    __shared__ float scratch[32];
    float s = 0.f;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += in[i];
    s = block_reduce_sum(s, scratch);
    if (threadIdx.x == 0) finish_norm(io, s, clip, host_norm);
}

// dst = SR(scale * (a + b))
template <typename T>
__global__ void __launch_bounds__(512)
vector_add_sr_kernel(T* dst, const T* a, const T* b, float scale, long long n, uint32_t seed) {
    const long long nvec = n / 8;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < nvec;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        float fa[8], fb[8];
        load8<T>(fa, a + i * 8);
        load8<T>(fb, b + i * 8);
#pragma unroll
        for (int k = 0; k < 8; ++k) fa[k] = scale * (fa[k] + fb[k]);
        store8_sr<T>(dst + i * 8, fa, static_cast<uint64_t>(i * 8), seed);
    }
}

// dst = SR(scale * (sum_{k != skip} src[k * shard_stride + i] (+ dst[i] if accumulate)))
template <typename T>
__global__ void __launch_bounds__(512)
vector_reduce_sr_kernel(T* dst, const T* src, float scale, int n_shards, int skip, long long shard_stride, int accumulate,
                        long long n, uint32_t seed) {
    const long long nvec = n / 8;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < nvec;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        float acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.f;
        if (accumulate) load8<T>(acc, dst + i * 8);
        for (int sh = 0; sh < n_shards; ++sh) {
            if (sh == skip) continue;
            float f[8];
            load8<T>(f, src + sh * shard_stride + i * 8);
#pragma unroll
            for (int k = 0; k < 8; ++k) acc[k] += f[k];
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] *= scale;
        store8_sr<T>(dst + i * 8, acc, static_cast<uint64_t>(i * 8), seed);
    }
}

}  // namespace

// dtype codes: param/grad: 0 bf16 | 3 fp32;  m: 0 | 3 | 1 (e4m3, needs m_scales and n % 128 == 0);  v: 0 | 3
extern "C" int llmq_adamw_hyper(void*, const void*, void*, void*, float*, long long, float, float, float, int, float, float, const float*, float*,
                                unsigned int, long long, int, int, int, int, int, const float*, cudaStream_t);

extern "C" int llmq_adamw(void* param, const void* grad, void* m, void* v, float* m_scales, long long n, float lr, float beta1,
                          float beta2, int step, float eps, float wd, const float* grad_scale, float* absmax_out,
                          unsigned int seed, long long elem_offset, int p_dtype, int g_dtype, int m_dtype, int v_dtype,
                          int num_sms, cudaStream_t s) {
    return llmq_adamw_hyper(param, grad, m, v, m_scales, n, lr, beta1, beta2, step, eps, wd, grad_scale, absmax_out, seed, elem_offset,
                            p_dtype, g_dtype, m_dtype, v_dtype, num_sms, nullptr, s);
}

// Fills the 8 host floats that `hyper` points the kernel at, with the same arithmetic as the by-value launch.
extern "C" void llmq_adamw_fill_hyper(float* out, float lr, float beta1, float beta2, int step, float eps, float wd, unsigned int seed) {
    out[0] = lr; out[1] = beta1; out[2] = beta2;
    out[3] = 1.f / (1.f - powf(beta1, static_cast<float>(step)));
    out[4] = 1.f / (1.f - powf(beta2, static_cast<float>(step)));
    out[5] = eps; out[6] = wd;
    memcpy(out + 7, &seed, sizeof(seed));
}

// Same, with the step-dependent scalars optionally read from 8 floats in device memory (see adamw_kernel).
extern "C" int llmq_adamw_hyper(void* param, const void* grad, void* m, void* v, float* m_scales, long long n, float lr, float beta1,
                                float beta2, int step, float eps, float wd, const float* grad_scale, float* absmax_out,
                                unsigned int seed, long long elem_offset, int p_dtype, int g_dtype, int m_dtype, int v_dtype,
                                int num_sms, const float* hyper, cudaStream_t s) {
    if (n <= 0) return 0;
    if (n % 8) return -1;
    if (m_dtype == 1 && (n % 128 || !m_scales)) return -2;
    const float bc1 = 1.f / (1.f - powf(beta1, static_cast<float>(step)));
    const float bc2 = 1.f / (1.f - powf(beta2, static_cast<float>(step)));
    // fp32 moments: one round of the loop per block.  With just the resident blocks (8 per SM) these stride through the same few megabytes of
    // every stream in step: 67.9 M elements 263 us, 216 this way; 4.2 M 13.0 / 12.4.  16-bit and 8-bit moments are the same either way (156 / 167
    // and 195 / 194 us): resident blocks.
    const long long rounds = ceil_div_ll(n / 8, 256);
    const int g = m_dtype == 3 && v_dtype == 3 && rounds < (1ll << 30) ? static_cast<int>(rounds) : grid_for(n / 8, 256, num_sms);
#define A_CASE(P, PC, G, GC, M, MC, V, VC)                                                                          \
    if (p_dtype == PC && g_dtype == GC && m_dtype == MC && v_dtype == VC) {                                         \
        launch_chained(adamw_kernel<P, G, M, V>, g, 256, 0, s, static_cast<P*>(param), static_cast<const G*>(grad), static_cast<M*>(m), \
                                                   static_cast<V*>(v), m_scales, n, lr, beta1, beta2, bc1, bc2, eps, wd,   \
                                                   grad_scale, absmax_out, seed, elem_offset, hyper);               \
        return LLMQ_LAUNCH_CHECK();                                                                                 \
    }
    A_CASE(bf16, 0, bf16, 0, bf16, 0, bf16, 0)
    A_CASE(bf16, 0, bf16, 0, float, 3, float, 3)
    A_CASE(bf16, 0, bf16, 0, float, 3, bf16, 0)
    A_CASE(bf16, 0, bf16, 0, bf16, 0, float, 3)
    A_CASE(bf16, 0, bf16, 0, e4m3, 1, bf16, 0)
    A_CASE(bf16, 0, bf16, 0, e4m3, 1, float, 3)
    A_CASE(float, 3, float, 3, float, 3, float, 3)
    A_CASE(float, 3, float, 3, bf16, 0, bf16, 0)
    A_CASE(float, 3, bf16, 0, float, 3, float, 3)
    A_CASE(float, 3, bf16, 0, bf16, 0, bf16, 0)
#undef A_CASE
    return -10;
}

// All tensors of a step: `tensors` is a device array of AdamTensor, first_chunk counts chunks of llmq_adamw_chunk() elements.  Every
// tensor has the given types; sizes are multiples of 8 (128 with e4m3 moments).
extern "C" int llmq_adamw_chunk() { return kAdamChunk; }
extern "C" int llmq_adamw_multi(const void* tensors, int n_tensors, long long n_chunks, float lr, float beta1, float beta2, int step, float eps, float wd,
                                const float* grad_scale, unsigned int seed, int p_dtype, int g_dtype, int m_dtype, int v_dtype, int num_sms,
                                const float* hyper, cudaStream_t s) {
    if (n_tensors <= 0 || n_chunks <= 0) return 0;
    const float bc1 = 1.f / (1.f - powf(beta1, static_cast<float>(step)));
    const float bc2 = 1.f / (1.f - powf(beta2, static_cast<float>(step)));
    const int g = static_cast<int>(n_chunks < (1ll << 30) ? n_chunks : (1ll << 30));
    const AdamTensor* t = static_cast<const AdamTensor*>(tensors);
#define A_CASE(P, PC, G, GC, M, MC, V, VC)                                                                          \
    if (p_dtype == PC && g_dtype == GC && m_dtype == MC && v_dtype == VC) {                                         \
        launch_chained(adamw_multi_kernel<P, G, M, V>, g, 256, 0, s, t, n_tensors, n_chunks, lr, beta1, beta2, bc1, bc2, eps, wd, grad_scale, seed, hyper); \
        return LLMQ_LAUNCH_CHECK();                                                                                 \
    }
    A_CASE(bf16, 0, bf16, 0, bf16, 0, bf16, 0)
    A_CASE(bf16, 0, bf16, 0, float, 3, float, 3)
    A_CASE(bf16, 0, bf16, 0, float, 3, bf16, 0)
    A_CASE(bf16, 0, bf16, 0, bf16, 0, float, 3)
    A_CASE(bf16, 0, bf16, 0, e4m3, 1, bf16, 0)
    A_CASE(bf16, 0, bf16, 0, e4m3, 1, float, 3)
    A_CASE(float, 3, float, 3, float, 3, float, 3)
    A_CASE(float, 3, float, 3, bf16, 0, bf16, 0)
    A_CASE(float, 3, bf16, 0, float, 3, float, 3)
    A_CASE(float, 3, bf16, 0, bf16, 0, bf16, 0)
#undef A_CASE
    return -10;
}

extern "C" int llmq_norm_squared_multi(float* partials, const void* tensors, int n_tensors, int dtype, int num_partials, cudaStream_t s) {
    if (n_tensors <= 0) return 0;
    const AdamTensor* t = static_cast<const AdamTensor*>(tensors);
    if (dtype == 0) launch_chained(norm_squared_multi_kernel<bf16>, num_partials, 512, 0, s, partials, t, n_tensors);
    else if (dtype == 3) launch_chained(norm_squared_multi_kernel<float>, num_partials, 512, 0, s, partials, t, n_tensors);
    else return -10;
    return LLMQ_LAUNCH_CHECK();
}

extern "C" int llmq_norm_squared(float* partials, const void* x, long long n, int dtype, int num_partials, cudaStream_t s) {
    if (n <= 0) return 0;
    if (dtype != 0 && dtype != 3) return -10;
    const bool many = n / (dtype == 0 ? 8 : 4) >= 4LL * 512 * num_partials;
    const bf16* h = static_cast<const bf16*>(x);
    const float* f = static_cast<const float*>(x);
#define GO(P, ...) launch_chained(norm_squared_kernel<__VA_ARGS__>, num_partials, 512, 0, s, partials, P, n)
    if (dtype == 0)               { if (many) GO(h, bf16, 4, true, 4); else GO(h, bf16, 1, false, 4); }
    else if (!many)               GO(f, float, 1, false, 4);
    else if (n * 4 <= 126LL << 20) GO(f, float, 4, false, 4);
    else                          GO(f, float, 4, true, 0);
#undef GO
    return LLMQ_LAUNCH_CHECK();
}

extern "C" int llmq_deterministic_sum(float* out, const float* in, int n, cudaStream_t s) {
    launch_chained(deterministic_sum_kernel, 1, 512, 0, s, out, in, n);
    return LLMQ_LAUNCH_CHECK();
}

extern "C" int llmq_norm_finish(float* io, float clip, float* host_norm, cudaStream_t s) {
    launch_chained(norm_finish_kernel, 1, 1, 0, s, io, clip, host_norm);
    return LLMQ_LAUNCH_CHECK();
}

// io[0] <- norm of which `in` holds the partial squares, io[1] <- the multiplier of llmq_norm_finish
extern "C" int llmq_norm_sum_finish(float* io, const float* in, int n, float clip, float* host_norm, cudaStream_t s) {
    launch_chained(norm_sum_finish_kernel, 1, 512, 0, s, io, in, n, clip, host_norm);
    return LLMQ_LAUNCH_CHECK();
}

extern "C" int llmq_vector_add_sr(void* dst, const void* a, const void* b, float scale, long long n, unsigned int seed, int dtype,
                                  int num_sms, cudaStream_t s) {
    if (n <= 0) return 0;
    if (n % 8) return -1;
    int g = grid_for(n / 8, 512, num_sms);
    if (dtype == 0) vector_add_sr_kernel<bf16><<<g, 512, 0, s>>>(static_cast<bf16*>(dst), static_cast<const bf16*>(a), static_cast<const bf16*>(b), scale, n, seed);
    else if (dtype == 3) vector_add_sr_kernel<float><<<g, 512, 0, s>>>(static_cast<float*>(dst), static_cast<const float*>(a), static_cast<const float*>(b), scale, n, seed);
    else return -10;
    return LLMQ_LAUNCH_CHECK();
}

extern "C" int llmq_vector_reduce_sr(void* dst, const void* src, float scale, int n_shards, int skip, long long shard_stride,
                                     int accumulate, long long n, unsigned int seed, int dtype, int num_sms, cudaStream_t s) {
    if (n <= 0) return 0;
    if (n % 8) return -1;
    int g = grid_for(n / 8, 512, num_sms);
    if (dtype == 0) vector_reduce_sr_kernel<bf16><<<g, 512, 0, s>>>(static_cast<bf16*>(dst), static_cast<const bf16*>(src), scale, n_shards, skip, shard_stride, accumulate, n, seed);
    else if (dtype == 3) vector_reduce_sr_kernel<float><<<g, 512, 0, s>>>(static_cast<float*>(dst), static_cast<const float*>(src), scale, n_shards, skip, shard_stride, accumulate, n, seed);
    else return -10;
    return LLMQ_LAUNCH_CHECK();
}
