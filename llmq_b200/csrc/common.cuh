// Device helpers shared by all kernels: 16-byte vector access, warp/block reductions, abs-max
// atomics, a counter-based hash RNG for stochastic rounding, and fp8 conversion.
#pragma once
#include <cstdint>
#include <utility>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

typedef __nv_bfloat16 bf16;
typedef __nv_fp8_e4m3 e4m3;
typedef __nv_fp8_e5m2 e5m2;

#define LLMQ_LAUNCH_CHECK() static_cast<int>(cudaGetLastError())

// ------------------------------------------------------------------------------------------------
// Programmatic dependent launch.  A kernel launched with launch_chained() is set up while the kernel before it on the stream still runs, and may
// start then: launch overhead, block scheduling and whatever it does before grid_wait() (barriers, tensor memory) overlap with that
// kernel.  It must not touch global memory before grid_wait(), which returns when the kernel before it is complete and its
// writes are visible; as that one has waited for its own predecessor, the order of the whole stream holds.  In a kernel that was launched the
// ordinary way the wait is a no-op.
// Without more the next kernel starts when every block of this one has left.  grid_release() lets it start once every block has called it, which
// pays for kernels that keep an SM to themselves and have a long way to their first load: GEMM and attention (GEMMs that leave many SMs idle for
// long do not, see gemm_tcgen05.cu).  Elsewhere blocks of the next kernel, put beside running ones, end up several on one SM with another
// SM idle, and for grids of many small blocks the call itself costs time.  us with / without the release, launched behind themselves in a graph:
// AdamW tables of 2.4 M elements 21.5 / 9.6, gradient norm, clipping and that AdamW 36.4 / 21.4, bias gradient 7308 x 1000 8.2 / 6.4, RoPE of 60 tokens 2.1 / 1.7,
// RMSNorm forward 8165 x 512 9.2 / 6.1.  A kernel that waits for other GPUs must not call it.
// Launched this way: attention, RoPE, GEMM, their small second passes, the embedding, the norm and the AdamW launches of an update.  A pass over
// rope, attention forward, backward (then three kernels) and rope, launched plainly / this way: 333 tokens, 12 / 2 heads of 128 in a graph 66 / 39, 8 x 1024
// tokens, 14 / 2 heads of 64 221 / 175.  The long streaming kernels (SwiGLU, RMSNorm, quantise, transposes, classifier) are not:
// what the compiler loses by the two functions below costs them more than a launch (RMSNorm pass 186 -> 195 us, SwiGLU 793 -> 811).
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Loads through const __restrict__ pointers (and __ldg, __ldcs) count as loads of memory that nothing writes while the kernel runs: the compiler
// may move them in front of the wait.  It cannot when their address comes out of it, so everything that is loaded is either found through a
// block or thread index (or a zero) that went through after_wait(), or through one of `pointers`.  (All pointers that way would also lose their
// __restrict__, and the kernels the freedom to load ahead of their stores or to load again instead of keeping a register: AdamW 204 -> 218 us.)
template <typename... P>
__device__ __forceinline__ void grid_wait(P&... pointers) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    ((void)([&] { asm volatile("" : "+l"(pointers)); }()), ...);
}
__device__ __forceinline__ int after_wait(unsigned int index) {
    asm volatile("" : "+r"(index));
    return static_cast<int>(index);
}
// `cluster` > 1: blocks per cluster along x.  As with <<<>>>, the caller takes the status with LLMQ_LAUNCH_CHECK(), which also clears it: one
// that stayed behind would be reported again by the launch check of a later, unrelated kernel.
template <typename... P, typename... A>
void launch_chained_cluster(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cudaLaunchAttribute attr[2]{};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = cluster > 1 ? 2 : 1;
    static_cast<void>(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}
template <typename... P, typename... A>
void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    launch_chained_cluster(kernel, grid, block, smem, stream, 1, std::forward<A>(args)...);
}

__host__ __device__ constexpr long long ceil_div_ll(long long a, long long b) { return (a + b - 1) / b; }
// SMs of the current device
inline int device_sms() {
    static int sms[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& n = sms[dev & 63];
    if (n <= 0 && (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)) n = 148;
    return n;
}
__host__ __device__ constexpr int ceil_div_i(int a, int b) { return (a + b - 1) / b; }

// ------------------------------------------------------------------------------------------------
// Reductions
__device__ __forceinline__ float warp_reduce_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_reduce_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// Block-wide reductions; `scratch` holds at least 32 floats of shared memory. All threads get the result.
__device__ __forceinline__ float block_reduce_sum(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_reduce_sum(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float r = (lane < nw) ? scratch[lane] : 0.f;
    return warp_reduce_sum(r);
}
__device__ __forceinline__ float block_reduce_max(float v, float* scratch) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_reduce_max(v);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float r = (lane < nw) ? scratch[lane] : -INFINITY;
    return warp_reduce_max(r);
}

// abs-max values are non-negative floats, whose bit patterns order like unsigned integers
__device__ __forceinline__ void atomic_max_float(float* addr, float v) {
    atomicMax(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v));
}
// Reduces a per-thread abs-max over the block and merges it into *dst (if dst != null).
__device__ __forceinline__ void block_absmax_commit(float* dst, float tmax, float* scratch) {
    if (!dst) return;
    tmax = block_reduce_max(tmax, scratch);
    if (threadIdx.x == 0 && tmax > 0.f) atomic_max_float(dst, tmax);
}

// ------------------------------------------------------------------------------------------------
// Element access for the supported storage types
template <typename T> __device__ __forceinline__ float to_float(T v);
template <> __device__ __forceinline__ float to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_float<bf16>(bf16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_float<e4m3>(e4m3 v) { return static_cast<float>(v); }
template <> __device__ __forceinline__ float to_float<e5m2>(e5m2 v) { return static_cast<float>(v); }

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ bf16 from_float<bf16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ e4m3 from_float<e4m3>(float v) { return e4m3(v); }   // saturating
template <> __device__ __forceinline__ e5m2 from_float<e5m2>(float v) { return e5m2(v); }

// Two floats -> two e4m3 bytes with one conversion instruction (saturating, round to nearest even).
__device__ __forceinline__ uint32_t pack_e4m3x2(float lo, float hi) {
    return static_cast<uint32_t>(__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3));
}
__device__ __forceinline__ uint2 pack_e4m3x8(const float (&f)[8]) {
    uint2 r;
    r.x = pack_e4m3x2(f[0], f[1]) | (pack_e4m3x2(f[2], f[3]) << 16);
    r.y = pack_e4m3x2(f[4], f[5]) | (pack_e4m3x2(f[6], f[7]) << 16);
    return r;
}

// 16-byte vector of T
template <typename T>
struct alignas(16) Vec16 {
    static constexpr int N = 16 / sizeof(T);
    T v[N];
    __device__ __forceinline__ static Vec16 load(const T* p) {
        Vec16 r;
        *reinterpret_cast<uint4*>(r.v) = *reinterpret_cast<const uint4*>(p);
        return r;
    }
    __device__ __forceinline__ static Vec16 load_stream(const T* p) {   // read-once data
        Vec16 r;
        *reinterpret_cast<uint4*>(r.v) = __ldcs(reinterpret_cast<const uint4*>(p));
        return r;
    }
    __device__ __forceinline__ void store(T* p) const { *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(v); }
    __device__ __forceinline__ void store_stream(T* p) const { __stcs(reinterpret_cast<uint4*>(p), *reinterpret_cast<const uint4*>(v)); }
};

// ------------------------------------------------------------------------------------------------
// Division of a 31-bit index by a loop-invariant divisor with one multiply-high and a shift (the per-element
// index arithmetic of the streaming kernels would otherwise cost more instructions than their math).
struct FastDiv {
    uint32_t d, mul, shr;
    FastDiv() : d(1), mul(0), shr(0) {}
    explicit FastDiv(uint32_t div) : d(div), mul(0), shr(0) {
        if (div > 1) {
            uint32_t lg = 0;
            while ((1ull << lg) < div) ++lg;
            const uint32_t p = 31 + lg;
            mul = static_cast<uint32_t>(((1ull << p) + div - 1) / div);
            shr = p - 32;
        }
    }
    // n < 2^31
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return d == 1 ? n : (__umulhi(n, mul) >> shr); }
    __device__ __forceinline__ void divmod(uint32_t n, uint32_t& q, uint32_t& r) const { q = div(n); r = n - q * d; }
};

// ------------------------------------------------------------------------------------------------
// Counter-based hash RNG.  The value depends only on (counter, seed), never on launch geometry, so
// that recomputation and different chunkings reproduce the same rounding decisions.
__device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
    x ^= x >> 16; x *= 0x7feb352du;
    x ^= x >> 15; x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}
__device__ __forceinline__ uint32_t rng_u32(uint64_t counter, uint32_t seed) {
    uint32_t lo = static_cast<uint32_t>(counter), hi = static_cast<uint32_t>(counter >> 32);
    return hash_u32(lo ^ hash_u32(hi + 0x9e3779b9u * (seed + 1u)) ^ (seed * 0x85ebca6bu));
}

// Stochastic rounding fp32 -> bf16: add 16 random bits below the bf16 mantissa and truncate.
__device__ __forceinline__ bf16 sr_bf16(float x, uint32_t rnd) {
    uint32_t bits = __float_as_uint(x);
    if ((bits & 0x7f800000u) == 0x7f800000u) return __float2bfloat16_rn(x);   // inf / nan
    bits += (rnd & 0xFFFFu);
    bits &= 0xFFFF0000u;
    return __float2bfloat16_rn(__uint_as_float(bits));    // exact
}
// Two values at once, packed (lo in the low half): the same bits as two calls of sr_bf16 with r and r >> 16, in about half the
// instructions (one finiteness branch and one byte permute per pair).
__device__ __forceinline__ uint32_t sr_bf16x2(float lo, float hi, uint32_t r) {
    constexpr float kMax = 3.402823466e38f;
    if (fabsf(lo) <= kMax && fabsf(hi) <= kMax)
        return __byte_perm(__float_as_uint(lo) + (r & 0xFFFFu), __float_as_uint(hi) + (r >> 16), 0x7632);
    const bf16 a = sr_bf16(lo, r), b = sr_bf16(hi, r >> 16);
    return static_cast<uint32_t>(__bfloat16_as_ushort(a)) | (static_cast<uint32_t>(__bfloat16_as_ushort(b)) << 16);
}
// Stochastic rounding to e4m3 of a value already scaled into the representable range.
__device__ __forceinline__ e4m3 sr_e4m3(float x, uint32_t rnd) {
    // e4m3 has 3 mantissa bits: make the rounding increment relative to the fp32 exponent
    float ax = fabsf(x);
    if (!(ax < 448.f)) return e4m3(x);
    if (ax < 0.015625f) {                 // subnormal range: fixed quantum 2^-9
        float q = 0.001953125f;
        float lo = floorf(x / q) * q;
        float frac = (x - lo) / q;
        float u = (rnd >> 8) * (1.0f / 16777216.0f);
        return e4m3(frac > u ? lo + q : lo);
    }
    uint32_t bits = __float_as_uint(x);
    bits += (rnd & 0xFFFFFu);             // 20 dropped mantissa bits
    bits &= 0xFFF00000u;
    return e4m3(__uint_as_float(bits));
}
// Two values at once, packed (lo in the low byte): the same bits as two calls of sr_e4m3, with one conversion and one branch where both are normal and
// finite, as nearly all are.
__device__ __forceinline__ uint32_t sr_e4m3x2(float lo, float hi, uint32_t r_lo, uint32_t r_hi) {
    const float a = fabsf(lo), b = fabsf(hi);
    if (fminf(a, b) >= 0.015625f && a < 448.f && b < 448.f)
        return pack_e4m3x2(__uint_as_float((__float_as_uint(lo) + (r_lo & 0xFFFFFu)) & 0xFFF00000u), __uint_as_float((__float_as_uint(hi) + (r_hi & 0xFFFFFu)) & 0xFFF00000u));
    const e4m3 x = sr_e4m3(lo, r_lo), y = sr_e4m3(hi, r_hi);
    return static_cast<uint32_t>(x.__x) | static_cast<uint32_t>(y.__x) << 8;
}
template <typename T> __device__ __forceinline__ T sr_round(float x, uint32_t rnd);
template <> __device__ __forceinline__ float sr_round<float>(float x, uint32_t) { return x; }
template <> __device__ __forceinline__ bf16 sr_round<bf16>(float x, uint32_t rnd) { return sr_bf16(x, rnd); }

// 32 bytes (16 bf16), aligned to as much: a whole sector per lane and instruction
__device__ __forceinline__ void store_sector(void* p, const uint32_t* r) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"l"(p), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// 1 / (1 + e^-x) = 1 / (1 + 2^(-x log2 e)).  The exponent in fp32 (its rounding and that of log2 e) makes the result of a negative x wrong by up to 1.23 |x| 2^-24 of itself, the approximations by
// a few times 2^-23; subnormal numbers are flushed: of the power, which vanishes in the sum, and of the result, which is 0 below 2^-126.
__device__ __forceinline__ float fast_sigmoid(float x) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(-x * 1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
    return r;
}
