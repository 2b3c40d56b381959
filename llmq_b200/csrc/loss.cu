// Fused softmax cross-entropy over the vocabulary with in-place logit gradients, plus the small
// statistics kernels that go with it (per-position loss groups, log-sum-exp monitoring).
// Behavioural counterpart of src/kernels/fused_classifier.cu:20-342 and fused_classifier_tma.cu:40-273:
//   loss[row] += lse - logit[target];   dlogit = p * (dloss + z_reg * lse) - 1[target] * dloss;
//   rows whose target is -100 - or any other id outside [0, V), e.g. from a token file of a larger tokenizer - get
//   zero loss and zero gradient; the id never indexes memory.
// Pass 1 streams a row once and keeps an online (max, sum); pass 2 re-reads the row (still L2 resident: a bf16 row of 152k
// logits is 300 KB) and overwrites it with the gradient using streaming stores, so HBM sees one read and one write per logit.
// bf16 rows are shared by the two CTAs of a cluster, fp32 rows belong to one CTA of 1024 threads.
#include "api.h"
#include "common.cuh"

namespace {

constexpr int CE_THREADS = 1024;

template <typename T>
__global__ void __launch_bounds__(CE_THREADS, 1)
fused_ce_kernel(T* logits, float* __restrict__ losses, float* __restrict__ lse_out, const int* __restrict__ targets,
                float dloss, float z_reg, int rows, int V, long long ld, int write_dlogits) {
    __shared__ float s_max[32], s_sum[32];
    using Vt = Vec16<T>;
    const long long row = rows - 1 - static_cast<long long>(blockIdx.x);   // newest GEMM output first: L2 hits
    T* x = logits + row * ld;
    const int tgt = targets[row];
    const int nvec = V / Vt::N;
    if (tgt < 0 || tgt >= V) {                  // -100 = masked; other out-of-range ids are treated the same way
        if (write_dlogits) {
            Vt z;
#pragma unroll
            for (int k = 0; k < Vt::N; ++k) z.v[k] = from_float<T>(0.f);
            for (int i = threadIdx.x; i < nvec; i += CE_THREADS) z.store_stream(x + i * Vt::N);
            for (int i = nvec * Vt::N + threadIdx.x; i < V; i += CE_THREADS) x[i] = from_float<T>(0.f);
        }
        if (threadIdx.x == 0 && lse_out) lse_out[row] = 0.f;
        return;
    }
    constexpr float kLog2e = 1.4426950408889634f;
    // pass 1: online max / sum (base-2 domain).  The maximum starts at the lowest finite value: -inf logits then give exponentials of
    // -inf, which are 0, before the first finite logit too.
    float m = -3.402823466e38f, s = 0.f;
    for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
        Vt v = Vt::load(x + i * Vt::N);
        float lm = -INFINITY;
#pragma unroll
        for (int k = 0; k < Vt::N; ++k) lm = fmaxf(lm, to_float(v.v[k]));
        if (lm > m) { s *= exp2f((m - lm) * kLog2e); m = lm; }
#pragma unroll
        for (int k = 0; k < Vt::N; ++k) s += exp2f((to_float(v.v[k]) - m) * kLog2e);
    }
    for (int i = nvec * Vt::N + threadIdx.x; i < V; i += CE_THREADS) {
        float f = to_float(x[i]);
        if (f > m) { s *= exp2f((m - f) * kLog2e); m = f; }
        s += exp2f((f - m) * kLog2e);
    }
    // combine (max, sum) pairs across the block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
        float nm = fmaxf(m, om);
        s = s * exp2f((m - nm) * kLog2e) + os * exp2f((om - nm) * kLog2e);
        m = nm;
    }
    if (lane == 0) { s_max[warp] = m; s_sum[warp] = s; }
    __syncthreads();
    m = s_max[lane]; s = s_sum[lane];          // CE_THREADS / 32 == 32 warps
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
        float nm = fmaxf(m, om);
        s = s * exp2f((m - nm) * kLog2e) + os * exp2f((om - nm) * kLog2e);
        m = nm;
    }
    const float lse = logf(s) + m;
    const float tgt_logit = to_float(x[tgt]);
    __syncthreads();                            // everyone has read x[tgt] before it is overwritten
    if (threadIdx.x == 0) {
        losses[row] += lse - tgt_logit;
        if (lse_out) lse_out[row] = lse;
    }
    if (!write_dlogits) return;
    // pass 2: p * gscale = exp2(x*log2e + shift)
    const float gscale = dloss + z_reg * lse;
    const float shift = (gscale > 0.f ? log2f(gscale) : -INFINITY) - lse * kLog2e;
    for (int i = threadIdx.x; i < nvec; i += CE_THREADS) {
        Vt v = Vt::load(x + i * Vt::N);
        const int base = i * Vt::N;
#pragma unroll
        for (int k = 0; k < Vt::N; ++k) {
            float g = exp2f(to_float(v.v[k]) * kLog2e + shift);
            if (base + k == tgt) g -= dloss;
            v.v[k] = from_float<T>(g);
        }
        v.store_stream(x + base);
    }
    for (int i = nvec * Vt::N + threadIdx.x; i < V; i += CE_THREADS) {
        float g = exp2f(to_float(x[i]) * kLog2e + shift);
        if (i == tgt) g -= dloss;
        x[i] = from_float<T>(g);
    }
}

// bf16 rows, two CTAs of a cluster per row and three CTAs on an SM: the passes over one row (a stream of loads, two reductions, a
// stream of loads and stores) overlap with those of other rows, while the rows in flight (222 of up to 300 KB) still fit the L2
// between their two passes.  The CTAs exchange their warps' (maximum, sum) pairs through distributed shared memory.  Exponentials are the
// hardware's directly (with a range step around it, exp2f costs four instructions more and two of them are spent per logit).
// Bound by the two exponentials per logit (280 us of MUFU time at 4096 x 152064) and by memory (375 us for one read and one write):
// 430-459 us there, 622 us with one 1024-thread CTA per row and SM, whose loads, reductions and stores followed one another.  A row kept
// in registers (clusters of eight CTAs, one read) took 819 us: its CTAs live 4 us, most of it start-up and cluster barriers.
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// two floats into the same shared-memory variable of CTA `rank` of the cluster
__device__ __forceinline__ void st_cluster_f32x2(float2* local, int rank, float a, float b) {
    uint32_t dst;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(local))), "r"(rank));
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(dst), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ float ce_exp2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 ce_unpack(uint32_t w) {
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

constexpr int CE_ROW_THREADS = 512;

// Thread t of CTA `part` does what thread part * 512 + t of a 1024-thread block would: vectors part * 512 + t, + 1024, ..., one after
// the other, and the CTAs' 32 warp results are combined in every warp in the order of that block, so the sums have its bits.
// Rows of up to 512 vectors (V < 4104) have no work for the second CTA: PARTS = 1 leaves it out, and the cluster's barriers with it
// (148 x 1000 4.5 us with two CTAs a row, 2.9 with one, 3.6 with one of 1024 threads; 1000 x 1000 19.1, 8.1, 19.9).
template <int PARTS>
__global__ void __launch_bounds__(CE_ROW_THREADS, 3)
fused_ce_row_kernel(bf16* logits, float* __restrict__ losses, float* __restrict__ lse_out, const int* __restrict__ targets,
                    float dloss, float z_reg, int rows, int V, long long ld, int write_dlogits) {
    constexpr int STRIDE = 2 * CE_ROW_THREADS;
    __shared__ float2 s_part[32];               // (maximum, sum) of every warp of the 1024-thread block
    const int part = blockIdx.x % PARTS, tid = threadIdx.x;
    const long long row = rows - 1 - static_cast<long long>(blockIdx.x / PARTS);     // newest GEMM output first: L2 hits
    bf16* x = logits + row * ld;
    const int tgt = targets[row];
    const int nvec = V / 8, first = part * CE_ROW_THREADS + tid;
    const int tail = part == 0 ? V - nvec * 8 : 0;                 // elements behind the last whole vector
    if (tgt < 0 || tgt >= V) {                  // masked row: the same decision in every CTA of the cluster
        if (write_dlogits) {
            for (int i = first; i < nvec; i += STRIDE) __stcs(reinterpret_cast<uint4*>(x) + i, make_uint4(0u, 0u, 0u, 0u));
            if (tid < tail) x[nvec * 8 + tid] = __float2bfloat16_rn(0.f);
        }
        if (part == 0 && tid == 0 && lse_out) lse_out[row] = 0.f;
        return;
    }
    if constexpr (PARTS > 1) cluster_arrive_relaxed();
    constexpr float kLog2e = 1.4426950408889634f;
    const float tgt_logit = (part == 0 && tid == 0) ? __bfloat162float(x[tgt]) : 0.f;    // read before anyone overwrites it
    // pass 1: online maximum and sum of exponentials (base-2 domain), four vectors in flight
    float m = -INFINITY, s = 0.f;
    auto add = [&](const uint4& w) {
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
        const __nv_bfloat162 mx2 = __hmax2(__hmax2(h[0], h[1]), __hmax2(h[2], h[3]));
        const float lm = fmaxf(__low2float(mx2), __high2float(mx2));
        if (lm > m) { s *= ce_exp2((m - lm) * kLog2e); m = lm; }
        const float moff = m == -INFINITY ? 0.f : m;           // nothing but -inf so far: every exponential is 0
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float2 f = ce_unpack(u[q]);
            s += ce_exp2((f.x - moff) * kLog2e);
            s += ce_exp2((f.y - moff) * kLog2e);
        }
    };
    int i = first;
    for (; i + 3 * STRIDE < nvec; i += 4 * STRIDE) {
        uint4 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = *(reinterpret_cast<const uint4*>(x) + i + j * STRIDE);
#pragma unroll
        for (int j = 0; j < 4; ++j) add(w[j]);
    }
    for (; i < nvec; i += STRIDE) add(*(reinterpret_cast<const uint4*>(x) + i));
    const float xt = tid < tail ? __bfloat162float(x[nvec * 8 + tid]) : -INFINITY;
    if (tid < tail) {
        if (xt > m) { s *= ce_exp2((m - xt) * kLog2e); m = xt; }
        if (m != -INFINITY) s += ce_exp2((xt - m) * kLog2e);
    }
    auto combine = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
            const float nm = fmaxf(m, om);
            s = (m == -INFINITY ? 0.f : s * ce_exp2((m - nm) * kLog2e)) + (om == -INFINITY ? 0.f : os * ce_exp2((om - nm) * kLog2e));
            m = nm;
        }
    };
    combine();
    const int lane = tid & 31, warp = tid >> 5;
    if constexpr (PARTS > 1) {
        cluster_wait();                                        // every CTA of the cluster has started
        if (lane < PARTS) st_cluster_f32x2(&s_part[part * (CE_ROW_THREADS / 32) + warp], lane, m, s);
        cluster_arrive();
        cluster_wait();
    } else {
        if (lane == 0) { s_part[warp] = make_float2(m, s); s_part[CE_ROW_THREADS / 32 + warp] = make_float2(-INFINITY, 0.f); }
        __syncthreads();
    }
    m = s_part[lane].x; s = s_part[lane].y;
    combine();
    const float lse = logf(s) + m;
    if (part == 0 && tid == 0) {
        losses[row] += lse - tgt_logit;
        if (lse_out) lse_out[row] = lse;
    }
    if (!write_dlogits) return;
    // pass 2: p * gscale = exp2(x * log2e + shift).  The hardware's exponential flushes results below 2^-126, which bf16 gradients can
    // still hold: vectors with such an element take exp2f.  (In pass 1 every sum holds a 1 beside them.)  4096 x 152064: 430 us with and
    // without the test where no vector has one, 449 us where nearly all have.
    constexpr float kSubnormal = -125.f;
    const float gscale = dloss + z_reg * lse;
    const float shift = (gscale > 0.f ? log2f(gscale) : -INFINITY) - lse * kLog2e;
    const int tv = tgt / 8;                                    // vector that holds the target
    auto grad = [&](uint4 w, int at) {
        uint32_t u[4] = {w.x, w.y, w.z, w.w};
        float g[8];
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
        const __nv_bfloat162 mn2 = __hmin2(__hmin2(h[0], h[1]), __hmin2(h[2], h[3]));
        if (fmaf(fminf(__low2float(mn2), __high2float(mn2)), kLog2e, shift) < kSubnormal) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = ce_unpack(u[j]);
                g[2 * j] = exp2f(fmaf(f.x, kLog2e, shift));
                g[2 * j + 1] = exp2f(fmaf(f.y, kLog2e, shift));
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 f = ce_unpack(u[j]);
                g[2 * j] = ce_exp2(fmaf(f.x, kLog2e, shift));
                g[2 * j + 1] = ce_exp2(fmaf(f.y, kLog2e, shift));
            }
        }
        if (at == tv) {
#pragma unroll
            for (int j = 0; j < 8; ++j) if (at * 8 + j == tgt) g[j] -= dloss;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 h = __floats2bfloat162_rn(g[2 * j], g[2 * j + 1]);
            u[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        __stcs(reinterpret_cast<uint4*>(x) + at, make_uint4(u[0], u[1], u[2], u[3]));
    };
    for (i = first; i + 3 * STRIDE < nvec; i += 4 * STRIDE) {
        uint4 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = __ldcs(reinterpret_cast<const uint4*>(x) + i + j * STRIDE);
#pragma unroll
        for (int j = 0; j < 4; ++j) grad(w[j], i + j * STRIDE);
    }
    for (; i < nvec; i += STRIDE) grad(__ldcs(reinterpret_cast<const uint4*>(x) + i), i);
    if (tid < tail) {
        float g = exp2f(fmaf(xt, kLog2e, shift));
        if (nvec * 8 + tid == tgt) g -= dloss;
        x[nvec * 8 + tid] = __float2bfloat16_rn(g);
    }
}

// max and sum of the per-token LSE values (z-loss monitoring); out = {max, sum}
__global__ void __launch_bounds__(1024) lse_stats_kernel(float* __restrict__ out, const float* __restrict__ lse, long long n, int accumulate) {
    grid_wait(out, lse);
    __shared__ float scratch[32];
    float m = -INFINITY, s = 0.f;
    for (long long i = threadIdx.x; i < n; i += blockDim.x) { float v = lse[i]; m = fmaxf(m, v); s += v; }
    m = block_reduce_max(m, scratch);
    s = block_reduce_sum(s, scratch);
    if (threadIdx.x == 0) {
        if (accumulate) { out[0] = fmaxf(out[0], m); out[1] += s; }
        else { out[0] = m; out[1] = s; }
    }
}

// out[g] = sum over batch and over positions [g*group, (g+1)*group) of losses(B, T)
__global__ void __launch_bounds__(256) grouped_loss_kernel(float* __restrict__ out, const float* __restrict__ losses, int B, int T, int group) {
    grid_wait();
    const int bx = after_wait(blockIdx.x), tx = after_wait(threadIdx.x);
    __shared__ float scratch[32];
    const int g = bx;
    const int t0 = g * group, t1 = min(T, t0 + group);
    float s = 0.f;
    for (int b = 0; b < B; ++b)
        for (int t = t0 + tx; t < t1; t += blockDim.x) s += losses[static_cast<long long>(b) * T + t];
    s = block_reduce_sum(s, scratch);
    if (tx == 0) out[g] = s;
}

}  // namespace

extern "C" int llmq_fused_classifier(void* logits, float* losses, float* lse_out, const int* targets, float dloss, float z_reg,
                                     int rows, int V, long long ld, int dtype, int write_dlogits, cudaStream_t s) {
    if (rows <= 0) return 0;
    if (dtype == 0) {
        if (ld % 8) return -1;
        if (V / 8 <= CE_ROW_THREADS) {
            fused_ce_row_kernel<1><<<rows, CE_ROW_THREADS, 0, s>>>(static_cast<bf16*>(logits), losses, lse_out, targets, dloss, z_reg, rows, V, ld, write_dlogits);
            return LLMQ_LAUNCH_CHECK();
        }
        if (rows > (1 << 30) - 1) return -1;                   // a grid of pairs has no more; such logits would take 8.8 TB
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned int>(rows) * 2); cfg.blockDim = dim3(CE_ROW_THREADS); cfg.stream = s;
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr; cfg.numAttrs = 1;
        const cudaError_t e = cudaLaunchKernelEx(&cfg, fused_ce_row_kernel<2>, static_cast<bf16*>(logits), losses, lse_out, targets, dloss, z_reg, rows, V, ld,
                                                 write_dlogits);
        if (e != cudaSuccess) return static_cast<int>(e);
    } else if (dtype == 3) {
        if (ld % 4) return -1;
        fused_ce_kernel<float><<<rows, CE_THREADS, 0, s>>>(static_cast<float*>(logits), losses, lse_out, targets, dloss, z_reg, rows, V, ld, write_dlogits);
    } else return -10;
    return LLMQ_LAUNCH_CHECK();
}

extern "C" int llmq_lse_stats(float* out, const float* lse, long long n, int accumulate, cudaStream_t s) {
    launch_chained(lse_stats_kernel, 1, 1024, 0, s, out, lse, n, accumulate);
    return LLMQ_LAUNCH_CHECK();
}

extern "C" int llmq_grouped_loss_sum(float* out, const float* losses, int B, int T, int group, cudaStream_t s) {
    int groups = ceil_div_i(T, group);
    if (groups <= 0) return 0;
    launch_chained(grouped_loss_kernel, groups, 256, 0, s, out, losses, B, T, group);
    return LLMQ_LAUNCH_CHECK();
}
