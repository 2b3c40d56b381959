// RMSNorm kernels: (fused residual +) RMSNorm forward with abs-max / direct fp8 emission, and the
// backward pass with a deterministic weight-gradient reduction.
// Behavioural counterpart of src/kernels/rmsnorm.cu:17-460 in the reference: y = T(x * rstd) * w with
// the intermediate rounded to the storage type (matches the HF modelling code), abs-max of y fused.
#include "api.h"
#include "common.cuh"
#include "ptx_sm100.cuh"

namespace {

constexpr int NORM_THREADS = 256;

// One CTA per token row.  Pass 1 reads the row (adding the two residual inputs when fused, and writing
// the sum), pass 2 re-reads it from L1/L2 to normalise.  HBM traffic is one read + one write per tensor.
template <typename T>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_fwd_kernel(T* __restrict__ residual_out,      // may be null when not fused
                   T* __restrict__ y_out,             // may be null when only fp8 output is wanted
                   e4m3* __restrict__ q_out,          // optional direct fp8 output (needs known abs-max)
                   float* __restrict__ rstd_out,
                   const T* __restrict__ in_a, const T* __restrict__ in_b,   // in_b null -> plain norm of in_a
                   const T* __restrict__ weight, float eps, int C,
                   float* __restrict__ absmax_out, const float* __restrict__ known_absmax,
                   float* __restrict__ q_scale_out) {
    __shared__ float scratch[32];
    using V = Vec16<T>;
    const long long row = blockIdx.x;
    const T* a = in_a + row * C;
    const T* b = in_b ? in_b + row * C : nullptr;
    T* res = residual_out ? residual_out + row * C : nullptr;
    const T* x = res ? res : a;

    float ss = 0.f;
    for (int c = threadIdx.x * V::N; c < C; c += NORM_THREADS * V::N) {
        V va = V::load(a + c);
        if (b) {
            V vb = V::load_stream(b + c);
#pragma unroll
            for (int i = 0; i < V::N; ++i) va.v[i] = from_float<T>(to_float(va.v[i]) + to_float(vb.v[i]));
        }
        if (res) va.store(res + c);
#pragma unroll
        for (int i = 0; i < V::N; ++i) { float f = to_float(va.v[i]); ss += f * f; }
    }
    ss = block_reduce_sum(ss, scratch);     // contains __syncthreads: the residual writes are visible below
    const float rstd = rsqrtf(ss / C + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;

    float qmul = 0.f;
    if (q_out) {
        float am = fmaxf(*known_absmax, 1e-10f);
        qmul = 448.f / am;
        if (row == 0 && threadIdx.x == 0 && q_scale_out) *q_scale_out = am / 448.f;
    }
    float tmax = 0.f;
    for (int c = threadIdx.x * V::N; c < C; c += NORM_THREADS * V::N) {
        V vx = V::load(x + c);
        V vw = V::load(weight + c);
        V vy;
        alignas(8) e4m3 q[V::N];
#pragma unroll
        for (int i = 0; i < V::N; ++i) {
            T n = from_float<T>(to_float(vx.v[i]) * rstd);
            vy.v[i] = from_float<T>(to_float(n) * to_float(vw.v[i]));
            float f = to_float(vy.v[i]);
            tmax = fmaxf(tmax, fabsf(f));
            if (q_out) q[i] = e4m3(f * qmul);
        }
        if (y_out) vy.store(y_out + row * C + c);
        if (q_out) {
            if constexpr (V::N == 8) *reinterpret_cast<uint2*>(q_out + row * C + c) = *reinterpret_cast<uint2*>(q);
            else *reinterpret_cast<uint32_t*>(q_out + row * C + c) = *reinterpret_cast<uint32_t*>(q);
        }
    }
    block_absmax_commit(absmax_out, tmax, scratch);
}

// The sum of 8 warp sums in the order of block_reduce_sum's shuffle tree: the kernels below give the bits of a 256-thread block
// reduction whatever their own shape is.
__device__ __forceinline__ float tree8(const float* w) { return ((w[0] + w[4]) + (w[2] + w[6])) + ((w[1] + w[5]) + (w[3] + w[7])); }

// Same contract for rows of up to 8 column vectors per thread: the row is read once (all loads of a thread in flight at once),
// stays in registers across the reduction and is neither stored first nor read again.  A CTA is one row and, where there are enough
// rows, as small as the row allows (64 threads up to 512 vectors), so that many rows share an SM and one row's reduction hides
// behind the others' loads.
// Bound by memory: 16384 x 3584 with the residual add, 470 MB, 77 us (6.1 TB/s) against 92 us for the two-pass kernel above.
template <typename T, int THREADS, int VPT>
__global__ void __launch_bounds__(THREADS)
rmsnorm_fwd_reg_kernel(T* __restrict__ residual_out, T* __restrict__ y_out, e4m3* __restrict__ q_out, float* __restrict__ rstd_out,
                       const T* __restrict__ in_a, const T* __restrict__ in_b, const T* __restrict__ weight, float eps, int C,
                       float* __restrict__ absmax_out, const float* __restrict__ known_absmax, float* __restrict__ q_scale_out) {
    __shared__ float scratch[8], scratch_max[THREADS / 32];
    using V = Vec16<T>;
    const long long row = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    V x[VPT];
    {
        const T* a = in_a + row * C;
        V b[VPT];
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int c = (k * THREADS + threadIdx.x) * V::N;
            if (c < C) x[k] = V::load_stream(a + c);
        }
        if (in_b) {
#pragma unroll
            for (int k = 0; k < VPT; ++k) {
                const int c = (k * THREADS + threadIdx.x) * V::N;
                if (c < C) b[k] = V::load_stream(in_b + row * C + c);
            }
#pragma unroll
            for (int k = 0; k < VPT; ++k) {
                const int c = (k * THREADS + threadIdx.x) * V::N;
                if (c < C) {
#pragma unroll
                    for (int i = 0; i < V::N; ++i) x[k].v[i] = from_float<T>(to_float(x[k].v[i]) + to_float(b[k].v[i]));
                }
            }
        }
    }
    // Vector v of the row belongs to virtual thread v mod 256, which adds its vectors up in ascending order; with 64 threads a thread
    // stands for four virtual threads.
    constexpr int CHAINS = 256 / THREADS;
    float ss[CHAINS];
#pragma unroll
    for (int q = 0; q < CHAINS; ++q) ss[q] = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        const int c = (k * THREADS + threadIdx.x) * V::N;
        if (c < C) {
            if (residual_out) x[k].store(residual_out + row * C + c);
#pragma unroll
            for (int i = 0; i < V::N; ++i) { const float f = to_float(x[k].v[i]); ss[k % CHAINS] += f * f; }
        }
    }
#pragma unroll
    for (int q = 0; q < CHAINS; ++q) {
        const float s = warp_reduce_sum(ss[q]);
        if (lane == 0) scratch[q * (THREADS / 32) + warp] = s;
    }
    __syncthreads();
    const float sum = tree8(scratch);
    const float rstd = rsqrtf(sum / C + eps);
    if (threadIdx.x == 0 && rstd_out) rstd_out[row] = rstd;
    float qmul = 0.f;
    if (q_out) {
        const float am = fmaxf(*known_absmax, 1e-10f);
        qmul = 448.f / am;
        if (row == 0 && threadIdx.x == 0 && q_scale_out) *q_scale_out = am / 448.f;
    }
    float tmax = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        const int c = (k * THREADS + threadIdx.x) * V::N;
        if (c < C) {
            const V vw = V::load(weight + c);
            V vy;
            alignas(8) e4m3 q[V::N];
#pragma unroll
            for (int i = 0; i < V::N; ++i) {
                const T n = from_float<T>(to_float(x[k].v[i]) * rstd);
                vy.v[i] = from_float<T>(to_float(n) * to_float(vw.v[i]));
                const float f = to_float(vy.v[i]);
                tmax = fmaxf(tmax, fabsf(f));
                if (q_out) q[i] = e4m3(f * qmul);
            }
            if (y_out) vy.store(y_out + row * C + c);
            if (q_out) {
                if constexpr (V::N == 8) *reinterpret_cast<uint2*>(q_out + row * C + c) = *reinterpret_cast<uint2*>(q);
                else *reinterpret_cast<uint32_t*>(q_out + row * C + c) = *reinterpret_cast<uint32_t*>(q);
            }
        }
    }
    if (absmax_out) {
        tmax = warp_reduce_max(tmax);
        if (lane == 0) scratch_max[warp] = tmax;
        __syncthreads();
        if (threadIdx.x == 0) {
#pragma unroll
            for (int w = 1; w < THREADS / 32; ++w) tmax = fmaxf(tmax, scratch_max[w]);
            // a plain read first: once the running maximum has grown, most rows have nothing to add to it
            if (tmax > *reinterpret_cast<volatile float*>(absmax_out)) atomic_max_float(absmax_out, tmax);
        }
    }
}

// Backward.  Persistent CTAs walk over rows; each thread owns up to VPT 16-byte column vectors and keeps
// its share of the weight gradient in registers.  Partials go to scratch[gridDim.x][C] and a second
// kernel sums them in a fixed order (deterministic, no atomics).
template <typename T, int VPT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_bwd_kernel(T* __restrict__ dinp,               // in: upstream residual gradient, out: += norm gradient
                   float* __restrict__ dw_partial,     // [gridDim.x, C]
                   const T* __restrict__ dout, const T* __restrict__ inp, const T* __restrict__ weight,
                   const float* __restrict__ rstd, int rows, int C, float* __restrict__ absmax_out) {
    __shared__ float scratch[32];
    using V = Vec16<T>;
    float dw[VPT][V::N];
#pragma unroll
    for (int k = 0; k < VPT; ++k)
#pragma unroll
        for (int i = 0; i < V::N; ++i) dw[k][i] = 0.f;
    float tmax = 0.f;

    for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
        const T* dy = dout + row * C;
        const T* x = inp + row * C;
        T* dx = dinp + row * C;
        const float rs = rstd[row];
        // pass 1: dot = sum(w * dy * xhat)
        float dot = 0.f;
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            int c = (k * NORM_THREADS + threadIdx.x) * V::N;
            if (c < C) {
                V vdy = V::load(dy + c), vx = V::load(x + c), vw = V::load(weight + c);
#pragma unroll
                for (int i = 0; i < V::N; ++i) {
                    float xh = to_float(vx.v[i]) * rs;
                    float g = to_float(vdy.v[i]);
                    dot += to_float(vw.v[i]) * g * xh;
                    dw[k][i] += g * xh;
                }
            }
        }
        dot = block_reduce_sum(dot, scratch) / C;
        // pass 2 (operands are L1/L2 resident)
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            int c = (k * NORM_THREADS + threadIdx.x) * V::N;
            if (c < C) {
                V vdy = V::load(dy + c), vx = V::load(x + c), vw = V::load(weight + c), vd = V::load(dx + c);
#pragma unroll
                for (int i = 0; i < V::N; ++i) {
                    float xh = to_float(vx.v[i]) * rs;
                    float g = (to_float(vw.v[i]) * to_float(vdy.v[i]) - xh * dot) * rs;
                    float r = to_float(vd.v[i]) + g;
                    vd.v[i] = from_float<T>(r);
                    tmax = fmaxf(tmax, fabsf(to_float(vd.v[i])));
                }
                vd.store(dx + c);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        int c = (k * NORM_THREADS + threadIdx.x) * V::N;
        if (c < C) {
#pragma unroll
            for (int i = 0; i < V::N; ++i) dw_partial[static_cast<long long>(blockIdx.x) * C + c + i] = dw[k][i];
        }
    }
    block_absmax_commit(absmax_out, tmax, scratch);
}

// 16 bytes from global to shared memory, asynchronously; a thread waits for its own copies in groups, in order
__device__ __forceinline__ void copy_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// `bytes` (a multiple of 16, both addresses aligned to 16) from global to shared memory by the copy engine; counted by the barrier
__device__ __forceinline__ void copy_row_async(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Same contract, for fp32 rows of two to four column vectors per thread, for short rows and for blocks with one or two (launch_bwd has the lines): the row's dout,
// inp and residual gradient are loaded once and stay in registers across the block-wide dot product.  fp32 4000 x 4096 51.6 us, 53.2 with the rows in shared memory (below), 1000 x 2048 12.2 / 13.2.
// STAGES > 0: that many rows to come are on their way into shared memory; every thread copies and reads back its own vectors, so that no row waits for a barrier
// or for the thread that issues.
template <typename T, int VPT, int STAGES>
__global__ void __launch_bounds__(NORM_THREADS, VPT <= 2 ? 3 : 2)
rmsnorm_bwd_reg_kernel(T* __restrict__ dinp, float* __restrict__ dw_partial, const T* __restrict__ dout, const T* __restrict__ inp,
                       const T* __restrict__ weight, const float* __restrict__ rstd, int rows, int C, float* __restrict__ absmax_out) {
    __shared__ float scratch[32];
    __shared__ float dots[2][NORM_THREADS / 32];             // alternating, so that one barrier per row is enough
    extern __shared__ __align__(16) uint8_t ring[];          // [STAGES][dout, inp, dinp][C]
    using V = Vec16<T>;
    float dw[VPT][V::N];
    V vw[VPT];
    auto slot = [&](int stage, int what, int c) { return reinterpret_cast<T*>(ring) + (stage * 3 + what) * C + c; };
    auto fetch = [&](long long row, int stage) {
        if (row < rows) {
#pragma unroll
            for (int k = 0; k < VPT; ++k) {
                const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
                if (c < C) {
                    copy_async16(slot(stage, 0, c), dout + row * C + c);
                    copy_async16(slot(stage, 1, c), inp + row * C + c);
                    copy_async16(slot(stage, 2, c), dinp + row * C + c);
                }
            }
        }
        copy_async_commit();                                 // a group per row, empty beyond the last one
    };
    if constexpr (STAGES > 0) {
#pragma unroll
        for (int st = 0; st < STAGES; ++st) fetch(blockIdx.x + static_cast<long long>(st) * gridDim.x, st);
    }
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
        if (c < C) vw[k] = V::load(weight + c);
#pragma unroll
        for (int i = 0; i < V::N; ++i) dw[k][i] = 0.f;
    }
    float tmax = 0.f;
    const float inv_c = 1.f / C;
    int par = 0, stage = 0;
    for (long long row = blockIdx.x; row < rows; row += gridDim.x, par ^= 1) {
        const T* dy = dout + row * C;
        const T* x = inp + row * C;
        T* dx = dinp + row * C;
        V vdy[VPT], vx[VPT], vd[STAGES > 0 ? 1 : VPT];
        if constexpr (STAGES > 0) copy_async_wait<STAGES - 1>();
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
            if constexpr (STAGES > 0) {
                if (c < C) { vdy[k] = V::load(slot(stage, 0, c)); vx[k] = V::load(slot(stage, 1, c)); }
            } else {
                if (c < C) { vdy[k] = V::load_stream(dy + c); vx[k] = V::load_stream(x + c); vd[k] = V::load_stream(dx + c); }
            }
        }
        const float rs = rstd[row];
        float dot = 0.f;
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
            if (c < C) {
#pragma unroll
                for (int i = 0; i < V::N; ++i) {
                    const float xh = to_float(vx[k].v[i]) * rs;
                    const float g = to_float(vdy[k].v[i]);
                    dot += to_float(vw[k].v[i]) * g * xh;
                    dw[k][i] += g * xh;
                }
            }
        }
        dot = warp_reduce_sum(dot);
        if ((threadIdx.x & 31) == 0) dots[par][threadIdx.x >> 5] = dot;
        __syncthreads();
        dot = tree8(dots[par]) * inv_c;
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
            if (c < C) {
                V& d = vd[STAGES > 0 ? 0 : k];
                if constexpr (STAGES > 0) d = V::load(slot(stage, 2, c));
#pragma unroll
                for (int i = 0; i < V::N; ++i) {
                    const float xh = to_float(vx[k].v[i]) * rs;
                    const float g = (to_float(vw[k].v[i]) * to_float(vdy[k].v[i]) - xh * dot) * rs;
                    d.v[i] = from_float<T>(to_float(d.v[i]) + g);
                    tmax = fmaxf(tmax, fabsf(to_float(d.v[i])));
                }
                d.store(dx + c);
            }
        }
        if constexpr (STAGES > 0) {
            fetch(row + static_cast<long long>(STAGES) * gridDim.x, stage);
            if (++stage == STAGES) stage = 0;
        }
    }
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
        if (c < C) {
#pragma unroll
            for (int i = 0; i < V::N; ++i) dw_partial[static_cast<long long>(blockIdx.x) * C + c + i] = dw[k][i];
        }
    }
    block_absmax_commit(absmax_out, tmax, scratch);
}

// Waits for a row's copies; false when the limit ran out, in this thread or (in later rows) in another one
__device__ __forceinline__ bool row_wait(uint32_t bar, uint32_t parity, volatile uint32_t* gave_up) {
    return sm100::mbar_try_wait(bar, parity) || (!*gave_up && sm100::mbar_wait(bar, parity, gave_up));
}

// The end of a block whose copies did not come: what may still be under way, the copies of the STAGES rows from `first_lost` on, has to land before the block
// gives its shared memory back, and its rows become NaN
template <int STAGES, typename T>
__device__ __noinline__ void give_up_rows(T* dinp, int rows, int C, uint32_t full, long long first_lost) {
    const long long step = gridDim.x;
    if (threadIdx.x == 0) {
        const uint64_t t0 = sm100::globaltimer_ns();
        long long n = (first_lost - blockIdx.x) / step;
        for (int i = 0; i < STAGES; ++i, ++n)
            while (blockIdx.x + n * step < rows && !sm100::mbar_try_wait(full + 8 * static_cast<uint32_t>(n % STAGES), (n / STAGES) & 1) &&
                   sm100::globaltimer_ns() - t0 < sm100::kWaitLimitNs) {}
    }
    for (long long row = blockIdx.x; row < rows; row += step)
        for (int c = threadIdx.x; c < C; c += NORM_THREADS) dinp[row * C + c] = from_float<T>(NAN);
}

// Same contract, for rows of up to 4 column vectors per thread.  Rows to come are on their way into shared memory: three bulk copies per row, issued by one
// thread, so that neither registers nor load instructions are spent on what is in flight, and the registers hold the weight gradient and little
// else (both passes over a row read it from shared memory).  One barrier per row; it also says that the row before has been read, whose place the next
// copies take.  Memory is the limit for long rows.  us, rows in registers (two vectors a thread) or copied thread by thread (one, four) / now:
// 16384 x 3584, 470 MB, 98.7 / 77.9;  16384 x 3072 91 / 71;  4096 x 3584 31.6 / 30.3;  16384 x 5120 191 / 146;  4000 x 8192 91 / 66;  16384 x 2048 66 / 54;  16384 x 896 42.5 / 37.5;
// 4096 x 896 16.3 / 14.7;  fp32 4096 x 896 18.7 / 17.3.  Two rows per turn and barrier, with two CTAs per SM: 16384 x 3584 84.
// A copy that does not come within the limit of the waits: the status word says so, and the weight gradient and all rows of its block become NaN, so that
// callers without a status word see it too.  (Leaving the loop there costs 1 to 10 % where nothing is wrong.)
template <typename T, int VPT, int STAGES, int CTAS>
__global__ void __launch_bounds__(NORM_THREADS, CTAS)
rmsnorm_bwd_ring_kernel(T* __restrict__ dinp, float* __restrict__ dw_partial, const T* __restrict__ dout, const T* __restrict__ inp,
                        const T* __restrict__ weight, const float* __restrict__ rstd, int rows, int C, float* __restrict__ absmax_out,
                        unsigned int* __restrict__ status) {
    __shared__ float scratch[32];
    static_assert(STAGES >= 2, "the row in use and the ones on their way");
    __shared__ float dots[2][NORM_THREADS / 32];             // alternating, so that one barrier per row is enough
    extern __shared__ __align__(16) uint8_t ring[];          // [STAGES][dout, inp, dinp][C]
    __shared__ uint64_t full[STAGES];
    __shared__ uint32_t gave_up;
    __shared__ long long first_lost;                         // where thread 0's wait ran out
    using V = Vec16<T>;
    float dw[VPT][V::N];
    V vw[VPT];
    const uint32_t row_bytes = C * sizeof(T);
    int fetch_end = rows;
    auto slot = [&](int stage, int what) { return ring + (stage * 3 + what) * row_bytes; };
    auto fetch = [&](long long row, int stage) {             // one thread
#ifdef LLMQ_TEST_LOST_ROW
        if (row == LLMQ_TEST_LOST_ROW) return;               // builds for tests: a row whose copies never come
#endif
        if (row < fetch_end) {
            const uint32_t bar = sm100::smem_u32(full + stage);
            sm100::mbar_expect_tx(bar, 3 * row_bytes);
            copy_row_async(sm100::smem_u32(slot(stage, 0)), dout + row * C, row_bytes, bar);
            copy_row_async(sm100::smem_u32(slot(stage, 1)), inp + row * C, row_bytes, bar);
            copy_row_async(sm100::smem_u32(slot(stage, 2)), dinp + row * C, row_bytes, bar);
        }
    };
    const long long step = gridDim.x;
    if (threadIdx.x == 0) {
        for (int st = 0; st < STAGES; ++st) sm100::mbar_init(sm100::smem_u32(full + st), 1);
        gave_up = 0;
        first_lost = rows;
        sm100::mbar_init_fence();
        for (int st = 0; st < STAGES; ++st) fetch(blockIdx.x + st * step, st);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
        if (c < C) vw[k] = V::load(weight + c);
#pragma unroll
        for (int i = 0; i < V::N; ++i) dw[k][i] = 0.f;
    }
    float tmax = 0.f;
    const float inv_c = 1.f / C;
    int par = 0, stage = 0;
    uint32_t phase = 0;
    for (long long row = blockIdx.x; row < rows; row += step, par ^= 1) {
        const float rs = rstd[row];
        float dot = 0.f;
        if (!row_wait(sm100::smem_u32(full + stage), phase, &gave_up)) {
            if (threadIdx.x == 0 && fetch_end) first_lost = row;
            fetch_end = 0;                                   // nothing is fetched any more
        }
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
            if (c < C) {
                const V vdy = V::load(reinterpret_cast<const T*>(slot(stage, 0)) + c), vx = V::load(reinterpret_cast<const T*>(slot(stage, 1)) + c);
#pragma unroll
                for (int i = 0; i < V::N; ++i) {
                    const float xh = to_float(vx.v[i]) * rs;
                    const float g = to_float(vdy.v[i]);
                    dot += to_float(vw[k].v[i]) * g * xh;
                    dw[k][i] += g * xh;
                }
            }
        }
        dot = warp_reduce_sum(dot);
        if ((threadIdx.x & 31) == 0) dots[par][threadIdx.x >> 5] = dot;
        __syncthreads();
        // every thread is through with the row before: the row STAGES behind that one takes its place
        if (threadIdx.x == 0 && row != blockIdx.x) fetch(row + (STAGES - 1) * step, stage == 0 ? STAGES - 1 : stage - 1);
        dot = tree8(dots[par]) * inv_c;
        T* dx = dinp + row * C;
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
            if (c < C) {
                const V vdy = V::load(reinterpret_cast<const T*>(slot(stage, 0)) + c), vx = V::load(reinterpret_cast<const T*>(slot(stage, 1)) + c);
                V vd = V::load(reinterpret_cast<const T*>(slot(stage, 2)) + c);
#pragma unroll
                for (int i = 0; i < V::N; ++i) {
                    const float xh = to_float(vx.v[i]) * rs;
                    const float g = (to_float(vw[k].v[i]) * to_float(vdy.v[i]) - xh * dot) * rs;
                    vd.v[i] = from_float<T>(to_float(vd.v[i]) + g);
                    tmax = fmaxf(tmax, fabsf(to_float(vd.v[i])));
                }
                vd.store(dx + c);
            }
        }
        if (++stage == STAGES) { stage = 0; phase ^= 1u; }
    }
    // Set before the barrier of a row, so the same for all threads here
    const bool lost = *static_cast<volatile uint32_t*>(&gave_up) != 0;
    if (lost) {
        tmax = 0.f;
        if (threadIdx.x == 0 && status) atomicOr(status, static_cast<unsigned int>(sm100::kErrOther));
        give_up_rows<STAGES>(dinp, rows, C, sm100::smem_u32(full), first_lost);
    }
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
        const int c = (k * NORM_THREADS + threadIdx.x) * V::N;
        if (c < C) {
#pragma unroll
            for (int i = 0; i < V::N; ++i) dw_partial[static_cast<long long>(blockIdx.x) * C + c + i] = lost ? NAN : dw[k][i];
        }
    }
    block_absmax_commit(absmax_out, tmax, scratch);
}

// Column sums of the per-CTA partial rows.  A CTA owns 32 columns; its 16 thread rows walk the partial rows with a stride
// of 16 (28 loads per thread for 444 partial rows instead of 444 dependent loads in one thread) and are summed through
// shared memory in a fixed order, so the result does not depend on the schedule.
constexpr int RED_COLS = 32, RED_GROUPS = 16;
template <typename T>
__global__ void __launch_bounds__(RED_COLS * RED_GROUPS)
rmsnorm_bwd_reduce_kernel(T* __restrict__ dweight, const float* __restrict__ dw_partial, int nparts, int C, int accumulate) {
    grid_wait();
    const int bx = after_wait(blockIdx.x), tx = after_wait(threadIdx.x);
    __shared__ float part[RED_GROUPS][RED_COLS];
    const int x = tx % RED_COLS, y = tx / RED_COLS;
    const int c = bx * RED_COLS + x;
    float s = 0.f;
    if (c < C) {
#pragma unroll 4
        for (int p = y; p < nparts; p += RED_GROUPS) s += dw_partial[static_cast<long long>(p) * C + c];
    }
    part[y][x] = s;
    __syncthreads();
    if (y == 0 && c < C) {
        float t = 0.f;
#pragma unroll
        for (int g = 0; g < RED_GROUPS; ++g) t += part[g][x];
        if (accumulate) t += to_float(dweight[c]);
        dweight[c] = from_float<T>(t);
    }
}

template <typename T>
int launch_fwd(void* residual_out, void* y_out, void* q_out, float* rstd, const void* a, const void* b, const void* w,
               float eps, int rows, int C, float* absmax, const float* known_absmax, float* q_scale, cudaStream_t s) {
    using V = Vec16<T>;
    if (C % V::N) return -1;
#define LAUNCH(KERNEL, THREADS)                                                                                                \
    KERNEL<<<rows, THREADS, 0, s>>>(static_cast<T*>(residual_out), static_cast<T*>(y_out), static_cast<e4m3*>(q_out), rstd,   \
                                    static_cast<const T*>(a), static_cast<const T*>(b), static_cast<const T*>(w), eps, C,     \
                                    absmax, known_absmax, q_scale)
#define LAUNCH_VPT(VPT, THREADS) LAUNCH((rmsnorm_fwd_reg_kernel<T, THREADS, VPT>), THREADS)
    const int vecs = C / V::N;
    // Short rows: 64 threads a row put the most rows on an SM.  With few rows that only makes every row slower, so 256 threads take them
    // while one wave of such CTAs (8 per SM) holds all rows.  With 8 vectors a thread the registers leave room for 12 rows of 64 threads
    // on an SM: in the second and third wave of those, 256 threads are faster too.  bf16, with / without the residual add, us for 64
    // and for 256 threads: 1 x 4096 5.14 / 4.87 and 2.65 / 2.73, 300 x 3584 5.16 / 4.83 and 3.35 / 3.15, 1000 x 1536 4.17 / 3.72 and 3.77 /
    // 3.42, 1200 x 1536 4.11 / 3.83 and 4.06 / 3.92, 4096 x 1536 8.1 / 6.9 and 9.7 / 8.6;  2000 x 4096 11.9 / 9.7 and 9.6 / 7.7, 4096 x 4096
    // 23.9 / 15.3 and 20.9 / 14.6, 16384 x 4096 85.3 / 50.6 and 82.6 / 51.7.
    constexpr int kWave256 = 8 * 148, kWave64 = 12 * 148;
    const bool few = rows <= kWave256 || (vecs > 7 * 64 && rows > kWave64 && rows <= 4096);
    // 7 vectors a thread have an instance of their own: 16384 x 3584 without a residual add 42.7 us, 45.9 with the one for 8.
    if (vecs <= 256 && few) LAUNCH_VPT(1, 256);
    else if (vecs <= 512 && few) LAUNCH_VPT(2, 256);
    else if (vecs <= 2 * 64) LAUNCH_VPT(2, 64);
    else if (vecs <= 4 * 64) LAUNCH_VPT(4, 64);
    else if (vecs <= 6 * 64) LAUNCH_VPT(6, 64);
    else if (vecs <= 7 * 64) LAUNCH_VPT(7, 64);
    else if (vecs <= 8 * 64) LAUNCH_VPT(8, 64);
    else if (vecs <= 4 * 256) LAUNCH_VPT(4, 256);
    else if (vecs <= 6 * 256) LAUNCH_VPT(6, 256);
    else if (vecs <= 8 * 256) LAUNCH_VPT(8, 256);
    else LAUNCH(rmsnorm_fwd_kernel<T>, NORM_THREADS);
#undef LAUNCH_VPT
#undef LAUNCH
    return LLMQ_LAUNCH_CHECK();
}

template <typename T, int VPT, int STAGES, int CTAS>
int launch_bwd_ring(T* dinp, float* scratch, const T* dout, const T* inp, const T* w, const float* rstd, int rows, int C, float* absmax, int blocks, unsigned int* status, cudaStream_t s) {
    static bool attr_set[64] = {};          // per device
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_set[dev & 63]) {
        cudaError_t e = cudaFuncSetAttribute(rmsnorm_bwd_ring_kernel<T, VPT, STAGES, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGES * 3 * VPT * NORM_THREADS * 16);
        if (e != cudaSuccess) return static_cast<int>(e);
        attr_set[dev & 63] = true;
    }
    rmsnorm_bwd_ring_kernel<T, VPT, STAGES, CTAS><<<blocks, NORM_THREADS, STAGES * 3 * C * sizeof(T), s>>>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax, status);
    return LLMQ_LAUNCH_CHECK();
}

template <typename T>
int launch_bwd(void* dinp_, void* dweight, float* scratch, const void* dout_, const void* inp_, const void* w_,
               const float* rstd, int rows, int C, float* absmax, int accumulate_dw, int num_blocks, unsigned int* status, cudaStream_t s) {
    using V = Vec16<T>;
    if (C % V::N) return -1;
    const int vecs = ceil_div_i(C / V::N, NORM_THREADS);
    // Blocks: few rows go to few blocks, whose rows follow one another through the ring; every block costs a partial row that the second kernel has to read.
    // us with one / two / three blocks per SM:  444 x 3072 8.6 / 9.8 / 11.9,  444 x 4096 9.8 / 11.4 / 13.9,  888 x 4096
    // 14.4 / 16.0 / 18.2,  888 x 1536 8.3 / 8.6 / 9.3,  1200 x 3072 15.0 / 14.9 / 16.4,  2500 x 4096 25.9 / 24.0 / 26.3,  4000 x 3072 31.8 / 26.5 / 25.8,
    // 8000 x 2048 49 / 35 / 33;  three or four vectors a thread, of which two blocks reside: 888 x 5120 17.6 / 18.1 / 22.7,  8000 x 5120 90 / 66 / 79.
    // Rows of up to 1024 columns keep three: their sums over the rows, and with them the weight gradients, keep their order.
    if (sizeof(T) == 2 && C > 1024 && C <= 4 * NORM_THREADS * V::N) {
        const int sms = device_sms();
        const int most = (rows <= 7 * sms ? 1 : vecs > 2 || rows <= 24 * sms ? 2 : 3) * sms;
        if (num_blocks > most) num_blocks = most;
    }
    if (num_blocks > rows) num_blocks = rows;
    T* dinp = static_cast<T*>(dinp_);
    const T *dout = static_cast<const T*>(dout_), *inp = static_cast<const T*>(inp_), *w = static_cast<const T*>(w_);
    int rc;
    // stages and CTAs per SM: as much shared memory as fits
    // Rows of one vector a thread.  Blocks with one or two of them have nothing to fetch ahead, and setting up the ring costs 0.3 us: us with / without it, bf16: 20 x 896 4.2 / 3.9,
    // 113 x 1536 5.7 / 5.2, 888 x 256 7.3 / 7.0.  Short rows spend a turn of the ring on its barriers and its one issuing thread, which shows where the operands lie in the L2 already.  bf16
    // rows of up to 768 channels are copied by their threads, which is as fast from HBM until the operands are larger than the L2; us, rows by bulk copies / by their threads, from L2
    // and from HBM: 4096 x 256 12.1 / 10.9, 16384 x 256 28.6 / 24.5 and 29.4 / 29.9, 8192 x 512 19.0 / 16.9 and 19.8 / 20.2, 8192 x 768 20.8 / 19.1 and 21.8 / 21.8;  65536 x 256 (101 MB)
    // 99.2 / 99.9 and 99.2 / 101.8;  8192 x 896 20.8 / 19.6 and 22.2 / 23.0, 4096 x 896 14.0 / 13.6 and 15.3 / 16.1.  fp32 rows, from L2 and from HBM, by bulk copies / in
    // registers: 2000 x 1024 10.8 / 9.9 and 13.5 / 13.8, 3000 x 768 (28 MB) 11.5 / 10.5 and 14.2 / 15.4, 4096 x 256 11.3 / 10.4 and 12.0 / 14.5;  beyond 32 MB, where they
    // rarely lie in the L2 as a whole, 8192 x 512 (50 MB) 16.9 / 15.1 and 18.8 / 24.6, 8192 x 768 (75 MB) 18.3 / 20.5 and 23.6 / 27.6.
    const long long bytes = 3ll * rows * C * static_cast<long long>(sizeof(T));
    const bool in_registers = rows <= 2 * num_blocks || (sizeof(T) == 4 && bytes <= (32ll << 20)), by_threads = C <= 768 && bytes <= (96ll << 20);
    if (vecs <= 1 && (in_registers || (sizeof(T) == 2 && by_threads))) {
        constexpr int stages = sizeof(T) == 2 ? 4 : 0;       // 18 KB at most
        if (in_registers) rmsnorm_bwd_reg_kernel<T, 1, 0><<<num_blocks, NORM_THREADS, 0, s>>>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax);
        else rmsnorm_bwd_reg_kernel<T, 1, stages><<<num_blocks, NORM_THREADS, stages * 3 * C * sizeof(T), s>>>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax);
        rc = LLMQ_LAUNCH_CHECK();
    }
    else if (vecs <= 1) rc = launch_bwd_ring<T, 1, 4, 3>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax, num_blocks, status, s);
    else if (vecs <= 4) {
        if constexpr (sizeof(T) == 2) {
            if (vecs <= 2) rc = launch_bwd_ring<T, 2, 3, 3>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax, num_blocks, status, s);
            else           rc = launch_bwd_ring<T, 4, 2, 2>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax, num_blocks, status, s);
        } else {
            if (vecs <= 2) rmsnorm_bwd_reg_kernel<T, 2, 0><<<num_blocks, NORM_THREADS, 0, s>>>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax);
            else           rmsnorm_bwd_reg_kernel<T, 4, 0><<<num_blocks, NORM_THREADS, 0, s>>>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax);
            rc = LLMQ_LAUNCH_CHECK();
        }
    }
    else if (vecs <= 8) {
        rmsnorm_bwd_kernel<T, 8><<<num_blocks, NORM_THREADS, 0, s>>>(dinp, scratch, dout, inp, w, rstd, rows, C, absmax);
        rc = LLMQ_LAUNCH_CHECK();
    } else return -2;
    if (rc) return rc;
    launch_chained(rmsnorm_bwd_reduce_kernel<T>, ceil_div_i(C, RED_COLS), RED_COLS * RED_GROUPS, 0, s, static_cast<T*>(dweight), scratch, num_blocks, C, accumulate_dw);
    return LLMQ_LAUNCH_CHECK();
}

}  // namespace

extern "C" int llmq_rmsnorm_forward(void* residual_out, void* y_out, void* q_out, float* rstd, const void* in_a,
                                    const void* in_b, const void* weight, float eps, int rows, int C, int dtype,
                                    float* absmax, const float* known_absmax, float* q_scale, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (dtype == 0) return launch_fwd<bf16>(residual_out, y_out, q_out, rstd, in_a, in_b, weight, eps, rows, C, absmax, known_absmax, q_scale, stream);
    if (dtype == 3) return launch_fwd<float>(residual_out, y_out, q_out, rstd, in_a, in_b, weight, eps, rows, C, absmax, known_absmax, q_scale, stream);
    return -10;
}

// scratch must hold num_blocks * C floats.  status: optional device word that takes a bit when a wait of the kernel runs out.
extern "C" int llmq_rmsnorm_backward(void* dinp, void* dweight, float* scratch, const void* dout, const void* inp,
                                     const void* weight, const float* rstd, int rows, int C, int dtype, float* absmax,
                                     int accumulate_dweight, int num_blocks, unsigned int* status, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (dtype == 0) return launch_bwd<bf16>(dinp, dweight, scratch, dout, inp, weight, rstd, rows, C, absmax, accumulate_dweight, num_blocks, status, stream);
    if (dtype == 3) return launch_bwd<float>(dinp, dweight, scratch, dout, inp, weight, rstd, rows, C, absmax, accumulate_dweight, num_blocks, status, stream);
    return -10;
}

// ------------------------------------------------------------------------------------------------
// RMSNorm backward for callers that must not allocate (see noalloc.h).
//
// The weight-gradient partials live in a file-scope device array instead of a caller-provided buffer.
// Every GPU that loads this library keeps the array resident until the process exits.
#include "noalloc.h"
#include <mutex>

static __device__ __align__(256) float g_noalloc_norm_scratch[LLMQ_NOALLOC_SCRATCH_FLOATS];

namespace {
std::mutex g_noalloc_mutex;
float* g_noalloc_scratch_ptr[64] = {};     // device address of the array, per device ordinal
}  // namespace

extern "C" int llmq_rmsnorm_backward_noalloc(void* dinp, void* dweight, const void* dout, const void* inp,
                                             const void* weight, const float* rstd, int rows, int C, int dtype,
                                             float* absmax, int accumulate_dweight, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (C <= 0 || C > LLMQ_NOALLOC_MAX_C) return LLMQ_NOALLOC_ERR_TOO_LARGE;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    if (dev < 0 || dev >= 64) return LLMQ_NOALLOC_ERR_DEVICE;
    float* scratch = nullptr;
    int sms = 0;
    {
        // One-time set-up per device, with that device current.  In host code the array's name is only a
        // handle for the runtime; the address a kernel can use comes from cudaGetSymbolAddress.
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_scratch_ptr[dev]) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_norm_scratch);
            if (e != cudaSuccess) return static_cast<int>(e);
            g_noalloc_scratch_ptr[dev] = static_cast<float*>(p);
        }
        scratch = g_noalloc_scratch_ptr[dev];
    }
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    // as many row-walking CTAs as the array can hold partial rows for, at most two per SM
    long long blocks = 2LL * sms;
    const long long fit = LLMQ_NOALLOC_SCRATCH_FLOATS / C;
    if (blocks > fit) blocks = fit;
    if (blocks < 1) return LLMQ_NOALLOC_ERR_TOO_LARGE;
    if (dtype == 0) return launch_bwd<bf16>(dinp, dweight, scratch, dout, inp, weight, rstd, rows, C, absmax, accumulate_dweight, static_cast<int>(blocks), nullptr, stream);
    if (dtype == 3) return launch_bwd<float>(dinp, dweight, scratch, dout, inp, weight, rstd, rows, C, absmax, accumulate_dweight, static_cast<int>(blocks), nullptr, stream);
    return -10;
}
