// Persistent, warp-specialised tcgen05 GEMM for sm_100a.
//
//   C[M,N] (+)= alpha * A * B^T (+ bias[N]),   fp32 accumulation in tensor memory.
//
// Operands are bf16, 8-bit floats (e4m3 / e5m2) or - one-CTA kernel only - fp32 multiplied as tf32 (the GEMMs of an
// fp32 model: src/kernels/matmul.cpp:46-153 of the reference runs those through cuBLASLt).  Each operand may be stored K-major
// (row = M/N index, K contiguous) or MN-major (row = K index, M/N contiguous); the MN-major
// form is what lets the backward GEMMs (dX = dY * W, dW = dY^T * X) read the very same tensors
// as the forward pass without any transpose kernel.  alpha is the product of two optional
// per-tensor dequantisation factors read from device memory, so no host synchronisation is
// needed between the abs-max reduction and the GEMM.
//
// Replaces the cuBLASLt wrapper and the mma.sync kernel of the reference
// (src/kernels/matmul.cpp:46-153, src/kernels/gemm_mma.cu:21-291).
//
// Structure (192 threads per CTA, one CTA per SM):
//   warp 0     TMA producer: fills a 4-stage ring of 128x(128 B) A and 256x(128 B) B tiles (6 stages with 128-wide B tiles)
//   warp 1     MMA issuer (one elected lane): 4 tcgen05.mma per stage into one of two
//              128x256 (or 128x128) fp32 accumulators in TMEM, tcgen05.commit to free the stage
//   warps 2-5  epilogue: tcgen05.ld the finished accumulator (while the other one is being
//              computed), scale, add bias, optionally add the previous C, track abs-max, store
// Outputs with few tiles and a long K cut the K loop; the parts of a tile are summed by the CTAs of a cluster or by a second kernel.
#include <type_traits>
#include "ptx_sm100.cuh"
#include "api.h"
#include "common.cuh"
#include "gemm_common.cuh"

using namespace sm100;

namespace {

constexpr int BM = 128;
constexpr int ROW_BYTES = 128;            // one swizzle row
constexpr int A_STAGE_BYTES = BM * ROW_BYTES;   // 16 KiB
constexpr int NUM_THREADS = 192;
// Tile width BN is 256, or 128 for outputs with so few tiles that half the SMs would idle.  Two accumulators of BN columns.
template <int BN> struct Tile {
    static constexpr int STAGES = BN == 256 ? 4 : 6;
    static constexpr int B_STAGE_BYTES = BN * ROW_BYTES;
    static constexpr int STAGE_BYTES = A_STAGE_BYTES + B_STAGE_BYTES;
    static constexpr int TMEM_COLS = 2 * BN;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
    // outputs that are added to: two blocks of previous values of C per epilogue warp behind the barriers.  Only then, since a kernel that is launched
    // early starts sooner the less shared memory is taken (the second kernel of a cut K loop: 1152 x 896 x 4096 23.4 us, 22.5 without).
    static constexpr int OLD_OFFSET = STAGES * STAGE_BYTES + 256;
    static constexpr int SMEM_BYTES_ADDED = SMEM_BYTES + 4 * 2 * OLD_BLOCK_BYTES;
};


__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
    // Grouped rasterisation: 16 row tiles share every column tile while it is hot in L2.
    constexpr int G = 16;
    int per_group = G * tiles_n;
    int group = t / per_group;
    int first_m = group * G;
    int gsz = min(tiles_m - first_m, G);
    int r = t - group * per_group;
    tm = first_m + (r % gsz);
    tn = r / gsz;
}

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// Split K, the parts of a tile in one cluster: every CTA has put its fp32 accumulator [128][BN] at the start of its shared memory (16-byte pieces, piece index ^
// (row % 8)).  CTA `part` adds up its share of the rows of all of them, in the order of the parts like the two-kernel form (same bits), and writes the
// result.  What it saves is the latency of a second kernel and of parts x M x N floats through the L2; see the rule in gemm_impl.
template <int BN>
__device__ __forceinline__ void cluster_reduce(const GemmParams& p, uint32_t smem_base, int tm, int tn, int part, int parts, float alpha, float& tmax) {
    // only the rows and columns that exist, the pieces of a row rounded up to 8, 16, 32 or 64 (208 x 32 x 1216: all of them 9.7 us, these 7.6, a second kernel 7.8;  16 x 3168 x 3584 11.8, 10.0, 11.3)
    const int in_m = min(BM, p.M - tm * BM), in_n = min(BN, p.N - tn * BN);
    const int shift = in_n > 128 ? 6 : in_n > 64 ? 5 : in_n > 32 ? 4 : 3;
    const int row0 = in_m * part / parts, total = (in_m * (part + 1) / parts - row0) << shift;
    uint32_t base[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) base[q] = map_to_cta(smem_base, q < parts ? q : 0);
    // four pieces per thread at a time: all their loads, from the other CTAs and of the old values, are under way together
    constexpr int U = 4;
    for (int i0 = after_wait(threadIdx.x); i0 < total; i0 += U * NUM_THREADS) {
        uint4 old[U];
        float4 x[U][8];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * NUM_THREADS, r = row0 + (i >> shift), piece = i & ((1 << shift) - 1), row = tm * BM + r, col = tn * BN + piece * 4;
            const bool inside = i < total && col < p.N;
            if (p.accumulate && inside) {
                if (p.c_dtype == 0) {
                    const uint2 o = *reinterpret_cast<const uint2*>(static_cast<bf16*>(p.C) + row * p.ldc + col);
                    old[u].x = o.x; old[u].y = o.y;            // as they are: what is computed from a load here would wait for it
                } else {
                    old[u] = *reinterpret_cast<const uint4*>(static_cast<float*>(p.C) + row * p.ldc + col);
                }
            }
            const uint32_t at = r * (BN * 4) + ((piece ^ (r & 7)) << 4);
#pragma unroll
            for (int q = 0; q < 8; ++q) if (q < parts && inside) x[u][q] = ld_cluster_f32x4(base[q] + at);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * NUM_THREADS, r = row0 + (i >> shift), piece = i & ((1 << shift) - 1), row = tm * BM + r, col = tn * BN + piece * 4;
            if (i >= total || col >= p.N) continue;
            float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int q = 0; q < 8; ++q) if (q < parts) { v[0] += x[u][q].x; v[1] += x[u][q].y; v[2] += x[u][q].z; v[3] += x[u][q].w; }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] *= alpha;
                if (p.bias) v[k] += p.bias_dtype == 0 ? __bfloat162float(static_cast<const bf16*>(p.bias)[col + k]) : static_cast<const float*>(p.bias)[col + k];
            }
            if (p.accumulate && p.c_dtype == 0) {
                v[0] += __uint_as_float(old[u].x << 16); v[1] += __uint_as_float(old[u].x & 0xffff0000u);
                v[2] += __uint_as_float(old[u].y << 16); v[3] += __uint_as_float(old[u].y & 0xffff0000u);
            } else if (p.accumulate) {
                v[0] += __uint_as_float(old[u].x); v[1] += __uint_as_float(old[u].y); v[2] += __uint_as_float(old[u].z); v[3] += __uint_as_float(old[u].w);
            }
            if (p.c_dtype == 0) {
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
                *reinterpret_cast<uint2*>(static_cast<bf16*>(p.C) + row * p.ldc + col) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
            } else {
                *reinterpret_cast<float4*>(static_cast<float*>(p.C) + row * p.ldc + col) = make_float4(v[0], v[1], v[2], v[3]);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) tmax = fmaxf(tmax, fabsf(v[k]));
        }
    }
}

// Kind: MMA kind of ptx_sm100.cuh's mma_issue (0 bf16, 1 8-bit floats, 2 tf32 on fp32 operands).
// Mode: kCluster, the CTAs of a cluster are the K parts of one tile (grid = tiles x parts, one work item per CTA); kAdded, a bf16 C that is added to, in
// whole sectors (GemmParams::c_sectors);  kAddedNarrow, the same with up to 32 columns, whose old values every lane loads for its row.
enum { kPlain, kCluster, kAdded, kAddedNarrow };
template <int Kind, int BN, int Mode>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const GemmParams p) {
    constexpr int STAGES = Tile<BN>::STAGES, B_STAGE_BYTES = Tile<BN>::B_STAGE_BYTES, STAGE_BYTES = Tile<BN>::STAGE_BYTES;
    constexpr int TMEM_COLS = Tile<BN>::TMEM_COLS;
    constexpr bool Cluster = Mode == kCluster, Added = Mode == kAdded;
    extern __shared__ uint8_t smem_raw[];
    // 128B-swizzled tiles must start on a 1024-byte boundary
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
    // bars[0..S) full, [S..2S) empty, [2S..2S+2) tmem_full, [2S+2..2S+4) tmem_empty
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);      // uniform, and known to be
    const int lane = threadIdx.x & 31;
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (STAGES + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * STAGES + 2 + a); };

    const int bk = ROW_BYTES / p.elem_bytes;          // K elements per stage (K-major row)
    const int k_iters = (p.K + bk - 1) / bk;
    const int tiles_m = (p.M + BM - 1) / BM;
    const int tiles_n = (p.N + BN - 1) / BN;
    const int splits = p.k_splits > 1 ? p.k_splits : 1;
    const int k_per_split = (k_iters + splits - 1) / splits;
    const int num_tiles = tiles_m * tiles_n * splits;           // work items: (tile, K split)

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(tfull_bar(a), 1); mbar_init(tempty_bar(a), 128); }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    grid_release();
    grid_wait();

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        // the whole warp runs the loop, the elected lane issues (see gemm_tcgen05_2cta.cu)
        {
            const bool leader = elect_one();
            if (leader) { tma_prefetch_desc(&tmap_a); tma_prefetch_desc(&tmap_b); }
            int stage = 0; uint32_t phase = 0;
            const int mn_chunk = ROW_BYTES / p.elem_bytes;     // M/N elements per 128-byte row (MN-major)
            bool ok = true;
            for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
                int tm, tn; tile_coords(t / splits, tiles_m, tiles_n, tm, tn);
                const int k_begin = (t % splits) * k_per_split, k_end = min(k_iters, k_begin + k_per_split);
                for (int k = k_begin; k < k_end; ++k) {
                    if (!mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag)) { if (leader) atomicOr(p.status, kErrEmptyWait); ok = false; break; }
                    uint32_t sa = smem_base + stage * STAGE_BYTES;
                    uint32_t sb = sa + A_STAGE_BYTES;
                    if (leader) {
                        mbar_expect_tx(full_bar(stage), STAGE_BYTES);
                        if (!p.a_mn_major) {
                            tma_load_2d(sa, &tmap_a, full_bar(stage), k * bk, tm * BM);
                        } else if (p.a_box3) {
                            tma_load_3d(sa, &tmap_a, full_bar(stage), 0, k * bk, tm * (BM / mn_chunk));
                        } else {
                            // boxes of [bk K-rows][128 B of M]; BM*elem_bytes/128 boxes side by side
                            int nbox = BM * p.elem_bytes / ROW_BYTES;
                            for (int b = 0; b < nbox; ++b)
                                tma_load_2d(sa + b * (A_STAGE_BYTES / nbox), &tmap_a, full_bar(stage), tm * BM + b * mn_chunk, k * bk);
                        }
                        if (!p.b_mn_major) {
                            tma_load_2d(sb, &tmap_b, full_bar(stage), k * bk, tn * BN);
                        } else if (p.b_box3) {
                            tma_load_3d(sb, &tmap_b, full_bar(stage), 0, k * bk, tn * (BN / mn_chunk));
                        } else {
                            int nbox = BN * p.elem_bytes / ROW_BYTES;
                            for (int b = 0; b < nbox; ++b)
                                tma_load_2d(sb + b * (B_STAGE_BYTES / nbox), &tmap_b, full_bar(stage), tn * BN + b * mn_chunk, k * bk);
                        }
                    }
                    __syncwarp();
                    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        {
            const bool leader = elect_one();
            const uint32_t idesc = make_instr_desc(p.a_fmt, p.b_fmt, p.a_mn_major, p.b_mn_major, BM, BN);
            // K-major: 8-row groups are 1024 B apart, a K step of one MMA is 32 B inside the row.
            // MN-major: a K step of one MMA is (mma_k rows * 128 B); next 128 B chunk along M/N
            //           is one whole box (bk rows * 128 B) further on.
            const int mma_k = 32 / p.elem_bytes;
            const uint32_t box_bytes = static_cast<uint32_t>(bk) * ROW_BYTES;
            const uint32_t a_step = p.a_mn_major ? mma_k * ROW_BYTES : 32;
            const uint32_t b_step = p.b_mn_major ? mma_k * ROW_BYTES : 32;
            const uint32_t a_lbo = p.a_mn_major ? box_bytes : 16;
            const uint32_t b_lbo = p.b_mn_major ? box_bytes : 16;
            const uint32_t a_hi = desc_hi(1024), b_hi = desc_hi(1024);
            const uint32_t a_lo0 = desc_lo(smem_base, a_lbo), b_lo0 = desc_lo(smem_base + A_STAGE_BYTES, b_lbo);
            const uint32_t a_inc = a_step >> 4, b_inc = b_step >> 4;
            int stage = 0; uint32_t phase = 0;
            int acc = 0; uint32_t acc_phase = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < num_tiles && ok; t += gridDim.x) {
                if (!mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, abort_flag)) { if (leader) atomicOr(p.status, kErrTmemEmpty); ok = false; break; }
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + acc * BN;
                const int k_begin = (t % splits) * k_per_split, k_end = min(k_iters, k_begin + k_per_split);
                for (int k = k_begin; k < k_end; ++k) {
                    if (!mbar_wait_warp(full_bar(stage), phase, abort_flag)) { if (leader) atomicOr(p.status, kErrFullWait); ok = false; break; }
                    tc_fence_after_sync();
                    const uint32_t alo = a_lo0 + stage * (STAGE_BYTES >> 4);
                    const uint32_t blo = b_lo0 + stage * (STAGE_BYTES >> 4);
                    if (leader) {
                        mma_issue<Kind, false>(d_tmem, alo, a_hi, blo, b_hi, idesc, k > k_begin ? 1u : 0u);
                        mma_issue<Kind, false>(d_tmem, alo + a_inc, a_hi, blo + b_inc, b_hi, idesc, 1u);
                        mma_issue<Kind, false>(d_tmem, alo + 2 * a_inc, a_hi, blo + 2 * b_inc, b_hi, idesc, 1u);
                        mma_issue<Kind, false>(d_tmem, alo + 3 * a_inc, a_hi, blo + 3 * b_inc, b_hi, idesc, 1u);
                        mma_commit(empty_bar(stage));          // stage reusable once these MMAs have read it
                    }
                    __syncwarp();
                    if (++stage == STAGES) { stage = 0; phase ^= 1u; }
                }
                if (!ok) break;
                if (leader) mma_commit(tfull_bar(acc));    // accumulator complete
                __syncwarp();
                if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (4 warps)
        const int q = warp & 3;                            // TMEM lane quarter this warp may access
        float alpha = p.alpha;
        if (p.scale_a) alpha *= *p.scale_a;
        if (p.scale_b) alpha *= *p.scale_b;
        float tmax = 0.f;
        int acc = 0; uint32_t acc_phase = 0;
        bool ok = true;
        auto origin = [&](int t, int& row, int& col) {
            int tm, tn; tile_coords(t, tiles_m, tiles_n, tm, tn);
            row = tm * BM + q * 32;
            col = tn * BN;
        };
        std::conditional_t<Added, OldBlocks<decltype(origin)>, NoOldBlocks> old(p, origin, smem + Tile<BN>::OLD_OFFSET + q * 2 * OLD_BLOCK_BYTES, after_wait(blockIdx.x),
                                                                                gridDim.x, num_tiles, BN);
        for (int t = after_wait(blockIdx.x); t < num_tiles && ok; t += gridDim.x) {
            int tm, tn; tile_coords(t / splits, tiles_m, tiles_n, tm, tn);
            if (!mbar_wait(tfull_bar(acc), acc_phase, abort_flag)) { if (lane == 0) atomicOr(p.status, kErrTmemFull); ok = false; break; }
            tc_fence_after_sync();
            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BN;
            if constexpr (Mode == kAddedNarrow) epilogue_rows_sectors<true>(p, t_row, tm * BM + q * 32 + lane, tn * BN, BN, alpha, tmax);
            else if constexpr (Added) epilogue_rows_added(p, t_row, tm * BM + q * 32 + lane, tn * BN, BN, alpha, tmax, old);
            else if constexpr (Cluster) {
                uint8_t* const mine = smem + (q * 32 + lane) * (BN * 4);
                const int in_n = min(BN, p.N - tn * BN);
#pragma unroll 1
                for (int c = 0; c < in_n; c += 32) {
                    uint32_t r[32];
                    tmem_ld_32x32b_x32(t_row + c, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        *reinterpret_cast<uint4*>(mine + (((c / 4 + i) ^ (lane & 7)) << 4)) = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
                }
            }
            else if (splits > 1) epilogue_rows_partial(p, t_row, tm * BM + q * 32 + lane, tn * BN, BN, t % splits);
            else             epilogue_rows(p, t_row, tm * BM + q * 32 + lane, tn * BN, BN, alpha, tmax);
            tc_fence_before_sync();
            mbar_arrive(tempty_bar(acc));                  // 128 arrivals release the accumulator
            if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        }
        if constexpr (Added) old.drain();
        if (!Cluster && p.absmax_out) {
            tmax = warp_reduce_max(tmax);
            if (lane == 0 && tmax > 0.f) atomic_max_float(p.absmax_out, tmax);
        }
    }
    if constexpr (Cluster) {
        // Every CTA of a cluster gets here, also one that gave up on a wait (the status word says so and the output is void)
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        float alpha = p.alpha, tmax = 0.f;
        if (p.scale_a) alpha *= *p.scale_a;
        if (p.scale_b) alpha *= *p.scale_b;
        int tm, tn; tile_coords(after_wait(blockIdx.x) / splits, tiles_m, tiles_n, tm, tn);
        cluster_reduce<BN>(p, smem_base, tm, tn, blockIdx.x % splits, splits, alpha, tmax);
        if (p.absmax_out) {
            tmax = warp_reduce_max(tmax);
            if (lane == 0 && tmax > 0.f) atomic_max_float(p.absmax_out, tmax);
        }
        __syncwarp();
        cluster_arrive();                                      // the others may still read this CTA's accumulator
        cluster_wait();
    }

    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Sum of the split-K parts + the normal epilogue (alpha, bias, accumulate, bf16 / fp32 store, abs-max).
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const GemmParams p, float alpha_host) {
    grid_wait();
    __shared__ float scratch[32];
    float alpha = alpha_host;
    if (p.scale_a) alpha *= *p.scale_a;
    if (p.scale_b) alpha *= *p.scale_b;
    const long long total = static_cast<long long>(p.M) * p.N;
    float tmax = 0.f;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += static_cast<long long>(gridDim.x) * 256) {
        const int col = static_cast<int>(i % p.N);
        const long long row = i / p.N;
        float v = 0.f;
        for (int s = 0; s < p.k_splits; ++s) v += p.partial[static_cast<long long>(s) * total + i];
        v *= alpha;
        if (p.bias) v += p.bias_dtype == 0 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col]) : static_cast<const float*>(p.bias)[col];
        if (p.c_dtype == 0) {
            __nv_bfloat16* c = static_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col;
            if (p.accumulate) v += __bfloat162float(*c);
            *c = __float2bfloat16_rn(v);
        } else {
            float* c = static_cast<float*>(p.C) + row * p.ldc + col;
            if (p.accumulate) v += *c;
            *c = v;
        }
        tmax = fmaxf(tmax, fabsf(v));
    }
    if (p.absmax_out) block_absmax_commit(p.absmax_out, tmax, scratch);
}

// The same, four columns per thread, for bf16 / fp32 outputs with rows of whole 16-byte partial vectors (N and ldc multiples of
// 4, aligned C): 16-byte loads of the parts, and a multiply instead of a 64-bit division per element.  1152 x 896 from two parts:
// 3.8 us against 14.
__global__ void __launch_bounds__(256) splitk_reduce_vec_kernel(const GemmParams p, float alpha_host, const FastDiv fd) {
    grid_wait();
    __shared__ float scratch[32];
    float alpha = alpha_host;
    if (p.scale_a) alpha *= *p.scale_a;
    if (p.scale_b) alpha *= *p.scale_b;
    const long long total = static_cast<long long>(p.M) * p.N;
    const uint32_t nvec = static_cast<uint32_t>(total / 4);
    float tmax = 0.f;
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < nvec; i += gridDim.x * 256u) {
        uint32_t row, cv;
        fd.divmod(i, row, cv);
        const int col = static_cast<int>(cv) * 4;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < p.k_splits; ++s) {
            const float4 q = *reinterpret_cast<const float4*>(p.partial + static_cast<long long>(s) * total + static_cast<long long>(i) * 4);
            v[0] += q.x; v[1] += q.y; v[2] += q.z; v[3] += q.w;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] *= alpha;
            if (p.bias) v[k] += p.bias_dtype == 0 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.bias)[col + k]) : static_cast<const float*>(p.bias)[col + k];
        }
        if (p.c_dtype == 0) {
            uint2* c = reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(p.C) + row * p.ldc + col);
            if (p.accumulate) {
                const uint2 old = *c;
                v[0] += __uint_as_float(old.x << 16); v[1] += __uint_as_float(old.x & 0xffff0000u);
                v[2] += __uint_as_float(old.y << 16); v[3] += __uint_as_float(old.y & 0xffff0000u);
            }
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
            *c = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        } else {
            float4* c = reinterpret_cast<float4*>(static_cast<float*>(p.C) + row * p.ldc + col);
            if (p.accumulate) { const float4 old = *c; v[0] += old.x; v[1] += old.y; v[2] += old.z; v[3] += old.w; }
            *c = make_float4(v[0], v[1], v[2], v[3]);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) tmax = fmaxf(tmax, fabsf(v[k]));
    }
    if (p.absmax_out) block_absmax_commit(p.absmax_out, tmax, scratch);
}

// Launches the one-CTA kernel for `items` (tile, K part) pairs: `cluster` = the parts of a tile in one cluster
template <int Kind, int BN>
int launch_one_cta(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, int items, bool cluster, int num_sms, cudaStream_t stream) {
    static bool attr_set[64] = {};          // the attribute is per device
    constexpr int smem = Tile<BN>::SMEM_BYTES, smem_added = Tile<BN>::SMEM_BYTES_ADDED;
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_set[dev & 63]) {
        const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
        cudaError_t e = cudaFuncSetAttribute(gemm_tcgen05_kernel<Kind, BN, kPlain>, at, smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_tcgen05_kernel<Kind, BN, kCluster>, at, smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_tcgen05_kernel<Kind, BN, kAdded>, at, smem_added);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(gemm_tcgen05_kernel<Kind, BN, kAddedNarrow>, at, smem);
        if (e != cudaSuccess) return static_cast<int>(e);
        attr_set[dev & 63] = true;
    }
    const int grid = items < num_sms ? items : num_sms;
    if (cluster) launch_chained_cluster(gemm_tcgen05_kernel<Kind, BN, kCluster>, items, NUM_THREADS, smem, stream, p.k_splits, ta, tb, p);
    // up to 32 columns, added to, us with blocks of old values / this way: 32 x 16 x 256 3.35 / 3.14, 8192 x 16 x 64 3.18 / 3.03
    else if (p.accumulate && p.c_sectors && p.k_splits <= 1 && p.N <= 32) launch_chained(gemm_tcgen05_kernel<Kind, BN, kAddedNarrow>, grid, NUM_THREADS, smem, stream, ta, tb, p);
    else if (p.accumulate && p.c_sectors && p.k_splits <= 1) launch_chained(gemm_tcgen05_kernel<Kind, BN, kAdded>, grid, NUM_THREADS, smem_added, stream, ta, tb, p);
    else         launch_chained(gemm_tcgen05_kernel<Kind, BN, kPlain>, grid, NUM_THREADS, smem, stream, ta, tb, p);
    return LLMQ_LAUNCH_CHECK();
}

// Clusters of `parts` CTAs of the one-CTA kernel that reside at once (the same for all operand types: one CTA per SM)
int resident_clusters(int parts) {
    static int known[64][9] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& n = known[dev & 63][parts];
    if (n > 0) return n;
    constexpr int smem = Tile<256>::SMEM_BYTES;
    if (cudaFuncSetAttribute(gemm_tcgen05_kernel<0, 256, kCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) { cudaGetLastError(); return 0; }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = 64 * parts; cfg.blockDim = NUM_THREADS; cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1]{};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = parts; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int found = 0;
    if (cudaOccupancyMaxActiveClusters(&found, gemm_tcgen05_kernel<0, 256, kCluster>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    return n = found;
}

// ------------------------------------------------------------------------------------------------
// Host side: tensor-map encoding through the driver entry point (no link-time libcuda dependency).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess || !ptr)
            return nullptr;
        fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

}  // namespace

// Encodes a 2-D tiled map over a row-major [rows, cols] matrix with leading dimension ld (elements).
// The box is [box_rows][128 bytes] with the 128-byte swizzle.  Returns 0 on success.
int llmq_encode_tmap_2d(CUtensorMap* out, const void* base, int elem_bytes, long long rows, long long cols,
                        long long ld, int box_rows) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -1;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * elem_bytes};
    cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / elem_bytes), static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUtensorMapDataType dt = elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                             : (elem_bytes == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT8);
    CUresult r = fn(out, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

// 3-D view of an MN-major operand [rows = K, cols = M or N], cols a multiple of the 128-byte chunk: (column inside the chunk,
// K row, chunk).  The box is `chunks` chunks of [box_rows][128 bytes] one behind the other, the layout of that many 2-D boxes.
static int encode_tmap_chunks(CUtensorMap* out, const void* base, int elem_bytes, long long rows, long long cols, long long ld, int box_rows, int chunks) {
    EncodeTiledFn fn = get_encode_fn();
    if (!fn) return -1;
    const int chunk = 128 / elem_bytes;
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(chunk), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(cols / chunk)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(ld) * elem_bytes, 128};
    cuuint32_t box[3] = {static_cast<cuuint32_t>(chunk), static_cast<cuuint32_t>(box_rows), static_cast<cuuint32_t>(chunks)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(out, elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : static_cast<int>(r);
}

int llmq_gemm_2cta_launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tc, const GemmParams& p, int num_sms, cudaStream_t stream);

// Tile-shape selection: 0 = automatic, 1 = force the one-CTA kernel, 2 = force the CTA-pair kernel.
static int g_gemm_mode = 0;
static int g_gemm_tma_store = 1;
extern "C" void llmq_gemm_set_tma_store(int on) { g_gemm_tma_store = on; }
extern "C" void llmq_gemm_set_mode(int mode) { g_gemm_mode = mode; }
// Columns of a tile of the CTA-pair kernel: 0 = automatic, 224 or 256 = forced where the operands allow it (tests, measurements).  Other widths are
// refused (-1): the number goes into the MMA's descriptor and the byte counts of its barriers.
static int g_gemm_pair_bn = 0;
extern "C" int llmq_gemm_set_pair_bn(int bn) {
    if (bn != 0 && bn != 224 && bn != 256) return -1;
    g_gemm_pair_bn = bn;
    return 0;
}

static long long waves(long long tiles, int at_once) { return (tiles + at_once - 1) / at_once; }
static long long tiles_of(int M, int N, int bm, int bn) { return static_cast<long long>((M + bm - 1) / bm) * ((N + bn - 1) / bn); }

// The CTA-pair kernel runs GEMMs of at least 32 tiles of 256 x 256, and those that carry a collective or a fused epilogue (`fused`).
// Per round of tiles on all SMs it is 1.1 to 1.2 times as fast as the one-CTA kernel, whose 128 x 256 tiles it loses to where its own leave
// most of the last round idle: 896 x 4864 x 4096, both operands MN-major, is 76 pair tiles (two rounds of 74, 48.5 us) or 133 of the others
// (one round of 148, 36.4 us); with equally many rounds 16384 x 4608 x 3584 351 / 388 us, 4096 x 896 x 9728 60.8 / 66.4, 4096 x 4864 x 896
// 33.7 / 40.6.  With that many tiles the one-CTA kernel does not cut the K loop, so the sums have the same bits.
// Where they leave half of the GPU idle, with 48 or more K steps of 128 bytes, the one-CTA kernel in two K parts wins, pairs / parts in us: 1062 x 2048 x 3072 bf16 22 / 20,
// x 8192 46 / 33;  614 x 3584 x 12288 both MN-major 85 / 55;  1536 x 1536 x 8192 e4m3 26 / 23;  with 32 steps 17.4 / 17.5, with 16 12.7 / 14.8.  Where K may
// not be cut (no workspace) it walks the whole of K on tiles of 128 columns, in 0.73 to 1.02 of the pairs' time over 30 shapes (two took 1.08): 880 x 2448 x 5088 21.0 / 27.4, 1112 x 2048 x 6784
// B MN-major 35.7 / 37.6, 1000 x 2256 x 6368 A MN-major 41.4 / 42.6.  With both MN-major it takes 1.02 to 1.34 of it (14 shapes: 1512 x 1520 x 5904 49.5 / 44.5, 2208 x 1024 x 28224 e4m3
// 107 / 80), and the pairs keep them (`few_tiles` false).
static bool uses_pair_kernel(int M, int N, int K, int elem_bytes, bool fused, bool few_tiles, int num_sms) {
    if (elem_bytes == 4) return false;
    if (fused || g_gemm_mode == 2) return true;
    if (g_gemm_mode != 0 || M < 256 || static_cast<long long>(M) * N < 256LL * 256 * 32) return false;
    if (few_tiles && 2 * tiles_of(M, N, 128, 256) <= num_sms && K > 47 * (128 / elem_bytes)) return false;
    const long long pair = waves(tiles_of(M, N, 256, 256), num_sms / 2);
    return pair < 2 || 5 * waves(tiles_of(M, N, 128, 256), num_sms) >= 4 * pair;
}

// GEMMs of that many tiles that the one-CTA kernel is better at all the same.  Short K: what bounds them is the output, which its epilogue writes (and, where it is
// added to, reads) straight from the accumulators while a tile of a pair has twice the rows to drain before its successor.  Up to 8 K steps of 128 bytes it takes 0.75 to 0.98 of the
// pairs' time, one / pair tiles in us: 37888 x 3584 x 256 bf16 88 / 103, added to 130 / 165;  9728 x 896 x 512 0.88;  37888 x 3584 x 512 both MN-major 1.01;  with 10 steps 0.96
// (both MN-major 1.05), with 12 1.02 (1.10).  And one round of tiles on all SMs with up to 64 K steps, 16 with both operands MN-major: a pair starts later than
// a CTA, 2976 x 1536 x 1536 13.6 / 16.1, 1232 x 2048 x 2048 e4m3 10.4 / 11.9, 1960 x 2048 x 2048 15.5 / 17.1;  longer walks are bound by the loads, of which a pair has fewer:
// 743 x 5120 x 13824 92 / 80, 2048 x 2048 x 4746 both MN-major 37 / 31.  Neither cuts K, so the sums have the same bits.
// `line`: bytes, up to 128, that all rows of A and B start at a multiple of.  Rows that do not start with a 128-byte line cost the loads more, and the walk at which they are the bound is
// shorter.  One / pair tiles over 890 shapes: one round, rows of whole lines 0.63-1.05 up to 64 steps;  of 64 bytes 0.76-1.04 up to 34 steps, then up to 1.14;  of 32 0.76-1.01 up to 24, 1.10
// with 28, 1.20 with 46;  of 16 (8-bit elements) 0.92-1.06 up to 14, 1.13 with 28, 1.30 with 60 (1728 x 2080 x 7632 e4m3 38.8 / 29.8).  Short K with rows of 16 0.67-0.99 up to 6 steps, up to 1.13 with
// 7 and 8 (2784 x 7632 x 1008 e4m3 30.0 / 26.4).
// `output`: bf16 that is not added to and not made of whole sectors leaves the epilogue of this kernel 16 bytes a lane or less, that of the pairs through TMA or coalesced stores, and the pairs keep
// it (73 shapes with N a multiple of 4 or 8, 0.67-1.27 of the pairs' time, 1.04 on average: 7744 x 312 x 736 10.4 / 9.2, 6704 x 4280 x 104 31.7 / 28.7).  fp32: 0.54-1.03 up to 32 steps, up to 1.06 behind.
enum GemmOutput { kOutSectors, kOutPieces, kOutFp32 };          // bf16 in whole sectors or added to, other bf16, fp32
static bool better_with_one_cta(int M, int N, int K, int elem_bytes, bool both_mn, int line, int output, int num_sms) {
    if (g_gemm_mode != 0 || output == kOutPieces) return false;
    const int bk = 128 / elem_bytes, k_iters = (K + bk - 1) / bk;
    const long long tiles = tiles_of(M, N, 128, 256);
    int walk = line >= 128 ? 64 : line >= 64 ? 32 : line >= 32 ? 24 : 12;
    if (output == kOutFp32 && walk > 32) walk = 32;
    return k_iters <= (line >= 32 ? 8 : 6) || (tiles <= num_sms && 2 * tiles > num_sms && k_iters <= (both_mn && walk > 16 ? 16 : walk));
}

static bool takes_pair_kernel(int M, int N, int K, int elem_bytes, bool both_mn, int line, int output, bool fused, bool may_cut, int num_sms) {
    return uses_pair_kernel(M, N, K, elem_bytes, fused, may_cut || !both_mn, num_sms) && (fused || !better_with_one_cta(M, N, K, elem_bytes, both_mn, line, output, num_sms));
}
// CTAs that work on a tile of a plain GEMM of this shape (output: a GemmOutput): 2 or 1 (for tests; nothing is launched)
extern "C" int llmq_gemm_tile_ctas(int M, int N, int K, int elem_bytes, int both_mn_major, int line, int output, int may_cut, int num_sms) {
    return takes_pair_kernel(M, N, K, elem_bytes, both_mn_major != 0, line, output, false, may_cut != 0, num_sms) ? 2 : 1;
}

// Tile rows of 256 that the pair kernel works through together.  B is read from memory once per group, so a group is as large as its rows of A
// stay in the L2 beside the B tiles that stream past: up to 40 MB, but at least 4 and at most 32 tile rows.  Sustained, us with 4 / 8 / 16 / 32 tile
// rows (in brackets the MB of A in 8):  16384 x 37888 x 3584 e4m3 (7) 1840 / 1790 / 1718 / 1687, 16384 x 18944 x 3584 e4m3 (7) 940 / 896 / 868 / 854,
// 4096 x 152064 x 3584 bf16 (15) 3444 / 3299 / 3229 / 3207, 4096 x 151936 x 896 bf16 (4) 984 / 946 / 918 / 918, 16384 x 3584 x 18944 e4m3 (39)
// 919 / 912 / 914 / 985.  With a longer K no group's rows of A stay, and 4, 8 and 16 take the same time within the spread of 2 % (9 interleaved runs each, medians):
// 17920 x 1536 x 16384 bf16 (67) 719 / 719 / 719, 16384 x 3584 x 18944 bf16 (74) 1740 / 1748 / 1757, 4096 x 2048 x 128256 bf16 (501) 1818 / 1806 / 1779,
// 4096 x 3584 x 152064 bf16 (594) 4109 / 4098 / 4081, 16384 x 8192 x 32768 e4m3 (64) 3679 / 3681 / 3687.
// The order of the tiles is all that changes; kernels with a collective or a SwiGLU epilogue (`fused`) keep groups of 8.
static int pair_group_rows(int K, int elem_bytes, bool fused) {
    if (fused) return 8;
    int rows = 32;
    while (rows > 4 && static_cast<long long>(rows) * 256 * K * elem_bytes > (40ll << 20)) rows /= 2;
    return rows;
}

// Columns of a pair tile: 224 instead of 256 where that saves time, K-major B.  A round of 224-column tiles takes 0.93-0.95 of the time (the
// loads of A are the same), so it may need at most 3 % more rounds (none below 34), and 3 % more columns beyond N, which cost loads.  256 / 224 columns, us:
// 4096 x 896 x 151936 863 / 797 (896 is 4 x 224), 151936 x 896 x 4096 850 / 792, 4096 x 896 x 4864 33.5 / 31.1, 2048 x 3072 x 3072 39.8 / 37.3 (two
// rounds either way);  left at 256: 16384 x 3584 x 3584 275 / 278 (13 / 14 rounds), 4096 x 1152 x 896 15.5 / 16.1 (1280 / 1344 columns).
// 192, 160 and 128 columns are slower still per column: a K step takes 0.85, 0.83, 0.79 of the time of one of 256.
static int pair_tile_columns(int M, int N, int num_sms) {
    const long long w256 = waves(tiles_of(M, N, 256, 256), num_sms / 2), w224 = waves(tiles_of(M, N, 256, 224), num_sms / 2);
    const long long c256 = (N + 255) / 256 * 256LL, c224 = (N + 223) / 224 * 224LL;
    return 100 * w224 <= 103 * w256 && 100 * c224 <= 103 * c256 ? 224 : 256;
}

// Parts that the one-CTA kernel cuts the K loop into: more than one for outputs with at most half as many 256-column tiles as SMs and a
// long K.  The parts' sums, parts x M x N fp32 values, are limited to 64 MB.
constexpr long long kSplitFloats = 16ll << 20;
static int splitk_parts(int M, int N, int K, int elem_bytes, int num_sms) {
    const long long tiles = static_cast<long long>((M + BM - 1) / BM) * ((N + 255) / 256);
    const int bk = 128 / elem_bytes, k_iters = (K + bk - 1) / bk;
    if (tiles * 2 > num_sms || k_iters < 16) return 1;
    int parts = num_sms / static_cast<int>(tiles);
    if (parts > 8) parts = 8;
    if (parts > k_iters / 8) parts = k_iters / 8;
    while (parts > 1 && static_cast<long long>(parts) * M * N > kSplitFloats) --parts;
    // every part must get at least one K step
    while (parts > 1 && (parts - 1) * ((k_iters + parts - 1) / parts) >= k_iters) --parts;
    return parts;
}

// The parts of a tile form a cluster, which adds them up in distributed shared memory, where all clusters reside at once (148 SMs hold 74 / 45 / 33 / 26 /
// 22 / 15 / 15 of 2 .. 8 CTAs) and rows are whole 16-byte vectors of sums.  Otherwise the parts go through the workspace to a second kernel:
// a second round of clusters costs more than that.  us in a graph, two kernels / clusters: 1001 x 896 x 1152 12.9 / 9.9, 1152 x 896 x 1001 added to C
// 14.6 / 11.2, 896 x 896 x 1024 13.8 / 10.1, 339 x 3584 x 3584 added 22.4 / 16.4, 117 x 17920 x 1536 19.5 / 14.2, 576 x 1536 x 8960 30.4 / 24.4, 256 x 256 x 8192
// 11.1 / 9.2, 1966 x 896 x 9728 42 / 35 (50 shapes whose clusters reside: 0.68 to 1.02, 0.85 on average);  with more tiles 1152 x 896 x 4096 (36 of 4 parts) 22.6 / 28.4,
// 287 x 3072 x 8192 (36 of 4) 25.8 / 36.2, 256 x 2048 x 8192 e4m3 (16 of 8) 15.2 / 23.5.
struct SplitPlan {
    int parts, bn;                            // parts of K, columns of a tile
    bool cluster;                             // the parts of a tile are added up by a cluster
    int tiles;
};
static SplitPlan split_plan(const void* C, int M, int N, int K, int elem_bytes, long long ldc, int c_dtype, bool may_cut, int num_sms) {
    SplitPlan s;
    s.parts = may_cut ? splitk_parts(M, N, K, elem_bytes, num_sms) : 1;
    const int tiles128 = static_cast<int>(tiles_of(M, N, BM, 128));
    s.bn = elem_bytes != 4 && static_cast<long long>(tiles128) * s.parts <= num_sms ? 128 : 256;
    s.tiles = s.bn == 128 ? tiles128 : static_cast<int>(tiles_of(M, N, BM, 256));
    const int out_bytes = c_dtype == 0 ? 8 : 16;                           // four columns
    const bool vec = N % 4 == 0 && ldc % 4 == 0 && reinterpret_cast<uintptr_t>(C) % out_bytes == 0;
    s.cluster = s.parts > 1 && vec && s.tiles <= resident_clusters(s.parts);
    return s;
}

// Floats of the workspace with which a plain GEMM of this shape (A and B of `elem_bytes` an element) cuts its K loop; 0: it does not.
extern "C" long long llmq_gemm_splitk_floats(int M, int N, int K, int elem_bytes, int num_sms) {
    if (M <= 0 || N <= 0 || K <= 0 || elem_bytes <= 0 || uses_pair_kernel(M, N, K, elem_bytes, false, true, num_sms)) return 0;
    const int parts = splitk_parts(M, N, K, elem_bytes, num_sms);
    return parts > 1 ? static_cast<long long>(parts) * M * N : 0;
}

// How a plain GEMM with this output cuts its K loop if it may: 0 not at all, 1 in parts that clusters add up, 2 in parts that go through a workspace of
// llmq_gemm_splitk_floats.  Launches nothing; the stream is not used.
extern "C" int llmq_gemm_split_mode(const void* C, int M, int N, int K, int elem_bytes, long long ldc, int c_dtype, int num_sms, cudaStream_t) {
    if (llmq_gemm_splitk_floats(M, N, K, elem_bytes, num_sms) == 0) return 0;
    return split_plan(C, M, N, K, elem_bytes, ldc, c_dtype, true, num_sms).cluster ? 1 : 2;
}

extern "C" int llmq_gemm_ready(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, long long, long long, long long, int, int, int,
                               const float*, const float*, float, float*, unsigned int*, int, const unsigned int*, unsigned int, int, double, float*, long long,
                               cudaStream_t);
static int gemm_impl(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, long long, long long, long long, int, int, int,
                     const float*, const float*, float, float*, unsigned int*, int, const unsigned int*, unsigned int, int, double, const GemmParams*,
                     float*, long long, cudaStream_t);

extern "C" int llmq_gemm(const void* A, const void* B, void* C, const void* bias,
                         int M, int N, int K,
                         int ab_dtype,            // 0 bf16, 1 e4m3, 2 e5m2 (A), B shares the width
                         int b_dtype,
                         int a_mn_major, int b_mn_major,
                         long long lda, long long ldb, long long ldc,
                         int c_dtype, int bias_dtype, int accumulate,
                         const float* scale_a, const float* scale_b, float alpha,
                         float* absmax_out, unsigned int* status, int num_sms, cudaStream_t stream) {
    return llmq_gemm_ready(A, B, C, bias, M, N, K, ab_dtype, b_dtype, a_mn_major, b_mn_major, lda, ldb, ldc, c_dtype, bias_dtype, accumulate,
                           scale_a, scale_b, alpha, absmax_out, status, num_sms, nullptr, 0u, 0, 0.0, nullptr, 0, stream);
}

// Same, with the fused all-gather hook: rows of the stored B matrix are written by peer GPUs; ready_flags[src]
// reaching ready_gen marks source src's rows complete.  The producer warps poll the flags tile by tile.
// splitk_ws (optional): `splitk_floats` fp32 elements that no other work in flight uses; with fewer than llmq_gemm_splitk_floats
// of them the K loop stays whole.  splitk_floats = -1: it is cut where that needs no workspace (llmq_gemm_split_mode 1).
extern "C" int llmq_gemm_ready(const void* A, const void* B, void* C, const void* bias,
                               int M, int N, int K, int ab_dtype, int b_dtype, int a_mn_major, int b_mn_major,
                               long long lda, long long ldb, long long ldc, int c_dtype, int bias_dtype, int accumulate,
                               const float* scale_a, const float* scale_b, float alpha, float* absmax_out, unsigned int* status,
                               int num_sms, const unsigned int* ready_flags, unsigned int ready_gen, int ready_rows_per_src,
                               double ready_limit_s, float* splitk_ws, long long splitk_floats, cudaStream_t stream) {
    return gemm_impl(A, B, C, bias, M, N, K, ab_dtype, b_dtype, a_mn_major, b_mn_major, lda, ldb, ldc, c_dtype, bias_dtype, accumulate, scale_a,
                     scale_b, alpha, absmax_out, status, num_sms, ready_flags, ready_gen, ready_rows_per_src, ready_limit_s, nullptr, splitk_ws,
                     splitk_floats, stream);
}

// GEMM whose epilogue reduce-scatters the result over the data-parallel ranks (see gemm_tcgen05_2cta.cu).
// landing / counters: the landing buffer and the arrival counter of every rank (peer addresses); M must split
// into `world` row shards of a multiple of 32 rows, the output is bf16 with ldc == N.  `counter_target` is the
// value the local counter reaches after this call: every call adds world * (M / world / 32) * ceil(N / 256).
extern "C" int llmq_gemm_rs(const void* A, const void* B, void* C, int M, int N, int K, int ab_dtype, int b_dtype, int a_mn_major,
                            int b_mn_major, long long lda, long long ldb, int accumulate, const float* scale_a, const float* scale_b,
                            float alpha, unsigned int* status, int num_sms, void* const* landing, void* const* counters, int rank, int world,
                            unsigned int counter_target, void* shard_dst, int shard_accumulate, float shard_scale, float* norm_partials,
                            int num_partials, unsigned int seed, double limit_s, cudaStream_t stream) {
    if (world < 2 || world > 8 || M % world || (M / world) % 32 || M < 256 || N % 8) return -20;
    GemmParams rs{};
    rs.rs_world = world; rs.rs_rank = rank; rs.rs_shard_rows = M / world;
    for (int i = 0; i < world; ++i) { rs.rs_landing[i] = landing[i]; rs.rs_counter[i] = static_cast<unsigned int*>(counters[i]); }
    rs.rs_target = counter_target; rs.rs_dst = shard_dst; rs.rs_accumulate = shard_accumulate; rs.rs_scale = shard_scale;
    rs.rs_norm_partials = norm_partials; rs.rs_num_partials = num_partials > 0 ? num_partials : 1; rs.rs_seed = seed;
    rs.rs_limit_ns = static_cast<unsigned long long>(limit_s * 1e9);
    return gemm_impl(A, B, C, nullptr, M, N, K, ab_dtype, b_dtype, a_mn_major, b_mn_major, lda, ldb, N, 0, 0, accumulate, scale_a, scale_b, alpha,
                     nullptr, status, num_sms, nullptr, 0u, 0, 0.0, &rs, nullptr, 0, stream);
}

// GEMM with SwiGLU in the epilogue (see GemmParams::ep_mode).  mode 1: C[M, 2D] = A @ B^T with B = [up | gate] rows,
// aux[M, D] = swiglu(C).  mode 2: aux[M, 2D] ([up | gate] -> [d_up | d_gate], in place) from d(out) = A @ B^T, N = D.
// bf16 results; M >= 256, D a multiple of 128 (mode 1) / 8 (mode 2).  absmax_out follows the epilogue's output.
extern "C" int llmq_gemm_swiglu(const void* A, const void* B, void* C, void* aux, int mode, int M, int D, int K, int ab_dtype, int b_dtype,
                                int a_mn_major, int b_mn_major, long long lda, long long ldb, const float* scale_a, const float* scale_b,
                                float alpha, float* absmax_out, unsigned int* status, int num_sms, cudaStream_t stream) {
    if ((mode != 1 && mode != 2) || M < 256 || D % 8 || (mode == 1 && D % 128) || !aux || (mode == 1 && !C)) return -30;
    GemmParams ep{};
    ep.ep_mode = mode; ep.ep_ptr = aux; ep.ep_D = D;
    const int N = mode == 1 ? 2 * D : D;
    return gemm_impl(A, B, mode == 1 ? C : aux, nullptr, M, N, K, ab_dtype, b_dtype, a_mn_major, b_mn_major, lda, ldb, N, 0, 0, 0, scale_a, scale_b,
                     alpha, absmax_out, status, num_sms, nullptr, 0u, 0, 0.0, &ep, nullptr, 0, stream);
}

extern "C" unsigned int llmq_gemm_rs_arrivals(int M, int N, int world) {
    return static_cast<unsigned int>(world) * static_cast<unsigned int>(M / world / 32) * static_cast<unsigned int>((N + 255) / 256);
}

static int gemm_impl(const void* A, const void* B, void* C, const void* bias,
                     int M, int N, int K, int ab_dtype, int b_dtype, int a_mn_major, int b_mn_major,
                     long long lda, long long ldb, long long ldc, int c_dtype, int bias_dtype, int accumulate,
                     const float* scale_a, const float* scale_b, float alpha, float* absmax_out, unsigned int* status,
                     int num_sms, const unsigned int* ready_flags, unsigned int ready_gen, int ready_rows_per_src,
                     double ready_limit_s, const GemmParams* rs, float* splitk_ws, long long splitk_floats, cudaStream_t stream) {
    auto width = [](int dt) { return dt == 0 ? 2 : (dt == 1 || dt == 2) ? 1 : (dt == 3 ? 4 : 0); };
    const int eb = width(ab_dtype);
    if (eb == 0 || width(b_dtype) != eb) return -2;
    if (eb == 4 && (rs != nullptr || ready_flags != nullptr)) return -2;      // fp32 operands: one-CTA kernel without fused collectives
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    // TMA needs 16-byte aligned bases and row pitches
    if ((reinterpret_cast<uintptr_t>(A) & 15u) || (reinterpret_cast<uintptr_t>(B) & 15u)) return -3;
    if ((lda * eb) % 16 || (ldb * eb) % 16) return -4;

    CUtensorMap ta, tb;
    const int bk = 128 / eb;
    int rc;
    // The CTA-pair kernel stages 128 rows of B per CTA; the one-CTA kernel stages all 256.
    const bool fused = rs != nullptr || ready_flags != nullptr;
    const bool may_cut = splitk_floats < 0 ? split_plan(C, M, N, K, eb, ldc, c_dtype, true, num_sms).cluster
                                           : splitk_ws && static_cast<long long>(splitk_parts(M, N, K, eb, num_sms)) * M * N <= splitk_floats;
    const uintptr_t starts = reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | static_cast<uintptr_t>(lda * eb) | static_cast<uintptr_t>(ldb * eb) | 128u;
    const bool sectors = c_dtype == 0 && N % 16 == 0 && ldc % 16 == 0 && (reinterpret_cast<uintptr_t>(C) & 31u) == 0;
    const int output = c_dtype != 0 ? kOutFp32 : sectors || accumulate ? kOutSectors : kOutPieces;
    const bool pair_kernel = takes_pair_kernel(M, N, K, eb, a_mn_major && b_mn_major, static_cast<int>(starts & (~starts + 1)), output, fused, may_cut, num_sms);
    // An MN-major stage that is several 128-byte chunks wide (16-bit operands; the 256 rows of B of the one-CTA kernel) is fetched with
    // one 3-D load instead of one 2-D load per chunk: the loads of a stage were issued one after the other for longer than its MMAs
    // run.  bf16, CTA pairs, TFLOP/s with 2-D loads / 3-D loads / 3-D loads and a K loop per kind of load (gemm_tcgen05_2cta.cu), K-major
    // 1540: 17920 x 1536 x 16384 both operands 968-1062 / 1327 / 1435-1523, 16384 x 3584 x 4096 both 1052 / 1328 / 1520, B only 1352 / 1520 /
    // 1545, 4096^3 both 906 / 1184 / 1427.  With a ragged last chunk the 2-D boxes stay (its columns beyond the matrix would lie in the
    // next row), and for one chunk a 3-D box gains nothing.
    // One-CTA kernel: the K loop is cut into parts for outputs with fewer 256-column tiles than half of the SMs and a long K; where the
    // GPU then still has room for twice as many CTAs the tiles are 128 columns wide (half the MMA time per stage, more stages in
    // flight).  The cut depends on the 256-column tiles alone, so the sums have the same bits with both widths.  1001 x 896 x 1152 and
    // 1152 x 896 x 1001, the QKV gradients of a short batch, launch included: 46 -> 20-24 us with the vector form of the second pass.
    // Kernel times of the two widths, 128 / 256 columns, bf16, both operands K-major: with items for at most one CTA per SM
    // 256 x 896 x 896 8.4 / 11.9 us, 2304 x 896 x 896 9.6 / 12.5, 1001 x 896 x 1152 (112 items) 13.1 / 17.8, 512 x 1536 x 1536 (144 items)
    // 12.8 / 17.6;  with more 1024 x 1536 x 1536 (288) 19.2 / 19.2, 2048 x 896 x 4864 (224) 30.2 / 28.1, 256 x 7168 x 3584 (224) 25.3 /
    // 23.6;  both MN-major 512 x 1536 x 1536 14.3 / 18.5, 2048 x 896 x 4864 45.4 / 33.1, 512 x 3584 x 3584 (224) 36.2 / 28.7.
    const SplitPlan plan = split_plan(C, M, N, K, eb, ldc, c_dtype, may_cut, num_sms);
    const int splits = plan.parts, bn = plan.bn;
    int pair_bn = 256;
    if (pair_kernel && rs == nullptr && ready_flags == nullptr && !b_mn_major) pair_bn = g_gemm_pair_bn ? g_gemm_pair_bn : pair_tile_columns(M, N, num_sms);
    const int b_rows = pair_kernel ? pair_bn / 2 : bn;
    const bool a_box3 = a_mn_major && eb < 4 && BM > bk && M % bk == 0, b_box3 = b_mn_major && eb < 4 && b_rows > bk && N % bk == 0;
    if (!a_mn_major) rc = llmq_encode_tmap_2d(&ta, A, eb, M, K, lda, BM);
    else if (a_box3) rc = encode_tmap_chunks(&ta, A, eb, K, M, lda, bk, BM / bk);
    else             rc = llmq_encode_tmap_2d(&ta, A, eb, K, M, lda, bk);
    if (rc) return rc;
    if (!b_mn_major) rc = llmq_encode_tmap_2d(&tb, B, eb, N, K, ldb, b_rows);
    else if (b_box3) rc = encode_tmap_chunks(&tb, B, eb, K, N, ldb, bk, b_rows / bk);
    else             rc = llmq_encode_tmap_2d(&tb, B, eb, K, N, ldb, bk);
    if (rc) return rc;

    GemmParams p{};
    p.M = M; p.N = N; p.K = K; p.elem_bytes = eb;
    p.a_mn_major = a_mn_major; p.b_mn_major = b_mn_major; p.a_box3 = a_box3; p.b_box3 = b_box3;
    p.a_fmt = ab_dtype == 3 ? 2 : (ab_dtype == 0 ? 1 : (ab_dtype == 1 ? 0 : 1));
    p.b_fmt = b_dtype == 3 ? 2 : (b_dtype == 0 ? 1 : (b_dtype == 1 ? 0 : 1));
    p.C = C; p.ldc = ldc; p.c_dtype = c_dtype; p.accumulate = accumulate;
    p.bias = bias; p.bias_dtype = bias_dtype;
    p.group_rows = pair_group_rows(K, eb, rs != nullptr || ready_flags != nullptr);
    p.bn = pair_bn; p.b_stage_bytes = b_rows * 128;
    p.c_sectors = rs == nullptr && (accumulate || !pair_kernel) && sectors;
    p.scale_a = scale_a; p.scale_b = scale_b; p.alpha = alpha;
    p.absmax_out = absmax_out; p.status = status;
    p.ready_flags = ready_flags; p.ready_gen = ready_gen; p.ready_rows_per_src = ready_rows_per_src > 0 ? ready_rows_per_src : 1;
    p.ready_limit_ns = static_cast<unsigned long long>(ready_limit_s * 1e9);
    if (rs) {
        p.ep_mode = rs->ep_mode; p.ep_ptr = rs->ep_ptr; p.ep_D = rs->ep_D;
        p.rs_world = rs->rs_world; p.rs_rank = rs->rs_rank; p.rs_shard_rows = rs->rs_shard_rows;
        for (int i = 0; i < 8; ++i) { p.rs_landing[i] = rs->rs_landing[i]; p.rs_counter[i] = rs->rs_counter[i]; }
        p.rs_target = rs->rs_target; p.rs_dst = rs->rs_dst; p.rs_accumulate = rs->rs_accumulate; p.rs_scale = rs->rs_scale;
        p.rs_norm_partials = rs->rs_norm_partials; p.rs_num_partials = rs->rs_num_partials; p.rs_seed = rs->rs_seed;
        p.rs_limit_ns = rs->rs_limit_ns;
    }

    if (pair_kernel) {
        // A kernel that waits for other GPUs keeps its successor off the SMs.  So does one that leaves a third of them idle for long: the CTA pairs of
        // the next GEMM would be put onto just these, which is a worse choice of SMs than one among all.  Behind itself, us, with / without the release:
        // 640 x 3584 x 18944 96.5 / 91.6, 773 x 3072 x 16384 90.1 / 86.4, 2048 x 1536 x 10752 61.0 / 58.3;  with fewer than 64 K steps, or more tiles, it is 2 to 5 %
        // faster with it.
        const bool idle_sms = 10 * tiles_of(M, N, 256, pair_bn) < 7 * (num_sms / 2) && K >= 64 * bk;
        p.early_release = ready_flags == nullptr && p.rs_world == 0 && !idle_sms;
        // plain bf16 outputs leave the epilogue through TMA stores: a tensor map of C with 64-column x 32-row boxes
        CUtensorMap tc = ta;
        if (c_dtype == 0 && !accumulate && p.rs_world == 0 && p.ep_mode == 0 && (N % 8) == 0 && (ldc % 8) == 0 &&
            (reinterpret_cast<uintptr_t>(C) & 15u) == 0 && g_gemm_tma_store) {
            if (llmq_encode_tmap_2d(&tc, C, 2, M, N, ldc, 32) == 0) p.c_tma = 1;
        }
        return llmq_gemm_2cta_launch(ta, tb, tc, p, num_sms, stream);
    }

    const int tiles = plan.tiles;
    const bool cluster = plan.cluster;
    if (splits > 1) { p.k_splits = splits; p.partial = splitk_ws; }
    if (bn == 128) rc = eb == 1 ? launch_one_cta<1, 128>(ta, tb, p, tiles * splits, cluster, num_sms, stream) : launch_one_cta<0, 128>(ta, tb, p, tiles * splits, cluster, num_sms, stream);
    else if (eb == 1) rc = launch_one_cta<1, 256>(ta, tb, p, tiles * splits, cluster, num_sms, stream);
    else if (eb == 2) rc = launch_one_cta<0, 256>(ta, tb, p, tiles * splits, cluster, num_sms, stream);
    else              rc = launch_one_cta<2, 256>(ta, tb, p, tiles * splits, cluster, num_sms, stream);
    if (rc || cluster) return rc;
    if (splits > 1) {
        const long long total = static_cast<long long>(M) * N;             // at most kSplitFloats / 2
        const int out_bytes = c_dtype == 0 ? 8 : 16;                       // four columns
        if (N % 4 == 0 && ldc % 4 == 0 && reinterpret_cast<uintptr_t>(C) % out_bytes == 0) {
            long long blocks = (total / 4 + 255) / 256;
            if (blocks > 8LL * num_sms) blocks = 8LL * num_sms;
            launch_chained(splitk_reduce_vec_kernel, static_cast<unsigned int>(blocks), 256, 0, stream, p, p.alpha, FastDiv(static_cast<uint32_t>(N / 4)));
            return static_cast<int>(cudaGetLastError());
        }
        long long blocks = (total + 255) / 256;
        if (blocks > 4LL * num_sms) blocks = 4LL * num_sms;
        launch_chained(splitk_reduce_kernel, static_cast<unsigned int>(blocks), 256, 0, stream, p, p.alpha);
    }
    return static_cast<int>(cudaGetLastError());
}
