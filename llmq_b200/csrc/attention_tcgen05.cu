// Causal grouped-query flash attention, forward and backward, on tcgen05 tensor cores (sm_100a).
//
// Operates directly on the packed post-RoPE tensor qkv (B, T, Hq + 2*Hkv, HS) through strided TMA maps,
// writes out (B, T, Hq, HS) and the per-row log-sum-exp (B, Hq, T); the backward pass produces the
// packed gradient dqkv with the same layout.  It takes the place of the cuDNN SDPA graphs and the
// scalar fallback kernel of the reference (src/kernels/cudnn_att.cpp:46-263, src/kernels/attention.cu).
//
// The forward kernel is in attention_fwd_pingpong.cu.  The two kinds of gradient CTAs share one organisation.  A CTA owns a 128-row tile
// (keys for dK / dV, queries for dQ) and walks over 64-column score tiles.  16 compute warps form two groups that take the tiles in
// turn, two warps issue MMAs, the others load by TMA.  Everything is handed over through mbarriers (one arrival per warp); score tiles
// are double buffered in tensor memory, the streamed operand (Q / dO for dK / dV, K / V for dQ) sits in a ring of shared-memory buffers.
// P^T, dS^T and dS never leave tensor memory: the bf16 values take the place of the scores they were computed from and are the A
// operands of the accumulating MMAs.  Q and dO of the dQ CTAs, and with head size 64 K and V of the others, are A operands in tensor
// memory too.  The shared-memory tile of V / K / Q / dO doubles as an MN-major B operand, so no transposed copy is ever made.
//
// Backward is made of two kinds of CTAs, both deterministic (no atomics):
//   * dK/dV: one CTA per (batch, kv head, 128 keys) walks over all query heads of the group and all query blocks at or below the
//     diagonal; dK and dV accumulate in TMEM across the whole walk.  With few items a cluster shares the heads (split_heads).
//   * dQ   : one CTA per (batch, kv head, 128 queries) and part of the group walks over its query heads and their key blocks; dQ
//     accumulates in TMEM and is drained once per head.
// A small pre-pass computes delta = rowsum(dO * O).  Both kinds are launched as one grid: neither needs what the other writes, so the dQ CTAs
// start on the SMs that the dK / dV CTAs leave idle, at the end of their longest walks or, with few items, from the start.  The CTAs with the longest walks
// of each kind come first.  attention_backward in us, a launch for each kind / one:  8 x 1024 tokens, 14 / 2 heads of 64 112 / 80;  4 x 1024 94 / 73;  1 x 333, 12 / 2
// heads of 128 21.9 / 15.1;  2 x 700, 24 / 8 of 128 54 / 38;  where each kind alone fills the SMs for many rounds, 8 x 2048, 28 / 4 of 128, 761 / 758.
//
// What bounds it, head size 128: a tile of dK / dV takes 1190 cycles (clock stamps, 8 x 2048 tokens, 28 / 4 heads).  Its MMAs need 1024 of the tensor pipe and 1024 of shared memory: 16 of N = 64
// with both operands in shared memory, 32 cycles of the pipe and 48 of reading them, 8 of N = 128 with A in tensor memory, 64 and 32; one after the other they take 1300.  A tile of dQ
// takes 880, its MMAs 768.  At head size 64 no unit is saturated.  The rest is the chain of
// hand-overs of a tile.  A wait on an mbarrier costs a warp about 150 cycles even when the phase is complete, and several times that
// while MMAs with both operands in shared memory run: those take nearly all of its bandwidth.  Hence two groups of compute warps, two
// issuing warps, row statistics in few wide loads, and everything that comes from global memory (Q / dO and the statistics of the next
// head or tile) fetched a tile or a head ahead by a warp of its own; the statistics that the producer used to wait for tile by tile alone
// cost 10 to 20 % of dK / dV.  Times of the two kinds as two launches, one after the other, before they shared a grid, us, one group and one issuing warp / two:
//                                          dK / dV      dQ
//   8 x 2048 tokens, 28 / 4 heads of 128   425 / 364   403 / 331
//   1 x 8192, 32 / 8 heads of 128          880 / 752   708 / 620
//   8 x 1024, 14 / 2 heads of 64            87 / 68     56 / 42
//   2 x 4096, 32 / 8 heads of 64           368 / 285   300 / 221
//   1 x 333, 12 / 2 heads of 128            37 / 30     10 / 9      (one CTA per item; with a cluster dK / dV took 14)
// Not better: score tiles of 128 columns without a second buffer; with head size 64 P^T in columns of its own and S issued before the sums
// of the tile two before (dK / dV 68 -> 77: the groups then meet at the exponentials).
#include <cstdlib>
#include "ptx_sm100.cuh"
#include "api.h"
#include "common.cuh"

using namespace sm100;

namespace {

constexpr float kLog2e = 1.4426950408889634f;
// Backward kernels: two groups of two warpgroups; in a tile a thread of a group handles 32 score columns of its row(s)
constexpr int kBwdWarpgroups = 4;
constexpr int kBwdComputeThreads = 128 * kBwdWarpgroups;
constexpr int kBwdComputeWarps = kBwdComputeThreads / 32;
constexpr int kBwdGroupWarps = kBwdComputeWarps / 2;              // two groups, alternating score tiles
// + four helper warps: two MMA issuers and one (dK / dV) or two (dQ) TMA producers
constexpr int kBwdThreads = kBwdComputeThreads + 128;
// A block's code is used twice: barriers and tensor memory before the wait for the kernel before (nothing of global memory is touched), the walk after it
enum { kBwdSetup, kBwdRun };
// One arrival per warp (512 single arrivals on one shared-memory word would serialise): the lanes' earlier
// writes and fences are ordered before lane 0's releasing arrive by the warp barrier.
__device__ __forceinline__ void warp_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}
// 2^x with the hardware approximation (-inf -> 0)
__device__ __forceinline__ float fast_exp2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

#define kDescHi desc_hi(1024)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess || !ptr) return nullptr;
        fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    return fn;
}

// bf16 tensor viewed as (B, T, W) with W contiguous; box = [box_rows along T][64 elements of W], 128B swizzle.
int encode_btw(CUtensorMap* out, const void* base, int B, int T, long long W, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return -1;
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(W), static_cast<cuuint64_t>(T), static_cast<cuuint64_t>(B)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(W) * 2, static_cast<cuuint64_t>(W) * 2 * T};
    cuuint32_t box[3] = {64, static_cast<cuuint32_t>(box_rows), 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 1000 + static_cast<int>(r);
}

// not __ldg: the compiler may move such a load in front of grid_wait()
template <typename V>
__device__ __forceinline__ V load_plain(const V* p) { return *p; }

struct AttnParams {
    int B, T, Hq, Hkv;
    float scale;                 // 1/sqrt(HS)
    float* lse;                  // (B,Hq,T), natural log
    const float* delta;          // (B,Hq,T)
    bf16* dqkv;                  // packed gradient
    const bf16* qkv;             // packed inputs as a plain pointer
    unsigned int* status;
};

// ------------------------------------------------------------------------------------------------
// delta[b,h,t] = sum_d dO[b,t,h,d] * O[b,t,h,d]; HS / 8 lanes per row (one 16-byte load of each tensor per lane), so a
// warp covers 2 (HS = 128) or 4 (HS = 64) rows and every lane has work
template <int HS>
__global__ void __launch_bounds__(256)
attn_delta_kernel(float* __restrict__ delta, const bf16* __restrict__ o, const bf16* __restrict__ d_o, int B, int T, int Hq) {
    grid_release();
    grid_wait();
    const int bx = after_wait(blockIdx.x), tx = after_wait(threadIdx.x);
    constexpr int LANES = HS / 8;                       // lanes per row
    static_assert(LANES == 8 || LANES == 16, "head sizes 64 and 128");
    const long long gid = bx * static_cast<long long>(blockDim.x) + tx;
    const long long w = gid / LANES;                    // row index over (b, t, h)
    const int sub = static_cast<int>(gid % LANES);
    const long long total = static_cast<long long>(B) * T * Hq;
    const bool active = w < total;
    float s = 0.f;
    if (active) {
        Vec16<bf16> a = Vec16<bf16>::load(o + w * HS + sub * 8), g = Vec16<bf16>::load(d_o + w * HS + sub * 8);
#pragma unroll
        for (int k = 0; k < 8; ++k) s += __bfloat162float(a.v[k]) * __bfloat162float(g.v[k]);
    }
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (active && sub == 0) {
        const int h = static_cast<int>(w % Hq);
        const long long bt = w / Hq;
        const int t = static_cast<int>(bt % T);
        const long long b = bt / T;
        delta[(b * Hq + h) * T + t] = s;
    }
}

// ------------------------------------------------------------------------------------------------
// 16 fp32 accumulator values of one row -> 16 bf16 in global memory: one store of 32 bytes where the gradient is aligned to as much (a lane that writes 16
// bytes at a time touches every sector twice; us, 16 / 32 bytes: 8 x 2048 tokens, 28 / 4 heads of 128 761 / 741, 8 x 1024, 14 / 2 of 64 80.0 / 78.1, 2 x 700, 24 / 8
// of 128 38.2 / 34.9, 8 x 100, 32 / 8 of 128 20.1 / 18.0)
__device__ __forceinline__ void store16_bf16(bf16* dst, const uint32_t (&r)[16]) {
    uint32_t v[8];
#pragma unroll
    for (int jj = 0; jj < 8; ++jj) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(r[2 * jj]), __uint_as_float(r[2 * jj + 1]));
        v[jj] = *reinterpret_cast<const uint32_t*>(&h);
    }
    if (reinterpret_cast<uintptr_t>(dst) % 32 == 0) {
        store_sector(dst, v);
    } else {
        *reinterpret_cast<uint4*>(dst) = make_uint4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<uint4*>(dst + 8) = make_uint4(v[4], v[5], v[6], v[7]);
    }
}
__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ float4 ld_cluster_f32x4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}

// ------------------------------------------------------------------------------------------------
// dK / dV.  Walk over the (query head, query block) tiles.  Q / dO tiles sit in a ring of shared-memory buffers, P^T / dS^T go back to
// tensor memory.  The thread layout of the score tiles (16 x 256 bit TMEM accesses) gives a thread two of every eight columns of four
// rows, so that the statistics of its columns are four 16-byte shared-memory loads a tile instead of sixteen: loads from shared
// memory all but stop while MMAs with both operands there run.
// With HS = 64 K and V live in tensor memory as A operands; with HS = 128 scores and accumulators fill it.
template <int HS>
struct DkdvShape {
    static constexpr bool kTmemKV = HS == 64;
    static constexpr int NBUF = HS == 64 ? 6 : 4;
    static constexpr int KV_BYTES = 128 * HS * 2, Q_BYTES = 64 * HS * 2;
    static constexpr int STAT_OFFSET = (kTmemKV ? 0 : 2 * KV_BYTES) + 2 * NBUF * Q_BYTES;
    static constexpr int SMEM_BYTES = STAT_OFFSET + NBUF * 64 * 8 + 256;
};

template <int HS, int Phase>
__device__ __forceinline__ void
bwd_dkdv_block(const CUtensorMap& tmap_kv128,                          // qkv, box 128 rows (K and V tiles)
               const CUtensorMap& tmap_q64,                            // qkv, box 64 rows (Q tiles)
               const CUtensorMap& tmap_do64,                           // dO, box 64 rows
               const AttnParams& p, const int parts,                   // CTAs of a cluster that share the query heads of an item
               const int block) {
    using Shape = DkdvShape<HS>;
    constexpr int BKV = 128, BQ = 64, NCH = HS / 64, NBUF = Shape::NBUF;
    constexpr int KV_BYTES = Shape::KV_BYTES, Q_BYTES = Shape::Q_BYTES;
    constexpr bool kTmemKV = Shape::kTmemKV;
    constexpr uint32_t TMEM_COLS = 512;                       // S0 S1 | dP0 dP1 | dV | dK (| K | V)
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;                                       // HS = 128
    uint8_t* sV = sK + KV_BYTES;
    uint8_t* sQ = smem + (kTmemKV ? 0 : 2 * KV_BYTES);        // NBUF buffers
    uint8_t* sdO = sQ + NBUF * Q_BYTES;                       // NBUF buffers
    float2* sStat = reinterpret_cast<float2*>(smem + Shape::STAT_OFFSET);  // [NBUF][64] (lse * log2(e), delta * softmax scale)
    uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + NBUF * BQ);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);       // uniform, and known to be
    const int role = warp - kBwdComputeWarps;                 // 0, 1: MMA issuers (one elected lane); 2: TMA loads and row statistics; 3: none
    const int wg = tid >> 7, r = tid & 127;                   // compute threads: warpgroup, TMEM lane
    // 1-D grid, key block slowest: the blocks with the longest walks (small kb) start first on every SM
    const int item = block / parts, part = block % parts;
    const int kb = item / (p.Hkv * p.B);
    const int kvh = (item % (p.Hkv * p.B)) % p.Hkv, b = (item % (p.Hkv * p.B)) / p.Hkv;
    const int G = p.Hq / p.Hkv;
    const int h0 = kvh * G + G * part / parts, nh = G * (part + 1) / parts - G * part / parts;      // query heads [h0, h0 + nh)
    const int kv0 = kb * BKV;
    const int nqb = (p.T + BQ - 1) / BQ;
    const int qb_first = kv0 / BQ;
    const int n_it = (nqb - qb_first) * nh;
    const int kcol = (p.Hq + kvh) * HS, vcol = (p.Hq + p.Hkv + kvh) * HS;

    // barriers: 0 K / V in place | 1-2 S ready | 3-4 dP ready | 5-6 P^T in tensor memory | 7-8 dS^T in tensor memory | 9 all done |
    //           10.. q/dO ring (TMA bytes + row statistics) | 16.. q/dO buffer free.  Two-entry sets alternate with the tile parity: the
    //           commit of tile it+2 needs the group of tile it to have handed it over, so a waiter can never miss a phase.
    const uint32_t bar0 = smem_u32(bars);
    const uint32_t kv_bar = bar0, done_bar = bar0 + 72;
    auto score_bar = [&](int which, int it) { return bar0 + 8 + 16 * which + 8 * (it & 1); };      // 0: S, 1: dP
    auto ready_bar = [&](int which, int it) { return bar0 + 40 + 16 * which + 8 * (it & 1); };     // 0: P^T, 1: dS^T
    auto qdo_bar = [&](int buf) { return bar0 + 80 + 8 * buf; };
    auto qdo_free = [&](int buf) { return bar0 + 128 + 8 * buf; };
    if constexpr (Phase == kBwdSetup) {
        if (tid == 0) {
            mbar_init(kv_bar, kTmemKV ? kBwdComputeWarps : 1); mbar_init(done_bar, 2);
            for (int i = 0; i < NBUF; ++i) { mbar_init(qdo_bar(i), 2); mbar_init(qdo_free(i), 2); }
            for (int w = 0; w < 2; ++w)
                for (int i = 0; i < 2; ++i) { mbar_init(score_bar(w, i), 1); mbar_init(ready_bar(w, i), kBwdGroupWarps); }
            *abort_flag = 0;
            mbar_init_fence();
        }
        if (role == 0) { tmem_alloc(smem_u32(tmem_slot), TMEM_COLS); tmem_relinquish(); }
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
        return;
    }
    const uint32_t tmem = *tmem_slot;
    const uint32_t tdV = tmem + 4 * BQ, tdK = tdV + HS;
    const uint32_t tK = tdK + HS, tV = tK + HS / 2;           // HS = 64
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    auto tS = [&](int it) { return tmem + (it & 1) * BQ; };
    auto tdP = [&](int it) { return tmem + 2 * BQ + (it & 1) * BQ; };
    uint4* const sums = reinterpret_cast<uint4*>(smem);       // parts > 1: [dK, dV][128 rows][32] after the walk
    bool ok = true;

    if (role == 2) {
        // ============================================================ TMA producer warp
        const int lane = tid & 31;
        if (lane == 0) {
            tma_prefetch_desc(&tmap_q64); tma_prefetch_desc(&tmap_do64);
            if (!kTmemKV && n_it > 0) {
                tma_prefetch_desc(&tmap_kv128);
                mbar_expect_tx(kv_bar, 2 * KV_BYTES);
                for (int c = 0; c < NCH; ++c) {
                    tma_load_3d(smem_u32(sK) + c * (BKV * 128), &tmap_kv128, kv_bar, kcol + c * 64, kv0, b);
                    tma_load_3d(smem_u32(sV) + c * (BKV * 128), &tmap_kv128, kv_bar, vcol + c * 64, kv0, b);
                }
            }
        }
        int hq = h0, qb = qb_first;
        // lse and delta of a tile's 64 queries, two per lane, read one tile ahead; rows beyond the sequence get probability 0
        float2 stat[2], stat_next[2];
        auto load_stats = [&](float2 (&st)[2]) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int q = qb * BQ + lane + 32 * i;
                const long long si = (static_cast<long long>(b) * p.Hq + hq) * p.T + q;
                st[i] = q < p.T ? make_float2(load_plain(p.lse + si), load_plain(p.delta + si)) : make_float2(INFINITY, 0.f);
            }
        };
        if (n_it > 0) load_stats(stat);
        for (int it = 0; it < n_it; ++it) {
            const int buf = it % NBUF, hq_now = hq, qb_now = qb;
            if (++qb == nqb) { qb = qb_first; ++hq; }
            if (it + 1 < n_it) load_stats(stat_next);
            // the buffer's previous tile, it - NBUF, has been consumed by its dV / dK MMAs
            if (it >= NBUF) {
                bool got = true;
                if (lane == 0) got = mbar_wait(qdo_free(buf), ((it / NBUF) - 1) & 1, abort_flag);
                if (!__shfl_sync(0xffffffffu, static_cast<int>(got), 0)) { if (lane == 0) atomicOr(p.status, kErrOther); break; }
            }
            if (lane == 0) {
                mbar_expect_tx(qdo_bar(buf), 2 * Q_BYTES);
                for (int c = 0; c < NCH; ++c) {
                    tma_load_3d(smem_u32(sQ) + buf * Q_BYTES + c * (BQ * 128), &tmap_q64, qdo_bar(buf), hq_now * HS + c * 64, qb_now * BQ, b);
                    tma_load_3d(smem_u32(sdO) + buf * Q_BYTES + c * (BQ * 128), &tmap_do64, qdo_bar(buf), hq_now * HS + c * 64, qb_now * BQ, b);
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                sStat[buf * BQ + lane + 32 * i] = make_float2(stat[i].x * kLog2e, stat[i].y * p.scale);
                stat[i] = stat_next[i];
            }
            warp_arrive(qdo_bar(buf));
        }
    } else if (role == 0 || role == 1) {
        // ============================================================ MMA issuer warps
        // Warp 0 issues S^T = K Q^T and dV += P^T dO, warp 1 dP^T = V dO^T and dK += dS^T Q: the same sequence, on other operands.  P^T (dS^T)
        // of tile it lies in the buffer of S (dP) of tile it + 2; MMAs of one thread execute in issue order, so a buffer that a later MMA
        // overwrites needs no barrier for the MMAs that read it.  One warp for both needs up to 1400 cycles a tile for its waits and the issue.
        if (n_it > 0) {
            const bool leader = elect_one();
            const uint32_t idesc_st = make_instr_desc(1, 1, false, false, BKV, BQ);
            const uint32_t idesc_acc = make_instr_desc(1, 1, false, true, BKV, HS);
            const uint32_t a_lo = desc_lo(smem_u32(role == 0 ? sK : sV), 16), a_tmem = role == 0 ? tK : tV;
            const uint32_t b_score = desc_lo(smem_u32(role == 0 ? sQ : sdO), 16), b_acc = desc_lo(smem_u32(role == 0 ? sdO : sQ), BQ * 128);
            const uint32_t t_score = role == 0 ? tS(0) : tdP(0), t_acc = role == 0 ? tdV : tdK;
            auto issue_scores = [&](int it, int buf) {
                const uint32_t d = t_score + (it & 1) * BQ, b_lo = b_score + buf * (Q_BYTES >> 4), bar = score_bar(role, it);
                if (leader) {
#pragma unroll
                    for (int k = 0; k < HS / 16; ++k) {
                        const uint32_t bk = b_lo + (((k / 4) * (BQ * 128) + (k % 4) * 32) >> 4);
                        if constexpr (kTmemKV) mma_issue_f16_tmem_a(d, a_tmem + k * 8, bk, kDescHi, idesc_st, k > 0);
                        else mma_issue<false, false>(d, a_lo + (((k / 4) * (BKV * 128) + (k % 4) * 32) >> 4), kDescHi, bk, kDescHi, idesc_st, k > 0);
                    }
                    mma_commit(bar);
                }
                __syncwarp();
            };
            ok = mbar_wait_warp(kv_bar, 0, abort_flag);
            for (int it = 0; it < 2 && it < n_it && ok; ++it) {
                ok = mbar_wait_warp(qdo_bar(it), 0, abort_flag);
                tc_fence_after_sync();
                if (ok) issue_scores(it, it);
            }
            for (int it = 0; it < n_it && ok; ++it) {
                const int buf = it % NBUF, buf2 = (it + 2) % NBUF;
                const uint32_t phase2 = ((it + 2) / NBUF) & 1;
                const bool loaded = it + 2 < n_it && mbar_test_wait(qdo_bar(buf2), phase2);          // asked early, answered by the time it is needed
                if (!mbar_wait_warp(ready_bar(role, it), (it >> 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after_sync();
                const uint32_t b_lo = b_acc + buf * (Q_BYTES >> 4), a_t = t_score + (it & 1) * BQ, bar = qdo_free(buf);
                const uint32_t acc0 = it > 0;
                if (leader) {
#pragma unroll
                    for (int k = 0; k < BQ / 16; ++k)
                        mma_issue_f16_tmem_a(t_acc, a_t + k * 16, b_lo + ((k * (16 * 128)) >> 4), kDescHi, idesc_acc, k > 0 ? 1u : acc0);
                    mma_commit(bar);
                }
                __syncwarp();
                if (it + 2 < n_it) {
                    if (!__all_sync(0xffffffffu, loaded)) ok = mbar_wait_warp(qdo_bar(buf2), phase2, abort_flag);
                    if (ok) issue_scores(it + 2, buf2);
                }
            }
            if (leader) {
                if (ok) mma_commit(done_bar);
                else { *abort_flag = 1u; atomicOr(p.status, kErrOther); }
            }
            __syncwarp();
        }
    } else if (role < 0) {
        // ============================================================ compute warps
        // Two groups of two warpgroups take turns: group g works on the tiles of parity g, warpgroup `half` of it on 32 of their columns.
        const float sl2 = p.scale * kLog2e;
        const int lane = tid & 31, grp = wg >> 1, half = wg & 1;
        const int kv_row = kv0 + r;
        if constexpr (kTmemKV) {
            // rows of K (group 0) and V (group 1) into tensor memory, 16 packed words per thread; zeros beyond the sequence
            if (n_it > 0) {
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = 0u;
                if (kv_row < p.T) {
                    const uint4* src = reinterpret_cast<const uint4*>(p.qkv + (static_cast<long long>(b) * p.T + kv_row) * (p.Hq + 2 * p.Hkv) * HS +
                                                                      (grp == 0 ? kcol : vcol) + half * 32);
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        const uint4 x = load_plain(src + q4);
                        w[4 * q4] = x.x; w[4 * q4 + 1] = x.y; w[4 * q4 + 2] = x.z; w[4 * q4 + 3] = x.w;
                    }
                }
                __syncwarp();
                tmem_st_32x32b_x16((grp == 0 ? tK : tV) + lane_off + half * 16, w);
                tmem_st_wait();
                tc_fence_before_sync();
                warp_arrive(kv_bar);
            }
        }
        int qb = qb_first + grp;
        while (qb >= nqb) qb -= nqb - qb_first;
        const int row_l = (warp & 3) * 32 + (lane >> 2), col_l = half * 32 + 2 * (lane & 3);  // tile row / column of this thread's first value
        for (int it = grp; it < n_it; it += 2) {
            const int buf = it % NBUF;
            if (!mbar_wait(qdo_bar(buf), (it / NBUF) & 1, abort_flag)) { ok = false; break; }
            float4 st[4];                                       // (lse, delta) of columns col_l + 8 i and + 1
#pragma unroll
            for (int i = 0; i < 4; ++i) st[i] = *reinterpret_cast<const float4*>(sStat + buf * BQ + col_l + 8 * i);
            if (!mbar_wait(score_bar(0, it), (it >> 1) & 1, abort_flag)) { ok = false; break; }
            tc_fence_after_sync();
            float pv[2][16];                                    // 16-row halves: [4 i + 2 r8 + c] = row + 8 r8, column 8 i + c
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) tmem_ld_16x256b_x4(tS(it) + lane_off + (h << 20) + half * 32, *reinterpret_cast<uint32_t(*)[16]>(pv[h]));
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < 16; ++i) pv[h][i] = fast_exp2(fmaf(pv[h][i], sl2, -((i & 1) ? st[i / 4].z : st[i / 4].x)));
            if (qb * BQ < kv0 + BKV) {                          // only tiles that touch the diagonal pay for the mask
                const int lim = kv0 + row_l - qb * BQ - col_l;  // columns below lim (+ the row's offset) are above the diagonal (q < kv)
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < 16; ++i) if (8 * (i / 4) + (i & 1) < lim + 16 * h + 8 * ((i >> 1) & 1)) pv[h][i] = 0.f;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int k = 0; k < 2; ++k) {                   // K steps of 16 queries
                    const float* v = pv[h] + 8 * k;
                    tmem_st_16x128b_x2(tS(it) + lane_off + (h << 20) + (2 * half + k) * 16, pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                                       pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
                }
            tmem_st_wait();
            tc_fence_before_sync();
            warp_arrive(ready_bar(0, it));
            if (!mbar_wait(score_bar(1, it), (it >> 1) & 1, abort_flag)) { ok = false; break; }
            tc_fence_after_sync();
            uint32_t rp[2][16];
            __syncwarp();
#pragma unroll
            for (int h = 0; h < 2; ++h) tmem_ld_16x256b_x4(tdP(it) + lane_off + (h << 20) + half * 32, rp[h]);
            tmem_ld_wait();
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    uint32_t d[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {               // j = 2 (column group) + (row + 8)
                        const int i = 8 * k + 2 * j;
                        d[j] = pack_bf16x2(pv[h][i] * fmaf(__uint_as_float(rp[h][i]), p.scale, -st[i / 4].y),
                                           pv[h][i + 1] * fmaf(__uint_as_float(rp[h][i + 1]), p.scale, -st[i / 4].w));
                    }
                    tmem_st_16x128b_x2(tdP(it) + lane_off + (h << 20) + (2 * half + k) * 16, d[0], d[1], d[2], d[3]);
                }
            tmem_st_wait();
            tc_fence_before_sync();
            warp_arrive(ready_bar(1, it));
            qb += 2;
            while (qb >= nqb) qb -= nqb - qb_first;
        }
        if (ok && n_it > 0) ok = mbar_wait(done_bar, 0, abort_flag);
        tc_fence_after_sync();
        if (!ok && r == 0) atomicOr(p.status, kErrOther);
        if (ok && n_it > 0) {
            // The TMEM loads are warp-collective: every lane executes them, only the stores are predicated.
            const bool row_ok = kv_row < p.T;
            bf16* dk = p.dqkv + ((static_cast<long long>(b) * p.T + (row_ok ? kv_row : 0)) * (p.Hq + 2 * p.Hkv)) * HS + kcol;
            bf16* dv = dk + (vcol - kcol);
            __syncwarp();
            constexpr int ECW = HS / kBwdWarpgroups;           // output columns per thread
#pragma unroll
            for (int c = 0; c < ECW; c += 16) {
                const int col = wg * ECW + c;
                uint32_t rk[16], rv[16];
                tmem_ld_32x32b_x16(tdK + lane_off + col, rk);
                tmem_ld_32x32b_x16(tdV + lane_off + col, rv);
                tmem_ld_wait();
                if (HS == 128 && parts > 1) {
                    // every MMA and load of this CTA is complete: the sums of its heads go over K, V and the ring, rows of 32 16-byte
                    // pieces, swizzled
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int at = r * 32 + ((col / 4 + i) ^ lane);
                        sums[at] = make_uint4(rk[4 * i], rk[4 * i + 1], rk[4 * i + 2], rk[4 * i + 3]);
                        sums[128 * 32 + at] = make_uint4(rv[4 * i], rv[4 * i + 1], rv[4 * i + 2], rv[4 * i + 3]);
                    }
                } else if (row_ok) {
                    store16_bf16(dk + col, rk);
                    store16_bf16(dv + col, rv);
                }
            }
        }
    }
    if constexpr (HS == 128) {
        if (parts > 1) {
            // Rows [part * 128 / parts, ...) of dK and dV: the sum over the cluster's CTAs, in the order of their heads
            __syncwarp();
            cluster_arrive();
            cluster_wait();
            if (role < 0) {
                const int row0 = 128 * part / parts, rows = 128 * (part + 1) / parts - row0;
                for (int i = tid; i < rows * 64; i += kBwdComputeThreads) {
                    const int what = (i >> 5) & 1, row = row0 + (i >> 6), c4 = i & 31;       // dK / dV, row, four columns
                    const uint32_t local = smem_u32(sums + what * 128 * 32 + row * 32 + (c4 ^ (row & 31)));
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    for (int q = 0; q < parts; ++q) {
                        const float4 x = ld_cluster_f32x4(map_to_cta(local, q));
                        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
                    }
                    if (ok && kv0 + row < p.T) {
                        bf16* dst = p.dqkv + ((static_cast<long long>(b) * p.T + kv0 + row) * (p.Hq + 2 * p.Hkv)) * HS + (what == 0 ? kcol : vcol) + 4 * c4;
                        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
                    }
                }
            }
            __syncwarp();
            cluster_arrive();                                 // the others may still read this CTA's sums
            cluster_wait();
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (role == 0) tmem_dealloc(tmem, TMEM_COLS);
}

// ------------------------------------------------------------------------------------------------
// dQ.  One CTA owns 128 query rows and walks over `heads_per_cta` query heads of one kv head, and for every head over
// the key tiles up to the diagonal.  Q and dO of the current head live in tensor memory as the A operands of the score
// MMAs (they are constant during a key walk), K / V tiles stream through a ring of shared-memory buffers, S / dP are double buffered in
// TMEM, dS takes the place of the dP tile it was computed from (A operand of dQ += dS K), dQ accumulates in TMEM and is drained once
// per head while the scores of the next head's first tiles are computed.
template <int HS>
struct DqShape {
    static constexpr int NBUF = HS == 64 ? 6 : 4;
    static constexpr int KV_BYTES = 64 * HS * 2, Q_BYTES = 128 * HS * 2;
    static constexpr int STAT_OFFSET = 2 * NBUF * KV_BYTES + 2 * Q_BYTES;
    static constexpr int SMEM_BYTES = STAT_OFFSET + 128 * 8 + 256;
};

template <int HS, int Phase>
__device__ __forceinline__ void
bwd_dq_block(const CUtensorMap& tmap_qkv64,                          // qkv, box 64 rows (K, V and Q tiles)
             const CUtensorMap& tmap_do64,                           // dO, box 64 rows
             const AttnParams& p, const int heads_per_cta, const int block) {
    constexpr int BQ = 128, BKV = 64, NCH = HS / 64, NBUF = DqShape<HS>::NBUF;
    constexpr int KV_BYTES = DqShape<HS>::KV_BYTES, Q_BYTES = DqShape<HS>::Q_BYTES;
    constexpr uint32_t TMEM_COLS = 512;                       // Q | dO (bf16 pairs, A operands) | S0 S1 | dP0 dP1 | dQ
    constexpr int CW = 16;                                    // columns of one K step of the dQ MMA
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;                       // NBUF buffers
    uint8_t* sV = sK + NBUF * KV_BYTES;       // NBUF buffers
    uint8_t* sQ = sV + NBUF * KV_BYTES;       // Q and dO of the next head, on their way to tensor memory
    uint8_t* sdO = sQ + Q_BYTES;
    float2* sStat = reinterpret_cast<float2*>(smem + DqShape<HS>::STAT_OFFSET);   // (lse * log2(e), delta * softmax scale) of its rows
    uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + BQ);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);       // uniform, and known to be
    const int role = warp - kBwdComputeWarps;                 // 0, 1: MMA issuers (one elected lane); 2: TMA loads of K / V, 3: of Q / dO and row statistics
    const int wg = tid >> 7, r = tid & 127;
    const int nqb = (p.T + BQ - 1) / BQ;
    const int G = p.Hq / p.Hkv;
    const int parts = (G + heads_per_cta - 1) / heads_per_cta;
    const int per_qb = p.Hkv * p.B * parts;
    const int qb = nqb - 1 - block / per_qb;                    // longest key walks first
    const int rest = block % per_qb;
    const int kvh = rest % p.Hkv, b = (rest / p.Hkv) % p.B, part = rest / (p.Hkv * p.B);
    const int h0 = kvh * G + part * heads_per_cta;              // query heads [h0, h0 + nh)
    const int nh = min(heads_per_cta, G - part * heads_per_cta);
    const int q0 = qb * BQ;
    const int n_kv = min((p.T + BKV - 1) / BKV, (q0 + BQ) / BKV);
    const int total = n_kv * nh;                                // tiles of the whole walk, t = g * n_kv + j
    const int kcol = (p.Hq + kvh) * HS, vcol = (p.Hq + p.Hkv + kvh) * HS;

    // barriers: 0 Q of a head in place | 1 dO of a head in place | 2-3 S ready | 4-5 dP ready | 6-7 dS in tensor memory | 8-9 S has been
    //           read | 10 dQ of a head done | 11 dQ of a head drained | 12.. k/v ring | 18.. k/v buffer free | 24 Q / dO of a head staged |
    //           25 staging free.  Two-entry sets alternate with the tile parity.
    const uint32_t bar0 = smem_u32(bars);
    const uint32_t q_ready = bar0, do_ready = bar0 + 8, dq_bar = bar0 + 80, dq_drained = bar0 + 88;
    auto s_bar = [&](int t) { return bar0 + 16 + 8 * (t & 1); };
    auto dp_bar = [&](int t) { return bar0 + 32 + 8 * (t & 1); };
    auto p_ready = [&](int t) { return bar0 + 48 + 8 * (t & 1); };
    auto s_free = [&](int t) { return bar0 + 64 + 8 * (t & 1); };
    auto kv_bar = [&](int buf) { return bar0 + 96 + 8 * buf; };
    auto kv_free = [&](int buf) { return bar0 + 144 + 8 * buf; };
    const uint32_t staged = bar0 + 192, stage_free = bar0 + 200;
    if constexpr (Phase == kBwdSetup) {
        if (tid == 0) {
            mbar_init(q_ready, kBwdGroupWarps); mbar_init(do_ready, kBwdGroupWarps);
            mbar_init(dq_drained, kBwdGroupWarps); mbar_init(dq_bar, 1);
            mbar_init(staged, 2); mbar_init(stage_free, kBwdComputeWarps);
            for (int i = 0; i < NBUF; ++i) { mbar_init(kv_bar(i), 1); mbar_init(kv_free(i), 1); }
            for (int i = 0; i < 2; ++i) { mbar_init(s_bar(i), 1); mbar_init(dp_bar(i), 1); mbar_init(p_ready(i), kBwdGroupWarps); mbar_init(s_free(i), kBwdGroupWarps); }
            *abort_flag = 0;
            mbar_init_fence();
        }
        if (role == 0) { tmem_alloc(smem_u32(tmem_slot), TMEM_COLS); tmem_relinquish(); }
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
        return;
    }
    const uint32_t tmem = *tmem_slot;
    const uint32_t tQ = tmem, tdO = tmem + HS / 2, tdQ = tmem + HS + 4 * BKV;
    auto tS = [&](int t) { return tmem + HS + (t & 1) * BKV; };
    auto tdP = [&](int t) { return tmem + HS + 2 * BKV + (t & 1) * BKV; };
    const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
    bool ok = true;

    if (role == 2) {
        // ============================================================ TMA producer warp
        if ((tid & 31) == 0 && total > 0) {
            tma_prefetch_desc(&tmap_qkv64);
            int j = 0;
            for (int t = 0; t < total; ++t) {
                const int buf = t % NBUF;
                // the buffer's previous tile, t - NBUF, has been consumed by its dQ MMA
                if (t >= NBUF && !mbar_wait(kv_free(buf), ((t / NBUF) - 1) & 1, abort_flag)) { atomicOr(p.status, kErrOther); break; }
                mbar_expect_tx(kv_bar(buf), 2 * KV_BYTES);
                for (int c = 0; c < NCH; ++c) {
                    tma_load_3d(smem_u32(sK) + buf * KV_BYTES + c * (BKV * 128), &tmap_qkv64, kv_bar(buf), kcol + c * 64, j * BKV, b);
                    tma_load_3d(smem_u32(sV) + buf * KV_BYTES + c * (BKV * 128), &tmap_qkv64, kv_bar(buf), vcol + c * 64, j * BKV, b);
                }
                if (++j == n_kv) j = 0;
            }
        }
    } else if (role == 3) {
        // ============================================================ Q / dO of a head at a time, while the head before is worked on
        const int lane = tid & 31;
        if (lane == 0) { tma_prefetch_desc(&tmap_qkv64); tma_prefetch_desc(&tmap_do64); }
        for (int g = 0; g < nh && total > 0; ++g) {
            const int hq = h0 + g;
            float2 st[4];                                       // rows beyond the sequence get probability 0
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int q = q0 + lane + 32 * i;
                const long long si = (static_cast<long long>(b) * p.Hq + hq) * p.T + q;
                st[i] = q < p.T ? make_float2(load_plain(p.lse + si), load_plain(p.delta + si)) : make_float2(INFINITY, 0.f);
            }
            if (g > 0 && !mbar_wait_warp(stage_free, (g - 1) & 1, abort_flag)) { if (lane == 0) atomicOr(p.status, kErrOther); break; }
            if (lane == 0) {
                mbar_expect_tx(staged, 2 * Q_BYTES);
                for (int c = 0; c < NCH; ++c)
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t off = c * (BQ * 128) + h * (64 * 128);
                        tma_load_3d(smem_u32(sQ) + off, &tmap_qkv64, staged, hq * HS + c * 64, q0 + h * 64, b);
                        tma_load_3d(smem_u32(sdO) + off, &tmap_do64, staged, hq * HS + c * 64, q0 + h * 64, b);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) sStat[lane + 32 * i] = make_float2(st[i].x * kLog2e, st[i].y * p.scale);
            warp_arrive(staged);
        }
    } else if (role >= 0) {
        // ============================================================ MMA issuer warps
        // Warp 0 issues S two tiles ahead of the sums (its buffer is free once the scores have been read), across the heads: Q of the next
        // head comes when the last S of the head before is complete.  Warp 1 issues dQ += dS K and then dP two tiles ahead into the buffer
        // of the dS just read; dO of the next head comes after the last dP of a head, so its first tiles follow the head's last sums.
        if (total > 0) {
            const bool leader = elect_one();
            const uint32_t idesc_s = make_instr_desc(1, 1, false, false, BQ, BKV);
            const uint32_t idesc_dq = make_instr_desc(1, 1, false, true, BQ, HS);
            auto scores = [&](uint32_t d, uint32_t a, uint32_t b_lo, uint32_t bar) {
                if (leader) {
#pragma unroll
                    for (int k = 0; k < HS / 16; ++k)
                        mma_issue_f16_tmem_a(d, a + k * 8, b_lo + (((k / 4) * (BKV * 128) + (k % 4) * 32) >> 4), kDescHi, idesc_s, k > 0);
                    mma_commit(bar);
                }
                __syncwarp();
            };
            if (role == 0) {
                const uint32_t k_lo = desc_lo(smem_u32(sK), 16);
                int j = 0, head = 0, buf = 0;
                uint32_t phase = 0;
                for (int t = 0; t < total; ++t) {
                    const bool loaded = mbar_test_wait(kv_bar(buf), phase);
                    if (j == 0) ok = mbar_wait_warp(q_ready, head & 1, abort_flag);
                    if (ok && t >= 2) ok = mbar_wait_warp(s_free(t), ((t - 2) >> 1) & 1, abort_flag);
                    if (ok && !__all_sync(0xffffffffu, loaded)) ok = mbar_wait_warp(kv_bar(buf), phase, abort_flag);
                    if (!ok) break;
                    tc_fence_after_sync();
                    scores(tS(t), tQ, k_lo + buf * (KV_BYTES >> 4), s_bar(t));
                    if (++buf == NBUF) { buf = 0; phase ^= 1u; }
                    if (++j == n_kv) { j = 0; ++head; }
                }
            } else {
                const uint32_t k_lo = desc_lo(smem_u32(sK), BKV * 128), v_lo = desc_lo(smem_u32(sV), 16);
                int dp = 0, dp_buf = 0;                         // next dP tile
                uint32_t dp_phase = 0;
                // dP tiles up to tile `upto`, before tile `end`
                auto issue_dp = [&](int upto, int end, bool loaded) -> bool {
                    for (; dp <= upto && dp < end; ++dp) {
                        if (!__all_sync(0xffffffffu, loaded) && !mbar_wait_warp(kv_bar(dp_buf), dp_phase, abort_flag)) return false;
                        tc_fence_after_sync();
                        scores(tdP(dp), tdO, v_lo + dp_buf * (KV_BYTES >> 4), dp_bar(dp));
                        if (++dp_buf == NBUF) { dp_buf = 0; dp_phase ^= 1u; }
                        loaded = false;
                    }
                    return true;
                };
                ok = mbar_wait_warp(do_ready, 0, abort_flag) && issue_dp(1, n_kv, false);
                int t = 0, buf = 0;
                for (int g = 0; g < nh && ok; ++g) {
                    const int head_end = (g + 1) * n_kv;
                    for (int j = 0; j < n_kv; ++j, ++t) {
                        const bool loaded = t + 2 < head_end && mbar_test_wait(kv_bar(dp_buf), dp_phase);
                        if (!mbar_wait_warp(p_ready(t), (t >> 1) & 1, abort_flag)) { ok = false; break; }
                        // the first dQ MMA of a head overwrites the accumulator: the previous head's must have been read
                        if (j == 0 && g > 0 && !mbar_wait_warp(dq_drained, (g - 1) & 1, abort_flag)) { ok = false; break; }
                        tc_fence_after_sync();
                        const uint32_t b_lo = k_lo + buf * (KV_BYTES >> 4), dp_t = tdP(t), bar = kv_free(buf);
                        const uint32_t acc0 = j > 0;
                        if (leader) {
#pragma unroll
                            for (int k = 0; k < BKV / 16; ++k)
                                mma_issue_f16_tmem_a(tdQ, dp_t + k * CW, b_lo + ((k * (16 * 128)) >> 4), kDescHi, idesc_dq, k > 0 ? 1u : acc0);
                            mma_commit(bar);
                        }
                        __syncwarp();
                        if (++buf == NBUF) buf = 0;
                        if (!issue_dp(t + 2, head_end, loaded)) { ok = false; break; }
                    }
                    if (!ok) break;
                    if (leader) mma_commit(dq_bar);
                    __syncwarp();
                    if (g + 1 < nh) ok = mbar_wait_warp(do_ready, (g + 1) & 1, abort_flag) && issue_dp(t + 1, head_end + n_kv, false);
                }
            }
            if (!ok && leader) { *abort_flag = 1u; atomicOr(p.status, kErrOther); }
            __syncwarp();
        }
    } else {
        // ============================================================ compute warps
        // Two groups of two warpgroups take turns: group g works on the tiles of parity g, a thread on 32 columns of its row.
        const float sl2 = p.scale * kLog2e;
        const int row = q0 + r;
        const bool row_ok = row < p.T;
        const int grp = wg >> 1, c0 = (wg & 1) * 2 * CW;
        const int H = p.Hq + 2 * p.Hkv;
        constexpr int ECW = HS / 2;                             // dQ columns per thread
        // Q and dO of head g are moved to tensor memory by one group each: dO by the group of the last tile before the head, Q by the other
        // one, which is through with its last tile earlier.  A thread moves half a row, and reads the statistics of its row.
        auto writes_do = [&](int g) { return ((g * n_kv - 1) & 1) == grp; };
        float lse2 = 0.f, delta_s = 0.f;
        auto move_half_row = [&](int g) -> bool {
            if (!mbar_wait(staged, g & 1, abort_flag)) return false;
            const bool is_do = writes_do(g);
            const uint8_t* src = (is_do ? sdO : sQ) + r * 128;
#pragma unroll
            for (int c = 0; c < HS / 64; ++c) {                 // 32 elements: four 16-byte pieces, swizzled
                const int e = (wg & 1) * (HS / 2) + c * 32;     // first element
                uint32_t w[16];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint4 x = *reinterpret_cast<const uint4*>(src + (e / 64) * (BQ * 128) + ((((e % 64) / 8 + i) ^ (r & 7)) << 4));
                    w[4 * i] = x.x; w[4 * i + 1] = x.y; w[4 * i + 2] = x.z; w[4 * i + 3] = x.w;
                }
                __syncwarp();
                tmem_st_32x32b_x16((is_do ? tdO : tQ) + lane_off + e / 2, w);
            }
            const float2 st = sStat[r];
            lse2 = st.x; delta_s = st.y;
            tmem_st_wait();
            tc_fence_before_sync();
            warp_arrive(is_do ? do_ready : q_ready);
            warp_arrive(stage_free);
            return true;
        };
        ok = total > 0 && move_half_row(0);
        for (int g = 0; g < nh && ok; ++g) {
            const int t0 = g * n_kv;
            for (int j = (t0 & 1) ^ grp; j < n_kv; j += 2) {
                const int t = t0 + j;
                if (!mbar_wait(s_bar(t), (t >> 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after_sync();
                float pv[2][CW];
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h) tmem_ld_32x32b_x16(tS(t) + lane_off + c0 + h * CW, *reinterpret_cast<uint32_t(*)[CW]>(pv[h]));
                tmem_ld_wait();
                tc_fence_before_sync();
                warp_arrive(s_free(t));
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int i = 0; i < CW; ++i) pv[h][i] = fast_exp2(fmaf(pv[h][i], sl2, -lse2));
                if ((j + 1) * BKV > q0) {
                    const int lim = row - j * BKV - c0;         // columns above lim are beyond the diagonal (kv > q)
#pragma unroll
                    for (int h = 0; h < 2; ++h)
#pragma unroll
                        for (int i = 0; i < CW; ++i) if (h * CW + i > lim) pv[h][i] = 0.f;
                }
                if (!mbar_wait(dp_bar(t), (t >> 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after_sync();
                __syncwarp();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t rv[CW], dsp[CW / 2];
                    tmem_ld_32x32b_x16(tdP(t) + lane_off + c0 + h * CW, rv);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < CW; i += 2)
                        dsp[i / 2] = pack_bf16x2(pv[h][i] * fmaf(__uint_as_float(rv[i]), p.scale, -delta_s),
                                                 pv[h][i + 1] * fmaf(__uint_as_float(rv[i + 1]), p.scale, -delta_s));
                    // into the first half of the 16 columns this thread has just read: one K step of the dQ MMA
                    tmem_st_32x32b_x8(tdP(t) + lane_off + c0 + h * CW, dsp);
                }
                tmem_st_wait();
                tc_fence_before_sync();
                warp_arrive(p_ready(t));
            }
            if (!ok) break;
            // ---- this group's part of the head's walk is over.  Q / dO of the next head may be written once the last MMA that reads this
            // head's is complete: the last S tile (the other group's, waited for here) for Q, the last dP tile for dO.
            if (g + 1 < nh) {
                const int tl = t0 + n_kv - 1;
                if (!mbar_wait(writes_do(g + 1) ? dp_bar(tl) : s_bar(tl), (tl >> 1) & 1, abort_flag)) { ok = false; break; }
                tc_fence_after_sync();
                if (!move_half_row(g + 1)) { ok = false; break; }
            }
            // Then the group of the last tile drains dQ; the other one is already at the next head's first tile.
            if (!writes_do(g + 1)) continue;
            if (!mbar_wait(dq_bar, g & 1, abort_flag)) { ok = false; break; }
            tc_fence_after_sync();
            bf16* dq = p.dqkv + ((static_cast<long long>(b) * p.T + row) * H + h0 + g) * HS + (wg & 1) * ECW;
            __syncwarp();
#pragma unroll
            for (int c = 0; c < ECW; c += 32) {
                uint32_t acc[32];
                tmem_ld_32x32b_x32(tdQ + lane_off + (wg & 1) * ECW + c, acc);
                tmem_ld_wait();
                if (c + 32 == ECW) {
                    tc_fence_before_sync();
                    warp_arrive(dq_drained);
                }
                if (row_ok) {
                    store16_bf16(dq + c, *reinterpret_cast<const uint32_t(*)[16]>(acc));
                    store16_bf16(dq + c + 16, *reinterpret_cast<const uint32_t(*)[16]>(acc + 16));
                }
            }
        }
        if (!ok && r == 0) atomicOr(p.status, kErrOther);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (role == 0) tmem_dealloc(tmem, TMEM_COLS);
}

// Blocks [0, n_dkdv) are the dK / dV CTAs, clusters of `parts`; the n_dq blocks behind them are the dQ CTAs, the last cluster filled up with idle ones.
template <int HS>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_kv128, const __grid_constant__ CUtensorMap tmap_qkv64,
                const __grid_constant__ CUtensorMap tmap_do64, const AttnParams p, const int parts, const int n_dkdv, const int heads_per_cta,
                const int n_dq) {
    extern __shared__ __align__(1024) uint8_t smem[];
    if (smem_u32(smem) & 1023u) { if (threadIdx.x == 0) atomicOr(p.status, kErrOther); return; }
    const int block = static_cast<int>(blockIdx.x);
    if (block >= n_dkdv + n_dq) return;
    const bool dkdv = block < n_dkdv;
    if (dkdv) bwd_dkdv_block<HS, kBwdSetup>(tmap_kv128, tmap_qkv64, tmap_do64, p, parts, block);
    else      bwd_dq_block<HS, kBwdSetup>(tmap_qkv64, tmap_do64, p, heads_per_cta, block - n_dkdv);
    grid_release();
    grid_wait();
    if (dkdv) bwd_dkdv_block<HS, kBwdRun>(tmap_kv128, tmap_qkv64, tmap_do64, p, parts, block);
    else      bwd_dq_block<HS, kBwdRun>(tmap_qkv64, tmap_do64, p, heads_per_cta, block - n_dkdv);
}

// Tag makes the static flag unique per kernel instantiation (several kernels share one signature).
template <int Tag, typename K>
int set_smem(K kernel, int bytes) {
    static bool done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!done[dev & 63]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return 2000 + static_cast<int>(e);
        done[dev & 63] = true;
    }
    return 0;
}

template <int HS>
constexpr int bwd_smem() {
    return one_block_per_sm(DkdvShape<HS>::SMEM_BYTES > DqShape<HS>::SMEM_BYTES ? DkdvShape<HS>::SMEM_BYTES : DqShape<HS>::SMEM_BYTES);
}

// Query heads of a group that a dQ CTA walks over; `base` = (query block, kv head, batch) items.  A CTA that walks a whole group pays its
// start-up once, but few items leave SMs idle: the group is cut into the fewest parts that give 1.5 CTAs per SM.  Heads do not share
// sums, so the results do not depend on the cut.
int dq_heads(int G, int base) {
    int heads = G;
    for (int parts = 1; parts <= G; ++parts) {
        heads = (G + parts - 1) / parts;
        if (2 * base * ((G + heads - 1) / heads) >= 3 * device_sms()) break;
    }
    return heads;
}

// Clusters of `parts` CTAs (plain CTAs for one) that reside at once
template <int HS>
int resident_clusters(int parts, int smem) {
    static int known[64][9] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    int& n = known[dev & 63][parts];
    if (n > 0) return n;
    int found = device_sms();
    if (parts > 1) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = device_sms() * parts; cfg.blockDim = kBwdThreads; cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1]{};
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = parts; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&found, attn_bwd_kernel<HS>, &cfg) != cudaSuccess) { cudaGetLastError(); return 0; }
    }
    return n = found;
}

// How the query heads of a group are shared out.  dkdv: CTAs of one cluster that share the heads of a dK / dV item (key block, kv head, batch); they
// add their sums up through distributed shared memory, in the order of the heads.  dq: heads that a dQ CTA walks over.
struct HeadSplit {
    int dkdv, dq;
};

// With head size 64 the sum over the heads stays in one accumulator, so that its results keep their bits, and the dQ CTAs follow dq_heads (within 0.3 % of the best
// cut over 20 shapes).  With head size 128 the pair is the one with the smallest estimate, in us: a dK / dV CTA costs 5, with a cluster 2 + 0.5
// per part more for its sums, 0.25 a head and 0.85 a tile; a dQ CTA 4.2, 1.7 a head (Q and dO in, dQ out) and 0.6 a tile; all of them together take the longest CTA
// or, if that is longer and they do not all reside at once, the average of the resident CTAs and half a CTA behind it (clusters do not fill the SMs:
// of 7 CTAs 15 reside, of 2 74).  Over 55 shapes (20 to 6731 tokens, 1 to 8 sequences, groups of 1 to 12 heads) the picked pair
// takes 1.03 of the time of the best one on average, the rules for two launches one after the other took 1.10.  attention_backward, us, with those / picked:
// 1 x 1024 tokens, 32 / 8 heads 58 / 42;  6 x 405, 12 / 2 35 / 31;  2 x 683, 28 / 4 58 / 44;  3 x 2048, 28 / 4 312 / 284;  4 x 1024, 16 / 2 86 / 70.
// For sequences of one key block, whose few tiles the estimate of a tile says little about (7 x 33 tokens, 12 / 2 heads 10.7 by the rules for two launches, 12.0 by the estimate), those rules
// stay unless the estimate of what they give is 1.45 times that of the best pair; over 19 such shapes that takes 1.04 of the best one. Both:  8 x 100, 32 / 8 30 / 21, 12 x 128, 28 / 4 34.5 / 24.3,
// 9 x 16, 28 / 4 16.1 / 12.3.
template <int HS>
HeadSplit split_heads(int G, int base, int T, int smem) {
    const int heads_rule = dq_heads(G, base);
    if constexpr (HS == 64) return {1, heads_rule};
    const int nqb = (T + 63) / 64, nkb = (T + 127) / 128;
    const double mean_tiles = nqb - (nkb - 1);               // query blocks at or below the diagonal, mean over the key blocks
    const auto estimate = [&](int parts, int dq, int resident) {
        const int heads = (G + parts - 1) / parts, cut = (G + dq - 1) / dq;              // dQ CTAs of an item
        const double sums = parts > 1 ? 2. + 0.5 * parts : 0.;
        const double longest_dkdv = 5. + sums + heads * (0.25 + 0.85 * nqb), longest_dq = 4.2 + dq * (1.7 + 0.6 * nqb);
        const double us = longest_dkdv > longest_dq ? longest_dkdv : longest_dq;
        const double ctas = static_cast<double>(base) * (parts + cut), at_once = static_cast<double>(resident) * parts;
        if (ctas <= at_once) return us;
        const double work = base * (parts * (5. + sums) + G * (0.25 + 0.85 * mean_tiles) + cut * 4.2 + G * (1.7 + 0.6 * (nkb + 1)));
        const double mean = work / ctas, shared = work / at_once + 0.5 * (us < mean ? us : mean);
        return shared > us ? shared : us;
    };
    HeadSplit best{1, heads_rule}, rule{1, heads_rule};      // rule: that of two launches, which looks at dK / dV alone
    double best_us = 0., rule_us = 0., rule_estimate = 0.;
    for (int parts = 1; parts <= 8 && parts <= G; ++parts) {
        const int resident = resident_clusters<HS>(parts, smem);
        if (resident <= 0) continue;
        for (int dq = G; dq >= 1; --dq) {
            if (dq > 1 && (G + dq - 2) / (dq - 1) == (G + dq - 1) / dq) continue;        // the smallest `dq` of every cut is looked at
            const double us = estimate(parts, dq, resident);
            if (best_us == 0. || us < best_us) { best = {parts, dq}; best_us = us; }
        }
        const int heads = (G + parts - 1) / parts;
        const double rounds = (base + resident - 1) / resident, longest = static_cast<double>(nqb) * heads, average = mean_tiles * heads * base / resident;
        const double us = rounds * (5. + (parts > 1 ? 2. + 0.6 * parts : 0.)) + 0.9 * (longest > average ? longest : average);
        if (rule_us == 0. || us < rule_us) { rule_us = us; rule.dkdv = parts; rule_estimate = estimate(parts, heads_rule, resident); }
    }
    return nkb == 1 && rule_estimate <= 1.45 * best_us ? rule : best;
}

template <int HS>
int bwd_impl(void* dqkv, float* delta, const void* d_out, const void* out, const float* lse, const void* qkv, int B, int T,
             int Hq, int Hkv, unsigned int* status, cudaStream_t s) {
    const int H = Hq + 2 * Hkv;
    {
        long long rows = static_cast<long long>(B) * T * Hq;
        long long blocks = (rows * (HS / 8) + 255) / 256;
        launch_chained(attn_delta_kernel<HS>, static_cast<unsigned int>(blocks), 256, 0, s, delta, static_cast<const bf16*>(out), static_cast<const bf16*>(d_out), B, T, Hq);
        int rc = LLMQ_LAUNCH_CHECK();
        if (rc) return rc;
    }
    CUtensorMap t128, t64, tdo64;
    int rc = encode_btw(&t128, qkv, B, T, static_cast<long long>(H) * HS, 128);
    if (!rc) rc = encode_btw(&t64, qkv, B, T, static_cast<long long>(H) * HS, 64);
    if (!rc) rc = encode_btw(&tdo64, d_out, B, T, static_cast<long long>(Hq) * HS, 64);
    if (rc) return rc;
    AttnParams p{};
    p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.scale = 1.f / sqrtf(static_cast<float>(HS));
    p.lse = const_cast<float*>(lse); p.delta = delta; p.dqkv = static_cast<bf16*>(dqkv); p.status = status;
    p.qkv = static_cast<const bf16*>(qkv);
    const int base = ((T + 127) / 128) * Hkv * B, G = Hq / Hkv;
    constexpr int smem = bwd_smem<HS>();
    rc = set_smem<1000 + HS>(attn_bwd_kernel<HS>, smem);
    if (rc) return rc;
    const HeadSplit split = split_heads<HS>(G, base, T, smem);
    const int parts = split.dkdv, n_dkdv = base * parts, n_dq = base * ((G + split.dq - 1) / split.dq);
    launch_chained_cluster(attn_bwd_kernel<HS>, n_dkdv + (n_dq + parts - 1) / parts * parts, kBwdThreads, smem, s, parts, t128, t64, tdo64, p, parts,
                           n_dkdv, split.dq, n_dq);
    rc = LLMQ_LAUNCH_CHECK();
    return rc;
}

}  // namespace

int llmq_attention_forward_pingpong(void* out, float* lse, const void* qkv, int B, int T, int Hq, int Hkv, int HS, float* absmax,
                                    unsigned int* status, cudaStream_t s);

// qkv (B,T,Hq+2Hkv,HS) bf16 -> out (B,T,Hq,HS) bf16, lse (B,Hq,T) fp32.  HS in {64, 128}.
// absmax (optional): atomic maximum of |out|, for the fp8 quantisation of the output.
extern "C" int llmq_attention_forward(void* out, float* lse, const void* qkv, int B, int T, int Hq, int Hkv, int HS,
                                      float* absmax, unsigned int* status, cudaStream_t s) {
    if (B <= 0 || T <= 0) return 0;
    if (Hq % Hkv) return -1;
    if (HS == 64 || HS == 128) return llmq_attention_forward_pingpong(out, lse, qkv, B, T, Hq, Hkv, HS, absmax, status, s);
    return -2;
}

// CTAs that share the query heads of a dK / dV item in llmq_attention_backward of this shape; negative: an error of the runtime
extern "C" int llmq_attention_dkdv_parts(int B, int T, int Hq, int Hkv, int HS) {
    if (HS != 128) return 1;
    constexpr int smem = bwd_smem<128>();
    const int rc = set_smem<1000 + 128>(attn_bwd_kernel<128>, smem);
    return rc ? -rc : split_heads<128>(Hq / Hkv, ((T + 127) / 128) * Hkv * B, T, smem).dkdv;
}

// dqkv (B,T,Hq+2Hkv,HS) is fully overwritten.  delta is scratch of B*Hq*T floats.
extern "C" int llmq_attention_backward(void* dqkv, float* delta, const void* d_out, const void* out, const float* lse,
                                       const void* qkv, int B, int T, int Hq, int Hkv, int HS, unsigned int* status,
                                       cudaStream_t s) {
    if (B <= 0 || T <= 0) return 0;
    if (Hq % Hkv) return -1;
    if (HS == 64) return bwd_impl<64>(dqkv, delta, d_out, out, lse, qkv, B, T, Hq, Hkv, status, s);
    if (HS == 128) return bwd_impl<128>(dqkv, delta, d_out, out, lse, qkv, B, T, Hq, Hkv, status, s);
    return -2;
}
