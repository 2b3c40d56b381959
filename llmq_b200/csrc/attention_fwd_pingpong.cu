// Causal grouped-query flash attention forward (head sizes 64 and 128): two query tiles per CTA, processed alternately.
//
// A CTA owns 256 consecutive queries of one (batch, query head) as two 128-row tiles A and B.  Each tile has its own
// softmax warpgroup (thread r owns row r = TMEM lane r and sees the whole 128-key score row, so the row maximum and the
// row sum need no exchange between threads), its own MMA-issuing thread and its own tensor-memory columns:
//
//     columns   0..127  S_A   (fp32 scores of the current key tile; the bf16 probabilities P_A overwrite columns 0..63)
//     columns 128..255  S_B
//     columns 256 ..    O_A   (fp32 output accumulator, head size columns)
//     then              O_B
//
// Per 128-key tile j and query tile X the chain is  S_X = Q_X K_j^T  ->  softmax warpgroup X: max, exp2, bf16, P_X into
// tensor memory (handed over in two halves of 64 keys)  ->  O_X += P_X V_j (P is the A operand straight from tensor memory).  The two chains are independent,
// so while one tile's warpgroup computes exponentials the tensor core runs the other tile's MMAs.  us, where the 168 registers of an even split made the
// score rows spill (which waits for the L1) and the output left in 16-byte stores, each an access of its own / now:  8 x 2048 tokens, 28 / 4 heads of
// 128 274 / 238 (clock counters: 6000 cycles from the end of a walk to the next item, 2500 now),  1 x 8192, 32 / 8 of 128 471 / 454,  8 x 1024, 14 / 2
// of 64 39.1 / 33.2,  1 x 8192, 32 / 8 of 64 412 / 385,  1 x 333, 12 / 2 of 128 12.4 / 8.8.  A tile takes 3800 cycles at head size 128 (1600 of them
// exponentials, 1100 from P to the next scores, 500 the maximum) and two tiles are under way; 3200 at head size 64, bound by the exponentials of both.
// K and V tiles stream through two (head size 128) or three shared-memory stages each (TMA, 128-byte swizzle); Q_A and Q_B stay in shared memory
// for the whole walk.  O is rescaled only when a row maximum moved by more than 2^8 since the last rescale (the stale
// maximum keeps P <= 256, which is exact after the final normalisation), and then by the row's own thread.
// Every wait is bounded: a wait that runs out sets the CTA's abort flag and the status word and all roles leave.
//
// Takes the place of the cuDNN SDPA forward graph of the reference (src/kernels/cudnn_att.cpp:46-160).
#include "ptx_sm100.cuh"
#include "api.h"
#include "common.cuh"

using namespace sm100;

namespace {

constexpr int BQ = 128;                      // rows per query tile
constexpr int BKV = 128;                     // keys per tile
constexpr int CHUNK_BYTES = 128 * 128;       // 128 rows x 64 columns of a Q, K or V tile; a tile has HS / 64 of them
template <int HS> constexpr int KV_STAGES = HS == 64 ? 3 : 2;
constexpr int NUM_THREADS = 384;             // 4 + 4 softmax warps, TMA producer, MMA issuer A, MMA issuer B, an idle warp
constexpr int SOFTMAX_REGS = 208, OTHER_REGS = 80;        // registers of a thread: 2 x 128 x 208 + 128 x 80 of the 384 x 168 the block starts with
static_assert(256 * SOFTMAX_REGS + 128 * OTHER_REGS <= NUM_THREADS * 168);
constexpr uint32_t TMEM_COLS = 512;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kRescaleThreshold = 8.f;     // in log2 units

struct FwdParams {
    int B, T, Hq, Hkv;
    float scale;
    int turns;                   // 1: the two softmax warpgroups take turns with their exponentials
    int wide;                    // 1: the output is aligned to 32 bytes
    __nv_bfloat16* out;          // (B, T, Hq, HS)
    float* lse;                  // (B, Hq, T), natural log
    float* absmax;               // optional
    unsigned int* status;
};

// The register count of a warpgroup; executed by all of its warps.  inc waits until the block's other warpgroups have given up as many.
template <int N> __device__ __forceinline__ void set_max_regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void set_max_regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void warp_arrive(uint32_t bar) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
}

// One work item = 256 consecutive queries of one (batch, query head).  Items are numbered with the longest key walks first
// (query block descending); a CTA walks the items  c, 2G-1-c, 2G+c, 4G-1-c, ...  (G = grid size): in every round of G items the
// order of the CTAs flips, which evens out the total walk length per CTA.
// Sequences of up to 128 tokens fill one query tile only.  With more heads than SMs an item is then two query heads of one group, which
// share K and V: tile B holds the next head instead of the next 128 queries.  64 x 64 tokens, 14 / 2 heads of 64: 15.1 us, 22.1 with a head
// per item (17.9 with the former kernel, whose small CTAs shared an SM); 32 x 128, 32 / 8 heads of 128: 22.0 and 36.2 us.  With at most as
// many heads as SMs a head per item is faster or the same (every item is resident at once).  Groups of one head have nothing to pair.
struct Item {
    int h, b, kvh, n_max;
    int row_a, row_b, n_a, n_b;              // first query and number of key tiles of pipeline A's and B's query tile
    __device__ int row(int x) const { return x ? row_b : row_a; }
    __device__ int n(int x) const { return x ? n_b : n_a; }
};
// The later query tile of an item has one key tile more.  Pipeline B takes it in the first item of a CTA that has both, A in the second, and so on: the
// pipelines have walked the same number of tiles after every second item and one is never more than one tile ahead, so they go on in
// turn across the items.  Tiles of neighbouring stages are then walked at once, which takes a third stage: head size 64 only (3 x 700, 32 / 8 heads 20.0 -> 18.8 us, 4 x 1024, 14 / 2
// 20.6 -> 20.1; head size 128, whose stages fill the shared memory, 244 -> 258 us for 8 x 2048, 28 / 4).
struct Order { int items = 0; };             // items with both query tiles so far
__host__ __device__ __forceinline__ int pairs_of_group(const FwdParams& p) { return (p.Hq / p.Hkv + 1) / 2; }
__device__ __forceinline__ int item_of(int it, int cta, int grid) { return it * grid + ((it & 1) ? grid - 1 - cta : cta); }
template <bool PAIRED, bool ALTERNATE>
__device__ __forceinline__ Item decode_item(int item, const FwdParams& p, int nqb, Order& order) {
    Item w;
    if constexpr (PAIRED) {
        const int G = p.Hq / p.Hkv, pairs = pairs_of_group(p);
        const int rem = item % (p.Hkv * pairs);
        w.b = item / (p.Hkv * pairs);
        w.kvh = rem / pairs;
        w.h = w.kvh * G + 2 * (rem % pairs);
        w.row_a = w.row_b = 0;
        w.n_a = w.n_max = 1;
        w.n_b = 2 * (rem % pairs) + 1 < G ? 1 : 0;
        return w;
    }
    const int per_qb = p.Hq * p.B;
    const int qb = nqb - 1 - item / per_qb;
    const int rem = item % per_qb;
    w.h = rem % p.Hq;
    w.b = rem / p.Hq;
    w.kvh = w.h / (p.Hq / p.Hkv);
    // key tiles each query tile walks over: everything up to and including its diagonal tile.  Only the last query block of a sequence, whose
    // items come first, may lack its second tile.
    const int q0 = qb * 2 * BQ, n0 = 2 * qb + 1, n1 = q0 + BQ < p.T ? n0 + 1 : 0;
    const bool swap = ALTERNATE && n1 > 0 && (order.items & 1);
    w.row_a = swap ? q0 + BQ : q0; w.row_b = swap ? q0 : q0 + BQ;
    w.n_a = swap ? n1 : n0;        w.n_b = swap ? n0 : n1;
    w.n_max = max(n0, n1);
    order.items += n1 > 0;
    return w;
}

// Persistent: one CTA per SM walks its items with every pipeline running across the item boundary.  The producer loads the
// next item's Q tiles as soon as the last score MMAs of the current item have read them and keeps the K / V stages rolling;
// an issuer starts the next item's first score tile while the softmax warpgroup still normalises and stores the current
// item's rows (it only has to wait for that before the first P V product overwrites O); tile A moves on to the next item
// while tile B walks its extra key tile.  All barrier phases are counted over the whole kernel.
template <int HS, bool PAIRED>
__global__ void __launch_bounds__(NUM_THREADS, 1)
attn_fwd_pingpong_kernel(const __grid_constant__ CUtensorMap tmap_qkv,     // qkv as (B, T, W), box 128 rows x 64 columns
                         const FwdParams p) {
    constexpr int NCH = HS / 64, TILE_BYTES = NCH * CHUNK_BYTES, ST = KV_STAGES<HS>;
    constexpr bool ALTERNATE = HS == 64 && !PAIRED, SPLIT = HS == 64 && !PAIRED;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;                                   // [2 tiles][TILE_BYTES]
    uint8_t* sK = sQ + 2 * TILE_BYTES;                    // [ST][TILE_BYTES]
    uint8_t* sV = sK + ST * TILE_BYTES;                  // [ST][TILE_BYTES]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + ST * TILE_BYTES);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 28);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;       // warp: uniform, and known to be
    if (smem_u32(smem) & 1023u) { if (tid == 0) atomicOr(p.status, kErrOther); return; }

    const int nqb = (p.T + 2 * BQ - 1) / (2 * BQ);
    const int total = PAIRED ? pairs_of_group(p) * p.Hkv * p.B : nqb * p.Hq * p.B;
    const int cta = blockIdx.x, grid = gridDim.x;

    // barriers: 0-1 q_full[X] | 2-3 q_empty[X] | 4-5 s_full[X] | 6-7 p_ready[X] (first 64 keys) | 8-9 p_ready2[X] (second 64 keys) | 10-11 o_done[X]
    //           | 12-13 turn[X] (the exponentials of X may start) | 14-15 o_free[X] (the rows of X's previous item are stored, O may be overwritten)
    //           | 16-18 k_full | 19-21 k_empty | 22-24 v_full | 25-27 v_empty.
    //           A waiter can be at most one completed phase behind on every barrier, so the parity test stays unambiguous.
    const uint32_t bar0 = smem_u32(bars);
    auto q_full = [&](int x) { return bar0 + 8u * x; };
    auto q_empty = [&](int x) { return bar0 + 8u * (2 + x); };
    auto s_full = [&](int x) { return bar0 + 8u * (4 + x); };
    auto p_ready = [&](int x) { return bar0 + 8u * (6 + x); };
    auto p_ready2 = [&](int x) { return bar0 + 8u * (8 + x); };
    auto o_done = [&](int x) { return bar0 + 8u * (10 + x); };
    auto turn = [&](int x) { return bar0 + 8u * (12 + x); };
    auto o_free = [&](int x) { return bar0 + 8u * (14 + x); };
    auto k_full = [&](int s) { return bar0 + 8u * (16 + s); };
    auto k_empty = [&](int s) { return bar0 + 8u * (19 + s); };
    auto v_full = [&](int s) { return bar0 + 8u * (22 + s); };
    auto v_empty = [&](int s) { return bar0 + 8u * (25 + s); };
    if (tid == 0) {
        for (int s = 0; s < 3; ++s) {
            mbar_init(k_full(s), 1); mbar_init(v_full(s), 1);
            mbar_init(k_empty(s), 2); mbar_init(v_empty(s), 2);          // both issuers, every key tile (used or not)
        }
        for (int x = 0; x < 2; ++x) {
            mbar_init(q_full(x), 1); mbar_init(q_empty(x), 1);
            mbar_init(s_full(x), 1); mbar_init(p_ready(x), 4); mbar_init(p_ready2(x), 4); mbar_init(o_done(x), 1);
            mbar_init(turn(x), 4); mbar_init(o_free(x), 4);
        }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 8) { tmem_alloc(smem_u32(tmem_slot), TMEM_COLS); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;
    grid_release();
    grid_wait();

    if (warp >= 8) {
    set_max_regs_dec<OTHER_REGS>();
    if (warp == 8) {
        // ============================================================ TMA producer
        if (lane == 0) {
            tma_prefetch_desc(&tmap_qkv);
            uint32_t kv = 0, walks_a = 0, walks_b = 0;       // K / V stage fills and Q tiles so far
            Order order;
            bool ok = true;
            for (int it = 0; ok; ++it) {
                const int item = item_of(it, cta, grid);
                if (item >= total) break;
                const Item w = decode_item<PAIRED, ALTERNATE>(item, p, nqb, order);
                const int qcol = w.h * HS, kcol = (p.Hq + w.kvh) * HS, vcol = (p.Hq + p.Hkv + w.kvh) * HS;
                auto load_q = [&](int x, uint32_t& walks) {
                    if (w.n(x) == 0) return true;
                    if (walks > 0 && !mbar_wait(q_empty(x), (walks - 1) & 1, abort_flag)) return false;
                    ++walks;
                    mbar_expect_tx(q_full(x), TILE_BYTES);
                    for (int c = 0; c < NCH; ++c)
                        tma_load_3d(smem_u32(sQ) + x * TILE_BYTES + c * CHUNK_BYTES, &tmap_qkv, q_full(x), qcol + (PAIRED ? x * HS : 0) + c * 64, w.row(x), w.b);
                    return true;
                };
                // A is the first to leave an item: its query tile, then the first key tile, then B's query tile
                if (!load_q(0, walks_a)) { ok = false; break; }
                for (int j = 0; j < w.n_max; ++j, ++kv) {
                    const int st = kv % ST;
                    const uint32_t par = ((kv / ST) - 1) & 1;
                    if (kv >= ST && !mbar_wait(k_empty(st), par, abort_flag)) { ok = false; break; }
                    mbar_expect_tx(k_full(st), TILE_BYTES);
                    for (int c = 0; c < NCH; ++c)
                        tma_load_3d(smem_u32(sK) + st * TILE_BYTES + c * CHUNK_BYTES, &tmap_qkv, k_full(st), kcol + c * 64, j * BKV, w.b);
                    if (kv >= ST && !mbar_wait(v_empty(st), par, abort_flag)) { ok = false; break; }
                    mbar_expect_tx(v_full(st), TILE_BYTES);
                    for (int c = 0; c < NCH; ++c)
                        tma_load_3d(smem_u32(sV) + st * TILE_BYTES + c * CHUNK_BYTES, &tmap_qkv, v_full(st), vcol + c * 64, j * BKV, w.b);
                    if (j == 0 && !load_q(1, walks_b)) { ok = false; break; }
                }
            }
            if (!ok) { *abort_flag = 1u; atomicOr(p.status, kErrOther); }
        }
    } else if (warp < 11) {
        // ============================================================ MMA issuer of query tile x
        const int x = warp - 9;
        {
            const bool leader = elect_one();
            const uint32_t idesc_s = make_instr_desc(1, 1, false, false, BQ, BKV);       // S = Q K^T
            const uint32_t idesc_o = make_instr_desc(1, 1, false, true, BQ, HS);         // O += P V  (V read as MN-major B)
            const uint32_t hi = desc_hi(1024);
            const uint32_t tS = tmem + x * BKV, tO = tmem + 2 * BKV + x * HS;
            const uint32_t q_lo = desc_lo(smem_u32(sQ) + x * TILE_BYTES, 16);
            const uint32_t idesc_half = make_instr_desc(1, 1, false, false, BQ, BKV / 2);
            // scores of the keys from `key` on, as many as idesc says
            auto scores = [&](int st, int key, uint32_t idesc) {
                const uint32_t k_lo = desc_lo(smem_u32(sK) + st * TILE_BYTES + key * 128, 16);
#pragma unroll
                for (int k = 0; k < HS / 16; ++k)
                    mma_issue<0, false>(tS + key, q_lo + (((k / 4) * CHUNK_BYTES + (k % 4) * 32) >> 4), hi, k_lo + (((k / 4) * CHUNK_BYTES + (k % 4) * 32) >> 4), hi, idesc, k > 0);
            };
            uint32_t kv = 0, tiles = 0, walks = 0;           // stage uses, key tiles of this query tile, items in which it had any
            Order order;
            bool ok = true;
            for (int it = 0; ok; ++it) {
                const int item = item_of(it, cta, grid);
                if (item >= total) break;
                const Item w = decode_item<PAIRED, ALTERNATE>(item, p, nqb, order);
                const int n = w.n(x);
                if (n > 0 && !mbar_wait_warp(q_full(x), walks & 1, abort_flag)) { ok = false; break; }
                for (int j = 0; j < n && ok; ++j, ++kv, ++tiles) {
                    const int st = kv % ST;
                    const uint32_t par = (kv / ST) & 1;
                    if (j == 0 || !SPLIT) {
                        if (!mbar_wait_warp(k_full(st), par, abort_flag)) { ok = false; break; }
                        tc_fence_after_sync();
                    }
                    const uint32_t ke = k_empty(st);
                    const bool last = j == n - 1;
                    if (leader) {
                        if (j == 0 || !SPLIT) scores(st, 0, idesc_s);
                        else                  scores(st, 0, idesc_half);         // the other keys were issued during the previous tile
                        mma_commit(s_full(x));
                        mma_commit(ke);
                        if (last) mma_commit(q_empty(x));        // the item's last read of this Q tile
                    }
                    __syncwarp();
                    if (!mbar_wait_warp(v_full(st), par, abort_flag)) { ok = false; break; }
                    // the first product of an item overwrites O: the warpgroup must have stored the previous item's rows
                    if (j == 0 && walks > 0 && !mbar_wait_warp(o_free(x), (walks - 1) & 1, abort_flag)) { ok = false; break; }
                    const uint32_t v_lo = desc_lo(smem_u32(sV) + st * TILE_BYTES, CHUNK_BYTES), ve = v_empty(st);
                    const uint32_t acc0 = j > 0;
                    // P arrives in two halves of 64 keys (a barrier each): the first half's MMAs run while the warpgroup still
                    // exponentiates the second half
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        if (!mbar_wait_warp(half == 0 ? p_ready(x) : p_ready2(x), tiles & 1, abort_flag)) { ok = false; break; }
                        tc_fence_after_sync();
                        if (leader) {
#pragma unroll
                            for (int k = half * 4; k < half * 4 + 4; ++k)
                                mma_issue_f16_tmem_a(tO, tS + k * 8, v_lo + ((k * (16 * 128)) >> 4), hi, idesc_o, k > 0 ? 1u : acc0);
                            if (half == 1) { mma_commit(o_done(x)); mma_commit(ve); }
                        }
                        __syncwarp();
                        // The first half of P is there, so the score row has been read: the scores of the next tile's last 64 keys, whose columns P does not
                        // use, need not wait for this tile's products.  Head size 64: 1 x 8192, 32 / 8 heads 392 -> 385 us.  Head size 128, where products
                        // of 64 columns take more than half the time of 128: 239 -> 241 us for 8 x 2048, 28 / 4.
                        if (SPLIT && half == 0 && j + 1 < n) {
                            const int next = (kv + 1) % ST;
                            if (!mbar_wait_warp(k_full(next), ((kv + 1) / ST) & 1, abort_flag)) { ok = false; break; }
                            tc_fence_after_sync();
                            if (leader) scores(next, BKV / 2, idesc_half);
                            __syncwarp();
                        }
                    }
                    if (!ok) break;
                }
                // the other tile may walk further: its stages still need this tile's arrival (wait for the stage's load first:
                // it is only issued once the stage's previous use was released by both tiles, so this arrival cannot be counted
                // towards that earlier phase)
                for (int j = n; j < w.n_max && ok; ++j, ++kv) {
                    const int st = kv % ST;
                    const uint32_t par = (kv / ST) & 1;
                    if (!mbar_wait_warp(k_full(st), par, abort_flag)) { ok = false; break; }
                    if (leader) mbar_arrive(k_empty(st));
                    if (!mbar_wait_warp(v_full(st), par, abort_flag)) { ok = false; break; }
                    if (leader) mbar_arrive(v_empty(st));
                }
                if (n > 0) ++walks;
            }
            if (!ok && leader) { *abort_flag = 1u; atomicOr(p.status, kErrOther); }
            __syncwarp();
        }
    }
    } else {
        set_max_regs_inc<SOFTMAX_REGS>();
        // ============================================================ softmax warpgroup of query tile x
        const int x = warp >> 2;
        const int r = tid & 127;
        const uint32_t lane_off = static_cast<uint32_t>((warp & 3) * 32) << 16;
        const uint32_t tS = tmem + x * BKV + lane_off, tO = tmem + 2 * BKV + x * HS + lane_off;
        const float sl2 = p.scale * kLog2e;
        float omax = 0.f;
        uint32_t tiles = 0, turns = 0;                       // key tiles of this query tile so far; those in turn with the other tile's
        Order order;
        bool ok = true;
        for (int it = 0; ok; ++it) {
            const int item = item_of(it, cta, grid);
            if (item >= total) break;
            const Item w = decode_item<PAIRED, ALTERNATE>(item, p, nqb, order);
            const int n = w.n(x);
            const int q0 = w.row(x), h = w.h + (PAIRED ? x : 0), b = w.b;
            const int row = q0 + r;
            const bool row_ok = row < p.T;
            // The two warpgroups take turns with their exponentials: a warp alone on its SM sub-partition keeps the MUFU unit nearly busy, two at once
            // halve each other's rate and then wait for the tensor pipe together (1 x 8192, 32 / 8 heads of 64: 493 us without turns).  A goes first.
            // A warpgroup hands the turn over when its exponentials are issued, at head size 64, where the exponentials are the bound, before the last 32 keys:
            // that covers the way through the barrier (388 us, 404 after the last; at head size 128 464, 454 after the last).  A's k-th wait (k >= 1) consumes
            // B's arrival k-1, B's k-th wait A's arrival k.  With the extra tiles alternating (see Order) every tile has its turn, across the items; only the
            // very last one of B may have no partner.  Otherwise the tiles of an item that both walk do.
            const bool both = p.turns && w.n_a > 0 && w.n_b > 0;
            const int n_turn = !both ? 0 : ALTERNATE ? n : min(w.n_a, w.n_b);
            const bool alone = ALTERNATE && w.n_b > w.n_a && item_of(it + 1, cta, grid) >= total;
            float m_ref = -INFINITY, l_sum = 0.f, l4[4] = {0.f, 0.f, 0.f, 0.f};       // l4: head size 64 only, see below
            for (int j = 0; j < n && ok; ++j, ++tiles) {
                if (!mbar_wait(s_full(x), tiles & 1, abort_flag)) { ok = false; break; }
                tc_fence_after_sync();
                const bool diag = PAIRED || (j + 1) * BKV > q0;      // some keys of this tile lie beyond some rows of the tile
                const int lim = row - j * BKV;                      // columns above lim are masked (key > query)
                // ---- the whole score row at once: four loads in flight, one wait (the row stays in registers for both passes)
                uint32_t rs[128];
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) tmem_ld_32x32b_x32(tS + ch * 32, *reinterpret_cast<uint32_t(*)[32]>(rs + ch * 32));
                tmem_ld_wait();
                if (diag) {
#pragma unroll
                    for (int i = 0; i < 128; ++i) if (i > lim) rs[i] = __float_as_uint(-INFINITY);
                }
                float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;      // 0, 1: first 64 keys, 2, 3: the others
#pragma unroll
                for (int i = 0; i < 64; i += 2) {
                    mx0 = fmaxf(mx0, __uint_as_float(rs[i]));      mx1 = fmaxf(mx1, __uint_as_float(rs[i + 1]));
                    mx2 = fmaxf(mx2, __uint_as_float(rs[64 + i])); mx3 = fmaxf(mx3, __uint_as_float(rs[64 + i + 1]));
                }
                const float mx_first = fmaxf(mx0, mx1), mx = fmaxf(mx_first, fmaxf(mx2, mx3));
                // The reference of the exponentials starts as the maximum of the first key tile; with head size 64 as that of its first
                // 64 keys unless the others exceed it by the threshold.  That gives the bits of a walk in 64-key tiles as long as no
                // later tile moves the reference: such a walk would decide per 64 keys, this one decides per 128.
                const bool early = HS == 64 && j == 0 && (mx - mx_first) * sl2 <= kRescaleThreshold;
                // ---- lazy rescale of O (warp-collective tensor-memory accesses: the warp decides together)
                const bool need = j == 0 || (mx - m_ref) * sl2 > kRescaleThreshold;
                if (__any_sync(0xffffffffu, need)) {
                    const float m_new = need ? (early ? mx_first : fmaxf(m_ref, mx)) : m_ref;
                    if (j > 0) {
                        const float alpha = need ? ex2((m_ref - m_new) * sl2) : 1.f;
                        l_sum *= alpha;
                        if constexpr (HS == 64) {
#pragma unroll
                            for (int q = 0; q < 4; ++q) l4[q] *= alpha;
                        }
                        if (!mbar_wait(o_done(x), (tiles - 1) & 1, abort_flag)) { ok = false; break; }      // PV of tile j-1 has landed
                        tc_fence_after_sync();
#pragma unroll 1
                        for (int ch = 0; ch < HS / 32; ++ch) {
                            uint32_t ro[32];
                            tmem_ld_32x32b_x32(tO + ch * 32, ro);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 32; ++i) ro[i] = __float_as_uint(__uint_as_float(ro[i]) * alpha);
                            tmem_st_32x32b_x32(tO + ch * 32, ro);
                        }
                        tmem_st_wait();
                    }
                    m_ref = m_new;
                }
                // ---- this warpgroup's turn
                const bool in_turn = j < n_turn;
                if (in_turn && (x == 0 ? turns > 0 : !(alone && j == n - 1))) {
                    if (!mbar_wait(turn(x), (x == 0 ? turns - 1 : turns) & 1, abort_flag)) { ok = false; break; }
                }
                // ---- probabilities -> bf16 -> tensor memory (over the first 64 score columns, which are in registers by now)
                const float moff = m_ref * sl2;
                float sum0 = 0.f, sum1 = 0.f;
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    uint32_t pw[16];
                    float part = 0.f;
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        const float p0 = ex2(fmaf(__uint_as_float(rs[ch * 32 + i]), sl2, -moff));         // masked scores are -inf -> 0
                        const float p1 = ex2(fmaf(__uint_as_float(rs[ch * 32 + i + 1]), sl2, -moff));
                        if constexpr (HS == 64) {
                            // with the early reference above, the row sum too is that of 64-key tiles: one sum per 16 columns of a tile
                            part += p0 + p1;
                            if (i == 14 || i == 30) { l4[(2 * ch + i / 16) % 4] += part; part = 0.f; }
                        } else {
                            sum0 += p0; sum1 += p1;
                        }
                        pw[i / 2] = pack2(p0, p1);
                    }
                    tmem_st_32x32b_x16(tS + ch * 16, pw);
                    if (in_turn && ch == (HS == 64 ? 2 : 3)) warp_arrive(turn(1 - x));      // the other tile's turn
                    if (ch == 1) {                                  // first 64 keys of P are complete: hand them over
                        tmem_st_wait();
                        tc_fence_before_sync();
                        warp_arrive(p_ready(x));
                    }
                }
                turns += in_turn;
                const float sum = sum0 + sum1;
                l_sum += sum;
                tmem_st_wait();
                tc_fence_before_sync();
                warp_arrive(p_ready2(x));
            }
            // ---- the walk is over: normalise and store this tile's rows, then release O to the next item
            if (ok && n > 0) ok = mbar_wait(o_done(x), (tiles - 1) & 1, abort_flag);
            tc_fence_after_sync();
            if (ok && n > 0) {
                if constexpr (HS == 64) l_sum = ((l4[0] + l4[1]) + l4[2]) + l4[3];
                const float inv = 1.f / l_sum;
                __nv_bfloat16* o = p.out + ((static_cast<long long>(b) * p.T + (row_ok ? row : 0)) * p.Hq + h) * HS;
                uint32_t ro[HS];
#pragma unroll
                for (int ch = 0; ch < HS / 32; ++ch) tmem_ld_32x32b_x32(tO + ch * 32, *reinterpret_cast<uint32_t(*)[32]>(ro + ch * 32));
                tmem_ld_wait();
                tc_fence_before_sync();                             // O is in registers
                warp_arrive(o_free(x));
                if (row_ok) {
#pragma unroll
                    for (int g = 0; g < HS / 16; ++g) {
                        uint32_t v[8];
#pragma unroll
                        for (int jj = 0; jj < 8; ++jj) {
                            const __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(ro[g * 16 + 2 * jj]) * inv, __uint_as_float(ro[g * 16 + 2 * jj + 1]) * inv);
                            v[jj] = *reinterpret_cast<const uint32_t*>(&h2);
                        }
                        if (p.absmax) {
#pragma unroll
                            for (int jj = 0; jj < 8; ++jj) omax = fmaxf(omax, fmaxf(fabsf(__uint_as_float(v[jj] << 16)), fabsf(__uint_as_float(v[jj] & 0xffff0000u))));
                        }
                        if (p.wide) {
                            store_sector(o + g * 16, v);
                        } else {
                            *reinterpret_cast<uint4*>(o + g * 16) = make_uint4(v[0], v[1], v[2], v[3]);
                            *reinterpret_cast<uint4*>(o + g * 16 + 8) = make_uint4(v[4], v[5], v[6], v[7]);
                        }
                    }
                }
                if (row_ok) p.lse[(static_cast<long long>(b) * p.Hq + h) * p.T + row] = m_ref * p.scale + logf(l_sum);
            }
        }
        if (!ok) { *abort_flag = 1u; if (r == 0) atomicOr(p.status, kErrOther); }
        if (p.absmax) {
            omax = warp_reduce_max(omax);
            if (lane == 0 && omax > 0.f) atomic_max_float(p.absmax, omax);
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 8) tmem_dealloc(tmem, TMEM_COLS);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

template <int HS>
int launch(void* out, float* lse, const void* qkv, int B, int T, int Hq, int Hkv, float* absmax, unsigned int* status, cudaStream_t s) {
    static EncodeTiledFn encode = nullptr;
    if (!encode) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess || !ptr) return -1;
        encode = reinterpret_cast<EncodeTiledFn>(ptr);
    }
    const long long W = static_cast<long long>(Hq + 2 * Hkv) * HS;
    CUtensorMap tmap;
    cuuint64_t dims[3] = {static_cast<cuuint64_t>(W), static_cast<cuuint64_t>(T), static_cast<cuuint64_t>(B)};
    cuuint64_t strides[2] = {static_cast<cuuint64_t>(W) * 2, static_cast<cuuint64_t>(W) * 2 * T};
    cuuint32_t box[3] = {64, 128, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = encode(&tmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(qkv), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return 1000 + static_cast<int>(r);
    constexpr int smem = one_block_per_sm((2 + 2 * KV_STAGES<HS>) * (HS / 64) * CHUNK_BYTES + 256);
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_done[dev & 63]) {
        cudaError_t e = cudaFuncSetAttribute(attn_fwd_pingpong_kernel<HS, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(attn_fwd_pingpong_kernel<HS, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return 2000 + static_cast<int>(e);
        attr_done[dev & 63] = true;
    }
    FwdParams p{};
    p.B = B; p.T = T; p.Hq = Hq; p.Hkv = Hkv; p.scale = 1.f / sqrtf(static_cast<float>(HS));
    p.out = static_cast<__nv_bfloat16*>(out); p.lse = lse; p.absmax = absmax; p.status = status;
    static const bool no_turns = [] { const char* e = getenv("LLMQ_ATTN_FWD_TURNS"); return e && e[0] == '0'; }();      // for A/B measurements
    p.turns = no_turns ? 0 : 1;
    p.wide = reinterpret_cast<uintptr_t>(out) % 32 == 0;
    const int nqb = (T + 2 * BQ - 1) / (2 * BQ);
    static int sms[64] = {};
    if (!sms[dev & 63]) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return -2;
        sms[dev & 63] = n;
    }
    const bool paired = T <= BQ && Hq / Hkv > 1 && static_cast<long long>(Hq) * B > sms[dev & 63];
    const long long total = paired ? static_cast<long long>(pairs_of_group(p)) * Hkv * B : static_cast<long long>(nqb) * Hq * B;
    const int grid = static_cast<int>(total < sms[dev & 63] ? total : sms[dev & 63]);       // one CTA per SM (tensor memory)
    if (paired) launch_chained(attn_fwd_pingpong_kernel<HS, true>, grid, NUM_THREADS, smem, s, tmap, p);
    else        launch_chained(attn_fwd_pingpong_kernel<HS, false>, grid, NUM_THREADS, smem, s, tmap, p);
    return LLMQ_LAUNCH_CHECK();
}

}  // namespace

// Same contract as llmq_attention_forward (which dispatches here); head size 64 or 128.
int llmq_attention_forward_pingpong(void* out, float* lse, const void* qkv, int B, int T, int Hq, int Hkv, int HS, float* absmax,
                                    unsigned int* status, cudaStream_t s) {
    return HS == 64 ? launch<64>(out, lse, qkv, B, T, Hq, Hkv, absmax, status, s) : launch<128>(out, lse, qkv, B, T, Hq, Hkv, absmax, status, s);
}
