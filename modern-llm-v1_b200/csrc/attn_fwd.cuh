// Causal grouped-query attention forward for sm_100a: O = softmax(scale * Q K^T) V and
// L = logsumexp of the scaled scores (natural log), the pair of outputs of the
// reference's flash_attn_forward (llm/src/model/flash_attn.h:25-28,
// llm/src/model/flash_attn.cu:28-131), computed tile-wise on the tensor cores.
//
// Persistent CTAs, two per SM.  A CTA walks a static list of work items (item = one 128-row
// query tile of one (batch, query head); items are ordered heaviest first and dealt by a host-built
// table, see ItemTable) and, per item, the key tiles of K/V up to the diagonal (tiles above it are
// never loaded).  Every pipeline keeps running across item boundaries: the K/V ring prefetches
// the next item's tiles and the MMA warp issues the next item's first Q K^T products while the
// softmax warps write the previous item's output rows.  GQA is an index: the K/V tensor maps are
// addressed with h_kv = h_q / group (llm/src/model/attention.cu:406), nothing is replicated.
//
// Roles (256 threads = two warpgroups, so that setmaxnreg can move registers from the
// second group to the first):
//   warps 0-3  softmax + epilogue, thread r owns query row r == TMEM lane r
//   warp  4    TMA producer (converged warp, one elected lane issues)
//   warp  5    TMEM allocation and tcgen05.mma issue (converged warp, one elected lane issues)
//   warps 6-7  idle (they only donate registers)
// TMEM (256 columns):
//   D = 64   S (128 FP32 columns), O (64), P (BF16 pairs, 64).  Tiles of 128 keys.
//   D = 128  S (64), P (32), columns 0-63 of Q (32), O (128).  Tiles of 64 keys.
// The softmax warps take a tile's scores into registers in one go and hand S back, so the next tile's Q K^T runs under this
// tile's exponentials; P V of a tile runs under the next tile's.
// What bounds it: at D = 64 the chain of a tile in the softmax warps (scores out of tensor memory, maximum, exponentials at 16 a
// clock, P back, three barriers of about 100 clocks each), two such chains per scheduler.  Hence 128 keys a tile, packed FP32
// arithmetic, and no commit whose completion another barrier implies.  In the steady state two CTAs take 2350 clocks for a tile
// each, of which the exponentials alone are 2048.  At D = 128 it is that chain and the tensor pipe alike: a Q K^T step of 64 keys
// takes 64 clocks of it with both operands in shared memory, 37 with Q in tensor memory, where beside S, P and O half of Q has
// room (copied there by the MMA warp, tcgen05.cp): 680 clocks a tile instead of 788, and a tile every 1450 to 1650 instead of
// 1700.  (Two S buffers of 64 columns with P over them, as before, leave no room for Q.)
// Measured on B200, us: against 64-key tiles with P over S and Q in tensor memory at D=64: B=2 T=128 6/2
// 6.0 -> 5.4, B=32 T=512 6/2 21.9 -> 20.6, B=16 T=1024 16/4 74.3 -> 69.2; one code path for both head dimensions, without the
// second S buffer: B=32 T=512 20.4 -> 19.4, B=16 T=1024 72.9 -> 68.8, B=8 T=2000 16/4 123.5 -> 115, B=1 T=2000 6/2 18.1 -> 16.5,
// and with half of Q in tensor memory at D=128: B=4 T=8192 16/4 1080 -> 1025, B=8 T=1024 16/4 46.1 -> 44.4, B=32 T=1001 1/1
// 20.0 -> 19.2, B=20 T=200 8/4 12.0 both.
// Measured and dropped: four epilogue warps of their own, as the dQ pass has (B=8 T=2000 121 -> 118, but B=32 T=512 20.1 -> 20.8,
// B=2 T=128 5.0 -> 5.5, D=128 137 -> 145: the softmax warps lose registers to them); exponentials against the reference of the
// tile before with the maximum taken under them (5 % slower); a warp of its own for Q K^T (no difference); Q copied by the
// softmax warps (D=128 T=200 12.0 -> 13.1).
#pragma once

#include "ptx.cuh"

namespace b200attn {

struct FwdParams {
    int B, T, Hq, Hkv, group;
    int n_qtiles;
    int kv_off;        // keys in front of the first query row: query row t sees keys 0 .. kv_off + t (0 when q and k
                       // cover the same tokens; the cached tokens' count when a chunk of new tokens attends over a KV cache)
    int split;         // CTAs (a cluster) that share an item's key tiles; 1 except in the split kernel
    FastDiv div_split;
    int early;         // whether the next kernel may start while this one's last items are worked on (see ptx.cuh)
    float scale;       // softmax scale
    float scale_log2;  // scale * log2(e)
    float* lse;        // [B, Hq, T]
    uint16_t* o;       // output, BF16
    long long o_st, o_sh, o_sb;  // element strides of o: token, head, batch
    int* status;       // device status word
    int* sched;        // two words of the device-wide item counter (see ptx.cuh)
    FastDiv div_bh, div_h, div_group;  // division by B * Hq, by Hq and by the group size
};

template <int D>
struct FwdCfg {
    static constexpr int kKeys = D == 64 ? 128 : 64;  // keys per K/V tile
    static constexpr int kStages = 2;
    static constexpr int kQBufs = 2;                  // the next item's Q is prefetched
    static constexpr bool kQTmem = D == 128;          // the first 64 columns of Q are in tensor memory
    static constexpr int kQTileBytes = 128 * D * 2;
    static constexpr int kQBoxBytes = 128 * 64 * 2;   // Q TMA box: 128 rows x 64 bf16
    static constexpr int kQStageBytes = kQTmem ? kQBoxBytes : 0;  // where those 64 columns land
    static constexpr int kQBytes = kQStageBytes + kQBufs * kQBoxBytes;
    static constexpr int kKVTileBytes = kKeys * D * 2;
    static constexpr int kKVBoxBytes = kKeys * 64 * 2;  // K/V TMA box: kKeys rows x 64 bf16
    static constexpr int kBoxes = D / 64;
    static constexpr int kBarBytes = 512;
    static constexpr int kSmemBytes = kQBytes + 2 * kStages * kKVTileBytes + kBarBytes;
    static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs per SM");
    static constexpr int kTmemCols = 256;
    static constexpr int kColS = 0, kColO = 128;
    static constexpr int kColP = D == 64 ? kColO + D : kKeys;
    static constexpr int kColQ = 96;  // kQTmem
    // registers per thread of the softmax warpgroup and of the other one: together the launch's 256 x 128
    static constexpr int kRegsSoftmax = D == 64 ? 192 : 168, kRegsOther = 256 - kRegsSoftmax;
};

// log2 of the growth of the row maximum that is tolerated before O and the row
// sum are rescaled; below it the stale maximum stays the exponent reference.
constexpr float kRescaleThresholdLog2 = 8.0f;

// SPLIT: few, long items (a chunk of new tokens behind a long cache, a single long sequence).  A CTA walks a share of ONE
// item's key tiles, and the CTAs of a cluster add up their (m, l, O) through distributed shared memory, each finishing
// 128 / split of the rows.  Measured on B200: 15 tokens behind 6000, B=1 6/2
// D=64 (6 items, 8 CTAs each) 57.2 -> 15.0 us; 720 behind 4000, B=1 8/1 D=64 (48 items, 4) 47.7 -> 26.8; 500 behind 3000,
// B=2 16/4 D=128 (128 items, 2) 47.4 -> 40.8.
template <int D, bool SPLIT>
__global__ void __launch_bounds__(256, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmV, const FwdParams p, const __grid_constant__ ItemTable tab) {
    using Cfg = FwdCfg<D>;
    constexpr int NST = Cfg::kStages;
    constexpr int NQB = Cfg::kQBufs;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;                         // kQTmem: columns 0-63 on their way to tensor memory
    uint8_t* sQb = sQ + Cfg::kQStageBytes;      // [NQB] Q as the products read it (kQTmem: columns 64-127)
    uint8_t* sK = sQb + NQB * Cfg::kQBoxBytes;
    uint8_t* sV = sK + NST * Cfg::kKVTileBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sV + NST * Cfg::kKVTileBytes);
    uint64_t* bar_q = bars + 0;        // [2] per Q buffer: Q of an item has landed              (phase: item / NQB)
    uint64_t* bar_q_free = bars + 2;   // [2] per Q buffer: every Q K^T product of the item done (phase: item / NQB)
    uint64_t* bar_s_full = bars + 4;   //                                                         (phase: tile)
    uint64_t* bar_s_loaded = bars + 5; // S is in registers                                       (phase: tile)
    uint64_t* bar_p_full = bars + 7;   // P written, O rescaled                                   (phase: tile)
    uint64_t* bar_qt_full = bars + 8;  // kQTmem: columns 0-63 of an item's Q are in tensor memory, the staging box is free (phase: item)
    uint64_t* bar_o_done = bars + 11;  // O of an item is complete                                (phase: item)
    uint64_t* bar_o_free = bars + 12;  // O has been read by the epilogue                         (phase: item)
    uint64_t* bar_k_full = bars + 13;            // [NST]
    uint64_t* bar_k_free = bars + 13 + NST;      // [NST] Q K^T of the tile is complete (a softmax thread that has seen it says so)
    uint64_t* bar_v_full = bars + 13 + 2 * NST;  // [NST]
    uint64_t* bar_v_free = bars + 13 + 3 * NST;  // [NST] P V of the tile is complete
    uint64_t* bar_item = bars + 32;    // [kItemRing] item ids handed out by the producer
    volatile int* item_ring = reinterpret_cast<volatile int*>(bars + 32 + kItemRing);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 30);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 31);

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;

    // item id -> (query tile, head, batch); ids are ordered by work, heaviest query tile first
    const int n_bh = p.B * p.Hq;
    const int n_items = p.n_qtiles * n_bh;
    auto get_item = [&](int n) { return item_get(bar_item, item_ring, n, abort_flag, p.status); };
    auto item_rest = [&](int id) { return id - int(fastdiv(unsigned(id), p.div_bh)) * n_bh; };  // b * Hq + h
    auto item_qt = [&](int id) { return p.n_qtiles - 1 - int(fastdiv(unsigned(id), p.div_bh)); };
    auto item_b = [&](int id) { return int(fastdiv(unsigned(item_rest(id)), p.div_h)); };
    auto item_h = [&](int id) { return item_rest(id) - item_b(id) * p.Hq; };
    auto item_all = [&](int id) { return (p.kv_off + min(p.T, item_qt(id) * 128 + 128) + Cfg::kKeys - 1) / Cfg::kKeys; };
    const int split_id = SPLIT ? int(fastdiv(blockIdx.x, p.div_split)) : 0, rank = SPLIT ? int(blockIdx.x) - split_id * p.split : 0;
    // key tiles of an item that are this CTA's: [j_first, j_first + item_nkv)
    const int j_first = SPLIT ? int(fastdiv(unsigned(item_all(split_id) * rank), p.div_split)) : 0;
    auto item_nkv = [&](int id) {
        return SPLIT ? int(fastdiv(unsigned(item_all(id) * (rank + 1)), p.div_split)) - j_first : item_all(id);
    };
    float split_m = -INFINITY, split_l = 0.f;  // SPLIT: this thread's row

    B200ATTN_TRACE_BEGIN(0);
    // Set-up with one CTA-wide barrier: one lane of the producer warp initialises every mbarrier while
    // the MMA warp allocates TMEM; nothing touches global memory before grid_dep_wait().  The first item's Q and its first K and V
    // are requested at once then, so that the status word, the barrier and the roles' start pass under their latency (requested by
    // the producer's role behind the barrier, us: B=2 T=128 6/2 D=64 5.07 instead of 4.75, B=32 T=512 6/2 19.4 instead of 18.4, B=2 T=128 D=128
    // 6.1 instead of 5.8, B=32 T=1001 1/1 D=128 18.9 instead of 18.7).
    const int id_first = SPLIT ? split_id : sched_first(tab, p.sched, int(blockIdx.x));  // the first item needs no fetch
    const bool any = !SPLIT || item_nkv(id_first) > 0;
    auto load_q = [&](int n, int id) {  // one thread: Q of this CTA's n-th item into Q buffer n % NQB
        mbar_arrive_expect_tx(&bar_q[n % NQB], Cfg::kQTileBytes);
#pragma unroll
        for (int bx = 0; bx < Cfg::kBoxes; ++bx)
            tma_load_4d(bx + 1 < Cfg::kBoxes ? sQ : sQb + (n % NQB) * Cfg::kQBoxBytes, &tmQ, &bar_q[n % NQB], bx * 64, item_qt(id) * 128,
                        item_h(id), item_b(id));
    };
    auto load_kv = [&](uint8_t* tile, const CUtensorMap* map, uint64_t* full, int j, int hk, int b) {  // one thread
        mbar_arrive_expect_tx(full, Cfg::kKVTileBytes);
#pragma unroll
        for (int bx = 0; bx < Cfg::kBoxes; ++bx)
            tma_load_4d(tile + bx * Cfg::kKVBoxBytes, map, full, bx * 64, (j_first + j) * Cfg::kKeys, hk, b);
    };
    if (warp == 4 && lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_q[i], 1);
            mbar_init(&bar_q_free[i], 1);
        }
        mbar_init(bar_s_full, 1);
        mbar_init(bar_s_loaded, 128);
        mbar_init(bar_p_full, 128);
        mbar_init(bar_qt_full, 1);
        mbar_init(bar_o_done, 1);
        mbar_init(bar_o_free, 128);
        for (int s = 0; s < NST; ++s) {
            mbar_init(&bar_k_full[s], 1);
            mbar_init(&bar_k_free[s], 1);
            mbar_init(&bar_v_full[s], 1);
            mbar_init(&bar_v_free[s], 1);
        }
        for (int i = 0; i < kItemRing; ++i) mbar_init(&bar_item[i], 1);
        fence_mbar_init();
        *abort_flag = 0;
        item_publish(bar_item, item_ring, 0, any ? id_first : -1);
    }
    if (warp == 4) {
        __syncwarp();
        grid_dep_wait();  // first global access of this CTA comes next
        if (elect_one()) {
            if (any) {
                const int b = item_b(id_first), hk = int(fastdiv(unsigned(item_h(id_first)), p.div_group));
                load_q(0, id_first);
                load_kv(sK, &tmK, &bar_k_full[0], 0, hk, b);
                load_kv(sV, &tmV, &bar_v_full[0], 0, hk, b);
            }
            const int failed = *reinterpret_cast<volatile int*>(p.status);
            if (failed != 0) {  // behind an earlier failure the CTA leaves, but not before its loads have landed
                for (uint64_t* bar : {bar_q, bar_k_full, bar_v_full})
                    if (any) mbar_wait(bar, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                *abort_flag = failed;
            }
        }
        __syncwarp();
    }
    if (warp == 5) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    grid_dep_wait();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    if (*abort_flag != 0) {
        // an earlier CTA already failed: fall through to the teardown
    } else if (warp >= 6) {
        reg_dealloc<Cfg::kRegsOther>();  // idle warps
    } else if (warp == 4) {
        // ------------------------------------------------------------------ producer
        reg_dealloc<Cfg::kRegsOther>();
        int g = 0;  // key tiles issued so far by this CTA (ring position)
        bool ok = true;
        int id_next = 0;  // lane 0: the id fetched for the item after the next Q load
        // waits for Q buffer n % NQB and requests Q of the n-th item
        auto next_q = [&](int n, int id) {
            if (n >= NQB)
                ok = mbar_wait_warp(&bar_q_free[n % NQB], uint32_t(n / NQB - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
            if (Cfg::kQTmem && ok)  // the item before has left the staging box
                ok = mbar_wait_warp(bar_qt_full, uint32_t(n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
            if (!ok) return;
            if (elect_one()) load_q(n, id);
            __syncwarp();
        };
        int id = id_first;
        if (lane == 0) id_next = SPLIT ? n_items : sched_fetch(tab, p.sched, 1, int(blockIdx.x), int(gridDim.x));
        __syncwarp();
        ok = any;
        for (int n = 0; ok; ++n) {
            const int h = item_h(id), b = item_b(id), hk = int(fastdiv(unsigned(h), p.div_group)), n_kv = item_nkv(id);
            // The next item is taken, announced and its Q requested a few tiles before this item's loads end
            // (late, so that a CTA commits itself to little work ahead, but not before the ring has been
            // filled for this item).
            const int j_next = max(min(n_kv, NST) - 1, n_kv - 3);
            int id_new = n_items;
            for (int j = 0; j < n_kv; ++j, ++g) {
                const int s = g % NST;
                const uint32_t use = uint32_t(g / NST);
                if (g >= NST) ok = mbar_wait_warp(&bar_k_free[s], (use - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
                if (!ok) break;
                if (g > 0 && elect_one()) load_kv(sK + s * Cfg::kKVTileBytes, &tmK, &bar_k_full[s], j, hk, b);
                __syncwarp();
                if (g >= NST) ok = mbar_wait_warp(&bar_v_free[s], (use - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
                if (!ok) break;
                if (g > 0 && elect_one()) load_kv(sV + s * Cfg::kKVTileBytes, &tmV, &bar_v_full[s], j, hk, b);
                __syncwarp();
                if (j == j_next) {
                    id_new = __shfl_sync(0xffffffffu, id_next, 0);
                    const bool more = id_new < n_items;
                    if (lane == 0) {
                        item_publish(bar_item, item_ring, n + 1, more ? id_new : -1);
                        if (more) id_next = sched_fetch(tab, p.sched, n + 2, int(blockIdx.x), int(gridDim.x));
                    }
                    __syncwarp();
                    if (more) next_q(n + 1, id_new);
                    if (!ok) break;
                }
            }
            if (!ok || id_new >= n_items) break;
            id = id_new;
        }
        if (!SPLIT && ok && lane == 0) sched_finish(p.sched, int(gridDim.x));
        if (p.early) grid_dep_launch();
    } else if (warp == 5) {
        // ------------------------------------------------------------------ MMA issuer
        reg_dealloc<Cfg::kRegsOther>();
        constexpr uint32_t idesc_s = make_idesc_bf16(128, Cfg::kKeys, 0, 0);
        constexpr uint32_t idesc_o = make_idesc_bf16(128, D, 0, 1);
        // This CTA's key tiles are numbered g = 0, 1, ... across all its items: ring stage g % NST.  The cursor `sc`
        // walks that sequence for the products Q K^T, one tile ahead of the loop below that issues the products P V, also
        // across item boundaries.
        struct Cursor {
            int id, n, j, n_kv, g;  // item id, items before it on this CTA, tile in item, tiles of item, global tile
        };
        Cursor sc{get_item(0), 0, 0, 0, 0};
        if (sc.id >= 0) sc.n_kv = item_nkv(sc.id);
        bool ok = true;
        // Waits for what S(cursor) reads: its Q (first tile of an item) and K.  (The S buffer is free once the products before
        // it in the pipe have run.)
        auto wait_s = [&]() {
            if (sc.id < 0) return;
            const int s = sc.g % NST, qb = sc.n % NQB;
            if (sc.j == 0)
                ok = mbar_wait_warp(&bar_q[qb], uint32_t(sc.n / NQB) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
            if (ok) ok = mbar_wait_warp(&bar_k_full[s], uint32_t(sc.g / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
        };
        const uint32_t sq_addr = smem_u32(sQb), sk_addr = smem_u32(sK), sv_addr = smem_u32(sV);
        // S(cursor) = Q K^T
        auto issue_s = [&]() {
            tc_fence_after_sync();
            const int qb = sc.n % NQB;
            const uint64_t q_desc = make_sdesc_sw128(sq_addr + qb * Cfg::kQBoxBytes, 16, 1024);
            const uint64_t k_desc = make_sdesc_sw128(sk_addr + (sc.g % NST) * Cfg::kKVTileBytes, 16, 1024);
            if (elect_one()) {
                if (Cfg::kQTmem && sc.j == 0) {  // (the products of the item before have been read out of the S buffer)
                    const uint64_t stage_desc = make_sdesc_sw128(smem_u32(sQ), 16, 1024);
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks) tmem_copy_128x32b(tmem + Cfg::kColQ + ks * 8, stage_desc + kmajor_step(ks, 0));
                    umma_commit(bar_qt_full);
                }
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint64_t b_desc = k_desc + kmajor_step(ks, Cfg::kKVBoxBytes);
                    if (Cfg::kQTmem && ks < 4) umma_ts(tmem + Cfg::kColS, tmem + Cfg::kColQ + ks * 8, b_desc, idesc_s, ks > 0);
                    else umma_ss(tmem + Cfg::kColS, q_desc + kmajor_step(ks % 4, 0), b_desc, idesc_s, ks > 0);
                }
                umma_commit(bar_s_full);
                if (sc.j + 1 == sc.n_kv) umma_commit(&bar_q_free[qb]);  // no later product reads this item's Q
            }
            __syncwarp();
        };
        auto next_s = [&]() {
            ++sc.g;
            if (++sc.j == sc.n_kv) {
                sc.id = get_item(++sc.n);
                sc.j = 0;
                sc.n_kv = sc.id >= 0 ? item_nkv(sc.id) : 0;
            }
        };
        if (sc.id >= 0) {
            wait_s();
            if (ok) issue_s(), next_s();
        }
        int g = 0, n = 0;
        // (this warp has already waited for the ring entry of item n: the cursor above is never behind)
        for (int id; ok && (id = item_ring[n % kItemRing]) >= 0; ++n) {
            const int n_kv = item_nkv(id);
            for (int j = 0; j < n_kv; ++j, ++g) {
                // What P V needs besides P is waited for first: a wait costs 100 clocks even when the barrier is complete.
                const int s = g % NST;
                // S(g + 1) as soon as S(g) is in registers: it runs under the exponentials of tile g
                if (sc.id >= 0) {
                    wait_s();
                    if (ok) ok = mbar_wait_warp(bar_s_loaded, uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                    if (!ok) break;
                    issue_s();
                    next_s();
                }
                if (ok) ok = mbar_wait_warp(&bar_v_full[s], uint32_t(g / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                // the accumulator belongs to the previous item's epilogue until it has been read
                if (ok && j == 0 && n > 0) ok = mbar_wait_warp(bar_o_free, uint32_t(n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                if (!ok) break;
                const uint64_t v_desc = make_sdesc_sw128(sv_addr + s * Cfg::kKVTileBytes, Cfg::kKVBoxBytes, 1024);
                ok = mbar_wait_warp(bar_p_full, uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                if (!ok) break;
                B200ATTN_STAMP(lane == 0, 16 + 8 * g + 4);
                tc_fence_after_sync();
                if (elect_one()) {
                    // O += P V : 16 keys per K step, 8 columns of BF16 pairs each
#pragma unroll
                    for (int ks = 0; ks < Cfg::kKeys / 16; ++ks)
                        umma_ts(tmem + Cfg::kColO, tmem + Cfg::kColP + ks * 8, v_desc + uint64_t(ks * 128), idesc_o, (j > 0) || (ks > 0));
                    umma_commit(&bar_v_free[s]);
                    if (j + 1 == n_kv) umma_commit(bar_o_done);
                }
                __syncwarp();
                B200ATTN_STAMP(lane == 0, 16 + 8 * g + 6);
            }
        }
        // nothing may be in flight when TMEM is freed: the last commit covers every MMA issued above
        if (ok && n > 0) mbar_wait_warp(bar_o_done, uint32_t(n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
    } else {
        // ------------------------------------------------------------------ softmax + epilogue
        reg_alloc<Cfg::kRegsSoftmax>();
        const int row = tid;                                   // query row inside the tile == TMEM lane
        const uint32_t lane_base = uint32_t(warp * 32) << 16;  // this warp's TMEM lane quadrant
        const uint32_t t_o = tmem + lane_base + Cfg::kColO;
        bool ok = true;
        // Epilogue of one item: O / l -> BF16 -> global memory, logsumexp.  (bar_v_free cannot be used for
        // "O is complete": P V of the last TWO tiles may still be in flight, and a parity wait is only
        // unambiguous when the waiter is at most one phase behind; bar_o_done completes once per item.)
        auto epilogue = [&](int n_item, int id, float m_ref, float l) -> bool {
            B200ATTN_STAMP(tid == 0, 400 + 4 * n_item + 0);
            if (!mbar_wait_warp(bar_o_done, uint32_t(n_item) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA)) return false;
            B200ATTN_STAMP(tid == 0, 400 + 4 * n_item + 1);
            tc_fence_after_sync();
            const float inv_l = 1.f / l;
            const int q0 = item_qt(id) * 128, b = item_b(id), h = item_h(id);
            const bool in_range = q0 + row < p.T;
            uint16_t* orow = p.o + size_t(b) * p.o_sb + size_t(h) * p.o_sh + size_t(q0 + row) * p.o_st;
            // every thread owns one contiguous row of D elements, written 64 columns at a time
#pragma unroll
            for (int hh = 0; hh < D / 64; ++hh) {
                uint32_t ow[32];  // 64 columns as BF16 pairs
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t orr[32];
                    tmem_ld_x32(t_o + hh * 64 + c * 32, orr);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        ow[c * 16 + i] = pack_bf16x2(__uint_as_float(orr[2 * i]) * inv_l, __uint_as_float(orr[2 * i + 1]) * inv_l);
                }
                if (hh + 1 == D / 64) {
                    // the accumulator has been read: the next item's first P V may overwrite it
                    tc_fence_before_sync();
                    mbar_arrive(bar_o_free);
                }
                B200ATTN_STAMP(tid == 0, 440 + 4 * n_item + 0);
                if (in_range) {
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        *reinterpret_cast<uint4*>(orow + hh * 64 + c * 8) =
                            make_uint4(ow[c * 4], ow[c * 4 + 1], ow[c * 4 + 2], ow[c * 4 + 3]);
                }
            }
            B200ATTN_STAMP(tid == 0, 440 + 4 * n_item + 1);
            if (in_range) p.lse[(size_t(b) * p.Hq + h) * p.T + q0 + row] = m_ref * p.scale + logf(l);
            B200ATTN_STAMP(tid == 0, 400 + 4 * n_item + 2);
            return true;
        };
        // The epilogue of an item is deferred until the softmax of the next item's first tile has been handed
        // to the MMA warp: the wait for the item's last P V then overlaps useful work.
        bool pending = false;
        int pend_id = 0;
        float pend_m = 0.f, pend_l = 1.f;
        int g = 0, n = 0;
        for (int id; ok && (id = get_item(n)) >= 0; ++n) {
            const int qt = item_qt(id), h = item_h(id), b = item_b(id), n_kv = item_nkv(id);
            const int q0 = qt * 128;
            float m_ref = -INFINITY;  // exponent reference (a past row maximum), raw score units
            float l = 0.f;            // running sum of exp2((s - m_ref) * scale_log2)
            for (int j = 0; j < n_kv; ++j, ++g) {
                const uint32_t t_s = tmem + lane_base + Cfg::kColS;
                ok = mbar_wait_warp(bar_s_full, uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                if (!ok) break;
                B200ATTN_STAMP(tid == 0, 16 + 8 * g + 0);
                if (tid == 0) mbar_arrive(&bar_k_free[g % NST]);
                tc_fence_after_sync();
                constexpr int KEYS = Cfg::kKeys;
                uint32_t sr[KEYS];
#pragma unroll
                for (int c = 0; c < KEYS; c += 32) tmem_ld_x32(t_s + c, &sr[c]);
                tmem_wait_ld();
                tc_fence_before_sync();
                mbar_arrive(bar_s_loaded);  // the buffer goes back to the MMA warp at once
                const int kbase = (j_first + j) * KEYS;  // first key of this tile
                if (kbase + KEYS - 1 > q0 + p.kv_off) {
                    // tile touches the diagonal: key kbase + c is visible to query q0 + row iff it is <= the query's
                    // own position kv_off + q0 + row
                    const int lim = p.kv_off + q0 + row - kbase;  // columns c <= lim are visible
                    // 32 columns at a time: those that the whole warp sees (it does from its first row on) need no look.  The
                    // comparisons of all columns cost such a tile 550 of 3600 clocks at D = 64.
#pragma unroll
                    for (int c32 = 0; c32 < KEYS; c32 += 32)
                        if (c32 + 31 > lim - lane) {
#pragma unroll
                            for (int c = c32; c < c32 + 32; ++c)
                                if (c > lim) sr[c] = 0xff800000u;  // -inf
                        }
                }
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < KEYS; c += 8)
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        mx[k] = fmaxf(mx[k], fmaxf(__uint_as_float(sr[c + 2 * k]), __uint_as_float(sr[c + 2 * k + 1])));
                const float m_new = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), m_ref);
                float alpha = 1.f;
                if ((m_new - m_ref) * p.scale_log2 > kRescaleThresholdLog2) {  // also true for m_ref == -inf
                    alpha = ex2_approx((m_ref - m_new) * p.scale_log2);
                    m_ref = m_new;
                }
                // (a share of an item may hold no key that a row sees: its exponentials are 0 then, not NaN)
                const float neg_m = SPLIT && m_ref == -INFINITY ? 0.f : -m_ref * p.scale_log2;
                const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2), neg2 = pack_f32x2(neg_m, neg_m);
                uint64_t sum2[2] = {0ull, 0ull};
                // 32 columns at a time: exponentials, sums and BF16 pairs
                auto chunk = [&](int c, uint32_t (&pk)[16]) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float a0, a1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sr[c + 2 * i]), __uint_as_float(sr[c + 2 * i + 1])), scale2, neg2), a0, a1);
                        a0 = ex2_approx(a0);
                        a1 = ex2_approx(a1);
                        sum2[i & 1] = add_f32x2(sum2[i & 1], pack_f32x2(a0, a1));
                        pk[i] = pack_bf16x2(a0, a1);
                    }
                };
                // P V of the previous tile: it reads the columns P goes to and adds to O, which may have to be rescaled.
                // (At most one phase of this barrier is outstanding here: P V of this tile cannot start before this warp has
                // arrived on bar_p_full below.)
                uint64_t* bar_pv = &bar_v_free[(g - 1) % NST];
                const uint32_t pv_par = uint32_t((g - 1) / NST) & 1;
                const bool pv_seen = g == 0 || mbar_try_wait(bar_pv, pv_par);  // (looked at again below)
                auto wait_pv = [&]() {
                    if (!__all_sync(0xffffffffu, pv_seen)) ok = mbar_wait_warp(bar_pv, pv_par, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                    if (ok) tc_fence_after_sync();
                };
                const uint32_t t_p = tmem + lane_base + Cfg::kColP;
                {
                    uint32_t pk[16];
                    chunk(0, pk);
                    wait_pv();
                    if (!ok) break;
                    tmem_st_x16(t_p, pk);
                }
#pragma unroll
                for (int c = 1; c < KEYS / 32; ++c) {
                    uint32_t pk[16];
                    chunk(c * 32, pk);
                    tmem_st_x16(t_p + c * 16, pk);
                }
                const bool rescale = j > 0 && __any_sync(0xffffffffu, alpha != 1.f);  // (in front of the exponentials the vote holds them up)
                {
                    float s0, s1;
                    unpack_f32x2(add_f32x2(sum2[0], sum2[1]), s0, s1);
                    l = l * alpha + (s0 + s1);
                }
                B200ATTN_STAMP(tid == 0, 16 + 8 * g + 1);
                if (rescale) {
#pragma unroll
                    for (int c = 0; c < D / 32; ++c) {
                        uint32_t orr[32];
                        tmem_ld_x32(t_o + c * 32, orr);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) orr[i] = __float_as_uint(__uint_as_float(orr[i]) * alpha);
                        tmem_st_x32(t_o + c * 32, orr);
                    }
                }
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive(bar_p_full);
                B200ATTN_STAMP(tid == 0, 16 + 8 * g + 2);
                if (j == 0 && pending) {
                    ok = epilogue(n - 1, pend_id, pend_m, pend_l);
                    pending = false;
                    if (!ok) break;
                }
            }
            if (!ok) break;
            pending = true;
            pend_id = id, pend_m = m_ref, pend_l = l;
        }
        if constexpr (SPLIT) {
            if (ok && pending) ok = mbar_wait_warp(bar_o_done, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            if (ok && pending) split_m = pend_m, split_l = pend_l;
        } else if (ok && pending) {
            epilogue(n - 1, pend_id, pend_m, pend_l);
        }
        tc_fence_before_sync();
    }

    if constexpr (SPLIT) {
        // Every role comes here, also after a wait that gave up and when the status word was set before the launch.  Row r is
        // finished by CTA r / rows of the cluster; the K/V ring holds the arrivals, so all CTAs must be through with theirs
        // first.  A CTA that has failed sends a negative row sum instead of its share, and nobody writes the item.
        const int rows = 128 / p.split;
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (tid < 128) {
            const bool failed = *abort_flag != 0;  // (final: every warp of the CTA has passed the barrier)
            tc_fence_after_sync();
            const int to = (tid * p.split) >> 7, r = tid - to * rows;
            uint8_t* own = sK + (rank * rows + r) * D * 4;
            const uint32_t dst = cluster_addr(own, to);
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                if (failed) break;
                uint32_t v[32];
                tmem_ld_x32(tmem + (uint32_t(warp * 32) << 16) + Cfg::kColO + c * 32, v);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 8; ++i) {  // 16-byte pieces swizzled by the row: the rows of a warp would share a bank
                    const int at = ((c * 8 + i) ^ (r & 7)) << 4;
                    if (to == rank)
                        *reinterpret_cast<uint4*>(own + at) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    else
                        cluster_store_4(dst + at, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
            }
            cluster_store_f2(sQ + (rank * rows + r) * 8, to, failed ? make_float2(-INFINITY, -1.f) : make_float2(split_m, split_l));
            tc_fence_before_sync();
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (tid < 128) {
            const float2* ml = reinterpret_cast<const float2*>(sQ);
            const int q0 = item_qt(split_id) * 128 + rank * rows, b = item_b(split_id), h = item_h(split_id);
            // `split` threads per row, each with D / split columns, 16 at a time (8 when there are no more)
            const int r = fastdiv(unsigned(tid), p.div_split), part = tid - r * p.split, cols = fastdiv(unsigned(D), p.div_split);
            float m = -INFINITY;
            bool good = q0 + r < p.T;
            for (int k = 0; k < p.split; ++k) {
                m = fmaxf(m, ml[k * rows + r].x);
                if (ml[k * rows + r].y < 0.f) good = false;
            }
            if (good) {
                float l = 0.f;
                for (int k = 0; k < p.split; ++k) {
                    const float2 s = ml[k * rows + r];
                    // a share without a key for the row has l = 0, one whose scores are all NaN l = NaN: that must not get lost
                    l += s.x == -INFINITY ? s.y : ex2_approx((s.x - m) * p.scale_log2) * s.y;
                }
                if (m == -INFINITY) l = __int_as_float(0x7fffffff);  // no score above -inf: NaN, as 0 / 0 is
                const float inv_l = 1.f / l;
                uint16_t* orow = p.o + size_t(b) * p.o_sb + size_t(h) * p.o_sh + size_t(q0 + r) * p.o_st + part * cols;
                for (int c = 0; c < cols; c += 16) {
                    const bool two = c + 8 < cols;
                    float acc[16];
#pragma unroll
                    for (int e = 0; e < 16; ++e) acc[e] = l != l ? l : 0.f;
                    for (int k = 0; k < p.split; ++k) {
                        const float mk = ml[k * rows + r].x;
                        if (mk == -INFINITY) continue;  // no key of the row, or no tile at all: nothing valid was sent
                        const float f = ex2_approx((mk - m) * p.scale_log2) * inv_l;
                        const uint8_t* row = sK + (k * rows + r) * D * 4;
                        float4 v[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (e < 2 || two) v[e] = *reinterpret_cast<const float4*>(row + ((((part * cols + c) / 4 + e) ^ (r & 7)) << 4));
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (e < 2 || two) {
                                acc[e * 4 + 0] += f * v[e].x, acc[e * 4 + 1] += f * v[e].y;
                                acc[e * 4 + 2] += f * v[e].z, acc[e * 4 + 3] += f * v[e].w;
                            }
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e)
                        if (e == 0 || two)
                            *reinterpret_cast<uint4*>(orow + c + e * 8) =
                                make_uint4(pack_bf16x2(acc[e * 8], acc[e * 8 + 1]), pack_bf16x2(acc[e * 8 + 2], acc[e * 8 + 3]),
                                           pack_bf16x2(acc[e * 8 + 4], acc[e * 8 + 5]), pack_bf16x2(acc[e * 8 + 6], acc[e * 8 + 7]));
                }
                if (part == 0) p.lse[(size_t(b) * p.Hq + h) * p.T + q0 + r] = m * p.scale + logf(l);
            }
        }
    }
    // teardown: every role falls through to here, also after a wait that gave up
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, Cfg::kTmemCols);
    }
    B200ATTN_TRACE_END(0);
}

}  // namespace b200attn
