// Causal grouped-query attention backward for sm_100a, the three steps of the
// reference's flash_attn_backward (llm/src/model/flash_attn.cu:428-504, math :137-146):
//   1. preprocess  D[i] = sum_d O[i,d] dO[i,d]            (flash_attn_compute_D_kernel, :150-172)
//                  - done by the dQ pass for its own rows, no separate kernel
//   2. dQ pass     query tile stationary, walks key tiles  (flash_attn_dq_kernel, :175-274)
//   3. dK/dV pass  key tile stationary, walks query tiles  (flash_attn_dkdv_kernel, :277-379)
// with  P = exp(s - L),  dP = dO V^T,  dS = P (dP - D),  dQ = scale dS K,
//       dK = scale dS^T Q,  dV = P^T dO.
// Both passes recompute P from the saved logsumexp on the tensor cores; neither uses
// atomics, so results are bit-reproducible.  GQA: the dK/dV CTA of a KV head loops over
// the query heads of its group and keeps one accumulator, which replaces
// accumulate_kv_grads (llm/src/model/attention.cu:412-429,510-543).
//
// Roles in the dK/dV pass (640 threads; the dQ pass is described at its kernel):
//   warps 0-15  compute: thread owns TMEM lane (warp % 4) * 32 + lane and 32 of the 128 score columns (warp / 4); four warps
//               per scheduler hide the TMEM and MUFU latencies of one another
//   warp  16    TMA producer (converged warp, one elected lane issues)
//   warp  17    TMEM allocation and the products S^T (converged warp, one elected lane issues)
//   warp  18    the other products
//   warp  19    D = 64: the row vectors as MMA operands (see there); else idle
// TMEM (512 columns): S [0,128), dP blocks of 128 columns (two at D = 64, one at D = 128), then the dV and dK accumulators.
//   The compute warps take a unit's scores into registers in one go and hand the S buffer back at once, so the next S^T runs
//   under this unit's exponentials; P^T and dS^T go over the unit's dP block.
// The compute step has two phases so that it can start on S before dP has arrived:
//   A: P = exp2(S * scale*log2e - L*log2e)   (kept in registers)
//   B: dS = P * (dP - D)                      (stored over dP as BF16, in the dK/dV pass beside P)
#pragma once

#include "ptx.cuh"

namespace b200attn {

struct BwdParams {
    int B, T, Tpad, Hq, Hkv, group, n_tiles;
    float scale, scale_log2;
    const float* lse2;  // [B, Hq, Tpad]  logsumexp * log2(e); +inf in the padding rows   (read by the dK/dV pass)
    const float* dvec;  // [B, Hq, Tpad]  rowsum(O * dO);       0 in the padding rows     (read by the dK/dV pass)
    float* lse2_w;      // the same two vectors, written by the dQ pass
    float* dvec_w;
    const float* lse;       // [B, Hq, T]
    const uint16_t* o;      // forward output, q layout
    const uint16_t* dout;   // upstream gradient, q layout
    uint16_t* dq;           // q layout
    long long q_st, q_sh, q_sb;  // element strides of the q layout: token, head, batch
    int* status;
    uint16_t* dk;           // k layout
    uint16_t* dv;           // k layout
    long long k_st, k_sh, k_sb;  // element strides of the k layout: token, head, batch
    int* sched;   // two words of the device-wide item counter of the persistent dQ pass (see ptx.cuh), or nullptr
    int* sched2;  // the same for the dK/dV pass
    int split;    // CTAs (a cluster) that share an item's key tiles (dQ pass) or units (dK/dV pass); 1 except in the split kernels
    FastDiv div_split;
    FastDiv div_bhq, div_hq, div_bhkv, div_hkv, div_group;  // division by B * Hq, Hq, B * Hkv, Hkv and the group size
    int early;    // whether the next kernel may start while this one's last items are worked on (see ptx.cuh)
};

template <int D>
struct BwdCfg {
    static constexpr int kStages = D == 64 ? 4 : 2;   // streamed operand pairs (Q, dO) in shared memory
    static constexpr int kTileBytes = 128 * D * 2;
    static constexpr int kBoxBytes = 128 * 64 * 2;
    static constexpr int kBoxes = D / 64;
    static constexpr int kVecBytes = kStages * 2 * 512;  // per stage (lse2, dvec) of 128 rows
    static constexpr int kBarBytes = 512;
    static constexpr int kKvBufs = D == 64 ? 2 : 1;      // K/V tile pairs in shared memory (the next item's are prefetched)
    static constexpr int kPartCols = 16;                 // score columns whose P^T and dS^T lie side by side
    static constexpr int kCols = 32;                     // score columns per compute thread
    static constexpr int kComputeThreads = 512;
    static constexpr int kThreads = kComputeThreads + 128;
    // registers per thread of the compute warps and of the others: together the launch's kThreads x 96
    static constexpr int kRegsCompute = 104, kRegsOther = 64;
    static_assert(kRegsCompute * kComputeThreads + kRegsOther * 128 <= 96 * kThreads, "more registers than the launch has");
    static constexpr bool kVecOps = D == 64;             // the row vectors enter the products (see the row-vector warp)
    static constexpr int kOpBytes = 128 * 16;            // a row vector as MMA operand: 8 BF16 per row
    static constexpr int kOpsBytes = kVecOps ? (2 * kStages + 2) * kOpBytes : 0;  // two per stage, ones, zeros
    static constexpr int kOutBytes = D == 64 ? 0 : (kComputeThreads / 32) * kRowStageBytes;  // D = 64: in the item's own K/V tiles
    static constexpr int kSmemBytes = (2 * kKvBufs + 2 * kStages) * kTileBytes + kOutBytes + kVecBytes + kOpsBytes + kBarBytes;
    static_assert(kSmemBytes <= 232448, "shared memory of an SM");
    static constexpr int kTmemCols = 512;
    static constexpr int kDpBufs = D == 64 ? 2 : 1;
    static constexpr int kColS = 0;
    static constexpr int kColAcc0 = 128 + 128 * kDpBufs;  // dV
    static constexpr int kColAcc1 = kColAcc0 + D;         // dK
    static_assert(kColAcc1 + D <= kTmemCols, "tensor memory");
    __host__ __device__ static constexpr int col_dp(int buf) { return 128 + 128 * buf; }
};

// D[tmem] = A[smem, K-major] * B[smem, K-major]^T over the head dimension; a_desc / b_desc
// describe K step 0 of each operand.
template <int D>
__device__ __forceinline__ void issue_ss_over_headdim(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                                      uint32_t idesc) {
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks)
        umma_ss(d_tmem, a_desc + kmajor_step(ks, BwdCfg<D>::kBoxBytes), b_desc + kmajor_step(ks, BwdCfg<D>::kBoxBytes),
                idesc, ks > 0);
}

// D[tmem] (+)= A[tmem, BF16 pairs] * B[smem, MN-major] over 128 rows of B (b_desc describes
// rows 0..15).  The A operand lies in pieces of 16 values (8 columns) that are kPartCols columns apart.
template <int D>
__device__ __forceinline__ void issue_ts_over_rows(uint32_t d_tmem, uint32_t a_col, uint64_t b_desc, uint32_t idesc,
                                                   bool accumulate) {
#pragma unroll
    for (int ks = 0; ks < 8; ++ks)
        umma_ts(d_tmem, a_col + ks * BwdCfg<D>::kPartCols, b_desc + uint64_t(ks * 128), idesc, accumulate || ks > 0);
}

template <int D>
__device__ __forceinline__ uint64_t kmajor_desc(const void* tile) {
    return make_sdesc_sw128(smem_u32(tile), 16, 1024);
}
template <int D>
__device__ __forceinline__ uint64_t mnmajor_desc(const void* tile) {
    return make_sdesc_sw128(smem_u32(tile), BwdCfg<D>::kBoxBytes, 1024);
}

// The end of an item that a cluster shares (SPLIT): every CTA holds the dQ sums of its key tiles in tensor memory (32 columns from t_acc on
// per part of the compute warps).  Query row r of the tile is finished by CTA r / rows, which adds the shares up in their order.  The
// compute warps come here, also after a wait that gave up, and all other warps of the cluster to dq_exchange_idle; the tiles in shared
// memory make room for the arrivals, so all CTAs must be through with theirs first.  Nobody writes an item of which a CTA has failed.
__device__ __forceinline__ void dq_exchange_idle(const BwdParams& p, volatile uint32_t* fail, int rank) {
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (int(threadIdx.x) < p.split) cluster_store_1(const_cast<uint32_t*>(fail) + rank, threadIdx.x, 1u);  // the CTA left at its start
    __syncwarp();
    cluster_arrive();
    cluster_wait();
}
template <int D, typename Begin>
__device__ __forceinline__ void dq_exchange(const BwdParams& p, uint8_t* smem, volatile uint32_t* fail, const volatile int* abort_flag, uint32_t t_acc,
                                            int id, int rank, bool any, Begin share_begin) {
    constexpr int kThreads = 4 * D;  // the compute warps: 128 rows x D / 32 parts
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rows = 128 / p.split;
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    const bool failed = *abort_flag != 0;  // (final: every warp of the CTA has passed the barrier)
    if (tid < p.split) cluster_store_1(const_cast<uint32_t*>(fail) + rank, tid, failed);
    __syncwarp();
    if (tid < kThreads && !failed && any) {
        tc_fence_after_sync();
        const int row = (warp & 3) * 32 + lane, part = warp >> 2, to = (row * p.split) >> 7, r = row - to * rows;
        // [source CTA][row][D] FP32, 16-byte pieces swizzled by the row: the rows of a warp would share a bank
        uint8_t* own = smem + (rank * rows + r) * D * 4;
        const uint32_t dst = cluster_addr(own, to);
        uint32_t v[32];
        tmem_ld_x32(t_acc + (uint32_t((warp & 3) * 32) << 16) + part * 32, v);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = ((part * 8 + i) ^ (r & 7)) << 4;
            if (to == rank)
                *reinterpret_cast<uint4*>(own + at) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            else
                cluster_store_4(dst + at, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
        tc_fence_before_sync();
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    bool good = true;
    for (int k = 0; k < p.split; ++k) good = good && fail[k] == 0;
    if (tid < kThreads && good) {
        const int n_bh = p.B * p.Hq, qt = int(fastdiv(unsigned(id), p.div_bhq)), bh = id - qt * n_bh, b = int(fastdiv(unsigned(bh), p.div_hq));
        const int q0 = (p.n_tiles - 1 - qt) * 128 + rank * rows;
        uint16_t* out = p.dq + size_t(b) * p.q_sb + size_t(bh - b * p.Hq) * p.q_sh + size_t(q0) * p.q_st;
        for (int i = tid; i < rows * (D / 8); i += kThreads) {  // eight columns each
            const int r = i / (D / 8), c8 = i % (D / 8);
            if (q0 + r >= p.T) break;
            float acc[8] = {};
#pragma unroll 2
            for (int k = 0; k < p.split; ++k) {
                if (share_begin(k + 1) == share_begin(k)) continue;  // nothing was sent
                const uint8_t* src = smem + (k * rows + r) * D * 4;
                const float4 v0 = *reinterpret_cast<const float4*>(src + (((c8 * 2) ^ (r & 7)) << 4));
                const float4 v1 = *reinterpret_cast<const float4*>(src + (((c8 * 2 + 1) ^ (r & 7)) << 4));
                acc[0] += v0.x, acc[1] += v0.y, acc[2] += v0.z, acc[3] += v0.w;
                acc[4] += v1.x, acc[5] += v1.y, acc[6] += v1.z, acc[7] += v1.w;
            }
            *reinterpret_cast<uint4*>(out + size_t(r) * p.q_st + c8 * 8) =
                make_uint4(pack_bf16x2(acc[0] * p.scale, acc[1] * p.scale), pack_bf16x2(acc[2] * p.scale, acc[3] * p.scale),
                           pack_bf16x2(acc[4] * p.scale, acc[5] * p.scale), pack_bf16x2(acc[6] * p.scale, acc[7] * p.scale));
        }
    }
}

// ---------------------------------------------------------------------------------------
// dQ pass (D = 64): persistent CTAs, two per SM.  A CTA walks a list of work items (item = one 128-row query tile
// of one (batch, query head); items are ordered heaviest first), and every pipeline keeps running across item
// boundaries.  The O tile travels with Q and dO, so the preprocess D = rowsum(O * dO)
// (flash_attn_compute_D_kernel, llm/src/model/flash_attn.cu:150-172) is shared-memory work once per item; D and L * log2(e)
// are also left in the workspace for the dK/dV pass, which therefore has to run after this kernel.
//
// Q and dO in tensor memory.  Every D = 64 kernel here is bound by the shared-memory data path (a product M128 N64
// K16 with both operands in shared memory fetches 4 KB of A and 2 KB of B for 32 clocks of math), and Q and dO are
// the A operands of every S = Q K^T and dP = dO V^T product of an item.  The two tiles are therefore copied
// once per item from shared memory into tensor memory (tcgen05.cp, issued by the MMA warp in front of the products that read
// them), all three products of a key tile take their A operand from tensor memory, and the shared-memory tiles are free for
// the NEXT item's loads while this item is still being worked on.
//
// Row warps.  What happens once per item - the preprocess, the dQ rows on their way out - has four warps of its own, beside the
// compute warps that go from one item's last tile to the next item's first; the next item's first scores are computed under the
// last tile.  Done by the compute warps, the copy into tensor memory too, it kept them from 3400 clocks of tiles per item (1250 a
// tile).  Measured on B200, us for both passes of the backward, with the row warps and then with the copies as tcgen05.cp: B=32
// T=512 6/2 47.0 -> 45.4 -> 44.7, B=16 T=1024 16/4 163.5 -> 161.0 -> 158.3, B=8 T=2000 16/4 279 -> 275.7 -> 274.5, B=2 T=128 6/2
// 12.15 -> 12.26 -> 12.06.  dS through shared memory instead of over the dP block, so that the next dP need not wait for dQ, was slower
// (B=16 T=1024: 168 against 162): the tiles of two CTAs cover that wait already.
//
// SPLIT: few, long items (few sequences and heads).  A CTA works on a share of ONE item's key tiles, and the CTAs of a cluster that share it
// exchange their dQ sums through distributed shared memory at the end (dq_exchange); the sums are in a fixed order, so dQ is
// bit-reproducible.  What bounds it: the chain of the longest share's tiles, 0.43 us each, and 2 us for the exchange.  At B=1 T=4000 2/1 both
// passes took 61 us with an item per CTA and take 44.
//
// Roles (512 threads): warps 0-7 compute (thread owns query row (warp % 4) * 32 + lane == TMEM lane and the 32 key
// columns of its part warp / 4), warps 8-11 rows, warp 12 TMA producer, warp 13 TMEM allocation + MMA issue (converged
// warps, one elected lane issues), warps 14-15 idle (they complete a warpgroup, the unit in which registers are dealt).
// TMEM (256 columns): S [0,64), dP [64,128) (dS as BF16 over the first 16 columns of each part's range), dQ
// accumulator [128,192), Q [192,224), dO [224,256).  There is one S buffer: the compute warps read a tile's scores
// into registers in one go and hand the buffer back at once, so the next tile's Q K^T runs under this tile's
// exponentials; dS overwrites dP, so the next dP product follows the dQ product that consumes it.
// ---------------------------------------------------------------------------------------
template <int D>
struct DqCfg {
    static constexpr int kKeys = 64;
    static constexpr int kStages = 3;
    static constexpr int kQTileBytes = 128 * D * 2;
    static constexpr int kQBoxBytes = 128 * 64 * 2;
    static constexpr int kKVTileBytes = kKeys * D * 2;
    static constexpr int kKVBoxBytes = kKeys * 64 * 2;
    static constexpr int kBoxes = D / 64;
    static constexpr int kOutBytes = 4 * kRowStageBytes;  // per row warp: its output rows on their way to global memory
    static constexpr int kVecBytes = 2 * 128 * 8;         // (L * log2(e), D) of the rows of two items
    static constexpr int kSmemBytes = 3 * kQTileBytes + 2 * kStages * kKVTileBytes + kOutBytes + kVecBytes + 512;  // Q, dO, O + ring + barriers
    static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs per SM");
    static constexpr int kTmemCols = 256;
    static constexpr int kCtasPerSm = 2;
    static constexpr int kColS = 0, kColDP = 64, kColAcc = 128, kColQ = 192, kColDO = 224;
    static constexpr int kParts = 2;
    static constexpr int kPartCols = kKeys / kParts;  // 32
    static constexpr int kComputeThreads = 128 * kParts;
    static constexpr int kThreads = kComputeThreads + 256;
    static constexpr int kRowWarp = 4 * kParts, kProducerWarp = kRowWarp + 4, kMmaWarp = kProducerWarp + 1;
    // registers per thread of the compute warps, the row warps and the others: together the launch's kThreads x 64
    static constexpr int kRegsCompute = 80, kRegsRow = 56, kRegsOther = 40;
    static_assert(kRegsCompute * kComputeThreads + (kRegsRow + kRegsOther) * 128 <= 64 * kThreads, "more registers than the launch has");
};

template <int D, bool SPLIT>
__global__ void __launch_bounds__(DqCfg<D>::kThreads, DqCfg<D>::kCtasPerSm)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmO, const BwdParams p, const __grid_constant__ ItemTable tab) {
    static_assert(D == 64, "the persistent dQ pass keeps Q and dO in 64 tensor-memory columns: D = 64 only");
    using Cfg = DqCfg<D>;
    constexpr int NST = Cfg::kStages;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;
    uint8_t* sdO = sQ + Cfg::kQTileBytes;
    uint8_t* sO = sdO + Cfg::kQTileBytes;
    uint8_t* sK = sO + Cfg::kQTileBytes;         // [NST]
    uint8_t* sV = sK + NST * Cfg::kKVTileBytes;  // [NST]
    uint8_t* sOut = sV + NST * Cfg::kKVTileBytes;  // [4 row warps]
    float2* sVec = reinterpret_cast<float2*>(sOut + Cfg::kOutBytes);  // [2][128], by item parity
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + Cfg::kOutBytes + Cfg::kVecBytes);
    uint64_t* bar_q = bars + 0;         // Q, dO, O of an item have landed in shared memory      (phase: item)
    uint64_t* bar_qs_free = bars + 1;   // those three tiles have been read                       (phase: item)
    uint64_t* bar_vec = bars + 10;      // [2] by item parity: the item's row vectors are in sVec (phase: item / 2)
    uint64_t* bar_s_full = bars + 3;    //                                                         (phase: tile)
    uint64_t* bar_s_loaded = bars + 4;  // S is in registers: the buffer may be overwritten       (phase: tile)
    uint64_t* bar_dp_full = bars + 5;   //                                                         (phase: tile)
    uint64_t* bar_ds_full = bars + 6;   // dS written over dP                                      (phase: tile)
    uint64_t* bar_acc = bars + 8;       // dQ accumulator of an item complete                      (phase: item)
    uint64_t* bar_acc_free = bars + 9;  // dQ accumulator read by the epilogue                     (phase: item)
    uint64_t* bar_kv_full = bars + 14;        // [NST]
    uint64_t* bar_kv_free = bars + 14 + NST;  // [NST]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14 + 2 * NST);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 15 + 2 * NST);
    uint64_t* bar_item = bars + 24;     // [kItemRing] item ids handed out by the producer
    volatile int* item_ring = reinterpret_cast<volatile int*>(bars + 24 + kItemRing);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_bh = p.B * p.Hq;
    const int n_items = p.n_tiles * n_bh;
    // item id -> (query tile, head, batch); ids are ordered by work, heaviest query tile first
    auto item_rest = [&](int id) { return id - int(fastdiv(unsigned(id), p.div_bhq)) * n_bh; };  // b * Hq + h
    auto item_qt = [&](int id) { return p.n_tiles - 1 - int(fastdiv(unsigned(id), p.div_bhq)); };
    auto item_b = [&](int id) { return int(fastdiv(unsigned(item_rest(id)), p.div_hq)); };
    auto item_h = [&](int id) { return item_rest(id) - item_b(id) * p.Hq; };
    auto item_all = [&](int id) { return (min(p.T, item_qt(id) * 128 + 128) + Cfg::kKeys - 1) / Cfg::kKeys; };
    // SPLIT: a CTA's tiles of an item, of cluster CTA r [tiles r / split, tiles (r + 1) / split)
    const int split_id = SPLIT ? int(fastdiv(blockIdx.x, p.div_split)) : 0, rank = SPLIT ? int(blockIdx.x) - split_id * p.split : 0;
    auto share_begin = [&](int r) { return int(fastdiv(unsigned(item_all(split_id) * r), p.div_split)); };
    const int j_first = SPLIT ? share_begin(rank) : 0;
    auto item_nkv = [&](int id) { return SPLIT ? share_begin(rank + 1) - j_first : item_all(id); };
    auto get_item = [&](int n) { return item_get(bar_item, item_ring, n, abort_flag, p.status); };

    B200ATTN_TRACE_BEGIN(1);
    const int id_first = SPLIT ? split_id : sched_first(tab, p.sched, int(blockIdx.x));  // the first item needs no fetch
    const bool any = !SPLIT || item_nkv(id_first) > 0;
    // one thread: Q, dO and O of an item; a tile of K and V
    auto load_rows = [&](int id) {
        const int q0 = item_qt(id) * 128, h = item_h(id), b = item_b(id);
        mbar_arrive_expect_tx(bar_q, 3 * Cfg::kQTileBytes);
        tma_load_4d(sQ, &tmQ, bar_q, 0, q0, h, b);
        tma_load_4d(sdO, &tmdO, bar_q, 0, q0, h, b);
        tma_load_4d(sO, &tmO, bar_q, 0, q0, h, b);
    };
    auto load_kv = [&](int s, int j, int hk, int b) {
        mbar_arrive_expect_tx(&bar_kv_full[s], 2 * Cfg::kKVTileBytes);
        tma_load_4d(sK + s * Cfg::kKVTileBytes, &tmK, &bar_kv_full[s], 0, j * Cfg::kKeys, hk, b);
        tma_load_4d(sV + s * Cfg::kKVTileBytes, &tmV, &bar_kv_full[s], 0, j * Cfg::kKeys, hk, b);
    };
    if (warp == Cfg::kProducerWarp && lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmdO);
        tma_prefetch_desc(&tmO);
        mbar_init(bar_q, 1);
        mbar_init(bar_qs_free, 128 + 1);  // the row warps, and the MMA warp's copies
        mbar_init(&bar_vec[0], 128);
        mbar_init(&bar_vec[1], 128);
        mbar_init(bar_s_full, 1);
        mbar_init(bar_s_loaded, Cfg::kComputeThreads);
        mbar_init(bar_dp_full, 1);
        mbar_init(bar_ds_full, Cfg::kComputeThreads);
        mbar_init(bar_acc, 1);
        mbar_init(bar_acc_free, 128);
        for (int s = 0; s < NST; ++s) {
            mbar_init(&bar_kv_full[s], 1);
            mbar_init(&bar_kv_free[s], 1);
        }
        for (int i = 0; i < kItemRing; ++i) mbar_init(&bar_item[i], 1);
        fence_mbar_init();
        *abort_flag = 0;
        item_publish(bar_item, item_ring, 0, any ? id_first : -1);
    }
    if (warp == Cfg::kProducerWarp) {
        __syncwarp();
        grid_dep_wait();  // first global access of this CTA comes next
        // The first loads: the status word, the barrier and the roles' start pass under their latency (both passes, us: B=32 T=512 6/2 44.9 -> 44.2,
        // at D = 128 B=20 T=200 8/4 33.6 -> 32.6).
        if (any && elect_one()) {
            load_rows(id_first);
            load_kv(0, j_first, int(fastdiv(unsigned(item_h(id_first)), p.div_group)), item_b(id_first));
            const int failed = *reinterpret_cast<volatile int*>(p.status);
            if (failed != 0) {  // behind an earlier failure the CTA leaves, but not before its loads have landed
                mbar_wait(bar_q, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                mbar_wait(&bar_kv_full[0], 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                *abort_flag = failed;
            }
        }
        __syncwarp();
    }
    if (warp == Cfg::kMmaWarp) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    grid_dep_wait();
    grid_dep_launch();  // the dK/dV pass: only now, see there
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    const bool left = *abort_flag != 0;
    if (left) {
        // an earlier CTA already failed: fall through to the teardown
    } else if (warp > Cfg::kMmaWarp) {
        reg_dealloc<Cfg::kRegsOther>();  // idle warps
    } else if (warp == Cfg::kProducerWarp) {
        // ------------------------------------------------------------------ producer
        reg_dealloc<Cfg::kRegsOther>();
        int g = 0;  // tiles issued so far by this CTA (ring position)
        bool ok = any;
        int id = id_first;
        int id_next = 0;      // lane 0: the id fetched for the next item
        if (lane == 0) id_next = SPLIT ? n_items : sched_fetch(tab, p.sched, 1, int(blockIdx.x), int(gridDim.x));
        __syncwarp();
        for (int n = 0; ok; ++n) {
            const int h = item_h(id), b = item_b(id), hk = int(fastdiv(unsigned(h), p.div_group)), n_kv = item_nkv(id);
            // the next item is taken and announced shortly before this item's loads end, but not before the
            // ring has been filled for this item
            const int j_next = max(min(n_kv, NST) - 1, n_kv - 2);
            int id_new = n_items;
            // the three tiles in shared memory are free as soon as the previous item has been copied out of them
            if (n > 0) ok = mbar_wait_warp(bar_qs_free, (n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
            if (!ok) break;
            if (n > 0 && elect_one()) load_rows(id);
            __syncwarp();
            for (int j = 0; j < n_kv; ++j, ++g) {
                const int s = g % NST;
                if (g >= NST) ok = mbar_wait_warp(&bar_kv_free[s], ((g / NST) - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
                if (!ok) break;
                if (g > 0 && elect_one()) load_kv(s, j_first + j, hk, b);
                __syncwarp();
                if (j == j_next) {
                    id_new = __shfl_sync(0xffffffffu, id_next, 0);
                    if (lane == 0) {
                        item_publish(bar_item, item_ring, n + 1, id_new < n_items ? id_new : -1);
                        if (id_new < n_items) id_next = sched_fetch(tab, p.sched, n + 2, int(blockIdx.x), int(gridDim.x));
                    }
                    __syncwarp();
                }
            }
            if (!ok || id_new >= n_items) break;
            id = id_new;
        }
        if (!SPLIT && ok && lane == 0) sched_finish(p.sched, int(gridDim.x));
    } else if (warp == Cfg::kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer
        reg_dealloc<Cfg::kRegsOther>();
        constexpr uint32_t idesc_s = make_idesc_bf16(128, Cfg::kKeys, 0, 0);  // A in TMEM, B (K or V tile) K-major
        constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);         // A in TMEM, B (K tile) MN-major
        // g numbers this CTA's key tiles across all its items: ring stage g % NST
        // S(g) = Q K^T; the buffer still holds S(g - 1) until it has been read.  first: of an item, whose Q is copied into tensor
        // memory in front (the products that read the Q before it are complete: their scores have been read)
        auto issue_s = [&](int g, bool first) -> bool {
            const int s = g % NST;
            if (g > 0 && !mbar_wait_warp(bar_s_loaded, uint32_t(g - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX))
                return false;
            if (!mbar_wait_warp(&bar_kv_full[s], (g / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD)) return false;
            tc_fence_after_sync();
            const uint64_t k_desc = make_sdesc_sw128(smem_u32(sK + s * Cfg::kKVTileBytes), 16, 1024);
            const uint64_t q_desc = make_sdesc_sw128(smem_u32(sQ), 16, 1024);
            if (elect_one()) {
                if (first) {
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks) tmem_copy_128x32b(tmem + Cfg::kColQ + ks * 8, q_desc + kmajor_step(ks, 0));
                }
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ts(tmem + Cfg::kColS, tmem + Cfg::kColQ + ks * 8, k_desc + kmajor_step(ks, Cfg::kKVBoxBytes), idesc_s, ks > 0);
                umma_commit(bar_s_full);
            }
            __syncwarp();
            return true;
        };
        // dP(g) = dO V^T; tile g's loads have landed (S(g) was issued), and the product that read dS(g - 1) out of
        // this block was issued before (the products execute in order).  first: of an item, whose dO is copied into tensor memory
        // in front (the products that read the dO before it are complete: dS has been made of them)
        auto issue_dp = [&](int g, bool first) {
            const int s = g % NST;
            const uint64_t v_desc = make_sdesc_sw128(smem_u32(sV + s * Cfg::kKVTileBytes), 16, 1024);
            const uint64_t do_desc = make_sdesc_sw128(smem_u32(sdO), 16, 1024);
            if (elect_one()) {
                if (first) {
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks) tmem_copy_128x32b(tmem + Cfg::kColDO + ks * 8, do_desc + kmajor_step(ks, 0));
                    umma_commit(bar_qs_free);
                }
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ts(tmem + Cfg::kColDP, tmem + Cfg::kColDO + ks * 8, v_desc + kmajor_step(ks, Cfg::kKVBoxBytes), idesc_s, ks > 0);
                umma_commit(bar_dp_full);
            }
            __syncwarp();
        };
        int g = 0, n = 0;
        bool ok = true;
        int id = get_item(0);
        // S of the first tile of this CTA's n-th item
        auto start_item = [&]() {
            B200ATTN_STAMP(lane == 0, 440 + 2 * n);
            ok = mbar_wait_warp(bar_q, uint32_t(n) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
            B200ATTN_STAMP(lane == 0, 441 + 2 * n);
            if (ok) ok = issue_s(g, true);
        };
        if (id >= 0) start_item();
        while (ok && id >= 0) {
            const int n_kv = item_nkv(id);
            issue_dp(g, true);
            int id_next = -1;
            for (int j = 0; j < n_kv; ++j) {
                const int s = g % NST;
                ++g;
                if (j + 1 < n_kv) {
                    ok = issue_s(g, false);  // as soon as the tile's scores are in registers
                } else {
                    id_next = get_item(n + 1);
                    ++n;
                    if (id_next >= 0) start_item();
                }
                if (ok) ok = mbar_wait_warp(bar_ds_full, uint32_t(g - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                if (!ok) break;
                B200ATTN_STAMP(lane == 0, 240 + 8 * (g - 1) + 5);
                // the accumulator still belongs to the previous item's epilogue until it has been read
                if (j == 0 && n - (n_kv == 1) > 0) {
                    ok = mbar_wait_warp(bar_acc_free, uint32_t(n - (n_kv == 1) - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                    if (!ok) break;
                }
                tc_fence_after_sync();
                const uint64_t kmn_desc = make_sdesc_sw128(smem_u32(sK + s * Cfg::kKVTileBytes), Cfg::kKVBoxBytes, 1024);
                if (elect_one()) {
                    // dQ += dS K : 64 keys = 4 K steps; part q keeps its BF16 dS in the first 16 columns of its range
#pragma unroll
                    for (int ks = 0; ks < Cfg::kKeys / 16; ++ks) {
                        constexpr int kStepsPerPart = Cfg::kPartCols / 16;
                        const uint32_t a_col = Cfg::kColDP + (ks / kStepsPerPart) * Cfg::kPartCols + (ks % kStepsPerPart) * 8;
                        umma_ts(tmem + Cfg::kColAcc, tmem + a_col, kmn_desc + uint64_t(ks * 128), idesc_acc, (j > 0) || (ks > 0));
                    }
                    umma_commit(&bar_kv_free[s]);
                    if (j + 1 == n_kv) umma_commit(bar_acc);
                }
                __syncwarp();
                B200ATTN_STAMP(lane == 0, 240 + 8 * (g - 1) + 6);
                if (j + 1 < n_kv) issue_dp(g, false);
            }
            id = id_next;
        }
        // drain: nothing may be in flight when TMEM is freed
        if (ok && n > 0) mbar_wait_warp(bar_acc, (n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
    } else if (warp >= Cfg::kRowWarp) {
        // ------------------------------------------------------------------ rows: what happens once per item
        reg_dealloc<Cfg::kRegsRow>();
        const int w4 = warp & 3;
        const int row = w4 * 32 + lane;  // query row in the tile == TMEM lane
        const uint32_t lane_base = uint32_t(w4 * 32) << 16;
        const uint32_t sw = uint32_t(row & 7) << 4;  // the tiles' swizzle
        bool ok = true;
        // dQ rows of the CTA's n_item-th item (times scale) -> BF16 -> global memory
        auto epilogue = [&](int n_item, int id) {
            ok = mbar_wait_warp(bar_acc, uint32_t(n_item) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            if (!ok) return;
            B200ATTN_STAMP(tid == Cfg::kRowWarp * 32, 400 + 4 * n_item + 2);
            tc_fence_after_sync();
            const int q0 = item_qt(id) * 128;
            uint16_t* out = p.dq + size_t(item_b(id)) * p.q_sb + size_t(item_h(id)) * p.q_sh + size_t(q0 + w4 * 32) * p.q_st;
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                uint32_t v[32], w[16];
                tmem_ld_x32(tmem + lane_base + Cfg::kColAcc + c * 32, v);
                tmem_wait_ld();
                if (c + 1 == D / 32) {
                    tc_fence_before_sync();
                    mbar_arrive(bar_acc_free);  // the MMA warp may start the next item's accumulation
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]) * p.scale, __uint_as_float(v[2 * i + 1]) * p.scale);
                store_rows_64b(sOut + w4 * kRowStageBytes, w, lane, out + c * 32, p.q_st, p.T - (q0 + w4 * 32));
            }
            B200ATTN_STAMP(tid == Cfg::kRowWarp * 32, 400 + 4 * n_item + 3);
        };
        int n = 0, id_prev = -1;
        for (int id; ok && (id = get_item(n)) >= 0; ++n) {
            const int q0 = item_qt(id) * 128;
            const size_t bh = size_t(item_b(id)) * p.Hq + item_h(id);
            const bool in_range = q0 + row < p.T;
            // (issued here and first used after the wait below, so that its latency overlaps the wait)
            const float lse_raw = in_range ? p.lse[bh * p.T + q0 + row] : 0.f;
            B200ATTN_STAMP(tid == Cfg::kRowWarp * 32, 400 + 4 * n + 0);
            ok = mbar_wait_warp(bar_q, uint32_t(n) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
            if (!ok) break;
            B200ATTN_STAMP(tid == Cfg::kRowWarp * 32, 400 + 4 * n + 1);
            // the preprocess of this row, D = rowsum(O * dO) and L * log2(e)
            float acc = 0.f;
#pragma unroll
            for (int c = 0; c < D / 8; ++c) {
                const uint32_t off = row * 128 + ((uint32_t(c) << 4) ^ sw);
                const uint4 a = *reinterpret_cast<const uint4*>(sO + off);
                const uint4 gq = *reinterpret_cast<const uint4*>(sdO + off);
                const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
                const uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    acc = fmaf(__uint_as_float(aw[e] << 16), __uint_as_float(gw[e] << 16), acc);
                    acc = fmaf(__uint_as_float(aw[e] & 0xffff0000u), __uint_as_float(gw[e] & 0xffff0000u), acc);
                }
            }
            // exp2(x - inf) = 0: padding query rows contribute nothing
            const float2 vec = make_float2(in_range ? lse_raw * 1.4426950408889634f : INFINITY, in_range ? acc : 0.f);
            // (Every compute warp has passed the barrier and read what the buffer held by the end of that item's epilogue below.  With
            // one barrier for all items a row warp could be an item ahead of another and arrive for both.)
            sVec[(n & 1) * 128 + row] = vec;
            mbar_arrive(&bar_vec[n & 1]);
            const size_t vrow = bh * p.Tpad + q0 + row;
            if (!SPLIT || rank == p.split - 1) {  // (the last share is never empty)
                p.lse2_w[vrow] = vec.x;
                p.dvec_w[vrow] = vec.y;
            }
            // The tiles were read with ordinary loads and will be overwritten by TMA, which works through the async
            // proxy: without this fence the producer's next load, issued the moment the last thread has arrived, may
            // overtake reads that are still in flight (the producer is parked at the barrier whenever the item before
            // was short; dQ rows of whole warps, sometimes of single lanes, then came out wrong once in a few launches).
            fence_proxy_async_smem();
            mbar_arrive(bar_qs_free);  // the three tiles may be overwritten by the next item's loads
            if (n > 0) epilogue(n - 1, id_prev);
            id_prev = id;
        }
        if (!SPLIT && ok && n > 0) epilogue(n - 1, id_prev);
    } else {
        // ------------------------------------------------------------------ compute
        reg_alloc<Cfg::kRegsCompute>();
        const int w4 = warp & 3, part = warp >> 2;
        const int row = w4 * 32 + lane;  // query row in the tile == TMEM lane
        const uint32_t lane_base = uint32_t(w4 * 32) << 16;
        const int c0 = part * Cfg::kPartCols;  // first key column of this thread's part
        bool ok = true;
        const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
        int g = 0, n = 0;
        for (int id; ok && (id = get_item(n)) >= 0; ++n) {
            const int q0 = item_qt(id) * 128, n_kv = item_nkv(id);
            ok = mbar_wait_warp(&bar_vec[n & 1], uint32_t(n >> 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
            if (!ok) break;
            const float2 vec = sVec[(n & 1) * 128 + row];
            const float lse2 = vec.x, dv = vec.y;
            for (int j = 0; j < n_kv; ++j, ++g) {
                ok = mbar_wait_warp(bar_s_full, uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                if (!ok) break;
                B200ATTN_STAMP(tid == 0, 240 + 8 * g + 0);
                tc_fence_after_sync();
                // phase A: P from S (the scores leave tensor memory in one go)
                float pr[32];
                {
                    uint32_t sv[32];
                    tmem_ld_x32(tmem + lane_base + Cfg::kColS + c0, sv);
                    tmem_wait_ld();
                    tc_fence_before_sync();
                    mbar_arrive(bar_s_loaded);
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float x0, x1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), scale2, pack_f32x2(-lse2, -lse2)), x0, x1);
                        pr[i] = ex2_approx(x0);
                        pr[i + 1] = ex2_approx(x1);
                    }
                }
                const int kbase = (j_first + j) * Cfg::kKeys;
                if (kbase + Cfg::kKeys - 1 > q0) {
                    const int lim = q0 + row - kbase - c0;  // columns i <= lim of this part are visible
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (i > lim) pr[i] = 0.f;
                }
                B200ATTN_STAMP(tid == 0, 240 + 8 * g + 1);
                ok = mbar_wait_warp(bar_dp_full, uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                if (!ok) break;
                B200ATTN_STAMP(tid == 0, 240 + 8 * g + 2);
                tc_fence_after_sync();
                // phase B: dS = P (dP - D), written as BF16 over the part's first 16 columns of the dP block
                {
                    uint32_t dp[32], pk[16];
                    const uint32_t t_dp = tmem + lane_base + Cfg::kColDP + c0;
                    tmem_ld_x32(t_dp, dp);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float y0, y1;
                        unpack_f32x2(mul_f32x2(pack_f32x2(pr[i], pr[i + 1]),
                                               add_f32x2(pack_f32x2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), pack_f32x2(-dv, -dv))), y0, y1);
                        pk[i / 2] = pack_bf16x2(y0, y1);
                    }
                    tmem_st_x16(t_dp, pk);
                }
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive(bar_ds_full);
                B200ATTN_STAMP(tid == 0, 240 + 8 * g + 3);
            }
        }
        if constexpr (SPLIT) {
            if (ok && n > 0) mbar_wait_warp(bar_acc, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            dq_exchange<D>(p, smem, reinterpret_cast<volatile uint32_t*>(sVec), abort_flag, tmem + Cfg::kColAcc, split_id, rank, any, share_begin);
        }
    }

    if (SPLIT && (warp >= Cfg::kRowWarp || left)) dq_exchange_idle(p, reinterpret_cast<volatile uint32_t*>(sVec), rank);
    tc_fence_before_sync();
    __syncthreads();
    if (warp == Cfg::kMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, Cfg::kTmemCols);
    }
    B200ATTN_TRACE_END(1);
}

// ---------------------------------------------------------------------------------------
// dQ pass for D = 128: persistent CTAs, one per SM, that walk a list of the same items; 128-key tiles loaded by TMA and worked
// on as two halves of 64 keys.  As in the D = 64 kernel, Q and dO are copied once per item from shared memory into tensor memory,
// so that S = Q K^T, dP = dO V^T and dQ += dS K all take their A operand from there (a 128-wide product with
// A in shared memory fetches 4 KB of A and 4 KB of B per K step).
// The halves are two streams with their own barriers: S of the next tile's half follows as soon as this one's scores are in
// registers, and dP of the next tile's half as soon as dQ has read dS out of its block, so one half's products run under the
// other half's arithmetic.  (With whole tiles and one dP block, dS, dQ and the next dP followed one another: 3900 clocks per
// 128 x 128 block for 1800 of tensor-pipe time, against 2020 now.  There is no room for a second dP block beside S, dQ, Q and dO.)
// The halves' dQ products are issued by one warp in a fixed order, so dQ is bit-reproducible.
// What bounds it: the tensor pipe inside an item.  Between two items a CTA of its own for each left the pipe idle for 3 us (its
// start, the preprocess from global memory, Q and dO, K and V, the way out of dQ); now the ring of loads runs on into the next item,
// whose Q and dO take one place in it, and row warps of their own do the preprocess and the dQ rows, as in the D = 64 kernel.
// SPLIT as in the D = 64 kernel: the exchange is 64 KB of every CTA, 5.6 us (B=1 T=4000 2/1 77 -> 65 us for both passes).
// Measured on B200, us for both passes of the backward: B=8 T=512 6/2 39.0 -> 33.6, B=20 T=200 8/4 41.2 -> 33.4, B=8 T=1024 16/4
// 168 -> 146, B=32 T=1001 1/1 48.2 -> 43.2, B=4 T=2048 16/4 267 -> 245, B=4 T=8192 16/4 3437 -> 3375; one item per CTA: B=2 T=128 6/2
// 15.7 both, B=1 T=2000 6/2 53.2 -> 53.5.
//
// Roles (736 threads): warps 0-15 compute (thread owns row (warp % 4) * 32 + lane and 32 of the half's 64 columns: half
// warp / 8, part (warp / 4) % 2), warps 16-19 rows, warp 20 TMA producer, warp 21 TMEM allocation and S, warp 22 dQ and dP.
// A CTA's first preprocess and its last dQ rows, which nothing hides, are the sixteen compute warps' instead.
// Shared memory: three ring places of 64 KB, Q and dO of an item or K and V of a tile.
// TMEM (512 columns): S [0,128), dP [128,256) (dS as BF16 over the first 16 columns of each part's range), dQ
// accumulator [256,384), Q [384,448), dO [448,512).
// ---------------------------------------------------------------------------------------
template <int D>
struct DqWideCfg {
    static constexpr int kStages = 3;  // ring places
    static constexpr int kTileBytes = 128 * D * 2;
    static constexpr int kBoxBytes = 128 * 64 * 2;
    static constexpr int kBoxes = D / 64;
    static constexpr int kComputeThreads = 512, kStreamThreads = 256, kRowThreads = 128, kThreads = kComputeThreads + kRowThreads + 96;
    static constexpr int kOutBytes = 4 * kRowStageBytes;  // per row warp: its output rows on their way to global memory
    static constexpr int kVecBytes = 2 * 128 * 8 + 512;   // (L * log2(e), D) of the rows of two items; D of the first
    static constexpr int kSmemBytes = 2 * kStages * kTileBytes + kOutBytes + kVecBytes + 512;
    static_assert(kSmemBytes <= 232448, "shared memory of an SM");
    static constexpr int kTmemCols = 512;
    static constexpr int kColS = 0, kColDP = 128, kColAcc = 256, kColQ = 384, kColDO = 448;
};

// D = rowsum(O * dO) of PASSES * 256 / D rows of a tile from r0 on, by one warp from global memory, D / 8 lanes to a row
template <int D, int PASSES>
struct RowSums {
    static constexpr int LPR = D / 8, RPP = 32 / LPR;
    uint4 a[PASSES], g[PASSES];
    __device__ __forceinline__ void load(const BwdParams& p, size_t tile_off, int q0, int r0, int lane) {
#pragma unroll
        for (int i = 0; i < PASSES; ++i) {
            const int r = r0 + i * RPP + lane / LPR;
            a[i] = g[i] = make_uint4(0u, 0u, 0u, 0u);
            if (q0 + r < p.T) {
                const size_t off = tile_off + size_t(q0 + r) * p.q_st + (lane % LPR) * 8;
                a[i] = *reinterpret_cast<const uint4*>(p.o + off);
                g[i] = *reinterpret_cast<const uint4*>(p.dout + off);
            }
        }
    }
    template <typename Use>  // `use(r, D)` by the first lane of a row
    __device__ __forceinline__ void sum(int r0, int lane, Use use) const {
#pragma unroll
        for (int i = 0; i < PASSES; ++i) {
            const uint32_t aw[4] = {a[i].x, a[i].y, a[i].z, a[i].w};
            const uint32_t gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
            float acc = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc = fmaf(__uint_as_float(aw[e] << 16), __uint_as_float(gw[e] << 16), acc);
                acc = fmaf(__uint_as_float(aw[e] & 0xffff0000u), __uint_as_float(gw[e] & 0xffff0000u), acc);
            }
#pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane % LPR == 0) use(r0 + i * RPP + lane / LPR, acc);
        }
    }
};
template <int D, int PASSES, typename Use>
__device__ __forceinline__ void row_sums(const BwdParams& p, size_t tile_off, int q0, int r0, int lane, Use use) {
    RowSums<D, PASSES> s;
    s.load(p, tile_off, q0, r0, lane);
    s.sum(r0, lane, use);
}

template <int D, bool SPLIT>
__global__ void __launch_bounds__(DqWideCfg<D>::kThreads, 1)
attn_bwd_dq_wide_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const BwdParams p, const __grid_constant__ ItemTable tab) {
    static_assert(D == 128, "Q and dO take 2 x 64 tensor-memory columns: D = 128 only");
    using Cfg = DqWideCfg<D>;
    constexpr int NST = Cfg::kStages;
    extern __shared__ __align__(1024) uint8_t smem[];
    auto place_a = [&](int e) { return smem + (e % NST) * 2 * Cfg::kTileBytes; };  // Q or K of ring entry e
    auto place_b = [&](int e) { return smem + (e % NST) * 2 * Cfg::kTileBytes + Cfg::kTileBytes; };  // dO or V
    uint8_t* sOut = smem + 2 * NST * Cfg::kTileBytes;                 // [4 row warps]
    float2* sVec = reinterpret_cast<float2*>(sOut + Cfg::kOutBytes);  // [2][128], by item parity
    float* sD = reinterpret_cast<float*>(sVec + 2 * 128);             // [128] rowsum(O * dO) of the CTA's first item
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOut + Cfg::kOutBytes + Cfg::kVecBytes);
    uint64_t* bar_full = bars + 0;      // [NST] a ring entry has landed                       (phase: entry / NST)
    uint64_t* bar_free = bars + 3;      // [NST] both MMA warps are through with it            (phase: entry / NST)
    uint64_t* bar_s_full = bars + 6;    // [2] per half                                        (phase: tile)
    uint64_t* bar_s_loaded = bars + 8;  // [2] S is in registers: the half may be overwritten  (phase: tile)
    uint64_t* bar_dp_full = bars + 10;  // [2]                                                 (phase: tile)
    uint64_t* bar_ds_full = bars + 12;  // [2] dS written over dP                              (phase: tile)
    uint64_t* bar_vec = bars + 14;      // [2] by item parity: the row vectors are in sVec     (phase: (item - 1) / 2)
    uint64_t* bar_acc = bars + 16;      // dQ accumulator of an item complete                  (phase: item)
    uint64_t* bar_acc_free = bars + 17; // dQ accumulator read by the row warps                (phase: item)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 19);
    uint64_t* bar_item = bars + 24;     // [kItemRing] item ids handed out by the producer
    volatile int* item_ring = reinterpret_cast<volatile int*>(bars + 24 + kItemRing);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kRowWarp = Cfg::kComputeThreads / 32, kProducerWarp = kRowWarp + 4, kMmaSWarp = kProducerWarp + 1;
    const int n_bh = p.B * p.Hq;
    const int n_items = p.n_tiles * n_bh;
    // item id -> (query tile, head, batch); ids are ordered by work, heaviest query tile first
    auto item_rest = [&](int id) { return id - int(fastdiv(unsigned(id), p.div_bhq)) * n_bh; };  // b * Hq + h
    auto item_qt = [&](int id) { return p.n_tiles - 1 - int(fastdiv(unsigned(id), p.div_bhq)); };
    auto item_b = [&](int id) { return int(fastdiv(unsigned(item_rest(id)), p.div_hq)); };
    auto item_h = [&](int id) { return item_rest(id) - item_b(id) * p.Hq; };
    auto item_all = [&](int id) { return item_qt(id) + 1; };
    // SPLIT: a CTA's tiles of an item, of cluster CTA r [tiles r / split, tiles (r + 1) / split)
    const int split_id = SPLIT ? int(fastdiv(blockIdx.x, p.div_split)) : 0, rank = SPLIT ? int(blockIdx.x) - split_id * p.split : 0;
    auto share_begin = [&](int r) { return int(fastdiv(unsigned(item_all(split_id) * r), p.div_split)); };
    const int j_first = SPLIT ? share_begin(rank) : 0;
    auto item_nkv = [&](int id) { return SPLIT ? share_begin(rank + 1) - j_first : item_all(id); };
    auto get_item = [&](int n) { return item_get(bar_item, item_ring, n, abort_flag, p.status); };
    auto q_offset = [&](int id) { return size_t(item_b(id)) * p.q_sb + size_t(item_h(id)) * p.q_sh; };

    B200ATTN_TRACE_BEGIN(1);
    const int id_first = SPLIT ? split_id : sched_first(tab, p.sched, int(blockIdx.x));  // the first item needs no fetch
    const bool any = !SPLIT || item_nkv(id_first) > 0;
    // one thread: ring entry e
    auto load = [&](int e, const CUtensorMap* ma, const CUtensorMap* mb, int row, int head, int b) {
        uint64_t* full = &bar_full[e % NST];
        mbar_arrive_expect_tx(full, 2 * Cfg::kTileBytes);
#pragma unroll
        for (int bx = 0; bx < Cfg::kBoxes; ++bx) {
            tma_load_4d(place_a(e) + bx * Cfg::kBoxBytes, ma, full, bx * 64, row, head, b);
            tma_load_4d(place_b(e) + bx * Cfg::kBoxBytes, mb, full, bx * 64, row, head, b);
        }
    };
    if (warp == kProducerWarp && lane == 0) {
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmdO);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_s_full[i], 1);
            mbar_init(&bar_s_loaded[i], Cfg::kStreamThreads);
            mbar_init(&bar_dp_full[i], 1);
            mbar_init(&bar_ds_full[i], Cfg::kStreamThreads);
            mbar_init(&bar_vec[i], Cfg::kRowThreads);
        }
        mbar_init(bar_acc, 1);
        mbar_init(bar_acc_free, Cfg::kRowThreads);
        for (int s = 0; s < NST; ++s) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_free[s], 2);
        }
        for (int i = 0; i < kItemRing; ++i) mbar_init(&bar_item[i], 1);
        fence_mbar_init();
        *abort_flag = 0;
        item_publish(bar_item, item_ring, 0, any ? id_first : -1);
    }
    if (warp == kProducerWarp) {
        __syncwarp();
        // launched with programmatic stream serialization: wait for the previous kernel before any global access
        grid_dep_wait();
        if (any && elect_one()) {  // the first loads: the status word, the barrier and the roles' start pass under their latency
            const int h = item_h(id_first), b = item_b(id_first);
            load(0, &tmQ, &tmdO, item_qt(id_first) * 128, h, b);
            load(1, &tmK, &tmV, j_first * 128, int(fastdiv(unsigned(h), p.div_group)), b);
            const int failed = *reinterpret_cast<volatile int*>(p.status);
            if (failed != 0) {  // behind an earlier failure the CTA leaves, but not before its loads have landed
                for (int e = 0; e < 2; ++e) mbar_wait(&bar_full[e], 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                *abort_flag = failed;
            }
        }
        __syncwarp();
    }
    if (warp == kMmaSWarp) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    grid_dep_wait();
    grid_dep_launch();  // the dK/dV pass: only now, see there
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    const bool left = *abort_flag != 0;
    if (left) {
        // an earlier CTA already failed: fall through to the teardown
    } else if (warp == kProducerWarp) {
        // ------------------------------------------------------------------ producer (whole warp, one lane issues)
        int e = 0;  // ring entries issued so far by this CTA
        bool ok = any;
        int id = id_first;
        int id_next = 0;  // lane 0: the id fetched for the next item
        if (lane == 0) id_next = SPLIT ? n_items : sched_fetch(tab, p.sched, 1, int(blockIdx.x), int(gridDim.x));
        __syncwarp();
        auto next_entry = [&](const CUtensorMap* ma, const CUtensorMap* mb, int row, int head, int b) {
            if (e >= NST) ok = mbar_wait_warp(&bar_free[e % NST], uint32_t(e / NST - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
            if (!ok) return;
            if (e >= 2 && elect_one()) load(e, ma, mb, row, head, b);  // (the first two are under way)
            __syncwarp();
            ++e;
        };
        for (int n = 0; ok; ++n) {
            const int h = item_h(id), b = item_b(id), hk = int(fastdiv(unsigned(h), p.div_group)), n_kv = item_nkv(id);
            // the next item is taken and announced shortly before this item's loads end, but not before the
            // ring has been filled for this item
            const int j_next = max(min(n_kv, NST - 1) - 1, n_kv - 2);
            int id_new = n_items;
            next_entry(&tmQ, &tmdO, item_qt(id) * 128, h, b);
            for (int j = 0; j < n_kv && ok; ++j) {
                next_entry(&tmK, &tmV, (j_first + j) * 128, hk, b);
                if (ok && j == j_next) {
                    id_new = __shfl_sync(0xffffffffu, id_next, 0);
                    if (lane == 0) {
                        item_publish(bar_item, item_ring, n + 1, id_new < n_items ? id_new : -1);
                        if (id_new < n_items) id_next = sched_fetch(tab, p.sched, n + 2, int(blockIdx.x), int(gridDim.x));
                    }
                    __syncwarp();
                }
            }
            if (!ok || id_new >= n_items) break;
            id = id_new;
        }
        if (!SPLIT && ok && lane == 0) sched_finish(p.sched, int(gridDim.x));
    } else if (warp >= kMmaSWarp) {
        // ------------------------------------------------------------------ MMA issuers (whole warps, one lane issues)
        constexpr uint32_t idesc_s = make_idesc_bf16(128, 64, 0, 0);    // A in TMEM, B (64 rows of the K or V tile) K-major
        constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);   // A in TMEM, B (K tile) MN-major
        bool ok = true;
        int e = 0, g = 0;  // ring entry, and tile across all items of the CTA
        auto wait_entry = [&](int entry) {
            ok = mbar_wait_warp(&bar_full[entry % NST], uint32_t(entry / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
        };
        // an operand of the item from its ring entry into tensor memory
        auto copy_operand = [&](const uint8_t* tile, uint32_t col) {
            tc_fence_after_sync();
            const uint64_t desc = kmajor_desc<D>(tile);
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) tmem_copy_128x32b(tmem + col + ks * 8, desc + kmajor_step(ks, Cfg::kBoxBytes));
                umma_commit(&bar_free[e % NST]);
            }
            __syncwarp();
        };
        // D[tmem, 64 columns] = A[tmem] * (rows 64 half .. + 64 of the tile)^T
        auto issue_half = [&](uint32_t d_col, uint32_t a_col, const uint8_t* tile, int half, uint64_t* full, uint64_t* free) {
            const uint64_t desc = kmajor_desc<D>(tile + half * 64 * 128);
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    umma_ts(tmem + d_col + half * 64, tmem + a_col + ks * 8, desc + kmajor_step(ks, Cfg::kBoxBytes), idesc_s, ks > 0);
                umma_commit(full);
                if (free) umma_commit(free);
            }
            __syncwarp();
        };
        if (warp == kMmaSWarp) {
            for (int n = 0, id; ok && (id = get_item(n)) >= 0; ++n) {
                const int n_kv = item_nkv(id);
                // (the products that read the Q before are complete when their scores have been read)
                for (int half = 0; half < 2 && ok && g > 0; ++half)
                    ok = mbar_wait_warp(&bar_s_loaded[half], uint32_t(g - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                if (ok) wait_entry(e);
                if (!ok) break;
                copy_operand(place_a(e), Cfg::kColQ);
                ++e;
                for (int j = 0; j < n_kv && ok; ++j, ++g, ++e) {
                    wait_entry(e);
                    for (int half = 0; half < 2 && ok; ++half) {
                        if (j > 0) ok = mbar_wait_warp(&bar_s_loaded[half], uint32_t(g - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                        if (!ok) break;
                        tc_fence_after_sync();
                        issue_half(Cfg::kColS, Cfg::kColQ, place_a(e), half, &bar_s_full[half], half ? &bar_free[e % NST] : nullptr);
                    }
                }
            }
        } else {
            int n = 0;
            for (int id; ok && (id = get_item(n)) >= 0; ++n) {
                const int n_kv = item_nkv(id);
                wait_entry(e);
                if (!ok) break;
                copy_operand(place_b(e), Cfg::kColDO);  // (dS of the item before has been made of all its dP)
                ++e;
                wait_entry(e);
                if (!ok) break;
                tc_fence_after_sync();
                for (int half = 0; half < 2; ++half) issue_half(Cfg::kColDP, Cfg::kColDO, place_b(e), half, &bar_dp_full[half], nullptr);
                for (int j = 0; j < n_kv && ok; ++j, ++g, ++e) {
                    const bool more = j + 1 < n_kv;
                    const uint64_t k_desc = mnmajor_desc<D>(place_a(e));
                    if (more) wait_entry(e + 1);
                    for (int half = 0; half < 2 && ok; ++half) {
                        ok = mbar_wait_warp(&bar_ds_full[half], uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                        // the accumulator belongs to the previous item's rows until they have been read
                        if (ok && j == 0 && half == 0 && n > 0)
                            ok = mbar_wait_warp(bar_acc_free, uint32_t(n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                        if (!ok) break;
                        tc_fence_after_sync();
                        if (elect_one()) {
                            // dQ += dS K over the half's 64 keys: 4 K steps, two per part
#pragma unroll
                            for (int ks = 0; ks < 4; ++ks)
                                umma_ts(tmem + Cfg::kColAcc, tmem + Cfg::kColDP + half * 64 + (ks >> 1) * 32 + (ks & 1) * 8,
                                        k_desc + uint64_t((half * 4 + ks) * 128), idesc_acc, j > 0 || half > 0 || ks > 0);
                            if (half == 1) umma_commit(&bar_free[e % NST]);
                            if (half == 1 && !more) umma_commit(bar_acc);
                        }
                        __syncwarp();
                        // behind the product that reads dS out of the block
                        if (more) issue_half(Cfg::kColDP, Cfg::kColDO, place_b(e + 1), half, &bar_dp_full[half], nullptr);
                    }
                }
            }
            // nothing may be in flight when TMEM is freed (the compute warps have waited for the other warp's products)
            if (ok && n > 0) mbar_wait_warp(bar_acc, uint32_t(n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
        }
    } else if (warp >= kRowWarp) {
        // ------------------------------------------------------------------ rows: what happens once per item
        const int w4 = warp & 3, row = w4 * 32 + lane;  // query row in the tile == TMEM lane
        bool ok = true;
        int id_prev = get_item(0);
        for (int n = 1, id; ok && id_prev >= 0 && (id = get_item(n)) >= 0; ++n) {
            // preprocess of the next item
            const int q0 = item_qt(id) * 128;
            const size_t bh = size_t(item_b(id)) * p.Hq + item_h(id);
            const float lse2 = q0 + row < p.T ? p.lse[bh * p.T + q0 + row] * 1.4426950408889634f : INFINITY;  // exp2(x - inf) = 0: padding
            // (Every compute warp has passed the barrier and read what the buffer held by the end of that item's rows below.  With one
            // barrier for all items a row warp could be an item ahead of another and arrive for both.)
            float2* vec = sVec + (n & 1) * 128;
#pragma unroll 1
            for (int r = 0; r < 32; r += 8) row_sums<D, 4>(p, q_offset(id), q0, w4 * 32 + r, lane, [&](int r, float d) { vec[r].y = d; });
            __syncwarp();
            vec[row].x = lse2;
            mbar_arrive(&bar_vec[n & 1]);
            const size_t vrow = bh * p.Tpad + q0 + row;
            p.lse2_w[vrow] = lse2;
            p.dvec_w[vrow] = vec[row].y;
            // dQ rows of the item before (times scale) -> BF16 -> global memory
            ok = mbar_wait_warp(bar_acc, uint32_t(n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            if (!ok) break;
            tc_fence_after_sync();
            const int q_prev = item_qt(id_prev) * 128 + w4 * 32;
            uint16_t* out = p.dq + q_offset(id_prev) + size_t(q_prev) * p.q_st;
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                uint32_t v[32], w[16];
                tmem_ld_x32(tmem + (uint32_t(w4 * 32) << 16) + Cfg::kColAcc + c * 32, v);
                tmem_wait_ld();
                if (c + 1 == D / 32) {
                    tc_fence_before_sync();
                    mbar_arrive(bar_acc_free);  // the MMA warp may start the next item's accumulation
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]) * p.scale, __uint_as_float(v[2 * i + 1]) * p.scale);
                store_rows_64b(sOut + w4 * kRowStageBytes, w, lane, out + c * 32, p.q_st, p.T - q_prev);
            }
            id_prev = id;
        }
    } else {
        // ------------------------------------------------------------------ compute
        const int w4 = warp & 3, part = (warp >> 2) & 1, half = warp >> 3;
        const int row = w4 * 32 + lane;  // query row in the tile == TMEM lane
        const uint32_t lane_base = uint32_t(w4 * 32) << 16;
        const int c0 = half * 64 + part * 32;  // first key column of this thread
        const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
        bool ok = true;
        int g = 0, n = 0, id_last = -1;
        for (int id; ok && (id = get_item(n)) >= 0; ++n) {
            const int qt = item_qt(id), n_kv = item_nkv(id), q0 = qt * 128;
            float lse2, dv;
            if (n == 0) {
                // preprocess D = rowsum(O * dO) of the first item: the four warps that share 32 rows take 8 each
                const size_t bh = size_t(item_b(id)) * p.Hq + item_h(id);
                const float lse_raw = q0 + row < p.T ? p.lse[bh * p.T + q0 + row] : INFINITY;
                row_sums<D, 4>(p, q_offset(id), q0, w4 * 32 + (warp >> 2) * 8, lane, [&](int r, float d) { sD[r] = d; });
                lse2 = lse_raw * 1.4426950408889634f;
                named_bar_sync(1, Cfg::kComputeThreads);
                dv = sD[row];
                if (warp < 4 && (!SPLIT || rank == p.split - 1)) {  // (the last share is never empty)
                    const size_t vrow = bh * p.Tpad + q0 + row;
                    p.lse2_w[vrow] = lse2;
                    p.dvec_w[vrow] = dv;
                }
            } else {
                ok = mbar_wait_warp(&bar_vec[n & 1], uint32_t((n - 1) >> 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                if (!ok) break;
                const float2 vec = sVec[(n & 1) * 128 + row];
                lse2 = vec.x, dv = vec.y;
            }
            const uint64_t neg_l2 = pack_f32x2(-lse2, -lse2), neg_d2 = pack_f32x2(-dv, -dv);
            for (int j = 0; j < n_kv; ++j, ++g) {
                ok = mbar_wait_warp(&bar_s_full[half], uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                if (!ok) break;
                tc_fence_after_sync();
                // phase A: P from S (the scores leave tensor memory in one go)
                float pr[32];
                {
                    uint32_t sv[32];
                    tmem_ld_x32(tmem + lane_base + Cfg::kColS + c0, sv);
                    tmem_wait_ld();
                    tc_fence_before_sync();
                    mbar_arrive(&bar_s_loaded[half]);
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float x0, x1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), scale2, neg_l2), x0, x1);
                        pr[i] = ex2_approx(x0);
                        pr[i + 1] = ex2_approx(x1);
                    }
                }
                if (j_first + j == qt) {
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if (c0 + i > row) pr[i] = 0.f;  // key above the diagonal
                }
                ok = mbar_wait_warp(&bar_dp_full[half], uint32_t(g) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                if (!ok) break;
                tc_fence_after_sync();
                // phase B: dS = P (dP - D), written as BF16 over the first 16 of the thread's dP columns
                {
                    uint32_t dp[32], pk[16];
                    const uint32_t t_dp = tmem + lane_base + Cfg::kColDP + c0;
                    tmem_ld_x32(t_dp, dp);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; i += 2) {
                        float y0, y1;
                        unpack_f32x2(mul_f32x2(pack_f32x2(pr[i], pr[i + 1]),
                                               add_f32x2(pack_f32x2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])), neg_d2)), y0, y1);
                        pk[i / 2] = pack_bf16x2(y0, y1);
                    }
                    tmem_st_x16(t_dp, pk);
                }
                tmem_wait_st();
                tc_fence_before_sync();
                mbar_arrive(&bar_ds_full[half]);
            }
            id_last = id;
        }
        if (ok && n > 0) ok = mbar_wait_warp(bar_acc, uint32_t(n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
        if (!SPLIT && ok && n > 0) {
            // dQ rows of the last item through the ring, which nothing reads or loads any more
            tc_fence_after_sync();
            uint32_t v[32], w[16];
            tmem_ld_x32(tmem + lane_base + Cfg::kColAcc + c0, v);
            tmem_wait_ld();
            tc_fence_before_sync();
#pragma unroll
            for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]) * p.scale, __uint_as_float(v[2 * i + 1]) * p.scale);
            const int q0 = item_qt(id_last) * 128 + w4 * 32;
            store_rows_64b(smem + warp * kRowStageBytes, w, lane, p.dq + q_offset(id_last) + size_t(q0) * p.q_st + c0, p.q_st, p.T - q0);
        }
        if constexpr (SPLIT)
            dq_exchange<D>(p, smem, reinterpret_cast<volatile uint32_t*>(sVec), abort_flag, tmem + Cfg::kColAcc, split_id, rank, any, share_begin);
    }

    if (SPLIT && (warp >= kRowWarp || left)) dq_exchange_idle(p, reinterpret_cast<volatile uint32_t*>(sVec), rank);
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kMmaSWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, Cfg::kTmemCols);
    }
    B200ATTN_TRACE_END(1);
}


// ---------------------------------------------------------------------------------------
// dK/dV pass: persistent CTAs, one per SM.  An item is one 128-key tile of one (batch, KV head); its
// units are the (query head of the group, 128-query tile at or below the diagonal) pairs, each a
// 128 x 128 block of scores.  Items are ordered heaviest first (key tile 0 sees every query tile) and
// handed out as described in ptx.cuh.  All pipelines run across item boundaries: the next item's K and V
// tiles (second buffer, D = 64) and its first Q / dO tiles are loaded, and its first S^T and dP^T
// products issued, while the compute warps still drain the accumulators of the previous item.
// What bounds it: D = 128 the tensor pipe (two products with both operands in shared memory, two with one in tensor memory);
// D = 64 a unit's chain, scores -> exponentials -> dP -> dS -> products, of which S^T and dP^T of the following units are off
// the chain because there is one more dP block than units in work and S goes back as soon as it is in registers.  Measured
// against two S buffers (P^T and dS^T over the scores), one dP block, one MMA warp and row vectors read by the compute warps,
// us: B=16 T=1024 16/4 D=64 94.7 -> 84.5, B=8 T=2000 16/4 D=64 171 -> 148, B=4 T=4096 16/4 D=128 496 -> 468.  Two groups of eight
// warps on alternate units (64 columns a thread) were slower: 93 to 117 at the first of these, they spill.
// ---------------------------------------------------------------------------------------
// SPLIT: few, long items (few sequences and key/value heads).  A CTA works on a share of ONE item's units, and the CTAs of a
// cluster add up their accumulators through distributed shared memory in the order of the units, each finishing
// 128 / split of the key rows.
template <int D, bool SPLIT>
__global__ void __launch_bounds__(BwdCfg<D>::kThreads, 1)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO, const BwdParams p) {
    using Cfg = BwdCfg<D>;
    constexpr int NST = Cfg::kStages;
    constexpr int NKV = Cfg::kKvBufs;
    constexpr int NDP = Cfg::kDpBufs;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;                         // [NKV]
    uint8_t* sV = sK + NKV * Cfg::kTileBytes;   // [NKV]
    uint8_t* sQ = sV + NKV * Cfg::kTileBytes;   // [NST]
    uint8_t* sdO = sQ + NST * Cfg::kTileBytes;  // [NST]
    uint8_t* sOut = sdO + NST * Cfg::kTileBytes;  // per compute warp: a piece of its output rows (D = 128)
    float* sLse = reinterpret_cast<float*>(sOut + Cfg::kOutBytes);        // [NST][128]
    float* sDv = sLse + NST * 128;                                        // [NST][128]
    uint8_t* sOps = reinterpret_cast<uint8_t*>(sLse) + Cfg::kVecBytes;    // kVecOps: [NST] L and D operands; ones; zeros
    uint8_t* sOnes = sOps + 2 * NST * Cfg::kOpBytes;
    uint8_t* sZero = sOnes + Cfg::kOpBytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(sOps + Cfg::kOpsBytes);
    uint64_t* bar_kv = bars + 0;        // [2] per K/V buffer: K, V of an item have landed      (phase: item / NKV)
    uint64_t* bar_kv_free = bars + 2;   // [2] per K/V buffer: every MMA reading them is done   (phase: item / NKV)
    uint64_t* bar_s_full = bars + 4;    //                                                       (phase: unit)
    uint64_t* bar_s_loaded = bars + 5;  // S^T is in registers, the buffer is free               (phase: unit)
    uint64_t* bar_dp_full = bars + 6;   // [2] by unit parity                                    (phase: unit / 2)
    uint64_t* bar_pds_full = bars + 8;  // [2] by unit parity: P^T and dS^T written              (phase: unit / 2)
    uint64_t* bar_acc = bars + 10;      // accumulators of an item complete                      (phase: item)
    uint64_t* bar_acc_free = bars + 11; // accumulators read by the epilogue                     (phase: item)
    uint64_t* bar_full = bars + 12;     // [4] per stage: Q, dO and the two row vectors of a unit have landed (phase: unit / NST;
                                        // of the CTA's first unit: they may be used as soon as bar_kv[0] is complete too)
    uint64_t* bar_free = bars + 16;     // [4] per stage                                         (phase: unit / NST)
    uint64_t* bar_vec = bars + 20;      // [4] per stage, kVecOps: the row vectors are there as operands (phase: unit / NST)
    uint64_t* bar_item = bars + 24;     // [kItemRing] item ids handed out by the producer
    volatile int* item_ring = reinterpret_cast<volatile int*>(bars + 24 + kItemRing);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 40);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 41);
    static_assert(NST <= 4, "the barriers are laid out for four stages");

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int kProducerWarp = Cfg::kComputeThreads / 32, kMmaSWarp = kProducerWarp + 1, kMmaWarp = kProducerWarp + 2,
                  kVecWarp = kProducerWarp + 3;
    // item id -> (key tile, KV head, batch); ids are ordered by work: key tile 0 has the most query tiles below it
    const int n_bh = p.B * p.Hkv;
    const int n_items = p.n_tiles * n_bh;
    auto item_kt = [&](int id) { return int(fastdiv(unsigned(id), p.div_bhkv)); };
    auto item_rest = [&](int id) { return id - item_kt(id) * n_bh; };  // b * Hkv + hk
    auto item_b = [&](int id) { return int(fastdiv(unsigned(item_rest(id)), p.div_hkv)); };
    auto item_hk = [&](int id) { return item_rest(id) - item_b(id) * p.Hkv; };
    // units of an item that are this CTA's: [u_first, u_first + item_units); SPLIT: of cluster CTA r, [units r / split, ...)
    const int split_id = SPLIT ? int(fastdiv(blockIdx.x, p.div_split)) : 0, rank = SPLIT ? int(blockIdx.x) - split_id * p.split : 0;
    auto item_all = [&](int id) { return p.group * (p.n_tiles - item_kt(id)); };
    auto share_begin = [&](int r) { return int(fastdiv(unsigned(item_all(split_id) * r), p.div_split)); };
    const int u_first = SPLIT ? share_begin(rank) : 0;
    auto item_units = [&](int id) { return SPLIT ? share_begin(rank + 1) - u_first : item_all(id); };
    auto get_item = [&](int n) { return item_get(bar_item, item_ring, n, abort_flag, p.status); };

    B200ATTN_TRACE_BEGIN(2);
    if (warp == kProducerWarp && lane == 0) {
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmdO);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_kv[i], 1);
            // each of the MMA warps reads K or V; at D = 64 the epilogue stages its rows in the item's tiles
            mbar_init(&bar_kv_free[i], 2 + (Cfg::kOutBytes == 0 && !SPLIT ? Cfg::kComputeThreads : 0));
            mbar_init(&bar_dp_full[i], 1);
            mbar_init(&bar_pds_full[i], Cfg::kComputeThreads);
        }
        mbar_init(bar_s_full, 1);
        mbar_init(bar_s_loaded, Cfg::kComputeThreads);
        mbar_init(bar_acc, 1);
        mbar_init(bar_acc_free, Cfg::kComputeThreads);
        for (int s = 0; s < NST; ++s) {
            mbar_init(&bar_full[s], 1);
            mbar_init(&bar_free[s], 1);
            mbar_init(&bar_vec[s], 32);
        }
        for (int i = 0; i < kItemRing; ++i) mbar_init(&bar_item[i], 1);
        fence_mbar_init();
        *abort_flag = *reinterpret_cast<volatile int*>(p.status);
    }
    if (Cfg::kVecOps && warp == kVecWarp) {  // ones: 1, 1, 1, 0, ... per row; zeros
        for (int r = lane; r < 128; r += 32) {
            reinterpret_cast<uint4*>(sOnes)[r] = make_uint4(0x3f803f80u, 0x3f80u, 0u, 0u);
            reinterpret_cast<uint4*>(sZero)[r] = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_proxy_async_smem();
    }
    if (warp == kMmaSWarp) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
    }
    // No wait for the previous kernel of the stream here: it is the dQ pass, and that lets this grid in only when all its CTAs
    // have passed their own wait, so everything before it is complete.  What it writes itself, the two row vectors, is waited
    // for by the producer in front of their first load; K, V and the first Q and dO load meanwhile.  The status word is looked
    // at twice: here, to leave at once behind an earlier failure, and by the producer behind that wait, because a dQ pass that
    // gave up leaves row vectors of an earlier call.
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    if (*abort_flag != 0) {
        // an earlier kernel failed: fall through to the teardown, but not ahead of the dQ pass (what follows this grid may
        // start when it ends)
        grid_dep_wait();
    } else if (warp == kProducerWarp) {
        // ------------------------------------------------------------------ producer (whole warp, one lane issues)
        reg_dealloc<Cfg::kRegsOther>();
        int u = 0;  // units issued so far by this CTA (ring position)
        bool ok = true;
        int id = SPLIT ? split_id : blockIdx.x;  // the first item needs no fetch
        int id_next = 0;      // lane 0: the id fetched for the next item
        if (SPLIT && item_units(id) == 0) ok = false;
        if (lane == 0) {
            item_publish(bar_item, item_ring, 0, ok ? id : -1);
            id_next = SPLIT ? n_items : sched_fetch(p.sched2, 1, int(blockIdx.x), int(gridDim.x));
        }
        __syncwarp();
        for (int n = 0; ok; ++n) {
            const int kt = item_kt(id), hk = item_hk(id), b = item_b(id), k0 = kt * 128;
            const int n_it = item_units(id), n_i = p.n_tiles - kt, h_skip = SPLIT ? u_first / n_i : 0;
            const int kb = n % NKV;
            if (n >= NKV) ok = mbar_wait_warp(&bar_kv_free[kb], uint32_t(n / NKV - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
            if (!ok) break;
            if (elect_one()) {
                // (all loads of the CTA's first unit complete on this barrier: see there)
                mbar_arrive_expect_tx(&bar_kv[kb], n == 0 ? 4 * Cfg::kTileBytes + 1024 : 2 * Cfg::kTileBytes);
#pragma unroll
                for (int bx = 0; bx < Cfg::kBoxes; ++bx) {
                    tma_load_4d(sK + kb * Cfg::kTileBytes + bx * Cfg::kBoxBytes, &tmK, &bar_kv[kb], bx * 64, k0, hk, b);
                    tma_load_4d(sV + kb * Cfg::kTileBytes + bx * Cfg::kBoxBytes, &tmV, &bar_kv[kb], bx * 64, k0, hk, b);
                }
            }
            __syncwarp();
            // the next item is taken and announced shortly before this item's loads end, but not before the
            // ring has been filled for this item
            const int j_next = max(min(n_it, NST) - 1, n_it - 2);
            int id_new = n_items;
            for (int it = 0, h = hk * p.group + h_skip, i = kt + u_first - h_skip * n_i; it < n_it; ++it, ++u, i = (i + 1 == p.n_tiles ? kt : i + 1), h += (i == kt)) {
                const int s = u % NST;
                if (u >= NST) ok = mbar_wait_warp(&bar_free[s], uint32_t(u / NST - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
                if (!ok) break;
                // The first unit's loads complete on bar_kv[0], which whoever needs them waits for too; bar_full[0] is arrived
                // on once the dQ pass is complete and the status word, read under the loads' latency, is still clear.
                uint64_t* full = u == 0 ? &bar_kv[0] : &bar_full[s];
                int failed = 0;
                if (elect_one()) {
                    if (u > 0) mbar_arrive_expect_tx(full, 2 * Cfg::kTileBytes + 1024);
#pragma unroll
                    for (int bx = 0; bx < Cfg::kBoxes; ++bx) {
                        tma_load_4d(sQ + s * Cfg::kTileBytes + bx * Cfg::kBoxBytes, &tmQ, full, bx * 64, i * 128, h, b);
                        tma_load_4d(sdO + s * Cfg::kTileBytes + bx * Cfg::kBoxBytes, &tmdO, full, bx * 64, i * 128, h, b);
                    }
                    if (u == 0) grid_dep_wait();  // (the same lane issues all loads)
                    const size_t voff = (size_t(b) * p.Hq + h) * p.Tpad + size_t(i) * 128;
                    bulk_load_1d(sLse + s * 128, p.lse2 + voff, 512, full);
                    bulk_load_1d(sDv + s * 128, p.dvec + voff, 512, full);
                    if (u == 0) {
                        failed = *reinterpret_cast<volatile int*>(p.status);
                        if (failed == 0) mbar_arrive(&bar_full[0]);
                    }
                }
                __syncwarp();
                if (u == 0 && __any_sync(0xffffffffu, failed != 0)) {
                    // the other roles stand at bar_full[0]: they are sent home once the loads in flight have landed
                    mbar_wait_warp(&bar_kv[0], 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                    if (failed != 0) *abort_flag = failed;
                    ok = false;
                    break;
                }
                if (it == j_next) {
                    id_new = __shfl_sync(0xffffffffu, id_next, 0);
                    if (lane == 0) {
                        item_publish(bar_item, item_ring, n + 1, id_new < n_items ? id_new : -1);
                        if (id_new < n_items) id_next = sched_fetch(p.sched2, n + 2, int(blockIdx.x), int(gridDim.x));
                    }
                    __syncwarp();
                }
            }
            if (!ok || id_new >= n_items) break;
            id = id_new;
        }
        if (!SPLIT && ok && lane == 0) sched_finish(p.sched2, int(gridDim.x));
        if (p.early) grid_dep_launch();
    } else if (warp == kVecWarp) {
        // ------------------------------------------------------------------ row vectors
        // L and D are the same for a whole column of S^T and dP^T, so reading them costs the compute warps 32 shared-memory
        // loads per unit and warp, in the pipe that the products' operands come through: 10 % of the kernel at D = 64.  There
        // they enter the products as one more K step instead, ones[128 keys x 16] times the vector, split into three BF16 terms
        // (24 bits), so that S^T arrives as s - L / scale and dP^T as dP - D.  This warp turns a unit's two vectors into such
        // operands.  (At D = 128 the tensor pipe sets the pace: two more K steps per unit cost 10 %.)
        reg_dealloc<Cfg::kRegsOther>();
        if constexpr (Cfg::kVecOps) {
            const float to_scores = -1.f / p.scale_log2;
            auto split = [](float v) {
                const float hi = __bfloat162float(__float2bfloat16_rn(v)), r = fabsf(hi) == INFINITY ? 0.f : v - hi;  // (NaN stays NaN)
                const float mid = __bfloat162float(__float2bfloat16_rn(r));
                return make_uint4(pack_bf16x2(hi, mid), pack_bf16x2(r - mid, 0.f), 0u, 0u);
            };
            int u = 0;
            bool ok = true;
            for (int n = 0, id; ok && (id = get_item(n)) >= 0; ++n) {
                for (int it = item_units(id); it > 0; --it, ++u) {
                    const int s = u % NST;
                    ok = mbar_wait_warp(u == 0 ? &bar_kv[0] : &bar_full[s], uint32_t(u / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                    if (!ok) break;
                    uint4* op_l = reinterpret_cast<uint4*>(sOps + 2 * s * Cfg::kOpBytes);
                    uint4* op_d = op_l + 128;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int r = i * 32 + lane;
                        op_l[r] = split(sLse[s * 128 + r] * to_scores);  // padding rows: L = inf, so S^T = -inf and P = 0
                        op_d[r] = split(-sDv[s * 128 + r]);
                    }
                    fence_proxy_async_smem();  // ordinary accesses before the products' reads and the next loads' writes
                    if (u == 0) ok = mbar_wait_warp(&bar_full[0], 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);  // the status word
                    if (!ok) break;
                    mbar_arrive(&bar_vec[s]);
                }
            }
        }
    } else if (warp == kMmaSWarp || warp == kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuers (whole warps, one lane issues)
        // Two warps share the products: the first issues S^T, the second dV, dK and, into the block whose operands these have
        // read, dP^T of the unit kDpBufs ahead.  (Between two products a warp spends 100 clocks on every wait and every commit.)
        reg_dealloc<Cfg::kRegsOther>();
        constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);
        constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);
        // This CTA's units are numbered u = 0, 1, ... across all its items: ring stage u % NST, dP block u % NDP.
        struct Cursor {
            int n, it, n_it, u;  // items before this one on this CTA, unit in item, units of item (0: list ended), unit number
        };
        bool ok = true;
        auto cursor_start = [&]() {
            const int id = get_item(0);
            return Cursor{0, 0, id >= 0 ? item_units(id) : 0, 0};
        };
        auto cursor_next = [&](Cursor& c) {
            ++c.u;
            if (++c.it == c.n_it) {
                ++c.n;
                c.it = 0;
                const int id = get_item(c.n);
                c.n_it = id >= 0 ? item_units(id) : 0;
            }
        };
        // Q, dO and the row vectors of the unit (and K and V of its item) have landed
        auto wait_loaded = [&](const Cursor& c) {
            const int s = c.u % NST, kb = c.n % NKV;
            if (c.it == 0) ok = mbar_wait_warp(&bar_kv[kb], uint32_t(c.n / NKV) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
            if (ok)
                ok = mbar_wait_warp(Cfg::kVecOps ? &bar_vec[s] : &bar_full[s], uint32_t(c.u / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
        };
        // One thread: D[tmem] = A B^T over the head dimension, plus the row vector `which` of stage s (0 L, 1 D; kVecOps).  After
        // the item's last unit this warp's products read its K or V no more.
        const uint64_t ones_desc = make_sdesc_plain(smem_u32(sOnes), uint32_t(sZero - sOnes), 128);
        auto issue_block = [&](uint32_t d_tmem, const uint8_t* key_tile, const uint8_t* query_tile, const Cursor& c, int which, uint64_t* full) {
            tc_fence_after_sync();
            if (elect_one()) {
                issue_ss_over_headdim<D>(d_tmem, kmajor_desc<D>(key_tile), kmajor_desc<D>(query_tile), idesc_s);
                if constexpr (Cfg::kVecOps) {
                    const uint8_t* op = sOps + (2 * (c.u % NST) + which) * Cfg::kOpBytes;
                    umma_ss(d_tmem, ones_desc, make_sdesc_plain(smem_u32(op), uint32_t(sZero - op), 128), idesc_s, 1);  // (second half of the K step: zeros)
                }
                umma_commit(full);
                if (c.it + 1 == c.n_it) umma_commit(&bar_kv_free[c.n % NKV]);
            }
            __syncwarp();
        };
        if (warp == kMmaSWarp) {
            for (Cursor c = cursor_start(); ok && c.n_it > 0; cursor_next(c)) {
                wait_loaded(c);
                // the buffer holds S^T of the unit before until the compute warps have read it into registers
                if (ok && c.u > 0) ok = mbar_wait_warp(bar_s_loaded, uint32_t(c.u - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                if (!ok) break;
                issue_block(tmem + Cfg::kColS, sK + (c.n % NKV) * Cfg::kTileBytes, sQ + (c.u % NST) * Cfg::kTileBytes, c, 0, bar_s_full);
            }
        } else {
            Cursor ca = cursor_start(), cd = ca;
            auto next_dp = [&]() {
                wait_loaded(cd);
                if (!ok) return;
                issue_block(tmem + Cfg::col_dp(cd.u % NDP), sV + (cd.n % NKV) * Cfg::kTileBytes, sdO + (cd.u % NST) * Cfg::kTileBytes, cd, 1,
                            &bar_dp_full[cd.u & 1]);
                cursor_next(cd);
            };
            for (int i = 0; i < NDP && ok && cd.n_it > 0; ++i) next_dp();
            int n_done = 0;  // items whose accumulators have been completed
            while (ok && ca.n_it > 0) {
                const int s = ca.u % NST;
                ok = mbar_wait_warp(&bar_pds_full[ca.u & 1], uint32_t(ca.u >> 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                // the accumulators belong to the previous item's epilogue until it has read them
                if (ok && ca.it == 0 && ca.n > 0)
                    ok = mbar_wait_warp(bar_acc_free, uint32_t(ca.n - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                if (!ok) break;
                B200ATTN_STAMP(lane == 0, 16 + 8 * ca.u + 4);
                tc_fence_after_sync();
                if (elect_one()) {
                    // dV += P^T dO ; dK += dS^T Q   (P^T and dS^T sit side by side over the unit's dP block)
                    const uint32_t a_pds = tmem + Cfg::col_dp(ca.u % NDP);
                    issue_ts_over_rows<D>(tmem + Cfg::kColAcc0, a_pds, mnmajor_desc<D>(sdO + s * Cfg::kTileBytes), idesc_acc, ca.it > 0);
                    issue_ts_over_rows<D>(tmem + Cfg::kColAcc1, a_pds + Cfg::kPartCols / 2, mnmajor_desc<D>(sQ + s * Cfg::kTileBytes),
                                          idesc_acc, ca.it > 0);
                    umma_commit(&bar_free[s]);
                    if (ca.it + 1 == ca.n_it) umma_commit(bar_acc);
                }
                __syncwarp();
                B200ATTN_STAMP(lane == 0, 16 + 8 * ca.u + 5);
                if (ca.it + 1 == ca.n_it) ++n_done;
                if (cd.n_it > 0) next_dp();  // overwrites this unit's P^T and dS^T: behind the two products just issued
                cursor_next(ca);
            }
            // nothing may be in flight when TMEM is freed: the last commit covers every product issued here, and the other warp's
            // were waited for by the compute warps
            if (ok && n_done > 0) mbar_wait_warp(bar_acc, uint32_t(n_done - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
        }
    } else {
        // ------------------------------------------------------------------ compute
        reg_alloc<Cfg::kRegsCompute>();
        const int w4 = warp & 3, part = warp >> 2;
        const int row = w4 * 32 + lane;  // key row in the tile == TMEM lane
        const uint32_t lane_base = uint32_t(w4 * 32) << 16;
        constexpr int NC = Cfg::kCols;
        const int c0 = part * NC;  // first query column of this thread
        bool ok = true;
        // Epilogue of an item.  It is deferred until the first unit of the next item has been handed to the MMA
        // warp, so that the wait for the item's last products overlaps that unit's arithmetic.  Parts 0, 1 write dV, parts 2, 3
        // dK (times scale); each takes D / 2 columns of its key row, which are contiguous in global memory.
        auto epilogue = [&](int n_item, int id_item) -> bool {
            B200ATTN_STAMP(tid == 0, 460 + 4 * n_item + 0);
            ok = mbar_wait_warp(bar_acc, uint32_t(n_item) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            if (!ok) return false;
            B200ATTN_STAMP(tid == 0, 460 + 4 * n_item + 1);
            tc_fence_after_sync();
            // (the values below are derived from copies the compiler cannot see through, so that it does not
            // compute them ahead of the unit loop and keep them in registers there)
            int part_e = part, id_e = id_item;
            asm volatile("" : "+r"(part_e), "+r"(id_e));
            constexpr int kCols = D / 2;
            const bool is_dk = part_e >= 2;
            const uint32_t acc = is_dk ? Cfg::kColAcc1 : Cfg::kColAcc0;
            const float mul = is_dk ? p.scale : 1.f;
            const int col0 = (part_e & 1) * kCols;
            const int k0 = item_kt(id_e) * 128;
            uint8_t* stage = Cfg::kOutBytes > 0 ? sOut + warp * kRowStageBytes
                                                : (is_dk ? sV : sK) + (n_item % NKV) * Cfg::kTileBytes + (warp & 7) * kRowStageBytes;
            uint16_t* out = (is_dk ? p.dk : p.dv) + size_t(item_b(id_e)) * p.k_sb + size_t(item_hk(id_e)) * p.k_sh +
                            size_t(k0 + w4 * 32) * p.k_st + col0;
#pragma unroll
            for (int c = 0; c < kCols / 32; ++c) {
                uint32_t v[32], w[16];
                tmem_ld_x32(tmem + lane_base + acc + col0 + c * 32, v);
                tmem_wait_ld();
                if (c + 1 == kCols / 32) {
                    tc_fence_before_sync();
                    mbar_arrive(bar_acc_free);  // the MMA warp may start the next item's accumulation
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]) * mul, __uint_as_float(v[2 * i + 1]) * mul);
                store_rows_64b(stage, w, lane, out + c * 32, p.k_st, p.T - (k0 + w4 * 32));
            }
            if constexpr (Cfg::kOutBytes == 0) {
                fence_proxy_async_smem();  // ordinary accesses before the next load (TMA) into the tiles
                mbar_arrive(&bar_kv_free[n_item % NKV]);
            }
            B200ATTN_STAMP(tid == 0, 460 + 4 * n_item + 2);
            return true;
        };
        const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
        bool pending = false;
        int pend_id = 0;
        int u = 0, n = 0;
        for (int id; ok && (id = get_item(n)) >= 0; ++n) {
            const int n_i = p.n_tiles - item_kt(id);
            // units of the item: for each query head of the group, the query tiles from the diagonal down
            for (int it = item_units(id), i_in = SPLIT ? u_first % n_i : 0; it > 0; --it, ++u, i_in = (i_in + 1 == n_i ? 0 : i_in + 1)) {
                const int s = u % NST;
                const bool diag = i_in == 0;
                ok = mbar_wait_warp(bar_s_full, uint32_t(u) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                if (!ok) break;
                B200ATTN_STAMP(tid == 0, 16 + 8 * u + 0);
                tc_fence_after_sync();
                const float4* lse4 = reinterpret_cast<const float4*>(sLse + s * 128 + c0);
                const float4* dv4 = reinterpret_cast<const float4*>(sDv + s * 128 + c0);
                const uint32_t t_dp = tmem + lane_base + Cfg::col_dp(u % NDP) + c0;
                // phase A: the scores leave tensor memory in one go and the buffer goes back to the MMA warp at once; P^T stays
                // in registers until phase B
                float pr[NC];
                {
                    uint32_t sv[NC];
                    tmem_ld_x32(tmem + lane_base + Cfg::kColS + c0, sv);
                    tmem_wait_ld();
                    tc_fence_before_sync();
                    mbar_arrive(bar_s_loaded);
#pragma unroll
                    for (int i = 0; i < NC; i += 2) {
                        uint64_t x = pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1]));
                        float x0, x1;
                        if constexpr (Cfg::kVecOps) {
                            unpack_f32x2(mul_f32x2(x, scale2), x0, x1);
                        } else {
                            const float4 l4 = lse4[i / 4];
                            unpack_f32x2(fma_f32x2(x, scale2, i % 4 ? pack_f32x2(-l4.z, -l4.w) : pack_f32x2(-l4.x, -l4.y)), x0, x1);
                        }
                        pr[i] = ex2_approx(x0);
                        pr[i + 1] = ex2_approx(x1);
                    }
                }
                if (diag) {
#pragma unroll
                    for (int i = 0; i < NC; ++i)
                        if (c0 + i < row) pr[i] = 0.f;  // query above the key: masked
                }
                B200ATTN_STAMP(tid == 0, 16 + 8 * u + 1);
                ok = mbar_wait_warp(&bar_dp_full[u & 1], uint32_t(u >> 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
                if (!ok) break;
                B200ATTN_STAMP(tid == 0, 16 + 8 * u + 2);
                tc_fence_after_sync();
                // phase B: 16 columns of dP^T at a time into registers, then P^T and dS^T = P^T (dP^T - D) as BF16 side by side
                // over those columns (P^T in the first 8, dS^T in the second 8)
#pragma unroll
                for (int h = 0; h < NC / 16; ++h) {
                    uint32_t dp[16], pk[8];
                    tmem_ld_x16(t_dp + h * 16, dp);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 16; i += 2) {
                        uint64_t d = pack_f32x2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1]));
                        if constexpr (!Cfg::kVecOps) {
                            const float4 d4 = dv4[h * 4 + i / 4];
                            d = add_f32x2(d, i % 4 ? pack_f32x2(-d4.z, -d4.w) : pack_f32x2(-d4.x, -d4.y));
                        }
                        float y0, y1;
                        unpack_f32x2(mul_f32x2(pack_f32x2(pr[h * 16 + i], pr[h * 16 + i + 1]), d), y0, y1);
                        pk[i / 2] = pack_bf16x2(y0, y1);
                    }
                    tmem_st_x8(t_dp + h * 16 + 8, pk);
#pragma unroll
                    for (int i = 0; i < 8; ++i) pk[i] = pack_bf16x2(pr[h * 16 + 2 * i], pr[h * 16 + 2 * i + 1]);
                    tmem_st_x8(t_dp + h * 16, pk);
                }
                tmem_wait_st();
                tc_fence_before_sync();
                // the unit's row vectors were read from shared memory with ordinary loads; the stage goes back to TMA (async
                // proxy) through the products this arrival lets go
                if constexpr (!Cfg::kVecOps) fence_proxy_async_smem();
                mbar_arrive(&bar_pds_full[u & 1]);
                B200ATTN_STAMP(tid == 0, 16 + 8 * u + 3);
                if (pending) {  // first unit of this item: now the previous item's epilogue
                    pending = false;
                    if (!epilogue(n - 1, pend_id)) break;
                }
            }
            if (!ok) break;
            pending = true;
            pend_id = id;
        }
        if constexpr (SPLIT) {
            if (ok && pending) mbar_wait_warp(bar_acc, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
        } else if (ok && pending) {
            epilogue(n - 1, pend_id);
        }
    }

    if constexpr (SPLIT) {
        // Every role comes here, also after a wait that gave up and when the status word was set before the launch.  Key row r
        // is finished by CTA r / rows of the cluster; the tiles in shared memory make room for the arrivals, so all CTAs must be
        // through with theirs first.  Nobody writes an item of which a CTA has failed.
        const int rows = 128 / p.split;
        volatile uint32_t* fail = reinterpret_cast<volatile uint32_t*>(sLse);  // [CTA of the cluster]
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        const bool failed = *abort_flag != 0;  // (final: every warp of the CTA has passed the barrier)
        if (tid < p.split) cluster_store_1(const_cast<uint32_t*>(fail) + rank, tid, failed);
        __syncwarp();
        if (tid < Cfg::kComputeThreads && !failed && item_units(split_id) > 0) {
            tc_fence_after_sync();
            const int row = (warp & 3) * 32 + lane, part = warp >> 2, to = (row * p.split) >> 7, r = row - to * rows;
            // [source CTA][row][dV: D, dK: D] FP32, 16-byte pieces swizzled by the row: the rows of a warp would share a bank
            uint8_t* own = smem + (rank * rows + r) * D * 8;
            const uint32_t dst = cluster_addr(own, to);
            const uint32_t t_acc = tmem + (uint32_t((warp & 3) * 32) << 16) + (part < 2 ? Cfg::kColAcc0 : Cfg::kColAcc1) + (part & 1) * (D / 2);
#pragma unroll
            for (int c = 0; c < D / 64; ++c) {
                uint32_t v[32];
                tmem_ld_x32(t_acc + c * 32, v);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int at = ((part * (D / 8) + c * 8 + i) ^ (r & 7)) << 4;
                    if (to == rank)
                        *reinterpret_cast<uint4*>(own + at) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                    else
                        cluster_store_4(dst + at, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
                }
            }
            tc_fence_before_sync();
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        bool good = true;
        for (int k = 0; k < p.split; ++k) good = good && fail[k] == 0;
        if (tid < Cfg::kComputeThreads && good) {
            const int k0 = item_kt(split_id) * 128 + rank * rows, b = item_b(split_id), hk = item_hk(split_id);
            for (int i = tid; i < rows * (D / 4); i += Cfg::kComputeThreads) {  // eight columns each: dV, then dK
                const int r = i / (D / 4), c8 = i % (D / 4);
                if (k0 + r >= p.T) break;
                float acc[8] = {};
#pragma unroll 2
                for (int k = 0; k < p.split; ++k) {
                    if (share_begin(k + 1) == share_begin(k)) continue;  // nothing was sent
                    const uint8_t* src = smem + (k * rows + r) * D * 8;
                    const float4 v0 = *reinterpret_cast<const float4*>(src + (((c8 * 2) ^ (r & 7)) << 4));
                    const float4 v1 = *reinterpret_cast<const float4*>(src + (((c8 * 2 + 1) ^ (r & 7)) << 4));
                    acc[0] += v0.x, acc[1] += v0.y, acc[2] += v0.z, acc[3] += v0.w;
                    acc[4] += v1.x, acc[5] += v1.y, acc[6] += v1.z, acc[7] += v1.w;
                }
                const bool is_dk = c8 >= D / 8;
                const float mul = is_dk ? p.scale : 1.f;
                uint16_t* out = (is_dk ? p.dk : p.dv) + size_t(b) * p.k_sb + size_t(hk) * p.k_sh + size_t(k0 + r) * p.k_st + (c8 % (D / 8)) * 8;
                *reinterpret_cast<uint4*>(out) = make_uint4(pack_bf16x2(acc[0] * mul, acc[1] * mul), pack_bf16x2(acc[2] * mul, acc[3] * mul),
                                                            pack_bf16x2(acc[4] * mul, acc[5] * mul), pack_bf16x2(acc[6] * mul, acc[7] * mul));
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kMmaSWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, Cfg::kTmemCols);
    }
    B200ATTN_TRACE_END(2);
}

}  // namespace b200attn
