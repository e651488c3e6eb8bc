// Causal grouped-query attention backward of sequences that fit one tile (T <= 128) for sm_100a, in one launch.
//
// The two passes of attn_bwd.cuh exist because a query tile's dQ and a key tile's dK, dV are sums over different tiles.  With one
// tile they are not: a CTA takes one query head, or one (batch, key/value head) and goes through the query heads of its group, and
// computes S, P, dP and dS of a head once for all of
//      dQ = scale dS K        dV += P^T dO        dK += scale dS^T Q
// (the steps of the reference's flash_attn_backward, llm/src/model/flash_attn.cu:428-504, math :137-146).  D = rowsum(O dO) and
// L log2(e) are computed by the CTA, too.  Nothing is added to global memory, so results are bit-reproducible.
// What bounds it: latency, a chain of loads, two products, the exponentials, three products and the way out of dQ per head (2.8 us
// at D = 64 and 5.5 at D = 128 behind 3 us of start), and with the heads of a group in a cluster the exchange of dV and dK at 13 bytes
// a clock of distributed shared memory.  Measured on B200 against the two passes, us: B=2 T=128 6/2 D=64 12.0 -> 9.4, D=128 15.9 ->
// 14.0, B=1 T=100 4/4 D=64 10.0 -> 5.2, B=16 6/2 13.0 -> 10.2, B=64 T=100 6/2 17.7 -> 13.3 (by group), D=128 T=128 32.2 -> 25.9; more
// beside the rule that chooses.  L and D of the next head by two warps of their own were no faster (2.8 us a head).
//
// Roles (576 threads): warps 0-15 compute (thread owns TMEM lane (warp % 4) * 32 + lane, a key row of S^T and dP^T and a query
// row of dQ, and of the 128 query columns the 32 of its part warp / 4), warp 16 TMA producer, warp 17 TMEM allocation + MMA issue.
// TMEM (512 columns): S [0,128), dP [128,256) with P^T and dS^T over it as in the dK/dV pass, dV and dK from 256, dQ [384,448) at
// D = 64 and over S at D = 128.  dS^T also goes to shared memory: in dQ the query index is the M dimension.
#pragma once

#include "attn_bwd.cuh"

namespace b200attn {

template <int D>
struct BwdTileCfg {
    static constexpr int kStages = 2;  // heads whose Q and dO are in shared memory or on the way
    static constexpr int kTileBytes = 128 * D * 2;
    static constexpr int kBoxBytes = 128 * 64 * 2;
    static constexpr int kBoxes = D / 64;
    static constexpr int kDsBytes = 2 * kBoxBytes;       // dS^T: two [128 keys][64 queries] boxes
    static constexpr int kVecBytes = 2 * 2 * 128 * 4;    // L log2(e) and D of the rows of two heads
    static constexpr int kMaxCluster = 8;
    static constexpr int kSmemBytes = (2 + 2 * kStages) * kTileBytes + kDsBytes + kVecBytes + 256;
    static_assert(kSmemBytes <= 232448, "shared memory of an SM");
    static constexpr int kComputeThreads = 512, kThreads = kComputeThreads + 64;
    static constexpr int kProducerWarp = 16, kMmaWarp = 17;
    static constexpr int kTmemCols = 512;
    static constexpr int kColS = 0, kColDP = 128, kColDV = 256, kColDK = 256 + D, kColDQ = D == 64 ? 384 : kColS;
};

// ONE: a CTA takes one query head, and the CTAs of a group are a cluster that adds up dV and dK through distributed shared memory in
// the order of the heads, each finishing its share of the key rows.
template <int D, bool ONE>
__global__ void __launch_bounds__(BwdTileCfg<D>::kThreads, 1)
attn_bwd_tile_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                     const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmdO, const BwdParams p) {
    using Cfg = BwdTileCfg<D>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sK = smem;
    uint8_t* sV = sK + Cfg::kTileBytes;
    constexpr int NST = Cfg::kStages;
    uint8_t* sQ = sV + Cfg::kTileBytes;         // [NST]
    uint8_t* sdO = sQ + NST * Cfg::kTileBytes;  // [NST]
    uint8_t* sdS = sdO + NST * Cfg::kTileBytes;
    float* sLse = reinterpret_cast<float*>(sdS + Cfg::kDsBytes);  // [2][128]
    float* sDv = sLse + 2 * 128;                                  // [2][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sDv + 2 * 128);
    uint64_t* bar_kv = bars + 0;        // K and V have landed
    uint64_t* bar_full = bars + 1;      // [NST] Q and dO of a head have landed                  (phase: head / NST)
    uint64_t* bar_free = bars + 5;      // [NST] every product reading them is done              (phase: head / NST)
    uint64_t* bar_s_full = bars + 9;    //                                                       (phase: head)
    uint64_t* bar_s_loaded = bars + 10; // S^T is in registers                                   (phase: head)
    uint64_t* bar_dp_full = bars + 11;  //                                                       (phase: head)
    uint64_t* bar_pds_full = bars + 12; // P^T and dS^T are written                              (phase: head)
    uint64_t* bar_dq_full = bars + 13;  //                                                       (phase: head)
    uint64_t* bar_dq_free = bars + 14;  // dQ has been read                                      (phase: head)
    uint64_t* bar_acc = bars + 15;      // dV and dK are complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 17);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = int(fastdiv(blockIdx.x, ONE ? p.div_hq : p.div_hkv)), rest = int(blockIdx.x) - b * (ONE ? p.Hq : p.Hkv);
    const int hk = ONE ? int(fastdiv(unsigned(rest), p.div_group)) : rest;
    const int h0 = ONE ? rest : hk * p.group, n_heads = ONE ? 1 : p.group;  // this CTA's query heads
    const int rank = h0 - hk * p.group;                                     // ONE: in the cluster

    auto load_tile = [&](uint8_t* tile, const CUtensorMap* map, int h, uint64_t* full) {  // one thread
#pragma unroll
        for (int bx = 0; bx < Cfg::kBoxes; ++bx) tma_load_4d(tile + bx * Cfg::kBoxBytes, map, full, bx * 64, 0, h, b);
    };
    auto load_head = [&](int u) {  // one thread
        const int s = u % NST;
        mbar_arrive_expect_tx(&bar_full[s], 2 * Cfg::kTileBytes);
        load_tile(sQ + s * Cfg::kTileBytes, &tmQ, h0 + u, &bar_full[s]);
        load_tile(sdO + s * Cfg::kTileBytes, &tmdO, h0 + u, &bar_full[s]);
    };
    if (warp == Cfg::kProducerWarp && lane == 0) {
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmdO);
        mbar_init(bar_kv, 1);
        for (int i = 0; i < NST; ++i) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_free[i], 1);
        }
        mbar_init(bar_s_full, 1);
        mbar_init(bar_s_loaded, Cfg::kComputeThreads);
        mbar_init(bar_dp_full, 1);
        mbar_init(bar_pds_full, Cfg::kComputeThreads);
        mbar_init(bar_dq_full, 1);
        mbar_init(bar_dq_free, Cfg::kComputeThreads);
        mbar_init(bar_acc, 1);
        fence_mbar_init();
        *abort_flag = 0;
    }
    if (warp == Cfg::kProducerWarp) {
        __syncwarp();
        grid_dep_wait();  // first global access of this CTA comes next
        if (elect_one()) {  // the first loads: the status word, the barrier and the roles' start pass under their latency
            mbar_arrive_expect_tx(bar_kv, 2 * Cfg::kTileBytes);
            load_tile(sK, &tmK, hk, bar_kv);
            load_head(0);
            load_tile(sV, &tmV, hk, bar_kv);
            const int failed = *reinterpret_cast<volatile int*>(p.status);
            if (failed != 0) {  // behind an earlier failure the CTA leaves, but not before its loads have landed
                mbar_wait(bar_kv, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
                mbar_wait(&bar_full[0], 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
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
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = *tmem_slot;

    if (*abort_flag != 0) {
        // an earlier kernel failed: fall through to the teardown
    } else if (warp == Cfg::kProducerWarp) {
        // ------------------------------------------------------------------ producer (whole warp, one lane issues)
        for (int u = 1; u < n_heads; ++u) {
            if (u >= NST && !mbar_wait_warp(&bar_free[u % NST], uint32_t(u / NST - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE)) break;
            if (elect_one()) load_head(u);
            // (O comes into L2, where the compute warps will look for it)
            for (int i = lane; i < p.T * (D / 64); i += 32)
                prefetch_l2(p.o + size_t(b) * p.q_sb + size_t(h0 + u) * p.q_sh + size_t(i / (D / 64)) * p.q_st + (i % (D / 64)) * 64);
            __syncwarp();
        }
        if (p.early) grid_dep_launch();
    } else if (warp == Cfg::kMmaWarp) {
        // ------------------------------------------------------------------ MMA issuer (whole warp, one lane issues)
        constexpr uint32_t idesc_s = make_idesc_bf16(128, 128, 0, 0);   // S^T, dP^T: K-major operands
        constexpr uint32_t idesc_acc = make_idesc_bf16(128, D, 0, 1);   // dV, dK: A in TMEM, B MN-major
        constexpr uint32_t idesc_dq = make_idesc_bf16(128, D, 1, 1);    // dQ: dS^T (M = query) and K both MN-major
        const uint64_t ds_desc = make_sdesc_sw128(smem_u32(sdS), Cfg::kBoxBytes, 1024);
        const uint64_t k_desc = mnmajor_desc<D>(sK);
        auto issue_block = [&](uint32_t col, const uint8_t* key_tile, const uint8_t* query_tile, uint64_t* full) {
            tc_fence_after_sync();
            if (elect_one()) {
                issue_ss_over_headdim<D>(tmem + col, kmajor_desc<D>(key_tile), kmajor_desc<D>(query_tile), idesc_s);
                umma_commit(full);
            }
            __syncwarp();
        };
        bool ok = mbar_wait_warp(bar_kv, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
        if (ok) ok = mbar_wait_warp(&bar_full[0], 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
        if (ok) {
            issue_block(Cfg::kColS, sK, sQ, bar_s_full);
            issue_block(Cfg::kColDP, sV, sdO, bar_dp_full);
        }
        for (int u = 0; u < n_heads && ok; ++u) {
            const int s = u % NST, s1 = (u + 1) % NST;
            const bool more = u + 1 < n_heads;
            const uint32_t par = uint32_t(u) & 1;
            auto wait_next = [&]() { ok = mbar_wait_warp(&bar_full[s1], uint32_t((u + 1) / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD); };
            if (D == 64 && more) {  // the next head's S^T under this head's exponentials
                wait_next();
                if (ok) ok = mbar_wait_warp(bar_s_loaded, par, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
                if (ok) issue_block(Cfg::kColS, sK, sQ + s1 * Cfg::kTileBytes, bar_s_full);
            }
            if (ok) ok = mbar_wait_warp(bar_pds_full, par, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX);
            if (ok && D == 64 && u > 0) ok = mbar_wait_warp(bar_dq_free, uint32_t(u - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
            if (!ok) break;
            tc_fence_after_sync();
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)  // dQ = dS K, 16 keys a step
                    umma_ss(tmem + Cfg::kColDQ, ds_desc + uint64_t(ks * 128), k_desc + uint64_t(ks * 128), idesc_dq, ks > 0);
                umma_commit(bar_dq_full);
                issue_ts_over_rows<D>(tmem + Cfg::kColDV, tmem + Cfg::kColDP, mnmajor_desc<D>(sdO + s * Cfg::kTileBytes), idesc_acc, u > 0);
                issue_ts_over_rows<D>(tmem + Cfg::kColDK, tmem + Cfg::kColDP + BwdCfg<D>::kPartCols / 2, mnmajor_desc<D>(sQ + s * Cfg::kTileBytes),
                                      idesc_acc, u > 0);
                umma_commit(more ? &bar_free[s] : bar_acc);
            }
            __syncwarp();
            if (!more) break;
            if (D == 128) wait_next();
            if (!ok) break;
            issue_block(Cfg::kColDP, sV, sdO + s1 * Cfg::kTileBytes, bar_dp_full);  // behind the products that read P^T and dS^T there
            if (D == 128) {  // dQ lies over S
                ok = mbar_wait_warp(bar_dq_free, par, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
                if (ok) issue_block(Cfg::kColS, sK, sQ + s1 * Cfg::kTileBytes, bar_s_full);
            }
        }
        // nothing may be in flight when TMEM is freed: the last commit covers every product
        if (ok) mbar_wait_warp(bar_acc, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
    } else {
        // ------------------------------------------------------------------ compute
        const int w4 = warp & 3, part = warp >> 2;
        const int row = w4 * 32 + lane;
        const uint32_t lane_base = uint32_t(w4 * 32) << 16;
        const int c0 = part * 32;  // first query column of this thread
        const uint64_t scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
        const uint32_t t_s = tmem + lane_base + Cfg::kColS + c0, t_dp = tmem + lane_base + Cfg::kColDP + c0;
        uint8_t* ds_row = sdS + (part >> 1) * Cfg::kBoxBytes + row * 128;  // this key's queries, 16-byte pieces swizzled by the row
        bool ok = true;
        // L log2(e) (exp2(x - inf) = 0: padding query rows contribute nothing) and D = rowsum(O dO), eight rows a warp
        RowSums<D, 8 * D / 256> rs;
        float lse_raw;
        auto load_rows = [&](int h) {
            lse_raw = tid < 128 && tid < p.T ? p.lse[(size_t(b) * p.Hq + h) * p.T + tid] : INFINITY;
            rs.load(p, size_t(b) * p.q_sb + size_t(h) * p.q_sh, 0, warp * 8, lane);
        };
        // dQ rows of head u (times scale), D / 4 columns each
        auto write_dq = [&](int u) {
            ok = mbar_wait_warp(bar_dq_full, uint32_t(u) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            if (!ok) return;
            tc_fence_after_sync();
            constexpr int kCols = D / 4;
            uint32_t v[kCols];
            if constexpr (kCols == 16) tmem_ld_x16(tmem + lane_base + Cfg::kColDQ + part * kCols, v);
            else tmem_ld_x32(tmem + lane_base + Cfg::kColDQ + part * kCols, v);
            tmem_wait_ld();
            tc_fence_before_sync();
            mbar_arrive(bar_dq_free);
            if (row < p.T) {
                uint16_t* out = p.dq + size_t(b) * p.q_sb + size_t(h0 + u) * p.q_sh + size_t(row) * p.q_st + part * kCols;
#pragma unroll
                for (int g = 0; g < kCols / 8; ++g) {
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        w[e] = pack_bf16x2(__uint_as_float(v[g * 8 + 2 * e]) * p.scale, __uint_as_float(v[g * 8 + 2 * e + 1]) * p.scale);
                    *reinterpret_cast<uint4*>(out + g * 8) = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        };
        load_rows(h0);
        for (int u = 0; u < n_heads; ++u) {
            const uint32_t par = uint32_t(u) & 1;
            float* lse = sLse + (u & 1) * 128;
            float* dv = sDv + (u & 1) * 128;
            if (tid < 128) lse[tid] = lse_raw * 1.4426950408889634f;
            rs.sum(warp * 8, lane, [&](int r, float d) { dv[r] = d; });
            named_bar_sync(1, Cfg::kComputeThreads);
            ok = mbar_wait_warp(bar_s_full, par, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            if (!ok) break;
            tc_fence_after_sync();
            float pr[32];
            {
                uint32_t sv[32];
                tmem_ld_x32(t_s, sv);
                tmem_wait_ld();
                tc_fence_before_sync();
                mbar_arrive(bar_s_loaded);
                const float4* lse4 = reinterpret_cast<const float4*>(lse + c0);
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    const float4 l4 = lse4[i / 4];
                    float x0, x1;
                    unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sv[i]), __uint_as_float(sv[i + 1])), scale2,
                                           i % 4 ? pack_f32x2(-l4.z, -l4.w) : pack_f32x2(-l4.x, -l4.y)), x0, x1);
                    pr[i] = ex2_approx(x0);
                    pr[i + 1] = ex2_approx(x1);
                }
            }
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (c0 + i < row) pr[i] = 0.f;  // query above the key: masked
            ok = mbar_wait_warp(bar_dp_full, par, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
            if (!ok) break;
            tc_fence_after_sync();
            // P^T and dS^T = P^T (dP^T - D) as BF16 side by side over the dP columns, 16 at a time, and dS^T into shared memory
            const float4* dv4 = reinterpret_cast<const float4*>(dv + c0);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t dp[16], pk[8];
                tmem_ld_x16(t_dp + c * 16, dp);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; i += 2) {
                    const float4 d4 = dv4[c * 4 + i / 4];
                    const uint64_t d = add_f32x2(pack_f32x2(__uint_as_float(dp[i]), __uint_as_float(dp[i + 1])),
                                                 i % 4 ? pack_f32x2(-d4.z, -d4.w) : pack_f32x2(-d4.x, -d4.y));
                    float y0, y1;
                    unpack_f32x2(mul_f32x2(pack_f32x2(pr[c * 16 + i], pr[c * 16 + i + 1]), d), y0, y1);
                    pk[i / 2] = pack_bf16x2(y0, y1);
                }
                tmem_st_x8(t_dp + c * 16 + 8, pk);
#pragma unroll
                for (int g = 0; g < 2; ++g)
                    *reinterpret_cast<uint4*>(ds_row + ((((part & 1) * 4 + c * 2 + g) ^ (row & 7)) << 4)) =
                        make_uint4(pk[4 * g], pk[4 * g + 1], pk[4 * g + 2], pk[4 * g + 3]);
#pragma unroll
                for (int i = 0; i < 8; ++i) pk[i] = pack_bf16x2(pr[c * 16 + 2 * i], pr[c * 16 + 2 * i + 1]);
                tmem_st_x8(t_dp + c * 16, pk);
            }
            fence_proxy_async_smem();  // ordinary stores before the product's reads
            tmem_wait_st();
            tc_fence_before_sync();
            mbar_arrive(bar_pds_full);
            if (u + 1 < n_heads) load_rows(h0 + u + 1);  // under the products
            write_dq(u);
            if (!ok) break;
        }
        // parts 0, 1 write dV, parts 2, 3 dK (times scale); each takes D / 2 columns of its key row
        if (ok) ok = mbar_wait_warp(bar_acc, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_MMA);
        if (ok && (!ONE || p.group == 1)) {
            tc_fence_after_sync();
            const bool is_dk = part >= 2;
            const float mul = is_dk ? p.scale : 1.f;
            const int col0 = (part & 1) * (D / 2);
            uint16_t* out = (is_dk ? p.dk : p.dv) + size_t(b) * p.k_sb + size_t(hk) * p.k_sh + size_t(w4 * 32) * p.k_st + col0;
            uint8_t* stage = sdS + warp * kRowStageBytes;  // (32 KB; every product is done)
#pragma unroll
            for (int c = 0; c < D / 64; ++c) {
                uint32_t v[32], w[16];
                tmem_ld_x32(tmem + lane_base + (is_dk ? Cfg::kColDK : Cfg::kColDV) + col0 + c * 32, v);
                tmem_wait_ld();
#pragma unroll
                for (int i = 0; i < 16; ++i) w[i] = pack_bf16x2(__uint_as_float(v[2 * i]) * mul, __uint_as_float(v[2 * i + 1]) * mul);
                store_rows_64b(stage, w, lane, out + c * 32, p.k_st, p.T - w4 * 32);
            }
        }
    }

    if (ONE && p.group > 1) {
        // Every role comes here, also after a wait that gave up and when the status word was set before the launch.  Key row r is
        // finished by CTA r group / 128 of the cluster; the tiles in shared memory make room for the arrivals, so all CTAs must be
        // through with theirs first.  Nobody writes dV and dK of a group of which a CTA has failed.
        const int n = p.group, max_rows = (128 + n - 1) / n;
        auto first_row = [&](int c) { return (128 * c + n - 1) / n; };
        volatile uint32_t* fail = reinterpret_cast<volatile uint32_t*>(sLse);  // [CTA of the cluster]
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        const bool failed = *abort_flag != 0;  // (final: every warp of the CTA has passed the barrier)
        if (tid < n) cluster_store_1(const_cast<uint32_t*>(fail) + rank, tid, failed);
        __syncwarp();
        if (tid < Cfg::kComputeThreads && !failed) {
            tc_fence_after_sync();
            const int row = (warp & 3) * 32 + lane, part = warp >> 2, to = (row * n) >> 7, r = row - first_row(to);
            // [source CTA][row][dV: D, dK: D] FP32, 16-byte pieces swizzled by the row: the rows of a warp would share a bank
            uint8_t* own = smem + (rank * max_rows + r) * D * 8;
            const uint32_t dst = cluster_addr(own, to);
            const uint32_t t_acc = tmem + (uint32_t((warp & 3) * 32) << 16) + (part < 2 ? Cfg::kColDV : Cfg::kColDK) + (part & 1) * (D / 2);
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
        for (int k = 0; k < n; ++k) good = good && fail[k] == 0;
        if (tid < Cfg::kComputeThreads && good) {
            const int k0 = first_row(rank), rows = first_row(rank + 1) - k0;
            for (int i = tid; i < rows * (D / 4); i += Cfg::kComputeThreads) {  // eight columns each: dV, then dK
                const int r = i / (D / 4), c8 = i % (D / 4);
                if (k0 + r >= p.T) break;
                float acc[8] = {};
#pragma unroll 2
                for (int k = 0; k < n; ++k) {
                    const uint8_t* src = smem + (k * max_rows + r) * D * 8;
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
    if (warp == Cfg::kMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, Cfg::kTmemCols);
    }
}

}  // namespace b200attn
