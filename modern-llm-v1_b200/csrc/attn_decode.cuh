// Split-KV decode for sm_100a: one query token per sequence against a KV cache.
// The reference has no such path (infer_modern_gpt re-runs the whole forward per token,
// llm/apps/infer_modern_gpt.cu:253-255); the math is row L-1 of its causal attention
// (llm/src/model/flash_attn.cu:28-131) with T = L.
//
// Large caches are bound by HBM (every K and V byte is read exactly once), small ones by latency.  A unit is one
// (batch, KV head, chunk of at most 16 query heads of the group): all its query heads are served from the same K/V tile,
// which is the bandwidth win of GQA.  One launch does everything; it deals the units' tiles in one of two ways
// (decode_plan in b200attn_api.cu chooses):
//  * shares: a unit's tiles are split evenly over 1, 2, 4 or 8 CTAs, a cluster, which exchange their partial results
//    through distributed shared memory, each CTA finishing a slice of the outputs.  (A caller may ask for any other number of
//    shares; their partial results go through the workspace as in the next deal.)
//  * ranges: the tiles of all units are numbered through and CTA c of n takes tiles [c total / n, (c + 1) total / n), the
//    same number for every CTA (to one) whatever the units' lengths are.  A range falls into pieces at unit boundaries; a
//    piece that is a whole unit is written at once, the pieces of a unit that several CTAs share are left un-normalised
//    (m, l, O) in the workspace, and the CTA that finishes last (a counter per shared unit) adds them up in the order of
//    the tiles, so the result does not depend on who was last.
//
// K/V tiles stream through a 96 KB shared-memory ring filled by TMA (128-byte swizzle, which also makes the row-per-thread
// reads bank-conflict free); the ring runs on across pieces.  Two CTAs share an SM: one streams while the other is at the end
// of a piece.
//
// Roles (192 threads): warps 0-3 compute with warp-level BF16 MMAs (m16n8k16), each on its own quarter of a tile's keys.  Keys
// and head dimension are the rows and the unit's query heads the columns, S^T = K Q^T and O^T = V^T P^T, eight heads at a time
// (NH = 1 or 2): with the heads as rows the usual four of sixteen would be used, at twice the instructions.  Warp 4 = TMA
// producer (converged, one elected lane issues: from a diverged lane a TMA instruction cost 160 clocks).  Warp 5 counts the
// shared piece that a range begins with, so that the compute warps go on to the next piece at once (fence, counter and
// addition are a chain of 3 us through L2).
//
// Measured on B200 against one CTA per (unit, split), heads as MMA rows and a second kernel for the partial results, us per
// call back to back: B=1 L=110 6/2 D=64 4.1 -> 2.9; B=1 L=1500 16/4 D=128 8.5 -> 5.5; B=1 L=8192 16/4 D=128 23.8 -> 11.1;
// B=48 L=300 16/4 D=64 7.9 -> 5.3; B=300 L=200 8/8 D=64 39.3 -> 24.6; B=64 L=4096 16/4 D=64 45.2 -> 42.1 (6.39 TB/s).
// Eight compute warps in one CTA per SM, taking tiles in two groups, were slower at every piece's end (B=300: 42.8).
#pragma once

#include <algorithm>

#include "ptx.cuh"

namespace b200attn {

struct DecodeParams {
    int B, L, Hq, Hkv, group;
    int G;         // query heads per unit (a divisor of group, <= 16)
    int n_chunks;  // group / G
    int units_per_seq;  // Hkv * n_chunks
    FastDiv div_units, div_chunks, div_shares, div_tiles, div_slice;  // by units_per_seq, n_chunks, shares, tiles of L, output pairs per CTA of a cluster
    int shares;         // CTAs per unit, or 0: ranges
    int cluster;        // CTAs per cluster: shares where they exchange through distributed shared memory, else 1
    int whole;          // ranges: they begin and end at unit boundaries (all sequences have length L)
    int slot_mode;      // where a shared unit's pieces lie in the workspace, see decode_slot
    float scale, scale_log2;
    const int* lens;    // [B] cache length per sequence (1 <= lens[b]; clamped to L), or nullptr: every sequence has L
    const uint16_t* q;  // [B, Hq, D]
    uint16_t* o;        // [B, Hq, D]
    float* lse;         // [B, Hq] or nullptr
    float* part_o;      // [slot][G][D]  un-normalised
    float* part_m;      // [slot][G]     row maximum, raw score units
    float* part_l;      // [slot][G]     sum of exp2((s - m) * scale_log2)
    unsigned long long* counters;  // one per CTA, see decode_count: pieces finished of the shared unit that begins in that CTA
                                   // (not where a cluster shares it)
    unsigned long long tag;        // of this launch
    int* status;                   // status word and epoch
};

constexpr int kDecodeMaxCtas = 320, kDecodeMaxCluster = 8, kDecodeThreads = 192;
// Workspace slot of CTA c's piece of a shared unit: one per tile when there are as many slots (mode 0), one per CTA in the deal
// by shares (mode 1), else two per CTA (mode 2: a range may end one shared unit and begin another).
enum { kDecodeSlotTile = 0, kDecodeSlotCta = 1, kDecodeSlotTwo = 2 };

template <int D>
struct DecodeCfg {
    static constexpr int kKeys = D == 64 ? 128 : 64;  // per tile
    static constexpr int kTileBytes = kKeys * D * 2;  // 16 KB
    static constexpr int kStages = 3;
    static constexpr int kBoxBytes = kKeys * 64 * 2;
    static constexpr int kBoxes = D / 64;
    static constexpr int kQRow = D * 2;
    static constexpr int kQBytes = 16 * kQRow;          // rows >= G stay zero
    static constexpr int kMlBytes = 4 * 16 * 8;         // (m, l) of the four warps' heads
    // from the cluster: O slices (over the second q buffer, which a CTA with one piece does not use) and (m, l) rows
    static constexpr int kXBytes = 16 * D * 4, kXMlBytes = kDecodeMaxCluster * 16 * 8;
    static_assert(4 * 16 * D * 4 <= 2 * kTileBytes, "the warps' O rows are merged in one K/V stage");
    static constexpr int kSmemBytes = 2 * kStages * kTileBytes + kQBytes + kXBytes + kMlBytes + kXMlBytes + 256 + 1024;
    static_assert(kXBytes >= kQBytes, "the second q buffer lies in the cluster's region");
    static_assert(2 * (kSmemBytes + 1024) <= 228 * 1024, "two CTAs per SM");
};

// ---- warp-level tensor-core pieces (mma.sync is enough here: the kernel is bound by HBM and latency, and a unit has
// ---- at most sixteen query heads, an eighth of a tcgen05 tile)
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
// Byte offset of the 16-byte chunk `chunk` (8 BF16 of the head dimension) of row `r` inside a tile of
// [rows][64]-boxes written by TMA with the 128-byte swizzle.
__device__ __forceinline__ uint32_t swz_off(int r, int chunk, int box_bytes) {
    return uint32_t((chunk >> 3) * box_bytes + r * 128 + (((chunk & 7) ^ (r & 7)) << 4));
}

// Walks one CTA's pieces.  Executed by each warp on its own (all lanes alike); every warp sees the same pieces.
struct DecodeWalk {
    int t, t_end;        // next tile and end of this CTA's range, in the numbering over all units
    int b, u, j0;        // unit at t: sequence, unit within the sequence, tile within the unit
    int len, n_tiles;    // length and tiles per unit of sequence b
    int total, n_ctas;   // tiles of all units (shares: of the unit), CTAs that share them
    int cta0;            // the first of those CTAs
};

// EARLY: in front of the wait for the kernel that may write the lengths; read through L2, so that no stale copy stays in L1
template <bool EARLY = false>
__host__ __device__ __forceinline__ int decode_len(const DecodeParams& p, int b) {
#ifdef __CUDA_ARCH__
    return p.lens ? max(1, min(EARLY ? __ldcg(p.lens + b) : __ldg(p.lens + b), p.L)) : p.L;
#else
    return p.lens ? std::max(1, std::min(p.lens[b], p.L)) : p.L;
#endif
}
// First tile of CTA c's range, and the CTA whose range holds tile t.
__host__ __device__ __forceinline__ int decode_range(const DecodeWalk& w, int c) {
    const unsigned n = unsigned(w.n_ctas), q = unsigned(w.total) / n;
    return int(unsigned(c) * q + unsigned(c) * (unsigned(w.total) - q * n) / n);
}
__device__ __forceinline__ int decode_cta_of(const DecodeWalk& w, int t) {
    return int(((unsigned long long)(unsigned)(t + 1) * (unsigned)w.n_ctas - 1) / (unsigned)w.total);
}

template <int KEYS, bool EARLY = false>
__device__ __forceinline__ DecodeWalk decode_walk_start(const DecodeParams& p, int cta, int n_ctas, int lane) {
    DecodeWalk w;
    if (p.shares) {  // one piece: this CTA's share of its unit's tiles, possibly none
        const int unit = int(fastdiv(cta, p.div_shares)), rank = cta - unit * p.shares;
        w.b = int(fastdiv(unit, p.div_units));
        w.u = unit - w.b * p.units_per_seq;
        w.len = decode_len<EARLY>(p, w.b);
        w.n_tiles = (w.len + KEYS - 1) / KEYS;
        w.total = w.n_tiles;
        w.cta0 = unit * p.shares;
        w.n_ctas = p.shares;
        w.t = w.j0 = int(fastdiv(w.n_tiles * rank, p.div_shares));
        w.t_end = int(fastdiv(w.n_tiles * (rank + 1), p.div_shares));
        if (p.cluster == 1 && w.n_tiles < p.shares) {  // a sequence shorter than that: the pieces are counted, none may be empty
            w.n_ctas = w.n_tiles;
            w.t = w.j0 = min(rank, w.n_tiles);
            w.t_end = min(rank + 1, w.n_tiles);
        }
        return w;
    }
    w.cta0 = 0;
    if (!p.lens) {
        w.len = p.L;
        w.n_tiles = (p.L + KEYS - 1) / KEYS;
        w.total = p.B * p.units_per_seq * w.n_tiles;
    } else {
        int sum = 0;
        for (int b = lane; b < p.B; b += 32) sum += (decode_len<EARLY>(p, b) + KEYS - 1) / KEYS;
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        w.total = sum * p.units_per_seq;
    }
    w.n_ctas = min(n_ctas, w.total);
    w.t = cta < w.n_ctas ? decode_range(w, cta) : 0;
    w.t_end = cta < w.n_ctas ? decode_range(w, cta + 1) : 0;
    if (p.whole) {  // (rounding the ends of all ranges down alike; at least one unit per CTA)
        w.t -= w.t % w.n_tiles;
        w.t_end -= w.t_end % w.n_tiles;
    }
    if (!p.lens) {
        const int unit = int(fastdiv(w.t, p.div_tiles));
        w.j0 = w.t - unit * w.n_tiles;
        w.b = int(fastdiv(unit, p.div_units));
        w.u = unit - w.b * p.units_per_seq;
    } else {
        // the sequence that holds tile t: 32 sequences at a time
        const int target = int(fastdiv(w.t, p.div_units));  // in tiles of one unit per sequence
        int before = 0;
        w.b = p.B - 1, w.len = 1, w.n_tiles = 1, w.u = 0, w.j0 = 0;
        for (int b0 = 0; b0 < p.B; b0 += 32) {
            const int len = b0 + lane < p.B ? decode_len<EARLY>(p, b0 + lane) : 0;
            const int n = (len + KEYS - 1) / KEYS;
            int incl = n;
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += up;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, before + incl > target);
            if (hit) {
                const int src = __ffs(hit) - 1;
                w.b = b0 + src;
                w.len = __shfl_sync(0xffffffffu, len, src);
                w.n_tiles = __shfl_sync(0xffffffffu, n, src);
                const int start = (before + __shfl_sync(0xffffffffu, incl, src) - w.n_tiles) * p.units_per_seq;
                w.u = (w.t - start) / w.n_tiles;
                w.j0 = w.t - start - w.u * w.n_tiles;
                break;
            }
            before += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    return w;
}
// Tiles of the piece at w.t
__host__ __device__ __forceinline__ int decode_piece(const DecodeWalk& w) {
    const int range = w.t_end - w.t, unit = w.n_tiles - w.j0;
    return range < unit ? range : unit;
}
template <int KEYS, bool EARLY = false>
__host__ __device__ __forceinline__ void decode_walk_next(const DecodeParams& p, DecodeWalk& w, int n) {
    w.t += n;
    w.j0 = 0;  // the piece ended at its unit's end, or the range is over
    if (w.t < w.t_end && ++w.u == p.units_per_seq) {
        w.u = 0;
        ++w.b;
        // (the range's end and this sequence may come from different lengths, see decode_first_tiles)
        if (EARLY && w.b == p.B) {
            w.t = w.t_end;
            return;
        }
        w.len = decode_len<EARLY>(p, w.b);
        w.n_tiles = (w.len + KEYS - 1) / KEYS;
    }
}
// The range's first `left` tiles, for a look at them in front of the wait: visit(sequence, unit within it, tile).  The kernel in
// front may write the lengths meanwhile, so w.t_end, w.b and what is read here need not fit together: the tiles are a guess, all
// inside the cache, and the walk ends at the last sequence at the latest.
#pragma nv_exec_check_disable
template <int KEYS, typename Visit>
__host__ __device__ __forceinline__ void decode_first_tiles(const DecodeParams& p, DecodeWalk w, int left, Visit visit) {
    while (w.t < w.t_end && left > 0) {
        const int tiles = decode_piece(w);
        for (int i = 0; i < tiles && left > 0; ++i, --left) visit(w.b, w.u, w.j0 + i);
        decode_walk_next<KEYS, true>(p, w, tiles);
    }
}
__device__ __forceinline__ int decode_slot(const DecodeParams& p, const DecodeWalk& w, int c, int first_cta, int unit_start) {
    if (p.slot_mode == kDecodeSlotTile) return max(unit_start, decode_range(w, c));
    if (p.slot_mode == kDecodeSlotCta) return w.cta0 + c;
    return 2 * c + (c == first_cta ? 1 : 0);
}

// One state of the online softmax over the unit's outputs, in the MMA's register layout (see the kernel): this lane's heads
// are nh * 8 + (lane % 4) * 2 + {0, 1}, its head-dim rows of tile mt mt * 16 + lane / 4 + {0, 8}.  m is the same in the eight
// lanes that share a head, l is each lane's share of the sum.
template <int D, int NH>
struct DecodeState {
    float m[NH][2], l[NH][2];
    float o[D / 16][NH][4];  // {row, head}: 0 {0, 0}, 1 {0, 1}, 2 {8, 0}, 3 {8, 1}
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int nh = 0; nh < NH; ++nh) {
            m[nh][0] = m[nh][1] = -INFINITY;
            l[nh][0] = l[nh][1] = 0.f;
#pragma unroll
            for (int mt = 0; mt < D / 16; ++mt) o[mt][nh][0] = o[mt][nh][1] = o[mt][nh][2] = o[mt][nh][3] = 0.f;
        }
    }
};

// The CTA's start: barriers initialised, status word read.  Producer and compute warps wait for each other; the counter warp, which
// is late when it has looked ahead, waits for them and they not for it (waiting for it took 2 us where no kernel in front hides
// the look: first pass on new buffers of B=300 L=200 8/8 D=64 44.1 us against 42.1, append + decode B=48 L<=6000 16/4 70.9 against 67.0).
constexpr int kDecodeStartBar = 2, kDecodeCountBar = 3;
__device__ __forceinline__ void decode_started() {
    named_bar_sync(kDecodeStartBar, kDecodeThreads - 32);
    named_bar_arrive(kDecodeCountBar, kDecodeThreads);
}
// barrier over the four compute warps that also tells every thread whether any of them has given up
__device__ __forceinline__ bool decode_bar_ok(bool ok) {
    uint32_t bad;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.eq.u32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred q, 1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t"
        "}\n"
        : "=r"(bad)
        : "r"(uint32_t(ok))
        : "memory");
    return bad == 0;
}
// Column swizzle of the merge scratch [warp][16 heads][D] FP32: the four heads a warp writes at once would share a bank
__device__ __forceinline__ int decode_merge_col(int head, int col) { return col ^ (((head >> 1) & 3) << 3); }

// The warps' states -> one, through shared memory; `use(g, d, acc0, acc1, m, l)` is called once per pair of output elements.
template <int D, int NH, typename Use>
__device__ __forceinline__ void decode_merge(DecodeState<D, NH>& s, float* sO, float2* sMl, int warp, int lane, int tid, int G,
                                             float scale_log2, Use use) {
    {
        const int r = lane >> 2, c = (lane & 3) * 2;
        float* mine = sO + warp * 16 * D;
#pragma unroll
        for (int nh = 0; nh < NH; ++nh)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float l = s.l[nh][e];
                l += __shfl_xor_sync(0xffffffffu, l, 4);
                l += __shfl_xor_sync(0xffffffffu, l, 8);
                l += __shfl_xor_sync(0xffffffffu, l, 16);
                const int g = nh * 8 + c + e;
                if (g >= G) continue;
#pragma unroll
                for (int mt = 0; mt < D / 16; ++mt) {
                    mine[g * D + decode_merge_col(g, mt * 16 + r)] = s.o[mt][nh][e];
                    mine[g * D + decode_merge_col(g, mt * 16 + r + 8)] = s.o[mt][nh][e + 2];
                }
                if (r == 0) sMl[warp * 16 + g] = make_float2(s.m[nh][e], l);
            }
    }
    named_bar_sync(1, 128);
    for (int i = tid; i < G * (D / 2); i += 128) {
        const int g = i / (D / 2), d = (i % (D / 2)) * 2;
        float2 ml[4], v[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            ml[w] = sMl[w * 16 + g];
            v[w] = *reinterpret_cast<const float2*>(sO + (w * 16 + g) * D + decode_merge_col(g, d));
        }
        const float m = fmaxf(fmaxf(ml[0].x, ml[1].x), fmaxf(ml[2].x, ml[3].x));
        float a0 = 0.f, a1 = 0.f, l = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float f = (ml[w].x == -INFINITY) ? 0.f : ex2_approx((ml[w].x - m) * scale_log2);
            a0 += f * v[w].x;
            a1 += f * v[w].y;
            l += f * ml[w].y;
        }
        use(g, d, a0, a1, m, l);
    }
}

// One pair of output elements of a shared unit from its pieces in the workspace, in the order of the tiles.  `own`: the CTA
// whose piece is passed in registers instead (the same values it would have stored), or -1.
template <int D, typename Write>
__device__ __forceinline__ void decode_add_pieces(const DecodeParams& p, const DecodeWalk& w, int first, int last, int unit_start, int g,
                                                  int d, int own, float own0, float own1, float own_m, float own_l, Write write) {
    float m = -INFINITY, l = 0.f, a0 = 0.f, a1 = 0.f;
    for (int c0 = first; c0 <= last; c0 += 4) {
        float pm[4], pl[4];
        float2 po[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int c = c0 + k;
            pm[k] = own_m, pl[k] = own_l, po[k] = make_float2(own0, own1);
            if (c <= last && c != own) {
                const size_t row = size_t(decode_slot(p, w, c, first, unit_start)) * p.G + g;
                pm[k] = __ldcg(p.part_m + row);
                pl[k] = __ldcg(p.part_l + row);
                po[k] = __ldcg(reinterpret_cast<const float2*>(p.part_o + row * D + d));
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (c0 + k > last) break;
            const float mn = fmaxf(m, pm[k]);  // finite: every piece has a key
            const float fa = ex2_approx((m - mn) * p.scale_log2), fb = ex2_approx((pm[k] - mn) * p.scale_log2);
            m = mn;
            l = l * fa + fb * pl[k];
            a0 = a0 * fa + fb * po[k].x;
            a1 = a1 * fa + fb * po[k].y;
        }
    }
    write(g, d, a0, a1, m, l);
}
__device__ __forceinline__ unsigned long long decode_ld_acquire(const unsigned long long* a) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(a) : "memory");
    return v;
}
// The counters lie in the caller's workspace, so that launches which may overlap (other streams, other graphs) never share one,
// and nobody clears them: a word is launch tag (40 bits), epoch (14 bits) and count (10 bits), and one with another tag or epoch,
// whatever the workspace held before, counts as zero.  The last piece of a unit puts its count back to zero, so a captured
// launch, which keeps its tag, can be replayed; what a launch that gave up leaves behind has the epoch before, which ends when
// the host takes the error off the status word.  (Words that nobody has counted in: one in 2^54 would pass.)
constexpr int kDecodeCountBits = 10, kDecodeEpochBits = 14;
static_assert(kDecodeMaxCtas < (1 << kDecodeCountBits), "a count fits");
// One more piece finished; returns how many there are now.  `seen`: what the word held at some point of this launch.
__device__ __forceinline__ int decode_count(unsigned long long* word, unsigned long long tag, unsigned long long seen) {
    if ((seen >> kDecodeCountBits) != (tag >> kDecodeCountBits)) {
        if (atomicCAS(word, seen, tag + 1) == seen) return 1;
        // another CTA of this launch has tagged it meanwhile
    }
    return int(atomicAdd(word, 1ull) - tag) + 1;
}

// PF: tiles that a CTA brings into L2 while the kernel in front of this one ends
template <int D, int NH, int PF>
__global__ void __launch_bounds__(kDecodeThreads, 2)
attn_decode_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const DecodeParams p) {
    using Cfg = DecodeCfg<D>;
    constexpr int KEYS = Cfg::kKeys;
    constexpr int NST = Cfg::kStages;
    constexpr int KS = D / 16;     // k-steps of Q K^T
    constexpr int MT = D / 16;     // 16-row output tiles of V^T P^T
    constexpr int KT = KEYS / 64;  // 16-key tiles per warp
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* sKV = smem;                                                 // [NST] K tile, V tile
    uint8_t* sQ = sKV + NST * 2 * Cfg::kTileBytes;                       // [2][16 rows]
    float2* sX = reinterpret_cast<float2*>(sQ + Cfg::kQBytes);           // [CTA of the cluster][slice of the output pairs]
    float2* sMl = reinterpret_cast<float2*>(sQ + Cfg::kQBytes + Cfg::kXBytes);  // [4 warps][16 heads]
    float2* sXMl = sMl + 4 * 16;                                         // [CTA of the cluster][16 heads]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sXMl + kDecodeMaxCluster * 16);
    uint64_t* bar_full = bars;              // [NST]
    uint64_t* bar_free = bars + NST;        // [NST]
    uint64_t* bar_q = bars + 2 * NST;       // [2] the q rows of a piece have landed   (phase: piece / 2)
    uint64_t* bar_q_free = bar_q + 2;       // [2] they are in registers               (phase: piece / 2)
    uint64_t* bar_part = bar_q_free + 2;    // the shared piece at the range's beginning has been stored
    volatile int* abort_flag = reinterpret_cast<volatile int*>(bar_part + 1);
    volatile int* last_flag = abort_flag + 1;
    volatile int* fail_flag = abort_flag + 2;
    volatile int* epoch = abort_flag + 3;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = p.G;

    // The next kernel of the stream may be brought in as soon as every CTA of this one has started (all at once where they fit
    // the device, else with the last round): its set-up then runs under this kernel, and it waits for this kernel's end before
    // it touches global memory.
    grid_dep_launch();
    if (p.cluster > 1) cluster_arrive();  // waited for in front of the first access to another CTA's shared memory
    if (warp == 4) {
        // ------------------------------------------------------------------ producer
        if (elect_one()) {
            tma_prefetch_desc(&tmK);
            tma_prefetch_desc(&tmV);
            *abort_flag = 0;
        }
        if (lane < 2 * NST + 5) {  // in the order of `bars`: full, free, q, q_free, part
            mbar_init(bars + lane, lane < NST ? 1 : lane < 2 * NST ? 128 : lane < 2 * NST + 2 ? 1 : 128);
            fence_mbar_init();
        }
        __syncwarp();
        // everything above overlaps the previous kernel's end (the cache append that wrote q and the newest K / V row)
        grid_dep_wait();
        DecodeWalk w = decode_walk_start<KEYS>(p, int(blockIdx.x), int(gridDim.x), lane);
        int j = 0;  // tiles issued so far (ring position)
        bool synced = false, ok = true;
        for (int n = 0; w.t < w.t_end && ok; ++n) {
            const int tiles = decode_piece(w);
            const int hk = int(fastdiv(w.u, p.div_chunks)), h0 = hk * p.group + (w.u - hk * p.n_chunks) * G;
            for (int i = 0; i < tiles; ++i, ++j) {
                const int s = j % NST;
                if (j >= NST) {
                    if (!synced) decode_started(), synced = true;  // the other warps have started
                    ok = mbar_wait_warp(&bar_free[s], ((j / NST) - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
                    if (!ok) break;
                }
                if (elect_one()) {
                    mbar_arrive_expect_tx(&bar_full[s], 2 * Cfg::kTileBytes);
                    uint8_t* k = sKV + s * 2 * Cfg::kTileBytes;
#pragma unroll
                    for (int bx = 0; bx < Cfg::kBoxes; ++bx) {
                        tma_load_4d(k + bx * Cfg::kBoxBytes, &tmK, &bar_full[s], bx * 64, (w.j0 + i) * KEYS, hk, w.b);
                        tma_load_4d(k + Cfg::kTileBytes + bx * Cfg::kBoxBytes, &tmV, &bar_full[s], bx * 64, (w.j0 + i) * KEYS, hk, w.b);
                    }
                }
                __syncwarp();
                if (i == 0) {  // behind the first tile's requests: the piece's q rows
                    if (n >= 2) {
                        if (!synced) decode_started(), synced = true;
                        ok = mbar_wait_warp(&bar_q_free[n & 1], ((n >> 1) - 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_FREE);
                        if (!ok) break;
                    }
                    if (elect_one()) {
                        mbar_arrive_expect_tx(&bar_q[n & 1], G * D * 2);
                        bulk_load_1d(sQ + (n & 1) * Cfg::kQBytes, p.q + (size_t(w.b) * p.Hq + h0) * D, G * D * 2, &bar_q[n & 1]);
                    }
                    __syncwarp();
                }
            }
            decode_walk_next<KEYS>(p, w, tiles);
        }
        if (!synced) decode_started();
        return;
    }

    auto write_rows_of = [&](const DecodeWalk& w) {  // final rows of the unit at w
        const int hk = int(fastdiv(w.u, p.div_chunks));
        const size_t row0 = size_t(w.b) * p.Hq + hk * p.group + (w.u - hk * p.n_chunks) * G;
        return [&p, row0](int g, int d, float a0, float a1, float m, float l) {
            const float inv = 1.f / l;
            reinterpret_cast<uint32_t*>(p.o)[(row0 + g) * (D / 2) + d / 2] = pack_bf16x2(a0 * inv, a1 * inv);
            if (p.lse && d == 0) p.lse[row0 + g] = m * p.scale + logf(l);
        };
    };
    if (warp == 5) {
        // ------------------------------------------------------------------ counter of the range's first piece
        // First, while the kernel in front is still at work: this CTA's first tiles into L2 (coherent: what that kernel still
        // writes there is what the loads behind the wait find).
        if constexpr (PF > 0) {
            const DecodeWalk w = decode_walk_start<KEYS, true>(p, int(blockIdx.x), int(gridDim.x), lane);
            decode_first_tiles<KEYS>(p, w, PF, [&](int b, int u, int tile) {
                const int hk = int(fastdiv(u, p.div_chunks));
                if (elect_one()) {
#pragma unroll
                    for (int bx = 0; bx < Cfg::kBoxes; ++bx) {
                        tma_prefetch_4d(&tmK, bx * 64, tile * KEYS, hk, b);
                        tma_prefetch_4d(&tmV, bx * 64, tile * KEYS, hk, b);
                    }
                }
                __syncwarp();
            });
        }
        grid_dep_wait();
        const DecodeWalk w = decode_walk_start<KEYS>(p, int(blockIdx.x), int(gridDim.x), lane);
        named_bar_sync(kDecodeCountBar, kDecodeThreads);
        if (p.shares || *fail_flag != 0 || w.t >= w.t_end) return;
        const int tiles = decode_piece(w);
        if (tiles == w.n_tiles || w.t + tiles == w.t_end) return;
        const int unit_start = w.t - w.j0;
        const int first = decode_cta_of(w, unit_start), last = decode_cta_of(w, unit_start + w.n_tiles - 1);
        const unsigned long long tag = p.tag + ((unsigned long long)*epoch << kDecodeCountBits);
        const unsigned long long seen = decode_ld_acquire(p.counters + first);
        if (!mbar_wait_warp(bar_part, 0, abort_flag, p.status, DEV_WAIT_TIMEOUT_SOFTMAX)) return;
        int is_last = 0;
        if (lane == 0) {
            __threadfence();
            is_last = decode_count(p.counters + first, tag, seen) == last - first + 1;
            if (is_last) p.counters[first] = tag;
            __threadfence();
        }
        if (!__shfl_sync(0xffffffffu, is_last, 0)) return;
        const auto write = write_rows_of(w);
        for (int i = lane; i < G * (D / 2); i += 32)
            decode_add_pieces<D>(p, w, first, last, unit_start, i / (D / 2), (i % (D / 2)) * 2, -1, 0.f, 0.f, 0.f, 0.f, write);
        return;
    }

    // ---------------------------------------------------------------------- compute warps
    for (int i = tid; i < (p.cluster > 1 ? 1 : 2) * (16 - G) * (D / 8); i += 128) {  // rows >= G of the q buffers
        const int buf = i / ((16 - G) * (D / 8)), r = i % ((16 - G) * (D / 8));
        *reinterpret_cast<uint4*>(sQ + buf * Cfg::kQBytes + (G + r / (D / 8)) * Cfg::kQRow + (r % (D / 8)) * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    grid_dep_wait();
    // (a launch behind a failure writes nothing; its loads are harmless, but shared memory has to outlive them)
    if (tid == 0) {
        *fail_flag = *reinterpret_cast<volatile int*>(p.status);
        *epoch = *reinterpret_cast<volatile int*>(p.status + 1);
    }
    DecodeWalk w = decode_walk_start<KEYS>(p, int(blockIdx.x), int(gridDim.x), lane);
    decode_started();
    const bool failed = *fail_flag != 0;
    bool ok = true;
    const int rank = p.cluster > 1 ? int(blockIdx.x) % p.cluster : 0;
    bool sent = false;
    int j = 0;  // tiles before this piece (ring position)
    for (int n = 0; w.t < w.t_end; ++n) {
        const int tiles = decode_piece(w);
        DecodeState<D, NH> st;
        st.clear();
        uint32_t bq[KS][NH][2];  // B fragments of Q^T (columns = heads)
        if (ok) ok = mbar_wait_warp(&bar_q[n & 1], (n >> 1) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
        {
            const uint32_t q_base = smem_u32(sQ + (n & 1) * Cfg::kQBytes);
#pragma unroll
            for (int nh = 0; nh < NH; ++nh)
#pragma unroll
                for (int ks = 0; ks < KS; ks += 2)  // matrices 0-3: head-dim chunks 2ks .. 2ks+3 of heads nh * 8 .. + 8
                    ldsm_x4(q_base + (nh * 8 + (lane & 7)) * Cfg::kQRow + (ks * 2 + (lane >> 3)) * 16, bq[ks][nh][0], bq[ks][nh][1],
                            bq[ks + 1][nh][0], bq[ks + 1][nh][1]);
            fence_proxy_async_smem();
            mbar_arrive(&bar_q_free[n & 1]);
        }
        const int kw = warp * (KEYS / 4);  // this warp's keys inside a tile
        for (int i = 0; i < tiles; ++i, ++j) {
            const int s = j % NST;
            ok = ok && mbar_wait_warp(&bar_full[s], (j / NST) & 1, abort_flag, p.status, DEV_WAIT_TIMEOUT_LOAD);
            if (!ok) break;
            const uint32_t k_base = smem_u32(sKV + s * 2 * Cfg::kTileBytes);
            const uint32_t v_base = k_base + Cfg::kTileBytes;
            // ---- S^T[keys x heads] = K Q^T, the keys of this warp in tiles of 16
            float sc[KT][NH][4];  // {key, head}: 0 {0, 0}, 1 {0, 1}, 2 {8, 0}, 3 {8, 1} of key lane / 4, head (lane % 4) * 2
#pragma unroll
            for (int kt = 0; kt < KT; ++kt) {
                float odd[NH][4];  // a second accumulator: half the chain of dependent products
#pragma unroll
                for (int nh = 0; nh < NH; ++nh)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sc[kt][nh][e] = odd[nh][e] = 0.f;
                const int key = kw + kt * 16 + (lane & 15);
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) {
                    uint32_t a[4];
                    ldsm_x4(k_base + swz_off(key, ks * 2 + (lane >> 4), Cfg::kBoxBytes), a[0], a[1], a[2], a[3]);
#pragma unroll
                    for (int nh = 0; nh < NH; ++nh) mma_bf16_16816((ks & 1) ? odd[nh] : sc[kt][nh], a, bq[ks][nh][0], bq[ks][nh][1]);
                }
#pragma unroll
                for (int nh = 0; nh < NH; ++nh)
#pragma unroll
                    for (int e = 0; e < 4; ++e) sc[kt][nh][e] += odd[nh][e];
            }
            // ---- mask keys beyond the cache length (a unit's last tile only)
            const int tile_key = (w.j0 + i) * KEYS;
            if (tile_key + KEYS > w.len) {
#pragma unroll
                for (int kt = 0; kt < KT; ++kt) {
                    const int key = tile_key + kw + kt * 16 + (lane >> 2);
#pragma unroll
                    for (int nh = 0; nh < NH; ++nh) {
                        if (key >= w.len) sc[kt][nh][0] = sc[kt][nh][1] = -INFINITY;
                        if (key + 8 >= w.len) sc[kt][nh][2] = sc[kt][nh][3] = -INFINITY;
                    }
                }
            }
            // ---- online softmax per head over this warp's keys; P^T becomes the B operand of the second product: rows and
            // columns of its 8 x 8 blocks change places (movmatrix)
            uint32_t bp[KT][NH][2];
#pragma unroll
            for (int nh = 0; nh < NH; ++nh) {
                float alpha[2], nb[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float mx = -INFINITY;
#pragma unroll
                    for (int kt = 0; kt < KT; ++kt) mx = fmaxf(mx, fmaxf(sc[kt][nh][e], sc[kt][nh][e + 2]));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                    const float mn = fmaxf(st.m[nh][e], mx);
                    // a warp whose keys are all beyond the cache has mn = -inf: keep its state neutral
                    alpha[e] = (mn == -INFINITY) ? 1.f : ex2_approx((st.m[nh][e] - mn) * p.scale_log2);
                    nb[e] = (mn == -INFINITY) ? 0.f : -mn * p.scale_log2;
                    st.m[nh][e] = mn;
                    st.l[nh][e] *= alpha[e];
                }
#pragma unroll
                for (int kt = 0; kt < KT; ++kt) {
                    const float p0 = ex2_approx(fmaf(sc[kt][nh][0], p.scale_log2, nb[0]));
                    const float p1 = ex2_approx(fmaf(sc[kt][nh][1], p.scale_log2, nb[1]));
                    const float p2 = ex2_approx(fmaf(sc[kt][nh][2], p.scale_log2, nb[0]));
                    const float p3 = ex2_approx(fmaf(sc[kt][nh][3], p.scale_log2, nb[1]));
                    st.l[nh][0] += p0 + p2;
                    st.l[nh][1] += p1 + p3;
                    bp[kt][nh][0] = movmatrix_trans(pack_bf16x2(p0, p1));
                    bp[kt][nh][1] = movmatrix_trans(pack_bf16x2(p2, p3));
                }
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    st.o[mt][nh][0] *= alpha[0];
                    st.o[mt][nh][1] *= alpha[1];
                    st.o[mt][nh][2] *= alpha[0];
                    st.o[mt][nh][3] *= alpha[1];
                }
            }
            // ---- O^T[D x heads] += V^T P^T
#pragma unroll
            for (int kt = 0; kt < KT; ++kt) {
                const int key = kw + kt * 16 + (lane & 7) + ((lane >> 4) << 3);  // matrices 0,1: keys 0-7; 2,3: 8-15
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    uint32_t a[4];  // matrices 0,2: head-dim rows 0-7; 1,3: 8-15
                    ldsm_x4_trans(v_base + swz_off(key, mt * 2 + ((lane >> 3) & 1), Cfg::kBoxBytes), a[0], a[1], a[2], a[3]);
#pragma unroll
                    for (int nh = 0; nh < NH; ++nh) mma_bf16_16816(st.o[mt][nh], a, bp[kt][nh][0], bp[kt][nh][1]);
                }
            }
            if (i + 1 < tiles) {
                // ordinary (ldmatrix) reads of a stage that TMA will overwrite: ordered before the async proxy's write
                fence_proxy_async_smem();
                mbar_arrive(&bar_free[s]);
            }
        }
        // ---- end of the piece.  Its last stage stays with the compute warps as scratch until the piece is written.
        ok = decode_bar_ok(ok);
        if (!ok) break;
        const int s_last = (j - 1) % NST;
        if (failed) {
            // every piece's loads are waited for, nothing is written
            if (p.cluster > 1) break;  // (one piece)
            fence_proxy_async_smem();
            mbar_arrive(&bar_free[s_last]);
            decode_walk_next<KEYS>(p, w, tiles);
            continue;
        }
        float* sO = reinterpret_cast<float*>(sKV + s_last * 2 * Cfg::kTileBytes);
        const auto write_rows = write_rows_of(w);
        if (p.cluster > 1) {
            // output pair e belongs to CTA e / slice of the cluster; every CTA needs everyone's (m, l)
            const int slice = int(p.div_slice.d);
            cluster_wait();
            decode_merge<D, NH>(st, sO, sMl, warp, lane, tid, G, p.scale_log2, [&](int g, int d, float a0, float a1, float m, float l) {
                const int e = g * (D / 2) + d / 2, to = int(fastdiv(e, p.div_slice));
                cluster_store_f2(&sX[rank * slice + e - to * slice], to, make_float2(a0, a1));
                if (d == 0)
                    for (int c = 0; c < p.cluster; ++c) cluster_store_f2(&sXMl[rank * 16 + g], c, make_float2(m, l));
            });
            sent = true;
            break;
        } else if (tiles == w.n_tiles) {
            decode_merge<D, NH>(st, sO, sMl, warp, lane, tid, G, p.scale_log2, write_rows);
        } else {
            const int cta = int(blockIdx.x) - w.cta0;
            const int unit_start = w.t - w.j0;
            const int first = decode_cta_of(w, unit_start), last = decode_cta_of(w, unit_start + w.n_tiles - 1);
            const size_t slot = decode_slot(p, w, cta, first, unit_start);
            const bool ends_range = w.t + tiles == w.t_end;
            // At the range's end nothing is left to hide latency behind.  Usually all other pieces have been stored by then
            // (they lie at the beginning of their CTAs' ranges): one look at the counter instead of store, fence and count.
            unsigned long long* const counter = p.counters + w.cta0 + first;
            const unsigned long long tag = p.tag + ((unsigned long long)*epoch << kDecodeCountBits);
            unsigned long long seen = 0;
            if (tid == 0 && ends_range) seen = decode_ld_acquire(counter);
            if (tid == 0) *last_flag = ends_range && seen == tag + (last - first);
            decode_merge<D, NH>(st, sO, sMl, warp, lane, tid, G, p.scale_log2, [&](int g, int d, float a0, float a1, float m, float l) {
                if (*last_flag) {
                    decode_add_pieces<D>(p, w, first, last, unit_start, g, d, cta, a0, a1, m, l, write_rows);
                    return;
                }
                *reinterpret_cast<float2*>(p.part_o + (slot * G + g) * D + d) = make_float2(a0, a1);
                if (d == 0) {
                    p.part_m[slot * G + g] = m;
                    p.part_l[slot * G + g] = l;
                }
            });
            if (!ends_range) {
                mbar_arrive(bar_part);
            } else if (*last_flag) {
                if (tid == 0) *counter = tag;
            } else {
                __threadfence();
                named_bar_sync(1, 128);
                if (tid == 0) {
                    const bool is_last = decode_count(counter, tag, seen) == last - first + 1;
                    if (is_last) *counter = tag;
                    *last_flag = is_last;
                    __threadfence();
                }
                named_bar_sync(1, 128);
                if (*last_flag)
                    for (int i = tid; i < G * (D / 2); i += 128)
                        decode_add_pieces<D>(p, w, first, last, unit_start, i / (D / 2), (i % (D / 2)) * 2, -1, 0.f, 0.f, 0.f, 0.f, write_rows);
            }
        }
        // the scratch was written and read with ordinary accesses; the stage goes back to TMA
        fence_proxy_async_smem();
        mbar_arrive(&bar_free[s_last]);
        named_bar_sync(1, 128);  // sMl and the flag are rewritten at the next piece's end
        decode_walk_next<KEYS>(p, w, tiles);
    }
    if (p.cluster <= 1) return;
    // ---- the cluster's partial results: this CTA finishes its slice of the outputs.  A CTA without tiles sends weight zero, one
    // that has failed a negative row sum, upon which nobody writes the unit; nobody leaves before everybody's stores have landed.
    if (!sent) {
        cluster_wait();
        for (int i = tid; i < G * p.cluster; i += 128)
            cluster_store_f2(&sXMl[rank * 16 + i / p.cluster], i % p.cluster, make_float2(-INFINITY, failed || !ok ? -1.f : 0.f));
    }
    cluster_arrive();
    cluster_wait();
    const int slice = int(p.div_slice.d);
    const auto write_rows = write_rows_of(w);
    for (int i = tid; i < slice; i += 128) {
        const int e = rank * slice + i, g = e / (D / 2), d2 = e - g * (D / 2);
        float2 ml[kDecodeMaxCluster], v[kDecodeMaxCluster];
#pragma unroll
        for (int c = 0; c < kDecodeMaxCluster; ++c) {
            ml[c] = c < p.cluster ? sXMl[c * 16 + g] : make_float2(-INFINITY, 0.f);
            v[c] = c < p.cluster ? sX[c * slice + i] : make_float2(0.f, 0.f);
        }
        float m = ml[0].x;
        bool good = !(ml[0].y < 0.f);
#pragma unroll
        for (int c = 1; c < kDecodeMaxCluster; ++c) {
            m = fmaxf(m, ml[c].x);
            good = good && !(ml[c].y < 0.f);
        }
        if (!good) return;  // a CTA has failed (and said so for every head)
        float a0 = 0.f, a1 = 0.f, l = 0.f;
#pragma unroll
        for (int c = 0; c < kDecodeMaxCluster; ++c) {
            if (ml[c].x == -INFINITY && ml[c].y == 0.f) continue;  // no tiles: its slots hold nothing (all scores NaN: l is NaN)
            const float f = ex2_approx((ml[c].x - m) * p.scale_log2);
            a0 += f * v[c].x;
            a1 += f * v[c].y;
            l += f * ml[c].y;
        }
        write_rows(g, d2 * 2, a0, a1, m, l);
    }
}

}  // namespace b200attn
