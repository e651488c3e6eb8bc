// C-ABI launcher for the sm_100a attention kernels (see include/b200attn.h for
// the contract).  Host side only validates, builds TMA tensor maps and enqueues.
#include "../../include/b200attn.h"
#include "b200attn_debug.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <functional>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>

#include "attn_bwd.cuh"
#include "attn_bwd_onepass.cuh"
#include "attn_bwd_tile.cuh"
#include "attn_decode.cuh"
#include "attn_fwd.cuh"
#include "kv_cache.cuh"
#include "rope_norm.cuh"
#include "tmap.h"

using namespace b200attn;

namespace {

// One status word per device, living in the library's device image, and behind it the epoch: how many errors have been taken
// off the word (see decode_count).
__device__ int g_status_word[2];

constexpr int kMaxDevices = 64;
std::atomic<int*> g_status_ptr[kMaxDevices] = {};  // (the words are zero at load)

// Item counters of the persistent kernels (two words per launch, see ptx.cuh), also in the device
// image (zero at load).  A kernel leaves its two words zero again when it ends, so one pair would do
// for launches that follow each other on one stream; consecutive launches take consecutive pairs so
// that launches running at the same time on different streams do not share one.  (Two launches
// kSchedSlots launches apart that overlap in time, or one captured graph replayed concurrently with
// itself, would share a pair: serialise those.)  A kernel that gave up on a wait may leave its pair
// non-zero; b200attn_last_device_status clears all pairs when it reports such a failure, and until
// then every kernel exits at once because the status word is set.
constexpr int kSchedSlots = 64;
__device__ int g_sched_words[2 * kSchedSlots];
std::atomic<int*> g_sched_ptr[kMaxDevices] = {};
std::atomic<unsigned> g_sched_seq{0};

// What tells a decode launch's counters from those of every other launch (see decode_count).  The sequence starts anywhere, so
// that the counters of another process in recycled memory are as unlikely to pass as anything else.
std::atomic<unsigned long long> g_decode_seq{0};
unsigned long long next_decode_tag() {
    static const unsigned long long start = [] {
        unsigned long long x = (unsigned long long)std::chrono::steady_clock::now().time_since_epoch().count() +
                               (unsigned long long)reinterpret_cast<uintptr_t>(&g_decode_seq);
        x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;  // the finaliser of SplitMix64 (Steele, Lea and Flood)
        x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
        return x ^ (x >> 31);
    }();
    return (start + g_decode_seq.fetch_add(1, std::memory_order_relaxed)) << (kDecodeCountBits + kDecodeEpochBits);
}

// Returns the device address of the status word of the current device (resolved once per device).
int* status_ptr(int* err) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        *err = B200ATTN_ERR_NO_DEVICE;
        return nullptr;
    }
    int* status = g_status_ptr[dev].load(std::memory_order_acquire);
    if (!status) {  // several threads may come here at once: all find the same addresses
        void *p = nullptr, *sp = nullptr;
        if (cudaGetSymbolAddress(&p, g_status_word) != cudaSuccess || cudaGetSymbolAddress(&sp, g_sched_words) != cudaSuccess) {
            cudaGetLastError();
            *err = B200ATTN_ERR_NO_DEVICE;
            return nullptr;
        }
        status = static_cast<int*>(p);
        g_sched_ptr[dev].store(static_cast<int*>(sp), std::memory_order_relaxed);
        g_status_ptr[dev].store(status, std::memory_order_release);
    }
    return status;
}

// The counter pair for the next launch of a persistent kernel on the current device (status_ptr()
// has resolved the device's addresses before).
// Returns nullptr when the items should be dealt statically: with only a few items per CTA a static
// deal in rounds of alternating direction balances better than first come, first served, because a CTA
// takes its next item before it has finished the current one.  (B200ATTN_ITEMS=static|dynamic overrides.)
int* next_sched_pair(long long n_items, unsigned n_ctas) {
    static const int forced = [] {
        const char* e = getenv("B200ATTN_ITEMS");
        return !e ? 0 : (e[0] == 's' ? 1 : (e[0] == 'd' ? 2 : 0));
    }();
    if (forced == 1 || (forced == 0 && n_items < 4LL * n_ctas)) return nullptr;
    int dev = 0;
    cudaGetDevice(&dev);
    return g_sched_ptr[dev].load(std::memory_order_relaxed) + 2 * (g_sched_seq.fetch_add(1, std::memory_order_relaxed) % kSchedSlots);
}

// The static deal of the forward and the dQ pass (two CTAs per SM) as a table: items (ids are heaviest first;
// item id covers query tile n_qtiles - 1 - id / n_groups, i.e. that many 64-key tiles plus item_cost half tiles
// for its loads and epilogue; the deal at the training shapes is the same for costs from 1 to 8) go, longest first, to the list with the least work; then the lists are handed out by
// falling work, so that block i (one of the first n_SMs blocks) and block i + n_SMs, which share an SM, get a
// heavy and a light list.  Returns a table with per_cta == 0 when the deal does not fit the table (the kernel
// then uses the closed formula) or when B200ATTN_ITEMS=static asks for the formula.
const ItemTable& item_table_for(long long n_items, unsigned n_ctas, int n_groups, int n_qtiles, int T, int item_cost) {
    static const ItemTable none = [] {
        ItemTable t;
        t.per_cta = 0;
        return t;
    }();
    static const bool formula = [] {
        const char* e = getenv("B200ATTN_ITEMS");
        return e && e[0] == 's';
    }();
    if (formula || n_ctas > (unsigned)kItemTableCtas || n_items >= 0xffff || n_items < (long long)n_ctas) return none;
    struct Entry {
        long long n_items = -1;
        unsigned n_ctas = 0;
        int n_groups = 0, n_qtiles = 0, T = 0, cost = 0;
        ItemTable tab;
    };
    thread_local Entry cache[4];
    thread_local unsigned next = 0;
    for (Entry& e : cache)
        if (e.n_items == n_items && e.n_ctas == n_ctas && e.n_groups == n_groups && e.n_qtiles == n_qtiles && e.T == T &&
            e.cost == item_cost)
            return e.tab.per_cta >= 0 ? e.tab : none;
    Entry& e = cache[next++ % 4];
    e.n_items = n_items, e.n_ctas = n_ctas, e.n_groups = n_groups, e.n_qtiles = n_qtiles, e.T = T, e.cost = item_cost;
    // longest processing time first; work in half tiles: an item costs its tiles plus half a tile.  (Fixed arrays: this runs
    // under C entry points, which never throw.)
    struct List {  // on the heap: least work first, then lowest index
        long long work;
        unsigned index;
        bool operator>(const List& o) const { return work != o.work ? work > o.work : index > o.index; }
    };
    List heap[kItemTableCtas];
    unsigned short ids[kItemTableCtas][kItemTableMaxPerCta];
    int count[kItemTableCtas] = {}, longest = 0;
    for (unsigned c = 0; c < n_ctas; ++c) heap[c] = {0, c};
    for (long long id = 0; id < n_items; ++id) {
        const int qt = n_qtiles - 1 - (int)(id / n_groups);
        const int rows = std::min(T, qt * 128 + 128);
        std::pop_heap(heap, heap + n_ctas, std::greater<List>());
        List& l = heap[n_ctas - 1];
        if (count[l.index] == kItemTableMaxPerCta) {
            e.tab.per_cta = -1;  // remembered as "no table"
            return none;
        }
        ids[l.index][count[l.index]++] = (unsigned short)id;
        longest = std::max(longest, count[l.index]);
        l.work += 2 * ((rows + 63) / 64) + item_cost;
        std::push_heap(heap, heap + n_ctas, std::greater<List>());
    }
    std::sort(heap, heap + n_ctas, [](const List& a, const List& b) { return a.work != b.work ? a.work > b.work : a.index < b.index; });
    e.tab.per_cta = longest;
    for (unsigned c = 0; c < n_ctas; ++c)
        for (int n = 0; n < longest; ++n)
            e.tab.ids[c * longest + n] = n < count[heap[c].index] ? ids[heap[c].index][n] : kItemTableEnd;
    return e.tab;
}

// SM count of the current device (cached per device).
int sm_count() {
    static int cached[kMaxDevices] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return cached[dev];
}

struct Strides {
    long long t, h, b;  // element strides
};

inline Strides strides_for(int layout, int H, int T, int D) {
    Strides s;
    if (layout == B200ATTN_LAYOUT_BHTD) {
        s.t = D;
        s.h = (long long)T * D;
        s.b = (long long)H * T * D;
    } else {
        s.t = (long long)H * D;
        s.h = D;
        s.b = (long long)T * H * D;
    }
    return s;
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int check_common(int B, int T, int Hq, int Hkv, int D, int layout) {
    if (B <= 0 || T <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0) return B200ATTN_ERR_INVALID_ARG;
    if (Hq % Hkv != 0) return B200ATTN_ERR_INVALID_ARG;
    if (layout != B200ATTN_LAYOUT_BHTD && layout != B200ATTN_LAYOUT_BTHD) return B200ATTN_ERR_INVALID_ARG;
    if (D != 64 && D != 128) return B200ATTN_ERR_UNSUPPORTED;
    return B200ATTN_OK;
}

// Launch with programmatic stream serialization: the kernel may become resident while the
// previous kernel of the stream drains; it calls griddepcontrol.wait before touching global memory.
// cluster > 1: in thread-block clusters of that many blocks.
template <typename... KArgs, typename... Args>
cudaError_t launch_cluster(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, int cluster,
                           Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, Args&&... args) {
    return launch_cluster(kernel, grid, block, smem, st, 1, args...);
}

template <typename K>
int set_smem_once(K kernel, int bytes, bool* done) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (!done[dev]) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
            cudaGetLastError();
            return B200ATTN_ERR_CUDA;
        }
        done[dev] = true;
    }
    return B200ATTN_OK;
}

// The SMs that clusters can have: those of four and eight do not fill the last SMs of a GPC and get 132 and 120 of 148.
double cluster_slots(int cluster) { return sm_count() * (cluster <= 2 ? 1.0 : cluster <= 4 ? 0.892 : 0.811); }

// Early launch of the next kernel (`early`): a kernel whose CTAs have one item each lets the next one start once their last loads are
// issued, which hides the 1.3 us from the last CTA's end to the next kernel's first instruction.  The next kernel's CTAs then go to
// whatever SMs are free, so kernels with room for two CTAs on an SM and no more CTAs than SMs ask for more shared memory than half
// an SM has (spread_smem): without that they came to lie in pairs (forward and backward, us, released at the end / early / early and
// spread: B=1 T=1500 8/8 D=64 49.4 / 51.1 / 47.4, B=8 T=128 16/4 D=128 23.0 / 23.3 / 21.8).  Both together: B=2 T=128 6/2 D=64 14.1 ->
// 13.1, B=11 15.3 -> 14.1, B=36 19.7 -> 18.6, B=2 T=700 8/2 35.7 -> 33.6, D=128 B=1 T=500 6/2 35.3 -> 33.2, B=8 T=512 6/2 45.5 -> 43.7,
// B=32 T=1001 1/1 60.5 -> 58.8.
// Not early: kernels with several items per CTA (the next kernel's CTAs, dealt their work in pairs per SM, then share SMs as it happens:
// forward of B=32 T=512 6/2 D=64 18.3 -> 18.7), clusters beyond one CTA per SM (forward of B=1 T=2000 4/4 D=128 18.0 -> 20.7), a dK/dV
// pass whose forward has more CTAs than SMs (B=3 T=2000 6/2 D=64 83.3 -> 86.0; also with other kernels behind, below), the tile kernel by head in
// clusters on more than half the SMs (B=14 T=128 6/2 D=128 20.5 -> 21.2), by group on more than half the SMs or at D = 128 (T=128 6/2, released at
// the end / early, forward and backward; RoPE + QK-Norm, forward, backward and back: B=27 T=100 18.0 / 17.2; 28.1 / 28.25, B=36 19.5 / 19.1; 31.6 /
// 31.85, B=48 20.15 / 19.95; 33.9 / 34.9, B=60 22.0 / 22.8; 37.7 / 37.9, D=128 B=36 30.1 / 30.75; 46.6 / 46.7, B=60 34.6 / 36.0; 58.0 / 59.2), and a forward at D = 64 of more than three query tiles and more CTAs than SMs, whose dQ pass shares SMs in
// pairs of a heavy and a light CTA (B=8 T=512 6/2 34.5 -> 35.3, B=5 T=500 10/10 31.2 -> 32.0; of three, B=16 T=300 6/2, 33.8 -> 32.7).
// For the release of the dK/dV pass and of the tile kernel by head it matters what follows: with attention behind it gains up to 2 %, with the RoPE +
// QK-Norm backward behind it costs up to 2 % (spreading that kernel over the SMs, too, does not help), a matrix product of a library waits
// for the end anyway.  us, released at the end / early, forward and backward; RoPE + QK-Norm, forward, backward and back; backwards in a row:
//   B=2 T=700 8/2 35.2 / 34.9; 43.15 / 43.2; 24.9 / 24.5      B=8 T=300 6/2 28.3 / 28.1; 37.4 / 38.05; 20.2 / 19.8
//   B=1 T=500 6/2 D=128 34.5 / 34.4; 41.5 / 41.8; 24.9 / 24.4  B=2 T=128 6/2 14.1 / 13.9; 19.8 / 20.0; 9.6 / 9.5
//   and where the rule says no: B=3 T=2000 6/2 82.8 / 86.5; 97.3 / 98.1; 59.1 / 64.5   B=8 T=512 6/2 34.5 / 35.3; 46.0 / 47.1; 23.9 / 26.3
// The forward's release, with the backward behind, alone and in that chain: B=32 T=1001 1/1 D=128 60.6 / 58.6; 92.7 / 87.6, B=2 T=700 8/2 35.5 / 34.8;
// 43.0 / 42.8; with the RoPE + QK-Norm forward of another call behind it costs 0.1 to 0.5 us (B=8 T=300 6/2 10.7 / 11.2).
constexpr int kAloneSmemBytes = 114 * 1024;
inline size_t spread_smem(int bytes, bool one_per_sm) { return one_per_sm ? std::max(bytes, kAloneSmemBytes) : bytes; }

// How many CTAs of a cluster share an item (forward: its key tiles, dK/dV pass: its units): the number with the smallest
// estimate of the kernel's time, 1 unless another one is at least 5 % better.  Not only few items are split: 126 items of
// 126 to 2 units on 148 SMs are bound by the longest one (dK/dV at B=1 T=8000 4/2 D=128: 229 -> 134 us).  Held against every
// number of shares at forty shapes from 2 to 2048 items, 15 to 8000 tokens, the pick was the fastest at each; some of them, us
// for 1 / 2 / 4 / 8 shares: forward B=2 T=128 6/2 D=64 5.4 / 8.2 / 8.2 / 8.7, B=1 T=2000 6/2 D=64 22.5 / 18.2 / 23.9 / 36.6, 15 tokens
// behind 6000 6/2 D=64 57.4 / 35.1 / 21.3 / 14.7, 500 behind 3000 B=2 16/4 D=128 43.6 / 36.2 / 50.6 / 86.5; dQ pass and dK/dV pass
// B=1 T=2000 6/2 D=64 78.0 / 56.3 / 43.8 / 58.3, B=8 T=512 6/2 D=64 26.8 / 23.7 / 32.7 / 62.9, B=1 T=4096 8/2 D=128 264 / 162 / 121 /
// 167, B=32 T=1001 1/1 D=128 44.2 / 77.9 / 136 / 262.  The costs of the forward and of the dK/dV pass at D=128 are those of the kernels with one
// S buffer and copies by tcgen05.cp, fitted at 32 shapes with every number of shares and 95 whose pick they change; with the costs of the
// kernels before, us: forward B=1 T=3870 6/2 D=64 37.7 instead of 28.6, T=5151 2/1 28.7 instead of 22.6, B=2 T=512 8/1 8.7 instead of 7.5, B=2 T=906 6/2
// D=128 14.9 instead of 13.2; both passes of the backward B=5 T=4257 2/1 D=128 181 instead of 163.  The order of the estimates is what counts: they are within some 12 % of the
// time in one round of items, and up to half too low where shared items run in many rounds.  They do not see how items of
// different lengths pack.
struct SplitCosts {
    int per_sm;                // CTAs of the kernel that fit an SM
    float tile_one, tile_all;  // us per tile in a CTA that has the SM to itself, and with a second CTA beside it
    float exchange, start;     // us: the exchange in a cluster of two, a CTA's start
};
int pick_split(long long items, int longest, double total, const SplitCosts& c, int most = 8) {
    const int sms = sm_count();
    int best = 1;
    double best_us = 1e30;
    for (int split = 1; split <= most; split *= 2) {
        const double slots = c.per_sm * cluster_slots(split), ctas = (double)items * split;
        const double shared = c.per_sm > 1 ? std::min(1.0, std::max(0.0, ctas / sms - 1)) : 0.0;  // SMs with two CTAs
        const double share = (longest + split - 1) / split * (c.tile_one + (c.tile_all - c.tile_one) * shared);
        const double all = total * c.tile_all / slots;
        // in one round the longest share decides; in several the work, and what the last CTAs leave uneven
        double us = split == 1 ? std::max(share, all) + c.start : (ctas <= slots ? share : all + 0.5 * share) + c.start * ceil(ctas / slots);
        if (split > 1) us += c.exchange * (1 + shared) + (split == 4 ? 1.5 : split == 8 ? 4.0 : 0.0);
        if (split == 1 || us < 0.95 * best_us) best = split, best_us = us;
        if (ctas >= 4 * slots) break;
    }
    return best;
}
// tiles of all items of a causal problem: query tiles of 128 rows behind kv_off keys, key tiles of `keys`
double fwd_total_tiles(int n_qtiles, int kv_off, int T, int keys) {
    const double last = (kv_off + T + keys - 1) / keys, first = (kv_off + std::min(T, 128) + keys - 1) / keys;
    return n_qtiles * (first + last) / 2;
}

// CTAs (a cluster) that share an item of the forward
template <int D>
int fwd_split(int B, int Hq, int T, int kv_off, int n_qtiles) {
    constexpr int keys = FwdCfg<D>::kKeys;
    constexpr SplitCosts kCosts = D == 64 ? SplitCosts{2, 1.35f, 1.6f, 2.8f, 3.5f} : SplitCosts{2, 0.9f, 1.05f, 4.f, 3.5f};
    return pick_split((long long)n_qtiles * Hq * B, (kv_off + T + keys - 1) / keys, (double)B * Hq * fwd_total_tiles(n_qtiles, kv_off, T, keys), kCosts);
}

template <int D>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdParams& p,
               cudaStream_t st) {
    using Cfg = FwdCfg<D>;
    const long long items = (long long)p.n_qtiles * p.Hq * p.B;
    FwdParams pl = p;
    pl.div_bh = fastdiv_make((unsigned)(p.B * p.Hq));
    pl.div_h = fastdiv_make((unsigned)p.Hq);
    pl.div_group = fastdiv_make((unsigned)p.group);
    pl.split = fwd_split<D>(p.B, p.Hq, p.T, p.kv_off, p.n_qtiles);
    pl.div_split = fastdiv_make((unsigned)pl.split);
    cudaError_t e;
    if (pl.split > 1) {
        static bool set[kMaxDevices] = {false};
        if (int rc = set_smem_once(attn_fwd_kernel<D, true>, std::max(Cfg::kSmemBytes, kAloneSmemBytes), set)) return rc;
        pl.sched = nullptr;
        pl.early = items * pl.split <= cluster_slots(pl.split);
        e = launch_cluster(attn_fwd_kernel<D, true>, dim3((unsigned)(items * pl.split)), 256, spread_smem(Cfg::kSmemBytes, pl.early), st, pl.split, tq, tk, tv, pl,
                           item_table_for(-1, 1, 1, 1, 1, 1));
    } else {
        static bool set[kMaxDevices] = {false};
        if (int rc = set_smem_once(attn_fwd_kernel<D, false>, std::max(Cfg::kSmemBytes, kAloneSmemBytes), set)) return rc;
        // persistent CTAs, two per SM, each walking a heaviest-first list of (query tile, head, batch) items
        const unsigned grid = (unsigned)std::min<long long>(items, 2LL * sm_count());
        pl.sched = next_sched_pair(items, grid);
        pl.early = items <= sm_count() || (items <= grid && (D == 128 || p.n_qtiles <= 3));
        const ItemTable& tab = item_table_for(pl.sched ? -1 : items, grid, p.B * p.Hq, p.n_qtiles, p.T, 1);
        e = launch_pdl(attn_fwd_kernel<D, false>, grid, 256, spread_smem(Cfg::kSmemBytes, grid <= (unsigned)sm_count()), st, tq, tk, tv, pl, tab);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    return B200ATTN_OK;
}

}  // namespace

namespace {

// The forward with K and V at their own strides (sk): the training call passes the strides of `layout`, the
// prefill over a KV cache those of the cache.
int fwd_run(const void* q, const void* k, const void* v, void* o, float* lse, int B, int T, int kv_off, int Hq, int Hkv, int D,
            int layout, const Strides& sk, float softmax_scale, void* stream) {
    int rc = check_common(B, T, Hq, Hkv, D, layout);
    if (rc) return rc;
    if (!q || !k || !v || !o || !lse) return B200ATTN_ERR_INVALID_ARG;
    if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o)) return B200ATTN_ERR_ALIGNMENT;
    int* status = status_ptr(&rc);
    if (!status) return rc;
    const Strides sq = strides_for(layout, Hq, T, D);
    const int keys = D == 64 ? FwdCfg<64>::kKeys : FwdCfg<128>::kKeys;
    CUtensorMap tq, tk, tv;
    if (!make_tmap_bf16_4d(&tq, q, D, T, Hq, B, sq.t, sq.h, sq.b, 128) ||
        !make_tmap_bf16_4d(&tk, k, D, kv_off + T, Hkv, B, sk.t, sk.h, sk.b, keys) ||
        !make_tmap_bf16_4d(&tv, v, D, kv_off + T, Hkv, B, sk.t, sk.h, sk.b, keys))
        return B200ATTN_ERR_TENSOR_MAP;
    FwdParams p;
    p.B = B;
    p.T = T;
    p.Hq = Hq;
    p.Hkv = Hkv;
    p.group = Hq / Hkv;
    p.n_qtiles = (T + 127) / 128;
    p.kv_off = kv_off;
    p.scale = softmax_scale > 0.f ? softmax_scale : 1.f / sqrtf((float)D);
    p.scale_log2 = p.scale * 1.4426950408889634f;
    p.lse = lse;
    p.o = static_cast<uint16_t*>(o);
    p.o_st = sq.t;
    p.o_sh = sq.h;
    p.o_sb = sq.b;
    p.status = status;
    p.sched = nullptr;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return D == 64 ? launch_fwd<64>(tq, tk, tv, p, st) : launch_fwd<128>(tq, tk, tv, p, st);
}

}  // namespace

extern "C" int b200attn_fwd(const void* q, const void* k, const void* v, void* o, float* lse, int B, int T, int Hq,
                            int Hkv, int D, int layout, float softmax_scale, void* stream) {
    if (T <= 0 || Hkv <= 0 || D <= 0) return B200ATTN_ERR_INVALID_ARG;
    return fwd_run(q, k, v, o, lse, B, T, 0, Hq, Hkv, D, layout, strides_for(layout, Hkv, T, D), softmax_scale, stream);
}

extern "C" int b200attn_fwd_kvcache(const void* q, const void* kcache, const void* vcache, void* o, float* lse, int B,
                                    int T, int L_cap, int Hq, int Hkv, int D, int q_layout, float softmax_scale,
                                    void* stream) {
    return b200attn_fwd_kvcache_at(q, kcache, vcache, o, lse, B, T, 0, L_cap, Hq, Hkv, D, q_layout, softmax_scale, stream);
}

extern "C" int b200attn_fwd_kvcache_at(const void* q, const void* kcache, const void* vcache, void* o, float* lse, int B,
                                       int T, int pos0, int L_cap, int Hq, int Hkv, int D, int q_layout,
                                       float softmax_scale, void* stream) {
    if (T <= 0 || pos0 < 0 || Hkv <= 0 || D <= 0 || (long long)pos0 + T > L_cap) return B200ATTN_ERR_INVALID_ARG;
    return fwd_run(q, kcache, vcache, o, lse, B, T, pos0, Hq, Hkv, D, q_layout,
                   strides_for(B200ATTN_LAYOUT_BHTD, Hkv, L_cap, D), softmax_scale, stream);
}

namespace {

inline size_t bwd_vec_elems(int B, int T, int Hq) { return (size_t)B * Hq * (size_t)((T + 127) / 128 * 128); }

cudaEvent_t g_bwd_events[4] = {nullptr, nullptr, nullptr, nullptr};

inline void record_bwd_event(int i, cudaStream_t st) {
    if (g_bwd_events[i]) cudaEventRecord(g_bwd_events[i], st);
}

// Which backward runs.  The one-pass kernel (attn_bwd_onepass.cuh) exists for D = 64; it needs the FP32 dQ
// accumulator behind the two row vectors in the workspace.  AUTO is the two-pass backward: measured on B200 the
// one-pass kernel moves as many bytes through shared memory per block of scores as the two passes together (the
// limiter of every D = 64 kernel here) and pays two HBM-bound kernels around it, so it only draws level from
// T = 4096 on.  The environment variable B200ATTN_BWD=two_pass|one_pass overrides AUTO.
inline size_t bwd_acc_bytes(int B, int T, int Hq, int D) { return bwd_vec_elems(B, T, Hq) * (size_t)D * sizeof(float); }
inline size_t bwd_vec_bytes_padded(int B, int T, int Hq) { return (2 * bwd_vec_elems(B, T, Hq) * sizeof(float) + 255) & ~(size_t)255; }

int bwd_forced_mode() {
    static const int forced = [] {
        const char* e = getenv("B200ATTN_BWD");
        return !e ? 0 : (e[0] == 't' ? B200ATTN_BWD_TWO_PASS : (e[0] == 'o' ? B200ATTN_BWD_ONE_PASS : 0));
    }();
    return forced;
}
int bwd_resolve_mode(int mode, int B, int T, int Hq, int D) {
    const int forced = bwd_forced_mode();
    if (mode == B200ATTN_BWD_AUTO) {
        mode = forced ? forced : B200ATTN_BWD_TWO_PASS;
        if (D != 64) mode = B200ATTN_BWD_TWO_PASS;
        (void)B, (void)T, (void)Hq;
    }
    return mode;
}

// Whether AUTO takes the kernel for sequences of one tile (attn_bwd_tile.cuh): a CTA per query head, the group's CTAs in a
// cluster, or a CTA per key/value head that goes through its group.  Measured at T = 128, us, two passes / group / head:
//   heads without a group, always by head: 20 10.3 / 6.3 / 5.4, 300 21.2 / 20.5 / 18.5, 1500 75 / 72 / 65; D=128 1500 123 / 128 / 113
//   by head while the clusters run in one round: 40 x 2 (B x group) 11.7 / 9.3 / 9.1, 20 x 4 13.9 / 15.0 / 10.0, 12 x 8 16.0 / 26.5 /
//     10.8, D=128 30 x 2 14.7 / 14.8 / 12.9, 12 x 8 21.7 / 46 / 16; in two rounds no longer: 37 x 4 15.2 / 15.2 / 19.3, D=128 20.9 / 26 / 30
//   by group from a tenth of the SMs per head of the group on (fewer CTAs are slower than the two passes' many: 40 x 8 21.3 / 27.3, D=128
//     38 / 49): 120 x 2 15.8 / 10.5, 60 x 3 14.3 / 12.3, 100 x 4 19.8 / 17.1, 148 x 8 33.5 / 30.7; D=128 120 x 2 23.6 / 19.7, 100 x 4
//     33.3 / 29.8, 444 x 4 117 / 91, 300 x 8 162 / 151; at D=64 in one round only: 444 x 4 48.6 / 51.0, 300 x 8 66 / 83
enum BwdTile { kTileNo, kTileGroup, kTileHead };
BwdTile bwd_tile(int B, int T, int Hq, int Hkv, int D) {
    if (T > 128) return kTileNo;
    const int sms = sm_count(), group = Hq / Hkv;
    const long long items = (long long)B * Hkv, heads = (long long)B * Hq;
    if (group == 1) return kTileHead;
    // (clusters of three and more do not fill the last SMs of a GPC)
    if (group <= BwdTileCfg<64>::kMaxCluster && heads <= sms * (group == 2 ? 1.0 : group <= 4 ? 0.89 : 0.81)) return kTileHead;
    return items * 10 >= (long long)group * sms && (D == 128 || items <= sms) ? kTileGroup : kTileNo;
}

// One-pass backward (D = 64): row vectors + cleared accumulator, the fused kernel, accumulator -> dq.
int launch_bwd_onepass(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                       const BwdParams& p, float* dq_acc, cudaStream_t st) {
    static bool set[kMaxDevices] = {false};
    int rc = set_smem_once(attn_bwd_onepass_kernel, OnePassCfg::kSmemBytes, set);
    if (rc) return rc;
    record_bwd_event(0, st);
    const unsigned q_tiles = (unsigned)(p.n_tiles * p.Hq * p.B);
    if (launch_pdl(attn_bwd_prep_kernel<64>, q_tiles, 256, 0, st, p, dq_acc) != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    record_bwd_event(1, st);
    const unsigned kv_items = (unsigned)(p.n_tiles * p.Hkv * p.B);
    const unsigned kv_grid = std::min(kv_items, (unsigned)sm_count());
    BwdParams pk = p;
    pk.sched2 = next_sched_pair(kv_items, kv_grid);
    if (launch_pdl(attn_bwd_onepass_kernel, kv_grid, OnePassCfg::kThreads, OnePassCfg::kSmemBytes, st, tk, tv, tq, tdo, pk,
                   dq_acc) != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    record_bwd_event(2, st);
    const float* acc_c = dq_acc;
    if (launch_pdl(attn_bwd_dq_convert_kernel<64>, q_tiles, 128, 0, st, p, acc_c) != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    record_bwd_event(3, st);
    return B200ATTN_OK;
}

// Sequences of one tile: one launch (attn_bwd_tile.cuh).
template <int D, bool ONE>
int launch_bwd_tile(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const BwdParams& p,
                    cudaStream_t st) {
    using Cfg = BwdTileCfg<D>;
    static bool set[kMaxDevices] = {false};
    if (int rc = set_smem_once(attn_bwd_tile_kernel<D, ONE>, Cfg::kSmemBytes, set)) return rc;
    record_bwd_event(0, st);
    const int ctas = p.B * (ONE ? p.Hq : p.Hkv);
    BwdParams pt = p;
    pt.early = (ONE && p.group == 1) || ((ONE || D == 64) && 2 * ctas <= sm_count());
    const cudaError_t e = launch_cluster(attn_bwd_tile_kernel<D, ONE>, dim3((unsigned)ctas), Cfg::kThreads, Cfg::kSmemBytes, st, ONE ? p.group : 1,
                                         tk, tv, tq, tdo, pt);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    record_bwd_event(1, st);
    record_bwd_event(2, st);
    return B200ATTN_OK;
}

// own: what the dQ pass at D = 64 alone reads through TMA: K and V in boxes of 64 rows, and O.
template <int D>
int launch_bwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap (&own)[3],
               const BwdParams& p, cudaStream_t st) {
    static bool dq_set[kMaxDevices] = {false}, dq_split_set[kMaxDevices] = {false}, dkdv_set[kMaxDevices] = {false};
    // D = 64: 64-key tiles.  D = 128: 128-key tiles (tensor-pipe bound).
    constexpr bool kWide = (D == 128);
    int rc;
    rc = set_smem_once(attn_bwd_dkdv_kernel<D, false>, BwdCfg<D>::kSmemBytes, dkdv_set);
    if (rc) return rc;
    record_bwd_event(0, st);
    // the dQ pass also writes the two per-row vectors the dK/dV pass reads
    const unsigned dq_items = (unsigned)(p.n_tiles * p.Hq * p.B);
    cudaError_t e;
    // It is persistent: two CTAs per SM at D = 64, one at D = 128, walk the item list.
    const unsigned dq_grid = std::min(dq_items, (kWide ? 1u : 2u) * (unsigned)sm_count());
    BwdParams pq = p;
    // Few, long items are shared by clusters (both passes of the backward, us for 1 / 2 / 4 / 8 CTAs of the dQ pass: B=1 T=4000 2/1 D=64 61.3 / 51.0 /
    // 44.1 / 52.2, D=128 76.9 / 65.2 / 68.4 / 102; T=2000 6/2 D=64 41.7 / 37.9 / 43.1 / 54.3, D=128 54.1 / 56.0 / 70.1 / 115; T=1000 8/8 D=64 23.4 / 22.6 /
    // 24.1 / 33.1; T=500 6/2 D=64 18.6 / 19.0 / 18.4 / 19.9, B=2 T=700 8/2 D=64 23.9 / 26.0 / 31.9 / 44.3).  Four at most: the costs
    // never ask for eight (1 to 296 heads of up to 38400 tokens), which was the slowest wherever it was measured but at T=4000 D=64.
    constexpr SplitCosts kDqCosts = D == 64 ? SplitCosts{2, 0.43f, 0.6f, 2.f, 4.f} : SplitCosts{1, 1.06f, 1.06f, 5.6f, 4.f};
    constexpr int kDqKeys = D == 64 ? 64 : 128;
    pq.split = pick_split(dq_items, (p.T + kDqKeys - 1) / kDqKeys, (double)p.B * p.Hq * fwd_total_tiles(p.n_tiles, 0, p.T, kDqKeys), kDqCosts, 4);
    pq.div_split = fastdiv_make((unsigned)pq.split);
    pq.sched = pq.split > 1 ? nullptr : next_sched_pair(dq_items, dq_grid);
    // (no table where every CTA has one item: one line of constants less in front of its first load)
    const ItemTable& tab = item_table_for(pq.split > 1 || pq.sched || dq_items <= dq_grid ? -1 : (long long)dq_items, dq_grid, p.B * p.Hq, p.n_tiles, p.T, 4);
    auto launch_dq = [&](auto kernel, bool* set, int bytes, int threads, bool one_per_sm, auto&&... maps) {
        if ((rc = set_smem_once(kernel, std::max(bytes, kAloneSmemBytes), set))) return cudaErrorInvalidValue;
        return launch_cluster(kernel, dim3(pq.split > 1 ? dq_items * (unsigned)pq.split : dq_grid), threads, spread_smem(bytes, one_per_sm), st, pq.split,
                              maps..., pq, tab);
    };
    const bool dq_spread = pq.split > 1 ? (double)dq_items * pq.split <= cluster_slots(pq.split) : dq_grid <= (unsigned)sm_count();
    if constexpr (kWide) {
        using Cfg = DqWideCfg<D>;
        e = pq.split > 1 ? launch_dq(attn_bwd_dq_wide_kernel<D, true>, dq_split_set, Cfg::kSmemBytes, Cfg::kThreads, false, tq, tk, tv, tdo)
                         : launch_dq(attn_bwd_dq_wide_kernel<D, false>, dq_set, Cfg::kSmemBytes, Cfg::kThreads, false, tq, tk, tv, tdo);
    } else {
        using Cfg = DqCfg<D>;
        e = pq.split > 1 ? launch_dq(attn_bwd_dq_kernel<D, true>, dq_split_set, Cfg::kSmemBytes, Cfg::kThreads, dq_spread, tq, own[0], own[1], tdo, own[2])
                         : launch_dq(attn_bwd_dq_kernel<D, false>, dq_set, Cfg::kSmemBytes, Cfg::kThreads, dq_spread, tq, own[0], own[1], tdo, own[2]);
    }
    if (rc) return rc;
    if (e != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    record_bwd_event(1, st);
    // the dK/dV pass is persistent too: one CTA per SM walks the list of (key tile, KV head, batch) items
    const unsigned kv_items = (unsigned)(p.n_tiles * p.Hkv * p.B);
    BwdParams pk = p;
    // (the exchange is 64 KB in and out of every CTA at D = 128, at the 13 bytes a clock of distributed shared memory)
    constexpr SplitCosts kCosts = D == 64 ? SplitCosts{1, 1.4f, 1.4f, 3.f, 3.5f} : SplitCosts{1, 1.8f, 1.8f, 5.6f, 3.5f};
    pk.split = pick_split(kv_items, p.group * p.n_tiles, (double)p.B * p.Hq * p.n_tiles * (p.n_tiles + 1) / 2, kCosts);
    pk.div_split = fastdiv_make((unsigned)pk.split);
    const int fs = fwd_split<D>(p.B, p.Hq, p.T, 0, p.n_tiles);
    pk.early = (pk.split > 1 || kv_items <= (unsigned)sm_count()) && (long long)dq_items * fs <= cluster_slots(fs);
    if (pk.split > 1) {
        static bool set[kMaxDevices] = {false};
        if ((rc = set_smem_once(attn_bwd_dkdv_kernel<D, true>, BwdCfg<D>::kSmemBytes, set))) return rc;
        e = launch_cluster(attn_bwd_dkdv_kernel<D, true>, dim3(kv_items * (unsigned)pk.split), BwdCfg<D>::kThreads, BwdCfg<D>::kSmemBytes, st,
                           pk.split, tk, tv, tq, tdo, pk);
    } else {
        const unsigned kv_grid = std::min(kv_items, (unsigned)sm_count());
        pk.sched2 = next_sched_pair(kv_items, kv_grid);
        e = launch_pdl(attn_bwd_dkdv_kernel<D, false>, kv_grid, BwdCfg<D>::kThreads, BwdCfg<D>::kSmemBytes, st, tk, tv, tq, tdo, pk);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    record_bwd_event(2, st);
    return B200ATTN_OK;
}

}  // namespace

// ---------------------------------------------------------------------------------------
// Fused RoPE + QK-Norm (rope_norm.cuh)
// ---------------------------------------------------------------------------------------
namespace {

constexpr int kRopeNormMaxCtasPerSm = 8;  // of the backward, as far as its workspace goes
static_assert(kRopeNormBwdBlocks <= kRopeNormMaxCtasPerSm, "a partial sum per CTA");

int rope_norm_check(int B, int T, int H, int D, int x_dtype, int x_layout, int y_layout) {
    if (B <= 0 || T <= 0 || H <= 0 || D <= 0) return B200ATTN_ERR_INVALID_ARG;
    if (x_dtype != B200ATTN_DTYPE_BF16 && x_dtype != B200ATTN_DTYPE_F32) return B200ATTN_ERR_INVALID_ARG;
    for (int l : {x_layout, y_layout})
        if (l != B200ATTN_LAYOUT_BHTD && l != B200ATTN_LAYOUT_BTHD) return B200ATTN_ERR_INVALID_ARG;
    if (D != 64 && D != 128) return B200ATTN_ERR_UNSUPPORTED;
    if ((long long)B * T * H >= (1LL << 31)) return B200ATTN_ERR_TOO_LARGE;  // rows are counted in 32 bits
    return B200ATTN_OK;
}

// Heads per item: eight of them share a token's cosines and sines and addresses, fewer when that leaves less than four items
// for a resident warp (one eighth of a wave is then the most that the last round can waste).
void rope_norm_plan(RopeNormParams* p, int n_tensors, int D, unsigned warps) {
    int chunk = 8;
    auto items = [&](const RopeNormParams& q) { return (long long)((q.n_tokens + 256u / D - 1) / (256u / D)) * ((q.H + chunk - 1) / chunk); };
    auto all = [&] { return items(p[0]) + (n_tensors > 1 ? items(p[1]) : 0); };
    while (chunk > 1 && all() < (chunk > 4 ? 4LL : 1LL) * warps) chunk /= 2;
    for (int i = 0; i < n_tensors; ++i) {
        p[i].chunk = chunk;
        p[i].n_items = (unsigned)items(p[i]);
        p[i].div_chunks = fastdiv_make((unsigned)((p[i].H + chunk - 1) / chunk));
    }
}

// CTAs that the device keeps resident at once, never more than the items need
inline unsigned rope_norm_grid(const RopeNormParams* p, int n_tensors, int blocks) {
    const long long items = (long long)p[0].n_items + (n_tensors > 1 ? p[1].n_items : 0);
    const long long need = (items + kRopeNormThreads / 32 - 1) / (kRopeNormThreads / 32);
    return (unsigned)std::min<long long>(need, (long long)blocks * sm_count());
}

template <int D, bool F32>
void rope_norm_launch_fwd(RopeNormParams* p, int n_tensors, cudaStream_t st) {
    rope_norm_plan(p, n_tensors, D, (unsigned)(kRopeNormFwdBlocks * (kRopeNormThreads / 32) * sm_count()));
    launch_pdl(rope_norm_fwd_kernel<D, F32>, dim3(rope_norm_grid(p, n_tensors, kRopeNormFwdBlocks)), kRopeNormThreads, 0, st, p[0], p[1], n_tensors);
}
template <int D, bool F32>
void rope_norm_launch_bwd(RopeNormParams* p, int n_tensors, float* workspace, cudaStream_t st) {
    rope_norm_plan(p, n_tensors, D, (unsigned)(kRopeNormBwdBlocks * (kRopeNormThreads / 32) * sm_count()));
    const unsigned grid = rope_norm_grid(p, n_tensors, kRopeNormBwdBlocks);
    p[0].partial = workspace;
    p[1].partial = workspace + (size_t)kRopeNormMaxCtasPerSm * sm_count() * D;
    launch_pdl(rope_norm_bwd_kernel<D, F32>, dim3(grid), kRopeNormThreads, 0, st, p[0], p[1], n_tensors);
    const float* part0 = p[0].partial;
    const float* part1 = p[1].partial;
    launch_pdl(rope_norm_dgamma_kernel<D>, dim3(n_tensors * (D / 8)), kDgammaThreads, 0, st, part0, p[0].d_gamma, part1,
               p[1].d_gamma, (int)grid);
}

void rope_norm_fill(RopeNormParams& p, int B, int T, int H, int D, int x_layout, int y_layout) {
    const Strides sx = strides_for(x_layout, H, T, D), sy = strides_for(y_layout, H, T, D);
    p.B = B;
    p.T = T;
    p.H = H;
    p.n_tokens = (unsigned)B * (unsigned)T;
    p.x_st = sx.t, p.x_sh = sx.h, p.x_sb = sx.b;
    p.y_st = sy.t, p.y_sh = sy.h, p.y_sb = sy.b;
    p.div_t = fastdiv_make((unsigned)T);
}

struct RopeNormTensor {  // what differs between q and k
    const void* x;
    void* y;            // forward: y; backward: d_x
    const void* dy;     // backward only
    float* rstd;
    const float* gamma;
    float* d_gamma;     // backward only
    int H;
};

int rope_norm_run(bool backward, const RopeNormTensor* t, int n_tensors, int x_dtype, int x_layout, int y_layout,
                  const float* cos_t, const float* sin_t, int B, int T, int D, float eps, void* workspace,
                  size_t workspace_bytes, void* stream) {
    RopeNormParams p[2] = {};
    for (int i = 0; i < n_tensors; ++i) {
        int rc = rope_norm_check(B, T, t[i].H, D, x_dtype, x_layout, y_layout);
        if (rc) return rc;
        if (!t[i].x || !t[i].y || !t[i].rstd || !t[i].gamma || (backward && (!t[i].dy || !t[i].d_gamma)))
            return B200ATTN_ERR_INVALID_ARG;
        if (!aligned16(t[i].x) || !aligned16(t[i].y) || (backward && !aligned16(t[i].dy))) return B200ATTN_ERR_ALIGNMENT;
        rope_norm_fill(p[i], B, T, t[i].H, D, x_layout, y_layout);
        p[i].x = t[i].x;
        p[i].y = t[i].y;
        p[i].dy = static_cast<const uint16_t*>(t[i].dy);
        p[i].rstd = t[i].rstd;
        p[i].gamma = t[i].gamma;
        p[i].d_gamma = t[i].d_gamma;
        p[i].cos_t = cos_t;
        p[i].sin_t = sin_t;
        p[i].eps = eps;
    }
    if (!cos_t || !sin_t) return B200ATTN_ERR_INVALID_ARG;
    if (backward && (!workspace || workspace_bytes < b200attn_rope_norm_bwd_workspace_bytes(D) ||
                     (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0))
        return B200ATTN_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool f32 = x_dtype == B200ATTN_DTYPE_F32;
    float* ws = static_cast<float*>(workspace);
    if (!backward) {
        if (D == 64) {
            if (f32) rope_norm_launch_fwd<64, true>(p, n_tensors, st);
            else rope_norm_launch_fwd<64, false>(p, n_tensors, st);
        } else {
            if (f32) rope_norm_launch_fwd<128, true>(p, n_tensors, st);
            else rope_norm_launch_fwd<128, false>(p, n_tensors, st);
        }
    } else {
        if (D == 64) {
            if (f32) rope_norm_launch_bwd<64, true>(p, n_tensors, ws, st);
            else rope_norm_launch_bwd<64, false>(p, n_tensors, ws, st);
        } else {
            if (f32) rope_norm_launch_bwd<128, true>(p, n_tensors, ws, st);
            else rope_norm_launch_bwd<128, false>(p, n_tensors, ws, st);
        }
    }
    if (cudaGetLastError() != cudaSuccess) return B200ATTN_ERR_CUDA;
    return B200ATTN_OK;
}

}  // namespace

extern "C" int b200attn_rope_table(int T, int D, float base, float* cos_host, float* sin_host) {
    if (T <= 0 || D <= 0 || (D & 1) || !cos_host || !sin_host || !(base > 0.f)) return B200ATTN_ERR_INVALID_ARG;
    const int half = D / 2;
    // the same single-precision arithmetic as make_rope_cache (llm/src/model/rope.cu:112-128)
    for (int t = 0; t < T; ++t)
        for (int i = 0; i < half; ++i) {
            const float theta = powf(base, -static_cast<float>(2 * i) / static_cast<float>(D));
            const float angle = static_cast<float>(t) * theta;
            cos_host[(size_t)t * half + i] = cosf(angle);
            sin_host[(size_t)t * half + i] = sinf(angle);
        }
    return B200ATTN_OK;
}

extern "C" size_t b200attn_rope_norm_bwd_workspace_bytes(int D) {
    if (D <= 0) return 0;
    return (size_t)2 * kRopeNormMaxCtasPerSm * sm_count() * D * sizeof(float);  // partial sums for up to two tensors
}

extern "C" int b200attn_rope_norm_fwd(const void* x, int x_dtype, int x_layout, void* y, int y_layout, float* rstd,
                                      const float* gamma, const float* cos_t, const float* sin_t, int B, int T, int H,
                                      int D, float eps, void* stream) {
    const RopeNormTensor t = {x, y, nullptr, rstd, gamma, nullptr, H};
    return rope_norm_run(false, &t, 1, x_dtype, x_layout, y_layout, cos_t, sin_t, B, T, D, eps, nullptr, 0, stream);
}

extern "C" int b200attn_rope_norm_bwd(const void* dy, int y_layout, const void* x, int x_dtype, int x_layout,
                                      const float* rstd, const float* gamma, const float* cos_t, const float* sin_t,
                                      void* dx, float* d_gamma, int B, int T, int H, int D, void* workspace,
                                      size_t workspace_bytes, void* stream) {
    const RopeNormTensor t = {x, dx, dy, const_cast<float*>(rstd), gamma, d_gamma, H};
    return rope_norm_run(true, &t, 1, x_dtype, x_layout, y_layout, cos_t, sin_t, B, T, D, 0.f, workspace, workspace_bytes,
                         stream);
}

extern "C" int b200attn_rope_norm_fwd_qk(const void* xq, const void* xk, int x_dtype, int x_layout, void* yq, void* yk,
                                         int y_layout, float* rstd_q, float* rstd_k, const float* gamma_q,
                                         const float* gamma_k, const float* cos_t, const float* sin_t, int B, int T,
                                         int Hq, int Hkv, int D, float eps, void* stream) {
    const RopeNormTensor t[2] = {{xq, yq, nullptr, rstd_q, gamma_q, nullptr, Hq}, {xk, yk, nullptr, rstd_k, gamma_k, nullptr, Hkv}};
    return rope_norm_run(false, t, 2, x_dtype, x_layout, y_layout, cos_t, sin_t, B, T, D, eps, nullptr, 0, stream);
}

extern "C" int b200attn_rope_norm_bwd_qk(const void* dyq, const void* dyk, int y_layout, const void* xq, const void* xk,
                                         int x_dtype, int x_layout, const float* rstd_q, const float* rstd_k,
                                         const float* gamma_q, const float* gamma_k, const float* cos_t,
                                         const float* sin_t, void* dxq, void* dxk, float* d_gamma_q, float* d_gamma_k,
                                         int B, int T, int Hq, int Hkv, int D, void* workspace, size_t workspace_bytes,
                                         void* stream) {
    const RopeNormTensor t[2] = {{xq, dxq, dyq, const_cast<float*>(rstd_q), gamma_q, d_gamma_q, Hq},
                                 {xk, dxk, dyk, const_cast<float*>(rstd_k), gamma_k, d_gamma_k, Hkv}};
    return rope_norm_run(true, t, 2, x_dtype, x_layout, y_layout, cos_t, sin_t, B, T, D, 0.f, workspace, workspace_bytes,
                         stream);
}

extern "C" int b200attn_set_bwd_profile_events4(void* e0, void* e1, void* e2, void* e3) {
    void* ev[4] = {e0, e1, e2, e3};
    const int n_set = (e0 != nullptr) + (e1 != nullptr) + (e2 != nullptr);
    if (n_set != 0 && n_set != 3) return B200ATTN_ERR_INVALID_ARG;
    if (n_set == 0 && e3 != nullptr) return B200ATTN_ERR_INVALID_ARG;
    for (int i = 0; i < 4; ++i) g_bwd_events[i] = static_cast<cudaEvent_t>(ev[i]);
    return B200ATTN_OK;
}

extern "C" int b200attn_set_bwd_profile_events(void* e0, void* e1, void* e2) {
    return b200attn_set_bwd_profile_events4(e0, e1, e2, nullptr);
}

extern "C" size_t b200attn_bwd_workspace_bytes_mode(int B, int T, int Hq, int Hkv, int D, int mode) {
    (void)Hkv;
    if (B <= 0 || T <= 0 || Hq <= 0 || D <= 0) return 0;
    if (mode != B200ATTN_BWD_AUTO && mode != B200ATTN_BWD_TWO_PASS && mode != B200ATTN_BWD_ONE_PASS) return 0;
    if (bwd_resolve_mode(mode, B, T, Hq, D) == B200ATTN_BWD_ONE_PASS) return bwd_vec_bytes_padded(B, T, Hq) + bwd_acc_bytes(B, T, Hq, D);
    return 2 * bwd_vec_elems(B, T, Hq) * sizeof(float);
}

extern "C" size_t b200attn_bwd_workspace_bytes(int B, int T, int Hq, int Hkv, int D) {
    return b200attn_bwd_workspace_bytes_mode(B, T, Hq, Hkv, D, B200ATTN_BWD_AUTO);
}

extern "C" int b200attn_bwd(const void* q, const void* k, const void* v, const void* o, const float* lse,
                            const void* dout, void* dq, void* dk, void* dv, int B, int T, int Hq, int Hkv, int D,
                            int layout, float softmax_scale, void* workspace, size_t workspace_bytes, void* stream) {
    return b200attn_bwd_mode(q, k, v, o, lse, dout, dq, dk, dv, B, T, Hq, Hkv, D, layout, softmax_scale, B200ATTN_BWD_AUTO,
                             workspace, workspace_bytes, stream);
}

extern "C" int b200attn_bwd_mode(const void* q, const void* k, const void* v, const void* o, const float* lse,
                                 const void* dout, void* dq, void* dk, void* dv, int B, int T, int Hq, int Hkv, int D,
                                 int layout, float softmax_scale, int mode, void* workspace, size_t workspace_bytes,
                                 void* stream) {
    int rc = check_common(B, T, Hq, Hkv, D, layout);
    if (rc) return rc;
    if (!q || !k || !v || !o || !lse || !dout || !dq || !dk || !dv) return B200ATTN_ERR_INVALID_ARG;
    if (!aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(o) || !aligned16(dout) || !aligned16(dq) ||
        !aligned16(dk) || !aligned16(dv))
        return B200ATTN_ERR_ALIGNMENT;
    if (mode != B200ATTN_BWD_AUTO && mode != B200ATTN_BWD_TWO_PASS && mode != B200ATTN_BWD_ONE_PASS)
        return B200ATTN_ERR_INVALID_ARG;
    if (mode == B200ATTN_BWD_ONE_PASS && D != 64) return B200ATTN_ERR_UNSUPPORTED;
    const size_t two_pass_bytes = 2 * bwd_vec_elems(B, T, Hq) * sizeof(float);
    const size_t one_pass_bytes = bwd_vec_bytes_padded(B, T, Hq) + bwd_acc_bytes(B, T, Hq, D);
    if (!workspace || workspace_bytes < two_pass_bytes || (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
        return B200ATTN_ERR_WORKSPACE;
    // AUTO falls back to the two-pass kernels when the workspace only holds the row vectors
    const bool auto_mode = mode == B200ATTN_BWD_AUTO;
    mode = bwd_resolve_mode(mode, B, T, Hq, D);
    if (mode == B200ATTN_BWD_ONE_PASS && workspace_bytes < one_pass_bytes) {
        if (!auto_mode) return B200ATTN_ERR_WORKSPACE;
        mode = B200ATTN_BWD_TWO_PASS;
    }
    const BwdTile tile = auto_mode && bwd_forced_mode() == 0 ? bwd_tile(B, T, Hq, Hkv, D) : kTileNo;
    int* status = status_ptr(&rc);
    if (!status) return rc;
    const Strides sq = strides_for(layout, Hq, T, D), sk = strides_for(layout, Hkv, T, D);
    CUtensorMap tq, tk, tv, tdo, own[3];
    bool maps = make_tmap_bf16_4d(&tq, q, D, T, Hq, B, sq.t, sq.h, sq.b, 128) &&
                make_tmap_bf16_4d(&tk, k, D, T, Hkv, B, sk.t, sk.h, sk.b, 128) &&
                make_tmap_bf16_4d(&tv, v, D, T, Hkv, B, sk.t, sk.h, sk.b, 128) &&
                make_tmap_bf16_4d(&tdo, dout, D, T, Hq, B, sq.t, sq.h, sq.b, 128);
    if (mode == B200ATTN_BWD_TWO_PASS && D == 64 && tile == kTileNo)
        maps = maps && make_tmap_bf16_4d(&own[0], k, D, T, Hkv, B, sk.t, sk.h, sk.b, 64) &&
               make_tmap_bf16_4d(&own[1], v, D, T, Hkv, B, sk.t, sk.h, sk.b, 64) &&
               make_tmap_bf16_4d(&own[2], o, D, T, Hq, B, sq.t, sq.h, sq.b, 128);
    if (!maps) return B200ATTN_ERR_TENSOR_MAP;
    float* ws = static_cast<float*>(workspace);
    const size_t nvec = bwd_vec_elems(B, T, Hq);
    BwdParams p;
    p.B = B;
    p.T = T;
    p.Tpad = (T + 127) / 128 * 128;
    p.Hq = Hq;
    p.Hkv = Hkv;
    p.group = Hq / Hkv;
    p.n_tiles = (T + 127) / 128;
    p.scale = softmax_scale > 0.f ? softmax_scale : 1.f / sqrtf((float)D);
    p.scale_log2 = p.scale * 1.4426950408889634f;
    p.lse2 = ws;
    p.dvec = ws + nvec;
    p.lse2_w = ws;
    p.dvec_w = ws + nvec;
    p.lse = lse;
    p.o = static_cast<const uint16_t*>(o);
    p.dout = static_cast<const uint16_t*>(dout);
    p.dq = static_cast<uint16_t*>(dq);
    p.q_st = sq.t;
    p.q_sh = sq.h;
    p.q_sb = sq.b;
    p.dk = static_cast<uint16_t*>(dk);
    p.dv = static_cast<uint16_t*>(dv);
    p.k_st = sk.t;
    p.k_sh = sk.h;
    p.k_sb = sk.b;
    p.status = status;
    p.sched = nullptr;
    p.sched2 = nullptr;
    p.div_bhq = fastdiv_make((unsigned)(B * Hq));
    p.div_hq = fastdiv_make((unsigned)Hq);
    p.div_bhkv = fastdiv_make((unsigned)(B * Hkv));
    p.div_hkv = fastdiv_make((unsigned)Hkv);
    p.div_group = fastdiv_make((unsigned)p.group);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (tile == kTileHead) return D == 64 ? launch_bwd_tile<64, true>(tq, tk, tv, tdo, p, st) : launch_bwd_tile<128, true>(tq, tk, tv, tdo, p, st);
    if (tile == kTileGroup) return D == 64 ? launch_bwd_tile<64, false>(tq, tk, tv, tdo, p, st) : launch_bwd_tile<128, false>(tq, tk, tv, tdo, p, st);
    if (mode == B200ATTN_BWD_ONE_PASS) {
        float* dq_acc = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + bwd_vec_bytes_padded(B, T, Hq));
        return launch_bwd_onepass(tq, tk, tv, tdo, p, dq_acc, st);
    }
    return D == 64 ? launch_bwd<64>(tq, tk, tv, tdo, own, p, st) : launch_bwd<128>(tq, tk, tv, tdo, own, p, st);
}

// ---------------------------------------------------------------------------------------
// Backward with its scratch in the library's own device image: no allocation anywhere.
// ---------------------------------------------------------------------------------------
namespace {

// Two FP32 vectors of B200ATTN_BWD_STATIC_MAX_ROWS rows (logsumexp * log2(e) and rowsum(O * dO)).
// In host code this name is only a handle for cudaGetSymbolAddress, never a device pointer.
static __device__ __align__(256) float g_bwd_static_scratch[2 * B200ATTN_BWD_STATIC_MAX_ROWS];

std::atomic<float*> g_bwd_static_ptr[kMaxDevices] = {};

// Device address of the array on the current device, resolved once per device.
float* bwd_static_scratch(int* err) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        *err = B200ATTN_ERR_NO_DEVICE;
        return nullptr;
    }
    if (!g_bwd_static_ptr[dev]) {
        float* ptr = nullptr;
        if (cudaGetSymbolAddress((void**)&ptr, g_bwd_static_scratch) != cudaSuccess || ptr == nullptr) {
            cudaGetLastError();
            *err = B200ATTN_ERR_CUDA;
            return nullptr;
        }
        g_bwd_static_ptr[dev] = ptr;
    }
    return g_bwd_static_ptr[dev];
}

}  // namespace

extern "C" int b200attn_bwd_static(const void* q, const void* k, const void* v, const void* o, const float* lse,
                                   const void* dout, void* dq, void* dk, void* dv, int B, int T, int Hq, int Hkv, int D,
                                   int layout, float softmax_scale, void* stream) {
    int rc = check_common(B, T, Hq, Hkv, D, layout);
    if (rc) return rc;
    if (bwd_vec_elems(B, T, Hq) > (size_t)B200ATTN_BWD_STATIC_MAX_ROWS) return B200ATTN_ERR_TOO_LARGE;
    float* scratch = bwd_static_scratch(&rc);
    if (!scratch) return rc;
    // Always the two passes; the dQ pass rewrites every row of the row vectors (padding included) that the dK/dV pass reads, so
    // stale contents of an earlier call are never seen.  b200attn_bwd may take the one-tile kernel for T <= 128 (bwd_tile), whose
    // sums are grouped in another way: the two may differ there by roundings.
    return b200attn_bwd_mode(q, k, v, o, lse, dout, dq, dk, dv, B, T, Hq, Hkv, D, layout, softmax_scale,
                             B200ATTN_BWD_TWO_PASS, scratch, 2 * sizeof(float) * (size_t)B200ATTN_BWD_STATIC_MAX_ROWS, stream);
}

namespace {

// Query heads served per decode CTA: the largest divisor of the group size that is <= 16
// (the row count of the kernel's MMA shape).
inline int decode_heads_per_cta(int group) {
    for (int g = 16; g >= 1; --g)
        if (group % g == 0) return g;
    return 1;
}

inline int decode_tile_keys(int D) { return D == 64 ? DecodeCfg<64>::kKeys : DecodeCfg<128>::kKeys; }
inline int decode_max_ctas() { return std::min(2 * sm_count(), kDecodeMaxCtas); }  // two fit an SM: all are resident at once

struct DecodePlan {
    int G, n_chunks;
    int slots;    // workspace slots per unit for partial results
    int splits;   // and with the room for the counters behind them
    int shares;   // CTAs per unit, or 0: ranges of tiles
    int cluster;  // CTAs per cluster
    bool whole;   // ranges of whole units
    int n_ctas, slot_mode;
};

// The deal (see attn_decode.cuh).
//
// Ranges cost about 3 us at the end (partial results through memory, a counter, the last CTA's additions), clusters
// about 1 us, whole units nothing.  So units stay whole or in clusters unless that leaves the memory system idle for longer
// than that: some 60 SMs saturate HBM, so what counts is how many CTAs the last round has (all, where the units are fewer
// than the SMs) and how long a unit is, and, for sequences of different lengths, how much memory there is to read at all.
// kRangesBytes is what HBM delivers in those 3 us.
//
// A cluster is the smallest that leaves a CTA at most two tiles, as far as that is one CTA per SM: more of them saturate
// HBM by themselves.
//
// n_splits > 0 asks for that many shares per unit (at most 64, none empty): a cluster where it can have that size.
constexpr long long kRangesBytes = 16ll << 20;
constexpr int kSaturatingCtas = 60;

DecodePlan decode_plan(int B, int L, int Hq, int Hkv, int D, int n_splits, bool ragged) {
    DecodePlan d;
    const int group = Hq / Hkv, cap = decode_max_ctas();
    d.G = decode_heads_per_cta(group);
    d.n_chunks = group / d.G;
    const long long units = (long long)B * Hkv * d.n_chunks;
    const int keys = decode_tile_keys(D), n_all = (L + keys - 1) / keys, n_128 = (L + 127) / 128;
    const long long unit_bytes = 4ll * L * D, tiles = units * n_all;
    d.shares = d.cluster = 1;
    d.whole = false;
    d.slot_mode = kDecodeSlotTile;
    long long counters = 0;
    if (n_splits > 0) {
        const int want = std::min(std::min(n_splits, n_128), 64), per = (n_128 + want - 1) / want;
        d.slots = d.shares = (n_128 + per - 1) / per;
        if (d.shares <= kDecodeMaxCluster && (d.shares & (d.shares - 1)) == 0) {
            d.cluster = d.shares;
        } else {
            d.slot_mode = kDecodeSlotCta;
            counters = units * d.shares;
        }
    } else {
        d.slots = (int)std::min<long long>(n_all, (2 * cap + units - 1) / units);
        if (n_all > 1) counters = std::min<long long>(tiles, cap);  // (a single tile is never shared)
        while (d.cluster < kDecodeMaxCluster && units * d.cluster * 2 <= sm_count() && n_all > 2 * d.cluster) d.cluster *= 2;
        d.shares = d.cluster;
        const long long ctas = units * d.cluster, last = ctas % cap ? ctas % cap : cap;
        const long long idle = last < kSaturatingCtas ? unit_bytes / d.cluster * (kSaturatingCtas - last) : 0;
        if (tiles > d.cluster * units && (idle > kRangesBytes || (ragged && units * unit_bytes > kRangesBytes))) {
            d.shares = 0;
            d.cluster = 1;
            d.slot_mode = d.slots == n_all ? kDecodeSlotTile : kDecodeSlotTwo;
        }
    }
    // the counters behind the slots, in units of a slot of every (batch, query head)
    const long long slot_bytes = (long long)B * Hq * (D + 2) * 4;
    d.splits = d.slots + (int)((8 * counters + slot_bytes - 1) / slot_bytes);
    if (d.shares == 0) {
        d.n_ctas = (int)std::min<long long>(tiles, cap);
        return d;
    }
    d.n_ctas = (int)std::min<long long>(units * d.shares, 1ll << 30);
    if (d.shares == 1 && units > cap && !ragged) {  // the ring of a CTA then runs on from unit to unit
        d.shares = 0;
        d.whole = true;
        d.n_ctas = cap;
    }
    return d;
}

template <int D, int NH, int PF>
int launch_decode_pf(const CUtensorMap& tk, const CUtensorMap& tv, const DecodeParams& p, int n_ctas, cudaStream_t st) {
    using Cfg = DecodeCfg<D>;
    static bool set[kMaxDevices] = {false};
    int rc = set_smem_once(attn_decode_kernel<D, NH, PF>, Cfg::kSmemBytes, set);
    if (rc) return rc;
    if (launch_cluster(attn_decode_kernel<D, NH, PF>, dim3(n_ctas), kDecodeThreads, Cfg::kSmemBytes, st, p.cluster, tk, tv, p) != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    return B200ATTN_OK;
}

// Where the CTAs fill most of the device the launch is bound by HBM, and the first two tiles of each come into L2 while the kernel
// in front ends, provided that it lets this one start early, as the append of one token and the decode itself do (us per call over
// caches larger than L2 in turn, without / with: append + decode B=48 L<=6000 16/4 D=64 35.6 / 34.3, B=64 L<=4096 33.5 / 31.8, B=20 L<=1500
// D=128 19.3 / 18.0; decode behind decode B=64 L=4096 16/4 D=64 41.9 / 41.3, B=300 L=200 8/8 24.0 / 22.8, B=64 L=1000 6/2 9.0 / 8.5, B=8
// L=2000 8/8 D=128, 128 CTAs, 14.3 / 14.1).  With a matrix product in front of each append + decode, the product included: 40.6 / 39.9,
// 38.3 / 37.5, 23.4 / 23.0.  Behind a kernel that does not release this one early the tiles are asked for twice: product and decode
// 46.1 / 46.0, 29.8 / 29.5, 13.3 / 13.4, 19.1 / 19.3; a first pass on new buffers on an idle device gains nothing (host's time of a call,
// B=300 41.8 / 42.1, append + decode B=48 67.3 / 67.0).  With three tiles the gain is smaller, with six it is gone.
// Fewer CTAs are bound by latency, of which this hides nothing: B=6 L<=3000 8/1 D=128 8.5 -> 8.6, B=1 L=1500 16/4 5.26 -> 5.30.
constexpr int kPrefetchCtas = 128;
template <int D, int NH>
int launch_decode(const CUtensorMap& tk, const CUtensorMap& tv, const DecodeParams& p, int n_ctas, cudaStream_t st) {
    return n_ctas >= kPrefetchCtas ? launch_decode_pf<D, NH, 2>(tk, tv, p, n_ctas, st) : launch_decode_pf<D, NH, 0>(tk, tv, p, n_ctas, st);
}

}  // namespace

extern "C" int b200attn_decode_default_splits(int B, int L, int Hq, int Hkv, int D) {
    if (B <= 0 || L <= 0 || Hq <= 0 || Hkv <= 0 || Hq % Hkv != 0) return 0;
    return decode_plan(B, L, Hq, Hkv, D, 0, false).splits;
}

extern "C" size_t b200attn_decode_workspace_bytes(int B, int L, int Hq, int Hkv, int D, int n_splits) {
    if (B <= 0 || L <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0 || Hq % Hkv != 0) return 0;
    const int s = decode_plan(B, L, Hq, Hkv, D, n_splits, false).splits;
    return (size_t)B * Hq * s * (size_t)(D + 2) * sizeof(float);
}

extern "C" int b200attn_decode(const void* q, const void* kcache, const void* vcache, void* o, float* lse, int B, int L,
                               int Hq, int Hkv, int D, float softmax_scale, int n_splits, void* workspace,
                               size_t workspace_bytes, void* stream) {
    return b200attn_decode_cached(q, kcache, vcache, o, lse, B, L, L, Hq, Hkv, D, softmax_scale, n_splits, workspace,
                                  workspace_bytes, stream);
}

extern "C" int b200attn_decode_cached(const void* q, const void* kcache, const void* vcache, void* o, float* lse, int B,
                                      int L, int L_cap, int Hq, int Hkv, int D, float softmax_scale, int n_splits,
                                      void* workspace, size_t workspace_bytes, void* stream) {
    return b200attn_decode_ragged(q, kcache, vcache, o, lse, nullptr, B, L, L_cap, Hq, Hkv, D, softmax_scale, n_splits,
                                  workspace, workspace_bytes, stream);
}

extern "C" int b200attn_decode_ragged(const void* q, const void* kcache, const void* vcache, void* o, float* lse,
                                      const int* lens, int B, int L, int L_cap, int Hq, int Hkv, int D,
                                      float softmax_scale, int n_splits, void* workspace, size_t workspace_bytes,
                                      void* stream) {
    int rc = check_common(B, L, Hq, Hkv, D, B200ATTN_LAYOUT_BHTD);
    if (rc) return rc;
    if (L_cap < L) return B200ATTN_ERR_INVALID_ARG;
    if (!q || !kcache || !vcache || !o) return B200ATTN_ERR_INVALID_ARG;
    if (!aligned16(q) || !aligned16(kcache) || !aligned16(vcache) || !aligned16(o)) return B200ATTN_ERR_ALIGNMENT;
    if (!workspace || workspace_bytes < b200attn_decode_workspace_bytes(B, L, Hq, Hkv, D, n_splits) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u) != 0)
        return B200ATTN_ERR_WORKSPACE;
    int* status = status_ptr(&rc);
    if (!status) return rc;
    const DecodePlan d = decode_plan(B, L, Hq, Hkv, D, n_splits, lens != nullptr);
    // the maps end at row L of every (batch, head): rows of the cache beyond it are never read (TMA fills zeros)
    const Strides sk = strides_for(B200ATTN_LAYOUT_BHTD, Hkv, L_cap, D);
    CUtensorMap tk, tv;
    if (!make_tmap_bf16_4d(&tk, kcache, D, L, Hkv, B, sk.t, sk.h, sk.b, decode_tile_keys(D)) ||
        !make_tmap_bf16_4d(&tv, vcache, D, L, Hkv, B, sk.t, sk.h, sk.b, decode_tile_keys(D)))
        return B200ATTN_ERR_TENSOR_MAP;
    DecodeParams p;
    p.B = B;
    p.L = L;
    p.Hq = Hq;
    p.Hkv = Hkv;
    p.group = Hq / Hkv;
    p.G = d.G;
    p.n_chunks = d.n_chunks;
    p.units_per_seq = Hkv * d.n_chunks;
    p.div_units = fastdiv_make((unsigned)p.units_per_seq);
    p.div_chunks = fastdiv_make((unsigned)d.n_chunks);
    p.div_shares = fastdiv_make((unsigned)std::max(d.shares, 1));
    p.div_tiles = fastdiv_make((unsigned)((L + decode_tile_keys(D) - 1) / decode_tile_keys(D)));
    p.div_slice = fastdiv_make((unsigned)(d.G * (D / 2) / d.cluster));
    p.shares = d.shares;
    p.cluster = d.cluster;
    p.whole = d.whole;
    p.slot_mode = d.slot_mode;
    p.scale = softmax_scale > 0.f ? softmax_scale : 1.f / sqrtf((float)D);
    p.scale_log2 = p.scale * 1.4426950408889634f;
    p.lens = lens;
    p.q = static_cast<const uint16_t*>(q);
    p.o = static_cast<uint16_t*>(o);
    p.lse = lse;
    const size_t rows = (size_t)B * Hq * d.slots;  // slots x heads per slot
    p.part_o = static_cast<float*>(workspace);
    p.part_m = p.part_o + rows * D;
    p.part_l = p.part_m + rows;
    p.counters = reinterpret_cast<unsigned long long*>(p.part_l + rows);  // (D + 2 is even: 8-byte aligned)
    p.tag = next_decode_tag();
    p.status = status;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (D == 64) return d.G <= 8 ? launch_decode<64, 1>(tk, tv, p, d.n_ctas, st) : launch_decode<64, 2>(tk, tv, p, d.n_ctas, st);
    return d.G <= 8 ? launch_decode<128, 1>(tk, tv, p, d.n_ctas, st) : launch_decode<128, 2>(tk, tv, p, d.n_ctas, st);
}

namespace {

template <int D, bool F32>
int launch_kv_append(const KvAppendParams& p, cudaStream_t st) {
    const long long rows = (long long)p.rows_q + 2LL * p.rows_kv;
    const long long rows_per_cta = (kKvAppendThreads / 32) * (256 / D);
    long long grid = (rows + rows_per_cta - 1) / rows_per_cta;
    const long long cap = 8LL * sm_count();  // 8 CTAs of 256 threads are resident per SM
    if (grid > cap) grid = cap;
    if (launch_pdl(kv_append_kernel<D, F32>, dim3((unsigned)grid, 1, 1), kKvAppendThreads, 0, st, p) != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    return B200ATTN_OK;
}

}  // namespace

namespace {
int kv_append_run(const void* xq, const void* xk, const void* xv, int x_dtype, void* q_out, void* kcache, void* vcache,
                  const float* gamma_q, const float* gamma_k, const float* cos_t, const float* sin_t, const int* pos,
                  int B, int n_new, int pos0, int L_cap, int Hq, int Hkv, int D, float eps, void* stream);
}

extern "C" int b200attn_kv_append(const void* xq, const void* xk, const void* xv, int x_dtype, void* q_out, void* kcache,
                                  void* vcache, const float* gamma_q, const float* gamma_k, const float* cos_t,
                                  const float* sin_t, int B, int n_new, int pos0, int L_cap, int Hq, int Hkv, int D,
                                  float eps, void* stream) {
    return kv_append_run(xq, xk, xv, x_dtype, q_out, kcache, vcache, gamma_q, gamma_k, cos_t, sin_t, nullptr, B, n_new, pos0,
                         L_cap, Hq, Hkv, D, eps, stream);
}

extern "C" int b200attn_kv_append_at(const void* xq, const void* xk, const void* xv, int x_dtype, void* q_out, void* kcache,
                                     void* vcache, const float* gamma_q, const float* gamma_k, const float* cos_t,
                                     const float* sin_t, const int* pos, int B, int n_new, int L_cap, int Hq, int Hkv,
                                     int D, float eps, void* stream) {
    if (!pos) return B200ATTN_ERR_INVALID_ARG;
    return kv_append_run(xq, xk, xv, x_dtype, q_out, kcache, vcache, gamma_q, gamma_k, cos_t, sin_t, pos, B, n_new, 0, L_cap,
                         Hq, Hkv, D, eps, stream);
}

namespace {
int kv_append_run(const void* xq, const void* xk, const void* xv, int x_dtype, void* q_out, void* kcache, void* vcache,
                  const float* gamma_q, const float* gamma_k, const float* cos_t, const float* sin_t, const int* pos,
                  int B, int n_new, int pos0, int L_cap, int Hq, int Hkv, int D, float eps, void* stream) {
    if (B <= 0 || n_new <= 0 || pos0 < 0 || L_cap <= 0 || Hq <= 0 || Hkv <= 0 || D <= 0) return B200ATTN_ERR_INVALID_ARG;
    if (Hq % Hkv != 0 || (long long)pos0 + n_new > L_cap) return B200ATTN_ERR_INVALID_ARG;
    if (x_dtype != B200ATTN_DTYPE_BF16 && x_dtype != B200ATTN_DTYPE_F32) return B200ATTN_ERR_INVALID_ARG;
    if (D != 64 && D != 128) return B200ATTN_ERR_UNSUPPORTED;
    if (!xq || !xk || !xv || !q_out || !kcache || !vcache || !gamma_q || !gamma_k || !cos_t || !sin_t)
        return B200ATTN_ERR_INVALID_ARG;
    if (!aligned16(xq) || !aligned16(xk) || !aligned16(xv) || !aligned16(q_out) || !aligned16(kcache) ||
        !aligned16(vcache) || !aligned16(gamma_q) || !aligned16(gamma_k) || !aligned16(cos_t) || !aligned16(sin_t))
        return B200ATTN_ERR_ALIGNMENT;
    const long long rows_q = (long long)B * n_new * Hq, rows_kv = (long long)B * n_new * Hkv;
    if (rows_q + 2 * rows_kv >= (1LL << 31)) return B200ATTN_ERR_TOO_LARGE;
    int rc = 0;
    int* status = status_ptr(&rc);
    if (!status) return rc;
    KvAppendParams p;
    p.pos = pos;
    p.status = status;
    p.xq = xq;
    p.xk = xk;
    p.xv = xv;
    p.q_out = static_cast<uint16_t*>(q_out);
    p.kcache = static_cast<uint16_t*>(kcache);
    p.vcache = static_cast<uint16_t*>(vcache);
    p.gamma_q = gamma_q;
    p.gamma_k = gamma_k;
    p.cos_t = cos_t;
    p.sin_t = sin_t;
    p.B = B;
    p.n_new = n_new;
    p.pos0 = pos0;
    p.L_cap = L_cap;
    p.Hq = Hq;
    p.Hkv = Hkv;
    p.rows_q = (unsigned)rows_q;
    p.rows_kv = (unsigned)rows_kv;
    p.div_hq = fastdiv_make((unsigned)Hq);
    p.div_hkv = fastdiv_make((unsigned)Hkv);
    p.div_n = fastdiv_make((unsigned)n_new);
    p.eps = eps;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool f32 = x_dtype == B200ATTN_DTYPE_F32;
    if (D == 64) return f32 ? launch_kv_append<64, true>(p, st) : launch_kv_append<64, false>(p, st);
    return f32 ? launch_kv_append<128, true>(p, st) : launch_kv_append<128, false>(p, st);
}
}  // namespace

extern "C" int b200attn_item_deal(int n_groups, int n_qtiles, int T, int n_ctas, int item_cost, unsigned short* ids,
                                  int* per_cta) {
    if (n_groups <= 0 || n_qtiles <= 0 || T <= 0 || n_ctas <= 0 || item_cost < 0 || !ids || !per_cta)
        return B200ATTN_ERR_INVALID_ARG;
    const ItemTable& tab = item_table_for((long long)n_groups * n_qtiles, (unsigned)n_ctas, n_groups, n_qtiles, T, item_cost);
    *per_cta = tab.per_cta;
    for (int i = 0; i < n_ctas * tab.per_cta; ++i) ids[i] = tab.ids[i];
    return B200ATTN_OK;
}

extern "C" int b200attn_last_device_status(void* stream) {
    int rc = 0;
    int* status = status_ptr(&rc);
    if (!status) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaStreamSynchronize(st) != cudaSuccess) {
        cudaGetLastError();
        return B200ATTN_ERR_CUDA;
    }
    int host[2] = {0, 0};  // status word and epoch
    if (cudaMemcpy(host, status, sizeof(host), cudaMemcpyDeviceToHost) != cudaSuccess) return B200ATTN_ERR_CUDA;
    if (host[0] != 0) {
        // a kernel that gave up may have left its item counters behind: wait for everything else on the
        // device (kernels exit at once while the status word is set), then clear counters and status
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceSynchronize();
        cudaMemset(g_sched_ptr[dev].load(), 0, sizeof(int) * 2 * kSchedSlots);
        const int next[2] = {0, (host[1] + 1) & ((1 << kDecodeEpochBits) - 1)};
        cudaMemcpy(status, next, sizeof(next), cudaMemcpyHostToDevice);
        return host[0];
    }
    return B200ATTN_OK;
}

extern "C" const char* b200attn_strerror(int status) {
    switch (status) {
        case B200ATTN_OK: return "ok";
        case B200ATTN_ERR_INVALID_ARG: return "invalid argument (null pointer, non-positive size, Hq % Hkv != 0 or bad layout)";
        case B200ATTN_ERR_UNSUPPORTED: return "unsupported head dimension (only 64 and 128)";
        case B200ATTN_ERR_ALIGNMENT: return "a base pointer is not 16-byte aligned";
        case B200ATTN_ERR_WORKSPACE: return "workspace missing, misaligned or too small";
        case B200ATTN_ERR_CUDA: return "a CUDA runtime call or kernel launch failed";
        case B200ATTN_ERR_TENSOR_MAP: return "the driver refused a TMA tensor map";
        case B200ATTN_ERR_DEVICE_WAIT: return "a kernel gave up on a bounded wait";
        case B200ATTN_ERR_NO_DEVICE: return "no usable CUDA device is current";
        case B200ATTN_ERR_TOO_LARGE:
            return "problem too large: beyond the fixed scratch of b200attn_bwd_static (B*Hq*ceil(T/128)*128 > 524288), or "
                   "2^31 or more rows in a RoPE / QK-Norm / KV-append call";
        case DEV_WAIT_TIMEOUT_LOAD: return "device: a TMA load barrier never completed";
        case DEV_WAIT_TIMEOUT_MMA: return "device: a tensor-core completion barrier never completed";
        case DEV_WAIT_TIMEOUT_SOFTMAX: return "device: a softmax hand-off barrier never completed";
        case DEV_WAIT_TIMEOUT_FREE: return "device: a buffer-free barrier never completed";
        case DEV_KV_CACHE_OVERFLOW: return "device: a KV-cache position plus the new tokens exceeds the cache capacity";
        default: return "unknown status";
    }
}

extern "C" int b200attn_version(void) { return 1; }

#ifdef B200ATTN_PROBE
// Tuning builds only: copies the phase timestamps of the last launch to the host.
extern "C" int b200attn_debug_read_probe(long long* host, int n) {
    if (n > 512) n = 512;
    return cudaMemcpyFromSymbol(host, b200attn::g_probe, sizeof(long long) * n) == cudaSuccess ? 0 : B200ATTN_ERR_CUDA;
}
extern "C" int b200attn_debug_read_trace(unsigned long long* host, int n_ctas) {
    if (n_ctas > 8192) n_ctas = 8192;
    return cudaMemcpyFromSymbol(host, b200attn::g_trace, sizeof(unsigned long long) * 3 * n_ctas) == cudaSuccess
               ? 0 : B200ATTN_ERR_CUDA;
}
extern "C" int b200attn_debug_read_trace_clk(long long* host, int n_ctas) {
    if (n_ctas > 8192) n_ctas = 8192;
    return cudaMemcpyFromSymbol(host, b200attn::g_trace_clk, sizeof(long long) * 2 * n_ctas) == cudaSuccess
               ? 0 : B200ATTN_ERR_CUDA;
}
#endif
