// Onesweep LSD radix sort of the 63-bit Morton keys with a 32-bit payload
// (the body's previous position), and the permutation of the body arrays.
//
// Replaces sortBodiesByMortonKey (include/utility.h:23-52).  The reference
// index-sorts with std::sort and gathers pos/mass/vel/ids/keys; here the
// sort is a stable 8-pass LSD radix sort (8-bit digits) whose digit
// histograms for all passes come from the key kernel, and each pass is one
// kernel: tiles claim an id in launch order, rank their keys warp by warp,
// publish per-digit tile counts, and obtain their global offsets by a decoupled
// look-back over earlier tiles.  Every wait
// in the look-back is bounded; on expiry the kernel raises kErrTimeout
// and still publishes, so no tile can wait forever.
//
// Up to some 100,000 keys one thread-block cluster sorts in distributed shared
// memory instead (cluster_sort_kernel below).
#include <cooperative_groups.h>

#include <utility>

#include "bh_internal.cuh"
#include "bh_per_device.h"

namespace bh {
namespace {

constexpr int kWarps = kSortThreads / 32;  // 16
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagIncl = 2u << 30;
constexpr uint32_t kCountMask = (1u << 30) - 1;
constexpr int kSpinLimit = 1 << 22;
constexpr int kBatch = 4;  // look-back: predecessors read per round

struct SortSmem {
    uint32_t warp_hist[kWarps][kRadix];  // per-warp digit counts, then warp prefixes
    uint32_t warp_mask[kWarps][kRadix];  // lanes per digit, for rank_item
    uint32_t tile_hist[kRadix];          // the tile's digit counts
    uint32_t digit_excl[kRadix];         // tile-local start of each digit
    uint32_t global_base[kRadix];        // global start minus tile-local start
    uint32_t scan[kRadix / 32];
    uint32_t tile;
    uint64_t keys[kSortTile];
    uint32_t vals[kSortTile];
};

// One item of a warp's ranking: the lane's rank among the warp's keys of its
// digit so far, and its digit's count moved on.  Every lane sets its bit in the
// digit's word of `mask` (zero before and after) and reads there which lanes
// hold the same digit.  (A ballot per digit bit does without the words, but a
// vote takes the SM about four cycles: 64 of them a thread bounded the ranking,
// 4,400 cycles a tile.)
template <typename Count>
__device__ __forceinline__ uint32_t rank_item(uint32_t d, bool valid, unsigned lt, int lane, uint32_t* mask,
                                              Count* hist)
{
    if (valid) atomicOr(&mask[d], 1u << lane);
    __syncwarp();
    uint32_t peers = 0, old = 0;
    if (valid) {
        peers = mask[d];
        old = hist[d];
    }
    __syncwarp();
    if (valid && (peers & lt) == 0u) {  // the lowest peer
        mask[d] = 0;
        hist[d] = (Count)(old + __popc(peers));
    }
    __syncwarp();
    return old + __popc(peers & lt);
}

// Exclusive scan over 256 values held one per thread by 8 consecutive warps,
// the first 256 threads of a block or those from a multiple of 256 on.
__device__ uint32_t scan256(uint32_t v, uint32_t* tmp)
{
    const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 7;
    uint32_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) tmp[w] = x;
    __syncwarp();
    // 8 warps: a tiny serial pass by each thread over the warp totals.
    asm volatile("bar.sync 1, 256;" ::: "memory");
    uint32_t before = 0;
    for (int k = 0; k < w; ++k) before += tmp[k];
    return before + x - v;
}

__global__ void hist_scan_kernel(uint32_t* __restrict__ hist)
{
    __shared__ uint32_t tmp[kRadix / 32];
    uint32_t* h = hist + blockIdx.x * kRadix;
    const uint32_t v = h[threadIdx.x];
    const uint32_t e = scan256(v, tmp);
    h[threadIdx.x] = e;
}

// 16 warps rank the tile's keys and put them in order in shared memory; 8 more
// publish its digit counts and look back while they do.  Latency bounds a tile:
// what its successors wait for is kept short (no fence, since a flag and its
// count are one word; four predecessors a round, where 8 read more that is not
// there yet: 135 and 128 us at 1M).  Sort phase per step with one set of warps,
// ballots for the ranking and a fence, and now: 100,000 keys 96 -> 84 us,
// 300,149 110 -> 93, 1M 173 -> 128, 4M 420 -> 332.
constexpr int kLookThreads = kRadix;  // a thread per digit
constexpr int kTileThreads = kSortThreads + kLookThreads;

template <bool kFirst>
__global__ void __launch_bounds__(kTileThreads, 2) onesweep_kernel(
    int64_t n, int shift, const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
    uint64_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out, const uint32_t* __restrict__ bucket_start,
    uint32_t* lookback, uint32_t* tile_ctr, unsigned* err)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortSmem& s = *reinterpret_cast<SortSmem*>(smem_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool ranks = threadIdx.x < kSortThreads;

    if (threadIdx.x == 0) s.tile = atomicAdd(tile_ctr, 1u);
    for (int k = threadIdx.x; k < (2 * kWarps + 1) * kRadix; k += kTileThreads) (&s.warp_hist[0][0])[k] = 0;
    __syncthreads();
    const uint32_t tile = s.tile;
    const int64_t base = (int64_t)tile * kSortTile;
    const int64_t rem = n - base;
    const int cnt = rem < kSortTile ? (int)rem : kSortTile;

    // Warp w owns keys [w*256, w*256+256) of the tile, item k at lane l is
    // key w*256 + k*32 + l, so (w, k, l) is the input order.
    uint64_t key[kSortItems];
    uint32_t val[kSortItems], rank[kSortItems / 2] = {};  // rank: 16 bits an item
    const unsigned lt = (1u << lane) - 1u;
    const int first = w * (32 * kSortItems) + lane;
    if (ranks) {
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) key[k] = first + k * 32 < cnt ? keys_in[base + first + k * 32] : ~0ull;
#pragma unroll
        for (int k = 0; k < kSortItems; ++k)
            rank[k / 2] |= rank_item((uint32_t)(key[k] >> shift) & 0xFFu, first + k * 32 < cnt, lt, lane,
                                     s.warp_mask[w], s.warp_hist[w])
                           << 16 * (k & 1);
#pragma unroll
        for (int k = 0; k < kSortItems; ++k)
            val[k] = kFirst ? (uint32_t)base + first + k * 32 : first + k * 32 < cnt ? vals_in[base + first + k * 32] : 0;
        asm volatile("bar.sync 2, %0;" ::"n"(kSortThreads) : "memory");
        // Two threads per digit: exclusive prefix over the warps.
        const int d = threadIdx.x >> 1, h = threadIdx.x & 1;
        uint32_t sum = 0;
#pragma unroll
        for (int k = 0; k < kWarps / 2; ++k) sum += s.warp_hist[h * (kWarps / 2) + k][d];
        uint32_t run = __shfl_up_sync(0xffffffffu, sum, 1);
        if (h == 0) run = 0;
#pragma unroll
        for (int k = 0; k < kWarps / 2; ++k) {
            const uint32_t c = s.warp_hist[h * (kWarps / 2) + k][d];
            s.warp_hist[h * (kWarps / 2) + k][d] = run;
            run += c;
        }
        if (h == 1) s.tile_hist[d] = run;
    }
    __syncthreads();
    if (ranks) {
        // ... and the digits' starts from the other warps.
        asm volatile("bar.sync 3, %0;" ::"n"(kTileThreads) : "memory");
        // Into shared memory in tile-sorted order.
#pragma unroll
        for (int k = 0; k < kSortItems; ++k) {
            if (first + k * 32 < cnt) {
                const uint32_t d = (uint32_t)(key[k] >> shift) & 0xFFu;
                const uint32_t p = s.digit_excl[d] + s.warp_hist[w][d] + (rank[k / 2] >> 16 * (k & 1) & 0xFFFFu);
                if (p < (uint32_t)kSortTile) {
                    s.keys[p] = key[k];
                    s.vals[p] = val[k];
                }
            }
        }
    } else {
        // Decoupled look-back: thread d sums earlier tiles' counts of digit d,
        // reading kBatch predecessors per round (independent loads in flight)
        // and stopping at the nearest inclusive prefix.  A predecessor that
        // has not published yet is read again (bounded).
        const int d = threadIdx.x - kSortThreads;
        const uint32_t tile_count = s.tile_hist[d];
        volatile uint32_t* lb = lookback + (size_t)tile * kRadix;
        lb[d] = (tile == 0 ? kFlagIncl : kFlagAgg) | tile_count;
        const uint32_t bucket = bucket_start[d];
        const uint32_t start = scan256(tile_count, s.scan);
        s.digit_excl[d] = start;
        asm volatile("bar.arrive 3, %0;" ::"n"(kTileThreads) : "memory");
        uint32_t excl = 0;
        if (tile > 0) {
            const volatile uint32_t* lbv = lookback;
            int k = (int)tile - 1;
            int spins = 0;
            while (k >= 0) {
                uint32_t v[kBatch];
#pragma unroll
                for (int q = 0; q < kBatch; ++q) v[q] = k - q >= 0 ? lbv[(size_t)(k - q) * kRadix + d] : kFlagIncl;
                int used = 0;
                bool found = false, stall = false;
#pragma unroll
                for (int q = 0; q < kBatch; ++q) {
                    if (!found && !stall && k - q >= 0) {
                        const uint32_t f = v[q] & ~kCountMask;
                        if (f == 0u) {
                            stall = true;  // not published yet: read again from here
                        } else {
                            excl += v[q] & kCountMask;
                            ++used;
                            found = f == kFlagIncl;
                        }
                    }
                }
                if (found) break;
                if (stall) {
                    if (++spins > kSpinLimit) {
                        atomicOr(err, kErrTimeout);
                        break;
                    }
                }
                k -= used;
            }
            // (flag and count are one word: nothing to order it with)
            lb[d] = kFlagIncl | ((excl + tile_count) & kCountMask);
        }
        s.global_base[d] = bucket + excl - start;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < cnt; j += kTileThreads) {
        const uint64_t kk = s.keys[j];
        const uint32_t d = (uint32_t)((kk >> shift) & 0xFF);
        const uint32_t g = s.global_base[d] + (uint32_t)j;
        if ((int64_t)g < n) {  // always true unless a look-back wait gave up
            keys_out[g] = kk;
            vals_out[g] = s.vals[j];
        }
    }
}

// Small sets: one cluster of 1 to 16 blocks holds all keys in its shared
// memory.  The onesweep passes above cost a launch, a look-back chain and a
// trip through memory each, 60 us and more however few the keys are; here a
// pass is two cluster barriers around a scatter over the blocks' shared
// memory.  A block owns `per` consecutive positions; the digits are ranked as
// above, the blocks exchange their digit counts, and every key goes straight
// to the block and place it sorts to.
//
// The high 32 bits of the key are sorted first, in four passes.  Morton keys
// equal there share a cell of the tenth level, so in most sets few are left to
// order.  Runs of equal high bits are then ordered in place: up to kTieRun keys
// by a thread's insertion (stable, as the passes are), up to kTieWarp by a
// warp.  With a longer run the set is sorted by all eight digits instead; where
// a sample of the keys shows that (an outlier makes the box wide for the rest,
// and the LET codes of the upper cells have no high bits), at once.
// Sort phase per step, us, before -> after: 1,000 keys 71 -> 14, 19,054 92 -> 28,
// 65,536 95 -> 48 (68 with 8 blocks, 79 with key and payload as two words).
// With one body at 200 / 1,000 / 10,000 AU (runs of 20 / 331 / 33,623 keys at
// 65,537): 60 / 70 / 69 (onesweep 93), and 103 / 102 / 97 when every run above
// kTieRun had the set sorted by four digits and then by eight; at 98,304 83 / 86
// / 84 (93), and 129 / 127 / 120 so.
// At the large end the remote stores bound it (a block's 4,096 words in 2.3 us
// a pass); staging a pass's words in digit order before they leave the block
// gained nothing.
constexpr int kCThreads = 1024;
constexpr int kCWarps = kCThreads / 32;
constexpr int kCMax = 16;      // blocks, where the device takes clusters beyond the portable 8
constexpr int kCPortable = 8;
constexpr int kBlockKeys = 8192;
// With 16 blocks the cluster is ahead of the onesweep passes up to here (sort and
// key phases together, us: 65,537 keys 102 / 59, 98,304 103 / 75, 110,000 107 /
// 82 with a step 1 % faster, 131,000 108 / 91 with a step 2 % slower; with
// long ties 98,304 107 / 100).
constexpr int64_t kClusterSortMax = 98304;
constexpr int kTieRun = 16;
constexpr int kTieWarp = 256;  // the words of a warp's row of warp_mask
constexpr int kSampleSlots = 2 * kCMax * kRadix;  // 16-bit counters in `totals`
// The sample takes 1 to 2 us.  Below three keys to a thread (32,768) all twelve
// passes stay under the onesweep ones without it (19,054 keys 63 and 91 us).
constexpr int kSampleItems = 3;
constexpr int kMaxTieRuns = kBlockKeys / (kTieRun + 1) + 1;  // longer than kTieRun, starting in one block
constexpr int kHistRow = kRadix + 2;  // 129 words: the four quarters of a digit's column fall in four bank groups

struct ClusterSmem {
    uint64_t words[kBlockKeys];  // 32 bits of the key over the key's index
    uint16_t warp_hist[kCWarps][kHistRow];
    uint32_t warp_mask[kCWarps][kRadix];
    uint32_t totals[kCMax][kRadix];  // every block's digit counts
    uint32_t base[kRadix];           // where the block's keys of a digit go
    uint32_t scan[kRadix / 32];
    int flags[kCMax];
    int tied, runs;
};
static_assert(kMaxTieRuns <= kCMax * kRadix, "the list of runs in `totals`");

template <int I>
__global__ void __launch_bounds__(kCThreads) cluster_sort_kernel(int n, int per, const uint64_t* keys_in,
                                                                 uint64_t* keys_out, uint32_t* __restrict__ vals_out)
{
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterSmem& s = *reinterpret_cast<ClusterSmem*>(smem_raw);
    const cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), r = (int)cluster.block_rank();
    constexpr bool kSample = I >= kSampleItems;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int start = r * per;
    const int cnt = n - start < 0 ? 0 : (n - start < per ? n - start : per);
    const unsigned lt = (1u << lane) - 1u;
    // g / per for g < 2^17, per <= 2^13 (exact: the excess of the reciprocal
    // times g stays below 2^32; per == 1 is a single key, 2^32 wraps to 0)
    const uint32_t recip = (uint32_t)(((1ull << 32) + per - 1) / per);
    const auto sync = [&] {
        if (C > 1) cluster.sync();
        else __syncthreads();
    };
    const auto at = [&](int g) -> uint64_t* {
        const int c = (int)__umulhi((uint32_t)g, recip);
        return cluster.map_shared_rank(s.words, c) + (g - c * per);
    };
    const auto half = [&](int g) { return (uint32_t)(*at(g) >> 32); };
    // A run of equal high halves that starts at g: its length up to
    // kTieWarp + 1, 0 if none starts here or it is one key.
    const auto run_at = [&](int g) {
        const uint32_t t = half(g);
        if (g + 1 >= n || half(g + 1) != t || (g > 0 && half(g - 1) == t)) return 0;
        int e = g + 2;
        while (e < n && e - g <= kTieRun && half(e) == t) ++e;
        if (e - g <= kTieRun || e == n || half(e) != t) return e - g;
        int end = n < g + kTieWarp + 1 ? n : g + kTieWarp + 1;  // e is in the run; [e + 1, end] holds its end
        for (++e; e < end;) {
            const int mid = (e + end) / 2;
            if (half(mid) == t) e = mid + 1;
            else end = mid;
        }
        return e - g;
    };

    for (int k = threadIdx.x; k < kCWarps * kRadix; k += kCThreads) (&s.warp_mask[0][0])[k] = 0;
    if (threadIdx.x == 0) s.runs = 0;
    if (kSample) {
        for (int k = threadIdx.x; k < kSampleSlots / 2; k += kCThreads) (&s.totals[0][0])[k] = 0;
        __syncthreads();
    }
    // Round 0 sorts by the high halves; rounds 1 and 2, where needed, by the
    // low and then by the high halves.
    for (int round = 0; round < 3; ++round) {
        uint32_t sample = 0;  // the high half of one of the thread's keys
        bool sampled = false;
#pragma unroll
        for (int k = 0; k < I; ++k) {
            const int i = k * kCThreads + threadIdx.x;
            if (i < cnt) {
                const uint32_t v = round == 2 ? (uint32_t)s.words[i] : (uint32_t)(start + i);
                const uint64_t key = keys_in[v];
                s.words[i] = (round == 1 ? key << 32 : key >> 32 << 32) | v;
                if (k == (int)(threadIdx.x % I)) {
                    sample = (uint32_t)(key >> 32);
                    sampled = true;
                }
            }
        }
        if (kSample && round == 0) {
            // Long ties show in a sample of one key in I, evenly spread: the
            // keys of a high half (or, rarely, of two that share a counter)
            // are then as many as half of kTieWarp neighbours would give.
            uint32_t* slots = &s.totals[0][0];
            const uint32_t h = sample * 0x9E3779B1u >> 19;
            static_assert(kSampleSlots == 1 << 13 && kCThreads < 1 << 16, "13 bits of the hash, 16-bit counters");
            if (sampled) atomicAdd(&slots[h >> 1], 1u << 16 * (h & 1));
            __syncthreads();
            const int count = sampled ? (int)(slots[h >> 1] >> 16 * (h & 1) & 0xFFFFu) : 0;
            const int tied = __syncthreads_or(I * count > kTieWarp / 2);
            if (threadIdx.x == 0) s.tied = tied;
        }
        sync();
        if (kSample && round == 0 && __syncthreads_or((int)threadIdx.x < C && *cluster.map_shared_rank(&s.tied, threadIdx.x)))
            continue;
        for (int shift = 32; shift < 64; shift += 8) {
            // Warp w holds positions w*32*I + k*32 + lane of the block.
            uint64_t word[I];
            uint16_t rank[I];
#pragma unroll
            for (int k = 0; k < I; ++k) {
                const int i = w * (32 * I) + k * 32 + lane;
                word[k] = i < cnt ? s.words[i] : 0;
            }
            for (int k = lane; k < kHistRow / 2; k += 32) reinterpret_cast<uint32_t*>(s.warp_hist[w])[k] = 0;
            __syncwarp();
#pragma unroll
            for (int k = 0; k < I; ++k)
                rank[k] = (uint16_t)rank_item((uint32_t)(word[k] >> shift) & 0xFFu,
                                              w * (32 * I) + k * 32 + lane < cnt, lt, lane, s.warp_mask[w],
                                              s.warp_hist[w]);
            __syncthreads();
            {
                // Four threads per digit: exclusive prefix over the warps,
                // and the block's count to every block.
                const int d = threadIdx.x >> 2, q = threadIdx.x & 3;
                uint32_t c[kCWarps / 4], sum = 0;
#pragma unroll
                for (int k = 0; k < kCWarps / 4; ++k) {
                    c[k] = s.warp_hist[q * (kCWarps / 4) + k][d];
                    sum += c[k];
                }
                uint32_t inc = sum;
                uint32_t y = __shfl_up_sync(0xffffffffu, inc, 1);
                if (q >= 1) inc += y;
                y = __shfl_up_sync(0xffffffffu, inc, 2);
                if (q >= 2) inc += y;
                uint32_t run = inc - sum;
#pragma unroll
                for (int k = 0; k < kCWarps / 4; ++k) {
                    s.warp_hist[q * (kCWarps / 4) + k][d] = (uint16_t)run;
                    run += c[k];
                }
                const uint32_t total = __shfl_sync(0xffffffffu, inc, lane | 3);
                for (int b = q; b < C; b += 4) cluster.map_shared_rank(&s.totals[0][0], b)[r * kRadix + d] = total;
            }
            sync();  // counts there; every block has its words in registers
            if (threadIdx.x < kRadix) {
                const int d = threadIdx.x;
                uint32_t before = 0, total = 0;
                for (int b = 0; b < C; ++b) {
                    const uint32_t v = s.totals[b][d];
                    if (b < r) before += v;
                    total += v;
                }
                s.base[d] = scan256(total, s.scan) + before;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < I; ++k) {
                if (w * (32 * I) + k * 32 + lane < cnt) {
                    const uint32_t d = (uint32_t)(word[k] >> shift) & 0xFFu;
                    *at((int)(s.base[d] + s.warp_hist[w][d] + rank[k])) = word[k];
                }
            }
            sync();
        }
        if (round != 0) continue;

        // Ties of the high halves: a thread looks for runs that start at its
        // positions.  flags: 1 up to kTieWarp long, 2 longer.  Runs above
        // kTieRun go to a list (in `totals`), for the warps.
        int f = 0;
        for (int i = threadIdx.x; i < cnt; i += kCThreads) {
            const int len = run_at(start + i);
            if (len) f |= len > kTieWarp ? 2 : 1;
            if (len > kTieRun && len <= kTieWarp)
                (&s.totals[0][0])[atomicAdd(&s.runs, 1)] = (uint32_t)(start + i) | (uint32_t)len << 17;
        }
        const int shorts = __syncthreads_or(f & 1), longs = __syncthreads_or(f & 2);
        if ((int)threadIdx.x < C)
            cluster.map_shared_rank(s.flags, threadIdx.x)[r] = (shorts ? 1 : 0) | (longs ? 2 : 0);
        sync();
        int any = 0;
        for (int b = 0; b < C; ++b) any |= s.flags[b];
        if (any >= 2) continue;
        if (any) {
            for (int i = threadIdx.x; i < cnt; i += kCThreads) {
                const int g = start + i, len = run_at(g);
                if (len > kTieRun) continue;
                for (int e = g + 1; e < g + len; ++e) {
                    const uint64_t x = *at(e);
                    const uint32_t xl = (uint32_t)keys_in[(uint32_t)x];
                    int j = e;
                    for (; j > g; --j) {
                        const uint64_t y = *at(j - 1);
                        if ((uint32_t)keys_in[(uint32_t)y] <= xl) break;
                        *at(j) = y;
                    }
                    *at(j) = x;
                }
            }
            // A warp to a run: a key's place is the number of keys before it,
            // by the low halves and then by the order they stand in.
            for (int k = w; k < s.runs; k += kCWarps) {
                const uint32_t run = (&s.totals[0][0])[k];
                const int g = (int)(run & 0x1FFFFu), len = (int)(run >> 17);
                uint32_t* low = s.warp_mask[w];
                constexpr int kPer = kTieWarp / 32;
                uint64_t x[kPer];
                uint32_t mine[kPer], place[kPer] = {};
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const int i = 32 * q + lane;
                    if (i >= len) continue;
                    x[q] = *at(g + i);
                    low[i] = mine[q] = (uint32_t)keys_in[(uint32_t)x[q]];
                }
                __syncwarp();
                for (int j = 0; j < len; ++j) {
                    const uint32_t v = low[j];
#pragma unroll
                    for (int q = 0; q < kPer; ++q) {
                        if (32 * q >= len) break;
                        if (32 * q + lane < len && (v < mine[q] || (v == mine[q] && j < 32 * q + lane))) ++place[q];
                    }
                }
#pragma unroll
                for (int q = 0; q < kPer; ++q)
                    if (32 * q + lane < len) *at(g + (int)place[q]) = x[q];
                __syncwarp();
            }
        }
        sync();
        break;
    }
    // keys_out may be keys_in: every block reads before any writes.
    uint64_t key[I];
#pragma unroll
    for (int k = 0; k < I; ++k) {
        const int i = k * kCThreads + threadIdx.x;
        if (i < cnt) key[k] = keys_in[(uint32_t)s.words[i]];
    }
    sync();
#pragma unroll
    for (int k = 0; k < I; ++k) {
        const int i = k * kCThreads + threadIdx.x;
        if (i < cnt) {
            keys_out[start + i] = key[k];
            vals_out[start + i] = (uint32_t)s.words[i];
        }
    }
}

template <int I>
int launch_cluster_sort_items(int n, int C, int per, const uint64_t* in, uint64_t* out, uint32_t* vals,
                              cudaStream_t stream)
{
    BH_CUDA_TRY(cudaFuncSetAttribute(cluster_sort_kernel<I>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(ClusterSmem)));
    if (C > kCPortable)
        BH_CUDA_TRY(cudaFuncSetAttribute(cluster_sort_kernel<I>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)C);
    cfg.blockDim = dim3(kCThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterSmem);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    BH_CUDA_TRY(cudaLaunchKernelEx(&cfg, cluster_sort_kernel<I>, n, per, in, out, vals));
    return BH_OK;
}

// Blocks of the current device's largest cluster: kCMax where it has room for
// one; asked once per device.
int cluster_blocks_max()
{
    static PerDevice most;
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    return most.get(dev, kCPortable, [] {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kCMax);
        cfg.blockDim = dim3(kCThreads);
        cfg.dynamicSmemBytes = sizeof(ClusterSmem);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = kCMax;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int clusters = 0;
        const bool fits =
            cudaFuncSetAttribute(cluster_sort_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(ClusterSmem)) == cudaSuccess &&
            cudaFuncSetAttribute(cluster_sort_kernel<8>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&clusters, cluster_sort_kernel<8>, &cfg) == cudaSuccess && clusters > 0;
        cudaGetLastError();
        return fits ? kCMax : kCPortable;
    });
}

// 1 <= n, !sort_uses_hist(n); in and out may be the same.
int launch_cluster_sort(int64_t n64, const uint64_t* in, uint64_t* out, uint32_t* vals, cudaStream_t stream)
{
    const int n = (int)n64, most = cluster_blocks_max();
    int C = 1;
    while (C < most && C * kCThreads < n) C *= 2;
    const int per = (n + C - 1) / C;
    if (per <= kCThreads) return launch_cluster_sort_items<1>(n, C, per, in, out, vals, stream);
    if (per <= 2 * kCThreads) return launch_cluster_sort_items<2>(n, C, per, in, out, vals, stream);
    if (per <= 3 * kCThreads) return launch_cluster_sort_items<3>(n, C, per, in, out, vals, stream);
    if (per <= 4 * kCThreads) return launch_cluster_sort_items<4>(n, C, per, in, out, vals, stream);
    if (per <= 6 * kCThreads) return launch_cluster_sort_items<6>(n, C, per, in, out, vals, stream);
    return launch_cluster_sort_items<8>(n, C, per, in, out, vals, stream);
}

constexpr int kPermThreads = 256;

// out[i] = in[perm[i]] for positions, velocities, masses and ids.
__global__ void __launch_bounds__(kPermThreads) permute_kernel(
    int64_t n, const uint32_t* __restrict__ perm, const double* __restrict__ px, const double* __restrict__ py,
    const double* __restrict__ pz, const double* __restrict__ vx, const double* __restrict__ vy,
    const double* __restrict__ vz, const double* __restrict__ m, const uint64_t* __restrict__ id,
    double* __restrict__ px2, double* __restrict__ py2, double* __restrict__ pz2, double* __restrict__ vx2,
    double* __restrict__ vy2, double* __restrict__ vz2, double* __restrict__ m2, uint64_t* __restrict__ id2)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t j = perm[i];
        if ((int64_t)j >= n) j = (uint32_t)i;  // only after a failed sort (error word set)
        px2[i] = px[j];
        py2[i] = py[j];
        pz2[i] = pz[j];
        vx2[i] = vx[j];
        vy2[i] = vy[j];
        vz2[i] = vz[j];
        m2[i] = m[j];
        id2[i] = id[j];
    }
}

}  // namespace

size_t sort_smem_bytes() { return sizeof(SortSmem); }

bool sort_uses_hist(int64_t n)
{
    const int64_t room = (int64_t)cluster_blocks_max() * kBlockKeys;
    return n > (room < kClusterSortMax ? room : kClusterSortMax);
}

int launch_sort(bh_context* ctx)
{
    const int64_t n = ctx->n;
    if (n <= 1) {
        if (n == 1) BH_CUDA_TRY(cudaMemsetAsync(ctx->perm, 0, sizeof(uint32_t), ctx->stream));
        return BH_OK;
    }
    if (!sort_uses_hist(n)) {
        const int rc = launch_cluster_sort(n, ctx->key, ctx->key, ctx->perm, ctx->stream);
        if (rc) return rc;
        BH_LAUNCH_CHECK(ctx);
        return BH_OK;
    }
    const size_t smem = sizeof(SortSmem);
    BH_CUDA_TRY(cudaFuncSetAttribute(onesweep_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    BH_CUDA_TRY(cudaFuncSetAttribute(onesweep_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    BH_CUDA_TRY(cudaMemsetAsync(ctx->lookback, 0, sizeof(uint32_t) * kSortPasses * tiles * kRadix, ctx->stream));
    BH_CUDA_TRY(cudaMemsetAsync(ctx->tile_ctr, 0, sizeof(uint32_t) * kSortPasses, ctx->stream));
    hist_scan_kernel<<<kSortPasses, kRadix, 0, ctx->stream>>>(ctx->hist);
    BH_LAUNCH_CHECK(ctx);
    uint64_t* kin = ctx->key;
    uint64_t* kout = ctx->key_alt;
    uint32_t* vin = ctx->perm;
    uint32_t* vout = ctx->perm_alt;
    for (int p = 0; p < kSortPasses; ++p) {
        uint32_t* lb = ctx->lookback + (size_t)p * tiles * kRadix;
        if (p == 0)
            onesweep_kernel<true><<<(unsigned)tiles, kTileThreads, smem, ctx->stream>>>(
                n, 8 * p, kin, vin, kout, vout, ctx->hist + p * kRadix, lb, ctx->tile_ctr + p, ctx->err);
        else
            onesweep_kernel<false><<<(unsigned)tiles, kTileThreads, smem, ctx->stream>>>(
                n, 8 * p, kin, vin, kout, vout, ctx->hist + p * kRadix, lb, ctx->tile_ctr + p, ctx->err);
        BH_LAUNCH_CHECK(ctx);
        uint64_t* tk = kin; kin = kout; kout = tk;
        uint32_t* tv = vin; vin = vout; vout = tv;
    }
    // After an even number of passes the result is back in key / perm.
    return BH_OK;
}

int sort_passes_raw(int64_t n, const uint64_t* keys_in, uint64_t* keys_out, uint32_t* vals_out, uint64_t* key_alt,
                    uint32_t* val_alt, uint32_t* hist, uint32_t* lookback, uint32_t* tile_ctr, unsigned* err,
                    cudaStream_t stream)
{
    // The eight onesweep passes over caller-provided buffers: digit starts
    // from `hist` (counts on entry), pass 0 reads keys_in and writes the
    // alternate buffers, the last pass writes keys_out / vals_out.  Where
    // !sort_uses_hist(n) only the three outer buffers are used.
    if (n > 0 && !sort_uses_hist(n)) return launch_cluster_sort(n, keys_in, keys_out, vals_out, stream);
    const size_t smem = sizeof(SortSmem);
    BH_CUDA_TRY(cudaFuncSetAttribute(onesweep_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    BH_CUDA_TRY(cudaFuncSetAttribute(onesweep_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    hist_scan_kernel<<<kSortPasses, kRadix, 0, stream>>>(hist);
    BH_CUDA_TRY(cudaGetLastError());
    const uint64_t* kin = keys_in;
    const uint32_t* vin = nullptr;
    for (int p = 0; p < kSortPasses; ++p) {
        const bool to_out = (p & 1) != 0;
        uint64_t* kout = to_out ? keys_out : key_alt;
        uint32_t* vout = to_out ? vals_out : val_alt;
        uint32_t* lb = lookback + (size_t)p * tiles * kRadix;
        if (p == 0)
            onesweep_kernel<true><<<(unsigned)tiles, kTileThreads, smem, stream>>>(
                n, 8 * p, kin, vin, kout, vout, hist + p * kRadix, lb, tile_ctr + p, err);
        else
            onesweep_kernel<false><<<(unsigned)tiles, kTileThreads, smem, stream>>>(
                n, 8 * p, kin, vin, kout, vout, hist + p * kRadix, lb, tile_ctr + p, err);
        BH_CUDA_TRY(cudaGetLastError());
        kin = kout;
        vin = vout;
    }
    return BH_OK;
}

int launch_permute(bh_context* ctx)
{
    const int64_t n = ctx->n;
    if (n == 0) return BH_OK;
    int64_t want = (n + kPermThreads - 1) / kPermThreads;
    const int blocks = (int)(want > 8 * bh::num_sms() ? 8 * bh::num_sms() : want);
    permute_kernel<<<blocks, kPermThreads, 0, ctx->stream>>>(n, ctx->perm, ctx->px, ctx->py, ctx->pz, ctx->vx, ctx->vy,
                                                             ctx->vz, ctx->m, ctx->id, ctx->px2, ctx->py2, ctx->pz2,
                                                             ctx->vx2, ctx->vy2, ctx->vz2, ctx->m2, ctx->id2);
    BH_LAUNCH_CHECK(ctx);
    swap_body_sets(ctx);
    return BH_OK;
}

void swap_body_sets(bh_context* ctx)
{
    std::swap(ctx->px, ctx->px2);
    std::swap(ctx->py, ctx->py2);
    std::swap(ctx->pz, ctx->pz2);
    std::swap(ctx->vx, ctx->vx2);
    std::swap(ctx->vy, ctx->vy2);
    std::swap(ctx->vz, ctx->vz2);
    std::swap(ctx->m, ctx->m2);
    std::swap(ctx->id, ctx->id2);
}

}  // namespace bh
