// Parallel bottom-up octree construction from the sorted Morton keys, with
// a level-synchronous monopole pass (no global atomics).
//
// Replaces buildOctreeBottomUp (src/linear_octree.cpp:13-107) followed by the
// single-rank full-tree exchange (src/exchange.cpp:9-29, whose effect is
// mergeRecordsIntoTree into an empty map, src/linear_octree.cpp:178-204).
//
// The reference's tree is uncompressed: every (depth, prefix) cell that holds
// a body exists, so most bodies hang below a chain of single-child cells.
// A single-child cell has exactly its child's mass and weighted position
// sums (the reference starts every sum at +0.0, and 0.0 + c == c for every c
// such a sum can hold), hence the same centre of mass.  This build therefore
// materialises only the cells with two or more children ("branching nodes")
// and the leaves; each stored node stands for the chain above it (depth
// range [top, depth]).  bh_export_tree expands the chains back into the
// reference's node set for parity checks.
//
// Terminology: leaves are the distinct keys K[0..L).  Boundary j (1 <= j < L)
// sits between leaves j-1 and j; cdep[j] is the deepest depth at which the
// two keys share a cell.  A branching node at depth D spanning leaves [a, e)
// has all interior boundaries with cdep >= D and at least one with
// cdep == D; its children are the depth-(D+1) cells inside it.  The node is
// identified by its first child boundary ("representative").
//
// Sums follow the reference's order exactly: a leaf sums its bodies in
// sorted order, a parent sums its children in octant order (= key order),
// each starting from 0.0; then com = sum/mass when mass > 0, then the merge
// step mass' = 0 + mass, com' = (0*0 + mass*com) / mass'.  All with IEEE
// double intrinsics (no contraction), so masses and centres of mass are bit
// for bit the reference's.
//
// Below some 100,000 bodies the launches bound the build (3 to 5 us each, and
// every stage needs the one before), so a stage carries what the next needs
// from it in its blocks' sums: the representatives' and children's numbers
// come from the resolve and split passes themselves, with no scans of their
// own.  Build per step, before -> after: 1,000 bodies 89 -> 60 us, 19,054
// 97 -> 72, 300,149 182 -> 123, 1M 257 -> 234, 4M 728 -> 707.
#include <climits>
#include <utility>

#include "bh_internal.cuh"

namespace bh {
namespace {

constexpr int kThreads = 256;

// 0.0 + v in round-to-nearest: v itself, except -0.0 -> +0.0.
__device__ __forceinline__ double plus_zero(double v)
{
    const long long b = __double_as_longlong(v);
    return __longlong_as_double(b == (long long)0x8000000000000000ull ? 0ll : b);
}

inline int grid_for(int64_t n, int threads, int max_blocks)
{
    int64_t b = (n + threads - 1) / threads;
    if (b < 1) b = 1;
    return (int)(b > max_blocks ? max_blocks : b);
}

// ---- Tree structure from the boundary depths ---------------------------
// With d(j) = cdep[j] for the boundaries 1 <= j < L and d(0) = d(L) = -1,
// the branching node that boundary j splits (the cell of depth d(j) holding
// leaves j-1 and j) spans the leaves [pl(j), pr(j)) between the nearest
// shallower boundaries
//   pl(j) = max{k < j : d(k) < d(j)},   pr(j) = min{k > j : d(k) < d(j)};
// its splits are the boundaries of depth d(j) in between (at most 7: eight
// octants), and the first of them represents it (j is first exactly when
// max{k < j : d(k) <= d(j)} is pl(j)).  next(j) = min{k > j : d(k) <= d(j)}
// is j's next split when d(next(j)) = d(j).  These nearest-value queries are
// answered per warp, block and grid: a query looks inside its own warp first
// (the lanes below its depth, from ballots on the depth's bits), then in the
// other warps of its block (prefix / suffix over the warps' last and first
// positions below each of the 22 thresholds t, d <= t - 1, t = 0..21), then
// in the other blocks (prefix / suffix over the blocks' extreme positions,
// from a pass over block summaries).  No searches and no atomics.
constexpr int kNT = kMaxDepth + 1;  // thresholds t: d <= t - 1
constexpr int kBT = 1024;           // boundary positions per block
constexpr int kBW = kBT / 32;
// Up to this many blocks the resolve pass scans the blocks' summaries itself
// instead of reading bnd_scan_kernel's result (a launch, about 3 us, against
// four loads a lane).
constexpr int kDirectBlocks = 128;

__device__ __forceinline__ int bnd_depth(const int8_t* __restrict__ cdep, int L, int64_t j)
{
    return j <= L ? (int)cdep[j] : 127;  // cdep[0] = cdep[L] = -1; past L: no threshold
}

// A warp's last and first position below each threshold t (v < t, i.e.
// d <= t - 1), into wl[t] and wf[t] (-1 / INT_MAX where none is): lane l is
// the last below t exactly for t in (v_l, min of the later lanes' v], and
// the first for t in (v_l, min of the earlier lanes' v]; thresholds up to
// the warp's minimum have neither.  Two min-scans and a short loop per lane
// instead of one ballot per threshold.
__device__ __forceinline__ void warp_threshold_ends(int v, int lane, int wbase, int* wl, int* wf)
{
    int suf = v, pre = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_down_sync(0xffffffffu, suf, off);
        if (lane + off < 32) suf = min(suf, y);
        const int z = __shfl_up_sync(0xffffffffu, pre, off);
        if (lane >= off) pre = min(pre, z);
    }
    int s_next = __shfl_down_sync(0xffffffffu, suf, 1);
    if (lane == 31) s_next = 127;
    int p_prev = __shfl_up_sync(0xffffffffu, pre, 1);
    if (lane == 0) p_prev = 127;
    const int wmin = __shfl_sync(0xffffffffu, pre, 31);
    if (lane < kNT && lane <= wmin) {
        wl[lane] = -1;
        wf[lane] = INT_MAX;
    }
    const int lo = v + 1;  // v >= -1
    for (int t = lo; t <= min(s_next, kNT - 1); ++t) wl[t] = wbase + lane;
    for (int t = lo; t <= min(p_prev, kNT - 1); ++t) wf[t] = wbase + lane;
}

// Leaf sums in body order (linear_octree.cpp:28-38), boundary depths, and per
// block, for every threshold, the last and the first position at or below it.
// A thread per boundary position; two blocks to an SM (32 registers) for the
// loads in flight: 107 us at 4M with one, 70 with two.
// kMoments: also the leaf's second moment about its centre of mass (the
// learned criterion's spread feature), sum_b m_b |x_b - c|^2.
// nzero > 0: the bodies with id < nzero count as massless (the FP32 forms'
// far-field tree, which leaves the Sun and planets to the direct terms).
template <bool kMoments>
__global__ void __launch_bounds__(kBT, 2) leaf_bnd_kernel(
    const int32_t* __restrict__ counts, const int32_t* __restrict__ leaf_first, const uint64_t* __restrict__ leaf_key,
    const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
    const double* __restrict__ m, const uint64_t* __restrict__ id, int nzero, double4_32a* __restrict__ ls,
    int8_t* __restrict__ cdep, double* __restrict__ lq, int32_t* __restrict__ blast, int32_t* __restrict__ bfirst)
{
    static_assert(kNT <= 32, "one lane per threshold");
    __shared__ int wl[kBW][kNT], wf[kBW][kNT];
    auto mass = [&](int b) { return nzero > 0 && id[b] < (uint64_t)nzero ? 0.0 : m[b]; };
    const int L = counts[0];
    const int64_t j = (int64_t)blockIdx.x * kBT + threadIdx.x;
    int v = 127;  // past the sentinel: no threshold
    if (j < L) {
        const int l = (int)j;
        double sm = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
        const int b0 = leaf_first[l], b1 = leaf_first[l + 1];
        v = l == 0 ? -1 : common_depth(leaf_key[l - 1], leaf_key[l]);
        cdep[l] = (int8_t)v;
        if (b1 == b0 + 1) {
            // One body: each sum is 0.0 + v, which is v except that -0.0
            // becomes +0.0; decided on the bit patterns (no FP64 addition).
            const double mb = mass(b0);
            sm = plus_zero(mb);
            sx = plus_zero(__dmul_rn(px[b0], mb));
            sy = plus_zero(__dmul_rn(py[b0], mb));
            sz = plus_zero(__dmul_rn(pz[b0], mb));
        } else {
#pragma unroll 1
            for (int b = b0; b < b1; ++b) {
                const double mb = mass(b);
                sm = __dadd_rn(sm, mb);
                sx = __dadd_rn(sx, __dmul_rn(px[b], mb));
                sy = __dadd_rn(sy, __dmul_rn(py[b], mb));
                sz = __dadd_rn(sz, __dmul_rn(pz[b], mb));
            }
        }
        ls[l] = double4_32a{sx, sy, sz, sm};
        if (kMoments) {
            double q = 0.0;
            if (b1 - b0 > 1 && sm > 0) {
                const double is = rcp_nr(sm);
                const double cx = sx * is, cy = sy * is, cz = sz * is;
#pragma unroll 1
                for (int b = b0; b < b1; ++b) {
                    const double dx = px[b] - cx, dy = py[b] - cy, dz = pz[b] - cz;
                    q += mass(b) * (dx * dx + dy * dy + dz * dz);
                }
            }
            lq[l] = q;
        }
    } else if (j == L) {
        v = -1;  // right sentinel of the boundary pass
        cdep[L] = -1;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wbase = (int)(j - lane);
    warp_threshold_ends(v, lane, wbase, wl[w], wf[w]);
    __syncthreads();
    // Warp t reduces threshold t over the block's warps (lane = warp).
    static_assert(kBW == 32 && kNT <= kBW, "one lane per warp, one warp per threshold");
    if (w < kNT) {
        const int t = w;
        int l = wl[lane][t], f = wf[lane][t];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            l = max(l, __shfl_xor_sync(0xffffffffu, l, off));
            f = min(f, __shfl_xor_sync(0xffffffffu, f, off));
        }
        if (lane == 0) {
            blast[(int64_t)blockIdx.x * kNT + t] = l;
            bfirst[(int64_t)blockIdx.x * kNT + t] = f;
        }
    }
}

// Exclusive scan of one int per thread over the block (max, or min with
// kMin), continued from `carry`; returns the thread's exclusive value and
// advances `carry` past the whole block.
template <bool kMin>
__device__ int block_excl_extreme(int x, int& carry, int* wsum)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    auto op = [](int a, int b) { return kMin ? min(a, b) : max(a, b); };
    const int ident = kMin ? INT_MAX : -1;
    int inc = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc = op(inc, y);
    }
    int ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = ident;
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    if (w == 0) {
        int sw = lane < (int)(blockDim.x >> 5) ? wsum[lane] : ident;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, sw, off);
            if (lane >= off) sw = op(sw, y);
        }
        wsum[lane] = sw;
    }
    __syncthreads();
    const int res = op(carry, op(w ? wsum[w - 1] : ident, ex));
    carry = op(carry, wsum[(blockDim.x >> 5) - 1]);
    __syncthreads();
    return res;
}

// Two blocks per threshold: the blocks' exclusive prefix of last positions
// (max; blocks 0..kNT-1) and exclusive suffix of first positions (min;
// blocks kNT..2 kNT-1).
__global__ void __launch_bounds__(1024) bnd_scan_kernel(int nblk, const int32_t* __restrict__ blast,
                                                        const int32_t* __restrict__ bfirst,
                                                        int32_t* __restrict__ bpre, int32_t* __restrict__ bsuf)
{
    __shared__ int wsum[32];
    const int t = blockIdx.x % kNT;
    if (blockIdx.x < kNT) {
        int carry = -1;
        for (int base = 0; base < nblk; base += blockDim.x) {
            const int b = base + threadIdx.x;
            const int x = b < nblk ? blast[(int64_t)b * kNT + t] : -1;
            const int ex = block_excl_extreme<false>(x, carry, wsum);
            if (b < nblk) bpre[(int64_t)b * kNT + t] = ex;
        }
    } else {
        int carry = INT_MAX;
        for (int base = 0; base < nblk; base += blockDim.x) {
            const int b = nblk - 1 - (base + (int)threadIdx.x);
            const int x = b >= 0 ? bfirst[(int64_t)b * kNT + t] : INT_MAX;
            const int ex = block_excl_extreme<true>(x, carry, wsum);
            if (b >= 0) bsuf[(int64_t)b * kNT + t] = ex;
        }
    }
}

// Per boundary: the representative flag (flag[j], 0 for j = 0 and j >= L up
// to cap), pl, pr and next; per block the number of representatives.
// scanned: blast / bfirst hold bnd_scan_kernel's prefixes and suffixes; else
// the blocks' own positions, which the block scans for itself.
__global__ void __launch_bounds__(kBT) bnd_resolve_kernel(const int32_t* __restrict__ counts,
                                                          const int8_t* __restrict__ cdep,
                                                          const int32_t* __restrict__ blast,
                                                          const int32_t* __restrict__ bfirst, int scanned,
                                                          int32_t* __restrict__ flag, int32_t* __restrict__ pl,
                                                          int32_t* __restrict__ pr, int32_t* __restrict__ nxt,
                                                          int32_t* __restrict__ bsum, int64_t cap)
{
    __shared__ int wl[kBW][kNT], wf[kBW][kNT];
    const int L = counts[0];
    const int64_t j = (int64_t)blockIdx.x * kBT + threadIdx.x;
    const int v = bnd_depth(cdep, L, j);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int wbase = (int)(j - lane);
    warp_threshold_ends(v, lane, wbase, wl[w], wf[w]);
    // Inside the warp: the lanes whose depth is below this lane's (LT) and
    // at or below it (LE), from five ballots on the bits of v + 1 (past the
    // end, v = 127, counts as 30: above every depth).
    const int vq = min(v, 30) + 1;
    unsigned lt_m = 0u, eq_m = 0xffffffffu;
#pragma unroll
    for (int k = 4; k >= 0; --k) {
        const bool bit = (vq >> k) & 1;
        const unsigned b = __ballot_sync(0xffffffffu, bit);
        if (bit) {
            lt_m |= eq_m & ~b;
            eq_m &= b;
        } else {
            eq_m &= ~b;
        }
    }
    const unsigned le_m = lt_m | eq_m;
    __syncthreads();
    // Each warp's answer from outside it: exclusive prefix (max) and suffix
    // (min) over the warps, started from the other blocks'.  Warp t scans
    // threshold t, one lane per warp of the block.
    if (w < kNT) {
        const int t = w;
        int inc = wl[lane][t];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc = max(inc, y);
        }
        int ex = __shfl_up_sync(0xffffffffu, inc, 1);
        if (lane == 0) ex = -1;
        int before = -1, after = INT_MAX;
        if (scanned) {
            before = blast[(int64_t)blockIdx.x * kNT + t];
            after = bfirst[(int64_t)blockIdx.x * kNT + t];
        } else {
            for (int b = lane; b < (int)gridDim.x; b += 32) {
                if (b < (int)blockIdx.x) before = max(before, blast[b * kNT + t]);
                if (b > (int)blockIdx.x) after = min(after, bfirst[b * kNT + t]);
            }
            before = __reduce_max_sync(0xffffffffu, before);
            after = __reduce_min_sync(0xffffffffu, after);
        }
        wl[lane][t] = max(before, ex);
        int sinc = wf[lane][t];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_down_sync(0xffffffffu, sinc, off);
            if (lane + off < 32) sinc = min(sinc, y);
        }
        int sex = __shfl_down_sync(0xffffffffu, sinc, 1);
        if (lane == 31) sex = INT_MAX;
        wf[lane][t] = min(after, sex);
    }
    __syncthreads();
    int f = 0;
    if (j >= 1 && j < L) {
        const unsigned below = (1u << lane) - 1u, above = ~below & ~(1u << lane);
        auto prev = [&](unsigned mask, int t) {
            const unsigned m = mask & below;
            return m ? wbase + 31 - __clz(m) : wl[w][t];
        };
        auto next = [&](unsigned mask, int t) {
            const unsigned m = mask & above;
            return m ? wbase + __ffs(m) - 1 : wf[w][t];
        };
        const int PL = prev(lt_m, v), PLE = prev(le_m, v + 1);
        f = PLE == PL ? 1 : 0;
        pl[j] = PL;
        pr[j] = next(lt_m, v);
        nxt[j] = next(le_m, v + 1);
    }
    if (j < cap) flag[j] = f;
    const int reps = __syncthreads_count(f);
    if (threadIdx.x == 0) bsum[blockIdx.x] = reps;
}

// Each branching node from its representative (a thread per boundary; node
// ids count the representatives, so the blocks' numbers before come from
// bnd_resolve_kernel's sums): depth, leaf range and its splits (at most 7)
// with their ranks; child count = splits + 1, its first child's place among
// the children of the block's nodes (cs), and the block's child count (csum).
__global__ void __launch_bounds__(kBT) node_split_kernel(
    int32_t* counts, const int8_t* __restrict__ cdep, const int32_t* __restrict__ flag,
    const int32_t* __restrict__ bsum, const int32_t* __restrict__ pl, const int32_t* __restrict__ pr,
    const int32_t* __restrict__ nxt, int32_t* __restrict__ rep_node, int32_t* __restrict__ node_rep,
    int32_t* __restrict__ node_a, int32_t* __restrict__ node_e, uint8_t* __restrict__ node_depth,
    int32_t* __restrict__ node_nchild, int32_t* __restrict__ split_node, int8_t* __restrict__ split_rank,
    int32_t* __restrict__ cs, int32_t* __restrict__ csum, unsigned* __restrict__ err)
{
    static_assert(kBW == 32, "one lane per warp");
    __shared__ int w_before[kBW], w_reps[kBW], w_children[kBW];
    const int L = counts[0];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t jj = (int64_t)blockIdx.x * kBT + threadIdx.x;
    const bool rep = jj >= 1 && jj < L && flag[jj];
    const unsigned reps = __ballot_sync(0xffffffffu, rep);
    int before = 0;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += kBT) before += bsum[k];
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) {
        w_before[w] = before;
        w_reps[w] = __popc(reps);
    }
    __syncthreads();
    before = __reduce_add_sync(0xffffffffu, w_before[lane] + (lane < w ? w_reps[lane] : 0));
    const int b = before + __popc(reps & ((1u << lane) - 1u));
    int children = 0;
    if (jj < L) {
        const int j = (int)jj;
        rep_node[j] = b;
        if (rep) {
            const int c = cdep[j];
            node_rep[b] = j;
            node_a[b] = pl[j];
            node_e[b] = pr[j];
            node_depth[b] = (uint8_t)c;
            int k = j, r = 0;
            for (;;) {
                split_node[k] = b;
                split_rank[k] = (int8_t)r;
                ++r;
                k = nxt[k];
                if (k >= L || cdep[k] != c || r >= 7) break;
            }
            if (k < L && cdep[k] == c) atomicOr(err, kErrOverflow);  // an eighth split: impossible for an octree
            children = r + 1;
            node_nchild[b] = children;
        }
    }
    int inc = children;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += y;
    }
    if (lane == 31) w_children[w] = inc;
    __syncthreads();
    const int ahead = __reduce_add_sync(0xffffffffu, lane < w ? w_children[lane] : 0);
    if (rep) cs[b] = ahead + inc - children;
    if (threadIdx.x == kBT - 1) {
        csum[blockIdx.x] = ahead + inc;
        if (blockIdx.x == gridDim.x - 1) counts[1] = b + (rep ? 1 : 0);
    }
}

// The sum of the blocks' child counts before each block, for node_place_kernel
// where its blocks don't form it for themselves; one block.
__global__ void __launch_bounds__(1024) child_offset_kernel(int nb, int32_t* __restrict__ csum)
{
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int carry = 0;
    for (int base = 0; base < nb; base += 1024) {
        const int k = base + (int)threadIdx.x;
        const int x = k < nb ? csum[k] : 0;
        int inc = x;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += y;
        }
        if (lane == 31) wsum[w] = inc;
        __syncthreads();
        const int ahead = __reduce_add_sync(0xffffffffu, lane < w ? wsum[lane] : 0);
        const int total = __reduce_add_sync(0xffffffffu, wsum[lane]);
        if (k < nb) csum[k] = carry + ahead + inc - x;
        carry += total;
        __syncthreads();
    }
    if (threadIdx.x == 0) csum[nb] = carry;
}

// Child slots: every leaf and branching node finds its parent from the
// boundaries at its two ends (the deeper one splits the parent; both
// sentinels: the root) and its place among the parent's children from that
// split's rank.  Slot 0 is the root.  A node's first child slot (node_cs) is
// its place in its block (cs) behind the children of the blocks before, which
// every block here sums from csum first (kOffBlocks of them at most; beyond,
// child_offset_kernel has).
constexpr int kOffBlocks = 4096;

__global__ void __launch_bounds__(kThreads) node_place_kernel(
    int32_t* counts, const int8_t* __restrict__ cdep, const int32_t* __restrict__ node_a,
    const int32_t* __restrict__ node_e, const uint8_t* __restrict__ node_depth, const int32_t* __restrict__ node_rep,
    const int32_t* __restrict__ cs, const int32_t* __restrict__ csum, int nb, int32_t* __restrict__ node_cs,
    const int32_t* __restrict__ split_node, const int8_t* __restrict__ split_rank, int32_t* __restrict__ slot_ref,
    uint8_t* __restrict__ slot_top, unsigned* __restrict__ err)
{
    __shared__ int off_s[kOffBlocks];
    __shared__ int wsum[kThreads / 32];
    const bool own = nb <= kOffBlocks;
    int total;
    if (own) {
        // Thread t takes the blocks [t q, t q + q).
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        const int q = (nb + kThreads - 1) / kThreads, k0 = (int)threadIdx.x * q, k1 = min(k0 + q, nb);
        int sum = 0;
        for (int k = k0; k < k1; ++k) sum += csum[k];
        int inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) wsum[w] = inc;
        __syncthreads();
        int run = inc - sum;
        total = 0;
        for (int k = 0; k < kThreads / 32; ++k) {
            if (k < w) run += wsum[k];
            total += wsum[k];
        }
        for (int k = k0; k < k1; ++k) {
            off_s[k] = run;
            run += csum[k];
        }
        __syncthreads();
    } else {
        total = csum[nb];
    }
    const int* off = own ? off_s : csum;
    const auto first_child = [&](int b) { return cs[b] + off[node_rep[b] / kBT]; };
    const int L = counts[0], B = counts[1], S = total + 1;  // the root and every child
    if (blockIdx.x == 0 && threadIdx.x == 0) counts[2] = S;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < L + B; i += gridDim.x * blockDim.x) {
        int a, e, ref;
        if (i < L) {
            a = i; e = i + 1; ref = i;
        } else {
            const int b = i - L;
            a = node_a[b]; e = node_e[b]; ref = ~b;
            node_cs[b] = first_child(b);
        }
        const int ca = a == 0 ? -1 : cdep[a];
        const int ce = e >= L ? -1 : cdep[e];
        int P = -1, s = 0, top = 0;
        if (ca >= 0 || ce >= 0) {
            const bool left = ca >= ce;
            const int k = left ? a : e;
            P = split_node[k];
            if ((unsigned)P >= (unsigned)B) {  // every boundary splits a node: a broken invariant
                atomicOr(err, kErrOverflow);
                continue;
            }
            s = first_child(P) + 1 + split_rank[k] + (left ? 1 : 0);
            top = node_depth[P] + 1;
            if (s < 1 || s >= S) {
                atomicOr(err, kErrOverflow);
                continue;
            }
        }
        slot_ref[s] = ref;
        slot_top[s] = (uint8_t)top;
    }
}

// ---- Monopole pass ------------------------------------------------------
// Every branching node's sums from its children's, in slot (= octant) order
// from 0.0 (linear_octree.cpp:69-87), deepest level first.  A block takes
// kChunk consecutive leaves and all the nodes inside them: it sorts those by
// depth and works up level by level in shared memory, with a block barrier
// between levels.  The nodes that reach past the chunk (at most 21 around each
// end) are left for the next stage, whose blocks take kFan chunks each, and so
// on until one block holds the rest.  No atomics on global memory, and two
// launches up to 32,768 bodies or three up to two million, where one launch
// per depth took 21, and three more to sort the nodes by depth.  Bound: the
// FP64 additions (a node has 3.3 children on average) and, in the later
// stages, their latency.  The whole build, ms: 4,000,000 bodies 0.81 -> 0.73,
// 1,000,000 with second moments 0.51 -> 0.41, 300,149 0.28 -> 0.18, 19,054
// 0.20 -> 0.10, 1,000 0.17 -> 0.09.  512 leaves per block: 256 and 1,024 gave
// the same within 3 %.
constexpr int kChunk = 512;          // leaves per block of the first stage
constexpr int kChunkThreads = 256;
constexpr int kFan = 64;             // groups per block of a later stage
constexpr int kRestThreads = 512;
constexpr int kRestItems = 384;      // nodes of a later stage's block with their sums in shared memory
constexpr int kMaxSpan = 2 * kMaxDepth;  // nodes left over per group
constexpr int kDepths = kMaxDepth;       // branching depths 0..20

__device__ __forceinline__ double4_32a load_sums(const double4_32a* p)
{
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    return double4_32a{a.x, a.y, b.x, b.y};
}

// acc + child, the first child's 0.0 + v decided on the bit patterns.
__device__ __forceinline__ double add_sum(double acc, double v, bool first)
{
    return first ? plus_zero(v) : __dadd_rn(acc, v);
}
__device__ __forceinline__ void add_sums(double4_32a& acc, const double4_32a& v, bool first)
{
    acc.x = add_sum(acc.x, v.x, first);
    acc.y = add_sum(acc.y, v.y, first);
    acc.z = add_sum(acc.z, v.z, first);
    acc.w = add_sum(acc.w, v.w, first);
}

// Four consecutive lanes work on a node: one sum each (a dependent FP64
// addition takes about 100 cycles here, so a level's time is its longest chain;
// one lane with the four sums takes up to four times as long).  The second
// moment's terms are formed four children at a time and added by each lane.
__device__ __forceinline__ double quad_get(double v, int j)  // lane j's of the four
{
    const int lane = threadIdx.x & 31;
    return __shfl_sync(0xFu << (lane & 28), v, (lane & 28) + j);
}

// A node's second moment by the parallel-axis rule, one child's share:
// m_c |c_c - c|^2 = |w_c - m_c c|^2 / m_c: u = w_c - m_c c by FMA keeps the
// cancellation in FP64; the division by m_c needs only the feature's precision
// (an FP32 reciprocal, 2^-22).  Masses are >= 0, so "> 0" is a test on the bit
// pattern.
__device__ __forceinline__ double moment_uu(const double4_32a& v, double gx, double gy, double gz)  // |u|^2
{
    const double ux = fma(-v.w, gx, v.x), uy = fma(-v.w, gy, v.y), uz = fma(-v.w, gz, v.z);
    return fma(ux, ux, fma(uy, uy, uz * uz));
}
__device__ __forceinline__ double moment_add(double uu, double mass, double cq)
{
    if (__double_as_longlong(mass) <= 0) return 0.0;
    return fma(uu, widen(__frcp_rn(narrow_trunc(mass))), cq);
}
__device__ __forceinline__ double moment_share(const double4_32a& v, double cq, double gx, double gy, double gz)
{
    return moment_add(moment_uu(v, gx, gy, gz), v.w, cq);
}

// The order a block takes its nodes in: deepest first, and within a depth by
// child count, so that the lanes of a warp add equally many children (the FP64
// pipe takes an addition for one lane as long as for 32).
constexpr int kBins = 8 * kDepths;
__device__ __forceinline__ int bin_of(int depth, int nchild) { return 8 * (kDepths - 1 - depth) + (8 - nchild); }

// Exclusive prefix of the bin counts (and the total behind it), by warp 0.
__device__ __forceinline__ void bin_offsets(const int* cnt, int* off)
{
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int carry = 0;
        for (int base = 0; base < kBins; base += 32) {
            const int v = base + lane < kBins ? cnt[base + lane] : 0;
            int x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (base + lane < kBins) off[base + lane] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) off[kBins] = carry;
    }
}

template <bool kMoments>
struct ChunkSmem {
    double4_32a leaf[kChunk];
    double4_32a node[kChunk];
    double uu[kMoments ? 2 * kChunk + 8 * kMaxSpan : 1];  // per child slot
    int child[2 * kChunk + 8 * kMaxSpan];  // child slots' refs of the chunk's nodes
    int cs[kChunk + 1];                    // first child of each node in `child`
    uint16_t order[kChunk];                // local nodes, deepest first
    int cnt[kBins], pos[kBins], off[kBins + 1];
    int span;
};

template <bool kMoments>
__global__ void __launch_bounds__(kChunkThreads) monopole_chunk_kernel(
    const int32_t* __restrict__ counts, const int32_t* __restrict__ rep_node, const int32_t* __restrict__ node_a,
    const int32_t* __restrict__ node_e, const uint8_t* __restrict__ node_depth, const int32_t* __restrict__ node_cs,
    const int32_t* __restrict__ node_nchild, const int32_t* __restrict__ slot_ref, const double4_32a* __restrict__ ls,
    double4_32a* __restrict__ ns, const double* __restrict__ lq, double* __restrict__ nq,
    int32_t* __restrict__ span_cnt, int32_t* __restrict__ span)
{
    extern __shared__ __align__(32) unsigned char smem_raw[];
    ChunkSmem<kMoments>& m = *reinterpret_cast<ChunkSmem<kMoments>*>(smem_raw);
    const int L = counts[0], B = counts[1];
    const int c0 = blockIdx.x * kChunk, c1 = min(c0 + kChunk, L);
    if (c0 >= L) {
        if (threadIdx.x == 0) span_cnt[blockIdx.x] = 0;
        return;
    }
    // The nodes whose first split lies in the chunk (numbered in that order).
    const int n0 = rep_node[c0], n1 = c1 < L ? rep_node[c1] : B;
    const int nn = n1 - n0;
    for (int k = threadIdx.x; k < c1 - c0; k += kChunkThreads) {
        m.leaf[k] = ls[c0 + k];
    }
    for (int k = threadIdx.x; k < kBins; k += kChunkThreads) m.cnt[k] = m.pos[k] = 0;
    if (threadIdx.x == 0) m.span = 0;
    __syncthreads();
    const int s0 = nn > 0 ? node_cs[n0] : 0;
    int bin[kChunk / kChunkThreads];  // -1: not a node inside the chunk
#pragma unroll
    for (int q = 0; q < kChunk / kChunkThreads; ++q) {
        const int k = threadIdx.x + q * kChunkThreads;
        bin[q] = -1;
        if (k < nn) {
            const int b = n0 + k, f = node_cs[b], nc = node_nchild[b];
            m.cs[k] = f - s0;
            if (k == nn - 1) m.cs[nn] = f - s0 + nc;
            if (node_a[b] >= c0 && node_e[b] <= c1) {
                bin[q] = bin_of(node_depth[b], nc);
                atomicAdd(&m.cnt[bin[q]], 1);
            } else {
                const int at = atomicAdd(&m.span, 1);
                if (at < kMaxSpan) span[(int64_t)blockIdx.x * kMaxSpan + at] = b;
            }
        }
    }
    __syncthreads();
    bin_offsets(m.cnt, m.off);
    if (threadIdx.x == 0) span_cnt[blockIdx.x] = min(m.span, kMaxSpan);
    const int children = nn > 0 ? m.cs[nn] : 0;
    for (int k = threadIdx.x; k < children; k += kChunkThreads) m.child[k] = slot_ref[s0 + 1 + k];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kChunk / kChunkThreads; ++q)
        if (bin[q] >= 0)
            m.order[m.off[bin[q]] + atomicAdd(&m.pos[bin[q]], 1)] = (uint16_t)(threadIdx.x + q * kChunkThreads);
    __syncthreads();
    for (int level = 0; level < kDepths; ++level) {
        const int lo = m.off[8 * level], hi = m.off[8 * level + 8];
        if (lo == hi) continue;
        for (int t = 4 * lo + threadIdx.x; t < 4 * hi; t += kChunkThreads) {
            const int k = m.order[t >> 2];
            const int f = m.cs[k], e = m.cs[k + 1];
            double sum = 0.0;
            for (int c = f; c < e; ++c) {
                const int r = m.child[c];
                sum = add_sum(sum, (r >= 0 ? &m.leaf[r - c0].x : &m.node[~r - n0].x)[t & 3], c == f);
            }
            (&m.node[k].x)[t & 3] = sum;
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < kChunk / kChunkThreads; ++q) {
        const int k = threadIdx.x + q * kChunkThreads;
        if (bin[q] >= 0) ns[n0 + k] = m.node[k];
    }
    if (kMoments) {
        // The distances of the children from the centres need only the sums:
        // all nodes at once, with full warps.  Then the moments themselves,
        // level by level, in place of the sums' x.
        for (int t = threadIdx.x; t < m.off[kBins]; t += kChunkThreads) {
            const int k = m.order[t];
            const double4_32a sum = m.node[k];
            if (__double_as_longlong(sum.w) <= 0) continue;
            const double is = rcp_nr(sum.w);
            const double gx = sum.x * is, gy = sum.y * is, gz = sum.z * is;
            for (int c = m.cs[k]; c < m.cs[k + 1]; ++c) {
                const int r = m.child[c];
                m.uu[c] = moment_uu(r >= 0 ? m.leaf[r - c0] : m.node[~r - n0], gx, gy, gz);
            }
        }
        __syncthreads();
        for (int k = threadIdx.x; k < c1 - c0; k += kChunkThreads) m.leaf[k].x = lq[c0 + k];
        __syncthreads();
        for (int level = 0; level < kDepths; ++level) {
            const int lo = m.off[8 * level], hi = m.off[8 * level + 8];
            if (lo == hi) continue;
            for (int t = 4 * lo + threadIdx.x; t < 4 * hi; t += kChunkThreads) {
                const int k = m.order[t >> 2], j = t & 3;
                double q = 0.0;
                if (__double_as_longlong(m.node[k].w) > 0) {
                    const int f = m.cs[k], e = m.cs[k + 1];
                    for (int c = f; c < e; c += 4) {
                        double share = 0.0;
                        if (c + j < e) {
                            const int r = m.child[c + j];
                            const double4_32a& v = r >= 0 ? m.leaf[r - c0] : m.node[~r - n0];
                            share = moment_add(m.uu[c + j], v.w, v.x);
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const double x = quad_get(share, i);
                            if (c + i < e) q += x;
                        }
                    }
                }
                if (j == 0) {
                    m.node[k].x = q;
                    nq[n0 + k] = q;
                }
            }
            __syncthreads();
        }
    }
}

// A node's sums (and second moment) from its children's in memory, for the
// nodes of a later stage that do not fit its table.
template <bool kMoments>
__device__ __noinline__ void node_sums(int b, const int32_t* __restrict__ node_cs,
                                       const int32_t* __restrict__ node_nchild, const int32_t* __restrict__ slot_ref,
                                       const double4_32a* ls, double4_32a* ns, const double* lq, double* nq)
{
    const int s0 = node_cs[b] + 1, nc = node_nchild[b];
    double4_32a sum;
    for (int c = 0; c < nc; ++c) {
        const int r = slot_ref[s0 + c];
        add_sums(sum, load_sums(r >= 0 ? ls + r : ns + ~r), c == 0);
    }
    ns[b] = sum;
    if (kMoments) {
        double q = 0.0;
        if (__double_as_longlong(sum.w) > 0) {
            const double is = rcp_nr(sum.w);
            const double gx = sum.x * is, gy = sum.y * is, gz = sum.z * is;
            for (int c = 0; c < nc; ++c) {
                const int r = slot_ref[s0 + c];
                q += moment_share(load_sums(r >= 0 ? ls + r : ns + ~r), __ldcg(r >= 0 ? lq + r : nq + ~r), gx, gy, gz);
            }
        }
        nq[b] = q;
    }
}

// A later stage: the nodes left over by kFan groups of `leaves` leaves each.
// Children whose sums are known already (leaves, nodes of earlier stages) are
// loaded before the levels begin, the others' come through shared memory, so
// that a level waits for no memory.  node_item: scratch, the place of a node in the order.
template <bool kMoments>
struct RestSmem {
    double4_32a sum[kRestItems];  // (kMoments: then the second moment in x)
    int32_t order[kFan * kMaxSpan];  // local nodes, in bin order
    int cnt[kBins], pos[kBins], off[kBins + 1], spans;
};

template <bool kMoments>
__global__ void __launch_bounds__(kRestThreads) monopole_rest_kernel(
    const int32_t* __restrict__ counts, int groups, int64_t leaves, const int32_t* __restrict__ in_cnt,
    const int32_t* __restrict__ in, const int32_t* __restrict__ node_a, const int32_t* __restrict__ node_e,
    const uint8_t* __restrict__ node_depth, const int32_t* __restrict__ node_cs,
    const int32_t* __restrict__ node_nchild, const int32_t* __restrict__ slot_ref, const double4_32a* ls,
    double4_32a* ns, const double* lq, double* nq, int32_t* node_item, int32_t* __restrict__ span_cnt,
    int32_t* __restrict__ span)
{
    static_assert(kRestThreads % kFan == 0, "equal shares of a list");
    extern __shared__ __align__(32) unsigned char smem_raw[];
    RestSmem<kMoments>& m = *reinterpret_cast<RestSmem<kMoments>*>(smem_raw);
    const int L = counts[0];
    const int64_t c0 = (int64_t)blockIdx.x * kFan * leaves;
    const int64_t c1 = min((int64_t)L, c0 + kFan * leaves);
    for (int k = threadIdx.x; k < kBins; k += kRestThreads) m.cnt[k] = m.pos[k] = 0;
    if (threadIdx.x == 0) m.spans = 0;
    __syncthreads();
    // Thread t reads every (kRestThreads / kFan)th entry of list t % kFan.
    const int g = blockIdx.x * kFan + threadIdx.x % kFan;
    const int entries = g < groups ? in_cnt[g] : 0;
    const int32_t* list = in + (int64_t)g * kMaxSpan;
    auto place = [&](int b) { return node_a[b] >= c0 && node_e[b] <= c1 ? bin_of(node_depth[b], node_nchild[b]) : -1; };
    for (int e = threadIdx.x / kFan; e < entries; e += kRestThreads / kFan) {
        const int b = list[e], bin = place(b);
        if (bin >= 0) {
            atomicAdd(&m.cnt[bin], 1);
        } else {
            const int at = atomicAdd(&m.spans, 1);
            if (at < kMaxSpan) span[(int64_t)blockIdx.x * kMaxSpan + at] = b;
        }
    }
    __syncthreads();
    bin_offsets(m.cnt, m.off);
    if (threadIdx.x == 0) span_cnt[blockIdx.x] = min(m.spans, kMaxSpan);
    __syncthreads();
    for (int e = threadIdx.x / kFan; e < entries; e += kRestThreads / kFan) {
        const int b = list[e], bin = place(b);
        if (bin >= 0) {
            const int k = m.off[bin] + atomicAdd(&m.pos[bin], 1);
            m.order[k] = b;
            node_item[b] = k;
        }
    }
    __syncthreads();
    // Lane j of four takes component j of the items (thread / 4) + i kQuads.
    constexpr int kQuads = kRestThreads / 4, kItems = kRestItems / kQuads;
    const int j = threadIdx.x & 3, quad = threadIdx.x >> 2, total = m.off[kBins];
    const bool fits = total <= kRestItems;
    int node[kItems], nc[kItems];
    double v[kItems][8] = {};        // the children's component j
    int16_t src[kItems][8];          // child c: its place in the order, or -1 with v[c] loaded
    double cq[kMoments ? kItems : 1][2];  // second moments of children j and j + 4
    if (fits) {
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            const int k = quad + i * kQuads;
            node[i] = nc[i] = 0;
            if (k >= total) continue;
            node[i] = m.order[k];
            nc[i] = node_nchild[node[i]];
            const int s0 = node_cs[node[i]] + 1;
            int ref[8], at[8];
#pragma unroll
            for (int c = 0; c < 8; ++c) ref[c] = c < nc[i] ? slot_ref[s0 + c] : 0;
#pragma unroll
            for (int c = 0; c < 8; ++c) at[c] = c < nc[i] && ref[c] < 0 ? __ldcg(node_item + ~ref[c]) : -1;
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                // (node_item of a node of another stage or block is stale)
                if ((unsigned)at[c] >= (unsigned)total || m.order[at[c]] != ~ref[c]) at[c] = -1;
                src[i][c] = (int16_t)at[c];
                if (c < nc[i] && at[c] < 0)
                    v[i][c] = __ldcg(&(ref[c] >= 0 ? ls + ref[c] : ns + ~ref[c])->x + j);
                if (kMoments && c < nc[i] && at[c] < 0 && (c & 3) == j)
                    cq[i][c >> 2] = __ldcg(ref[c] >= 0 ? lq + ref[c] : nq + ~ref[c]);
            }
        }
    }
    for (int level = 0; level < kDepths; ++level) {
        const int lo = m.off[8 * level], hi = m.off[8 * level + 8];
        if (lo == hi) continue;
        if (fits) {
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                const int k = quad + i * kQuads;
                if (k < lo || k >= hi) continue;
                double sum = 0.0;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    if (c >= nc[i]) break;
                    if (src[i][c] >= 0) v[i][c] = (&m.sum[src[i][c]].x)[j];
                    sum = add_sum(sum, v[i][c], c == 0);
                }
                (&m.sum[k].x)[j] = sum;
                (&ns[node[i]].x)[j] = sum;
            }
        } else {
            for (int k = lo + threadIdx.x; k < hi; k += kRestThreads)
                node_sums<kMoments>(m.order[k], node_cs, node_nchild, slot_ref, ls, ns, lq, nq);
        }
        __syncthreads();  // also orders the block's global writes
    }
    if (kMoments && fits) {
        // As in the first stage: the distances for all nodes at once (kept by
        // the lane that takes the child's term), then the moments level by
        // level, in the place of the sums' x.
        double uu[kItems][2], mass[kItems][2];
        bool some[kItems];
#pragma unroll
        for (int i = 0; i < kItems; ++i) {
            const int k = quad + i * kQuads;
            some[i] = k < total && __double_as_longlong(m.sum[k < total ? k : 0].w) > 0;
            if (!some[i]) continue;
            const double4_32a sum = m.sum[k];
            const double is = rcp_nr(sum.w);
            const double gx = sum.x * is, gy = sum.y * is, gz = sum.z * is;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (4 * h >= nc[i]) break;
                double4_32a w{0.0, 0.0, 0.0, 0.0};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double x = quad_get(v[i][4 * h + c], 0), y = quad_get(v[i][4 * h + c], 1);
                    const double z = quad_get(v[i][4 * h + c], 2), u = quad_get(v[i][4 * h + c], 3);
                    if (c == j) w = double4_32a{x, y, z, u};
                }
                uu[i][h] = moment_uu(w, gx, gy, gz);
                mass[i][h] = w.w;
            }
        }
        __syncthreads();
        for (int level = 0; level < kDepths; ++level) {
            const int lo = m.off[8 * level], hi = m.off[8 * level + 8];
            if (lo == hi) continue;
#pragma unroll
            for (int i = 0; i < kItems; ++i) {
                const int k = quad + i * kQuads;
                if (k < lo || k >= hi) continue;
                double q = 0.0;
                if (some[i]) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (4 * h >= nc[i]) break;
                        const int at = j == 0 ? src[i][4 * h] : j == 1 ? src[i][4 * h + 1]
                                     : j == 2 ? src[i][4 * h + 2] : src[i][4 * h + 3];
                        double share = 0.0;
                        if (4 * h + j < nc[i])
                            share = moment_add(uu[i][h], mass[i][h], at >= 0 ? m.sum[at].x : cq[i][h]);
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const double x = quad_get(share, c);
                            if (4 * h + c < nc[i]) q += x;
                        }
                    }
                }
                if (j == 0) {
                    m.sum[k].x = q;
                    nq[node[i]] = q;
                }
            }
            __syncthreads();
        }
    }
}

// com = w/m when m > 0 (linear_octree.cpp:95-104), then the merge of
// linear_octree.cpp:194-202 with m0 = com0 = 0.  A one-body leaf passes its
// body's position (one = true): its w is 0 + x m, so w/m is merge_div(m, x).
__device__ inline void finish_com(double m, double wx, double wy, double wz, TreeRec& r, int merge, bool one,
                                  double x, double y, double z)
{
    double cx = wx, cy = wy, cz = wz;
    if (m > 0) {
        if (one) { cx = merge_div(m, x); cy = merge_div(m, y); cz = merge_div(m, z); }
        else {
            const double r = rcp_nr(m);
            cx = div_exact(wx, m, r); cy = div_exact(wy, m, r); cz = div_exact(wz, m, r);
        }
    }
    if (!merge) {  // buildOctreeBottomUp's own output, before any exchange
        r.cx = cx; r.cy = cy; r.cz = cz; r.m = m;
        return;
    }
    const double tot = __dadd_rn(0.0, m);
    if (tot == 0) {
        r.cx = r.cy = r.cz = r.m = 0.0;
        return;
    }
    r.cx = merge_div(tot, cx);
    r.cy = merge_div(tot, cy);
    r.cz = merge_div(tot, cz);
    r.m = tot;
}

// The far-field tree of the FP32 forms (direct bodies' masses zeroed) is not
// the reference's tree, so its centres of mass need no bit-exact quotient:
// w times the refined reciprocal of m (within 2 ulps), no merge step.  The
// kernel also writes the FP32 walk's node records (hi + lo split of the
// centre, G m and the topology word), which the walk would otherwise make in
// a pass of its own.
// Masses are >= 0, so "m > 0" is a test on the bit pattern.  A leaf of one
// body takes the body's position (the quotient w/m would round it).
__device__ inline void far_com(double m, double wx, double wy, double wz, TreeRec& r)
{
    if (__double_as_longlong(m) > 0) {
        const double q = rcp_nr(m);
        r.cx = wx * q; r.cy = wy * q; r.cz = wz * q;
    } else {
        r.cx = wx; r.cy = wy; r.cz = wz;
    }
    r.m = m;
}

struct FarOut {
    float4* A;       // {hi.x, hi.y, hi.z, G m}
    float4* B;       // {lo.x, lo.y, lo.z, bits of child or leaf id}
    uint32_t* meta;  // nchild | depth << 8 | leaf << 16 | massless << 17 | chain above the leaf << 18
    double G;
};

template <bool kMoments, bool kFar>
__global__ void finalize_kernel(const int32_t* __restrict__ counts, const int32_t* __restrict__ slot_ref,
                                const uint8_t* __restrict__ slot_top, const double4_32a* __restrict__ ls,
                                const double4_32a* __restrict__ ns, const int32_t* __restrict__ node_cs,
                                const int32_t* __restrict__ node_nchild, const uint8_t* __restrict__ node_depth,
                                TreeRec* __restrict__ rec, const double* __restrict__ lq,
                                const double* __restrict__ nq, float* __restrict__ spread, int merge,
                                const int32_t* __restrict__ leaf_first, const double* __restrict__ px,
                                const double* __restrict__ py, const double* __restrict__ pz, FarOut far)
{
    const int S = counts[2];
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
        const int r = slot_ref[s];
        TreeRec o;
        o.top = slot_top[s];
        o.pad0 = 0;
        o.pad1 = 0;
        const double4_32a v = r >= 0 ? ls[r] : ns[~r];
        if (r >= 0) {
            if (kFar) {
                const int b = leaf_first[r];
                if (leaf_first[r + 1] == b + 1 && __double_as_longlong(v.w) > 0) {
                    o.cx = px[b]; o.cy = py[b]; o.cz = pz[b]; o.m = v.w;
                } else {
                    far_com(v.w, v.x, v.y, v.z, o);
                }
            } else {
                const int b = leaf_first[r];
                const bool one = leaf_first[r + 1] == b + 1;
                finish_com(v.w, v.x, v.y, v.z, o, merge, one, one ? px[b] : 0.0, one ? py[b] : 0.0,
                           one ? pz[b] : 0.0);
            }
            o.child = -1;
            o.leaf = r;
            o.nchild = 0;
            o.depth = (uint8_t)kMaxDepth;
        } else {
            const int b = ~r;
            if (kFar) far_com(v.w, v.x, v.y, v.z, o);
            else finish_com(v.w, v.x, v.y, v.z, o, merge, false, 0.0, 0.0, 0.0);
            o.child = node_cs[b] + 1;
            o.leaf = -1;
            o.nchild = (uint8_t)node_nchild[b];
            o.depth = node_depth[b];
        }
        // The fused far-field build feeds only the FP32 walks, which read
        // the FP32 records below: the FP64 record is left out (ensure_rec
        // writes it when a diagnostic or export asks for it).
        if (!kFar) rec[s] = o;
        if (kFar) {  // the FP32 walk's records, as fp32_nodes_kernel makes them
            const bool leaf = o.child < 0;
            far.A[s] = make_float4(narrow_trunc(o.cx), narrow_trunc(o.cy), narrow_trunc(o.cz),
                                   narrow_trunc(far.G * o.m));
            far.B[s] = make_float4(low_part(o.cx), low_part(o.cy), low_part(o.cz),
                                   __int_as_float(leaf ? o.leaf : o.child));
            far.meta[s] = (uint32_t)o.nchild | ((uint32_t)o.depth << 8) | ((leaf ? 1u : 0u) << 16) |
                          ((__double_as_longlong(o.m) << 1) == 0 ? 1u << 17 : 0u) |
                          (leaf && o.top <= kMaxDepth - 1 ? 1u << 18 : 0u);
        }
        if (kMoments) {  // a feature: FP32 after narrowing on the bit patterns
            const double m = v.w;
            const double q = r >= 0 ? lq[r] : nq[~r];
            spread[s] = __double_as_longlong(m) > 0 ? sqrtf(narrow_trunc(q) * __frcp_rn(narrow_trunc(m))) : 0.0f;
        }
    }
}

template <bool kMoments>
int launch_monopoles(bh_context* ctx)
{
    cudaStream_t st = ctx->stream;
    const size_t smem = sizeof(ChunkSmem<kMoments>);
    BH_CUDA_TRY(cudaFuncSetAttribute(monopole_chunk_kernel<kMoments>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    static_assert(sizeof(RestSmem<true>) <= 48 * 1024, "no opt-in needed");
    int64_t groups = (ctx->n + kChunk - 1) / kChunk;
    // Two stages' lists in turn: counts, then kMaxSpan nodes per group.
    const int64_t half = monopole_ints(ctx->cap) / 2;
    int32_t* in = ctx->mono_span;
    int32_t* out = ctx->mono_span + half;
    monopole_chunk_kernel<kMoments><<<(unsigned)groups, kChunkThreads, smem, st>>>(
        ctx->counts, ctx->rep_node, ctx->node_a, ctx->node_e, ctx->node_depth, ctx->node_cs, ctx->node_nchild,
        ctx->slot_ref, ctx->leaf_s, ctx->node_s, ctx->leaf_q, ctx->node_q, in, in + groups);
    BH_LAUNCH_CHECK(ctx);
    for (int64_t leaves = kChunk; groups > 1; leaves *= kFan) {
        const int64_t next = (groups + kFan - 1) / kFan;
        monopole_rest_kernel<kMoments><<<(unsigned)next, kRestThreads, sizeof(RestSmem<kMoments>), st>>>(
            ctx->counts, (int)groups, leaves, in, in + groups, ctx->node_a, ctx->node_e, ctx->node_depth, ctx->node_cs,
            ctx->node_nchild, ctx->slot_ref, ctx->leaf_s, ctx->node_s, ctx->leaf_q, ctx->node_q, ctx->head, out,
            out + next);
        BH_LAUNCH_CHECK(ctx);
        std::swap(in, out);
        groups = next;
    }
    return BH_OK;
}

}  // namespace

int64_t monopole_ints(int64_t n)
{
    return 2 * ((n + kChunk - 1) / kChunk) * (kMaxSpan + 1);
}

int64_t boundary_pass_ints(int64_t n)
{
    const int64_t nb = (n + 1 + kBT - 1) / kBT;
    return 4 * kNT * nb;
}

int launch_build(bh_context* ctx, const double* mass, bool moments, bool far_fused, double G, bool far_masses)
{
    const int nzero = far_masses ? (ctx->num_direct < 64 ? ctx->num_direct : 64) : 0;
    ctx->fnodes_fused = false;
    const int64_t n = ctx->n;
    if (n == 0) return BH_OK;
    cudaStream_t st = ctx->stream;
    const int maxb = 8 * bh::num_sms();

    // 1. leaves: ids, first bodies and keys from a scan of the keys' head flags
    int rc = device_number_leaves(ctx, ctx->key, n, ctx->counts + 0, ctx->body_leaf, ctx->leaf_first, ctx->leaf_key);
    if (rc) return rc;

    // 2. leaf sums and branching nodes: the boundary pass (representative
    // flags, node ranges, split chains) -> node ids and child counts -> slots
    const int nb = (int)((n + 1 + kBT - 1) / kBT);
    int32_t* blast = ctx->ansv_blk;
    int32_t* bfirst = blast + (int64_t)nb * kNT;
    int32_t* bpre = bfirst + (int64_t)nb * kNT;
    int32_t* bsuf = bpre + (int64_t)nb * kNT;
    int32_t* bsum = ctx->scan_tmp;
    int32_t* csum = blast;  // free after the boundary pass; nb + 1
    int32_t* cs = reinterpret_cast<int32_t*>(ctx->perm_alt);  // free after the sort
    if (moments)
        leaf_bnd_kernel<true><<<nb, kBT, 0, st>>>(ctx->counts, ctx->leaf_first, ctx->leaf_key, ctx->px, ctx->py, ctx->pz,
                                                  mass, ctx->id, nzero, ctx->leaf_s, ctx->cdep, ctx->leaf_q, blast,
                                                  bfirst);
    else
        leaf_bnd_kernel<false><<<nb, kBT, 0, st>>>(ctx->counts, ctx->leaf_first, ctx->leaf_key, ctx->px, ctx->py, ctx->pz,
                                                   mass, ctx->id, nzero, ctx->leaf_s, ctx->cdep, ctx->leaf_q, blast,
                                                   bfirst);
    BH_LAUNCH_CHECK(ctx);
    const bool scanned = nb > kDirectBlocks;
    if (scanned) {
        bnd_scan_kernel<<<2 * kNT, 1024, 0, st>>>(nb, blast, bfirst, bpre, bsuf);
        BH_LAUNCH_CHECK(ctx);
    }
    bnd_resolve_kernel<<<nb, kBT, 0, st>>>(ctx->counts, ctx->cdep, scanned ? bpre : blast, scanned ? bsuf : bfirst,
                                           scanned ? 1 : 0, ctx->head, ctx->bnd_pl, ctx->bnd_pr, ctx->bnd_next, bsum,
                                           n);
    BH_LAUNCH_CHECK(ctx);
    node_split_kernel<<<nb, kBT, 0, st>>>(ctx->counts, ctx->cdep, ctx->head, bsum, ctx->bnd_pl, ctx->bnd_pr,
                                          ctx->bnd_next, ctx->rep_node, ctx->node_rep, ctx->node_a, ctx->node_e,
                                          ctx->node_depth, ctx->node_nchild, ctx->split_node, ctx->split_rank, cs,
                                          csum, ctx->err);
    BH_LAUNCH_CHECK(ctx);
    if (nb > kOffBlocks) {
        child_offset_kernel<<<1, 1024, 0, st>>>(nb, csum);
        BH_LAUNCH_CHECK(ctx);
    }
    node_place_kernel<<<grid_for(2 * n, kThreads, maxb), kThreads, 0, st>>>(
        ctx->counts, ctx->cdep, ctx->node_a, ctx->node_e, ctx->node_depth, ctx->node_rep, cs, csum, nb, ctx->node_cs,
        ctx->split_node, ctx->split_rank, ctx->slot_ref, ctx->slot_top, ctx->err);
    BH_LAUNCH_CHECK(ctx);

    // 3./4. monopoles (and second moments): chunks of leaves, then what reaches
    // past them
    if ((rc = moments ? launch_monopoles<true>(ctx) : launch_monopoles<false>(ctx))) return rc;

    // 5. traversal records
    const int gs = grid_for(2 * n, kThreads, maxb);
    const FarOut far{ctx->fA, ctx->fB, ctx->fmeta, G};
#define BH_FINALIZE(M, F)                                                                                      \
    finalize_kernel<M, F><<<gs, kThreads, 0, st>>>(                                                            \
        ctx->counts, ctx->slot_ref, ctx->slot_top, ctx->leaf_s, ctx->node_s, ctx->node_cs, ctx->node_nchild,     \
        ctx->node_depth,                                                                                       \
        ctx->rec, ctx->leaf_q, ctx->node_q, ctx->fspread, ctx->build_merge ? 1 : 0, ctx->leaf_first, ctx->px,  \
        ctx->py, ctx->pz, far)
    if (far_fused) {
        if (moments) BH_FINALIZE(true, true);
        else BH_FINALIZE(false, true);
    } else {
        if (moments) BH_FINALIZE(true, false);
        else BH_FINALIZE(false, false);
    }
#undef BH_FINALIZE
    BH_LAUNCH_CHECK(ctx);
    if (far_fused) {
        ctx->fnodes_fused = true;
        ctx->fnodes_G = G;
    }
    ctx->tree_rec = !far_fused;
    return BH_OK;
}

int ensure_rec(bh_context* ctx)
{
    if (ctx->tree_rec || ctx->n == 0) return BH_OK;
    return launch_build(ctx, ctx->m, ctx->tree_moments, false, 0.0, ctx->tree_far);
}

}  // namespace bh
