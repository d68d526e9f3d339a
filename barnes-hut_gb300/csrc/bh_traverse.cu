// Warp-cooperative Barnes-Hut traversal.
//
// Replaces computeAccelerations (src/traversal.cpp:13-103).
//
// BH_MODE_PLAIN_FP64 (exact): a warp owns 32 / P Morton-consecutive bodies, P
// lanes to a body, and walks the compressed octree once for all of them.
//
// Walk.  The reference's per-body stack pops children last-in-first-out, in
// descending octant order, so a body meets the nodes it accepts in descending
// key order.  The warp's stack holds items in that order, the next one on
// top: nodes still to be tested, and nodes some bodies have accepted.  A pass
// takes the top 32 items, one per lane, tests the untested ones all at once
// and puts the children of an opened node in its place; the accepted items in
// front of the first opened node are next for every body, and go to the
// bodies' lists.  (One node per pass, as a plain depth-first walk takes them,
// left the warp waiting on one node record at a time: 34 passes instead of
// about 950 at 100,003 bodies.)  A node is classified against the bodies' box
// in FP32 with allowances for rounding: accepted by all, opened by all, or
// undecided; an undecided one each body tests itself, in FP32 and, where that
// cannot tell either, in FP64 with the reference's rounding.
//
// Evaluation.  Every term is rounded as the reference rounds it and every body
// adds its terms in the reference's order, so the accelerations are the
// reference's bit for bit.  P lanes evaluate P consecutive terms of a body;
// then one lane per component adds them one after the other.  The FP64 pipe
// bounds this (two lanes per cycle: 16 to 19 cycles of the SM per warp
// instruction), so the products, the square root and the reciprocal run as
// integer code beside it (bh_soft64.cuh): 11 FP64 instructions per 32 terms
// are left at P = 4 (the differences, two squares, the sum of squares and the P
// additions) instead of 36.
//
// Measured (theta 1.05, ms of forces; before: one node per pass, 32 bodies
// per warp, IEEE operations on the FP64 pipe):
//   300,149 bodies 12.66 -> 2.84, 19,054 7.71 -> 1.11, 1,000 1.23 -> 0.071.
#include <cfloat>
#include <climits>

#include "bh_internal.cuh"
#include "bh_soft64.cuh"

namespace bh {
namespace {

constexpr int kTravWarps = 4;
constexpr int kTravThreads = 32 * kTravWarps;

struct TravParams {
    int64_t n;
    const double* px;
    const double* py;
    const double* pz;
    const int32_t* body_leaf;
    ExactTree tree;
    const double* bbox;
    double theta2;
    double soft2;
    double kick_h;  // > 0: also apply the second half kick v += kick_h * a
    double one;        // 1.0, as a run-time value: RN(a 1 + b) stays an FMA
    int64_t max_passes;  // above the nodes a walk can meet
    double* ax;
    double* ay;
    double* az;
    double* vx;
    double* vy;
    double* vz;
    unsigned long long* inter_count;
    int32_t* body_count;
    unsigned* err;
};

// side(d)^2 = (L / 2^d)^2 with L the largest bbox span (traversal.cpp:31-43).
__device__ inline void fill_side2(const double* bbox, double* side2)
{
    if (threadIdx.x <= kMaxDepth) {
        const double dx = __dsub_rn(bbox[3], bbox[0]);
        const double dy = __dsub_rn(bbox[4], bbox[1]);
        const double dz = __dsub_rn(bbox[5], bbox[2]);
        double L = dx;
        if (L < dy) L = dy;
        if (L < dz) L = dz;
        const double side = __ddiv_rn(L, (double)(1ull << threadIdx.x));
        side2[threadIdx.x] = __dmul_rn(side, side);
    }
}

// Stack items {node | kDecided, lane mask}: a node still to be tested by the
// lanes of its mask, or (kDecided) one those lanes have accepted.
constexpr int kDecided = 1 << 31;
constexpr int kStk = 384;
// Nodes other than the first undecided one are opened only while the stack
// stays below this; the first one always may, which adds at most 8 items per
// level of one root path (21 levels), so the stack never passes kStk.
constexpr int kSoftStk = kStk - 21 * 8 - 8;
// FP32 tests: a relative margin on the squares (eight roundings of 2^-24 each
// and a square root's 2^-22 are below 1e-6) with an absolute one against
// underflow (of squares below 2^-126, which sqrt_est takes as zero, too), and
// the error of a group-relative distance relative to the coordinates'
// magnitudes: each component of a difference is off by at most 2^-24 (3 |c| + 2 |r|), so the
// distance by sqrt(3) times that, below 3.2e-7 (|c| + |r|); the hi + lo
// split of an absolute coordinate adds 2^-46 of it, so sqrt(3) 2^-46, below
// 2.5e-14, of the group's distance from the origin (and of |c|).
constexpr float kMargin = 2e-6f, kTiny = 1e-36f;
constexpr float kAbsErr = 4e-7f;
// Where a square or a product overflows (distances above 1.8e19), an infinite
// bound says nothing about one that is finite in FP64: sure_below asks for a
// finite right side, and the table's side^2 ends at FLT_MAX, which sure_below
// never accepts and sure_above still bounds from below.
__device__ __forceinline__ bool sure_below(float side2, float theta2, float dist2)  // side^2 < theta^2 dist^2
{
    const float right = theta2 * dist2;
    return fmaf(side2, 1.0f + kMargin, kTiny) < right && right <= FLT_MAX;
}
__device__ __forceinline__ bool sure_above(float side2, float theta2, float dist2)  // side^2 > theta^2 dist^2
{
    return side2 * (1.0f - kMargin) > fmaf(theta2, dist2, kTiny);
}

// Shared memory of a block.  Per-body ordered interaction lists: kCap entries
// per body (P lanes to a body), slots modulo kCap.
template <int P>
struct ExactSmem {
    static constexpr int kBodies = 32 / P;
    // The first lane of each body: masks of bodies have their bits there.
    static constexpr unsigned kFirst = 0xffffffffu / ((1u << (P - 1) << 1) - 1u);
    static constexpr int kCap = 128;  // a power of two, over 33
    int2 stack[kTravWarps][kStk];
    int plist[kTravWarps][kCap][kBodies];
    // A warp to a body: the block's warps evaluate together, and the first takes
    // the sums of all.
    static constexpr bool kShare = P == 32;
    static constexpr int kSumBodies = kShare ? kTravWarps * kBodies : kBodies;
    double term[kShare ? 2 : 1][kTravWarps][3][32];  // the terms of one step of an evaluation
    // Nodes the box cannot decide: {centre, allowance}, {depth of the test,
    // node, leaf id or -1, a chain above the leaf}.
    float4 und[kTravWarps][32];
    int4 und2[kTravWarps][32];
    double side2[kMaxDepth + 1];
    float side2f[kMaxDepth + 1];
};

// The factor G m / r^3 with the reference's operations, for the terms whose
// exponents soft::term leaves out.  A call of its own: inlined, it becomes
// predicated instructions that take the FP64 pipe although no lane needs them.
__device__ __noinline__ double ieee_scale(double dx, double dy, double dz, double soft2, double gm)
{
    const double r2 =
        __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)), soft2);
    const double invR = __drcp_rn(__dsqrt_rn(r2));
    return __dmul_rn(gm, __dmul_rn(__dmul_rn(invR, invR), invR));
}

// One interaction term with the reference's rounding (src/traversal.cpp:
// 80-88): displacement, r^2 and the three products sc d.
// `beside`: work that does not depend on it, done in its waits.
template <bool kSoft, typename F>
__device__ __forceinline__ void exact_term(const double4_32a& r, double px, double py, double pz, double soft2,
                                           bool on, double one, double& tx, double& ty, double& tz, F beside)
{
    const double dx = fma(r.x, one, -px), dy = fma(r.y, one, -py), dz = fma(r.z, one, -pz);
    // One of the three squares on the integer pipes balances them with the
    // FP64 pipe (300,149 bodies: none 3.05 ms, one 2.96, two 2.96, three 3.06).
    const double zz = soft::square(soft::bits_of(dz));
    double r2 = fma(fma(__dmul_rn(dx, dx), one, __dmul_rn(dy, dy)), one, zz);
    if (kSoft) r2 = fma(r2, one, soft2);
    beside();
    if (!soft::term(dx, dy, dz, r2, r.w, tx, ty, tz) && on) {
        const double sc = ieee_scale(dx, dy, dz, soft2, r.w);
        tx = __dmul_rn(sc, dx);
        ty = __dmul_rn(sc, dy);
        tz = __dmul_rn(sc, dz);
    }
}

// Blocks per SM of the form that loads records ahead.
constexpr int kAheadBlocks = 5;

template <int P, bool kSoft, bool kAhead>
__global__ void __launch_bounds__(kTravThreads, kAhead ? kAheadBlocks : 0) traverse_exact_kernel(TravParams p)
{
    using Smem = ExactSmem<P>;
    constexpr int kBodies = Smem::kBodies;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
    fill_side2(p.bbox, sm.side2);
    __syncthreads();
    if (threadIdx.x <= kMaxDepth) sm.side2f[threadIdx.x] = fminf((float)sm.side2[threadIdx.x], FLT_MAX);
    __syncthreads();

    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t group = (int64_t)blockIdx.x * kTravWarps + w;
    const int64_t base = group * kBodies;
    if (!Smem::kShare && base >= p.n) return;  // whole warp past the end
    const int body = lane / P, phase = lane % P;
    const int64_t i = base + body;
    const bool valid = i < p.n;
    const int64_t ii = valid ? i : base < p.n ? base : 0;
    const double px = p.px[ii], py = p.py[ii], pz = p.pz[ii];
    const int my_leaf = valid ? p.body_leaf[i] : -2;
    const double theta2 = p.theta2, soft2 = p.soft2;
    const float theta2f = (float)theta2, soft2f = (float)soft2;
    // Group box in group-relative FP32 coordinates (for the group tests).
    const float gx = __double2float_rn(__shfl_sync(0xffffffffu, px, 0));
    const float gy = __double2float_rn(__shfl_sync(0xffffffffu, py, 0));
    const float gz = __double2float_rn(__shfl_sync(0xffffffffu, pz, 0));
    const float rx = __double2float_rn(px - (double)gx);
    const float ry = __double2float_rn(py - (double)gy);
    const float rz = __double2float_rn(pz - (double)gz);
    float bminx = rx, bminy = ry, bminz = rz, bmaxx = rx, bmaxy = ry, bmaxz = rz;
    int leaf_lo = valid ? my_leaf : INT_MAX, leaf_hi = valid ? my_leaf : INT_MIN;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        bminx = fminf(bminx, __shfl_xor_sync(0xffffffffu, bminx, off));
        bminy = fminf(bminy, __shfl_xor_sync(0xffffffffu, bminy, off));
        bminz = fminf(bminz, __shfl_xor_sync(0xffffffffu, bminz, off));
        bmaxx = fmaxf(bmaxx, __shfl_xor_sync(0xffffffffu, bmaxx, off));
        bmaxy = fmaxf(bmaxy, __shfl_xor_sync(0xffffffffu, bmaxy, off));
        bmaxz = fmaxf(bmaxz, __shfl_xor_sync(0xffffffffu, bmaxz, off));
        leaf_lo = min(leaf_lo, __shfl_xor_sync(0xffffffffu, leaf_lo, off));
        leaf_hi = max(leaf_hi, __shfl_xor_sync(0xffffffffu, leaf_hi, off));
    }
    const float bmag = fmaxf(fmaxf(fmaxf(fabsf(bminx), fabsf(bmaxx)), fmaxf(fabsf(bminy), fabsf(bmaxy))),
                             fmaxf(fabsf(bminz), fabsf(bmaxz))) +
                       (5e-14f / kAbsErr) * fmaxf(fmaxf(fabsf(gx), fabsf(gy)), fabsf(gz));
    int2* stk = sm.stack[w];
    int (*PL)[kBodies] = sm.plist[w];
    const unsigned lt = (1u << lane) - 1u;

    // This body's list: entries done .. cnt - 1, in slots modulo kCap.
    int cnt = 0, done = 0;
    const unsigned full = __ballot_sync(0xffffffffu, valid) & Smem::kFirst;
    int sp = full ? 1 : 0;
    const double one = __shfl_sync(0xffffffffu, p.one, 0);
    if (lane == 0) stk[0] = make_int2(0, (int)full);
    __syncwarp();
    bool overflow = false;
    int64_t passes = 0;

    // Evaluates the bodies' lists in order until none holds more than `left`
    // entries.  P lanes evaluate P consecutive terms of a body.  The sums run
    // over them one after the other, each waiting for the one before (68
    // cycles), so they take the terms of the step before while the next ones
    // are evaluated (19,054 bodies 1.18 -> 1.15 ms, 8,000 0.46 -> 0.42).
    // Lane l < 3 kSumBodies sums the component l / kSumBodies of a body.  An
    // addition takes the FP64 pipe 19 cycles however few lanes it is for, and a
    // warp's own sums are P of them a step, at P = 32 32 of 39 FP64
    // instructions: there the block's four warps evaluate together, a barrier
    // to a step, and the first takes the sums of all (2,000 bodies 0.135 ->
    // 0.103 ms, 4,000 0.285 -> 0.170; with 16 lanes 0.208 -> 0.238, with 8
    // 0.27 -> 0.29).
    constexpr int kSumBodies = Smem::kSumBodies;
    const bool sums = !Smem::kShare || w == 0;
    const int sum_body = lane % kSumBodies;  // of the block, or of the warp
    const int sum_comp = lane < 3 * kSumBodies ? lane / kSumBodies : 2;
    double sum = 0.0;
    int par = 0;  // the half of `term` the next step fills
    for (int h = 0; h < (Smem::kShare ? 2 : 1); ++h)
        sm.term[h][w][0][lane] = sm.term[h][w][1][lane] = sm.term[h][w][2][lane] = 0.0;
    if (Smem::kShare) __syncthreads();
    else __syncwarp();
    // where they stand in a half of `term`
    const int from = (Smem::kShare ? sum_body / kBodies : w) * 96 + sum_comp * 32 + sum_body % kBodies * P;
    constexpr int kHalf = kTravWarps * 96;
    auto add = [&] {
        const double* t = &sm.term[0][0][0][0] + from + (Smem::kShare ? (par ^ 1) * kHalf : 0);
#pragma unroll
        for (int k = 0; k < P; ++k) sum = fma(sum, one, t[k]);
    };
    auto record = [&](int q) { return p.tree.d4[q < cnt ? PL[q & (Smem::kCap - 1)][body] : 0]; };
    auto step = [&](double4_32a& next, auto beside) {
        const int q = done + phase;
        const bool on = q < cnt;
        const double4_32a r = kAhead ? next : record(q);
        if (kAhead) next = record(q + P);
        double tx, ty, tz;
        exact_term<kSoft>(r, px, py, pz, soft2, on, one, tx, ty, tz, beside);
        if (!Smem::kShare) __syncwarp();
        // (a sum is never -0, so adding +0 leaves it as it is)
        auto T = sm.term[Smem::kShare ? par : 0][w];
        T[0][lane] = on ? tx : 0.0;
        T[1][lane] = on ? ty : 0.0;
        T[2][lane] = on ? tz : 0.0;
        done = min(done + P, cnt);
    };
    // kShare: every warp of the block calls it equally often, walking or not;
    // returns whether any still walks.
    auto flush = [&](int left, bool walking) {
        if (Smem::kShare) {
            while (__syncthreads_or(cnt - done > left)) {
                double4_32a none;
                if (sums) step(none, add);
                else step(none, [] {});
                par ^= 1;
            }
            return __syncthreads_or(walking) != 0;
        }
        int most = cnt - done;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, off));
        double4_32a next;
        if (kAhead) next = record(done + phase);
        for (; most > left; most -= P) {
            step(next, add);
            __syncwarp();
        }
        return false;
    };

    while (sp > 0) {
        if (++passes > p.max_passes) {
            overflow = true;
            break;
        }
        // The window: the top items of the stack, lane 0 the first in walk
        // order.
        const int m = sp < 32 ? sp : 32;
        int node = 0, nc = 0, ref = 0, depth = 0;
        unsigned M = 0, A = 0;
        bool test = false, leaf = false, chain = false, mixed = false;
        float cx = 0.f, cy = 0.f, cz = 0.f, nerr = 0.f;  // group-relative centre, its allowance
        if (lane < m) {
            const int2 it = stk[sp - 1 - lane];
            node = it.x & ~kDecided;
            M = (unsigned)it.y;
            if (it.x & kDecided) {
                A = M;
            } else {
                test = true;
                const float4 a = __ldg(p.tree.A + node);
                const float4 b = __ldg(p.tree.B + node);
                const uint32_t mt = __ldg(p.tree.meta + node);
                cx = (a.x - gx) + b.x;
                cy = (a.y - gy) + b.y;
                cz = (a.z - gz) + b.z;
                ref = __float_as_int(b.w);
                leaf = (mt >> 16) & 1u;
                chain = (mt >> 18) & 1u;
                depth = (mt >> 8) & 0xFF;
                nerr = kAbsErr * (fmaxf(fabsf(cx), fmaxf(fabsf(cy), fabsf(cz))) + bmag);
                if ((mt >> 17) & 1u) {
                    M = 0;  // massless: skipped with its subtree (traversal.cpp:66)
                } else if (leaf) {
                    A = M;
                } else {
                    nc = (int)(mt & 0xFF);
                    const float ex = fmaxf(0.0f, fmaxf(bminx - cx, cx - bmaxx));
                    const float ey = fmaxf(0.0f, fmaxf(bminy - cy, cy - bmaxy));
                    const float ez = fmaxf(0.0f, fmaxf(bminz - cz, cz - bmaxz));
                    const float fx = fmaxf(fabsf(cx - bminx), fabsf(cx - bmaxx));
                    const float fy = fmaxf(fabsf(cy - bminy), fabsf(cy - bmaxy));
                    const float fz = fmaxf(fabsf(cz - bminz), fabsf(cz - bmaxz));
                    const float dlo = fmaxf(sqrt_est(ex * ex + ey * ey + ez * ez) - nerr, 0.0f);
                    const float dhi = sqrt_est(fx * fx + fy * fy + fz * fz) + nerr;
                    const float s2 = sm.side2f[depth];
                    if (sure_below(s2, theta2f, dlo * dlo + soft2f)) A = M;
                    else mixed = !sure_above(s2, theta2f, dhi * dhi + soft2f);
                }
            }
        }
        // Nodes the box cannot decide, and the leaves that may hold one of
        // the bodies: each body tests them itself, P at a time, in FP32 with
        // the same allowance and in FP64 with the reference's rounding where
        // that cannot decide either.  A body skips its own leaf at depth 21,
        // but a chain cell above it (depths top..20) may already accept it;
        // any other leaf it accepts.
        const bool own = test && leaf && A != 0 && ref >= leaf_lo && ref <= leaf_hi;
        const unsigned ub = __ballot_sync(0xffffffffu, mixed || own);
        if (ub) {
            const int k = __popc(ub & lt);
            if (mixed || own) {
                sm.und[w][k] = make_float4(cx, cy, cz, nerr);
                sm.und2[w][k] = make_int4(own ? kMaxDepth - 1 : depth, node, own ? ref : -1, chain ? 1 : 0);
            }
            __syncwarp();
            const int nu = __popc(ub);
            for (int k0 = 0; k0 < nu; k0 += P) {
                bool acc = false;
                const int kk = k0 + phase;
                if (kk < nu) {
                    const float4 u = sm.und[w][kk];
                    const int4 v = sm.und2[w][kk];
                    const float dxf = u.x - rx, dyf = u.y - ry, dzf = u.z - rz;
                    const float df = sqrt_est(dxf * dxf + dyf * dyf + dzf * dzf);
                    const float lo = fmaxf(df - u.w, 0.0f), hi = df + u.w;
                    const float s2 = sm.side2f[v.x];
                    if (v.z >= 0 ? v.z != my_leaf : sure_below(s2, theta2f, lo * lo + soft2f)) {
                        acc = true;
                    } else if (!sure_above(s2, theta2f, hi * hi + soft2f)) {
                        const double4_32a r = p.tree.d4[v.y];
                        const double dx = __dsub_rn(r.x, px), dy = __dsub_rn(r.y, py), dz = __dsub_rn(r.z, pz);
                        const double r2 = __dadd_rn(
                            __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)), soft2);
                        acc = (v.z < 0 || v.w != 0) && sm.side2[v.x] < __dmul_rn(theta2, r2);
                    }
                }
                const unsigned res = __ballot_sync(0xffffffffu, acc);
                if ((mixed || own) && k >= k0 && k < k0 + P) A = (res >> (k - k0)) & Smem::kFirst & M;
            }
            __syncwarp();
        }
        // Opened nodes leave their children in their place.  Where they would
        // not fit, the later ones wait (an untested item again).
        const unsigned O = leaf ? 0u : M & ~A;
        bool open = test && O != 0;
        const unsigned opened = __ballot_sync(0xffffffffu, open);
        const int first = opened ? __ffs(opened) - 1 : 32;
        int out = (A != 0 ? 1 : 0) + (open ? nc : 0);
        int incl = out;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off) incl += t;
        }
        const int below = sp - m;
        if (__any_sync(0xffffffffu, open && lane > first && below + incl + (m - 1 - lane) > kSoftStk)) {
            if (open && lane > first && below + incl + (m - 1 - lane) > kSoftStk) {
                open = false;
                A = M;
                nc = -1;  // not decided: the item goes back as it was
                out = 1;
            }
            incl = out;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += t;
            }
        }
        // Accepted items before the first opened node, and its own accepted
        // part, are next in walk order: they go to the lists.  All else goes
        // back on the stack.
        const bool emit = A != 0 && lane <= first;
        if (emit) --out;
        const unsigned em = __ballot_sync(0xffffffffu, emit);
        const int total = __shfl_sync(0xffffffffu, incl, 31) - __popc(em);
        const int pos = incl - __popc(em & (lt | (1u << lane))) - out;  // outputs put back before this lane's
        if (below + total > kStk) {
            overflow = true;
            break;
        }
        __syncwarp();
        int top = below + total - 1 - pos;
        if (A != 0 && !emit) stk[top--] = make_int2(nc < 0 ? node : node | kDecided, (int)A);
        if (open)
            for (int c = nc - 1; c >= 0; --c) stk[top--] = make_int2(ref + c, (int)O);
        sp = below + total;
        if (em) {
            if (__any_sync(0xffffffffu, cnt - done > Smem::kCap - 33)) {
                __syncwarp();
                flush(Smem::kCap / 4, true);
            }
            // Body by body: the lanes whose item it takes append it.
#pragma unroll
            for (int b = 0; b < kBodies; ++b) {
                const bool take = emit && ((A >> (b * P)) & 1u);
                const unsigned tb = __ballot_sync(0xffffffffu, take);
                const int at = __shfl_sync(0xffffffffu, cnt, b * P);
                if (take) PL[(at + __popc(tb & lt)) & (Smem::kCap - 1)][b] = node;
                if (body == b) cnt += __popc(tb);
            }
        }
        __syncwarp();
    }
    while (flush(0, false)) {}
    add();
    if (overflow && lane == 0) atomicOr(p.err, kErrOverflow);
    if (sums && lane < 3 * kSumBodies) {
        const int64_t k = (Smem::kShare ? (int64_t)blockIdx.x * kTravWarps * kBodies : base) + sum_body;
        if (k < p.n) {
            double* a = sum_comp == 0 ? p.ax : sum_comp == 1 ? p.ay : p.az;
            double* v = sum_comp == 0 ? p.vx : sum_comp == 1 ? p.vy : p.vz;
            a[k] = sum;
            if (p.kick_h > 0.0) v[k] = __dadd_rn(v[k], __dmul_rn(p.kick_h, sum));
        }
    }
    const bool counts = valid && phase == 0;
    if (counts && p.body_count) p.body_count[i] = cnt;
    if (p.inter_count) {
        unsigned long long c = counts ? (unsigned long long)cnt : 0ull;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) c += __shfl_down_sync(0xffffffffu, c, off);
        if (lane == 0) atomicAdd(p.inter_count, c);
    }
}

template <int P, bool kSoft, bool kAhead>
int launch_exact(bh_context* ctx, const TravParams& p)
{
    auto kernel = traverse_exact_kernel<P, kSoft, kAhead>;
    const size_t smem = sizeof(ExactSmem<P>);
    BH_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    BH_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     (int)cudaSharedmemCarveoutMaxShared));
    const int64_t groups = (p.n + 32 / P - 1) / (32 / P);
    const int64_t blocks = (groups + kTravWarps - 1) / kTravWarps;
    kernel<<<(unsigned)blocks, kTravThreads, smem, ctx->stream>>>(p);
    BH_LAUNCH_CHECK(ctx);
    return BH_OK;
}

// soft2 = 0 leaves r^2 as it is (r^2 + 0 = r^2): one FP64 addition less.
template <int P, bool kAhead = false>
int launch_exact_p(bh_context* ctx, const TravParams& p)
{
    return p.soft2 == 0.0 ? launch_exact<P, false, kAhead>(ctx, p) : launch_exact<P, true, kAhead>(ctx, p);
}

}  // namespace

int launch_exact_walk(bh_context* ctx, const ExactTree& tree, double theta, double soft2, double kick_h,
                      int32_t* body_count, unsigned long long* inter_count, unsigned* err)
{
    const int64_t n = ctx->n;
    if (n == 0) return BH_OK;
    TravParams p;
    p.n = n;
    p.px = ctx->px; p.py = ctx->py; p.pz = ctx->pz;
    p.body_leaf = ctx->body_leaf;
    p.tree = tree;
    p.bbox = ctx->bbox;
    p.theta2 = theta * theta;
    p.soft2 = soft2;
    p.kick_h = kick_h;
    p.one = 1.0;
    p.max_passes = 2 * tree.nodes + 2;
    p.ax = ctx->ax; p.ay = ctx->ay; p.az = ctx->az;
    p.vx = ctx->vx; p.vy = ctx->vy; p.vz = ctx->vz;
    p.inter_count = inter_count;
    p.body_count = body_count;
    p.err = err;
    // Lanes to a body: 4 (the evaluation's sums fill 24 lanes and the bodies
    // share a walk) while that gives the chip 12 warps per SM, and more below,
    // where a warp's own latency counts.  Forces in ms with 4 / 8 / 16 / 32
    // lanes: 300,149 bodies 2.84 / 3.67 / 5.36 / -, 19,054 1.11 / 1.18 / 1.30 /
    // 1.29, 14,000 0.90 / 0.72 / - / 0.88, 8,000 0.63 / 0.41 / 0.42 / 0.43, 7,000
    // - / 0.36 / - / 0.39, 4,000 0.40 / 0.27 / 0.21 / 0.17, 2,000 0.27 / 0.17 / 0.13 / 0.10, 1,000 0.18 /
    // 0.12 / 0.086 / 0.071 (16 is not built: never ahead of both neighbours by
    // more than 1 %).  With 4 lanes and all blocks on the chip at once, five to an
    // SM, the next step's records are loaded ahead, which takes 92 registers
    // for 72 (19,054 bodies 1.15 -> 1.11; 30,000 0.312 -> 0.344, in two rounds).
    const int64_t want = 12 * (int64_t)num_sms() * 32;
    if (n > kAheadBlocks * kTravWarps * 8 * (int64_t)num_sms()) return launch_exact_p<4>(ctx, p);
    if (n * 4 >= want) return launch_exact_p<4, true>(ctx, p);
    if (n * 8 >= want - want / 8) return launch_exact_p<8>(ctx, p);
    return launch_exact_p<32>(ctx, p);
}

int launch_traverse(bh_context* ctx, double theta, double G, double soft2, int mode, double kick_h)
{
    const int64_t n = ctx->n;
    if (n == 0) return BH_OK;
    BH_CUDA_TRY(cudaMemsetAsync(ctx->inter_count, 0, sizeof(unsigned long long), ctx->stream));
    switch (mode) {
    case BH_MODE_PLAIN_FP64: {
        const int rc = launch_fp32_nodes(ctx, G, true);
        if (rc) return rc;
        return launch_exact_walk(ctx, ExactTree{2 * n, ctx->fA, ctx->fB, ctx->fmeta, ctx->d4}, theta, soft2, kick_h,
                                 ctx->body_count, ctx->inter_count, ctx->err);
    }
    case BH_MODE_FP64_LIST:
        return launch_traverse_masked(ctx, theta, G, soft2, kick_h, true);
    case BH_MODE_FP32_FAR:
        return launch_traverse_masked(ctx, theta, G, soft2, kick_h, false);
    case BH_MODE_LEARNED:
        return launch_traverse_learned(ctx, theta, G, soft2, kick_h);
    case BH_MODE_FP32_GROUP:
        return launch_traverse_masked(ctx, theta, G, soft2, kick_h, false, true);
    default:
        return bh_fail(BH_ERR_INVALID_ARGUMENT, "bh_compute_accelerations: mode not available");
    }
}

}  // namespace bh
