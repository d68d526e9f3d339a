// Training of the acceptance network on the GPU with hand-written forward,
// backward and Adam kernels.  No reference counterpart.
//
// Loss: mean squared error of the standardised log10 error label.  Forward
// numerics are those of the inference path fused into the traversal: BF16
// weights and BF16 layer inputs, FP32 accumulation, bias first.  Gradients
// are taken with respect to the FP32 master weights (the BF16 rounding is
// treated as the identity), reduced deterministically (no atomics).
#include <algorithm>
#include <cmath>
#include <numeric>
#include <random>
#include <string>
#include <vector>

#include "bh_internal.cuh"
#include "bh_mlp.cuh"

namespace bh {
namespace {

// A batch's samples are dealt to four row sets, sample b to row b / 4 of set
// b % 4 (the four interleaved partial sums of dW2); `rows` rows are allotted to
// each set, a multiple of kRowStep.
constexpr int kFbSamples = 32;  // samples per block of the forward/backward kernel
constexpr int kFbThreads = 256;
constexpr int kRowStep = 64;

struct Scratch {
    int rows;
    float* h1;    // [4][rows][64] layer-1 outputs
    float* xb;    // [4][rows][8] inputs
    float* dh1;   // [4][64][rows] layer deltas and layer-2 outputs, by unit
    float* dh2;
    float* h2;
    float* dy;    // [4][rows]
    float* loss_part;  // per 32 samples
    float* p_w2;  // [4][64 * 64] partial sums of the gradient
    float* p_w1;  // [32][64 * 8]
    float* p_b;   // [64][193]: b1, b2, W3, b3
};
constexpr int kBiasParts = 3 * kHid + 1;

constexpr int kW2tRow = kHid + 4;
struct FbSmem {
    float W2[kHid * kHid];   // [i][j]
    float W2t[kHid * kW2tRow];  // [j][i], rows padded against bank conflicts
    float h1[kHid][kFbSamples];
    float h2[kHid][kFbSamples];
    float d2[kHid][kFbSamples];
    float W1[kHid * kFeat], b1[kHid], b2[kHid], W3[kHid];
    float b3;
};

// A batch is a chain of three short kernels, each waiting for the one before.
// They are launched so that a kernel's blocks are set up, and what does not
// depend on the chain is loaded, while its predecessor runs; wait_for_chain()
// returns when that one has completed, and lets the next be set up.  A kernel
// waits before it writes anything or reads what the chain writes (past L1, whose
// lines may be older than the wait), so it also knows all earlier ones complete.
__device__ __forceinline__ void wait_for_chain()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
cudaError_t launch_in_chain(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t stream, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Forward, loss and backward to the layer deltas for 32 samples: lane = sample,
// warp w computes units 8 w .. 8 w + 7 of each layer, so that eight independent
// sums run beside one another and every weight is read by broadcast.  Each sum
// keeps the order of its terms.  What bounds it is latency (a block's 32
// samples are a chain of three small layers); with one thread per sample, 32
// blocks of 128 on the whole chip, a batch of 4,096 took 135 us over its three
// kernels, and takes 22 (30 before they were chained; in ncu 11 here, 12 in
// the sums, 6 in Adam).
__global__ void __launch_bounds__(kFbThreads) mlp_fwd_bwd_kernel(const float* __restrict__ X,
                                                                const float* __restrict__ T,
                                                                const int32_t* __restrict__ idx, int64_t off,
                                                                int B, float inv_b, const float* P,
                                                                Scratch s)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FbSmem& m = *reinterpret_cast<FbSmem*>(smem_raw);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, u0 = 8 * w;
    const int b = blockIdx.x * kFbSamples + lane;
    const bool live = b < B;
    const int64_t sidx = live ? (idx ? (int64_t)idx[off + b] : off + b) : 0;
    float xb[kFeat];
#pragma unroll
    for (int k = 0; k < kFeat; ++k) xb[k] = live ? bf16r(X[sidx * kFeat + k]) : 0.0f;
    const float target = live ? T[sidx] : 0.0f;
    wait_for_chain();
    static_assert(kOffW2 % 4 == 0, "rows of W2 are read as float4");
#pragma unroll
    for (int q = 0; q < kHid * kHid / 4 / kFbThreads; ++q) {
        const int k = 4 * (threadIdx.x + q * kFbThreads), i = k / kHid, j = k % kHid;
        float4 v = __ldcg(reinterpret_cast<const float4*>(P + kOffW2 + k));
        v.x = bf16r(v.x); v.y = bf16r(v.y); v.z = bf16r(v.z); v.w = bf16r(v.w);
        *reinterpret_cast<float4*>(&m.W2[k]) = v;
        m.W2t[j * kW2tRow + i] = v.x;
        m.W2t[(j + 1) * kW2tRow + i] = v.y;
        m.W2t[(j + 2) * kW2tRow + i] = v.z;
        m.W2t[(j + 3) * kW2tRow + i] = v.w;
    }
    for (int k = threadIdx.x; k < kHid * kFeat; k += kFbThreads) m.W1[k] = bf16r(__ldcg(P + kOffW1 + k));
    if (threadIdx.x < kHid) {
        m.b1[threadIdx.x] = __ldcg(P + kOffB1 + threadIdx.x);
        m.b2[threadIdx.x] = __ldcg(P + kOffB2 + threadIdx.x);
        m.W3[threadIdx.x] = bf16r(__ldcg(P + kOffW3 + threadIdx.x));
    }
    if (threadIdx.x == 0) m.b3 = __ldcg(P + kOffB3);
    __syncthreads();
    float h1[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        float a = m.b1[u0 + u];
#pragma unroll
        for (int k = 0; k < kFeat; ++k) a = fmaf(m.W1[(u0 + u) * kFeat + k], xb[k], a);
        h1[u] = bf16r(fmaxf(a, 0.0f));
        m.h1[u0 + u][lane] = h1[u];
    }
    __syncthreads();
    float acc[8], h2[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u] = m.b2[u0 + u];
#pragma unroll 8
    for (int j = 0; j < kHid; ++j) {
        const float h = m.h1[j][lane];
        const float4 v0 = *reinterpret_cast<const float4*>(&m.W2t[j * kW2tRow + u0]);
        const float4 v1 = *reinterpret_cast<const float4*>(&m.W2t[j * kW2tRow + u0 + 4]);
        acc[0] = fmaf(v0.x, h, acc[0]); acc[1] = fmaf(v0.y, h, acc[1]);
        acc[2] = fmaf(v0.z, h, acc[2]); acc[3] = fmaf(v0.w, h, acc[3]);
        acc[4] = fmaf(v1.x, h, acc[4]); acc[5] = fmaf(v1.y, h, acc[5]);
        acc[6] = fmaf(v1.z, h, acc[6]); acc[7] = fmaf(v1.w, h, acc[7]);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        h2[u] = bf16r(fmaxf(acc[u], 0.0f));
        m.h2[u0 + u][lane] = h2[u];
    }
    __syncthreads();
    float y = m.b3;  // in every warp
#pragma unroll 16
    for (int i = 0; i < kHid; ++i) y = fmaf(m.W3[i], m.h2[i][lane], y);
    const float diff = y - target;
    const float dy = 2.0f * diff * inv_b;
    float d2[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        d2[u] = h2[u] > 0.0f ? dy * m.W3[u0 + u] : 0.0f;
        m.d2[u0 + u][lane] = d2[u];
        acc[u] = 0.0f;
    }
    __syncthreads();
#pragma unroll 8
    for (int i = 0; i < kHid; ++i) {
        const float d = m.d2[i][lane];
        const float4 v0 = *reinterpret_cast<const float4*>(&m.W2[i * kHid + u0]);
        const float4 v1 = *reinterpret_cast<const float4*>(&m.W2[i * kHid + u0 + 4]);
        acc[0] = fmaf(d, v0.x, acc[0]); acc[1] = fmaf(d, v0.y, acc[1]);
        acc[2] = fmaf(d, v0.z, acc[2]); acc[3] = fmaf(d, v0.w, acc[3]);
        acc[4] = fmaf(d, v1.x, acc[4]); acc[5] = fmaf(d, v1.y, acc[5]);
        acc[6] = fmaf(d, v1.z, acc[6]); acc[7] = fmaf(d, v1.w, acc[7]);
    }
    if (live) {
        const int q = b & 3, r = b >> 2;
        float4* o = reinterpret_cast<float4*>(s.h1 + ((int64_t)q * s.rows + r) * kHid + u0);
        o[0] = make_float4(h1[0], h1[1], h1[2], h1[3]);
        o[1] = make_float4(h1[4], h1[5], h1[6], h1[7]);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int64_t k = ((int64_t)q * kHid + u0 + u) * s.rows + r;
            s.dh1[k] = h1[u] > 0.0f ? acc[u] : 0.0f;
            s.dh2[k] = d2[u];
            s.h2[k] = h2[u];
        }
        if (w == 0) {
            float4* x = reinterpret_cast<float4*>(s.xb + ((int64_t)q * s.rows + r) * kFeat);
            x[0] = make_float4(xb[0], xb[1], xb[2], xb[3]);
            x[1] = make_float4(xb[4], xb[5], xb[6], xb[7]);
            s.dy[(int64_t)q * s.rows + r] = dy;
        }
    }
    if (w == 0) {
        float l2 = live ? diff * diff : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l2 += __shfl_down_sync(0xffffffffu, l2, o);
        if (lane == 0) s.loss_part[blockIdx.x] = l2;
    }
}

__device__ __forceinline__ void copy16(void* smem, const void* global)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)),
                 "l"(global)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The gradient's sums over the batch, to partial sums (one term after the
// other within each, in batch order).  Blocks 0..63: dW2[i][j] = sum dh2[i]
// h1[j] for four units i and one row set, one sum per thread: a chain of B / 4
// FMAs, four cycles each, which is what bounds it (a batch of 4,096: 4,096
// cycles, 2.1 us), while the rows stream through shared memory four steps
// ahead.  Blocks 64..95: the sums over 32 (dW1) and 64 (biases, W3) interleaved
// parts for eight units and one row set.
constexpr int kReduceThreads = 256;
constexpr int kW2Units = 4;                       // units per block
constexpr int kW2Blocks = 4 * kHid / kW2Units;    // 64
constexpr int kSmallUnits = 8;
constexpr int kSmallBlocks = 4 * kHid / kSmallUnits;  // 32
constexpr int kSteps = 4;  // copies in flight

struct W2Step {
    float h1[kRowStep][kHid];
    float d2[kW2Units][kRowStep];
};
struct SmallTile {
    float dh1[kSmallUnits][kRowStep], dh2[kSmallUnits][kRowStep], h2[kSmallUnits][kRowStep];
    float xb[kRowStep][kFeat];
    float dy[kRowStep];
};
// More than half of an SM's shared memory, which keeps the blocks one to an SM.
// They are set up while the forward blocks still hold most SMs; three to each
// of the free ones, a batch of 4,096 took 36 us instead of 22.
constexpr size_t kReduceSmem = 118 * 1024;
static_assert(kReduceSmem >= kSteps * sizeof(W2Step) && kReduceSmem >= kSteps * sizeof(SmallTile) &&
                  kReduceSmem + sizeof(FbSmem) + 2048 <= 228 * 1024,
              "a reducing block beside a forward one");

__global__ void __launch_bounds__(kReduceThreads) mlp_grad_reduce_kernel(int B, Scratch s)
{
    wait_for_chain();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x;
    const bool small = blockIdx.x >= kW2Blocks;
    const int q = blockIdx.x & 3;
    const int g = (small ? blockIdx.x - kW2Blocks : blockIdx.x) >> 2;
    const int n = (B - q + 3) / 4;  // rows of this set
    const int steps = (n + kRowStep - 1) / kRowStep;
    if (!small) {
        W2Step* st = reinterpret_cast<W2Step*>(smem_raw);
        const int j = t & 63, ii = t >> 6, i0 = g * kW2Units;
        const float* h1 = s.h1 + (int64_t)q * s.rows * kHid;
        const float* d2 = s.dh2 + ((int64_t)q * kHid + i0) * s.rows;
        auto fetch = [&](int k) {
            if (k < steps) {
                W2Step& c = st[k % kSteps];
                const float* src = h1 + (int64_t)k * kRowStep * kHid;
#pragma unroll
                for (int o = 0; o < kRowStep * kHid / 4; o += kReduceThreads)
                    copy16(&c.h1[0][0] + 4 * (o + t), src + 4 * (o + t));
                if (t < kW2Units * kRowStep / 4)
                    copy16(&c.d2[t / 16][4 * (t % 16)], d2 + (int64_t)(t / 16) * s.rows + k * kRowStep + 4 * (t % 16));
            }
            copy_commit();
        };
        static_assert(kRowStep == 64 && kReduceThreads == kW2Units * kHid, "copy shape");
        for (int k = 0; k < kSteps - 1; ++k) fetch(k);
        float a = 0.0f;
        for (int k = 0; k < steps; ++k) {
            copy_wait<kSteps - 2>();
            __syncthreads();  // step k is here for all, step k - 1 read by all
            fetch(k + kSteps - 1);
            const W2Step& c = st[k % kSteps];
            const int rows = n - k * kRowStep < kRowStep ? n - k * kRowStep : kRowStep;
            if (rows == kRowStep) {
#pragma unroll 16
                for (int r = 0; r < kRowStep; ++r) a = fmaf(c.d2[ii][r], c.h1[r][j], a);
            } else {
                for (int r = 0; r < rows; ++r) a = fmaf(c.d2[ii][r], c.h1[r][j], a);
            }
        }
        s.p_w2[(int64_t)q * kHid * kHid + (i0 + ii) * kHid + j] = a;
        return;
    }
    SmallTile* st = reinterpret_cast<SmallTile*>(smem_raw);
    const int i0 = g * kSmallUnits;
    const int64_t u0 = ((int64_t)q * kHid + i0) * s.rows;
    auto fetch = [&](int k) {
        if (k < steps) {
            SmallTile& c = st[k % kSteps];
            const int64_t r0 = (int64_t)k * kRowStep;
            if (t < kSmallUnits * kRowStep / 4) {
                const int u = t / 16, r = 4 * (t % 16);
                copy16(&c.dh1[u][r], s.dh1 + u0 + (int64_t)u * s.rows + r0 + r);
                copy16(&c.dh2[u][r], s.dh2 + u0 + (int64_t)u * s.rows + r0 + r);
                copy16(&c.h2[u][r], s.h2 + u0 + (int64_t)u * s.rows + r0 + r);
                copy16(&c.xb[0][0] + 4 * t, s.xb + ((int64_t)q * s.rows + r0) * kFeat + 4 * t);
            }
            if (t < kRowStep / 4) copy16(&c.dy[4 * t], s.dy + (int64_t)q * s.rows + r0 + 4 * t);
        }
        copy_commit();
    };
    static_assert(kRowStep * kFeat == kSmallUnits * kRowStep, "copy shape");
    for (int k = 0; k < kSteps - 1; ++k) fetch(k);
    // dW1: unit t / 32, part v = (t / 4) % 8 (rows v, v + 8, ...), features
    // t % 4 and t % 4 + 4.  Biases and W3: 3 x 8 units x 16 parts, two per
    // thread (t and t + 256); b3: 16 more parts, in unit group 0.
    const int wu = t >> 5, wv = (t >> 2) & 7, wk = t & 3;
    float a0 = 0.0f, a1 = 0.0f, c0 = 0.0f, c1 = 0.0f;
    const int e1 = t + kReduceThreads;
    const int kind0 = t / 128, unit0 = (t >> 4) & 7, v0 = t & 15;
    const int kind1 = e1 / 128, unit1 = (e1 >> 4) & 7, v1 = e1 & 15;  // kind 2: dW3, 3: db3 (e1 >= 384)
    for (int k = 0; k < steps; ++k) {
        copy_wait<kSteps - 2>();
        __syncthreads();
        fetch(k + kSteps - 1);
        const SmallTile& c = st[k % kSteps];
        const int rows = n - k * kRowStep < kRowStep ? n - k * kRowStep : kRowStep;
        for (int r = wv; r < rows; r += 8) {
            const float d = c.dh1[wu][r];
            a0 = fmaf(d, c.xb[r][wk], a0);
            a1 = fmaf(d, c.xb[r][wk + 4], a1);
        }
        for (int r = v0; r < rows; r += 16) c0 += kind0 ? c.dh2[unit0][r] : c.dh1[unit0][r];
        if (kind1 == 2) {
            for (int r = v1; r < rows; r += 16) c1 = fmaf(c.dy[r], c.h2[unit1][r], c1);
        } else if (g == 0 && e1 < 400) {
            for (int r = v1; r < rows; r += 16) c1 += c.dy[r];
        }
    }
    // part u = b mod 32 (or 64) is row set q, rows v modulo 8 (or 16)
    float* pw = s.p_w1 + (int64_t)(q + 4 * wv) * kHid * kFeat + (i0 + wu) * kFeat;
    pw[wk] = a0;
    pw[wk + 4] = a1;
    s.p_b[(q + 4 * v0) * kBiasParts + kind0 * kHid + i0 + unit0] = c0;
    if (kind1 == 2) s.p_b[(q + 4 * v1) * kBiasParts + 2 * kHid + i0 + unit1] = c1;
    else if (g == 0 && e1 < 400) s.p_b[(q + 4 * v1) * kBiasParts + 3 * kHid] = c1;
}

// One more block than these sums the loss.
constexpr int kParamThreads = 128;
constexpr int kParamBlocks = (kParams + kParamThreads - 1) / kParamThreads;

// kParts values in order, all loads in flight at once.
template <int kParts>
__device__ __forceinline__ float sum_parts(const float* p, int stride)
{
    float x[kParts], r = 0.0f;
#pragma unroll
    for (int u = 0; u < kParts; ++u) x[u] = __ldcg(p + u * stride);
#pragma unroll
    for (int u = 0; u < kParts; ++u) r += x[u];
    return r;
}

// Parameter k's gradient from the partial sums, added in part order.
__device__ __forceinline__ float grad_of(const Scratch& s, int k)
{
    if (k >= kOffW2 && k < kOffB2) {
        const float* p = s.p_w2 + (k - kOffW2);
        constexpr int n = kHid * kHid;
        return (__ldcg(p) + __ldcg(p + n)) + (__ldcg(p + 2 * n) + __ldcg(p + 3 * n));
    }
    if (k < kOffB1) return sum_parts<32>(s.p_w1 + k, kHid * kFeat);
    return sum_parts<64>(s.p_b + (k < kOffW2 ? k - kOffB1 : kHid + (k - kOffB2)), kBiasParts);
}

// The batch's loss from the per-32-sample sums, by one warp: groups of four,
// one per lane, added in order; the running sum over an epoch in loss_out[1].
__device__ __forceinline__ void sum_loss(const Scratch& s, int B, float inv_b, float* loss_out)
{
    const int lane = threadIdx.x & 31;
    const int np = (B + kFbSamples - 1) / kFbSamples;
    float l = 0.0f;
    for (int u0 = 0; u0 < np; u0 += 128) {
        float t = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int u = u0 + 4 * lane + k;
            t += u < np ? __ldcg(s.loss_part + u) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < 32; ++k) l += __shfl_sync(0xffffffffu, t, k);  // past the end: + 0
    }
    if (lane == 0) {
        loss_out[0] = l * inv_b;
        loss_out[1] = __ldcg(loss_out + 1) + l * inv_b;
    }
}

__global__ void grad_kernel(int B, float inv_b, Scratch s, float* __restrict__ g, float* __restrict__ loss_out)
{
    if (blockIdx.x == kParamBlocks) {
        if (threadIdx.x < 32) sum_loss(s, B, inv_b, loss_out);
        return;
    }
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < kParams) g[k] = grad_of(s, k);
}

__global__ void __launch_bounds__(kParamThreads) adam_kernel(int B, float inv_b, Scratch s, float* P, float* m,
                                                             float* v, float lr, float b1, float b2, float c1,
                                                             float c2, float eps, float* loss_out)
{
    // The parameter and its moments are those of the step before, which has
    // completed (the kernels between have waited for it).
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = k < kParams;
    const float p0 = live ? __ldcg(P + k) : 0.0f, m0 = live ? __ldcg(m + k) : 0.0f, v0 = live ? __ldcg(v + k) : 0.0f;
    wait_for_chain();
    if (blockIdx.x == kParamBlocks) {
        if (threadIdx.x < 32) sum_loss(s, B, inv_b, loss_out);
        return;
    }
    if (!live) return;
    const float gk = grad_of(s, k);
    const float mk = fmaf(1.0f - b1, gk, b1 * m0);
    const float vk = fmaf((1.0f - b2) * gk, gk, b2 * v0);
    m[k] = mk;
    v[k] = vk;
    P[k] = p0 - lr * (mk * c1) / (sqrtf(vk * c2) + eps);
}

// Standardisation of the features and labels (FP64 sums, as the scaling's
// definition; one thread per feature and row class, columns 8 = the label).
constexpr int kStdBlocks = 128, kStdThreads = 288;  // 32 rows x 9 columns
struct StdScratch {
    double sum[kStdBlocks][9], sq[kStdBlocks][9];
    float lo[kStdBlocks][kFeat], hi[kStdBlocks][kFeat];
    MlpScale sc;
    float loss[2];
};

__global__ void __launch_bounds__(kStdThreads) std_sum_kernel(int64_t n, const float* __restrict__ X,
                                                             const float* __restrict__ T, StdScratch* s)
{
    __shared__ double ps[kStdThreads], pq[kStdThreads];
    const int c = threadIdx.x % 9, r = threadIdx.x / 9;
    double a = 0.0, q = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * 32 + r; i < n; i += 32 * kStdBlocks) {
        const double v = c < kFeat ? X[i * kFeat + c] : T[i];
        a += v;
        q += v * v;
    }
    ps[threadIdx.x] = a;
    pq[threadIdx.x] = q;
    __syncthreads();
    if (threadIdx.x < 9) {
        for (int k = 1; k < 32; ++k) {
            a += ps[9 * k + c];
            q += pq[9 * k + c];
        }
        s->sum[blockIdx.x][c] = a;
        s->sq[blockIdx.x][c] = q;
    }
}

// Warp c: column c.
__global__ void __launch_bounds__(kStdThreads) std_scale_kernel(int64_t n, StdScratch* s)
{
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double a = 0.0, q = 0.0;
#pragma unroll
    for (int k = lane; k < kStdBlocks; k += 32) {
        a += s->sum[k][c];
        q += s->sq[k][c];
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        q += __shfl_xor_sync(0xffffffffu, q, off);
    }
    if (lane > 0) return;
    const double mu = a / n, v = q / n - mu * mu, var = v < 1e-12 ? 1e-12 : v;
    if (c < kFeat) {
        s->sc.mean[c] = (float)mu;
        s->sc.inv_std[c] = (float)(1.0 / sqrt(var));
    } else {
        s->sc.lmean = (float)mu;
        s->sc.lstd = (float)sqrt(var);
    }
}

__global__ void __launch_bounds__(kStdThreads) std_apply_kernel(int64_t n, float* __restrict__ X, float* __restrict__ T,
                                                               StdScratch* s)
{
    __shared__ float pl[kStdThreads], ph[kStdThreads];
    const int c = threadIdx.x % 9, r = threadIdx.x / 9;
    const float mean = c < kFeat ? s->sc.mean[c] : s->sc.lmean, inv = c < kFeat ? s->sc.inv_std[c] : 0.0f;
    const float lstd = s->sc.lstd;
    float lo = 1e30f, hi = -1e30f;
    for (int64_t i = (int64_t)blockIdx.x * 32 + r; i < n; i += 32 * kStdBlocks) {
        if (c < kFeat) {
            const float z = (X[i * kFeat + c] - mean) * inv;
            X[i * kFeat + c] = z;
            lo = z < lo ? z : lo;
            hi = hi < z ? z : hi;
        } else {
            T[i] = __fdiv_rn(T[i] - mean, lstd);
        }
    }
    pl[threadIdx.x] = lo;
    ph[threadIdx.x] = hi;
    __syncthreads();
    if (threadIdx.x < kFeat) {
        for (int k = 1; k < 32; ++k) {
            lo = fminf(lo, pl[9 * k + c]);
            hi = fmaxf(hi, ph[9 * k + c]);
        }
        s->lo[blockIdx.x][c] = lo;
        s->hi[blockIdx.x][c] = hi;
    }
}

__global__ void __launch_bounds__(32 * kFeat) std_range_kernel(StdScratch* s)
{
    const int c = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float lo = 1e30f, hi = -1e30f;
#pragma unroll
    for (int k = lane; k < kStdBlocks; k += 32) {
        lo = fminf(lo, s->lo[k][c]);
        hi = fmaxf(hi, s->hi[k][c]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
    }
    if (lane == 0) {
        s->sc.lo[c] = lo;
        s->sc.hi[c] = hi;
    }
}

struct DevBuf {
    std::vector<void*> ptrs;
    ~DevBuf()
    {
        for (void* p : ptrs) cudaFree(p);
    }
    template <class T>
    T* alloc(size_t count)
    {
        void* p = nullptr;
        if (cudaMalloc(&p, sizeof(T) * std::max<size_t>(count, 1)) != cudaSuccess) return nullptr;
        ptrs.push_back(p);
        return static_cast<T*>(p);
    }
};

bool alloc_scratch(DevBuf& d, int B, Scratch& s)
{
    s.rows = ((B + 3) / 4 + kRowStep - 1) / kRowStep * kRowStep;
    const size_t r = 4 * (size_t)s.rows;
    // One allocation: the arrays above, each a multiple of 64 floats.
    const size_t len[] = {r * kHid, r * kFeat, r * kHid, r * kHid, r * kHid, r, (size_t)(B / kFbSamples + 64),
                          (size_t)4 * kHid * kHid, (size_t)32 * kHid * kFeat, (size_t)64 * kBiasParts};
    float** to[] = {&s.h1, &s.xb, &s.dh1, &s.dh2, &s.h2, &s.dy, &s.loss_part, &s.p_w2, &s.p_w1, &s.p_b};
    size_t total = 0;
    for (size_t n : len) total += (n + 63) / 64 * 64;
    float* p = d.alloc<float>(total);
    if (!p) return false;
    for (int k = 0; k < 10; ++k) {
        *to[k] = p;
        p += (len[k] + 63) / 64 * 64;
    }
    return true;
}

// Forward, backward and the gradient's partial sums of one batch.
int fwd_bwd(const float* X, const float* T, const int32_t* idx, int64_t off, int B, const float* P, Scratch& s,
            cudaStream_t st)
{
    BH_CUDA_TRY(cudaFuncSetAttribute(mlp_fwd_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(FbSmem)));
    BH_CUDA_TRY(cudaFuncSetAttribute(mlp_grad_reduce_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kReduceSmem));
    BH_CUDA_TRY(launch_in_chain(mlp_fwd_bwd_kernel, (B + kFbSamples - 1) / kFbSamples, kFbThreads, sizeof(FbSmem), st, X,
                                T, idx, off, B, 1.0f / (float)B, P, s));
    BH_CUDA_TRY(launch_in_chain(mlp_grad_reduce_kernel, kW2Blocks + kSmallBlocks, kReduceThreads, kReduceSmem, st, B,
                                s));
    return BH_OK;
}

}  // namespace
}  // namespace bh

using namespace bh;

extern "C" int bh_mlp_gradient(const float* params, const float* X, const float* T, int64_t n, float* grad_out,
                               float* loss_out)
{
    if (!params || !X || !T || !grad_out || n <= 0 || n > (1 << 20))
        return bh_fail(BH_ERR_INVALID_ARGUMENT, "bh_mlp_gradient: bad arguments (n in [1, 2^20])");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return bh_fail(BH_ERR_NO_DEVICE, "bh_mlp_gradient: no CUDA device");
    }
    DevBuf d;
    float* dP = d.alloc<float>(kParams);
    float* dX = d.alloc<float>((size_t)n * kFeat);
    float* dT = d.alloc<float>(n);
    float* dG = d.alloc<float>(kParams);
    float* dL = d.alloc<float>(2);
    Scratch s;
    if (!dP || !dX || !dT || !dG || !dL || !alloc_scratch(d, (int)n, s))
        return bh_fail(BH_ERR_OUT_OF_MEMORY, "bh_mlp_gradient: device allocation failed");
    BH_CUDA_TRY(cudaMemcpy(dP, params, sizeof(float) * kParams, cudaMemcpyHostToDevice));
    BH_CUDA_TRY(cudaMemcpy(dX, X, sizeof(float) * n * kFeat, cudaMemcpyHostToDevice));
    BH_CUDA_TRY(cudaMemcpy(dT, T, sizeof(float) * n, cudaMemcpyHostToDevice));
    int rc = fwd_bwd(dX, dT, nullptr, 0, (int)n, dP, s, 0);
    if (rc) return rc;
    grad_kernel<<<kParamBlocks + 1, kParamThreads>>>((int)n, 1.0f / (float)n, s, dG, dL);
    BH_CUDA_TRY(cudaGetLastError());
    BH_CUDA_TRY(cudaMemcpy(grad_out, dG, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
    if (loss_out) BH_CUDA_TRY(cudaMemcpy(loss_out, dL, sizeof(float), cudaMemcpyDeviceToHost));
    return BH_OK;
}

extern "C" int bh_mlp_train(const float* features, const float* labels, int64_t n, int epochs, int batch, float lr,
                            uint64_t seed, float* params_out, float* scale_out, float* loss_out)
{
    if (!features || !labels || !params_out || !scale_out || n < 16 || epochs < 1 || batch < 16 || batch > (1 << 16) ||
        !(lr > 0))
        return bh_fail(BH_ERR_INVALID_ARGUMENT, "bh_mlp_train: bad arguments");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return bh_fail(BH_ERR_NO_DEVICE, "bh_mlp_train: no CUDA device");
    }
    // He-normal initialisation, zero biases.
    std::mt19937_64 rng(seed);
    std::normal_distribution<double> nd(0.0, 1.0);
    std::vector<float> P(kParams, 0.0f);
    for (int k = 0; k < kHid * kFeat; ++k) P[kOffW1 + k] = (float)(nd(rng) * std::sqrt(2.0 / kFeat));
    for (int k = 0; k < kHid * kHid; ++k) P[kOffW2 + k] = (float)(nd(rng) * std::sqrt(2.0 / kHid));
    for (int k = 0; k < kHid; ++k) P[kOffW3 + k] = (float)(nd(rng) * std::sqrt(1.0 / kHid));

    DevBuf d;
    float* dP = d.alloc<float>(3 * kParams);  // parameters and the two moments
    float* dM = dP + kParams;
    float* dV = dM + kParams;
    float* dX = d.alloc<float>((size_t)n * (kFeat + 2));  // features, labels, order
    float* dT = dX + (size_t)n * kFeat;
    int32_t* dI = reinterpret_cast<int32_t*>(dT + n);
    StdScratch* dS = d.alloc<StdScratch>(1);
    Scratch s;
    const int B = (int)std::min<int64_t>(batch, n);
    if (!dP || !dX || !dS || !alloc_scratch(d, B, s))
        return bh_fail(BH_ERR_OUT_OF_MEMORY, "bh_mlp_train: device allocation failed");
    float* dL = dS->loss;
    BH_CUDA_TRY(cudaMemcpy(dP, P.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice));
    BH_CUDA_TRY(cudaMemsetAsync(dM, 0, sizeof(float) * 2 * kParams));
    BH_CUDA_TRY(cudaMemcpy(dX, features, sizeof(float) * n * kFeat, cudaMemcpyHostToDevice));
    BH_CUDA_TRY(cudaMemcpy(dT, labels, sizeof(float) * n, cudaMemcpyHostToDevice));
    // Standardisation in place.
    std_sum_kernel<<<kStdBlocks, kStdThreads>>>(n, dX, dT, dS);
    BH_CUDA_TRY(cudaGetLastError());
    std_scale_kernel<<<1, kStdThreads>>>(n, dS);
    BH_CUDA_TRY(cudaGetLastError());
    std_apply_kernel<<<kStdBlocks, kStdThreads>>>(n, dX, dT, dS);
    BH_CUDA_TRY(cudaGetLastError());
    std_range_kernel<<<1, 32 * kFeat>>>(dS);
    BH_CUDA_TRY(cudaGetLastError());
    std::vector<int32_t> order(n);
    std::iota(order.begin(), order.end(), 0);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    int64_t step = 0;
    const int64_t nb = n / B;  // full batches only
    std::shuffle(order.begin(), order.end(), rng);
    for (int e = 0; e < epochs; ++e) {
        BH_CUDA_TRY(cudaMemcpy(dI, order.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice));
        BH_CUDA_TRY(cudaMemset(dL, 0, 2 * sizeof(float)));
        for (int64_t k = 0; k < nb; ++k) {
            int rc = fwd_bwd(dX, dT, dI, k * B, B, dP, s, 0);
            if (rc) return rc;
            ++step;
            const float c1 = 1.0f / (1.0f - std::pow(b1, (float)step));
            const float c2 = 1.0f / (1.0f - std::pow(b2, (float)step));
            BH_CUDA_TRY(launch_in_chain(adam_kernel, kParamBlocks + 1, kParamThreads, 0, 0, B, 1.0f / (float)B, s, dP,
                                        dM, dV, lr, b1, b2, c1, c2, eps, dL));
        }
        // the next epoch's order, while the device works on this one
        if (e + 1 < epochs) std::shuffle(order.begin(), order.end(), rng);
        float l[2] = {0.f, 0.f};
        BH_CUDA_TRY(cudaMemcpy(l, dL, 2 * sizeof(float), cudaMemcpyDeviceToHost));
        if (loss_out) loss_out[e] = l[1] / (float)std::max<int64_t>(nb, 1);  // mean batch loss of the epoch
    }
    BH_CUDA_TRY(cudaMemcpy(params_out, dP, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
    BH_CUDA_TRY(cudaMemcpy(scale_out, &dS->sc, sizeof(MlpScale), cudaMemcpyDeviceToHost));
    return BH_OK;
}
