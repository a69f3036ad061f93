// nbh_theta.cu — learned per-body opening angle (no counterpart in the reference).
//
// A small MLP 12 -> 64 -> 64 -> 1 (ReLU) maps per-body features of the current tree and
// of the previous force walk to log(theta).  Inference runs once per step between the sort
// and the force stages: BF16 weights and activations on the tensor cores (mma.sync
// m16n8k16, FP32 accumulation), one warp per 32 bodies of the depth-first order.  Training
// uses the FP32 kernels at the end of this file (forward, backward, batch reductions, Adam).
//
// Parameter layout (row-major FP32, kMlpParams floats):
//   W1[64][12] b1[64] W2[64][64] b2[64] W3[64] b3
#include "nbh_common.cuh"
#include "nbh_kernels.h"
#include "nbh_theta.h"

#include <algorithm>

#include <cuda_bf16.h>

namespace nbh {

// ---- features -------------------------------------------------------------------------
// Per body, from the current tree (after sort) and the previous force walk (acc: previous
// acceleration, acc.w: its quadrupole error bound; theta_prev: the angle that walk used):
//   0 log10|a|             1 log10(bound/|a|)      2 log10 theta_prev
//   3 log10(d/R)           4 log10(n_leaf + 1)     5 level(leaf)/20
//   6 log10(n_up2 + 1)     7 log10(n_leaf/h^3)     8 log10(m_leaf/M)
//   9 log10(|a| d^2 / M)  10 log10(eps/h)         11 log10(h/d)
// d: distance to the universe's centre of mass, R and M: root half-width and mass, leaf:
// the cell holding the body, h: its half-width, up2: the leaf's parent (or the leaf if it
// is the root).
__device__ __forceinline__ void body_features(const StepParams& p, const ThetaDev& m, int b, int u, float4 a,
                                              float theta_prev, float f[kMlpIn]) {
    const int nbody = p.nbody;
    const float4 x = p.node4[b];
    const int root = p.nnodes - u;
    const float4 rc = p.node4[root];
    const float R = p.uradius[u];
    const float M = rc.w;
    const int leaf = p.parent[b];
    const int up = p.parent[leaf] >= 0 ? p.parent[leaf] : leaf;
    const int lv = p.clevel[leaf - nbody];
    const float h = ldexpf(R, -lv);
    const float nl = (float)p.count[leaf - nbody];
    const float nu = (float)p.count[up - nbody];
    const float ml = p.node4[leaf].w;
    const float dx = x.x - rc.x, dy = x.y - rc.y, dz = x.z - rc.z;
    const float d = sqrtf(dx * dx + dy * dy + dz * dz) + 1e-12f;
    const float am = sqrtf(a.x * a.x + a.y * a.y + a.z * a.z) + 1e-30f;
    const float eps = sqrtf(p.eps2);
    f[0] = log10f(am);
    f[1] = log10f(fmaxf(a.w, 0.0f) / am + 1e-30f);
    f[2] = log10f(fmaxf(theta_prev, 1e-6f));
    f[3] = log10f(d / R + 1e-12f);
    f[4] = log10f(nl + 1.0f);
    f[5] = (float)lv * 0.05f;
    f[6] = log10f(nu + 1.0f);
    f[7] = log10f(nl / (h * h * h) + 1e-30f);
    f[8] = log10f(fmaxf(ml, 0.0f) / M + 1e-30f);
    f[9] = log10f(am * d * d / M + 1e-30f);
    f[10] = log10f(eps / h);
    f[11] = log10f(h / d);
}

// ---- BF16 tensor-core inference -------------------------------------------------------
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const unsigned*>(&v);
}

__device__ __forceinline__ void mma_bf16(float c[4], const unsigned a[4], const unsigned b[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

constexpr int kThetaThreads = 128;

// Shared-memory image of the model: weights as BF16 (W1 padded to K = 16, W3 as an 8 x 64
// tile whose row 0 is W3), biases FP32.
struct ThetaSmem {
    __nv_bfloat16 w1[kMlpHid * 16];
    __nv_bfloat16 w2[kMlpHid * kMlpHid];
    __nv_bfloat16 w3[8 * kMlpHid];
    float b1[kMlpHid];
    float b2[kMlpHid];
    float x[kThetaThreads / 32][32][16];   // normalized features of the warp's 32 bodies
};

// One warp: 32 bodies (rows) through the three layers.  Fragment layouts of
// mma.m16n8k16: A reg0 = (row g, k 2t..2t+1), reg1 = (row g+8, ...), reg2 = (row g, k+8),
// reg3 = (row g+8, k+8); B reg0 = (k 2t..2t+1, col g), reg1 = (k+8); C c0,c1 = (row g,
// cols 2t, 2t+1), c2,c3 = (row g+8).  A C tile pair (cols 16k..16k+15) is the A fragment
// of the next layer's k-tile k.
__device__ __forceinline__ void mlp_warp(const ThetaSmem& S, const float (*xs)[16], float b3, int lane,
                                         float out[2][2]) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
        const int r0 = mt * 16 + g, r1 = r0 + 8;
        unsigned a1[4];
        a1[0] = pack_bf16(xs[r0][2 * t], xs[r0][2 * t + 1]);
        a1[1] = pack_bf16(xs[r1][2 * t], xs[r1][2 * t + 1]);
        a1[2] = pack_bf16(xs[r0][2 * t + 8], xs[r0][2 * t + 9]);
        a1[3] = pack_bf16(xs[r1][2 * t + 8], xs[r1][2 * t + 9]);
        // layer 1
        unsigned a2[4][4];
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
            float c[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int nt = 2 * kt + h;
                const int n = nt * 8 + g;
                unsigned bf[2];
                bf[0] = *reinterpret_cast<const unsigned*>(&S.w1[n * 16 + 2 * t]);
                bf[1] = *reinterpret_cast<const unsigned*>(&S.w1[n * 16 + 2 * t + 8]);
                c[h][0] = c[h][1] = c[h][2] = c[h][3] = 0.f;
                mma_bf16(c[h], a1, bf);
                const float bb0 = S.b1[nt * 8 + 2 * t], bb1 = S.b1[nt * 8 + 2 * t + 1];
                c[h][0] = fmaxf(c[h][0] + bb0, 0.f);
                c[h][1] = fmaxf(c[h][1] + bb1, 0.f);
                c[h][2] = fmaxf(c[h][2] + bb0, 0.f);
                c[h][3] = fmaxf(c[h][3] + bb1, 0.f);
            }
            a2[kt][0] = pack_bf16(c[0][0], c[0][1]);
            a2[kt][1] = pack_bf16(c[0][2], c[0][3]);
            a2[kt][2] = pack_bf16(c[1][0], c[1][1]);
            a2[kt][3] = pack_bf16(c[1][2], c[1][3]);
        }
        // layer 2, with layer 3 folded in k-tile by k-tile
        float c3[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int kt3 = 0; kt3 < 4; ++kt3) {
            float c[2][4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int nt = 2 * kt3 + h;
                const int n = nt * 8 + g;
                c[h][0] = c[h][1] = c[h][2] = c[h][3] = 0.f;
#pragma unroll
                for (int kt = 0; kt < 4; ++kt) {
                    unsigned bf[2];
                    bf[0] = *reinterpret_cast<const unsigned*>(&S.w2[n * kMlpHid + kt * 16 + 2 * t]);
                    bf[1] = *reinterpret_cast<const unsigned*>(&S.w2[n * kMlpHid + kt * 16 + 2 * t + 8]);
                    mma_bf16(c[h], a2[kt], bf);
                }
                const float bb0 = S.b2[nt * 8 + 2 * t], bb1 = S.b2[nt * 8 + 2 * t + 1];
                c[h][0] = fmaxf(c[h][0] + bb0, 0.f);
                c[h][1] = fmaxf(c[h][1] + bb1, 0.f);
                c[h][2] = fmaxf(c[h][2] + bb0, 0.f);
                c[h][3] = fmaxf(c[h][3] + bb1, 0.f);
            }
            unsigned a3[4];
            a3[0] = pack_bf16(c[0][0], c[0][1]);
            a3[1] = pack_bf16(c[0][2], c[0][3]);
            a3[2] = pack_bf16(c[1][0], c[1][1]);
            a3[3] = pack_bf16(c[1][2], c[1][3]);
            unsigned bf[2];
            bf[0] = *reinterpret_cast<const unsigned*>(&S.w3[g * kMlpHid + kt3 * 16 + 2 * t]);
            bf[1] = *reinterpret_cast<const unsigned*>(&S.w3[g * kMlpHid + kt3 * 16 + 2 * t + 8]);
            mma_bf16(c3, a3, bf);
        }
        // column 0 of the output tile: thread t == 0 holds rows g (c3[0]) and g+8 (c3[2])
        out[mt][0] = c3[0] + b3;
        out[mt][1] = c3[2] + b3;
    }
}

__device__ __forceinline__ void load_model(ThetaSmem& S, const ThetaDev& m) {
    for (int i = threadIdx.x; i < kMlpHid * 16; i += blockDim.x) S.w1[i] = m.w1[i];
    for (int i = threadIdx.x; i < kMlpHid * kMlpHid; i += blockDim.x) S.w2[i] = m.w2[i];
    for (int i = threadIdx.x; i < 8 * kMlpHid; i += blockDim.x) S.w3[i] = m.w3[i];
    for (int i = threadIdx.x; i < kMlpHid; i += blockDim.x) {
        S.b1[i] = m.b1[i];
        S.b2[i] = m.b2[i];
    }
}

// Per-body theta of this step.  Up to the step at which the model was switched on
// (theta_since; the first step after a load) there is no previous walk with error bounds:
// every body gets the fixed theta.  Otherwise theta = clamp(exp(MLP(features)), min, max).
__global__ void __launch_bounds__(kThetaThreads) theta_kernel(StepParams p, const ThetaDev* __restrict__ mdl,
                                                              float* theta_out) {
    if (load_status(p.st)) return;
    __shared__ ThetaSmem S;
    const ThetaDev& m = *mdl;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int step = p.st->step;
    const bool use_fixed = step <= p.st->theta_since;   // no previous walk with bounds yet
    if (!use_fixed && !theta_model_step(p.st, step)) return;   // angles kept from the last evaluation
    const float fixed = sqrtf(p.theta2);
    if (!use_fixed) load_model(S, m);
    __syncthreads();
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int item = blockIdx.x * (blockDim.x >> 5) + wid; item < p.nwarps; item += warps) {
        const int2 wi = p.warps[item];
        const int u = wi.y;
        const int s = wi.x + lane;
        const bool valid = s < p.ubody[u + 1];
        const int b = p.sorted[valid ? s : wi.x];
        if (use_fixed) {
            if (valid) theta_out[b] = fixed;
            continue;
        }
        float f[kMlpIn];
        body_features(p, m, b, u, p.acc[b], theta_out[b], f);
#pragma unroll
        for (int k = 0; k < kMlpIn; ++k) S.x[wid][lane][k] = (f[k] - m.mean[k]) * m.inv_std[k];
#pragma unroll
        for (int k = kMlpIn; k < 16; ++k) S.x[wid][lane][k] = 0.f;
        __syncwarp();
        float out[2][2];
        mlp_warp(S, S.x[wid], m.b3, lane, out);
        __syncwarp();
        if ((lane & 3) == 0) {
            const int g = lane >> 2;
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int row = mt * 16 + g + 8 * h;
                    if (wi.x + row < p.ubody[u + 1]) {
                        const int br = p.sorted[wi.x + row];
                        theta_out[br] = fminf(fmaxf(__expf(out[mt][h]), m.theta_min), m.theta_max);
                    }
                }
        }
    }
}

// Raw features of every body (for training data and tests).  src: previous acceleration
// and bound per body; theta_prev: per-body angle of that walk.
__global__ void features_kernel(StepParams p, const ThetaDev* __restrict__ mdl, const float4* src,
                                const float* theta_prev, float* feat) {
    const int stride = gridDim.x * blockDim.x;
    for (int item = blockIdx.x * blockDim.x + threadIdx.x; item < p.nbody; item += stride) {
        // position item of the depth-first order, so neighbouring threads share cells
        int u = 0;
        while (p.ubody[u + 1] <= item) ++u;
        const int b = p.sorted[item];
        float f[kMlpIn];
        body_features(p, *mdl, b, u, src[b], theta_prev[b], f);
#pragma unroll
        for (int k = 0; k < kMlpIn; ++k) feat[(size_t)b * kMlpIn + k] = f[k];
    }
}

// Model upload: FP32 parameters -> BF16 tiles + FP32 biases.
__global__ void model_convert_kernel(const float* __restrict__ prm, ThetaDev* mdl) {
    const float* W1 = prm;
    const float* b1 = W1 + kMlpHid * kMlpIn;
    const float* W2 = b1 + kMlpHid;
    const float* b2 = W2 + kMlpHid * kMlpHid;
    const float* W3 = b2 + kMlpHid;
    const float b3 = W3[kMlpHid];
    for (int i = threadIdx.x; i < kMlpHid * 16; i += blockDim.x) {
        const int n = i / 16, k = i % 16;
        mdl->w1[i] = __float2bfloat16_rn(k < kMlpIn ? W1[n * kMlpIn + k] : 0.f);
    }
    for (int i = threadIdx.x; i < kMlpHid * kMlpHid; i += blockDim.x) mdl->w2[i] = __float2bfloat16_rn(W2[i]);
    for (int i = threadIdx.x; i < 8 * kMlpHid; i += blockDim.x)
        mdl->w3[i] = __float2bfloat16_rn(i < kMlpHid ? W3[i] : 0.f);
    for (int i = threadIdx.x; i < kMlpHid; i += blockDim.x) {
        mdl->b1[i] = b1[i];
        mdl->b2[i] = b2[i];
    }
    if (threadIdx.x == 0) mdl->b3 = b3;
}

void launch_theta(const StepParams& p, const ThetaDev* mdl, float* theta_out, int grid, cudaStream_t s) {
    theta_kernel<<<grid, kThetaThreads, 0, s>>>(p, mdl, theta_out);
}
void launch_features(const StepParams& p, const ThetaDev* mdl, const float4* src, const float* theta_prev,
                     float* feat, int grid, cudaStream_t s) {
    features_kernel<<<grid, 256, 0, s>>>(p, mdl, src, theta_prev, feat);
}
void launch_model_convert(const float* prm, ThetaDev* mdl, cudaStream_t s) {
    model_convert_kernel<<<1, 256, 0, s>>>(prm, mdl);
}

// ---- FP32 training kernels ------------------------------------------------------------
// One pass over the batch takes three kernels.  The sample kernel runs tiles of 64 samples
// through both layers, the loss and the backward pass in shared memory (64 x 64 x 64 products,
// 8 x 4 outputs per thread from 16-byte shared loads) and writes the tiles' activations and
// their gradients out once.  The weight kernel contracts them over the samples, in at most 64
// chunks, each output one chain of multiply-adds in sample order; a last kernel adds the
// chunks and takes the Adam step.  13,900 multiply-adds per sample, 35 us for 100,000
// samples at the FMA rate.  The order of every sum is fixed.
constexpr int kTrainThreads = 128;
constexpr int kTile = 64;              // samples per tile
constexpr int kRow = kTile + 4;        // floats per row: neighbouring rows 4 banks apart
constexpr int kTrainBlocksPerSm = 3;

// What the sample kernel leaves of a tile (feature- and unit-major).
struct TrainTile {
    float h1[kMlpHid][kRow], h2[kMlpHid][kRow], d2[kMlpHid][kRow], d1[kMlpHid][kRow];
    float x[kMlpIn][kRow];
    float dy[kRow];
};
static_assert(sizeof(TrainTile) % 16 == 0, "tiles are copied 16 bytes at a time");

struct TrainSmem {
    float w1[kMlpHid][kMlpIn];
    float w2[kMlpHid][kRow];
    float b1[kMlpHid], b2[kMlpHid], w3[kMlpHid];
    float x[kMlpIn][kRow];
    float h1[kMlpHid][kRow];
    float d[kMlpHid][kRow];            // h2, then its gradient, then h1's
    float dy[kRow];
    float b3, red[2];
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float* v) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
// acc[0..7] += w * (lo, hi): the thread's eight samples 4 ts .. 4 ts + 3 and those 32 further
__device__ __forceinline__ void fma8(float (&acc)[8], const float w, const float4 lo, const float4 hi) {
    acc[0] = fmaf(w, lo.x, acc[0]), acc[1] = fmaf(w, lo.y, acc[1]);
    acc[2] = fmaf(w, lo.z, acc[2]), acc[3] = fmaf(w, lo.w, acc[3]);
    acc[4] = fmaf(w, hi.x, acc[4]), acc[5] = fmaf(w, hi.y, acc[5]);
    acc[6] = fmaf(w, hi.z, acc[6]), acc[7] = fmaf(w, hi.w, acc[7]);
}
template <int THREADS>
__device__ __forceinline__ void copy_rows(float* dst, const float* src, int rows, int t) {
    for (int i = 4 * t; i < rows * kRow; i += 4 * THREADS)
        *reinterpret_cast<float4*>(dst + i) = ld4(src + i);
}

// GRAD: pinball (quantile q) loss against T, mean over the batch (one partial sum per block),
// and the tiles with their gradients; otherwise the outputs into Y.
template <bool GRAD>
__global__ void __launch_bounds__(kTrainThreads, kTrainBlocksPerSm)
    mlp_samples_kernel(const float* __restrict__ prm, const float* __restrict__ X, const float* __restrict__ T, int n,
                       float q, float* __restrict__ Y, TrainTile* __restrict__ out, float* __restrict__ lossp) {
    extern __shared__ __align__(16) unsigned char train_smem[];
    TrainSmem& S = *reinterpret_cast<TrainSmem*>(train_smem);
    const int tid = threadIdx.x;
    const int ts = tid & 7, tu = tid >> 3;            // sample group, unit group
    {
        const float* g = prm;
        for (int i = tid; i < kMlpHid * kMlpIn; i += kTrainThreads) S.w1[i / kMlpIn][i % kMlpIn] = g[i];
        g += kMlpHid * kMlpIn;
        for (int i = tid; i < kMlpHid; i += kTrainThreads) S.b1[i] = g[i];
        g += kMlpHid;
        for (int i = tid; i < kMlpHid * kMlpHid; i += kTrainThreads) S.w2[i / kMlpHid][i % kMlpHid] = g[i];
        g += kMlpHid * kMlpHid;
        for (int i = tid; i < kMlpHid; i += kTrainThreads) S.b2[i] = g[i], S.w3[i] = g[kMlpHid + i];
        if (tid == 0) S.b3 = g[2 * kMlpHid];
    }
    float lsum = 0.f;
    const float inv_n = 1.0f / (float)n;
    const int tiles = (n + kTile - 1) / kTile;
    // the features and targets of a tile are on their way while the tile before is worked on
    constexpr int kPerThread = kTile * kMlpIn / kTrainThreads;
    float nx[kPerThread], nt = 0.f;
    auto fetch = [&](int tile) {
        const size_t first = (size_t)tile * kTile;
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
            const int i = tid + k * kTrainThreads;
            nx[k] = first + i / kMlpIn < (size_t)n ? X[first * kMlpIn + i] : 0.f;
        }
        if (GRAD && tid < kTile) nt = first + tid < (size_t)n ? T[first + tid] : 0.f;
    };
    fetch(blockIdx.x);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int first = tile * kTile;
        __syncthreads();                              // the last tile's readers are done
#pragma unroll
        for (int k = 0; k < kPerThread; ++k) {
            const int i = tid + k * kTrainThreads;
            S.x[i % kMlpIn][i / kMlpIn] = nx[k];
        }
        const float target = nt;
        __syncthreads();
        fetch(tile + (int)gridDim.x);                 // past the last tile: zeros
        // layers 1 and 2: units tu + 16 i
        float acc[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[i][e] = S.b1[tu + 16 * i];
#pragma unroll
        for (int f = 0; f < kMlpIn; ++f) {
            const float4 lo = ld4(&S.x[f][4 * ts]), hi = ld4(&S.x[f][4 * ts + 32]);
#pragma unroll
            for (int i = 0; i < 4; ++i) fma8(acc[i], S.w1[tu + 16 * i][f], lo, hi);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[i][e] = fmaxf(acc[i][e], 0.f);
            st4(&S.h1[tu + 16 * i][4 * ts], acc[i]);
            st4(&S.h1[tu + 16 * i][4 * ts + 32], acc[i] + 4);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[i][e] = S.b2[tu + 16 * i];
#pragma unroll 2
        for (int k = 0; k < kMlpHid; k += 4) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = ld4(&S.w2[tu + 16 * i][k]);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const float4 lo = ld4(&S.h1[k + kk][4 * ts]), hi = ld4(&S.h1[k + kk][4 * ts + 32]);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    fma8(acc[i], kk == 0 ? w[i].x : (kk == 1 ? w[i].y : (kk == 2 ? w[i].z : w[i].w)), lo, hi);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[i][e] = fmaxf(acc[i][e], 0.f);
            st4(&S.d[tu + 16 * i][4 * ts], acc[i]);
            st4(&S.d[tu + 16 * i][4 * ts + 32], acc[i] + 4);
        }
        __syncthreads();
        // layer 3 and the loss on half of the threads; the others write the activations out
        if (tid < kTile) {
            float y = S.b3;
#pragma unroll 16
            for (int j = 0; j < kMlpHid; ++j) y = fmaf(S.w3[j], S.d[j][tid], y);
            const int s = first + tid;
            if constexpr (GRAD) {
                float dy = 0.f;
                if (s < n) {
                    const float r = target - y;
                    lsum += r > 0.f ? q * r : (q - 1.f) * r;
                    dy = (r > 0.f ? -q : 1.f - q) * inv_n;
                }
                S.dy[tid] = dy;
                out[tile].dy[tid] = dy;
            } else {
                if (s < n) Y[s] = y;
            }
        } else if constexpr (GRAD) {
            copy_rows<kTrainThreads - kTile>(out[tile].x[0], S.x[0], kMlpIn, tid - kTile);
            copy_rows<kTrainThreads - kTile>(out[tile].h1[0], S.h1[0], kMlpHid, tid - kTile);
            copy_rows<kTrainThreads - kTile>(out[tile].h2[0], S.d[0], kMlpHid, tid - kTile);
        }
        if constexpr (GRAD) {
            __syncthreads();
            // dh2 = dy W3 (h2 > 0)
            {
                const float4 lo = ld4(&S.dy[4 * ts]), hi = ld4(&S.dy[4 * ts + 32]);
                const float dy[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float w = S.w3[tu + 16 * i];
#pragma unroll
                    for (int e = 0; e < 8; ++e) acc[i][e] = acc[i][e] > 0.f ? dy[e] * w : 0.f;
                    st4(&S.d[tu + 16 * i][4 * ts], acc[i]);
                    st4(&S.d[tu + 16 * i][4 * ts + 32], acc[i] + 4);
                }
            }
            __syncthreads();
            // dh1 = W2^T dh2 (h1 > 0): units 4 tu + i
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[i][e] = 0.f;
#pragma unroll 8
            for (int j = 0; j < kMlpHid; ++j) {
                const float4 lo = ld4(&S.d[j][4 * ts]), hi = ld4(&S.d[j][4 * ts + 32]);
                const float4 w = ld4(&S.w2[j][4 * tu]);
                fma8(acc[0], w.x, lo, hi);
                fma8(acc[1], w.y, lo, hi);
                fma8(acc[2], w.z, lo, hi);
                fma8(acc[3], w.w, lo, hi);
            }
            copy_rows<kTrainThreads>(out[tile].d2[0], S.d[0], kMlpHid, tid);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 lo = ld4(&S.h1[4 * tu + i][4 * ts]), hi = ld4(&S.h1[4 * tu + i][4 * ts + 32]);
                const float h[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[i][e] = h[e] > 0.f ? acc[i][e] : 0.f;
            }
            // straight from the registers: eight lanes cover the 128 bytes of a row's half
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                st4(&out[tile].d1[4 * tu + i][4 * ts], acc[i]);
                st4(&out[tile].d1[4 * tu + i][4 * ts + 32], acc[i] + 4);
            }
        }
    }
    if constexpr (GRAD) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        if ((tid & 31) == 0 && tid < kTile) S.red[tid >> 5] = lsum;
        __syncthreads();
        if (tid == 0) lossp[blockIdx.x] = (S.red[0] + S.red[1]) * inv_n;
    }
}

// Weight gradients of one chunk of samples, each output one chain of multiply-adds in sample
// order.  blockIdx.x < 64 / R * Q: R rows of gW2 (and gb2) by 64 / Q columns, a thread rows
// tid % 8 + 8 i by every (THREADS / 8)-th column; the next Q blocks 64 / Q units of gW1 and gb1;
// the last Q as many of gW3, and gb3.  Tiles come in through stages of asynchronous copies (with
// two the kernel waited for them: 67 us a pass at 100,000 samples).
// <16, 1, 128, 4> for many chunks, bound by shared-memory loads (6 for 32 multiply-adds; 8 for 32
// with 256 threads: 135 us a training step at 100,000 samples against 125).
// <8, 4, 128, 8> for few chunks (small batches), whose blocks leave SMs idle while each walks its
// chunk tile after tile: smaller blocks copy and load a third per tile, and a
// warp's few instructions per tile (the steps unrolled, the copies' places worked out once) are
// what takes the time.  A training step at 5,000 samples 65.7 -> 41 us against <8, 1, 128, 4>, at
// 20,000 70 -> 57; at 100,000 (the copies' places only) 125 -> 122.
template <int R, int Q, int THREADS, int STAGES>
struct WeightSplit {
    static constexpr int kUnits = kMlpHid / Q;                            // columns or units of a block
    static constexpr int kRowBlocks = kMlpHid / R, kBlocks = kRowBlocks * Q + 2 * Q;
    static constexpr int kColGroups = THREADS / 8, kCols = kUnits / kColGroups;   // gW2 columns of a thread
    static constexpr int kFeatGroups = THREADS / kUnits;
    static constexpr int kFeat = (kMlpIn + kFeatGroups - 1) / kFeatGroups;        // gW1 features of a thread
    static constexpr int kRows = kUnits + (R > kMlpIn ? R : kMlpIn);              // of a stage
    static constexpr size_t kSmem = sizeof(float) * STAGES * kRows * kRow;
    static_assert(kCols * kColGroups == kUnits && kFeat * kFeatGroups >= kMlpIn && kUnits < THREADS,
                  "every output has a thread");
};
__device__ __forceinline__ void chain4(float& acc, const float4 a, const float4 b) {
    acc = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
__device__ __forceinline__ void sum4(float& acc, const float4 a) { acc = (((acc + a.x) + a.y) + a.z) + a.w; }

template <int R, int Q, int THREADS, int STAGES>
__global__ void __launch_bounds__(THREADS) mlp_weights_kernel(const TrainTile* __restrict__ in, int n,
                                                              float* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char train_smem[];
    using Split = WeightSplit<R, Q, THREADS, STAGES>;
    constexpr int kUnits = Split::kUnits, kCols = Split::kCols, kColGroups = Split::kColGroups, kFeat = Split::kFeat;
    constexpr int kStageFloats = Split::kRows * kRow;
    float* const buf = reinterpret_cast<float*>(train_smem);
    constexpr int RI = R / 8, kSteps = Q > 1 ? kTile / 4 : 4;      // four samples each, unrolled
    const int tid = threadIdx.x;
    const int chunk = (n + gridDim.y - 1) / gridDim.y;
    const int s0 = blockIdx.y * chunk, s1 = min(n, s0 + chunk);
    float* const g = part + (size_t)blockIdx.y * kMlpParams;
    const int bx = (int)blockIdx.x - Split::kRowBlocks * Q;
    const int kind = bx < 0 ? 0 : (bx < Q ? 1 : 2);                // gW2 rows, gW1, gW3
    const int row0 = R * ((int)blockIdx.x % Split::kRowBlocks);
    const int q = bx < 0 ? (int)blockIdx.x / Split::kRowBlocks : bx % Q;
    const int u0 = q * kUnits;                                     // first column or unit
    const int arows = kind == 0 ? R : (kind == 1 ? kUnits : 1);    // gradients; activations follow
    const int t0 = s0 / kTile, t1 = s1 > s0 ? (s1 + kTile - 1) / kTile : t0;
    // a tile comes as two runs of rows; this thread's 16-byte pieces of them
    constexpr int kTileFloats = sizeof(TrainTile) / sizeof(float);
    const float* const first = kind == 0 ? in->d2[row0] : (kind == 1 ? in->d1[u0] : in->dy);
    const float* const second = kind == 0 ? in->h1[u0] : (kind == 1 ? in->x[0] : in->h2[u0]);
    const int split = arows * kRow, floats = split + (kind == 1 ? kMlpIn : kUnits) * kRow;
    constexpr int kPieces = (kStageFloats / 4 + THREADS - 1) / THREADS;
    int from[kPieces];
#pragma unroll
    for (int i = 0; i < kPieces; ++i) {
        const int e = 4 * (tid + i * THREADS);
        from[i] = e < split ? e : e - split + (int)(second - first);
    }
    const unsigned dst = (unsigned)__cvta_generic_to_shared(buf) + 16 * tid;
    auto fetch = [&](int t) {
        if (t < t1) {
            const unsigned d = dst + (t % STAGES) * (unsigned)(kStageFloats * sizeof(float));
            const float* const src = first + (size_t)t * kTileFloats;
#pragma unroll
            for (int i = 0; i < kPieces; ++i) {
                if (4 * (tid + i * THREADS) < floats)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * i * THREADS),
                                 "l"(src + from[i])
                                 : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");       // perhaps empty
    };
    const int r = tid % 8, c = tid / 8;                            // gW2
    const int unit = tid % kUnits, f0 = tid / kUnits * kFeat;      // gW1, gW3
    float acc[RI][kCols] = {}, gb[RI] = {};
    float w1[kFeat] = {}, u = 0.f;
#pragma unroll
    for (int k = 0; k < STAGES - 1; ++k) fetch(t0 + k);
    for (int t = t0; t < t1; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                              // tile t is here, tile t - 1 done with
        fetch(t + STAGES - 1);
        float* const a = buf + (t % STAGES) * kStageFloats;
        const float* const b = a + arows * kRow;
        const int lo = max(0, s0 - t * kTile), hi = min(kTile, s1 - t * kTile);
        if (lo > 0 || hi < kTile) {
            // samples of the neighbouring chunks (or none) count as zero gradients
            for (int i = tid; i < arows * kTile; i += THREADS) {
                const int s = i % kTile;
                if (s < lo || s >= hi) a[(i / kTile) * kRow + s] = 0.f;
            }
            __syncthreads();
        }
        if (kind == 0) {
#pragma unroll kSteps
            for (int s = 0; s < kTile; s += 4) {
                float4 av[RI], bv[kCols];
#pragma unroll
                for (int i = 0; i < RI; ++i) av[i] = ld4(a + (r + 8 * i) * kRow + s);
#pragma unroll
                for (int k = 0; k < kCols; ++k) bv[k] = ld4(b + (c + kColGroups * k) * kRow + s);
#pragma unroll
                for (int i = 0; i < RI; ++i)
#pragma unroll
                    for (int k = 0; k < kCols; ++k) chain4(acc[i][k], av[i], bv[k]);
                if (c == 0 && q == 0)
#pragma unroll
                    for (int i = 0; i < RI; ++i) sum4(gb[i], av[i]);
            }
        } else if (kind == 1) {
            if (f0 < kMlpIn) {
#pragma unroll kSteps
                for (int s = 0; s < kTile; s += 4) {
                    const float4 dv = ld4(a + unit * kRow + s);
#pragma unroll
                    for (int f = 0; f < kFeat; ++f) chain4(w1[f], dv, ld4(b + (f0 + f) * kRow + s));
                    sum4(u, dv);
                }
            }
        } else if (tid <= kUnits) {
            // unit tid of gW3; the thread after them gb3
#pragma unroll 4
            for (int s = 0; s < kTile; s += 4) {
                const float4 yv = ld4(a + s);
                if (tid < kUnits) chain4(u, yv, ld4(b + tid * kRow + s));
                else sum4(u, yv);
            }
        }
    }
    float* const gb1 = g + kMlpHid * kMlpIn;
    float* const gw2 = gb1 + kMlpHid;
    float* const gb2 = gw2 + kMlpHid * kMlpHid;
    if (kind == 0) {
#pragma unroll
        for (int i = 0; i < RI; ++i) {
#pragma unroll
            for (int k = 0; k < kCols; ++k) gw2[(row0 + r + 8 * i) * kMlpHid + u0 + c + kColGroups * k] = acc[i][k];
            if (c == 0 && q == 0) gb2[row0 + r + 8 * i] = gb[i];
        }
    } else if (kind == 1) {
        if (f0 < kMlpIn) {
#pragma unroll
            for (int f = 0; f < kFeat; ++f) g[(u0 + unit) * kMlpIn + f0 + f] = w1[f];
        }
        if (f0 == 0) gb1[u0 + unit] = u;
    } else if (tid < kUnits || (tid == kUnits && q == Q - 1)) {
        gb2[kMlpHid + u0 + tid] = u;                  // gW3, then gb3
    }
}

// Adds the chunks, in order (many of them in FP64), into grad, or (grad null) into one Adam step of prm
// (whose rate may have fallen to zero); the last block adds the loss.
struct AdamStep {
    float *prm, *m1, *m2;
    float lr, b1, b2, eps, c1, c2;
};
constexpr int kReduceThreads = 32;
__global__ void __launch_bounds__(kReduceThreads)
    mlp_reduce_kernel(const float* __restrict__ part, int chunks, const float* __restrict__ lossp, int nloss,
                      float* __restrict__ grad, float* __restrict__ loss, AdamStep ad) {
    if (blockIdx.x == gridDim.x - 1) {
        float l = 0.f;
        for (int k = threadIdx.x; k < nloss; k += kReduceThreads) l += lossp[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (threadIdx.x == 0) *loss = l;
        return;
    }
    const int i = blockIdx.x * kReduceThreads + threadIdx.x;
    if (i >= kMlpParams) return;
    float gi = 0.f;
    if (chunks <= 16) {
#pragma unroll 8
        for (int c = 0; c < chunks; ++c) gi += part[(size_t)c * kMlpParams + i];
    } else {
        double sum = 0.0;                             // one rounding instead of up to 63
#pragma unroll 16
        for (int c = 0; c < chunks; ++c) sum += (double)part[(size_t)c * kMlpParams + i];
        gi = (float)sum;
    }
    if (!grad) {
        const float a = ad.b1 * ad.m1[i] + (1.f - ad.b1) * gi;
        const float v = ad.b2 * ad.m2[i] + (1.f - ad.b2) * gi * gi;
        ad.m1[i] = a;
        ad.m2[i] = v;
        ad.prm[i] -= ad.lr * (a / ad.c1) / (sqrtf(v / ad.c2) + ad.eps);
    } else {
        grad[i] = gi;
    }
}

namespace {
int train_tiles(int n) { return (n + kTile - 1) / kTile; }
int train_grid(int n, int sms) { return std::max(1, std::min(train_tiles(n), kTrainBlocksPerSm * sms)); }
int train_chunks(int n) { return std::max(1, std::min(64, n / 2048)); }

using Many = WeightSplit<16, 1, 128, 4>;
using Few = WeightSplit<8, 4, 128, 8>;

void train_pass(const float* prm, const float* X, const float* T, int n, float q, TrainWork w, float* grad,
                float* loss, AdamStep ad, int sms, cudaStream_t s) {
    TrainTile* tiles = static_cast<TrainTile*>(w.tiles);
    const int grid = train_grid(n, sms), chunks = train_chunks(n);
    mlp_samples_kernel<true><<<grid, kTrainThreads, sizeof(TrainSmem), s>>>(prm, X, T, n, q, nullptr, tiles, w.lossp);
    if (chunks * Many::kBlocks >= sms)
        mlp_weights_kernel<16, 1, 128, 4><<<dim3(Many::kBlocks, chunks), 128, Many::kSmem, s>>>(tiles, n, w.part);
    else
        mlp_weights_kernel<8, 4, 128, 8><<<dim3(Few::kBlocks, chunks), 128, Few::kSmem, s>>>(tiles, n, w.part);
    mlp_reduce_kernel<<<(kMlpParams + kReduceThreads - 1) / kReduceThreads + 1, kReduceThreads, 0, s>>>(
        w.part, chunks, w.lossp, grid, grad, loss, ad);
}
}  // namespace

size_t train_work_bytes(int n, int sms, TrainWork* w, void* base) {
    const size_t tiles = sizeof(TrainTile) * train_tiles(n);
    const size_t part = (sizeof(float) * kMlpParams * train_chunks(n) + 15) / 16 * 16;
    if (w) {
        w->tiles = base;
        w->part = reinterpret_cast<float*>(static_cast<char*>(base) + tiles);
        w->lossp = reinterpret_cast<float*>(static_cast<char*>(base) + tiles + part);
    }
    return tiles + part + sizeof(float) * train_grid(n, sms);
}

cudaError_t prepare_train_kernels() {
    cudaError_t e;
    const auto a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((e = cudaFuncSetAttribute(mlp_samples_kernel<true>, a, (int)sizeof(TrainSmem))) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(mlp_samples_kernel<false>, a, (int)sizeof(TrainSmem))) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(mlp_weights_kernel<8, 4, 128, 8>, a, (int)Few::kSmem)) != cudaSuccess) return e;
    return cudaFuncSetAttribute(mlp_weights_kernel<16, 1, 128, 4>, a, (int)Many::kSmem);
}

void mlp_forward(const float* prm, const float* X, int n, float* Y, int sms, cudaStream_t s) {
    mlp_samples_kernel<false><<<train_grid(n, sms), kTrainThreads, sizeof(TrainSmem), s>>>(prm, X, nullptr, n, 0.5f, Y,
                                                                                          nullptr, nullptr);
}

// One forward and backward pass: gradient (kMlpParams) and loss of the batch.
void mlp_grad(const float* prm, const float* X, const float* T, int n, float q, TrainWork w, float* grad, float* loss,
              int sms, cudaStream_t s) {
    train_pass(prm, X, T, n, q, w, grad, loss, AdamStep{}, sms, s);
}

// The same, with the gradient taken into the Adam step t (from 1) of prm.
void mlp_train_step(float* prm, const float* X, const float* T, int n, float q, TrainWork w, float* loss, float* m1,
                    float* m2, float lr, int t, int sms, cudaStream_t s) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
    train_pass(prm, X, T, n, q, w, nullptr, loss, AdamStep{prm, m1, m2, lr, b1, b2, 1e-8f, c1, c2}, sms, s);
}

}  // namespace nbh
