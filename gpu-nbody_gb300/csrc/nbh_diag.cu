// nbh_diag.cu — diagnostics of each universe as GPU reductions
// (GPUBarnesHutNBodySimulation.java:305-365: printEnergy, printDepth, printImpulse).
//
// Per universe, in FP64: mass, mass-weighted position (centre of mass), momentum sum m v
// (printImpulse, :347-365), angular momentum sum m x cross v, kinetic energy sum m |v|^2/2
// (:318-324) and, on request, the potential energy sum over pairs i < j of -G m_i m_j / r,
// softened (r^2 + eps^2, the potential of the force the step integrates) and unsoftened (the
// form of :326-335, which adds each pair twice -- `2 * e` at :334 -- and is counted once
// here).  Reductions run in a fixed order (warp shuffles, then warps in order, then chunks
// in order), so the results do not depend on scheduling.
#include "nbh_common.cuh"
#include "nbh_kernels.h"

namespace nbh {

constexpr int kDiagThreads = 256;   // one block per 256-body chunk

// Sums v over the block into red[field] of thread 0's view, in a fixed order.
template <int F>
__device__ __forceinline__ void block_sum(double (&v)[F], double (*red)[F], double* out) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[f] += __shfl_xor_sync(0xffffffffu, v[f], o);
    if (lane == 0)
#pragma unroll
        for (int f = 0; f < F; ++f) red[wid][f] = v[f];
    __syncthreads();
    if (threadIdx.x < F) {
        double a = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) a += red[w][threadIdx.x];
        out[threadIdx.x] = a;
    }
    __syncthreads();
}

// Moments of one chunk: its partial row.
__global__ void __launch_bounds__(kDiagThreads) diag_moments_kernel(const float4* __restrict__ node4,
                                                                    const float4* __restrict__ vel,
                                                                    const int4* __restrict__ chunks, double* part) {
    __shared__ double red[kDiagThreads / 32][kDiagMoments];
    const int4 ck = chunks[blockIdx.x];
    const int b = ck.y + threadIdx.x;
    double v[kDiagMoments];
#pragma unroll
    for (int f = 0; f < kDiagMoments; ++f) v[f] = 0.0;
    if (b < ck.z) {
        const float4 q = node4[b];
        const float4 w = vel[b];
        const double m = q.w, x = q.x, y = q.y, z = q.z, vx = w.x, vy = w.y, vz = w.z;
        v[0] = m;
        v[1] = m * x; v[2] = m * y; v[3] = m * z;
        v[4] = m * vx; v[5] = m * vy; v[6] = m * vz;
        v[7] = m * (y * vz - z * vy); v[8] = m * (z * vx - x * vz); v[9] = m * (x * vy - y * vx);
        v[10] = 0.5 * m * (vx * vx + vy * vy + vz * vz);
    }
    block_sum<kDiagMoments>(v, red, part + (size_t)blockIdx.x * kDiagMoments);
}

// Pair potential: sum over pairs of -m_i m_j / r_ij, softened and unsoftened, each pair once
// (counted twice, the caller halves the sum of m_i phi_i).  A universe's 256-body chunks form
// a ring of K; chunk a meets chunks a, a + 1, ... a + K/2 (mod K), so that every pair of
// chunks meets once and every block has the same work (with K even, the chunks half a ring
// apart meet on the first K/2 blocks only).  blockIdx.y takes one of gridDim.y slices of these
// offsets.  A thread keeps two bodies, so one 16-byte shared load serves two pairs.  Pair terms
// are FP32 (1/sqrt of the FP32 squared distance), summed per 256-source tile in FP32 and the
// tile sums in FP64.  Bound by the two inverse square roots of a pair (16 lanes per clock and
// SM: 8.1 ms at 200,003 bodies, measured 9.6; 38.0 with every pair evaluated from both
// sides and one body per thread).
//
// 1/sqrt flushes subnormal squared distances (bodies closer than 1e-19, or coincident): a
// tile in which a thread met one is summed again with the full-range function.
constexpr int kPotThreads = kDiagThreads / 2;
__device__ __forceinline__ float rsqrt_normal(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float pair_r2(const float4 q, const float4 qi) {
    const float dx = q.x - qi.x, dy = q.y - qi.y, dz = q.z - qi.z;
    return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

__global__ void __launch_bounds__(kPotThreads) diag_potential_kernel(const float4* __restrict__ node4,
                                                                     const int4* __restrict__ chunks,
                                                                     const int* __restrict__ ubody, float eps2,
                                                                     double* pot) {
    __shared__ float4 tile[kDiagThreads];
    __shared__ double red[kPotThreads / 32][2];
    const int4 ck = chunks[blockIdx.x];
    const int lo = ubody[ck.x], hi = ubody[ck.x + 1];
    const int K = (hi - lo + kDiagThreads - 1) / kDiagThreads;
    const int a = (ck.y - lo) / kDiagThreads;
    const int offsets = K / 2 + (K % 2 == 0 && a >= K / 2 ? 0 : 1);
    const int d0 = (int)((long long)offsets * blockIdx.y / gridDim.y);
    const int d1 = (int)((long long)offsets * (blockIdx.y + 1) / gridDim.y);
    const bool flushed = eps2 < 1.17549435e-38f;      // softened squares may be subnormal too
    int i[2];
    bool valid[2];
    float4 qi[2];
    double ps[2] = {0.0, 0.0}, pu[2] = {0.0, 0.0};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        i[t] = ck.y + threadIdx.x + t * kPotThreads;
        valid[t] = i[t] < ck.z;
        qi[t] = node4[valid[t] ? i[t] : ck.y];
    }
    for (int d = d0; d < d1; ++d) {
        const int base = lo + (a + d < K ? a + d : a + d - K) * kDiagThreads;
        const int cnt = min(kDiagThreads, hi - base);
        __syncthreads();
        for (int j = threadIdx.x; j < cnt; j += kPotThreads) tile[j] = node4[base + j];
        __syncthreads();
        float ts[2] = {0.0f, 0.0f}, tu[2] = {0.0f, 0.0f};
        bool full = d == 0 || flushed;
        if (!full) {
            float least = 1.0f;
#pragma unroll 8
            for (int k = 0; k < cnt; ++k) {
                const float4 q = tile[k];
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const float r2 = pair_r2(q, qi[t]);
                    least = fminf(least, r2);
                    ts[t] = fmaf(q.w, rsqrt_normal(r2 + eps2), ts[t]);
                    tu[t] = fmaf(q.w, rsqrt_normal(r2), tu[t]);
                }
            }
            full = least < 1.17549435e-38f;
        }
        if (full) {
            // the chunk against itself (a body skips itself), or a subnormal squared distance
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                ts[t] = tu[t] = 0.0f;
                for (int k = 0; k < cnt; ++k) {
                    const float4 q = tile[k];
                    const float r2 = pair_r2(q, qi[t]);
                    const bool other = base + k != i[t];
                    ts[t] += other ? q.w * rsqrtf(r2 + eps2) : 0.0f;
                    tu[t] += other ? q.w * rsqrtf(r2) : 0.0f;
                }
            }
        }
        const double w = d == 0 ? 1.0 : 2.0;          // both sides of a pair of two chunks
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            ps[t] = fma(w, (double)ts[t], ps[t]);
            pu[t] = fma(w, (double)tu[t], pu[t]);
        }
    }
    double v[2] = {0.0, 0.0};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        if (!valid[t]) continue;
        v[0] -= (double)qi[t].w * ps[t];
        v[1] -= (double)qi[t].w * pu[t];
    }
    block_sum<2>(v, red, pot + 2 * ((size_t)blockIdx.x * gridDim.y + blockIdx.y));
}

// One block per universe: its chunks' rows summed in chunk order.
__global__ void __launch_bounds__(kDiagThreads) diag_reduce_kernel(const int4* __restrict__ chunks, int nchunks,
                                                                   const double* __restrict__ part,
                                                                   const double* __restrict__ pot, int slices,
                                                                   double* out) {
    __shared__ double red[kDiagThreads / 32][kDiagFields];
    const int u = blockIdx.x;
    // chunks are ordered by universe: binary search for [c0, c1)
    int a = 0, b = nchunks;
    while (a < b) {
        const int m = (a + b) >> 1;
        if (chunks[m].x < u) a = m + 1;
        else b = m;
    }
    const int c0 = a;
    b = nchunks;
    while (a < b) {
        const int m = (a + b) >> 1;
        if (chunks[m].x <= u) a = m + 1;
        else b = m;
    }
    const int c1 = a;
    double v[kDiagFields];
#pragma unroll
    for (int f = 0; f < kDiagFields; ++f) v[f] = 0.0;
    for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
#pragma unroll
        for (int f = 0; f < kDiagMoments; ++f) v[f] += part[(size_t)c * kDiagMoments + f];
        for (int y = 0; y < slices; ++y) {            // none without the potential
            v[kDiagMoments] += pot[2 * ((size_t)c * slices + y)];
            v[kDiagMoments + 1] += pot[2 * ((size_t)c * slices + y) + 1];
        }
    }
    block_sum<kDiagFields>(v, red, out + (size_t)u * kDiagFields);
}

// Slices of a chunk's ring of tiles: enough blocks for several per SM (a 30,000-body universe
// has 118 chunks), but four tiles each at least.
int diag_slices(int nchunks, int max_chunks, int sms) {
    const int want = (32 * sms + nchunks - 1) / nchunks;
    const int most = max_chunks / 8 > 1 ? max_chunks / 8 : 1;
    return want < 1 ? 1 : (want < most ? want : most);
}

void launch_diagnostics(const float4* node4, const float4* vel, const int4* chunks, int nchunks, const int* ubody,
                        int nuniv, int slices, float eps2, double* part, double* out, cudaStream_t s) {
    double* pot = part + (size_t)kDiagMoments * nchunks;
    diag_moments_kernel<<<nchunks, kDiagThreads, 0, s>>>(node4, vel, chunks, part);
    if (slices > 0)
        diag_potential_kernel<<<dim3(nchunks, slices), kPotThreads, 0, s>>>(node4, chunks, ubody, eps2, pot);
    diag_reduce_kernel<<<nuniv, kDiagThreads, 0, s>>>(chunks, nchunks, part, pot, slices, out);
}

}  // namespace nbh
