// nbh_direct.cuh — one tile of the FP64 direct sum (nbh_direct_f64, nbh_direct_f64_static).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace nbh {

constexpr int kDirectTile = 256;
struct Src64 {
    double x, y, z, m;
};

// Slices of the sources for `targets` blocks of target bodies: 32 blocks per SM in all (four
// are resident), so that the last wave is short.
inline int direct_slices(int targets, int sms) {
    const int want = (32 * sms + targets - 1) / targets;
    return want < 1 ? 1 : (want < 256 ? want : 256);
}

// m d2^(-3/2), for d2 in the range of normal floats.
//
// FP64 runs at 2 operations per clock and SM (measured: one warp instruction in 64.6 cycles
// of a scheduler), integer and FP32 at 64 and 128, so the estimate and its powers are made in
// integers: y0 ~ d2^(-1/2) is the FP32 approximation rounded to 17 bits (relative error below
// 2^-16.9), i its 17-bit significand, and y0^2 (34 bits) and y0^3 (51 bits) are exact doubles
// assembled from i^2 and i^3.  With e = 1 - d2 y0^2 (one rounding, |e| < 2^-15.9) the binomial
// series gives d2^(-3/2) = y0^3 (1 - e)^(-3/2) = y0^3 (1 + 3/2 e + 15/8 e^2 + 35/16 e^3 + ...);
// the terms from e^4 on are below 2^-62, and those of e^2 and e^3, below 2^-30.8 together, are
// formed in FP32.  Four FP64 operations in place of a square root, a division and three
// products.  In a host replay of 5 million draws the result was at most 2.3 x 2^-53 off
// (relative); m * inv * inv * inv with inv = 1 / sqrt(d2) was up to 6.9 x 2^-53 off.
__device__ __forceinline__ double mass_over_cube(const double d2, const double m) {
    const int hi = __double2hiint(d2), lo = __double2loint(d2);
    // the float below d2: exponent bias 1023 -> 127, the low 29 significand bits dropped
    const float x = __uint_as_float(__funnelshift_l((unsigned)lo, (unsigned)hi, 3) + 0x40000000u);
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    const unsigned yb = __float_as_uint(y) + 0x40u;
    const unsigned i = ((yb >> 7) & 0xffffu) | 0x10000u;          // y0 = i 2^(E - 143)
    const int E = (int)(yb >> 23);
    const unsigned long long i2 = (unsigned long long)i * i;      // [2^32, 2^34)
    const unsigned long long i3 = i2 * i;                         // [2^48, 2^51)
    const int t2 = (int)(i2 >> 33);                               // leading bit at 32 + t2
    const int t3 = 31 - __clz((int)(i3 >> 32));                   // leading bit at 32 + t3
    // significand with its leading bit at 52, added to the exponent field less one
    const double y2 = __longlong_as_double(
        (long long)((i2 << (20 - t2)) + ((unsigned long long)(1023 + 32 + t2 + 2 * (E - 143) - 1) << 52)));
    const double y3 = __longlong_as_double(
        (long long)((i3 << (20 - t3)) + ((unsigned long long)(1023 + 32 + t3 + 3 * (E - 143) - 1) << 52)));
    const double e = __fma_rn(-d2, y2, 1.0);
    // float of e and double of the series' tail by their bits too: a conversion costs as much as
    // an FP64 operation.  |e| below 2^-40 counts as zero (its square is below 2^-80), and a zero
    // tail becomes 2^-127.
    const unsigned eh = (unsigned)__double2hiint(e);
    const unsigned eb = __funnelshift_l((unsigned)__double2loint(e), eh, 3) + 0x40000000u;
    const float ef = __uint_as_float(((eh & 0x7fffffffu) >= (983u << 20) ? eb : 0u) | (eh & 0x80000000u));
    const unsigned tail = __float_as_uint(ef * ef * fmaf(ef, 2.1875f, 1.875f));
    const double g = __fma_rn(e, 1.5, __hiloint2double((int)((tail >> 3) + 0x38000000u), (int)(tail << 29)));
    const double w = m * y3;
    return __fma_rn(w, g, w);
}

// Adds the attraction of tile[k0, k1) on a body at (xi, yi, zi) to s.  Squared distances above
// the largest float (or not finite) take the library's square root and division for the whole
// tile, as do softenings below 2^-100, where d2 could leave the normal floats downwards.
__device__ __forceinline__ void direct_tile(const Src64* tile, const int k0, const int k1, const double xi,
                                            const double yi, const double zi, const double eps2, double (&s)[3]) {
    double ax = s[0], ay = s[1], az = s[2];
    unsigned most = eps2 < 0x1p-100 ? 0xffffffffu : 0u;
    if (most == 0u) {
#pragma unroll 2
        for (int k = k0; k < k1; ++k) {
            const Src64 q = tile[k];
            const double dx = q.x - xi, dy = q.y - yi, dz = q.z - zi;
            const double d2 = __fma_rn(dx, dx, __fma_rn(dy, dy, __fma_rn(dz, dz, eps2)));
            most = max(most, (unsigned)__double2hiint(d2));
            const double f = mass_over_cube(d2, q.m);
            ax = __fma_rn(dx, f, ax);
            ay = __fma_rn(dy, f, ay);
            az = __fma_rn(dz, f, az);
        }
    }
    if (most >= 0x47e00000u) {                        // 2^127
        ax = s[0], ay = s[1], az = s[2];
        for (int k = k0; k < k1; ++k) {
            const Src64 q = tile[k];
            const double dx = q.x - xi, dy = q.y - yi, dz = q.z - zi;
            const double d2 = dx * dx + dy * dy + dz * dz + eps2;
            const double inv = 1.0 / sqrt(d2);
            const double f = q.m * inv * inv * inv;
            ax += dx * f;
            ay += dy * f;
            az += dz * f;
        }
    }
    s[0] = ax, s[1] = ay, s[2] = az;
}

}  // namespace nbh
