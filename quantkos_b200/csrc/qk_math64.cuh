// FP64 elementary functions of the path kernels (sm_100a).
//
// What bounds an FP64 path-step is the number of instructions it issues: the FP64 pipe
// takes one warp instruction per two cycles and scheduler, and the CUDA library's log,
// sincospi, exp, sqrt and divisions cost about 70 FP64 and 160 other instructions per
// Euler step (argument checks, range reduction and special cases that a path-step never
// meets).  The functions here are written for the arguments that occur:
//
//   * logarithm and power of two by a table of 256 points and a short Taylor polynomial
//     (Tang, ACM TOMS 16, 1990 and 15, 1989), the reduced argument formed exactly by an
//     FMA; the table point next to 1 is 1 itself, so -2 ln u keeps its relative accuracy
//     as u approaches 1.  The steps of the argument reduction on the bits (subtracting an
//     offset's high word to get exponent and table index at once, pairs of 1 / c and log c,
//     a shift by 1.5 * 2^52 / N whose low word is the index) are those of Arm's Optimized
//     Routines (log and exp2); polynomials and tables are formed here;
//   * sine and cosine of 2 pi (u - 1/2) from the integer word behind u: its top 9 bits
//     pick a table angle, the other 23 are the (exact) remainder, and the addition
//     theorem joins them;
//   * reciprocal, square root and reciprocal square root from the 2^-20 hardware
//     approximations by one third-order step (Householder), without the library's
//     special-case branches: callers guard the arguments.
//
// Largest relative errors against long double (a million arguments each): -2 ln u 3.7e-16, 2^x
// 2.5e-16, reciprocal and reciprocal square root 1.2e-16, square root 1.7e-16, a normal
// 4.6e-16 of its radius.  The tables (14 KB) live in shared memory, filled at the start of a
// kernel by the block's threads with the CUDA functions: about 0.5 us, no table in global
// memory to load.  Plain FP64 Heston Euler European, 1,048,576 x 252: 286 warp instructions
// per 32 path-steps and 2.77 ms with the library's functions on the spot, 106 and 1.21 ms
// with these on its logarithm (FP64 pipe 53% busy in both, 52% now at less than half the
// work: FP64 and the generator's wide multiplies share issue and register ports).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace qk {

struct Tab64 {
    double2 sct[512];   // sin, cos of pi t_j, t_j = 2 (j + 1/2) / 512 - 1
    double2 logt[256];  // 1 / c_i (rounded), -2 ln of the reciprocal of that
    double ex[256];     // 2^(j / 256)
};

// The mantissa interval [m, 2m) a logarithm's argument is brought into starts at
// m = 0.7002, placed so that 1 is the centre of one of the 256 sub-intervals.
constexpr int kLogOff = 0x3FE66800;

__device__ __forceinline__ void fill_tab64(Tab64 &t) {
    for (int j = threadIdx.x; j < 512; j += blockDim.x) {
        double s, c;
        ::sincospi((2 * j + 1) * (1.0 / 512.0) - 1.0, &s, &c);
        t.sct[j] = make_double2(s, c);
        if (j < 256) {
            const double inv = 1.0 / __hiloint2double(kLogOff + (j << 12) + 0x800, 0);
            t.logt[j] = make_double2(inv, 2.0 * ::log(inv));
            t.ex[j] = ::exp2(j * (1.0 / 256.0));
        }
    }
}

// 2^52 + k and 2^51 + k / 2 as doubles, built from their bits.
__device__ __forceinline__ double magic52(uint32_t k) { return __hiloint2double(0x43300000, static_cast<int>(k)); }
__device__ __forceinline__ double magic51(uint32_t k) { return __hiloint2double(0x43200000, static_cast<int>(k)); }

// -2 ln x of a positive normal x.  x = 2^k z, z in [0.7002, 1.4004); z c_i^-1 = 1 + r
// with |r| <= 2^-9, and -2 ln(1 + r) = -2r + r^2 (1 - 2r/3 + r^2/2 - 2r^3/5 + r^4/3),
// truncated at 2e-19 (8e-18 relative next to x = 1).
__device__ __forceinline__ double neg2_log64(const Tab64 &t, double x, int k_off) {
    const int tmp = __double2hiint(x) - kLogOff;
    const int k = tmp >> 20;
    const double z = __hiloint2double(__double2hiint(x) - (tmp & static_cast<int>(0xFFF00000)), __double2loint(x));
    const double2 e = t.logt[(tmp >> 12) & 255];
    const double kd = magic52(static_cast<uint32_t>(k + 2048)) - (4503599627370496.0 + 2048.0 + k_off);
    const double r = fma(z, e.x, -1.0);
    double q = fma(r, 1.0 / 3.0, -0.4);
    q = fma(q, r, 0.5);
    q = fma(q, r, -2.0 / 3.0);
    q = fma(q, r, 1.0);
    const double b = fma(kd, -2.0 * 0.693147180559945309417, e.y);
    return fma(r * r, q, fma(r, -2.0, b));
}

// 2^x.  x = n/256 + r, |r| <= 2^-9, 2^(n mod 256 / 256) from the table, 2^r by Taylor
// (truncated at 4e-17 relative); |x| beyond 1000 (and NaN) goes to the library.
__device__ __noinline__ inline double exp2_slow64(double x) { return ::exp2(x); }
__device__ __forceinline__ double exp2_64(const Tab64 &t, double x) {
    if ((__double2hiint(x) & 0x7FFFFFFF) >= 0x408F4000) return exp2_slow64(x);
    constexpr double kShift = 6755399441055744.0 / 256.0;  // 1.5 * 2^52 / 256: the low word then holds n
    const double s = x + kShift;
    const int n = __double2loint(s);
    const double r = x - (s - kShift);
    constexpr double L = 0.693147180559945309417;
    double p = fma(r, L * L * L * L / 24.0, L * L * L / 6.0);
    p = fma(p, r, L * L / 2.0);
    p = fma(p, r, L);
    const double T = t.ex[n & 255];
    const double y = fma(T * r, p, T);
    return __hiloint2double(__double2hiint(y) + ((n >> 8) << 20), __double2loint(y));
}

// 1/x, 1/sqrt(x), sqrt(x) from the hardware approximation y0 (relative error e0 <= 2^-19):
// with e = 1 - x y0 (or 1 - x y0^2), y0 (1 + e + e^2) resp. y0 (1 + e/2 + 3 e^2/8) has
// error of order e^3.  rcp and rsqrt: x positive (or negative for rcp) and normal.
__device__ __forceinline__ double rcp64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double rsqrt_approx64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double rsqrt64(double x) {
    const double y = rsqrt_approx64(x);
    const double e = fma(-x, y * y, 1.0);  // y * y is exact: the approximation's low word is zero
    return fma(y * e, fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ double sqrt_from64(double x, double y) {
    const double h = x * y;
    const double e = fma(-h, y, 1.0);
    return fma(h * e, fma(e, 0.375, 0.5), h);
}
// x > 0 and normal
__device__ __forceinline__ double sqrt_pos64(double x) { return sqrt_from64(x, rsqrt_approx64(x)); }
// x >= 0: the approximation reads only the high word, which is kept normal, so x = 0 gives 0.
__device__ __forceinline__ double sqrt64(double x) {
    return sqrt_from64(x, rsqrt_approx64(__hiloint2double(max(__double2hiint(x), 0x00100000), __double2loint(x))));
}

// max(x, 0) on the sign and exponent bits, 0 for NaN (as fmax): no FP64 compare.
__device__ __forceinline__ double max0_64(double x) {
    const bool keep = static_cast<uint32_t>(__double2hiint(x)) <= 0x7FF00000u;
    return __hiloint2double(keep ? __double2hiint(x) : 0, keep ? __double2loint(x) : 0);
}

// Box-Muller of two 32-bit words: u = (w + 1/2) / 2^32, R = sqrt(-2 ln u1), angle
// 2 pi (u2 - 1/2).
__device__ __forceinline__ void box_muller64(const Tab64 &t, uint32_t w1, uint32_t w2, double &z1, double &z2) {
    const double u = magic52(w1) - (4503599627370496.0 - 0.5);  // w1 + 1/2, exact
    const double rad = sqrt_pos64(neg2_log64(t, u, 32));
    // angle remainder in units of 2 pi / 2^32: the low 23 bits + 1/2 - 2^22, exact
    const double d = magic51(((w2 << 1) & 0xFFFFFFu) | 1u) - (2251799813685248.0 + 4194304.0);
    constexpr double a = 6.283185307179586476925 / 4294967296.0;
    const double D = d * d;
    double sd = fma(D, a * a * a * a * a / 120.0, -a * a * a / 6.0);
    sd = fma(sd, D, a);
    sd *= d;                                                        // sin of the remainder
    const double cm = D * fma(D, a * a * a * a / 24.0, -a * a / 2.0);  // cos of the remainder - 1
    const double2 sc = t.sct[w2 >> 23];
    z2 = rad * fma(sc.y, sd, fma(sc.x, cm, sc.x));
    z1 = rad * fma(-sc.x, sd, fma(sc.y, cm, sc.y));
}

}  // namespace qk
