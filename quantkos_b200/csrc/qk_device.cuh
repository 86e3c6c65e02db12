// Device building blocks of the Monte Carlo hot path (sm_100a).
//
//   * Philox4x32-10 counter-based generator and the fixed draw layout that makes
//     every path reproducible whatever the launch shape;
//   * the Heston / Bates step functions under Euler, implicit Milstein and
//     Andersen QE, written once, templated on the arithmetic type and on the
//     draw source (Philox in the pricing kernels, fed draws in the parity trace);
//   * payoff trackers and final payoffs for the ten forward option types;
//   * FP64 statistics helpers (Welford / Chan merge).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "qk_internal.h"
#include "qk_math64.cuh"

namespace qk {

// ============================================================================
// Philox4x32-10 (J. Salmon, M. Moraes, R. Dror, D. Shaw, "Parallel random
// numbers: as easy as 1, 2, 3", SC'11): 10 rounds of two 32x32->64 multiplies
// with a Weyl-sequence key schedule.  Counter = (block, path, stream, domain),
// key = (lo32(seed), hi32(seed)).
// ============================================================================
struct U4 {
    uint32_t x, y, z, w;
};

__device__ __forceinline__ U4 philox4x32_10(U4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        // one 32x32 -> 64-bit multiply per product (IMAD.WIDE.U32)
        const uint64_t p0 = static_cast<uint64_t>(kPhiloxM0) * c.x;
        const uint64_t p1 = static_cast<uint64_t>(kPhiloxM1) * c.z;
        const uint32_t lo0 = static_cast<uint32_t>(p0), hi0 = static_cast<uint32_t>(p0 >> 32);
        const uint32_t lo1 = static_cast<uint32_t>(p1), hi1 = static_cast<uint32_t>(p1 >> 32);
        c = U4{hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0};
        k0 += kPhiloxW0;
        k1 += kPhiloxW1;
    }
    return c;
}

// Round keys k_r = (k0 + r W0, k1 + r W1), r = 0..9, precomputed on the host and
// passed by value as a kernel parameter: the XORs then read them straight from
// the parameter bank, with no key arithmetic per round.
struct PhiloxRoundKeys {
    uint32_t k[20];
};

inline PhiloxRoundKeys philox_round_keys(uint32_t k0, uint32_t k1) {
    PhiloxRoundKeys rk;
    for (int r = 0; r < 10; ++r) {
        rk.k[2 * r] = k0 + static_cast<uint32_t>(r) * kPhiloxW0;
        rk.k[2 * r + 1] = k1 + static_cast<uint32_t>(r) * kPhiloxW1;
    }
    return rk;
}

// Round keys of a launch whose tasks share the seed (from the parameter bank), or of the
// task's own key.
struct ParamKeys {
    const PhiloxRoundKeys &rk;
    __device__ __forceinline__ uint32_t k0(int r) const { return rk.k[2 * r]; }
    __device__ __forceinline__ uint32_t k1(int r) const { return rk.k[2 * r + 1]; }
};
struct RegKeys {
    uint32_t key0, key1;
    __device__ __forceinline__ uint32_t k0(int r) const { return key0 + static_cast<uint32_t>(r) * kPhiloxW0; }
    __device__ __forceinline__ uint32_t k1(int r) const { return key1 + static_cast<uint32_t>(r) * kPhiloxW1; }
};

// The path loop's Philox.  A 32x32->64 multiply occupies the FMA pipe for four cycles (an
// FP32 FMA: one), so the generator's 20 per block are 40 of the pipe's cycles per
// path-step, more than any step's arithmetic.  In the first three rounds most of the state
// does not depend on both counter words: with the counter (block, path, stream, domain),
//   round 1: x = hi(M1 stream) ^ path ^ k0 (per path), z, w from M0 block (per block),
//   round 2: M0 x per path, M1 z per block,
//   round 3: M0 x per block, M1 z the first multiply that needs both.
// What depends on the path alone is computed once per path (PhiloxPath), what depends on
// the block alone once per warp: lane l of a warp computes the row of block l of the next
// 32 blocks (64 steps) into shared memory, and a step pair reads its row with one
// broadcast load.  A block then costs 15 multiplies and 17 XORs instead of 20 and 20.
// The same words as philox4x32_10.
struct PhiloxPath {
    uint32_t hi, lo;  // M0 x after round 1
};
__device__ __forceinline__ PhiloxPath philox_path_of(uint32_t x) {
    const uint64_t p = static_cast<uint64_t>(kPhiloxM0) * x;
    return PhiloxPath{static_cast<uint32_t>(p >> 32), static_cast<uint32_t>(p)};
}
template <class Keys>
__device__ __forceinline__ uint4 philox_row(const Keys &k, uint32_t block, uint32_t stream, uint32_t domain) {
    const uint64_t p0 = static_cast<uint64_t>(kPhiloxM0) * block;
    const uint32_t y1 = kPhiloxM1 * stream;
    const uint64_t p1 = static_cast<uint64_t>(kPhiloxM1) * (static_cast<uint32_t>(p0 >> 32) ^ domain ^ k.k1(0));
    const uint64_t p2 = static_cast<uint64_t>(kPhiloxM0) * (static_cast<uint32_t>(p1 >> 32) ^ y1 ^ k.k0(1));
    return make_uint4(static_cast<uint32_t>(p0) ^ k.k1(1), static_cast<uint32_t>(p1) ^ k.k0(2),
                      static_cast<uint32_t>(p2 >> 32) ^ k.k1(2), static_cast<uint32_t>(p2) ^ k.k1(3));
}
template <class Keys>
__device__ __forceinline__ U4 philox_rest(const Keys &k, const uint4 &row, const PhiloxPath &pp) {
    const uint64_t q = static_cast<uint64_t>(kPhiloxM1) * (pp.hi ^ row.x);  // round 3
    uint32_t x = static_cast<uint32_t>(q >> 32) ^ row.y, y = static_cast<uint32_t>(q), z = row.z ^ pp.lo, w = row.w;
#pragma unroll
    for (int r = 3; r < 10; ++r) {
        const uint64_t p0 = static_cast<uint64_t>(kPhiloxM0) * x;
        const uint64_t p1 = static_cast<uint64_t>(kPhiloxM1) * z;
        x = static_cast<uint32_t>(p1 >> 32) ^ y ^ k.k0(r);
        y = static_cast<uint32_t>(p1);
        z = r == 3 ? static_cast<uint32_t>(p0 >> 32) ^ w : static_cast<uint32_t>(p0 >> 32) ^ w ^ k.k1(r);  // row.w holds k1(3)
        w = static_cast<uint32_t>(p0);
    }
    return U4{x, y, z, w};
}

// Rows of a warp: 32 normal blocks, then (FP64 Bates) 16 first-Poisson-word blocks, of the
// 64 steps from n0 (a multiple of 64).  Every lane of the warp takes part in fill.
constexpr int kRowSteps = 64;
template <class R, int MODEL>
constexpr int philox_rows() {
    return 32 + (sizeof(R) == 8 && MODEL == kBates ? 16 : 0);
}
template <int ROWS, class Keys>
struct WarpPhilox {
    Keys keys;
    uint4 *rows;  // this warp's, in shared memory
    uint32_t stream;
    __device__ __forceinline__ void fill(int n0) const {
        const uint32_t lane = threadIdx.x & 31u;
        __syncwarp();  // the rows of the previous 64 steps have been read
        rows[lane] = philox_row(keys, static_cast<uint32_t>(n0 >> 1) + lane, stream, 0u);
        if (ROWS > 32 && lane < 16) rows[32 + lane] = philox_row(keys, static_cast<uint32_t>(n0 >> 2) + lane, stream, 2u);
        __syncwarp();
    }
    // x after round 1
    __device__ __forceinline__ uint32_t path_word(uint32_t path) const {
        return static_cast<uint32_t>((static_cast<uint64_t>(kPhiloxM1) * stream) >> 32) ^ path ^ keys.k0(0);
    }
    __device__ __forceinline__ PhiloxPath path(uint32_t path) const { return philox_path_of(path_word(path)); }
    __device__ __forceinline__ U4 block(const uint4 *row, const PhiloxPath &pp) const {
        return philox_rest(keys, *row, pp);
    }
};

// ============================================================================
// Arithmetic policy.  FP32 uses the SFU (MUFU) approximations explicitly; FP64 uses the
// functions of qk_math64.cuh in the path loop, the CUDA library in rare code and in
// step_spot64.
// ============================================================================
template <class R>
struct Math;

// Single SFU instructions (hand-written PTX): approximate base-2 exponential and
// logarithm, reciprocal and square root, flushing subnormals to zero.
__device__ __forceinline__ float ptx_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ptx_lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ptx_rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ptx_sqrt(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <>
struct Math<float> {
    static constexpr float kLog2e = 1.44269504088896341f;
    static constexpr float kLn2 = 0.693147180559945309f;
    static __device__ __forceinline__ float exp(float x) { return ptx_ex2(x * kLog2e); }
    static __device__ __forceinline__ float log(float x) { return ptx_lg2(x) * kLn2; }
    // arguments are >= 0 here (variances, moment ratios); sqrt.approx(0) = 0
    static __device__ __forceinline__ float sqrt(float x) { return ptx_sqrt(x); }
    static __device__ __forceinline__ float rcp(float x) { return ptx_rcp(x); }
    static __device__ __forceinline__ float div(float a, float b) { return a * ptx_rcp(b); }
    static __device__ __forceinline__ float erf(float x) { return erff(x); }
    // uniform in (0,1): (k + 1/2) / 2^23, k = top 23 bits of the word.  The float
    // 1 + k 2^-23 is built from its bits (k as the mantissa) and 1 - 2^-24 subtracted;
    // both are exact and so is the difference (2k + 1) 2^-24, so this equals
    // k * 2^-23 + 2^-24 bit for bit without an integer-to-float conversion.
    static __device__ __forceinline__ float u01(uint32_t w) {
        return __fsub_rn(mantissa(w), 0.99999994039535522f);
    }
    // 1 + k 2^-23 (one funnel shift: the exponent bits come in from the left)
    static __device__ __forceinline__ float mantissa(uint32_t w) {
        return __uint_as_float(__funnelshift_r(w, 0x7Fu, 9));
    }
    static constexpr float kU01Offset = 0.99999994039535522f;  // 1 - 2^-24
    static constexpr float kTwoPi = 6.28318530717958648f;
    // Box-Muller pair: R = sqrt(-2 ln u1), angle = 2*pi*(u2 - 1/2); IEEE-rounded
    // operations in a fixed order (box_muller_two repeats them on pairs).  With
    // f = 1 + k 2^-23, u2 - 1/2 = (f - 3/2) + 2^-24 exactly, so the angle is one FMA.
    static __device__ __forceinline__ void box_muller(uint32_t w1, uint32_t w2, float &z1, float &z2) {
        const float rad = ptx_sqrt(__fmul_rn(-2.0f * kLn2, ptx_lg2(u01(w1))));
        float s, c;
        __sincosf(__fmaf_rn(__fadd_rn(mantissa(w2), -1.5f), kTwoPi, kTwoPi / 16777216.0f), &s, &c);
        z1 = __fmul_rn(rad, c);
        z2 = __fmul_rn(rad, s);
    }
    // Two independent Box-Muller pairs, (a1, a2) and (b1, b2): the same operations as
    // box_muller with the FP32 multiplies and adds on the paired pipe, so each pair
    // gets the same bits as from box_muller.  z1 = (z1 of a, z1 of b), z2 likewise.
    static __device__ __forceinline__ void box_muller_two(uint32_t a1, uint32_t a2, uint32_t b1, uint32_t b2,
                                                          float2 &z1, float2 &z2) {
        const float2 u1 = __fadd2_rn(make_float2(mantissa(a1), mantissa(b1)), make_float2(-kU01Offset, -kU01Offset));
        const float2 g = __fadd2_rn(make_float2(mantissa(a2), mantissa(b2)), make_float2(-1.5f, -1.5f));
        const float2 t = __fmul2_rn(make_float2(-2.0f * kLn2, -2.0f * kLn2),
                                    make_float2(ptx_lg2(u1.x), ptx_lg2(u1.y)));
        const float2 rad = make_float2(ptx_sqrt(t.x), ptx_sqrt(t.y));
        const float2 ang = __ffma2_rn(g, make_float2(kTwoPi, kTwoPi),
                                      make_float2(kTwoPi / 16777216.0f, kTwoPi / 16777216.0f));
        float sa, ca, sb, cb;
        __sincosf(ang.x, &sa, &ca);
        __sincosf(ang.y, &sb, &cb);
        z1 = __fmul2_rn(rad, make_float2(ca, cb));
        z2 = __fmul2_rn(rad, make_float2(sa, sb));
    }
};

template <>
struct Math<double> {
    static __device__ __forceinline__ double exp(double x) { return ::exp(x); }
    static __device__ __forceinline__ double sqrt(double x) { return ::sqrt(x); }
    static __device__ __forceinline__ double u01(uint32_t w) {
        return (static_cast<double>(w) + 0.5) * (1.0 / 4294967296.0);
    }
    static __device__ __forceinline__ void box_muller(uint32_t w1, uint32_t w2, double &z1, double &z2) {
        const double u1 = u01(w1);
        const double u2 = u01(w2);
        const double rad = ::sqrt(-2.0 * ::log(u1));
        double s, c;
        ::sincospi(2.0 * u2 - 1.0, &s, &c);
        z1 = rad * c;
        z2 = rad * s;
    }
};

template <class R>
__device__ __forceinline__ R rmax(R a, R b) { return fmax(a, b); }
template <class R>
__device__ __forceinline__ R rmin(R a, R b) { return fmin(a, b); }

// ============================================================================
// Draw sources.  A step asks for: one normal pair (Z1, Z2); Bates steps then ask
// for Poisson uniforms one at a time and, when a jump occurred, one jump normal.
//
// Philox layout per path p of stream s (counter = (block, p, s, domain)):
//   normal pair of step n:        domain 0, block floor(n/2), words (x,y) if n even, (z,w) if odd;
//   1st Poisson uniform of step n: FP64 domain 2, block floor(n/4), word n mod 4;
//                                  FP32 23 bits: the low 9 bits of each of the step's two
//                                  normal words (18 bits), then the top 5 bits of that
//                                  domain-2 word, drawn only when the first 18 cannot
//                                  decide the jump test;
//   jump normal of step n:         domain 1, block n, Box-Muller of words (x,y), first output;
//   Poisson uniforms 2, 3:         domain 1, block n, words z, w;
//   Poisson uniform k >= 4:        domain 3 + (k-4)/4, block n, word (k-4) mod 4.
// A step costs half a Philox block for the normals and, under Bates in FP64, a
// quarter block for the jump test (in FP32 nearly nothing); the rest is drawn only
// on the rare steps with a jump.
// ============================================================================
template <class R>
struct PhiloxJumpDraws {
    uint32_t k0, k1, path, stream, step;
    R first;    // the step's first Poisson uniform
    int used;   // Poisson uniforms consumed so far in this step
    int domain; // block currently held in wx (0 = none)
    U4 wx;

    __device__ __forceinline__ U4 block(uint32_t d) {
        return philox4x32_10(U4{step, path, stream, d}, k0, k1);
    }
    __device__ __forceinline__ R uniform() {
        const int k = used++;
        if (k == 0) return first;
        const int d = (k < 3) ? 1 : 3 + (k - 3) / 4;
        if (domain != d) {
            wx = block(static_cast<uint32_t>(d));
            domain = d;
        }
        const int slot = (k < 3) ? k + 1 : ((k - 3) & 3);
        const uint32_t word = slot == 0 ? wx.x : (slot == 1 ? wx.y : (slot == 2 ? wx.z : wx.w));
        return Math<R>::u01(word);
    }
    __device__ __forceinline__ R jump_normal() {
        const U4 j = domain == 1 ? wx : block(1u);  // the block of the 2nd and 3rd uniforms
        R z1, z2;
        Math<R>::box_muller(j.x, j.y, z1, z2);
        return z1;
    }
};

// Fed draws for the parity trace: z[3] = {Z1, Z2, Zjump}; u[umax] Poisson uniforms.
template <class R>
struct FedStep {
    const double *z;
    const double *u;
    int umax;
    int used;
    int overflow;
    __device__ __forceinline__ void normal_pair(R &z1, R &z2) {
        z1 = static_cast<R>(z[0]);
        z2 = static_cast<R>(z[1]);
    }
    __device__ __forceinline__ R uniform() {
        if (used >= umax) {
            overflow = 1;
            return R(0);
        }
        return static_cast<R>(u[used++]);
    }
    __device__ __forceinline__ R jump_normal() { return static_cast<R>(z[2]); }
};

// ============================================================================
// Scheme steps: Heston + Euler (include/core/schemes/markovian/MSchemes.hpp:133-156),
// + implicit Milstein (MSchemes.hpp:229-253), + Andersen QE with martingale correction
// (MSchemes.hpp:363-442), in FP32 on the spot and in FP64 on its logarithm (step_spot64: on
// the spot).  QE's
// quadratic-branch martingale term log(exp(X)/sqrt(t)) is evaluated as X - log(t)/2 (the
// same quantity without an exp/rsqrt/log round trip).
// ============================================================================

// ----------------------------------------------------------------------------
// FP32 steps with an explicit rounding order.  Every FP32 operation below
// is an IEEE-rounded intrinsic (no compiler contraction), and the paired two-path
// forms further down perform the same operations on float2 pairs with the sm_100
// paired FP32 instructions, so one path gives the same bits whichever form
// simulates it.
__device__ __forceinline__ void qe_quadratic_f32(const StepConst<float> &p, float m, float m2, float s2, float Zv,
                                                 float &vn, float &logM) {
    const float two_ip = __fmul_rn(__fmul_rn(2.0f, m2), ptx_rcp(s2));
    const float t1 = __fadd_rn(two_ip, -1.0f);
    const float b2 = __fadd_rn(t1, ptx_sqrt(__fmul_rn(two_ip, t1)));
    const float a = __fmul_rn(m, ptx_rcp(__fadd_rn(1.0f, b2)));
    const float bz = __fadd_rn(ptx_sqrt(b2), Zv);
    vn = __fmul_rn(__fmul_rn(a, bz), bz);
    const float Aa = fminf(__fmul_rn(p.A, a), __fmaf_rn(-p.eps, a, 0.5f));
    const float term = __fmaf_rn(-2.0f, Aa, 1.0f);
    logM = __fmaf_rn(__fmul_rn(Aa, b2), ptx_rcp(term), __fmul_rn(-0.5f * Math<float>::kLn2, ptx_lg2(term)));
}

__device__ __forceinline__ void qe_spot_f32(const StepConst<float> &p, float &S, float v, float vn, float logM,
                                            float Zind) {
    const float K0n = __fmaf_rn(p.K1_half_K3, v, logM);  // -K0
    const float isig = __fmaf_rn(p.K3, v, __fmul_rn(p.K4, vn));
    const float e12 = __fadd_rn(__fadd_rn(p.r_minus_q_dt, -K0n), __fmaf_rn(p.K1, v, __fmul_rn(p.K2, vn)));
    const float ex = __fmaf_rn(ptx_sqrt(isig), Zind, e12);
    S = __fmul_rn(S, ptx_ex2(__fmul_rn(ex, Math<float>::kLog2e)));
}

__device__ __forceinline__ void step_qe_f32(const StepConst<float> &p, float &S, float &v, float Zv, float Zind) {
    const float m = __fmaf_rn(v, p.exp_mkdt, p.theta_m);
    const float s2 = __fmaf_rn(v, p.s2f1, p.s2f2);
    const float m2 = __fmul_rn(m, m);
    // the quadratic regime unconditionally (the common case, no branch before its
    // SFU chain); the other regimes overwrite its result
    float vn, logM;
    qe_quadratic_f32(p, m, m2, s2, Zv, vn, logM);
    if (m <= p.eps) {
        vn = 0.0f;
        logM = 0.0f;
    } else if (s2 <= __fmul_rn(p.eps, m2)) {
        vn = m;
        logM = 0.0f;
    } else if (!(s2 <= __fmul_rn(p.psi_c, m2))) {
        // exponential branch (rare at the usual parameters)
        const float inv_m = ptx_rcp(m);
        const float psi = s2 * inv_m * inv_m;
        const float pz = Math<float>::div(psi - 1.0f, psi + 1.0f);
        const float beta = (1.0f - pz) * inv_m;
        const float U = 0.5f * (1.0f + erff(Zv * p.inv_sqrt2));
        if (U <= pz) {
            vn = 0.0f;
        } else {
            const float safe_U = fminf(U, 1.0f - p.eps);
            vn = Math<float>::div(Math<float>::log(Math<float>::div(1.0f - pz, 1.0f - safe_U)), beta);
        }
        const float safe_A = fminf(p.A, beta - p.eps);
        const float M = pz + Math<float>::div(beta * (1.0f - pz), beta - safe_A);
        logM = Math<float>::log(M);
    }
    qe_spot_f32(p, S, v, vn, logM, Zind);
    v = vn;
}

__device__ __forceinline__ void step_euler_f32(const StepConst<float> &p, float &S, float &v, float Z1, float Z2) {
    const float ZS = __fmaf_rn(p.rho, Z1, __fmul_rn(p.rho_c, Z2));
    const float sqv = ptx_sqrt(v);
    const float ex = __fmaf_rn(__fmul_rn(sqv, p.sqrt_dt), ZS, __fmaf_rn(v, -p.half_dt, p.r_minus_q_dt));
    S = __fmul_rn(S, ptx_ex2(__fmul_rn(ex, Math<float>::kLog2e)));
    v = fmaxf(__fmaf_rn(__fmul_rn(p.sigma_sqrt_dt, sqv), Z1, __fmaf_rn(v, p.one_minus_k_dt, p.k_theta_dt)), 0.0f);
}

// Implicit Milstein variance update with an explicit rounding order.
__device__ __forceinline__ float milstein_variance_f32(const StepConst<float> &p, float v, float sqv, float Z1) {
    const float corr = __fmul_rn(p.quarter_sigma_sq_dt, __fmaf_rn(Z1, Z1, -1.0f));
    const float t = __fadd_rn(__fmaf_rn(__fmul_rn(p.sigma_sqrt_dt, sqv), Z1, __fadd_rn(v, p.k_theta_dt)), corr);
    return fmaxf(__fmul_rn(p.implicit_den, t), 0.0f);
}

__device__ __forceinline__ void step_milstein_f32(const StepConst<float> &p, float &S, float &v, float Z1, float Z2) {
    const float ZS = __fmaf_rn(p.rho, Z1, __fmul_rn(p.rho_c, Z2));
    const float sqv = ptx_sqrt(v);
    const float ex = __fmaf_rn(__fmul_rn(sqv, p.sqrt_dt), ZS, __fmaf_rn(v, -p.half_dt, p.r_minus_q_dt));
    S = __fmul_rn(S, ptx_ex2(__fmul_rn(ex, Math<float>::kLog2e)));
    v = milstein_variance_f32(p, v, sqv, Z1);
}

// Paired FP32: component-wise IEEE operations on two paths at once.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 rcp2(float2 x) { return make_float2(ptx_rcp(x.x), ptx_rcp(x.y)); }
__device__ __forceinline__ float2 sqrt2(float2 x) { return make_float2(ptx_sqrt(x.x), ptx_sqrt(x.y)); }
__device__ __forceinline__ float2 lg2_2(float2 x) { return make_float2(ptx_lg2(x.x), ptx_lg2(x.y)); }
__device__ __forceinline__ float2 ex2_2(float2 x) { return make_float2(ptx_ex2(x.x), ptx_ex2(x.y)); }
__device__ __forceinline__ float2 max0_2(float2 a) { return make_float2(fmaxf(a.x, 0.0f), fmaxf(a.y, 0.0f)); }

// Where the paired QE step takes 1 / term and log2 term from, term = 1 - 2 A a: the SFU, or
// a shared-memory table of the SFU's results for every float of the task's range
// [lo, lo + n) of bit patterns (term moves by a few hundred millionths, so at daily steps
// that is a few thousand floats).  The same bits for two of the step's twelve SFU
// operations less, on the unit that bounds QE: five-payoff Bates QE, 16,777,216 x 252,
// 14.00 -> 13.41 ms; Heston QE Asian, 5,000,000 x 365, 5.62 -> 5.33 ms.
struct TermSfu {
    static constexpr bool kTable = false;
};
struct TermTable {
    static constexpr bool kTable = true;
    const float2 *tab;  // kTermTableMax + 1 entries; the last one stands for all terms beyond
    uint32_t lo;
    __device__ __forceinline__ static TermTable fill(float2 *tab, uint32_t lo) {
        for (uint32_t i = threadIdx.x; i <= kTermTableMax; i += blockDim.x) {
            const float x = __uint_as_float(lo + i);
            tab[i] = make_float2(ptx_rcp(x), __fmul_rn(-0.5f * Math<float>::kLn2, ptx_lg2(x)));
        }
        __syncthreads();
        return TermTable{tab, lo};
    }
};

// QE step of two paths (spot S, variance v as pairs): paired when both take the
// quadratic branch (the common case), otherwise each path through step_qe_f32.
template <class Term>
__device__ __forceinline__ void step_qe_two_f32(const Term &tt, const StepConst<float> &p, float2 &S, float2 &v,
                                                float2 Zv, float2 Zind) {
    const float2 m = __ffma2_rn(v, f2(p.exp_mkdt), f2(p.theta_m));
    const float2 h = __ffma2_rn(v, f2(p.h_f1), f2(p.h_f2));  // s^2 / 2
    const float2 m2 = __fmul2_rn(m, m);
    // the quadratic form for both paths first (no branch before the long SFU chain);
    // a pair not both in the quadratic regime is redone per path below
    const float2 S_old = S, v_old = v;
    // qe_quadratic_f32, paired: m2 rcp(s^2 / 2) has the bits of 2 m2 rcp(s^2), and where
    // ip_lo admits the step min(A a, 1/2 - eps a) is A a
    const float2 two_ip = __fmul2_rn(m2, rcp2(h));
    // the regime from 2 / psi itself, a little inside its bounds (StepConst::ip_lo), instead of
    // from s^2 against eps m^2 and psi_c m^2; the task of a term table has m > eps on every
    // step (term_range_lo).  Same bits.  Five-payoff Bates QE 13.41 -> 13.21 ms, Heston QE Asian
    // 5.32 -> 5.15 ms, American put FP32 4.19 -> 4.12 ms.
    bool quad = two_ip.x >= p.ip_lo && two_ip.y >= p.ip_lo && two_ip.x < p.ip_hi && two_ip.y < p.ip_hi;
    if constexpr (!Term::kTable) quad = quad && m.x > p.eps && m.y > p.eps;
    const float2 t1 = __fadd2_rn(two_ip, f2(-1.0f));
    const float2 b2 = __fadd2_rn(t1, sqrt2(__fmul2_rn(two_ip, t1)));
    const float2 a = __fmul2_rn(m, rcp2(__fadd2_rn(f2(1.0f), b2)));
    const float2 bz = __fadd2_rn(sqrt2(b2), Zv);
    const float2 vn = __fmul2_rn(__fmul2_rn(a, bz), bz);
    const float2 Aa = __fmul2_rn(f2(p.A), a);
    const float2 term = __ffma2_rn(f2(-2.0f), Aa, f2(1.0f));
    float2 rterm, lterm;  // 1 / term, -ln(term) / 2
    if constexpr (Term::kTable) {
        const uint32_t ia = __float_as_uint(term.x) - tt.lo, ib = __float_as_uint(term.y) - tt.lo;
        quad = quad && ia < kTermTableMax && ib < kTermTableMax;
        const float2 ta = tt.tab[min(ia, kTermTableMax)], tb = tt.tab[min(ib, kTermTableMax)];
        rterm = make_float2(ta.x, tb.x);
        lterm = make_float2(ta.y, tb.y);
    } else {
        rterm = rcp2(term);
        lterm = __fmul2_rn(f2(-0.5f * Math<float>::kLn2), lg2_2(term));
    }
    const float2 logM = __ffma2_rn(__fmul2_rn(Aa, b2), rterm, lterm);
    // qe_spot_f32, paired
    const float2 K0n = __ffma2_rn(f2(p.K1_half_K3), v, logM);
    const float2 isig = __ffma2_rn(f2(p.K3), v, __fmul2_rn(f2(p.K4), vn));
    const float2 e12 = __fadd2_rn(__ffma2_rn(K0n, f2(-1.0f), f2(p.r_minus_q_dt)),
                                  __ffma2_rn(f2(p.K1), v, __fmul2_rn(f2(p.K2), vn)));
    const float2 ex = __ffma2_rn(sqrt2(isig), Zind, e12);
    S = __fmul2_rn(S, ex2_2(__fmul2_rn(ex, f2(Math<float>::kLog2e))));
    v = vn;
    if (!quad) {
        // one copy of the one-path step for both paths (rare; keeps the loop body small)
        S = S_old;
        v = v_old;
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
            float Si = i ? S.y : S.x, vi = i ? v.y : v.x;
            step_qe_f32(p, Si, vi, i ? Zv.y : Zv.x, i ? Zind.y : Zind.x);
            if (i) {
                S.y = Si;
                v.y = vi;
            } else {
                S.x = Si;
                v.x = vi;
            }
        }
    }
}

// Milstein for two paths: the spot update (the same as Euler's) paired, the
// variance update per path.
__device__ __forceinline__ void step_milstein_two_f32(const StepConst<float> &p, float2 &S, float2 &v, float2 Z1,
                                                      float2 Z2) {
    const float2 ZS = __ffma2_rn(f2(p.rho), Z1, __fmul2_rn(f2(p.rho_c), Z2));
    const float2 sqv = sqrt2(v);
    const float2 ex = __ffma2_rn(__fmul2_rn(sqv, f2(p.sqrt_dt)), ZS, __ffma2_rn(v, f2(-p.half_dt), f2(p.r_minus_q_dt)));
    S = __fmul2_rn(S, ex2_2(__fmul2_rn(ex, f2(Math<float>::kLog2e))));
    v = make_float2(milstein_variance_f32(p, v.x, sqv.x, Z1.x), milstein_variance_f32(p, v.y, sqv.y, Z1.y));
}

__device__ __forceinline__ void step_euler_two_f32(const StepConst<float> &p, float2 &S, float2 &v, float2 Z1,
                                                   float2 Z2) {
    const float2 ZS = __ffma2_rn(f2(p.rho), Z1, __fmul2_rn(f2(p.rho_c), Z2));
    const float2 sqv = sqrt2(v);
    const float2 ex = __ffma2_rn(__fmul2_rn(sqv, f2(p.sqrt_dt)), ZS, __ffma2_rn(v, f2(-p.half_dt), f2(p.r_minus_q_dt)));
    S = __fmul2_rn(S, ex2_2(__fmul2_rn(ex, f2(Math<float>::kLog2e))));
    v = max0_2(__ffma2_rn(__fmul2_rn(f2(p.sigma_sqrt_dt), sqv), Z1,
                          __ffma2_rn(v, f2(p.one_minus_k_dt), f2(p.k_theta_dt))));
}

template <int SCHEME>
__device__ __forceinline__ void heston_step_f32(const StepConst<float> &p, float &S, float &v, float Z1, float Z2) {
    if constexpr (SCHEME == kEuler) step_euler_f32(p, S, v, Z1, Z2);
    else if constexpr (SCHEME == kMilstein) step_milstein_f32(p, S, v, Z1, Z2);
    else step_qe_f32(p, S, v, Z1, Z2);
}

// ----------------------------------------------------------------------------
// FP64 steps on the base-2 logarithm x of S / S0: one path-step then needs no
// exponential (a spot is formed only where something reads it), and every operation is
// one of qk_math64.cuh's.
//
// QE, quadratic regime, with h = s^2 / 2, G = sqrt(m^2 - h) (h < m^2 as psi <= psi_c < 2)
// and q = m + G.  The textbook's b^2 = 2/psi - 1 + sqrt(2/psi (2/psi - 1)) and
// a = m / (1 + b^2) are, multiplied out, a b^2 = G and a = h / q, so that
//   vn = a (b + Zv)^2,  b = G / sqrt(a G),
//   1 - 2 A a = u / q,  u = q - 2 A h,   w = a b^2 / (1 - 2 A a) = G q / u,
// and one reciprocal of q u serves both q and u: a square root, a reciprocal and a
// reciprocal square root in place of three reciprocals and two square roots.
//
// Two sums are ordered by their rounding.  K2 vn - A w, nearly equal products of numbers of
// the order of rho / sigma, is K2 (vn - w) + (K2 - A) w: nothing of the order of rho / sigma
// is rounded but the constants, and those as the reference rounds them.  The martingale
// factor's sqrt(1 - 2 A a) goes into a running product P, folded into x by one logarithm per
// 16 steps (fewer where P could fall below 1/2 before, qe_fold_steps); its factors are next
// to 1, so what is accumulated is E = (1 - P) / (2 A), the sum of a P, whose rounding is that
// of numbers of the order of E.  Errors against long double, Heston QE Asian, ten contracts of
// 100,003 x 126 (rms): price 3.9e-16 with step_spot64's formulas, 3.4e-16 with these (3.8e-15
// with A w rounded apart from K2 vn), vomma 1.2e-10 and 4.3e-11 (1.4e-10 with the factors
// multiplied up themselves).
// ----------------------------------------------------------------------------
struct Path64 {
    double x, P, E, v;  // log2(S / S0) = x + log2(P) / 2, P = 1 - 2 A E
};
constexpr double kLog2e64 = 1.44269504088896340736;

// The regimes of a QE step as the reference branches between them (MSchemes.hpp:363-442);
// (vn, log M).  Reached when a step is not plainly inside the quadratic regime.
__device__ __noinline__ inline double2 qe_regimes64(double m, double s2, double Zv, double psi_c, double eps, double A) {
    if (m <= eps) return make_double2(0.0, 0.0);
    const double m2 = m * m;
    if (s2 <= eps * m2) return make_double2(m, 0.0);
    if (s2 <= psi_c * m2) {
        const double two_ip = 2.0 * m2 / s2;
        const double b2 = two_ip - 1.0 + ::sqrt(two_ip * (two_ip - 1.0));
        const double a = m / (1.0 + b2);
        const double bz = ::sqrt(b2) + Zv;
        const double Aa = fmin(A * a, 0.5 - eps * a);  // min(A, 1/(2a) - eps) a
        const double term = 1.0 - 2.0 * Aa;
        return make_double2(a * bz * bz, Aa * b2 / term - 0.5 * ::log(term));
    }
    const double inv_m = 1.0 / m;
    const double psi = s2 * inv_m * inv_m;
    const double pz = (psi - 1.0) / (psi + 1.0);
    const double beta = (1.0 - pz) * inv_m;
    const double U = 0.5 * (1.0 + ::erf(Zv * 0.70710678118654752440));
    const double vn = U <= pz ? 0.0 : ::log((1.0 - pz) / (1.0 - fmin(U, 1.0 - eps))) / beta;
    const double safe_A = fmin(A, beta - eps);
    return make_double2(vn, ::log(pz + beta * (1.0 - pz) / (beta - safe_A)));
}

__device__ __forceinline__ bool below_hi64(double a, double b) { return __double2hiint(a) < __double2hiint(b); }

template <int SCHEME>
__device__ __forceinline__ void step64(const StepConst<double> &p, Path64 &s, double Z1, double Z2) {
    const double v = s.v;
    if constexpr (SCHEME != kQE) {
        const double sq = sqrt64(v);
        const double ZS = fma(p.rho, Z1, p.rho_c * Z2);
        s.x += fma(sq * p.l_sqrt_dt, ZS, fma(v, -p.l_half_dt, p.l_drift));
        const double noise = (p.sigma_sqrt_dt * sq) * Z1;
        if constexpr (SCHEME == kEuler) {
            s.v = max0_64(fma(v, p.one_minus_k_dt, p.k_theta_dt) + noise);
        } else {
            const double corr = p.quarter_sigma_sq_dt * fma(Z1, Z1, -1.0);
            s.v = max0_64(p.implicit_den * (((v + p.k_theta_dt) + noise) + corr));
        }
    } else {
        const double m = fma(v, p.exp_mkdt, p.theta_m);
        const double h = fma(v, p.h_f1, p.h_f2);
        const double m2 = m * m;
        const double G = sqrt_pos64(m2 - h);
        const double q = m + G;
        const double u = fma(-p.two_A, h, q);
        const double R = rcp64(q * u);
        double a = h * (u * R);
        const double b = G * rsqrt64(a * G);
        const double bz = b + Z1;
        double vn = (a * bz) * bz;
        double w = (G * q) * (q * R);
        // Inside the quadratic regime (m > eps, eps m^2 < s^2 <= psi_c m^2), no clamp possible?
        // Compared by the high words (positive values order as integers), strictly, so a value
        // next to a threshold, and NaN, take the exact branches.
        const bool quad = below_hi64(p.eps, m) && below_hi64(p.h_eps * m2, h) && below_hi64(h, p.h_psi_plain * m2);
        if (!quad) {
            const double2 r = qe_regimes64(m, 2.0 * h, Z1, p.psi_c, p.eps, p.A);
            vn = r.x;
            s.x = fma(r.y, -kLog2e64, s.x);
            w = a = 0.0;
        }
        s.E = fma(a, s.P, s.E);
        s.P = fma(-p.two_A, s.E, 1.0);
        s.x += fma(sqrt64(v + vn), p.l_sqrt_K3 * Z2, fma(p.l_K2, vn - w, fma(p.l_c2, w, fma(p.l_c1, v, p.l_drift))));
        s.v = vn;
    }
}

// P into x (every TaskDev::fold_steps steps).
template <int SCHEME>
__device__ __forceinline__ void fold64(const Tab64 &t, Path64 &s) {
    if constexpr (SCHEME == kQE) {
        s.x = fma(neg2_log64(t, s.P, 0), -0.25 * kLog2e64, s.x);
        s.P = 1.0;
        s.E = 0.0;
    }
}

// S / S0
template <int SCHEME>
__device__ __forceinline__ double rel_spot64(const Tab64 &t, const Path64 &s) {
    if constexpr (SCHEME == kQE) return exp2_64(t, s.x) * sqrt_pos64(s.P);
    else return exp2_64(t, s.x);
}

// ----------------------------------------------------------------------------
// FP64 steps on the spot itself with the CUDA library's functions: the paths of American
// contracts in the reference's mode (Laguerre basis) and of the path dump.  An American
// price hangs on exercise decisions, and in that mode those come from unscaled normal
// equations whose smallest pivot is 1e-7 beside sums of 1e5: last bits of the spots reach
// the fit, one flipped decision spreads to a thousand at earlier dates, and the price moves
// by 1e-4 of itself (with step64's paths on 3 of 164 contracts tried, up to 4e-4).  These
// steps keep the spots, and with them those prices, bit for bit.  The six-term basis is
// centred, scaled and solved with a condition check: 400 of its contracts priced with
// step64's paths differ by at most 3e-13, and they keep those paths.  300,001 x 100 on every
// date, Laguerre: Heston Milstein 1,134 us with step64's paths, 1,261 us with these; six
// terms, 25 dates: Heston QE 509 us, 840 us.
// ----------------------------------------------------------------------------
template <int SCHEME>
__device__ __forceinline__ void step_spot64(const StepConst<double> &p, double &S, double &v, double Z1, double Z2) {
    if constexpr (SCHEME != kQE) {
        const double ZS = p.rho * Z1 + p.rho_c * Z2;
        const double sqv = ::sqrt(v);
        const double ex = p.r_minus_q_dt - v * p.half_dt + (sqv * p.sqrt_dt) * ZS;
        const double Sn = S * ::exp(ex);
        double vn;
        if constexpr (SCHEME == kEuler) {
            vn = v * p.one_minus_k_dt + p.k_theta_dt + (p.sigma_sqrt_dt * sqv) * Z1;
        } else {
            const double corr = p.quarter_sigma_sq_dt * (Z1 * Z1 - 1.0);
            vn = p.implicit_den * (v + p.k_theta_dt + (p.sigma_sqrt_dt * sqv) * Z1 + corr);
        }
        S = Sn;
        v = fmax(vn, 0.0);
    } else {
        const double m = v * p.exp_mkdt + p.theta_m;
        const double s2 = v * p.s2f1 + p.s2f2;
        double vn, logM;  // logM: log of the martingale factor
        if (m <= p.eps) {
            vn = 0.0;
            logM = 0.0;
        } else {
            const double m2 = m * m;
            if (s2 <= p.eps * m2) {
                vn = m;
                logM = 0.0;
            } else if (s2 <= p.psi_c * m2) {
                const double two_ip = 2.0 * m2 * (1.0 / s2);  // 2 / psi
                const double b2 = two_ip - 1.0 + ::sqrt(two_ip * (two_ip - 1.0));
                const double a = m * (1.0 / (1.0 + b2));
                const double bz = ::sqrt(b2) + Z1;
                vn = a * bz * bz;
                const double Aa = fmin(p.A * a, 0.5 - p.eps * a);  // min(A, 1/(2a) - eps) a
                const double term = 1.0 - 2.0 * Aa;
                logM = Aa * b2 * (1.0 / term) - 0.5 * ::log(term);
            } else {
                const double inv_m = 1.0 / m;
                const double psi = s2 * inv_m * inv_m;
                const double pz = (psi - 1.0) / (psi + 1.0);
                const double beta = (1.0 - pz) * inv_m;
                const double U = 0.5 * (1.0 + ::erf(Z1 * p.inv_sqrt2));
                if (U <= pz) {
                    vn = 0.0;
                } else {
                    const double safe_U = fmin(U, 1.0 - p.eps);
                    vn = ::log((1.0 - pz) / (1.0 - safe_U)) / beta;
                }
                const double safe_A = fmin(p.A, beta - p.eps);
                const double M = pz + (beta * (1.0 - pz)) / (beta - safe_A);
                logM = ::log(M);
            }
        }
        const double K0 = -logM - p.K1_half_K3 * v;
        const double isig = p.K3 * v + p.K4 * vn;
        const double ex = p.r_minus_q_dt + K0 + (p.K1 * v + p.K2 * vn) + ::sqrt(isig) * Z2;
        S = S * ::exp(ex);
        v = vn;
    }
}

// Bates jump part after the (drift-compensated) Heston step: MSchemes.hpp:493-526.
// Knuth's Poisson draw: multiply uniforms until the product drops below exp(-lambda dt).
// `prod` holds the first uniform, already known to be >= exp(-lambda dt) (a jump).
template <class R, class Draws>
__device__ __noinline__ R jump_factor(const StepConst<R> &p, R prod, Draws &d) {
    int N = 0;
    do {
        ++N;
        prod *= d.uniform();
    } while (prod >= p.exp_m_lambda_dt && N < kMaxJumpsPerStep);
    const R Z = d.jump_normal();
    const R rN = static_cast<R>(N);
    return Math<R>::exp(rN * p.mu_j + Math<R>::sqrt(rN) * p.sigma_j * Z);
}


// Both members of an antithetic pair: the same jump count, jump sizes with the
// normal of opposite sign.
template <class R, class Draws>
__device__ __noinline__ void jump_factor_pair(const StepConst<R> &p, R prod, Draws &d, R &fa, R &fb) {
    int N = 0;
    do {
        ++N;
        prod *= d.uniform();
    } while (prod >= p.exp_m_lambda_dt && N < kMaxJumpsPerStep);
    const R Z = d.jump_normal();
    const R rN = static_cast<R>(N);
    const R m = rN * p.mu_j;
    const R s = Math<R>::sqrt(rN) * p.sigma_j * Z;
    fa = Math<R>::exp(m + s);
    fb = Math<R>::exp(m - s);
}

template <class R, class Draws>
__device__ __forceinline__ void bates_jump(const StepConst<R> &p, R &S, Draws &d) {
    const R first = d.uniform();
    if (first >= p.exp_m_lambda_dt) S *= jump_factor<R>(p, first, d);
}

// One step on the spot itself for the fed-draw trace: the pricing kernels' scheme steps, but
// with the martingale product folded and the spot formed after every step, and in FP64 the
// jumps of jump_factor on the fed draws (the pricing kernels': jump_log2_f64).
template <class R, int MODEL, int SCHEME, class Draws>
__device__ __forceinline__ void evolve_step(const Tab64 *tab, const StepConst<R> &p, R &S, R &v, Draws &d) {
    R Z1, Z2;
    d.normal_pair(Z1, Z2);
    if constexpr (sizeof(R) == 4) {
        heston_step_f32<SCHEME>(p, S, v, Z1, Z2);
    } else {
        Path64 s{0.0, 1.0, 0.0, v};
        step64<SCHEME>(p, s, Z1, Z2);
        fold64<SCHEME>(*tab, s);
        S *= exp2_64(*tab, s.x);
        v = s.v;
    }
    if constexpr (MODEL == kBates) bates_jump<R>(p, S, d);
}

// ============================================================================
// Payoffs: include/core/options/Payoff.hpp:35-243.  Trackers (running sum in
// double, running max / min started at S0) are kept for every path; the final
// payoff per requested contract leg reads the ones it needs.
// ============================================================================
template <class R>
__device__ __forceinline__ R intrinsic(int right, R S, R K) {
    return right == kCall ? (S > K ? S - K : R(0)) : (K > S ? K - S : R(0));
}

template <class R>
__device__ __forceinline__ R final_payoff(const PayoffSpec &ps, R S, double ssum, R smax, R smin, int n_steps) {
    const R K = static_cast<R>(ps.K);
    const R B = static_cast<R>(ps.B);
    switch (ps.type) {
        case kEuropean: return intrinsic<R>(ps.right, S, K);
        case kAsian: return intrinsic<R>(ps.right, static_cast<R>(ssum / static_cast<double>(n_steps)), K);
        case kBarrierUpOut: return smax < B ? intrinsic<R>(ps.right, S, K) : R(0);
        case kBarrierDownOut: return smin > B ? intrinsic<R>(ps.right, S, K) : R(0);
        case kBarrierUpIn: return smax >= B ? intrinsic<R>(ps.right, S, K) : R(0);
        case kBarrierDownIn: return smin <= B ? intrinsic<R>(ps.right, S, K) : R(0);
        case kLookbackFloating:
            return ps.right == kCall ? intrinsic<R>(kCall, S, smin) : intrinsic<R>(kPut, S, smax);
        case kLookbackFixed:
            return ps.right == kCall ? intrinsic<R>(kCall, smax, K) : intrinsic<R>(kPut, smin, K);
        case kBinaryCash:
            return ps.right == kCall ? (S > K ? R(1) : R(0)) : (S < K ? R(1) : R(0));
        case kBinaryAsset:
            return ps.right == kCall ? (S > K ? S : R(0)) : (S < K ? S : R(0));
        default: return intrinsic<R>(ps.right, S, K);  // American legs priced at maturity only here
    }
}

// ============================================================================
// FP64 statistics: (n, mean, M2) merged with Chan et al.'s parallel update.
// ============================================================================
__device__ __forceinline__ Moments chan_merge(const Moments &a, const Moments &b) {
    const double n = a.n + b.n;
    if (n <= 0.0) return Moments{0.0, 0.0, 0.0, 0.0};
    if (a.n <= 0.0) return b;
    if (b.n <= 0.0) return a;
    const double d = b.mean - a.mean;
    Moments r;
    r.n = n;
    r.mean = a.mean + d * (b.n / n);
    r.m2 = a.m2 + b.m2 + d * d * (a.n * b.n / n);
    r.itm = a.itm + b.itm;
    return r;
}

__device__ __forceinline__ Moments shfl_down_moments(const Moments &m, int off) {
    Moments r;
    r.n = __shfl_down_sync(0xffffffffu, m.n, off);
    r.mean = __shfl_down_sync(0xffffffffu, m.mean, off);
    r.m2 = __shfl_down_sync(0xffffffffu, m.m2, off);
    r.itm = __shfl_down_sync(0xffffffffu, m.itm, off);
    return r;
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    return x;
}

// Exact two-pass moments of the 32 values of a warp (inactive lanes excluded):
// the values are in registers, so the second pass costs one more shuffle tree.
__device__ __forceinline__ Moments warp_moments(double x, bool active, bool itm) {
    const unsigned act = __ballot_sync(0xffffffffu, active);
    const unsigned im = __ballot_sync(0xffffffffu, active && itm);
    const double n = static_cast<double>(__popc(act));
    const double s = warp_sum(active ? x : 0.0);
    const double mean = n > 0.0 ? s / n : 0.0;
    const double dv = active ? x - mean : 0.0;
    const double m2 = warp_sum(dv * dv);
    return Moments{n, mean, m2, static_cast<double>(__popc(im))};
}

// Moments of the 32 pair averages of a warp (antithetic sampling): each lane's
// value is (x_a + x_b) / 2 and its in-the-money weight (1{a} + 1{b}) / 2.
__device__ __forceinline__ Moments warp_moments_pair(double y, bool active, bool itm_a, bool itm_b) {
    const unsigned act = __ballot_sync(0xffffffffu, active);
    const unsigned ia = __ballot_sync(0xffffffffu, active && itm_a);
    const unsigned ib = __ballot_sync(0xffffffffu, active && itm_b);
    const double n = static_cast<double>(__popc(act));
    const double s = warp_sum(active ? y : 0.0);
    const double mean = n > 0.0 ? s / n : 0.0;
    const double dv = active ? y - mean : 0.0;
    const double m2 = warp_sum(dv * dv);
    return Moments{n, mean, m2, 0.5 * static_cast<double>(__popc(ia) + __popc(ib))};
}

}  // namespace qk
