// Device arithmetic shared by the photon kernels: the counter-based RNG, the Fresnel reflectance
// of an interface and the Henyey-Greenstein spin. Everything here is FP32 except the
// near-critical-angle Fresnel branch, which is FP64.
#pragma once

#include <cmath>
#include <cstdint>

namespace xmc {

// Philox4x32-10 (Salmon, Moraes, Dror, Shaw: "Parallel random numbers: as easy as 1, 2, 3", SC'11):
// ten rounds of the published round function and Weyl key schedule.
__host__ __device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint32_t k0, uint32_t k1) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
#ifdef __CUDA_ARCH__
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
#else
        const uint64_t p0 = (uint64_t)0xD2511F53u * c.x, p1 = (uint64_t)0xCD9E8D57u * c.z;
        const uint32_t lo0 = (uint32_t)p0, hi0 = (uint32_t)(p0 >> 32);
        const uint32_t lo1 = (uint32_t)p1, hi1 = (uint32_t)(p1 >> 32);
#endif
        c = make_uint4(hi1 ^ c.y ^ k0, lo1, hi0 ^ c.w ^ k1, lo0);
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
    }
    return c;
}

// The same with the key schedule worked out beforehand (philox_round_keys): the round keys come from the
// kernel's parameters as operands of the rounds' XORs instead of two additions per round.
struct PhiloxKeys {
    uint32_t k0[10], k1[10];
};
inline PhiloxKeys philox_round_keys(uint32_t k0, uint32_t k1) {
    PhiloxKeys k;
    for (int r = 0; r < 10; ++r) {
        k.k0[r] = k0 + (uint32_t)r * 0x9E3779B9u;
        k.k1[r] = k1 + (uint32_t)r * 0xBB67AE85u;
    }
    return k;
}
#ifdef __CUDACC__
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, const PhiloxKeys& k) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint32_t lo0 = 0xD2511F53u * c.x, hi0 = __umulhi(0xD2511F53u, c.x);
        const uint32_t lo1 = 0xCD9E8D57u * c.z, hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k.k0[r], lo1, hi0 ^ c.w ^ k.k1[r], lo0);
    }
    return c;
}
#endif

// 24-bit uniform in (0,1), exactly the value the FP64 oracle uses.
__host__ __device__ __forceinline__ float u24(uint32_t x) { return fmaf((float)(x >> 8), 0x1p-24f, 0x1p-25f); }

// Sums of products with the rounding of every term written out. Left to the compiler, which of two products is
// rounded on its own differs from kernel to kernel with the registers at hand; a photon is walked by more than one
// kernel, by which one is a matter of timing, and has to take the same path in each.
__host__ __device__ __forceinline__ float mul_rn(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fmul_rn(a, b);
#else
    return a * b;
#endif
}
// a b + c d, a b - c d, and the dot product of two vectors
__host__ __device__ __forceinline__ float sum2(float a, float b, float c, float d) { return fmaf(a, b, mul_rn(c, d)); }
__host__ __device__ __forceinline__ float diff2(float a, float b, float c, float d) { return fmaf(a, b, -mul_rn(c, d)); }
__host__ __device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
    return fmaf(az, bz, sum2(ax, bx, ay, by));
}

#ifdef __CUDACC__
// Reflectance of an interface for incidence cosine ci (0 < ci <= 1) from index ni into nt:
// GetCriticalCos, ComputeTransmitCosine and ComputeFrenselReflectance of the reference
// (base/xmcml/xmcml/mcml_kernel.cpp:497-564, :644-661). Total internal reflection gives 1; within
// 1e-3 of the critical cosine the unpolarised Fresnel formula is evaluated in FP64.
__device__ __forceinline__ float fresnel_reflectance(float ni, float nt, float ci) {
    if (ni == nt) return 0.0f;
    const float cc = ni > nt ? sqrtf(1.0f - (nt * nt) / (ni * ni)) : 0.0f;
    if (ci <= cc) return 1.0f;
    if (ci > 1.0f - 1e-6f) {
        const float r = (nt - ni) / (nt + ni);
        return r * r;
    }
    if (ci < 1e-6f) return 1.0f;
    if (ni > nt && ci - cc < 1e-3f) {
        const double Ci = ci, Ni = ni, Nt = nt;
        const double Si = sqrt(1.0 - Ci * Ci);
        const double St = Ni * Si / Nt;
        if (St >= 1.0) return 1.0f;
        const double Ct = sqrt(1.0 - St * St);
        const double pc = __dmul_rn(Si, St), ps = __dmul_rn(Ci, St);
        const double cs = __fma_rn(Ci, Ct, -pc), cd = __fma_rn(Ci, Ct, pc);
        const double ss = __fma_rn(Si, Ct, ps), sd = __fma_rn(Si, Ct, -ps);
        return (float)(0.5 * sd * sd * __fma_rn(cd, cd, __dmul_rn(cs, cs)) / (ss * ss * cd * cd));
    }
    const float si = sqrtf(1.0f - ci * ci);
    const float st = ni * si / nt;
    if (st >= 1.0f) return 1.0f;
    const float ct = sqrtf(1.0f - st * st);
    const float pc = __fmul_rn(si, st), ps = __fmul_rn(si, ct);
    const float cs = __fmaf_rn(ci, ct, -pc), cd = __fmaf_rn(ci, ct, pc);
    const float ss = __fmaf_rn(ci, st, ps), sd = __fmaf_rn(-ci, st, ps);
    return 0.5f * sd * sd * __fmaf_rn(cd, cd, __fmul_rn(cs, cs)) / (ss * ss * cd * cd);
}

// sqrt(x^2 + y^2) with the rounding written out, for the same reason.
__device__ __forceinline__ float radius_xy(float x, float y) { return sqrtf(__fmaf_rn(x, x, __fmul_rn(y, y))); }

// Deflection of an interaction (ComputeCosineTheta, mcml_kernel.cpp:442-463): Henyey-Greenstein
// cos(theta) from u1 by the inverse CDF (hg_* = 1 - g^2, 1 + g^2, 1 / 2g, 1 - g, 2g; isotropic when
// hg_e == 0) and sin(theta); sine and cosine of the azimuth 2 pi u2. It does not depend on the direction.
__device__ __forceinline__ void hg_angles(float hg_a, float hg_b, float hg_c, float hg_d, float hg_e, float u1, float u2,
                                          float& cost, float& sint, float& sp, float& cp) {
    const float t = hg_a / (hg_d + hg_e * u1);
    cost = hg_e != 0.0f ? (hg_b - t * t) * hg_c : 2.0f * u1 - 1.0f;
    cost = fminf(1.0f, fmaxf(-1.0f, cost));
    sint = sqrtf(fmaxf(0.0f, 1.0f - cost * cost));
    float a = u2;
    a = a > 0.5f ? a - 1.0f : a;  // same angle as 2*pi*u, reduced to [-pi, pi]
    __sincosf(6.283185307179586f * a, &sp, &cp);
}

// GetNewPhotonDirection (mcml_kernel.cpp:464-495): rotation of (dx, dy, dz) by these angles, with the
// near-vertical special case.
__device__ __forceinline__ void hg_rotate(float cost, float sint, float sp, float cp, float& dx, float& dy, float& dz) {
    const float ux = dx, uy = dy, uz = dz;
    // the rounding of every sum is written out (see fresnel_reflectance), and both cases are computed: a branch
    // for the rare one would end the straight line that the compiler schedules the random numbers into
    const float rho2 = __fmaf_rn(uy, uy, __fmul_rn(ux, ux));
    const float irho = rsqrtf(rho2);
    const float rho = __fmul_rn(rho2, irho);
    const float ax = __fmaf_rn(__fmul_rn(ux, uz), cp, -__fmul_rn(uy, sp)), ay = __fmaf_rn(ux, sp, __fmul_rn(__fmul_rn(uy, uz), cp));
    const bool slanted = rho2 > 1e-12f;
    const float nx = slanted ? __fmaf_rn(ux, cost, __fmul_rn(__fmul_rn(sint, ax), irho)) : __fmul_rn(sint, cp);
    const float ny = slanted ? __fmaf_rn(uy, cost, __fmul_rn(__fmul_rn(sint, ay), irho)) : __fmul_rn(sint, sp);
    const float nz = slanted ? __fmaf_rn(uz, cost, __fmul_rn(__fmul_rn(-sint, cp), rho)) : uz >= 0.0f ? cost : -cost;
    const float on = rsqrtf(__fmaf_rn(nz, nz, __fmaf_rn(nx, nx, __fmul_rn(ny, ny))));
    dx = __fmul_rn(nx, on);
    dy = __fmul_rn(ny, on);
    dz = __fmul_rn(nz, on);
}

__device__ __forceinline__ void hg_spin(float hg_a, float hg_b, float hg_c, float hg_d, float hg_e, float u1, float u2,
                                        float& dx, float& dy, float& dz) {
    float cost, sint, sp, cp;
    hg_angles(hg_a, hg_b, hg_c, hg_d, hg_e, u1, u2, cost, sint, sp, cp);
    hg_rotate(cost, sint, sp, cp, dx, dy, dz);
}
#endif

}  // namespace xmc
