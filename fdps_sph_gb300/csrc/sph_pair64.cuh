// FP64 pair arithmetic shared by the device-resident passes (sph_pairs.cu) and the functor kernels
// (sph_batch64.cu).
//
// What bounds every FP64 pair kernel on this GPU is the FP64 pipe: one warp instruction per SM every 16
// cycles, about 1/40 of the FP32 rate, and an FP64 divide or square root costs 7.5 of them (measured with an
// operation loop: sqrt 150, divide 148, rsqrt 97 against 20 for a fused multiply-add).  So the pair terms are
// written for few FP64 instructions: square roots and reciprocals start from the hardware's approximate
// seeds (an MUFU instruction, off the FP64 pipe) and take one or two Newton / Householder steps
// (error below 2^-53 before the last rounding), constants are folded out of the sums, tests and clamps run on
// the integer pipe.
#pragma once

#include "sph_physics.cuh"

namespace sph {

// exponent field of x well inside the normal range and x positive: the seeds and the steps below neither
// overflow nor lose bits
__device__ __forceinline__ bool mid_range(double x) {
    return (unsigned)(__double2hiint(x) - 0x10000000) < 0x60000000u;
}

// 1 / x: seed y (relative error e below 2^-18), then y (1 + e + e^2) with e = 1 - x y
__device__ __forceinline__ double rcp64(double x) {
    if (!mid_range(x)) return 1.0 / x;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// r = sqrt(x) and y = 1 / sqrt(x) (y = 0 at x = 0), within 2 units of 2^-53 each: seed y0, e = 1 - x y0^2,
// both times (1 + e / 2 + 3 e^2 / 8)
__device__ __forceinline__ void sqrt_rsqrt64(double x, double &r, double &y) {
    const bool zero = ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;   // (-0 too)
    if (!zero && !mid_range(x)) {
        r = sqrt(x);
        y = 1.0 / r;
        return;
    }
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
    if (zero) y0 = 0.0;
    const double t = x * y0;
    const double e = fma(-t, y0, 1.0);
    const double ec = e * fma(0.375, e, 0.5);
    r = fma(t, ec, t);
    y = fma(y0, ec, y0);
}

// sqrt(x) with the last step on the exact residual x - r^2, so the result is the rounded root but for rare
// ties: the density's and the derivative's weights amplify its error
__device__ __forceinline__ double sqrt64(double x) {
    const bool zero = (__double2hiint(x) | __double2loint(x)) == 0;
    if (!zero && !mid_range(x)) return sqrt(x);
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(x));
    double h0 = __hiloint2double(__double2hiint(y0) - 0x00100000, __double2loint(y0));   // y0 / 2
    if (zero) y0 = h0 = 0.0;
    const double t = x * y0;
    const double e = fma(-t, h0, 0.5);
    const double r = fma(t, e, t), h = fma(h0, e, h0);
    return fma(fma(-r, r, x), h, r);
}

// 1 / H as hi + lo (lo: the remainder of hi): r hi alone would carry hi's rounding into every weight of the
// particle with the same sign
struct Inv64 {
    double hi, lo;
};
__device__ __forceinline__ Inv64 inv64(double H) {
    Inv64 v;
    v.hi = 1.0 / H;
    v.lo = fma(-H, v.hi, 1.0) * v.hi;
    return v;
}

// max(1 - s, 0) without an FP64 compare (a NaN stays a NaN or becomes 0; its product with the polynomial is a
// NaN either way, as with fmax)
__device__ __forceinline__ double kernel_q(double s) {
    const double p = 1.0 - s;
    return __double2hiint(p) < 0 ? 0.0 : p;
}

// CalcDensity's pair (force.h:9-23): m_j W / norm added to sum
__device__ __forceinline__ void dens_pair64(double dx, double dy, double dz, double mj, Inv64 invH, double &sum) {
    const double r = sqrt64(fma(dx, dx, fma(dy, dy, dz * dz)));
    const double s = fma(r, invH.hi, r * invH.lo), q = kernel_q(s);
    const double q2 = q * q, q4 = q2 * q2;
    sum = fma(mj, fma(s, fma(s, fma(s, 32.0, 25.0), 8.0), 1.0) * (q4 * q4), sum);
}

// CalcDerivative's pair (force.h:89-106), kernel constants left out: with g = r (1 + 7 s + 16 s^2) q^7 /
// (r H + 1e-6 h) (gradW = -22 norm / H g dr, kernel.h:22-34), D[0] += m g v.dr, D[1..3] += m g (v x dr),
// D[4] += m w, D[5] += m g r^2 with v = v_i - v_j
__device__ __forceinline__ void drvt_pair64(double dx, double dy, double dz, double vx, double vy, double vz, double mj,
                                            Inv64 invH, double H, double ceps, double D[6]) {
    const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
    const double r = sqrt64(r2);
    const double s = fma(r, invH.hi, r * invH.lo), q = kernel_q(s);
    const double q2 = q * q, q4 = q2 * q2, q7 = q4 * (q2 * q);
    const double w = fma(s, fma(s, fma(s, 32.0, 25.0), 8.0), 1.0) * (q7 * q);
    const double mg = mj * ((r * fma(s, fma(s, 16.0, 7.0), 1.0)) * (q7 * rcp64(fma(r, H, ceps))));
    D[0] = fma(mg, fma(vx, dx, fma(vy, dy, vz * dz)), D[0]);
    D[1] = fma(mg, fma(vy, dz, -(vz * dy)), D[1]);
    D[2] = fma(mg, fma(vz, dx, -(vx * dz)), D[2]);
    D[3] = fma(mg, fma(vx, dy, -(vy * dx)), D[3]);
    D[4] = fma(mj, w, D[4]);
    D[5] = fma(mg, r2, D[5]);
}

// a particle's constants for the hydro pair: qn = -22 norm / H, H, 1 / H, 1e-6 h, A = f P / rho^2, f, rho,
// b = -Bal / 4, c_s
struct Hydro64 {
    double qn, H, invH, ceps, A, f, rho, b, c;
};

__device__ __forceinline__ Hydro64 hydro64_consts(double h, double rho, double pres, double gradh, double bal,
                                                  double snds) {
    Hydro64 k;
    k.H = SUPPORT * h;
    k.invH = rcp64(k.H);
    k.qn = (-22.0 * WNORM / PI_D) * ((k.invH * k.invH) * (k.invH * k.invH));
    k.ceps = 1.0e-6 * h;
    k.A = gradh * pres * rcp64(rho * rho);
    k.f = gradh;
    k.rho = rho;
    k.b = -0.25 * bal;
    k.c = snds;
    return k;
}

// dW/dr / r of one side: qn r (1 + 7 s + 16 s^2) q^7 / (r H + 1e-6 h)
__device__ __forceinline__ double hydro_gf64(double r, double qn, double H, double invH, double ceps) {
    const double s = r * invH, q = kernel_q(s);
    const double q2 = q * q, q7 = q2 * q2 * (q2 * q);
    return (qn * r) * fma(s, fma(s, 16.0, 7.0), 1.0) * (q7 * rcp64(fma(r, H, ceps)));
}

// CalcHydroForce's pair (force.h:113-147): D[0..2] -= acceleration terms, D[3] += twice the du/dt term, vmax
// the signal velocity.  AV / 2 = u = (-Bal_i/4 - Bal_j/4) v_sig w / (rho_i + rho_j).
__device__ __forceinline__ void hydro_pair64(double dx, double dy, double dz, double vx, double vy, double vz, double mj,
                                             const Hydro64 &I, const Hydro64 &J, double D[4], double &vmax) {
    double r, y;
    sqrt_rsqrt64(fma(dx, dx, fma(dy, dy, dz * dz)), r, y);
    const double dvdr = fma(vx, dx, fma(vy, dy, vz * dz));
    const double w = dvdr < 0 ? dvdr * y : 0.0;
    const double vsig = fma(-3.0, w, I.c + J.c);
    vmax = fmax(vmax, vsig);
    const double u = (I.b + J.b) * (vsig * w) * rcp64(I.rho + J.rho);
    const double gi = hydro_gf64(r, I.qn, I.H, I.invH, I.ceps), gj = hydro_gf64(r, J.qn, J.H, J.invH, J.ceps);
    const double coef = mj * fma(gi, fma(u, I.f, I.A), gj * fma(u, J.f, J.A));
    D[0] = fma(-coef, dx, D[0]);
    D[1] = fma(-coef, dy, D[1]);
    D[2] = fma(-coef, dz, D[2]);
    D[3] = fma(mj * (I.A + u) * fma(gi, I.f, gj * J.f), dvdr, D[3]);
}

// CalcGravityForce's pair (force.h:154-168): dx.. = x_i - x_j, gm = G m_j
__device__ __forceinline__ void grav_pair64(double dx, double dy, double dz, double eps2, double gm, double A[4]) {
    const double y = rsqrt(fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2))));
    const double gmr = gm * y;
    const double gmr3 = gmr * (y * y);
    A[0] = fma(-gmr3, dx, A[0]);
    A[1] = fma(-gmr3, dy, A[1]);
    A[2] = fma(-gmr3, dz, A[2]);
    A[3] -= gmr;
}

__device__ __forceinline__ double warp_sum64(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// four sums over the warp with 6 additions a lane instead of 20: the lanes split the values between them as
// the distance halves.  Returns the sum of v[lane >> 3] in every lane.
__device__ __forceinline__ double warp_sum64x4(const double v[4]) {
    const int lane = threadIdx.x & 31;
    const bool up = lane & 16;
    double a = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
    double b = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
    const bool up2 = lane & 8;
    a = (up2 ? b : a) + __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

}  // namespace sph
