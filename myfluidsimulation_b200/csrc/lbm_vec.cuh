// One cell's arithmetic and two cells' (Blackwell's paired FP32 instructions, or
// a pair of doubles), every operation with its rounding spelled out: the same
// expression gives the same bits whichever kernel it is compiled into.
#pragma once

#include "lbm_common.cuh"

namespace lbm {

// ---- scalar and paired FP32 arithmetic with identical rounding -------------
__device__ __forceinline__ float vadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vsplat(float s, float) { return s; }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 vsub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 vmul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 vsplat(float s, float2) { return make_float2(s, s); }
// FP64 (the reference form): one double, or a pair of doubles with the same
// interface as float2
struct D2 {
    double x, y;
};
__device__ __forceinline__ double vadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double vsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double vmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double vfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double vsplat(float s, double) { return s; }
__device__ __forceinline__ D2 vadd(D2 a, D2 b) { return {__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y)}; }
__device__ __forceinline__ D2 vsub(D2 a, D2 b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y)}; }
__device__ __forceinline__ D2 vmul(D2 a, D2 b) { return {__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)}; }
__device__ __forceinline__ D2 vfma(D2 a, D2 b, D2 c) { return {__fma_rn(a.x, b.x, c.x), __fma_rn(a.y, b.y, c.y)}; }
__device__ __forceinline__ D2 vsplat(float s, D2) { return {(double)s, (double)s}; }
__device__ __forceinline__ D2 vsplat(double s, D2) { return {s, s}; }
__device__ __forceinline__ double vsplat(double s, double) { return s; }
__device__ __forceinline__ D2 mulk(D2 x, float hi, float lo) { return {mulk(x.x, hi, lo), mulk(x.y, hi, lo)}; }

// -3 r where a = 3 r is at hand: a sign for one cell, a product for two
__device__ __forceinline__ float vneg3(float, float a) { return -a; }
__device__ __forceinline__ double vneg3(double, double a) { return -a; }
__device__ __forceinline__ float2 vneg3(float2 r, float2) { return vmul(vsplat(-3.0f, float2{}), r); }
__device__ __forceinline__ D2 vneg3(D2, D2 a) { return {-a.x, -a.y}; }
// a b - c, one rounding
__device__ __forceinline__ float vfms(float a, float b, float c) { return __fmaf_rn(a, b, -c); }
__device__ __forceinline__ float2 vfms(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, make_float2(-c.x, -c.y)); }
__device__ __forceinline__ double vfms(double a, double b, double c) { return __fma_rn(a, b, -c); }
__device__ __forceinline__ D2 vfms(D2 a, D2 b, D2 c) { return {__fma_rn(a.x, b.x, -c.x), __fma_rn(a.y, b.y, -c.y)}; }

// one aligned pair in shared memory
__device__ __forceinline__ void st_pair(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }
__device__ __forceinline__ void st_pair(double* p, D2 v) { *reinterpret_cast<double2*>(p) = make_double2(v.x, v.y); }
__device__ __forceinline__ float2 ld_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ D2 ld_pair(const double* p) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    return {v.x, v.y};
}
// 1/r where r > 0, else 0 (u = 0 for an empty cell, home.cu:258-262)
__device__ __forceinline__ float2 vrcp_pos(float2 r) {
    return make_float2(r.x > 0.f ? __frcp_rn(r.x) : 0.f, r.y > 0.f ? __frcp_rn(r.y) : 0.f);
}
__device__ __forceinline__ D2 vrcp_pos(D2 r) { return {r.x > 0.0 ? 1.0 / r.x : 0.0, r.y > 0.0 ? 1.0 / r.y : 0.0}; }

// scalar reciprocal with the same rule
__device__ __forceinline__ float vrcp_pos(float r) { return r > 0.f ? __frcp_rn(r) : 0.f; }
__device__ __forceinline__ double vrcp_pos(double r) { return r > 0.0 ? 1.0 / r : 0.0; }
// and without it
__device__ __forceinline__ float vrcp(float r) { return __frcp_rn(r); }
__device__ __forceinline__ double vrcp(double r) { return 1.0 / r; }

// ---- BGK on one cell (V = float, double) or two (V = float2, D2) -----------
template <class V>
struct CellV {
    V r, ux, uy, uz;
};

// Pre-collision moments with the velocity-shift force (legacy.cu:78-90).
// Opposite pairs are summed first: s = f_q + f_opp, d = f_q - f_opp.
// EMPTY: u = F where rho is not positive, as in the solvers; otherwise u = j / rho + F
// there too, which is what the adjoint differentiates (one cell only).
template <bool EMPTY = true, class V, class R>
__device__ __forceinline__ CellV<V> moments(const V (&f)[19], R fx, R fy, R fz) {
    // pairs with their positive member: (1,2) x, (3,4) y, (5,6) z, (7,10) +x+y,
    // (9,8) +x-y, (11,14) +x+z, (13,12) +x-z, (15,18) +y+z, (17,16) +y-z
    const V s12 = vadd(f[1], f[2]), d12 = vsub(f[1], f[2]);
    const V s34 = vadd(f[3], f[4]), d34 = vsub(f[3], f[4]);
    const V s56 = vadd(f[5], f[6]), d56 = vsub(f[5], f[6]);
    const V s7 = vadd(f[7], f[10]), d7 = vsub(f[7], f[10]);
    const V s9 = vadd(f[9], f[8]), d9 = vsub(f[9], f[8]);
    const V s11 = vadd(f[11], f[14]), d11 = vsub(f[11], f[14]);
    const V s13 = vadd(f[13], f[12]), d13 = vsub(f[13], f[12]);
    const V s15 = vadd(f[15], f[18]), d15 = vsub(f[15], f[18]);
    const V s17 = vadd(f[17], f[16]), d17 = vsub(f[17], f[16]);
    CellV<V> c;
    c.r = vadd(vadd(f[0], vadd(vadd(s12, s34), vadd(s56, s7))), vadd(vadd(vadd(s9, s11), vadd(s13, s15)), s17));
    const V jx = vadd(vadd(vadd(d12, d7), vadd(d9, d11)), d13);
    const V jy = vadd(vsub(vadd(d34, d7), d9), vadd(d15, d17));
    const V jz = vadd(vsub(vadd(d56, d11), d13), vsub(d15, d17));
    V inv = vrcp_pos(c.r);
    // (behind a test: taken unconditionally it costs the adjoint's reverse step 80 registers for 64)
    if constexpr (!EMPTY)
        if (!(c.r > V(0))) inv = vrcp(c.r);
    c.ux = vfma(jx, inv, vsplat(fx, V{}));
    c.uy = vfma(jy, inv, vsplat(fy, V{}));
    c.uz = vfma(jz, inv, vsplat(fz, V{}));
    return c;
}

// BGK collision f* = f + w (feq - f) for every direction, the equilibrium
// evaluated per opposite pair: feq_(+-) = w rho (1 - 1.5u^2 + 4.5 t^2) +- 3 w rho t.
// (The Hybrid's "HOME form" of hybrid.cu:148-152 is this with w = omega_shear.)
template <class V>
__device__ __forceinline__ void collide(V (&f)[19], const CellV<V>& c, V omega) {
    const V uu = vfma(c.uz, c.uz, vfma(c.ux, c.ux, vmul(c.uy, c.uy)));
    const V A = vfma(vsplat(-1.5f, V{}), uu, vsplat(1.0f, V{}));
    // w_q rho with the weights' own rounding compensated (mulk): no mass or momentum bias per step
    const V r0 = mulk(c.r, K3_HI, K3_LO), r1 = mulk(c.r, K18_HI, K18_LO), r2 = mulk(c.r, K36_HI, K36_LO);
    const V a1 = vmul(vsplat(3.0f, V{}), r1), a2 = vmul(vsplat(3.0f, V{}), r2);
    const V n1 = vneg3(r1, a1), n2 = vneg3(r2, a2);
    auto pair = [&](int qp, int qm, V t, V wr, V w3, V n3) {
        const V sym = vmul(wr, vfma(vmul(vsplat(4.5f, V{}), t), t, A));
        f[qp] = vfma(omega, vsub(vfma(w3, t, sym), f[qp]), f[qp]);
        f[qm] = vfma(omega, vsub(vfma(n3, t, sym), f[qm]), f[qm]);
    };
    f[0] = vfma(omega, vfms(r0, A, f[0]), f[0]);
    pair(1, 2, c.ux, r1, a1, n1);
    pair(3, 4, c.uy, r1, a1, n1);
    pair(5, 6, c.uz, r1, a1, n1);
    pair(7, 10, vadd(c.ux, c.uy), r2, a2, n2);
    pair(9, 8, vsub(c.ux, c.uy), r2, a2, n2);
    pair(11, 14, vadd(c.ux, c.uz), r2, a2, n2);
    pair(13, 12, vsub(c.ux, c.uz), r2, a2, n2);
    pair(15, 18, vadd(c.uy, c.uz), r2, a2, n2);
    pair(17, 16, vsub(c.uy, c.uz), r2, a2, n2);
}

}  // namespace lbm
