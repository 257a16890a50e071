// interact.cuh -- one sink against one staged source record, FP32.
//
// The arithmetic is the reference's multipole recurrence
// (do_gravph_avx8, nln/do_grav_avx8.c:1779-1904; pH, nln/pgrav.cu:49-213):
// with d = sink - source and the normalised traceless moments q_l / R^l,
// order l contributes
//     eq  = t_l * (q_l contracted with d^(l-1)),   t_l = -(2l-1)!! R^l / r^(2l+1)
//     phi += c_l eq.d,          c_l = 1/2, 1/3, 1/4
//     a   += d (2l+1) c_l eq.d / r^2 - eq
// The constant -(2l-1)!! R^l is folded into the moments once per source when
// a tile is staged (stage_* below), so the inner loop only multiplies by
// powers of 1/r.  Staged record layouts (floats, 16-byte aligned):
//   P (points, 4):      x y z m
//   Q (quadrupole, 12): x y z m | Qxx Qxy Qyy Qxz Qyz Qzz | - -
//   H (order 4, 32):    x y z m | Qxx Qxy Qyy Qxz Qyz Qzz | O[7] Osum1 Osum2 |
//                       X[9] Xsum | - - -
// with Q = -3 R^2 q2, O = -15 R^3 q3, X = -105 R^4 q4 and the sums
// Qzz = -(Qxx+Qyy), Osum1 = Oxxx+Oxyy, Osum2 = Oxxy+Oyyy, Xsum = Xxyyy+Xxxxy.
#pragma once

#include "common.cuh"

constexpr int REC_P = 4, REC_Q = 12, REC_H = 32;

struct Acc4 {
    float ax, ay, az, phi;
};

// Softening laws of the monopole term.
enum Soft { SOFT_PLUMMER = 0, SOFT_NONE = 1, SOFT_MASKED = 2, SOFT_K1 = 3 };

// Staging: raw fields -> folded record.  q2[5], q3[7], q4[9] in the
// reference order (qxx qxy qyy qxz qyz; qxxx qxxy qxyy qyyy qxxz qxyz qyyz;
// qxxxx qxxxy qxxyy qxyyy qyyyy qxxxz qxxyz qxyyz qyyyz).
__device__ __forceinline__ void stage_quad(float *o, float R, const float *q2) {
    const float c2 = -3.0f * R * R;
    float Qxx = c2 * q2[0], Qxy = c2 * q2[1], Qyy = c2 * q2[2], Qxz = c2 * q2[3],
          Qyz = c2 * q2[4];
    o[4] = Qxx;
    o[5] = Qxy;
    o[6] = Qyy;
    o[7] = Qxz;
    o[8] = Qyz;
    o[9] = -(Qxx + Qyy);
    o[10] = 0.0f;
    o[11] = 0.0f;
}

__device__ __forceinline__ void stage_hexa(float *o, float R, const float *q3, const float *q4) {
    const float c3 = -15.0f * R * R * R;
    const float c4 = -105.0f * R * R * R * R;
    float O[7], X[9];
#pragma unroll
    for (int k = 0; k < 7; k++) O[k] = c3 * q3[k];
#pragma unroll
    for (int k = 0; k < 9; k++) X[k] = c4 * q4[k];
#pragma unroll
    for (int k = 0; k < 7; k++) o[12 + k] = O[k];
    o[19] = O[0] + O[2];  // Oxxx + Oxyy
    o[20] = O[1] + O[3];  // Oxxy + Oyyy
#pragma unroll
    for (int k = 0; k < 9; k++) o[21 + k] = X[k];
    o[30] = X[3] + X[1];  // Xxyyy + Xxxxy
    o[31] = 0.0f;
}

// Monopole term: its potential pm and radial coefficient kr (the term adds
// pm to phi and d * kr to the acceleration), and ri = 1/r, ri2 for the
// higher orders.
template <int SOFT>
__device__ __forceinline__ void mono_terms(float x, float y, float z, float m, float e, float &pm,
                                           float &kr, float &ri, float &ri2) {
    if (SOFT == SOFT_PLUMMER || SOFT == SOFT_NONE) {
        // nln/do_grav_avx8.c:2181-2210, e = eps^2
        float r2 = fmaf(x, x, fmaf(y, y, SOFT == SOFT_PLUMMER ? fmaf(z, z, e) : z * z));
        ri = rsqrt_fast(r2);
        ri2 = ri * ri;
        float mri = m * ri;
        pm = -mri;
        kr = -mri * ri2;
    } else if (SOFT == SOFT_MASKED) {
        // do_grav_avx8: pairs closer than e contribute nothing (nln/do_grav_avx8.c:978-990)
        float r2 = fmaf(x, x, fmaf(y, y, z * z));
        ri = (r2 >= e * e) ? rsqrt_fast(r2) : 0.0f;
        ri2 = ri * ri;
        float mri = m * ri;
        pm = -mri;
        kr = -mri * ri2;
    } else {
        // Dehnen K1 inside r < eps, e = 1/eps (nln/do_grav_avx8.c:1013-1045, nln/pgrav.cu:441-461)
        float r2 = fmaf(x, x, fmaf(y, y, z * z));
        float pf, af;
        if (r2 * e * e < 1.0f) {
            float u2 = fmaf(r2, e * e, -1.0f);
            pf = fmaf(fmaf(fmaf(-45.0f / 32.0f, u2, 3.0f / 8.0f), u2, -0.5f), u2, 1.0f) * e;
            af = fmaf(fmaf(135.0f / 16.0f, u2, -1.5f), u2, 1.0f) * e * e * e;
            ri = 0.0f;
        } else {
            ri = rsqrt_fast(r2);
            pf = ri;
            af = ri * ri * ri;
        }
        ri2 = ri * ri;
        pm = -m * pf;
        kr = -m * af;
    }
}

template <int SOFT>
__device__ __forceinline__ void mono(float x, float y, float z, float m, float e, Acc4 &a,
                                     float &ri, float &ri2) {
    float pm, kr;
    mono_terms<SOFT>(x, y, z, m, e, pm, kr, ri, ri2);
    a.phi += pm;
    a.ax = fmaf(x, kr, a.ax);
    a.ay = fmaf(y, kr, a.ay);
    a.az = fmaf(z, kr, a.az);
}

// Quadrupole contraction: Q.d and d.Q.d.
__device__ __forceinline__ void quad_vec(float x, float y, float z, const float *__restrict__ r,
                                         float &Qx, float &Qy, float &Qz, float &dQd) {
    const float4 q0 = *reinterpret_cast<const float4 *>(r + 4);  // Qxx Qxy Qyy Qxz
    const float2 q1 = *reinterpret_cast<const float2 *>(r + 8);  // Qyz Qzz
    Qx = fmaf(q0.x, x, fmaf(q0.y, y, q0.w * z));
    Qy = fmaf(q0.y, x, fmaf(q0.z, y, q1.x * z));
    Qz = fmaf(q0.w, x, fmaf(q1.x, y, q1.y * z));
    dQd = fmaf(x, Qx, fmaf(y, Qy, z * Qz));
}

// Octupole and hexadecapole contractions with d^2 and d^3 (e, h) and their
// products with d (nln/do_grav_avx8.c:1853-1898), traceless moments.
__device__ __forceinline__ void hexa_vec(float x, float y, float z, const float *__restrict__ r,
                                         float e[3], float &d3, float h[3], float &d4) {
    const float4 o0 = *reinterpret_cast<const float4 *>(r + 12);  // Oxxx Oxxy Oxyy Oyyy
    const float4 o1 = *reinterpret_cast<const float4 *>(r + 16);  // Oxxz Oxyz Oyyz S1
    const float4 o2 = *reinterpret_cast<const float4 *>(r + 20);  // S2 Xxxxx Xxxxy Xxxyy
    const float4 x0 = *reinterpret_cast<const float4 *>(r + 24);  // Xxyyy Xyyyy Xxxxz Xxxyz
    const float4 x1 = *reinterpret_cast<const float4 *>(r + 28);  // Xxyyz Xyyyz XS -
    const float third = 1.0f / 3.0f;
    float xx = 0.5f * x * x, yy = 0.5f * y * y, zz = 0.5f * z * z;
    float xy = x * y, xz = x * z, yz = y * z;
    float xxx = x * fmaf(xx, third, -zz);
    float xxz = z * fmaf(zz, -third, xx);
    float yyy = y * fmaf(yy, third, -zz);
    float yyz = z * fmaf(zz, -third, yy);
    xx -= zz;
    yy -= zz;
    e[0] = fmaf(o0.x, xx, fmaf(o0.z, yy, fmaf(o0.y, xy, fmaf(o1.x, xz, o1.y * yz))));
    e[1] = fmaf(o0.z, xy, fmaf(o0.y, xx, fmaf(o0.w, yy, fmaf(o1.z, yz, o1.y * xz))));
    e[2] = fmaf(-o1.w, xz, fmaf(-o2.x, yz, fmaf(o1.x, xx, fmaf(o1.z, yy, o1.y * xy))));
    d3 = fmaf(x, e[0], fmaf(y, e[1], z * e[2]));
    float xxy = y * xx, xyy = x * yy, xyz = xy * z;
    // X order: xxxx(o2.y) xxxy(o2.z) xxyy(o2.w) xyyy(x0.x) yyyy(x0.y) xxxz(x0.z) xxyz(x0.w)
    //          xyyz(x1.x) yyyz(x1.y), XS = xyyy + xxxy (x1.z)
    h[0] = fmaf(o2.y, xxx, fmaf(x0.x, yyy, fmaf(o2.z, xxy, fmaf(x0.z, xxz,
           fmaf(o2.w, xyy, fmaf(x0.w, xyz, x1.x * yyz))))));
    h[1] = fmaf(x0.x, xyy, fmaf(o2.z, xxx, fmaf(x0.y, yyy, fmaf(x1.y, yyz,
           fmaf(o2.w, xxy, fmaf(x0.w, xxz, x1.x * xyz))))));
    h[2] = fmaf(-o2.y, xxz, fmaf(-x1.z, xyz, fmaf(-x0.y, yyz, fmaf(x0.z, xxx,
           fmaf(x1.y, yyy, fmaf(-o2.w, xxz + yyz, fmaf(x0.w, xxy, x1.x * xyy)))))));
    d4 = fmaf(x, h[0], fmaf(y, h[1], z * h[2]));
}

// One staged record of order ORDER (0, 2, 4) against a sink at (sx, sy, sz).
// The orders' terms are summed before they reach the accumulators: with
// eq_l = r^-(2l+1) (moment contracted with d^(l-1)),
//     phi += pm + qsh eq_2.d + eq_3.d/3 + eq_4.d/4
//     a   += d (kr + r^-2 (5 qsh' eq_2.d + 7/3 eq_3.d + 9/4 eq_4.d)) - (eq_2 + eq_3 + eq_4)
// (qsh' = 1/2: the acceleration does not take the potential's sign
// convention) and eq_2 + eq_3 + eq_4 = r^-5 (Q.d + r^-2 (e + r^-2 h)).
template <int ORDER, int SOFT>
__device__ __forceinline__ void interact(const float *__restrict__ r, float sx, float sy,
                                         float sz, float e, float qsh, Acc4 &a) {
    const float4 p = *reinterpret_cast<const float4 *>(r);
    float x = sx - p.x, y = sy - p.y, z = sz - p.z;
    float ri, ri2;
    if (ORDER == 0) {
        mono<SOFT>(x, y, z, p.w, e, a, ri, ri2);
        return;
    }
    float pm, kr;
    mono_terms<SOFT>(x, y, z, p.w, e, pm, kr, ri, ri2);
    float Qx, Qy, Qz, dQd;
    quad_vec(x, y, z, r, Qx, Qy, Qz, dQd);
    const float ri5 = ri * ri2 * ri2;
    const float eqd2 = ri5 * dQd;
    float tx = Qx, ty = Qy, tz = Qz, K;
    if (ORDER >= 4) {
        float ev[3], hv[3], d3, d4;
        hexa_vec(x, y, z, r, ev, d3, hv, d4);
        const float ri7 = ri5 * ri2, ri9 = ri7 * ri2;
        const float eqd3 = ri7 * d3, eqd4 = ri9 * d4;
        a.phi = fmaf(0.25f, eqd4, fmaf(1.0f / 3.0f, eqd3, fmaf(qsh, eqd2, a.phi + pm)));
        K = fmaf(ri2, fmaf(2.25f, eqd4, fmaf(7.0f / 3.0f, eqd3, 2.5f * eqd2)), kr);
        tx = fmaf(ri2, fmaf(ri2, hv[0], ev[0]), Qx);
        ty = fmaf(ri2, fmaf(ri2, hv[1], ev[1]), Qy);
        tz = fmaf(ri2, fmaf(ri2, hv[2], ev[2]), Qz);
    } else {
        a.phi = fmaf(qsh, eqd2, a.phi + pm);
        K = fmaf(2.5f * ri2, eqd2, kr);
    }
    a.ax = fmaf(x, K, fmaf(-ri5, tx, a.ax));
    a.ay = fmaf(y, K, fmaf(-ri5, ty, a.ay));
    a.az = fmaf(z, K, fmaf(-ri5, tz, a.az));
}

// ---------------------------------------------------------------- record pairs
//
// Two source records against one sink with Blackwell's paired FP32
// instructions (fma/add/mul .f32x2): the .x halves belong to one record, the
// .y halves to the other.  Both records stay in this lane's registers while
// the warp walks its group's sinks, whose negated offsets come in as splat
// pairs (nsx, nsx).  Everything works in v = source - sink = -d.
//
// What bounds them is the register file, not the FMA pipe: on a B200 a
// paired FMA with three distinct operands takes 3.05 to 3.3 cycles a warp, by
// the registers it gets (45 to 49 of 74 TFLOP/s), with two 2.05; a scalar one
// 1.1 to 1.5, and 1.04.  So the forms below count operand reads, not only
// operations.
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 splat2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 rsqrt2(float2 a) { return f2(rsqrt_fast(a.x), rsqrt_fast(a.y)); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Running sums of one sink over this lane's records (nphi: -phi).
struct Sum2 {
    float2 ax, ay, az, nphi;
    // (ax, ay, az, phi) of both halves together
    __device__ __forceinline__ float4 total() const {
        return make_float4(ax.x + ax.y, ay.x + ay.y, az.x + az.y, -(nphi.x + nphi.y));
    }
};

struct MonoPair {
    float2 x, y, z, m;
};

// Monopoles, the arithmetic of mono<SOFT_PLUMMER>; FIRST starts the sums.
template <bool FIRST>
__device__ __forceinline__ void mono_pair(const MonoPair &r, float2 nsx, float2 nsy, float2 nsz,
                                          float2 e2, Sum2 &A) {
    const float2 x = add2(r.x, nsx), y = add2(r.y, nsy), z = add2(r.z, nsz);
    const float2 ri = rsqrt2(fma2(x, x, fma2(y, y, fma2(z, z, e2))));
    const float2 mri = mul2(r.m, ri), mri3 = mul2(mri, mul2(ri, ri));
    if (FIRST) {
        A.nphi = mri;
        A.ax = mul2(x, mri3);
        A.ay = mul2(y, mri3);
        A.az = mul2(z, mri3);
    } else {
        A.nphi = add2(A.nphi, mri);
        A.ax = fma2(x, mri3, A.ax);
        A.ay = fma2(y, mri3, A.ay);
        A.az = fma2(z, mri3, A.az);
    }
}

// Quadrupole cells: q = Qxx Qxy Qyy Qxz Qyz Qzz with Q = -3 R^2 q2.  With
// U = Q.v:  a = v (m r^-3 - 5/2 r^-2 eq_2.d) + r^-5 U,  -phi = m/r - qsh eq_2.d.
struct QuadPair {
    float2 x, y, z, m, q[6];
};

template <bool FIRST>
__device__ __forceinline__ void cell_pair(const QuadPair &r, float2 nsx, float2 nsy, float2 nsz,
                                          float2 e2, float qsh, Sum2 &A) {
    const float2 x = add2(r.x, nsx), y = add2(r.y, nsy), z = add2(r.z, nsz);
    const float2 ri = rsqrt2(fma2(x, x, fma2(y, y, fma2(z, z, e2))));
    const float2 ri2 = mul2(ri, ri), ri3 = mul2(ri, ri2), ri5 = mul2(ri3, ri2);
    const float2 Ux = fma2(r.q[0], x, fma2(r.q[1], y, mul2(r.q[3], z)));
    const float2 Uy = fma2(r.q[1], x, fma2(r.q[2], y, mul2(r.q[4], z)));
    const float2 Uz = fma2(r.q[3], x, fma2(r.q[4], y, mul2(r.q[5], z)));
    const float2 eqd = mul2(ri5, fma2(x, Ux, fma2(y, Uy, mul2(z, Uz))));
    A.nphi = fma2(r.m, ri, FIRST ? mul2(splat2(-qsh), eqd) : fma2(splat2(-qsh), eqd, A.nphi));
    const float2 K = fma2(mul2(splat2(-2.5f), ri2), eqd, mul2(r.m, ri3));
    A.ax = fma2(x, K, FIRST ? mul2(ri5, Ux) : fma2(ri5, Ux, A.ax));
    A.ay = fma2(y, K, FIRST ? mul2(ri5, Uy) : fma2(ri5, Uy, A.ay));
    A.az = fma2(z, K, FIRST ? mul2(ri5, Uz) : fma2(ri5, Uz, A.az));
}

// Order-4 cells.  Staged per record: q = Q (xx xy yy xz yz), o = -O/2 (the
// seven of stage_hexa) and the two sums (Oxxx+Oxyy)/2, (Oxxy+Oyyy)/2, h = X/6
// (nine) and -(Xxxxx+Xxxyy)/6, -(Xyyyy+Xxxyy)/6, -(Xxxxy+Xxyyy)/6 (the xxzz,
// yyzz and xyzz components).  With the harmonic second-degree monomials
// s = (x^2 - z^2, y^2 - z^2, 2xy, 2xz, 2yz):
//   e = o : s          v.e = d3     (octupole vector)
//   M = h : s          M : s = d4   (hexadecapole as a traceless matrix)
//   U = (Q + r^-4 M).v + r^-2 e,    v.U = T = d2 + r^-2 d3 + r^-4 d4
// and with t = r^-2 (d3 + 3/2 r^-2 d4), P = T - t/3 (twice the multipole
// potential over r^-5):
//   -phi = m/r - r^-5 P / 2,   a = v (m r^-3 - r^-7 (4 T + P) / 2) + r^-5 U.
// Contracting the hexadecapole to a matrix once folds its 3x3 product into
// the quadrupole's: 105 operations against 111 for separate order-2, 3 and 4
// vectors, 274 against 285 cycles a pair by the operand reads.
struct HexaPair {
    float2 x, y, z, m, q[5], o[9], h[12];
};

__device__ __forceinline__ float2 dot5(const float2 *c, const float2 *s) {
    return fma2(c[0], s[0], fma2(c[1], s[1], fma2(c[2], s[2], fma2(c[3], s[3], mul2(c[4], s[4])))));
}

// PHYS: the physical potential (qsh = 1/2); otherwise the quadrupole's enters
// with qsh, the other sign convention.
template <bool PHYS>
__device__ __forceinline__ void cell_pair(const HexaPair &r, float2 nsx, float2 nsy, float2 nsz,
                                          float2 e2, float qsh, Sum2 &A) {
    const float2 x = add2(r.x, nsx), y = add2(r.y, nsy), z = add2(r.z, nsz);
    const float2 ri = rsqrt2(fma2(x, x, fma2(y, y, fma2(z, z, e2))));
    const float2 nzz = neg2(mul2(z, z)), x2 = add2(x, x), y2 = add2(y, y);
    const float2 s[5] = {fma2(x, x, nzz), fma2(y, y, nzz), mul2(x2, y), mul2(x2, z), mul2(y2, z)};
    // o: xxx xxy xyy yyy xxz xyz yyz, sums; h: xxxx xxxy xxyy xyyy yyyy xxxz xxyz xyyz yyyz,
    // xxzz yyzz xyzz
    const float2 *o = r.o, *h = r.h;
    const float2 c0[5] = {o[0], o[2], o[1], o[4], o[5]}, c1[5] = {o[1], o[3], o[2], o[5], o[6]},
                 c2[5] = {o[4], o[6], o[5], o[7], o[8]};
    const float2 ex = dot5(c0, s), ey = dot5(c1, s), ez = dot5(c2, s);
    const float2 mxx[5] = {h[0], h[2], h[1], h[5], h[6]}, mxy[5] = {h[1], h[3], h[2], h[6], h[7]},
                 myy[5] = {h[2], h[4], h[3], h[7], h[8]}, mxz[5] = {h[5], h[7], h[6], h[9], h[11]},
                 myz[5] = {h[6], h[8], h[7], h[11], h[10]};
    const float2 M[5] = {dot5(mxx, s), dot5(myy, s), dot5(mxy, s), dot5(mxz, s), dot5(myz, s)};
    const float2 ri2 = mul2(ri, ri), ri4 = mul2(ri2, ri2), ri5 = mul2(ri4, ri);
    const float2 mri = mul2(r.m, ri);
    const float2 d3 = fma2(x, ex, fma2(y, ey, mul2(z, ez)));
    const float2 d4 = dot5(M, s);
    const float2 qxx = fma2(ri4, M[0], r.q[0]), qyy = fma2(ri4, M[1], r.q[2]),
                 qxy = fma2(ri4, M[2], r.q[1]), qxz = fma2(ri4, M[3], r.q[3]),
                 qyz = fma2(ri4, M[4], r.q[4]);
    float2 Ux = fma2(qxx, x, fma2(qxy, y, mul2(qxz, z)));
    float2 Uy = fma2(qxy, x, fma2(qyy, y, mul2(qyz, z)));
    float2 Uz = fma2(qxz, x, fma2(qyz, y, mul2(neg2(add2(qxx, qyy)), z)));
    Ux = fma2(ri2, ex, Ux);
    Uy = fma2(ri2, ey, Uy);
    Uz = fma2(ri2, ez, Uz);
    const float2 T = fma2(x, Ux, fma2(y, Uy, mul2(z, Uz)));
    const float2 q1 = mul2(ri2, d4);
    const float2 t = mul2(ri2, fma2(splat2(1.5f), q1, d3));
    float2 P = fma2(splat2(-1.f / 3.f), t, T);
    const float2 c = fma2(splat2(4.f), T, P);
    if (!PHYS) {
        const float2 d2 = fma2(neg2(ri2), add2(d3, q1), T);
        P = fma2(splat2(2.f * qsh - 1.f), d2, P);
    }
    const float2 nri5h = mul2(splat2(-0.5f), ri5);
    A.nphi = fma2(nri5h, P, mri);
    const float2 K = fma2(mul2(nri5h, c), ri2, mul2(mri, ri2));
    A.ax = fma2(x, K, mul2(ri5, Ux));
    A.ay = fma2(y, K, mul2(ri5, Uy));
    A.az = fma2(z, K, mul2(ri5, Uz));
}
