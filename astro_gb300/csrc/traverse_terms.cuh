// Interaction terms shared by the traversal kernels (traverse.cu,
// traverse_group.cu): the fast 1/sqrt, the cell and particle terms, the
// far-node expansion and compensated accumulators.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace astro {

// The fast traversal's 1/sqrt: a single rsqrt.approx.ftz operation. It is
// used only where the argument is a normal float (r^2 >= eps^2 >= FLT_MIN);
// there it returns what rsqrtf() returns, without the fix-up rsqrtf() wraps
// around the same operation for subnormal arguments.
constexpr float kFltMin = 1.17549435e-38f;
__device__ __forceinline__ float rsqrt_ftz(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Interaction terms of the PHYSICAL preset (G = g):
//   particle / monopole:  t = G m d / (r^2 + eps^2)^(3/2)
//   quadrupole addition:  t += G [ 5/2 (d.Qd) d / r^7 - Qd / r^5 ]
// with d the displacement towards the source and Q traceless
// (Qzz = -Qxx - Qyy). kExact rounds every operation separately, in the
// order of the CPU restatement; otherwise rsqrt and FMAs are used.
template <bool kExact>
__device__ __forceinline__ void cell_term(float dx, float dy, float dz, float r2t, float m,
                                          bool quad, float4 q, float qyz, float g, float eps2,
                                          float& tx, float& ty, float& tz) {
    if (kExact) {
        const float r2 = __fadd_rn(r2t, eps2);
        const float inv = __fdiv_rn(1.0f, __fsqrt_rn(r2));
        const float inv2 = __fmul_rn(inv, inv);
        const float inv3 = __fmul_rn(inv2, inv);
        const float sc = __fmul_rn(__fmul_rn(g, m), inv3);
        tx = __fmul_rn(dx, sc);
        ty = __fmul_rn(dy, sc);
        tz = __fmul_rn(dz, sc);
        if (quad) {
            const float inv5 = __fmul_rn(inv3, inv2), inv7 = __fmul_rn(inv5, inv2);
            const float qzz = -__fadd_rn(q.x, q.y);
            const float qx = __fadd_rn(__fadd_rn(__fmul_rn(q.x, dx), __fmul_rn(q.z, dy)), __fmul_rn(q.w, dz));
            const float qy = __fadd_rn(__fadd_rn(__fmul_rn(q.z, dx), __fmul_rn(q.y, dy)), __fmul_rn(qyz, dz));
            const float qz = __fadd_rn(__fadd_rn(__fmul_rn(q.w, dx), __fmul_rn(qyz, dy)), __fmul_rn(qzz, dz));
            const float dqd = __fadd_rn(__fadd_rn(__fmul_rn(dx, qx), __fmul_rn(dy, qy)), __fmul_rn(dz, qz));
            const float w = __fmul_rn(__fmul_rn(2.5f, dqd), inv7);
            tx = __fadd_rn(tx, __fmul_rn(g, __fsub_rn(__fmul_rn(w, dx), __fmul_rn(qx, inv5))));
            ty = __fadd_rn(ty, __fmul_rn(g, __fsub_rn(__fmul_rn(w, dy), __fmul_rn(qy, inv5))));
            tz = __fadd_rn(tz, __fmul_rn(g, __fsub_rn(__fmul_rn(w, dz), __fmul_rn(qz, inv5))));
        }
    } else {
        const float inv = rsqrtf(r2t + eps2);
        const float inv2 = inv * inv;
        const float inv3 = inv2 * inv;
        const float sc = g * m * inv3;
        tx = dx * sc;
        ty = dy * sc;
        tz = dz * sc;
        if (quad) {
            const float inv5 = inv3 * inv2, inv7 = inv5 * inv2;
            const float qzz = -(q.x + q.y);
            const float qx = fmaf(q.x, dx, fmaf(q.z, dy, q.w * dz));
            const float qy = fmaf(q.z, dx, fmaf(q.y, dy, qyz * dz));
            const float qz = fmaf(q.w, dx, fmaf(qyz, dy, qzz * dz));
            const float dqd = fmaf(dx, qx, fmaf(dy, qy, dz * qz));
            const float w = 2.5f * dqd * inv7;
            const float gi5 = g * inv5, gw = g * w;
            tx = fmaf(gw, dx, fmaf(-gi5, qx, tx));
            ty = fmaf(gw, dy, fmaf(-gi5, qy, ty));
            tz = fmaf(gw, dz, fmaf(-gi5, qz, tz));
        }
    }
}

template <bool kExact>
__device__ __forceinline__ void particle_term(float dx, float dy, float dz, float m, float g,
                                              float eps2, float& tx, float& ty, float& tz) {
    if (kExact) {
        const float r2t =
            __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
        cell_term<true>(dx, dy, dz, r2t, m, false, make_float4(0.f, 0.f, 0.f, 0.f), 0.f, g, eps2,
                        tx, ty, tz);
    } else {
        const float inv = rsqrtf(fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, eps2))));
        const float sc = g * m * (inv * inv * inv);
        tx = dx * sc;
        ty = dy * sc;
        tz = dz * sc;
    }
}

// ---------------------------------------------------------- far nodes ----
// The field of an accepted node at d = D - rho, D = com - group centre, to
// second order in the offset rho (the same terms as cell_term, without G):
//   a_i(D - rho) = a_i - J_ij rho_j + 1/2 H_ijk rho_j rho_k
// With R = (|D|^2 + eps^2)^(-1/2), q = QD, s = D.QD:
//   a_i   = al D_i - R^5 q_i
//   J_ij  = ga (q_i D_j + q_j D_i) - be D_i D_j - R^5 Q_ij + al [i=j]
//   H_ijk = nu D_i D_j D_k + ka S(qDD) + ga (S(QD) + S(q delta)) - be S(delta D)
// al = m R^3 + 5/2 s R^7, be = 3 m R^5 + 35/2 s R^9, ga = 5 R^7,
// ka = -35 R^9, nu = 15 m R^7 + 315/2 s R^11; S(.) sums the three distinct
// placements of the indices. Coefficients: a {x, y, z}, J {xx, yy, zz, xy,
// xz, yz}, H {xxx, yyy, zzz, xxy, xxz, xyy, yyz, xzz, yzz, xyz}. The exact
// form rounds every product and sum separately in the CPU restatement's
// order (fma(a, b, c) there is a * b + c); the fast form uses FMAs and rsqrt.
constexpr int kFarCoefs = 19;

template <bool kExact>
__device__ __forceinline__ float xmul(float a, float b) { return kExact ? __fmul_rn(a, b) : a * b; }
template <bool kExact>
__device__ __forceinline__ float xadd(float a, float b) { return kExact ? __fadd_rn(a, b) : a + b; }
template <bool kExact>
__device__ __forceinline__ float xfma(float a, float b, float c) {
    return kExact ? __fadd_rn(__fmul_rn(a, b), c) : fmaf(a, b, c);
}

struct FarTerms {
    float D[3], qv[3], Q[3][3], R5, al, be, ga, ka, nu;
};

template <int i, int j>
__device__ __forceinline__ float far_j(const FarTerms& f) {
    float v = xfma<true>(f.ga, xfma<true>(f.qv[i], f.D[j], __fmul_rn(f.qv[j], f.D[i])),
                         -xfma<true>(f.be, __fmul_rn(f.D[i], f.D[j]), __fmul_rn(f.R5, f.Q[i][j])));
    if (i == j) v = __fadd_rn(v, f.al);
    return v;
}

template <int i, int j, int k>
__device__ __forceinline__ float far_h(const FarTerms& f) {
    const float dij = __fmul_rn(f.D[i], f.D[j]);
    const float sqdd =
        xfma<true>(f.qv[i], __fmul_rn(f.D[j], f.D[k]),
                   xfma<true>(f.qv[j], __fmul_rn(f.D[i], f.D[k]), __fmul_rn(f.qv[k], dij)));
    const float sqd = xfma<true>(f.Q[i][j], f.D[k],
                                 xfma<true>(f.Q[i][k], f.D[j], __fmul_rn(f.Q[j][k], f.D[i])));
    const float ddd = __fmul_rn(dij, f.D[k]);
    // The restatement multiplies by the 0/1 Kronecker factors.
    constexpr float cij = i == j ? 1.f : 0.f, cik = i == k ? 1.f : 0.f, cjk = j == k ? 1.f : 0.f;
    const float sqdel = xfma<true>(cjk, f.qv[i], xfma<true>(cik, f.qv[j], __fmul_rn(cij, f.qv[k])));
    const float sdel = xfma<true>(cij, f.D[k], xfma<true>(cik, f.D[j], __fmul_rn(cjk, f.D[i])));
    return xfma<true>(f.nu, ddd,
                      xfma<true>(f.ka, sqdd,
                                 xfma<true>(f.ga, __fadd_rn(sqd, sqdel), -__fmul_rn(f.be, sdel))));
}

// Adds the far-node coefficients of a node (centre of mass and mass cm,
// quadrupole {Qxx, Qyy, Qxy, Qxz}, Qyz, Qzz) about the group centre gc into
// fc: the exact form.
template <bool kQuad>
__device__ __forceinline__ void far_coefs_exact(float4 cm, float4 q, float qyz, float qzz, float gcx,
                                                float gcy, float gcz, float eps2,
                                                float (&fc)[kFarCoefs]) {
    FarTerms f;
    f.D[0] = __fadd_rn(cm.x, -gcx);
    f.D[1] = __fadd_rn(cm.y, -gcy);
    f.D[2] = __fadd_rn(cm.z, -gcz);
    const float m = cm.w;
    const float r2 = __fadd_rn(
        xfma<true>(f.D[0], f.D[0], xfma<true>(f.D[1], f.D[1], __fmul_rn(f.D[2], f.D[2]))), eps2);
    const float R = __fdiv_rn(1.0f, __fsqrt_rn(r2));
    const float R2 = __fmul_rn(R, R), R3 = __fmul_rn(R2, R), R5 = __fmul_rn(R3, R2),
                R7 = __fmul_rn(R5, R2);
    f.R5 = R5;
    const float qxx = kQuad ? q.x : 0.f, qyy = kQuad ? q.y : 0.f, qxy = kQuad ? q.z : 0.f,
                qxz = kQuad ? q.w : 0.f, qyz_ = kQuad ? qyz : 0.f, qzz_ = kQuad ? qzz : -0.f;
    f.Q[0][0] = qxx; f.Q[0][1] = qxy; f.Q[0][2] = qxz;
    f.Q[1][0] = qxy; f.Q[1][1] = qyy; f.Q[1][2] = qyz_;
    f.Q[2][0] = qxz; f.Q[2][1] = qyz_; f.Q[2][2] = qzz_;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        f.qv[i] = xfma<true>(f.Q[i][0], f.D[0],
                             xfma<true>(f.Q[i][1], f.D[1], __fmul_rn(f.Q[i][2], f.D[2])));
    const float sq = xfma<true>(f.D[0], f.qv[0], xfma<true>(f.D[1], f.qv[1], __fmul_rn(f.D[2], f.qv[2])));
    const float R9 = __fmul_rn(R7, R2), R11 = __fmul_rn(R9, R2);
    f.al = xfma<true>(m, R3, __fmul_rn(__fmul_rn(2.5f, sq), R7));
    f.be = xfma<true>(__fmul_rn(3.0f, m), R5, __fmul_rn(__fmul_rn(17.5f, sq), R9));
    f.ga = __fmul_rn(5.0f, R7);
    f.ka = -__fmul_rn(35.0f, R9);
    f.nu = xfma<true>(__fmul_rn(15.0f, m), R7, __fmul_rn(__fmul_rn(157.5f, sq), R11));
#pragma unroll
    for (int i = 0; i < 3; ++i)
        fc[i] = __fadd_rn(fc[i], xfma<true>(f.al, f.D[i], -__fmul_rn(R5, f.qv[i])));
    fc[3] = __fadd_rn(fc[3], far_j<0, 0>(f));
    fc[4] = __fadd_rn(fc[4], far_j<1, 1>(f));
    fc[5] = __fadd_rn(fc[5], far_j<2, 2>(f));
    fc[6] = __fadd_rn(fc[6], far_j<0, 1>(f));
    fc[7] = __fadd_rn(fc[7], far_j<0, 2>(f));
    fc[8] = __fadd_rn(fc[8], far_j<1, 2>(f));
    fc[9] = __fadd_rn(fc[9], far_h<0, 0, 0>(f));
    fc[10] = __fadd_rn(fc[10], far_h<1, 1, 1>(f));
    fc[11] = __fadd_rn(fc[11], far_h<2, 2, 2>(f));
    fc[12] = __fadd_rn(fc[12], far_h<0, 0, 1>(f));
    fc[13] = __fadd_rn(fc[13], far_h<0, 0, 2>(f));
    fc[14] = __fadd_rn(fc[14], far_h<0, 1, 1>(f));
    fc[15] = __fadd_rn(fc[15], far_h<1, 1, 2>(f));
    fc[16] = __fadd_rn(fc[16], far_h<0, 2, 2>(f));
    fc[17] = __fadd_rn(fc[17], far_h<1, 2, 2>(f));
    fc[18] = __fadd_rn(fc[18], far_h<0, 1, 2>(f));
}

// The fast form's sums, turned into the coefficients above once per walk
// (far_finish). Per node, with u = ga q, v = u - be D, w = u + v,
// t = nu/3 D + ka q and B_ij = ga Q_ij + (t_i D_j + t_j D_i) / 2,
//   J_ij  = (w_i D_j + w_j D_i) / 2 - R^5 Q_ij + al [i=j]
//   H_ijk = B_ij D_k + B_ik D_j + B_jk D_i + v_k [i=j] + v_j [i=k] + v_i [j=k]
// and the traces are cheaper than the components with two z's: the field is
// harmonic but for the softening, J_ii = eps^2 be and
// H_iik = -eps^2 (nu D_k + ka q_k). Sums kept: a; Jxx, Jyy, be, 2 Jxy, 2 Jxz,
// 2 Jyz; Hxxx, Hyyy, trace z, Hxxy, Hxxz, Hxyy, Hyyz, trace x, trace y,
// 2 Hxyz. About 115 operations a node, against 170 with all 19 components
// formed apart.
template <bool kQuad>
__device__ __forceinline__ void far_coefs_fast(float4 cm, float4 q, float qyz, float gcx, float gcy,
                                               float gcz, float eps2, float (&fc)[kFarCoefs]) {
    const float D[3] = {cm.x - gcx, cm.y - gcy, cm.z - gcz};
    const float m = cm.w;
    const float R = rsqrtf(fmaf(D[0], D[0], fmaf(D[1], D[1], fmaf(D[2], D[2], eps2))));
    const float R2 = R * R, R3 = R2 * R, R5 = R3 * R2, R7 = R5 * R2;
    const float ga = 5.0f * R7, m3 = 3.0f * m;
    float al, be, nu, t[3], v[3], w[3];
    float b00, b11, c01, c02, c12;  // B00, B11, 2 B01, 2 B02, 2 B12
    if constexpr (kQuad) {
        const float qzz = -(q.x + q.y);
        const float qv[3] = {fmaf(q.x, D[0], fmaf(q.z, D[1], q.w * D[2])),
                             fmaf(q.z, D[0], fmaf(q.y, D[1], qyz * D[2])),
                             fmaf(q.w, D[0], fmaf(qyz, D[1], qzz * D[2]))};
        const float hs = 0.5f * fmaf(D[0], qv[0], fmaf(D[1], qv[1], D[2] * qv[2]));
        const float R9 = R7 * R2, k35 = 35.0f * R9;
        al = fmaf(ga, hs, m * R3);
        be = fmaf(k35, hs, m3 * R5);
        nu = fmaf(9.0f * k35 * R2, hs, m3 * ga);
        const float nu3 = nu * (1.0f / 3.0f);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float u = ga * qv[i];
            t[i] = fmaf(nu3, D[i], -k35 * qv[i]);
            v[i] = fmaf(-be, D[i], u);
            w[i] = u + v[i];
            fc[i] = fmaf(al, D[i], fmaf(-R5, qv[i], fc[i]));
        }
        const float ga2 = 2.0f * ga, r52 = -2.0f * R5;
        b00 = fmaf(t[0], D[0], ga * q.x);
        b11 = fmaf(t[1], D[1], ga * q.y);
        c01 = fmaf(t[0], D[1], fmaf(t[1], D[0], ga2 * q.z));
        c02 = fmaf(t[0], D[2], fmaf(t[2], D[0], ga2 * q.w));
        c12 = fmaf(t[1], D[2], fmaf(t[2], D[1], ga2 * qyz));
        fc[3] = fmaf(-R5, q.x, fc[3]);
        fc[4] = fmaf(-R5, q.y, fc[4]);
        fc[6] = fmaf(r52, q.z, fc[6]);
        fc[7] = fmaf(r52, q.w, fc[7]);
        fc[8] = fmaf(r52, qyz, fc[8]);
    } else {
        al = m * R3;
        be = m3 * R5;
        nu = m3 * ga;
        const float nu3 = nu * (1.0f / 3.0f);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            t[i] = nu3 * D[i];
            v[i] = w[i] = -be * D[i];
            fc[i] = fmaf(al, D[i], fc[i]);
        }
        b00 = t[0] * D[0];
        b11 = t[1] * D[1];
        c01 = 2.0f * t[0] * D[1];
        c02 = 2.0f * t[0] * D[2];
        c12 = 2.0f * t[1] * D[2];
    }
    const float nu23 = nu * (2.0f / 3.0f);
    fc[3] = fmaf(w[0], D[0], fc[3] + al);
    fc[4] = fmaf(w[1], D[1], fc[4] + al);
    fc[5] += be;
    fc[6] = fmaf(w[0], D[1], fmaf(w[1], D[0], fc[6]));
    fc[7] = fmaf(w[0], D[2], fmaf(w[2], D[0], fc[7]));
    fc[8] = fmaf(w[1], D[2], fmaf(w[2], D[1], fc[8]));
    fc[9] = fmaf(3.0f, fmaf(b00, D[0], v[0]), fc[9]);
    fc[10] = fmaf(3.0f, fmaf(b11, D[1], v[1]), fc[10]);
    fc[11] = fmaf(nu23, D[2], fc[11] + t[2]);
    fc[12] = fmaf(c01, D[0], fmaf(b00, D[1], fc[12] + v[1]));
    fc[13] = fmaf(c02, D[0], fmaf(b00, D[2], fc[13] + v[2]));
    fc[14] = fmaf(c01, D[1], fmaf(b11, D[0], fc[14] + v[0]));
    fc[15] = fmaf(c12, D[1], fmaf(b11, D[2], fc[15] + v[2]));
    fc[16] = fmaf(nu23, D[0], fc[16] + t[0]);
    fc[17] = fmaf(nu23, D[1], fc[17] + t[1]);
    fc[18] = fmaf(c01, D[2], fmaf(c02, D[1], fmaf(c12, D[0], fc[18])));
}
__device__ __forceinline__ void far_finish(float eps2, float (&fc)[kFarCoefs]) {
    fc[5] = eps2 * fc[5] - fc[3] - fc[4];
    fc[6] *= 0.5f;
    fc[7] *= 0.5f;
    fc[8] *= 0.5f;
    const float tx = fc[16], ty = fc[17], tz = fc[11];
    fc[16] = -eps2 * tx - fc[9] - fc[14];
    fc[17] = -eps2 * ty - fc[12] - fc[10];
    fc[11] = -eps2 * tz - fc[13] - fc[15];
    fc[18] *= 0.5f;
}

// The expansion fc at offset rho from the group centre (without G).
template <bool kExact>
__device__ __forceinline__ void far_eval(const float (&fc)[kFarCoefs], float rx, float ry, float rz,
                                         float& ox, float& oy, float& oz) {
    const float pxx = xmul<kExact>(rx, rx), pyy = xmul<kExact>(ry, ry), pzz = xmul<kExact>(rz, rz);
    const float pxy = xmul<kExact>(rx, ry), pxz = xmul<kExact>(rx, rz), pyz = xmul<kExact>(ry, rz);
    const float* J = fc + 3;
    const float* H = fc + 9;
    auto comp = [&](float a, float j0, float j1, float j2, float h0, float h1, float h2, float h3,
                    float h4, float h5) {
        const float jr = xfma<kExact>(j0, rx, xfma<kExact>(j1, ry, xmul<kExact>(j2, rz)));
        const float cross = xfma<kExact>(h3, pxy, xfma<kExact>(h4, pxz, xmul<kExact>(h5, pyz)));
        const float hh = xfma<kExact>(
            h0, pxx, xfma<kExact>(h1, pyy, xfma<kExact>(h2, pzz, xmul<kExact>(2.0f, cross))));
        return xfma<kExact>(0.5f, hh, xadd<kExact>(a, -jr));
    };
    // Rows: J {x: xx xy xz, y: xy yy yz, z: xz yz zz}; H {x: xxx xyy xzz xxy xxz xyz,
    // y: xxy yyy yzz xyy xyz yyz, z: xxz yyz zzz xyz xzz yzz}.
    ox = comp(fc[0], J[0], J[3], J[4], H[0], H[5], H[7], H[3], H[4], H[9]);
    oy = comp(fc[1], J[3], J[1], J[5], H[3], H[1], H[8], H[5], H[9], H[6]);
    oz = comp(fc[2], J[4], J[5], J[2], H[4], H[6], H[2], H[9], H[7], H[8]);
}

// Per-lane acceleration sum: plain or compensated (Kahan) per component.
template <bool kExact, bool kKahan>
struct Accum {
    float ax = 0.f, ay = 0.f, az = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;

    __device__ __forceinline__ void add1(float& s, float& c, float t) {
        if (kKahan) {
            if (kExact) {
                const float y = __fsub_rn(t, c);
                const float u = __fadd_rn(s, y);
                c = __fsub_rn(__fsub_rn(u, s), y);
                s = u;
            } else {
                const float y = t - c;
                const float u = s + y;
                c = (u - s) - y;
                s = u;
            }
        } else {
            s = kExact ? __fadd_rn(s, t) : s + t;
        }
    }
    __device__ __forceinline__ void add(float tx, float ty, float tz) {
        add1(ax, cx, tx);
        add1(ay, cy, ty);
        add1(az, cz, tz);
    }

    // Blocked form (group walk, exact): with Kahan, terms are added plainly
    // within blocks of 32 consecutive list positions and each block's
    // partial is Kahan-added by step(); every position steps, including a
    // particle's own skipped one. Without Kahan, push() is add().
    float bx = 0.f, by = 0.f, bz = 0.f;
    uint32_t k = 0;
    __device__ __forceinline__ void push(float tx, float ty, float tz) {
        if (kKahan) {
            bx = kExact ? __fadd_rn(bx, tx) : bx + tx;
            by = kExact ? __fadd_rn(by, ty) : by + ty;
            bz = kExact ? __fadd_rn(bz, tz) : bz + tz;
        } else {
            add(tx, ty, tz);
        }
    }
    __device__ __forceinline__ void close() {
        add(bx, by, bz);
        bx = by = bz = 0.f;
    }
    __device__ __forceinline__ void step() {
        if (kKahan && (++k & 31u) == 0u) close();
    }
    __device__ __forceinline__ void finish() {
        if (kKahan && (k & 31u) != 0u) close();
    }
};


}  // namespace astro
