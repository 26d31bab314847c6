// pencil.cuh -- the enumeration's certified filter for candidate tetrahedra
// of one triangle: the alpha test and the early refutation in a few
// operations each, with a proof per decision that the general path (the
// reference's binary32 formulas, refarith.cuh, or the exact polynomials,
// exactpred.cuh) would decide the same.
//
// Geometry.  For the triangle of balls p, v2, v3 and any ball z let
// z' = z - p (A, B for v2, v3), n = A x B, and the lift
//     s(z) = |z'|^2 - w_z + w_p.
// The spheres orthogonal to the three balls form a pencil; its smallest one
// is centred at p + Q/2 with Q in the triangle's plane, Q.A = s(A),
// Q.B = s(B).  With
//     h(z) = n . z'            g(z) = s(z) - Q . z'
// the pencil's sphere through z is centred at p + Q/2 + (t/2) n, t = g/h,
// its power is rho(z) = |Q|^2/4 - w_p + t^2 |n|^2 / 4, and the power of a ball
// y with respect to it is g(y) - t(z) h(y).  Hence, exactly,
//     alpha tetrahedron  <=>  g^2 - k h^2 <= 0,  k = 4 (alpha + w_p - |Q|^2/4) / |n|^2
//     y violates (p, v2, v3, x)  <=>  sign(h(x)) (g(y) h(x) - g(x) h(y)) < 0
// and g(y) h(x) - g(x) h(y) is the lifted determinant insphere_w evaluates
// (up to sign), h(x) the one orient3d evaluates.
//
// Bounds (u = 2^-24).  L bounds every alpha edge's length, W every weight, R
// the grown radius sqrt(w + alpha), C the distance of the four vertices from
// the origin, q = |Q| <= 2.03 R (larger ones certify nothing);
// l = |A| |A - B|, N = |n|, H = N L >= |h|, G = L^2 + W + q L >= |g|.  All
// candidates z of a triangle are joined to its three vertices by alpha edges,
// so |z'|, |z - v2|, |z - v3| <= L.
//  * This file's rounding.  z' and s are rounded once from exact values, n and
//    Q are computed in double (Q's division in single) and rounded; a three
//    term FMA chain each:  |dh| <= Eh = 6 u H,
//    |dg| <= Eg = u (4.2 (L^2 + W) + 8.2 q L).
//  * insphere_w in binary32 is off by at most 18 u P (certify.cuh; 21 u P when
//    contraction keeps its weights unrounded), P its expression over magnitudes.
//    Each 3 x 3 minor's permanent is at most 1.155 times the product of its
//    rows' lengths (n!/n^(n/2), n = 3), the rows are differences from y: L for
//    p, v2, v3 and 2 L for x, so P <= 1.155 L^3 (10 L^2 + 7 W).  Refutation is
//    certain when sign(h(x)) (g(y) h(x) - g(x) h(y)) < -rg with
//    rg >= 21 u P + 2 (G Eh + H Eg) + 4 u G H, and the sign of orient3d, off
//    by at most 9 u 1.155 L^3, is certain (|h| >= hmin).
//  * markRealTets in binary32.  Its centre X^ is Cramer's rule over rows
//    a_i = p - v2, v2 - v3, v3 - x (lengths l_1, l_2 with l_1 l_2 = l, and at most
//    L) and b_i, half the differences of |z|^2 - w.  Those squares are rounded
//    once per ball: the filter takes the rounded squares as the data
//    (s~ = s + e(z) - e(p), e(z) the rounding of z's squares; X~, g~, Q~ from
//    them), which leaves |db_i| <= u (5 l_i C + W).  A numerator's terms carry at
//    most 9 roundings besides b's, their magnitudes sum to at most
//    sum_i |b_i| |a_j'| |a_k'| (a' the two other coordinates), |b_i| <= l_i C + W/2,
//    and over the three numerators the 2-norm of |a_j'| |a_k'| is at most
//    sqrt(2) |a_j| |a_k|; the denominator carries 11 u 1.155 l L, the quotient u.
//    So with S = l + 2 L^2 >= l_1 l_2 + (l_1 + l_2) L and D = |X~ - v2|
//      |X^ - X~| <= (e1 + e2 D) / |h|,
//      e1 = u (68 l L C + 8 W S),   e2 = 14 u l L.
//    (With contraction a square of a difference may or may not be rounded, and
//    a weight too: half of e(z) is taken, and e1 grows by 0.51 u C^2 S + 2.2 u W S.
//    The unperturbed centre X is within u C^2 S / |h| of X~.)  With
//    e = e1 + 2 e2 R the reference's power compares with alpha as X~'s does when
//    |rho - alpha| > 2.2 R e / |h|; near alpha D <= 2 R, and far above it
//    (t N > 4 R, so rho - alpha >= 3 R^2) the same margin holds when e / |h| is
//    below R / 8, which the alpha test's own limit kappa hmin ensures.
//    The comparison is made as |g~^2 - k h^2| > ea |h|, ea |n|^2 four times that
//    margin plus the roundings of dist and of this file.
//  * The reference's window of the tetrahedron (27 cells around X^) surely
//    holds y when every coordinate of y - X^ is below 0.99 cell steps
//    (pipeline.cu).  A violator is within R of X, so it suffices that
//    R + 2.3 e / |h| + 2.2 u C^2 S / |h| <= 0.99 step, which hmin ensures (the
//    factors above one for a power not certainly below alpha); where R is
//    too large for that, or C makes it costly, the caller checks that y lies
//    within 0.86 steps of X~ on every axis (violators are within R, about 0.8
//    steps), and hmin leaves 0.125 steps for e / |h| and the rounding of that check.
//  * Attachment of the triangle itself.  markRealTriangles' centre Xt^ (upstream
//    formulas) is Cramer's rule over p - v2, v2 - v3 and the computed normal n^,
//    b3 = n^ . p; checkDanglingTris compares, for a ball e,
//    |e - Xt^|^2 - w_e with |p - Xt^|^2 - w_p, which differ by s(e) - 2 e' . (Xt^ - p),
//    and 2 (Xt~ - p) = Q~.  Counting as above (the third row has length N, the
//    determinant is N^2, a tilt of n^ by 3.6 u |A| |B| / N moves Xt^ along n by
//    that times |Q| / 2),
//      |Xt^ - Xt~| <= d = u (65 l C + 16 W L + 26 l R + 3.7 L^2 R) / N + 1.05 u (C + R)
//    (with contraction + u C^2 L / N), so e attaches the triangle in binary32 when
//    s(e) - Q~ . e' = g~(e) + (s(e) - s~(e)) < -mt, mt the sum of 2 L d, Eg and the
//    rounding of the two powers.  Such a ball lies within 1.005 R of Xt (rho <= alpha + 0.01 R^2 is
//    checked), hence in the window of Xt^ when 1.01 R + 2.1 u C^2 L / N + d is
//    below 0.99 step; where C or R make that costly, the caller checks that e lies
//    within 0.95 steps of Xt~ on every axis, and d stays below 0.04 steps.
// So every bound is affine in N and l with coefficients that depend on the
// ball p alone.  They are evaluated in binary32 with factors that cover their
// own rounding; NaN and overflow compare false, so nothing is certified then.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define PAC_PENCIL_FN __host__ __device__ __forceinline__
#else
#define PAC_PENCIL_FN inline
#endif

namespace pac {
namespace pencil {

constexpr float kU = 5.9604645e-08f;  // 2^-24

// What holds for every triangle of one ball p: the three bounds as
// c[0] + c[1] N + c[2] l, and the limits below which a triangle is fine.
struct Bounds {
    float rg[2];      // refutation (no l term)
    float m4[3];      // alpha test, times |n|^2
    float hmin[3];
    float nmin2;      // |n|^2 below this: needle triangles (double's rounding of n would show)
    float mt[3];      // attachment: (mt[0] + mt[1] l) / N + mt[2]
    float mw, mtmax;  // its use needs mw / N + mt < mtmax
    float mreach;     // 0.95 step where its window needs the check by distance, else 0
    float base4;      // 4 (w + alpha) + 0.04 R^2
    float kappa;      // the alpha test's limit in |h| is kappa hmin
    float q2max;      // |Q|^2 above this certifies nothing
    float alpha;
    float reach;      // 0.86 step where the window needs the check by distance, else 0
};

// p's centre and weight; maxlen2: largest squared length of an alpha edge (binary32); wmax: upper
// bound of every weight; contracted: markRealTets compiled with FMA contraction.
PAC_PENCIL_FN Bounds bounds(float px, float py, float pz, float wp, float alpha, float maxlen2,
                            float wmax, float step, bool contracted) {
    Bounds b;
    const float L = sqrtf(maxlen2) * 1.001f, L2 = L * L, W = wmax;
    const float R = sqrtf(fmaxf(W + alpha, 0.0f)) * 1.001f, R2 = R * R;
    const float C = sqrtf(px * px + py * py + pz * pz) * 1.001f + L;
    const float q = 2.03f * R;
    const float G = L2 + W + q * L;
    const float Eg = kU * (4.2f * (L2 + W) + 8.2f * q * L);
    const float eh = 6.0f * kU * L;  // Eh = eh N
    const float insphere = 21.0f * 1.16f * kU * L * L2 * (10.0f * L2 + 7.0f * W);
    b.rg[0] = 1.02f * insphere + 1e-20f;
    b.rg[1] = 1.02f * (2.0f * (G * eh + L * Eg) + 4.0f * kU * G * L);
    // e = ea + eb l, C^2 S = ca + cb l
    const float ca = kU * C * C * 2.0f * L2, cb = kU * C * C;
    const float ws = (contracted ? 10.2f : 8.0f) * kU * W;
    const float ea = ws * 2.0f * L2 + (contracted ? 0.51f * ca : 0.0f);
    const float eb = kU * (68.0f * L * C + 28.0f * L * R) + ws + (contracted ? 0.51f * cb : 0.0f);
    b.m4[0] = 1.02f * 9.2f * R * ea + 1e-20f;
    b.m4[2] = 1.02f * 9.2f * R * eb;
    b.m4[1] = 1.02f * (32.0f * kU * (2.0f * R2 + W) * L + 8.0f * R * Eg + 8.0f * R2 * eh +
                       kU * L * (100.0f * R2 + 16.0f * (q * q + W + fabsf(alpha))));
    const float slack = 0.99f * step - R;
    const bool win_ok = slack > 0.02f * R && 2.2f * (ca + cb * L2) < 3.0f * slack;
    b.reach = win_ok ? 0.0f : 0.86f * step;
    // hmin: the sum of the conditions above (each at least, so their sum),
    // those of the firsts and of refutation; the alpha test's are kappa times it
    const float iR = 1.0f / R, iR2 = 0.5f * iR * iR;
    const float iw = win_ok ? 1.0f / slack : 1.0f / (0.125f * step);
    const float we = win_ok ? 2.3f : 1.05f, wc = win_ok ? 2.2f : 0.0f;
    b.hmin[0] = 1.02f * (12.0f * kU * L * L2 + iw * (we * ea + wc * ca));
    b.hmin[1] = 1.02f * (1025.0f * eh + 16.0f * Eg * iR + (win_ok ? 0.0f : 2.0f * iw * Eg));
    b.hmin[2] = 1.02f * (iw * (we * eb + wc * cb));
    const float a0 = 1.02f * (9.0f * iR * ea + iR2 * b.m4[0] + 12.0f * kU * L * L2);
    const float a1 = 1.02f * (1025.0f * eh + 16.0f * Eg * iR + iR2 * b.m4[1]);
    const float a2 = 1.02f * (1024.0f * 14.0f * kU * L + 9.0f * iR * eb + iR2 * b.m4[2]);
    b.kappa = 1.0001f * fmaxf(fmaxf(1.0f, a0 / b.hmin[0]), fmaxf(a1 / b.hmin[1], a2 / b.hmin[2]));
    b.alpha = alpha;
    const float ct = contracted ? 1.05f * kU * C * C * L : 0.0f;
    b.mt[0] = 1.02f * 2.0f * L * (kU * (16.0f * W * L + 3.7f * L2 * R) + ct);
    b.mt[1] = 1.02f * kU * 2.0f * L * (65.0f * C + 26.0f * R);
    b.mt[2] = 1.02f * (kU * (2.1f * L * (C + R) + 16.0f * (2.0f * R2 + W)) + Eg) + 1e-20f;
    const float aslack = 0.99f * step - 1.01f * R;
    const bool near_ok = aslack > 0.02f * R && 10.0f * kU * C * C < 0.3f * aslack * L;
    b.mreach = near_ok ? 0.0f : 0.95f * step;
    b.mw = near_ok ? 2.2f * kU * C * C * L * 2.0f * L : 0.0f;
    b.mtmax = 2.0f * L * (near_ok ? aslack : 0.04f * step);
    b.base4 = 4.0f * (wp + alpha) + 0.04f * R2;
    b.nmin2 = fmaxf(1e-6f * L2 * L2, 1e-18f);
    b.q2max = 4.1f * R2;
    // sizes the bounds were not written for certify nothing
    if (!(L < 1e3f && W < 1e6f && R < 1e3f && C < 1e5f)) b.q2max = -1.0f;
    return b;
}

struct Group {
    float nx, ny, nz, hmin;  // below hmin in |h| nothing is certified (alpha: kappa hmin)
    float qx, qy, qz, rg;    // Q, the refutation's margin
    float tx, ty, tz, k;     // Q~, the alpha test's k
    float ea;                // and margin
    float mt;                // attachment's margin
};

// A neighbour of p: its position relative to p, its lift s and the lift s~ of
// the rounded squares (the same where they do not apply).
struct Point {
    double x, y, z, s, st;
};

// The triangle of p, A and B; wp the weight of p.
PAC_PENCIL_FN Group group(const Bounds &b, const Point &A, const Point &B, float wp) {
    Group g;
    const double nx = fma(A.y, B.z, -(A.z * B.y)), ny = fma(A.z, B.x, -(A.x * B.z)),
                 nz = fma(A.x, B.y, -(A.y * B.x));
    // B x n and n x A
    const double ux = fma(B.y, nz, -(B.z * ny)), uy = fma(B.z, nx, -(B.x * nz)),
                 uz = fma(B.x, ny, -(B.y * nx));
    const double vx = fma(ny, A.z, -(nz * A.y)), vy = fma(nz, A.x, -(nx * A.z)),
                 vz = fma(nx, A.y, -(ny * A.x));
    g.nx = (float)nx, g.ny = (float)ny, g.nz = (float)nz;
    const float N2 = fmaf(g.nx, g.nx, fmaf(g.ny, g.ny, g.nz * g.nz)), inv = 1.0f / N2;
    g.qx = (float)fma(A.s, ux, B.s * vx) * inv;
    g.qy = (float)fma(A.s, uy, B.s * vy) * inv;
    g.qz = (float)fma(A.s, uz, B.s * vz) * inv;
    g.tx = (float)fma(A.st, ux, B.st * vx) * inv;
    g.ty = (float)fma(A.st, uy, B.st * vy) * inv;
    g.tz = (float)fma(A.st, uz, B.st * vz) * inv;
    // power at the pencil's base about v2: |Q~|^2/4 - w_p + (s(A) - s~(A))
    const float t2 = fmaf(g.tx, g.tx, fmaf(g.ty, g.ty, g.tz * g.tz));
    const float base = fmaf(0.25f, t2, (float)(A.s - A.st) - wp);
    const float q2 = fmaxf(t2, fmaf(g.qx, g.qx, fmaf(g.qy, g.qy, g.qz * g.qz)));
    const float ax = (float)A.x, ay = (float)A.y, az = (float)A.z;
    const float cx = (float)(A.x - B.x), cy = (float)(A.y - B.y), cz = (float)(A.z - B.z);
    const float l = sqrtf(fmaf(ax, ax, fmaf(ay, ay, az * az)) *
                          fmaf(cx, cx, fmaf(cy, cy, cz * cz))) * 1.0001f;
    const float N = sqrtf(N2) * 1.0001f;
    g.rg = fmaf(b.rg[1], N, b.rg[0]);
    g.ea = fmaf(b.m4[1], N, fmaf(b.m4[2], l, b.m4[0])) * inv;
    g.k = 4.0f * (b.alpha - base) * inv;
    const float hm = fmaf(b.hmin[1], N, fmaf(b.hmin[2], l, b.hmin[0]));
    const float mt = fmaf(fmaf(b.mt[1], l, b.mt[0]), N * inv, b.mt[2]);
    const bool fine = N2 > b.nmin2 && q2 < b.q2max && hm < 1e18f;
    g.hmin = fine ? hm : INFINITY;
    g.mt = fine && q2 < b.base4 && fmaf(b.mw, N * inv, mt) < b.mtmax ? mt : INFINITY;
    return g;
}

PAC_PENCIL_FN float height(float nx, float ny, float nz, float x, float y, float z) {
    return fmaf(nz, z, fmaf(ny, y, nx * x));
}
PAC_PENCIL_FN float power(float qx, float qy, float qz, float s, float x, float y, float z) {
    return fmaf(-qz, z, fmaf(-qy, y, fmaf(-qx, x, s)));
}

// Whether z lies within reach, per axis, of the triangle's centre Xt~.
PAC_PENCIL_FN bool in_box(float tx, float ty, float tz, float x, float y, float z, float reach) {
    return fmaxf(fabsf(fmaf(-0.5f, tx, x)),
                 fmaxf(fabsf(fmaf(-0.5f, ty, y)), fabsf(fmaf(-0.5f, tz, z)))) <= reach;
}

// Alpha test of x (a = |h(x)| >= kappa hmin, gt = g~(x)): certainly alpha, certainly
// not, or neither.
PAC_PENCIL_FN void alpha_test(float a, float gt, float k, float ea, bool &in, bool &out) {
    const float m = ea * a, f = fmaf(gt, gt, -(k * a) * a);
    in = f < -m;
    out = f > m;
}

// Whether ball v lies within reach, per axis, of the orthosphere centre X~ of x
// (all relative to p; h = h(x), gt = g~(x)).
PAC_PENCIL_FN bool within_reach(float nx, float ny, float nz, float tx, float ty, float tz, float h,
                                float gt, float vx, float vy, float vz, float reach) {
    const float t = 0.5f * gt / h;
    return fmaxf(fabsf(fmaf(t, nx, 0.5f * tx) - vx),
                 fmaxf(fabsf(fmaf(t, ny, 0.5f * ty) - vy), fabsf(fmaf(t, nz, 0.5f * tz) - vz))) <= reach;
}

// Whether ball y certainly violates the tetrahedron of x (|h(x)| >= hmin).
PAC_PENCIL_FN bool refutes(float hx, float gx, float hy, float gy, float rg) {
    const float v = fmaf(gy, hx, -(gx * hy));
    return (hx < 0.0f ? -v : v) < -rg;
}

}  // namespace pencil
}  // namespace pac
