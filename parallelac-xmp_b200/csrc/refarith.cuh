// refarith.cuh -- the reference's single-precision filter arithmetic.
//
// Each function performs the float operations of one reference kernel in
// the reference's statement and operand order.  The translation unit that
// includes this header is compiled twice:
//   strict     : every operation is one IEEE binary32 op (-fmad=false, the
//                oracle-identical flavour), and
//   contracted : (PAC_CONTRACTED) multiply-adds are fused as nvcc fuses them
//                by default, the flavour that follows the reference built
//                with default flags.
// The formulas themselves have to be the reference's for the decisions to
// match bit for bit; the statement layout is kept for the same reason.
//
// Which multiply-adds nvcc fuses depends on the code around an expression, so
// the contracted flavour does not leave it to the compiler: every product that
// meets a sum is written with its rounding (diff, sum, plus, minus below), by a
// sequence per place (the At... structs).  The sequences are those nvcc 12.9
// gave the kernels that first had this flavour, found by comparing their
// results -- the spheres of 600,000 tetrahedra bit for bit, some 90 million
// decisions of lattices and clusters whose last radius sits within a few ulps
// of the decision's flip -- with every choice of sequence.  A place that was
// compiled twice with two sequences (balls of at most 64 upper neighbours and
// others) keeps both; the as-run enumeration, whose counting and writing
// passes had disagreed by one term, keeps the writing pass's in both.
//
// Citations: LD = AlphaComplexLargeData.cu, PLAIN = AlphaComplexParallel.cu,
//            PRED = predicates.h.
#pragma once
#include <cmath>
#include <cstdint>

namespace pac {

struct Ball {
    float x, y, z, r;  // r = raw radius + solvent radius (LD:1085)
};

__device__ __forceinline__ Ball ld_ball(const float4 *p) {
    float4 v = __ldg(p);
    return Ball{v.x, v.y, v.z, v.w};
}

// formula sets; kExact selects the decision-exact predicates (exactpred.cuh)
enum : int { kUpstream = 0, kPlainXmp = 1, kExact = 2 };

// The reference compares binary32 results in double precision: THRES and
// ATHRES are the double literal 0.0 (LD:48-49), so `x <= (alpha + ATHRES)`
// (LD:185, 347, 588) and `powDist + THRES <= currentDist` (LD:829, 968)
// convert their binary32 operands to double.  That conversion is exact and
// adding +0.0 changes no value a comparison sees, so each such test has the
// outcome of the binary32 comparison x <= y, NaNs included; that is what is
// evaluated here.  (Tests whose right-hand side is a double product, in the
// plain-xmp formulas, stay in double.)
__device__ __forceinline__ bool le_as_double(float x, float y) { return x <= y; }

// ------------------------------------------------------------- contraction
#ifdef PAC_CONTRACTED
constexpr bool kFused = true;
#else
constexpr bool kFused = false;
#endif

#ifdef __CUDACC__
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float mul_rn(float a, float b) { return kFused ? __fmul_rn(a, b) : a * b; }
__device__ __forceinline__ float add_rn(float a, float b) { return kFused ? __fadd_rn(a, b) : a + b; }
__device__ __forceinline__ float sub_rn(float a, float b) { return kFused ? __fsub_rn(a, b) : a - b; }
#else  // host checks, built without contraction
inline float fma_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
inline float mul_rn(float a, float b) { return a * b; }
inline float add_rn(float a, float b) { return a + b; }
inline float sub_rn(float a, float b) { return a - b; }
#endif

// a b - c d and a b + c d; M says which product is fused (0: both are rounded)
template <int M>
__device__ __forceinline__ float diff(float a, float b, float c, float d) {
    if constexpr (kFused && M == 1) return fma_rn(a, b, -mul_rn(c, d));
    else if constexpr (kFused && M == 2) return fma_rn(-c, d, mul_rn(a, b));
    else return sub_rn(mul_rn(a, b), mul_rn(c, d));
}
template <int M>
__device__ __forceinline__ float sum(float a, float b, float c, float d) {
    if constexpr (kFused && M == 1) return fma_rn(a, b, mul_rn(c, d));
    else if constexpr (kFused && M == 2) return fma_rn(c, d, mul_rn(a, b));
    else return add_rn(mul_rn(a, b), mul_rn(c, d));
}
// s + a b and s - a b; M = 1: fused
template <int M>
__device__ __forceinline__ float plus(float s, float a, float b) {
    if constexpr (kFused && M == 1) return fma_rn(a, b, s);
    else return add_rn(s, mul_rn(a, b));
}
template <int M>
__device__ __forceinline__ float minus(float s, float a, float b) {
    if constexpr (kFused && M == 1) return fma_rn(-a, b, s);
    else return sub_rn(s, mul_rn(a, b));
}

// The sequences, by place.  b1, b2, b3: the three differences of squares, the
// - r^2 and the + r^2 of a difference of powers (power_diff); b1w: b1 for balls
// of more than 64 upper neighbours; det: the first sum of D, Dx, Dy and Dz (the
// other terms are fused); dist: the first sum of squares, the third square, the
// - r^2 of a power.
struct AtEdge {  // alpha test of an edge
    static constexpr int b1[5] = {2, 2, 2, 0, 1};
};
template <int V>
struct AtLink {  // alpha test of a triangle, balls of at most 64 upper neighbours
    static constexpr int b1[5] = {0, 0, 0, 0, 1}, b2[5] = {2, 2, 2, 1, 1};
    static constexpr int det[4] = {1, V == kPlainXmp ? 1 : 2, 2, 1};
    static constexpr int dist[3] = {1, 1, V == kPlainXmp ? 1 : 0};
};
template <int V>
struct AtLinkWide {  // and of the others
    static constexpr int b1[5] = {0, 0, 0, 0, 0}, b2[5] = {2, 2, 2, 0, 1};
    static constexpr int det[4] = {1, 1, 2, 1};
    static constexpr int dist[3] = {1, 1, V == kPlainXmp ? 1 : 0};
};
template <int V>
struct AtAttach {  // the triangle's sphere in its attachment test
    static constexpr int b1[5] = {1, 1, 1, 0, 1}, b2[5] = {2, 2, 2, 1, 1};
    static constexpr int det[4] = {1, V == kPlainXmp ? 1 : 2, 2, 1};
    static constexpr int dist[3] = {1, 1, V == kPlainXmp ? 1 : 0};
};
struct AtFoot {  // an edge's radical foot in its attachment test
    static constexpr int b1[5] = {1, 1, 1, 0, 1}, dist[3] = {1, 1, 0};
};
struct AtPower {  // a ball's power in both attachment tests
    static constexpr int dist[3] = {1, 1, 1};
};
struct AtEnum {  // alpha test and sphere of a tetrahedron, as written
    static constexpr int b1[5] = {1, 1, 1, 0, 0}, b1w[5] = {0, 0, 1, 0, 0};
    static constexpr int b2[5] = {2, 2, 2, 0, 1}, b3[5] = {1, 1, 1, 1, 1};
    static constexpr int det[4] = {1, 1, 2, 1}, dist[3] = {1, 1, 0};
};
struct AtRun {  // the same as run
    static constexpr int b1[5] = {2, 2, 1, 0, 1}, b1w[5] = {2, 2, 1, 0, 1};
    static constexpr int b2[5] = {1, 1, 1, 0, 0}, b3[5] = {2, 2, 2, 0, 1};
    static constexpr int det[4] = {1, 1, 1, 2}, dist[3] = {2, 1, 0};
};
struct AtSos {  // where exact zeros are resolved
    static constexpr int b1[5] = {1, 1, 1, 0, 0}, b1w[5] = {1, 1, 1, 0, 0};
    static constexpr int b2[5] = {0, 0, 0, 0, 0}, b3[5] = {2, 2, 2, 0, 0};
    static constexpr int det[4] = {2, 1, 2, 2}, dist[3] = {1, 1, 1};
    static constexpr int dab = 2;
};
struct AtScan {  // the empty-orthosphere test
    static constexpr int dab = 1;
};

// (|a|^2 - r_a^2) - (|b|^2 - r_b^2), summed as the reference does
template <int X, int Y, int Z, int P, int Q>
__device__ __forceinline__ float power_diff(const Ball a, const Ball b) {
    const float s = add_rn(add_rn(diff<X>(a.x, a.x, b.x, b.x), diff<Y>(a.y, a.y, b.y, b.y)),
                           diff<Z>(a.z, a.z, b.z, b.z));
    return plus<Q>(minus<P>(s, a.r, a.r), b.r, b.r);
}
#define PAC_POWER_DIFF(F, a, b) power_diff<F[0], F[1], F[2], F[3], F[4]>(a, b)

// u^2 + v^2 + w^2 - r^2
template <class F>
__device__ __forceinline__ float power(float u, float v, float w, float r) {
    return minus<F::dist[2]>(plus<F::dist[1]>(sum<F::dist[0]>(u, u, v, v), w, w), r, r);
}

// p0 q0 + p1 q1 + p2 q2 - p3 q3 - p4 q4 - p5 q5
template <int M>
__device__ __forceinline__ float six(float p0, float q0, float p1, float q1, float p2, float q2,
                                     float p3, float q3, float p4, float q4, float p5, float q5) {
    return minus<1>(minus<1>(minus<1>(plus<1>(sum<M>(p0, q0, p1, q1), p2, q2), p3, q3), p4, q4), p5, q5);
}

// Cramer's determinants of the rows (a_k1, a_k2, a_k3 | b_k) (LD:325-338, 569-576)
struct Cramer {
    float D, X, Y, Z;
};
template <class F>
__device__ __forceinline__ Cramer cramer(float a11, float a12, float a13, float b1, float a21,
                                         float a22, float a23, float b2, float a31, float a32,
                                         float a33, float b3) {
    Cramer c;
    c.D = six<F::det[0]>(mul_rn(a11, a22), a33, mul_rn(a12, a23), a31, mul_rn(a13, a21), a32,
                         mul_rn(a13, a22), a31, mul_rn(a12, a21), a33, mul_rn(a11, a23), a32);
    c.X = six<F::det[1]>(mul_rn(b1, a22), a33, mul_rn(a12, a23), b3, mul_rn(a13, b2), a32,
                         mul_rn(a13, a22), b3, mul_rn(a12, b2), a33, mul_rn(b1, a23), a32);
    c.Y = six<F::det[2]>(mul_rn(a11, b2), a33, mul_rn(b1, a23), a31, mul_rn(a13, a21), b3,
                         mul_rn(a13, b2), a31, mul_rn(b1, a21), a33, mul_rn(a11, a23), b3);
    c.Z = six<F::det[3]>(mul_rn(a11, a22), b3, mul_rn(a12, b2), a31, mul_rn(b1, a21), a32,
                         mul_rn(b1, a22), a31, mul_rn(a12, a21), b3, mul_rn(a11, b2), a32);
    return c;
}

// ---------------------------------------------------------------- formulas
// markRealEdges: LD:173-189 (upstream) / PLAIN:209-229 (plain-xmp).
template <int V>
__device__ __forceinline__ bool edge_alpha(const Ball a1, const Ball a2, float alpha) {
    float a = a1.x - a2.x;
    float b = a1.y - a2.y;
    float c = a1.z - a2.z;
    float d = PAC_POWER_DIFF(AtEdge::b1, a1, a2);
    d = mul_rn(d, 0.5f);
    // (contracted: d was fused as its half, which rounds a a1.x)
    float t = minus<1>(minus<1>(sub_rn(d, mul_rn(a, a1.x)), b, a1.y), c, a1.z);
    float l = plus<1>(sum<1>(a, a, b, b), c, c);
    if (V == kUpstream) {
        float currentDist = sub_rn(mul_rn(t, t) / l, mul_rn(a1.r, a1.r));
        return le_as_double(currentDist, alpha);
    } else {
        float currentDistTerm = diff<1>(t, t, mul_rn(a1.r, a1.r), l);
        return currentDistTerm <= ((double)alpha + 0.0) * l;
    }
}

// markRealTriangles: LD:308-347 (upstream) / PLAIN:320-370 (plain-xmp).
// Returns the alpha mark and writes the orthosphere (X, Y, Z, power).
template <int V, class F = AtAttach<V>>
__device__ __forceinline__ bool tri_alpha(const Ball a1, const Ball a2, const Ball a3,
                                          float alpha, float4 &ortho) {
    float a11 = a1.x - a2.x;
    float a12 = a1.y - a2.y;
    float a13 = a1.z - a2.z;
    float b1 = PAC_POWER_DIFF(F::b1, a1, a2);
    if (V == kUpstream) b1 = mul_rn(b1, 0.5f);
    float a21 = a2.x - a3.x;
    float a22 = a2.y - a3.y;
    float a23 = a2.z - a3.z;
    float b2 = PAC_POWER_DIFF(F::b2, a2, a3);
    if (V == kUpstream) b2 = mul_rn(b2, 0.5f);
    float a31 = diff<1>(a2.y - a1.y, a3.z - a1.z, a3.y - a1.y, a2.z - a1.z);
    float a32 = diff<1>(a2.z - a1.z, a3.x - a1.x, a3.z - a1.z, a2.x - a1.x);
    float a33 = diff<1>(a2.x - a1.x, a3.y - a1.y, a3.x - a1.x, a2.y - a1.y);
    float b3 = sum<1>(a31, a1.x, a32, a1.y);
    if (V == kUpstream)
        b3 = plus<1>(b3, a33, a1.z);
    else
        b3 = add_rn(b3, mul_rn(mul_rn(a33, a1.z), 2.0f));
    const Cramer c = cramer<F>(a11, a12, a13, b1, a21, a22, a23, b2, a31, a32, a33, b3);
    if (V == kUpstream) {
        float X = c.X / c.D;
        float Y = c.Y / c.D;
        float Z = c.Z / c.D;
        float dist = power<F>(a1.x - X, a1.y - Y, a1.z - Z, a1.r);
        ortho = make_float4(X, Y, Z, dist);
        return le_as_double(dist, alpha);
    } else {
        float D = mul_rn(c.D, 2.0f);
        float u = minus<1>(c.X, a1.x, D), v = minus<1>(c.Y, a1.y, D), w = minus<1>(c.Z, a1.z, D);
        float dist = plus<F::dist[1]>(sum<F::dist[0]>(u, u, v, v), w, w);
        dist = minus<F::dist[2]>(dist, mul_rn(mul_rn(a1.r, a1.r), D), D);
        bool mark = dist <= ((double)alpha + 0.0) * D * D;
        ortho = make_float4(c.X / D, c.Y / D, c.Z / D, dist / mul_rn(D, D));
        return mark;
    }
}

// markRealTets: LD:542-590 (the same in both binaries).  wide: a1 has more
// than 64 upper neighbours.
template <class F = AtEnum>
__device__ __forceinline__ bool tet_alpha(const Ball a1, const Ball a2, const Ball a3,
                                          const Ball a4, float alpha, float4 &ortho, bool wide = false) {
    float a11 = a1.x - a2.x;
    float a12 = a1.y - a2.y;
    float a13 = a1.z - a2.z;
    float b1 = PAC_POWER_DIFF(F::b1, a1, a2);
    if (kFused && wide) b1 = PAC_POWER_DIFF(F::b1w, a1, a2);
    b1 = mul_rn(b1, 0.5f);
    float a21 = a2.x - a3.x;
    float a22 = a2.y - a3.y;
    float a23 = a2.z - a3.z;
    float b2 = mul_rn(PAC_POWER_DIFF(F::b2, a2, a3), 0.5f);
    float a31 = a3.x - a4.x;
    float a32 = a3.y - a4.y;
    float a33 = a3.z - a4.z;
    float b3 = mul_rn(PAC_POWER_DIFF(F::b3, a3, a4), 0.5f);
    const Cramer c = cramer<F>(a11, a12, a13, b1, a21, a22, a23, b2, a31, a32, a33, b3);
    if (c.D == 0.0) {
        ortho = make_float4(0, 0, 0, 0);
        return true;
    }
    float X = c.X / c.D;
    float Y = c.Y / c.D;
    float Z = c.Z / c.D;
    float dist = power<F>(a2.x - X, a2.y - Y, a2.z - Z, a2.r);
    ortho = make_float4(X, Y, Z, dist);
    return le_as_double(dist, alpha);
}

// orient3d determinant (PRED:2015-2045); the error bound there is dead.  M: its
// minors (in the empty-orthosphere test they are rounded apart where the
// window's centre names no cell).
template <int M = 1>
__device__ __forceinline__ float orient3d(const float *pa, const float *pb, const float *pc,
                                          const float *pd) {
    float adx = pa[0] - pd[0];
    float bdx = pb[0] - pd[0];
    float cdx = pc[0] - pd[0];
    float ady = pa[1] - pd[1];
    float bdy = pb[1] - pd[1];
    float cdy = pc[1] - pd[1];
    float adz = pa[2] - pd[2];
    float bdz = pb[2] - pd[2];
    float cdz = pc[2] - pd[2];
    float bc = diff<M>(bdx, cdy, cdx, bdy);
    float ca = diff<M>(cdx, ady, adx, cdy);
    float ab = diff<M>(adx, bdy, bdx, ady);
    return plus<1>(sum<1>(adz, bc, bdz, ca), cdz, ab);
}

// insphere_w determinant (PRED:4250-4322) from the differences of the weights;
// the error bound there is dead.
template <class F>
__device__ __forceinline__ float insphere_d(const float *pa, const float *pb, const float *pc,
                                            const float *pd, const float *pe, float aew, float bew,
                                            float cew, float dew) {
    float aex = pa[0] - pe[0];
    float bex = pb[0] - pe[0];
    float cex = pc[0] - pe[0];
    float dex = pd[0] - pe[0];
    float aey = pa[1] - pe[1];
    float bey = pb[1] - pe[1];
    float cey = pc[1] - pe[1];
    float dey = pd[1] - pe[1];
    float aez = pa[2] - pe[2];
    float bez = pb[2] - pe[2];
    float cez = pc[2] - pe[2];
    float dez = pd[2] - pe[2];
    float ab = diff<1>(aex, bey, bex, aey);
    float bc = diff<1>(bex, cey, cex, bey);
    float cd = diff<1>(cex, dey, dex, cey);
    float da = diff<1>(dex, aey, aex, dey);
    float ac = diff<1>(aex, cey, cex, aey);
    float bd = diff<1>(bex, dey, dex, bey);
    float abc = plus<1>(diff<1>(aez, bc, bez, ac), cez, ab);
    float bcd = plus<1>(diff<1>(bez, cd, cez, bd), dez, bc);
    float cda = plus<1>(sum<1>(cez, da, dez, ac), aez, cd);
    float dab = plus<1>(sum<F::dab>(dez, ab, aez, bd), bez, da);
    float alift = plus<1>(sum<1>(aex, aex, aey, aey), aez, aez);
    float blift = plus<1>(sum<1>(bex, bex, bey, bey), bez, bez);
    float clift = plus<1>(sum<1>(cex, cex, cey, cey), cez, cez);
    float dlift = plus<1>(sum<1>(dex, dex, dey, dey), dez, dez);
    float alw = sub_rn(alift, aew);
    float blw = sub_rn(blift, bew);
    float clw = sub_rn(clift, cew);
    float dlw = sub_rn(dlift, dew);
    return add_rn(diff<1>(dlw, abc, clw, dab), diff<1>(blw, cda, alw, bcd));
}
template <class F = AtScan>
__device__ __forceinline__ float insphere_w(const float *pa, const float *pb, const float *pc,
                                            const float *pd, const float *pe, float wa,
                                            float wb, float wc, float wd, float we) {
    return insphere_d<F>(pa, pb, pc, pd, pe, sub_rn(wa, we), sub_rn(wb, we), sub_rn(wc, we),
                         sub_rn(wd, we));
}

// Attachment test of checkDanglingTris / checkDanglingEdges
// (LD:825-829, 964-968): true when ball e is at least as close (in power
// distance) to (px, py, pz) as the simplex's own balls.
__device__ __forceinline__ bool attached(const Ball e, float px, float py, float pz,
                                         float currentDist) {
    return le_as_double(power<AtPower>(e.x - px, e.y - py, e.z - pz, e.r), currentDist);
}

// Foot of the radical plane of an edge and its power (LD:936-949).
__device__ __forceinline__ void edge_foot(const Ball a1, const Ball a2, float &px, float &py,
                                          float &pz, float &currentDist) {
    float a = a1.x - a2.x;
    float b = a1.y - a2.y;
    float c = a1.z - a2.z;
    float d = mul_rn(PAC_POWER_DIFF(AtFoot::b1, a1, a2), 0.5f);
    float t = minus<1>(minus<1>(sub_rn(d, mul_rn(a, a1.x)), b, a1.y), c, a1.z) /
              plus<1>(sum<1>(a, a, b, b), c, c);
    px = plus<1>(a1.x, a, t);
    py = plus<1>(a1.y, b, t);
    pz = plus<1>(a1.z, c, t);
    currentDist = power<AtFoot>(a1.x - px, a1.y - py, a1.z - pz, a1.r);
}

// Cell coordinate of a point (LD:72-74, 621-623): float subtract, IEEE
// divide, truncating conversion (NaN -> 0, saturating).
__device__ __forceinline__ int cell_coord(float p, float lo, float step) {
    return (int)((p - lo) / step);
}

}  // namespace pac
