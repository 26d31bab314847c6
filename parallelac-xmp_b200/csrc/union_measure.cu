// union_measure.cu -- volume and surface area of a union of balls by
// inclusion-exclusion over a fixed complex, with the gradient with respect
// to every centre and radius.
//
//   vol(U)  = sum_s (-1)^dim(s) vol(B_s),       B_s = intersection of the balls of s
//   area(U) = sum_s (-1)^dim(s) area(dB_s)
// summed over the vertices, edges, triangles and tetrahedra of the complex
// (Edelsbrunner 1995: exact when the complex is the dual complex of the
// balls, i.e. the weighted alpha complex with radii sqrt(r^2 + alpha)).
//
// Per simplex, the boundary of B_s is a set of spherical patches F_i (the
// part of sphere i inside the other balls of s), bounded by circle arcs
// ("ridges") that meet at triple points.  For every patch the kernel
// computes its area A_i (Gauss-Bonnet: R^2 (2 pi - sum_arcs phi cos(theta)
// - sum_corners exterior angle)) and its vector area M_i (half the loop
// integral of p x dp); the volume follows from the divergence theorem,
// vol = 1/3 sum_i (R_i A_i + (c_i - x0) . M_i).
//
// Gradient (the adjoint), from the first variation of volume and area:
//   d vol  / d R_i = A_i                 d vol  / d c_i = M_i
//   d area / d R_i = 2 A_i / R_i + sum_j r_ij l_ij
//   d area / d c_i = 2 M_i / R_i + sum_j r_ij N_ij
// where l_ij is the length of the ridge on circle ij, N_ij the integral of
// sphere i's unit normal along it, and r_ij = (d_ij^2 - (R_i - R_j)^2) /
// (2 d_ij rho_ij) the rate at which a ridge of two spheres at distance d_ij
// (circle radius rho_ij) changes the area per unit normal motion.  Every
// term is accumulated with the simplex's sign, so the result is the exact
// gradient of the inclusion-exclusion sum for the complex held fixed.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>

#include "pac_internal.h"

namespace pac_union {

struct V3 {
    double x, y, z;
};
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 operator*(double s, V3 a) { return {s * a.x, s * a.y, s * a.z}; }
__device__ __forceinline__ double dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

constexpr double kPi = 3.14159265358979323846;

// circle of spheres i and j
struct Circle {
    V3 u;          // unit axis from c_i towards c_j
    double d;      // centre distance
    double ti, tj; // signed distance of the circle's plane from c_i along u, from c_j along -u
    double rho;    // circle radius
    double g;      // (d^2 - (R_i - R_j)^2) / (2 d) = r rho
};
__device__ __forceinline__ Circle make_circle(V3 a, double Ri, double Rj) {  // a = c_j - c_i
    Circle C;
    C.d = sqrt(dot(a, a));
    const double h = 0.5 / C.d;
    C.u = (2 * h) * a;
    C.ti = (C.d * C.d + Ri * Ri - Rj * Rj) * h;
    C.tj = C.d - C.ti;
    C.rho = sqrt(fmax(Ri * Ri - C.ti * C.ti, 0.0));
    C.g = (C.d * C.d - (Ri - Rj) * (Ri - Rj)) * h;
    return C;
}

// the two points common to spheres i, j, m: x +- eta nh (x relative to c_i).
// A complex decided in single precision holds triples whose spheres just miss
// each other: eta is then 0, or with miss the negative square R^2 - |x|^2.
struct Triple {
    V3 x, nh;
    double eta, nl;  // nl = |(c_j - c_i) x (c_m - c_i)|
};
__device__ __forceinline__ Triple make_triple(V3 a, V3 b, double Ri, double Rj, double Rm, bool miss, bool &missing) {
    // a = c_j - c_i, b = c_m - c_i; x in the plane of the centres with equal power
    V3 n = cross(a, b);
    double nn = dot(n, n);
    double a1 = 0.5 * (dot(a, a) + Ri * Ri - Rj * Rj);
    double a2 = 0.5 * (dot(b, b) + Ri * Ri - Rm * Rm);
    Triple T;
    T.x = (1.0 / nn) * (a1 * cross(b, n) + a2 * cross(n, a));
    T.nl = sqrt(nn);
    T.nh = (1.0 / T.nl) * n;
    const double e2 = Ri * Ri - dot(T.x, T.x);
    missing |= e2 < 0;
    T.eta = miss && e2 < 0 ? e2 : sqrt(fmax(e2, 0.0));
    return T;
}

struct Terms {
    double V;
    double A[4];
    V3 M[4];
    double rl[4];  // sum_j r_ij l_ij
    V3 rN[4];      // sum_j r_ij N_ij
};

// Patch quantities of K balls, centres relative to c[0].
//
// A ridge is an arc of the circle of two spheres; both spheres share it, one
// running it backwards.  Its ends are triple points, so the chord between
// them needs no sine or cosine: with w the unit direction from the circle's
// axis u to the third centre, the arc inside that ball ends at the triple
// points, along +-u x w = +-nh of the triple.  The exterior angle of patch i at
// a triple point is atan2(eta R_i |u_ij x u_im|, R_i^2 u_ij . u_im - t_ij t_im), the same
// at both points.  Where the three spheres just miss each other, both points
// are x, outside the spheres by eps R^2 = |x|^2 - R^2: the arcs vanish or close
// at the foot of x on the circle, and the angle between the circles' tangent
// directions there is atan2(eps R^2 |u_ij x u_im|, R^2 u_ij . u_im - t_ij t_im (1 - eps)).
// With K a template parameter every index is static, so what the
// registers hold stays there (at 128 a thread, 0.2 KB of a triangle and 1.5 KB
// of a tetrahedron spill: see k_union).  One ordered pair at a time, with
// arrays indexed at run time (local memory), four sines and cosines, three
// atan2 and normalised tangents per pair: 1.13 ms at 100,008 balls for volume,
// area and gradients, now 0.58; bound by FP64 latency then and now (at 40,000
// balls the tetrahedra issue on 36 % of the cycles with 15 of 64 warps).
//
// Returns whether three of the spheres miss each other: the terms are then right
// only with miss.
template <int K>
__device__ __forceinline__ bool simplex_terms(const V3 *c, const double *R, bool miss, Terms &T) {
    bool missing = false;
#pragma unroll
    for (int i = 0; i < K; i++) {
        T.A[i] = 0;
        T.M[i] = {0, 0, 0};
        T.rl[i] = 0;
        T.rN[i] = {0, 0, 0};
    }
    if constexpr (K == 1) {
        T.V = 4.0 / 3.0 * kPi * R[0] * R[0] * R[0];
        T.A[0] = 4 * kPi * R[0] * R[0];
    } else if constexpr (K == 2) {
        const Circle C = make_circle(c[1] - c[0], R[0], R[1]);
        double h0 = R[0] - C.ti, h1 = R[1] - C.tj;
        T.V = kPi * h0 * h0 * (3 * R[0] - h0) / 3 + kPi * h1 * h1 * (3 * R[1] - h1) / 3;
        T.A[0] = 2 * kPi * R[0] * h0;
        T.A[1] = 2 * kPi * R[1] * h1;
        double disk = kPi * C.rho * C.rho;
        T.M[0] = disk * C.u;
        T.M[1] = -disk * C.u;
        // full circle: l = 2 pi rho, N_i = t_i l u_i / R_i
        T.rl[0] = T.rl[1] = C.g * 2 * kPi;
        T.rN[0] = (C.g * 2 * kPi * C.ti / R[0]) * C.u;
        T.rN[1] = (C.g * 2 * kPi * C.tj / R[1]) * (-1.0 * C.u);
    } else {
        // pairs (i, j), i < j, in lexicographic order; the triples by their
        // missing ball (K = 3: one), each seen from its first ball
        constexpr int kPairs = K * (K - 1) / 2, kTriples = K == 3 ? 1 : 4;
        constexpr int PI[6] = {0, 0, K == 3 ? 1 : 0, 1, 1, 2}, PJ[6] = {1, 2, K == 3 ? 2 : 3, 2, 3, 3};
        constexpr int TA[4] = {K == 3 ? 0 : 1, 0, 0, 0}, TB[4] = {K == 3 ? 1 : 2, 2, 1, 1},
                      TC[4] = {K == 3 ? 2 : 3, 3, 3, 2};
        Circle C[kPairs];
        Triple P[kTriples];
#pragma unroll
        for (int e = 0; e < kPairs; e++) C[e] = make_circle(c[PJ[e]] - c[PI[e]], R[PI[e]], R[PJ[e]]);
#pragma unroll
        for (int f = 0; f < kTriples; f++)
            P[f] = make_triple(c[TB[f]] - c[TA[f]], c[TC[f]] - c[TA[f]], R[TA[f]], R[TB[f]], R[TC[f]], miss,
                               missing);
        double gb[K];  // sum of arc angle times cosine, and the exterior angles
#pragma unroll
        for (int i = 0; i < K; i++) gb[i] = 0;
#pragma unroll
        for (int e = 0; e < kPairs; e++) {
            const int i = PI[e], j = PJ[e];
            const V3 u = C[e].u, o = c[i] + C[e].ti * u;  // the circle's centre
            // the arc inside each other ball m: ends at E[..][0] (start) and
            // E[..][1] about u, half-width b
            V3 w[K - 2], E[K - 2][2];
            double b[K - 2];
            int at = 0;
#pragma unroll
            for (int m = 0; m < K; m++) {
                if (m == i || m == j) continue;
                const int f = K == 3 ? 0 : 6 - i - j - m;
                // nh points along u x (c_m - c_i) when (i, j, m) is an even
                // order of the triple's (TA, TB, TC)
                const double s = (i < m && m < j) ? -1.0 : 1.0;
                const V3 nh = s * P[f].nh;
                const V3 x = c[TA[f]] + P[f].x - o;
                w[at] = cross(nh, u);
                const double xw = dot(x, w[at]);
                b[at] = atan2(miss ? fmax(P[f].eta, 0.0) : P[f].eta, xw);
                E[at][0] = x - P[f].eta * nh;
                E[at][1] = x + P[f].eta * nh;
                if (miss && P[f].eta < 0) E[at][0] = E[at][1] = (xw < 0 ? -C[e].rho : C[e].rho) * w[at];
                at++;
            }
            double phi = 2 * b[0];
            V3 chord = E[0][1] - E[0][0];
            if constexpr (K == 4) {
                // overlap of [-b0, b0] with [dl - b1, dl + b1] on the circle
                const double dl = atan2(dot(cross(w[0], w[1]), u), dot(w[1], w[0]));
                double best = 0;
                V3 qs = {0, 0, 0}, qe = {0, 0, 0};
#pragma unroll
                for (int t = -1; t <= 1; t++) {
                    const double l1 = dl - b[1] + 2 * kPi * t, h1 = dl + b[1] + 2 * kPi * t;
                    const double l2 = fmax(-b[0], l1), h2 = fmin(b[0], h1);
                    if (h2 - l2 > best) {
                        best = h2 - l2;
                        qs = l1 > -b[0] ? E[1][0] : E[0][0];
                        qe = h1 < b[0] ? E[1][1] : E[0][1];
                    }
                }
                phi = best;
                chord = qe - qs;
            }
            const V3 uc = cross(u, chord);
            const V3 disk = (0.5 * C[e].rho * C[e].rho * phi) * u;
            gb[i] += phi * C[e].ti / R[i];
            gb[j] += phi * C[e].tj / R[j];
            T.M[i] = T.M[i] + disk + (0.5 * C[e].ti) * uc;
            T.M[j] = T.M[j] - disk + (0.5 * C[e].tj) * uc;
            T.rl[i] += C[e].g * phi;
            T.rl[j] += C[e].g * phi;
            T.rN[i] = T.rN[i] + (C[e].g / R[i]) * ((C[e].ti * phi) * u - uc);
            T.rN[j] = T.rN[j] - (C[e].g / R[j]) * ((C[e].tj * phi) * u + uc);
        }
        // exterior angles: each triple's, for each of its balls; both points
        // when K = 3, the one inside the fourth ball when K = 4
#pragma unroll
        for (int e = 0; e < kPairs; e++)
#pragma unroll
            for (int g = e + 1; g < kPairs; g++) {
                const int i = PI[e] == PI[g] || PI[e] == PJ[g] ? PI[e]
                              : PJ[e] == PI[g] || PJ[e] == PJ[g] ? PJ[e] : -1;
                if (i < 0) continue;
                const int j = PI[e] + PJ[e] - i, m = PI[g] + PJ[g] - i;
                const int f = K == 3 ? 0 : 6 - i - j - m;
                const double te = i < j ? C[e].ti : C[e].tj, tg = i < m ? C[g].ti : C[g].tj;
                const double cu = ((i < j) == (i < m) ? 1.0 : -1.0) * dot(C[e].u, C[g].u);
                const double eta = P[f].eta;
                double y = eta * R[i], tt = te * tg;
                if (miss && eta < 0) y = -eta, tt += tt * eta / (R[i] * R[i]);
                const double x = atan2(y * P[f].nl, (R[i] * R[i] * cu - tt) * (C[e].d * C[g].d));
                gb[i] += K == 3 ? 2 * x : x;
            }
        V3 x0 = {0, 0, 0};
#pragma unroll
        for (int i = 0; i < K; i++) x0 = x0 + c[i];
        x0 = (1.0 / K) * x0;
        double vol = 0;
#pragma unroll
        for (int i = 0; i < K; i++) {
            T.A[i] = R[i] * R[i] * (2 * kPi - gb[i]);
            vol += R[i] * T.A[i] + dot(c[i] - x0, T.M[i]);
        }
        T.V = vol / 3.0;
    }
    return missing;
}

// double-double accumulation (TwoSum), so the totals do not depend on the
// order in which the blocks finish: each block reduces its simplices in a
// fixed shuffle/shared-memory order and writes one (hi, lo) pair; one block
// then sums the pairs in index order.
__device__ __forceinline__ void dd_add(double &hi, double &lo, double bh, double bl) {
    double s = hi + bh;
    double v = s - hi;
    double e = (hi - (s - v)) + (bh - v);
    e += lo + bl;
    hi = s + e;
    lo = e - (hi - s);
}

// Sums v over the run of consecutive lanes of act (a prefix of the warp, all of
// which call) with the same id, in lane order; true for the run's first lane, which then holds the sum.  The lists
// group simplices by their first vertex (in the complex's own order runs of 5
// to 11), whose atomics, a quarter to a half of all, shrink by that much:
// 224 us of atomics for 2.3 M simplices without it.
__device__ __forceinline__ bool run_sum(unsigned act, uint32_t id, double (&v)[8]) {
    const int lane = threadIdx.x & 31;
    const uint32_t left = __shfl_up_sync(act, id, 1);
    const bool head = lane == 0 || left != id;
    const unsigned heads = __ballot_sync(act, head);
    // lanes up to the next head
    const unsigned above = lane == 31 ? 0u : heads & (0xfffffffeu << lane);
    const int end = above ? __ffs((int)above) - 1 : __popc(act);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const bool in = lane + o < end;
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const double x = __shfl_down_sync(act, v[t], o);
            if (in) v[t] += x;
        }
    }
    return head;
}

// one thread per simplex of K vertices, indices in idx[K * s + ...]
// (blocks per SM: four for triangles and tetrahedra, although they spill 0.2 and
// 1.5 KB at 128 registers -- two or three blocks without spills leave the
// FP64 latency uncovered: tetrahedra 354 and 304 us against 286)
template <int K>
__global__ void __launch_bounds__(128, K >= 3 ? 4 : 8) k_union(uint64_t ns, const uint32_t *idx, const double4 *balls,
                                               double4 *partial, double *dV, double *dA,
                                               int want_grad, unsigned *miss) {
    __shared__ double4 wpart[4];
    uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double vh = 0, vl = 0, ah = 0, al = 0;
    const unsigned act = __ballot_sync(0xffffffffu, s < ns);
    if (s < ns) {
        uint32_t id[K];
        V3 c[K];
        double R[K];
#pragma unroll
        for (int q = 0; q < K; q++) {
            id[q] = K == 1 ? (uint32_t)s : idx[(uint64_t)K * s + q];
            double4 b = balls[id[q]];
            R[q] = b.w;
            c[q] = {b.x, b.y, b.z};
        }
        V3 c0 = c[0];
#pragma unroll
        for (int q = 0; q < K; q++) c[q] = c[q] - c0;
        Terms T;
        const bool missing = simplex_terms<K>(c, R, false, T);
        if constexpr (K >= 3) {
            const unsigned m = __ballot_sync(act, missing);
            if ((threadIdx.x & 31) == 0) miss[4 * blockIdx.x + (threadIdx.x >> 5)] = m;
        }
        constexpr double sg = (K & 1) ? 1.0 : -1.0;
        vh = sg * T.V;
#pragma unroll
        for (int q = 0; q < K; q++) dd_add(ah, al, sg * T.A[q], 0.0);
        if (want_grad) {
#pragma unroll
            for (int q = 0; q < K; q++) {
                double *gv = dV + 4 * (uint64_t)id[q], *ga = dA + 4 * (uint64_t)id[q];
                const double inv = 2.0 / R[q];
                double v[8] = {sg * T.M[q].x, sg * T.M[q].y, sg * T.M[q].z, sg * T.A[q],
                               sg * (inv * T.M[q].x + T.rN[q].x), sg * (inv * T.M[q].y + T.rN[q].y),
                               sg * (inv * T.M[q].z + T.rN[q].z), sg * (inv * T.A[q] + T.rl[q])};
                bool lead = true;
                if constexpr (K > 1)
                    if (q == 0) lead = run_sum(act, id[0], v);
                if (lead) {
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        atomicAdd(gv + t, v[t]);
                        atomicAdd(ga + t, v[4 + t]);
                    }
                }
            }
        }
    }
    if (K >= 3 && !act && (threadIdx.x & 31) == 0) miss[4 * blockIdx.x + (threadIdx.x >> 5)] = 0;
    for (int o = 16; o; o >>= 1) {
        double h1 = __shfl_xor_sync(0xffffffffu, vh, o), l1 = __shfl_xor_sync(0xffffffffu, vl, o);
        double h2 = __shfl_xor_sync(0xffffffffu, ah, o), l2 = __shfl_xor_sync(0xffffffffu, al, o);
        dd_add(vh, vl, h1, l1);
        dd_add(ah, al, h2, l2);
    }
    if ((threadIdx.x & 31) == 0) wpart[threadIdx.x >> 5] = make_double4(vh, vl, ah, al);
    __syncthreads();
    if (threadIdx.x == 0) {
        double4 r = wpart[0];
        for (int w = 1; w < 4; w++) {
            dd_add(r.x, r.y, wpart[w].x, wpart[w].y);
            dd_add(r.z, r.w, wpart[w].z, wpart[w].w);
        }
        partial[blockIdx.x] = r;
    }
}

// Corrects the terms of the simplices whose spheres just miss each other, one in a
// million or fewer: a thread per block of k_union reads its four masks and adds,
// for each bit, the right terms less those that were added.  In k_union itself
// these cases cost every simplex registers (100,008 balls: 590 to 650 us instead
// of 560), here 575.
template <int K>
__device__ void correct(const uint32_t *id, const double4 *balls, double4 &sum, double *dV, double *dA,
                        int want_grad) {
    V3 c[K];
    double R[K];
    const double4 b0 = balls[id[0]];
#pragma unroll
    for (int q = 0; q < K; q++) {
        const double4 b = balls[id[q]];
        R[q] = b.w;
        c[q] = {b.x - b0.x, b.y - b0.y, b.z - b0.z};
    }
#pragma unroll 1
    for (int w = 0; w < 2; w++) {
        Terms T;
        simplex_terms<K>(c, R, w != 0, T);
        const double sg = ((K & 1) != 0) == (w != 0) ? 1.0 : -1.0;
        dd_add(sum.x, sum.y, sg * T.V, 0.0);
#pragma unroll
        for (int q = 0; q < K; q++) dd_add(sum.z, sum.w, sg * T.A[q], 0.0);
        if (!want_grad) continue;
#pragma unroll
        for (int q = 0; q < K; q++) {
            double *gv = dV + 4 * (uint64_t)id[q], *ga = dA + 4 * (uint64_t)id[q];
            const double inv = 2.0 / R[q];
            atomicAdd(gv, sg * T.M[q].x), atomicAdd(ga, sg * (inv * T.M[q].x + T.rN[q].x));
            atomicAdd(gv + 1, sg * T.M[q].y), atomicAdd(ga + 1, sg * (inv * T.M[q].y + T.rN[q].y));
            atomicAdd(gv + 2, sg * T.M[q].z), atomicAdd(ga + 2, sg * (inv * T.M[q].z + T.rN[q].z));
            atomicAdd(gv + 3, sg * T.A[q]), atomicAdd(ga + 3, sg * (inv * T.A[q] + T.rl[q]));
        }
    }
}

// miss: of the bt blocks of triangles, then of the bq of tetrahedra, as partial
__global__ void __launch_bounds__(128) k_union_miss(uint32_t bt, const uint32_t *tris, uint32_t bq, const uint32_t *tets,
                                                    const double4 *balls, double4 *partial, double *dV, double *dA,
                                                    int want_grad, const unsigned *miss) {
    const uint32_t b = blockIdx.x * 128 + threadIdx.x;
    if (b >= bt + bq) return;
    for (int w = 0; w < 4; w++)
        for (unsigned m = miss[4 * (uint64_t)b + w]; m; m &= m - 1) {
            const uint64_t at = 32 * w + (__ffs((int)m) - 1);
            if (b < bt)
                correct<3>(tris + 3 * (128 * (uint64_t)b + at), balls, partial[b], dV, dA, want_grad);
            else
                correct<4>(tets + 4 * (128 * (uint64_t)(b - bt) + at), balls, partial[b], dV, dA, want_grad);
        }
}

__global__ void __launch_bounds__(1024) k_union_total(const double4 *partial, uint64_t np, double *out) {
    __shared__ double4 sp[32];
    double vh = 0, vl = 0, ah = 0, al = 0;
    for (uint64_t i = threadIdx.x; i < np; i += 1024) {
        double4 r = partial[i];
        dd_add(vh, vl, r.x, r.y);
        dd_add(ah, al, r.z, r.w);
    }
    // a fixed tree: lanes by shuffle, then the 32 warps in order
    for (int o = 16; o; o >>= 1) {
        const double h1 = __shfl_xor_sync(0xffffffffu, vh, o), l1 = __shfl_xor_sync(0xffffffffu, vl, o);
        const double h2 = __shfl_xor_sync(0xffffffffu, ah, o), l2 = __shfl_xor_sync(0xffffffffu, al, o);
        dd_add(vh, vl, h1, l1);
        dd_add(ah, al, h2, l2);
    }
    if ((threadIdx.x & 31) == 0) sp[threadIdx.x >> 5] = make_double4(vh, vl, ah, al);
    __syncthreads();
    if (threadIdx.x == 0) {
        double4 r = sp[0];
        for (int t = 1; t < 32; t++) {
            dd_add(r.x, r.y, sp[t].x, sp[t].y);
            dd_add(r.z, r.w, sp[t].z, sp[t].w);
        }
        out[0] = r.x + r.y;
        out[1] = r.z + r.w;
    }
}

// All kernels of one measure on stream s: counts and lists by vertices less one,
// partial and miss (four words) per block of 128.  Returns the launches.
inline int launch(cudaStream_t s, const uint64_t (&counts)[4], const uint32_t *const (&lists)[4],
                  const double4 *balls, double4 *partial, unsigned *miss, double *dV, double *dA, int want_grad,
                  double *totals) {
    uint32_t blocks[4], off = 0;
    int launches = 1;
    for (int k = 0; k < 4; k++) {
        const uint32_t nb = blocks[k] = (uint32_t)((counts[k] + 127) / 128);
        if (!nb) continue;
        const uint64_t ns = counts[k];
        const uint32_t *idx = lists[k];
        double4 *p = partial + off;
        unsigned *m = miss + 4 * (uint64_t)off;
        switch (k) {
            case 0: k_union<1><<<nb, 128, 0, s>>>(ns, idx, balls, p, dV, dA, want_grad, m); break;
            case 1: k_union<2><<<nb, 128, 0, s>>>(ns, idx, balls, p, dV, dA, want_grad, m); break;
            case 2: k_union<3><<<nb, 128, 0, s>>>(ns, idx, balls, p, dV, dA, want_grad, m); break;
            default: k_union<4><<<nb, 128, 0, s>>>(ns, idx, balls, p, dV, dA, want_grad, m);
        }
        off += nb;
        launches++;
    }
    if (const uint32_t nb = blocks[2] + blocks[3]) {
        const uint32_t at = blocks[0] + blocks[1];
        k_union_miss<<<(nb + 127) / 128, 128, 0, s>>>(blocks[2], lists[2], blocks[3], lists[3], balls, partial + at, dV,
                                                      dA, want_grad, miss + 4 * (uint64_t)at);
        launches++;
    }
    k_union_total<<<1, 1024, 0, s>>>(partial, off, totals);
    return launches;
}

}  // namespace pac_union

namespace pac {

// Runs the measure on device-resident balls and lists.  Gradients go to the
// device buffers d_dV / d_dA (n x 4 each) when given; vol/area to the host.
int union_measure_device(Ctx &ctx, const double4 *d_balls, uint32_t n, const uint32_t *d_edges,
                         uint64_t ne, const uint32_t *d_tris, uint64_t nt, const uint32_t *d_tets,
                         uint64_t nq, double *vol, double *area, double *d_dV, double *d_dA,
                         float *ms) {
    cudaStream_t s = ctx.stream;
    double *acc = ctx.arena.alloc_n<double>(2);
    bool grad = d_dV || d_dA;
    double *dV = d_dV, *dA = d_dA;
    if (grad && !dV) dV = ctx.arena.alloc_n<double>(4 * (size_t)n);
    if (grad && !dA) dA = ctx.arena.alloc_n<double>(4 * (size_t)n);
    const uint32_t *lists[4] = {nullptr, d_edges, d_tris, d_tets};
    uint64_t counts[4] = {n, ne, nt, nq};
    uint64_t nblocks = 0;
    for (int k = 0; k < 4; k++) nblocks += (counts[k] + 127) / 128;
    double4 *partial = ctx.arena.alloc_n<double4>(nblocks);
    unsigned *miss = ctx.arena.alloc_n<unsigned>(4 * nblocks);
    if (!acc || !partial || !miss || (grad && (!dV || !dA))) return PAC_ERR_OOM;
    // two timing events, destroyed on every return path
    struct Events {
        cudaEvent_t e[2] = {nullptr, nullptr};
        Events() {
            cudaEventCreate(&e[0]);
            cudaEventCreate(&e[1]);
        }
        ~Events() {
            for (cudaEvent_t x : e)
                if (x) cudaEventDestroy(x);
        }
    } ev;
    cudaEvent_t e0 = ev.e[0], e1 = ev.e[1];
    cudaEventRecord(e0, s);
    if (grad) {
        cudaMemsetAsync(dV, 0, 4 * sizeof(double) * n, s);
        cudaMemsetAsync(dA, 0, 4 * sizeof(double) * n, s);
    }
    ctx.launches += pac_union::launch(s, counts, lists, d_balls, partial, miss, dV, dA, grad ? 1 : 0, acc);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        cudaStreamSynchronize(s);  // the launches that did start finish first
        return set_error(PAC_ERR_CUDA, std::string("union measure launch: ") + cudaGetErrorString(e));
    }
    cudaEventRecord(e1, s);
    double h[2];
    cudaMemcpyAsync(h, acc, sizeof(h), cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return set_error(PAC_ERR_CUDA, std::string("union measure: ") + cudaGetErrorString(e));
    if (ms) cudaEventElapsedTime(ms, e0, e1);
    if (vol) *vol = h[0];
    if (area) *area = h[1];
    return PAC_OK;
}

}  // namespace pac

// ---------------------------------------------------------------------------
// pac_union_measure_noalloc: the same measure for callers that cannot
// allocate device memory.
//
// Some callers cannot call cudaMalloc: a process whose device memory is
// reserved up front by another allocator (a framework's caching pool that
// owns nearly all of the GPU), or a latency-bound loop that cannot afford
// cudaMalloc's implicit device synchronisation.  This entry point allocates
// nothing: the caller passes the balls, the complex and the gradient buffers
// in device memory, and the only scratch -- one partial (volume, area) sum
// and one mask per block of 128 simplices and the two totals -- lives in the
// file-scope array below, which every GPU that loads this library holds until
// the process exits (3 MiB).
//
// Limit: the four simplex lists together may need at most kNoAllocBlocks
// blocks of 128, i.e. sum over vertices, edges, triangles and tetrahedra of
// ceil(count / 128) <= 65,536 (about 8.4 million simplices); larger
// complexes are rejected with PAC_ERR_CAPACITY before anything runs.
// ---------------------------------------------------------------------------
namespace {

constexpr uint64_t kNoAllocBlocks = 65536;
constexpr int kMaxDevices = 64;

// partial sums (one double4 per block), one slot for the two totals, then the
// blocks' masks (16 bytes each)
static __device__ __align__(256) double4 g_noalloc_scratch[kNoAllocBlocks + 1 + kNoAllocBlocks / 2];

std::mutex g_noalloc_mutex;
double4 *g_noalloc_ptr[kMaxDevices] = {};

// Device address of the scratch array on `device` (which must be current).
// The first call on each device looks it up with cudaGetSymbolAddress; in
// host code the array's name only stands in for the symbol.
int noalloc_scratch(int device, double4 **out) {
    if (device < 0 || device >= kMaxDevices)
        return pac::set_error(PAC_ERR_INVALID_ARG, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[device]) {
        void *ptr = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
        if (e != cudaSuccess)
            return pac::set_error(PAC_ERR_CUDA, std::string("cudaGetSymbolAddress: ") +
                                                    cudaGetErrorString(e));
        g_noalloc_ptr[device] = static_cast<double4 *>(ptr);
    }
    *out = g_noalloc_ptr[device];
    return PAC_OK;
}

}  // namespace

extern "C" int pac_union_measure_noalloc(pac_ctx *ctx, const double *d_xyzr, uint32_t n,
                                         const pac_complex *cx, double *vol, double *area,
                                         double *d_dvol, double *d_darea) {
    if (!ctx || !cx || (n && !d_xyzr))
        return pac::set_error(PAC_ERR_INVALID_ARG, "null argument");
    if ((d_dvol == nullptr) != (d_darea == nullptr))
        return pac::set_error(PAC_ERR_INVALID_ARG,
                              "pass both gradient buffers or neither (nothing is allocated)");
    // The kernels read the lists in place: they must be device lists of this
    // many balls (host lists would be dereferenced as device addresses).
    if (cx->on_device != 1)
        return pac::set_error(PAC_ERR_INVALID_ARG,
                              "pac_union_measure_noalloc needs device lists (on_device = 1)");
    if (cx->n_vertices && cx->n_vertices != n)
        return pac::set_error(PAC_ERR_INVALID_ARG, "complex and balls differ in size");
    if ((cx->n_edges && !cx->edges) || (cx->n_tris && !cx->tris) || (cx->n_tets && !cx->tets))
        return pac::set_error(PAC_ERR_INVALID_ARG, "a non-empty list has a null pointer");
    const uint32_t *lists[4] = {nullptr, cx->edges, cx->tris, cx->tets};
    const uint64_t counts[4] = {n, cx->n_edges, cx->n_tris, cx->n_tets};
    uint64_t blocks = 0;
    for (int k = 0; k < 4; k++) blocks += (counts[k] + 127) / 128;
    if (blocks > kNoAllocBlocks)
        return pac::set_error(PAC_ERR_CAPACITY,
                              "complex too large for pac_union_measure_noalloc: needs " +
                                  std::to_string(blocks) + " blocks of 128 simplices, the fixed "
                                  "scratch holds " + std::to_string(kNoAllocBlocks));
    pac::Ctx &c = pac_ctx_internal(ctx);
    cudaError_t e = cudaSetDevice(c.device);
    if (e != cudaSuccess)
        return pac::set_error(PAC_ERR_CUDA, std::string("cudaSetDevice: ") + cudaGetErrorString(e));
    double4 *scratch = nullptr;
    int rc = noalloc_scratch(c.device, &scratch);
    if (rc) return rc;
    cudaStream_t s = c.stream;
    const bool grad = d_dvol != nullptr;
    if (grad) {
        // the gradients accumulate: they must start at zero
        cudaMemsetAsync(d_dvol, 0, 4 * sizeof(double) * n, s);
        cudaMemsetAsync(d_darea, 0, 4 * sizeof(double) * n, s);
    }
    // every partial and mask slot used is written; the totals slot is written here
    double *totals = reinterpret_cast<double *>(scratch + kNoAllocBlocks);
    unsigned *miss = reinterpret_cast<unsigned *>(scratch + kNoAllocBlocks + 1);
    pac_union::launch(s, counts, lists, reinterpret_cast<const double4 *>(d_xyzr), scratch, miss, d_dvol, d_darea,
                      grad ? 1 : 0, totals);
    e = cudaGetLastError();
    if (e != cudaSuccess)
        return pac::set_error(PAC_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e));
    double h[2] = {0, 0};
    e = cudaMemcpyAsync(h, totals, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return pac::set_error(PAC_ERR_CUDA, std::string("union measure: ") + cudaGetErrorString(e));
    if (vol) *vol = h[0];
    if (area) *area = h[1];
    return PAC_OK;
}
