// pipeline.cu -- the single device pass: balls in, weighted alpha complex out.
//
// Compiled twice: with -DPAC_NS=pac_strict -fmad=false (IEEE op-by-op, the
// oracle-identical flavour) and with -DPAC_NS=pac_fma -DPAC_CONTRACTED (nvcc's
// default contraction, the flavour that follows the reference binary built
// with default flags; its fused operations are written out in refarith.cuh).
//
// Layout in HBM (n balls, molecules back to back):
//   at[n]        float4 (x, y, z, r + sol) in (molecule, cell, input index)
//                order -- the reference's stable sort by cell key
//                (AlphaComplexLargeData.cu:1174-1177)
//   orig[n]      molecule-local 0-based input index of each sorted ball
//   cellbeg[]    CSR cell ranges over the sorted balls (all molecules)
//   eoff[n+1], ER[]   alpha edges (i, ER[k]) with i < ER[k], CSR by i,
//                each row ascending (= the reference's sorted edge list)
//   loff[n+1], link[] per ball i, a deg(i) x deg(i) bit matrix over the
//                row of i in ER: bit (a, b) set <=> (i, ER[a], ER[b]) is an
//                alpha triangle.  faces[] has the same shape and marks final
//                triangles.
// Candidate tetrahedra are never stored: one kernel enumerates them from
// the link matrices, applies the alpha filter and the empty-orthosphere
// test, and writes only the survivors.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "certify.cuh"
#include "exactpred.cuh"
#include "pac_internal.h"
#include "pencil.cuh"
#include "refarith.cuh"
#include "sos.cuh"

#ifndef PAC_NS
#error "PAC_NS must name the arithmetic flavour namespace"
#endif

namespace PAC_NS {

using pac::Ball;

constexpr int kMaxDeg = 256;  // upper neighbours per ball supported
constexpr int kMaxW = kMaxDeg / 64;
constexpr unsigned kFull = 0xffffffffu;

// device-side counters (one slot each)
enum Counter {
    C_CAND_E, C_ALPHA_E, C_CAND_T, C_ALPHA_T, C_CAND_Q, C_ALPHA_Q, C_INSPHERE, C_SOS,
    C_OOB, C_SURV, C_PEND, C_MAXDEG, C_SOS_RANGE, C_NONFINITE, C_NEXT, C_FILTER, C_FALLBACK,
    C_KILLED, C_KTESTS, C_CERT, C_CERT_BAD,
    C_MAXLEN,                 // largest squared alpha-edge length (bits of a binary32)
    C_CLASS, C_TAKE = C_CLASS + 4,  // balls per degree class, and handed out of each
    C_NCOUNTERS = C_TAKE + 4
};

struct MolGrid {
    float minx, miny, minz, step;
    int gx, gy, gz;
    float wmax;  // upper bound on every ball's binary32 weight (r + sol)^2
    uint64_t cell_base;  // first global cell of this molecule
    uint64_t ncell;
    uint64_t atom_base;  // first ball (sorted and input) of this molecule
};

#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess)                                                            \
            return pac::set_error(PAC_ERR_CUDA, std::string(#call) + ": " +               \
                                                    cudaGetErrorString(e_));              \
    } while (0)

#define LAUNCH_CHECK(ctx)                                                                 \
    do {                                                                                  \
        (ctx).launches++;                                                                 \
        cudaError_t e_ = cudaGetLastError();                                              \
        if (e_ != cudaSuccess)                                                            \
            return pac::set_error(PAC_ERR_CUDA, std::string("launch: ") +                 \
                                                    cudaGetErrorString(e_));              \
    } while (0)

// ------------------------------------------------------------------ utils
__device__ __forceinline__ int fkey(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float funkey(int k) {
    return __int_as_float(k >= 0 ? k : k ^ 0x7fffffff);
}
__device__ __forceinline__ uint32_t mol_of(const uint32_t *mol, uint64_t i) {
    return mol ? mol[i] : 0u;
}
// 32-bit wrapping linear cell index, as the reference's int arithmetic
// behaves on the GPU (AlphaComplexLargeData.cu:625-626).
__device__ __forceinline__ int lin3(int X, int Y, int Z, int gx, int gy) {
    return (int)((unsigned)Z * (unsigned)gx * (unsigned)gy + (unsigned)Y * (unsigned)gx +
                 (unsigned)X);
}
// lower_bound of v in sorted a[0..n)
__device__ __forceinline__ int lbound(const uint32_t *a, int n, uint32_t v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        int m = (lo + hi) >> 1;
        if (__ldg(&a[m]) < v)
            lo = m + 1;
        else
            hi = m;
    }
    return lo;
}
// position of the k-th set bit (0-based) of a W-word mask, or -1
__device__ __forceinline__ int select_bit(const uint64_t *m, int W, int k) {
    for (int w = 0; w < W; w++) {
        int c = __popcll(m[w]);
        if (k < c) {
            uint32_t lo = (uint32_t)m[w], hi = (uint32_t)(m[w] >> 32);
            int cl = __popc(lo);
            if (k < cl) return w * 64 + __fns(lo, 0, k + 1);
            return w * 64 + 32 + __fns(hi, 0, k - cl + 1);
        }
        k -= c;
    }
    return -1;
}
// position of the k-th set bit (0-based) of x, k < popcount(x): halve the
// word by popcounts
__device__ __forceinline__ int select64(uint64_t x, int k) {
    uint32_t v = (uint32_t)x;
    int pos = 0;
    const int pl = __popc(v);
    if (k >= pl) {
        k -= pl;
        v = (uint32_t)(x >> 32);
        pos = 32;
    }
    int q = __popc(v & 0xffffu);
    if (k >= q) k -= q, v >>= 16, pos += 16;
    q = __popc(v & 0xffu);
    if (k >= q) k -= q, v >>= 8, pos += 8;
    q = __popc(v & 0xfu);
    if (k >= q) k -= q, v >>= 4, pos += 4;
    q = __popc(v & 0x3u);
    if (k >= q) k -= q, v >>= 2, pos += 2;
    return pos + (k >= (int)(v & 1u) ? 1 : 0);
}
// the same over a KW-word mask, k < its popcount
template <int KW>
__device__ __forceinline__ int select_kw(const uint64_t *m, int k) {
    int w = 0;
    uint64_t x = m[0];
#pragma unroll
    for (int v = 0; v + 1 < KW; v++) {
        const int q = __popcll(x);
        if (k < q) break;
        k -= q;
        w = v + 1;
        x = m[v + 1];
    }
    return w * 64 + select64(x, k);
}
// bits of word w whose global position is greater than b
__device__ __forceinline__ uint64_t above_mask(int b, int w) {
    if (w * 64 + 63 <= b) return 0ull;
    if (w * 64 > b) return ~0ull;
    int j = b & 63;
    return j == 63 ? 0ull : (~0ull << (j + 1));
}
__device__ __forceinline__ void bump(unsigned long long *ctr, int which, unsigned long long v) {
    if (v) atomicAdd(&ctr[which], v);
}
__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// ------------------------------------------------------------------ decisions
// Each test of the pipeline in one of two arithmetics: the reference's
// single-precision formulas (V = kUpstream, kPlainXmp; refarith.cuh) or the
// decision-exact cascade (V = kExact; exactpred.cuh).  In the exact mode the
// "weight" slots of the insphere/orientation helpers carry radii, squared
// exactly inside the predicates.
using pac::ex::Tally;

template <int V>
__device__ __forceinline__ float wt(float r) {
    if constexpr (V == pac::kExact) return r;
    else return pac::mul_rn(r, r);
}

template <int V>
__device__ __forceinline__ bool dec_edge(const Ball a, const Ball b, float alpha, Tally &t) {
    if constexpr (V == pac::kExact) return pac::ex::edge_alpha(a, b, alpha, t);
    else return pac::edge_alpha<V>(a, b, alpha);
}

// alpha mark of a triangle; the orthosphere (centre, power) goes to o.  (F, here
// and below: the place in refarith.cuh whose contraction applies.)
template <int V, class F>
__device__ __forceinline__ bool dec_tri(const Ball a, const Ball b, const Ball c, float alpha,
                                        float4 &o, Tally &t) {
    if constexpr (V == pac::kExact) {
        o = make_float4(0.f, 0.f, 0.f, 0.f);
        return pac::ex::tri_alpha(a, b, c, alpha, t);
    } else {
        return pac::tri_alpha<V, F>(a, b, c, alpha, o);
    }
}

// window centre (and the reference's power) of an alpha triangle
template <int V>
__device__ __forceinline__ float4 tri_sphere(const Ball a, const Ball b, const Ball c, float alpha) {
    if constexpr (V == pac::kExact) {
        const float3 q = pac::ex::tri_centre(a, b, c);
        return make_float4(q.x, q.y, q.z, 0.f);
    } else {
        float4 o;
        pac::tri_alpha<V>(a, b, c, alpha, o);
        return o;
    }
}

// alpha mark of a tetrahedron; its orthosphere centre goes to o (zeros when
// the tetrahedron is flat, as in the reference).  wide: a has more than 64
// upper neighbours.
template <int V, class F>
__device__ __forceinline__ bool dec_tet(const Ball a, const Ball b, const Ball c, const Ball d,
                                        float alpha, float4 &o, bool wide, Tally &t) {
    if constexpr (V == pac::kExact) {
        bool flat = false;
        const bool m = pac::ex::tet_alpha(a, b, c, d, alpha, flat, t);
        o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m && !flat) {
            const float3 q = pac::ex::tet_centre(a, b, c, d);
            o = make_float4(q.x, q.y, q.z, 0.f);
        }
        return m;
    } else {
        return pac::tet_alpha<F>(a, b, c, d, alpha, o, wide);
    }
}

template <int V>
__device__ __forceinline__ float dec_orient(const float *pa, const float *pb, const float *pc,
                                            const float *pd, float wa, float wb, float wc, float wd,
                                            Tally &t) {
    if constexpr (V == pac::kExact)
        return (float)pac::ex::orient_sign(Ball{pa[0], pa[1], pa[2], wa}, Ball{pb[0], pb[1], pb[2], wb},
                                           Ball{pc[0], pc[1], pc[2], wc}, Ball{pd[0], pd[1], pd[2], wd}, t);
    else
        return pac::orient3d(pa, pb, pc, pd);
}

template <int V, class F>
__device__ __forceinline__ float dec_insphere(const float *pa, const float *pb, const float *pc,
                                              const float *pd, const float *pe, float wa, float wb,
                                              float wc, float wd, float we, Tally &t) {
    if constexpr (V == pac::kExact)
        return (float)pac::ex::insphere_sign(
            Ball{pa[0], pa[1], pa[2], wa}, Ball{pb[0], pb[1], pb[2], wb}, Ball{pc[0], pc[1], pc[2], wc},
            Ball{pd[0], pd[1], pd[2], wd}, Ball{pe[0], pe[1], pe[2], we}, t);
    else
        return pac::insphere_w<F>(pa, pb, pc, pd, pe, wa, wb, wc, wd, we);
}

// Attachment of the triangle (a0, v1, v2) by ball q; (px, py, pz, cur) is
// the reference's orthosphere of the triangle (unused in the exact mode).
template <int V>
__device__ __forceinline__ bool dec_tri_attached(const Ball a0, const float4 *at, uint32_t v1,
                                                 uint32_t v2, const Ball q, float px, float py,
                                                 float pz, float cur, Tally &t) {
    if constexpr (V == pac::kExact)
        return pac::ex::tri_attached(a0, pac::ld_ball(&at[v1]), pac::ld_ball(&at[v2]), q, t);
    else
        return pac::attached(q, px, py, pz, cur);
}

// Window centre of an alpha edge and the reference's power there.
template <int V>
__device__ __forceinline__ void edge_sphere(const Ball a1, const Ball a2, float &px, float &py,
                                            float &pz, float &cur) {
    if constexpr (V == pac::kExact) {
        const float3 c = pac::ex::edge_centre(a1, a2);
        px = c.x, py = c.y, pz = c.z, cur = 0.f;
    } else {
        pac::edge_foot(a1, a2, px, py, pz, cur);
    }
}

template <int V>
__device__ __forceinline__ bool dec_edge_attached(const Ball a1, const Ball a2, const Ball q,
                                                  float px, float py, float pz, float cur,
                                                  Tally &t) {
    if constexpr (V == pac::kExact) return pac::ex::edge_attached(a1, a2, q, t);
    else return pac::attached(q, px, py, pz, cur);
}

// End of a warp-per-ball kernel (all lanes present): add the lanes'
// tallies to the counters.
template <int V>
__device__ __forceinline__ void flush_tally(const Tally &t, unsigned long long *ctr) {
    if constexpr (V == pac::kExact) {
        const unsigned long long e = warp_sum(t.evals), f = warp_sum(t.fallbacks);
        const bool r = __any_sync(kFull, t.range != 0);
        if ((threadIdx.x & 31) == 0) {
            bump(ctr, C_FILTER, e);
            bump(ctr, C_FALLBACK, f);
            if (r) bump(ctr, C_SOS_RANGE, 1);
        }
    }
}
// The same from a single thread.
template <int V>
__device__ __forceinline__ void flush_tally_thread(const Tally &t, unsigned long long *ctr) {
    if constexpr (V == pac::kExact) {
        if (t.evals) atomicAdd(&ctr[C_FILTER], (unsigned long long)t.evals);
        if (t.fallbacks) atomicAdd(&ctr[C_FALLBACK], (unsigned long long)t.fallbacks);
        if (t.range) atomicAdd(&ctr[C_SOS_RANGE], 1ull);
    }
}

// ------------------------------------------------------------------ scan
// Exclusive prefix sum of n values into out[0..n], out[n] = total.  A block
// of 8 warps takes kScanTile values, a warp 512 consecutive ones held in
// registers (16 coalesced loads), scanned by shuffles.  What bounds it at the
// sizes of one molecule is launches and barriers: one tile is one launch, up to
// kScanWide tiles are two (each block adds up the sums of the tiles before
// it), more are three.  Against three launches with shared-memory scans of 20
// barriers per 1,024 values: 13 -> 5 us of kernel time a scan at 211 balls, 16 ->
// 13 us at 25,000 (of that about 2.5 us per launch).
constexpr int kScanTile = 4096;
constexpr uint64_t kScanWide = 1024;

// sum of the block's values v (all threads get it)
__device__ __forceinline__ unsigned long long block_sum(unsigned long long v) {
    __shared__ unsigned long long s[8];
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) v += s[w];
    return v;
}
template <class Tin>
__global__ void __launch_bounds__(256) k_scan_reduce(const Tin *in, uint64_t n, uint64_t *bsum) {
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
    unsigned long long acc = 0;
#pragma unroll
    for (int k = 0; k < kScanTile / 256; k++) {
        const uint64_t i = base + (uint64_t)k * 256 + threadIdx.x;
        if (i < n) acc += (unsigned long long)in[i];
    }
    acc = block_sum(acc);
    if (threadIdx.x == 0) bsum[blockIdx.x] = acc;
}
// exclusive prefix sums of the nb tile sums, in place, in one block
__global__ void __launch_bounds__(256) k_scan_blocks(uint64_t *bsum, uint64_t nb) {
    __shared__ unsigned long long s[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (uint64_t base = 0; base < nb; base += 256) {
        const uint64_t i = base + threadIdx.x;
        const unsigned long long v = i < nb ? bsum[i] : 0;
        unsigned long long incl = v;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        __syncthreads();
        if (lane == 31) s[warp] = incl;
        __syncthreads();
        unsigned long long before = carry, tot = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) {
            if (w < warp) before += s[w];
            tot += s[w];
        }
        if (i < nb) bsum[i] = before + incl - v;
        carry += tot;
    }
}
// bsum: the tiles' sums (summed = false) or their prefix sums (true); unused
// when there is one tile
template <class Tin, class Tout>
__global__ void __launch_bounds__(256) k_scan_apply(const Tin *in, uint64_t n, const uint64_t *bsum,
                                                    bool summed, Tout *out) {
    __shared__ unsigned long long s[8];
    constexpr int kPer = kScanTile / 256;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile + (uint64_t)warp * (32 * kPer);
    unsigned long long carry = 0;
    if (summed) {
        carry = bsum[blockIdx.x];
    } else {
        for (uint64_t b = threadIdx.x; b < blockIdx.x; b += 256) carry += bsum[b];
        if (blockIdx.x) carry = block_sum(carry);
    }
    Tin v[kPer];
    unsigned long long mine = 0;
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const uint64_t i = base + (uint64_t)k * 32 + lane;
        v[k] = i < n ? in[i] : Tin(0);
        mine += (unsigned long long)v[k];
    }
    mine = warp_sum(mine);
    if (lane == 0) s[warp] = mine;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; w++)
        if (w < warp) carry += s[w];
#pragma unroll
    for (int k = 0; k < kPer; k++) {
        const uint64_t i = base + (uint64_t)k * 32 + lane;
        unsigned long long incl = (unsigned long long)v[k];
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += t;
        }
        if (i < n) out[i] = (Tout)(carry + incl - (unsigned long long)v[k]);
        if (i + 1 == n) out[n] = (Tout)(carry + incl);
        carry += __shfl_sync(kFull, incl, 31);
    }
    if (n == 0 && threadIdx.x == 0) out[0] = 0;
}

template <class Tin, class Tout>
static int exclusive_scan(pac::Ctx &ctx, const Tin *in, uint64_t n, Tout *out) {
    const uint64_t nb = std::max<uint64_t>(1, (n + kScanTile - 1) / kScanTile);
    uint64_t *bsum = nullptr;
    if (nb > 1) {
        bsum = ctx.arena.alloc_n<uint64_t>(nb);
        if (!bsum) return PAC_ERR_OOM;
        k_scan_reduce<Tin><<<(unsigned)nb, 256, 0, ctx.stream>>>(in, n, bsum);
        LAUNCH_CHECK(ctx);
    }
    if (nb > kScanWide) {
        k_scan_blocks<<<1, 256, 0, ctx.stream>>>(bsum, nb);
        LAUNCH_CHECK(ctx);
    }
    k_scan_apply<Tin, Tout><<<(unsigned)nb, 256, 0, ctx.stream>>>(in, n, bsum, nb > kScanWide, out);
    LAUNCH_CHECK(ctx);
    return PAC_OK;
}

// ------------------------------------------------------------------ grid
__global__ void k_mol_ids(const uint64_t *off, uint32_t n_mol, uint32_t *mol) {
    uint32_t m = blockIdx.x;
    if (m >= n_mol) return;
    for (uint64_t i = off[m] + threadIdx.x; i < off[m + 1]; i += blockDim.x) mol[i] = m;
}

// min/max of raw x, y, z, r per molecule (AlphaComplexLargeData.cu:1088-1110).
// Floats are compared through an order-preserving int key.  Non-finite
// coordinates and radii are reported in ctr[C_NONFINITE].
__global__ void k_bbox(const float4 *balls, uint64_t n, const uint32_t *mol, int *mm,
                       unsigned long long *ctr) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool act = i < n;
    uint32_t m = act ? mol_of(mol, i) : 0xffffffffu;
    float4 b = act ? balls[i] : make_float4(0, 0, 0, 0);
    if (!isfinite(b.x) || !isfinite(b.y) || !isfinite(b.z) || !isfinite(b.w)) ctr[C_NONFINITE] = 1;
    int k[4] = {fkey(b.x), fkey(b.y), fkey(b.z), fkey(b.w)};
    uint32_t m0 = __shfl_sync(kFull, m, 0);
    bool uniform = __all_sync(kFull, act && m == m0);
    for (int q = 0; q < 4; q++) {
        if (uniform) {
            int lo = k[q], hi = k[q];
            for (int o = 16; o; o >>= 1) {
                lo = min(lo, __shfl_xor_sync(kFull, lo, o));
                hi = max(hi, __shfl_xor_sync(kFull, hi, o));
            }
            if ((threadIdx.x & 31) == 0) {
                atomicMin(&mm[m * 8 + q], lo);
                atomicMax(&mm[m * 8 + 4 + q], hi);
            }
        } else if (act) {
            atomicMin(&mm[m * 8 + q], k[q]);
            atomicMax(&mm[m * 8 + 4 + q], k[q]);
        }
    }
}

// grid parameters per molecule (AlphaComplexLargeData.cu:1119-1123)
__global__ void k_grid(const int *mm, uint32_t n_mol, float sol, float alpha, MolGrid *g,
                       uint64_t *ncell) {
    uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n_mol) return;
    float minX = funkey(mm[m * 8 + 0]), minY = funkey(mm[m * 8 + 1]),
          minZ = funkey(mm[m * 8 + 2]);
    float maxX = funkey(mm[m * 8 + 4]), maxY = funkey(mm[m * 8 + 5]),
          maxZ = funkey(mm[m * 8 + 6]), maxRadius = funkey(mm[m * 8 + 7]);
    float possibleMaxRadius = __fsqrt_rn(__fadd_rn(__fmul_rn(maxRadius, maxRadius), alpha));
    float stepSize = __fmul_rn(2.0f, possibleMaxRadius);
    int gx = (int)__fdiv_rn(__fsub_rn(maxX, minX), stepSize) + 1;
    int gy = (int)__fdiv_rn(__fsub_rn(maxY, minY), stepSize) + 1;
    int gz = (int)__fdiv_rn(__fsub_rn(maxZ, minZ), stepSize) + 1;
    MolGrid r;
    r.minx = minX;
    r.miny = minY;
    r.minz = minZ;
    r.step = stepSize;
    r.gx = gx;
    r.gy = gy;
    r.gz = gz;
    // r + sol is rounded monotonically, so the extreme radii bound every
    // ball's weight; the margin covers the rounding of the square
    const float rlo = fabsf(__fadd_rn(funkey(mm[m * 8 + 3]), sol)), rhi = fabsf(__fadd_rn(maxRadius, sol));
    const float rm = fmaxf(rlo, rhi);
    r.wmax = __fmul_rn(__fmul_rn(rm, rm), 1.0f + 1.0f / 1024.0f);
    r.cell_base = 0;
    r.ncell = (uint64_t)max(gx, 0) * (uint64_t)max(gy, 0) * (uint64_t)max(gz, 0);
    r.atom_base = 0;
    g[m] = r;
    ncell[m] = r.ncell;
}

// cell key (AlphaComplexLargeData.cu:65-78) and a slot within the cell
__global__ void k_cellkey(const float4 *balls, uint64_t n, const uint32_t *mol, const MolGrid *g,
                          uint32_t *gcell, uint32_t *slot, uint32_t *cellcnt) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const MolGrid G = g[mol_of(mol, i)];
    float4 b = balls[i];
    int cellX = (int)__fdiv_rn(__fsub_rn(b.x, G.minx), G.step);
    int cellY = (int)__fdiv_rn(__fsub_rn(b.y, G.miny), G.step);
    int cellZ = (int)__fdiv_rn(__fsub_rn(b.z, G.minz), G.step);
    int cell = cellX + G.gx * cellY + G.gx * G.gy * cellZ;
    uint32_t gc = (uint32_t)(G.cell_base + (uint64_t)cell);
    gcell[i] = gc;
    slot[i] = atomicAdd(&cellcnt[gc], 1u);
}

__global__ void k_scatter(uint64_t n, const uint32_t *gcell, const uint32_t *slot,
                          const uint32_t *cellbeg, uint32_t *perm) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    perm[cellbeg[gcell[i]] + slot[i]] = (uint32_t)i;
}

// order each cell by input index: the stable sort's tie order
__global__ void k_cellsort(uint64_t ncell, const uint32_t *cellbeg, uint32_t *perm) {
    uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= ncell) return;
    uint32_t b = cellbeg[c], e = cellbeg[c + 1];
    for (uint32_t i = b + 1; i < e; i++) {
        uint32_t v = perm[i];
        uint32_t j = i;
        while (j > b && perm[j - 1] > v) {
            perm[j] = perm[j - 1];
            j--;
        }
        perm[j] = v;
    }
}

__global__ void k_gather(uint64_t n, const uint32_t *perm, const float4 *balls, float sol,
                         const uint32_t *gcell, const uint32_t *mol, const MolGrid *g,
                         float4 *at, uint32_t *orig, uint32_t *cellof) {
    uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    uint32_t i = perm[p];
    float4 b = balls[i];
    at[p] = make_float4(b.x, b.y, b.z, __fadd_rn(b.w, sol));
    orig[p] = (uint32_t)(i - g[mol_of(mol, i)].atom_base);
    cellof[p] = gcell[i];
}

// ------------------------------------------------------------------ edges
// One warp per ball i: the candidates are the balls l > i of the 27 cells
// around i's cell whose linear index is >= i's (AlphaComplexLargeData.cu:
// 80-165); each passes the power filter (markRealEdges) or not.  Lane k < 27
// owns neighbour cell k in the reference's loop order, so a warp prefix sum
// over the cell sizes enumerates the candidates in ascending l.
template <int V, bool FILL>
__global__ void __launch_bounds__(256) k_edges(uint64_t n, const float4 *__restrict__ at,
                                               const uint32_t *__restrict__ cellof,
                                               const uint32_t *__restrict__ cellbeg,
                                               const uint32_t *__restrict__ mol,
                                               const MolGrid *__restrict__ grids, float alpha,
                                               uint32_t *ecount, const uint64_t *eoff,
                                               uint32_t *ER, unsigned long long *ctr) {
    const int lane = threadIdx.x & 31;
    uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long cand_acc = 0, alpha_acc = 0;
    float len2 = 0.f;  // FILL: the longest alpha edge
    Tally tally;
    for (uint64_t p = warp; p < n; p += nwarps) {
        const MolGrid G = grids[mol_of(mol, p)];
        int cell = (int)(cellof[p] - G.cell_base);
        int gX = cell % G.gx, t = cell / G.gx, gY = t % G.gy, gZ = t / G.gy;
        uint32_t beg = 0, cnt = 0;
        if (lane < 27) {
            int i = lane / 9 - 1, j = (lane / 3) % 3 - 1, k = lane % 3 - 1;
            bool ok = !((gZ + i >= G.gz) || (gY + j >= G.gy) || (gX + k >= G.gx)) &&
                      !((gZ + i < 0) || (gY + j < 0) || (gX + k < 0));
            if (ok) {
                int adj = (gZ + i) * G.gx * G.gy + (gY + j) * G.gx + (gX + k);
                if (adj >= cell) {
                    uint64_t gc = G.cell_base + (uint64_t)adj;
                    uint32_t b = cellbeg[gc], e = cellbeg[gc + 1];
                    if (adj == cell) b = (uint32_t)p + 1;
                    if (e > b) {
                        beg = b;
                        cnt = e - b;
                    }
                }
            }
        }
        uint32_t incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t v = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += v;
        }
        uint32_t total = __shfl_sync(kFull, incl, 31);
        const Ball A = pac::ld_ball(&at[p]);
        uint64_t out = FILL ? eoff[p] : 0;
        uint32_t kept = 0;
        for (uint32_t base = 0; base < total; base += 32) {
            uint32_t s = base + lane;
            bool act = s < total;
            // segment owning slot s: first lane whose inclusive sum exceeds s
            int lo = 0;
            for (int step = 16; step; step >>= 1) {
                uint32_t v = __shfl_sync(kFull, incl, lo + step - 1);
                if (v <= s) lo += step;
            }
            uint32_t sinc = __shfl_sync(kFull, incl, lo & 31);
            uint32_t sbeg = __shfl_sync(kFull, beg, lo & 31);
            uint32_t scnt = __shfl_sync(kFull, cnt, lo & 31);
            bool pass = false;
            uint32_t l = 0;
            if (act) {
                l = sbeg + (s - (sinc - scnt));
                const Ball B = pac::ld_ball(&at[l]);
                pass = dec_edge<V>(A, B, alpha, tally);
                if (FILL && pass) {
                    const float x = A.x - B.x, y = A.y - B.y, z = A.z - B.z;
                    len2 = fmaxf(len2, x * x + y * y + z * z);
                }
            }
            unsigned m = __ballot_sync(kFull, pass);
            if (FILL && pass) ER[out + kept + __popc(m & ((1u << lane) - 1))] = l;
            kept += __popc(m);
        }
        if (lane == 0) {
            if (!FILL) ecount[p] = kept;
            cand_acc += total;
            alpha_acc += kept;
        }
    }
    if (FILL) {
        const unsigned bits = __reduce_max_sync(kFull, __float_as_uint(len2));
        if (lane == 0 && bits > (unsigned)*(volatile unsigned long long *)&ctr[C_MAXLEN])
            atomicMax(&ctr[C_MAXLEN], (unsigned long long)bits);
    }
    if (!FILL) flush_tally<V>(tally, ctr);
    if (!FILL && lane == 0) {
        bump(ctr, C_CAND_E, cand_acc);
        bump(ctr, C_ALPHA_E, alpha_acc);
    }
}

// words of link matrix per ball; the largest degree through one atomic per
// block (one per ball serialised on its address: 18 us at 25,000 balls)
__global__ void __launch_bounds__(256) k_link_size(uint64_t n, const uint32_t *ecount, uint64_t *lsize,
                                                   unsigned long long *ctr) {
    __shared__ unsigned m[8];
    const uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t deg = p < n ? ecount[p] : 0;
    if (p < n) lsize[p] = deg * ((deg + 63) >> 6);
    const unsigned w = __reduce_max_sync(kFull, (unsigned)deg);
    if ((threadIdx.x & 31) == 0) m[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x) return;
    unsigned top = 0;
    for (int k = 0; k < 8; k++) top = max(top, m[k]);
    if (top > *(volatile unsigned long long *)&ctr[C_MAXDEG]) atomicMax(&ctr[C_MAXDEG], (unsigned long long)top);
}

// The balls of [lo, hi) by class (0, 1, 2: at most 64, 128, 256 upper neighbours;
// 3: at most `sparse`; of at least `least`): list[class * n ..], counted in
// ctr[C_CLASS + class].
constexpr int kSparse = 3;
__global__ void k_classes(uint64_t lo, uint64_t hi, uint64_t n, const uint64_t *eoff,
                          const uint64_t *loff, uint64_t *attached, int least, int sparse,
                          uint32_t *list, unsigned long long *ctr) {
    const uint64_t p = lo + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int deg = p < hi ? (int)(eoff[p + 1] - eoff[p]) : 0;
    if (attached && deg > 0 && deg < 3)  // no class: its rows are not written there
        for (int a = 0; a < deg; a++) attached[loff[p] + a] = 0;
    const int mine = deg < least ? -1 : deg <= sparse ? kSparse : deg <= 64 ? 0 : deg <= 128 ? 1 : 2;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const unsigned m = __ballot_sync(kFull, mine == c);
        if (!m) continue;
        unsigned long long b = 0;
        if (lane == 0) b = atomicAdd(&ctr[C_CLASS + c], (unsigned long long)__popc(m));
        b = __shfl_sync(kFull, b, 0);
        if (mine == c) list[c * n + b + __popc(m & ((1u << lane) - 1))] = (uint32_t)p;
    }
}

// ------------------------------------------------------------------ triangles
// Bit (a, b) of ball i's link matrix is set when (i, v1 = N[a], v2 = N[b]) is a
// candidate triangle -- edge v1v2 is an alpha edge (AlphaComplexLargeData.cu:
// 192-296) -- and passes markRealTriangles.  A block per ball of one class (see
// k_classes).  The edges among a ball's neighbours come from one table look-up
// per neighbour of a neighbour (a binary search in global memory per pair took
// half of the time); the candidates are then cut into equal shares over the
// block's threads, so that every lane evaluates markRealTriangles.
// What bounds it: instruction issue, most of it markRealTriangles.  A warp per
// ball searching pair by pair, 21 of 32 lanes: 1.98 ms at 100,000 balls, 105 us
// at 211.

// Slot of ball x in a table of 2^bits, for attempt t: the neighbours of a ball
// are a few runs of consecutive indices, which the low bits usually keep apart
// and else a multiplication, which spreads a run evenly (of the 24,832 balls of a
// 25,013-ball globule with a probe 23,612 settle by the low bits, 1,220 by a
// multiplication; eight attempts are for indices that are no runs).
constexpr int kHashTries = 8;
__device__ __forceinline__ uint32_t hash_slot(uint32_t x, int t, int bits) {
    return t == 0 ? x & ((1u << bits) - 1) : (x * (2654435769u * (2u * t + 1u))) >> (32 - bits);
}

// A table from ball indices to positions in the list ids[0..deg), whose entries
// are written for attempt 0: tries others until no two of the list collide.
// Returns the attempt, or kHashTries when all collide (block-uniform; ends
// with a barrier).
__device__ __forceinline__ int settle_table(uint8_t *tab, const uint32_t *ids, int deg, int bits) {
    int tries = 0;
    while (true) {
        bool clash = false;
        for (int c = threadIdx.x; c < deg; c += blockDim.x)
            clash |= tab[hash_slot(ids[c], tries, bits)] != (uint8_t)c;
        if (!__syncthreads_or(clash) || ++tries == kHashTries) return tries;
        for (int c = threadIdx.x; c < deg; c += blockDim.x)
            tab[hash_slot(ids[c], tries, bits)] = (uint8_t)c;
        __syncthreads();
    }
}
// The position of x in the list, or some other position (compare ids there):
// a slot that no listed ball wrote holds anything.  size: of ids' array, a
// power of two.
__device__ __forceinline__ int table_find(const uint8_t *tab, const uint32_t *ids, int deg, int size,
                                          int bits, int tries, uint32_t x) {
    if (tries < kHashTries) return tab[hash_slot(x, tries, bits)] & (size - 1);
    int lo = 0, hi = deg;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ids[mid] <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <int KW>
struct LinkSmem {
    static constexpr int kDeg = 64 * KW, kBits = KW == 1 ? 10 : KW == 2 ? 11 : 13, kWords = 2 * KW;
    float4 ball[kDeg];           // the upper neighbours
    uint64_t e2[kDeg];           // each one's first upper neighbour's index
    uint32_t edge[kDeg * kWords + 1];  // bits b of row a: alpha edge (N[a], N[b]); all ones at the end
    uint32_t tri[kDeg * kWords]; // the link rows
    uint32_t id[kDeg];
    uint32_t rowpre[kDeg + 1];   // candidates before each row
    uint32_t next;
    uint16_t d2[kDeg];           // upper degrees
    uint8_t tab[1 << kBits];
};

template <int V, int KW>
__global__ void __launch_bounds__(128) k_link(const uint32_t *list, int cls,
                                              const float4 *__restrict__ at,
                                              const uint64_t *__restrict__ eoff,
                                              const uint32_t *__restrict__ ER,
                                              const uint64_t *__restrict__ loff, uint64_t *link,
                                              float alpha, unsigned long long *ctr) {
    using Smem = LinkSmem<KW>;
    using Place = std::conditional_t<KW == 1, pac::AtLink<V>, pac::AtLinkWide<V>>;
    constexpr int kWords = Smem::kWords, kThreads = 128, kWarps = 4;
    __shared__ Smem S;
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    uint32_t cand_acc = 0, alpha_acc = 0;
    Tally tally;
    const uint64_t count = ctr[C_CLASS + cls];
    while (true) {
        __syncthreads();  // the previous ball's shared memory is free
        if (tid == 0) {
            const unsigned long long u = atomicAdd(&ctr[C_TAKE + cls], 1ull);
            S.next = u < count ? list[u] : 0xffffffffu;
        }
        __syncthreads();
        const uint32_t p = S.next;
        if (p == 0xffffffffu) break;
        const uint64_t e0 = eoff[p];
        const int deg = (int)(eoff[p + 1] - e0);
        const Ball A = pac::ld_ball(&at[p]);
        for (int c = tid; c < deg; c += kThreads) {
            const uint32_t x = __ldg(&ER[e0 + c]);
            S.id[c] = x;
            S.ball[c] = __ldg(&at[x]);
            const uint64_t e2 = eoff[x];
            S.e2[c] = e2;
            S.d2[c] = (uint16_t)(eoff[x + 1] - e2);
            S.tab[hash_slot(x, 0, Smem::kBits)] = (uint8_t)c;
        }
        for (int k = tid; k < deg * kWords; k += kThreads) S.tri[k] = 0;
        __syncthreads();
        const int tries = settle_table(S.tab, S.id, deg, Smem::kBits);
        // ---- the edges among the neighbours: lanes over the list of N[a]
        for (int a = wib; a < deg; a += kWarps) {
            const uint32_t *N2 = ER + S.e2[a];
            const int deg2 = S.d2[a];
            uint32_t mine[kWords];
#pragma unroll
            for (int w = 0; w < kWords; w++) mine[w] = 0;
            for (int k = lane; k < deg2; k += 32) {
                const uint32_t x = __ldg(&N2[k]);
                const int c = table_find(S.tab, S.id, deg, Smem::kDeg, Smem::kBits, tries, x);
                const bool hit = c < deg && S.id[c] == x;
#pragma unroll
                for (int w = 0; w < kWords; w++)
                    if (hit && (c >> 5) == w) mine[w] |= 1u << (c & 31);
            }
            uint32_t cnt = 0;
#pragma unroll
            for (int w = 0; w < kWords; w++) {
                const uint32_t all = __reduce_or_sync(kFull, mine[w]);
                if (lane == 0) S.edge[a * kWords + w] = all;
                cnt += __popc(all);
            }
            if (lane == 0) S.rowpre[a + 1] = cnt;
        }
        if (tid == 0) {
            S.rowpre[0] = 0;
            S.edge[deg * kWords] = 0xffffffffu;  // ends every walk
        }
        __syncthreads();
        if (wib == 0) {
            uint32_t carry = 0;
            for (int a0 = 0; a0 < deg; a0 += 32) {
                const int a = a0 + lane;
                uint32_t incl = a < deg ? S.rowpre[a + 1] : 0;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += v;
                }
                if (a < deg) S.rowpre[a + 1] = carry + incl;
                carry += __shfl_sync(kFull, incl, 31);
            }
        }
        __syncthreads();
        // ---- markRealTriangles, an equal share of the candidates per thread
        const int total = (int)S.rowpre[deg];
        const int steps = (total + kThreads - 1) / kThreads;
        const int start = tid * steps, left = max(0, min(total - start, steps));
        if (left > 0) {
            int lo = 0, hi = deg;  // rowpre[lo] <= start < rowpre[lo + 1]
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if ((int)S.rowpre[mid] <= start) lo = mid;
                else hi = mid;
            }
            int skip = start - (int)S.rowpre[lo];
            uint32_t k = (uint32_t)lo * kWords, bits = S.edge[k];
            for (int q; skip >= (q = __popc(bits)); skip -= q) bits = S.edge[++k];
            for (; skip > 0; skip--) bits &= bits - 1;
            for (int s = 0; s < left; s++) {
                while (!bits) bits = S.edge[++k];
                const int a = (int)(k / kWords), b = (int)(k % kWords) * 32 + __ffs((int)bits) - 1;
                bits &= bits - 1;
                const float4 b1 = S.ball[a], b2 = S.ball[b];
                float4 o;
                if (dec_tri<V, Place>(A, Ball{b1.x, b1.y, b1.z, b1.w}, Ball{b2.x, b2.y, b2.z, b2.w}, alpha,
                                      o, tally)) {
                    atomicOr(&S.tri[k], 1u << (b & 31));
                    alpha_acc++;
                }
            }
            cand_acc += left;
        }
        __syncthreads();
        const int W = (deg + 63) >> 6;
        uint64_t *L = link + loff[p];
        for (int k = tid; k < deg * W; k += kThreads) {
            const int a = k / W, w = k % W;
            const uint32_t *t = &S.tri[a * kWords + 2 * w];
            L[k] = (uint64_t)t[0] | (uint64_t)t[1] << 32;
        }
    }
    const unsigned long long cs = warp_sum(cand_acc), as = warp_sum(alpha_acc);
    flush_tally<V>(tally, ctr);
    if (lane == 0) {
        bump(ctr, C_CAND_T, cs);
        bump(ctr, C_ALPHA_T, as);
    }
}

// The same for balls of few upper neighbours, a warp per ball: its pairs
// (a, b) flattened over the lanes, row a's deg - 1 - a of them after the
// P(a) = a (2 deg - 1 - a) / 2 before it, each looked up by a search in N[a]'s
// list.  A block spends most of such a ball on barriers and on the chain of
// loads before them: all links of 231,086 balls without a probe (8.6 upper
// neighbours on average) 0.60 ms by blocks, 0.29 / 0.25 / 0.235 / 0.24 with balls
// of at most 12 / 16 / 24 / 32 here; with a probe (41) 1.36 -> 1.33 ms at 100,000.
// Passes of few balls are as long as their slowest ball and keep to blocks
// (with 24 here: 28 -> 40 us at 211 balls, 110 -> 120 at 5,003, 396 -> 400 at
// 25,000 with a probe; 173 -> 87 at 60,000 without).
constexpr int kLinkWarpDeg = 24;
constexpr uint64_t kSparseBalls = 1 << 15;  // (links and enumeration)
template <int V>
__global__ void __launch_bounds__(256) k_link_warp(const uint32_t *list, const float4 *__restrict__ at,
                                                   const uint64_t *__restrict__ eoff,
                                                   const uint32_t *__restrict__ ER,
                                                   const uint64_t *__restrict__ loff, uint64_t *link,
                                                   float alpha, unsigned long long *ctr) {
    __shared__ uint32_t rows[8][32];
    static_assert(kLinkWarpDeg <= 32, "a word per row");
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t count = ctr[C_CLASS + kSparse];
    uint32_t cand_acc = 0, alpha_acc = 0;
    Tally tally;
    for (uint64_t u = warp; u < count; u += nwarps) {
        const uint32_t p = list[u];
        const uint64_t e0 = eoff[p];
        const int deg = (int)(eoff[p + 1] - e0);
        const uint32_t *N = ER + e0;
        const Ball A = pac::ld_ball(&at[p]);
        rows[wib][lane] = 0;
        __syncwarp();
        const int total = deg * (deg - 1) / 2;
        for (int s = lane; s < total; s += 32) {
            const float D = (float)(2 * deg - 1);
            int a = (int)((D - sqrtf(D * D - 8.0f * (float)s)) * 0.5f);
            a = max(0, min(a, deg - 2));
            while (a > 0 && a * (2 * deg - 1 - a) / 2 > s) a--;
            while (a + 1 <= deg - 2 && (a + 1) * (2 * deg - 2 - a) / 2 <= s) a++;
            const int b = a + 1 + (s - a * (2 * deg - 1 - a) / 2);
            const uint32_t v1 = __ldg(&N[a]), v2 = __ldg(&N[b]);
            const uint64_t e1 = eoff[v1];
            const int deg1 = (int)(eoff[v1 + 1] - e1);
            const int pos = lbound(ER + e1, deg1, v2);
            if (pos == deg1 || __ldg(&ER[e1 + pos]) != v2) continue;
            cand_acc++;
            float4 o;
            if (dec_tri<V, pac::AtLink<V>>(A, pac::ld_ball(&at[v1]), pac::ld_ball(&at[v2]), alpha, o, tally)) {
                atomicOr(&rows[wib][a], 1u << b);
                alpha_acc++;
            }
        }
        __syncwarp();
        if (lane < deg) link[loff[p] + lane] = rows[wib][lane];
        __syncwarp();
    }
    const unsigned long long cs = warp_sum(cand_acc), as = warp_sum(alpha_acc);
    flush_tally<V>(tally, ctr);
    if (lane == 0) {
        bump(ctr, C_CAND_T, cs);
        bump(ctr, C_ALPHA_T, as);
    }
}

// ------------------------------------------------------------------ tetrahedra
struct TetArgs {
    uint64_t n;
    const float4 *at;
    const uint32_t *orig;
    const uint64_t *eoff;
    const uint32_t *ER;
    const uint64_t *loff;
    const uint64_t *link;
    uint64_t *faces;
    const uint32_t *cellbeg;
    const uint32_t *mol;
    const MolGrid *grids;
    float alpha;
    // survivors (as-written) / ordered output (as-run fill)
    uint2 *surv;          // (ball, packed a | b << 8 | c << 16)
    uint64_t surv_cap;
    uint32_t *tcount;     // per ball
    uint2 *pend;          // tetrahedra waiting for the exact SoS
    uint64_t pend_cap;
    const uint64_t *toff; // as-run fill: output offsets per ball
    uint32_t *tets_out;   // as-run fill: sorted-space vertex quadruples
    unsigned long long *ctr;   // the pass's counters, or a chunk's (enumeration)
    const unsigned long long *maxlen;  // C_MAXLEN of the pass
    uint64_t *attached;        // enumeration: alpha triangles a neighbour attaches (shape of
                               // link), or null
    int refute;                // enumeration: refute early against the group's firsts
    int verify;                // scan: replay every certified decision and count disagreements
    int scan_claim;            // queue entries a scan warp claims at a time
};

__device__ __forceinline__ void mark_face(uint64_t *F, uint64_t row_base, int W, int a, int b) {
    atomicOr((unsigned long long *)&F[row_base + (uint64_t)a * W + (b >> 6)],
             1ull << (b & 63));
}

// One warp per ball v1.  For each upper neighbour v2 = N[a] the lanes take
// the alpha triangles (v1, v2, v3 = N[b]); the fourth vertices v4 = N[c]
// (c > b) are the common bits of rows a and b of v1's link matrix whose
// face (v2, v3, v4) is also an alpha triangle -- exactly the reference's
// candidate tetrahedra (AlphaComplexLargeData.cu:350-529).  Each candidate
// then passes markRealTets and, as written, the empty-orthosphere test.
// As run (the orthosphere test skipped; both modes decide by one sequence of
// operations, or rows would not fit their count): MODE 1 counts per ball, MODE 2
// writes in reference order (needs MODE 1's offsets).
template <int V, int MODE>
__global__ void __launch_bounds__(256) k_tets(TetArgs A) {
    __shared__ uint16_t smap[8][kMaxDeg];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long cand_acc = 0, alpha_acc = 0;
    Tally tally;
    for (uint64_t p = warp; p < A.n; p += nwarps) {
        const uint64_t e0 = A.eoff[p];
        const int deg = (int)(A.eoff[p + 1] - e0);
        uint32_t ball_count = 0;
        if (deg >= 3) {
            const int W = (deg + 63) >> 6;
            const uint32_t *N = A.ER + e0;
            const uint64_t lp = A.loff[p];
            const uint64_t *Lp = A.link + lp;
            const Ball B1 = pac::ld_ball(&A.at[p]);
            uint64_t out_base = (MODE == 2) ? A.toff[p] : 0;
            for (int a = 0; a < deg - 2; a++) {
                uint64_t ra[kMaxW];
                int nb = 0;
#pragma unroll
                for (int w = 0; w < kMaxW; w++) {
                    ra[w] = w < W ? Lp[(uint64_t)a * W + w] : 0;
                    nb += __popcll(ra[w]);
                }
                if (nb < 2) continue;
                const uint32_t v2 = __ldg(&N[a]);
                const uint64_t e2 = A.eoff[v2];
                const int deg2 = (int)(A.eoff[v2 + 1] - e2);
                const int W2 = (deg2 + 63) >> 6;
                const uint64_t l2 = A.loff[v2];
                const uint64_t *L2 = A.link + l2;
                for (int c = a + 1 + lane; c < deg; c += 32) {
                    uint32_t x = __ldg(&N[c]);
                    int pos = lbound(A.ER + e2, deg2, x);
                    smap[wib][c] = (pos < deg2 && __ldg(&A.ER[e2 + pos]) == x) ? (uint16_t)pos
                                                                               : (uint16_t)0xffff;
                }
                __syncwarp();
                const Ball B2 = pac::ld_ball(&A.at[v2]);
                for (int k0 = 0; k0 < nb; k0 += 32) {
                    int b = (k0 + lane < nb) ? select_bit(ra, W, k0 + lane) : -1;
                    uint32_t lane_cnt = 0;
                    // MODE 2 needs each lane's count first to place its rows
                    uint64_t lane_off = 0;
                    for (int sweep = (MODE == 2 ? 0 : 1); sweep < 2; sweep++) {
                        if (MODE == 2 && sweep == 1) {
                            uint32_t incl = lane_cnt;
                            for (int o = 1; o < 32; o <<= 1) {
                                uint32_t v = __shfl_up_sync(kFull, incl, o);
                                if (lane >= o) incl += v;
                            }
                            lane_off = out_base + ball_count + (incl - lane_cnt);
                            ball_count += __shfl_sync(kFull, incl, 31);
                            lane_cnt = 0;
                        }
                        if (b >= 0) {
                            const uint32_t v3 = __ldg(&N[b]);
                            const Ball B3 = pac::ld_ball(&A.at[v3]);
                            const int mb = smap[wib][b];
                            uint64_t m[kMaxW];
#pragma unroll
                            for (int w = 0; w < kMaxW; w++)
                                m[w] = w < W ? (ra[w] & Lp[(uint64_t)b * W + w] & above_mask(b, w))
                                             : 0;
                            const uint64_t *R2 = L2 + (uint64_t)mb * W2;
                            for (int w = 0; w < kMaxW; w++) {
                                uint64_t bits = m[w];
                                while (bits) {
                                    int c = w * 64 + __ffsll((long long)bits) - 1;
                                    bits &= bits - 1;
                                    int mc = smap[wib][c];
                                    if (mb == 0xffff || mc == 0xffff) continue;
                                    if (!((__ldg(&R2[mc >> 6]) >> (mc & 63)) & 1ull)) continue;
                                    if (sweep == 1) cand_acc++;
                                    const uint32_t v4 = __ldg(&N[c]);
                                    const Ball B4 = pac::ld_ball(&A.at[v4]);
                                    float4 o;
                                    if (!dec_tet<V, pac::AtRun>(B1, B2, B3, B4, A.alpha, o, false, tally)) continue;
                                    if (sweep == 1) alpha_acc++;
                                    if (MODE == 1) {
                                        lane_cnt++;
                                        continue;
                                    }
                                    if (MODE == 2) {
                                        if (sweep == 0) {
                                            lane_cnt++;
                                            continue;
                                        }
                                        uint64_t q = lane_off + lane_cnt++;
                                        uint4 t4 = make_uint4((uint32_t)p, v2, v3, v4);
                                        *(uint4 *)&A.tets_out[4 * q] = t4;
                                        mark_face(A.faces, lp, W, a, b);
                                        mark_face(A.faces, lp, W, a, c);
                                        mark_face(A.faces, lp, W, b, c);
                                        mark_face(A.faces, l2, W2, mb, mc);
                                        continue;
                                    }
                                }
                            }
                        }
                    }
                    if (MODE != 2) {
                        uint32_t s = lane_cnt;
                        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(kFull, s, o);
                        ball_count += s;
                    }
                }
                __syncwarp();
            }
        }
        if (lane == 0 && MODE != 2) A.tcount[p] = ball_count;
    }
    cand_acc = warp_sum(cand_acc);
    alpha_acc = warp_sum(alpha_acc);
    if (MODE == 1) flush_tally<V>(tally, A.ctr);  // MODE 2 repeats MODE 1's tests
    if (lane == 0) {
        bump(A.ctr, C_CAND_Q, cand_acc);
        bump(A.ctr, C_ALPHA_Q, alpha_acc);
    }
}

// Records one tetrahedron that passed the orthosphere test (or, pending,
// one whose window held an exact zero): the survivor list, the per-ball
// count, and the marks of its four faces in the `faces` matrices.
__device__ __noinline__ void emit_survivor(const uint64_t *__restrict__ eoff,
                                           const uint32_t *__restrict__ ER,
                                           const uint64_t *__restrict__ loff, uint64_t *faces,
                                           uint2 *surv, uint64_t surv_cap, uint2 *pend,
                                           uint64_t pend_cap, unsigned long long *ctr,
                                           uint32_t *tcount, uint32_t p, uint32_t key, uint32_t v2,
                                           uint32_t v3, uint32_t v4, bool pending) {
    if (pending) {
        unsigned long long q = atomicAdd(&ctr[C_PEND], 1ull);
        if (q < pend_cap) pend[q] = make_uint2(p, key);
        return;
    }
    unsigned long long q = atomicAdd(&ctr[C_SURV], 1ull);
    if (q < surv_cap) surv[q] = make_uint2(p, key);
    atomicAdd(&tcount[p], 1u);
    const int W = (int)((eoff[p + 1] - eoff[p] + 63) >> 6);
    const uint64_t lp = loff[p];
    const int a = key & 0xff, b = (key >> 8) & 0xff, c = (key >> 16) & 0xff;
    mark_face(faces, lp, W, a, b);
    mark_face(faces, lp, W, a, c);
    mark_face(faces, lp, W, b, c);
    const uint64_t e2 = eoff[v2];
    const int deg2 = (int)(eoff[v2 + 1] - e2);
    const int mb = lbound(ER + e2, deg2, v3), mc = lbound(ER + e2, deg2, v4);
    mark_face(faces, loff[v2], (deg2 + 63) >> 6, mb, mc);
}

// The 27-cell window of the orthosphere and attachment tests, visited as
// the centre cell first (window_centre) and then ten parts (window_part):
// the two side cells of the centre row, then the eight other x-rows -- for
// z and y offsets (i, j) the cells (gX-1 .. gX+1, gY+j, gZ+i), clipped to
// the grid, are consecutive in the cell order, so their balls form one range
// of the sorted balls.  Faces before corners, so the balls nearest the
// window centre come first and most tests end early.  Together these are the
// reference's window (AlphaComplexLargeData.cu:621-733): the centre cell
// through its wrapped linear index, the 26 neighbours range-checked per
// axis; the same cells in another order, and the tests' outcome does not
// depend on the order.
constexpr int kWindowParts = 10;
// rows 2..9 as (i + 1) | (j + 1) << 2, 4 bits each:
// (0,-1) (0,1) (-1,0) (1,0) (-1,-1) (-1,1) (1,-1) (1,1)
constexpr uint64_t kRowOrder = 0x1ull | 0x9ull << 4 | 0x4ull << 8 | 0x6ull << 12 | 0x0ull << 16 |
                               0x8ull << 20 | 0x2ull << 24 | 0xAull << 28;

// [beg, end) of window part r, or false when it lies outside the grid.
__device__ __forceinline__ bool window_part(const MolGrid &G, const uint32_t *cellbeg, int gX,
                                            int gY, int gZ, int r, uint32_t &beg, uint32_t &end) {
    long long zz = gZ, yy = gY, xlo, xhi;
    if (r < 2) {  // a side cell of the centre row
        xlo = xhi = (long long)gX + (r == 0 ? -1 : 1);
    } else {
        const int code = (int)((kRowOrder >> (4 * (r - 2))) & 0xf);
        zz += (code & 3) - 1;
        yy += (code >> 2) - 1;
        xlo = (long long)gX - 1;
        xhi = (long long)gX + 1;
    }
    if (zz < 0 || zz >= G.gz || yy < 0 || yy >= G.gy) return false;
    xlo = max(xlo, 0ll);
    xhi = min(xhi, (long long)G.gx - 1);
    if (xlo > xhi) return false;
    const uint64_t row = G.cell_base + (uint64_t)(zz * G.gy + yy) * (uint64_t)G.gx;
    beg = cellbeg[row + (uint64_t)xlo];
    end = cellbeg[row + (uint64_t)xhi + 1];
    return true;
}

// The window's centre cell as the reference reads it, through its wrapped
// linear index cl.w: [beg, end), or an empty range (counted) when cl.w names
// no cell (out-of-range read in the reference, AlphaComplexLargeData.cu:
// 625-627).  When the centre (cl.x, cl.y, cl.z) lies inside the grid this is
// the centre cell itself, which no part holds; when it lies outside, the
// parts hold the window's in-grid cells and this is the extra cell the
// wrapped index names.
__device__ __forceinline__ void window_centre(const MolGrid &G, const uint32_t *cellbeg, int4 cl,
                                              uint32_t &beg, uint32_t &end,
                                              unsigned long long &oob) {
    beg = end = 0;
    if (cl.w < 0 || (uint64_t)cl.w >= G.ncell) {
        oob++;
        return;
    }
    beg = cellbeg[G.cell_base + (uint64_t)cl.w];
    end = cellbeg[G.cell_base + (uint64_t)cl.w + 1];
}

// Cell coordinate (int)((p - lo) / step) of the reference (LD:621-623), with
// the IEEE division replaced by a multiplication by inv = fl(1 / step)
// whenever that provably truncates to the same integer: the product is
// within 3.1 ulp of the quotient, so when no integer lies within 16 ulp of
// it both truncate alike.  Otherwise (and for huge or non-finite values)
// the division itself.
__device__ __forceinline__ int cell_coord_fast(float p, float lo, float step, float inv) {
    const float d = __fsub_rn(p, lo);
    const float q = __fmul_rn(d, inv);
    const float t = truncf(q);
    const float f = fabsf(__fsub_rn(q, t));
    if (fabsf(q) < 4194304.0f && fminf(f, __fsub_rn(1.0f, f)) > 16.0f * pac::cert::kU * fabsf(q) + 1e-30f)
        return (int)t;
    return pac::cell_coord(p, lo, step);
}

// The window cell of an orthosphere centre: (gridX, gridY, gridZ, wrapped
// linear index), as the reference forms it (LD:621-626).
__device__ __forceinline__ int4 window_cell(const MolGrid &G, float x, float y, float z) {
    const float inv = __frcp_rn(G.step);
    const int gX = cell_coord_fast(x, G.minx, G.step, inv);
    const int gY = cell_coord_fast(y, G.miny, G.step, inv);
    const int gZ = cell_coord_fast(z, G.minz, G.step, inv);
    return make_int4(gX, gY, gZ, lin3(gX, gY, gZ, G.gx, G.gy));
}

// Whether the reference's window of an orthosphere centre (x, y, z) holds
// a ball at (bx, by, bz) in the grid: certainly so when the two are less
// than 0.99 cell steps apart on every axis.  The cells are truncations of
// the monotone binary32 map v -> (v - lo) / step (LD:72-74, 621-623), so the
// two quotients differ by less than one (the rounding is far below the 1 %
// margin for grids of at most 16384 cells per axis); the ball's quotient is
// non-negative, so the centre's truncated cell is never below -0 and the
// ball's cell lies within one of it per axis.  A centre cell inside the grid
// is read as itself; outside the grid the ball's cell differs from it and is
// one of the 26 in-grid neighbours.  Either way the reference visits it.
__device__ __forceinline__ bool surely_in_window(float x, float y, float z, float bx, float by,
                                                 float bz, float reach) {
    return fmaxf(fabsf(bx - x), fmaxf(fabsf(by - y), fabsf(bz - z))) <= reach;
}

// Queue slots are handed out to warps in blocks (one atomic per block, not
// per batch: a single counter served every warp).  Slots a warp reserved
// but did not fill are marked with this ball index, and the scan skips them.
constexpr uint32_t kNoTet = 0xffffffffu;
constexpr uint64_t kQBlock = 128;

// ---- the as-written tetrahedra: enumeration, then a scan over an HBM queue
// Enumeration (k_tets_enum): ball p's candidate tetrahedra are the
// (p, v2 = N[a], v3 = N[b], v4 = N[c]), a < b < c, with (p, v2, v3),
// (p, v2, v4), (p, v3, v4) alpha triangles (bits of p's link rows) and
// (v2, v3, v4) one too (a bit of v2's link matrix) -- exactly the
// reference's candidates (AlphaComplexLargeData.cu:350-529).
//
// Each candidate needs two answers: is it an alpha tetrahedron (counted),
// and can it be refuted here, by a ball already at hand that violates its
// orthosphere?  Within one triangle group (a, b) the fourth vertices lie in
// the pencil of spheres orthogonal to p, v2, v3; on either side of the
// triangle's plane the one whose orthosphere comes first along the pencil
// lies inside the orthospheres of all the others, and the two sides' firsts
// refute each other unless they are in pencil order.  pencil.cuh gives both
// answers in some twenty operations, each with a certificate that the
// reference's arithmetic (or, in the exact mode, the exact polynomials) decides
// alike.  What it cannot certify, and what is not refuted, goes to the queue,
// and the scan decides it by the general path.
//
// What bounds it: instruction issue and shared memory (DRAM is nearly idle).
// The work of a ball is one list of its alpha triangles, taken 32 at a time
// by the warps of a block.  A lane sets up one triangle in shared memory; the
// 32 triangles' candidates are then cut into equal consecutive shares, a lane
// walking the bits of its share, so every lane is busy and finding a
// candidate costs a bit scan, not a search.  That first sweep decides the
// faces and the alpha tests, lists what is left and leaves each side's first
// candidate; the second tests the list against the firsts (testing against the
// best so far in one sweep queues twice as many).  A block per ball also keeps
// small molecules short: a ball's triangles run on 4 to 16 warps instead of one.
// Measured against one warp per ball or eight rows, markRealTets and a replayed
// insphere_w per candidate: the pass at 100,008 balls 18.98 -> 13.15 ms, at 211
// balls 1.52 -> 1.00 ms, the 2.5 M-ball assembly 340 -> 256 ms.
struct TetQueue {
    uint2 *ent;    // (ball, key): positions a | b << 8 | c << 16 in its list, and flags;
                   // ball = kNoTet marks an unused slot
    uint64_t cap;
};
constexpr uint32_t kAlphaOpen = 1u << 24;  // the alpha test is left to the scan (counted there)
constexpr uint32_t kRefuted = 1u << 25;    // refuted: the scan only counts it
// of pending entries, contracted flavour: see replay_violates; an insphere value
// was exactly 0
constexpr uint32_t kDisputed = 1u << 26, kTied = 1u << 27;
constexpr int kRingSteps = 2;              // candidate steps between writes to the queue

// One triangle of a chunk: pencil::Group and what the sweeps leave.  80 bytes
// apart, so that consecutive records' 16-byte reads meet no bank twice.
struct GroupRec {
    float4 nh;       // n, hmin
    float4 qe;       // Q, ea
    float4 tk;       // Q~, k
    float rg;
    uint32_t ab;     // a | b << 8 | attachment margin (16 bits); the sign: found attached
    uint32_t best[2];  // per side: pencil position (24 bits) | c of its first; then c | (refuted) << 8
    float2 first[2]; // h, g of the firsts
};
static_assert(sizeof(GroupRec) == 80, "bank layout");

// KW words per link row, D neighbours: balls of at most 64, 128 or 256 upper
// neighbours, or of at most 32 in passes of many balls.  Those have one or two
// chunks of triangles: a block of one warp each, 20 an SM, instead of four that
// wait at barriers (enumeration and scan of 231,086 balls without a probe, 2.2
// triangles an edge: 2.49 -> 1.74 ms; with balls of at most 16 or 24 here 1.80, 1.77;
// with a probe at 100,000 balls, 41 upper neighbours, 9.01 -> 8.99).  Below
// kSparseBalls the longest ball counts, and four warps share it (25,000 balls with a
// probe 2.11 ms, with one warp each 2.18; 211 balls 167 and 231 us).
template <int KW, int D = 64 * KW>
struct EnumSmem {
    static constexpr int kDeg = D, kTabBits = D == 32 ? 8 : KW == 1 ? 10 : KW == 2 ? 11 : 13;
    static constexpr int kSlots = D == 32 ? 96 : KW == 1 ? 216 : 256;  // candidates at a time (one group has fewer)
    static constexpr int kWords = 2 * KW;
    static constexpr int kGroups = D == 32 ? 512 : 1024;  // triangles listed at a time (one row has fewer)
    static constexpr int kWarps = D == 32 ? 1 : KW == 1 ? 4 : KW == 2 ? 12 : 16;
    static constexpr int kBlocks = D == 32 ? 20 : KW == 1 ? 6 : KW == 2 ? 2 : 1;  // per SM
    // records per warp: a chunk's 32 triangles and one past them, which ends
    // every walk and which lanes past their share read
    static constexpr int kRecs = 33;
    float4 rel[kDeg];            // upper neighbours relative to p, and their lifts s
    pac::pencil::Point pt[kDeg]; // the same in double
    uint64_t sL[kDeg * KW];      // p's link rows
    uint64_t e2[kDeg], l2[kDeg]; // per neighbour: its first upper neighbour's index, its link rows
    GroupRec group[kWarps][kRecs];  // the chunk's triangles
    float2 hg[kWarps][kSlots];   // per listed candidate: h, g
    uint32_t pm[kWarps][kRecs][kWords];  // per triangle: its fourth vertices (bits c); all ones past the last
    uint32_t face[kWarps][4][kRecs];     // and its row of v2's link matrix (128 bits)
    uint32_t ring[kWarps][32 * (kRingSteps + 1)];  // queue entries waiting for a full write
    uint16_t cand[kWarps][kSlots];  // listed candidates: group | c << 5 | kCand* bits
    float st[kDeg];              // lifts of the rounded squares
    uint32_t sN[kDeg];           // upper neighbours
    uint32_t att[kDeg * kWords]; // triangles found attached: bits b of row a
    uint32_t rowpre[kDeg + 1];   // triangles with fourth vertices before each row
    uint32_t next, chunk;        // the block's ball, its next chunk
    uint16_t tri[kGroups];       // p's triangles: a | b << 8
    pac::pencil::Bounds bounds;  // of the block's ball
    uint16_t d2[kDeg];           // per neighbour: its upper degree
    uint8_t tab[1 << kTabBits];  // positions of p's neighbours by a hash of their index
    uint8_t map[kDeg][kDeg];     // [a][c]: position of N[c] in the list of N[a] (alpha edges only)
};
// the sweeps index all three by the same record
template <int KW, int D = 64 * KW>
constexpr bool enum_records_match() {
    using S = EnumSmem<KW, D>;
    constexpr size_t n = S::kRecs;
    return n == 33 && std::extent<decltype(S::group), 1>::value == n &&
           std::extent<decltype(S::pm), 1>::value == n && std::extent<decltype(S::face), 2>::value == n;
}
static_assert(enum_records_match<1, 32>() && enum_records_match<1>() && enum_records_match<2>() &&
                  enum_records_match<kMaxW>(),
              "a record past the chunk's last in every array");
// a listed candidate's alpha test is open; |h| >= hmin (and refutation is on)
constexpr uint32_t kCandOpen = 1u << 13, kCandSure = 1u << 14;

// Per-warp state of the queue: the reserved block and the waiting entries.
struct QRes {
    uint64_t pos, end;  // next free slot of the warp's block, its end
    int wait;           // entries in the ring
};

// Writes the first k <= 32 waiting entries of ball p (warp-uniform call).
__device__ __forceinline__ void queue_write(const TetQueue &Q, unsigned long long *ctr, QRes &qr,
                                            uint32_t p, const uint32_t *ring, int k) {
    const int lane = threadIdx.x & 31;
    const uint64_t left = qr.end - qr.pos;
    uint64_t nb = 0;
    if ((uint64_t)k > left) {
        if (lane == 0) nb = atomicAdd(&ctr[C_SURV], (unsigned long long)kQBlock);
        nb = __shfl_sync(kFull, nb, 0);
    }
    if (lane < k) {
        const uint64_t pos = (uint64_t)lane < left ? qr.pos + lane : nb + (lane - left);
        if (pos < Q.cap) Q.ent[pos] = make_uint2(p, ring[lane]);
    }
    if ((uint64_t)k > left) {
        qr.pos = nb + (k - left);
        qr.end = nb + kQBlock;
    } else {
        qr.pos += k;
    }
}

// Writes the ring's full rows of 32 and moves the rest to its front.
__device__ __forceinline__ void queue_drain(const TetQueue &Q, unsigned long long *ctr, QRes &qr,
                                            uint32_t p, uint32_t *ring) {
    if (qr.wait < 32) return;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    int at = 0;
    for (; qr.wait >= 32; at += 32, qr.wait -= 32) queue_write(Q, ctr, qr, p, ring + at, 32);
    const uint32_t rest = lane < qr.wait ? ring[at + lane] : 0u;
    __syncwarp();
    if (lane < qr.wait) ring[lane] = rest;
}

// Marks the rest of the warp's block unused.
__device__ __forceinline__ void queue_close(const TetQueue &Q, QRes &qr) {
    const int lane = threadIdx.x & 31;
    for (uint64_t s = qr.pos + lane; s < qr.end; s += 32)
        if (s < Q.cap) Q.ent[s] = make_uint2(kNoTet, 0);
    qr.pos = qr.end;
}

// How the enumeration treats its inputs: weights and window centres of the
// exact mode or of the reference's arithmetic, every certified decision
// replayed or not (verify mode).
enum : int { kEnumFloat = 0, kEnumExact = 1, kEnumVerify = 2 };

// Sum over the coordinates of (binary32 square - square); each difference is
// exact.
__device__ __forceinline__ float square_rounding(float x, float y, float z) {
    const float xx = __fmul_rn(x, x), yy = __fmul_rn(y, y), zz = __fmul_rn(z, z);
    return -(fmaf(x, x, -xx) + fmaf(y, y, -yy) + fmaf(z, z, -zz));
}

// Verify mode: a certified alpha decision (alpha) and, when y >= 0, a
// certified refutation by ball y, against the general path; counted in
// C_CERT (decisions) and C_CERT_BAD (disagreements).
template <int M>
__device__ __noinline__ void enum_verify(const TetArgs &A, const MolGrid &G, const float4 b1,
                                         const float4 b2, const float4 b3, const float4 b4,
                                         bool wide, int alpha, const float4 *y) {
    constexpr int V = (M & kEnumExact) ? pac::kExact : pac::kUpstream;
    Tally tally;
    float4 sph;
    const Ball B1{b1.x, b1.y, b1.z, b1.w}, B2{b2.x, b2.y, b2.z, b2.w}, B3{b3.x, b3.y, b3.z, b3.w},
        B4{b4.x, b4.y, b4.z, b4.w};
    const bool mark = dec_tet<V, pac::AtEnum>(B1, B2, B3, B4, A.alpha, sph, wide, tally);
    if (alpha >= 0) {
        atomicAdd(&A.ctr[C_CERT], 1ull);
        if (mark != (alpha == 1)) atomicAdd(&A.ctr[C_CERT_BAD], 1ull);
    }
    if (y && mark) {
        const float pa[3] = {B1.x, B1.y, B1.z}, pb[3] = {B2.x, B2.y, B2.z};
        const float pc[3] = {B3.x, B3.y, B3.z}, pd[3] = {B4.x, B4.y, B4.z};
        const float pe[3] = {y->x, y->y, y->z};
        const float wa = wt<V>(B1.r), wb = wt<V>(B2.r), wc = wt<V>(B3.r), wd = wt<V>(B4.r);
        const float o = dec_orient<V>(pa, pb, pc, pd, wa, wb, wc, wd, tally);
        const float r = dec_insphere<V, pac::AtScan>(pa, pb, pc, pd, pe, wa, wb, wc, wd, wt<V>(y->w), tally);
        atomicAdd(&A.ctr[C_CERT], 1ull);
        if (!(o < 0 ? r < 0 : r > 0) ||
            !surely_in_window(sph.x, sph.y, sph.z, y->x, y->y, y->z, 0.99f * G.step))
            atomicAdd(&A.ctr[C_CERT_BAD], 1ull);
    }
}

// Verify mode: a certified attachment of the triangle by ball e.
template <int M>
__device__ __noinline__ void attach_verify(const TetArgs &A, const MolGrid &G, const float4 b1,
                                           const float4 b2, const float4 b3, const float4 e) {
    constexpr int V = (M & kEnumExact) ? pac::kExact : pac::kUpstream;
    Tally tally;
    const Ball B1{b1.x, b1.y, b1.z, b1.w}, B2{b2.x, b2.y, b2.z, b2.w}, B3{b3.x, b3.y, b3.z, b3.w},
        E{e.x, e.y, e.z, e.w};
    const float4 o = tri_sphere<V>(B1, B2, B3, A.alpha);
    bool att;
    if constexpr (V == pac::kExact) att = pac::ex::tri_attached(B1, B2, B3, E, tally);
    else att = pac::attached(E, o.x, o.y, o.z, o.w);
    atomicAdd(&A.ctr[C_CERT], 1ull);
    if (!att || !surely_in_window(o.x, o.y, o.z, e.x, e.y, e.z, 0.99f * G.step))
        atomicAdd(&A.ctr[C_CERT_BAD], 1ull);
}

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Whether ball v lies within reach, per axis, of the orthosphere centre of the
// candidate z (both relative to p) of a group.
__device__ __noinline__ bool within_reach(const float4 gA, const float4 gC, const float4 z, float st,
                                          const float4 v, float reach) {
    const float h = pac::pencil::height(gA.x, gA.y, gA.z, z.x, z.y, z.z);
    const float gt = pac::pencil::power(gC.x, gC.y, gC.z, st, z.x, z.y, z.z);
    return pac::pencil::within_reach(gA.x, gA.y, gA.z, gC.x, gC.y, gC.z, h, gt, v.x, v.y, v.z, reach);
}

// A block per ball of one class (list, counted in ctr[C_CLASS + cls], taken
// from ctr[C_TAKE + cls]).
template <int KW, int M, int D = 64 * KW>
__global__ void __launch_bounds__(EnumSmem<KW, D>::kWarps * 32, EnumSmem<KW, D>::kBlocks)
    k_tets_enum(TetArgs A, TetQueue Q, const uint32_t *list, int cls) {
    using Smem = EnumSmem<KW, D>;
    constexpr int kWarps = Smem::kWarps, kThreads = kWarps * 32, kSlots = Smem::kSlots;
    constexpr int kTabBits = Smem::kTabBits;
#ifdef PAC_CONTRACTED
    constexpr bool kContracted = !(M & kEnumExact);
#else
    constexpr bool kContracted = false;
#endif
    // (contracted: half of the squares' rounding, see pencil.cuh)
    constexpr bool kPerturbed = !(M & kEnumExact);
    constexpr double kShare = kContracted ? 0.5 : 1.0;
    // more than the 48 KB of static shared memory: dynamic, opted in by
    // enum_smem_optin()
    extern __shared__ __align__(16) unsigned char enum_smem[];
    Smem &S = *reinterpret_cast<Smem *>(enum_smem);
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1;
    uint32_t cand_acc = 0, open_acc = 0, listed_acc = 0, queued = 0;
    QRes qr{0, 0, 0};
    const uint64_t count = A.ctr[C_CLASS + cls];
    while (true) {
        // (the previous ball's shared memory is free: every warp passed the
        // barrier after its last chunk)
        if (tid == 0) {
            // stop handing out work once the queue has overflowed: the chunk
            // is rerun smaller
            unsigned long long u = count;
            if (!(*(volatile unsigned long long *)&A.ctr[C_SURV] > Q.cap))
                u = atomicAdd(&A.ctr[C_TAKE + cls], 1ull);
            S.next = u < count ? list[u] : kNoTet;
            S.chunk = 0;
        }
        __syncthreads();
        const uint32_t p = S.next;
        if (p == kNoTet) break;
        // (each thread clears what it wrote out for the previous ball)
        for (int k = tid; k < Smem::kDeg * KW; k += kThreads) *(uint64_t *)&S.att[2 * k] = 0;
        const uint64_t e0 = A.eoff[p];
        const int deg = (int)(A.eoff[p + 1] - e0);
        const MolGrid &G = A.grids[mol_of(A.mol, p)];
        const float4 b1 = __ldg(&A.at[p]);
        const float w1 = __fmul_rn(b1.w, b1.w);  // (its rounding in the exact mode is inside the bounds)
        const bool refute = A.refute && G.gx <= 16384 && G.gy <= 16384 && G.gz <= 16384;
        if (tid == 0)
            S.bounds = pac::pencil::bounds(b1.x, b1.y, b1.z, w1, A.alpha,
                                           __uint_as_float((uint32_t)*A.maxlen), G.wmax, G.step,
                                           kContracted);
        // ---- the ball's neighbours, relative to it, and its link rows
        {
            const double px = b1.x, py = b1.y, pz = b1.z;
            const double wp = (M & kEnumExact) ? (double)b1.w * b1.w : (double)w1;
            const float rp = kPerturbed ? square_rounding(b1.x, b1.y, b1.z) : 0.f;
            for (int c = tid; c < deg; c += kThreads) {
                const uint32_t x = __ldg(&A.ER[e0 + c]);
                const float4 b = __ldg(&A.at[x]);
                S.sN[c] = x;
                pac::pencil::Point P;
                P.x = b.x - px, P.y = b.y - py, P.z = b.z - pz;
                const double w = (M & kEnumExact) ? (double)b.w * b.w : (double)__fmul_rn(b.w, b.w);
                P.s = P.x * P.x + P.y * P.y + P.z * P.z - w + wp;
                P.st = kPerturbed ? P.s + kShare * (square_rounding(b.x, b.y, b.z) - rp) : P.s;
                S.pt[c] = P;
                S.rel[c] = make_float4((float)P.x, (float)P.y, (float)P.z, (float)P.s);
                S.st[c] = (float)P.st;
                const uint64_t e2 = A.eoff[x];
                S.e2[c] = e2;
                S.d2[c] = (uint16_t)(A.eoff[x + 1] - e2);
                S.l2[c] = A.loff[x];
                S.tab[hash_slot(x, 0, kTabBits)] = (uint8_t)c;
            }
            const int W = (deg + 63) >> 6;
            const uint64_t *Lg = A.link + A.loff[p];
            for (int k = tid; k < deg * KW; k += kThreads) {
                const int a = k / KW, w = k % KW;
                S.sL[k] = w < W ? Lg[(uint64_t)a * W + w] : 0ull;
            }
        }
        // (whether some neighbour's rows are wider than a staged face row)
        bool wide = false;
        for (int c = tid; c < deg; c += kThreads) wide |= S.d2[c] > 128;
        wide = __syncthreads_or(wide);
        // ---- a table without collisions, so that a lookup is one read
        const int tries = settle_table(S.tab, S.sN, deg, kTabBits);
        // ---- where each neighbour's neighbours stand in p's list: lanes
        // over the list of N[a], one lookup each (the last warp also counts
        // the triangles before each row: its bits but the highest, which has
        // no fourth vertex above)
        if (wib == kWarps - 1) {
            uint32_t base = 0;
            for (int a0 = 0; a0 < deg; a0 += 32) {
                const int a = a0 + lane;
                uint32_t nb = 0;
                if (a < deg)
#pragma unroll
                    for (int w = 0; w < KW; w++) nb += __popcll(S.sL[a * KW + w]);
                nb -= nb > 0;
                uint32_t incl = nb;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t v = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += v;
                }
                if (a < deg) S.rowpre[a] = base + incl - nb;
                base += __shfl_sync(kFull, incl, 31);
            }
            if (lane == 0) S.rowpre[deg] = base;
        }
        for (int a = wib; a < deg - 2; a += kWarps) {
            // (rows without a pair of triangles have no candidates: with the
            // plain-xmp formulas, whose alpha triangles are few, most rows)
            int nb = 0;
#pragma unroll
            for (int w = 0; w < KW; w++) nb += __popcll(S.sL[a * KW + w]);
            if (nb < 2) continue;
            const uint32_t *N2 = A.ER + S.e2[a];
            const int deg2 = S.d2[a];
            for (int k = lane; k < deg2; k += 32) {
                const uint32_t x = __ldg(&N2[k]);
                const int c = table_find(S.tab, S.sN, deg, Smem::kDeg, kTabBits, tries, x);
                if (S.sN[c] == x) S.map[a][c] = (uint8_t)k;
            }
        }
        __syncthreads();
        const bool slow = S.bounds.reach > 0.f || (M & kEnumVerify);
        const float kappa = S.bounds.kappa, mreach = S.bounds.mreach;
        // ---- the triangles (p, N[a], N[b]): rows [row0, row1) listed at a
        // time, 32 triangles per chunk
        for (int row0 = 0, row1; row0 < deg; row0 = row1) {
        const int listed = (int)S.rowpre[row0];
        row1 = deg;
        if (KW > 1 || (int)S.rowpre[deg] > Smem::kGroups) {
            int lo = row0 + 1, hi = deg;  // the last row whose end fits
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((int)S.rowpre[mid] - listed <= Smem::kGroups) lo = mid;
                else hi = mid - 1;
            }
            row1 = lo;
        }
        for (int a = row0 + tid; a < row1; a += kThreads) {
            uint16_t *out = &S.tri[S.rowpre[a] - listed];
            int left = (int)(S.rowpre[a + 1] - S.rowpre[a]);
            for (int w = 0; w < 2 * KW && left > 0; w++) {
                uint32_t bits = ((const uint32_t *)&S.sL[a * KW])[w];
                for (; bits && left > 0; left--) {
                    *out++ = (uint16_t)(a | ((w * 32 + __ffs((int)bits) - 1) << 8));
                    bits &= bits - 1;
                }
            }
        }
        const int ngroups = (int)S.rowpre[row1] - listed;
        __syncthreads();
        while (true) {
            int g0 = 0;
            if (lane == 0) g0 = (int)atomicAdd(&S.chunk, 32u);
            g0 = __shfl_sync(kFull, g0, 0);
            if (g0 >= ngroups) break;
            // lane: its triangle, and the fourth vertices c > b with the
            // three faces at p
            uint64_t pm[KW];
            int cnt = 0, a = 0, b = 0;
#pragma unroll
            for (int w = 0; w < KW; w++) pm[w] = 0ull;
            if (g0 + lane < ngroups) {
                const int ab = S.tri[g0 + lane];
                a = ab & 0xff, b = ab >> 8;
#pragma unroll
                for (int w = 0; w < KW; w++) {
                    pm[w] = S.sL[a * KW + w] & S.sL[b * KW + w] & above_mask(b, w);
                    cnt += __popcll(pm[w]);
                }
            }
            int incl = cnt;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(kFull, incl, 31);
            if (!total) continue;
            // the triangles with candidates, side by side in shared memory
            const unsigned used = __ballot_sync(kFull, cnt > 0);
            const int r = __popc(used & lt_mask);
            if (cnt > 0) {
                const int W2 = (S.d2[a] + 63) >> 6;
                const uint64_t *row = A.link + S.l2[a] + (uint64_t)S.map[a][b] * W2;
                const uint64_t f0 = __ldg(&row[0]), f1 = W2 > 1 ? __ldg(&row[1]) : 0ull;
                const pac::pencil::Group gr = pac::pencil::group(S.bounds, S.pt[a], S.pt[b], w1);
                GroupRec &R = S.group[wib][r];
                R.nh = make_float4(gr.nx, gr.ny, gr.nz, gr.hmin);
                R.qe = make_float4(gr.qx, gr.qy, gr.qz, gr.ea);
                R.tk = make_float4(gr.tx, gr.ty, gr.tz, gr.k);
                R.rg = gr.rg;
                // the attachment margin rounded up to 16 bits
                const float mt = A.attached ? gr.mt : INFINITY;
                R.ab = (uint32_t)a | ((uint32_t)b << 8) |
                       (min(__float_as_uint(mt) + 0xffffu, 0x7f800000u) & 0xffff0000u);
                R.best[0] = R.best[1] = 0xffffffffu;
                S.face[wib][0][r] = (uint32_t)f0;
                S.face[wib][1][r] = (uint32_t)(f0 >> 32);
                S.face[wib][2][r] = (uint32_t)f1;
                S.face[wib][3][r] = (uint32_t)(f1 >> 32);
#pragma unroll
                for (int w = 0; w < KW; w++) *(uint64_t *)&S.pm[wib][r][2 * w] = pm[w];
            }
            if (lane == 0) {  // ends every walk: lanes past their share read these
                S.pm[wib][__popc(used)][0] = 0xffffffffu;
                S.group[wib][__popc(used)].ab = 0;
            }
            __syncwarp();
            // as many whole triangles as the list holds at a time
            for (int base = 0; base < total;) {
                const unsigned fits = __ballot_sync(kFull, incl - base <= kSlots);
                const int end = __shfl_sync(kFull, incl, 31 - __clz((int)fits));
                const bool mine = cnt > 0 && incl > base && incl <= end;
                // equal shares: lane takes candidates [start, start + left)
                const int steps = (end - base + 31) >> 5;
                const int start = base + lane * steps, left = max(0, min(end - start, steps));
                int lo = 0;  // first lane whose inclusive count exceeds start
                for (int o = 16; o; o >>= 1) {
                    const int v = __shfl_sync(kFull, incl, lo + o - 1);
                    if (v <= start) lo += o;
                }
                const int skip = start - __shfl_sync(kFull, incl - cnt, lo & 31);
                const uint32_t *words = &S.pm[wib][0][0];
                // the share's first word, and what it holds of it (a lane
                // without a share walks along, its results unused)
                uint32_t k = (uint32_t)__popc(used) * Smem::kWords;
                uint32_t bits = 0xffffffffu;
                if (left > 0) {
                    const uint32_t j = __popc(used & ((1u << lo) - 1));
                    uint64_t m[KW];
#pragma unroll
                    for (int w = 0; w < KW; w++) m[w] = *(const uint64_t *)&S.pm[wib][j][2 * w];
                    const int c = select_kw<KW>(m, skip);
                    k = j * Smem::kWords + (c >> 5);
                    bits = words[k] & (~0u << (c & 31));
                }
                base = end;
                // ---- first sweep: faces, alpha tests, the firsts
                int n = 0;  // listed
                for (int s = 0; s < steps; s++) {
                    const bool act = s < left;
                    while (!bits) bits = words[++k];
                    const uint32_t j = k / Smem::kWords;
                    const uint32_t c = (k % Smem::kWords) * 32 + (uint32_t)__ffs((int)bits) - 1;
                    bits &= bits - 1;
                    GroupRec &R = S.group[wib][j];
                    const uint32_t ab = R.ab;
                    const uint32_t a = ab & 0xff, b = (ab >> 8) & 0xff;
                    const uint32_t mc = S.map[a][c];
                    uint32_t row = S.face[wib][(mc >> 5) & 3][j];
                    if (wide && act && S.d2[a] > 128)
                        row = ((const uint32_t *)&A.link[S.l2[a] + (uint64_t)S.map[a][b] *
                                                                       ((S.d2[a] + 63) >> 6)])[mc >> 5];
                    const bool face = act && ((row >> (mc & 31)) & 1u);
                    const float4 z = S.rel[c], nh = R.nh, qe = R.qe, tk = R.tk;
                    const float h = pac::pencil::height(nh.x, nh.y, nh.z, z.x, z.y, z.z);
                    const float q = pac::pencil::power(qe.x, qe.y, qe.z, z.w, z.x, z.y, z.z);
                    const float gt = kPerturbed
                                         ? pac::pencil::power(tk.x, tk.y, tk.z, S.st[c], z.x, z.y, z.z)
                                         : q;
                    // does this neighbour attach the triangle?  One or
                    // another does for most, at a few operations here;
                    // k_tri_attach tests the other triangles
                    if (gt + (z.w - S.st[c]) < -fabsf(__uint_as_float(ab & 0xffff0000u)) && act &&
                        (mreach == 0.f || pac::pencil::in_box(tk.x, tk.y, tk.z, z.x, z.y, z.z, mreach))) {
                        R.ab = ab | 0x80000000u;
                        if constexpr (M & kEnumVerify)
                            attach_verify<M>(A, G, b1, A.at[S.sN[a]], A.at[S.sN[b]], A.at[S.sN[c]]);
                    }
                    const float a0 = fabsf(h);
                    const bool sure = a0 >= nh.w;
                    bool in, out;
                    pac::pencil::alpha_test(a0, gt, tk.w, qe.w, in, out);
                    const bool certain = a0 >= kappa * nh.w;
                    in = in && certain, out = out && certain;
                    const int i = __float_as_int(q * rcp_approx(a0));
                    const uint32_t ord = (uint32_t)(i ^ ((i >> 31) | (int)0x80000000));
                    if (sure && act) atomicMin(&R.best[h > 0.f], (ord & ~0xffu) | c);
                    const bool live = face && !out, open = live && !in;
                    cand_acc += face;
                    open_acc += open;
                    if constexpr (M & kEnumVerify)
                        if (face)
                            enum_verify<M>(A, G, b1, A.at[S.sN[a]], A.at[S.sN[b]], A.at[S.sN[c]], KW > 1,
                                           in ? 1 : out ? 0 : -1, nullptr);
                    const unsigned m = __ballot_sync(kFull, live);
                    if (live) {
                        const int at = n + __popc(m & lt_mask);
                        S.cand[wib][at] = (uint16_t)(j | (c << 5) | (open ? kCandOpen : 0u) |
                                                     (sure ? kCandSure : 0u));
                        S.hg[wib][at] = make_float2(h, q);
                    }
                    n += __popc(m);
                }
                listed_acc += (uint32_t)n;
                __syncwarp();
                // ---- per triangle: its firsts, and whether they refute each other
                if (mine) {
                    GroupRec &R = S.group[wib][r];
                    const float4 nh = R.nh, qe = R.qe;
                    const uint32_t k0 = R.best[0], k1 = R.best[1];
                    const int y0 = k0 & 0xff, y1 = k1 & 0xff;
                    float h0 = 0.f, q0 = 0.f, h1 = 0.f, q1 = 0.f;
                    if (k0 != 0xffffffffu) {
                        const float4 z = S.rel[y0];
                        h0 = pac::pencil::height(nh.x, nh.y, nh.z, z.x, z.y, z.z);
                        q0 = pac::pencil::power(qe.x, qe.y, qe.z, z.w, z.x, z.y, z.z);
                    }
                    if (k1 != 0xffffffffu) {
                        const float4 z = S.rel[y1];
                        h1 = pac::pencil::height(nh.x, nh.y, nh.z, z.x, z.y, z.z);
                        q1 = pac::pencil::power(qe.x, qe.y, qe.z, z.w, z.x, z.y, z.z);
                    }
                    // (0 when either side is empty: nothing refuted)
                    const uint32_t both = pac::pencil::refutes(h0, q0, h1, q1, R.rg) ? 256u : 0u;
                    if (R.ab >> 31) atomicOr(&S.att[a * Smem::kWords + (b >> 5)], 1u << (b & 31));
                    R.first[0] = make_float2(h0, q0);
                    R.first[1] = make_float2(h1, q1);
                    R.best[0] = (uint32_t)y0 | both;
                    R.best[1] = (uint32_t)y1 | both;
                }
                __syncwarp();
                // ---- second sweep: refutation; the rest to the queue
                for (int i0 = 0; i0 < n; i0 += 32 * kRingSteps) {
#pragma unroll
                    for (int u = 0; u < kRingSteps; u++) {
                        const int i = i0 + 32 * u + lane;
                        bool take = false;
                        uint32_t key = 0;
                        if (i < n) {
                            const uint32_t e = S.cand[wib][i];
                            const int c = (e >> 5) & 0xff;
                            const float2 x = S.hg[wib][i];
                            const GroupRec &R = S.group[wib][e & 31];
                            const int side = x.x > 0.f;
                            const uint32_t own = R.best[side];
                            const float2 y = R.first[side];
                            bool dead = pac::pencil::refutes(x.x, x.y, y.x, y.y, R.rg);
                            if (c == (int)(own & 0xff)) dead = own >= 256u;
                            dead = dead && refute && (e & kCandSure);
                            if (slow) {
                                int v = own & 0xff;
                                if (v == c) v = R.best[side ^ 1] & 0xff;
                                if (dead && S.bounds.reach > 0.f)
                                    dead = within_reach(R.nh, R.tk, S.rel[c], S.st[c], S.rel[v],
                                                        S.bounds.reach);
                                if constexpr (M & kEnumVerify)
                                    if (dead)
                                        enum_verify<M>(A, G, b1, A.at[S.sN[R.ab & 0xff]],
                                                       A.at[S.sN[(R.ab >> 8) & 0xff]], A.at[S.sN[c]],
                                                       KW > 1, -1, &A.at[S.sN[v]]);
                            }
                            take = !dead || (e & kCandOpen);
                            if (take)
                                key = (R.ab & 0xffffu) | ((uint32_t)c << 16) |
                                      (e & kCandOpen ? kAlphaOpen : 0u) | (dead ? kRefuted : 0u);
                        }
                        const unsigned m = __ballot_sync(kFull, take);
                        if (take) S.ring[wib][qr.wait + __popc(m & lt_mask)] = key;
                        qr.wait += __popc(m);
                        queued += __popc(m);
                    }
                    queue_drain(Q, A.ctr, qr, p, S.ring[wib]);
                }
                __syncwarp();
            }
        }
        __syncthreads();  // every warp is done with the list
        if (row1 < deg) {
            if (tid == 0) S.chunk = 0;
            __syncthreads();
        }
        }
        if (A.attached) {
            const int W = (deg + 63) >> 6;
            uint64_t *out = A.attached + A.loff[p];
            for (int k = tid; k < deg * KW; k += kThreads)
                if (k % KW < W) out[(uint64_t)(k / KW) * W + k % KW] = *(const uint64_t *)&S.att[2 * k];
        }
        if (qr.wait) {
            __syncwarp();
            queue_write(Q, A.ctr, qr, p, S.ring[wib], qr.wait);
            qr.wait = 0;
            __syncwarp();
        }
    }
    queue_close(Q, qr);
    // into the chunk's counters: the host adds them to the pass's only when
    // the chunk is accepted (an overflowing chunk is rerun smaller)
    const unsigned long long cands = warp_sum(cand_acc), open = warp_sum(open_acc);
    const unsigned long long alphas = listed_acc - open;  // certain ones
    if (lane == 0) {
        bump(A.ctr, C_CAND_Q, cands);
        bump(A.ctr, C_ALPHA_Q, alphas);
        // every open one is queued, and of the certain ones what is not refuted
        bump(A.ctr, C_KILLED, alphas - (queued - open));
        if (A.refute) bump(A.ctr, C_KTESTS, listed_acc);
    }
}

constexpr int kScanStep = 4;
constexpr int kScanRefill = 16;  // idle lanes that trigger a refill

// Contracted flavour.  Its lists were first made by an enumeration that
// refuted a tetrahedron by replaying insphere_w against one suspect: the first of
// its side of the triangle (a, b) along the pencil among the candidates met so
// far, or the other side's first.  That replay fused v3's and v4's weights, the
// scan's rounds them, so a pair within rounding of zero could be a violation there
// alone, and the lists depend on it.  The scan therefore asks both for what the
// filter leaves open; a tetrahedron with a ball that violates by the replay only
// is pending, and k_sos_resolve settles whether that ball was its suspect.
__device__ __noinline__ bool replay_violates(const float4 *at, uint32_t p, uint32_t v2, uint32_t v3,
                                             uint32_t v4, uint32_t y) {
    const float4 a = __ldg(&at[p]), b = __ldg(&at[v2]), c = __ldg(&at[v3]), d = __ldg(&at[v4]),
                 e = __ldg(&at[y]);
    const float pa[3] = {a.x, a.y, a.z}, pb[3] = {b.x, b.y, b.z}, pc[3] = {c.x, c.y, c.z},
                pd[3] = {d.x, d.y, d.z}, pe[3] = {e.x, e.y, e.z};
    const float o = pac::orient3d(pa, pb, pc, pd), we = pac::mul_rn(e.w, e.w);
    const float r = pac::insphere_d<pac::AtScan>(
        pa, pb, pc, pd, pe, pac::sub_rn(pac::mul_rn(a.w, a.w), we), pac::sub_rn(pac::mul_rn(b.w, b.w), we),
        pac::fma_rn(c.w, c.w, -we), pac::fma_rn(d.w, d.w, -we));
    return o < 0 ? r < 0 : r > 0;
}

// Whether that enumeration refuted the tetrahedron of positions a, b, c in p's
// list.  It took the third vertices of row a 32 at a time and the candidates of
// those 32 triangles in order, 32 per step; a candidate met the suspects of its
// own step and of those before.
__device__ __noinline__ bool replay_refuted(const TetArgs &A, uint32_t p, int a, int b, int c) {
    const MolGrid &G = A.grids[mol_of(A.mol, p)];
    if (!A.refute || G.gx > 16384 || G.gy > 16384 || G.gz > 16384) return false;
    const uint64_t e0 = A.eoff[p];
    const int deg = (int)(A.eoff[p + 1] - e0), W = (deg + 63) >> 6;
    const uint32_t *N = A.ER + e0;
    const uint64_t *L = A.link + A.loff[p];
    const bool wide = deg > 64;
    // candidates of the triangle (a, x) in word w
    auto fourth = [&](int x, int w) {
        return L[(uint64_t)a * W + w] & L[(uint64_t)x * W + w] & above_mask(x, w);
    };
    int third = 0, before = 0, rank = 0;  // b's place in row a; candidates before the triangle; c's place
    for (int x = a + 1; x < b; x++) third += (int)((L[(uint64_t)a * W + (x >> 6)] >> (x & 63)) & 1ull);
    for (int x = a + 1, k = 0; x < b; x++) {
        if (!((L[(uint64_t)a * W + (x >> 6)] >> (x & 63)) & 1ull)) continue;
        if (k++ >= (third & ~31))
            for (int w = 0; w < W; w++) before += __popcll(fourth(x, w));
    }
    for (int w = 0; w < W; w++) rank += __popcll(fourth(b, w) & ~above_mask(c - 1, w));
    const int met = ((before + rank) / 32 + 1) * 32 - before;
    const Ball B1 = pac::ld_ball(&A.at[p]), B2 = pac::ld_ball(&A.at[N[a]]), B3 = pac::ld_ball(&A.at[N[b]]);
    const float ux = B2.x - B1.x, uy = B2.y - B1.y, uz = B2.z - B1.z;
    const float vx = B3.x - B1.x, vy = B3.y - B1.y, vz = B3.z - B1.z;
    const float nx = pac::diff<1>(uy, vz, uz, vy), ny = pac::diff<1>(uz, vx, ux, vz),
                nz = pac::diff<1>(ux, vy, uy, vx);
    unsigned long long best[2] = {~0ull, ~0ull};
    int side_c = -1;
    float4 sph_c = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int w = 0, i = 0; w < W; w++) {
        for (uint64_t bits = fourth(b, w); bits && i < met; bits &= bits - 1, i++) {
            const int x = w * 64 + __ffsll((long long)bits) - 1;
            const Ball B4 = pac::ld_ball(&A.at[N[x]]);
            float4 s;
            pac::tet_alpha<pac::AtEnum>(B1, B2, B3, B4, A.alpha, s, wide);
            const bool side = pac::plus<1>(pac::sum<1>(nx, B4.x - B1.x, ny, B4.y - B1.y), nz, B4.z - B1.z) > 0.f;
            float key = pac::plus<1>(pac::sum<1>(nx, s.x, ny, s.y), nz, s.z);
            if (!side) key = -key;
            if (!isfinite(key) || (s.x == 0.f && s.y == 0.f && s.z == 0.f)) continue;
            const uint32_t k = __float_as_uint(key);
            best[side] = min(best[side], (unsigned long long)((k & 0x80000000u) ? ~k : k | 0x80000000u) << 32 |
                                             (uint32_t)x);
            if (x == c) side_c = side, sph_c = s;
        }
    }
    if (side_c < 0) return false;
    int y = (int)(best[side_c] & 0xffffffffull);
    if (y == c && best[side_c ^ 1] != ~0ull) y = (int)(best[side_c ^ 1] & 0xffffffffull);
    if (y == c) return false;
    const float4 by = A.at[N[y]];
    return surely_in_window(sph_c.x, sph_c.y, sph_c.z, by.x, by.y, by.z, 0.99f * G.step) &&
           replay_violates(A.at, p, N[a], N[b], N[c], N[y]);
}

// k_tets_scan: the empty-orthosphere test (checkTetsOrthosphere,
// AlphaComplexLargeData.cu:606-734) of the queued tetrahedra.  An entry's
// orthosphere comes from markRealTets here (or its exact counterpart), which
// also settles the alpha tests the enumeration left open.  Each lane
// owns one tetrahedron at a time and tests kScanStep window balls per step; a warp
// claims a range of queue entries at a time and a lane takes the next
// unclaimed one as soon as its own is decided (claims of A.scan_claim
// entries: one counter serves every warp).  Each (tetrahedron, ball)
// decision is taken by the certified filter of certify.cuh when it can
// prove the reference's binary32 outcome, else by replaying that
// arithmetic; A.verify replays every certified decision too and counts
// disagreements (C_CERT_BAD).  Survivors are recorded and mark their faces.
template <int V>
__global__ void __launch_bounds__(256, V == pac::kExact ? 3 : 4) k_tets_scan(TetArgs A, TetQueue Q, const unsigned long long *queued,
                                                      uint64_t limit, unsigned long long *claim) {
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1;
    unsigned long long evals = 0, oob = 0, certd = 0, bad = 0;
    uint32_t late_alpha = 0, late_killed = 0;  // alpha tests left open by the enumeration
    const uint64_t nq = *queued;
    if (nq > limit) return;  // launched ahead of the count: the host sees to it
    // claims no larger than an equal share: a short queue occupies every warp
    const unsigned share = (unsigned)min(nq / (8ull * gridDim.x), (unsigned long long)A.scan_claim);
    const unsigned claim_size = max(32u, share);
    Tally tally;
    uint64_t head = 0, tail = 0;  // this warp's claimed range (warp-uniform)
    bool have = false, more = true;
    uint32_t p = 0, v2 = 0, v3 = 0, v4 = 0, key = 0;
    float ax = 0, ay = 0, az = 0, bx = 0, by = 0, bz = 0, cx = 0, cy = 0, cz = 0, dx = 0, dy = 0,
          dz = 0, wa = 0, wb = 0, wc = 0, wd = 0, orientation = 0;
    pac::cert::Insphere ct{};
    int gX = 0, gY = 0, gZ = 0, q = 0;
    uint32_t e = 0, end = 0;
    bool zero = false, disputed = false;
    const MolGrid *G = A.grids;
    while (true) {
        // claim: idle lanes take the next entries of the warp's range
        // idle lanes take new tetrahedra together, once enough of them
        // wait (or none works): the setup then runs for many lanes at once
        unsigned want = __ballot_sync(kFull, !have);
        if (!(__popc(want) >= kScanRefill || want == kFull)) want = 0u;
        if (want && head >= tail && more) {
            uint64_t b = 0;
            if (lane == 0) b = atomicAdd(claim, (unsigned long long)claim_size);
            b = __shfl_sync(kFull, b, 0);
            head = b;
            tail = min(nq, b + (uint64_t)claim_size);
            if (head >= tail) more = false;
            for (uint64_t k = head + 16 * lane; k < tail; k += 512)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(Q.ent + k));
        }
        if (want && head < tail) {
            const int r = __popc(want & lt_mask);
            if (!have && head + r < tail) {
                const uint64_t idx = head + r;
                const uint2 en = Q.ent[idx];
                if (en.x != kNoTet) {
                    p = en.x, key = en.y & 0xffffffu;
                    const uint64_t e0 = A.eoff[p];
                    const bool wide = pac::kFused && A.eoff[p + 1] - e0 > 64;
                    const uint32_t *N = A.ER + e0;
                    v2 = __ldg(&N[key & 0xff]), v3 = __ldg(&N[(key >> 8) & 0xff]),
                    v4 = __ldg(&N[key >> 16]);
                    const Ball a1 = pac::ld_ball(&A.at[p]), a2 = pac::ld_ball(&A.at[v2]),
                               a3 = pac::ld_ball(&A.at[v3]), a4 = pac::ld_ball(&A.at[v4]);
                    float4 sph;
                    bool mark = true, live = true;
                    if constexpr (V == pac::kExact) {
                        // an alpha test that FP64 cannot decide (a flat
                        // tetrahedron, a tie) waits for k_sos_resolve, so
                        // that no lane holds up its warp with integers
                        if (en.y & kAlphaOpen) {
                            const int t = pac::ex::tet_filter(a1, a2, a3, a4, A.alpha, tally);
                            mark = t > 0;
                            if (t == 0) {
                                const unsigned long long k = atomicAdd(&A.ctr[C_PEND], 1ull);
                                if (k < A.pend_cap) A.pend[k] = en;
                            }
                        }
                        const float3 x = pac::ex::tet_centre(a1, a2, a3, a4);
                        sph = make_float4(x.x, x.y, x.z, 0.f);
                    } else {
                        mark = pac::tet_alpha(a1, a2, a3, a4, A.alpha, sph, wide);
                    }
                    if (en.y & kAlphaOpen) {
                        live = mark && !(en.y & kRefuted);
                        late_alpha += mark;
                        late_killed += mark && (en.y & kRefuted);
                    }
                    if (live) {
                        G = A.grids + mol_of(A.mol, p);
                        ax = a1.x, ay = a1.y, az = a1.z, wa = wt<V>(a1.r);
                        bx = a2.x, by = a2.y, bz = a2.z, wb = wt<V>(a2.r);
                        cx = a3.x, cy = a3.y, cz = a3.z, wc = wt<V>(a3.r);
                        dx = a4.x, dy = a4.y, dz = a4.z, wd = wt<V>(a4.r);
                        const float pa[3] = {ax, ay, az}, pb[3] = {bx, by, bz}, pc[3] = {cx, cy, cz},
                                    pd[3] = {dx, dy, dz};
                        // (exact mode: where the filter's setup accepts it, the
                        // sign of the binary32 value is the exact one)
                        const int4 cl = window_cell(*G, sph.x, sph.y, sph.z);
                        orientation = pac::orient3d(pa, pb, pc, pd);
                        // contracted flavour: other minors where the centre names no
                        // cell (a flat tetrahedron's zero sphere; see refarith.cuh)
                        if (pac::kFused && (cl.w < 0 || (uint64_t)cl.w >= G->ncell))
                            orientation = pac::orient3d<0>(pa, pb, pc, pd);
                        ct = pac::cert::setup(ax, ay, az, a1.r * a1.r, bx, by, bz, a2.r * a2.r, cx, cy,
                                              cz, a3.r * a3.r, dx, dy, dz, a4.r * a4.r, orientation,
                                              sph.x, sph.y, sph.z, G->wmax);
                        if (V == pac::kExact && !ct.ok)
                            orientation = dec_orient<V>(pa, pb, pc, pd, wa, wb, wc, wd, tally);
                        gX = cl.x, gY = cl.y, gZ = cl.z;
                        q = 0;
                        zero = disputed = false;
                        window_centre(*G, A.cellbeg, cl, e, end, oob);
                        have = true;
                    }
                }
            }
            head = min(tail, head + (uint64_t)__popc(want));
        }
        if (!__any_sync(kFull, have)) {
            if (!more) break;
            continue;
        }
        if (!have) continue;
        if (e < end) {
            // kScanStep window balls per step: their loads overlap, and the
            // warp-wide bookkeeping above runs once per step
            const uint32_t cnt = min(end - e, (uint32_t)kScanStep);
            Ball bq[kScanStep];
#pragma unroll
            for (int t = 0; t < kScanStep; t++)
                bq[t] = pac::ld_ball(&A.at[e + min((uint32_t)t, cnt - 1)]);
            const uint32_t x0 = e;
            e += cnt;
            bool viol = false;
#pragma unroll
            for (int t = 0; t < kScanStep; t++) {
                const uint32_t x = x0 + t;
                const Ball bb = bq[t];
                if ((uint32_t)t >= cnt || viol || x == p || x == v2 || x == v3 || x == v4) continue;
                const float we = wt<V>(bb.r);
                int dec = pac::cert::test(ct, bb.x, bb.y, bb.z, bb.r * bb.r);
                evals++;
                if (dec >= 0) certd++;
                if (dec < 0 || A.verify) {
                    const float pa[3] = {ax, ay, az}, pb[3] = {bx, by, bz}, pc[3] = {cx, cy, cz},
                                pd[3] = {dx, dy, dz}, pe[3] = {bb.x, bb.y, bb.z};
                    float res;
                    if constexpr (V == pac::kExact) {
                        // the FP64 filter alone: what it cannot tell, a zero
                        // among it, waits for k_sos_resolve, so that no lane
                        // holds up its warp with integers
                        res = (float)pac::ex::insphere_filter(
                            Ball{ax, ay, az, wa}, Ball{bx, by, bz, wb}, Ball{cx, cy, cz, wc},
                            Ball{dx, dy, dz, wd}, Ball{bb.x, bb.y, bb.z, we}, tally);
                    } else {
                        res = dec_insphere<V, pac::AtScan>(pa, pb, pc, pd, pe, wa, wb, wc, wd, we, tally);
                    }
                    const int rdec = (orientation < 0 ? (res < 0) : (res > 0)) ? 1 : 0;
                    if (dec >= 0 && dec != rdec && !(V == pac::kExact && res == 0)) bad++;
                    if (dec < 0) {
                        dec = rdec;
                        if (res == 0) zero = true;
                        if constexpr (pac::kFused)
                            if (!rdec && A.refute && !disputed)
                                disputed = replay_violates(A.at, p, v2, v3, v4, x);
                    }
                }
                viol = dec == 1;
            }
            if (viol) have = false;
            continue;
        }
        bool found = false;
        while (q < kWindowParts && !found) found = window_part(*G, A.cellbeg, gX, gY, gZ, q++, e, end);
        if (!found) {
            const uint32_t open = pac::kFused ? (disputed ? kDisputed : 0u) | (zero ? kTied : 0u) : 0u;
            emit_survivor(A.eoff, A.ER, A.loff, A.faces, A.surv, A.surv_cap, A.pend, A.pend_cap,
                          A.ctr, A.tcount, p, key | open, v2, v3, v4, zero || disputed);
            have = false;
        }
    }
    evals = warp_sum(evals);
    oob = warp_sum(oob);
    certd = warp_sum(certd);
    bad = warp_sum(bad);
    const unsigned long long la = warp_sum(late_alpha), lk = warp_sum(late_killed);
    flush_tally<V>(tally, A.ctr);
    if (lane == 0) {
        bump(A.ctr, C_ALPHA_Q, la);
        bump(A.ctr, C_KILLED, lk);
        bump(A.ctr, C_INSPHERE, evals);
        bump(A.ctr, C_OOB, oob);
        bump(A.ctr, C_CERT, certd);
        bump(A.ctr, C_CERT_BAD, bad);
    }
}

// The tetrahedra that the scan left pending (no certain violator, but a ball
// whose insphere value is exactly 0 or, in the exact mode, beyond the FP64
// filters, or an alpha test beyond them): the test again, with the exact arithmetic and the reference's
// simulation of simplicity for the zeros (AlphaComplexLargeData.cu:645-652,
// 659-667).  A warp per tetrahedron, its lanes over the balls of a window
// cell, the cells in the reference's order: the few pending ones are a chain of
// integer evaluations each, so what counts is that they run beside each other
// and outside the scan's warps (25,000 lattice-snapped balls, 156 zeros: a thread
// per tetrahedron 2.4 ms, now 0.1; exact mode, 5,395 zeros and some 50,000 open
// alpha tests: 37 ms here and 37 ms in the scan's lanes, now 3.5 and 1.4).
template <int V>
__global__ void __launch_bounds__(128) k_sos_resolve(TetArgs A, uint64_t npend) {
    const int lane = threadIdx.x & 31;
    const uint64_t t = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (t >= npend) return;
    uint2 pk = A.pend[t];
    const uint64_t p = pk.x;
    const int a = pk.y & 0xff, b = (pk.y >> 8) & 0xff, c = (pk.y >> 16) & 0xff;
    const uint64_t e0 = A.eoff[p];
    const int deg = (int)(A.eoff[p + 1] - e0);
    const int W = (deg + 63) >> 6;
    const uint32_t *N = A.ER + e0;
    const uint32_t v[4] = {(uint32_t)p, N[a], N[b], N[c]};
    Ball B[4];
    for (int k = 0; k < 4; k++) B[k] = pac::ld_ball(&A.at[v[k]]);
    Tally tally;
    float4 sphere;
    const bool mark = dec_tet<V, pac::AtSos>(B[0], B[1], B[2], B[3], A.alpha, sphere, false, tally);
    bool tied = true;
    if constexpr (pac::kFused) {
        tied = pk.y & kTied;
        if ((pk.y & kDisputed) && replay_refuted(A, (uint32_t)p, a, b, c)) return;
        pk.y &= 0xffffffu;
    }
    if (pk.y & kAlphaOpen) {  // its alpha test was left open too
        const bool refuted = pk.y & kRefuted;
        if (lane == 0 && mark) {
            bump(A.ctr, C_ALPHA_Q, 1);
            bump(A.ctr, C_KILLED, refuted);
        }
        if (!mark || refuted) {
            flush_tally<V>(lane == 0 ? tally : Tally{}, A.ctr);
            return;
        }
        pk.y &= 0xffffffu;
    }
    const MolGrid G = A.grids[mol_of(A.mol, p)];
    float pts[5][3], ws[5];
    int idx[5];
    for (int k = 0; k < 4; k++) {
        pts[k][0] = B[k].x;
        pts[k][1] = B[k].y;
        pts[k][2] = B[k].z;
        ws[k] = wt<V>(B[k].r);
        idx[k] = (int)A.orig[v[k]] + 1;
    }
    const float orient = pac::orient3d(pts[0], pts[1], pts[2], pts[3]);
    const pac::cert::Insphere ct = pac::cert::setup(
        B[0].x, B[0].y, B[0].z, B[0].r * B[0].r, B[1].x, B[1].y, B[1].z, B[1].r * B[1].r, B[2].x,
        B[2].y, B[2].z, B[2].r * B[2].r, B[3].x, B[3].y, B[3].z, B[3].r * B[3].r, orient, sphere.x,
        sphere.y, sphere.z, G.wmax);
    const float orientation =
        dec_orient<V>(pts[0], pts[1], pts[2], pts[3], ws[0], ws[1], ws[2], ws[3], tally);
    if (lane) tally = Tally{};  // every lane took the same decisions so far
    int gridX = pac::cell_coord(sphere.x, G.minx, G.step);
    int gridY = pac::cell_coord(sphere.y, G.miny, G.step);
    int gridZ = pac::cell_coord(sphere.z, G.minz, G.step);
    int cc = lin3(gridX, gridY, gridZ, G.gx, G.gy);
    bool viol = false;
    uint32_t calls = 0;
    for (int q = 0; q < 27 && tied && !viol; q++) {
        uint32_t beg, end;
        if (q == 0) {
            if (cc < 0 || (uint64_t)cc >= G.ncell) continue;
            beg = A.cellbeg[G.cell_base + cc];
            end = A.cellbeg[G.cell_base + cc + 1];
        } else {
            int r = q - 1 + (q >= 14 ? 1 : 0);
            int i = r / 9 - 1, j = (r / 3) % 3 - 1, k = r % 3 - 1;
            int zz = (int)((unsigned)gridZ + (unsigned)i), yy = (int)((unsigned)gridY + (unsigned)j),
                xx = (int)((unsigned)gridX + (unsigned)k);
            if ((zz >= G.gz) || (yy >= G.gy) || (xx >= G.gx)) continue;
            if ((zz < 0) || (yy < 0) || (xx < 0)) continue;
            uint64_t gc = G.cell_base + (uint64_t)lin3(xx, yy, zz, G.gx, G.gy);
            beg = A.cellbeg[gc];
            end = A.cellbeg[gc + 1];
        }
        for (uint32_t base = beg; base < end && !viol; base += 32) {
            const uint32_t e = base + lane;
            bool hit = false, zero = false;
            if (e < end && e != v[0] && e != v[1] && e != v[2] && e != v[3]) {
                const Ball atom = pac::ld_ball(&A.at[e]);
                const int dec = pac::cert::test(ct, atom.x, atom.y, atom.z, atom.r * atom.r);
                hit = dec == 1;
                if (dec < 0) {
                    pts[4][0] = atom.x;
                    pts[4][1] = atom.y;
                    pts[4][2] = atom.z;
                    ws[4] = wt<V>(atom.r);
                    float result = dec_insphere<V, pac::AtSos>(pts[0], pts[1], pts[2], pts[3], pts[4], ws[0],
                                                               ws[1], ws[2], ws[3], ws[4], tally);
                    zero = result == 0;
                    if (zero) {
                        idx[4] = (int)A.orig[e] + 1;
                        int status = 0;
                        result = (float)pac::sos_orientation(pts, ws, idx, &status, V == pac::kExact);
                        if (status == 1) atomicAdd(&A.ctr[C_SOS_RANGE], 1ull);
                    }
                    hit = orientation < 0 ? (result < 0) : (result > 0);
                }
            }
            // the zeros up to the first violator: those the reference's loop
            // evaluates
            const unsigned hits = __ballot_sync(kFull, hit), zeros = __ballot_sync(kFull, zero);
            calls += __popc(hits ? zeros & (hits ^ (hits - 1)) : zeros);
            viol = hits != 0;
        }
    }
    flush_tally<V>(tally, A.ctr);
    if (lane) return;
    bump(A.ctr, C_SOS, calls);
    if (viol) return;
    unsigned long long q = atomicAdd(&A.ctr[C_SURV], 1ull);
    if (q < A.surv_cap) A.surv[q] = pk;
    atomicAdd(&A.tcount[p], 1u);
    const uint64_t lp = A.loff[p];
    mark_face(A.faces, lp, W, a, b);
    mark_face(A.faces, lp, W, a, c);
    mark_face(A.faces, lp, W, b, c);
    const uint32_t v2 = v[1];
    const uint64_t e2 = A.eoff[v2];
    const int deg2 = (int)(A.eoff[v2 + 1] - e2);
    const int mb = lbound(A.ER + e2, deg2, v[2]), mc = lbound(A.ER + e2, deg2, v[3]);
    mark_face(A.faces, A.loff[v2], (deg2 + 63) >> 6, mb, mc);
}

// Survivors to per-ball rows, ordered by (a, b, c) -- the order in which the
// reference enumerates them: k_tet_scatter collects each ball's keys, then a
// thread per tetrahedron counts the smaller keys of its ball (a few to a few
// tens, in L1) and writes its row there.  (A thread per ball sorting by
// insertion: 29 us at 211 balls, 56 at 25,000.)
__device__ __forceinline__ uint32_t key_order(uint32_t k) {
    return ((k & 0xff) << 16) | (k & 0xff00) | ((k >> 16) & 0xff);
}
__global__ void k_tet_scatter(const uint2 *surv, uint64_t ns, const uint64_t *toff,
                              uint32_t *cursor, uint32_t *keys, uint64_t p_lo, uint64_t p_hi) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ns) return;
    uint2 s = surv[t];
    if (s.x < p_lo || s.x >= p_hi) return;  // a slab's halo: not this pass's output
    keys[toff[s.x] + atomicAdd(&cursor[s.x], 1u)] = key_order(s.y);
}
__global__ void k_tet_emit(const uint2 *surv, uint64_t ns, const uint64_t *toff, const uint32_t *keys,
                           const uint64_t *eoff, const uint32_t *ER, const uint32_t *orig,
                           uint32_t *out, uint64_t p_lo, uint64_t p_hi) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ns) return;
    const uint2 s = surv[t];
    if (s.x < p_lo || s.x >= p_hi) return;
    const uint64_t b = toff[s.x], e = toff[s.x + 1];
    const uint32_t mine = key_order(s.y);
    uint64_t at = b;
    for (uint64_t i = b; i < e; i++) at += __ldg(&keys[i]) < mine;
    const uint32_t *N = ER + eoff[s.x];
    *(uint4 *)&out[4 * at] = make_uint4(orig[s.x], orig[N[s.y & 0xff]], orig[N[(s.y >> 8) & 0xff]],
                                        orig[N[(s.y >> 16) & 0xff]]);
}
__global__ void k_map4(uint64_t nq, const uint32_t *orig, uint32_t *tets) {
    uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nq) return;
    uint4 v = *(uint4 *)&tets[4 * t];
    *(uint4 *)&tets[4 * t] = make_uint4(orig[v.x], orig[v.y], orig[v.z], orig[v.w]);
}

// ------------------------------------------------------------------ attachment
// Final triangles of ball v1: tetrahedron faces, plus the alpha triangles
// that are neither faces nor found attached by the enumeration and whose orthosphere no other ball of the 27-cell
// window reaches (checkDanglingTris, AlphaComplexLargeData.cu:798-872).
// Work stealing: one warp per ball v1, balls handed out from a counter.  The alpha triangles
// of v1 that are not tetrahedron faces are queued in shared memory row by
// row; each lane takes one, recomputes its orthosphere (markRealTriangles)
// and tests one window ball per step (checkDanglingTris,
// AlphaComplexLargeData.cu:798-872), taking the next queued triangle as soon
// as its own is decided.  An unattached triangle sets its bit in `faces`.
// Then the warp counts v1's final triangles and marks their edges.
constexpr int kTQCap = 256;
constexpr int kTARefill = 24;  // idle lanes that trigger a refill

template <int V>
__global__ void __launch_bounds__(256, 4) k_tri_attach(uint64_t p_lo, uint64_t n,
                                                       const float4 *__restrict__ at,
                                                       const uint64_t *__restrict__ eoff,
                                                       const uint32_t *__restrict__ ER,
                                                       const uint64_t *__restrict__ loff,
                                                       const uint64_t *__restrict__ link,
                                                       const uint64_t *__restrict__ attached,
                                                       uint64_t *faces, uint32_t *tricount,
                                                       uint8_t *eflag, const uint32_t *cellbeg,
                                                       const uint32_t *mol, const MolGrid *grids,
                                                       float alpha, unsigned long long *ctr) {
    __shared__ uint16_t qa[8][kTQCap], qb[8][kTQCap];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1;
    unsigned long long oob = 0;
    Tally tally;
    while (true) {
        uint64_t p = 0;
        if (lane == 0) p = p_lo + atomicAdd(&ctr[C_NEXT], 1ull);
        p = __shfl_sync(kFull, p, 0);
        if (p >= n) break;
        const uint64_t e0 = eoff[p];
        const int deg = (int)(eoff[p + 1] - e0);
        uint32_t count = 0;
        if (deg >= 2) {
            const int W = (deg + 63) >> 6;
            const uint32_t *N = ER + e0;
            const uint64_t lp = loff[p];
            const Ball A0 = pac::ld_ball(&at[p]);
            const MolGrid *G = grids + mol_of(mol, p);
            int row = 0;       // next row to queue (warp-uniform)
            uint64_t rbits[kMaxW];  // unqueued candidate bits of `row`
            bool rloaded = false;
            // lane state
            bool have = false;
            int ta = 0, tb = 0;
            uint32_t v1 = 0, v2 = 0;
            float px = 0, py = 0, pz = 0, cur = 0;
            int gX = 0, gY = 0, gZ = 0, q = 0;
            uint32_t e = 0, end = 0;
            int qn = 0, head = 0;  // shared queue (warp-uniform)
            while (true) {
                // refill the queue from the remaining rows
                if (head >= qn) {
                    qn = 0;
                    head = 0;
                    while (row < deg - 1 && qn < kTQCap - 64) {
                        if (!rloaded) {
#pragma unroll
                            for (int w = 0; w < kMaxW; w++) {
                                const uint64_t k = lp + (uint64_t)row * W + w;
                                rbits[w] = w < W ? (link[k] & ~faces[k]) : 0;
                                // (never with the plain-xmp formulas)
                                if constexpr (V != pac::kPlainXmp)
                                    if (attached && w < W) rbits[w] &= ~attached[k];
                            }
                            rloaded = true;
                        }
                        int nc = 0;
#pragma unroll
                        for (int w = 0; w < kMaxW; w++) nc += __popcll(rbits[w]);
                        int take = min(nc, kTQCap - qn);
                        for (int k0 = 0; k0 < take; k0 += 32) {
                            int k = k0 + lane;
                            if (k < take) {
                                qa[wib][qn + k] = (uint16_t)row;
                                qb[wib][qn + k] = (uint16_t)select_bit(rbits, W, k);
                            }
                        }
                        qn += take;
                        if (take == nc) {
                            row++;
                            rloaded = false;
                        } else {
                            // drop the queued bits from the row, keep the rest
                            for (int k = 0; k < take; k++) {
                                int b = select_bit(rbits, W, 0);
                                rbits[b >> 6] &= ~(1ull << (b & 63));
                            }
                        }
                    }
                    __syncwarp();
                }
                // idle lanes take new triangles together, once enough of
                // them wait (or none works): the setup runs for many lanes
                // at a time instead of for a few in every step
                unsigned want = __ballot_sync(kFull, !have);
                if (want && head < qn && (__popc(want) >= kTARefill || want == kFull)) {
                    int r = __popc(want & lt_mask);
                    if (!have && head + r < qn) {
                        ta = qa[wib][head + r];
                        tb = qb[wib][head + r];
                        v1 = N[ta];
                        v2 = N[tb];
                        const float4 p1 =
                            tri_sphere<V>(A0, pac::ld_ball(&at[v1]), pac::ld_ball(&at[v2]), alpha);
                        px = p1.x;
                        py = p1.y;
                        pz = p1.z;
                        cur = p1.w;
                        gX = pac::cell_coord(p1.x, G->minx, G->step);
                        gY = pac::cell_coord(p1.y, G->miny, G->step);
                        gZ = pac::cell_coord(p1.z, G->minz, G->step);
                        q = 0;
                        window_centre(*G, cellbeg, make_int4(gX, gY, gZ, lin3(gX, gY, gZ, G->gx, G->gy)),
                                      e, end, oob);
                        have = true;
                    }
                    head = min(qn, head + __popc(want));
                }
                if (!__any_sync(kFull, have)) {
                    if (head >= qn && row >= deg - 1) break;
                    continue;
                }
                if (!have) continue;
                if (e < end) {
                    if constexpr (V != pac::kExact) {
                        // two window balls per step (independent loads)
                        const uint32_t x0 = e, x1 = (e + 1 < end) ? e + 1 : e;
                        e = x1 + 1;
                        const bool ok0 = !(x0 == (uint32_t)p || x0 == v1 || x0 == v2);
                        const bool ok1 = x1 != x0 && !(x1 == (uint32_t)p || x1 == v1 || x1 == v2);
                        const Ball b0 = pac::ld_ball(&at[x0]), b1 = pac::ld_ball(&at[x1]);
                        const bool t0 = pac::attached(b0, px, py, pz, cur);
                        const bool t1 = pac::attached(b1, px, py, pz, cur);
                        if ((ok0 && t0) || (ok1 && t1)) have = false;
                    } else {
                        uint32_t x = e++;
                        if (x == (uint32_t)p || x == v1 || x == v2) continue;
                        if (dec_tri_attached<V>(A0, at, v1, v2, pac::ld_ball(&at[x]), px, py, pz,
                                                cur, tally))
                            have = false;
                    }
                    continue;
                }
                bool found = false;
                while (q < kWindowParts && !found)
                    found = window_part(*G, cellbeg, gX, gY, gZ, q++, e, end);
                if (!found) {
                    atomicOr((unsigned long long *)&faces[lp + (uint64_t)ta * W + (tb >> 6)],
                             1ull << (tb & 63));
                    have = false;
                }
            }
            __syncwarp();
            __threadfence_block();
            // count the final triangles and mark their edges: a lane per
            // row, 32 rows at a time
            for (int a0 = 0; a0 < deg - 1; a0 += 32) {
                const int a = a0 + lane;
                uint64_t fin[kMaxW];
                int nf = 0;
#pragma unroll
                for (int w = 0; w < kMaxW; w++) {
                    fin[w] = (a < deg - 1 && w < W) ? faces[lp + (uint64_t)a * W + w] : 0;
                    nf += __popcll(fin[w]);
                }
                count += (uint32_t)warp_sum((unsigned long long)nf);
                if (!nf) continue;
                eflag[e0 + a] = 1;
                const uint32_t va = N[a];
                const uint64_t e1 = eoff[va];
                const int deg1 = (int)(eoff[va + 1] - e1);
#pragma unroll
                for (int w = 0; w < kMaxW; w++) {
                    uint64_t bits = fin[w];
                    while (bits) {
                        const int b = w * 64 + __ffsll((long long)bits) - 1;
                        bits &= bits - 1;
                        eflag[e0 + b] = 1;
                        const uint32_t vb = N[b];
                        const int pos = lbound(ER + e1, deg1, vb);
                        if (pos < deg1 && ER[e1 + pos] == vb) eflag[e1 + pos] = 1;
                    }
                }
            }
        }
        if (lane == 0) tricount[p] = count;
    }
    oob = warp_sum(oob);
    flush_tally<V>(tally, ctr);
    if (lane == 0) bump(ctr, C_OOB, oob);
}

// Final edges: edges of final triangles, plus the alpha edges whose radical
// foot no other ball reaches (checkDanglingEdges, AlphaComplexLargeData.cu:924-1011).
template <int V>
__global__ void __launch_bounds__(256) k_edge_final(uint64_t p_lo, uint64_t n,
                                                    const float4 *__restrict__ at,
                                                    const uint64_t *__restrict__ eoff,
                                                    const uint32_t *__restrict__ ER,
                                                    uint8_t *eflag, const uint32_t *cellbeg,
                                                    const uint32_t *mol, const MolGrid *grids,
                                                    unsigned long long *ctr) {
    const int lane = threadIdx.x & 31;
    unsigned long long oob = 0;
    Tally tally;
    // balls handed out by a counter (persistent warps)
    for (;;) {
        uint64_t p = 0;
        if (lane == 0) p = p_lo + atomicAdd(&ctr[C_NEXT], 1ull);
        p = __shfl_sync(kFull, p, 0);
        if (p >= n) break;
        const uint64_t e0 = eoff[p];
        const int deg = (int)(eoff[p + 1] - e0);
        if (!deg) continue;
        const Ball a1 = pac::ld_ball(&at[p]);
        const MolGrid G = grids[mol_of(mol, p)];
        for (int k = lane; k < deg; k += 32) {
            if (eflag[e0 + k]) continue;
            const uint32_t v2 = ER[e0 + k];
            float px, py, pz, currentDist;
            const Ball a2 = pac::ld_ball(&at[v2]);
            edge_sphere<V>(a1, a2, px, py, pz, currentDist);
            int gridX = pac::cell_coord(px, G.minx, G.step);
            int gridY = pac::cell_coord(py, G.miny, G.step);
            int gridZ = pac::cell_coord(pz, G.minz, G.step);
            int cc = lin3(gridX, gridY, gridZ, G.gx, G.gy);
            bool att = false;
            for (int q = 0; q < 27 && !att; q++) {
                uint32_t beg, end;
                if (q == 0) {
                    if (cc < 0 || (uint64_t)cc >= G.ncell) {
                        oob++;
                        continue;
                    }
                    beg = cellbeg[G.cell_base + cc];
                    end = cellbeg[G.cell_base + cc + 1];
                } else {
                    int r = q - 1 + (q >= 14 ? 1 : 0);
                    int i = r / 9 - 1, j = (r / 3) % 3 - 1, kk = r % 3 - 1;
                    int zz = (int)((unsigned)gridZ + (unsigned)i),
                        yy = (int)((unsigned)gridY + (unsigned)j),
                        xx = (int)((unsigned)gridX + (unsigned)kk);
                    if ((zz >= G.gz) || (yy >= G.gy) || (xx >= G.gx)) continue;
                    if ((zz < 0) || (yy < 0) || (xx < 0)) continue;
                    uint64_t gc = G.cell_base + (uint64_t)lin3(xx, yy, zz, G.gx, G.gy);
                    beg = cellbeg[gc];
                    end = cellbeg[gc + 1];
                }
                for (uint32_t e = beg; e < end; e++) {
                    if (e == p || e == v2) continue;
                    if (dec_edge_attached<V>(a1, a2, pac::ld_ball(&at[e]), px, py, pz,
                                             currentDist, tally)) {
                        att = true;
                        break;
                    }
                }
            }
            if (!att) eflag[e0 + k] = 1;
        }
    }
    oob = warp_sum(oob);
    flush_tally<V>(tally, ctr);
    if (lane == 0) bump(ctr, C_OOB, oob);
}

// ------------------------------------------------------------------ emission
// a warp per ball, its lanes over the ball's alpha edges (a thread per ball
// walking its row alone: 40 us at 211 balls, 112 at 25,000)
__global__ void __launch_bounds__(256) k_emit_edges(uint64_t n, const uint64_t *eoff, const uint32_t *ER,
                                                    const uint8_t *eflag, const uint64_t *epos,
                                                    const uint32_t *orig, uint32_t *out) {
    const int lane = threadIdx.x & 31;
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t p = warp; p < n; p += nwarps) {
        const uint32_t o = orig[p];
        const uint64_t end = eoff[p + 1];
        for (uint64_t k = eoff[p] + lane; k < end; k += 32)
            if (eflag[k]) *(uint2 *)&out[2 * epos[k]] = make_uint2(o, orig[ER[k]]);
    }
}
__global__ void __launch_bounds__(256) k_emit_tris(uint64_t p_lo, uint64_t n, const uint64_t *eoff,
                                                   const uint32_t *ER, const uint64_t *loff,
                                                   const uint64_t *faces, const uint64_t *tpos,
                                                   const uint32_t *orig, uint32_t *out) {
    const int lane = threadIdx.x & 31;
    uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t p = p_lo + warp; p < n; p += nwarps) {
        const int deg = (int)(eoff[p + 1] - eoff[p]);
        if (deg < 2) continue;
        const int W = (deg + 63) >> 6;
        const uint32_t *N = ER + eoff[p];
        const uint32_t o0 = orig[p];
        const uint64_t lp = loff[p];
        uint64_t q = tpos[p];
        // a lane per row, 32 rows at a time; rows in order, b ascending
        // within a row
        for (int a0 = 0; a0 < deg - 1; a0 += 32) {
            const int a = a0 + lane;
            uint64_t f[kMaxW];
            int nf = 0;
#pragma unroll
            for (int w = 0; w < kMaxW; w++) {
                f[w] = (a < deg - 1 && w < W) ? faces[lp + (uint64_t)a * W + w] : 0;
                nf += __popcll(f[w]);
            }
            int incl = nf;
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(kFull, incl, 31);
            if (nf) {
                const uint32_t o1 = orig[N[a]];
                uint64_t at = q + (uint64_t)(incl - nf);
#pragma unroll
                for (int w = 0; w < kMaxW; w++) {
                    uint64_t bits = f[w];
                    while (bits) {
                        const int b = w * 64 + __ffsll((long long)bits) - 1;
                        bits &= bits - 1;
                        out[3 * at] = o0;
                        out[3 * at + 1] = o1;
                        out[3 * at + 2] = orig[N[b]];
                        at++;
                    }
                }
            }
            q += (uint64_t)total;
        }
    }
}
// first output row of every molecule (and the totals at m = n_mol)
__global__ void k_mol_rows(uint32_t n_mol, const uint64_t *ball_off, uint64_t n,
                           const uint64_t *eoff, const uint64_t *epos, const uint64_t *tpos,
                           const uint64_t *toff, uint64_t *rows) {
    uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > n_mol) return;
    uint64_t b = m < n_mol ? ball_off[m] : n;
    rows[m] = epos[eoff[b]];
    rows[(n_mol + 1) + m] = tpos[b];
    rows[2 * (n_mol + 1) + m] = toff[b];
}

// ------------------------------------------------------------------ host
// The enumeration kernels' shared memory exceeds the static 48 KB: allow it
// once per context, whose options fix the kernels it launches (the attribute
// belongs to the kernel; another context setting it again, on whatever thread,
// changes nothing).
template <int M>
static int enum_smem_optin(pac::Ctx &ctx) {
    if (ctx.enum_optin) return PAC_OK;
    CK(cudaFuncSetAttribute(k_tets_enum<1, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)sizeof(EnumSmem<1>)));
    CK(cudaFuncSetAttribute(k_tets_enum<2, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)sizeof(EnumSmem<2>)));
    CK(cudaFuncSetAttribute(k_tets_enum<kMaxW, M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)sizeof(EnumSmem<kMaxW>)));
    ctx.enum_optin = true;
    return PAC_OK;
}

// The enumeration of the balls [lo, hi): their classes, then one launch per
// class that the pass's largest degree can reach, the longest blocks first.
template <int M>
static int enumerate(pac::Ctx &ctx, const pac::PipelineConfig &cfg, const TetArgs &A,
                     const TetQueue &Q, uint64_t lo, uint64_t hi, uint32_t *list, uint64_t maxdeg) {
    cudaStream_t s = ctx.stream;
    int rc = enum_smem_optin<M>(ctx);
    if (rc) return rc;
    const uint64_t balls = hi - lo;
    const bool sparse = balls >= kSparseBalls;
    k_classes<<<(unsigned)((balls + 255) / 256), 256, 0, s>>>(lo, hi, A.n, A.eoff, A.loff, A.attached, 3,
                                                               sparse ? 32 : 0, list, A.ctr);
    LAUNCH_CHECK(ctx);
    const unsigned light = (unsigned)std::min<uint64_t>(balls, 148u * (unsigned)std::max(1, cfg.enum_blocks));
    const unsigned heavy = (unsigned)std::min<uint64_t>(balls, 148u * (unsigned)std::max(1, cfg.heavy_blocks));
    // the few balls of the largest class take long one by one: beside the rest
    const bool aside = maxdeg > 128;
    if (aside) {
        rc = pac::side_stream(ctx);
        if (rc) return rc;
        CK(cudaEventRecord(ctx.side_ev[0], s));
        CK(cudaStreamWaitEvent(ctx.side, ctx.side_ev[0], 0));
        k_tets_enum<kMaxW, M><<<(unsigned)std::min<uint64_t>(heavy, 148), EnumSmem<kMaxW>::kWarps * 32,
                                sizeof(EnumSmem<kMaxW>), ctx.side>>>(A, Q, list + 2 * A.n, 2);
        LAUNCH_CHECK(ctx);
        CK(cudaEventRecord(ctx.side_ev[1], ctx.side));
    }
    if (maxdeg > 64) {
        k_tets_enum<2, M><<<heavy, EnumSmem<2>::kWarps * 32, sizeof(EnumSmem<2>), s>>>(
            A, Q, list + A.n, 1);
        LAUNCH_CHECK(ctx);
    }
    if (maxdeg >= 3) {
        k_tets_enum<1, M><<<light, EnumSmem<1>::kWarps * 32, sizeof(EnumSmem<1>), s>>>(A, Q, list, 0);
        LAUNCH_CHECK(ctx);
    }
    if (sparse) {
        using Smem = EnumSmem<1, 32>;
        k_tets_enum<1, M, 32><<<(unsigned)std::min<uint64_t>(balls, 148u * Smem::kBlocks), Smem::kWarps * 32,
                                sizeof(Smem), s>>>(A, Q, list + kSparse * A.n, kSparse);
        LAUNCH_CHECK(ctx);
    }
    if (aside) CK(cudaStreamWaitEvent(s, ctx.side_ev[1], 0));
    return PAC_OK;
}

struct Timer {
    pac::Ctx &ctx;
    int i = 0;
    explicit Timer(pac::Ctx &c) : ctx(c) {}
    void mark() {  // events 0..13 (14 and 15 time the orthosphere test)
        if (i < 14) cudaEventRecord(ctx.ev[i++], ctx.stream);
    }
    double ms(int a, int b) {
        float f = 0;
        if (a < i && b < i) cudaEventElapsedTime(&f, ctx.ev[a], ctx.ev[b]);
        return f;
    }
};

static unsigned blocks_for(uint64_t n, unsigned threads) {
    uint64_t b = (n + threads - 1) / threads;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(b, 0x7fffffffu));
}
static unsigned warp_blocks(uint64_t items) {
    // 8 warps per block, grid-stride: enough blocks to fill 148 SMs many times
    uint64_t b = (items + 7) / 8;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(b, 148ull * 64));
}

template <int V>
static int run_pass_v(pac::Ctx &ctx, const pac::PipelineConfig &cfg, const pac::PassInput &in,
                      pac::PassOutput &out, pac_stats *st) {
    cudaStream_t s = ctx.stream;
    pac::Arena &ar = ctx.arena;
    const uint64_t n = in.n;
    const uint32_t nm = in.n_mol;
    Timer tm(ctx);
    tm.mark();  // 0

    unsigned long long *ctr = ar.alloc_n<unsigned long long>(C_NCOUNTERS);
    int *mm = ar.alloc_n<int>(8 * (size_t)nm);
    MolGrid *grids = ar.alloc_n<MolGrid>(nm);
    uint64_t *ncell_d = ar.alloc_n<uint64_t>(nm);
    uint64_t *d_off = ar.alloc_n<uint64_t>(nm + 1);
    uint32_t *mol = nullptr;
    if (!ctr || !mm || !grids || !ncell_d || !d_off) return PAC_ERR_OOM;
    CK(cudaMemsetAsync(ctr, 0, sizeof(unsigned long long) * C_NCOUNTERS, s));
    {
        std::vector<int> init(8 * (size_t)nm);
        for (uint32_t m = 0; m < nm; m++)
            for (int q = 0; q < 4; q++) {
                init[8 * m + q] = 0x7fffffff;
                init[8 * m + 4 + q] = (int)0x80000000;
            }
        CK(cudaMemcpyAsync(mm, init.data(), sizeof(int) * init.size(), cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(d_off, in.h_offsets, sizeof(uint64_t) * (nm + 1),
                           cudaMemcpyHostToDevice, s));
        // (pageable sources are staged before the calls return)
    }
    if (nm > 1) {
        mol = ar.alloc_n<uint32_t>(n);
        if (!mol) return PAC_ERR_OOM;
        k_mol_ids<<<nm, 256, 0, s>>>(d_off, nm, mol);
        LAUNCH_CHECK(ctx);
    }
    k_bbox<<<blocks_for(n, 256), 256, 0, s>>>(in.d_balls, n, mol, mm, ctr);
    LAUNCH_CHECK(ctx);
    k_grid<<<blocks_for(nm, 128), 128, 0, s>>>(mm, nm, in.sol, in.alpha, grids, ncell_d);
    LAUNCH_CHECK(ctx);
    std::vector<MolGrid> hg(nm);
    unsigned long long bad = 0;
    CK(cudaMemcpyAsync(hg.data(), grids, sizeof(MolGrid) * nm, cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&bad, ctr + C_NONFINITE, sizeof(bad), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (bad) return pac::set_error(PAC_ERR_INVALID_ARG, "non-finite ball coordinate or radius");
    uint64_t total_cells = 0;
    for (uint32_t m = 0; m < nm; m++) {
        if (hg[m].gx <= 0 || hg[m].gy <= 0 || hg[m].gz <= 0 || hg[m].ncell > 0x7fffffffull)
            return pac::set_error(PAC_ERR_CAPACITY,
                                  "grid of molecule " + std::to_string(m) +
                                      " exceeds the reference's int cell index range");
        hg[m].cell_base = total_cells;
        hg[m].atom_base = in.h_offsets[m];
        total_cells += hg[m].ncell;
    }
    if (total_cells >= 0xffffffffull)
        return pac::set_error(PAC_ERR_CAPACITY, "more than 2^32 cells in one pass");
    CK(cudaMemcpyAsync(grids, hg.data(), sizeof(MolGrid) * nm, cudaMemcpyHostToDevice, s));

    // ---- binning
    uint32_t *gcell = ar.alloc_n<uint32_t>(n), *slot = ar.alloc_n<uint32_t>(n);
    uint32_t *cellcnt = ar.alloc_n<uint32_t>(total_cells);
    uint32_t *cellbeg = ar.alloc_n<uint32_t>(total_cells + 1);
    uint32_t *perm = ar.alloc_n<uint32_t>(n);
    float4 *at = ar.alloc_n<float4>(n);
    uint32_t *orig = ar.alloc_n<uint32_t>(n), *cellof = ar.alloc_n<uint32_t>(n);
    if (!gcell || !slot || !cellcnt || !cellbeg || !perm || !at || !orig || !cellof)
        return PAC_ERR_OOM;
    CK(cudaMemsetAsync(cellcnt, 0, sizeof(uint32_t) * total_cells, s));
    k_cellkey<<<blocks_for(n, 256), 256, 0, s>>>(in.d_balls, n, mol, grids, gcell, slot, cellcnt);
    LAUNCH_CHECK(ctx);
    int rc = exclusive_scan(ctx, cellcnt, total_cells, cellbeg);
    if (rc) return rc;
    k_scatter<<<blocks_for(n, 256), 256, 0, s>>>(n, gcell, slot, cellbeg, perm);
    LAUNCH_CHECK(ctx);
    k_cellsort<<<blocks_for(total_cells, 256), 256, 0, s>>>(total_cells, cellbeg, perm);
    LAUNCH_CHECK(ctx);
    k_gather<<<blocks_for(n, 256), 256, 0, s>>>(n, perm, in.d_balls, in.sol, gcell, mol, grids,
                                                at, orig, cellof);
    LAUNCH_CHECK(ctx);
    tm.mark();  // 1

    // ---- a slab of one molecule (cfg.slab_world > 1): this pass emits the
    // simplices whose smallest vertex in cell order lies in [own_lo, own_hi)
    // -- balls n r / world .. n (r + 1) / world rounded down to cell starts --
    // and computes the tetrahedron and triangle stages from work_lo, two cell
    // layers lower: every vertex of an alpha simplex lies in a cell adjacent
    // to its smallest vertex's (alpha edges join adjacent cells), so the
    // tetrahedra whose faces decide the owned triangles, and the triangles
    // whose edges decide the owned edges, all start at or above work_lo.
    uint64_t own_lo = 0, own_hi = n, work_lo = 0;
    if (cfg.slab_world > 1) {
        if (nm != 1)
            return pac::set_error(PAC_ERR_INVALID_ARG, "a slab pass takes one molecule");
        if (cfg.tet_mode != PAC_TETS_AS_WRITTEN)
            return pac::set_error(PAC_ERR_INVALID_ARG, "a slab pass applies the orthosphere test");
        if (cfg.slab_rank < 0 || cfg.slab_rank >= cfg.slab_world)
            return pac::set_error(PAC_ERR_INVALID_ARG, "slab rank out of range");
        auto cell_start = [&](uint64_t ball, uint64_t &out) -> int {
            if (ball >= n) {
                out = n;
                return PAC_OK;
            }
            uint32_t c = 0, b = 0;
            CK(cudaMemcpyAsync(&c, cellof + ball, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            CK(cudaMemcpyAsync(&b, cellbeg + c, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            out = b;
            return PAC_OK;
        };
        const uint64_t r = (uint64_t)cfg.slab_rank, w = (uint64_t)cfg.slab_world;
        if (r > 0 && (rc = cell_start(n * r / w, own_lo))) return rc;
        if (r + 1 < w && (rc = cell_start(n * (r + 1) / w, own_hi))) return rc;
        if (own_hi < own_lo) own_hi = own_lo;
        if (own_lo > 0) {
            uint32_t c = 0, b = 0;
            CK(cudaMemcpyAsync(&c, cellof + own_lo, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            const uint64_t layer = (uint64_t)hg[0].gx * hg[0].gy + hg[0].gx + 1;
            const uint64_t c0 = c > 2 * layer ? c - 2 * layer : 0;
            CK(cudaMemcpyAsync(&b, cellbeg + c0, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            work_lo = b;
        }
    }

    // ---- alpha edges
    uint32_t *ecount = ar.alloc_n<uint32_t>(n);
    uint64_t *eoff = ar.alloc_n<uint64_t>(n + 1);
    if (!ecount || !eoff) return PAC_ERR_OOM;
    k_edges<V, false><<<warp_blocks(n), 256, 0, s>>>(n, at, cellof, cellbeg, mol, grids, in.alpha,
                                                     ecount, nullptr, nullptr, ctr);
    LAUNCH_CHECK(ctx);
    rc = exclusive_scan(ctx, ecount, n, eoff);
    if (rc) return rc;
    uint64_t *lsize = ar.alloc_n<uint64_t>(n), *loff = ar.alloc_n<uint64_t>(n + 1);
    if (!lsize || !loff) return PAC_ERR_OOM;
    k_link_size<<<blocks_for(n, 256), 256, 0, s>>>(n, ecount, lsize, ctr);
    LAUNCH_CHECK(ctx);
    rc = exclusive_scan(ctx, lsize, n, loff);
    if (rc) return rc;
    uint64_t nE = 0, nL = 0;
    unsigned long long maxdeg = 0;
    CK(cudaMemcpyAsync(&nE, eoff + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&nL, loff + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&maxdeg, ctr + C_MAXDEG, sizeof(maxdeg), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (maxdeg > (unsigned long long)kMaxDeg)
        return pac::set_error(PAC_ERR_CAPACITY, "a ball has " + std::to_string(maxdeg) +
                                                    " alpha edges to higher balls; the limit is " +
                                                    std::to_string(kMaxDeg));
    uint32_t *ER = ar.alloc_n<uint32_t>(nE);
    uint8_t *eflag = ar.alloc_n<uint8_t>(nE);
    if (!ER || !eflag) return PAC_ERR_OOM;
    k_edges<V, true><<<warp_blocks(n), 256, 0, s>>>(n, at, cellof, cellbeg, mol, grids, in.alpha,
                                                    nullptr, eoff, ER, ctr);
    LAUNCH_CHECK(ctx);
    CK(cudaMemsetAsync(eflag, 0, nE ? nE : 1, s));
    tm.mark();  // 2

    // ---- alpha triangles (link matrices)
    uint64_t *link = ar.alloc_n<uint64_t>(nL), *faces = ar.alloc_n<uint64_t>(nL);
    if (!link || !faces) return PAC_ERR_OOM;
    CK(cudaMemsetAsync(faces, 0, sizeof(uint64_t) * (nL ? nL : 1), s));
    uint32_t *classes = ar.alloc_n<uint32_t>(4 * n);  // balls by degree (k_link, enumeration)
    if (!classes) return PAC_ERR_OOM;
    const bool sparse = n >= kSparseBalls;
    k_classes<<<blocks_for(n, 256), 256, 0, s>>>(0, n, n, eoff, loff, nullptr, 2, sparse ? kLinkWarpDeg : 0,
                                                 classes, ctr);
    LAUNCH_CHECK(ctx);
    if (sparse) {
        k_link_warp<V><<<148 * 8, 256, 0, s>>>(classes + kSparse * n, at, eoff, ER, loff, link, in.alpha, ctr);
        LAUNCH_CHECK(ctx);
    }
    const unsigned link_grid = (unsigned)std::min<uint64_t>(n, 148 * 10);
    if (maxdeg > 128) {
        k_link<V, kMaxW><<<std::min(link_grid, 148u * 4), 128, 0, s>>>(classes + 2 * n, 2, at, eoff, ER, loff,
                                                                       link, in.alpha, ctr);
        LAUNCH_CHECK(ctx);
    }
    if (maxdeg > 64) {
        k_link<V, 2><<<link_grid, 128, 0, s>>>(classes + n, 1, at, eoff, ER, loff, link, in.alpha, ctr);
        LAUNCH_CHECK(ctx);
    }
    if (maxdeg > 1) {
        k_link<V, 1><<<link_grid, 128, 0, s>>>(classes, 0, at, eoff, ER, loff, link, in.alpha, ctr);
        LAUNCH_CHECK(ctx);
    }
    tm.mark();  // 3

    // ---- tetrahedra
    TetArgs T{};
    T.n = n;
    T.at = at;
    T.orig = orig;
    T.eoff = eoff;
    T.ER = ER;
    T.loff = loff;
    T.link = link;
    T.faces = faces;
    T.cellbeg = cellbeg;
    T.mol = mol;
    T.grids = grids;
    T.alpha = in.alpha;
    T.ctr = ctr;
    T.maxlen = ctr + C_MAXLEN;
    T.refute = cfg.refute ? 1 : 0;
    T.verify = cfg.verify ? 1 : 0;
    T.scan_claim = std::max(32, cfg.scan_claim);
    T.tcount = ar.alloc_n<uint32_t>(n);
    uint64_t *toff = ar.alloc_n<uint64_t>(n + 1);
    if (!T.tcount || !toff) return PAC_ERR_OOM;
    // the accepted enumerations' counts; the scan adds what was left open to it
    constexpr int kEnumCounts[] = {C_CAND_Q, C_ALPHA_Q, C_KILLED, C_KTESTS, C_CERT, C_CERT_BAD};
    unsigned long long enum_total[C_NCOUNTERS] = {};
    uint64_t nQ = 0;      // tetrahedra output
    uint64_t nQ_all = 0;  // survivors, a slab's halo included
    uint32_t *tets_sorted = nullptr;
    if (cfg.tet_mode == PAC_TETS_AS_RUN) {
        k_tets<V, 1><<<warp_blocks(n), 256, 0, s>>>(T);
        LAUNCH_CHECK(ctx);
        rc = exclusive_scan(ctx, T.tcount, n, toff);
        if (rc) return rc;
        CK(cudaMemcpyAsync(&nQ, toff + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        tets_sorted = ar.alloc_n<uint32_t>(4 * nQ);
        if (!tets_sorted) return PAC_ERR_OOM;
        T.toff = toff;
        T.tets_out = tets_sorted;
        // the second sweep counts candidates again: reset those counters
        CK(cudaMemsetAsync(ctr + C_CAND_Q, 0, 2 * sizeof(unsigned long long), s));
        k_tets<V, 2><<<warp_blocks(n), 256, 0, s>>>(T);
        LAUNCH_CHECK(ctx);
    } else {
        // the enumeration settles most triangle attachments on its way (not
        // with the plain-xmp formulas, whose triangle centres are no
        // orthocentres, nor where the window lemma's grid limit is exceeded)
        bool small_grid = true;
        for (const MolGrid &g : hg) small_grid &= g.gx <= 16384 && g.gy <= 16384 && g.gz <= 16384;
        if (V != pac::kPlainXmp && small_grid) {
            T.attached = ar.alloc_n<uint64_t>(nL);
            if (!T.attached) return PAC_ERR_OOM;
        }
        // queue of alpha tetrahedra in HBM, processed in chunks of balls
        const uint64_t qcap = std::max<uint64_t>(1 << 16, cfg.queue_entries);
        TetQueue Q;
        Q.ent = ar.alloc_n<uint2>(qcap);
        Q.cap = qcap;
        // (at least what a molecule of some 15,000 balls queues: see `ahead`)
        uint64_t scap = std::max<uint64_t>(1 << 22, 16 * n);
        T.surv = ar.alloc_n<uint2>(scap);
        T.surv_cap = scap;
        T.pend_cap = std::max<uint64_t>(1 << 22, scap / 4);
        T.pend = ar.alloc_n<uint2>(T.pend_cap);
        unsigned long long *claim = ar.alloc_n<unsigned long long>(1);
        unsigned long long *ctrA = ar.alloc_n<unsigned long long>(C_NCOUNTERS);
        if (!Q.ent || !T.surv || !T.pend || !claim || !ctrA) return PAC_ERR_OOM;
        CK(cudaMemsetAsync(ctr + C_SURV, 0, 2 * sizeof(unsigned long long), s));
        CK(cudaMemsetAsync(ctr + C_INSPHERE, 0, sizeof(unsigned long long), s));
        CK(cudaMemsetAsync(faces, 0, sizeof(uint64_t) * (nL ? nL : 1), s));
        CK(cudaMemsetAsync(T.tcount, 0, sizeof(uint32_t) * n, s));
        // the empty-orthosphere test's share of the stage: ev[14], ev[15]
        // around each scan, read once the stream has passed them
        double ortho_ms = 0.0;
        bool ortho_pending = false;
        auto ortho_collect = [&]() {
            if (!ortho_pending) return;
            float f = 0.f;
            if (cudaEventElapsedTime(&f, ctx.ev[14], ctx.ev[15]) == cudaSuccess) ortho_ms += f;
            ortho_pending = false;
        };
        unsigned long long sp[2] = {0, 0};  // survivors, pending
        bool scanned = false;               // sp holds the final counts
        uint64_t lo = work_lo, chunk = n;
        {
            // first chunk: the whole range when its queue demand (a few
            // entries per alpha triangle) clearly fits, else a probe of 1/32
            // whose fill sizes the next chunks -- an overflowing chunk is
            // enumerated again, smaller
            // (about 0.5 entries per alpha triangle; 5 without refutation);
            // a ball has at most deg^2 / 2 triangles, which settles all but
            // the largest passes without reading the count back
            const double per = cfg.refute ? 1.0 : 8.0;
            unsigned long long atri = nE * maxdeg / 2;
            if (per * (double)atri > 0.85 * (double)qcap) {
                CK(cudaMemcpyAsync(&atri, ctr + C_ALPHA_T, sizeof(atri), cudaMemcpyDeviceToHost, s));
                CK(cudaStreamSynchronize(s));
            }
            const double span = (double)(own_hi - work_lo), share = span / (double)std::max<uint64_t>(1, n);
            if (per * (double)atri * share > 0.85 * (double)qcap)
                chunk = std::max<uint64_t>(1, (uint64_t)(span / 32.0));
        }
        // verbose: per-chunk enumeration and scan times
        unsigned long long late_before = 0;
        cudaEvent_t vev[3] = {nullptr, nullptr, nullptr};
        if (cfg.verbose)
            for (auto &e : vev) CK(cudaEventCreate(&e));
        while (lo < own_hi) {
            const uint64_t hi = std::min<uint64_t>(own_hi, lo + chunk);
            TetArgs TA = T;
            TA.ctr = ctrA;
            if (cfg.verbose) CK(cudaEventRecord(vev[0], s));
            CK(cudaMemsetAsync(ctrA, 0, sizeof(unsigned long long) * C_NCOUNTERS, s));
            constexpr int M = V == pac::kExact ? kEnumExact : kEnumFloat;
            rc = cfg.verify ? enumerate<M | kEnumVerify>(ctx, cfg, TA, Q, lo, hi, classes, maxdeg)
                            : enumerate<M>(ctx, cfg, TA, Q, lo, hi, classes, maxdeg);
            if (rc) return rc;
            if (cfg.verbose) CK(cudaEventRecord(vev[1], s));
            const unsigned scan_grid = 148u * (unsigned)std::max(1, cfg.scan_blocks);
            auto scan = [&](uint64_t limit) -> int {
                CK(cudaMemsetAsync(claim, 0, sizeof(unsigned long long), s));
                CK(cudaEventRecord(ctx.ev[14], s));
                k_tets_scan<V><<<scan_grid, 256, 0, s>>>(T, Q, ctrA + C_SURV, limit, claim);
                LAUNCH_CHECK(ctx);
                CK(cudaEventRecord(ctx.ev[15], s));
                ortho_pending = true;
                return PAC_OK;
            };
            // one chunk: the scan goes ahead of its queue's count, and does
            // nothing should that exceed what the lists hold (then it is
            // launched again below)
            const uint64_t room = std::min({qcap, T.surv_cap, T.pend_cap});
            const bool ahead = lo == work_lo && hi == own_hi;
            if (ahead && (rc = scan(room))) return rc;
            unsigned long long ha[C_NCOUNTERS];
            CK(cudaMemcpyAsync(ha, ctrA, sizeof(ha), cudaMemcpyDeviceToHost, s));
            CK(cudaMemcpyAsync(sp, ctr + C_SURV, sizeof(sp), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            ortho_collect();
            const unsigned long long queued = ha[C_SURV];
            if (queued > qcap) {
                if (hi - lo == 1)
                    return pac::set_error(PAC_ERR_CAPACITY,
                                          "the alpha tetrahedra of one ball exceed the queue");
                chunk = std::max<uint64_t>(1, (uint64_t)((double)(hi - lo) * 0.5));
                continue;
            }
            for (int k : kEnumCounts) enum_total[k] += ha[k];
            scanned = ahead && queued <= room;
            if (!scanned) {
                // every queued tetrahedron becomes at most one survivor or
                // one pending entry: grow either list (keeping its entries)
                // first; a list of scap entries beside a whole queue's lasts
                // for all later chunks, so that a list grows once to stay
                // within its third of the queue's bytes
                auto grow = [&](uint2 *&list, uint64_t &cap, unsigned long long used) -> int {
                    if (used + queued <= cap) return PAC_OK;
                    const uint64_t need = used + queued;
                    const uint64_t nc = std::max<uint64_t>(need, std::min<uint64_t>(2 * need, scap + qcap));
                    uint2 *nb = ar.alloc_n<uint2>(nc);
                    if (!nb) return PAC_ERR_OOM;
                    if (used)
                        CK(cudaMemcpyAsync(nb, list, sizeof(uint2) * used, cudaMemcpyDeviceToDevice, s));
                    list = nb;
                    cap = nc;
                    return PAC_OK;
                };
                if ((rc = grow(T.surv, T.surv_cap, sp[0]))) return rc;
                if ((rc = grow(T.pend, T.pend_cap, sp[1]))) return rc;
                if (queued && (rc = scan(qcap))) return rc;
            }
            if (cfg.verbose) {
                float me = 0.f, ms = 0.f;
                unsigned long long late = 0;  // alpha tests that the scan settled
                CK(cudaEventRecord(vev[2], s));
                CK(cudaMemcpyAsync(&late, ctr + C_ALPHA_Q, sizeof(late), cudaMemcpyDeviceToHost, s));
                CK(cudaStreamSynchronize(s));
                CK(cudaEventElapsedTime(&me, vev[0], vev[1]));
                CK(cudaEventElapsedTime(&ms, vev[1], vev[2]));
                std::fprintf(stderr,
                             "[pac] tetrahedra of balls [%llu, %llu): %llu candidates, %llu alpha, "
                             "%llu refuted early, %llu queued; enumeration %.3f ms, scan %.3f ms\n",
                             (unsigned long long)lo, (unsigned long long)hi, ha[C_CAND_Q],
                             ha[C_ALPHA_Q] + late - late_before, ha[C_KILLED], queued, me, ms);
                late_before = late;
            }
            // next chunk sized from this one's queue fill
            if (queued)
                chunk = std::max<uint64_t>(
                    1, (uint64_t)(0.85 * (double)qcap * (double)(hi - lo) / (double)queued));
            else
                chunk = n;
            lo = hi;
        }
        if (cfg.verbose)
            for (auto &e : vev) cudaEventDestroy(e);
        if (!scanned) {
            CK(cudaMemcpyAsync(sp, ctr + C_SURV, sizeof(sp), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            ortho_collect();
        }
        if (sp[0] > T.surv_cap || sp[1] > T.pend_cap)
            return pac::set_error(PAC_ERR_CAPACITY, "tetrahedron survivor buffer overflow");
        if (sp[1] && sp[0] + sp[1] > T.surv_cap) {  // resolved entries join the survivors
            uint2 *nb = ar.alloc_n<uint2>(sp[0] + sp[1]);
            if (!nb) return PAC_ERR_OOM;
            if (sp[0])
                CK(cudaMemcpyAsync(nb, T.surv, sizeof(uint2) * sp[0], cudaMemcpyDeviceToDevice, s));
            T.surv = nb;
            T.surv_cap = sp[0] + sp[1];
        }
        if (sp[1]) {
            CK(cudaEventRecord(ctx.ev[14], s));
            k_sos_resolve<V><<<blocks_for(sp[1], 4), 128, 0, s>>>(T, sp[1]);
            LAUNCH_CHECK(ctx);
            CK(cudaEventRecord(ctx.ev[15], s));
            ortho_pending = true;
            CK(cudaMemcpyAsync(sp, ctr + C_SURV, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
            ortho_collect();
        }
        if (st) st->ms_tet_orthosphere = ortho_ms;
        nQ = sp[0];
        if (cfg.slab_world > 1 && own_lo > 0)  // the halo's tetrahedra are not output
            CK(cudaMemsetAsync(T.tcount, 0, sizeof(uint32_t) * own_lo, s));
        rc = exclusive_scan(ctx, T.tcount, n, toff);
        if (rc) return rc;
        if (cfg.slab_world > 1) {
            nQ_all = nQ;
            CK(cudaMemcpyAsync(&nQ, toff + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
            CK(cudaStreamSynchronize(s));
        }
    }
    tm.mark();  // 4

    // ---- emission of the tetrahedra: final now, so with to_host their copy
    // crosses PCIe while the triangles and edges are decided
    out.d_tets = ar.alloc_n<uint32_t>(4 * nQ);
    if (!out.d_tets) return PAC_ERR_OOM;
    if (cfg.tet_mode == PAC_TETS_AS_RUN) {
        CK(cudaMemcpyAsync(out.d_tets, tets_sorted, sizeof(uint32_t) * 4 * (nQ ? nQ : 1),
                           cudaMemcpyDeviceToDevice, s));
        k_map4<<<blocks_for(nQ, 256), 256, 0, s>>>(nQ, orig, out.d_tets);
        LAUNCH_CHECK(ctx);
    } else {
        uint32_t *cursor = ar.alloc_n<uint32_t>(n), *keys = ar.alloc_n<uint32_t>(nQ);
        if (!cursor || !keys) return PAC_ERR_OOM;
        CK(cudaMemsetAsync(cursor, 0, sizeof(uint32_t) * n, s));
        const uint64_t ns = std::max(nQ, nQ_all);
        k_tet_scatter<<<blocks_for(ns, 256), 256, 0, s>>>(T.surv, ns, toff, cursor, keys, own_lo,
                                                          own_hi);
        LAUNCH_CHECK(ctx);
        k_tet_emit<<<blocks_for(ns, 256), 256, 0, s>>>(T.surv, ns, toff, keys, eoff, ER, orig,
                                                       out.d_tets, own_lo, own_hi);
        LAUNCH_CHECK(ctx);
    }
    if (in.to_host && (rc = pac::list_to_host_async(ctx, 2, out.d_tets, 4 * nQ, &out.h_tets)))
        return rc;
    tm.mark();  // 5

    // ---- final triangles
    uint32_t *tricount = ar.alloc_n<uint32_t>(n);
    uint64_t *tpos = ar.alloc_n<uint64_t>(n + 1);
    uint64_t *epos = ar.alloc_n<uint64_t>(nE + 1);
    if (!tricount || !tpos || !epos) return PAC_ERR_OOM;
    CK(cudaMemsetAsync(ctr + C_NEXT, 0, sizeof(unsigned long long), s));
    if (cfg.slab_world > 1) CK(cudaMemsetAsync(tricount, 0, sizeof(uint32_t) * n, s));
    k_tri_attach<V><<<std::min<unsigned>(warp_blocks(own_hi - work_lo), 148 * 4), 256, 0, s>>>(
        work_lo, own_hi, at, eoff, ER, loff, link, T.attached, faces, tricount, eflag, cellbeg, mol, grids,
        in.alpha, ctr);
    LAUNCH_CHECK(ctx);
    tm.mark();  // 6
    // only the owned balls' triangles are output
    if (cfg.slab_world > 1 && own_lo > work_lo)
        CK(cudaMemsetAsync(tricount + work_lo, 0, sizeof(uint32_t) * (own_lo - work_lo), s));
    rc = exclusive_scan(ctx, tricount, n, tpos);
    if (rc) return rc;
    uint64_t nT = 0, nEf = 0;
    auto emit_tris = [&]() -> int {
        out.d_tris = ar.alloc_n<uint32_t>(3 * nT);
        if (!out.d_tris) return PAC_ERR_OOM;
        k_emit_tris<<<warp_blocks(own_hi - own_lo), 256, 0, s>>>(own_lo, own_hi, eoff, ER, loff, faces,
                                                                tpos, orig, out.d_tris);
        LAUNCH_CHECK(ctx);
        return in.to_host ? pac::list_to_host_async(ctx, 1, out.d_tris, 3 * nT, &out.h_tris) : PAC_OK;
    };
    // the triangles leave before the edges are decided, except in passes of a
    // few thousand balls, where waiting for their count costs more than the
    // copy takes
    const bool early = nE > (1u << 20);
    if (early) {
        CK(cudaMemcpyAsync(&nT, tpos + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        if ((rc = emit_tris())) return rc;
    }
    tm.mark();  // 7

    // ---- final edges
    CK(cudaMemsetAsync(ctr + C_NEXT, 0, sizeof(unsigned long long), s));
    k_edge_final<V><<<std::min<unsigned>(warp_blocks(own_hi - own_lo), 148 * 5), 256, 0, s>>>(
        own_lo, own_hi, at, eoff, ER, eflag, cellbeg, mol, grids, ctr);
    LAUNCH_CHECK(ctx);
    if (cfg.slab_world > 1) {
        // only the owned balls' edges are output
        uint64_t eb[2] = {0, 0};
        CK(cudaMemcpyAsync(&eb[0], eoff + own_lo, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(&eb[1], eoff + own_hi, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        if (eb[0]) CK(cudaMemsetAsync(eflag, 0, eb[0], s));
        if (nE > eb[1]) CK(cudaMemsetAsync(eflag + eb[1], 0, nE - eb[1], s));
    }
    tm.mark();  // 8
    rc = exclusive_scan(ctx, eflag, nE, epos);
    if (rc) return rc;
    // every decision is made: the counters and the remaining lengths
    unsigned long long hc[C_NCOUNTERS];
    CK(cudaMemcpyAsync(hc, ctr, sizeof(hc), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&nT, tpos + n, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    CK(cudaMemcpyAsync(&nEf, epos + nE, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    for (int k : kEnumCounts) hc[k] += enum_total[k];
    if (!early && (rc = emit_tris())) return rc;
    out.d_edges = ar.alloc_n<uint32_t>(2 * nEf);
    if (!out.d_edges) return PAC_ERR_OOM;
    k_emit_edges<<<warp_blocks(n), 256, 0, s>>>(n, eoff, ER, eflag, epos, orig, out.d_edges);
    LAUNCH_CHECK(ctx);
    if (in.to_host && (rc = pac::list_to_host_async(ctx, 0, out.d_edges, 2 * nEf, &out.h_edges)))
        return rc;
    out.n_edges = nEf;
    out.n_tris = nT;
    out.n_tets = nQ;
    // per-molecule row offsets
    out.edge_off.assign(nm + 1, 0);
    out.tri_off.assign(nm + 1, 0);
    out.tet_off.assign(nm + 1, 0);
    if (nm == 1) {
        out.edge_off[1] = nEf;
        out.tri_off[1] = nT;
        out.tet_off[1] = nQ;
    } else {
        uint64_t *rows = ar.alloc_n<uint64_t>(3 * (size_t)(nm + 1));
        if (!rows) return PAC_ERR_OOM;
        k_mol_rows<<<blocks_for(nm + 1, 128), 128, 0, s>>>(nm, d_off, n, eoff, epos, tpos, toff,
                                                          rows);
        LAUNCH_CHECK(ctx);
        CK(cudaMemcpyAsync(out.edge_off.data(), rows, sizeof(uint64_t) * (nm + 1),
                           cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(out.tri_off.data(), rows + (nm + 1), sizeof(uint64_t) * (nm + 1),
                           cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(out.tet_off.data(), rows + 2 * (size_t)(nm + 1), sizeof(uint64_t) * (nm + 1),
                           cudaMemcpyDeviceToHost, s));
    }
    tm.mark();  // 9
    // the lists' copies that did not finish under the later stages
    if (in.to_host && (rc = pac::copies_join(ctx))) return rc;
    tm.mark();  // 10
    CK(cudaStreamSynchronize(s));
    if (hc[C_SOS_RANGE])
        return pac::set_error(PAC_ERR_EXACT_RANGE,
                              "coordinate range too wide for the exact SoS integers");
    if (st) {
        st->n_balls = n;
        st->n_cells = total_cells;
        st->cand_edges = hc[C_CAND_E];
        st->alpha_edges = hc[C_ALPHA_E];
        st->cand_tris = hc[C_CAND_T];
        st->alpha_tris = hc[C_ALPHA_T];
        st->cand_tets = hc[C_CAND_Q];
        st->alpha_tets = hc[C_ALPHA_Q];
        st->final_edges = nEf;
        st->final_tris = nT;
        st->final_tets = nQ;
        st->insphere_evals = hc[C_INSPHERE];
        st->sos_calls = hc[C_SOS];
        st->filter_evals = hc[C_FILTER];
        st->exact_fallbacks = hc[C_FALLBACK];
        st->early_refuted = hc[C_KILLED];
        st->early_tests = hc[C_KTESTS];
        st->cert_decisions = hc[C_CERT];
        st->cert_disagreements = hc[C_CERT_BAD];
        st->ortho_out_of_grid = hc[C_OOB];
        st->max_degree = maxdeg;
        st->ms_grid = tm.ms(0, 1);
        st->ms_edges = tm.ms(1, 2);
        st->ms_tris = tm.ms(2, 3);
        st->ms_tets = tm.ms(3, 4);
        st->ms_tri_attach = tm.ms(5, 6);
        st->ms_edge_attach = tm.ms(7, 8);
        st->ms_emit = tm.ms(4, 5) + tm.ms(6, 7) + tm.ms(8, 9);
        if (in.to_host) st->ms_d2h = tm.ms(9, 10);
        // the reference's data movement for this pass: balls in, lists out,
        // and every candidate list (edges 8 B, triangles 12 B + 16 B
        // orthosphere, tetrahedra 16 B + 16 B orthosphere) written and read
        // once -- independent of how this engine avoids storing them
        st->bytes_model = 16 * n + 8 * st->final_edges + 12 * st->final_tris +
                          16 * st->final_tets +
                          2 * (8 * st->cand_edges + 28 * st->cand_tris + 32 * st->cand_tets);
        if (nm == 1) {
            st->grid[0] = hg[0].gx;
            st->grid[1] = hg[0].gy;
            st->grid[2] = hg[0].gz;
            st->step = hg[0].step;
        }
    }
    if (cfg.verbose)
        std::fprintf(stderr,
                     "[pac] %llu balls: grid %.3f, edges %.3f, triangles %.3f, tetrahedra %.3f, "
                     "triangle attachment %.3f, edge attachment %.3f, emission %.3f ms\n",
                     (unsigned long long)n, tm.ms(0, 1), tm.ms(1, 2), tm.ms(2, 3), tm.ms(3, 4),
                     tm.ms(5, 6), tm.ms(7, 8), tm.ms(4, 5) + tm.ms(6, 7) + tm.ms(8, 9));
    return PAC_OK;
}

int run_pass(pac::Ctx &ctx, const pac::PipelineConfig &cfg, const pac::PassInput &in,
             pac::PassOutput &out, pac_stats *st) {
    if (cfg.exact) {
#if PAC_WITH_EXACT
        return run_pass_v<pac::kExact>(ctx, cfg, in, out, st);
#else
        return pac::set_error(PAC_ERR_INVALID_ARG, "exact predicates are built in the strict flavour");
#endif
    }
    if (cfg.formula == PAC_FORMULA_PLAIN_XMP) return run_pass_v<pac::kPlainXmp>(ctx, cfg, in, out, st);
    return run_pass_v<pac::kUpstream>(ctx, cfg, in, out, st);
}

}  // namespace PAC_NS
