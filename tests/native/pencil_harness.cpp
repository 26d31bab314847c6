// pencil_harness.cpp -- checks the enumeration's filter (pencil.cuh) against
// the arithmetic it stands for: whenever it claims an alpha decision or a
// refutation, markRealTets / orient3d / insphere_w in binary32 (refarith.cuh,
// built here without contraction) must decide the same, and the refuting ball
// must lie within 0.99 cell steps of the binary32 orthocentre; in the exact
// flavour the polynomials' exact signs (orc_exact_pred).  Built and run by
// tests/test_pencil.py.
//   pencil_harness SEED CLUSTERS OFFSET SOL LATTICE EXACT
//     -> "alpha N certified C bad B refutations R bad B attachments A bad B"
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#define __device__
#define __forceinline__ inline
struct float4 {
    float x, y, z, w;
};
static inline float4 make_float4(float x, float y, float z, float w) { return float4{x, y, z, w}; }
static inline float4 __ldg(const float4 *p) { return *p; }
#include "../../parallelac-xmp_b200/csrc/pencil.cuh"
#include "../../parallelac-xmp_b200/csrc/refarith.cuh"

extern "C" int orc_exact_pred(int kind, const float *balls, float alpha);

using pac::Ball;

static uint64_t g_state;
static double urand() {  // splitmix64 -> [0, 1)
    uint64_t z = (g_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

static double squares(const Ball &b) {  // rounded squares minus squares
    const double x = b.x, y = b.y, z = b.z;
    return ((double)(b.x * b.x) - x * x) + ((double)(b.y * b.y) - y * y) + ((double)(b.z * b.z) - z * z);
}

static int exact(int kind, std::initializer_list<Ball> b, float alpha) {
    std::vector<float> f;
    for (const Ball &x : b) f.insert(f.end(), {x.x, x.y, x.z, x.r});
    return orc_exact_pred(kind, f.data(), alpha);
}

int main(int argc, char **argv) {
    g_state = strtoull(argv[1], nullptr, 10);
    const int clusters = atoi(argv[2]);
    const double offset = atof(argv[3]), sol = atof(argv[4]);
    const bool lattice = atoi(argv[5]), ex = atoi(argv[6]);
    long tests = 0, certified = 0, bad = 0, refuted = 0, rbad = 0, attached = 0, abad = 0;
    for (int t = 0; t < clusters; t++) {
        const float alpha = t % 3 == 0 ? 0.0f : t % 3 == 1 ? 0.5f : 1.0f;
        const float step = 2.0f * std::sqrt(1.8f * 1.8f + alpha);
        const double reach = 1.2 * std::sqrt((1.7 + sol) * (1.7 + sol) + alpha);
        std::vector<Ball> b;
        for (int k = 0; k < 24; k++) {
            double c[3];
            for (double &v : c) {
                v = (2 * urand() - 1) * reach + offset;
                if (lattice) v = std::round(v * 4) / 4;
            }
            if (k % 6 == 5) c[2] = b[0].z + 1e-3 * urand();  // flat against b[0]'s plane z
            const float r = lattice ? 1.6f : (float)(1.52 + 0.28 * urand());
            b.push_back(Ball{(float)c[0], (float)c[1], (float)c[2], r + (float)sol});
        }
        const int n = (int)b.size();
        std::vector<char> edge(n * n, 0);
        float len2 = 0, wmax = 0;
        for (int i = 0; i < n; i++) {
            wmax = std::max(wmax, b[i].r * b[i].r * (1.0f + 1.0f / 1024.0f));
            for (int j = i + 1; j < n; j++) {
                if (b[i].x == b[j].x && b[i].y == b[j].y && b[i].z == b[j].z) continue;
                if (!pac::edge_alpha<pac::kUpstream>(b[i], b[j], alpha)) continue;
                edge[i * n + j] = edge[j * n + i] = 1;
                const float x = b[i].x - b[j].x, y = b[i].y - b[j].y, z = b[i].z - b[j].z;
                len2 = std::max(len2, x * x + y * y + z * z);
            }
        }
        const Ball &p = b[0];
        const pac::pencil::Bounds bounds =
            pac::pencil::bounds(p.x, p.y, p.z, p.r * p.r, alpha, len2, wmax, step, false);
        const double wp = ex ? (double)p.r * p.r : (double)(p.r * p.r);
        std::vector<pac::pencil::Point> P(n);
        for (int k = 0; k < n; k++) {
            pac::pencil::Point &q = P[k];
            q.x = (double)b[k].x - p.x, q.y = (double)b[k].y - p.y, q.z = (double)b[k].z - p.z;
            const double w = ex ? (double)b[k].r * b[k].r : (double)(b[k].r * b[k].r);
            q.s = q.x * q.x + q.y * q.y + q.z * q.z - w + wp;
            q.st = ex ? q.s : q.s + (squares(b[k]) - squares(p));
        }
        for (int i = 1; i < n; i++)
            for (int j = i + 1; j < n; j++) {
                if (!edge[i] || !edge[j] || !edge[i * n + j]) continue;
                const pac::pencil::Group g = pac::pencil::group(bounds, P[i], P[j], p.r * p.r);
                // attachment of the triangle by any other neighbour of p
                float4 to;
                if (ex ? exact(1, {p, b[i], b[j]}, alpha) != 0
                       : pac::tri_alpha<pac::kUpstream>(p, b[i], b[j], alpha, to))
                    for (int v = 1; v < n; v++) {
                        if (v == i || v == j || !edge[v]) continue;
                        const float s0 = (float)P[v].s, st = (float)P[v].st, x = (float)P[v].x,
                                    y = (float)P[v].y, zz = (float)P[v].z;
                        const float gt = pac::pencil::power(g.tx, g.ty, g.tz, st, x, y, zz);
                        if (!(gt + (s0 - st) < -g.mt)) continue;
                        if (bounds.mreach > 0 &&
                            !pac::pencil::in_box(g.tx, g.ty, g.tz, x, y, zz, bounds.mreach))
                            continue;
                        attached++;
                        if (ex) {
                            abad += exact(6, {p, b[i], b[j], b[v]}, alpha) == 0;
                            continue;
                        }
                        const float m = std::max(std::fabs(b[v].x - to.x), std::max(std::fabs(b[v].y - to.y),
                                                                                    std::fabs(b[v].z - to.z)));
                        abad += !pac::attached(b[v], to.x, to.y, to.z, to.w) || !(m <= 0.99f * step);
                    }
                std::vector<int> z;
                for (int k = 1; k < n; k++)
                    if (k != i && k != j && edge[k] && edge[i * n + k] && edge[j * n + k]) z.push_back(k);
                for (int c : z) {
                    const float x = (float)P[c].x, y = (float)P[c].y, zz = (float)P[c].z;
                    const float h = pac::pencil::height(g.nx, g.ny, g.nz, x, y, zz);
                    const float gt = pac::pencil::power(g.tx, g.ty, g.tz, (float)P[c].st, x, y, zz);
                    const float q = pac::pencil::power(g.qx, g.qy, g.qz, (float)P[c].s, x, y, zz);
                    float4 o;
                    const bool mark = ex ? exact(2, {p, b[i], b[j], b[c]}, alpha) != 0
                                         : pac::tet_alpha(p, b[i], b[j], b[c], alpha, o);
                    tests++;
                    const bool sure = std::fabs(h) >= g.hmin;
                    bool in = false, out = false;
                    pac::pencil::alpha_test(std::fabs(h), gt, g.k, g.ea, in, out);
                    in = in && std::fabs(h) >= bounds.kappa * g.hmin;
                    out = out && std::fabs(h) >= bounds.kappa * g.hmin;
                    if (in || out) {
                        certified++;
                        bad += mark != in;
                    }
                    if (!sure || !mark) continue;
                    for (int v : z) {  // every other candidate as the refuting ball
                        if (v == c) continue;
                        const float vx = (float)P[v].x, vy = (float)P[v].y, vz = (float)P[v].z;
                        const float hy = pac::pencil::height(g.nx, g.ny, g.nz, vx, vy, vz);
                        const float qy = pac::pencil::power(g.qx, g.qy, g.qz, (float)P[v].s, vx, vy, vz);
                        if (!(std::fabs(hy) >= g.hmin) || !pac::pencil::refutes(h, q, hy, qy, g.rg)) continue;
                        if (bounds.reach > 0 &&
                            !pac::pencil::within_reach(g.nx, g.ny, g.nz, g.tx, g.ty, g.tz, h, gt, vx, vy,
                                                       vz, bounds.reach))
                            continue;
                        refuted++;
                        const Ball &e = b[v];
                        if (ex) {
                            const int os = exact(3, {p, b[i], b[j], b[c]}, alpha);
                            const int is = exact(4, {p, b[i], b[j], b[c], e}, alpha);
                            rbad += !(os < 0 ? is < 0 : is > 0);
                            continue;
                        }
                        const float pa[3] = {p.x, p.y, p.z}, pb[3] = {b[i].x, b[i].y, b[i].z},
                                    pc[3] = {b[j].x, b[j].y, b[j].z}, pd[3] = {b[c].x, b[c].y, b[c].z},
                                    pe[3] = {e.x, e.y, e.z};
                        const float os = pac::orient3d(pa, pb, pc, pd);
                        const float is = pac::insphere_w(pa, pb, pc, pd, pe, p.r * p.r, b[i].r * b[i].r,
                                                         b[j].r * b[j].r, b[c].r * b[c].r, e.r * e.r);
                        const bool viol = os < 0 ? is < 0 : is > 0;
                        const float m = std::max(std::fabs(e.x - o.x),
                                                 std::max(std::fabs(e.y - o.y), std::fabs(e.z - o.z)));
                        rbad += !viol || !(m <= 0.99f * step);
                    }
                }
            }
    }
    std::printf("alpha %ld certified %ld bad %ld refutations %ld bad %ld attachments %ld bad %ld\n", tests, certified,
                bad, refuted, rbad, attached, abad);
    return 0;
}
