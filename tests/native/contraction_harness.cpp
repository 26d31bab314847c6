// contraction_harness.cpp -- checks the enumeration's filter (pencil.cuh, bounds
// of contracted arithmetic) against the written sequences of the contracted
// flavour (refarith.cuh with PAC_CONTRACTED): whenever it claims an alpha
// decision, a refutation or an attachment, every sequence that could decide it
// must agree, and the refuting or attaching ball must lie within 0.99 cell steps
// of each sequence's centre.  Built and run by tests/test_contraction.py.
//   contraction_harness SEED CLUSTERS OFFSET SOL FLAT
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

using pac::Ball;
namespace pn = pac::pencil;

static uint64_t g_state;
static double urand() {  // splitmix64 -> [0, 1)
    uint64_t z = (g_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

static float square_rounding(const Ball &b) {
    const double x = b.x, y = b.y, z = b.z;
    return (float)(((double)(b.x * b.x) - x * x) + ((double)(b.y * b.y) - y * y) + ((double)(b.z * b.z) - z * z));
}
static float reach_of(const Ball &e, const float4 &o) {
    return std::max(std::fabs(e.x - o.x), std::max(std::fabs(e.y - o.y), std::fabs(e.z - o.z)));
}
// violation by e: 0 as the scan decides it, 1 as exact zeros are resolved, 2 as
// the first enumeration replayed it
static bool violates(const Ball *t, const Ball &e, int how) {
    float q[5][3];
    for (int k = 0; k < 5; k++) {
        const Ball &b = k < 4 ? t[k] : e;
        q[k][0] = b.x, q[k][1] = b.y, q[k][2] = b.z;
    }
    const float we = e.r * e.r;
    const float o = pac::orient3d(q[0], q[1], q[2], q[3]);
    float s;
    if (how == 2)
        s = pac::insphere_d<pac::AtScan>(q[0], q[1], q[2], q[3], q[4], t[0].r * t[0].r - we, t[1].r * t[1].r - we,
                                         std::fmaf(t[2].r, t[2].r, -we), std::fmaf(t[3].r, t[3].r, -we));
    else if (how == 1)
        s = pac::insphere_w<pac::AtSos>(q[0], q[1], q[2], q[3], q[4], t[0].r * t[0].r, t[1].r * t[1].r,
                                        t[2].r * t[2].r, t[3].r * t[3].r, we);
    else
        s = pac::insphere_w<pac::AtScan>(q[0], q[1], q[2], q[3], q[4], t[0].r * t[0].r, t[1].r * t[1].r,
                                         t[2].r * t[2].r, t[3].r * t[3].r, we);
    return o < 0 ? s < 0 : s > 0;
}

int main(int argc, char **argv) {
    if (argc < 6) return 2;
    g_state = strtoull(argv[1], nullptr, 10);
    const int clusters = atoi(argv[2]);
    const double offset = atof(argv[3]), sol = atof(argv[4]);
    const bool flat = atoi(argv[5]);
    long tests = 0, certified = 0, bad = 0, refuted = 0, rbad = 0, attached = 0, abad = 0;
    for (int t = 0; t < clusters; t++) {
        const float alpha = t % 3 == 0 ? 0.0f : t % 3 == 1 ? 0.5f : 1.0f;
        const float step = 2.0f * std::sqrt(1.8f * 1.8f + alpha);
        const double reach = 1.2 * std::sqrt((1.7 + sol) * (1.7 + sol) + alpha);
        std::vector<Ball> b;
        for (int k = 0; k < 24; k++) {
            double c[3];
            for (double &v : c) v = (2 * urand() - 1) * reach + offset;
            if (k % (flat ? 2 : 6) == 1) c[2] = b[0].z + 1e-3 * urand();  // flat against b[0]'s plane z
            b.push_back(Ball{(float)c[0], (float)c[1], (float)c[2], (float)(1.52 + 0.28 * urand()) + (float)sol});
        }
        const int n = (int)b.size();
        std::vector<char> edge(n * n, 0);
        float len2 = 0, wmax = 0;
        for (int i = 0; i < n; i++) {
            wmax = std::max(wmax, b[i].r * b[i].r * (1.0f + 1.0f / 1024.0f));
            for (int j = i + 1; j < n; j++) {
                if (!pac::edge_alpha<pac::kUpstream>(b[i], b[j], alpha)) continue;
                edge[i * n + j] = edge[j * n + i] = 1;
                const float x = b[i].x - b[j].x, y = b[i].y - b[j].y, z = b[i].z - b[j].z;
                len2 = std::max(len2, x * x + y * y + z * z);
            }
        }
        const Ball &p = b[0];
        const pn::Bounds bounds = pn::bounds(p.x, p.y, p.z, p.r * p.r, alpha, len2, wmax, step, true);
        std::vector<pn::Point> P(n);
        for (int k = 0; k < n; k++) {
            pn::Point &q = P[k];
            q.x = (double)b[k].x - p.x, q.y = (double)b[k].y - p.y, q.z = (double)b[k].z - p.z;
            q.s = q.x * q.x + q.y * q.y + q.z * q.z - (double)(b[k].r * b[k].r) + (double)(p.r * p.r);
            q.st = q.s + 0.5 * (square_rounding(b[k]) - square_rounding(p));
        }
        for (int i = 1; i < n; i++)
            for (int j = i + 1; j < n; j++) {
                if (!edge[i] || !edge[j] || !edge[i * n + j]) continue;
                const pn::Group g = pn::group(bounds, P[i], P[j], p.r * p.r);
                float4 to;
                if (pac::tri_alpha<pac::kUpstream>(p, b[i], b[j], alpha, to))
                    for (int v = 1; v < n; v++) {
                        if (v == i || v == j || !edge[v] || !edge[i * n + v] || !edge[j * n + v]) continue;
                        const float x = (float)P[v].x, y = (float)P[v].y, z = (float)P[v].z, st = (float)P[v].st;
                        if (!(pn::power(g.tx, g.ty, g.tz, st, x, y, z) + ((float)P[v].s - st) < -g.mt)) continue;
                        if (bounds.mreach > 0 && !pn::in_box(g.tx, g.ty, g.tz, x, y, z, bounds.mreach)) continue;
                        attached++;
                        abad += !pac::attached(b[v], to.x, to.y, to.z, to.w) || !(reach_of(b[v], to) <= 0.99f * step);
                    }
                std::vector<int> z;
                for (int k = 1; k < n; k++)
                    if (k != i && k != j && edge[k] && edge[i * n + k] && edge[j * n + k]) z.push_back(k);
                for (int c : z) {
                    const float x = (float)P[c].x, y = (float)P[c].y, zz = (float)P[c].z, st = (float)P[c].st;
                    const float h = pn::height(g.nx, g.ny, g.nz, x, y, zz);
                    const float gt = pn::power(g.tx, g.ty, g.tz, st, x, y, zz);
                    const float q = pn::power(g.qx, g.qy, g.qz, (float)P[c].s, x, y, zz);
                    const Ball tet[4] = {p, b[i], b[j], b[c]};
                    float4 o[4];
                    const bool mark[4] = {
                        pac::tet_alpha<pac::AtEnum>(p, b[i], b[j], b[c], alpha, o[0], false),
                        pac::tet_alpha<pac::AtEnum>(p, b[i], b[j], b[c], alpha, o[1], true),
                        pac::tet_alpha<pac::AtRun>(p, b[i], b[j], b[c], alpha, o[2]),
                        pac::tet_alpha<pac::AtSos>(p, b[i], b[j], b[c], alpha, o[3])};
                    tests++;
                    const bool sure = std::fabs(h) >= g.hmin, certain = std::fabs(h) >= bounds.kappa * g.hmin;
                    bool in = false, out = false;
                    pn::alpha_test(std::fabs(h), gt, g.k, g.ea, in, out);
                    if (certain && (in || out)) {
                        certified++;
                        for (bool m : mark) bad += m != in;
                    }
                    if (!sure || !(mark[0] || mark[1])) continue;
                    for (int v : z) {
                        if (v == c) continue;
                        const float vx = (float)P[v].x, vy = (float)P[v].y, vz = (float)P[v].z;
                        const float hy = pn::height(g.nx, g.ny, g.nz, vx, vy, vz);
                        const float qy = pn::power(g.qx, g.qy, g.qz, (float)P[v].s, vx, vy, vz);
                        if (!(std::fabs(hy) >= g.hmin) || !pn::refutes(h, q, hy, qy, g.rg)) continue;
                        if (bounds.reach > 0 && !pn::within_reach(g.nx, g.ny, g.nz, g.tx, g.ty, g.tz, h, gt, vx, vy,
                                                                  vz, bounds.reach))
                            continue;
                        refuted++;
                        for (int how = 0; how < 3; how++) rbad += !violates(tet, b[v], how);
                        for (int k = 0; k < 2; k++) rbad += mark[k] && !(reach_of(b[v], o[k]) <= 0.99f * step);
                    }
                }
            }
    }
    std::printf("alpha %ld certified %ld bad %ld refutations %ld bad %ld attachments %ld bad %ld\n", tests, certified,
                bad, refuted, rbad, attached, abad);
    return 0;
}
