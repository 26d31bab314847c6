"""Workloads of the alpha complex engine, for timing and comparing builds.

Each case is one call of a public entry point on a synthetic molecule of the
kinds the benchmark and the tests use (self-avoiding-walk globules, their
lattice-snapped form, assemblies of globules, batches of molecules of uneven
size, the union measure over a complex).  listed() holds the cases that stand
for everyday use, draw() gives more of the same ranges, prepare() builds what
a program has in hand before the call and run() makes the call.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """parallelac-xmp_b200/ (not an identifier) as `parallelac_xmp_b200`."""
    name = "parallelac_xmp_b200"
    if name not in sys.modules:
        path = os.path.join(ROOT, "parallelac-xmp_b200")
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(path, "__init__.py"), submodule_search_locations=[path])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


def _case(name, kind, n, shape="globule", formula="upstream", tets="as-written", pred="strict",
          sol=1.4, alpha=1.0, molecules=0):
    c = {"kind": kind, "n": n, "shape": shape, "formula": formula, "tets": tets, "pred": pred,
         "sol": sol, "alpha": alpha, "molecules": molecules}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest molecules of a screening set, one call each: latency
        _case("host-211", "host", 211, alpha=0.5),
        # the plain method's own small case, solvent-free
        _case("host-plain-1300", "host", 1300, formula="plain-xmp", sol=0.0, alpha=0.0),
        # one ordinary protein with a solvent probe, a single host call
        _case("host-5003", "host", 5003, alpha=0.5),
        # the command-line tool's default semantics on a large protein
        _case("host-asrun-20011", "host", 20011, formula="plain-xmp", tets="as-run", sol=0.0),
        # the arithmetic that follows the contracted reference build
        _case("host-fma-25013", "host", 25013, pred="fma"),
        # co-spherical and co-planar input: exact ties everywhere
        _case("host-snapped-25000", "host", 25000, shape="snapped"),
        # the same input with every decision exact
        _case("host-exact-25000", "host", 25000, shape="snapped", pred="exact"),
        # the benchmark's molecule, balls and lists resident on the device
        _case("device-100008", "device", 100000, shape="padded"),
        # a screening set in one call
        _case("batch-256", "batch", 0, alpha=0.5, molecules=256),
        # the largest: a 2.5 M-ball assembly in one pass
        _case("device-assembly-2500000", "device", 400 * 6250, shape="assembly"),
        # volume, area and both gradients: one step of an optimisation, on the
        # device and, for an ordinary protein, through host arrays
        _case("union-device-100008", "union-device", 100000, shape="padded"),
        _case("union-host-5003", "union-host", 5003),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "host", "device", "device", "batch", "union-device",
                       "union-host"])
    if kind == "batch":
        return _case(None, kind, 0, alpha=rng.choice([0.5, 1.0]),
                     molecules=_log_uniform(rng, 8, 400))
    sol, alpha = rng.choice([(0.0, 0.0), (0.0, 1.0), (0.5, 2.0), (1.4, 0.5), (1.4, 1.0)])
    if kind.startswith("union"):
        n = _log_uniform(rng, 200, 150000 if kind == "union-device" else 30000)
        return _case(None, kind, n, sol=sol, alpha=alpha)
    shape = rng.choice(["globule", "globule", "snapped", "padded", "assembly"])
    formula = rng.choice(["upstream", "upstream", "plain-xmp"])
    tets = rng.choice(["as-written", "as-written", "as-written", "as-run"])
    pred = rng.choice(["strict", "strict", "strict", "fma", "exact"])
    if tets == "as-run":  # every alpha tetrahedron is listed: thousands per ball with a probe
        n = _log_uniform(rng, 200, 3000 if sol > 0 else 60000)
    elif pred == "exact":
        n = _log_uniform(rng, 200, 40000)
    else:
        n = _log_uniform(rng, 200, 400000)
    if shape == "assembly":
        n = max(8, n // 8) * 8
    return _case(None, kind, n, shape, formula, tets, pred, sol, alpha)


# One engine per set of options, kept as a program keeps it over many inputs
# (its device pool is gigabytes, so another set of options replaces it).
_ENGINE = [None, None]


def _engine(formula, tets, pred):
    key = (formula, tets, pred)
    if _ENGINE[0] != key:
        if _ENGINE[1] is not None:
            _ENGINE[1].close()
        _ENGINE[:] = [key, _package().Engine(device=torch.cuda.current_device(), formula=formula,
                                             tet_mode=tets, predicates=pred)]
    return _ENGINE[1]


def _balls(case, seed):
    pac = _package()
    seed, n = pac.SEED_BASE + 7919 * (seed % 1000003), case["n"]
    if case["shape"] == "snapped":
        return pac.snapped_globule(n, seed=seed)
    if case["shape"] == "assembly":
        if n == 400 * 6250:
            return pac.assembly(seed=seed)
        # 2 x 2 x 2 globules; the side holds 0.05 balls per cubic Angstrom
        side = max(12.0, (n / 8 / 0.034) ** (1.0 / 3.0))
        return pac.assembly(2, 2, 2, n // 8, pitch=side + 3.0, side=side, seed=seed)
    b = pac.globule(n, seed=seed)
    return pac.pad_corners(b) if case["shape"] == "padded" else b


class _View:
    """__cuda_array_interface__ over a device list of 32-bit indices."""

    def __init__(self, ptr, rows, k):
        addr = ctypes.cast(ptr, ctypes.c_void_p).value
        self.__cuda_array_interface__ = {"shape": (rows, k), "typestr": "<i4",
                                         "data": (addr, False), "version": 2}


def _lists(cx):
    """The lists of a device complex as tensors over the engine's memory."""
    return [torch.as_tensor(_View(p, rows, k), device="cuda") if rows else
            torch.zeros((0, k), dtype=torch.int32, device="cuda")
            for p, rows, k in ((cx.edges, cx.n_edges, 2), (cx.tris, cx.n_tris, 3),
                               (cx.tets, cx.n_tets, 4))]


def _sizes(case):
    """The molecules of a batch: the same sizes for every seed."""
    pac = _package()
    return pac.batch_sizes(case["molecules"], seed=pac.SEED_BASE + 3 + case["molecules"])


def _reach(case):
    """Upper neighbours of a ball within reach, at these generators' densities."""
    return 41.0 * (((1.65 + case["sol"]) ** 2 + case["alpha"]) / 10.3) ** 1.5


def _buffers(case, device):
    """The program's own arrays for the lists, wide enough for any molecule
    of the case's kind and size."""
    n = int(_sizes(case).sum()) if case["kind"] == "batch" else case["n"] + 8
    per = [12.0, 20.0, 10.0]
    if case["tets"] == "as-run":  # all alpha tetrahedra and their faces and edges
        m = _reach(case)
        per = [12 + 2 * m, 20 + m ** 2, 10 + 0.15 * m ** 3]
    return [torch.zeros((int(x * n) + 64, k), dtype=torch.int32, device=device)
            for x, k in zip(per, (2, 3, 4))]


def _keep(buffers, lists):
    """The lists into the program's arrays, and how many rows each holds."""
    for b, x in zip(buffers, lists):
        b[:len(x)].copy_(x)
    return {"rows": [len(x) for x in lists], "edges": buffers[0], "tris": buffers[1],
            "tets": buffers[2]}


def prepare(case, seed):
    pac = _package()
    eng = _engine(case["formula"], case["tets"], case["pred"])
    s = {"case": case}
    if not case["kind"].startswith("union"):
        s["out"] = _buffers(case, "cuda" if case["kind"] == "device" else "cpu")
    if case["kind"] == "batch":
        s["balls"], s["off"] = pac.batch(_sizes(case),
                                         seed=pac.SEED_BASE + 7919 * (seed % 1000003))
        return s
    balls = _balls(case, seed)
    sol, alpha = case["sol"], case["alpha"]
    if case["kind"] == "host":
        s["balls"] = balls
    elif case["kind"] == "device":
        s["balls"] = torch.from_numpy(balls).cuda()
    else:
        s["xyzr"] = pac.grown_radii(balls, sol, alpha)
        if case["kind"] == "union-host":
            s["complex"] = eng.alpha_complex(balls, sol, alpha)
        else:
            d = torch.from_numpy(balls).cuda()
            torch.cuda.synchronize()  # the engine's stream does not wait for torch's
            cx, _ = eng.alpha_complex_device(d.data_ptr(), len(balls), sol, alpha)
            s["lists"] = [t.clone() for t in _lists(cx)]
            u32 = ctypes.POINTER(ctypes.c_uint32)
            s["complex"] = pac.Complex(len(balls), 1, *[len(t) for t in s["lists"]],
                                       *[ctypes.cast(t.data_ptr(), u32) for t in s["lists"]])
            s["d_xyzr"] = torch.from_numpy(s["xyzr"]).cuda()
            s["dvol"] = torch.empty_like(s["d_xyzr"])
            s["darea"] = torch.empty_like(s["d_xyzr"])
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    eng = _engine(case["formula"], case["tets"], case["pred"])
    sol, alpha = case["sol"], case["alpha"]
    if case["kind"] == "host":
        r = eng.alpha_complex(s["balls"], sol, alpha)
        return _keep(s["out"], [torch.from_numpy(x.view(np.int32))
                                for x in (r.edges, r.tris, r.tets)])
    if case["kind"] == "device":
        cx, _ = eng.alpha_complex_device(s["balls"].data_ptr(), len(s["balls"]), sol, alpha)
        # the lists live until the engine's next call: copied on its stream
        with torch.cuda.stream(torch.cuda.ExternalStream(eng.stream())):
            return _keep(s["out"], _lists(cx))
    if case["kind"] == "batch":
        res, _ = eng.alpha_complex_batch(s["balls"], s["off"], sol, alpha)
        # the molecules' lists are consecutive slices of one array per kind
        whole = [torch.from_numpy(x.base.view(np.int32).reshape(-1, k))
                 for x, k in ((res[0].edges, 2), (res[0].tris, 3), (res[0].tets, 4))]
        return dict(_keep(s["out"], whole), molecules=np.array([r.counts() for r in res], np.int64))
    if case["kind"] == "union-host":
        vol, area, dv, da = eng.union_measure(s["xyzr"], s["complex"])
        return {"vol": vol, "area": area, "dvol": dv, "darea": da}
    vol, area = eng.union_measure_device(s["d_xyzr"].data_ptr(), len(s["d_xyzr"]), s["complex"],
                                         s["dvol"].data_ptr(), s["darea"].data_ptr())
    return {"vol": vol, "area": area, "dvol": s["dvol"], "darea": s["darea"]}


def work(case):
    """Bytes: balls in, lists out (per ball about 6.8 edges, 11 triangles, 5.3
    tetrahedra at these densities; the gradients out for the union measure).
    Operations: per ball m = upper neighbours within reach, about 0.4 m^2
    alpha triangles of 40 operations and 0.05 m^3 candidate tetrahedra of
    80 (the alpha test of each is part of what the complex is defined by)."""
    n = int(_sizes(case).sum()) if case["kind"] == "batch" else case["n"]
    lists = 4 * (2 * 6.8 + 3 * 11.0 + 4 * 5.3)
    if case["kind"].startswith("union"):
        return {"bytes": n * (32 + lists + 64), "flops": n * (60 * 6.8 + 900 * 11.0 + 3000 * 5.3)}
    m = _reach(case)
    out = lists
    if case["tets"] == "as-run":
        out += 16 * 0.04 * m ** 3
    return {"bytes": n * (16 + out), "flops": n * (20 * m + 40 * 0.4 * m ** 2 + 80 * 0.05 * m ** 3)}


# ------------------------------------------------------------ 64-bit values
def _unit(v):
    return v / v.square().sum(-1, keepdim=True).sqrt()


def _dot(a, b):
    return (a * b).sum(-1)


def _triple(a, b, Ri, Rj, Rm):
    """Points common to three spheres, relative to the first's centre."""
    n = torch.linalg.cross(a, b)
    nn = _dot(n, n)
    pa = 0.5 * (_dot(a, a) + Ri * Ri - Rj * Rj)
    pb = 0.5 * (_dot(b, b) + Ri * Ri - Rm * Rm)
    x = (pa[:, None] * torch.linalg.cross(b, n) + pb[:, None] * torch.linalg.cross(n, a)) / nn[:, None]
    eta = (Ri * Ri - _dot(x, x)).clamp(min=0).sqrt()
    return x, (eta / nn.sqrt())[:, None] * n


def _intersection(c, R):
    """The common part of k = 2, 3 or 4 balls per row: per ball i its patch's
    area A_i (Gauss-Bonnet) and vector area M_i, and over its ridges, with
    r = (d^2 - (R_i - R_j)^2) / (2 d rho), the sums of r times the ridge's
    length and of r times the integral of sphere i's normal along it."""
    k = c.shape[1]
    out = []
    for i in range(k):
        curv, turn, M, rl, rN = 0.0, 0.0, 0.0, 0.0, 0.0
        for j in range(k):
            if j == i:
                continue
            e = c[:, j] - c[:, i]
            d = _dot(e, e).sqrt()
            u = e / d[:, None]
            t = (d * d + R[:, i] ** 2 - R[:, j] ** 2) / (2 * d)
            rho = (R[:, i] ** 2 - t * t).clamp(min=0).sqrt()
            o = t[:, None] * u
            g = (d * d - (R[:, i] - R[:, j]) ** 2) / (2 * d)
            others = [m for m in range(k) if m not in (i, j)]
            if not others:
                phi, chord = 2 * math.pi * torch.ones_like(t), torch.zeros_like(u)
            else:
                arcs = []
                for m in others:
                    w = c[:, m] - c[:, i] - o
                    w = _unit(w - _dot(w, u)[:, None] * u)
                    x, up = _triple(e, c[:, m] - c[:, i], R[:, i], R[:, j], R[:, m])
                    arcs.append((w, torch.atan2(_dot(up, up).sqrt(), _dot(x - o, w))))
                w1, b1 = arcs[0]
                w2 = torch.linalg.cross(u, w1)
                lo, hi = -b1, b1
                if k == 4:
                    v, b = arcs[1]
                    mid = torch.atan2(_dot(v, w2), _dot(v, w1))
                    blo, bhi = torch.zeros_like(lo), torch.zeros_like(lo)
                    for turns in (-1, 0, 1):
                        l2 = torch.maximum(lo, mid - b + 2 * math.pi * turns)
                        h2 = torch.minimum(hi, mid + b + 2 * math.pi * turns)
                        more = h2 - l2 > bhi - blo
                        blo, bhi = torch.where(more, l2, blo), torch.where(more, h2, bhi)
                    lo, hi = blo, bhi
                phi = hi - lo
                chord = rho[:, None] * ((hi.cos() - lo.cos())[:, None] * w1 +
                                        (hi.sin() - lo.sin())[:, None] * w2)
            curv = curv + phi * t / R[:, i]
            M = M + 0.5 * ((rho * rho * phi)[:, None] * u + t[:, None] * torch.linalg.cross(u, chord))
            rl = rl + g * phi
            rN = rN + (g / R[:, i])[:, None] * ((t * phi)[:, None] * u - torch.linalg.cross(u, chord))
            for m in others:
                if m < j:
                    continue
                x, up = _triple(e, c[:, m] - c[:, i], R[:, i], R[:, j], R[:, m])
                um = _unit(c[:, m] - c[:, i])
                ends = [x + up, x - up]
                if k == 4:  # the end inside the fourth ball
                    f = c[:, 6 - i - j - m] - c[:, i]
                    near = (ends[0] - f).square().sum(-1) < (ends[1] - f).square().sum(-1)
                    ends = [torch.where(near[:, None], ends[0], ends[1])]
                for q in ends:
                    q = q / R[:, i, None]
                    na = _unit(u - _dot(u, q)[:, None] * q)
                    nb = _unit(um - _dot(um, q)[:, None] * q)
                    turn = turn + _dot(na, nb).clamp(-1, 1).acos()
        out.append((R[:, i] ** 2 * (2 * math.pi - curv - turn), M, rl, rN))
    return out


def exact(case, seed):
    """Union volume, area and gradients by inclusion-exclusion in 64 bits,
    the volume by the divergence theorem; the complexes are whole numbers."""
    if not case["kind"].startswith("union"):
        return None
    s = prepare(case, seed)
    cx = s["complex"]
    lists = s["lists"] if "lists" in s else [torch.from_numpy(x.astype(np.int32)).cuda()
                                             for x in (cx.edges, cx.tris, cx.tets)]
    b = torch.from_numpy(s["xyzr"]).cuda()
    r = b[:, 3]
    vol, area = 4 / 3 * math.pi * (r ** 3).sum(), 4 * math.pi * (r ** 2).sum()
    dvol, darea = torch.zeros_like(b), torch.zeros_like(b)
    dvol[:, 3], darea[:, 3] = 4 * math.pi * r * r, 8 * math.pi * r
    for rows in lists:
        sign = -1.0 if rows.shape[1] % 2 == 0 else 1.0
        for at in range(0, len(rows), 250000):
            idx = rows[at:at + 250000].long()
            c, R = b[idx][..., :3], b[idx][..., 3]
            c = c - c[:, :1]
            x0 = c.mean(1)
            for i, (A, M, rl, rN) in enumerate(_intersection(c, R)):
                vol = vol + sign / 3 * (R[:, i] * A + _dot(c[:, i] - x0, M)).sum()
                area = area + sign * A.sum()
                q = (2 / R[:, i])[:, None]
                dvol.index_add_(0, idx[:, i], sign * torch.cat([M, A[:, None]], 1))
                darea.index_add_(0, idx[:, i], sign * torch.cat([q * M + rN, q * A[:, None] + rl[:, None]], 1))
    dvol, darea = (t.cpu().numpy() if case["kind"] == "union-host" else t for t in (dvol, darea))
    return {"vol": float(vol), "area": float(area), "dvol": dvol, "darea": darea}
