"""The contracted flavour (predicates="fma"): its lists are those of the first
build that had it, list for list (tests/golden/contracted_lists.json), also on
inputs full of near ties, where one multiply-add fused or not changes a list;
its as-run lists hold what they counted; and on the CPU its certified filter
never disagrees with the written sequences of refarith.cuh."""
import hashlib
import json
import os
import subprocess

import numpy as np
import pytest

from conftest import GOLDEN, ROOT


def lattice(kind, m, spacing, jitter, radii, offset, seed):
    """A cubic lattice ("sc", "bcc", "fcc") of m cells a side, moved by jitter:
    co-spherical and co-planar up to a few last bits."""
    rng = np.random.default_rng(seed)
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3).astype(float)
    if kind == "bcc":
        g = np.concatenate([g, g + .5])
    if kind == "fcc":
        g = np.concatenate([g + b for b in ((0, 0, 0), (.5, .5, 0), (.5, 0, .5), (0, .5, .5))])
    g = g * spacing + rng.uniform(-jitter, jitter, g.shape) + np.array(offset)
    b = np.concatenate([g, rng.choice(np.array(radii), len(g))[:, None]], 1).astype(np.float32)
    return b[rng.permutation(len(b))]


def _globule(pac, n, seed, shift=(0, 0, 0)):
    b = pac.globule(n, seed=seed)
    b[:, :3] += np.float32(shift)
    return b


def inputs(pac, name):
    """balls, sol_rad, alpha, formula of a recorded case"""
    far, near = (311.3, -700.9, 120.7), (13.7, -21.3, 8.1)
    return {
        "globule-25013": lambda: (_globule(pac, 25013, 780), 1.4, 1.0, "upstream"),
        "globule-25013-far": lambda: (_globule(pac, 25013, 880, (400, -300, 700)), 1.4, 0.5, "upstream"),
        "globule-10007-far": lambda: (_globule(pac, 10007, 879, (400, -300, 700)), 1.4, 0.5, "upstream"),
        "globule-60001": lambda: (_globule(pac, 60001, 4021), 0.0, 1.0, "upstream"),
        "plain-globule-3001": lambda: (_globule(pac, 3001, 978), 0.0, 1.0, "plain-xmp"),
        "sc-near": lambda: (lattice("sc", 9, 1.9, 1e-5, (1.6,), near, 211), 0.3, 0.5, "upstream"),
        "sc-flat": lambda: (lattice("sc", 9, 1.9, 1e-6, (1.5, 1.6, 1.7), (0, 0, 0), 1), 0.0, 1.0, "upstream"),
        "sc-far": lambda: (lattice("sc", 9, 1.9, 1e-6, (1.6,), far, 900), 0.3, 0.5, "upstream"),
        "bcc-mixed": lambda: (lattice("bcc", 7, 2.3, 1e-5, (1.5, 1.6, 1.7), near, 12), 0.0, 1.0, "upstream"),
        "fcc-mixed": lambda: (lattice("fcc", 6, 2.9, 1e-5, (1.5, 1.6, 1.7), near, 23), 0.0, 1.0, "upstream"),
        "sc-wide": lambda: (lattice("sc", 8, 1.45, 1e-5, (1.5, 1.6, 1.7), (5.1, 3.3, -7.7), 301), 0.6, 1.0,
                            "upstream"),
        "plain-sc": lambda: (lattice("sc", 9, 2.47, 1e-5, (1.52, 1.7), near, 105), 0.7, 0.5, "plain-xmp"),
        "plain-sc-near": lambda: (lattice("sc", 9, 1.9, 1e-5, (1.6,), near, 205), 0.3, 0.5, "plain-xmp"),
        # flat tetrahedra whose window's centre names no cell
        "sc-flat-beside": lambda: (lattice("sc", 8, 1.908675471852929, 2.6489814044728684e-07, (1.5, 1.6, 1.7),
                                           (2.230977843233849, 4.63655287871564, -2.0192386464515844), 22009),
                                   0.0, 0.5, "upstream"),
        # zeros whose sphere's cell lies a few last bits from the next
        "fcc-zeros": lambda: (lattice("fcc", 5, 3.1095230816641637, 2.037890214557819e-06, (1.6,),
                                      (-0.055745524162997495, 0.20514445427019334, -0.16597770356890662), 31032),
                              0.7, 0.5, "upstream"),
        "sc-zeros": lambda: (lattice("sc", 8, 1.8865885658291435, 1.1941421051077662e-06, (1.5, 1.6, 1.7),
                                     (0.27711935683454136, -0.4374353934075288, 0.05114556876453136), 33084),
                             0.3, 0.5, "upstream"),
        "plain-fcc-zeros": lambda: (lattice("fcc", 5, 2.6177705613999813, 8.223267098573607e-08, (1.6,),
                                            (-2.7772292734515593, -3.878554559071259, 1.7090199477873946), 23053),
                                    0.7, 0.5, "plain-xmp"),
    }[name]()


AS_WRITTEN = ("globule-25013", "globule-25013-far", "globule-10007-far", "globule-60001", "plain-globule-3001",
              "sc-near", "sc-flat", "sc-far", "bcc-mixed", "fcc-mixed", "sc-wide", "plain-sc", "plain-sc-near",
              "sc-flat-beside", "fcc-zeros", "sc-zeros", "plain-fcc-zeros")


def sha(a):
    return hashlib.sha256(np.ascontiguousarray(a, dtype=np.uint32).tobytes()).hexdigest()


def record(pac, name):
    balls, sol, alpha, formula = inputs(pac, name)
    with pac.Engine(formula=formula, predicates="fma") as eng:
        r = eng.alpha_complex(balls, sol, alpha)
    return {"input": hashlib.sha256(balls.tobytes()).hexdigest(), "counts": list(r.counts()),
            "sha256": [sha(r.edges), sha(r.tris), sha(r.tets)],
            "stats": {k: r.stats[k] for k in ("alpha_edges", "alpha_tris", "cand_tets", "alpha_tets", "sos_calls")}}


@pytest.mark.gpu
@pytest.mark.parametrize("name", AS_WRITTEN)
def test_contracted_lists_are_the_recorded_ones(pac, name):
    want = json.load(open(os.path.join(GOLDEN, "contracted_lists.json")))[name]
    assert record(pac, name) == want


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["sc-far", "sc-run", "fcc-run"])
def test_contracted_as_run_lists_hold_what_was_counted(pac, name):
    """Counting and writing decide alike: no row past the list, none left out."""
    seed, kind, m, sp, radii, off = {
        "sc-far": (900, "sc", 9, 1.9, (1.6,), (311.3, -700.9, 120.7)),
        "sc-run": (901, "sc", 9, 1.9, (1.6,), (101.3, -70.9, 120.7)),
        "fcc-run": (910, "fcc", 5, 2.9, (1.5, 1.6), (311.3, -700.9, 120.7))}[name]
    balls = lattice(kind, m, sp, 1e-6, radii, off, seed)
    with pac.Engine(predicates="fma", tet_mode="as-run") as eng:
        r = eng.alpha_complex(balls, 0.3, 0.5)
    assert len(r.tets) == r.stats["alpha_tets"]
    assert r.tets.max() < len(balls)
    assert len(np.unique(np.sort(r.tets, axis=1), axis=0)) == len(r.tets)
    want = json.load(open(os.path.join(GOLDEN, "contracted_lists.json"))).get("as-run " + name)
    if want:
        assert sha(r.tets) == want["sha256"]


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    out = tmp_path_factory.mktemp("contraction") / "contraction_harness"
    subprocess.run(["g++", "-O2", "-mfma", "-std=c++17", "-ffp-contract=off", "-DPAC_CONTRACTED=1", "-o", str(out),
                    os.path.join(ROOT, "tests", "native", "contraction_harness.cpp")], check=True)
    return str(out)


@pytest.mark.parametrize("offset,sol,flat", [(0, 1.4, 0), (80, 1.4, 1), (300, 1.4, 0), (3000, 1.4, 1), (80, 0.0, 0),
                                             (20, 3.5, 1), (80, -1.2, 0)])
def test_contracted_filter_never_disagrees(harness, offset, sol, flat):
    """Certified decisions against every sequence that decides them."""
    r = subprocess.run([harness, "11", "60", str(offset), str(sol), str(flat)], capture_output=True, text=True,
                       check=True)
    print(r.stdout.strip())
    f = r.stdout.split()
    tests, cert, bad, refuted, rbad, attached, abad = (int(f[k]) for k in (1, 3, 5, 7, 9, 11, 13))
    assert (bad, rbad, abad) == (0, 0, 0)
    assert tests > 1000
    if offset > 1000:
        # a square rounded or not moves the centre by up to u C^2 (0.5 A here),
        # beyond every margin: the filter leaves all to the general path
        return
    assert refuted > 1000
    assert attached > 1000 or sol > 3  # (a window not certain leaves them to the general path)
    assert cert > 0.1 * tests
