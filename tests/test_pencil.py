"""The enumeration's certified filter (parallelac-xmp_b200/csrc/pencil.cuh): on
the CPU against the binary32 formulas it stands for and against the exact
predicates, at the origin and far from it, on generic, nearly flat and lattice
inputs; on the GPU in verify mode (every certified decision replayed) and list
for list against the restatement where the kernels' paths differ."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def harness(tmp_path_factory, orc):
    out = tmp_path_factory.mktemp("pencil") / "pencil_harness"
    lib = os.path.join(ROOT, "oracle", "_build")
    subprocess.run(["g++", "-O2", "-mfma", "-std=c++17", "-ffp-contract=off", "-o", str(out),
                    os.path.join(ROOT, "tests", "native", "pencil_harness.cpp"),
                    "-L", lib, "-loracle", "-Wl,-rpath," + lib], check=True)
    return str(out)


@pytest.mark.parametrize("offset,sol,lattice,exact", [
    (0, 1.4, 0, 0), (80, 1.4, 0, 0), (300, 1.4, 0, 0), (3000, 1.4, 0, 0),
    (80, 0.0, 0, 0), (20, 3.5, 0, 0), (40, 1.4, 1, 0), (80, 1.4, 0, 1), (40, 1.4, 1, 1)])
def test_pencil_filter_never_disagrees(harness, offset, sol, lattice, exact):
    """No certified decision differs from the arithmetic's; most alpha tests
    are certified (random clusters: nearly flat triangles are not)."""
    r = subprocess.run([harness, "7", "25" if exact else "120", str(offset), str(sol), str(lattice),
                        str(exact)], capture_output=True, text=True, check=True)
    f = r.stdout.split()
    print(r.stdout.strip())
    tests, cert, bad, refuted, rbad = (int(f[k]) for k in (1, 3, 5, 7, 9))
    assert bad == 0 and rbad == 0
    attached, abad = int(f[11]), int(f[13])
    assert abad == 0
    assert attached > 1000 or sol > 3  # (a window not certain leaves them to the general path)
    assert tests > 1000 and refuted > 1000
    assert cert > (0.5 if offset < 1000 else 0.2) * tests


def _clump(n, seed, side):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.uniform(0, side, (n, 3)), rng.uniform(1.5, 1.8, (n, 1))],
                          1).astype(np.float32)


def _inputs(pac, name):
    if name == "shifted":      # far from the origin: wide rounding of the reference's squares
        b = pac.globule(1500, seed=5)
        b[:, :3] += np.float32([900, -700, 1100])
        return b, 1.4, 0.5
    if name == "probe":        # probe radius beyond the grid step: the window is checked by distance
        return pac.globule(400, seed=6), 3.0, 0.5
    if name == "clump":        # degrees over 128: the widest class, face rows over 128 bits
        return _clump(150, 3, 5.5), 0.6, 0.5
    return _clump(90, 4, 5.0), 0.8, 0.5   # degrees of 65..89: the middle class


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["shifted", "probe", "clump", "middle"])
@pytest.mark.parametrize("predicates", ["strict", "exact"])
def test_enumeration_paths_match_restatement(pac, orc, name, predicates):
    balls, sol, alpha = _inputs(pac, name)
    e, t, q, st = orc.alpha_complex(balls, sol, alpha, exact=predicates == "exact")
    with pac.Engine(predicates=predicates) as eng:
        r = eng.alpha_complex(balls, sol, alpha)
    for got, want in ((r.edges, e), (r.tris, t), (r.tets, q)):
        np.testing.assert_array_equal(got, want)
    for k in ("cand_tets", "alpha_tets"):
        assert r.stats[k] == st[k], k
    if name == "clump":
        assert r.stats["max_degree"] > 128


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["shifted", "probe", "clump"])
@pytest.mark.parametrize("predicates", ["strict", "fma", "exact"])
def test_enumeration_certificates_hold_on_gpu(pac, name, predicates):
    """Verify mode with refutation on: every certified alpha decision and
    refutation replayed by the general path, no disagreement."""
    balls, sol, alpha = _inputs(pac, name)
    with pac.Engine(verify=True, predicates=predicates) as eng:
        st = eng.alpha_complex(balls, sol, alpha).stats
    print("%d certified decisions, %d refuted of %d alpha" % (st["cert_decisions"], st["early_refuted"],
                                                              st["alpha_tets"]))
    assert st["cert_disagreements"] == 0
    assert st["early_refuted"] > 0.25 * st["alpha_tets"]
