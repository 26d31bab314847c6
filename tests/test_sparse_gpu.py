"""Passes of many balls of few neighbours take other kernels (a warp per ball for
links, a block of one warp for the enumeration): the same lists as the
molecules one by one, which are too small for them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("formula", ["upstream", "plain-xmp"])
@pytest.mark.parametrize("predicates", ["strict", "fma", "exact"])
@pytest.mark.parametrize("sol,alpha", [(0.0, 0.0), (0.0, 1.0), (0.7, 1.0)])
def test_batch_of_sparse_molecules_equals_its_molecules(pac, formula, predicates, sol, alpha):
    """Upper degrees on average 8, 14 and 22, at most some 40, 56 and 80: balls on
    both sides of both kernels' limits (24 and 32)."""
    sizes = [2, 3, 1, 4099, 12001, 701, 16403]  # 33,210 balls: past the limit of 32,768
    mols = [pac.globule(n, seed=pac.SEED_BASE + 40 + k) for k, n in enumerate(sizes)]
    off = np.concatenate([[0], np.cumsum(sizes)])
    with pac.Engine(formula=formula, predicates=predicates) as eng:
        res, st = eng.alpha_complex_batch(np.concatenate(mols), off, sol, alpha)
        one = [eng.alpha_complex(m, sol, alpha) for m in mols]
    for a, b in zip(res, one):
        for k in ("edges", "tris", "tets"):
            np.testing.assert_array_equal(getattr(a, k), getattr(b, k))
    for k in ("cand_tris", "alpha_tris", "cand_tets", "alpha_tets"):
        assert st[k] == sum(r.stats[k] for r in one), k


@pytest.mark.parametrize("n", [32767, 32768])
def test_sides_of_the_limit_match_restatement(pac, orc, n):
    balls = pac.globule(n, seed=pac.SEED_BASE + 51)
    e, t, q, st = orc.alpha_complex(balls, 0.0, 1.0)
    with pac.Engine(verify=True) as eng:
        r = eng.alpha_complex(balls, 0.0, 1.0)
    for got, want in ((r.edges, e), (r.tris, t), (r.tets, q)):
        np.testing.assert_array_equal(got, want)
    assert r.stats["cert_disagreements"] == 0
