"""Exact ties whose inputs span many binary digits: the simulation of simplicity
and the exact predicates in 640-bit integers, and on both sides of the line to
256 bits (four times the span and 12 bits must fit)."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shell(k, seed):
    """The points (e, 1, 1.5), e = 2^-k (1 + 2^-20), with its coordinates in any
    order and the large ones of either sign: 24 points exactly on one sphere,
    in coordinates from 2^-(k + 20) to 1.5; and four balls inside and around."""
    e = np.float32(2.0 ** -k * (1 + 2.0 ** -20))
    pts = [[(e, 1.0 * s, 1.5 * t)[i] for i in p] for p in itertools.permutations(range(3))
           for s in (1, -1) for t in (1, -1)]
    extra = [[0.75, 0.5, 3.25], [-2.5, 2.75, 0.25], [2.5, -2.5, -2.0], [-2.25, -2.5, 2.0]]
    b = np.array([p + [1.5] for p in pts + extra], np.float32)
    return b[np.random.default_rng(seed).permutation(len(b))]


# spans of 71, 61 and 60 bits: 640-bit integers, the shortest span that takes
# them in the simulation, the longest that does not
@pytest.mark.parametrize("k", [50, 40, 39])
@pytest.mark.parametrize("predicates", ["strict", "exact"])
def test_wide_exact_ties_match_restatement(pac, orc, k, predicates):
    balls = _shell(k, k)
    e, t, q, st = orc.alpha_complex(balls, 0.0, 1.5, exact=predicates == "exact")
    with pac.Engine(predicates=predicates) as eng:
        r = eng.alpha_complex(balls, 0.0, 1.5)
    for got, want in ((r.edges, e), (r.tris, t), (r.tets, q)):
        np.testing.assert_array_equal(got, want)
    print(r.counts(), r.stats["sos_calls"], r.stats["exact_fallbacks"], st["sos_calls"])
    assert r.stats["alpha_tets"] == st["alpha_tets"]
    assert r.stats["sos_calls"] > 100
    if predicates == "exact":
        assert r.stats["exact_fallbacks"] > 100
