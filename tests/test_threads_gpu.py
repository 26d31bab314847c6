"""Contexts on several host threads, each making its first pass at once."""
from concurrent.futures import ThreadPoolExecutor
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("predicates", ["strict", "fma"])
def test_first_passes_on_several_threads(pac, predicates):
    balls = pac.globule(900, seed=pac.SEED_BASE + 23)
    gate = threading.Barrier(4)

    def first(_):
        with pac.Engine(predicates=predicates) as eng:
            gate.wait()
            return eng.alpha_complex(balls, 1.4, 1.0)

    with ThreadPoolExecutor(4) as ex:
        a, *others = list(ex.map(first, range(4)))
    for b in others:
        for k in ("edges", "tris", "tets"):
            np.testing.assert_array_equal(getattr(a, k), getattr(b, k))
