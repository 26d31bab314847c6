"""Device memory of a pass: the alpha-tetrahedron queue and the lists its entries
end in stay within the share of free memory that a context takes, so that a large
pass on a nearly full GPU runs in chunks."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pass_on_a_nearly_full_gpu_runs_in_chunks(pac):
    """2 GiB left free, an alpha tetrahedron queue that would need several times
    that (no early refutation): same lists as with the memory free.  The pool
    hands out blocks of 256 MiB: one for what precedes the queue; one for the
    queue (2 GiB / 4 / 24 B entries of 8 B) and the two first lists (2^22 of
    8 B each); one for each list grown to a whole queue beside its 2^22; one
    for the outputs."""
    torch = pytest.importorskip("torch")
    balls = pac.globule(60001, seed=pac.SEED_BASE + 17)
    with pac.Engine(refute=False) as eng:  # also loads the kernels
        want = eng.alpha_complex(balls, 1.4, 1.0)
    left = 2 << 30
    with pac.Engine(refute=False) as eng:
        gc.collect()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info(0)[0]
        hold = torch.empty(free - left, dtype=torch.uint8, device="cuda:0")
        try:
            before = torch.cuda.mem_get_info(0)[0]
            got = eng.alpha_complex(balls, 1.4, 1.0)
            used = before - torch.cuda.mem_get_info(0)[0]
        finally:
            del hold
            torch.cuda.empty_cache()
    print("free %d MiB, used %d MiB" % (before >> 20, used >> 20))
    for k in ("edges", "tris", "tets"):
        np.testing.assert_array_equal(getattr(got, k), getattr(want, k))
    assert got.stats["alpha_tets"] == want.stats["alpha_tets"]
    assert used <= 5 * (256 << 20)
