"""Balls whose neighbours' indices collide in every attempt of the kernels'
table, so that positions are found by search."""
import numpy as np
import pytest

SOL, ALPHA = 0.0, 0.0


def _mixed(count, tiny, seed):
    """Large balls that nearly all meet, over eight cells, between tiny ones that
    hardly any sphere meets: in the cells' order the neighbours of a ball are
    scattered, not runs of consecutive indices."""
    rng = np.random.default_rng(seed)
    big = np.concatenate([rng.uniform(2.8, 7.4, (count, 3)), rng.uniform(2.4, 2.6, (count, 1))], 1)
    small = np.concatenate([rng.uniform(0, 10.2, (tiny, 3)), np.full((tiny, 1), 0.003)], 1)
    small[0, :3], big[0, 3] = 0, 2.6  # the grid's corner and the largest radius
    b = np.concatenate([big, small]).astype(np.float32)
    return b[rng.permutation(len(b))]


def _searched(b):
    """Balls for which each of the eight attempts collides (restating the rule
    of hash_slot: the low bits, then seven multiplications)."""
    step = 2 * np.sqrt(b[:, 3].max() ** 2 + ALPHA)
    c = ((b[:, :3] - b[:, :3].min(0)) / step).astype(int)
    g = c.max(0) + 1
    o = np.argsort(c[:, 0] + g[0] * (c[:, 1] + g[1] * c[:, 2]), kind="stable")
    p, c = b[o].astype(float), c[o]
    r = np.sqrt((p[:, 3] + SOL) ** 2 + ALPHA)
    found = []
    for i in range(len(p)):
        j = np.arange(i + 1, len(p))
        d = np.linalg.norm(p[j, :3] - p[i, :3], axis=1)  # the spheres meet
        near = (d <= r[i] + r[j]) & (d >= np.abs(r[i] - r[j])) & (np.abs(c[j] - c[i]).max(1) <= 1)
        x = j[near].astype(np.uint64)
        if len(x) < 3:
            continue
        bits = 10 if len(x) <= 64 else 11 if len(x) <= 128 else 13
        slots = [x & np.uint64((1 << bits) - 1)]
        for t in range(1, 8):
            m = np.uint64(2654435769 * (2 * t + 1) & 0xffffffff)
            slots.append(((x * m) & np.uint64(0xffffffff)) >> np.uint64(32 - bits))
        if all(len(np.unique(s)) < len(x) for s in slots):
            found.append(len(x))
    return found


# large and tiny balls: degrees of at most 64, of 65 to 128 (the widest class's
# table, 8,192 slots, settles at every degree tried)
CASES = {"64": (60, 2500), "128": (110, 5000)}


@pytest.mark.parametrize("name", list(CASES))
def test_inputs_reach_the_search(name):
    deg = _searched(_mixed(*CASES[name], seed=7))
    print(len(deg), max(deg, default=0))
    assert any(int(name) // 2 < d <= int(name) for d in deg)


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("formula", ["upstream", "plain-xmp"])
def test_searched_positions_match_restatement(pac, orc, name, formula):
    b = _mixed(*CASES[name], seed=7)
    e, t, q, st = orc.alpha_complex(b, SOL, ALPHA, orc.UPSTREAM if formula == "upstream" else orc.PLAIN_XMP,
                                    tet_ortho=True)
    with pac.Engine(formula=formula) as eng:
        r = eng.alpha_complex(b, SOL, ALPHA)
    for got, want in ((r.edges, e), (r.tris, t), (r.tets, q)):
        np.testing.assert_array_equal(got, want)
    for k in ("alpha_tris", "cand_tets", "alpha_tets"):
        assert r.stats[k] == st[k], k
