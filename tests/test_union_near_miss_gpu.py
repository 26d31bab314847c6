"""Union measure of triangles and tetrahedra three of whose spheres just miss
each other, as a complex decided in single precision may hold them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _foot(c, R2):
    """|x|^2 - R^2 at the point of equal power in the plane of three centres."""
    a, b = c[1] - c[0], c[2] - c[0]
    n = np.cross(a, b)
    x = (0.5 * (a @ a + R2[0] - R2[1]) * np.cross(b, n) + 0.5 * (b @ b + R2[0] - R2[2]) * np.cross(n, a)) / (n @ n)
    return x @ x - R2[0]


def _simplex(k, miss, seed):
    """k balls of which the first three miss each other by miss (A^2), every
    pair's circle at least a fifth of its spheres: adding one constant to the
    squared radii moves no point of equal power."""
    rng = np.random.default_rng(seed)
    while True:
        c = rng.uniform(-2.2, 2.2, (k, 3))
        R2 = rng.uniform(1.7, 3.3, k) ** 2
        R2 = R2 + _foot(c[:3], R2[:3]) - miss
        if R2.min() < 1 or R2.max() > 16:
            continue
        ok = True
        for i in range(k):
            for j in range(k):
                d = np.linalg.norm(c[i] - c[j])
                ok &= i == j or (d > 1 and 1 - ((d * d + R2[i] - R2[j]) / (2 * d)) ** 2 / R2[i] > 0.04)
        if ok:
            return np.concatenate([c, np.sqrt(R2)[:, None]], 1)


@pytest.mark.parametrize("k", [3, 4])
@pytest.mark.parametrize("miss", [1e-9, 1e-4, 1e-3, 1e-2])
def test_spheres_that_just_miss_each_other(pac, orc, k, miss):
    none = [np.zeros((0, q), np.uint32) for q in (2, 3, 4)]
    lists = none[:k - 2] + [np.arange(k, dtype=np.uint32)[None]] + none[k - 1:]
    with pac.Engine() as eng:
        for seed in range(12):
            x = _simplex(k, miss, 100 * seed + k)
            v, a, dv, da = eng.union_measure(x, pac.Result(*lists, None))
            ov, oa, _, _ = orc.union_measure(x, *lists, grad=False)
            # the oracle's corners are arccosines of values off by 10 u / 0.04 at
            # most, near 1: k (k - 1) of them, sqrt(2 * 250 u) off each
            tol = k * (k - 1) * np.sqrt(500 * U) * (x[:, 3] ** 2).max()
            assert abs(a - oa) <= tol
            assert abs(v - ov) <= tol * x[:, 3].max() / 3
            # the areas of the patches are the derivatives by the radii
            assert abs(dv[:, 3].sum() - a) <= 1e-12 * oa
