"""The direct short-range sum over 4-cell cubes against the tree walk.

Groups cut from 8-cell cubes (tuning group_level 3) take the walk for every
particle; the default takes the direct sum wherever its rule allows. With an
opening angle that accepts no node both sum the same pairs, so the forces
differ by 32-bit rounding only: about 1e3 terms in another order (2e-6 of the
sum) and coordinates relative to another reference (2^-22 cells over a
softening of 0.05 cells: 5e-6 of a close pair). The tolerance is four times
the sum of the two.
"""
import numpy as np
import pytest

from lageunha_b200 import engine as E
from lageunha_b200 import ic

pytestmark = pytest.mark.gpu


def _points(kind, n, count):
    rng = np.random.Generator(np.random.PCG64(31 + n))
    p = rng.random((count, 3)) * n
    if kind == "blobs":
        # an isolated cube of 300 targets (three passes), one of 2000 and a
        # clump of 6000 that is left to the walk, on the periodic corner
        blob = lambda c, m, s: np.asarray(c) + s * rng.standard_normal((m, 3))  # noqa: E731
        p = np.concatenate([p, blob([22, 22, 22], 300, 0.3), blob([38, 10, 30], 2000, 0.6), blob([0, 0, 0], 6000, 0.8)])
    return ic.to_fixed_point(np.mod(p, n), n)


@pytest.mark.parametrize("kind,n,count,law,rsphere", [
    ("uniform", 16, 3000, "gaussian", 3.5),    # the reach spans the box
    ("uniform", 16, 1, "gaussian", 4.0),       # one particle
    ("uniform", 18, 5000, "reference", 4.0),   # last cubes two cells wide
    ("uniform", 20, 6000, "gaussian", 6.0),    # two cubes each way
    ("uniform", 45, 60000, "reference", 4.0),  # last cubes one cell wide, sparse
    ("uniform", 36, 90000, "gaussian", 5.5),   # 125 cubes in reach, some left to the walk
    ("uniform", 64, 2000, "gaussian", 3.0),    # mostly empty cubes
    ("blobs", 64, 20000, "gaussian", 3.5),
    ("blobs", 50, 20000, "reference", 4.0),
])
def test_direct_matches_walk(kind, n, count, law, rsphere):
    pu = _points(kind, n, count)
    with E.Engine(n, epsilon=0.05, theta=0.01, law=law, rsphere=rsphere, rs_split=0.8) as eng:
        eng.load_fixed(pu)
        eng.compute(E.PART_TREE)
        f = eng.forces().astype(np.float64)
        eng.compute(E.PART_TREE)
        assert np.array_equal(eng.forces(), f.astype(np.float32))  # the same bits on every call
        t = eng.tuning
        t.group_level = 3
        eng.tuning = t
        eng.compute(E.PART_TREE)
        w = eng.forces().astype(np.float64)
    if count == 1:
        assert np.all(f == 0) and np.all(w == 0)
        return
    assert np.linalg.norm(f - w) <= 3e-5 * np.linalg.norm(w)
