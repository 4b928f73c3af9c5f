"""The direct short-range sum over 4-cell cubes.

Against the tree walk: groups cut from 8-cell cubes (tuning group_level 3) take
the walk for every particle; the default takes the direct sum wherever its rule
allows. With an opening angle that accepts no node both sum the same pairs, so
the forces differ by 32-bit rounding only: about 1e3 terms in another order
(2e-6 of the sum) and coordinates relative to another reference (2^-22 cells
over a softening of 0.05 cells: 5e-6 of a close pair). The tolerance is four
times the sum of the two. The split is short enough for the law at the cut,
whose last bin may or may not be pruned, to be below 1e-3 of a pair's force.

On small boxes, where an 8-cell group's reach exceeds half the box, against an
FP64 sum over all pairs of the law as the engine's table ends it, within 2.8e-5
of a pair's Newtonian force; the tolerance is about four times that.
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


def _pair_sum(pu, n, rsphere, rs, eps):
    """Gaussian-split short-range force of unit masses, FP64, minimum image.
    The law ends as the engine's table does: linear to zero over the bin of
    2^-7 octaves of s = r^2 + 2^-20 that ends at the first bin edge past the
    cut."""
    from scipy.special import erf

    def law(r2):
        r = np.maximum(np.sqrt(r2), 1e-9)
        u = r / (2 * rs)
        return -((r2 + eps * eps) ** -1.5 - (erf(u) - 2 * u / np.sqrt(np.pi) * np.exp(-u * u)) / r ** 3)

    floor = 2.0 ** -20
    step = 2.0 ** (np.floor(np.log2(rsphere ** 2)) - 7)
    s1 = step * np.ceil((rsphere ** 2 + floor) / step)
    edge = law(s1 - step - floor)
    x = ic.from_fixed_point(pu, n)
    out = np.zeros_like(x)
    for i in range(0, len(x), 64):
        d = x[i:i + 64, None, :] - x[None, :, :]
        d -= n * np.round(d / n)
        r2 = (d ** 2).sum(-1)
        ramp = (s1 - floor - r2) / step
        w = np.where(ramp >= 1, law(r2), edge * np.maximum(ramp, 0.0))
        out[i:i + 64] = (d * np.where(r2 > 0, w, 0.0)[..., None]).sum(1)
    return out / n ** 2


@pytest.mark.parametrize("n,count,rsphere", [
    (16, 3000, 4.0),   # the reach spans the box
    (16, 1, 4.0),      # one particle
    (18, 5000, 3.5),   # last cubes two cells wide
    (20, 6000, 6.0),   # two cubes each way
])
def test_direct_matches_pair_sum(n, count, rsphere):
    pu = _points("uniform", n, count)
    rs, eps = np.float32(0.8).item(), np.float32(0.05).item()
    with E.Engine(n, epsilon=0.05, theta=0.3, law="gaussian", rsphere=rsphere, rs_split=0.8) as eng:
        eng.load_fixed(pu)
        eng.compute(E.PART_TREE)
        f = eng.forces().astype(np.float64)
    want = _pair_sum(pu, n, rsphere, rs, eps)
    assert np.linalg.norm(f - want) <= 1e-4 * np.linalg.norm(want)


@pytest.mark.parametrize("kind,n,count,law,rsphere", [
    ("uniform", 45, 60000, "reference", 4.0),  # last cubes one cell wide, sparse
    ("uniform", 36, 90000, "gaussian", 5.5),   # 125 cubes in reach, some left to the walk
    ("uniform", 64, 2000, "gaussian", 4.5),    # mostly empty cubes
    ("blobs", 64, 20000, "gaussian", 3.5),
    ("blobs", 50, 20000, "reference", 4.0),
])
def test_direct_matches_walk(kind, n, count, law, rsphere):
    pu = _points(kind, n, count)
    with E.Engine(n, epsilon=0.05, theta=0.01, law=law, rsphere=rsphere, rs_split=0.6) as eng:
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
    assert np.linalg.norm(f - w) <= 3e-5 * np.linalg.norm(w)
