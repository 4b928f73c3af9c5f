"""The single-sweep sort of a force evaluation: the permutation is the stable
argsort of the Morton keys and the keys are recomputed exactly, at the edges of
its 4096-particle tiles, for equal keys (one digit takes everything), for
already sorted and reversed sets, and over enough tiles that the look-back
passes several of them."""
import numpy as np
import pytest

from lageunha_b200 import engine as E
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _points(kind, count):
    rng = np.random.Generator(np.random.PCG64(count))
    p = rng.integers(0, 2 ** 32, (count, 3), dtype=np.uint64).astype(np.uint32)
    if kind == "equal":
        p[:] = p[0]
    elif kind == "few":  # three places: stability decides the order
        p = p[rng.integers(0, min(3, count), count)]
    elif kind in ("sorted", "reversed"):
        p = p[np.argsort(O.morton_keys(p, 32), kind="stable")]
        if kind == "reversed":
            p = p[::-1].copy()
    return p


@pytest.mark.parametrize("kind,count", [("random", 1), ("random", 2), ("random", 4095), ("random", 4096),
                                        ("random", 4097), ("random", 300001), ("equal", 5000), ("few", 70000),
                                        ("sorted", 12289), ("reversed", 12289)])
@pytest.mark.parametrize("n", [16, 135])
def test_permutation_is_the_stable_argsort(kind, count, n):
    pu = _points(kind, count)
    with E.Engine(n, epsilon=0.05) as eng:
        eng.load_fixed(pu)
        eng.compute(E.PART_PM)
        keys, perm = eng.order()
    want = O.morton_keys(pu, n)
    order = O.sort_order(want)
    assert np.array_equal(perm.astype(np.int64), order)
    assert np.array_equal(keys, want[order])
