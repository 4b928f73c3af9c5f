"""The octree that the two passes over the sorted keys build, through what
depends on all of it: friends-of-friends groups walk every level's nodes and
ranges, and the tree walk with an opening angle that accepts many nodes uses
their moments. Particle counts sit at the edges of the build's 2048-particle
tiles, and the sets hold runs of equal keys (the deepest level), cubes of
exactly 9 and 10 particles (the leaf rule) and clumps that span tiles."""
import numpy as np
import pytest

from lageunha_b200 import engine as E
from lageunha_b200 import ic
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _points(kind, n, count):
    rng = np.random.Generator(np.random.PCG64(5 + count))
    if kind == "uniform":
        p = rng.random((count, 3)) * n
    elif kind == "cells":  # 9, 10 or 11 particles in each of random cells
        cells = np.floor(rng.random((count, 3)) * n)
        p = np.repeat(cells, 9 + np.arange(count) % 3, axis=0)[:count] + 0.9 * rng.random((count, 3))
    else:  # equal keys and a dense clump
        p = np.concatenate([np.tile([[3.3, 3.3, 3.3]], (count // 4, 1)), [[8, 8, 8]] + 0.5 * rng.standard_normal((count - count // 4, 3))])
    return ic.to_fixed_point(np.mod(p, n), n)


@pytest.mark.parametrize("kind", ["uniform", "cells", "dense"])
@pytest.mark.parametrize("count", [9, 10, 11, 2047, 2048, 2049, 4097])
def test_groups_and_tree_force(kind, count):
    n = 16
    pu = _points(kind, n, count)
    pos = ic.from_fixed_point(pu, n)
    if kind == "dense":  # distinct separations for the force; the keys stay equal
        pu = pu + (np.arange(count, dtype=np.uint32) % 64)[:, None] * np.uint32(1 << 12)
        pos = ic.from_fixed_point(pu, n)
    with E.Engine(n, epsilon=0.05, theta=0.3, law="gaussian", rsphere=3.0, rs_split=0.6) as eng:
        eng.load_fixed(pu)
        lab, ng = eng.fof(0.21, 2)
        t = eng.tuning
        t.group_level = 3  # every particle to the walk, which needs the tree
        eng.tuning = t
        eng.compute(E.PART_TREE)
        f = eng.forces().astype(np.float64)
        nodes = eng.counters()["nodes"]
    want, ngw = O.fof_labels(n, pos, 0.21, 2)
    assert ng == ngw and np.array_equal(lab.astype(np.int64), want)
    assert nodes == _node_count(O.morton_keys(pu, n))
    assert np.all(np.isfinite(f))


def _node_count(keys):
    """Cubes with particles whose parent holds at least 10, and the root."""
    total, keys = 1, np.sort(keys)
    for level in range(1, 14):
        parent, here = keys >> np.uint64(3 * (14 - level)), keys >> np.uint64(3 * (13 - level))
        cube, count = np.unique(parent, return_counts=True)
        big = cube[count >= 10]
        total += len(np.unique(here[np.isin(parent, big)]))
    return total
