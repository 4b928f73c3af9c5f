"""The octree that the two passes over the sorted keys build: its node count
against the rule (a cube with particles whose parent holds at least 10), its
ranges through friends-of-friends groups, which walk every level's nodes, and its
moments through the force of an accepted node. The build has tiles of 256
particles below 2^20 particles and of 2048 from there on; the counts sit at the
edges of both, and the sets hold runs of equal keys (the deepest level), cubes of
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
@pytest.mark.parametrize("count", [9, 10, 11, 255, 256, 257, 2047, 2048, 2049, 4097])
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


@pytest.mark.parametrize("count", [2 ** 20 - 1, 2 ** 20, 2 ** 20 + 1, 2 ** 20 + 2049])
def test_groups_and_nodes_of_the_long_tiles(count):
    n = 100
    rng = np.random.Generator(np.random.PCG64(count))
    p = np.concatenate([rng.random((count - 23000, 3)) * n, np.tile([[50.0, 3.3, 96.0]], (3000, 1)),
                        [[0.0, 48.0, 63.9]] + 0.5 * rng.standard_normal((20000, 3))])
    pu = ic.to_fixed_point(np.mod(p, n), n)
    with E.Engine(n, epsilon=0.05) as eng:
        eng.load_fixed(pu)
        lab, ng = eng.fof(0.2, 2)
        eng.compute(E.PART_TREE)
        assert eng.counters()["nodes"] == _node_count(O.morton_keys(pu, n))
        assert np.all(np.isfinite(eng.forces()))
    want, ngw = O.fof_labels(n, ic.from_fixed_point(pu, n), 0.2, 2)
    assert ng == ngw and np.array_equal(lab.astype(np.int64), want)


@pytest.mark.parametrize("centre,scale", [([18.0, 18.0, 18.0], 1.0), ([0.9, 31.2, 14.6], 1.0),
                                          ([18 + 0.5 / 256, 18 + 1.5 / 256, 18 + 2.5 / 256], 1.5e-3)])
def test_moments_of_an_accepted_node(centre, scale):
    """A lopsided clump of 400 particles in one 4-cell cube, or shrunk into one
    cube of the deepest level (a leaf that a warp sums), and single ones
    around it that accept the cube's node as a whole (opening angle 0.9). Their
    force is the node's, with the clump's mass, centre and second moments, and
    the other single ones', all in FP64. The tolerance is four times the law
    tables' 2.8e-5 of the clump's Newtonian force, of which the terms of the
    second moments of the wide clump are 0.2-2.5% and those beyond up to 0.07%."""
    n, rs, eps = 32, np.float32(2.0).item(), np.float32(0.05).item()
    rng = np.random.Generator(np.random.PCG64(9))
    c = np.array(centre)
    clump = np.clip(rng.standard_normal((400, 3)), -2.4, 2.4) * [0.34, 0.2, 0.1] + 0.25 * (rng.random((400, 1)) < 0.3)
    clump = c + scale * clump
    d = rng.standard_normal((4000, 3))
    around = d / np.linalg.norm(d, axis=1)[:, None] * (3.2 + 1.4 * rng.random((4000, 1)))
    around = around[np.abs(around).max(1) > 2.9]
    cubes = {tuple(np.floor(np.mod(c, n) / 4))}
    keep = []
    for i, q in enumerate(np.floor(np.mod(c + around, n) / 4)):  # each alone in its cube: a group of its own
        if tuple(q) not in cubes:
            cubes.add(tuple(q))
            keep.append(i)
    around = c + around[keep]
    pu = ic.to_fixed_point(np.mod(np.concatenate([clump, around]), n), n)
    pos = ic.from_fixed_point(pu, n)
    with E.Engine(n, epsilon=0.05, theta=0.9, law="gaussian", rsphere=6.0, rs_split=2.0) as eng:
        eng.load_fixed(pu)
        eng.compute(E.PART_TREE)
        f = eng.forces()[400:].astype(np.float64)
    assert len(around) >= 8 and len(np.unique(np.floor(np.mod(clump, n) / 4), axis=0)) == 1
    assert scale == 1.0 or len(np.unique(O.morton_keys(pu[:400], n))) == 1

    from scipy.special import erf

    def law(r):  # the attraction of a unit mass, cells
        u = r / (2 * rs)
        return -(r / (r * r + eps * eps) ** 1.5 - (erf(u) - 2 * u / np.sqrt(np.pi) * np.exp(-u * u)) / r ** 2)

    def wrap(x):
        return x - n * np.round(x / n)

    rel = wrap(pos[:400] - c)
    com = rel.mean(0)
    Q = (rel - com).T @ (rel - com)
    want, newton = np.zeros_like(f), np.zeros(len(f))
    for i, x in enumerate(pos[400:]):
        v = wrap(x - c) - com
        r, h = np.linalg.norm(v), 1e-3
        g, g1, g2 = law(r), (law(r + h) - law(r - h)) / (2 * h), (law(r + h) - 2 * law(r) + law(r - h)) / h ** 2
        f1, f2, f3 = g / r, (g1 * r - g) / (2 * r ** 3), (g2 * r * r - 3 * g1 * r + 3 * g) / (2 * r ** 5)
        want[i] = v * (400 * f1 + np.trace(Q) * f2 + v @ Q @ v * f3) + 2 * f2 * (Q @ v)
        newton[i] = 400 / r ** 2
        for y in np.delete(pos[400:], i, 0):
            s = wrap(x - y)
            r = np.linalg.norm(s)
            if r < 6.0:
                want[i] += s * law(r) / r
    assert np.all(np.abs(f * n ** 2 - want).max(1) <= 1.12e-4 * newton)
