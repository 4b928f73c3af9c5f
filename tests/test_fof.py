"""Friends-of-friends groups (tpm_fof) against the FP64 oracle: the groups
are the connected components of "distance <= link" (FoF/fof.c:217-290), so
the partition is unique. Labels (smallest caller index of each group of
>= min_members, else -1) are compared exactly; the seeded sets have no pair
within float rounding of the link length."""
import numpy as np
import pytest

from lageunha_b200 import engine as E
from lageunha_b200 import ic
from oracle import oracle as O


def test_oracle_known_answer():
    # a chain of 5 linked across the periodic boundary, a pair, and loners
    n = 16
    pos = np.array([[15.95, 8, 8], [0.1, 8, 8], [0.25, 8, 8], [0.4, 8, 8], [15.8, 8, 8],  # chain (wraps)
                    [5, 5, 5], [5.15, 5, 5],                                                 # pair
                    [10, 10, 10], [12, 2, 7]], np.float64)
    lab, ng = O.fof_labels(n, pos, 0.2, 2)
    assert list(lab) == [0, 0, 0, 0, 0, 5, 5, -1, -1] and ng == 2
    lab, ng = O.fof_labels(n, pos, 0.2, 3)
    assert list(lab) == [0, 0, 0, 0, 0, -1, -1, -1, -1] and ng == 1


@pytest.mark.gpu
@pytest.mark.parametrize("name,n,link,minm", [("clustered256", 32, 0.2, 20), ("clustered256", 48, 0.1, 10),
                                              ("clustered256", 64, 0.15, 5), ("scale512", 32, 0.25, 3)])
def test_fof_matches_oracle(name, n, link, minm):
    ps = ic.workload(name, scale=n)
    pu = ps.positions_u32()
    pos = ic.from_fixed_point(pu, n)
    want, ngw = O.fof_labels(n, pos, link, minm)
    with E.Engine(n, epsilon=0.05) as eng:
        eng.load_fixed(pu)
        lab, ng = eng.fof(link, minm)
        # the context still evaluates forces afterwards
        eng.compute(E.PART_ALL)
        assert np.all(np.isfinite(eng.forces()))
    assert ng == ngw
    assert np.array_equal(lab.astype(np.int64), want)


@pytest.mark.gpu
def test_fof_singletons_and_no_groups():
    n = 16
    ps = ic.workload("plain64", scale=n)
    with E.Engine(n, epsilon=0.05) as eng:
        eng.load_fixed(ps.positions_u32())
        lab, ng = eng.fof(1e-4, 1)          # every particle its own group
        assert ng == ps.np and np.array_equal(lab, np.arange(ps.np, dtype=np.int32))
        lab, ng = eng.fof(1e-4, 2)          # no pair that close
        assert ng == 0 and np.all(lab == -1)
        with pytest.raises(E.EngineError):
            eng.fof(9.0, 2)                 # link of half the box


def _set(kind, n):
    """Positions for the cube search: clumps on the periodic corner and on
    cube faces, dense enough for whole nodes to lie within the link, a core
    with short links, or a sparse set with links across several cubes."""
    rng = np.random.Generator(np.random.PCG64(77 + n))
    if kind == "clumps":
        c = np.array([[0, 0, 0], [4, 8, 4], [n - 1, 4, 0.02]], np.float64)
        p = np.concatenate([c[i % 3] + 0.08 * rng.standard_normal((400, 3)) for i in range(3)] + [rng.random((300, 3)) * n])
    elif kind == "core":  # dense enough for a warp's particles to be split by octants
        p = np.array([[8.0, 4.0, 0.0]]) + 0.3 * rng.standard_normal((2500, 3))
    else:
        p = rng.random((500, 3)) * n
    return ic.to_fixed_point(np.mod(p, n), n)


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n,link,minm", [("clumps", 16, 0.2, 5), ("clumps", 45, 0.15, 2), ("clumps", 512, 0.25, 3),
                                              ("sparse", 45, 3.0, 2), ("sparse", 16, 1.2, 1), ("sparse", 18, 5.0, 2), ("core", 16, 0.02, 2),
                                              ("core", 45, 0.06, 2), ("core", 512, 0.004, 2)])
def test_fof_cubes_and_cliques(kind, n, link, minm):
    pu = _set(kind, n)
    pos = ic.from_fixed_point(pu, n)
    # no pair sits within the rounding of a 32-bit distance of the link
    d = pos[:, None, :] - pos[None, :, :]
    r = np.sqrt(((d - n * np.round(d / n)) ** 2).sum(-1))
    assert np.min(np.abs(r - link)) > 2e-7 * link
    want, ngw = O.fof_labels(n, pos, link, minm)
    with E.Engine(n, epsilon=0.05) as eng:
        eng.load_fixed(pu)
        lab, ng = eng.fof(link, minm)
    assert ng == ngw
    assert np.array_equal(lab.astype(np.int64), want)


@pytest.mark.gpu
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_fof_nodes_beyond_half_the_box_from_the_first_member(axis):
    """The two members of one 4-cell cube lie 3.8 cells apart; the node of the
    other ten is within the link of the second, and more than half the box from
    the first."""
    n, link = 16, 5.0
    x = np.concatenate([[0.1, 3.9], np.linspace(8.5, 8.8, 10)])
    pos = np.roll(np.stack([x, np.ones(12), np.ones(12)], 1), axis, axis=1)
    pu = ic.to_fixed_point(pos, n)
    want, ngw = O.fof_labels(n, ic.from_fixed_point(pu, n), link, 1)
    assert ngw == 1
    with E.Engine(n, epsilon=0.05) as eng:
        eng.load_fixed(pu)
        lab, ng = eng.fof(link, 1)
    assert ng == ngw and np.array_equal(lab.astype(np.int64), want)


def _stack_set():
    """5955 particles, five in each of some cells of a nested subdivision of the
    16-cell box, for which the search of the first warp (link 7.5: every 4-cell
    cube is near) opens 32 nodes on three levels, then single ones down to 544
    waiting nodes, then 32 more and one: 775 nodes wait, above the 768 that the
    wide steps alone can reach."""
    rng = np.random.Generator(np.random.PCG64(3))
    out = []

    def split(path):
        c, *o = path
        return (c >= 60, c == 63 and o[0] >= 4, c == 63 and o[0] == 5 and len(o) > 1 and o[1] < 4,
                c == 63 and o[0] == 5 and o[1:] == [3, 7, 7], False)[len(o) - 1]

    def cell(lo, side, path):
        for o in range(8):
            b = lo + side / 2 * np.array([o & 1, o >> 1 & 1, o >> 2])
            if split(path + (o,)):
                cell(b, side / 2, path + (o,))
            else:
                out.append(b + side / 2 * (0.1 + 0.8 * rng.random((5, 3))))

    for c in range(64):
        cell(4.0 * np.array([c % 4, c // 4 % 4, c // 16]), 4.0, (c,))
    return np.concatenate(out)


@pytest.mark.gpu
def test_fof_search_holds_every_node():
    n, link = 16, 7.5
    pos = _stack_set()
    assert len(pos) == 5955
    with E.Engine(n, epsilon=0.05) as eng:
        eng.load_fixed(ic.to_fixed_point(pos, n))
        lab, ng = eng.fof(link, 2)
    # neighbouring octants lie closer than the link: one group
    assert ng == 1 and np.all(lab == 0)
