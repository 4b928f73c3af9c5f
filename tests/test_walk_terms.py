"""The short-range force is the tree walk's, its node terms included: where the
opening test accepts a node, the node's moments stand for its particles, at any
density.

The forces of every fifth particle are compared with recorded ones of the same
walk (tests/golden/walk_terms.npz: clumps of 60 particles in a uniform box of
one particle per cell, both laws). Another order of the moments' sums changes
them by a few times 2^-24 of a term; the tolerance is 1e-5 of the forces' norm,
and 1e-4 of their rms for a single one. A sum over the particles of the accepted
nodes instead is 100 times as far away.
"""
import os

import numpy as np
import pytest

from lageunha_b200 import engine as E
from lageunha_b200 import ic

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "walk_terms.npz")
LAWS = {"gaussian": (24, {"law": "gaussian", "rs_split": 0.7, "rsphere": 3.5, "theta": 0.4}),
        "reference": (32, {"law": "reference", "rsphere": 4.0, "theta": 0.3})}


def _points(n):
    rng = np.random.Generator(np.random.PCG64(4100 + n))
    p = rng.random((n ** 3, 3)) * n
    c = rng.random((24, 3)) * n
    p = np.concatenate([p] + [q + 0.3 * rng.standard_normal((60, 3)) for q in c])
    return ic.to_fixed_point(np.mod(p, n), n)


@pytest.mark.parametrize("law", sorted(LAWS))
def test_walk_keeps_its_node_terms(law):
    n, prm = LAWS[law]
    want = np.load(GOLDEN)[law].astype(np.float64)
    with E.Engine(n, epsilon=0.05, **prm) as eng:
        eng.load_fixed(_points(n))
        eng.compute(E.PART_TREE)
        f = eng.forces()[::5].astype(np.float64)
        assert eng.counters()["pc"] > 0
    assert np.linalg.norm(f - want) <= 1e-5 * np.linalg.norm(want)
    assert np.abs(f - want).max() <= 1e-4 * np.sqrt((want ** 2).mean())
