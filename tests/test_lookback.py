"""The look-back of the single-sweep sort (lageunha_b200/csrc/lookback.h) on the
host: a tile learns the number of items before it from its predecessors' words,
at once, late or never published. A predecessor that never reports must not
change the number (a partial one would move the keys of later passes past their
buffers) nor hold the tile up."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "lageunha_b200", "csrc")


@pytest.fixture(scope="module")
def lookback(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    out = str(tmp_path_factory.mktemp("lookback") / "liblookback.so")
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-I", CSRC,
                    os.path.join(HERE, "lookback_harness.cpp"), "-o", out], check=True)
    fn = ctypes.CDLL(out).lookback
    fn.restype = ctypes.c_uint32
    fn.argtypes = [ctypes.c_int64, ctypes.c_uint32] + [ctypes.c_void_p] * 5

    def run(tile, limit, count, kind, after):
        count, after = np.array(count, np.uint32), np.array(after, np.uint32)
        kind = np.array(kind, np.uint8)
        counted, looked = np.zeros(len(count) + 1, np.uint32), np.zeros(1, np.uint64)
        r = fn(tile, limit, *(a.ctypes.data for a in (count, kind, after, counted, looked)))
        return r, counted, int(looked[0])
    return run


@pytest.mark.parametrize("tile", [0, 1, 2, 3, 4, 5, 8, 9, 37])
def test_every_word_published(lookback, tile):
    count = np.arange(tile) * 7 % 11
    for kind in (np.r_[2, np.ones(max(tile - 1, 0))][:tile], np.full(tile, 2)):
        r, counted, _ = lookback(tile, 100, count, kind, np.zeros(tile))
        assert r == count.sum() and not counted.any()


def test_a_word_that_comes_late(lookback):
    count = np.arange(1, 21)
    after = np.zeros(20)
    after[13] = 50
    r, counted, _ = lookback(20, 1000, count, np.r_[2, np.ones(19)], after)
    assert r == count.sum() and not counted.any()


@pytest.mark.parametrize("limit", [0, 3, 1000])
@pytest.mark.parametrize("missing", [[0], [19], [0, 1, 2, 3], [4, 5, 11], list(range(20))])
def test_words_that_never_come(lookback, limit, missing):
    count = np.arange(1, 21)
    kind = np.r_[2, np.ones(19)]
    kind[missing] = 0
    r, counted, looked = lookback(20, limit, count, kind, np.zeros(20))
    assert r == count.sum()
    # each missing tile is counted once (with no look to spare, others may be)
    assert all(counted[t] == 1 for t in missing) and counted.max() == 1
    assert looked <= 4 * (limit + 21)


def test_random_states(lookback):
    rng = np.random.default_rng(5)
    for _ in range(400):
        tile = int(rng.integers(1, 40))
        count = rng.integers(0, 4097, tile)
        kind = rng.integers(0, 3, tile)
        after = np.where(rng.random(tile) < 0.3, rng.integers(0, 20, tile), 0)
        r, _, looked = lookback(tile, int(rng.integers(0, 60)), count, kind, after)
        assert r == count.sum()
        assert looked <= 4 * (60 + 2 * tile + 1)
