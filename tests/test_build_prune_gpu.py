"""robustPrune's job classes (csrc/prune.cuh, csrc/build.cu) against the oracle's build: the same graph and the same
number of distance comparisons."""
import numpy as np
import pytest

import parlayann_b200 as P
from conftest import random_points
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def same_build(base, R, L, alpha, passes, metric):
    idx = P.Index(base, R, metric)
    st = idx.build(L, alpha, num_passes=passes)
    g = idx.get_graph()
    idx.close()
    o, tot = O.build_graph("oracle", base, R, L, alpha, passes, metric=metric)
    np.testing.assert_array_equal(g[:, 0], o[:, 0])
    np.testing.assert_array_equal(np.where(np.arange(R) < g[:, :1], g[:, 1:], 0),
                                  np.where(np.arange(R) < o[:, :1], o[:, 1:], 0))
    assert st.dist_cmps == tot


# degrees around a warp and a word of candidates, rows shorter and longer than one 128-byte line, alphas that keep
# (equal, larger for Euclidean) or drop (smaller, larger for mips) what the first pass proved about a row's pairs
@pytest.mark.parametrize("R,L,d,alpha", [(1, 4, 5, 1.2), (8, 12, 33, 1.0), (31, 40, 96, 1.2), (33, 40, 40, 0.9),
                                         (64, 100, 20, 1.1)])
@pytest.mark.parametrize("dtype,metric", [(np.uint8, P.L2), (np.int8, P.MIPS), (np.float32, P.L2),
                                          (np.float32, P.MIPS)])
def test_shapes(R, L, d, alpha, dtype, metric, lib_built):
    same_build(random_points(dtype, 3000, d, R + d), R, L, alpha, 2, metric)


@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
def test_repeated_points(dtype, lib_built):
    """Many equal points: equal distances, repeated candidates, kills at distance zero."""
    base = random_points(np.uint8, 40, 16, 5)[np.random.default_rng(6).integers(0, 40, 2000)].astype(dtype)
    same_build(base, 16, 24, 1.2, 2, P.L2)


@pytest.mark.parametrize("n,d,R,L", [(12000, 8, 16, 24), (230000, 4, 4, 6)])
def test_targets_of_many_edges(n, d, R, L, lib_built):
    """Inner product with three dominating points: a target takes every inserted point of a batch as a candidate
    (240: a block per job; 4,600: sorted in global memory)."""
    base = np.random.default_rng(1).integers(1, 20, (n, d)).astype(np.uint8)
    base[:3] = 255
    same_build(base, R, L, 1.2, 1, P.MIPS)
