"""The first search tier's row scoring (csrc/rowscore.cuh) and seen tables (csrc/search.cuh) at the ends of their
blocks, against the oracle: ids, distances, visited and comparison counts bit for bit."""
import numpy as np
import pytest

import parlayann_b200 as P
from conftest import random_points
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check(r, o):
    np.testing.assert_array_equal(r.ids, o["ids"])
    np.testing.assert_array_equal(r.dists, o["dists"])
    np.testing.assert_array_equal(r.visited, o["visited"])
    np.testing.assert_array_equal(r.cmps, o["cmps"])


# rows of a part of a 16-byte chunk up to several 128-byte column blocks and a remainder; degrees that leave rounds of
# 1 to 32 rows
@pytest.mark.parametrize("d", [1, 4, 15, 16, 17, 31, 32, 33, 64, 65, 96, 127, 129, 300])
@pytest.mark.parametrize("dtype,metric", [(np.uint8, P.L2), (np.int8, P.L2), (np.int8, P.MIPS), (np.float32, P.L2),
                                          (np.float32, P.MIPS)])
def test_row_lengths(d, dtype, metric, lib_built):
    n, R = 1500, 37
    base = random_points(dtype, n, d, d)
    q = random_points(dtype, 40, d, d + 1)
    g = O.random_graph(n, R, d + 2, min_deg=1)
    idx = P.Index(base, R, metric)
    idx.set_graph(g)
    check(idx.search(q, 5, 24), O.search("oracle", base, q, g, 5, 24, metric=metric))
    idx.close()


# (points, degree, slots): 16-bit tables with distances of up to 2, 30 and 510 buckets from home, tables that fill and
# spill, ids too wide for 16 bits (32-bit entries); beams whose frontier ends inside, at and past 32-entry words
@pytest.mark.parametrize("n,R,slots", [(200_000, 16, 128), (200_000, 16, 2048), (5000, 16, 128), (900, 8, 4096),
                                       (300_000, 16, 128)])
@pytest.mark.parametrize("L", [10, 32, 33, 150])
def test_seen_tables(n, R, slots, L, lib_built):
    base = random_points(np.uint8, n, 8, 3)
    q = random_points(np.uint8, 60, 8, 4)
    g = O.random_graph(n, R, 5, min_deg=R // 2)
    idx = P.Index(base, R)
    idx.set_graph(g)
    b = idx.batch(60, 10, L, seen_slots=slots)
    check(b.run(q, 10, L), O.search("oracle", base, q, g, 10, L))
    b.close()
    check(idx.search(q, 10, L), O.search("oracle", base, q, g, 10, L))
    idx.close()


def test_long_frontier(lib_built):
    """Frontiers past 1,024 entries (the unvisited flags no longer fit a warp's registers) and merges of more than 32
    candidates."""
    base = random_points(np.float32, 6000, 12, 7)
    q = random_points(np.float32, 8, 12, 8)
    g = O.random_graph(6000, 48, 9, min_deg=30)
    idx = P.Index(base, 48)
    idx.set_graph(g)
    for L in (1000, 1024, 1100):
        check(idx.search(q, 10, L), O.search("oracle", base, q, g, 10, L))
    idx.close()


# low-precision rows of a part of a 16-byte chunk up to several 128-byte column blocks, in 16-bit tables (many queries)
# and in wider ones (few): the same traversal, and re-ranked distances that are exactly Point::distance
@pytest.mark.parametrize("d", [1, 7, 16, 17, 33, 129, 300])
@pytest.mark.parametrize("precision", [P.PREC_BF16, P.PREC_FP8])
@pytest.mark.parametrize("metric", [P.L2, P.MIPS])
def test_low_precision_rows(d, precision, metric, lib_built):
    n, R = 4000, 37
    base = random_points(np.float32, n, d, d)
    q = random_points(np.float32, 3000, d, d + 1)
    idx = P.Index(base, R, metric)
    idx.set_graph(O.random_graph(n, R, d + 2, min_deg=1))
    idx.set_precision(precision)
    many = idx.search(q, 10, 40, precision=precision)
    few = idx.search(q[:50], 10, 40, precision=precision)
    for f in ("ids", "dists", "visited", "cmps"):
        np.testing.assert_array_equal(getattr(many, f)[:50], getattr(few, f))
    np.testing.assert_array_equal(few.dists, idx.score(q[:50], few.ids))
    idx.close()


@pytest.mark.parametrize("nq", [1, 2, 31, 32, 33, 64, 65])
def test_few_queries_with_growth(nq, lib_built):
    """Host calls on either side of the size up to which the later tiers are launched only when asked for, on queries
    of which some make the reference's hashset grow."""
    base = random_points(np.uint8, 20000, 8, 1)
    g = O.random_graph(20000, 64, 3, min_deg=60)
    q = random_points(np.uint8, 300, 8, 2)
    grew = O.search("oracle", base, q, g, 10, 40)["hash_grew"] > 0
    assert grew.any() and not grew.all()
    q = np.concatenate([q[grew], q[~grew]])[:nq]  # the first ones grow
    idx = P.Index(base, 64)
    idx.set_graph(g)
    o = O.search("oracle", base, q, g, 10, 40)
    r = idx.search(q, 10, 40)
    check(r, o)
    np.testing.assert_array_equal(r.flags == 1, o["hash_grew"] > 0)
    r = idx.search(q[-1:], 10, 40)  # a call after one that grew
    check(r, O.search("oracle", base, q[-1:], g, 10, 40))
    idx.close()


@pytest.mark.parametrize("n", [1 << 23, (1 << 23) + 9], ids=["16-bit", "32-bit"])
def test_widest_ids_of_4096_slots(n, lib_built):
    """Ids that just fit 16-bit entries at 4,096 slots (23 bits), and ids that do not."""
    rng = np.random.default_rng(6)
    R = 12
    base, q = random_points(np.uint8, n, 4, 7), random_points(np.uint8, 64, 4, 8)
    g = np.empty((n, R + 1), np.uint32)
    g[:, 0] = R
    g[:, 1:] = rng.integers(0, n, (n, R), dtype=np.uint32)
    idx = P.Index(base, R)
    idx.set_graph(g)
    o = O.search("oracle", base, q, g, 10, 60)
    assert (o["ids"] > n // 2).any()
    b = idx.batch(len(q), 10, 60, seen_slots=4096)
    check(b.run(q, 10, 60), o)
    b.close()
    check(idx.search(q, 10, 60), o)
    idx.close()


def test_every_query_resident_where_narrow_entries_allow_it(lib_built):
    """Few queries of long rows and beams: at 32-bit entries three of them fit on an SM, at 16 bits more; none of 500
    waits for another to finish."""
    n, d, R, nq = 1200, 3000, 32, 500
    base, q = random_points(np.float32, n, d, 1), random_points(np.float32, nq, d, 2)
    g = O.random_graph(n, R, 3, min_deg=24)
    idx = P.Index(base, R)
    idx.set_graph(g)
    b = idx.batch(nq, 10, 600)
    cfg = b.config()
    b.close()
    assert cfg["blocks"] * cfg["warps_per_block"] >= nq, cfg
    check(idx.search(q, 10, 600), O.search("oracle", base, q, g, 10, 600))
    idx.close()
