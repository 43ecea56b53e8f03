"""The tile search's shared-memory layout over every kind of accepted shape (thin tiles beside long rows above all),
and the search itself on thin tiles: the re-ranked distances are exactly Point::distance."""
import os
import subprocess

import numpy as np
import pytest

import parlayann_b200 as P
from conftest import random_points
from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_regions_hold_what_is_written(tmp_path):
    exe = str(tmp_path / "tile_layout_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "parlayann_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tile_layout_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1, 17, 512, 1000, 4096])
@pytest.mark.parametrize("R", [1, 2, 3, 8])
@pytest.mark.parametrize("precision", [P.PREC_BF16, P.PREC_FP8])
def test_thin_tiles(d, R, precision, lib_built):
    n, nq, beam = 600, 40, 20
    base = random_points(np.float32, n, d, d)
    q = random_points(np.float32, nq, d, d + 1)
    for metric in (P.L2, P.MIPS):
        idx = P.Index(base, R, metric)
        idx.set_graph(O.random_graph(n, R, d + 2, min_deg=R))
        idx.set_precision(precision)
        for parents in (1, 2, 4):
            for limit in sorted({1, min(2, R), R}):
                r = idx.search(q, 10, beam, degree_limit=limit, precision=precision, parents=parents, allow_short=True)
                live = r.ids != 0xFFFFFFFF
                assert live[:, 0].all()
                ids = np.where(live, r.ids, r.ids[:, :1])
                want = P.point_distances(q, base, ids, metric)
                np.testing.assert_array_equal(r.dists[live].view(np.uint32), want[live].view(np.uint32))
        idx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("d", [1, 7, 9, 15, 17, 33, 95])
@pytest.mark.parametrize("precision", [P.PREC_BF16, P.PREC_FP8])
def test_padded_dimensions_add_nothing(d, precision, lib_built):
    """Rows of any length score as the same rows with zeros up to a whole number of 16-byte chunks."""
    n, R = 3000, 24
    base, q = random_points(np.float32, n, d, d), random_points(np.float32, 200, d, d + 1)
    g = O.random_graph(n, R, d + 2, min_deg=8)
    pad = ((0, 0), (0, -d % 16))
    for metric in (P.L2, P.MIPS):
        got = []
        for b, x in ((base, q), (np.pad(base, pad), np.pad(q, pad))):
            idx = P.Index(b, R, metric)
            idx.set_graph(g)
            idx.set_precision(precision)
            got.append(idx.search(x, 10, 40, precision=precision, parents=3))
            idx.close()
        for f in ("ids", "dists", "visited", "cmps"):
            np.testing.assert_array_equal(getattr(got[0], f), getattr(got[1], f))
