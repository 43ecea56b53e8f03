"""Exact top-k on the tensor cores (csrc/gt_tensor.cu) against the plain FP64 / integer kernel, which answers the
same call with PANN_GT_PLAIN set: ids and distances equal bit for bit (both are exact, ties by id)."""
import ctypes
import threading

import numpy as np
import pytest

from conftest import has_gpu, random_points

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not has_gpu(), reason="needs a GPU")]

import parlayann_b200 as P  # noqa: E402

# points, queries, dimensions, k: ends of the 128-row tiles, of the 64..256-query blocks, of K's 32-byte steps and
# 64-byte chunks, of the candidate buffers (64, 256), rows too long for more than 64 queries a block, more k than points
SHAPES = [(1, 1, 1, 1), (50, 3, 7, 60), (127, 64, 16, 5), (129, 65, 33, 64), (4096, 256, 64, 65), (4097, 257, 65, 10),
          (20000, 300, 100, 256), (9000, 20, 700, 20), (3000, 10, 40, 257)]


def both(base, q, k, metric, monkeypatch):
    idx = P.Index(base, 4, metric)
    got = idx.groundtruth(q, k)
    monkeypatch.setenv("PANN_GT_PLAIN", "1")
    plain = idx.groundtruth(q, k)
    monkeypatch.delenv("PANN_GT_PLAIN")
    np.testing.assert_array_equal(got[0], plain[0])
    np.testing.assert_array_equal(got[1], plain[1])
    idx.close()
    return got


@pytest.mark.parametrize("metric", [P.L2, P.MIPS])
@pytest.mark.parametrize("dtype", [np.uint8, np.int8, np.float32])
@pytest.mark.parametrize("n,nq,d,k", SHAPES)
def test_equals_plain_kernel(n, nq, d, k, dtype, metric, lib_built, monkeypatch):
    both(random_points(dtype, n, d, n + d), random_points(dtype, nq, d, nq + d), k, metric, monkeypatch)


@pytest.mark.parametrize("dtype", [np.uint8, np.int8])
def test_equal_distances_by_id(dtype, lib_built, monkeypatch):
    """Few distinct 8-bit points: thousands of equal scores across tiles and slices."""
    rng = np.random.default_rng(3)
    both(rng.integers(0, 2, (30000, 5)).astype(dtype), rng.integers(0, 2, (200, 5)).astype(dtype), 70, P.L2, monkeypatch)


def test_float_scales(lib_built, monkeypatch):
    """Values far from 1, one query far from the others, a NaN point (never an answer)."""
    rng = np.random.default_rng(4)
    base = rng.standard_normal((6000, 48)).astype(np.float32)
    q = rng.standard_normal((40, 48)).astype(np.float32)
    both(base * np.float32(1e8), q * np.float32(1e8), 10, P.L2, monkeypatch)
    both(base * np.float32(1e-4), q * np.float32(1e-4), 10, P.MIPS, monkeypatch)
    far = q.copy()
    far[7] *= np.float32(1e9)
    both(base, far, 10, P.L2, monkeypatch)
    nan = np.concatenate([base, base[:1]])
    nan[-1, 5] = np.nan
    idx = P.Index(nan, 4)
    ids, dd = idx.groundtruth(q, 10)
    idx.close()
    want = both(base, q, 10, P.L2, monkeypatch)
    np.testing.assert_array_equal(ids, want[0])
    np.testing.assert_array_equal(dd, want[1])


def test_beside_searches_and_other_threads(lib_built):
    """Groundtruth calls of two threads beside device searches of padded rows on a third stream, all on one index."""
    import torch

    from oracle import oracle as O

    n, d, R, nq, k, L = 20000, 7, 24, 3000, 10, 60
    base, q = random_points(np.float32, n, d, 1), random_points(np.float32, nq, d, 2)
    idx = P.Index(base, R)
    idx.set_graph(O.random_graph(n, R, 3, min_deg=16))
    dq = torch.from_numpy(q).cuda()
    want = idx.search(q, k, L)
    parts = [(q[:700], 20), (q[700:1900], 5)]
    alone = [idx.groundtruth(*p) for p in parts]
    got = [[], []]

    def gt(i):
        for _ in range(12):
            got[i].append(idx.groundtruth(*parts[i]))

    ids = [torch.zeros((nq, k), dtype=torch.int32, device="cuda") for _ in range(12)]
    dists = [torch.zeros((nq, k), dtype=torch.float32, device="cuda") for _ in range(12)]
    flags = torch.zeros(nq, dtype=torch.int32, device="cuda")
    stream, qp, start = torch.cuda.Stream(), P.QueryParams(k, L, n, R, 0.125), np.zeros(1, np.uint32)
    torch.cuda.synchronize()
    threads = [threading.Thread(target=gt, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for i in range(12):
        rc = P.lib().pann_search_device(idx.handle, dq.data_ptr(), nq, ctypes.byref(qp), start.ctypes.data, 1,
                                        ids[i].data_ptr(), dists[i].data_ptr(), None, None, flags.data_ptr(),
                                        stream.cuda_stream)
        assert rc == 0
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(12):
        np.testing.assert_array_equal(ids[i].cpu().numpy().view(np.uint32), want.ids)
        np.testing.assert_array_equal(dists[i].cpu().numpy(), want.dists)
        for part in range(2):
            np.testing.assert_array_equal(got[part][i][0], alone[part][0])
            np.testing.assert_array_equal(got[part][i][1], alone[part][1])
    idx.close()


@pytest.mark.parametrize("metric", [P.L2, P.MIPS])
def test_half_of_the_queries_left_to_the_plain_kernel(metric, lib_built, monkeypatch):
    """Every second query lies near 3,000 copies of one point, whose equal scores its margin test cannot tell apart."""
    rng = np.random.default_rng(11)
    base = rng.standard_normal((20000, 24)).astype(np.float32)
    base[9000:12000] = 3 * base[5]
    q = rng.standard_normal((201, 24)).astype(np.float32)
    q[::2] = 3 * base[5] + np.float32(1e-3) * q[::2]
    both(base, q, 15, metric, monkeypatch)


def test_plain_kernel_works_in_place(lib_built):
    """k above 256 goes to the plain kernel whole. 4,000 queries on 300 points take it about 3 ms; a copy of each
    query's row, ids and distances (12,000 copies) would take at least 12 ms at 1 us a copy."""
    import time

    idx = P.Index(random_points(np.float32, 300, 16, 1), 4)
    q = random_points(np.float32, 4000, 16, 2)
    times = []
    for _ in range(6):
        t = time.perf_counter()
        idx.groundtruth(q, 257)
        times.append(time.perf_counter() - t)
    idx.close()
    assert min(times) < 12e-3, times


@pytest.mark.parametrize("metric", [P.L2, P.MIPS])
@pytest.mark.parametrize("d,offset", [(1, 1000), (33, 40), (96, 3000)])
def test_far_from_the_origin(d, offset, metric, lib_built, monkeypatch):
    """Points around a centre many spreads from the origin, some values not finite."""
    base = random_points(np.float32, 5000, d, d) + np.float32(offset)
    q = random_points(np.float32, 130, d, d + 1) + np.float32(offset)
    both(base, q, 10, metric, monkeypatch)
    base[::500, d // 2] = np.nan
    both(base[1:], q, 10, metric, monkeypatch)


def test_far_from_the_origin_takes_the_same_path(lib_built):
    """A common offset does not send queries to the plain kernel, which takes some 45 times as long for these sizes."""
    import time

    base, q = random_points(np.float32, 100_000, 32, 1), random_points(np.float32, 1000, 32, 2)
    best = []
    for offset in (0, 64):
        idx = P.Index(base + np.float32(offset), 4)
        times = []
        for _ in range(6):
            t = time.perf_counter()
            idx.groundtruth(q + np.float32(offset), 20)
            times.append(time.perf_counter() - t)
        best.append(min(times))
        idx.close()
    assert best[1] < 5 * best[0], best


@pytest.mark.parametrize("metric", [P.L2, P.MIPS])
def test_values_that_half_precision_splits_worst(metric, lib_built, monkeypatch):
    """Values 1 + j 2^-23 with odd j in (2048, 4096): the rest after the upper half has 13 bits, the lower half holds 11,
    so both halves miss the value by a whole float32 ulp. Random signs keep the mean at the origin; the distances of the
    points that share a query's signs differ in their last bits."""
    rng = np.random.default_rng(12)
    d = 40

    def rows(sign):
        j = 2 * rng.integers(1024, 2048, sign.shape) + 1
        return (sign * (1 + j * 2.0 ** -23)).astype(np.float32)

    sign = rng.choice([-1.0, 1.0], (100, d))
    both(rows(np.repeat(sign, 30, 0)), rows(sign), 20, metric, monkeypatch)


@pytest.mark.parametrize("dtype,d,k", [(np.float32, 256, 100), (np.uint8, 96, 200)])
def test_survivors_of_many_slices(dtype, d, k, lib_built, monkeypatch):
    """Few queries on many points are split into slices whose survivors number more than slices x C; they all fit, so
    the call does not fall back to the plain kernel (measured 25 to 300 times as long for these sizes)."""
    import time

    base, q = random_points(dtype, 300_000, d, 1), random_points(dtype, 100, d, 2)
    idx = P.Index(base, 4)
    took, answers = [], []
    for plain in ("", "", "", "1"):
        if plain:
            monkeypatch.setenv("PANN_GT_PLAIN", plain)
        t = time.perf_counter()
        answers.append(idx.groundtruth(q, k))
        took.append(time.perf_counter() - t)
    monkeypatch.delenv("PANN_GT_PLAIN")
    idx.close()
    for ids, dd in answers[:3]:
        np.testing.assert_array_equal(ids, answers[3][0])
        np.testing.assert_array_equal(dd, answers[3][1])
    assert max(took[1:3]) < took[3] / 5, took


@pytest.mark.parametrize("metric", [P.L2, P.MIPS])
@pytest.mark.parametrize("n,nq,d,k", [(100_000, 20, 700, 20), (2000, 30_001, 8, 256)], ids=["segments", "chunks"])
def test_more_than_one_segment_or_chunk(n, nq, d, k, metric, lib_built, monkeypatch):
    """Point images past 128 MB (three segments, the candidate buffers carried over) and candidate buffers past 128 MB
    (the queries in chunks)."""
    both(random_points(np.float32, n, d, 1), random_points(np.float32, nq, d, 2), k, metric, monkeypatch)
