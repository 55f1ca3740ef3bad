"""The symbolic phase at the edges of its scans and sort tiles, bit for bit
against the oracle: Hilbert orders with many equal keys, numberings with the
DOF classes mixed, patterns of random element DOF maps; indices out of range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 31, 33, 512, 4095, 4096, 4097, 8193, 100000])
def test_hilbert_order(femg, oracle, cuda, dim, n):
    rng = np.random.default_rng(n)
    pts = (rng.integers(0, 9, (n, dim)) / 8.0).astype(np.float32)  # few places: long runs of equal keys
    pts[::3] = rng.random((len(pts[::3]), dim), dtype=np.float32)
    mn, mx = np.full(dim, -1e-6, np.float32), np.full(dim, 1 + 1e-6, np.float32)
    assert np.array_equal(femg.hilbert_order(dim, pts, mn, mx), oracle.hilbert_order(dim, pts, mn, mx))


@pytest.mark.parametrize("n", [1, 4096, 4097, 50000])
def test_numbering_of_mixed_classes(femg, oracle, cuda, n):
    rng = np.random.default_rng(n)
    xyz = (rng.integers(0, 33, (n, 3)) / 32.0).astype(np.float32)
    types = rng.integers(0, 7, n).astype(np.int32)
    types[0] = femg.FG_AT_UNKNOWN
    bbox = np.array([0.0, 0.0, 0.0, 1.0, 1.0, 1.0])
    before = rng.integers(1, 1 << 40, n).astype(np.uint64)
    got = femg.hilbert_numbering(3, bbox, xyz, types, before)
    want = before.copy()
    first = 1
    for cls in (femg.FG_AT_UNKNOWN, femg.FG_AT_UNKNOWN_BUBBLE):
        ids = np.flatnonzero(types == cls)
        mn, mx = np.float32(bbox[:3]), np.float32(bbox[3:] + 1e-6)
        want[ids[oracle.hilbert_order(3, xyz[ids], mn, mx)]] = np.arange(first, first + len(ids), dtype=np.uint64)
        first += len(ids)
    assert np.array_equal(got, want)


def element_map(femg, n_rows, E, n, seed):
    rng = np.random.default_rng(seed)
    edof = np.stack([rng.choice(n_rows, n, replace=n > n_rows) for _ in range(E)]).astype(np.uint64)
    etype = np.full((E, n), femg.FG_AT_UNKNOWN, np.int32)
    etype[rng.random((E, n)) < 0.1] = femg.FG_AT_FIXED
    return edof, etype


@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("n_rows,E,n", [(1, 1, 1), (7, 3, 4), (2047, 900, 4), (2048, 900, 4), (2049, 700, 10), (5000, 1500, 20)])
def test_pattern_of_a_random_map(femg, oracle, cuda, n_rows, E, n, upper):
    edof, etype = element_map(femg, n_rows, E, n, n_rows + n)
    ai, aj = femg.pattern_build(edof, etype, n_rows, upper=upper)
    oi, oj = oracle.pattern(edof, etype, n_rows, upper=upper)
    assert np.array_equal(ai, oi) and np.array_equal(aj, oj)
    keep = aj[: len(aj) // 2]  # a part keeps the library's buffer
    copy = keep.copy()
    del aj
    femg.pattern_build(edof, etype, n_rows, upper=upper)
    assert np.array_equal(keep, copy)


def test_index_out_of_range(femg, cuda):
    edof, etype = element_map(femg, 100, 50, 4, 1)
    edof[7, 2], etype[7, 2] = 100, femg.FG_AT_UNKNOWN
    with pytest.raises(femg.FgError) as err:
        femg.pattern_build(edof, etype, 100)
    assert err.value.status == femg.FG_ERR_INDEX
    edof, etype = element_map(femg, 100, 50, 4, 1)
    edof[3, 1], etype[3, 1] = 2, femg.FG_AT_LINKED
    with pytest.raises(femg.FgError) as err:
        femg.pattern_build(edof, etype, 100, linked_row=np.array([5, 6], np.uint64))
    assert err.value.status == femg.FG_ERR_INDEX


def test_host_memory_is_given_back(femg, cuda):
    """Columns of 40 MB, built and dropped: the process does not grow."""
    edof, etype = element_map(femg, 20000, 13000, 20, 5)

    def resident():
        with open("/proc/self/statm") as f:
            return int(f.read().split()[1])

    import os
    for _ in range(3):
        femg.pattern_build(edof, etype, 20000)
    before = resident()
    for _ in range(10):
        ai, aj = femg.pattern_build(edof, etype, 20000)
    size = aj.nbytes
    del aj
    assert (resident() - before) * os.sysconf("SC_PAGE_SIZE") < 3 * size
