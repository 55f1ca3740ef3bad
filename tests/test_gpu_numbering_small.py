"""The Hilbert sort by one block (up to 8,192 items), the radix sort by small
tiles (up to 65,536), and their borders, bit for bit against the oracle: equal
keys, classes mixed, most DOFs without a number; two launches a small call, so
that it does not pay for the passes of a radix sort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def launches(femg, f):
    before = femg.lib().fg_launch_count()
    out = f()
    return out, femg.lib().fg_launch_count() - before


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 2049, 8191, 8192, 8193, 9217, 65535, 65536, 65537])
def test_order(femg, oracle, cuda, dim, n):
    rng = np.random.default_rng(n)
    pts = rng.random((n, dim), dtype=np.float32)
    pts[1::2] = (rng.integers(0, 5, pts[1::2].shape) / 4.0).astype(np.float32)  # long runs of equal keys
    mn, mx = np.full(dim, -1e-6, np.float32), np.full(dim, 1 + 1e-6, np.float32)
    got, count = launches(femg, lambda: femg.hilbert_order(dim, pts, mn, mx))
    assert np.array_equal(got, oracle.hilbert_order(dim, pts, mn, mx))
    assert (count == 2) == (n <= 8192)


@pytest.mark.parametrize("n,numbered", [(1, 1), (3000, 1), (3000, 3000), (40000, 8192), (40000, 8193), (8193, 8192), (70000, 70000)])
def test_numbering(femg, oracle, cuda, n, numbered):
    rng = np.random.default_rng(numbered)
    xyz = (rng.integers(0, 65, (n, 3)) / 64.0).astype(np.float32)
    types = rng.choice([femg.FG_AT_FIXED, femg.FG_AT_LINKED, femg.FG_AT_UNDEFINED, femg.FG_AT_UNKNOWN_GLOBAL], n).astype(np.int32)
    types[rng.choice(n, numbered, replace=False)] = rng.choice([femg.FG_AT_UNKNOWN, femg.FG_AT_UNKNOWN_BUBBLE], numbered)
    bbox = np.array([0.0, 0.0, 0.0, 1.0, 1.0, 1.0])
    before = rng.integers(1, 1 << 40, n).astype(np.uint64)
    got, count = launches(femg, lambda: femg.hilbert_numbering(3, bbox, xyz, types, before))
    want = before.copy()
    first = 1
    for cls in (femg.FG_AT_UNKNOWN, femg.FG_AT_UNKNOWN_BUBBLE):
        ids = np.flatnonzero(types == cls)
        mn, mx = np.float32(bbox[:3]), np.float32(bbox[3:] + 1e-6)
        if len(ids):
            want[ids[oracle.hilbert_order(3, xyz[ids], mn, mx)]] = np.arange(first, first + len(ids), dtype=np.uint64)
        first += len(ids)
    assert np.array_equal(got, want)
    assert (count == 2) == (numbered <= 8192)
