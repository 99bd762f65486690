"""The radix sort at the edges of its tiles of 4,096 records (below 2^18
records) and 8,192 (one record more and fewer, a last tile of one, more tiles than a look-back round takes), with
keys all equal, in order, in reverse and random, odd bit counts (an odd number
of passes copies the result back), through both entry points: the stable
order, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def keys(kind, n, bits, rng):
    if kind == "equal":
        return np.full(n, 7, dtype=np.uint32)
    if kind == "reverse":
        return np.arange(n, 0, -1, dtype=np.uint64).astype(np.uint32)
    if kind == "few":
        return rng.integers(0, 3, n).astype(np.uint32) << np.uint32(bits - 3)
    return rng.integers(0, 2 ** bits, n, dtype=np.uint64).astype(np.uint32)


@pytest.mark.parametrize("n", [2, 33, 4095, 4096, 4097, 17 * 4096 + 1, 2 ** 18 - 1, 2 ** 18, 40 * 8192 + 1, 2_500_003])
@pytest.mark.parametrize("kind,bits", [("random", 32), ("random", 24), ("few", 13), ("equal", 8), ("reverse", 32)])
def test_sort_tile_edges(dem, cuda, n, kind, bits):
    rng = np.random.default_rng(n + bits)
    k = keys(kind, n, bits, rng)
    kv = np.stack([k, np.arange(n, dtype=np.uint32)], 1)
    digits = 8 * ((bits + 7) // 8)
    order = np.argsort(k & np.uint32(2 ** digits - 1) if digits < 32 else k, kind="stable")
    for call in (dem.compat.RadixSort, dem.compat.RadixSortNoAlloc):
        d0 = cuda.from_numpy(kv.view(np.int32).copy()).cuda()
        d1 = cuda.zeros_like(d0)
        call(d0, d1, n, bits)
        cuda.cuda.synchronize()
        np.testing.assert_array_equal(d0.cpu().numpy().view(np.uint32), kv[order])
