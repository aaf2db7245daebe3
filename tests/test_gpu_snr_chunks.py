"""Boxcar S/N chunks at the edges of their two paths: rows around the chunk
sizes, widths up to the halo limit, integer rows inside the exact 32-bit path,
past its window limit (|sum| * width >= 2^31) and past float32's exact integers
(|x| > 2^24, factor 1: rounding as the float32 input of the oracle), many equal
windows, float32 rows.  S/N within rtol 1e-5 of the float64 oracle, peak index
equal (integer window sums are exact on both sides)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(orc, x, widths, factors):
    import torch

    from sigpyproc3_b200.search import boxcar_snr

    snr, idx = boxcar_snr(torch.from_numpy(x).cuda(), widths=widths, factors=factors)
    esnr, eidx = orc.boxcar_snr(x.astype(np.float32), factors, widths)
    np.testing.assert_allclose(snr.cpu().numpy(), esnr, rtol=1e-5)
    np.testing.assert_array_equal(idx.cpu().numpy(), eidx)


@pytest.mark.parametrize("rows,n", [(1, 300), (3, 1535), (2, 1537), (400, 6143), (399, 6145), (1, 40000)])
def test_integer_rows(orc, rows, n):
    rng = np.random.default_rng(n)
    x = np.rint(rng.normal(3000.0, 40.0, size=(rows, n))).astype(np.int32)
    x[0, n // 2:n // 2 + 20] += 200
    _check(orc, x, [1, 2, 7, 33, 256], [1, 2, 4])


@pytest.mark.parametrize("top", [1 << 20, 1 << 23, 1 << 26, (1 << 31) - 1])
def test_integer_range(orc, top):
    """Values up to `top` of both signs: the 32-bit path ends between the first
    and second for widths of 4096."""
    rng = np.random.default_rng(top)
    x = rng.integers(-top, top, size=(2, 9001), endpoint=True).astype(np.int32)
    _check(orc, x, [1, 16, 4096], [1])


def test_equal_windows(orc):
    """The first of many equal best windows, across chunks."""
    x = np.full((2, 20000), 5, dtype=np.int32)
    x[1, ::2] = 6
    _check(orc, x, list(range(1, 33)), [1, 2, 8])


@pytest.mark.parametrize("n", [1537, 30001])
def test_float_rows(orc, n):
    rng = np.random.default_rng(n)
    x = np.rint(rng.normal(0.0, 500.0, size=(3, n)) * 8).astype(np.float32) / 8  # sums exact in float64
    _check(orc, x, [1, 3, 64, 1000], [1, 2, 3])


@pytest.mark.parametrize("rows,n", [(1, 1536), (2, 5000), (400, 6500)])
@pytest.mark.parametrize("wmax", [255, 256, 257, 512, 1024])
def test_scan_runs(orc, rows, n, wmax):
    """Chunk and halo at the ends of the scan's run lengths (7, 13 and 25 words per
    thread, and past them)."""
    rng = np.random.default_rng(n + wmax)
    x = rng.integers(-2000, 2000, size=(rows, n), endpoint=True).astype(np.int32)
    _check(orc, x, [1, 5, wmax], [1, 2])


@pytest.mark.parametrize("sign", [1, -1])
def test_prefix_sums_wrap(orc, sign):
    """Large samples of one sign: a chunk's prefix sums pass 2^32 several times while
    every window stays below 2^31."""
    rng = np.random.default_rng(22)
    x = (sign * rng.integers((1 << 22) - 900, 1 << 22, size=(2, 13000))).astype(np.int32)
    _check(orc, x, [1, 3, 100, 256], [1, 2])


@pytest.mark.parametrize("rows", [111, 110, 74, 73])
@pytest.mark.parametrize("wmax", [256, 1024])
def test_chunk_rule(orc, rows, wmax):
    """222 chunks of 6144 samples, fewer (3072), 222 of 3072, fewer (1536; 3072 with
    halos of 1024); a last chunk of one sample."""
    rng = np.random.default_rng(rows)
    x = rng.integers(-2000, 2000, size=(rows, 6145), endpoint=True).astype(np.int32)
    _check(orc, x, [1, 5, wmax], [1])
    _check(orc, x.astype(np.float32), [1, 5, wmax], [1])


@pytest.mark.parametrize("rows,n,factors", [(1500, 130, [3]), (1500, 131, [1, 3]), (3, 3073, [1]), (1, 60001, [1, 2])])
@pytest.mark.parametrize("dtype", [np.int32, np.float32])
def test_chunks_per_row(orc, rows, n, factors, dtype):
    """One chunk a row (a lane each in the final pass), three and forty (four lanes, a
    warp); integer rows without a power-of-two factor."""
    rng = np.random.default_rng(rows + n)
    x = rng.integers(-2000, 2000, size=(rows, n), endpoint=True).astype(dtype)
    _check(orc, x, [1, 5, 32], factors)
