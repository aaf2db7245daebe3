"""Median / IQR selection of the robust S/N: rows split over CTAs (fewer than
148 series) and one CTA per row, at the sizes where the split changes, over
data whose keys span every pass (both signs, wide exponents, subnormals), ties
and constants.  Order statistics are exact, so the z-score differs from the
float64 oracle only by the rounding of the S/N itself.  (Peak indices do not
depend on the z-score and are tested elsewhere.)"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(kind, rng, shape):
    if kind == "sums":
        return np.rint(rng.normal(98304.0, 384.0, size=shape)).astype(np.int32)
    if kind == "wide":  # keys over the whole 32-bit range
        x = rng.normal(0.0, 1.0, size=shape) * 10.0 ** rng.uniform(-42, 6, size=shape)
        return x.astype(np.float32)
    x = np.full(shape, 7.25, dtype=np.float32)  # constant but for a few samples
    x[:, ::97] = -3.0
    return x


@pytest.mark.parametrize("kind", ["sums", "wide", "ties"])
@pytest.mark.parametrize("rows,n", [(1, 4095), (1, 4096), (2, 20011), (3, 70000), (148, 4100)])
def test_split_selection(orc, kind, rows, n):
    import torch

    from sigpyproc3_b200.search import boxcar_snr

    x = _data(kind, np.random.default_rng(rows * n), (rows, n))
    widths, factors = [1, 4, 32], [1] if rows == 148 else [1, 2, 3]
    snr, _ = boxcar_snr(torch.from_numpy(x).cuda(), widths=widths, factors=factors,
                          loc_scale="median_iqr")
    esnr, _ = orc.boxcar_snr(x.astype(np.float32), factors, widths, "median_iqr")
    np.testing.assert_allclose(snr.cpu().numpy(), esnr, rtol=1e-5)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 255, 256, 257, 4095, 4096, 4097])
@pytest.mark.parametrize("kind", ["wide", "ties", "int"])
def test_short_rows(n, kind):
    """The shortest rows, and both sides of the length up to which 256 bins are taken
    (4096): the same values as numpy's sorted row gives."""
    import torch

    from sigpyproc3_b200 import _lib

    rng = np.random.default_rng(n)
    rows = 7
    if kind == "wide":  # every exponent, both signs, zeros
        x = (np.exp(rng.uniform(-80, 80, (rows, n))) * rng.choice([-1, 1], (rows, n))).astype(np.float32)
        x[:, ::5] = 0.0
    elif kind == "ties":
        x = rng.integers(-2, 3, (rows, n)).astype(np.float32)
    else:
        x = rng.integers(-(1 << 31), 1 << 31, (rows, n)).astype(np.int32)
    dev = torch.from_numpy(x).cuda()
    out = torch.zeros((rows, 2), dtype=torch.float64, device="cuda")
    _lib.check(_lib.load().spp_row_loc_scale(
        dev.data_ptr(), _lib.OUT_I32 if kind == "int" else _lib.OUT_F32, rows, n, n, 1, out.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    y = x.astype(np.float32)
    loc = np.median(y, axis=1)
    q25, q75 = np.percentile(y.astype(np.float64), [25, 75], axis=1)
    scale = (q75 - q25) / 1.3489795003921634
    scale = np.where(np.abs(scale) <= 1e-8, 1.0, scale)
    got = out.cpu().numpy()
    # the median of an even row is the float32 mean of two float32 values, either way round
    np.testing.assert_allclose(got[:, 0], loc, rtol=2.0 ** -23, atol=0)
    # two interpolations and a difference in float64; differences of values up to |y|
    np.testing.assert_allclose(got[:, 1], scale, rtol=0, atol=8 * 2.0 ** -52 * (np.abs(q25) + np.abs(q75)).max() + 1e-300)
