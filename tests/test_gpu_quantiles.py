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
