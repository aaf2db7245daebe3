"""Float32 DM-time kernels whose last slab is short: the consumers take four
channels' offsets at a time and the remainder one by one.  Sums are float64 in
channel order in every path, so each output equals the oracle's bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nchans", [3, 18, 37])
@pytest.mark.parametrize("finite", [True, False])
def test_short_last_slab(orc, nchans, finite):
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan
    from sigpyproc3_b200.header import Header

    h = Header(nchans=nchans, fch1=1500.0, foff=-300.0 / nchans, tsamp=64e-6)
    d = np.atleast_2d(h.get_dmdelays(np.linspace(0.0, 20.0, 11))).astype(np.int32)
    nvalid = 1025  # one sample past a tile of 1024
    nsamps = nvalid + int(d.max())
    rng = np.random.default_rng(nchans)
    x = rng.normal(0.0, 1.0, size=(nsamps, nchans)).astype(np.float32)
    x[::7, 0] = 0.0
    x[::11, nchans - 1] = np.float32(1e-41)  # subnormal
    x[::13, nchans // 2] = np.float32(-3e38)
    if not finite:  # a sample no trial reads: the conversion-unit path, same outputs
        d[:, 0] = 0
        x[nsamps - 1, 0] = np.nan
    ref = orc.dmt(x.ravel(), d, nchans, nsamps, nvalid)
    plan = DMTPlan(d, nchans, nsamps, nbits=32)
    raw = torch.from_numpy(x.ravel()).cuda()
    assert plan.num_variants >= 6
    for v in range(plan.num_variants):
        plan.set_variant(v)
        out = plan.execute(raw, nsamps, check=True).cpu().numpy()
        np.testing.assert_array_equal(out, ref, err_msg=str(plan.describe()))
    plan.close()
