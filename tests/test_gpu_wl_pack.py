"""Work-list items at the edges of their packed sums: 16-bit rows added two
samples at a time for as many rows as stay below 65536 (`max_value`), rows at
that limit, and 8-bit groups whose uint16 output is stored straight from the
16-bit lanes (row starts of every alignment, a short last word, 257 channels =
the lanes' limit)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("max_value", [65535, 32767, 13107, 255])
@pytest.mark.parametrize("nrows", [1, 5, 33])
def test_sixteen_bit_pack(orc, max_value, nrows):
    import torch

    from sigpyproc3_b200 import _lib
    from sigpyproc3_b200.batch import WorkList, num_variants

    n = 2100
    rng = np.random.default_rng(nrows)
    vals = np.where(rng.random((nrows, n)) < 0.9, max_value,
                    rng.integers(0, max_value + 1, size=(nrows, n))).astype(np.uint16)
    d = rng.integers(0, 120, size=(9, nrows)).astype(np.int32)
    nv = n - int(d.max())
    expect = orc.dmt(np.ascontiguousarray(vals.T.astype(np.float32)), d, nrows, n, nv)
    for v in range(num_variants(16)):
        wl = WorkList(16, v)
        span = wl.span_of(d)
        slot = wl.slot_words(span)
        pitch = ((n + 1) // 2 + slot + wl.T // 2 + 16 + 3) // 4 * 4
        rows = np.zeros((nrows, pitch * 2), dtype=np.uint16)
        rows[:, :n] = vals
        planar = torch.from_numpy(rows.view(np.int32).copy()).cuda()
        dd = torch.from_numpy(d).cuda()
        out = torch.empty((9, nv), dtype=torch.int32, device="cuda")
        wl.add_job(planar_ptr=planar.data_ptr(), pitch_w=pitch, halo=0, nchans=nrows, delays_dev=dd,
                   delays_host=d, out_ptr=out.data_ptr(), out_stride=nv, out_start=0, out_elem=4,
                   nvalid=nv, out_kind=_lib.OUT_I32, max_value=max_value)
        wl.finalize(span)
        wl.launch()
        np.testing.assert_array_equal(out.cpu().numpy(), expect.astype(np.int32), err_msg=f"variant {v}")
        assert int(wl.status[0].item()) == 0


@pytest.mark.parametrize("nchans", [1, 32, 33, 257])
@pytest.mark.parametrize("shift,nvalid", [(0, 1024), (1, 1027), (2, 2049)])
def test_u16_lane_stores(orc, nchans, shift, nvalid):
    import torch

    from sigpyproc3_b200 import _lib
    from sigpyproc3_b200.batch import WorkList, num_variants

    rng = np.random.default_rng(nchans + shift)
    d = rng.integers(0, 50, size=(10, nchans)).astype(np.int32)
    n = nvalid + int(d.max())
    vals = rng.integers(200, 256, size=n * nchans, dtype=np.uint8)
    expect = orc.dmt(vals, d, nchans, n, nvalid)
    raw, dd = torch.from_numpy(vals).cuda(), torch.from_numpy(d).cuda()
    stride = nvalid + 5
    for v in range(num_variants(8)):
        wl = WorkList(8, v)
        span = wl.span_of(d)
        slot = wl.slot_words(span)
        halo, pitch, rpc = wl.layout(nvalid, 0, int(d.max()), slot)
        planar = torch.empty(nchans * rpc * pitch, dtype=torch.int32, device="cuda")
        wl.corner_turn(raw, _lib.BITORDER_BIG, nchans, n, halo, planar, pitch)
        out = torch.full((10 * stride + 8,), 7, dtype=torch.int16, device="cuda")
        wl.add_job(planar_ptr=planar.data_ptr(), pitch_w=pitch, halo=halo, nchans=nchans, delays_dev=dd,
                   delays_host=d, out_ptr=out.data_ptr() + 2 * shift, out_stride=stride, out_start=0,
                   out_elem=2, nvalid=nvalid, out_kind=_lib.OUT_U16)
        wl.finalize(span)
        wl.launch()
        got = out.cpu().numpy().view(np.uint16)[shift:shift + 10 * stride].reshape(10, stride)
        np.testing.assert_array_equal(got[:, :nvalid], np.minimum(expect, 65535), err_msg=f"variant {v}")
        assert (got[:, nvalid:] == 7).all()
