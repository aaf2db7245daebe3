"""Where a DM plan's working words lie behind its delay table.

The range passes of the interleaved kernels store pairs of 32-bit words there,
so the offset must be a multiple of 8 bytes whatever the table's size: an odd
channel count (8-bit rows only) times an odd trial count is an odd number of
words.  The plans themselves must equal the oracle's restatement of
kernels.dmt_block (src/sigpyproc/core/kernels.py:1155-1168) exactly.
"""

import ctypes

import numpy as np
import pytest


def _layout(nbits, nchans, ndm):
    from sigpyproc3_b200 import _lib

    off, total = ctypes.c_int64(), ctypes.c_int64()
    rc = _lib.load().spp_dmt_plan_layout(nbits, nchans, ndm, ctypes.byref(off), ctypes.byref(total))
    assert rc == _lib.SPP_OK
    return off.value, total.value


@pytest.mark.parametrize("nchans", [7, 8, 33, 34, 1024])
@pytest.mark.parametrize("ndm", [2, 3, 12, 13])
def test_work_words_aligned(nchans, ndm):
    off, total = _layout(8, nchans, ndm)
    assert off % 256 == 0 and off >= 4 * nchans * ndm
    # channel ranges are pairs of words; rows and scratch of up to 12 nchans pair rows
    assert total - off >= 4 * (2 * nchans + 2 * 12 * nchans)


def test_plans_without_row_tables():
    assert _layout(32, 33, 13) == (4 * 33 * 13, 4 * 33 * 13)
    assert _layout(8, 33, 1) == (4 * 33, 4 * 33)


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["dedisperse", "roll"])
@pytest.mark.parametrize("nchans,ndm", [(7, 3), (7, 13), (33, 3), (33, 13)])
def test_odd_channels_and_trials(orc, nchans, ndm, mode):
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan
    from sigpyproc3_b200.header import Header

    h = Header(nchans=nchans, fch1=1500.0, foff=-300.0 / nchans, tsamp=64e-6)
    d = np.atleast_2d(h.get_dmdelays(np.linspace(0.0, 20.0, ndm))).astype(np.int32)
    nsamps = 4001
    vals = np.random.default_rng(nchans + ndm).integers(0, 256, nsamps * nchans, dtype=np.uint8)
    if mode == "roll":
        expect = orc.dmt_roll(vals.astype(np.float32), d, nchans, nsamps).astype(np.int64)
    else:
        expect = orc.dmt(vals, d, nchans, nsamps).astype(np.int64)
    raw = torch.from_numpy(vals).cuda()
    plan = DMTPlan(d, nchans, nsamps, nbits=8, mode=mode, out_dtype=torch.int32)
    for v in range(plan.num_variants):
        plan.set_variant(v)
        out = plan.execute(raw, nsamps, check=True).cpu().numpy()
        np.testing.assert_array_equal(out.astype(np.int64), expect, err_msg=str(plan.describe()))
    plan.close()
