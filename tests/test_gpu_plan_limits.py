"""Tables and block lengths at the edge of what a DM plan takes.

The widest trial spreads fit one kernel shape only, and the longest blocks have
more time tiles of the shorter shapes than a grid's y extent (65535) holds: a
plan must offer the one and start from a shape that runs the other.  Sums as in
kernels.dmt_block (src/sigpyproc/core/kernels.py:1155-1168).
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_widest_1bit_spread(orc):
    """Trials 2500 samples apart: 17500 over a tile of eight."""
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan

    nchans, ndm, nvalid = 64, 8, 3001
    rng = np.random.default_rng(3)
    d = (2500 * np.arange(ndm)[:, None] + rng.integers(0, 40, nchans)[None, :]).astype(np.int32)
    nsamps = nvalid + int(d.max())
    bits = rng.integers(0, 2, nsamps * nchans, dtype=np.uint8)
    raw = torch.from_numpy(np.packbits(bits, bitorder="little")).cuda()
    expect = orc.dmt(bits, d, nchans, nsamps).astype(np.int64)
    plan = DMTPlan(d, nchans, nsamps, nbits=1, bitorder="little", out_dtype=torch.int32)
    out = plan.execute(raw, nsamps, check=True).cpu().numpy()
    np.testing.assert_array_equal(out.astype(np.int64), expect)
    plan.close()


@pytest.mark.parametrize("nbits,nchans,tile,step", [(32, 2, 256, 5), (8, 3, 1024, 2000)])
def test_more_tiles_than_a_grid(nbits, nchans, tile, step):
    """One output more than 65535 tiles of the shape that short blocks start from."""
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan

    nvalid = 65535 * tile + 1
    d = np.array([[0] * nchans, [step] * nchans], dtype=np.int32)
    nsamps = nvalid + step
    if nbits == 32:
        g = torch.Generator(device="cuda").manual_seed(1)
        raw = torch.randn(nsamps * nchans, device="cuda", generator=g)
        s = raw.view(nsamps, nchans).double().sum(1).float()
        dtype = torch.float32
    else:
        g = torch.Generator(device="cuda").manual_seed(2)
        raw = torch.randint(0, 256, (nsamps * nchans,), device="cuda", dtype=torch.uint8, generator=g)
        s = raw.view(nsamps, nchans).sum(1, dtype=torch.int32)
        dtype = torch.int32
    plan = DMTPlan(d, nchans, nsamps, nbits=nbits, out_dtype=dtype)
    out = plan.execute(raw, nsamps, check=True)
    assert torch.equal(out[0], s[:nvalid]) and torch.equal(out[1], s[step:])
    plan.close()


def test_no_memory_for_staging_tables(orc):
    """A grid whose staging tables (some 90 MB) do not fit what the delay table (66 MB)
    leaves of the device memory."""
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan

    nchans, ndm, nvalid = 2048, 8000, 4096
    d = (np.arange(ndm)[:, None] * np.arange(nchans)[None, :] // (1 << 19)).astype(np.int32)
    nsamps = nvalid + int(d.max())
    rng = np.random.default_rng(8)
    vals = rng.integers(0, 256, nsamps * nchans, dtype=np.uint8)
    rows = np.concatenate([np.arange(0, ndm, 997), [ndm - 1]])
    expect = orc.dmt(vals, np.ascontiguousarray(d[rows]), nchans, nsamps).astype(np.int64)
    raw = torch.from_numpy(vals).cuda()
    out = torch.zeros((ndm, nvalid), dtype=torch.int32, device="cuda")
    ws = torch.zeros(256 << 20, dtype=torch.uint8, device="cuda")
    torch.cuda.empty_cache()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (100 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 130 << 20
        plan = DMTPlan(d, nchans, nsamps, nbits=8, out_dtype=torch.int32)
    finally:
        del rest
        torch.cuda.empty_cache()
    plan.execute(raw, nsamps, out, ws=ws, check=True)
    np.testing.assert_array_equal(out.cpu().numpy()[rows].astype(np.int64), expect)
    plan.close()
