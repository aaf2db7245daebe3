"""Streaming single-DM kernel (spp_dedisperse_host) at its edges: row pitches of
every alignment, channel counts that leave a slab short, output counts around a
CTA's, more channels than one parameter size, negative delays (rows wrap at both
ends), blocks at an odd address, and spreads it refuses.  Integer sums equal the
oracle exactly; float32 sums are float64 in channel order, so they do too."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pack(vals, nbits):
    if nbits >= 8:
        return vals
    per = 8 // nbits
    v = vals.reshape(-1, per)
    out = np.zeros(v.shape[0], dtype=np.uint8)
    for k in range(per):
        out |= (v[:, k] << ((8 - (k + 1) * nbits) if nbits > 1 else k)).astype(np.uint8)
    return out


def _stream(raw, nbits, d, nchans, nsamps, nout):
    import torch

    from sigpyproc3_b200 import _lib

    out = torch.full((nout + 3,), -5.0, dtype=torch.float32, device="cuda")
    rc = _lib.load().spp_dedisperse_host(raw.data_ptr(), nbits, 1 if nbits == 1 else 0, nchans, nsamps,
                                         d.ctypes.data, out.data_ptr(), out.numel(), 2,
                                         torch.cuda.current_stream().cuda_stream)
    return rc, out.cpu().numpy()


@pytest.mark.parametrize("nbits,nchans", [(8, 4), (8, 31), (8, 336), (8, 1026), (8, 3000), (4, 38),
                                          (4, 1024), (2, 1020), (2, 4096), (1, 24), (1, 2048),
                                          (32, 5), (32, 336), (32, 1030)])
@pytest.mark.parametrize("nvalid,shift", [(1, 0), (129, 1), (5000, 3)])
def test_widths_and_alignments(orc, nbits, nchans, nvalid, shift):
    import torch

    rng = np.random.default_rng(nchans + nvalid)
    d = np.sort(rng.integers(0, 40 + 2 * nchans // 16, size=nchans)).astype(np.int32)
    nsamps = nvalid + int(d.max())
    if nbits == 32:
        x = rng.normal(0.0, 1.0, size=nsamps * nchans).astype(np.float32)
        raw = torch.from_numpy(x).cuda()
    else:
        x = rng.integers(0, 1 << nbits, size=nsamps * nchans, dtype=np.uint8)
        p = _pack(x, nbits)  # `shift` bytes into an allocation: any address
        raw = torch.from_numpy(np.concatenate([np.full(shift, 255, np.uint8), p])).cuda()[shift:]
    rc, out = _stream(raw, nbits, d, nchans, nsamps, nvalid)
    assert rc == 0
    np.testing.assert_array_equal(out[2:-1], orc.dedisperse(x, d, nchans, nsamps)[:nvalid])
    assert out[0] == out[1] == out[-1] == -5.0


@pytest.mark.parametrize("nbits", [8, 2, 32])
def test_negative_delays_wrap(orc, nbits):
    import torch

    nchans, nsamps = 160, 3000
    d = np.linspace(-300, 450, nchans).astype(np.int32)
    rng = np.random.default_rng(nbits)
    if nbits == 32:
        x = rng.normal(0.0, 1.0, size=nsamps * nchans).astype(np.float32)
    else:
        x = rng.integers(0, 1 << nbits, size=nsamps * nchans, dtype=np.uint8)
    rc, out = _stream(torch.from_numpy(_pack(x, nbits)).cuda(), nbits, d, nchans, nsamps, nsamps - 450)
    assert rc == 0
    np.testing.assert_array_equal(out[2:-1], orc.dedisperse(x, d, nchans, nsamps)[: nsamps - 450])


def test_wide_spreads_fall_back(orc):
    """One channel 9000 samples later than the rest of its slab: refused here,
    taken by dedisperse_block through the planar path."""
    import torch

    from sigpyproc3_b200 import _lib
    from sigpyproc3_b200.dedisp import dedisperse_block

    nchans, nsamps = 33, 12000
    d = np.zeros(nchans, dtype=np.int32)
    d[7] = 9000
    x = np.random.default_rng(3).integers(0, 256, size=nsamps * nchans, dtype=np.uint8)
    raw = torch.from_numpy(x).cuda()
    rc, _ = _stream(raw, 8, d, nchans, nsamps, nsamps - 9000)
    assert rc == _lib.SPP_ERR_UNSUPPORTED
    out = torch.zeros(nsamps - 9000, dtype=torch.float32, device="cuda")
    assert dedisperse_block(raw, d, nchans, nsamps, out) == nsamps - 9000
    np.testing.assert_array_equal(out.cpu().numpy(), orc.dedisperse(x, d, nchans, nsamps)[:3000])


@pytest.mark.parametrize("nbits", [8, 2])
def test_unknown_bit_order(nbits):
    """A block that writes nothing returns 0 whatever the order; a packed one
    that does is refused."""
    import torch

    from sigpyproc3_b200.dedisp import dedisperse_block

    d = np.array([0, 1, 2, 3], dtype=np.int32)
    raw = torch.zeros(64, dtype=torch.uint8, device="cuda")
    out = torch.zeros(8, dtype=torch.float32, device="cuda")
    assert dedisperse_block(raw, d, 4, 3, out, nbits=nbits, bitorder="x") == 0
    if nbits < 8:
        with pytest.raises(ValueError):
            dedisperse_block(raw, d, 4, 8, out, nbits=nbits, bitorder="x")


@pytest.mark.parametrize("nbits,nchans,nvalid,step,shift", [(32, 2048, 4147, 0, 0), (8, 512, 3001, 100, 4),
                                                            (8, 336, 20000, 1, 4), (2, 64, 20000, 60, 4)])
def test_blocks_left_to_two_passes(orc, nbits, nchans, nvalid, step, shift):
    """Short float32 blocks, delays `step` apart per channel (wide slabs) and
    8-bit rows aligned to 4 bytes: nothing is launched, and dedisperse_block
    takes them through spp_dedisperse."""
    import torch

    from sigpyproc3_b200 import _lib
    from sigpyproc3_b200.dedisp import dedisperse_block

    rng = np.random.default_rng(nchans)
    d = (step * np.arange(nchans)).astype(np.int32)
    nsamps = nvalid + int(d.max())
    if nbits == 32:
        x = rng.normal(0.0, 1.0, size=nsamps * nchans).astype(np.float32)
        raw = torch.from_numpy(x).cuda()
    else:
        x = rng.integers(0, 1 << nbits, size=nsamps * nchans, dtype=np.uint8)
        raw = torch.from_numpy(np.concatenate([np.zeros(shift, np.uint8), _pack(x, nbits)])).cuda()[shift:]
    out = torch.full((nvalid,), -5.0, dtype=torch.float32, device="cuda")
    args = (raw.data_ptr(), nbits, 0, nchans, nsamps, d.ctypes.data, _lib.ACC_F64, out.data_ptr(),
            out.numel(), 0, torch.cuda.current_stream().cuda_stream)
    assert _lib.load().spp_dedisperse_block(*args) == _lib.SPP_ERR_UNSUPPORTED
    assert bool((out == -5.0).all())
    assert dedisperse_block(raw, d, nchans, nsamps, out, nbits=nbits) == nvalid
    np.testing.assert_array_equal(out.cpu().numpy(), orc.dedisperse(x, d, nchans, nsamps))
