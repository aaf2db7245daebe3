"""Interleaved bit-plane DM-time kernels (bit i of word w = sample i * M + w).

Each case sits where the layout's arithmetic can go wrong: output lengths that
leave the last of the 32 runs short or the last word tile partly filled, trial
counts around a tile's, channel counts that do not fill a slab of groups (zero
rows), odd channel counts (no pairs), delay ranges many times the block (rows
of more than 32 runs), negative offsets and roll mode.  The sums are integers,
so every variant must equal the oracle's restatement of kernels.dedisperse /
kernels.dmt_block (src/sigpyproc/core/kernels.py:340-362, :1155-1168) exactly.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pack(vals, nbits):
    if nbits == 8:
        return vals
    per = 8 // nbits
    v = vals.reshape(-1, per)
    out = np.zeros(v.shape[0], dtype=np.uint8)
    for k in range(per):
        out |= (v[:, k] << ((8 - (k + 1) * nbits) if nbits > 1 else k)).astype(np.uint8)
    return out


def _run(orc, nbits, d, nchans, nsamps, mode="dedisperse", seed=0, ref_vals=None):
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan

    rng = np.random.default_rng(seed)
    vals = rng.integers(0, 1 << nbits, size=nsamps * nchans, dtype=np.uint8)
    vals[: nsamps * nchans // 3] = (1 << nbits) - 1  # saturated stretch: the top counter levels
    if mode == "roll":
        expect = orc.dmt_roll(vals.astype(np.float32), d, nchans, nsamps).astype(np.int64)
    else:
        expect = orc.dmt(vals, d, nchans, nsamps).astype(np.int64)
    raw = torch.from_numpy(_pack(vals, nbits)).cuda()
    seen = 0
    for dtype in (torch.int32, torch.float32):
        plan = DMTPlan(d, nchans, nsamps, nbits=nbits, bitorder="little" if nbits == 1 else "big",
                       mode=mode, out_dtype=dtype)
        for v in range(plan.num_variants):
            plan.set_variant(v)
            desc = plan.describe()
            if desc["R"] * 32 * desc["TW"] * 32 != desc["T"] or not desc["bit_sliced"]:
                continue
            seen += 1
            out = plan.execute(raw, nsamps, check=True).cpu().numpy()
            np.testing.assert_array_equal(out.astype(np.int64), expect, err_msg=str(desc))
        plan.close()
    return seen


def _delays(nchans, dm, ndm, fch1=1500.0, bw=300.0, ref="fch1"):
    from sigpyproc3_b200.header import Header

    h = Header(nchans=nchans, fch1=fch1, foff=-bw / nchans, tsamp=64e-6)
    return np.atleast_2d(h.get_dmdelays(np.linspace(0.0, dm, ndm), ref)).astype(np.int32)


@pytest.mark.parametrize("nbits", [1, 2, 4, 8])
@pytest.mark.parametrize("nvalid,ndm", [(1, 2), (31 * 256 + 5, 16), (32 * 256, 15), (32 * 264 + 1, 19)])
def test_tile_edges(orc, nbits, nvalid, ndm):
    """Last run short, one full word tile, one word past it; trials 16 = one
    past a 15-trial tile, 19 = one past two of nine."""
    nchans = 64
    d = _delays(nchans, 12.0, ndm)
    assert _run(orc, nbits, d, nchans, nvalid + int(d.max()), seed=nvalid) >= 4


@pytest.mark.parametrize("nbits,nchans", [(1, 8), (1, 24), (2, 36), (4, 38), (8, 7), (8, 21), (8, 34)])
def test_partial_slabs(orc, nbits, nchans):
    """Groups that do not fill the last slab read the zero row."""
    d = _delays(nchans, 15.0, 12)
    assert _run(orc, nbits, d, nchans, 3000 + int(d.max()), seed=nchans) >= 4


@pytest.mark.parametrize("nbits", [1, 2, 4, 8])
def test_rows_longer_than_32_runs(orc, nbits):
    """300 outputs behind delays of 12000 samples: a row is 1500 words of which
    16 carry outputs, so its words span dozens of 32-run blocks."""
    nchans = 16
    d = _delays(nchans, 800.0, 400)
    assert int(d.max()) > 11000
    assert _run(orc, nbits, d, nchans, 300 + int(d.max()), seed=5) >= 2


@pytest.mark.parametrize("nbits", [2, 8])
def test_negative_offsets_and_roll(orc, nbits):
    """Delays about the band centre (rows start before sample 0 and wrap) and
    circular rolls (offsets are -delay)."""
    nchans, ndm = 40, 13
    d = _delays(nchans, 25.0, ndm, ref="fcenter")
    assert d.min() < 0 < d.max()
    assert _run(orc, nbits, d, nchans, 5000, seed=1) >= 4
    d = _delays(nchans, 25.0, ndm)
    assert _run(orc, nbits, d, nchans, 4096, mode="roll", seed=2) >= 4


@pytest.mark.parametrize("nbits,nchans", [(1, 512), (2, 128), (4, 192), (8, 64)])
def test_long_rows_in_whole_sectors(orc, nbits, nchans):
    """The same where raw rows are read 32 bytes at a time: further blocks of 32
    runs are loaded one ahead."""
    d = _delays(nchans, 800.0, 400)
    assert _run(orc, nbits, d, nchans, 300 + int(d.max()), seed=6) >= 2


def test_long_rows_before_another_tile(orc):
    """69 channel groups x 70 word tiles of rows that just pass 32 runs: one CTA
    per group turns two tiles, the first of them with a further block."""
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan

    nchans, nvalid, ndm, step = 4368, 17900, 400, 44
    d = np.repeat(step * np.arange(ndm, dtype=np.int32)[:, None], nchans, axis=1)
    nsamps = nvalid + step * (ndm - 1)
    g = torch.Generator(device="cuda").manual_seed(4)
    raw = torch.randint(0, 256, (nsamps * nchans // 2,), device="cuda", dtype=torch.uint8, generator=g)
    b = raw.view(nsamps, nchans // 2).to(torch.int32)
    s = ((b >> 4) + (b & 15)).sum(1, dtype=torch.int32)
    del b
    expect = s.unfold(0, nvalid, step)
    plan = DMTPlan(d, nchans, nsamps, nbits=4, out_dtype=torch.int32)
    assert plan.describe()["bit_sliced"] and plan.describe()["T"] > 2048  # interleaved
    assert torch.equal(plan.execute(raw, nsamps, check=True), expect)
    plan.close()


@pytest.mark.parametrize("nbits,nchans", [(1, 336), (2, 256), (4, 340), (8, 65)])
def test_short_blocks_of_a_long_plan(orc, nbits, nchans):
    """Blocks far shorter than nsamps_max may run another shape than the plan's:
    the same sums, in the workspace that the plan asks for at that length or at
    its longest, from an aligned address and the next."""
    import torch

    from sigpyproc3_b200.dedisp import DMTPlan

    d = _delays(nchans, 600.0, 130)
    longest = 20000 + int(d.max())
    plan = DMTPlan(d, nchans, longest, nbits=nbits, bitorder="little" if nbits == 1 else "big",
                   out_dtype=torch.int32)
    for nvalid in (1, 257, 1900, 9999, 10001):
        nsamps = nvalid + int(d.max())
        vals = np.random.default_rng(nvalid).integers(0, 1 << nbits, nsamps * nchans, dtype=np.uint8)
        expect = orc.dmt(vals, d, nchans, nsamps).astype(np.int64)
        for shift, ws_samps in ((0, nsamps), (1, longest)):
            raw = torch.from_numpy(np.concatenate([np.zeros(shift, np.uint8), _pack(vals, nbits)])).cuda()[shift:]
            ws = torch.zeros(plan.workspace_bytes(ws_samps), dtype=torch.uint8, device="cuda")
            out = torch.full((plan.ndm, nvalid + 2), -7, dtype=torch.int32, device="cuda")
            got = plan.execute(raw, nsamps, out, out_start=1, ws=ws, check=True).cpu().numpy()
            np.testing.assert_array_equal(got[:, 1:-1].astype(np.int64), expect)
            assert (got[:, 0] == -7).all() and (got[:, -1] == -7).all()
        small = torch.zeros(256, dtype=torch.uint8, device="cuda")
        with pytest.raises(ValueError):
            plan.execute(raw, nsamps, out, out_start=1, ws=small)
    plan.close()


def _shapes(nbits, d, nchans, nsamps, mode="dedisperse"):
    """Whether channel and channel-pair rows are offered: interleaved tiles are of 3, 7,
    9, 11 or 15 trials, the others' of 1, 4 or 8."""
    from sigpyproc3_b200.dedisp import DMTPlan

    plan = DMTPlan(d, nchans, nsamps, nbits=nbits, mode=mode, bitorder="little" if nbits == 1 else "big")
    kinds = set()
    for v in range(plan.num_variants):
        plan.set_variant(v)
        if plan.describe()["DW"] not in (1, 4, 8):
            kinds.add(plan.describe()["paired"])
    plan.close()
    return kinds


@pytest.mark.parametrize("nbits,nchans,dm,ndm,nvalid,mode,ref", [
    (1, 64, 12.0, 16, 7941, "dedisperse", "fch1"), (2, 64, 12.0, 2, 1, "dedisperse", "fch1"),
    (4, 64, 12.0, 15, 8192, "dedisperse", "fch1"), (8, 64, 12.0, 19, 8449, "dedisperse", "fch1"),
    (1, 8, 15.0, 12, 3000, "dedisperse", "fch1"), (2, 36, 15.0, 12, 3000, "dedisperse", "fch1"),
    (4, 38, 15.0, 12, 3000, "dedisperse", "fch1"), (8, 7, 15.0, 12, 3000, "dedisperse", "fch1"),
    (8, 34, 15.0, 12, 3000, "dedisperse", "fch1"), (1, 16, 800.0, 400, 300, "dedisperse", "fch1"),
    (2, 16, 800.0, 400, 300, "dedisperse", "fch1"), (4, 16, 800.0, 400, 300, "dedisperse", "fch1"),
    (8, 16, 800.0, 400, 300, "dedisperse", "fch1"), (2, 40, 25.0, 13, 4096, "roll", "fch1"),
    (8, 40, 25.0, 13, 4096, "roll", "fch1"), (2, 40, 25.0, 13, 4500, "dedisperse", "fcenter"),
    (8, 40, 25.0, 13, 4500, "dedisperse", "fcenter")])
def test_tables_are_offered(nbits, nchans, dm, ndm, nvalid, mode, ref):
    """The tables above reach the interleaved kernels, those of 64 channels (few distinct
    offsets within a pair) the pairs' too."""
    d = _delays(nchans, dm, ndm, ref=ref)
    nsamps = nvalid + (0 if mode == "roll" else int(np.abs(d).max()))
    kinds = _shapes(nbits, d, nchans, nsamps, mode)
    assert 0 in kinds
    if nchans == 64:
        assert (1 in kinds) == (nbits > 1)


@pytest.mark.parametrize("nbits,nchans,mode", [(2, 36, "dedisperse"), (2, 68, "roll"), (4, 38, "dedisperse"),
                                               (8, 34, "roll"), (8, 66, "dedisperse")])
def test_partial_slabs_of_pairs(orc, nbits, nchans, mode):
    """Pairs that do not fill the last slab read the zero row of pair planes."""
    d = _delays(nchans, 2.0, 25)
    nsamps = 3000 + int(d.max())
    assert _shapes(nbits, d, nchans, nsamps, mode) == {0, 1}
    assert _run(orc, nbits, d, nchans, nsamps, mode=mode, seed=nchans) >= 4
