"""Blocks whose halo is taken from the previous block on the device, and the
folded cube's means, against the plain forms."""

import numpy as np
import pytest

from sigpyproc3_b200 import ArrayFilterbank, Filterbank, Header, _lib, readers

pytestmark = pytest.mark.gpu


class _Staged(Filterbank):
    """Read through pinned staging buffers."""

    def __init__(self, raw, header):
        self._raw, self.header = raw, header

    def _read_bytes(self, offset, view):
        part = self._raw[offset:offset + view.nbytes]
        view[:part.nbytes] = part
        return part.nbytes


@pytest.mark.parametrize("source", [ArrayFilterbank, _Staged])
@pytest.mark.parametrize("n,gulp,skipback,start", [
    (1000, 300, 100, 0),    # the last block shorter than the gulp
    (1000, 100, 99, 3),     # one new row in a block, to past the end
    (700, 300, 100, 0),     # the last block no longer than the halo
    (1000, 2000, 50, 0),    # one block
    (1000, 250, 0, 0),      # no halo
])
def test_halo_blocks(monkeypatch, source, n, gulp, skipback, start):
    monkeypatch.setattr(readers, "KEEP_HALO_MIN_BYTES", 1)
    raw = np.random.default_rng(n + gulp).integers(0, 256, size=n * 24, dtype=np.uint8)
    fb = source(raw, Header(nchans=24, fch1=1400.0, foff=-1.0, tsamp=1e-3, nbits=8, nsamples=n))
    blocks = {}
    for keep in (False, True):
        blocks[keep] = []
        try:
            for m, ii, blk in fb.stream_blocks(gulp, start, n - start, skipback, keep_halo=keep):
                blocks[keep].append((m, ii, blk.cpu().numpy().copy()))
        except ValueError as e:  # a plan that runs past the data: refused at the same block
            blocks[keep].append((str(e), len(blocks[keep]), np.empty(0)))
    assert [b[:2] for b in blocks[True]] == [b[:2] for b in blocks[False]]
    assert len(blocks[True]) > 0
    for a, b in zip(blocks[True], blocks[False]):
        np.testing.assert_array_equal(a[2], b[2])


@pytest.mark.parametrize("cells", [1, 255, 256, 257, 51200])
@pytest.mark.parametrize("exact", [True, False])
def test_fold_means(cells, exact):
    import torch

    rng = np.random.default_rng(cells)
    count = rng.integers(0, 1 << 30, size=cells).astype(np.int32)
    sums = rng.integers(0, 1 << 50, size=cells)
    count[::7], sums[::7] = 0, 0  # cells that no sample falls into
    f32 = sums.astype(np.float32)
    with np.errstate(divide="ignore", invalid="ignore"):
        ref = f32.copy()
        ref /= count
    dev_sums = torch.from_numpy(sums if exact else f32).cuda()
    dev_count, out = torch.from_numpy(count).cuda(), torch.empty(cells, device="cuda")
    _lib.check(_lib.load().spp_fold_finish(
        None if exact else dev_sums.data_ptr(), dev_sums.data_ptr() if exact else None,
        dev_count.data_ptr(), cells, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    np.testing.assert_array_equal(out.cpu().numpy(), ref)
