"""Scratch of the boxcar S/N calls: reserved for the longest series and the most
rows, it serves every smaller call, across the lengths and counts where the chunks
get shorter (1184 of a length) and the selection is split over CTAs (148 series)."""

import numpy as np
import pytest


@pytest.mark.parametrize("robust", [False, True])
def test_scratch_monotone(robust):
    from sigpyproc3_b200 import _lib

    lib = _lib.load()
    size = lib.spp_boxcar_snr_robust_workspace_bytes if robust else lib.spp_boxcar_snr_workspace_bytes
    for rows in (1, 7, 147, 148, 149, 200, 592, 1184, 3000):
        for nf in (1, 3):
            need = [size(rows, n, nf, 9) for n in range(1, 60000, 511)]
            assert need == sorted(need), (rows, nf)
    for n in (1000, 4096, 30720, 250001):
        need = [size(rows, n, 1, 9) for rows in range(1, 1300, 7)] + [size(r, n, 1, 9) for r in (146, 147, 148)]
        assert need[:-3] == sorted(need[:-3]) and need[-3:] == sorted(need[-3:]), n
        assert size(200, n, 1, 9) <= size(200, n, 2, 9) and size(200, n, 1, 8) <= size(200, n, 1, 9)


def test_few_rows_keep_long_chunks():
    """544 chunks of 6144 samples fill the chip: 32 rows of 100003 samples are not cut
    shorter, which took up to 1.8 times as long."""
    from sigpyproc3_b200 import _lib

    def up(v):
        return -(-v // 256) * 256

    chunks = 32 * 17
    assert _lib.load().spp_boxcar_snr_workspace_bytes(32, 100003, 1, 9) == \
        256 + up(chunks * 9 * 16) + up(chunks * 3 * 8)


@pytest.mark.gpu
@pytest.mark.parametrize("robust,rows,n,most_rows,most_n", [(False, 200, 30720, 200, 36864),
                                                           (False, 100, 20000, 1300, 20000),
                                                           (True, 147, 9000, 148, 9000),
                                                           (True, 3, 5000, 200, 4097)])
def test_scratch_of_a_larger_call(robust, rows, n, most_rows, most_n):
    import torch

    from sigpyproc3_b200 import _lib
    from sigpyproc3_b200.search import DEFAULT_WIDTHS, boxcar_snr

    lib = _lib.load()
    size, call = ((lib.spp_boxcar_snr_robust_workspace_bytes, lib.spp_boxcar_snr_robust) if robust
                  else (lib.spp_boxcar_snr_workspace_bytes, lib.spp_boxcar_snr))
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, n, device="cuda", generator=g)
    ws = torch.zeros(size(most_rows, max(n, most_n), 1, 9), dtype=torch.uint8, device="cuda")
    snr = torch.zeros((rows, 1, 9), dtype=torch.float32, device="cuda")
    one = np.ones(1, np.int32)
    wid = np.array(DEFAULT_WIDTHS, np.int32)
    rc = call(x.data_ptr(), _lib.OUT_F32, rows, n, n, one.ctypes.data, 1, wid.ctypes.data, 9,
              snr.data_ptr(), None, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    assert rc == _lib.SPP_OK
    expect, _ = boxcar_snr(x, loc_scale="median_iqr" if robust else "mean_std")
    assert torch.equal(snr, expect)
