"""Filterbank sources and the streaming drop-in path (R1, R5).

``Filterbank`` carries the reference's streaming operations
(src/sigpyproc/base.py) over a block schedule identical to
``FilReader.read_plan`` (src/sigpyproc/readers.py:171-233).  Blocks travel
as raw bytes: file -> pinned host buffer -> async H2D (copy stream) -> HBM,
double-buffered, and the GPU kernels unpack them in their load path.  The
``skipback`` halo leads every block as in the reference (read again, or copied
on the device where it is long), so results are identical block for block.
"""

from __future__ import annotations

import ctypes
import warnings
from collections.abc import Callable, Iterator
from pathlib import Path

import numpy as np
import torch

from . import _lib
from .block import FilterbankBlock
from .dedisp import (DMTPlan, dedisperse_block, status_check, status_clear, stream_handle,
                     workspace)
from .folded import FoldedData
from .header import Header
from .io.bits import bitorder_code
from .io.bits import unpack as gpu_unpack
from .timeseries import TimeSeries


def plan_blocks(nsamples: int, gulp: int, start: int, nsamps: int | None,
                skipback: int) -> tuple[int, list[tuple[int, int, int]]]:
    """Block schedule of read_plan: (gulp, [(ii, samples, skip)])."""
    if nsamps is None:
        nsamps = nsamples - start
    gulp = min(nsamps, gulp)
    skipback = abs(skipback)
    if skipback >= gulp:
        raise ValueError(f"readsamps ({gulp}) must be > skipback ({skipback})")
    nreads, lastread = divmod(nsamps, (gulp - skipback))
    if lastread < skipback:
        nreads -= 1
        lastread = nsamps - (nreads * (gulp - skipback))
    blocks = [(ii, gulp, -skipback) for ii in range(nreads)]
    if lastread != 0:
        blocks.append((nreads, lastread, 0))
    return gulp, blocks


# In-memory filterbanks up to this size are page-locked in place on first use.
REGISTER_MAX_BYTES = 8 << 30

# A halo of this size or more is copied from the previous block on the device:
# that copy, between two from the host, holds the copy stream up by 27 us
# whatever its size, in which the host link moves 1.5 MB (8-bit, 64 MB in 16384-row
# blocks or longer: 2.3 ms either way at 1.5 MB, 2.80 -> 2.23 ms at 2.5 MB).
KEEP_HALO_MIN_BYTES = 3 << 19


def pinned_allocator(nbytes: int) -> torch.Tensor:
    return torch.empty(nbytes, dtype=torch.uint8, pin_memory=True)


def _host_view(buf) -> np.ndarray:
    if torch.is_tensor(buf):
        return buf.numpy()
    return np.frombuffer(memoryview(buf), dtype=np.uint8)


def _allocate(allocator: Callable[[int], object], nbytes: int):
    """io/fileio.py:25-71 contract: positive size, buffer object of that size."""
    if nbytes <= 0:
        raise ValueError(f"Requested buffer size ({nbytes}) is invalid, should be > 0")
    try:
        buf = allocator(nbytes)
    except Exception as exc:
        raise RuntimeError(f"Failed to allocate buffer of size {nbytes}") from exc
    view = _host_view(buf)
    if view.nbytes != nbytes:
        raise ValueError(f"Allocated buffer is not the expected size: {view.nbytes} (actual) "
                         f"!= {nbytes} (expected)")
    return buf


class _DelayTable:
    """Delays on the device, uploaded (and the workspace's status words cleared)
    when a kernel that reads them is first launched: most blocks go through
    kernels that take the delays from the host."""

    def __init__(self, delays: np.ndarray, dev: torch.device, ws: torch.Tensor):
        self._delays, self._dev, self._ws = delays, dev, ws
        self._t: torch.Tensor | None = None

    @property
    def used(self) -> bool:
        return self._t is not None

    def data_ptr(self) -> int:
        if self._t is None:
            self._t = torch.from_numpy(self._delays).to(self._dev)
            status_clear(self._ws)
        return self._t.data_ptr()


class Filterbank:
    """Base of filterbank sources.  Subclasses provide ``header`` and
    ``_read_bytes(offset, view)`` (fill ``view`` from byte ``offset`` of the
    data stream, return the byte count)."""

    header: Header

    # --- geometry ---
    @property
    def row_bytes(self) -> int:
        h = self.header
        return h.nchans * 4 if h.nbits == 32 else h.nchans * h.nbits // 8

    @property
    def bitorder(self) -> str:
        return {1: "little", 2: "big", 4: "big"}.get(self.header.nbits, "big")

    def _read_bytes(self, offset: int, view: np.ndarray) -> int:  # pragma: no cover
        raise NotImplementedError

    def _device_source(self, offset: int, nbytes: int) -> torch.Tensor | None:
        """Bytes [offset, offset + nbytes) as a page-locked host tensor the GPU
        can copy from directly, or None: blocks are staged through pinned
        buffers filled by ``_read_bytes``."""
        return None

    def _bytes_available(self, offset: int, nbytes: int) -> int:
        """How many of the bytes [offset, offset + nbytes) exist (sources with
        a direct path report it when a block runs past the data)."""
        return 0

    # --- streaming (R5) ---
    def stream_blocks(self, gulp: int = 16384, start: int = 0, nsamps: int | None = None,
                      skipback: int = 0, *, allocator: Callable[[int], object] | None = None,
                      description: str | None = None, quiet: bool = False,
                      keep_halo: bool = False) -> Iterator[tuple[int, int, torch.Tensor]]:
        """Yields ``(nsamps_read, ii, raw)``: ``raw`` is a CUDA uint8 tensor of
        the block's raw bytes, valid until the next iteration.  Work the
        consumer enqueues on the current stream is ordered before the buffer
        is refilled.  ``keep_halo``: a consumer that leaves ``raw`` as it is
        lets each block take its first ``skipback`` rows from the previous
        block on the device, where they are many (the same bytes; a caller's
        allocator always sees whole blocks)."""
        gulp, blocks = plan_blocks(self.header.nsamples, gulp, start, nsamps, skipback)
        rb = self.row_bytes
        if self.header.nbits < 8 and (self.header.nchans * self.header.nbits) % 8:
            raise ValueError("nchans * nbits must be a multiple of 8")
        nbytes = gulp * rb
        alloc = pinned_allocator if allocator is None else allocator
        dev = torch.device("cuda", torch.cuda.current_device())
        # data already in page-locked host memory is copied straight from
        # there (default allocator only: a caller's allocator is always used)
        direct = allocator is None and self._device_source(0, 0) is not None
        host = hviews = None
        if not direct:
            host = [_allocate(alloc, nbytes) for _ in range(2)]
            hviews = [_host_view(h) for h in host]
        devbuf = [torch.empty(nbytes, dtype=torch.uint8, device=dev) for _ in range(2)]
        copy_stream = torch.cuda.Stream(dev)
        lib = _lib.load()
        handle = ctypes.c_void_p()
        _lib.check(lib.spp_blocks_create(ctypes.byref(handle), copy_stream.cuda_stream,
                                         stream_handle(None, dev)))
        dptr = [d.data_ptr() for d in devbuf]
        pos = start * rb
        back = abs(skipback) * rb if keep_halo and allocator is None else 0
        if back < KEEP_HALO_MIN_BYTES:
            back = 0
        try:
            for n, (ii, nsamp_blk, skip) in enumerate(blocks):
                k = n & 1
                want = nsamp_blk * rb
                # already on the device: only the last block is shorter than the gulp
                old = min(back, want) if n else 0
                src = self._device_source(pos + old, want - old) if direct else None
                if src is None:
                    if direct:
                        got = self._bytes_available(pos, want)
                        raise ValueError(f"Unexpected number of bytes read from file {got} "
                                         f"(actual) != {want} (expected)")
                    if n > 1:  # host buffer k is free once its copy landed
                        _lib.check(lib.spp_blocks_wait(handle, k))
                    got = old + self._read_bytes(pos + old, hviews[k][:want - old])
                    if got != want:
                        raise ValueError(f"Unexpected number of bytes read from file {got} "
                                         f"(actual) != {want} (expected)")
                    sptr = hviews[k].ctypes.data
                else:
                    sptr = src.data_ptr()
                pos += want + skip * rb
                _lib.check(lib.spp_blocks_put(handle, k, dptr[k], dptr[1 - k] + nbytes - back, old,
                                              sptr, want - old))
                yield nsamp_blk, ii, devbuf[k][:want]
            torch.cuda.current_stream(dev).synchronize()
        finally:
            _lib.check(lib.spp_blocks_destroy(handle))

    def read_plan(self, gulp: int = 16384, start: int = 0, nsamps: int | None = None,
                  skipback: int = 0, description: str | None = None, *, quiet: bool = False,
                  allocator: Callable[[int], object] | None = None
                  ) -> Iterator[tuple[int, int, np.ndarray]]:
        """Reference-compatible read_plan: yields host arrays of the block's
        samples (unpacked to one uint8 per sample for nbits < 8, on the GPU)."""
        h = self.header
        for nsamp_blk, ii, raw in self.stream_blocks(gulp, start, nsamps, skipback,
                                                     allocator=allocator):
            if h.nbits in (1, 2, 4):
                data = gpu_unpack(raw, h.nbits, self.bitorder).cpu().numpy()
            elif h.nbits == 32:
                data = raw.view(torch.float32).cpu().numpy()
            else:
                data = raw.cpu().numpy()
            yield nsamp_blk, ii, data

    # --- R1: single-DM dedispersion ---
    def dedisperse(self, dm: float, ref_freq: str | float = "fch1", gulp: int = 16384,
                   start: int = 0, nsamps: int | None = None, *, parallel: bool = False,
                   **plan_kwargs) -> TimeSeries:
        """Dedisperse and collapse to a time series (base.py:360-424).

        ``parallel`` is accepted for compatibility; the GPU path is always
        parallel.  Float32 data is accumulated in float64 like the reference.
        """
        del parallel
        h = self.header
        chan_delays = np.atleast_1d(h.get_dmdelays(dm, ref_freq)).astype(np.int32)
        max_delay = int(np.max(np.abs(chan_delays)))
        gulp = max(2 * max_delay, gulp)
        tim_len = h.nsamples - max_delay
        dev = torch.device("cuda", torch.cuda.current_device())
        tim = torch.zeros(max(tim_len, 0), dtype=torch.float32, device=dev)
        # one workspace for every block (a block never exceeds the gulp); its
        # device status words collect any kernel-side error over the whole run
        need = _lib.load().spp_dedisperse_workspace_bytes(
            h.nbits, h.nchans, min(gulp, h.nsamples), int(chan_delays.min()),
            int(chan_delays.max()))
        ws = workspace(max(int(need), 256), dev)
        table = _DelayTable(chan_delays, dev, ws)
        for nsamps_r, ii, raw in self.stream_blocks(gulp, start, nsamps, skipback=max_delay,
                                                    keep_halo=True, **plan_kwargs):
            dedisperse_block(raw, chan_delays, h.nchans, nsamps_r, tim, ii * (gulp - max_delay),
                             nbits=h.nbits, bitorder=self.bitorder, acc=_lib.ACC_F64,
                             delays_dev=table, ws=ws)
        if table.used:  # only kernels that read the table record a device status
            status_check(ws)
        return TimeSeries(tim, h.new_header({"nchans": 1, "dm": dm, "nsamples": tim_len}))

    # --- R3: DM-trial batch ---
    def dedisperse_batch(self, dms=None, *, dm: float | None = None, dmsteps: int = 512,
                         ref_freq: str | float = "fch1", gulp: int = 1 << 20, start: int = 0,
                         nsamps: int | None = None, out_dtype=None, **plan_kwargs):
        """DM-time array ``out[i][t] = dedisperse(dms[i])[t]`` over the valid
        samples common to every trial (``nsamples - max_i max_c |delay|``).

        Give ``dms`` explicitly or ``dm``/``dmsteps`` for the dmt_transform
        grid ``dm + linspace(-dm, dm, dmsteps)``.  Integer data defaults to
        exact int32 sums, float data to float32.  Returns (tensor, dms).
        """
        h = self.header
        if dms is None:
            if dm is None:
                raise ValueError("give dms or dm/dmsteps")
            dms = dm + np.linspace(-dm, dm, dmsteps)
        dms = np.atleast_1d(np.asarray(dms, dtype=np.float64))
        delays = np.atleast_2d(h.get_dmdelays(dms, ref_freq)).astype(np.int32)
        max_delay = int(np.max(np.abs(delays)))
        if out_dtype is None:
            out_dtype = torch.float32 if h.nbits == 32 else torch.int32
        gulp = max(2 * max_delay, gulp)
        span = (h.nsamples - start) if nsamps is None else nsamps
        nout = max(span - max_delay, 0)
        dev = torch.device("cuda", torch.cuda.current_device())
        out = torch.zeros((delays.shape[0], nout), dtype=out_dtype, device=dev)
        plan = DMTPlan(delays, h.nchans, min(gulp, span), nbits=h.nbits, bitorder=self.bitorder,
                       out_dtype=out_dtype)
        try:
            ws = workspace(plan.workspace_bytes(min(gulp, span)), dev)
            status_clear(ws)
            for nsamps_r, ii, raw in self.stream_blocks(gulp, start, nsamps, skipback=max_delay,
                                                        keep_halo=True, **plan_kwargs):
                plan.execute(raw, nsamps_r, out, out_start=ii * (gulp - max_delay), ws=ws)
            status_check(ws)
        finally:
            torch.cuda.current_stream(dev).synchronize()
            plan.close()
        return out, dms

    # --- channel statistics (R10 / N2) ---
    def bandpass(self, method: str = "sum", gulp: int = 16384, start: int = 0, *,
                 parallel: bool = False, nsamps: int | None = None, **plan_kwargs) -> TimeSeries:
        """Per-channel sum (or mean) over samples (base.py:308-358), float32
        accumulated in sample order exactly as the reference."""
        del parallel
        h = self.header
        dev = torch.device("cuda", torch.cuda.current_device())
        bp = torch.zeros(h.nchans, dtype=torch.float32, device=dev)
        total = 0
        for nsamps_r, _ii, raw in self.stream_blocks(gulp, start, nsamps, **plan_kwargs):
            _lib.call("spp_bandpass", raw.data_ptr(), h.nbits, bitorder_code(self.bitorder),
                      h.nchans, nsamps_r, bp.data_ptr(), stream_handle(None, dev))
            total += nsamps_r
        if method == "mean":
            bp /= total
        return TimeSeries(bp, h.new_header({"nchans": 1, "nsamples": h.nchans}))

    def collapse(self, method: str = "sum", gulp: int = 16384, start: int = 0,
                 nsamps: int | None = None, *, parallel: bool = False,
                 **plan_kwargs) -> TimeSeries:
        """Sum over channels per sample (base.py:256-306)."""
        del parallel
        h = self.header
        tim_len = (h.nsamples - start) if nsamps is None else nsamps
        dev = torch.device("cuda", torch.cuda.current_device())
        tim = torch.zeros(tim_len, dtype=torch.float32, device=dev)
        for nsamps_r, ii, raw in self.stream_blocks(gulp, start, nsamps, **plan_kwargs):
            # the reference offsets each block by ii * nsamps_r (base.py:292-298)
            _lib.call("spp_collapse", raw.data_ptr(), h.nbits, bitorder_code(self.bitorder),
                      h.nchans, nsamps_r, tim.data_ptr(), ii * nsamps_r, stream_handle(None, dev))
        if method == "mean":
            tim /= h.nchans
        return TimeSeries(tim, h.new_header({"nchans": 1, "dm": 0}))

    # --- file-writing operations (R7, R10, N2) ---
    def _block_values(self, raw: torch.Tensor, nsamps_r: int) -> torch.Tensor:
        """The block's samples in the reference's read_plan dtype: one uint8 per
        sample (packed data unpacked on the GPU) or float32."""
        h = self.header
        raw = raw[: nsamps_r * self.row_bytes]
        if h.nbits in (1, 2, 4):
            return gpu_unpack(raw, h.nbits, self.bitorder)
        if h.nbits == 32:
            return raw.view(torch.float32)
        return raw

    def remove_zerodm(self, outfile_name: str | None = None, gulp: int = 16384, start: int = 0,
                      nsamps: int | None = None, *, parallel: bool = False,
                      **plan_kwargs) -> str:
        """Remove the channel-weighted zero-DM signal and write a new file
        (base.py:961-1028; Eatough, Keane & Lyne 2009).

        As the reference: the bandpass is the sum over the whole file
        (``self.bandpass(**plan_kwargs)``), ``chanwts = bpass / sum(bpass)``
        in float32, and each block becomes ``x - zdm * chanwts + bpass``
        (float64, zdm the channel sum of the spectrum) in the file's own
        sample format: float32 rounded, 8-bit as the low eight bits of the
        truncated value (the reference's uint8 cast), 1/2/4-bit repacked."""
        del parallel
        h = self.header
        if outfile_name is None:
            outfile_name = f"{h.basename}_noZeroDM.fil"
        bp = self.bandpass(**plan_kwargs).data
        chanwts = (bp / bp.sum()).astype(np.float32)
        dev = torch.device("cuda", torch.cuda.current_device())
        bp_d = torch.from_numpy(bp).to(dev)
        w_d = torch.from_numpy(chanwts).to(dev)
        st = stream_handle(None, dev)
        with h.prep_outfile(outfile_name, nbits=h.nbits) as out_file:
            for nsamps_r, _ii, raw in self.stream_blocks(gulp, start, nsamps, **plan_kwargs):
                x = self._block_values(raw, nsamps_r)
                y = torch.empty_like(x)
                fn = "spp_zero_dm" if h.nbits == 32 else "spp_zero_dm_u8"
                _lib.call(fn, x.data_ptr(), y.data_ptr(), h.nchans, nsamps_r, bp_d.data_ptr(),
                          w_d.data_ptr(), st)
                out_file.cwrite(y.cpu().numpy())
        return outfile_name

    def downsample(self, tfactor: int = 1, ffactor: int = 1, outfile_name: str | None = None,
                   gulp: int = 16384, start: int = 0, nsamps: int | None = None, *,
                   compat: bool = False, **plan_kwargs) -> str:
        """Decimate in time and frequency and write a new file (base.py:585-654):
        means of ``tfactor`` samples x ``ffactor`` channels (float64 sums,
        kernels.downsample_2d_mean_flat core/kernels.py:207-252), in the
        file's sample format (8-bit and packed means truncated to integers),
        header tsamp * tfactor, nchans // ffactor, foff * ffactor.

        The reference's block loop passes (nchans, nsamps) where the kernel
        expects (samples, channels) of its time-major block, which averages
        across the wrong axes; ``compat=True`` repeats that call exactly,
        the default averages as documented."""
        h = self.header
        if outfile_name is None:
            outfile_name = f"{h.basename}_f{ffactor:d}_t{tfactor:d}.fil"
        if h.nchans % ffactor != 0:
            raise ValueError(f"Bad frequency factor given: {ffactor:d}")
        if tfactor < 1 or ffactor < 1:
            raise ValueError("Factors must be positive integers.")
        gulp = int(np.ceil(gulp / tfactor) * tfactor)
        updates = {"tsamp": h.tsamp * tfactor, "nchans": h.nchans // ffactor,
                   "foff": h.foff * ffactor}
        st = stream_handle(None, torch.device("cuda", torch.cuda.current_device()))
        with h.prep_outfile(outfile_name, updates=updates) as out_file:
            for nsamps_r, _ii, raw in self.stream_blocks(gulp, start, nsamps, **plan_kwargs):
                x = self._block_values(raw, nsamps_r)
                dims = (h.nchans, nsamps_r) if compat else (nsamps_r, h.nchans)
                fac = (tfactor, ffactor)
                y = torch.empty((dims[0] // fac[0]) * (dims[1] // fac[1]), dtype=x.dtype,
                                device=x.device)
                fn = "spp_downsample_2d_mean" if h.nbits == 32 else "spp_downsample_2d_mean_u8"
                _lib.call(fn, x.data_ptr(), dims[0], dims[1], fac[0], fac[1], y.data_ptr(), st)
                out_file.cwrite(y.cpu().numpy())
        return outfile_name

    def subband(self, dm: float, nsub: int, ref_freq: str | float = "fch1",
                outfile_name: str | None = None, gulp: int = 16384, start: int = 0,
                nsamps: int | None = None, **plan_kwargs) -> str:
        """Dedisperse into ``nsub`` subbands at one DM and write them as a
        32-bit file (base.py:1030-1107): channel c goes to subband
        ``c // (nchans // nsub)``, the read_plan blocks overlap by the maximum
        delay, header fch1 = ftop - new_foff / 2, foff = foff * nchans // nsub,
        refdm = dm, nchans = nsub.  Each block's sums start from zero (the
        reference never clears its output buffer between blocks)."""
        h = self.header
        subfactor = h.nchans // nsub
        chan_delays = np.atleast_1d(h.get_dmdelays(dm, ref_freq)).astype(np.int32)
        max_delay = int(np.max(np.abs(chan_delays)))
        gulp = max(2 * max_delay, gulp)
        new_foff = h.foff * h.nchans // nsub
        new_fch1 = h.ftop - new_foff / 2
        chan_to_sub = (np.arange(h.nchans, dtype=np.int32) // subfactor).astype(np.int32)
        if chan_to_sub.max() >= nsub:
            raise ValueError(f"nchans ({h.nchans}) is not a multiple of nsub ({nsub})")
        updates = {"fch1": new_fch1, "foff": new_foff, "refdm": dm, "nchans": nsub}
        if outfile_name is None:
            outfile_name = f"{h.basename}_DM{dm:06.2f}.subbands"
        dev = torch.device("cuda", torch.cuda.current_device())
        d_d = torch.from_numpy(chan_delays).to(dev)
        c_d = torch.from_numpy(chan_to_sub).to(dev)
        st = stream_handle(None, dev)
        with h.prep_outfile(outfile_name, updates=updates, nbits=32) as out_file:
            for nsamps_r, _ii, raw in self.stream_blocks(gulp, start, nsamps,
                                                        skipback=max_delay, keep_halo=True,
                                                        **plan_kwargs):
                nout = nsamps_r - max_delay
                if nout <= 0:
                    continue
                y = torch.empty(nout * nsub, dtype=torch.float32, device=dev)
                _lib.call("spp_subband", raw.data_ptr(), h.nbits, bitorder_code(self.bitorder),
                          h.nchans, nsamps_r, d_d.data_ptr(), max_delay, c_d.data_ptr(), nsub,
                          y.data_ptr(), st)
                out_file.cwrite(y.cpu().numpy())
        return outfile_name

    # --- N4: folding ---
    def fold(self, period: float, dm: float, accel: float = 0, nbins: int = 50, nints: int = 32,
             nbands: int = 32, gulp: int = 16384, start: int = 0, nsamps: int | None = None,
             **plan_kwargs) -> FoldedData:
        """Fold into (subintegration, subband, phase bin) cells (base.py:1109-1207).

        The same checks, warnings, block plan and block index as the reference;
        each block folds on the GPU (packed data is unpacked on the device
        first) into device cells, divided by the counts at the end.  Integer
        samples fold into exact 64-bit cells rounded to float32 once
        (``spp_fold_exact``): identical to the reference's float32 cells while
        a cell stays below 2^24, deterministic beyond.  Float32 samples fold
        into float32 cells with atomic adds, so their last bits depend on the
        order the adds land in (the reference adds sequentially): cubes agree
        to float32 rounding and can differ from run to run in the last bits.
        """
        import warnings

        h = self.header
        if np.isclose(np.modf(period / h.tsamp)[0], 0.001, atol=0):
            warnings.warn("Foldng interval is an integer multiple of the sampling time",
                          stacklevel=2)
        if nbins > period / h.tsamp:
            warnings.warn("Number of phase bins is greater than period/sampling time",
                          stacklevel=2)
        if (h.nsamples * h.nchans) // (nbands * nints * nbins) < 10:
            raise ValueError(f"nbands x nints x nbins is too large: {nbands * nints * nbins}")
        nbands = min(nbands, h.nchans)
        chan_delays = np.atleast_1d(h.get_dmdelays(dm)).astype(np.int32)
        max_delay = int(chan_delays.max())
        gulp = max(2 * max_delay, gulp)
        band_start = fold_band_start(h.nchans, nbands)
        dev = torch.device("cuda", torch.cuda.current_device())
        cells = nbins * nints * nbands
        exact = h.nbits != 32  # integer samples: 64-bit integer cells, rounded once at the end
        fold_ar = torch.zeros(cells, dtype=torch.int64 if exact else torch.float32, device=dev)
        count_ar = torch.zeros(cells, dtype=torch.int32, device=dev)
        tables = torch.from_numpy(np.concatenate([chan_delays, band_start])).to(dev)  # one upload
        ddev, bdev = tables[:h.nchans], tables[h.nchans:]
        lib = _lib.load()
        st = stream_handle(None, dev)
        for nsamps_r, ii, raw in self.stream_blocks(gulp, start, nsamps, skipback=max_delay,
                                                    keep_halo=True, **plan_kwargs):
            if h.nbits < 8:
                x, nb = gpu_unpack(raw[:nsamps_r * self.row_bytes], h.nbits, self.bitorder), 8
            else:
                x, nb = raw, h.nbits
            # the reference indexes each block by ii * (gulp - max_delay) (base.py:1202)
            if exact:
                _lib.check(lib.spp_fold_exact(x.data_ptr(), h.nchans, nsamps_r, ddev.data_ptr(),
                                              max_delay, h.tsamp, period, accel, h.nsamples,
                                              nbins, nints, nbands, ii * (gulp - max_delay),
                                              bdev.data_ptr(), fold_ar.data_ptr(),
                                              count_ar.data_ptr(), cells, st))
            else:
                _lib.check(lib.spp_fold(x.data_ptr(), nb, h.nchans, nsamps_r, ddev.data_ptr(),
                                        max_delay, h.tsamp, period, accel, h.nsamples, nbins,
                                        nints, nbands, ii * (gulp - max_delay), bdev.data_ptr(),
                                        fold_ar.data_ptr(), count_ar.data_ptr(), cells, st))
        mean = torch.empty(cells, dtype=torch.float32, device=dev)
        _lib.check(lib.spp_fold_finish(None if exact else fold_ar.data_ptr(),
                                       fold_ar.data_ptr() if exact else None, count_ar.data_ptr(),
                                       cells, mean.data_ptr(), st))
        f = mean.cpu().numpy()
        return FoldedData(f.reshape(nints, nbands, nbins), h.new_header(), period, dm, accel)


def fold_band_start(nchans: int, nbands: int) -> np.ndarray:
    """First channel of each of ``nbands`` subbands (plus ``nchans`` at the end),
    as kernels.fold assigns channels: ``ichan // (nchans / nbands)`` with
    Python's float floor division (core/kernels.py:424, :439)."""
    factor2 = nchans / nbands
    band = np.array([int(c // factor2) for c in range(nchans)], dtype=np.int64)
    if np.any(np.diff(band) < 0) or band.min() < 0 or band.max() >= nbands:
        raise ValueError("subband assignment out of range")
    return np.searchsorted(band, np.arange(nbands + 1)).astype(np.int32)


class FilReader(Filterbank):
    """Sigproc filterbank file(s) (readers.py:33-233)."""

    def __init__(self, filenames, *, check_contiguity: bool = True):
        if isinstance(filenames, (str, Path)):
            filenames = [filenames]
        self._filenames = [str(f) for f in filenames]
        self._header = Header.from_sigproc(self._filenames)
        del check_contiguity

    @property
    def header(self) -> Header:
        return self._header

    @property
    def filename(self) -> str:
        return self._filenames[0]

    def _read_bytes(self, offset: int, view: np.ndarray) -> int:
        info = self._header.stream
        done = 0
        want = view.nbytes
        base = 0
        for fname, hlen, dlen in zip(info.files, info.hdrlens, info.datalens):
            if offset + done < base + dlen and done < want:
                local = offset + done - base
                n = min(dlen - local, want - done)
                with open(fname, "rb") as fp:
                    fp.seek(hlen + local)
                    got = fp.readinto(memoryview(view[done:done + n]))
                done += got or 0
            base += dlen
        return done

    def read_block(self, start: int, nsamps: int, fch1: float | None = None,
                   nchans: int | None = None) -> FilterbankBlock:
        """(nchans, nsamps) float32 block in HBM (readers.py:98-130)."""
        h = self.header
        fch1 = h.fch1 if fch1 is None else fch1
        nchans = h.nchans if nchans is None else nchans
        if fch1 > h.fch1 or nchans > h.nchans:
            raise ValueError(f"requested block is out of range: fch1={fch1}, nchans={nchans}")
        if start < 0 or start + nsamps > h.nsamples:
            raise ValueError(f"requested block is out of range: start={start}, nsamps={nsamps}")
        raw = np.empty(nsamps * self.row_bytes, dtype=np.uint8)
        got = self._read_bytes(start * self.row_bytes, raw)
        raw_t = torch.from_numpy(raw[:got]).cuda()
        if h.nbits in (1, 2, 4):
            vals = gpu_unpack(raw_t, h.nbits, self.bitorder).view(-1, h.nchans).float()
        elif h.nbits == 32:
            vals = raw_t.view(torch.float32).view(-1, h.nchans)
        else:
            vals = raw_t.view(-1, h.nchans).float()
        chan_start = int((fch1 - h.fch1) / h.foff)
        data = vals.t()[chan_start:chan_start + nchans].contiguous()
        hdr = h.new_header({"tstart": h.mjd_after_nsamps(start), "nsamples": data.shape[1],
                            "fch1": fch1, "nchans": nchans})
        return FilterbankBlock(data, hdr)


class ArrayFilterbank(Filterbank):
    """A filterbank held in host memory (raw time-major bytes), e.g. synthetic data.

    On first use the array (up to REGISTER_MAX_BYTES) is page-locked in place,
    so each block is copied to the GPU by DMA straight from it rather than
    through a staging buffer; it is released when the object is collected.
    If the driver refuses (e.g. the memory is already registered elsewhere),
    blocks are staged as for files."""

    def __init__(self, raw: np.ndarray, header: Header):
        self._raw = np.ascontiguousarray(raw).view(np.uint8).ravel()
        self._header = header
        self._registered: bool | None = None  # None: not tried yet
        self._whole: torch.Tensor | None = None  # _raw as a tensor, once registered

    @property
    def header(self) -> Header:
        return self._header

    def _read_bytes(self, offset: int, view: np.ndarray) -> int:
        n = max(0, min(view.nbytes, self._raw.nbytes - offset))
        view[:n] = self._raw[offset:offset + n]
        return n

    def _bytes_available(self, offset: int, nbytes: int) -> int:
        return max(0, min(nbytes, self._raw.nbytes - offset))

    def _device_source(self, offset: int, nbytes: int) -> torch.Tensor | None:
        if self._registered is None:
            n = self._raw.nbytes
            self._registered = (0 < n <= REGISTER_MAX_BYTES and
                                _lib.load().spp_host_register(self._raw.ctypes.data, n) == 0)
        if not self._registered or offset + nbytes > self._raw.nbytes:
            return None
        if self._whole is None:
            with warnings.catch_warnings():  # read-only arrays: the view is only read
                warnings.simplefilter("ignore", UserWarning)
                self._whole = torch.from_numpy(self._raw)
        return self._whole[offset:offset + nbytes]

    def __del__(self):
        if getattr(self, "_registered", False):
            try:
                _lib.load().spp_host_unregister(self._raw.ctypes.data)
            except Exception:  # interpreter shutdown
                pass


class PulseExtractor:
    """A filterbank block centred on a pulse (readers.py:353-478): the pulse's
    time of arrival ``pulse_toa`` (samples, at ``toa_freq``, default the top of
    the band), width and DM fix the window (the DM sweep plus five widths on
    each side, at least ``min_nsamps`` decimated samples); samples beyond the
    file are padded with each channel's median or mean."""

    def __init__(self, filfile, pulse_toa: int, pulse_width: int, pulse_dm: float,
                 min_nsamps: int = 256, toa_freq: float | None = None,
                 nchans: int | None = None):
        self.filfile = filfile
        self.pulse_toa = pulse_toa
        self.pulse_width = pulse_width
        self.pulse_dm = pulse_dm
        self.min_nsamps = min_nsamps
        hdr = Header.from_sigproc(filfile)
        self.toa_freq = toa_freq or hdr.fch1
        self.nchans = nchans or hdr.nchans
        self.sub_hdr = hdr.new_header({"fch1": self.toa_freq, "nchans": self.nchans})
        self._disp_delay = int(np.max(np.abs(np.atleast_1d(
            self.sub_hdr.get_dmdelays(self.pulse_dm, in_samples=True))))) + self.pulse_width * 5

    @property
    def t_decimate(self) -> int:
        return max(1, self.pulse_width // 2)

    @property
    def disp_delay(self) -> int:
        return self._disp_delay

    @property
    def block_delay(self) -> int:
        return ((self.disp_delay // self.t_decimate) + 1) * self.t_decimate

    @property
    def nsamps(self) -> int:
        return max(2 * self.block_delay, self.min_nsamps * self.t_decimate)

    @property
    def nstart(self) -> int:
        return self.pulse_toa - self.nsamps // 2

    @property
    def nstart_file(self) -> int:
        return max(0, self.nstart)

    @property
    def nsamps_file(self) -> int:
        return min(self.nsamps + min(0, self.nstart), self.sub_hdr.nsamples - max(0, self.nstart))

    @property
    def pulse_toa_block(self) -> int:
        return self.pulse_toa - self.nstart

    def get_data(self, pad_mode: str = "median") -> FilterbankBlock:
        fil = FilReader(self.filfile)
        block = fil.read_block(start=self.nstart_file, nsamps=self.nsamps_file,
                               fch1=self.toa_freq, nchans=self.nchans)
        if self.nstart < 0 or self.nstart + self.nsamps > self.sub_hdr.nsamples:
            offset = abs(min(0, self.nstart))
            block = block.pad_samples(self.nsamps, offset, pad_mode=pad_mode)
        return block
