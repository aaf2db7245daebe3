"""Performance cases: the calls a dedispersion user's program makes, over the
sizes, sample widths and options it makes them with.

Every case goes through public entry points.  Inputs and plans are what such a
program already holds before the call (raw samples in HBM, a delay table and
its plan; host arrays for the calls that start from host memory).  Sizes come
from the benchmark workloads (synth.C1/C2/C3/C5, the streaming server's beams)
and odd lengths around them.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import sigpyproc3_b200 as spp
from sigpyproc3_b200 import synth
from sigpyproc3_b200.search import boxcar_snr
from sigpyproc3_b200.subband import SubbandPlan, SubbandSearch

TSAMP = 64e-6
BANDWIDTH = 300.0  # MHz, below 1500 MHz (the 4096-channel and served bands)


def listed() -> list[dict]:
    return [
        # one DM over one block of the default gulp: the smallest call, what a
        # streaming Filterbank.dedisperse issues per block
        {"name": "single_gulp", "kind": "single", "nbits": 8, "nchans": 256, "nsamps": 16384,
         "dm": 100.0},
        # one DM over a long 8-bit observation held in HBM
        {"name": "single_long", "kind": "single", "nbits": 8, "nchans": 1024, "nsamps": 262144,
         "dm": 300.0},
        # one DM over a packed block with an odd channel count and odd length
        {"name": "single_packed", "kind": "single", "nbits": 2, "nchans": 1020, "nsamps": 200003,
         "dm": 150.0},
        # the headline DM-time transform: 2-bit, 4096 channels, 1024 trials, 2^20 samples
        {"name": "batch_2bit", "kind": "batch", "nbits": 2, "nchans": 4096, "nsamps": 1048576,
         "dm_max": 2000.0, "ndm": 1024},
        # a blind-search grid over an 8-bit block
        {"name": "batch_8bit", "kind": "batch", "nbits": 8, "nchans": 1024, "nsamps": 150001,
         "dm_max": 1000.0, "ndm": 512},
        # a served chunk: 4-bit, few trials that are not a multiple of any tile, short block
        {"name": "batch_4bit_chunk", "kind": "batch", "nbits": 4, "nchans": 1024, "nsamps": 70001,
         "dm_max": 1100.0, "ndm": 333},
        # float32 samples with the zero-DM signal removed in the load
        {"name": "batch_f32_zerodm", "kind": "zerodm", "nchans": 1024, "nsamps": 65536,
         "dm_max": 500.0, "ndm": 256},
        # two-stage subband search of uneven beams, S/N peaks at the end
        {"name": "subband_search", "kind": "subband", "nsamps_a": 262144, "nsamps_b": 150001,
         "dm_max": 1000.0, "ndm": 512},
        # boxcar S/N of a block of DM-time rows, downsampled 1/2/4
        {"name": "snr_rows", "kind": "snr", "rows": 512, "n": 250001, "dtype": "int32",
         "nfactors": 3, "nwidths": 9, "loc_scale": "mean_std"},
        # robust S/N of one dedispersed time series
        {"name": "snr_series", "kind": "snr", "rows": 1, "n": 262144, "dtype": "float32",
         "nfactors": 1, "nwidths": 9, "loc_scale": "median_iqr"},
        # folding an 8-bit observation from host memory with the default cube
        {"name": "fold", "kind": "fold", "nbits": 8, "nchans": 256, "nsamps": 262144,
         "period": 0.0503, "dm": 100.0},
        # Filterbank.dedisperse from host memory, the reference's block plan
        {"name": "filterbank_dedisperse", "kind": "filterbank", "nbits": 8, "nchans": 256,
         "nsamps": 65536, "dm": 100.0},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    """Log-uniform integer; odd as often as not."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v))


def draw(rng) -> dict:
    kind = rng.choice(["single", "single", "batch", "batch", "batch", "zerodm", "subband", "snr",
                       "snr", "fold", "filterbank"])
    if kind == "single":
        nbits = rng.choice([8, 8, 1, 2, 4, 32])
        nchans = rng.choice([256, 336, 512, 1024, 1020, 2048])
        cap = min(300000, (256 << 20) * 8 // (nbits * nchans))
        return {"kind": kind, "nbits": nbits, "nchans": nchans,
                "nsamps": _log_int(rng, 16384, cap), "dm": round(rng.uniform(10.0, 300.0), 2)}
    if kind == "batch":
        nbits = rng.choice([1, 2, 2, 4, 8, 8])
        nchans = rng.choice([256, 1024, 1024, 4096])
        ndm = _log_int(rng, 64, 1024)
        dm_max = round(rng.uniform(300.0, 2000.0), 1)
        lo = 16384 + int(16.3 * dm_max)  # the largest delay of the band is about 16.2 per DM unit
        cap = int(1.2e12 / nbits / (ndm * nchans))
        return {"kind": kind, "nbits": nbits, "nchans": nchans,
                "nsamps": _log_int(rng, lo, max(lo + 1000, min(400000, cap))),
                "dm_max": dm_max, "ndm": ndm}
    if kind == "zerodm":
        nchans = rng.choice([256, 1024, 2048])
        return {"kind": kind, "nchans": nchans,
                "nsamps": _log_int(rng, 24000, (64 << 20) // nchans + 16000),
                "dm_max": round(rng.uniform(100.0, 600.0), 1), "ndm": _log_int(rng, 32, 512)}
    if kind == "subband":
        return {"kind": kind, "nsamps_a": _log_int(rng, 80000, 262144),
                "nsamps_b": _log_int(rng, 60000, 200000),
                "dm_max": round(rng.uniform(400.0, 1200.0), 1), "ndm": 16 * rng.randint(8, 32)}
    if kind == "snr":
        one = rng.random() < 0.4
        return {"kind": kind, "rows": 1 if one else _log_int(rng, 8, 512),
                "n": _log_int(rng, 16384, 400000), "dtype": rng.choice(["int32", "float32"]),
                "nfactors": rng.randint(1, 3), "nwidths": rng.randint(6, 10),
                "loc_scale": rng.choice(["mean_std", "median_iqr"])}
    if kind == "fold":
        return {"kind": kind, "nbits": rng.choice([8, 8, 2]), "nchans": rng.choice([128, 256, 336]),
                "nsamps": _log_int(rng, 32768, 262144),
                "period": round(rng.uniform(0.01, 0.4), 5), "dm": round(rng.uniform(5.0, 150.0), 2)}
    return {"kind": kind, "nbits": rng.choice([8, 8, 2]), "nchans": rng.choice([256, 512]),
            "nsamps": _log_int(rng, 20000, 131072), "dm": round(rng.uniform(10.0, 120.0), 2)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _header(nchans: int, nbits: int, nsamps: int = 0) -> spp.Header:
    if nchans <= 512:  # the 256 MHz band of the single-DM workload
        return spp.Header(nchans=nchans, fch1=1500.0, foff=-256.0 / nchans, tsamp=TSAMP,
                          nbits=nbits, nsamples=nsamps)
    return spp.Header(nchans=nchans, fch1=1500.0, foff=-BANDWIDTH / nchans, tsamp=TSAMP,
                      nbits=nbits, nsamples=nsamps)


def _raw(nchans: int, nsamps: int, nbits: int, seed: int) -> torch.Tensor:
    """Raw time-major samples in HBM: Gaussian counts (8-bit), N(0,1) (float32),
    uniform packed levels (1/2/4-bit)."""
    if nbits == 8:
        return synth.gauss_u8_device(nchans * nsamps, seed, 96.0, 12.0)
    if nbits == 32:
        return synth.gauss_f32_device(nchans * nsamps, seed)
    return synth.uniform_bytes_device(nchans * nsamps * nbits // 8, seed)


def _delays(h: spp.Header, dms) -> np.ndarray:
    return np.ascontiguousarray(np.atleast_2d(h.get_dmdelays(dms)).astype(np.int32))


def _grid(case: dict) -> np.ndarray:
    return np.linspace(0.0, case["dm_max"], case["ndm"])


WIDTHS = tuple(1 << k for k in range(10))


def _bitorder(nbits: int) -> str:
    return "little" if nbits == 1 else "big"


def prepare(case: dict, seed: int):
    kind = case["kind"]
    seed = int(seed) % (1 << 22)
    if kind == "single":
        h = _header(case["nchans"], case["nbits"])
        d = _delays(h, case["dm"])[0]
        n = case["nsamps"]
        return {"kind": kind, "case": case, "raw": _raw(case["nchans"], n, case["nbits"], seed),
                "d": d, "dd": torch.from_numpy(d).cuda(),
                "out": torch.zeros(n - int(d.max()), dtype=torch.float32, device="cuda")}
    if kind == "batch":
        h = _header(case["nchans"], case["nbits"])
        d = _delays(h, _grid(case))
        n = case["nsamps"]
        plan = spp.DMTPlan(d, case["nchans"], n, nbits=case["nbits"],
                           bitorder=_bitorder(case["nbits"]), out_dtype=torch.int32)
        return {"kind": kind, "case": case, "plan": plan,
                "raw": _raw(case["nchans"], n, case["nbits"], seed),
                "out": torch.empty((case["ndm"], plan.nvalid(n)), dtype=torch.int32,
                                   device="cuda")}
    if kind == "zerodm":
        h = _header(case["nchans"], 32)
        d = _delays(h, _grid(case))
        n = case["nsamps"]
        raw = _raw(case["nchans"], n, 32, seed)
        bpass = raw.view(n, -1).sum(0) + 3.0 * n
        plan = spp.DMTPlan(d, case["nchans"], n, nbits=32)
        return {"kind": kind, "case": case, "plan": plan, "raw": raw, "bpass": bpass,
                "wts": bpass / bpass.sum(),
                "out": torch.empty((case["ndm"], plan.nvalid(n)), dtype=torch.float32,
                                   device="cuda")}
    if kind == "subband":
        h = spp.Header(nchans=1024, fch1=1400.0, foff=-0.29296875, tsamp=TSAMP, nbits=8)
        plan = SubbandPlan(h, _grid(case), nsub=32, group=16)
        srch = SubbandSearch(plan, [case["nsamps_a"], case["nsamps_b"]])
        for i, b in enumerate(srch.beams):
            synth.gauss_u8_device(b.raw.numel(), 2 * seed + i, 96.0, 12.0, out=b.raw)
        return {"kind": kind, "case": case, "search": srch}
    if kind == "snr":
        n, rows = case["n"], case["rows"]
        if case["dtype"] == "int32":  # sums of 1024 8-bit channels
            x = synth.gauss_f32_device(rows * n, seed, 98304.0, 384.0).round_().to(torch.int32)
        else:
            x = synth.gauss_f32_device(rows * n, seed, 98304.0, 384.0)
        return {"kind": kind, "case": case, "rows": x.view(rows, n)}
    if kind in ("fold", "filterbank"):
        nchans, n = case["nchans"], case["nsamps"]
        raw = _raw(nchans, n, case["nbits"], seed).cpu().numpy()
        fb = spp.ArrayFilterbank(raw, _header(nchans, case["nbits"], n))
        return {"kind": kind, "case": case, "fb": fb}
    raise ValueError(f"unknown kind {kind!r}")


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "single":
        spp.dedisperse_block(state["raw"], state["d"], case["nchans"], case["nsamps"],
                             state["out"], nbits=case["nbits"],
                             bitorder=_bitorder(case["nbits"]), delays_dev=state["dd"])
        return state["out"]
    if kind == "batch":
        return state["plan"].execute(state["raw"], case["nsamps"], state["out"])
    if kind == "zerodm":
        return state["plan"].execute_zero_dm(state["raw"], case["nsamps"], state["bpass"],
                                             state["wts"], state["out"])
    if kind == "subband":
        srch = state["search"]
        srch.run()
        return {"dmt": [b.dmt for b in srch.beams], "snr": [b.snr for b in srch.beams],
                "idx": [b.idx for b in srch.beams]}
    if kind == "snr":
        snr, idx = boxcar_snr(state["rows"], widths=WIDTHS[:case["nwidths"]],
                              factors=(1, 2, 4)[:case["nfactors"]], loc_scale=case["loc_scale"])
        return {"snr": snr, "idx": idx}
    if kind == "fold":
        return state["fb"].fold(case["period"], case["dm"]).data
    return state["fb"].dedisperse(case["dm"]).data


# ---------------------------------------------------------------------------
# the work of one pass: each input read once, each output written once
# ---------------------------------------------------------------------------
def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("single", "filterbank", "fold"):
        nchans, n = case["nchans"], case["nsamps"]
        dmax = int(_delays(_header(nchans, case["nbits"]), case["dm"]).max())
        out = 4 * 50 * 32 * 32 if kind == "fold" else 4 * (n - dmax)
        return {"bytes": n * nchans * case["nbits"] / 8 + out, "flops": float((n - dmax) * nchans)}
    if kind in ("batch", "zerodm"):
        nbits = case.get("nbits", 32)
        nchans, n = case["nchans"], case["nsamps"]
        nv = n - int(_delays(_header(nchans, nbits), _grid(case)).max())
        return {"bytes": n * nchans * nbits / 8 + 4.0 * case["ndm"] * nv,
                "flops": float(case["ndm"]) * nv * nchans}
    if kind == "subband":
        h = spp.Header(nchans=1024, fch1=1400.0, foff=-0.29296875, tsamp=TSAMP, nbits=8)
        p = SubbandPlan(h, _grid(case), nsub=32, group=16)
        b = f = 0.0
        for n in (case["nsamps_a"], case["nsamps_b"]):
            nv = p.nvalid(n)
            b += 1024.0 * n + 4.0 * p.ndm * nv + p.ndm * 3 * 9 * 8
            f += 1024.0 * p.ngroups * n + 32.0 * p.ndm * nv + 2.0 * p.ndm * nv * 9 * 1.75
        return {"bytes": b, "flops": f}
    rows, n, nw = case["rows"], case["n"], case["nwidths"]
    fac = sum(1.0 / f for f in (1, 2, 4)[:case["nfactors"]])
    return {"bytes": 4.0 * rows * n + 8.0 * rows * case["nfactors"] * nw,
            "flops": 2.0 * rows * n * nw * fac}


# ---------------------------------------------------------------------------
# the same results in 64 bits, by plain torch / numpy
# ---------------------------------------------------------------------------
def _unpacked(raw: torch.Tensor, nchans: int, nbits: int) -> torch.Tensor:
    """(nsamps, nchans) samples of a packed block."""
    if nbits == 32:
        return raw.view(torch.float32).view(-1, nchans)
    if nbits == 8:
        return raw.view(-1, nchans)
    per = 8 // nbits
    sh = [k * nbits for k in range(per)]
    if nbits != 1:
        sh = sh[::-1]
    return torch.stack([(raw >> s) & ((1 << nbits) - 1) for s in sh], dim=1).view(-1, nchans)


def _sum_rows(x: torch.Tensor, d: np.ndarray, nv: int, scale=None) -> torch.Tensor:
    """out[i][t] = sum_c x[t + d[i][c]][c] in float64 (scale: x -> float64 column)."""
    out = torch.zeros((d.shape[0], nv), dtype=torch.float64, device=x.device)
    for c in range(x.shape[1]):
        col = x[:, c].double() if scale is None else scale(x[:, c], c)
        for i in range(d.shape[0]):
            a = int(d[i, c])
            out[i] += col[a:a + nv]
    return out


def _exact_snr(x: torch.Tensor, case: dict) -> torch.Tensor:
    rows = []
    for f in (1, 2, 4)[:case["nfactors"]]:
        m = x.shape[1] // f
        y = x[:, :m * f].double().view(x.shape[0], m, f).mean(2)
        if case["loc_scale"] == "mean_std":
            loc, sc = y.mean(1), y.std(1, unbiased=False)
        else:
            s = y.sort(1).values
            q = []
            for p in (0.25, 0.5, 0.75):
                v = (m - 1) * p
                lo = int(math.floor(v))
                hi = min(lo + 1, m - 1)
                q.append(s[:, lo] + (s[:, hi] - s[:, lo]) * (v - lo))
            loc, sc = q[1], (q[2] - q[0]) / 1.3489795003921634
        cs = torch.cat([torch.zeros_like(y[:, :1]), y.cumsum(1)], 1)
        peaks = [((cs[:, w:] - cs[:, :-w]).max(1).values - w * loc) / (sc * math.sqrt(w))
                 for w in WIDTHS[:case["nwidths"]]]
        rows.append(torch.stack(peaks, 1))
    return torch.stack(rows, 1)


def _exact_fold(state: dict, case: dict) -> np.ndarray:
    nchans, n = case["nchans"], case["nsamps"]
    h = state["fb"].header
    nbins, nints, nbands = 50, 32, 32
    d = _delays(h, case["dm"])[0].astype(np.int64)
    dmax = int(d.max())
    gulp = max(2 * dmax, 16384)
    x = _unpacked(torch.from_numpy(state["fb"]._raw), nchans, case["nbits"]).numpy()
    band = np.array([int(c // (nchans / nbands)) for c in range(nchans)])
    tsamp, period = float(np.float32(h.tsamp)), float(np.float32(case["period"]))
    cells = np.zeros(nints * nbands * nbins)
    count = np.zeros_like(cells)
    step = min(gulp, n) - dmax
    nblk, last = divmod(n, step)
    if last < dmax:
        nblk -= 1
        last = n - nblk * step
    blocks = [(i, min(gulp, n)) for i in range(nblk)] + ([(nblk, last)] if last else [])
    for i, ns in blocks:
        if ns - dmax <= 0:
            continue
        t = np.arange(ns - dmax, dtype=np.int64)
        s = t + i * (gulp - dmax)
        tj = s.astype(np.float64) * tsamp
        phase = nbins * tj * (1.0 + 0.0) / period + 0.5
        pb = np.abs(phase.astype(np.int64)) % nbins
        sub = np.floor_divide(s.astype(np.float64), n / nints)
        pos = (sub * nbins * nbands + pb).astype(np.int64)
        first = i * step
        for c in range(nchans):
            p = pos + band[c] * nbins
            v = x[first + t + d[c], c]
            cells += np.bincount(p, weights=v, minlength=cells.size)
            count += np.bincount(p, minlength=cells.size)
    with np.errstate(divide="ignore", invalid="ignore"):
        return (cells / count).reshape(nints, nbands, nbins)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("batch", "subband"):  # whole numbers (and S/N of them, too long to redo in 64 bits)
        return None
    if kind == "zerodm" and case["ndm"] * case["nchans"] > 300000:
        return None
    st = prepare(case, seed)
    if kind == "single":
        x = _unpacked(st["raw"], case["nchans"], case["nbits"])
        return _sum_rows(x, st["d"][None, :], st["out"].numel())[0]
    if kind == "filterbank":
        x = _unpacked(torch.from_numpy(st["fb"]._raw).cuda(), case["nchans"], case["nbits"])
        d = _delays(st["fb"].header, case["dm"])
        return _sum_rows(x, d, case["nsamps"] - int(d.max()))[0].cpu().numpy()
    if kind == "zerodm":
        x = st["raw"].view(-1, case["nchans"])
        z = x.double().sum(1)
        w, b = st["wts"].double(), st["bpass"].double()
        return _sum_rows(x, st["plan"].delays, st["out"].shape[1],
                         lambda col, c: col.double() - z * w[c] + b[c])
    if kind == "snr":
        return {"snr": _exact_snr(st["rows"], case), "idx": None}
    return _exact_fold(st, case)
