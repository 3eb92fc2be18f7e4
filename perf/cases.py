"""Performance cases of the channelizer: what a program that uses it asks of it.

Each case is one pass through a public entry point, on synthetic inputs made
from a seed (complex Gaussian noise plus tones, as the receivers deliver).
``listed`` holds the named cases, ``draw`` further ones of the same ranges;
``prepare`` / ``run`` make and use what a program keeps (handles, buffers),
``work`` counts the bytes and operations a pass cannot do without, ``exact``
gives a pass's outputs in 64 bits by plain torch / numpy.

Kinds:
  host      the drop-in call on host memory, a live stream in uneven blocks
  stream    one device-resident block of one handle (cf32 or raw int16 I/Q)
  front     block mean, raw block through the filterbank, W1 / W2 fused
  array     a coherent element array, then W1 / W2 over its block
  batch     many uneven streams in one launch
  served    one round of the serving loop
  extract   the overlap-save extractor, device buffers
  spectrum  the display reduction (one line, or the four statistics)
  cfar      the detector and burst tracker over a run of frames
"""

from __future__ import annotations

import ctypes
import math
import random

import numpy as np
import torch

import atkdsp_b200 as ak
from atkdsp_b200 import gpu
from atkdsp_b200.serve import Server

#: stopband that gives Kaiser beta 8 (the single-stream configuration)
ATTEN_BETA8 = 8.0 / 0.1102 + 8.7
ATTEN = 80.0
FS = 2.4e6
FRONT_FS = 40e6
EXTRACT_FS = 61.44e6
SCALE = {"ci16": 1.0 / 32768.0, "ci16q11": 1.0 / 2048.0}


def listed() -> list:
    return [
        # a live narrow-band stream through the drop-in host call, in the
        # uneven blocks a driver hands over: latency and launches count
        {"name": "host_blocks", "kind": "host", "nchan": 64, "os": 1, "taps": 16, "blocks": "1,999,4096,7"},
        # one short device block (about 14 ms at 2.4 MS/s): a launch and one
        # tile's latency
        {"name": "stream_short", "kind": "stream", "nchan": 256, "os": 2, "taps": 12, "n": 32768, "fmt": "cf32"},
        # a long recording's block on the device, ragged against the hop
        {"name": "stream_long", "kind": "stream", "nchan": 1024, "os": 2, "taps": 16, "n": 8388301, "fmt": "cf32"},
        # the widest in-tile filterbank, ragged block
        {"name": "stream_wide", "kind": "stream", "nchan": 4096, "os": 2, "taps": 12, "n": 2097911, "fmt": "cf32"},
        # a channel grid that is no power of two (1000 channels), the generic path
        {"name": "odd_channels", "kind": "stream", "nchan": 1000, "os": 2, "taps": 12, "n": 500003, "fmt": "cf32"},
        # the 40 MS/s receiver's 50 ms block: 12-bit samples, DC estimate,
        # 1024 channels, per-channel powers
        {"name": "front_end", "kind": "front", "nchan": 1024, "os": 2, "taps": 12, "n": 2000000, "fmt": "ci16q11"},
        # eight coherent elements, covariance and power per channel
        {"name": "array", "kind": "array", "nchan": 2048, "os": 2, "taps": 16, "nel": 8, "n": 524288},
        # uneven independent streams, nchan 64..4096, one launch for all
        {"name": "batch_uneven", "kind": "batch", "streams": 64, "min_log2": 14, "max_log2": 22, "plan": 4},
        # one serving round: a 1.6 ms int16 block of each live stream
        {"name": "served_round", "kind": "served", "streams": 256, "plan": 5},
        # 64 channels of mixed widths from one 61.44 MS/s stream
        {"name": "extractor", "kind": "extract", "nfft": 4096, "channels": 64, "nel": 1, "n": 1048576, "plan": 9},
        # the display's statistics over a long block, half-overlapped Hann frames
        {"name": "spectrum", "kind": "spectrum", "nfft": 4096, "hop": 2048, "n": 16777216, "op": "stats"},
        # W3 gating: 1024 lines of 4096 bins, hit masks kept on the device
        {"name": "cfar", "kind": "cfar", "nbins": 4096, "frames": 1024, "mode": "ca", "k_frames": 4},
    ]


def _log_int(rng: random.Random, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["host", "stream", "stream", "stream", "odd", "front", "array", "batch", "served", "extract",
                       "spectrum", "cfar"])
    taps = rng.choice([8, 12, 16])
    if kind == "host":
        blocks = [_log_int(rng, 64, 65536) for _ in range(3)]
        return {"kind": "host", "nchan": rng.choice([16, 64, 128, 256, 1024]), "os": rng.choice([1, 2]), "taps": taps,
                "blocks": ",".join(str(b) for b in blocks)}
    if kind == "stream":
        return {"kind": "stream", "nchan": 1 << rng.randint(4, 12), "os": rng.choice([1, 2, 2, 4]), "taps": taps,
                "n": _log_int(rng, 1 << 14, 1 << 22), "fmt": rng.choice(["cf32", "cf32", "ci16"])}
    if kind == "odd":
        nchan = rng.choice([24, 60, 96, 192, 200, 640, 800, 1000, 1920, 3000, 6000])
        return {"kind": "stream", "nchan": nchan, "os": rng.choice([1, 2]), "taps": taps,
                "n": _log_int(rng, 1 << 14, 1 << 19), "fmt": "cf32"}
    if kind == "front":
        return {"kind": "front", "nchan": rng.choice([256, 512, 1024, 2048]), "os": rng.choice([1, 2]), "taps": taps,
                "n": _log_int(rng, 200000, 4000000), "fmt": rng.choice(["ci16", "ci16q11"])}
    if kind == "array":
        return {"kind": "array", "nchan": rng.choice([256, 1024, 2048]), "os": rng.choice([1, 2]), "taps": taps,
                "nel": rng.randint(2, 8), "n": _log_int(rng, 1 << 16, 1 << 19)}
    if kind == "batch":
        return {"kind": "batch", "streams": rng.randint(8, 64), "min_log2": 14, "max_log2": rng.choice([16, 18, 20, 21]),
                "plan": rng.randrange(1 << 16)}
    if kind == "served":
        return {"kind": "served", "streams": _log_int(rng, 16, 256), "plan": rng.randrange(1 << 16)}
    if kind == "extract":
        return {"kind": "extract", "nfft": rng.choice([1024, 2048, 4096]), "channels": rng.randint(4, 64),
                "nel": rng.choice([1, 1, 2]), "n": _log_int(rng, 1 << 16, 1 << 19), "plan": rng.randrange(1 << 16)}
    if kind == "spectrum":
        nfft = 1 << rng.randint(8, 12)
        return {"kind": "spectrum", "nfft": nfft, "hop": rng.choice([nfft, nfft // 2, nfft // 4 + 3]),
                "n": _log_int(rng, 1 << 17, 1 << 23), "op": rng.choice(["stats", "avg", "max"])}
    return {"kind": "cfar", "nbins": rng.choice([256, 1000, 1024, 2048, 4096]), "frames": _log_int(rng, 16, 1024),
            "mode": rng.choice(["ca", "os", "go", "so"]), "k_frames": rng.choice([1, 4])}


# ---- inputs ------------------------------------------------------------------
def _dev() -> torch.device:
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed: int) -> torch.Generator:
    g = torch.Generator(device=_dev())
    g.manual_seed(int(seed))
    return g


def _signal(n: int, seed: int, ntones: int = 3, amp: float = 10.0) -> torch.Tensor:
    """Unit-variance complex noise and ntones tones, complex64 on the device."""
    x = torch.randn(n, dtype=torch.complex64, device=_dev(), generator=_gen(seed))
    rng = np.random.default_rng([int(seed), 7])
    t = torch.arange(n, device=x.device, dtype=torch.float64)
    for _ in range(ntones):
        f, ph = float(rng.uniform(-0.5, 0.5)), float(rng.uniform(0, 2 * math.pi))
        a = 2 * math.pi * (torch.frac(f * t) + ph / (2 * math.pi))
        x += torch.polar(torch.full_like(a, amp), a).to(torch.complex64)
    return x


def _raw(n: int, seed: int, fmt: str) -> torch.Tensor:
    """(2n,) int16 I/Q: noise, tones and a DC offset, at the format's scale."""
    full = 2047.0 if fmt == "ci16q11" else 32767.0
    x = torch.view_as_real(_signal(n, seed, 8 if fmt == "ci16q11" else 2, 3.0)) * (full / 40.0)
    x = x + torch.tensor([full * 0.058, -full * 0.039], device=x.device)
    return torch.clamp(torch.round(x), -full - 1, full).to(torch.int16).reshape(-1).contiguous()


def _plan_batch(case: dict) -> list:
    """(nchan, taps, length) per stream."""
    rng = np.random.default_rng(int(case["plan"]))
    return [(int(rng.choice([64, 256, 1024, 4096])), int(rng.choice([8, 12, 16])),
             int(2.0 ** rng.uniform(case["min_log2"], case["max_log2"]))) for _ in range(case["streams"])]


def _plan_served(case: dict) -> list:
    """(rate, nchan, block samples) per stream: 1.6 ms at the stream's rate."""
    rng = np.random.default_rng(int(case["plan"]))
    out = []
    for _ in range(case["streams"]):
        rate = float(rng.choice([2.4e6, 10e6, 40e6]))
        out.append((rate, int(rng.choice([256, 1024])), int(round(rate * 1.6e-3))))
    return out


def _plan_extract(case: dict) -> list:
    """(offset_hz, bw_hz, out_rate): odd channels land at their decimated
    rate, even ones through the arbitrary resampler."""
    rng = np.random.default_rng(int(case["plan"]))
    bws = (60e3, 120e3, 240e3, 960e3) if case["nfft"] < 4096 else (12.5e3, 25e3, 50e3, 200e3)
    return [(float(rng.uniform(-0.45, 0.45) * EXTRACT_FS), bws[i % 4], bws[i % 4] * (1.25 if i % 2 else 1.0))
            for i in range(case["channels"])]


def _window(n: int) -> np.ndarray:
    return (0.5 - 0.5 * np.cos(2 * math.pi * np.arange(n) / (n - 1))).astype(np.float32)


def _frames_db(case: dict, seed: int) -> torch.Tensor:
    """Exponential noise lines with a few bursts, in dB."""
    nf, nb = case["frames"], case["nbins"]
    p = torch.empty(nf, nb, device=_dev(), dtype=torch.float32)
    p.exponential_(1.0, generator=_gen(seed))
    rng = np.random.default_rng([int(seed), 11])
    for _ in range(12):
        f0, b0 = int(rng.integers(0, nf)), int(rng.integers(0, nb - 8))
        p[f0:f0 + int(rng.integers(4, 64)), b0:b0 + int(rng.integers(1, 8))] += 60.0
    return 10.0 * torch.log10(p.clamp_min(1e-20))


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st = {"case": case}
    if kind == "host":
        blocks = [int(b) for b in case["blocks"].split(",")]
        x = _signal(sum(blocks), seed).cpu().numpy()
        st["pfb"] = ak.Pfb(FS, case["nchan"], case["os"], case["taps"], ATTEN_BETA8)
        st["x"] = [np.ascontiguousarray(b) for b in np.split(x, np.cumsum(blocks)[:-1])]
    elif kind == "stream":
        p = st["pfb"] = ak.Pfb(FS, case["nchan"], case["os"], case["taps"], ATTEN)
        st["x"] = _signal(case["n"], seed) if case["fmt"] == "cf32" else _raw(case["n"], seed, case["fmt"])
        hops = case["n"] // (case["nchan"] // case["os"]) + 1
        st["out"] = torch.zeros(p.nchan * hops, dtype=torch.complex64, device=_dev())
    elif kind == "front":
        p = st["pfb"] = ak.Pfb(FRONT_FS, case["nchan"], case["os"], case["taps"], ATTEN)
        M, dev = case["nchan"], _dev()
        st["x"] = _raw(case["n"], seed, case["fmt"])
        st["offset"] = torch.tensor(_offset(), dtype=torch.float64, device=dev)
        st["mean"] = torch.zeros(2, dtype=torch.float64, device=dev)
        st["out"] = torch.zeros(M * (case["n"] // (M // case["os"]) + 1), dtype=torch.complex64, device=dev)
        st["R"] = torch.zeros(M, 1, 1, dtype=torch.complex64, device=dev)
        st["counts"] = torch.zeros(M, dtype=torch.int32, device=dev)
        st["pwr"] = torch.zeros(1, M, dtype=torch.float32, device=dev)
        st["mean_pwr"] = torch.zeros(M, dtype=torch.float32, device=dev)
        need = int(ak.load().atkdsp_gpu_pfb_w12_scratch_bytes(p.handle, case["n"] + M))
        st["scratch"] = torch.empty(max(need, 8), dtype=torch.uint8, device=dev)
        st["stream"] = torch.cuda.Stream()
    elif kind == "array":
        p = st["pfb"] = ak.Pfb(FS, case["nchan"], case["os"], case["taps"], ATTEN, case["nel"])
        M, nel, dev = case["nchan"], case["nel"], _dev()
        st["x"] = _elements(case, seed)
        st["out"] = torch.zeros(nel * M * (case["n"] // (M // case["os"]) + 1), dtype=torch.complex64, device=dev)
        st["R"] = torch.zeros(M, nel, nel, dtype=torch.complex64, device=dev)
        st["counts"] = torch.zeros(M, dtype=torch.int32, device=dev)
        st["pwr"] = torch.zeros(nel, M, dtype=torch.float32, device=dev)
        st["mean_pwr"] = torch.zeros(M, dtype=torch.float32, device=dev)
        st["stream"] = torch.cuda.Stream()
    elif kind == "batch":
        plan = _plan_batch(case)
        st["pfbs"] = [ak.Pfb(FS, M, 2, K, ATTEN) for M, K, _ in plan]
        st["batch"] = gpu.Batch(st["pfbs"])
        x = _signal(sum(n for _, _, n in plan), seed)
        st["x"] = list(torch.split(x, [n for _, _, n in plan]))
        caps = [M * (n // (M // 2) + 1) for M, _, n in plan]
        st["out"] = torch.zeros(sum(caps), dtype=torch.complex64, device=_dev())
        st["outs"] = list(torch.split(st["out"], caps))
    elif kind == "served":
        plan = _plan_served(case)
        st["server"] = Server(max_streams=max(64, len(plan)))
        st["ids"] = [st["server"].open(rate, M, 2, 16, ATTEN, "ci16") for rate, M, _ in plan]
        x = _raw(sum(n for _, _, n in plan), seed, "ci16")
        st["x"] = list(torch.split(x, [2 * n for _, _, n in plan]))
        caps = [M * (n // (M // 2) + 1) for _, M, n in plan]
        st["out"] = torch.zeros(sum(caps), dtype=torch.complex64, device=_dev())
        st["outs"] = list(torch.split(st["out"], caps))
    elif kind == "extract":
        plan = _plan_extract(case)
        x = st["osx"] = ak.Osx(EXTRACT_FS, case["nfft"], ATTEN, case["nel"])
        for ch in plan:
            x.add(*ch)
        st["x"] = [_signal(case["n"], seed + 1000 * e, 5) for e in range(case["nel"])]
        nel, ns = case["nel"], x.channels()
        cap = max(x.out_max(c, case["n"] + case["nfft"]) for c in range(ns))
        st["out"] = torch.zeros(nel, ns, cap, dtype=torch.complex64, device=_dev())
        st["ins"] = (ctypes.c_void_p * nel)(*[t.data_ptr() for t in st["x"]])
        st["outs"] = (ctypes.c_void_p * (nel * ns))(*[st["out"][e, c].data_ptr() for e in range(nel) for c in range(ns)])
        st["counts"] = (ctypes.c_size_t * ns)()
        st["cap"] = cap
    elif kind == "spectrum":
        st["spec"] = gpu.Spectrum(case["nfft"])
        st["x"] = _signal(case["n"], seed, 5)
        st["win"] = torch.from_numpy(_window(case["nfft"])).to(_dev())
    elif kind == "cfar":
        st["cfar"] = ak.Cfar(case["nbins"], mode=case["mode"], k_frames=case["k_frames"])
        st["x"] = _frames_db(case, seed)
        st["t"] = 0.0
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return st


def _offset() -> tuple:
    """The running DC estimate a front end holds, as float32 values."""
    return (0.0546875, -0.03515625)


def _elements(case: dict, seed: int) -> list:
    """Common tones with a phase per element, independent noise."""
    rng = np.random.default_rng([int(seed), 3])
    common = _signal(case["n"], seed, 4, 3.0)
    return [(common * complex(np.exp(2j * np.pi * rng.uniform())) +
             torch.randn(case["n"], dtype=torch.complex64, device=_dev(), generator=_gen(seed + 77 + e)))
            for e in range(case["nel"])]


# ---- one pass ------------------------------------------------------------------
def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "host":
        return [st["pfb"].process(b) for b in st["x"]]
    if kind == "stream":
        if case["fmt"] == "cf32":
            return gpu.process_n(st["pfb"], [st["x"]], 1, out=st["out"])
        return gpu.process_n_raw(st["pfb"], [st["x"]], 1, case["fmt"], 0.0546875 - 0.03515625j, out=st["out"])
    if kind == "front":
        s = st["stream"]
        y = gpu.process_w12(st["pfb"], st["x"], case["fmt"], st["offset"], out=st["out"], R=st["R"],
                            counts=st["counts"], pwr=st["pwr"], mean_pwr=st["mean_pwr"], scratch=st["scratch"],
                            stream=s)
        mean = gpu.block_mean(st["x"], case["fmt"], st["offset"], st["mean"], stream=s)
        return {"y": y, "R": st["R"], "counts": st["counts"], "pwr": st["pwr"], "mean_pwr": st["mean_pwr"],
                "mean": mean}
    if kind == "array":
        s, nel = st["stream"], case["nel"]
        y = gpu.process_n(st["pfb"], st["x"], nel, out=st["out"], stream=s)
        gpu.accumulate(y, nel, case["nchan"], st["R"], st["counts"], st["pwr"], st["mean_pwr"], stream=s)
        return {"y": y, "R": st["R"], "counts": st["counts"], "pwr": st["pwr"], "mean_pwr": st["mean_pwr"]}
    if kind == "batch":
        st["batch"].process(st["x"], st["outs"])
        return st["out"]
    if kind == "served":
        srv = st["server"]
        for sid, x, o in zip(st["ids"], st["x"], st["outs"]):
            srv.submit(sid, x, o)
        srv.drain()
        return st["out"]
    if kind == "extract":
        x = st["osx"]
        rc = ak.load().atkdsp_gpu_osx_process_n(x.handle, st["ins"], case["nel"], case["n"], st["outs"], st["counts"],
                                                st["cap"])
        if rc < 0:
            raise RuntimeError(f"extractor: {rc}")
        return {"y": st["out"], "counts": [int(c) for c in st["counts"]][:32]}
    if kind == "spectrum":
        if case["op"] == "stats":
            return st["spec"].stats(st["x"], case["hop"], st["win"])
        line, frames = st["spec"].reduce(st["x"], case["hop"], st["win"], case["op"])
        return {"line": line, "frames": frames}
    ev, hits = gpu.cfar_process(st["cfar"], st["x"], st["t"], 1e-3, hits=True)
    st["t"] += case["frames"] * 1e-3
    whole = _rows([[e["type"], e["id"], e["flags"], e["lo"], e["hi"], e["n_hits"]] for e in ev], 6, np.int64)
    times = _rows([[e["t0"], e["t1"]] for e in ev], 2, np.float64)
    levels = _rows([[e["fc_bin"], e["level_db"], e["noise_db"], e["snr_db"], e["band_snr_db"]] for e in ev], 5,
                   np.float32)
    return {"hits": hits, "n_events": len(ev), "events": whole, "times": times, "levels": levels}


def _rows(rows: list, width: int, dtype) -> np.ndarray:
    """The events' rows in a table of fixed height."""
    t = np.zeros((max(2048, len(rows)), width), dtype)
    if rows:
        t[:len(rows)] = rows
    return t


# ---- what a pass cannot do without ------------------------------------------------
def _pfb_work(n: float, M: int, os: int, K: int, in_bytes: int) -> tuple:
    """n input samples: read once, os outputs each written once; the fold's
    complex-by-real products and a split-radix transform per output."""
    return n * (in_bytes + 8 * os), n * os * (4 * K + 4 * math.log2(M))


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "host":
        b, f = _pfb_work(sum(int(v) for v in case["blocks"].split(",")), case["nchan"], case["os"], case["taps"], 8)
    elif kind == "stream":
        b, f = _pfb_work(case["n"], case["nchan"], case["os"], case["taps"], 8 if case["fmt"] == "cf32" else 4)
    elif kind == "front":
        b, f = _pfb_work(case["n"], case["nchan"], case["os"], case["taps"], 4)
        f += case["n"] * (2 + 4 * case["os"])
    elif kind == "array":
        nel = case["nel"]
        b, f = _pfb_work(case["n"] * nel, case["nchan"], case["os"], case["taps"], 8)
        f += case["n"] * case["os"] * nel * (nel + 1) * 4
        b += case["nchan"] * nel * nel * 16
    elif kind == "batch":
        each = [_pfb_work(n, M, 2, K, 8) for M, K, n in _plan_batch(case)]
        b, f = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind == "served":
        each = [_pfb_work(n, M, 2, 16, 4) for _, M, n in _plan_served(case)]
        b, f = sum(e[0] for e in each), sum(e[1] for e in each)
    elif kind == "extract":
        nel, nfft, n = case["nel"], case["nfft"], case["n"]
        b, f = nel * n * 8.0, nel * 2.0 * n * 4 * math.log2(nfft)
        for _, bw, rate in _plan_extract(case):
            b += nel * 8.0 * n * rate / EXTRACT_FS
            f += nel * 2.0 * n * 8
    elif kind == "spectrum":
        frames = (case["n"] - case["nfft"]) // case["hop"] + 1
        b = case["n"] * 8.0 + case["nfft"] * 16.0
        f = frames * case["nfft"] * (4.0 * math.log2(case["nfft"]) + 8)
    else:
        cells = case["frames"] * case["nbins"]
        b, f = cells * 5.0, cells * 2.0 * 32
    return {"bytes": float(b), "flops": float(f)}


# ---- the outputs in 64 bits ---------------------------------------------------------
def _kaiser_beta(atten: float) -> float:
    return 0.1102 * (atten - 8.7) if atten > 50 else 0.5842 * (atten - 21) ** 0.4 + 0.07886 * (atten - 21)


def _sinc_kaiser(n: int, fc: float, atten: float) -> np.ndarray:
    mid = (n - 1) * 0.5
    t = np.arange(n) - mid
    beta = _kaiser_beta(atten)
    w = np.i0(beta * np.sqrt(np.maximum(0.0, 1.0 - (t / mid) ** 2))) / np.i0(beta)
    h = 2 * fc * np.sinc(2 * fc * t) * w
    return h / h.sum()


def _pfb64(x: torch.Tensor, M: int, os: int, K: int, atten: float) -> torch.Tensor:
    """A fresh handle's output (M, m) for x, in complex128."""
    hop, L, dev = M // os, M * K, x.device
    h = torch.from_numpy(_sinc_kaiser(L, 0.5 / M, atten) * M).to(dev)
    s = torch.cat([torch.zeros(L - hop, dtype=torch.complex128, device=dev), x.to(torch.complex128)])
    m = x.numel() // hop
    out = torch.zeros(M, m, dtype=torch.complex128, device=dev)
    if m == 0:
        return out
    k = torch.arange(M, device=dev)
    rot = torch.polar(torch.ones(M, dtype=torch.float64, device=dev), -2 * math.pi * k.double() / M)
    frames = s.unfold(0, L, hop)[:m]
    step = max(1, (1 << 25) // L)
    for c0 in range(0, m, step):
        seg = frames[c0:c0 + step]
        X = torch.fft.fft((seg * h).view(seg.shape[0], K, M).sum(1), dim=1)
        shift = ((torch.arange(c0, c0 + seg.shape[0], device=dev) + 1) * hop) % M
        out[:, c0:c0 + seg.shape[0]] = (X * rot[(k[None, :] * shift[:, None]) % M]).T
    return out


def _unpack64(raw: torch.Tensor, fmt: str, offset: complex = 0j) -> torch.Tensor:
    v = raw.to(torch.float64).view(-1, 2) * SCALE[fmt]
    return torch.complex(v[:, 0], v[:, 1]) - offset


def _flat64(ys: list, caps: list) -> torch.Tensor:
    out = torch.zeros(sum(caps), dtype=torch.complex128, device=_dev())
    for y, o in zip(ys, torch.split(out, caps)):
        o[:y.numel()] = y.reshape(-1)
    return out


def _powers64(y: torch.Tensor) -> tuple:
    """(R, pwr, mean_pwr) of a (nel, M, m) block."""
    R = torch.einsum("akm,bkm->kab", y, y.conj())
    pwr = (y.abs() ** 2).mean(-1)
    return R, pwr, pwr.mean(0)


def _extract64(case: dict, seed: int) -> torch.Tensor:
    nfft, nel, n, dev = case["nfft"], case["nel"], case["n"], _dev()
    ov = hop = nfft // 2
    m = n // hop
    plan = _plan_extract(case)
    cap = max(int((n + nfft) * rate / EXTRACT_FS) + 64 for _, _, rate in plan)
    out = torch.zeros(nel, len(plan), cap, dtype=torch.complex128, device=dev)
    for e in range(nel):
        x = _signal(n, seed + 1000 * e, 5).to(torch.complex128)
        s = torch.cat([torch.zeros(ov, dtype=torch.complex128, device=dev), x])
        X = torch.fft.fft(s.unfold(0, nfft, hop)[:m], dim=1)
        for c, (off, bw, rate) in enumerate(plan):
            target, d = max(rate, 1.25 * bw), 1
            while EXTRACT_FS / (2 * d) >= target and ov % (2 * d) == 0:
                d *= 2
            crate = EXTRACT_FS / d
            taps = _lowpass(0.5 * bw, min(crate - 0.5 * bw, 0.5 * EXTRACT_FS), ATTEN, EXTRACT_FS)
            if taps.size > ov + 1:
                taps = taps[:ov + 1] / taps[:ov + 1].sum()
            H = torch.fft.fft(torch.from_numpy(taps).to(dev).to(torch.complex128), n=nfft)
            sh = math.floor(off / EXTRACT_FS * nfft + 0.5)
            delta = off - sh * EXTRACT_FS / nfft
            M = nfft // d
            y = torch.fft.ifft((torch.roll(X, -sh, 1) * H).view(m, d, M).sum(1), dim=1)[:, ov // d:] / d
            i = torch.arange(m, device=dev, dtype=torch.int64)[:, None]
            k = torch.arange(M - ov // d, device=dev, dtype=torch.int64)[None, :]
            a0 = ((sh * (i * hop - ov)) % nfft).double() / nfft
            ph = -2 * math.pi * (a0 + delta * (i * hop + k * d).double() / EXTRACT_FS)
            v = (y * torch.polar(torch.ones_like(ph), ph)).reshape(-1)
            if abs(crate - rate) > 1e-6 * rate:
                v = _resample64(v, crate, rate)
            out[e, c, :v.numel()] = v
    return out


def _lowpass(fp: float, fst: float, atten: float, rate: float) -> np.ndarray:
    dw = 2 * math.pi * (fst - fp) / rate
    n = math.ceil((atten - 8.0) / (2.285 * dw)) + 1
    n = max(3, n | 1)
    return _sinc_kaiser(n, 0.5 * (fp + fst) / rate, atten)


def _resample64(v: torch.Tensor, in_rate: float, out_rate: float, P: int = 64) -> torch.Tensor:
    """The polyphase resampler (P phases, coefficients interpolated linearly)."""
    nyq = 0.5 * min(in_rate, out_rate)
    p = _lowpass(0.8 * nyq, nyq, ATTEN, in_rate * P) * P
    Q = -(-p.size // P)
    p = torch.from_numpy(np.concatenate([p, np.zeros(P * Q + 1 - p.size)])).to(v.device)
    step = in_rate / out_rate
    K = torch.arange(int(v.numel() / step) + 2, device=v.device, dtype=torch.float64)
    pos = K * step
    pos = pos[pos < v.numel()]
    i = torch.floor(pos)
    ph = (pos - i) * P
    b = torch.clamp(ph.long(), max=P - 1)
    mu = ph - b
    pad = torch.cat([torch.zeros(Q, dtype=v.dtype, device=v.device), v])
    y = torch.zeros(pos.numel(), dtype=torch.complex128, device=v.device)
    for q in range(Q):
        c = p[b + q * P] * (1 - mu) + p[b + q * P + 1] * mu
        y += c * pad[i.long() - q + Q]
    return y


def _spectrum64(case: dict, seed: int) -> dict:
    nfft, hop = case["nfft"], case["hop"]
    x = _signal(case["n"], seed, 5)
    w = torch.from_numpy(_window(nfft).astype(np.float64)).to(x.device)
    fr = x.unfold(0, nfft, hop)
    F = fr.shape[0]
    mx = torch.zeros(nfft, dtype=torch.float64, device=x.device)
    mn = torch.full_like(mx, float("inf"))
    su, s2 = torch.zeros_like(mx), torch.zeros_like(mx)
    for c0 in range(0, F, 1024):
        X = torch.fft.fftshift(torch.fft.fft(fr[c0:c0 + 1024].to(torch.complex128) * w, dim=1), dim=1)
        p = (X.abs() / nfft) ** 2
        mx = torch.maximum(mx, p.max(0).values)
        mn = torch.minimum(mn, p.min(0).values)
        su += p.sum(0)
        s2 += (p * p).sum(0)
    db = lambda v: 10 * torch.log10(v + 1e-12)  # noqa: E731
    amp_db = lambda v: 20 * torch.log10(torch.sqrt(v) + 1e-12)  # noqa: E731
    if case["op"] == "stats":
        return {"max": db(mx), "avg": db(su / F), "min": db(mn), "sk": F * s2 / (su * su), "frames": None}
    return {"line": amp_db(mx if case["op"] == "max" else su / F), "frames": None}


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "host":
        blocks = [int(b) for b in case["blocks"].split(",")]
        hop = case["nchan"] // case["os"]
        y = _pfb64(_signal(sum(blocks), seed), case["nchan"], case["os"], case["taps"], ATTEN_BETA8).cpu()
        ends = [0] + [int(e) // hop for e in np.cumsum(blocks)]
        return [y[:, a:b].contiguous() for a, b in zip(ends, ends[1:])]
    if kind == "stream":
        x = _signal(case["n"], seed) if case["fmt"] == "cf32" else \
            _unpack64(_raw(case["n"], seed, case["fmt"]), case["fmt"], 0.0546875 - 0.03515625j)
        return _pfb64(x, case["nchan"], case["os"], case["taps"], ATTEN)[None]
    if kind == "front":
        x = _unpack64(_raw(case["n"], seed, case["fmt"]), case["fmt"])
        y = _pfb64(x - complex(*_offset()), case["nchan"], case["os"], case["taps"], ATTEN)[None]
        R, pwr, mp = _powers64(y)
        return {"y": y, "R": R, "counts": None, "pwr": pwr, "mean_pwr": mp, "mean": torch.view_as_real(x.mean())}
    if kind == "array":
        y = torch.stack([_pfb64(x, case["nchan"], case["os"], case["taps"], ATTEN) for x in _elements(case, seed)])
        R, pwr, mp = _powers64(y)
        return {"y": y, "R": R, "counts": None, "pwr": pwr, "mean_pwr": mp}
    if kind == "batch":
        plan = _plan_batch(case)
        xs = torch.split(_signal(sum(n for _, _, n in plan), seed), [n for _, _, n in plan])
        return _flat64([_pfb64(x, M, 2, K, ATTEN) for x, (M, K, _) in zip(xs, plan)],
                       [M * (n // (M // 2) + 1) for M, _, n in plan])
    if kind == "served":
        plan = _plan_served(case)
        xs = torch.split(_raw(sum(n for _, _, n in plan), seed, "ci16"), [2 * n for _, _, n in plan])
        return _flat64([_pfb64(_unpack64(x, "ci16"), M, 2, 16, ATTEN) for x, (_, M, _) in zip(xs, plan)],
                       [M * (n // (M // 2) + 1) for _, M, n in plan])
    if kind == "extract":
        return {"y": _extract64(case, seed), "counts": None}
    if kind == "spectrum":
        return _spectrum64(case, seed)
    return None
