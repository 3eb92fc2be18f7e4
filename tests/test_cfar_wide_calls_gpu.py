"""Calls of many CFAR cells take several frames a thread, calls of few one.
Both run every sum in the same order, so a long call and the same frames in
short calls give the same hit masks, events (their times to the rounding of
each call's own start), counters and last frame bit for bit: every statistic,
k_frames that are and are not a power of two, bin counts and frame counts that
leave partial CTAs and frame groups, a mask, several passes of the ring."""

from __future__ import annotations

import numpy as np
import pytest

import atkdsp_b200 as ak

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("mode,k,nbins,frames,n_ref,units", [
    ("ca", 4, 4096, 1021, 16, "db"), ("ca", 3, 4095, 300, 5, "db"), ("ca", 1, 1000, 3001, 16, "linear"),
    ("go", 8, 2048, 777, 16, "db"), ("so", 2, 1000, 2402, 7, "linear"), ("go", 5, 4096, 259, 4, "db"),
    ("os", 4, 2048, 601, 16, "db"), ("os", 1, 512, 2403, 40, "linear")])
def test_long_calls_equal_short_ones(mode, k, nbins, frames, n_ref, units):
    from atkdsp_b200 import gpu
    rng = np.random.default_rng(nbins + frames)
    p = rng.exponential(1.0, (frames, nbins))
    for _ in range(12):
        b, f = int(rng.integers(0, nbins - 6)), int(rng.integers(0, frames - 60))
        p[f:f + int(rng.integers(8, 60)), b:b + int(rng.integers(1, 6))] *= 300.0
    x = torch.from_numpy((10 * np.log10(p) if units == "db" else p).astype(np.float32)).cuda()
    mask = np.zeros(nbins, np.uint8)
    mask[nbins // 3:nbins // 3 + 9] = 1
    got = []
    for step in (frames, 23):
        c = ak.Cfar(nbins, mode=mode, k_frames=k, n_ref=n_ref)
        c.set_mask(mask)
        evs, hits = [], []
        for a in range(0, frames, step):
            ev, h = gpu.cfar_process(c, x[a:a + step], a * 1e-3, 1e-3, units=units, hits=True)
            evs += ev
            hits.append(h.cpu().numpy())
        got.append((evs, np.concatenate(hits), c.stats(), c.last()))
    (ea, ha, sa, la), (eb, hb, sb, lb) = got
    assert np.array_equal(ha, hb) and ha.sum() > 0
    assert sa == sb and len(ea) == len(eb) and len(ea) > 0
    for u, v in zip(ea, eb):
        for key in u:
            if key in ("t0", "t1"):
                assert np.allclose(u[key], v[key], rtol=0, atol=1e-9, equal_nan=True), key
            else:
                assert np.array_equal(u[key], v[key], equal_nan=True), key
    for u, v in zip(la, lb):
        assert np.array_equal(u, v, equal_nan=True)
