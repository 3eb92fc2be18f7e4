"""The spectrum kernel's frame groups: a CTA works on 4096/n frames at a time
(several to a warp below n 256) and takes a run of frames that need not fill
its last turn. Frame counts around one CTA's groups, and a length for every
barrier kind, against the C oracle with the bars of test_spectrum_gpu.py; and
a NaN, which a comparison never lets in except from the first frame."""

from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _t(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n", [16, 32, 128, 256, 512, 2048, 4096])
def test_frame_counts_around_a_turn(n):
    from atkdsp_b200.gpu import Spectrum
    groups = 4096 // n
    sp = Spectrum(n)
    for frames in sorted({1, max(1, groups - 1), groups, groups + 1, 3 * groups + 2, 700}):
        rng = np.random.default_rng(n + frames)
        hop = max(1, n // 2 - 1)
        N = (frames - 1) * hop + n
        x = (rng.standard_normal(N) + 1j * rng.standard_normal(N)).astype(np.complex64)
        w = O.oracle().window("hann", n)
        for det in ("max", "min", "avg"):
            line, fr = sp.reduce(_t(x), hop, _t(w), det)
            ref, _ = O.oracle().spectrum_reduce(x, n, hop, w, det)
            assert fr == frames and np.max(np.abs(line.cpu().numpy() - ref)) <= 1e-4, (frames, det)
        st, so = sp.stats(_t(x), hop, _t(w)), O.oracle().spectrum_stats(x, n, hop, w)
        for q in ("max", "avg", "min"):
            assert np.max(np.abs(st[q].cpu().numpy() - so[q])) <= 1e-4, (frames, q)
        assert np.max(np.abs(st["sk"].cpu().numpy() - so["sk"]) / so["sk"]) <= 1e-5, frames


@pytest.mark.parametrize("n", [64, 1024])
def test_nan_frames(n):
    """A NaN in a later frame is compared away by max and min and stays in the
    average; in the first frame it stays everywhere."""
    from atkdsp_b200.gpu import Spectrum
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(40 * n) + 1j * rng.standard_normal(40 * n)).astype(np.complex64)
    sp = Spectrum(n)
    for at in (0, 17 * n + 3):
        y = x.copy()
        y[at] = np.nan
        for det in ("max", "min", "avg"):
            line, _ = sp.reduce(_t(y), n, None, det)
            ref, _ = O.oracle().spectrum_reduce(y, n, n, None, det)
            got = line.cpu().numpy()
            assert np.array_equal(np.isnan(got), np.isnan(ref)), (at, det)
            assert np.nanmax(np.abs(got - ref), initial=0.0) <= 1e-4, (at, det)


@pytest.mark.parametrize("n", [16, 64, 256, 512, 4096])
def test_an_infinite_sample_reaches_every_bin(n):
    """A sample whose index is a multiple of n/8 meets only +-1, +-i and W8
    before the additions (leg 0 of every later pass), so no 0 x infinity
    arises: every bin of its frame is infinite, as the transform's sum is."""
    from atkdsp_b200.gpu import Spectrum
    rng = np.random.default_rng(n)
    x = (rng.standard_normal(9 * n) + 1j * rng.standard_normal(9 * n)).astype(np.complex64)
    sp = Spectrum(n)
    for at in (0, n // 8, n // 2, 7 * n // 8):
        y = x.copy()
        y[4 * n + at] = np.inf
        for det in ("max", "avg"):
            line, _ = sp.reduce(_t(y), n, None, det)
            assert np.all(np.isposinf(line.cpu().numpy())), (at, det)
        line, _ = sp.reduce(_t(y), n, None, "min")
        assert np.all(np.isfinite(line.cpu().numpy())), at
        st = sp.stats(_t(y), n, None)
        assert np.all(np.isposinf(st["max"].cpu().numpy())) and np.all(np.isfinite(st["min"].cpu().numpy())), at
