"""The extractor's fold takes its filter values in batches of eight and wraps
the spectrum's address; the resampler takes its taps in batches of eight up to
the kept history. Channels whose decimation is below one batch, one batch and
many, with frequency offsets that put the spectrum's wrap inside and between
batches, at nfft 64 to 4096, one block at a time and several: against the C
oracle within the extractor's bar."""

from __future__ import annotations

import numpy as np
import pytest

import atkdsp_b200 as ak
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FS = 1.024e6


@pytest.mark.parametrize("nfft", [64, 256, 1024, 4096])
@pytest.mark.parametrize("resampled", [False, True])
def test_channels_of_every_decimation(nfft, resampled):
    rng = np.random.default_rng(nfft + resampled)
    a, b = ak.Osx(FS, nfft, 60.0), O.oracle().Osx(FS, nfft, 60.0)
    n = 0
    for lg in range(1, 12):
        bw = FS / (1.3 * 2 ** lg)
        if 2 ** lg > nfft // 2:
            break
        for off in (0.0, 0.4999 * FS, -0.31 * FS):
            rate = bw * (1.27 if resampled else 1.0)
            try:
                b.add(off, bw, rate)
            except RuntimeError:
                with pytest.raises(ak.AtkDspError):
                    a.add(off, bw, rate)
                continue
            a.add(off, bw, rate)
            n += 1
    assert n >= 9
    got, want = [[] for _ in range(n)], [[] for _ in range(n)]
    for m in (nfft, 5 * nfft + 3, nfft // 2, 9 * nfft):
        x = (rng.standard_normal(m) + 1j * rng.standard_normal(m)).astype(np.complex64)
        for y, all_ in ((a.process_n([x], 1), got), (b.process_n([x], 1), want)):
            outs, cnts = y
            for c in range(n):
                all_[c].append(np.asarray(outs[c])[0][:cnts[c]])
    for c in range(n):
        u, v = np.concatenate(got[c]), np.concatenate(want[c])
        assert u.shape == v.shape, c
        assert np.max(np.abs(u - v), initial=0.0) <= 1e-5 * np.max(np.abs(v), initial=1e-30), c
