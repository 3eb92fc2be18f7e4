"""W1 / W2 of 2 to 8 elements go through the FP64 matrix instruction, 2 and 4
elements with several hop groups stacked in its rows. Against sums in extended
precision at the edges of its steps and of the warps' runs, each part of each
entry within one float rounding plus m double roundings of the products'
magnitudes (the sums are double, rounded once); coherent elements, whose
imaginary parts cancel; gated channels untouched; accumulation over two calls;
the power-only call; infinities and NaN where the products have them."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _sums(y):
    r, i = y.real.astype(np.longdouble), y.imag.astype(np.longdouble)
    re = np.einsum("akm,bkm->kab", r, r) + np.einsum("akm,bkm->kab", i, i)
    im = np.einsum("akm,bkm->kab", i, r) - np.einsum("akm,bkm->kab", r, i)
    mag = np.einsum("akm,bkm->kab", np.abs(r) + np.abs(i), np.abs(r) + np.abs(i))
    return re, im, mag


def _close(got, ref, mag, m):
    bar = 2.0 ** -24 * np.abs(ref) * (1 + 1e-6) + (m + 16) * 2.0 ** -52 * mag + 1e-45
    assert (np.abs(got.astype(np.longdouble) - ref) <= bar).all()


@pytest.mark.parametrize("coherent", [False, True])
@pytest.mark.parametrize("nel,M,ms", [(2, 24, (1, 15, 17, 513)), (3, 17, (3, 8, 33, 255)), (4, 600, (7, 129)),
                                      (5, 16, (4, 31, 2049)), (7, 33, (32, 127)), (8, 513, (5, 128, 301)),
                                      (8, 16, (6000,))])
def test_against_extended_precision(nel, M, ms, coherent):
    from atkdsp_b200 import gpu
    for m in ms:
        rng = np.random.default_rng(nel * 1000 + m)
        y = rng.standard_normal((nel, M, m)) + 1j * rng.standard_normal((nel, M, m))
        if coherent:
            y = y[:1] * rng.uniform(0.5, 2.0, (nel, M, 1)) + 1e-6 * y
        y = y.astype(np.complex64)
        gate = (rng.random(M) < 0.7).astype(np.uint8)
        d, dg = torch.from_numpy(y).cuda(), torch.from_numpy(gate).cuda()
        R = torch.zeros(M, nel, nel, dtype=torch.complex64, device="cuda")
        c = torch.zeros(M, dtype=torch.int32, device="cuda")
        gpu.cov_accumulate(d, nel, M, dg, R, c)
        torch.cuda.synchronize()
        got, re, im, mag = R.cpu().numpy(), *_sums(y)
        on = gate.astype(bool)
        assert not got[~on].any() and np.array_equal(c.cpu().numpy(), np.where(on, m, 0))
        _close(got.real[on], re[on], mag[on], m)
        _close(got.imag[on], im[on], mag[on], m)
        assert not np.diagonal(got.imag, axis1=1, axis2=2).any()
        gpu.cov_accumulate(d, nel, M, dg, R, c)
        torch.cuda.synchronize()
        again = got.astype(np.complex128) + (re + 1j * im).astype(np.complex128) * on[:, None, None]
        assert np.max(np.abs(R.cpu().numpy() - again)) <= 2e-7 * np.max(np.abs(again))
        pw, mean = gpu.channel_power(d, nel, M)
        torch.cuda.synchronize()
        pr = np.diagonal(re, axis1=1, axis2=2).T / m
        _close(pw.cpu().numpy(), pr, pr, m)
        _close(mean.cpu().numpy(), pr.mean(0), pr.mean(0), m + nel)


@pytest.mark.parametrize("nel", [2, 4, 8])
def test_infinities_and_nan_stay_in_their_entries(nel):
    from atkdsp_b200 import gpu
    rng = np.random.default_rng(nel)
    M, m = 16, 70
    y = (rng.standard_normal((nel, M, m)) + 1j * rng.standard_normal((nel, M, m))).astype(np.complex64)
    y[1, 3, 41] = complex(np.inf, 1.0)
    y[0, 5, 69] = complex(np.nan, 0.0)
    R = torch.zeros(M, nel, nel, dtype=torch.complex64, device="cuda")
    c = torch.zeros(M, dtype=torch.int32, device="cuda")
    gpu.cov_accumulate(torch.from_numpy(y).cuda(), nel, M, None, R, c)
    torch.cuda.synchronize()
    got = R.cpu().numpy()
    bad = np.zeros((M, nel, nel), bool)
    bad[3, 1, :] = bad[3, :, 1] = bad[5, 0, :] = bad[5, :, 0] = True
    assert np.isfinite(got[~bad]).all() and not np.isfinite(got[bad]).any()
    assert got[3, 1, 1].real == np.inf and np.isnan(got[5, 0, 0].real)


@pytest.mark.parametrize("nel,ms", [(2, (2047, 2048, 4095, 4097)), (3, (1023, 1024, 2049)), (4, (2047, 2048)),
                                    (5, (511, 1025)), (8, (511, 512, 1023, 1024, 9001))])
def test_runs_around_the_warp_counts(nel, ms):
    """4, 8 and 16 warps a channel: hop counts around the lines between them,
    where a warp's run is shortest and the last may be empty."""
    from atkdsp_b200 import gpu
    M = 5
    for m in ms:
        rng = np.random.default_rng(nel * 7 + m)
        y = (rng.standard_normal((nel, M, m)) + 1j * rng.standard_normal((nel, M, m))).astype(np.complex64)
        R = torch.zeros(M, nel, nel, dtype=torch.complex64, device="cuda")
        c = torch.zeros(M, dtype=torch.int32, device="cuda")
        d = torch.from_numpy(y).cuda()
        gpu.cov_accumulate(d, nel, M, None, R, c)
        pw, mean = gpu.channel_power(d, nel, M)
        torch.cuda.synchronize()
        got, re, im, mag = R.cpu().numpy(), *_sums(y)
        assert np.array_equal(c.cpu().numpy(), np.full(M, m)), m
        _close(got.real, re, mag, m)
        _close(got.imag, im, mag, m)
        want = np.diagonal(re, axis1=1, axis2=2).T / m
        assert (np.abs(pw.cpu().numpy() - want) <= 2.0 ** -23 * want).all(), m
