"""Filterbanks whose nchan is no power of two (or below 16): single handles run
a kernel of one CTA per few hops, batches the tile kernel, both through
the same mixed-radix passes (butterflies for 2, 3, 4, 5, 7, 8, a direct DFT for
other primes). Every radix, hop counts that leave a CTA's last group short,
one and two elements, cf32 and int16: device calls against a batch bit for bit
and against the C oracle within the filterbank's 1e-5."""

from __future__ import annotations

import numpy as np
import pytest

import atkdsp_b200 as ak
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FS = 2.4e6


@pytest.mark.parametrize("M,os_,K", [(2, 1, 4), (3, 3, 2), (7, 1, 5), (10, 2, 6), (24, 2, 8), (35, 5, 3), (48, 4, 9),
                                     (77, 7, 4), (169, 13, 2), (343, 1, 3), (1000, 2, 12), (1021, 1, 3),
                                     (1920, 3, 8), (6400, 2, 2)])
def test_device_calls_equal_batches_and_the_oracle(M, os_, K):
    from atkdsp_b200 import gpu
    rng = np.random.default_rng(M * 7 + os_)
    hop = M // os_
    a, b = ak.Pfb(FS, M, os_, K), ak.Pfb(FS, M, os_, K)
    batch, ref = gpu.Batch([b]), O.oracle().Pfb(FS, M, os_, K)
    for n in (3 * hop + 1, M * K + 601 * hop // 2, hop):
        x = (rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)
        d = torch.from_numpy(x).cuda()            # lives until both streams are done
        y = gpu.process_n(a, [d], 1)
        hops = b.out_hops(n)
        out = torch.zeros(max(M * hops, 1), dtype=torch.complex64, device="cuda")
        torch.cuda.synchronize()
        batch.process([d], [out])
        torch.cuda.synchronize()
        got = y.cpu().numpy()[0]
        assert np.array_equal(got.reshape(-1).view(np.uint32), out[:M * hops].cpu().numpy().view(np.uint32)), n
        r = ref.process(x)
        assert got.shape == r.shape
        assert np.max(np.abs(got - r), initial=0.0) <= 1e-5 * np.max(np.abs(r), initial=1e-30), n
    assert ak.load().atkdsp_gpu_pfb_faults(a.handle) == 0


@pytest.mark.parametrize("M,os_,K", [(24, 2, 12), (1000, 2, 12), (3000, 2, 8)])
def test_two_elements_and_int16(M, os_, K):
    from atkdsp_b200 import gpu
    rng = np.random.default_rng(M)
    n = M * K + 97 * M // 2
    cal = (rng.standard_normal((2, M)) + 1j * rng.standard_normal((2, M))).astype(np.complex64)
    raws = [rng.integers(-2000, 2000, 2 * n, dtype=np.int64).astype("<i2") for _ in range(2)]
    p, r = ak.Pfb(FS, M, os_, K, 80.0, 2), O.oracle().Pfb(FS, M, os_, K, 80.0, 2)
    p.set_cal(cal, 2)
    r.set_cal(cal, 2)
    off = 0.01 - 0.02j
    ds = [torch.from_numpy(v).cuda() for v in raws]
    y = gpu.process_n_raw(p, ds, 2, "ci16", off)
    torch.cuda.synchronize()
    yr = r.process_n([O.oracle().unpack_dc(v.tobytes(), "ci16", off)[0] for v in raws], 2)
    assert tuple(y.shape) == yr.shape
    assert np.max(np.abs(y.cpu().numpy() - yr)) <= 1e-5 * np.max(np.abs(yr))
