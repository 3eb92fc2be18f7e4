"""Device calls of one element and few output points run one CTA per hop
(pfb_hops1_kernel), larger ones and batches the tile kernel. Both fold every
branch in the same order and walk the same FFT plan with the same butterflies,
so the outputs and the carried state must agree bit for bit: a handle driven
by device calls against a handle in a batch of one, at one hop, at the line
between the two kernels and one hop past it, over two ragged blocks."""

from __future__ import annotations

import numpy as np
import pytest

import atkdsp_b200 as ak

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FS = 2.4e6
POINTS = 1 << 17            # hops x nchan up to which a device call runs per hop


@pytest.mark.parametrize("M,os_,K,fmt", [(16, 2, 5, "cf32"), (64, 1, 16, "cf32"), (128, 4, 12, "ci16"),
                                         (256, 2, 12, "ci16q11"), (512, 8, 3, "cf32"), (1024, 2, 16, "cf32")])
def test_device_calls_equal_the_tile_kernel(M, os_, K, fmt):
    from atkdsp_b200 import gpu
    rng = np.random.default_rng(M + K)
    hop = M // os_
    for m in (1, min(2048, POINTS // M), min(2048, POINTS // M) + 1):
        a, b = ak.Pfb(FS, M, os_, K), ak.Pfb(FS, M, os_, K)
        batch = gpu.Batch([b])
        for n in (m * hop, m * hop + hop // 2 + 1):
            if fmt == "cf32":
                x = torch.from_numpy((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)).cuda()
                y = gpu.process_n(a, [x], 1)
            else:
                x = torch.from_numpy(rng.integers(-2000, 2000, 2 * n, dtype=np.int64).astype("<i2")).cuda()
                y = gpu.process_n_raw(a, [x], 1, fmt)
            hops = b.out_hops(n)
            out = torch.zeros(max(M * hops, 1), dtype=torch.complex64, device="cuda")
            torch.cuda.synchronize()
            (batch.process([x], [out]) if fmt == "cf32" else batch.process_raw([x], [out], fmt))
            torch.cuda.synchronize()
            assert y.shape == (1, M, hops)
            assert np.array_equal(y.cpu().numpy().reshape(-1).view(np.uint32),
                                  out[:M * hops].cpu().numpy().view(np.uint32)), (m, n)
        assert ak.load().atkdsp_gpu_pfb_faults(a.handle) == 0


@pytest.mark.parametrize("M,os_,K,line", [(16, 2, 21, 1536), (32, 1, 32, 1536), (32, 2, 33, 1024), (16, 1, 40, 1024),
                                          (64, 8, 40, 2048)])
def test_long_prototypes_around_their_line(M, os_, K, line):
    """More taps a branch move the line to fewer hops; on both sides of it the
    outputs and the carried state are the tile kernel's."""
    from atkdsp_b200 import gpu
    rng = np.random.default_rng(M + K)
    hop = M // os_
    for m in (line, line + 1):
        a, b = ak.Pfb(FS, M, os_, K), ak.Pfb(FS, M, os_, K)
        batch = gpu.Batch([b])
        for n in (m * hop, 5 * hop + 1):
            x = torch.from_numpy((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)).cuda()
            y = gpu.process_n(a, [x], 1)
            hops = b.out_hops(n)
            out = torch.zeros(max(M * hops, 1), dtype=torch.complex64, device="cuda")
            torch.cuda.synchronize()
            batch.process([x], [out])
            torch.cuda.synchronize()
            assert np.array_equal(y.cpu().numpy().reshape(-1).view(np.uint32),
                                  out[:M * hops].cpu().numpy().view(np.uint32)), (m, n)
        assert ak.load().atkdsp_gpu_pfb_faults(a.handle) == 0
