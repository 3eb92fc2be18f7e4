"""A single handle's large call runs a kernel built for its tile shape alone, a
mixed batch the kernel of every shape. The shapes' code is shared, so outputs
and carried state must agree bit for bit: every kind of shape (one hop per
thread, paired, quad, the two-hop tile of nchan 4096, oversample 8), two
ragged blocks with more points than the per-hop kernel takes, cf32 and int16,
one and two elements."""

from __future__ import annotations

import numpy as np
import pytest

import atkdsp_b200 as ak

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FS = 2.4e6


@pytest.mark.parametrize("M,os_,K,choice,fmt", [
    (16, 2, 8, 2, "cf32"), (16, 1, 5, 1, "ci16"), (32, 4, 12, 1, "cf32"), (64, 2, 16, 5, "cf32"),
    (128, 1, 12, 0, "cf32"), (256, 2, 12, 1, "ci16"), (512, 1, 8, 2, "cf32"), (1024, 2, 16, 1, "cf32"),
    (1024, 8, 6, -1, "cf32"), (2048, 4, 7, 1, "cf32"), (2048, 2, 16, 0, "ci16"), (4096, 2, 12, -1, "cf32"),
    (4096, 1, 3, -1, "ci16"), (4096, 8, 4, -1, "cf32")])
def test_single_and_mixed_launches_agree(M, os_, K, choice, fmt):
    from atkdsp_b200 import gpu
    lib = ak.load()
    rng = np.random.default_rng(M + 13 * os_ + K)
    hop = M // os_
    if choice >= 0:
        assert lib.atkdsp_gpu_tune_set(M, os_, K, choice) == 0
    try:
        a, b = ak.Pfb(FS, M, os_, K), ak.Pfb(FS, M, os_, K)
        two = ak.Pfb(FS, M, os_, K, 80.0, 2)
    finally:
        if choice >= 0:
            lib.atkdsp_gpu_tune_set(M, os_, K, -1)
    other = ak.Pfb(FS, 64 if M != 64 else 32, 2, 4)          # another bank: the kernel of every shape
    batch = gpu.Batch([b, other])
    z = torch.zeros(0, dtype=torch.complex64, device="cuda")
    for extra in (0, hop // 2 + 1):
        n = ((1 << 17) // M + 9) * hop + extra
        if fmt == "cf32":
            x = torch.from_numpy((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)).cuda()
            y, y2 = gpu.process_n(a, [x], 1), gpu.process_n(two, [x, x], 2)
        else:
            x = torch.from_numpy(rng.integers(-2000, 2000, 2 * n, dtype=np.int64).astype("<i2")).cuda()
            y, y2 = gpu.process_n_raw(a, [x], 1, fmt), gpu.process_n_raw(two, [x, x], 2, fmt)
        hops = b.out_hops(n)
        out = torch.zeros(M * hops, dtype=torch.complex64, device="cuda")
        torch.cuda.synchronize()
        (batch.process([x, z], [out, z]) if fmt == "cf32" else batch.process_raw([x, z], [out, z], fmt))
        torch.cuda.synchronize()
        want = out.cpu().numpy().view(np.uint32)
        assert np.array_equal(y.cpu().numpy().reshape(-1).view(np.uint32), want), extra
        for e in range(2):
            assert np.array_equal(y2[e].cpu().numpy().reshape(-1).view(np.uint32), want), (extra, e)
    assert lib.atkdsp_gpu_pfb_faults(a.handle) == 0 and lib.atkdsp_gpu_batch_faults(batch._b) == 0
