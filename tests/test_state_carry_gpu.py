"""The state carry after a launch: launches of few jobs copy it in parts over
several CTAs, launches of many jobs whole. A stream in blocks gives the bits of
the stream in one call, whatever the block ends in: a part past the carry's
end, parts that straddle state and input, carries shorter than the parts, long
prototypes, int16 input, 2 and 33 elements, batches of 2 and 40 streams."""

from __future__ import annotations

import numpy as np
import pytest

import atkdsp_b200 as ak

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FS = 2.4e6


def _x(rng, n, fmt):
    if fmt == "cf32":
        return torch.from_numpy((rng.standard_normal(n) + 1j * rng.standard_normal(n)).astype(np.complex64)).cuda()
    return torch.from_numpy(rng.integers(-2000, 2000, 2 * n, dtype=np.int64).astype("<i2")).cuda()


def _run(p, xs, nel, fmt):
    from atkdsp_b200 import gpu
    y = gpu.process_n(p, xs, nel) if fmt == "cf32" else gpu.process_n_raw(p, xs, nel, fmt)
    gpu.sync(p)
    return y.cpu().numpy()


@pytest.mark.parametrize("M,os_,K,nel,fmt", [(2048, 1, 40, 1, "cf32"), (4096, 2, 8, 1, "ci16"), (16, 2, 2, 1, "cf32"),
                                             (1024, 4, 5, 2, "cf32"), (64, 1, 16, 33, "cf32"), (512, 2, 12, 1, "ci16")])
def test_blocks_equal_one_call(M, os_, K, nel, fmt):
    rng = np.random.default_rng(M + K)
    hop = M // os_
    per = 2 if fmt != "cf32" else 1
    big = max((1 << 17) // M + 9, 2100 if M < 64 else 0) * hop
    cuts = [big + 3, 2 * hop - 1, big + hop // 2, 1, big]
    xs = [_x(rng, sum(cuts), fmt) for _ in range(nel)]
    want = _run(ak.Pfb(FS, M, os_, K, 80.0, nel), xs, nel, fmt)
    p, at, got = ak.Pfb(FS, M, os_, K, 80.0, nel), 0, []
    for n in cuts:
        got.append(_run(p, [x[per * at:per * (at + n)].clone() for x in xs], nel, fmt))
        at += n
    got = np.concatenate(got, axis=2)
    assert got.shape == want.shape and np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert ak.load().atkdsp_gpu_pfb_faults(p.handle) == 0


@pytest.mark.parametrize("count", [2, 40])
def test_batches(count):
    from atkdsp_b200 import gpu
    rng = np.random.default_rng(count)
    specs = [(int(rng.choice([16, 64, 1000, 1024, 4096])), int(rng.choice([1, 2])), int(rng.choice([3, 12, 40])))
             for _ in range(count)]
    xs = [_x(rng, 3 * M * K + M + 5, "cf32") for M, _, K in specs]
    hs = [ak.Pfb(FS, M, o, K) for M, o, K in specs]
    batch = gpu.Batch(hs)
    got = [[] for _ in specs]
    for part in range(3):
        ins = [x[len(x) * part // 3:len(x) * (part + 1) // 3].clone() for x in xs]
        hops = [h.out_hops(len(i)) for h, i in zip(hs, ins)]
        outs = [torch.zeros(max(M * m, 1), dtype=torch.complex64, device="cuda") for (M, _, _), m in zip(specs, hops)]
        torch.cuda.synchronize()
        batch.process(ins, outs)
        torch.cuda.synchronize()
        for g, o, (M, _, _), m in zip(got, outs, specs, hops):
            g.append(o[:M * m].view(M, m).cpu().numpy())
    for g, x, (M, o, K) in zip(got, xs, specs):
        want = _run(ak.Pfb(FS, M, o, K), [x], 1, "cf32")[0]
        g = np.concatenate(g, axis=1)
        assert g.shape == want.shape and np.array_equal(g.view(np.uint32), want.view(np.uint32)), (M, o, K)
    assert ak.load().atkdsp_gpu_batch_faults(batch._b) == 0
