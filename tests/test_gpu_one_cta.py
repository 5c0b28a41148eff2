"""Launches of a single CTA, and launches without the CTA that scans the tiles'
sizes (which leaves its place where no other CTA came to work): every
tile still finds its place.  Streams must equal the oracle's."""
from __future__ import annotations

import numpy as np
import pytest

import zccl_gb300 as Z

pytestmark = pytest.mark.gpu
EB = float(np.float32(1e-3))


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


def wave(n, seed):
    rng = np.random.default_rng(seed)
    return np.cumsum(rng.normal(0, 0.01 * (1 + 10 * (np.arange(n) % 50000 < 20000)))).astype(np.float32)


@pytest.mark.parametrize("n,L,T", [(1000003, 32, 1), (1000003, 32, 72), (400009, 36, 3), (8200, 32, 1), (100, 32, 1)])
def test_one_cta(torch, port, monkeypatch, n, L, T):
    xs = [wave(n, k) for k in range(3)]
    want = [port.compress(x, EB, L, T) for x in xs]
    total = port.homadd(port.homadd(want[0], want[1], n, EB, L, T), want[2], n, EB, L, T)
    codec = Z.Codec(n, L, T)
    dx = [torch.from_numpy(x).cuda() for x in xs]
    monkeypatch.setenv("ZCCL_GPU_TEST_ONE_CTA", "1")
    for _ in range(2):
        ss = [codec.compress(x, EB) for x in dx]
        codec.check()
        assert [s.tobytes() for s in ss] == want
        o = codec.homadd(ss)
        codec.check()
        assert o.tobytes() == total
        outs, sums = [codec.new_stream() for _ in xs], [codec.new_stream() for _ in range(2)]
        b = Z.Batch(Z.BATCH_COMPRESS, [(x, EB, T, s) for x, s in zip(dx, outs)], L)
        b.run()
        b.check()
        assert [s.tobytes() for s in outs] == want
        b = Z.Batch(Z.BATCH_HOMADD, [(ss, T, s) for s in sums], L)
        b.run()
        b.check()
        assert [s.tobytes() for s in sums] == [total] * 2


@pytest.mark.parametrize("bs", [2, 4, 8])
def test_one_cta_szp3d(torch, port, monkeypatch, bs):
    from zccl_gb300.szp3d import Szp3D
    dims = (33, 40, 70)
    x = wave(33 * 40 * 70, bs)
    want = port.szp3d_compress(x, dims, bs, EB)
    codec = Szp3D(dims, bs)
    monkeypatch.setenv("ZCCL_GPU_TEST_ONE_CTA", "1")
    out, size = codec.compress(torch.from_numpy(x).cuda(), EB)
    codec.check()
    assert out[: codec.size(size)].cpu().numpy().tobytes() == want


@pytest.mark.parametrize("n,L,T", [(4000003, 32, 1), (1000003, 32, 72), (400009, 36, 3), (8200, 32, 1)])
def test_no_scanner(torch, port, monkeypatch, n, L, T):
    x = wave(n, 7)
    want = port.compress(x, EB, L, T)
    codec = Z.Codec(n, L, T)
    monkeypatch.setenv("ZCCL_GPU_TEST_NO_SCANNER", "1")
    for _ in range(3):
        s = codec.compress(torch.from_numpy(x).cuda(), EB)
        codec.check()
        assert s.tobytes() == want
