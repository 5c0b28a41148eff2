"""Calls from several host threads, each on a stream of its own, whose kernels
want different amounts of shared memory for the same code (long and short
blocks through the header walk, wide and narrow planes through the 3-D
decoder), must not disturb one another."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import zccl_gb300 as Z

pytestmark = pytest.mark.gpu


def test_threads_with_different_shapes(port):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zccl_gb300.szp3d import Szp3D
    rng = np.random.default_rng(3)
    x = np.cumsum(rng.normal(0, 0.01, 200000)).astype(np.float32)
    eb, errors = 1e-3, []
    wires = {L: port.compress(x, eb, L, 3) for L in (8, 32, 36, 256)}
    floats = {L: port.decompress(w, x.size, eb, L, 3).view(np.uint32) for L, w in wires.items()}
    dims = [(12, 40, 500), (30, 16, 64), (9, 160, 1200)]
    vols = [rng.normal(0, 1, d).astype(np.float32).ravel() for d in dims]
    streams = [port.szp3d_compress(v, d, 4, eb) for v, d in zip(vols, dims)]
    want = [port.szp3d_decompress(s, d, 4, eb).view(np.uint32) for s, d in zip(streams, dims)]

    def work(k):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                for i in range(6):
                    L = (8, 32, 36, 256)[(k + i) % 4]
                    codec = Z.Codec(x.size, L, 3)
                    y = torch.empty(x.size, dtype=torch.float32, device="cuda")
                    codec.decompress(Z.DeviceStream.from_bytes(codec, wires[L]), eb, out=y)
                    codec.check()
                    assert np.array_equal(y.cpu().numpy().view(np.uint32), floats[L])
                    j = (k + i) % 3
                    v = Szp3D(dims[j], 4)
                    b = torch.from_numpy(np.frombuffer(streams[j], np.uint8).copy()).cuda()
                    z = v.decompress(b, eb, avail=len(streams[j]))
                    v.check()
                    assert np.array_equal(z.cpu().numpy().view(np.uint32), want[j])
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
