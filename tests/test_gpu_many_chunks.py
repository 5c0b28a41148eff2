"""Streams of thousands of chunks of a few blocks each: most warps of a tile have
nothing to do and run ahead as far as their barriers let them, tile after tile.
Every call must end in order, with the oracle's bytes."""
from __future__ import annotations

import numpy as np
import pytest

import zccl_gb300 as Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [3, 9, 32, 36, 100])
def test_batches_of_short_chunks(port, L):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, T, P, eb = 256000, 3000, 9, 1.0e-3
    rng = np.random.default_rng(L)
    xs = [rng.normal(0, 1, n).astype(np.float32) for _ in range(P)]
    want = [port.compress(x, eb, L, T) for x in xs]
    total = want[0]
    for w in want[1:]:
        total = port.homadd(total, w, n, eb, L, T)
    codec = Z.Codec(n, L, T)
    dx = [torch.from_numpy(x).cuda() for x in xs]
    ss, ys, o = [codec.new_stream() for _ in xs], [torch.empty(n, device="cuda") for _ in xs], codec.new_stream()
    c = Z.Batch(Z.BATCH_COMPRESS, [(x, eb, T, s) for x, s in zip(dx, ss)], L)
    c.run()
    c.check()
    assert [s.tobytes() for s in ss] == want
    h = Z.Batch(Z.BATCH_HOMADD, [(ss, T, o)] + [([s, s], T, codec.new_stream()) for s in ss], L)
    d = Z.Batch(Z.BATCH_DECOMPRESS, [(s, eb, T, y, False) for s, y in zip(ss, ys)], L)
    for _ in range(200):
        c.run()
        h.run()
        d.run()
    for b in (c, h, d):
        b.check()
    assert [s.tobytes() for s in ss] == want and o.tobytes() == total
    for y, w in zip(ys, want):
        assert np.array_equal(y.cpu().numpy().view(np.uint32), port.decompress(w, n, eb, L, T).view(np.uint32))
