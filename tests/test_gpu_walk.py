"""GPU parity of the header walk (streams that arrive as bytes only) where its
windows, groups and lists can go wrong: runs of zero-width blocks that fill
windows or stop inside them, windows of narrow blocks with more headers than a
list holds, many windows per chunk, long blocks, many chunks, and bytes after
the stream's end that look like headers.  The index must place every block
exactly, so the decoded floats equal the oracle's bit for bit; a header that
can be none is reported."""
from __future__ import annotations

import numpy as np
import pytest

import zccl_gb300 as Z

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    Z.lib()
    return t


def data(kind, n):
    rng = np.random.default_rng(n)
    x = np.cumsum(rng.normal(0, 0.01, n)).astype(np.float32)
    if kind == "zeros":
        return np.zeros(n, np.float32)
    if kind == "runs":  # smooth stretches between zero runs of every length up to many windows
        at = 0
        while at < n:
            k = int(2 ** rng.uniform(3, 18))
            x[at: at + k] = 0
            at += k + int(2 ** rng.uniform(3, 14))
    if kind == "narrow":  # widths 0, 1 and 2
        x = (rng.integers(-2, 3, n) * rng.integers(0, 2, n) * 1e-3).astype(np.float32)
    if kind == "wide":  # widths up to the 20s
        x = (rng.normal(0, 1, n) * 10.0 ** rng.uniform(-3, 3, n)).astype(np.float32)
    return x


@pytest.mark.parametrize("kind", ["smooth", "zeros", "runs", "narrow", "wide"])
@pytest.mark.parametrize("n,L,T", [(1 << 22, 32, 1), (1000003, 32, 7), (1000003, 36, 72), (300007, 8, 2),
                                   (700001, 256, 3), (4099, 1, 1)])
def test_walk_places_every_block(torch, port, kind, n, L, T):
    x = data(kind, n)
    eb = 1.0e-3
    wire = port.compress(x, eb, L, T)
    want = port.decompress(wire, n, eb, L, T).view(np.uint32)
    codec = Z.Codec(n, L, T)
    out = torch.empty(n, dtype=torch.float32, device="cuda")
    for tail in (b"", b"\0" * 5000, b"\x01" * 5000, b"\x20" * 3):
        s = Z.DeviceStream.from_bytes(codec, wire + tail)
        codec.decompress(s, eb, out=out)
        codec.check()
        assert s.tobytes() == wire
        assert np.array_equal(out.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("kind", ["smooth", "zeros"])
def test_walk_reports_what_is_no_stream(torch, port, kind):
    n, L, T, eb = 200000, 32, 2, 1.0e-3
    wire = bytearray(port.compress(data(kind, n), eb, L, T))
    codec = Z.Codec(n, L, T)
    bad = bytearray(wire)
    bad[8 * T + 4] = 33  # the first block's header
    for cut in (bytes(bad), bytes(wire[:-40])):
        codec.build_index(Z.DeviceStream.from_bytes(codec, cut))
        with pytest.raises(Exception):
            codec.check()
    codec.build_index(Z.DeviceStream.from_bytes(codec, bytes(wire)))
    codec.check()
