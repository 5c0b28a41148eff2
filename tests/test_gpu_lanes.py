"""GPU parity of the codec kernels' two work layouts -- a lane per block of
32 elements, and eight elements a lane for every other block -- where they can
go wrong: block lengths around the lane groups' edges, buffers at every
16-byte phase, values and sums past what floats hold exactly, and enough tiles
for several rounds of the scan that places them.  Bytes and floats must equal
the oracle's (no tolerance)."""
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


def at_phase(torch, a, p):
    """a on the device, p floats past a 16-byte boundary."""
    buf = torch.zeros(a.size + 4, dtype=torch.float32, device="cuda")
    buf[p: p + a.size] = torch.from_numpy(a).cuda()
    return buf[p: p + a.size]


def walk(n, seed, amp=0.01):
    return np.cumsum(np.random.default_rng(seed).normal(0, amp, n)).astype(np.float32)


def roundtrip(torch, port, xs, eb, L, T, p):
    """Compress at phase p, decompress at phase p (written and added), the
    sum of all xs, from device-made and from byte streams."""
    n = xs[0].size
    codec = Z.Codec(n, L, T)
    ss = [port.compress(x, eb, L, T) for x in xs]
    devs = [codec.compress(at_phase(torch, x, p), eb) for x in xs]
    for d, s in zip(devs, ss):
        assert d.tobytes() == s
    want = port.decompress(ss[0], n, eb, L, T)
    y = at_phase(torch, xs[1], p)
    codec.decompress(devs[0], eb, out=y)
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    acc = at_phase(torch, xs[1], p)
    codec.decompress_accumulate(devs[0], eb, acc)
    assert np.array_equal(acc.cpu().numpy(), xs[1] + want)
    foreign = Z.DeviceStream.from_bytes(codec, ss[0])
    codec.decompress(foreign, eb, out=y)
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
    total = ss[0]
    for s in ss[1:]:
        total = port.homadd(total, s, n, eb, L, T)
    h = codec.homadd(devs)
    assert h.tobytes() == total
    codec.decompress(h, eb, out=y)
    codec.check()
    assert np.array_equal(y.cpu().numpy().view(np.uint32), port.decompress(total, n, eb, L, T).view(np.uint32))


@pytest.mark.parametrize("L", [1, 7, 8, 16, 31, 32, 33, 36, 40, 64, 100, 128, 250, 256])
@pytest.mark.parametrize("T", [1, 3])
def test_block_lengths_at_every_phase(torch, port, L, T):
    for p in range(4):
        n = 2 * 8192 + 1013 + 5 * p if L >= 8 else 1500 + p
        xs = [walk(n, 17 * L + k) for k in range(3)]
        roundtrip(torch, port, xs, float(np.float32(1e-4 * np.ptp(xs[0]))), L, T, p)


@pytest.mark.parametrize("L", [32, 36])
def test_values_and_sums_past_exact_floats(torch, port, L):
    """Quantized values beyond 2^23 and 2^24, deltas beyond 2^22, and sums of
    many inputs beyond 2^24, in some blocks of a group and in all of them."""
    n, T, eb = 3 * 8192 + 700, 2, 1.0e-3
    rng = np.random.default_rng(L)
    for level, jump in ((9.0e6, 0.0), (2.0e7, 0.0), (0.0, 5.0e6), (0.0, 1.2e7)):
        xs = []
        for k in range(4):
            x = rng.normal(0, 300, n) + level
            x[rng.integers(0, n, 40)] += jump
            xs.append((eb * np.trunc(x)).astype(np.float32))
        roundtrip(torch, port, xs, eb, L, T, 1)


@pytest.mark.parametrize("L,T", [(32, 1), (32, 72), (36, 5)])
def test_many_tiles(torch, port, L, T):
    n = 700 * 8192 + 4321
    xs = [walk(n, T + k) for k in range(2)]
    roundtrip(torch, port, xs, float(np.float32(1e-4 * np.ptp(xs[0]))), L, T, 0)


@pytest.mark.parametrize("L", [32, 36, 100])
def test_fixed_rate_layout(torch, port, L):
    n, T = 2 * 8192 + 300, 3
    x = walk(n, L)
    x[5000] += 40.0  # a wide block among narrow ones
    eb = float(np.float32(1e-5 * np.ptp(x)))
    codec = Z.Codec(n, L, T, fixed=True)
    for p in range(4):
        s = codec.compress(at_phase(torch, x, p), eb)
        want = port.compress_fixed(x, eb, L, T)
        assert s.tobytes() == want
        y = at_phase(torch, x, p)
        codec.decompress(s, eb, out=y)
        codec.check()
        assert np.array_equal(y.cpu().numpy().view(np.uint32), port.decompress_fixed(want, n, eb, L, T).view(np.uint32))
