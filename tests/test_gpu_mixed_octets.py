"""GPU parity where one eight-element part of a block has values or differences
past what floats hold exactly and the block's other parts have not: the parts
are quantized in different forms, and the block is packed as wide as its widest
part asks for.  Streams and floats must equal the oracle's (no tolerance)."""
from __future__ import annotations

import numpy as np
import pytest

import zccl_gb300 as Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("L", [9, 12, 24, 32, 36, 64, 100, 200, 256])
def test_one_wide_part_in_a_block(port, L, fixed):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, T, eb = 6007, 2, 2.0 ** -10
    codec = Z.Codec(n, L, T, fixed=fixed)
    rng = np.random.default_rng(L)
    for bits in range(20, 31):  # the widest difference's bits
        q = rng.integers(-2000, 2000, n).astype(np.float64)
        at = rng.integers(0, n, n // 50)
        q[at] += rng.choice([-1, 1], at.size) * (2.0 ** bits - 2.0 ** (bits - 6))
        x = (q * eb).astype(np.float32)
        want = port.compress_fixed(x, eb, L, T) if fixed else port.compress(x, eb, L, T)
        s = codec.compress(torch.from_numpy(x).cuda(), eb)
        codec.check()
        assert s.tobytes() == want, bits
        floats = port.decompress_fixed(want, n, eb, L, T) if fixed else port.decompress(want, n, eb, L, T)
        y = codec.decompress(s, eb)
        codec.check()
        assert np.array_equal(y.cpu().numpy().view(np.uint32), floats.view(np.uint32)), bits
