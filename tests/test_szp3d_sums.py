"""The 3-D codec's kernels where their units, chunks, pieces, parts and ragged
ends can go wrong, against the oracle bit for bit, and the decoder's float
reconstruction against the double steps on the CPU."""
from __future__ import annotations

import os
import shutil
import subprocess

import numpy as np
import pytest


def test_reconstruction_matches_double(tmp_path):
    """(float)((double)q * twice) from float pairs and the rounding test,
    restated in C: about 100 million random, near-tie and power-of-two
    results."""
    cc = shutil.which("gcc") or shutil.which("cc")
    if not cc:
        pytest.skip("no C compiler")
    exe = tmp_path / "sz3_value"
    src = os.path.join(os.path.dirname(__file__), "native", "sz3_value.c")
    subprocess.run([cc, "-O2", "-ffp-contract=off", "-o", str(exe), src, "-lm"], check=True)
    out = subprocess.run([str(exe), "400000"], capture_output=True, text=True, timeout=120)
    bad, checks, slow = map(int, out.stdout.split())
    assert bad == 0 and checks > 50_000_000
    assert slow < checks // 8  # the rounding test settles nearly all


def volume(dims, kind, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, dims)
    if kind == "smooth":
        for ax in range(3):
            x = np.cumsum(x, axis=ax)
        x = x / np.abs(x).max() + rng.normal(0, 0.002, dims)
    elif kind == "sparse":
        x = np.where(rng.random(dims) < 0.002, x, 0.0)
    elif kind == "wide":  # magnitudes from block to block over nine decades: rates 0 to 27
        b = [-(-d // 8) for d in dims]
        x = x * np.kron(10.0 ** rng.uniform(-6, 3, b), np.ones((8, 8, 8)))[: dims[0], : dims[1], : dims[2]]
    return np.ascontiguousarray(x, np.float32).ravel()


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [2, 4, 8])
@pytest.mark.parametrize("kind", ["smooth", "sparse", "wide"])
@pytest.mark.parametrize("dims", [(9, 41, 517), (16, 16, 256), (33, 70, 35), (8, 8, 8), (1, 1, 1), (3, 5, 7),
                                  (17, 9, 129), (5, 300, 20), (70, 3, 67), (12, 35, 300), (2, 2, 2050), (25, 50, 2)])
def test_decode_sums(torch, port, bs, kind, dims):
    from zccl_gb300.szp3d import Szp3D
    x = volume(dims, kind, sum(dims) + bs)
    eb = 2e-4 if kind != "wide" else 1e-5
    s = port.szp3d_compress(x, dims, bs, eb)
    want = port.szp3d_decompress(s, dims, bs, eb).view(np.uint32)
    codec = Szp3D(dims, bs)
    for at in (0, 5):  # the stream at any byte
        buf = torch.zeros(len(s) + 16, dtype=torch.uint8, device="cuda")
        buf[at: at + len(s)] = torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda()
        y = codec.decompress(buf[at:], eb, avail=len(s)).cpu().numpy()
        codec.check()
        assert np.array_equal(y.view(np.uint32), want)
    out, size = codec.compress(torch.from_numpy(x).cuda(), eb)
    assert out[: codec.size(size)].cpu().numpy().tobytes() == s


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [2, 4, 8])
@pytest.mark.parametrize("scale", [2.0 ** 18, 2.0 ** 19, 2.0 ** 23, 2.0 ** 29])
def test_encode_past_exact_floats(torch, port, bs, scale):
    """Quantized values on both sides of what the float steps hold, near ties,
    in some units of a tile and in all, at any 4-byte phase of the volume."""
    from zccl_gb300.szp3d import Szp3D
    dims, eb = (19, 21, 150), 2e-4
    rng = np.random.default_rng(bs)
    q = rng.normal(0, 40, dims)
    q[:, :, 40:70] += scale * rng.choice([-1.0, 0.0, 1.0], (19, 21, 30))
    q[11:] *= 1 + min(scale / 4000, 2.0)  # within int
    x = ((np.round(q) - 0.5 * (rng.random(dims) < 0.2)) * 2 * eb).astype(np.float32).ravel()
    s = port.szp3d_compress(x, dims, bs, eb)
    codec = Szp3D(dims, bs)
    for at in range(4):
        buf = torch.zeros(x.size + 8, dtype=torch.float32, device="cuda")
        buf[at: at + x.size] = torch.from_numpy(x).cuda()
        out, size = codec.compress(buf[at: at + x.size], eb)
        codec.check()
        assert out[: codec.size(size)].cpu().numpy().tobytes() == s


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [2, 4, 8])
def test_decode_reports_what_is_no_stream(torch, port, bs):
    from zccl_gb300.szp3d import Szp3D
    dims, eb = (20, 30, 70), 2e-4
    s = port.szp3d_compress(volume(dims, "smooth", 1), dims, bs, eb)
    bad = bytearray(s)
    bad[3] = 33  # a rate
    codec = Szp3D(dims, bs)
    for cut in (bytes(bad), s[:-1], s[: len(s) // 2], s[:4]):
        buf = torch.from_numpy(np.frombuffer(cut, np.uint8).copy()).cuda()
        codec.decompress(buf, eb, avail=len(cut))
        with pytest.raises(Exception):
            codec.check()
    codec.decompress(torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda(), eb, avail=len(s))
    codec.check()
