"""The 3-D decoder on volumes with few rows of blocks, whose rows are summed in
pieces along z (rows of one piece's length and around it, pieces with and
without the carry of the rows before them, planes of both sizes of the last
pass, outputs at every phase), and on flat volumes, some of which take another
decoder.  Floats must equal the oracle's bit for bit."""
from __future__ import annotations

import numpy as np
import pytest


def volume(dims, wide, seed):
    rng = np.random.default_rng(seed)
    x = np.cumsum(rng.normal(0, 0.02, dims), axis=2) + rng.normal(0, 1, dims[:2] + (1,))
    if wide:
        x = x * 10.0 ** rng.uniform(-4, 3, (dims[0], dims[1], 1))
    return np.ascontiguousarray(x, np.float32).ravel()


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [2, 4, 8])
@pytest.mark.parametrize("dims", [(1, 1, 70001), (3, 5, 20000), (9, 41, 5170), (8, 24, 9001), (17, 33, 2300), (2, 70, 2100),
                                  (40, 3, 1025), (4, 20, 256), (4, 20, 257), (5, 9, 64), (5, 9, 65), (33, 18, 129)])
def test_rows_in_pieces(port, bs, dims):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zccl_gb300.szp3d import Szp3D
    n = dims[0] * dims[1] * dims[2]
    codec = Szp3D(dims, bs)
    for wide in (False, True):
        x = volume(dims, wide, n + bs)
        eb = 1e-3 if bs != 4 else 0.00123456789
        wire = port.szp3d_compress(x, dims, bs, eb)
        want = port.szp3d_decompress(wire, dims, bs, eb).view(np.uint32).ravel()
        b = torch.from_numpy(np.frombuffer(wire, np.uint8).copy()).cuda()
        for p in (0, 3):
            buf = torch.full((n + 8,), 7.0, device="cuda")
            codec.decompress(b, eb, out=buf[p: p + n], avail=len(wire))
            codec.check()
            got = buf.cpu().numpy()
            assert np.array_equal(got[p: p + n].view(np.uint32), want)
            assert (got[:p] == 7).all() and (got[p + n:] == 7).all()


@pytest.mark.gpu
@pytest.mark.parametrize("bs", [2, 4, 8])
@pytest.mark.parametrize("dims", [(1500, 1501, 2), (600, 500, 5), (601, 603, 5), (380, 390, 8), (340, 340, 9), (3001, 3003, 1)])
def test_flat_volumes(port, bs, dims):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zccl_gb300.szp3d import Szp3D
    x, eb = volume(dims, False, bs), 1e-3
    codec = Szp3D(dims, bs)
    wire = port.szp3d_compress(x, dims, bs, eb)
    b = torch.from_numpy(np.frombuffer(wire, np.uint8).copy()).cuda()
    y = codec.decompress(b, eb, avail=len(wire))
    codec.check()
    assert np.array_equal(y.cpu().numpy().view(np.uint32), port.szp3d_decompress(wire, dims, bs, eb).view(np.uint32).ravel())


@pytest.mark.gpu
@pytest.mark.parametrize("dims,T", [((10, 34, 4000), 3), ((18, 18, 3000), 8)])
@pytest.mark.parametrize("bs", [2, 4, 8])
def test_sub_volumes_share_the_scratch(port, bs, dims, T):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from zccl_gb300.szp3d import Szp3D
    x, eb = volume(dims, False, bs), 1e-3
    codec = Szp3D(dims, bs, T=T)
    wire = port.szp3d_compress_split(x, dims, bs, eb, T)
    b = torch.from_numpy(np.frombuffer(wire, np.uint8).copy()).cuda()
    y = codec.decompress(b, eb, avail=len(wire))
    codec.check()
    want = port.szp3d_decompress_split(wire, dims, bs, eb, T)
    assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32).ravel())


def test_scratch_grows_with_the_volume():
    """A sub-volume never needs more scratch than the largest, which the
    OpenMP form's scratch is sized for."""
    import zccl_gb300 as Z
    try:
        ws = Z.lib().zccl_gpu_szp3d_workspace_bytes
    except OSError:
        pytest.skip("library not built")
    rng = np.random.default_rng(1)
    for _ in range(4000):
        d = [int(v) for v in 2 ** rng.uniform(0, 12, 3)]
        s = [max(1, int(v - rng.integers(0, 1 + v // 2))) for v in d]
        for bs in (2, 4, 8):
            assert ws(*s, bs) <= ws(*d, bs)
