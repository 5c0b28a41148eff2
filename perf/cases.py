"""The measured workloads: what programs that use this library call, over the
sizes, layouts and options they call it with.

The library sits where ZCCL's codec sits: a simulation's float32 field or a
rank's message buffer is compressed within an error bound, sent, summed in
compressed form, and decompressed.  Accordingly the cases are single codec
calls on resident data (the device API), streams that arrive as bytes, whole
reductions over P ranks' buffers, batches of uneven buffers, the 3-D codec,
the smallest messages, and the reference's own entry points on host memory.

Streams are written into buffers of the largest size a stream can take, which
start zeroed, and a stream is returned with its whole buffer.  Floats are compared with the codec's definition in 64
bits: q = trunc(x * (1.0f / eb)), x' = q * eb (3-D: q = floor(x * 0.5 / eb +
0.5), x' = q * 2 eb).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import zccl_gb300 as Z
from zccl_gb300.ring import RingAllreduce
from zccl_gb300.szp3d import Szp3D

DEV = "cuda"

# Compression ratios (4 bytes per float / stream bytes per float) these data
# reach at these relative bounds, rounded, to count a stream's bytes in work().
RATIO = {
    ("field", 1e-3): 9.5, ("field", 1e-4): 6.0, ("field", 1e-5): 4.1,
    ("signal", 1e-3): 5.5, ("signal", 1e-4): 3.5, ("signal", 1e-5): 2.6,
    ("ranks", 1e-3): 5.0, ("ranks", 1e-4): 3.3, ("ranks", 1e-5): 2.5,
    ("laplace", 0.0): 2.6,
}


# --------------------------------------------------------------------------
# Inputs
# --------------------------------------------------------------------------

def _gen(seed: int):
    return torch.Generator(device=DEV).manual_seed(seed & 0x7FFFFFFFFFFFFFFF)


def _field(dims, seed: int):
    """A log-normal random field with P(k) ~ k^-3 (a density-like snapshot of
    a simulation), flattened with the last axis fastest."""
    d1, d2, d3 = dims
    g = _gen(seed)
    k2 = (torch.fft.fftfreq(d1, device=DEV)[:, None, None] ** 2
          + torch.fft.fftfreq(d2, device=DEV)[None, :, None] ** 2
          + torch.fft.rfftfreq(d3, device=DEV)[None, None, :] ** 2)
    amp = torch.where(k2 > 0, k2.clamp_min(1e-12) ** (-0.75), torch.zeros_like(k2))
    spec = torch.complex(torch.randn(k2.shape, generator=g, device=DEV),
                         torch.randn(k2.shape, generator=g, device=DEV)) * amp
    f = torch.fft.irfftn(spec, s=(d1, d2, d3))
    f = (f - f.mean()) / f.std()
    return torch.exp(1.5 * f).reshape(-1).contiguous().float()


def _signal(n: int, seed: int):
    """Two sines and a little noise: an oscillating 1-D record."""
    i = torch.arange(n, device=DEV, dtype=torch.float64)
    x = torch.sin(i * (2 * math.pi / 4096)) + 0.3 * torch.sin(i * (2 * math.pi / 97))
    return (x + 0.01 * torch.randn(n, generator=_gen(seed), device=DEV, dtype=torch.float64)).float()


def _ranks(n: int, P: int, seed: int):
    """P ranks' buffers: a shared smooth base and each rank's own noise."""
    g = _gen(seed)
    i = torch.arange(n, device=DEV, dtype=torch.float64)
    period = (500 + 49500 * torch.rand(8, generator=g, device=DEV, dtype=torch.float64)).tolist()
    phase = (2 * math.pi * torch.rand(8, generator=g, device=DEV, dtype=torch.float64)).tolist()
    base = torch.zeros(n, device=DEV, dtype=torch.float64)
    for p, f in zip(period, phase):
        base += torch.sin(2 * math.pi * i / p + f)
    return [(base + 0.05 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64)).float() for _ in range(P)]


def _inputs(case, seed: int):
    """The case's P float32 arrays and their error bound, rel x range."""
    P = case.get("P", 1)
    if case["data"] == "field":
        xs = [_field(_dims(case), 1000003 * seed + p) for p in range(P)]
    elif case["data"] == "signal":
        xs = [_signal(case["n"], 1000003 * seed + p) for p in range(P)]
    else:
        xs = _ranks(case["n"], P, seed)
    lo = min(float(x.min()) for x in xs)
    hi = max(float(x.max()) for x in xs)
    return xs, float(np.float32(case["rel"] * (hi - lo)))


def _buckets(case, seed: int):
    """Pairs of equal-size gradient buckets: log-uniform sizes, Laplace
    values, one pair in twenty constant, a bound per pair."""
    rng = np.random.default_rng(case["shapes"])
    k = case["pairs"]
    sizes = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), k)).astype(np.int64)
    const = rng.random(k) < 0.05
    rel = rng.choice([1e-3, 1e-4, 1e-5], k)
    g = _gen(seed)
    pairs, ebs = [], []
    for n, c, r in zip(sizes.tolist(), const, rel):
        if c:
            xs = [torch.full((n,), 0.5, device=DEV), torch.full((n,), 0.25, device=DEV)]
            span = 0.25
        else:
            u = (torch.rand(2 * n, generator=g, device=DEV) - 0.5).clamp_(-0.4999999, 0.4999999)
            v = -1e-3 * torch.sign(u) * torch.log1p(-2 * u.abs())
            xs = [v[:n], v[n:].clone()]
            span = 0.02  # the spread of a Laplace(0, 1e-3) sample of these sizes
        pairs.append(xs)
        ebs.append(float(np.float32(r * span)))
    return pairs, ebs


def _dims(case):
    return case["d1"], case["d2"], case["d3"]


def _n(case) -> int:
    return math.prod(_dims(case)) if "d1" in case else case["n"]


# --------------------------------------------------------------------------
# The cases
# --------------------------------------------------------------------------

def listed():
    return [
        # A simulation snapshot of 512^3 floats compressed where it lies, as a
        # 16-thread writer lays the stream out: the largest single buffer.
        {"name": "compress-512cube", "kind": "compress", "data": "field", "d1": 512, "d2": 512, "d3": 512, "rel": 1e-4,
         "L": 32, "T": 16},
        # The same snapshot read back from its resident stream.
        {"name": "decompress-512cube", "kind": "decompress", "data": "field", "d1": 512, "d2": 512, "d3": 512, "rel": 1e-4,
         "L": 32, "T": 16},
        # Two ranks' snapshots summed in compressed form, the reduce step of
        # the homomorphic allreduce.
        {"name": "add-512cube", "kind": "add", "data": "field", "d1": 512, "d2": 512, "d3": 512, "rel": 1e-4,
         "L": 32, "T": 16, "P": 2},
        # A 1-D record that arrived over the wire: bytes only, so its index is
        # rebuilt before it is decompressed; an odd length with a remainder
        # segment.
        {"name": "wire-decompress-64M", "kind": "wire", "data": "signal", "n": 67108877, "rel": 1e-4,
         "L": 32, "T": 16},
        # One message of a small allreduce (4096 floats): compress, sum with a
        # peer's, decompress the sum; nothing but latency.
        {"name": "message-4K", "kind": "roundtrip", "data": "signal", "n": 4096, "rel": 1e-4, "L": 32, "T": 1, "P": 2},
        # The reference's own scripts run with blocks of 36 elements: the same
        # three calls on a 16M-float record of an odd length.
        {"name": "roundtrip-L36-16M", "kind": "roundtrip", "data": "signal", "n": 16777259, "rel": 1e-4,
         "L": 36, "T": 8, "P": 2},
        # The homomorphic ring allreduce of 8 ranks, 16M floats each.
        {"name": "ring-homomorphic-8x16M", "kind": "ring", "variant": "homomorphic", "data": "ranks", "n": 1 << 24,
         "rel": 1e-4, "L": 32, "T": 16, "P": 8},
        # The decompress-add-recompress ring it is measured against, on an
        # uneven count.
        {"name": "ring-doc-8x8M", "kind": "ring", "variant": "doc", "data": "ranks", "n": 8400001,
         "rel": 1e-4, "L": 32, "T": 16, "P": 8},
        # Gradient buckets of one training step, 1024 floats to 4M: all
        # compressed, then summed pair by pair, one launch each.
        {"name": "buckets-256", "kind": "batch", "pairs": 256, "lo": 1024, "hi": 4 << 20, "shapes": 7, "L": 32, "T": 1},
        # The 3-D codec on the snapshot, blocks of 4^3.
        {"name": "szp3d-compress-512cube-bs4", "kind": "szp-compress", "data": "field", "d1": 512, "d2": 512, "d3": 512,
         "rel": 1e-4, "bs": 4},
        # The 3-D codec's reader on a volume whose sides are no multiples of
        # its 8^3 blocks.
        {"name": "szp3d-decompress-ragged-bs8", "kind": "szp-decompress", "data": "field", "d1": 301, "d2": 450, "d3": 517,
         "rel": 1e-4, "bs": 8},
        # A program relinked from the reference library: its entry points on
        # ordinary host arrays, copies included.
        {"name": "host-dropin-4M", "kind": "host", "data": "signal", "n": 4194304, "rel": 1e-4, "L": 32, "T": 8, "P": 2},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["compress", "decompress", "add", "wire", "roundtrip", "ring", "batch", "szp-compress",
                       "szp-decompress", "host"])
    rel = rng.choice([1e-3, 1e-4, 1e-4, 1e-5])
    T = rng.choice([1, 8, 16, 16, 72])
    if kind in ("szp-compress", "szp-decompress"):
        return {"kind": kind, "data": "field", "d1": _log_int(rng, 40, 510), "d2": _log_int(rng, 40, 510),
                "d3": _log_int(rng, 40, 510), "rel": rel, "bs": rng.choice([2, 4, 4, 8, 8])}
    if kind == "batch":
        return {"kind": kind, "pairs": rng.randint(20, 250), "lo": 1024, "hi": _log_int(rng, 1 << 16, 4 << 20),
                "shapes": rng.randint(0, 1 << 30), "L": 32, "T": 1}
    if kind == "ring":
        return {"kind": kind, "variant": rng.choice(["homomorphic", "doc"]), "data": "ranks",
                "n": _log_int(rng, 1 << 16, 8 << 20), "rel": rel, "L": 32, "T": rng.choice([1, 8, 16]),
                "P": rng.randint(2, 8)}
    if kind in ("compress", "decompress", "add") and rng.random() < 0.5:
        c = {"kind": kind, "data": "field", "d1": _log_int(rng, 64, 500), "d2": _log_int(rng, 64, 500),
             "d3": _log_int(rng, 64, 500), "rel": rel, "L": 32, "T": T}
        if kind == "add":
            c["P"] = rng.randint(2, 4)
        return c
    c = {"kind": kind, "data": "signal", "n": _log_int(rng, 1 << 16, 64 << 20), "rel": rel,
         "L": rng.choice([32, 32, 32, 36]), "T": T}
    if kind == "add":
        c["P"] = rng.randint(2, 4)
    elif kind == "roundtrip":
        c["n"] = _log_int(rng, 1 << 12, 16 << 20)
        c["P"] = 2
    elif kind == "host":
        c["n"] = _log_int(rng, 1 << 14, 4 << 20)
        c["P"] = 2
    return c


def _stream_bytes(case) -> float:
    return 4.0 * _n(case) / RATIO[case["data"], case["rel"]]


def work(case):
    """Bytes: each input read and each output written once (streams at the
    ratios above).  Operations: one multiply per quantized and one per
    reconstructed float, one add per float summed."""
    kind = case["kind"]
    if kind == "batch":
        rng = np.random.default_rng(case["shapes"])
        n = float(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["pairs"])).astype(np.int64).sum())
        c = 4 * n / RATIO["laplace", 0.0]
        return {"bytes": 2 * (4 * n + c) + (2 * c + c), "flops": 3 * n}
    n, c, P = float(_n(case)), _stream_bytes(case), case.get("P", 1)
    if kind == "add":
        return {"bytes": (P + 1) * c, "flops": (P - 1) * n}
    if kind in ("roundtrip", "host"):  # compress, add, decompress
        return {"bytes": (4 * n + c) + 3 * c + (c + 4 * n), "flops": 3 * n}
    if kind == "ring":  # every rank's floats in, the reduced floats out
        return {"bytes": (P + 1) * 4 * n, "flops": (2 * P) * n}
    return {"bytes": 4 * n + c, "flops": n}


# --------------------------------------------------------------------------
# What a program has in hand, one pass, and the values in 64 bits
# --------------------------------------------------------------------------

def _arena(codecs):
    """A zeroed buffer that holds one stream of every codec, and the streams."""
    at = [0]
    for c in codecs:
        at.append(at[-1] + (c.max_stream_bytes + 255) // 256 * 256)
    buf = torch.zeros(at[-1], dtype=torch.uint8, device=DEV)
    return buf, [Z.DeviceStream(c, data=buf[o: o + c.max_stream_bytes]) for c, o in zip(codecs, at)]


def prepare(case, seed: int):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "batch":
        pairs, ebs = _buckets(case, seed)
        codecs = [Z.Codec(xs[0].numel(), case["L"], case["T"], device=DEV) for xs in pairs]
        arenas = [_arena(codecs) for _ in range(3)]
        comp, sums = [], []
        for k, (xs, eb) in enumerate(zip(pairs, ebs)):
            a, b, out = (streams[k] for _, streams in arenas)
            comp += [(xs[0], eb, case["T"], a), (xs[1], eb, case["T"], b)]
            sums.append(([a, b], case["T"], out))
        bc = Z.Batch(Z.BATCH_COMPRESS, comp, case["L"], device=DEV)
        bh = Z.Batch(Z.BATCH_HOMADD, sums, case["L"], device=DEV)
        bc.run()
        bh.run()
        bc.check()
        bh.check()
        for buf, _ in arenas:
            buf.zero_()
        st.update(bc=bc, bh=bh, keep=(pairs, arenas), bufs=[buf for buf, _ in arenas])
        return st
    xs, eb = _inputs(case, seed)
    st["eb"] = eb
    if kind == "ring":
        st["xs"] = xs
        st["ring"] = RingAllreduce(case["n"], case["P"], case["L"], case["T"], device=DEV)
        return st
    if kind in ("szp-compress", "szp-decompress"):
        codec = Szp3D(_dims(case), case["bs"], device=DEV)
        buf = torch.zeros(codec.max_bytes, dtype=torch.uint8, device=DEV)
        _, size = codec.compress(xs[0], eb, out=buf)
        nbytes = codec.size(size)
        codec.check()
        st["codec"] = codec
        if kind == "szp-compress":
            buf.zero_()
            st.update(x=xs[0], buf=buf)
        else:
            st.update(s=buf[:nbytes].clone(), y=torch.zeros(_n(case), dtype=torch.float32, device=DEV))
        return st
    if kind == "host":
        n = case["n"]
        st["x"] = xs[0].cpu().numpy()
        st["out"] = np.zeros(4 * n + 4096, np.uint8)
        st["sum"] = np.zeros(4 * n + 4096, np.uint8)
        st["y"] = np.zeros(n, np.float32)
        peer = np.zeros(4 * n + 4096, np.uint8)
        Z.set_omp_threads(case["T"])
        Z.ZCCL_float_openmp_threadblock_arg(peer, xs[1].cpu().numpy(), 0, eb, n, case["L"])
        st["peer"] = peer
        return st
    codec = Z.Codec(_n(case), case["L"], case["T"], device=DEV)
    st["codec"] = codec
    streams = [codec.compress(x, eb) for x in xs]
    if kind == "compress":
        streams[0].buf.zero_()
        st.update(x=xs[0], s=streams[0], bufs=[streams[0].buf])
    elif kind == "decompress":
        st.update(s=streams[0], y=torch.zeros(codec.n, dtype=torch.float32, device=DEV))
    elif kind == "wire":
        st.update(b=streams[0].buf[: streams[0].size()].clone(),
                  y=torch.zeros(codec.n, dtype=torch.float32, device=DEV))
    elif kind == "add":
        out = codec.homadd(streams)
        out.buf.zero_()
        st.update(ins=streams, out=out, bufs=[out.buf])
    else:  # roundtrip: this rank's floats, a peer's resident stream
        out = codec.homadd(streams)
        streams[0].buf.zero_()
        out.buf.zero_()
        st.update(x=xs[0], s=streams[0], peer=streams[1], out=out, bufs=[streams[0].buf, out.buf],
                  y=torch.zeros(codec.n, dtype=torch.float32, device=DEV))
    codec.check()
    return st


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["bc"].run()
        state["bh"].run()
        return state["bufs"]
    eb = state["eb"]
    if kind == "ring":
        ring = state["ring"]
        return ring.homomorphic(state["xs"], eb) if state["case"]["variant"] == "homomorphic" \
            else ring.doc(state["xs"], eb)
    if kind == "host":
        n, L = state["case"]["n"], state["case"]["L"]
        Z.set_omp_threads(state["case"]["T"])
        Z.ZCCL_float_openmp_threadblock_arg(state["out"], state["x"], 0, eb, n, L)
        Z.ZCCL_float_homomophic_add_openmp_threadblock(state["sum"], 0, n, eb, L, state["out"], state["peer"])
        Z.ZCCL_float_decompress_openmp_threadblock_arg(state["y"], n, eb, L, state["sum"])
        return [state["out"], state["sum"], state["y"]]
    codec = state["codec"]
    if kind == "szp-compress":
        codec.compress(state["x"], eb, out=state["buf"])
        return [state["buf"]]
    if kind == "szp-decompress":
        return [codec.decompress(state["s"], eb, out=state["y"])]
    if kind == "compress":
        codec.compress(state["x"], eb, out=state["s"])
        return state["bufs"]
    if kind == "decompress":
        return [codec.decompress(state["s"], eb, out=state["y"])]
    if kind == "wire":
        s = Z.DeviceStream.from_bytes(codec, state["b"])
        return [codec.decompress(s, eb, out=state["y"])]
    if kind == "add":
        codec.homadd(state["ins"], out=state["out"])
        return state["bufs"]
    codec.compress(state["x"], eb, out=state["s"])
    codec.homadd([state["s"], state["peer"]], out=state["out"])
    return state["bufs"] + [codec.decompress(state["out"], eb, out=state["y"])]


def _quantized(x, eb: float):
    """trunc of the exact product with the float reciprocal, as float64."""
    return torch.trunc(x.double() * float(np.float32(1.0) / np.float32(eb)))


def exact(case, seed: int):
    kind = case["kind"]
    if kind in ("batch", "compress", "add", "szp-compress"):
        return None  # streams: bytes
    xs, eb = _inputs(case, seed)
    if kind == "szp-decompress":
        return [torch.floor(xs[0].double() * (0.5 / eb) + 0.5) * (2 * eb)]
    if kind in ("decompress", "wire"):
        return [_quantized(xs[0], eb) * eb]
    if kind == "roundtrip":
        return [None, None, (_quantized(xs[0], eb) + _quantized(xs[1], eb)) * eb]
    if kind == "host":
        return [None, None, ((_quantized(xs[0], eb) + _quantized(xs[1], eb)) * eb).cpu().numpy()]
    if case["variant"] == "homomorphic":
        return sum(_quantized(x, eb) for x in xs) * eb
    # decompress-add-recompress: chunk c travels from rank c to rank c - 1
    # around the ring, each rank adding what it receives to its own floats
    P, n = case["P"], case["n"]
    c = (n + P - 1) // P
    out = []
    for k in range(P):
        lo, hi = min(k * c, n), min((k + 1) * c, n)
        acc = xs[(k + 1) % P][lo:hi].double()
        for i in range(2, P + 1):
            acc = _quantized(acc, eb) * eb + xs[(k + i) % P][lo:hi].double()
        out.append(_quantized(acc, eb) * eb)
    return torch.cat(out)
