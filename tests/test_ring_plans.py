"""The ring allreduce's kept plans: a bound that changes with every call does not
make them grow, and an input buffer that a plan does not fit -- other type,
stride or length, also at an address that was planned before -- is refused, not
read.  Results are those of the ring without plans."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, P = 24001, 4


@pytest.fixture(scope="module")
def torch():
    t = pytest.importorskip("torch")
    if not t.cuda.is_available():
        pytest.skip("no CUDA device")
    return t


def ranks(torch, seed):
    rng = np.random.default_rng(seed)
    base = np.cumsum(rng.normal(0, 0.01, COUNT))
    return [torch.from_numpy((base + rng.normal(0, 0.02, COUNT)).astype(np.float32)).cuda() for _ in range(P)]


@pytest.mark.parametrize("variant", ["homomorphic", "doc"])
def test_plans_do_not_grow_with_the_bounds(torch, variant):
    from zccl_gb300.ring import RingAllreduce
    ring, plain = RingAllreduce(COUNT, P), RingAllreduce(COUNT, P, batched=False)
    xs, most = ranks(torch, 1), 0
    bounds = [1e-3 * (1 + 0.1 * k) for k in range(12)] + [1.0, 2.0, 1e-3, 1e-3, 2e-3, 1e-3]
    for k, eb in enumerate(bounds):
        y = getattr(ring, variant)(xs, eb)
        assert torch.equal(y, getattr(plain, variant)(xs, eb))
        if k == 5:
            most = len(ring._plans)
        if k > 5:
            assert len(ring._plans) <= most
    # the bound before the last is still there (but for the one compression of the inputs)
    before = {k: b for k, b in ring._plans.items() if k[:2] != ("ho", "compress")}
    getattr(ring, variant)(xs, 2e-3)
    assert all(ring._plans.get(k) is b for k, b in before.items())


def test_inputs_that_do_not_fit_are_refused(torch):
    from zccl_gb300.ring import RingAllreduce
    ring = RingAllreduce(COUNT, P)
    flat = torch.zeros(P, 2 * COUNT + 8, device="cuda")
    xs = ranks(torch, 2)
    for row, x in zip(flat, xs):
        row[:COUNT] = x
    good = [row[:COUNT] for row in flat]
    want = ring.homomorphic(good, 1e-3).clone()
    bad = [[row[: COUNT - 1] for row in flat],            # too short, at the planned addresses
           [row[: 2 * COUNT: 2] for row in flat],         # every second float
           [row[:COUNT].view(torch.int32) for row in flat],
           [x.double() for x in xs], good[:-1] + [xs[-1].half()]]
    for b in bad:
        with pytest.raises(ValueError):
            ring.homomorphic(b, 1e-3)
    assert torch.equal(ring.homomorphic([row[: COUNT + 8] for row in flat], 1e-3), want)  # longer: its first floats
    assert torch.equal(ring.homomorphic(good, 1e-3), want)
