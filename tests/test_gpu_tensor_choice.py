"""Which batches send stripes to the tensor cores: those whose runs were measured
faster for it.  Codes near the lines between the drains, short rows and the share that
a mixed-loss batch leaves to the XOR networks (a launch of its own) were slower."""
import numpy as np
import pytest

from scenarios import device_stripes
from scrs_b200.api import Engine
from scrs_b200.batch import OP_DECODE, OP_ENCODE

pytestmark = pytest.mark.gpu

GOOD, TOWER = Engine.GOOD_CAUCHY, Engine.TOWER


def _random_loss(rng, k, m):
    return rng.permutation(k + m)[:k].tolist()


# (engine, k, m, symbol length, op, stripes): us of the whole run on the XOR networks, split
SLOWER = [
    (GOOD, 32, 4, 4096, OP_DECODE, 1280),   # 113, 138
    (GOOD, 44, 4, 4096, OP_DECODE, 930),    # 118, 149
    (GOOD, 56, 2, 4096, OP_DECODE, 731),    # 116, 129
    (TOWER, 12, 2, 1024, OP_DECODE, 8192),  # 245, 281 at 13653 stripes
    (TOWER, 12, 2, 2048, OP_DECODE, 6826),  # 134, 170
    (TOWER, 10, 1, 34, OP_ENCODE, 8192),    # 737, 932 at 65536 stripes
    (TOWER, 10, 1, 264, OP_DECODE, 8192),   # 888, 1100 at 63550 stripes
    (GOOD, 12, 3, 264, OP_DECODE, 8192),
]
# the same, on the XOR networks and with the tensor cores
FASTER = [
    (GOOD, 32, 8, 4096, OP_DECODE, 1280),   # 161, 131
    (TOWER, 32, 8, 4096, OP_DECODE, 1280),
    (GOOD, 32, 8, 1400, OP_DECODE, 3744),   # 632, 130
    (TOWER, 16, 4, 1024, OP_DECODE, 4096),
    (GOOD, 32, 8, 100, OP_ENCODE, 8192),
    (TOWER, 10, 1, 4102, OP_DECODE, 4096),
]


@pytest.mark.parametrize("case,taken", [(c, False) for c in SLOWER] + [(c, True) for c in FASTER])
def test_runs_measured_faster(gpu, case, taken):
    torch = pytest.importorskip("torch")
    from scrs_b200.batch import Stripe, StripeBatch

    engine, k, m, L, op, n = case
    rng = np.random.default_rng(n + k)
    d_in = torch.zeros(n * k * L, dtype=torch.uint8, device="cuda")
    d_out = torch.zeros(n * max(k, m) * L, dtype=torch.uint8, device="cuda")
    rows = k if op == OP_DECODE else m
    b = StripeBatch(gpu.lib, n)
    b.set_jit(False)
    b.set([Stripe(op, engine, k, m, L, d_in.data_ptr() + s * k * L, d_out.data_ptr() + s * rows * L,
                  _random_loss(rng, k, m) if op == OP_DECODE else None) for s in range(n)])
    assert (b.tensor_stripes > n // 2) if taken else b.tensor_stripes == 0


def test_unaligned_class_beside_others(gpu, oracle):
    """A few hundred stripes of unaligned rows are worth a launch beside other drains."""
    torch = pytest.importorskip("torch")
    from scrs_b200.batch import StripeBatch

    rng = np.random.default_rng(12)
    specs = [(OP_DECODE if s % 2 else OP_ENCODE, GOOD, 32, 8, 1400) for s in range(400)]
    specs += [(OP_DECODE, GOOD, 6, 3, 4096)] * 200
    stripes, outs, expect, keep = device_stripes(torch, oracle, specs, rng)
    b = StripeBatch(gpu.lib, len(stripes))
    b.set(stripes)
    assert 350 < b.tensor_stripes <= 400
    for graph in (False, True):
        for o in outs:
            o.zero_()
        b.run(graph=graph)
        torch.cuda.synchronize()
        b.check()
        assert all(np.array_equal(o.cpu().numpy(), e) for o, e in zip(outs, expect))
