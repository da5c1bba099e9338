"""The tensor-core drain's work items stay within the count that a set checks
against the batch's capacity (2 KiB of a row each), so that a set that fits allocates
nothing, whichever drain its stripes take."""
import numpy as np
import pytest

from scrs_b200.api import Engine
from scrs_b200.batch import OP_ENCODE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine,k,m", [(Engine.GOOD_CAUCHY, 32, 8), (Engine.TOWER, 16, 4)])
def test_items_within_capacity(gpu, engine, k, m):
    torch = pytest.importorskip("torch")
    from scrs_b200.batch import Stripe, StripeBatch

    n, L = 400, 4096  # 800 items of 2 KiB
    d_in = torch.zeros(200 * 4096 * 200, dtype=torch.uint8, device="cuda")
    d_out = torch.zeros(200 * 4096 * 100, dtype=torch.uint8, device="cuda")

    def stripes(codes):
        a = c = 0
        out = []
        for e, q, r in codes:
            out.append(Stripe(OP_ENCODE, e, q, r, L, d_in.data_ptr() + a * L, d_out.data_ptr() + c * L))
            a, c = a + q, c + r
        return out

    b = StripeBatch(gpu.lib, n, 2 * n)
    b.set_jit(False)
    # as many items on the XOR networks, and a larger coefficient table
    b.set(stripes([(engine, 4, 2)] * (n - 1) + [(Engine.STANDARD_CAUCHY, 100, 100)]))
    assert b.tensor_stripes == 0
    allocs = gpu.lib.alloc_count()
    b.set(stripes([(engine, k, m)] * n))
    assert b.tensor_stripes == n
    assert gpu.lib.alloc_count() == allocs
