"""Unaligned encodes with 24 inputs or more, which leave their specialised kernel for
the tensor cores: only where those are launched, and back in the specialised group
where they are not."""
import numpy as np
import pytest

from scenarios import device_stripes
from scrs_b200.api import Engine
from scrs_b200.batch import OP_DECODE, OP_ENCODE

pytestmark = pytest.mark.gpu

GOOD = Engine.GOOD_CAUCHY


@pytest.mark.parametrize("others,specialised", [
    ([(OP_ENCODE, GOOD, 10, 4, 4096)] * 100, 1200),  # the encodes alone do not pay for a launch
    ([(OP_DECODE, GOOD, 24, 1, 1400)] * 1200, 0),    # with the decodes they do
])
def test_specialised_where_the_tensor_cores_are_not_launched(gpu, oracle, others, specialised):
    torch = pytest.importorskip("torch")
    from scrs_b200.batch import StripeBatch

    rng = np.random.default_rng(51)
    specs = [(OP_ENCODE, GOOD, 24, 1, 1400)] * 1200 + others
    specs = [specs[i] for i in rng.permutation(len(specs))]
    stripes, outs, expect, keep = device_stripes(torch, oracle, specs, rng)
    b = StripeBatch(gpu.lib, len(stripes))
    b.set(stripes)
    assert b.jit_stripes == specialised
    # every encode and every decode that lost a row, or none
    lossy = sum(s.indices is not None and max(s.indices) >= s.k for s in stripes)
    assert b.tensor_stripes == (0 if specialised else 1200 + lossy)
    for graph in (False, True):
        for o in outs:
            o.zero_()
        b.run(graph=graph)
        torch.cuda.synchronize()
        b.check()
        assert all(np.array_equal(o.cpu().numpy(), e) for o, e in zip(outs, expect))
