"""Work items of the persistent XOR drain: a CTA's first item is its own, the others
are claimed; item counts around the grid's size, against the oracle."""
import numpy as np
import pytest

from scenarios import device_stripes
from scrs_b200.api import Engine
from scrs_b200.batch import OP_DECODE, OP_ENCODE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [1, 3])
def test_item_counts_around_the_grid(gpu, oracle, ctas):
    torch = pytest.importorskip("torch")
    from scrs_b200 import tune
    from scrs_b200.batch import StripeBatch

    grid = torch.cuda.get_device_properties(0).multi_processor_count * ctas
    rng = np.random.default_rng(7 + ctas)
    tune.clear(gpu.lib)
    try:
        for n in (1, grid - 1, grid, grid + 1, 2 * grid + 3):
            specs = [(OP_ENCODE if s % 2 == 0 else OP_DECODE, Engine.GOOD_CAUCHY, 5, 3, 1040) for s in range(n)]
            stripes, outs, expect, keep = device_stripes(torch, oracle, specs, rng)
            b = StripeBatch(gpu.lib, n)
            b.set_jit(False)
            b.set(stripes)
            tune.set_entry(gpu.lib, b.tune_key, tune.TuneParams(5, ctas))
            assert b.launch_params.ctas_per_sm == ctas
            b.run()
            torch.cuda.synchronize()
            b.check()
            assert all(np.array_equal(o.cpu().numpy(), e) for o, e in zip(outs, expect)), n
    finally:
        tune.clear(gpu.lib)
