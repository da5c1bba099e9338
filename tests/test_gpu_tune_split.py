"""The autotuner's key and the XOR drain's segment size follow the stripes of that drain,
not those that drain on the tensor cores beside them."""
import numpy as np
import pytest

from scrs_b200.api import Engine
from scrs_b200.batch import DESC_DTYPE, OP_DECODE

pytestmark = pytest.mark.gpu

STD, GOOD = Engine.STANDARD_CAUCHY, Engine.GOOD_CAUCHY


def _descs(specs, d_in, d_out):
    """Decodes of the first m data rows of (engine, k, m, L) specs."""
    desc = np.zeros(len(specs), dtype=DESC_DTYPE)
    idx = np.zeros((len(specs), 64), dtype=np.uint16)
    at = 0
    for s, (engine, k, m, L) in enumerate(specs):
        idx[s, :k] = np.arange(m, k + m)
        desc[s] = (OP_DECODE, int(engine), k, m, L, d_in + at, d_out + at, idx.ctypes.data + s * 128)
        at += k * L
    return desc, idx


def _batch(gpu, specs, d_in, d_out):
    from scrs_b200.batch import StripeBatch

    desc, idx = _descs(specs, d_in, d_out)
    b = StripeBatch(gpu.lib, len(specs))
    b.set_arrays(desc["op"], desc["engine"], desc["k"], desc["m"], desc["symbol_len"], desc["in_"], desc["out"], indices=idx)
    return b


def test_key_and_segment_of_the_xor_drain(gpu):
    torch = pytest.importorskip("torch")
    from scrs_b200 import tune

    wide, narrow = [(STD, 64, 16, 4096)] * 300, [(GOOD, 10, 4, 4096)] * 500
    total = sum(k * L for _, k, _, L in wide + narrow)
    d_in = torch.zeros(total, dtype=torch.uint8, device="cuda")
    d_out = torch.zeros(total, dtype=torch.uint8, device="cuda")
    a, c = d_in.data_ptr(), d_out.data_ptr()

    def key_of(specs):
        desc, idx = _descs(specs, a, c)
        return tune.key_of(gpu.lib, desc)  # reads idx, kept alive here

    tune.clear(gpu.lib)
    try:
        mixed, alone, all_wide = (_batch(gpu, s, a, c) for s in (wide + narrow, narrow, wide))
        assert (mixed.tensor_stripes, alone.tensor_stripes, all_wide.tensor_stripes) == (300, 0, 300)
        assert mixed.tune_key == alone.tune_key == key_of(narrow)
        assert all_wide.tune_key == key_of(wide)
        # one segment holds every row of the XOR drain's stripes
        assert mixed.launch_params.seg_rows == alone.launch_params.seg_rows == 10
        assert all_wide.launch_params.seg_rows == 16
        chosen = mixed.autotune(reps=2)
        torch.cuda.synchronize()
        assert chosen.seg_rows <= 10
        assert [k for k, _ in tune.entries(gpu.lib)] == [alone.tune_key]
        # a batch that holds all of them on the XOR networks keeps its own key
        assert key_of(wide + narrow) != mixed.tune_key
    finally:
        tune.clear(gpu.lib)
