"""Which stripes drain on the tensor cores, and their results: every batch here
asserts how many of its stripes do (``tensor_stripes``), so that each instance of
the drain (both fields, rows of 16-byte units, of 8-byte units, at any address)
runs, with items of one and of many blocks, beside the other drains and right after
the plan kernel.  Results are exact: the comparison is byte for byte with the
oracle's codewords."""
import numpy as np
import pytest

from scenarios import encode_word
from scrs_b200.api import Engine
from scrs_b200.batch import OP_DECODE, OP_ENCODE

pytestmark = pytest.mark.gpu

STD, GOOD, TOWER = Engine.STANDARD_CAUCHY, Engine.GOOD_CAUCHY, Engine.TOWER
OFFSETS = {16: (0, 0), 8: (8, 8), 1: (3, 1)}  # of the input and output rows from aligned addresses


def _stripes(torch, oracle, specs, rng, align=16):
    """Device buffers for (op, engine, k, m, L, lost) specs; a decode loses exactly
    `lost` data rows.  Returns (stripes, output tensors, expected bytes, kept)."""
    from scrs_b200.batch import Stripe

    a, c = OFFSETS[align]
    stripes, outs, expect, keep = [], [], [], []
    for op, engine, k, m, L, lost in specs:
        data = rng.integers(0, 256, k * L, dtype=np.uint8)
        word = encode_word(oracle, oracle.resolve(engine, k, m, L), data)
        idx = None
        if op == OP_ENCODE:
            given, exp = data, np.concatenate(word[k:])
        else:
            gone = rng.choice(k, lost, replace=False).tolist()
            idx = [i for i in range(k) if i not in gone] + [k + j for j in rng.choice(m, lost, replace=False).tolist()]
            idx = rng.permutation(idx).tolist()
            given, exp = np.concatenate([word[i] for i in idx]), data
        d_in = torch.zeros(len(given) + a, dtype=torch.uint8, device="cuda")
        d_in[a:] = torch.from_numpy(given)
        d_out = torch.zeros(len(exp) + c + 1, dtype=torch.uint8, device="cuda")
        stripes.append(Stripe(op, engine, k, m, L, d_in.data_ptr() + a, d_out.data_ptr() + c, idx))
        expect.append(np.concatenate([np.zeros(c, np.uint8), exp, np.zeros(1, np.uint8)]))
        outs.append(d_out)
        keep.append(d_in)
    return stripes, outs, expect, keep


def _run_and_check(torch, b, outs, expect, graph):
    for o in outs:
        o.zero_()
    b.run(graph=graph)
    torch.cuda.synchronize()
    b.check()
    bad = [i for i, (o, e) in enumerate(zip(outs, expect)) if not np.array_equal(o.cpu().numpy(), e)]
    assert not bad, (graph, len(bad), bad[:5])


def _batch(gpu, stripes, jit=False):
    from scrs_b200.batch import StripeBatch

    b = StripeBatch(gpu.lib, len(stripes))
    b.set_jit(jit)
    b.set(stripes)
    return b


@pytest.mark.parametrize("align", [16, 8, 1])
@pytest.mark.parametrize("engine,k,m", [(GOOD, 24, 8), (TOWER, 16, 4)])
def test_items_of_many_blocks(gpu, oracle, engine, k, m, align):
    """Rows of about 1 MiB: enough blocks for the longest items, ragged ends."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(1000 + align + int(engine))
    step = {16: 16, 8: 24, 1: 34 if engine == TOWER else 17}[align]
    specs = [(OP_ENCODE if s % 2 else OP_DECODE, engine, k, m, (1 << 20) + (s + 1) * step // align * align, m - s % 3)
             for s in range(10)]
    stripes, outs, expect, keep = _stripes(torch, oracle, specs, rng, align)
    b = _batch(gpu, stripes)
    assert b.tensor_stripes == len(stripes)
    _run_and_check(torch, b, outs, expect, False)
    _run_and_check(torch, b, outs, expect, True)


# on the tensor cores' side of the lines, and next to them on the other
NARROW = [
    (GOOD, 16, [(OP_ENCODE, 16, 16), (OP_ENCODE, 18, 8), (OP_DECODE, 21, 5), (OP_DECODE, 32, 4), (OP_ENCODE, 56, 2)],
     [(OP_ENCODE, 16, 12), (OP_ENCODE, 18, 6), (OP_DECODE, 21, 4), (OP_DECODE, 32, 3), (OP_ENCODE, 56, 1)]),
    (STD, 8, [(OP_DECODE, 8, 1), (OP_ENCODE, 8, 6), (OP_ENCODE, 16, 1)], [(OP_DECODE, 7, 3), (OP_ENCODE, 8, 5), (OP_ENCODE, 15, 1)]),
    (GOOD, 1, [(OP_DECODE, 12, 4), (OP_DECODE, 16, 1), (OP_ENCODE, 12, 8), (OP_ENCODE, 17, 1)],
     [(OP_DECODE, 12, 3), (OP_DECODE, 15, 3), (OP_ENCODE, 12, 7), (OP_ENCODE, 16, 7)]),
    (TOWER, 16, [(OP_ENCODE, 8, 4), (OP_DECODE, 12, 2), (OP_DECODE, 16, 1)], [(OP_ENCODE, 8, 3), (OP_DECODE, 12, 1), (OP_DECODE, 7, 4)]),
    (TOWER, 8, [(OP_DECODE, 6, 1), (OP_ENCODE, 6, 3), (OP_ENCODE, 10, 1)], [(OP_DECODE, 5, 2), (OP_ENCODE, 6, 2), (OP_ENCODE, 9, 1)]),
    (TOWER, 1, [(OP_DECODE, 8, 1), (OP_ENCODE, 8, 4), (OP_ENCODE, 10, 1)], [(OP_DECODE, 7, 3), (OP_ENCODE, 8, 3), (OP_ENCODE, 9, 3)]),
]


@pytest.mark.parametrize("engine,align,on,off", NARROW)
def test_both_sides_of_the_lines(gpu, oracle, engine, align, on, off):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(2000 + align + int(engine))
    L = {16: 4096, 8: 4104, 1: 4102 if engine == TOWER else 4101}[align]
    count = 400
    for codes, share in ((on, count), (off, 0)):
        for op, k, m in codes:
            stripes, outs, expect, keep = _stripes(torch, oracle, [(op, engine, k, m, L, m)] * count, rng, align)
            b = _batch(gpu, stripes)
            assert b.tensor_stripes == share, (op, k, m)
            _run_and_check(torch, b, outs, expect, False)


@pytest.mark.parametrize("engine", [GOOD, TOWER])
def test_start_beside_the_plans(gpu, oracle, engine):
    """Batches that run in the plan kernel and one drain: the drain starts beside the
    plans, in the first run after a set as in later ones, with other losses each
    time (a coefficient read too early would be the last set's)."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3000 + int(engine))
    specs = [(OP_ENCODE if s % 3 == 0 else OP_DECODE, engine, 32, 8, 4096, 4 + s % 5) for s in range(400)]
    b = None
    for graph in (False, True, False, True):
        stripes, outs, expect, keep = _stripes(torch, oracle, specs, rng)
        b = b or _batch(gpu, stripes)
        b.set(stripes)
        assert b.tensor_stripes == len(stripes)
        _run_and_check(torch, b, outs, expect, graph)
        assert b.last_launches == 2
        _run_and_check(torch, b, outs, expect, graph)


def test_all_drains_in_one_batch(gpu, oracle):
    """Four tensor-core launches beside a specialised encode and both fields' XOR drains."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(4000)
    groups = [((STD, 64, 16, 4096), 16, 200), ((GOOD, 32, 8, 4101), 1, 300), ((TOWER, 32, 8, 4096), 16, 300),
              ((TOWER, 24, 6, 4102), 1, 300), ((TOWER, 3, 2, 1000), 1, 50)]
    stripes, outs, expect, keep = [], [], [], []
    for (engine, k, m, L), align, count in groups:
        specs = [(OP_ENCODE if s % 2 else OP_DECODE, engine, k, m, L, m - s % 2) for s in range(count)]
        for whole, part in zip((stripes, outs, expect, keep), _stripes(torch, oracle, specs, rng, align)):
            whole.extend(part)
    specs = [(OP_ENCODE, GOOD, 10, 4, 4096, 0)] * 600 + [(OP_DECODE, GOOD, 10, 4, 4096, 2)] * 50
    for whole, part in zip((stripes, outs, expect, keep), _stripes(torch, oracle, specs, rng)):
        whole.extend(part)
    b = _batch(gpu, stripes, jit=True)
    assert (b.tensor_stripes, b.jit_stripes) == (1100, 600)
    _run_and_check(torch, b, outs, expect, False)
    _run_and_check(torch, b, outs, expect, True)
    assert b.last_launches == 9  # two plans, a specialised drain, two XOR drains, four tensor-core drains
