"""The tensor-core drain of stripe batches: geometries on both sides of its
tile edges (blocks of 256 columns, K = 64 steps of 8 or 4 input rows, units of
four steps, passes of 16 or 8 outputs, the largest input count it takes), with
rows of 16-byte units, 8-byte units and any length or address, encode and
decode, against the oracle.  Every batch holds enough blocks for the drain to be
chosen; its results are exact, so the comparison is byte for byte."""
import numpy as np
import pytest

from scenarios import device_stripes
from scrs_b200.api import Engine
from scrs_b200.batch import OP_DECODE, OP_ENCODE

pytestmark = pytest.mark.gpu

STRIPES = 1300  # one block or more each

GF8 = [(24, 12), (25, 16), (31, 9), (32, 8), (33, 17), (40, 32), (48, 6), (64, 16), (65, 5), (72, 33)]
TOWER = [(16, 2), (17, 3), (24, 8), (31, 1), (32, 9), (33, 8), (47, 16), (64, 7)]
LENGTHS = {16: (16, 240, 256, 272, 512, 1024), 8: (8, 120, 264, 504, 1400), 1: (1, 127, 255, 257, 513, 1001)}


def _specs(engine, geometries, lengths, rng):
    specs = []
    for s in range(STRIPES):
        k, m = geometries[int(rng.integers(len(geometries)))]
        L = int(lengths[int(rng.integers(len(lengths)))])
        if engine == Engine.TOWER:
            L += L & 1
        specs.append((OP_ENCODE if s % 2 == 0 else OP_DECODE, engine, k, m, L))
    return specs


def _check(torch, gpu, oracle, specs, rng):
    from scrs_b200.batch import StripeBatch

    stripes, outs, expect, keep = device_stripes(torch, oracle, specs, rng)
    b = StripeBatch(gpu.lib, len(stripes))
    b.set_jit(False)
    b.set(stripes)
    for graph in (False, True):
        for o in outs:
            o.zero_()
        b.run(graph=graph)
        torch.cuda.synchronize()
        b.check()
        bad = [specs[i] for i, (o, e) in enumerate(zip(outs, expect)) if not np.array_equal(o.cpu().numpy(), e)]
        assert not bad, (graph, len(bad), bad[:5])


@pytest.mark.parametrize("align", [16, 8, 1])
@pytest.mark.parametrize("engine", [Engine.STANDARD_CAUCHY, Engine.TOWER])
def test_geometries_and_alignments(gpu, oracle, engine, align):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(100 + align + int(engine))
    _check(torch, gpu, oracle, _specs(engine, TOWER if engine == Engine.TOWER else GF8, LENGTHS[align], rng), rng)


@pytest.mark.parametrize("align", [16, 8, 1])
@pytest.mark.parametrize("engine", [Engine.GOOD_CAUCHY, Engine.TOWER])
def test_narrow_codes(gpu, oracle, engine, align):
    """Codes on both sides of the lines between the two drains."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(300 + align + int(engine))
    codes = ([(5, 3), (6, 3), (8, 2), (8, 4), (10, 1), (12, 2), (16, 1)] if engine == Engine.TOWER else
             [(7, 4), (8, 6), (12, 4), (12, 8), (16, 16), (17, 1), (18, 8), (21, 5), (32, 4), (44, 4), (56, 2)])
    lengths = {16: (1008, 1040, 4096), 8: (1016, 1400, 2056), 1: (1023, 1401, 2049)}[align]
    _check(torch, gpu, oracle, _specs(engine, codes, lengths, rng), rng)


@pytest.mark.parametrize("engine,k,m", [(Engine.STANDARD_CAUCHY, 223, 16), (Engine.STANDARD_CAUCHY, 224, 16),
                                        (Engine.TOWER, 111, 8), (Engine.TOWER, 112, 8)])
def test_largest_input_counts(gpu, oracle, engine, k, m):
    """The most inputs the drain takes, and one more (the XOR networks)."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(k)
    specs = [(OP_ENCODE if s % 2 == 0 else OP_DECODE, engine, k, m, 4096) for s in range(160)]
    _check(torch, gpu, oracle, specs, rng)


def test_long_rows_and_mixed_classes(gpu, oracle):
    """Rows of many items, both fields and every alignment in one batch."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(9)
    specs = [(OP_ENCODE, Engine.GOOD_CAUCHY, 32, 8, 70000), (OP_DECODE, Engine.TOWER, 32, 8, 65536)] * 6
    specs += [(OP_DECODE, Engine.GOOD_CAUCHY, 32, 8, 70001), (OP_ENCODE, Engine.TOWER, 20, 5, 65544)] * 6
    specs += [(OP_ENCODE, Engine.GOOD_CAUCHY, 8, 3, 4096), (OP_DECODE, Engine.GOOD_CAUCHY, 64, 16, 66000)] * 6
    _check(torch, gpu, oracle, specs, rng)
