"""The work that a user of scrs_b200 has it do, as measurable cases.

Every case runs one pass through the public entry points (the codec factories
of ``scrs_b200`` and ``scrs_b200.batch.StripeBatch``) on buffers that the
user's program holds.  Payload bytes are uniform random, as coded storage and
transport payloads (compressed or encrypted) are.  A decode's received rows
are random bytes too: the codes are MDS, so any k rows are k symbols of
exactly one codeword.  All outputs are finite-field results, bytes without
rounding, so there is no value in 64 bits to compare them with beyond the
bytes themselves.

Kinds of cases (``kind``):

* ``call``         one GF(256) stripe through the block encoder and the block
                   decoder, device buffers: the smallest work, one object at a
                   time;
* ``batch``        many equal stripes, half encoded and half decoded, in one
                   stripe batch on the device: a storage node's bulk work;
* ``mixed``        a stripe batch of uneven geometries;
* ``host``         a stripe batch whose buffers are pinned host memory;
* ``stream``       the per-symbol surface: an incremental encoder fed symbol by
                   symbol, a lazy decoder pushed symbol by symbol;
* ``afft_encode``  one large GF(2^16) additive-FFT block;
* ``afft_decode``  the same block decoded with ``lost`` data symbols missing
                   (-1: a random k of the k + m symbols arrive).

``lost`` has the same meaning in the other decodes.
"""
import math

import numpy as np
import torch

import scrs_b200
from scrs_b200.api import Engine
from scrs_b200.batch import OP_DECODE, OP_ENCODE, StripeBatch

_ENGINE = {"standard": Engine.STANDARD_CAUCHY, "good": Engine.GOOD_CAUCHY, "tower": Engine.TOWER, "afft": Engine.AFFT}
_MIXED_LENS = (1024, 4096, 65536)  # symbol lengths of the mixed batches: small objects, pages, large extents


def listed():
    return [
        # one object of 40 KB at a time, each call on its own: latency
        {"name": "call_10_4", "kind": "call", "engine": "good", "k": 10, "m": 4, "symbol_len": 4096, "lost": -1},
        # the bulk work of a storage node on the common 10 + 4 code with 4 KiB symbols
        {"name": "batch_10_4", "kind": "batch", "engine": "good", "k": 10, "m": 4, "symbol_len": 4096,
         "stripes": 131072, "lost": -1},
        # wider codes, for which the arithmetic per byte grows with m
        {"name": "batch_32_8", "kind": "batch", "engine": "good", "k": 32, "m": 8, "symbol_len": 4096,
         "stripes": 4096, "lost": -1},
        {"name": "batch_64_16", "kind": "batch", "engine": "standard", "k": 64, "m": 16, "symbol_len": 4096,
         "stripes": 2048, "lost": -1},
        # packets: 1400-byte symbols, rows that are not 16-byte aligned
        {"name": "batch_1400", "kind": "batch", "engine": "good", "k": 32, "m": 8, "symbol_len": 1400,
         "stripes": 8192, "lost": -1},
        # tenants with codes and sizes of their own in one launch
        {"name": "mixed", "kind": "mixed", "k_max": 64, "m_max": 16, "stripes": 8192},
        # objects in host memory: copies in and out are part of the pass
        {"name": "host_10_4", "kind": "host", "engine": "good", "k": 10, "m": 4, "symbol_len": 4096,
         "stripes": 8192, "lost": -1},
        # a sender and a receiver of 64 KiB symbols over the tower field
        {"name": "stream_tower", "kind": "stream", "engine": "tower", "k": 32, "m": 8, "symbol_len": 65536, "lost": 8},
        # the same code in bulk
        {"name": "batch_tower", "kind": "batch", "engine": "tower", "k": 32, "m": 8, "symbol_len": 65536,
         "stripes": 256, "lost": 8},
        # large blocks: encode at a power-of-two k, decode with half of the symbols gone
        {"name": "afft_encode_4096", "kind": "afft_encode", "engine": "afft", "k": 4096, "m": 4096, "symbol_len": 1024},
        {"name": "afft_decode_32768", "kind": "afft_decode", "engine": "afft", "k": 32768, "m": 16384,
         "symbol_len": 256, "lost": -1},
        # a large block that lost only two symbols, the usual loss on a good link
        {"name": "afft_decode_few", "kind": "afft_decode", "engine": "afft", "k": 4096, "m": 4096, "symbol_len": 1024,
         "lost": 2},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _length(rng, lo, hi, even):
    """A symbol length: whole pages, whole 16-byte units, or anything."""
    n = _log(rng, lo, hi)
    unit = rng.choice([512, 16, 2, 1])
    n = max(unit, n // unit * unit)
    return n + (n & 1) if even else n


def draw(rng):
    kind = rng.choice(["call", "batch", "batch", "batch", "tower", "mixed", "host", "stream", "afft_encode",
                       "afft_decode", "afft_decode"])
    k, m = rng.randint(2, 64), rng.randint(1, 16)
    lost = rng.choice([-1, -1, rng.randint(1, min(k, m))])
    if kind == "call":
        return {"kind": "call", "engine": rng.choice(["standard", "good"]), "k": k, "m": m,
                "symbol_len": _length(rng, 64, 65536, False), "lost": lost}
    if kind in ("batch", "tower", "host"):
        n = _length(rng, 512, 65536, kind == "tower")
        total = _log(rng, 1 << 24, {"batch": 1 << 30, "tower": 1 << 29, "host": 1 << 28}[kind])
        stripes = max(4, min(131072, total // (k * n)) // 2 * 2)
        return {"kind": "host" if kind == "host" else "batch",
                "engine": "tower" if kind == "tower" else rng.choice(["standard", "good"]), "k": k, "m": m,
                "symbol_len": n, "stripes": stripes, "lost": lost}
    if kind == "mixed":
        return {"kind": "mixed", "k_max": rng.randint(8, 64), "m_max": rng.randint(2, 16),
                "stripes": _log(rng, 256, 8192) // 2 * 2}
    if kind == "stream":
        return {"kind": "stream", "engine": rng.choice(["good", "tower"]), "k": k, "m": m,
                "symbol_len": _length(rng, 1024, 65536, True), "lost": max(lost, 1)}
    k, m = _log(rng, 32, 32768), _log(rng, 16, 16384)
    n = min(_length(rng, 64, 4096, True), max(64, (1 << 23) // k // 2 * 2))
    if kind == "afft_encode":
        return {"kind": kind, "engine": "afft", "k": k, "m": m, "symbol_len": n}
    return {"kind": kind, "engine": "afft", "k": k, "m": m, "symbol_len": n,
            "lost": rng.choice([-1, -1, min(2, m), min(5, m)])}


def _random(gen, count, pinned=False):
    x = torch.randint(0, 256, (count,), dtype=torch.uint8, device="cuda", generator=gen)
    if not pinned:
        return x
    h = torch.empty(count, dtype=torch.uint8, pin_memory=True)
    h.copy_(x)
    return h


def _zeros(count, pinned=False):
    return torch.zeros(count, dtype=torch.uint8, pin_memory=True) if pinned else torch.zeros(
        count, dtype=torch.uint8, device="cuda")


def _received(rng, stripes, k, m, lost):
    """The k symbols that arrive for each stripe, in arrival order."""
    keys = rng.random((stripes, k + m))
    if lost >= 0:  # that many data symbols never arrive: as many repairs do
        gone = np.argsort(rng.random((stripes, k)), axis=1)[:, :lost]
        extra = np.argsort(rng.random((stripes, m)), axis=1)[:, lost:] + k
        np.put_along_axis(keys, gone, 2.0, axis=1)
        np.put_along_axis(keys, extra, 2.0, axis=1)
    return np.argsort(keys, axis=1)[:, :k]


def _mixed_geometry(case, rng):
    s = case["stripes"]
    k = rng.integers(min(4, case["k_max"]), case["k_max"] + 1, s)
    m = rng.integers(1, case["m_max"] + 1, s)
    n = rng.choice(np.array(_MIXED_LENS), s)
    engine = rng.choice(np.array([int(Engine.STANDARD_CAUCHY), int(Engine.GOOD_CAUCHY)]), s)
    return engine, k, m, n


def _geometry_seed(case):
    return case["stripes"] * 131 + case["k_max"] * 17 + case["m_max"]


def _prepare_batch(case, rng, gen):
    lib = scrs_b200.api_default().lib
    host = case["kind"] == "host"
    s = case["stripes"]
    if case["kind"] == "mixed":  # the geometries belong to the case, the bytes and losses to the seed
        engine, k, m, n = _mixed_geometry(case, np.random.default_rng(_geometry_seed(case)))
    else:
        engine, k, m, n = (np.full(s, v) for v in (int(_ENGINE[case["engine"]]), case["k"], case["m"],
                                                   case["symbol_len"]))
    half = s // 2
    op = np.where(np.arange(s) < half, OP_ENCODE, OP_DECODE)
    unit = 256 if case["kind"] == "mixed" else 1  # separate objects start where an allocator puts them
    in_len = -(-(k * n) // unit) * unit
    out_len = -(-(np.where(op == OP_ENCODE, m, k) * n) // unit) * unit
    split = int(out_len[:half].sum())
    data = _random(gen, int(in_len.sum()), host)
    repairs, decoded = _zeros(split, host), _zeros(int(out_len.sum()) - split, host)
    in_at = data.data_ptr() + np.concatenate([[0], np.cumsum(in_len)[:-1]])
    out_at = np.concatenate([[0], np.cumsum(out_len)[:-1]])
    out_at = np.where(op == OP_ENCODE, repairs.data_ptr() + out_at, decoded.data_ptr() + out_at - split)
    indices = np.zeros((s, int(k.max())), dtype=np.uint16)
    if case["kind"] == "mixed":
        keys = rng.random((s, int((k + m).max())))
        keys[np.arange(keys.shape[1])[None, :] >= (k + m)[:, None]] = 2.0
        indices[:] = np.argsort(keys, axis=1)[:, :indices.shape[1]]
    else:
        indices[half:] = _received(rng, s - half, case["k"], case["m"], case["lost"])
    batch = StripeBatch(lib, s)
    batch.set_arrays(op, engine, k, m, n, in_at.astype(np.uint64), out_at.astype(np.uint64), indices=indices,
                     host=host)
    return {"kind": "batch", "batch": batch, "data": data, "out": {"repairs": repairs, "decoded": decoded}}


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind in ("batch", "mixed", "host"):
        return _prepare_batch(case, rng, gen)
    k, m, n = case["k"], case["m"], case["symbol_len"]
    profile = scrs_b200.resolve(_ENGINE[case["engine"]], k, m, n)
    state = {"kind": kind, "data": _random(gen, k * n)}
    if kind == "stream":
        enc, dec = scrs_b200.incremental_encoder(profile), scrs_b200.decoder(profile)
        order = _received(rng, 1, k, m, case["lost"])[0].tolist()
        rows = _random(gen, k * n)
        state.update(enc=enc, dec=dec, scratch=dec.scratch(), repairs=list(range(m)),
                     feeds=[(i, state["data"][i * n:(i + 1) * n]) for i in range(k)],
                     pushes=[(i, rows[q * n:(q + 1) * n]) for q, i in enumerate(order)], decoded=_zeros(k * n))

        class Rows:  # the encoder's repair rows where they are, on the device
            __cuda_array_interface__ = {"shape": (m * n,), "typestr": "|u1", "version": 3,
                                        "data": (enc.repair_device_ptr(0), False)}

        state["encoded"] = torch.as_tensor(Rows(), device="cuda")
        return state
    if kind in ("call", "afft_encode"):
        enc = scrs_b200.batch_encoder(profile)
        state.update(enc=enc, enc_scratch=enc.scratch(), encoded=_zeros(m * n))
    if kind in ("call", "afft_decode"):
        dec = scrs_b200.batch_decoder(profile)
        indices = _received(rng, 1, k, m, case["lost"])[0].astype(np.uint64)
        state.update(dec=dec, dec_scratch=dec.scratch(), symbols=(indices, _random(gen, k * n)), decoded=_zeros(k * n))
    return state


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].run()
        return state["out"]
    if kind == "stream":
        enc, dec = state["enc"], state["dec"]
        enc.reset()
        for index, symbol in state["feeds"]:
            enc.feed(index, symbol)
        for j in state["repairs"]:
            enc.repair_device_ptr(j)
        dec.reset()
        for index, symbol in state["pushes"]:
            dec.push(index, symbol)
        dec.finalize_into_with(state["decoded"], state["scratch"])
        return {"encoded": state["encoded"], "decoded": state["decoded"]}
    out = {}
    if "enc" in state:
        state["enc"].encode_into_with(state["data"], state["encoded"], state["enc_scratch"])
        out["encoded"] = state["encoded"]
    if "dec" in state:
        state["dec"].decode_into_with(state["symbols"], state["decoded"], state["dec_scratch"])
        out["decoded"] = state["decoded"]
    return out


def work(case):
    """Encode reads k rows and writes m, decode reads k rows and writes k; the
    field arithmetic is integer work, not floating point."""
    kind = case["kind"]
    if kind == "mixed":
        _, k, m, n = _mixed_geometry(case, np.random.default_rng(_geometry_seed(case)))
        enc = np.arange(case["stripes"]) < case["stripes"] // 2
        return {"bytes": int((np.where(enc, k + m, 2 * k) * n).sum()), "flops": 0}
    k, m, n = case["k"], case["m"], case["symbol_len"]
    encode, decode = (k + m) * n, 2 * k * n
    if kind in ("batch", "host"):
        half = case["stripes"] // 2
        return {"bytes": half * encode + (case["stripes"] - half) * decode, "flops": 0}
    return {"bytes": {"afft_encode": encode, "afft_decode": decode}.get(kind, encode + decode), "flops": 0}
