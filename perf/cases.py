"""The work that programs have this engine do, as cases that can be timed.

A case is one call of a public ``Engine`` entry point on a batch, with the
sizes, precisions and options that the tests, the benchmark, the queries and
the drop-in header use:

* ``gate``       HomGate over device batches (key switch + lvl01 bootstrap)
* ``gate_host``  the same through the synchronous host-buffer call
* ``compare``    comparison chains of encrypted columns, lvl1 and lvl2
* ``keyswitch``  identity key switches lvl1 -> lvl0, lvl2 -> lvl0, lvl2 -> lvl1
* ``extprod``    external products, one TRGSW per product, lvl1 and lvl2
* ``arc``        ArcEDB digit comparisons
* ``transform``  the standalone transforms, both directions, lvl1 and lvl2

All cases of a process share one context with one key set, tuned once, as a
query program keeps it.  Ciphertexts come from the seed; where a path's cost
and results do not depend on what is encrypted (key switches, external
products, ArcEDB digits) they are uniform words, which is how ciphertexts
and TRGSWs are distributed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cufhedb_b200 import FP64, GATES, GEN_ALL, MU1, N0, N1, N2, SPLIT32, Engine
from cufhedb_b200.queries import encrypt_column

KEY_SEED = 0x5EED_B200
PRECISION = {"fp64": FP64, "split32": SPLIT32}
GATE_NAMES = sorted(GATES)
COMPARE_OPS = ["gt", "ge", "lt", "le", "eq"]

# bytes of the bootstrapping keys and algorithmic flop of one bootstrap
# (672 CMux of l digit transforms, two inverse transforms and the products)
BK01_BYTES, BK02_BYTES = 66_060_288, 176_160_768
PBS01_FLOP, PBS02_FLOP = 156_893_184, 432_144_384
EXTPROD_FLOP = {1: 233_472, 2: 643_072}
TRGSW_BYTES = {1: 98_304, 2: 262_144}

_engine = None


def engine() -> Engine:
    """the process's context: all keys, launch shapes measured once"""
    global _engine
    if _engine is None:
        _engine = Engine(0)
        _engine.keygen(KEY_SEED, GEN_ALL)
        _engine.autotune()
    return _engine


def listed():
    return [
        # one gate: the latency a program that evaluates a circuit gate by gate sees
        {"name": "gate_split32_1", "kind": "gate", "gate": "NAND", "precision": "split32", "rows": 1},
        # the rows of 48 host threads that arrive together, at the default precision
        {"name": "gate_fp64_48", "kind": "gate", "gate": "AND", "precision": "fp64", "rows": 48},
        # the benchmark's batch
        {"name": "gate_split32_1024", "kind": "gate", "gate": "NAND", "precision": "split32", "rows": 1024},
        # a longer, ragged batch at the default precision
        {"name": "gate_fp64_1500", "kind": "gate", "gate": "XOR", "precision": "fp64", "rows": 1500},
        # host buffers in, host buffer out, synchronous
        {"name": "gate_host_split32_1000", "kind": "gate_host", "gate": "OR", "precision": "split32", "rows": 1000},
        # a small column filter at lvl1 (three bootstraps a row)
        {"name": "compare_lvl1_6bit_300", "kind": "compare", "level": 1, "op": "le", "bits": 6, "logic": True,
         "precision": "split32", "rows": 300},
        # a few rows against an encrypted constant at lvl2, default precision
        {"name": "compare_lvl2_16bit_24", "kind": "compare", "level": 2, "op": "lt", "bits": 16, "logic": True,
         "precision": "fp64", "rows": 24},
        # the range filter over a 20-bit column (six lvl02 and three lvl01 bootstraps a row)
        {"name": "compare_lvl2_20bit_2048", "kind": "compare", "level": 2, "op": "le", "bits": 20, "logic": True,
         "precision": "split32", "rows": 2048},
        # the switch that takes a lvl2 result down to lvl1, a middling batch
        {"name": "keyswitch_21_200", "kind": "keyswitch", "switch": 21, "rows": 200},
        # the external-product benchmark's batch
        {"name": "extprod_lvl1_4096", "kind": "extprod", "level": 1, "precision": "split32", "rows": 4096},
        # a small ArcEDB comparison over two digits
        {"name": "arc_gt_2digits_1000", "kind": "arc", "op": "gt", "digits": 2, "precision": "split32", "rows": 1000},
        # polynomials into the frequency domain and back
        {"name": "transform_lvl2_2000", "kind": "transform", "level": 2, "rows": 2000},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    kind = rng.choice(["gate", "gate", "gate_host", "compare", "compare", "keyswitch", "extprod", "arc", "transform"])
    precision = rng.choice(["fp64", "split32"])
    if kind in ("gate", "gate_host"):
        return {"kind": kind, "gate": rng.choice(GATE_NAMES), "precision": precision, "rows": _log_int(rng, 1, 4096)}
    if kind == "compare":
        level = rng.choice([1, 2])
        bits = rng.randint(4, 9) if level == 1 else rng.randint(12, 32)
        rows = _log_int(rng, 1, 4096 if level == 1 else 36_000 // bits)
        op = rng.choice(COMPARE_OPS)
        if level == 2 and op == "eq":
            rows = (rows + 1) // 2   # two chains
        return {"kind": kind, "level": level, "op": op, "bits": bits, "logic": rng.random() < 0.75,
                "precision": precision, "rows": rows}
    if kind == "keyswitch":
        return {"kind": kind, "switch": rng.choice([10, 20, 21]), "rows": _log_int(rng, 1, 4096)}
    if kind == "extprod":
        level = rng.choice([1, 2])
        return {"kind": kind, "level": level, "precision": precision if level == 1 else "fp64",
                "rows": _log_int(rng, 1, 4096)}
    if kind == "arc":
        return {"kind": kind, "op": rng.choice(["gt", "lt", "eq", "lt_strict"]), "digits": rng.randint(1, 3),
                "precision": precision, "rows": _log_int(rng, 1, 2048)}
    return {"kind": kind, "level": rng.choice([1, 2]), "rows": _log_int(rng, 1, 8192)}


def _words32(seed, n):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-2 ** 31, 2 ** 31, (n,), generator=g, device="cuda", dtype=torch.int32)


def _words64(seed, n):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-2 ** 63, 2 ** 63 - 1, (n,), generator=g, device="cuda", dtype=torch.int64)


def _bits(seed, rows):
    """lvl1 encryptions of uniform random bits"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    b = torch.randint(0, 2, (rows,), generator=g, device="cuda", dtype=torch.int32)
    ct = torch.empty(rows * (N1 + 1), dtype=torch.int32, device="cuda")
    engine().encrypt_lvl1(seed, 0xCA, 0, (2 * b - 1) * MU1, ct)
    return ct


def prepare(case, seed):
    eng, kind, rows = engine(), case["kind"], case["rows"]
    s = {"case": case}
    if kind in ("gate", "gate_host"):
        s["a"], s["b"] = _bits(2 * seed, rows), _bits(2 * seed + 1, rows)
        if kind == "gate":
            s["out"] = torch.empty_like(s["a"])
        else:
            def pinned(t):
                h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
                h.copy_(t)
                return h.numpy().view(np.uint32).reshape(rows, N1 + 1)
            s["a"], s["b"] = pinned(s["a"]), pinned(s["b"])
            s["out"] = pinned(torch.zeros(rows * (N1 + 1), dtype=torch.int32))
    elif kind == "compare":
        rng = np.random.default_rng(seed)
        x = rng.integers(0, 2 ** case["bits"], rows).astype(np.uint64)
        const = np.full(rows, rng.integers(0, 2 ** case["bits"]), np.uint64)
        same = rng.random(rows) < 0.125
        x[same] = const[same]
        s["a"] = encrypt_column(eng, x, case["bits"], seed, 0xA0, 0, case["level"])
        s["b"] = encrypt_column(eng, const, case["bits"], seed, 0xB0, 0, case["level"])
        s["out"] = torch.empty(rows * (N1 + 1), dtype=torch.int32, device="cuda")
    elif kind == "keyswitch":
        narrow = case["switch"] == 10
        s["a"] = _words32(seed, rows * (N1 + 1)) if narrow else _words64(seed, rows * (N2 + 1))
        width = N1 + 1 if case["switch"] == 21 else N0 + 1
        s["out"] = torch.empty(rows * width, dtype=torch.int32, device="cuda")
    elif kind == "extprod":
        s["g"] = torch.empty(rows * TRGSW_BYTES[case["level"]] // 8, dtype=torch.float64, device="cuda")
        if case["level"] == 1:
            s["a"] = _words32(2 * seed, rows * 2 * N1)
            eng.trgsw_prepare_lvl1(_words32(2 * seed + 1, rows * 6 * 2 * N1), s["g"], PRECISION[case["precision"]])
        else:
            s["a"] = _words64(2 * seed, rows * 2 * N2)
            eng.trgsw_prepare_lvl2(_words64(2 * seed + 1, rows * 8 * 2 * N2), s["g"])
        s["out"] = torch.empty_like(s["a"])
    elif kind == "arc":
        n = rows * case["digits"]
        s["a"] = _words32(2 * seed, n * 2 * N1)
        s["g"] = torch.empty(n * TRGSW_BYTES[1] // 8, dtype=torch.float64, device="cuda")
        eng.trgsw_prepare_lvl1(_words32(2 * seed + 1, n * 6 * 2 * N1), s["g"], PRECISION[case["precision"]])
        s["out"] = torch.empty(rows * (N1 + 1), dtype=torch.int32, device="cuda")
    elif kind == "transform":
        n = N1 if case["level"] == 1 else N2
        words = _words32 if case["level"] == 1 else _words64
        s["a"] = words(2 * seed, rows * n)
        s["fd"] = torch.empty(rows * n, dtype=torch.float64, device="cuda")
        # the way back gets the frequency values of other polynomials
        back = eng.twist_ifft_lvl1 if case["level"] == 1 else eng.twist_ifft_lvl2
        s["fd_in"] = torch.empty(rows * n, dtype=torch.float64, device="cuda")
        back(words(2 * seed + 1, rows * n), s["fd_in"])
        s["out"] = torch.empty_like(s["a"])
    else:
        raise ValueError(kind)
    torch.cuda.current_stream().synchronize()   # the raw TRGSWs may go
    return s


def run(s):
    eng, c = engine(), s["case"]
    kind = c["kind"]
    if kind == "gate":
        eng.gate_lvl1(c["gate"], s["a"], s["b"], s["out"], PRECISION[c["precision"]])
    elif kind == "gate_host":
        return eng.gate_lvl1_host(c["gate"], s["a"], s["b"], PRECISION[c["precision"]], out=s["out"]).view(np.int32)
    elif kind == "compare":
        eng.compare(c["op"], c["level"], s["a"], s["b"], s["out"], c["bits"], c["logic"], PRECISION[c["precision"]])
    elif kind == "keyswitch":
        eng.iks(c["switch"], s["a"], s["out"])
    elif kind == "extprod":
        if c["level"] == 1:
            eng.extprod_lvl1(s["a"], s["g"], s["out"], precision=PRECISION[c["precision"]])
        else:
            eng.extprod_lvl2(s["a"], s["g"], s["out"])
    elif kind == "arc":
        eng.arc_compare(c["op"], s["a"], s["g"], s["out"], c["digits"], PRECISION[c["precision"]])
    else:
        if c["level"] == 1:
            eng.twist_ifft_lvl1(s["a"], s["fd"])
            eng.twist_fft_lvl1(s["fd_in"], s["out"])
        else:
            eng.twist_ifft_lvl2(s["a"], s["fd"])
            eng.twist_fft_lvl2(s["fd_in"], s["out"])
        return {"fd": s["fd"], "out": s["out"]}
    return s["out"]


def _switch_bytes(switch, rows):
    """the distinct key rows that `rows` uniform ciphertexts select, their input and their output"""
    places, digits, row = {10: (2 * N1, 1024, 4 * (N0 + 1)), 20: (2 * N2, 1024, 4 * (N0 + 1)),
                           21: (10 * N2, 8, 4 * (N1 + 1))}[switch]
    width_in = 4 * (N1 + 1) if switch == 10 else 8 * (N2 + 1)
    return places * (digits - 1) * (1.0 - (1.0 - 1.0 / digits) ** rows) * row + rows * (width_in + row)


def _chain(level, op, bits, logic):
    """(lvl01 bootstraps, lvl02 bootstraps, lvl1 -> lvl0, lvl2 -> lvl0, lvl2 -> lvl1 switches) of one comparison"""
    if op == "eq":
        a, b = _chain(level, "ge", bits, True), _chain(level, "le", bits, True)
        return tuple(x + y + z for x, y, z in zip(a, b, (1, 0, 1, 0, 0)))
    pb, p2, k21 = bits + 1, 0, 0
    if level == 2:
        while pb > 9:
            p2 += 2
            pb -= 5
        k21 = 1
    p1 = 1 if pb <= 5 else 3 if pb <= 9 else 5
    if op in ("ge", "le") and not logic:
        p1 += 1
    return p1, p2, p1, p2, k21


def work(case):
    kind, rows = case["kind"], case["rows"]
    if kind in ("gate", "gate_host"):
        # the second input beside the switch's own, the bootstrapping key, the output
        return {"bytes": _switch_bytes(10, rows) + rows * 8 * (N1 + 1) + BK01_BYTES, "flops": rows * PBS01_FLOP}
    if kind == "compare":
        p1, p2, k10, k20, k21 = _chain(case["level"], case["op"], case["bits"], case["logic"])
        wide = 8 * (N2 + 1) if case["level"] == 2 else 4 * (N1 + 1)
        return {"bytes": k10 * _switch_bytes(10, rows) + k20 * _switch_bytes(20, rows) + k21 * _switch_bytes(21, rows)
                + p1 * (BK01_BYTES + rows * 4 * (N1 + 1)) + p2 * (BK02_BYTES + rows * 8 * (N2 + 1)) + 2 * rows * wide,
                "flops": rows * (p1 * PBS01_FLOP + p2 * PBS02_FLOP)}
    if kind == "keyswitch":
        return {"bytes": _switch_bytes(case["switch"], rows), "flops": 0}
    if kind == "extprod":
        poly = 2 * 4 * N1 if case["level"] == 1 else 2 * 8 * N2
        return {"bytes": rows * (TRGSW_BYTES[case["level"]] + 2 * poly), "flops": rows * EXTPROD_FLOP[case["level"]]}
    if kind == "arc":
        d = case["digits"]
        boots = (d - 1) * (_switch_bytes(10, rows) + BK01_BYTES + rows * 8 * (N0 + N1))
        return {"bytes": rows * d * (TRGSW_BYTES[1] + 2 * 4 * N1) + boots + rows * 4 * (N1 + 1),
                "flops": rows * (d * EXTPROD_FLOP[1] + (d - 1) * PBS01_FLOP)}
    n, word = (N1, 4) if case["level"] == 1 else (N2, 8)
    return {"bytes": 2 * rows * n * (word + 8), "flops": 2 * rows * 2.5 * n * math.log2(n // 2)}


def exact(case, seed):
    """the frequency values of the transforms; every other output is made of whole words"""
    if case["kind"] != "transform":
        return None
    n = N1 if case["level"] == 1 else N2
    a = (_words32 if case["level"] == 1 else _words64)(2 * seed, case["rows"] * n).cpu().numpy().astype(np.float64)
    a = a.reshape(-1, n)
    half = n // 2
    m = np.arange(half)
    z = (a[:, :half] + 1j * a[:, half:]) * np.exp(1j * math.pi * m / n)
    v = np.fft.ifft(z, axis=1) * half
    bits = half.bit_length() - 1
    rev = np.array([int(format(q, "0%db" % bits)[::-1], 2) for q in range(half)])
    out = np.empty_like(a)
    out[:, rev] = v.real
    out[:, rev + half] = v.imag
    return {"fd": out.reshape(-1), "out": None}
