"""GPU: the lvl01 kernel with one ciphertext per SM, and batches divided over
two launches, against one launch of the one-warp-per-ciphertext kernel: equal
words for every row.  The lvl02 kernel with one and two ciphertexts per CTA and
its divided batches against one another."""
from __future__ import annotations

import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu
N0, N1, N2 = 672, 1024, 2048


@pytest.fixture(scope="module")
def engines(tmp_path_factory):
    """(engine whose table makes the 7-per-CTA shape the only short one, so
    every batch is one launch of it; engine with the untuned table)"""
    from cufhedb_b200 import GEN_BK01, Engine
    one_warp, divided = Engine(0), Engine(0)
    for e in (one_warp, divided):
        e.keygen(SEED, GEN_BK01)
    path = str(tmp_path_factory.mktemp("tbl") / "t.tbl")
    one_warp.autotune_save(path)
    lines = open(path).read().splitlines()
    for i, ln in enumerate(lines):
        if ln.startswith(("pbs01 fp64 ", "pbs01 split32 ")):
            f = ln.split()
            lines[i] = " ".join(f[:2] + [x for w in f[2::2] for x in (w, "0.001" if w == "7" else "1000.0")])
    open(path, "w").write("\n".join(lines) + "\n")
    assert one_warp.autotune_load(path)
    yield one_warp, divided
    one_warp.close()
    divided.close()


@pytest.fixture(scope="module")
def lvl2_engines(tmp_path_factory):
    """an untuned engine, and one each whose table makes shape 1, 2 or 3 of lvl02
    the only short one"""
    from cufhedb_b200 import GEN_BK02, Engine
    path = str(tmp_path_factory.mktemp("tbl2") / "t.tbl")
    engs = [Engine(0) for _ in range(4)]
    for k, e in enumerate(engs):
        e.keygen(SEED, GEN_BK02)
        if k == 0:
            e.autotune_save(path)
            continue
        lines = open(path).read().splitlines()
        for i, ln in enumerate(lines):
            if ln.startswith("pbs02 fp64 "):
                f = ln.split()
                lines[i] = " ".join(f[:2] + [x for w in f[2::2] for x in (w, "0.001" if w == str(k) else "1000.0")])
        forced = path + str(k)
        open(forced, "w").write("\n".join(lines) + "\n")
        assert e.autotune_load(forced)
    yield engs
    for e in engs:
        e.close()


@pytest.mark.parametrize("tv", ["const", "staircase", "poly"])
@pytest.mark.parametrize("rows", [1, 2, "sms+1", "3sms+1"])
def test_lvl02_words_equal_across_shapes(lvl2_engines, tv, rows):
    import torch
    from cufhedb_b200 import testvec_const, testvec_poly, testvec_staircase
    S = lvl2_engines[0].num_sms
    B = {"sms+1": S + 1, "3sms+1": 3 * S + 1}.get(rows, rows)
    poly = torch.arange(N2, device="cuda", dtype=torch.int64) * 4503599627370449
    vec = {"const": testvec_const(1 << 61), "staircase": testvec_staircase(44), "poly": testvec_poly(poly)}[tv]
    x = _inputs(B)
    outs = []
    for e in lvl2_engines:
        outs.append(torch.empty(B * (N2 + 1), dtype=torch.int64, device="cuda"))
        e.pbs_lvl02(x, outs[-1], vec)
        e.sync()
    assert all(torch.equal(outs[0], o) for o in outs[1:])


def _inputs(B):
    """uniform lvl0 words, with mask words that round to rotations 0 and N and
    an all-zero row among them"""
    import torch
    g = torch.Generator(device="cuda").manual_seed(B)
    x = torch.randint(-2 ** 31, 2 ** 31, (B, N0 + 1), generator=g, device="cuda", dtype=torch.int32)
    x[0, ::3] = (1 << 19) - 1            # rotation 0 at both levels: the CMux is skipped
    x[0, 1::3] = -(1 << 19)              # rounds up to 2 N, that is 0
    x[B // 2, 1::2] = -2 ** 31           # rotation N
    x[-1, :] = 0
    return x.reshape(-1)


@pytest.mark.parametrize("precision", ["split32", "fp64"])
@pytest.mark.parametrize("tv", ["const", "staircase", "poly"])
@pytest.mark.parametrize("rows", [1, 2, "sms", "sms+1", "8sms+3"])
def test_words_equal_the_one_warp_kernel(engines, precision, tv, rows):
    import torch
    from cufhedb_b200 import FP64, SPLIT32, testvec_const, testvec_poly, testvec_staircase
    one_warp, divided = engines
    prec = SPLIT32 if precision == "split32" else FP64
    S = divided.num_sms
    B = {"sms": S, "sms+1": S + 1, "8sms+3": 8 * S + 3}.get(rows, rows)
    poly = torch.arange(N1, device="cuda", dtype=torch.int32) * 2097143
    vec = {"const": testvec_const(1 << 29), "staircase": testvec_staircase(20), "poly": testvec_poly(poly)}[tv]
    x = _inputs(B)
    out = [torch.empty(B * (N1 + 1), dtype=torch.int32, device="cuda") for _ in range(2)]
    one_warp.pbs_lvl01(x, out[0], vec, prec)
    divided.pbs_lvl01(x, out[1], vec, prec)
    one_warp.sync()
    divided.sync()
    assert torch.equal(out[0], out[1])
