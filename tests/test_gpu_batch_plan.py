"""GPU: a bootstrap's words do not depend on the batch it is in.  lvl01: every
launch variant of the batch size (one, two to three, four and more ciphertexts
per SM) gives a row the words it has in a large batch.  lvl02: every shape, and
batches divided over two launches, give the same words."""
from __future__ import annotations

import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu
N0, N1, N2 = 672, 1024, 2048


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


def test_lvl02_words_equal_in_large_batches(lvl2_engines):
    """more than six ciphertexts per SM run one per block: the same words as in
    small batches, first and last rows, a skipped CMux and the all-zero row"""
    import torch
    from cufhedb_b200 import testvec_staircase
    e = lvl2_engines[0]
    B = 6 * e.num_sms + 1
    x = _inputs(B)
    want = torch.empty(B * (N2 + 1), dtype=torch.int64, device="cuda")
    e.pbs_lvl02(x, want, testvec_staircase(44))
    for at in (0, B // 2 - 2, B - 5):
        got = torch.empty(5 * (N2 + 1), dtype=torch.int64, device="cuda")
        e.pbs_lvl02(x[at * (N0 + 1): (at + 5) * (N0 + 1)].contiguous(), got, testvec_staircase(44))
        e.sync()
        assert torch.equal(got, want[at * (N2 + 1): (at + 5) * (N2 + 1)]), at


@pytest.mark.parametrize("rows", ["all", "pairs", "every other"])
def test_lvl02_runs_of_skipped_cmuxes(lvl2_engines, rows):
    """two ciphertexts per SM, three passes and an odd row at the end: rows whose
    masks all round to rotation 0 (no CMux of theirs runs, so a pair of them passes
    every round of the key without a transform) and rows between them have the
    words of one ciphertext per SM"""
    import torch
    from cufhedb_b200 import testvec_staircase
    S = lvl2_engines[0].num_sms
    B = 4 * S + 3
    x = _inputs(B).reshape(B, N0 + 1)
    skip = {"all": slice(0, B), "pairs": [i for i in range(B) if i // 2 % 2], "every other": slice(0, B, 2)}[rows]
    x[skip, :N0] = (1 << 19) - 1
    outs = []
    for e in lvl2_engines[1:3]:
        outs.append(torch.empty(B * (N2 + 1), dtype=torch.int64, device="cuda"))
        e.pbs_lvl02(x.reshape(-1), outs[-1], testvec_staircase(44))
        e.sync()
    assert torch.equal(*outs)


def test_lvl02_launch_shape_is_the_shape_of_the_launch(lvl2_engines):
    """untuned: the plan for a B200's times; a forced shape up to six ciphertexts per
    SM; one ciphertext per block above"""
    from cufhedb_b200 import FP64
    S = lvl2_engines[0].num_sms
    shape = lambda e, B: e.launch_shape(2, FP64, B)
    assert [shape(lvl2_engines[0], B) for B in (1, S, S + 1, 2 * S, 2 * S + 1, 3 * S)] == [1, 1, 2, 2, 3, 3]
    for k, e in enumerate(lvl2_engines[1:], 1):
        assert [shape(e, B) for B in (1, 3 * S, 6 * S)] == [k] * 3
    assert all(shape(e, B) == 1 for e in lvl2_engines for B in (6 * S + 1, 16384))


def test_one_row_bootstraps_in_place(lvl2_engines):
    """the output over the row that it is made from, whose last CMuxes (or all) are
    skipped: no barrier stands between them and the output"""
    import torch
    from cufhedb_b200 import FP64, GEN_BK01, SPLIT32, Engine, testvec_staircase
    rows = _inputs(64).reshape(64, N0 + 1)[8:24].clone()
    for k, row in enumerate(rows):
        row[N0 - 42 * k: N0] = (1 << 19) - 1
    with Engine(0) as eng:
        eng.keygen(SEED, GEN_BK01)
        for prec in (SPLIT32, FP64):
            for row in rows:
                want = torch.empty(N1 + 1, dtype=torch.int32, device="cuda")
                eng.pbs_lvl01(row, want, testvec_staircase(20), prec)
                buf = torch.zeros_like(want)
                buf[: N0 + 1] = row
                eng.pbs_lvl01(buf[: N0 + 1], buf, testvec_staircase(20), prec)
                eng.sync()
                assert torch.equal(buf, want)
    for e in lvl2_engines:
        for row in rows[::5]:
            want = torch.empty(N2 + 1, dtype=torch.int64, device="cuda")
            e.pbs_lvl02(row, want, testvec_staircase(44))
            buf = torch.zeros_like(want)
            buf.view(torch.int32)[: N0 + 1] = row
            e.pbs_lvl02(buf.view(torch.int32)[: N0 + 1], buf, testvec_staircase(44))
            e.sync()
            assert torch.equal(buf, want)


def test_split_block_transforms_equal_the_one_warp_forms():
    """the packed one-warp transforms and the block's, bit for bit: both are the same
    operations with the same roundings"""
    from cufhedb_b200 import Engine
    with Engine(0) as eng:
        for seed in (1, 2):
            assert eng.selftest_split_transforms(seed, 4096) == (0, 0)


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
def test_lvl01_words_do_not_depend_on_the_batch(precision, tv):
    import torch
    from cufhedb_b200 import FP64, GEN_BK01, SPLIT32, Engine, testvec_const, testvec_poly, testvec_staircase
    prec = SPLIT32 if precision == "split32" else FP64
    with Engine(0) as eng:
        eng.keygen(SEED, GEN_BK01)
        S = eng.num_sms
        B = 4 * S + 5
        poly = torch.arange(N1, device="cuda", dtype=torch.int32) * 2097143
        vec = {"const": testvec_const(1 << 29), "staircase": testvec_staircase(20), "poly": testvec_poly(poly)}[tv]
        x = _inputs(B)
        want = torch.empty(B * (N1 + 1), dtype=torch.int32, device="cuda")
        eng.pbs_lvl01(x, want, vec, prec)
        for n in (1, 2, S, S + 1, 2 * S + 1, 3 * S + 1):
            got = torch.empty(n * (N1 + 1), dtype=torch.int32, device="cuda")
            eng.pbs_lvl01(x[: n * (N0 + 1)].contiguous(), got, vec, prec)
            eng.sync()
            assert torch.equal(got, want[: n * (N1 + 1)]), n


@pytest.mark.parametrize("precision", ["split32", "fp64"])
def test_lvl1_products_do_not_depend_on_the_batch(precision):
    """external products: every launch variant of the batch size, a block's first
    and later products, in place, and one shared TRGSW"""
    import torch
    from cufhedb_b200 import FP64, SPLIT32, Engine
    prec = SPLIT32 if precision == "split32" else FP64
    with Engine(0) as eng:
        S = eng.num_sms
        B = 4 * S + 5
        g = torch.Generator(device="cuda").manual_seed(7)
        words = lambda n: torch.randint(-2 ** 31, 2 ** 31, (n,), generator=g, device="cuda", dtype=torch.int32)
        x, raw = words(B * 2 * N1), words(B * 6 * 2 * N1)
        x[: 2 * N1] = -2 ** 31                       # extreme digits against extreme words
        raw[: 12 * N1] = 2 ** 31 - 1
        prep = torch.empty(B * 12288, dtype=torch.float64, device="cuda")
        eng.trgsw_prepare_lvl1(raw, prep, prec)
        want = torch.empty_like(x)
        eng.extprod_lvl1(x, prep, want, precision=prec)
        for n in (1, S, S + 1, 2 * S + 1):
            got = x[: n * 2 * N1].clone()
            eng.extprod_lvl1(got, prep[: n * 12288].contiguous(), got, precision=prec)
            eng.sync()
            assert torch.equal(got, want[: n * 2 * N1]), n
        one = prep[:12288].contiguous()
        got, rep = torch.empty_like(x), torch.empty_like(x)
        eng.extprod_lvl1(x, one, got, shared=True, precision=prec)
        eng.extprod_lvl1(x, one.repeat(B), rep, precision=prec)
        eng.sync()
        assert torch.equal(got, rep)
