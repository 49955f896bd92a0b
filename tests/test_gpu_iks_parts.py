"""GPU: key switches divided over several CTAs per ciphertext (small and middling
batches) give the undivided kernel's words, for every kind, at the edges of the
rule that divides them."""
from __future__ import annotations

import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu
WIDTH = {10: (1025, 673), 20: (2049, 673), 21: (2049, 1025)}


@pytest.fixture(scope="module")
def ks_engine():
    from cufhedb_b200 import GEN_KSK10, GEN_KSK20, GEN_KSK21, Engine
    eng = Engine(0)
    eng.keygen(SEED, GEN_KSK10 | GEN_KSK20 | GEN_KSK21)
    yield eng
    eng.close()


@pytest.mark.parametrize("kind", [10, 20, 21])
def test_divided_switch_equals_undivided(ks_engine, kind):
    """rows of an undivided batch (1,000; 21: the key-stationary kernel) against
    the same rows in smaller batches"""
    import torch
    win, wout = WIDTH[kind]
    B = 1000
    g = torch.Generator(device="cuda").manual_seed(kind)
    dt, lim = (torch.int32, 2 ** 31) if kind == 10 else (torch.int64, 2 ** 63)
    x = torch.randint(-lim, lim - 1, (B, win), generator=g, device="cuda", dtype=dt)
    x[0] = 0                       # no digit selects a row
    x[1, :-1] = -1                 # every digit wraps to 0 or its highest value
    want = torch.empty(B, wout, dtype=torch.int32, device="cuda")
    ks_engine.iks(kind, x, want)
    for n in (1, 2, 9, 148, 149, 511, 592, 850):
        got = torch.full((n, wout), 0x55555555, dtype=torch.int32, device="cuda")
        ks_engine.iks(kind, x[:n].contiguous(), got)
        ks_engine.sync()
        assert torch.equal(got, want[:n]), n


@pytest.mark.parametrize("B", [128, 129, 256, 257, 511, 513, 1100, 2100])
def test_key_stationary_batches_equal_gather(ks_engine, B):
    """lvl21, batches at the edges of the key-stationary switch's tiles and parts:
    the words the gather gives (batches of 100); captured, a batch below 512 takes
    the gather"""
    import torch
    g = torch.Generator(device="cuda").manual_seed(B)
    x = torch.randint(-2 ** 63, 2 ** 63 - 1, (B, 2049), generator=g, device="cuda", dtype=torch.int64)
    x[B // 2] = 0                       # digits of the rounding offset alone
    x[B - 1] = -1
    got = torch.full((B, 1025), 7, dtype=torch.int32, device="cuda")
    want = torch.empty_like(got)
    ks_engine.iks(21, x, got)
    for at in range(0, B, 100):
        n = min(100, B - at)
        part = torch.empty((n, 1025), dtype=torch.int32, device="cuda")
        ks_engine.iks(21, x[at: at + n].contiguous(), part)
        ks_engine.sync()
        want[at: at + n] = part
    assert torch.equal(got, want)
    if B < 512:
        again = torch.full_like(got, 9)
        stream = torch.cuda.Stream()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            ks_engine.iks(21, x, again, stream=stream)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(again, want)


@pytest.mark.parametrize("kind", [10, 20, 21])
def test_one_row_switches_in_place(ks_engine, kind):
    """the output over the row that it is made from, at its start and further in"""
    import torch
    win, wout = WIDTH[kind]
    g = torch.Generator(device="cuda").manual_seed(100 + kind)
    dt, lim = (torch.int32, 2 ** 31) if kind == 10 else (torch.int64, 2 ** 63)
    x = torch.randint(-lim, lim - 1, (win,), generator=g, device="cuda", dtype=dt)
    want = torch.empty(wout, dtype=torch.int32, device="cuda")
    ks_engine.iks(kind, x, want)
    for at in (0, 300):
        row = x.clone()
        got = row.view(torch.int32)[at: at + wout]
        ks_engine.iks(kind, row, got)
        ks_engine.sync()
        assert torch.equal(got, want), at


@pytest.mark.parametrize("kind", [10, 20])
def test_switch_words_at_the_edges_of_one_wave(ks_engine, kind):
    """batches on both sides of every line of the rule (few, one wave, its tail)
    against the same rows in batches of 100, which are divided finely"""
    import torch
    win, wout = WIDTH[kind]
    S = ks_engine.num_sms
    few, wave, tail = {10: (5.75, 10, 12.8), 20: (5.4, 8, 12.5)}[kind]
    sizes = [int(x * S) + k for x in (few, wave, tail) for k in (0, 1)]
    g = torch.Generator(device="cuda").manual_seed(200 + kind)
    dt, lim = (torch.int32, 2 ** 31) if kind == 10 else (torch.int64, 2 ** 63)
    x = torch.randint(-lim, lim - 1, (max(sizes), win), generator=g, device="cuda", dtype=dt)
    want = torch.empty(len(x), wout, dtype=torch.int32, device="cuda")
    for at in range(0, len(x), 100):
        ks_engine.iks(kind, x[at: at + 100], want[at: at + 100])
    for n in sizes:
        got = torch.full((n, wout), 0x55555555, dtype=torch.int32, device="cuda")
        ks_engine.iks(kind, x[:n], got)
        ks_engine.sync()
        assert torch.equal(got, want[:n]), n
