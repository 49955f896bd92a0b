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
