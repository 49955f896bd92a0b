"""GPU: equality runs both orders as one chain for up to 1,024 rows and as two
above; a row's words are the same either way, at both levels and results."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import SEED

pytestmark = pytest.mark.gpu
N1 = 1024


@pytest.mark.parametrize("level, bits", [(1, 4), (1, 9), (2, 12)])
@pytest.mark.parametrize("logic", [True, False])
def test_equal_words_do_not_depend_on_the_row_count(level, bits, logic):
    import torch
    from cufhedb_b200 import GEN_ALL, SPLIT32, Engine
    from cufhedb_b200.queries import encrypt_column
    rng = np.random.default_rng(bits)
    B = 1025                                   # the smallest count that runs two chains
    x = rng.integers(0, 2 ** bits, B).astype(np.uint64)
    y = np.where(rng.random(B) < 0.5, x, rng.integers(0, 2 ** bits, B).astype(np.uint64)).astype(np.uint64)
    with Engine(0) as eng:
        eng.keygen(SEED, GEN_ALL)
        a, b = (encrypt_column(eng, v, bits, SEED, sid, 0, level) for v, sid in ((x, 0xE0), (y, 0xE1)))
        want = torch.empty(B * (N1 + 1), dtype=torch.int32, device="cuda")
        eng.compare("eq", level, a, b, want, bits, logic, SPLIT32)
        w = a.numel() // B
        for n in (1, 149, 1024):
            got = torch.empty(n * (N1 + 1), dtype=torch.int32, device="cuda")
            eng.compare("eq", level, a[: n * w].contiguous(), b[: n * w].contiguous(), got, bits, logic, SPLIT32)
            eng.sync()
            assert torch.equal(got, want[: n * (N1 + 1)]), n
        ph = torch.empty(B, dtype=torch.int32, device="cuda")
        eng.phase_lvl1(want, ph)
        eng.sync()
        if logic:                              # phases +-1/8
            assert np.array_equal((ph > 0).cpu().numpy(), x == y)
