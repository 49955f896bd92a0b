"""GPU: the standalone transforms on frequency arrays that are 16-byte aligned and
ones that are only 8-byte aligned (16- and 8-byte accesses) give the same
values, for one polynomial, a ragged last block and many."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level", [1, 2])
@pytest.mark.parametrize("rows", [1, 5, 301])
def test_alignment_does_not_change_the_values(level, rows):
    import torch
    from cufhedb_b200 import Engine
    n = 1024 if level == 1 else 2048
    dt, lim = (torch.int32, 2 ** 31) if level == 1 else (torch.int64, 2 ** 63)
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randint(-lim, lim - 1, (rows * n,), generator=g, device="cuda", dtype=dt)
    with Engine(0) as eng:
        ifft = eng.twist_ifft_lvl1 if level == 1 else eng.twist_ifft_lvl2
        fft = eng.twist_fft_lvl1 if level == 1 else eng.twist_fft_lvl2
        fd = [torch.full((rows * n + 1,), float("nan"), dtype=torch.float64, device="cuda")[off: off + rows * n]
              for off in (0, 1)]
        back = [torch.empty_like(x) for _ in fd]
        for f, b in zip(fd, back):
            ifft(x, f)
            fft(f, b)
        eng.sync()
        assert fd[0].data_ptr() % 16 == 0 and fd[1].data_ptr() % 16 == 8
        assert torch.equal(fd[0], fd[1]) and torch.equal(back[0], back[1])
        d = back[0] - x                       # the round trip, modulo the torus
        bound = 1 if level == 1 else 2 ** 14  # the reference's own bounds
        assert int(d.abs().max()) <= bound
