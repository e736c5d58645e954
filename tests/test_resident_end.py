"""How a resident solve ends (csrc/tse_resident.cuh res_team_sum, res_last) when a block's
wait runs out: a restatement of the blocks' steps on the CPU, and the waits themselves with
a short limit on a GPU."""
import ctypes as ct
import random

import pytest

from transportse_b200 import _native as N


def _solve(rng, nb, count):
    """One launch of nb blocks in which one block's edge wait runs out in a
    random iteration; True if the solve is reported good, and the blocks that
    stored their part of the result.  ``count``: by the last block to leave, from
    every block's own flag; else by block 0 from its own."""
    checks = sorted(rng.sample(range(1, 30), 6))
    last = checks[-1]                      # converged there, by every block's sums
    bad, when = rng.randrange(nb), rng.randint(1, last)
    flagged = [False] * nb                 # a block's own flag
    launch_flag = False
    gone, stored = set(), set()
    for it in range(1, last + 1):
        if it == when:
            flagged[bad] = launch_flag = True
        for b in range(nb):
            # another block looks at the launch's flag only while it waits long
            if b not in gone and launch_flag and b != bad and rng.random() < 0.02:
                flagged[b] = True
        if it in checks:
            # every block still there publishes its sum; block 0 needs all of them
            if gone and 0 not in gone:
                flagged[0] = True          # its wait for a block that left runs out
            for b in range(nb):
                if b not in gone and (flagged[b] or (flagged[0] and 0 in gone)):
                    gone.add(b)
            if flagged[0]:
                return False, stored
    stored = {b for b in range(nb) if b not in gone}
    return (not gone if count else True), stored


def test_a_solve_is_good_only_if_every_block_stored_its_part():
    """Where the blocks count themselves out no good solve lacks a block's
    part; where block 0 trusts its own flag some do."""
    rng = random.Random(4)
    for nb in (2, 5, 37):
        runs = [_solve(rng, nb, True) for _ in range(3000)]
        assert all(len(stored) == nb for ok, stored in runs if ok)
        runs = [_solve(rng, nb, False) for _ in range(3000)]
        assert any(len(stored) < nb for ok, stored in runs if ok)


@pytest.mark.gpu
def test_resident_waits_give_up_and_an_early_leaver_is_reported(cuda_device):
    import torch
    res = torch.full((5,), -1, dtype=torch.int32, device=cuda_device)
    ws = torch.empty(32768, dtype=torch.uint8, device=cuda_device)
    rc = N.lib().tse_selftest_resident_waits(ct.c_void_p(res.data_ptr()), 0.1, ct.c_void_p(ws.data_ptr()),
                                             ws.numel(),
                                             ct.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream))
    assert rc == 0
    assert res.cpu().tolist() == [1, 1, 1, 1, 1]
    x = torch.arange(1000, dtype=torch.float64, device=cuda_device)
    assert float((x * 2).sum().item()) == 999000.0


@pytest.mark.gpu
def test_selftest_refuses_what_it_cannot_run(cuda_device):
    import torch
    res = torch.zeros(5, dtype=torch.int32, device=cuda_device)
    ws = torch.empty(32768, dtype=torch.uint8, device=cuda_device)
    call = lambda r, t, w, n: N.lib().tse_selftest_resident_waits(r, t, w, n, None)
    r, w = ct.c_void_p(res.data_ptr()), ct.c_void_p(ws.data_ptr())
    assert call(None, 0.1, w, 32768) == -1 and call(r, 0.0, w, 32768) == -1
    assert call(r, 0.1, None, 32768) == -1 and call(r, 0.1, w, 512) == -1
