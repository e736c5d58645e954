"""The resident solves' bounded waits (csrc/tse_resident.cuh) and the overlapped sweep's, with
a short limit."""
import ctypes as ct

import pytest

from transportse_b200 import _native as N


@pytest.mark.gpu
def test_resident_waits_give_up(cuda_device):
    import torch
    res = torch.full((3,), -1, dtype=torch.int32, device=cuda_device)
    ws = torch.empty(32768, dtype=torch.uint8, device=cuda_device)
    rc = N.lib().tse_selftest_resident_waits(ct.c_void_p(res.data_ptr()), 0.1, ct.c_void_p(ws.data_ptr()),
                                             ws.numel(),
                                             ct.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream))
    assert rc == 0
    assert res.cpu().tolist() == [1, 1, 1]
    x = torch.arange(1000, dtype=torch.float64, device=cuda_device)
    assert float((x * 2).sum().item()) == 999000.0


@pytest.mark.gpu
def test_selftest_refuses_what_it_cannot_run(cuda_device):
    import torch
    res = torch.zeros(3, dtype=torch.int32, device=cuda_device)
    ws = torch.empty(32768, dtype=torch.uint8, device=cuda_device)
    call = lambda r, t, w, n: N.lib().tse_selftest_resident_waits(r, t, w, n, None)
    r, w = ct.c_void_p(res.data_ptr()), ct.c_void_p(ws.data_ptr())
    assert call(None, 0.1, w, 32768) == -1 and call(r, 0.0, w, 32768) == -1
    assert call(r, 0.1, None, 32768) == -1 and call(r, 0.1, w, 512) == -1
