"""Local NCC from several host threads at once, with windows of different
sizes: no thread's launch is refused for another's window."""

import ctypes
import threading

import pytest
import torch

from nanodrr_gb300 import _ffi

pytestmark = pytest.mark.gpu


def test_threads_with_different_windows():
    g = torch.Generator().manual_seed(0)
    H, W = 128, 130
    x, y = (torch.rand(1, 1, H, W, generator=g).cuda() for _ in range(2))
    go = torch.ones(1, device="cuda")
    lib = _ffi.load()

    def calls(p):
        """The window's forward and adjoint, with their own buffers."""
        score, g1, g2 = torch.zeros(1, device="cuda"), torch.zeros_like(x), torch.zeros_like(y)
        maps = torch.zeros(5, H - p + 1, W - p + 1, device="cuda", dtype=torch.float64)
        nb = ctypes.c_uint64(0)
        _ffi.check(lib.ndrr_ncc_patch_workspace_bytes(1, 1, H, W, p, ctypes.byref(nb)), "workspace")
        ws = torch.empty(int(nb.value), device="cuda", dtype=torch.uint8)
        stream = torch.cuda.Stream()
        fwd = (x.data_ptr(), y.data_ptr(), 1, 1, H, W, p, 1e-5, score.data_ptr(), maps.data_ptr(), ws.data_ptr(),
               ws.numel(), stream.cuda_stream)
        bwd = (go.data_ptr(), x.data_ptr(), y.data_ptr(), maps.data_ptr(), 1, 1, H, W, p, g1.data_ptr(), g2.data_ptr(),
               stream.cuda_stream)
        return fwd, bwd, (score, g1, g2), (maps, ws, stream)

    refused = []

    def work(n, fwd, bwd, out, held):
        for _ in range(n):
            if lib.ndrr_ncc_patch_fwd(*fwd) or lib.ndrr_ncc_patch_bwd(*bwd):
                refused.append(lib.ndrr_last_error().decode())
                return

    torch.cuda.synchronize()
    jobs = [calls(p) for p in (1, 2, 60, 128)]
    threads = [threading.Thread(target=work, args=(4000, *j)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not refused, refused
    for fwd, bwd, out, held in jobs:
        got = [t.clone() for t in out]
        work(1, fwd, bwd, out, held)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, out))
