"""Caller-owned workspaces of the plan-less entry points: what the library remembers about them, what it leaves in them."""
import resource

import pytest
import torch

pytestmark = pytest.mark.gpu


def _lib():
    from souffle_models_b200 import _lib
    return _lib.load()


def _stream():
    return torch.cuda.current_stream().cuda_stream


class _Mlp:
    """One fused MLP call (three stages, two grid barriers) on a workspace of its own."""
    M, C, F = 256, 512, 2048

    def __init__(self):
        g = torch.Generator().manual_seed(3)
        make = lambda *s: (torch.randn(*s, generator=g) * 0.05).half().cuda()
        self.src, self.w1, self.w2 = make(self.M, self.C), make(self.C, self.F), make(self.F, self.C)
        self.hidden, self.out = torch.empty(self.M, self.F).half().cuda(), torch.empty(self.M, self.C).half().cuda()
        n = _lib().souffle_swin_mlp_workspace_bytes(self.M, self.C, self.F)
        self.ws = torch.full((n // 4,), -1, dtype=torch.int32, device="cuda")      # the library clears what it needs
        self.forget()                             # fresh memory, whatever lived at this address before
        assert self.call() == 0 and self.status() == 0
        self.want = self.out.clone()

    def call(self, rows=None):
        return _lib().souffle_swin_mlp_forward(self.src.data_ptr(), self.w1.data_ptr(), self.w2.data_ptr(), self.hidden.data_ptr(),
                                               self.out.data_ptr(), rows or self.M, self.C, self.F, self.ws.data_ptr(),
                                               self.ws.numel() * 4, _stream())

    def status(self):
        return _lib().souffle_workspace_status(self.ws.data_ptr(), _stream())

    def forget(self):
        assert _lib().souffle_workspace_forget(self.ws.data_ptr()) == 0

    def spoil(self):
        """One arrival is missing from whichever barrier pair the next call uses: its waits run out (2 s)."""
        self.ws[0], self.ws[2] = -1, -1


def test_a_wait_that_runs_out_is_reported_once_and_to_its_owner():
    mlp, other = _Mlp(), _Mlp()
    mlp.spoil()
    assert mlp.call() == 0
    assert other.call() == 0 and other.status() == 0
    assert mlp.status() == 6
    assert mlp.call() == 0 and mlp.status() == 0 and torch.equal(mlp.out, mlp.want)
    assert other.status() == 0 and torch.equal(other.out, other.want)


def test_the_next_owner_of_an_address_is_not_told_of_the_last():
    mlp = _Mlp()
    mlp.spoil()
    assert mlp.call() == 0
    mlp.forget()
    assert mlp.call() == 0 and mlp.status() == 0 and torch.equal(mlp.out, mlp.want)


def test_given_up_workspaces_leave_nothing_behind():
    """300,000 workspaces used once each, none asked for its status: a record and a status block apiece were 15 MB."""
    lib = _lib()
    a, w, c = (torch.zeros(64, 64).half().cuda() for _ in range(3))
    n = lib.souffle_gemm_workspace_bytes()
    pool = torch.empty(300_000 * n, dtype=torch.uint8, device="cuda")

    def use(lo, hi):
        for i in range(lo, hi):
            ws = pool.data_ptr() + i * n
            assert lib.souffle_gemm_f16(a.data_ptr(), w.data_ptr(), c.data_ptr(), 64, 64, 64, ws, n, _stream()) == 0
            assert lib.souffle_workspace_forget(ws) == 0
        torch.cuda.synchronize()
        return resource.getrusage(resource.RUSAGE_SELF).ru_maxrss

    before = use(0, 2000)
    assert use(2000, 300_000) - before < 4096            # KiB
