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


def _graph(call):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    return graph


def _replays_and_calls(graph, call, check):
    """Replays and ordinary calls in every order of two, then two replays on end."""
    for step in "rcrrccr":
        graph.replay() if step == "r" else call()
        check()
    graph.replay()
    graph.replay()
    check()


@pytest.mark.parametrize("first_call_captured", [False, True])
def test_captured_call_between_ordinary_ones(first_call_captured):
    """A captured call with grid barriers runs as often as its graph is replayed, whatever was called since: it finds its
    barrier words clear, and the words of ordinary calls are none of its business."""
    mlp = _Mlp()
    if first_call_captured:
        mlp.forget()
        mlp.ws[:32] = -1                        # what it needs is cleared, on an unknown workspace too

    def call():
        assert mlp.call() == 0

    def check():
        assert mlp.status() == 0 and torch.equal(mlp.out, mlp.want)
        mlp.out.zero_()
        mlp.hidden.zero_()

    graph = _graph(call)
    if first_call_captured:
        call()                                  # in front of the first replay
    _replays_and_calls(graph, call, check)


def test_captured_squeeze_and_excite_on_an_unknown_workspace():
    from souffle_models_b200 import efficientnet
    g = torch.Generator().manual_seed(1)
    x, wr, we = torch.randn(2, 24, 30, 30, generator=g).cuda(), torch.randn(6, 24, generator=g).cuda(), torch.randn(24, 6, generator=g).cuda()
    want = efficientnet.se_module(x, wr, we)[1].clone()
    out, lib = torch.empty_like(x), _lib()
    ws = torch.full((lib.souffle_se_module_workspace_bytes(2, 24, 30, 30) // 4,), -1, dtype=torch.int32, device="cuda")
    lib.souffle_workspace_forget(ws.data_ptr())

    def call():
        assert lib.souffle_se_module_forward(x.data_ptr(), wr.data_ptr(), we.data_ptr(), out.data_ptr(), None, 2, 24, 30, 30, 6,
                                             ws.data_ptr(), ws.numel() * 4, _stream()) == 0

    def check():
        assert lib.souffle_workspace_status(ws.data_ptr(), _stream()) == 0 and torch.equal(out, want)
        out.zero_()

    _replays_and_calls(_graph(call), call, check)


def test_captured_plans_between_ordinary_calls():
    from oracle import souffle_oracle as so
    from souffle_models_b200 import bert, lstm, swin
    cfg = so.BertConfig(2, 64, 2, 64, 512, "std")
    layers = [{k: v.cuda() for k, v in w.items()} for w in so.make_bert_weights(cfg, 3, 2)]
    enc = bert.BertEncoder(2, 64, 2, 64, 512, layers)
    blk = swin.SwinBlock(1, 14, 128, 4, 7, 3, {k: v.cuda() for k, v in so.make_swin_params(so.SwinConfig(res=14, dim=128, heads=4, window=7), 5).items()})
    x, w_in, w_st = so.make_lstm_params(3, 64, 8, seed=2)
    stack = lstm.LstmStack(w_in.cuda(), w_st.cuda(), 8)
    for plan, arg in ((enc, torch.randn(2, 64, 128).half().cuda()), (blk, torch.randn(196, 128).half().cuda()), (stack, x.float().cuda())):
        want, out = plan.forward(arg).clone(), []

        def call():
            out.append(plan.forward(arg))

        def check():
            plan.status()
            assert torch.equal(out[0], want) and torch.equal(out[-1], want)
            out[0].zero_()                      # the graph's buffer; an ordinary call brings its own

        graph = _graph(call)
        for step in "rcrrccr":
            if step == "r":
                graph.replay()
            else:
                call()
                out[0].copy_(want)
            check()
        graph.replay()
        graph.replay()
        check()


def test_a_refused_call_uses_no_barrier_words():
    """Rows beyond the limit are refused after the workspace has been looked at; the call behind it must not land on the
    words that the call in front of it has used."""
    mlp = _Mlp()
    for _ in range(3):
        assert mlp.call(rows=(1 << 20) + 1) == 1 and mlp.call() == 0 and mlp.status() == 0
        assert torch.equal(mlp.out, mlp.want)
        mlp.out.zero_()
        mlp.hidden.zero_()
