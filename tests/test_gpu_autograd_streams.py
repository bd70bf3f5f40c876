"""The differentiable loss on streams: its calls, and other calls on the same
context, give the same losses and gradients whatever stream they are issued on
and whatever is still pending there, at widths with and without padding."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import cloverleaf_gb300 as cl
from cloverleaf_gb300 import _native
from cloverleaf_gb300.autograd import EPBatchLoss
from tests._cases import random_problem, rel_err, sample_batch

pytestmark = pytest.mark.gpu
WAIT = 40_000_000       # clock cycles of a pending kernel (about 20 ms)


def _loss(dims, n_feat=300, seed=5):
    prob = random_problem(seed, n=600, n_feat=n_feat, dims=dims, deg=(1, 12), feats=(1, 6))
    f = EPBatchLoss(prob["rows"], prob["cols"], prob["fptr"], prob["fids"], n_feat, dims, cl.EPLoss.starspace(0.5, 4))
    return prob, f


def _args(prob, B, seed, K=6):
    s = sample_batch(seed, prob, B=B, K=K, R=4)
    return s["anchors"], s["nbr_ptr"], s["nbr"], s["nbr_w"], s["neg"]


def _grad(f, table, args, dtype=torch.float32, stream=None):
    with torch.cuda.stream(stream):
        t = torch.tensor(table, device="cuda", dtype=dtype, requires_grad=True)
        lv = f(t, *args)
        lv.sum().backward()
        out = lv.detach().cpu().numpy(), t.grad.cpu().numpy()
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("dims", [1, 20, 33, 36, 64, 100, 130])
def test_backward_after_another_forward(oracle, dims, dtype):
    # the backward of a batch stages it again: another batch, larger (the
    # scratch grows) or smaller, and a backward of that one may lie between
    prob, f = _loss(dims)
    a, b = _args(prob, 40, 1), _args(prob, 500, 2, K=12)
    alone = [_grad(_loss(dims)[1], prob["table"], x, dtype) for x in (a, b)]
    cfg = oracle.loss_cfg(loss=1, gamma=0.5, grad_mode=1)
    og = oracle.batch(prob["fptr"], prob["fids"], 300, prob["table"], prob["rows"], *a, cfg, "f64")[2]
    if dims > 1:    # in one dimension every cosine is 1 or -1 and the gradient 0: nothing to be relative to
        assert rel_err(alone[0][1], og) < 1e-4
    for stream in (None, torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            ta, tb = (torch.tensor(prob["table"], device="cuda", dtype=dtype, requires_grad=True) for _ in range(2))
            la = f(ta, *a)
            lb = f(tb, *b)
            la.sum().backward(retain_graph=True)
            lb.sum().backward()
            first = ta.grad.cpu().numpy()
            ta.grad = None
            la.sum().backward()
            got = [(la.detach().cpu().numpy(), first), (lb.detach().cpu().numpy(), tb.grad.cpu().numpy())]
        for (l0, g0), (l1, g1) in zip(alone, got):
            assert np.array_equal(l0, l1, equal_nan=True) and np.array_equal(g0, g1)
        assert np.array_equal(ta.grad.cpu().numpy(), alone[0][1])


@pytest.mark.parametrize("dims", [20, 64])
def test_calls_after_a_pending_stage(dims):
    # ep_ag_stage returns with its copies pending on the caller's stream; the
    # next call, on another stream and larger, waits for them
    prob, f = _loss(dims)
    ctx = f.ctx
    small, large = _args(prob, 30, 3), _args(prob, 700, 4, K=12)
    want_small, want_large = (_grad(_loss(dims)[1], prob["table"], x) for x in (small, large))
    ref = _native.Context(ctx.cfg)
    for c in (ref, ctx):
        c.upload_graph(prob["rows"], prob["cols"], None)
        c.upload_features(prob["fptr"], prob["fids"], 300)
        c.set_table(prob["table"])
    want_rows = ref.batch_grad(_native.Context.samples(*small), 300, dims)
    table = torch.tensor(prob["table"], device="cuda")
    s_small, s_large = _native.Context.samples(*small), _native.Context.samples(*large)
    side, third = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def stage(s):
        with torch.cuda.stream(side):
            torch.cuda._sleep(WAIT)
        ctx.ag_stage(s, 0, table.data_ptr(), side.cuda_stream)
        return not side.query()

    # a forward on a third stream that grows scratch and page-locked memory
    assert stage(s_small)
    assert np.array_equal(_grad(f, prob["table"], large, stream=third)[1], want_large[1])
    # a call on the context's own stream
    assert stage(s_large)
    got = ctx.batch_grad(s_small, 300, dims)
    for x, y in zip(got, want_rows):
        assert np.array_equal(x, y, equal_nan=True)
    # stage after stage, then the backward of the last
    assert stage(s_large)
    ctx.ag_stage(s_small, 0, table.data_ptr(), third.cuda_stream)
    with torch.cuda.stream(third):
        grad = torch.empty_like(table)
        ones = torch.ones(30, device="cuda")
        ctx.ag_backward(ones.data_ptr(), grad.data_ptr(), third.cuda_stream)
    assert np.array_equal(grad.cpu().numpy(), want_small[1])
    # a context given back with its stage pending
    assert stage(s_large)
    f.ctx.close()
    torch.cuda.synchronize()


def test_first_batch_on_a_side_stream_behind_the_upload():
    # a new context still initialises a large table on its own stream while a
    # side stream stages the first batch and the scratch is cleared
    n_feat, dims = 2_000_000, 64
    prob = random_problem(8, n=600, n_feat=n_feat, dims=1, deg=(1, 12), feats=(1, 6))
    args = _args(prob, 200, 6)
    table = torch.randn(n_feat, dims, generator=torch.Generator("cuda").manual_seed(1), device="cuda")
    out = []
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream(), torch.cuda.Stream()):
        f = EPBatchLoss(prob["rows"], prob["cols"], prob["fptr"], prob["fids"], n_feat, dims, cl.EPLoss.starspace(0.5, 4))
        torch.cuda.synchronize()
        f.ctx.set_table(None)
        with torch.cuda.stream(stream):
            t = table.detach().requires_grad_()
            lv = f(t, *args)
            lv.sum().backward()
            out.append((lv.detach().cpu(), t.grad.cpu()))
    for lv, g in out[1:]:
        assert torch.equal(lv, out[0][0]) and torch.equal(g, out[0][1])


@pytest.mark.parametrize("dims", [20, 64])
@pytest.mark.parametrize("default", [True, False])
def test_table_and_upstream_gradient_still_being_computed(dims, default):
    # the kernels that write the table and the upstream gradient are pending on
    # the caller's stream, the default stream or another, when the call is made
    prob, f = _loss(dims)
    args = _args(prob, 100, 9)
    want_loss, want = _grad(_loss(dims)[1], prob["table"], args)
    src = torch.tensor(prob["table"], device="cuda")
    weight = torch.linspace(0.5, 2.0, 100, device="cuda")
    f(src, *args)                       # scratch is allocated
    stream = torch.cuda.default_stream() if default else torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        t = torch.full_like(src, 7.0).requires_grad_()
        torch.cuda._sleep(WAIT)
        with torch.no_grad():
            t.copy_(src)
        assert not stream.query()
        lv = f(t, *args)
        lv.sum().backward()
        assert np.array_equal(lv.detach().cpu().numpy(), want_loss, equal_nan=True)
        assert np.array_equal(t.grad.cpu().numpy(), want)
        # the same upstream gradient, late and at once
        grads = []
        for late in (False, True):
            t.grad = None
            lv = f(t, *args)
            torch.cuda.synchronize()
            up = torch.full_like(weight, 3.0)
            if late:
                torch.cuda._sleep(WAIT)
            up.copy_(weight)
            lv.backward(up)
            grads.append(t.grad.cpu().numpy())
        assert np.array_equal(grads[0], grads[1]) and not np.array_equal(grads[0], want)
