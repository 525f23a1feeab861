"""The pybind shim (csrc/shim.cpp: one native call per direction, native autograd node) with the block's
options against the stage-by-stage sequence of the registered ops on the same inputs."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
ATOMIC_TOL = 8e-3      # bf16 adds in no fixed order, on both sides


def _block(bias, capacity, n_shared, combine, train=True, d=576, e=76, k=6):
    from nanospeaker_b200 import MoEBlock
    m = MoEBlock(d, e, d_ff=192, top_k=k, n_shared=n_shared, capacity_factor=capacity, bias=bias)
    with torch.no_grad():
        for n, p in m.named_parameters():
            std = p.shape[1] ** -0.5 if n.startswith("W_") else (0.02 if n == "router.W" else 0.1)
            p.copy_(torch.randn_like(p) * std)
    m = m.to(torch.bfloat16).cuda().train(train)
    m.combine_mode = combine
    m.router.logit_bias = torch.randn(e, device="cuda") * 0.3
    return m


def _step(m, x, gout):
    xc = x.clone().requires_grad_(True)
    for p in m.parameters():
        p.grad = None
    torch.manual_seed(3)                       # the same exploration noise on both sides
    out = m(xc)
    torch.autograd.backward([out, m.aux_loss], [gout, torch.ones_like(m.aux_loss)])
    return dict(out=out.detach(), aux=m.aux_loss.detach().clone(), dx=xc.grad,
                **{n: p.grad for n, p in m.named_parameters()}), m.expert_counts, m.dropped


@pytest.mark.parametrize("T", [1, 129, 700])
@pytest.mark.parametrize("bias,capacity,n_shared,combine,noise", [
    (True, None, 2, "atomic", 0.0), (True, 1.0, 0, "store", 0.0), (False, 0.5, 2, "atomic", 0.5),
    (False, 1.25, 1, "store", 0.0), (False, None, 2, "store", 0.0)])
def test_native_block_equals_the_stage_sequence(T, bias, capacity, n_shared, combine, noise):
    from nanospeaker_b200 import kernels, moe_kernel as MK
    torch.manual_seed(T)
    m = _block(bias, capacity, n_shared, combine)
    m.router.noise_std = noise
    x = torch.randn(T, 576, device="cuda").bfloat16()
    gout = torch.randn(T, 576, device="cuda").bfloat16()
    got, counts, dropped = _step(m, x, gout)
    m(x)
    assert m.aux_loss.grad_fn.name() == "MoEBlockBackward"
    MK._ONE_CALL = False
    try:
        want, counts_w, dropped_w = _step(m, x, gout)
    finally:
        MK._ONE_CALL = True
    assert torch.equal(counts.long(), counts_w.long()) and int(dropped) == int(dropped_w)
    for n in want:
        if n == "aux":
            assert abs(float(got[n]) - float(want[n])) < 1e-5
        elif float(want[n].float().norm()) > 0:
            # (the router gradient is a sum of bf16-rounded d topk_w: 2e-2 here as everywhere)
            assert rel_l2(got[n], want[n]) < (2e-2 if n == "router.W" else ATOMIC_TOL), n
    kernels.check_status("cuda")


def test_native_block_without_autograd_and_without_the_balance_loss():
    from nanospeaker_b200 import moe_kernel as MK
    torch.manual_seed(0)
    m = _block(True, None, 2, "store", train=False)
    x = torch.randn(3, 7, 576, device="cuda").bfloat16()
    with torch.no_grad():
        out = m(x)
        aux, counts = m.aux_loss, m.expert_counts
        assert aux.dtype == x.dtype and float(aux) == 0.0 and int(counts.sum()) == 21 * 6
        MK._ONE_CALL = False
        try:
            assert rel_l2(out, m(x)) < 1e-5
        finally:
            MK._ONE_CALL = True
    # a frozen block on an input that needs a gradient, and one backward through each output alone
    for p in m.parameters():
        p.requires_grad_(False)
    xc = x.clone().requires_grad_(True)
    m(xc).float().sum().backward()
    assert torch.isfinite(xc.grad.float()).all() and m.W_in.grad is None


@pytest.mark.parametrize("combine,n_shared,T", [("atomic", 2, 300), ("store", 0, 1)])
def test_native_sublayer_equals_the_python_node(combine, n_shared, T):
    from nanospeaker_b200 import MoEFFNSublayer, moe_kernel as MK
    torch.manual_seed(T)
    sub = MoEFFNSublayer(_block(False, None, n_shared, combine)).to(torch.bfloat16).cuda()
    x = torch.randn(T, 576, device="cuda").bfloat16()
    gout = torch.randn(T, 576, device="cuda").bfloat16()
    res = []
    for native in (True, False):
        MK._ONE_CALL = native
        try:
            xc = x.clone().requires_grad_(True)
            for p in sub.parameters():
                p.grad = None
            out, aux = sub(xc)
            torch.autograd.backward([out, aux], [gout, torch.ones_like(aux)])
        finally:
            MK._ONE_CALL = True
        res.append(dict(out=out.detach(), dx=xc.grad, **{n: p.grad for n, p in sub.named_parameters()}))
    for n in res[0]:
        assert rel_l2(res[0][n], res[1][n]) < ATOMIC_TOL, n


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])   # (fp32: torch's graphed callable)
def test_graphed_gradients_stay_when_the_next_backward_replays(dtype):
    """Micro-steps that add up without clearing, against the block called directly; then gradients kept
    by the caller over more steps than the graphs have sets of buffers."""
    from nanospeaker_b200 import GraphedMoEBlock, kernels
    T = 200
    m = _block(False, None, 2, "store").to(dtype)
    g = GraphedMoEBlock(m)
    params = list(m.parameters())
    gouts = [torch.randn(T, 576, device="cuda").bfloat16() for _ in range(5)]
    xs = [torch.randn(T, 576, device="cuda").bfloat16() for _ in range(5)]

    def grads(call, i):
        x = xs[i].clone().requires_grad_(True)
        return torch.autograd.grad([call(x)], [x, *params], [gouts[i]])
    want = [grads(m, i) for i in range(5)]
    for _ in range(2):                                   # twice: cleared in between
        for p in params:
            p.grad = None
        total = [torch.zeros_like(p) for p in params]
        for i in range(4):
            g(xs[i].clone().requires_grad_(True)).backward(gouts[i])
            for t, w in zip(total, want[i][1:]):
                t.add_(w)
            for p, t in zip(params, total):
                assert torch.equal(p.grad, t), i
    kept = [grads(g, i) for i in range(5)]
    for a, b in zip(kept, want):
        assert all(torch.equal(u, v) for u, v in zip(a, b))
    kernels.check_status("cuda")


def test_graphed_block_runs_the_warm_up_it_is_asked_for():
    from nanospeaker_b200 import GraphedMoEBlock, kernels
    m = _block(False, None, 2, "store")
    x = torch.randn(64, 576, device="cuda").bfloat16().requires_grad_(True)
    launches = []
    for n in (1, 4):
        before = kernels.LAUNCHES
        g = GraphedMoEBlock(m, warmup_iters=n)
        g(x)
        launches.append(kernels.LAUNCHES - before)
    before = kernels.LAUNCHES
    g(x).float().sum().backward()
    assert launches[1] - launches[0] == 3 * (kernels.LAUNCHES - before)


@pytest.mark.parametrize("kind", ["plain", "bias", "capacity", "sublayer", "graphed"])
def test_forward_mode_is_refused(kind):
    import torch.autograd.forward_ad as fwad
    from nanospeaker_b200 import GraphedMoEBlock, MoEFFNSublayer
    m = _block(kind == "bias", 1.25 if kind == "capacity" else None, 2, "store")
    call = (MoEFFNSublayer(m).to(torch.bfloat16).cuda() if kind == "sublayer" else
            GraphedMoEBlock(m) if kind == "graphed" else m)
    x = torch.randn(16, 576, device="cuda").bfloat16()
    with fwad.dual_level(), pytest.raises(NotImplementedError, match="forward mode"):
        call(fwad.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("kind", ["plain", "bias", "capacity", "sublayer", "graphed"])
def test_gradients_are_not_differentiated_again(kind):
    """create_graph gives the same gradients, and an error where they would be differentiated (made without
    grad mode, they would pass for constants)."""
    from nanospeaker_b200 import GraphedMoEBlock, MoEFFNSublayer
    m = _block(kind == "bias", 1.25 if kind == "capacity" else None, 2, "store")
    call = (MoEFFNSublayer(m).to(torch.bfloat16).cuda() if kind == "sublayer" else
            GraphedMoEBlock(m) if kind == "graphed" else m)
    x = torch.randn(16, 576, device="cuda").bfloat16().requires_grad_(True)
    first = lambda: call(x)[0] if kind == "sublayer" else call(x)
    params = list(call.parameters())
    for loss in (lambda o: o.float().sum(), lambda o: o.float().square().sum()):
        want = torch.autograd.grad(loss(first()), [x, *params], allow_unused=True)
        got = torch.autograd.grad(loss(first()), [x, *params], create_graph=True, allow_unused=True)
        assert all((a is None) == (b is None) for a, b in zip(got, want))
        if kind != "sublayer":      # (there the bf16 sums of the norm's weight come in any order)
            assert all(torch.equal(a, b) for a, b in zip(got, want) if a is not None)
        with pytest.raises(RuntimeError, match="differentiated again"):
            (got[0].float().sum() + x.float().sum()).backward()
