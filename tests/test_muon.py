"""Muon's batched Newton-Schulz on the stacked expert weights (nanospeaker_b200/muon.py) against the
oracle's restatement of src/train/optim.py:27-105 and the golden the reference produced."""
import pytest
import torch

from conftest import rel_l2
from oracle import moe_oracle as O
from test_oracle import _muon_golden


def test_torch_path_matches_the_reference_golden_on_cpu():
    from nanospeaker_b200.muon import Muon, newton_schulz5
    g, t = _muon_golden()
    for tag, _ in O.MUON_SHAPES:
        assert torch.equal(newton_schulz5(t[f"g_{tag}"]), g[f"ns_{tag}"]), tag
        w = torch.nn.Parameter(t[f"w_{tag}"].clone())
        opt = Muon([w], lr=0.02, momentum=0.95, weight_decay=0.1, ns_steps=5)
        for step in range(2):
            w.grad = t[f"grad_{tag}_{step}"].clone()
            opt.step()
        assert torch.equal(w.detach().reshape(-1)[::7], g[f"w_{tag}_after"]), tag
        assert opt.update_norm_ratio() > 0
    one = newton_schulz5(t["g_out"][0])            # a single matrix
    assert torch.equal(one, g["ns_out"][0])


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(78, 576, 256), (78, 128, 576), (3, 256, 576), (2, 128, 256)])
def test_kernel_newton_schulz_matches_the_oracle(shape):
    """The stacked weight-gradient shapes of the block (dW_in and dW_sh_in together: 78 x [576, 256],
    dW_out: 78 x [128, 576]) through the grouped tcgen05 GEMMs: against the oracle's bf16 iteration
    and the fp32 iteration. Five bf16 Newton-Schulz steps are noisy by themselves: the reference's
    own bf16 result sits 2.5e-2 (rel-L2) from the fp32 iteration on these inputs, and the kernels
    round in fewer places (one rounding per a X + b Y), so the bars are 4e-2 against the bf16
    oracle and 3e-2 against fp32; plus the defining property (singular values near 1)."""
    from nanospeaker_b200 import kernels
    from nanospeaker_b200.muon import _kernel_ok, newton_schulz5
    torch.manual_seed(5)
    g = (torch.randn(*shape) * 0.02).bfloat16()
    assert _kernel_ok(g.cuda())
    before = kernels.LAUNCHES
    got = newton_schulz5(g.cuda()).cpu()
    assert kernels.LAUNCHES - before >= 2 + 5 * 5        # no per-expert loop: 5 launches an iteration
    want = O.newton_schulz5(g)
    assert got.shape == g.shape and got.dtype == torch.bfloat16
    assert rel_l2(got, want) < 4e-2
    # fp32 iteration on the same bf16 input
    x = g.float()
    tall = shape[1] > shape[2]
    x = x.mT if tall else x
    x = x / (x.norm(dim=(-2, -1), keepdim=True) + 1e-7)
    for _ in range(5):
        a = x @ x.mT
        x = 3.4445 * x + (-4.7750 * a + 2.0315 * (a @ a)) @ x
    x = x.mT if tall else x
    assert rel_l2(got, x) < 3e-2
    sv = torch.linalg.svdvals(got[0].float())
    assert 0.6 < float(sv.min()) and float(sv.max()) < 1.3
    kernels.check_status("cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(10, 576, 256), (13, 576, 128), (11, 576, 256)])
def test_kernel_newton_schulz_on_stacks_cut_into_chunks(shape):
    """More than eight matrices whose Gram products are cut into three chunks each: 30, 39 and 33 work items.
    Every matrix against the fp32 iteration, to the bar of the test above."""
    from nanospeaker_b200 import kernels
    from nanospeaker_b200.muon import _kernel_ok, newton_schulz5
    g = (torch.randn(*shape) * 0.02).bfloat16().cuda()
    assert _kernel_ok(g)
    got = newton_schulz5(g).float()
    x = g.double().mT
    x = x / (x.norm(dim=(-2, -1), keepdim=True) + 1e-7)
    for _ in range(5):
        a = x @ x.mT
        x = 3.4445 * x + (-4.7750 * a + 2.0315 * (a @ a)) @ x
    off = (got - x.mT).norm(dim=(-2, -1)) / x.norm(dim=(-2, -1))
    assert float(off.max()) < 3e-2
    kernels.check_status("cuda")


@pytest.mark.gpu
def test_muon_step_on_the_blocks_gradients():
    """One optimizer step on a block's stacked expert weights with the gradients its backward left,
    on the GPU (kernel Newton-Schulz) against the oracle's step on the CPU."""
    from nanospeaker_b200 import MoEBlock
    from nanospeaker_b200.muon import Muon
    torch.manual_seed(1)
    m = MoEBlock(576, 8, d_ff=192, top_k=2, n_shared=1, capacity_factor=None)
    m = m.to(torch.bfloat16).cuda()
    x = torch.randn(512, 576, device="cuda").bfloat16()
    (m(x).float().square().mean() + m.aux_loss).backward()
    params = [m.W_in, m.W_out, m.W_sh_in, m.W_sh_out]
    ref = [(p.detach().cpu().clone(), p.grad.cpu().clone()) for p in params]
    opt = Muon(params, lr=0.02)
    opt.step()
    for p, (w, gr) in zip(params, ref):
        decayed = w.float() * (1 - 0.02 * 0.1)
        delta = O.muon_step(w, gr, torch.zeros_like(w))          # updates w in place
        # (these gradients have rank <= rows per expert < 256: the iteration amplifies rounding
        # noise in the near-null directions, so the applied step is compared loosely)
        assert rel_l2(p.detach().cpu(), w) < 1e-2                # the updated weights
        assert rel_l2(p.detach().cpu().float() - decayed, delta.float()) < 0.2    # the applied step
    assert 0 < opt.update_norm_ratio() < 1


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_native_muon_step_equals_the_operations_one_by_one(dtype):
    """Several steps over stacks and a single matrix (whole and ragged tiles of the long side, all of it
    on chip and streamed, one shape that the fused iteration declines) against the step in torch operations on copies: momentum bit for bit, weights and the
    update / weight norm ratio within the iteration's bf16 noise."""
    from nanospeaker_b200 import kernels, muon as MU
    torch.manual_seed(3)
    shapes = [(5, 576, 256), (2, 256, 256), (1, 288, 256), (2, 1056, 256), (5, 128, 576), (128, 128),
              (2, 128, 768), (3, 128, 1056), (3, 96, 64)]
    a = [torch.nn.Parameter((torch.randn(*s) * 0.05).to(dtype).cuda()) for s in shapes]
    b = [torch.nn.Parameter(p.detach().clone()) for p in a]
    oa, ob = MU.Muon(a, lr=0.02), MU.Muon(b, lr=0.02)
    for step in range(3):
        for p, q in zip(a, b):
            p.grad = torch.randn_like(p)
            q.grad = p.grad.clone()
        version, before = a[0]._version, [p.detach().clone() for p in a]
        oa.step()
        assert a[0]._version > version
        native = MU._native_ok
        MU._native_ok = lambda p, buf: False
        try:
            ob.step()
        finally:
            MU._native_ok = native
        for p, q, p0 in zip(a, b, before):
            assert torch.equal(oa.state[p]["momentum"], ob.state[q]["momentum"])
            assert rel_l2(p.detach(), q.detach()) < 2e-3
            if dtype == torch.float32:
                decayed = p0 * (1 - 0.02 * 0.1)
                assert rel_l2(p.detach() - decayed, q.detach() - decayed) < 2e-2, tuple(p.shape)
            q.data.copy_(p.data)
        assert abs(oa.update_norm_ratio() / ob.update_norm_ratio() - 1) < 2e-2
    kernels.check_status("cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("value", [0.0, 1e-30, 1e25, float("inf"), float("nan")])
def test_native_muon_step_with_extreme_gradients(value):
    """Directions whose norm vanishes, overflows or is no number, beside ordinary ones, against the step in
    torch operations: where that leaves numbers the same numbers, where it leaves none, none."""
    from nanospeaker_b200 import kernels, muon as MU
    torch.manual_seed(4)
    shapes = [(3, 576, 256), (3, 128, 576)]
    res = []
    start = [(torch.randn(*s) * 0.05).bfloat16().cuda() for s in shapes]
    grads = [torch.randn_like(p) for p in start]
    finite = value == value and abs(value) != float("inf")
    for g in grads:
        if finite:
            g[1].sign_().mul_(value)
        else:
            g[1, 5, 7] = value
    for native in (True, False):
        params = [torch.nn.Parameter(p.clone()) for p in start]
        opt = MU.Muon(params, lr=0.02)
        for p, g in zip(params, grads):
            p.grad = g.clone()
        keep = MU._native_ok
        if not native:
            MU._native_ok = lambda p, buf: False
        try:
            opt.step()
        finally:
            MU._native_ok = keep
        res.append([p.detach() for p in params])
    for a, b in zip(*res):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b))
        assert bool(torch.isfinite(b[1]).all()) == finite
        if finite:
            assert rel_l2(a[1], b[1]) < 2e-3
        assert rel_l2(a[[0, 2]], b[[0, 2]]) < 2e-3
    kernels.check_status("cuda")
