"""The one-kernel stack of blocks (csrc/stack.cu) against the layer-by-layer path on the same inputs."""
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _blocks(n, d=576, e=76, k=6, s=2, normalize=True, act="silu", bias=False, seed=0):
    from nanospeaker_b200 import MoEBlock
    torch.manual_seed(seed)
    out = []
    for _ in range(n):
        m = MoEBlock(d, e, d_ff=192, top_k=k, n_shared=s, capacity_factor=None, activation=act,
                     normalize_weights=normalize)
        with torch.no_grad():
            for name, p in m.named_parameters():
                if name.startswith("W_"):
                    p.copy_(torch.randn_like(p) * p.shape[1] ** -0.5)
        m = m.to(torch.bfloat16).cuda().eval()
        if bias:
            m.router.logit_bias = torch.randn(e, device="cuda") * 1.5   # some experts idle, one full
        out.append(m)
    return out


def _layer(b, x):
    """The same layer by the separate kernels."""
    from nanospeaker_b200 import moe_kernel as MK
    wp = MK.pad_router_weight(b.router.W.detach(), x.dtype)
    return MK.moe_block_inference(x, wp, b.router.logit_bias, b.W_in.detach(), b.W_out.detach(),
                                  None if b.W_sh_in is None else b.W_sh_in.detach(),
                                  None if b.W_sh_out is None else b.W_sh_out.detach(), b.n_experts,
                                  b.router.top_k, b.router.normalize_weights, b._kernel_act,
                                  residual=x, combine="store")


@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17, 33, 64, 149, 256])
@pytest.mark.parametrize("kw", [dict(), dict(bias=True), dict(d=96, e=8, k=2, s=0, act="gelu"),
                                dict(d=1024, e=128, k=8, s=1, normalize=False),
                                dict(d=608, e=16, k=4, s=2, bias=True)])
def test_one_layer_equals_the_separate_kernels(T, kw):
    """One layer on the same input: outputs within bf16 rounding. (The router's logits are summed in
    another order here, so a pair of bf16-tied logits may be resolved differently: such tokens are
    few and left out.)"""
    from nanospeaker_b200 import kernels
    from nanospeaker_b200.decode import StackedMoEDecoder
    b, = _blocks(1, seed=T, **kw)
    x = torch.randn(T, b.d_model, device="cuda").bfloat16()
    stack = StackedMoEDecoder([b])
    assert stack._stack_plan(x) is not None
    got, want = stack.eager(x), _layer(b, x)
    assert torch.equal(got, stack.eager(x))                     # bit-reproducible
    kernels.check_status("cuda")
    off = (got.float() - want.float()).norm(dim=1) / want.float().norm(dim=1)
    assert int((off > 6e-3).sum()) <= max(1, T // 16), off
    same = off <= 6e-3
    assert rel_l2(got[same], want[same]) < 4e-3


def test_stack_runs_all_layers_and_in_a_graph():
    from nanospeaker_b200 import kernels
    from nanospeaker_b200.decode import StackedMoEDecoder
    blocks = _blocks(5)
    with torch.no_grad():
        for b in blocks:
            for p in (b.W_in, b.W_sh_in, b.W_out, b.W_sh_out):
                p.mul_(0.5)
    stack = StackedMoEDecoder(blocks)
    for T in (1, 20, 64, 300):                                  # 300: layer by layer
        x = torch.randn(T, 576, device="cuda").bfloat16()
        assert (stack._stack_plan(x) is not None) == (T <= 256)
        want = x
        for b in blocks:
            want = StackedMoEDecoder([b]).eager(want)
        got = stack.step(x)
        assert torch.equal(got, want) and torch.equal(stack.step(x), want)
        y = torch.randn(T, 576, device="cuda").bfloat16()
        assert torch.equal(stack.step(y), stack.eager(y))
    kernels.check_status("cuda")
