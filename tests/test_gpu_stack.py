"""The one-kernel stack of blocks (csrc/stack.cu) against the layer-by-layer path on the same inputs."""
import pytest
import torch

from conftest import rel_l2
from oracle import moe_oracle as O

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


def _logits(b, x):
    """fp64 router logits with the routing bias, and the size of a bf16 step at each of them."""
    z = x.double() @ b.router.W.detach().double()
    step = torch.exp2(torch.floor(torch.log2(z.abs().clamp(min=2.0 ** -60))) - 7)
    bias = b.router.logit_bias
    return z if bias is None else z + bias.double(), step


def _clear(b, x):
    """Tokens whose selection no order of summation can change: the k-th and the next logit, each off by
    half a bf16 step at most, lie more than two steps apart."""
    z, step = _logits(b, x)
    if b.top_k == b.n_experts:
        return torch.ones(x.shape[0], dtype=torch.bool, device=x.device)
    top, at = z.topk(b.top_k + 1, dim=1)
    step = step.gather(1, at)
    return top[:, -2] - top[:, -1] > 2 * torch.maximum(step[:, -2], step[:, -1])


def _clear_tokens(b, T):
    x = torch.randn(4 * T + 64, b.d_model, device="cuda").bfloat16()
    x = x[_clear(b, x)]
    assert x.shape[0] >= T
    return x[:T].contiguous()


def _token_errors(got, want):
    return (got.double() - want.double()).norm(dim=1) / want.double().norm(dim=1)


@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17, 33, 64, 149, 256])
@pytest.mark.parametrize("kw", [dict(), dict(bias=True), dict(d=96, e=8, k=2, s=0, act="gelu"),
                                dict(d=1024, e=128, k=8, s=1, normalize=False),
                                dict(d=608, e=16, k=4, s=2, bias=True)])
def test_one_layer_equals_the_separate_kernels(T, kw):
    """One layer on the same input: every token within bf16 rounding. (The router's logits are summed in
    another order here, so the tokens are ones whose selection that cannot change.)"""
    from nanospeaker_b200 import kernels
    from nanospeaker_b200.decode import StackedMoEDecoder
    b, = _blocks(1, seed=T, **kw)
    x = _clear_tokens(b, T)
    stack = StackedMoEDecoder([b])
    assert stack._stack_plan(x) is not None
    got, want = stack.eager(x), _layer(b, x)
    assert torch.equal(got, stack.eager(x))                     # bit-reproducible
    kernels.check_status("cuda")
    # both round the sum to bf16 (2^-9 of a value at most), the separate kernels each of its terms before
    off = _token_errors(got, want)
    assert float(off.max()) < 6e-3, off
    assert rel_l2(got, want) < 4e-3


def _oracle_layer(b, x, swap):
    """x + block(x) in fp32 on the CPU, selecting from bf16-rounded logits; swap: the k-th and the next
    expert change places."""
    f = lambda t: None if t is None else t.detach().float().cpu()
    z = (x.double() @ b.router.W.detach().double()).bfloat16().float()
    if b.router.logit_bias is not None:
        z = z + b.router.logit_bias
    z = z.cpu()
    idx = O.canonical_topk(z, b.top_k + 1)
    idx = torch.cat([idx[:, :b.top_k - 1], idx[:, b.top_k:]], 1) if swap else idx[:, :b.top_k]
    w, idx, _ = O.router_select(z, b.top_k, b.router.normalize_weights, False, idx)
    return f(x) + O.experts_forward(f(x), f(b.W_in), f(b.W_out), w.bfloat16().float(), idx, b.activation,
                                    f(b.W_sh_in), f(b.W_sh_out))


@pytest.mark.parametrize("T", [1, 8, 64, 200])
@pytest.mark.parametrize("kw", [dict(), dict(d=608, e=16, k=4, s=1, act="gelu", bias=True),
                                dict(d=1024, e=128, k=8, s=0, normalize=False)])
def test_every_layer_of_the_stack_equals_the_fp32_oracle(T, kw):
    """The stack's output behind each of its layers (the stacks of the first 1, 2, ... blocks: results are
    bit-reproducible) against the oracle on what the layer before has left. A token whose k-th and next
    logit are within two bf16 steps may have either of the two experts; none is left out."""
    from nanospeaker_b200 import kernels
    from nanospeaker_b200.decode import StackedMoEDecoder
    blocks = _blocks(4, seed=T + 1, **kw)
    before = x = _clear_tokens(blocks[0], T)
    with torch.no_grad():
        for n, b in enumerate(blocks, 1):
            got = StackedMoEDecoder(blocks[:n]).eager(x)
            clear = _clear(b, before).cpu()
            off = _token_errors(got.cpu(), _oracle_layer(b, before, False))
            if not clear.all():
                other = _token_errors(got.cpu(), _oracle_layer(b, before, True))
                off = torch.where(clear, off, torch.minimum(off, other))
            # the hidden units, the logits, the weights and the result are each rounded to bf16: 2^-9 at
            # most, 2^-9 / sqrt(3) in the norm, together 2^-9 * sqrt(4 / 3); twice that for a single token
            # (a wrong expert: 8.5e-3 and more)
            assert float(off.max()) < 2 * 2.0 ** -9 * (4 / 3) ** 0.5, (n, off)
            before = got
    kernels.check_status("cuda")


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


def test_the_one_kernel_stack_needs_no_padded_router_weights():
    from nanospeaker_b200 import kernels
    from nanospeaker_b200.decode import StackedMoEDecoder
    blocks = _blocks(2)
    stack = StackedMoEDecoder(blocks)
    x = torch.randn(3, 576, device="cuda").bfloat16()
    before = kernels.LAUNCHES
    assert stack._stack_plan(x) is not None and kernels.LAUNCHES == before
    want = _layer(blocks[1], _layer(blocks[0], x))              # layer by layer they are made, and kept
    kept = [stack._fast_args(b, x)[0] for b in blocks]
    assert all(stack._fast_args(b, x)[0] is w for b, w in zip(blocks, kept))
    from nanospeaker_b200 import moe_kernel as MK
    MK._ONE_CALL = False
    try:
        assert rel_l2(stack.eager(x), want) < 1e-6
    finally:
        MK._ONE_CALL = True


def test_a_router_weight_at_any_address():
    from nanospeaker_b200.decode import StackedMoEDecoder
    b, = _blocks(1)
    x = torch.randn(5, 576, device="cuda").bfloat16()
    want = StackedMoEDecoder([b]).eager(x)
    flat = torch.zeros(576 * 76 + 8, device="cuda", dtype=torch.bfloat16)
    w = flat[3:3 + 576 * 76].view(576, 76)
    w.copy_(b.router.W.detach())
    b.router.W = torch.nn.Parameter(w)
    assert b.router.W.data_ptr() % 16
    stack = StackedMoEDecoder([b])
    assert stack._stack_plan(x) is not None and torch.equal(stack.eager(x), want)
