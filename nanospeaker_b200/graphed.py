"""CUDA-graph replay of a MoE block behind the module interface.

A block's training step is 15 to 17 launches; one native call per direction issues them in about
160 us of host time with autograd, which is what a step takes up to 2048 tokens. Nothing in the kernel
path reads a value on the host or has a data-dependent shape, so forward and backward can each be
captured once per input shape and replayed: 129 us at 300 tokens (167 eager), 146 at 2048 (162). Past that the copies into the graphs' buffers cost more
than the launches (16384: 421 against 390), and the block called directly is the faster one.
`GraphedMoEBlock` does that and stays a drop-in for the block: same call, same post-forward
attributes (`aux_loss`, `expert_counts`, `dropped`), autograd works as usual (the two graphs are
tied together by a native autograd node; by torch.cuda.make_graphed_callables where the weights are
cast on every call), parameters stay those of the wrapped block.

The caller loop this serves is the reference's micro-step, `loss, aux = model(x, y); (loss + aux)
.backward()` (src/train/train.py:317-324), where the block is called once per layer and step with a
fixed [batch, seq, d_model] shape.
"""
from typing import Dict, Tuple

import torch
from torch import nn

from . import moe_kernel as MK
from .moe import MoEBlock


class _BlockWithAux(nn.Module):
    """(out, aux_loss as fp32, expert_counts as fp32): the tensors a graph has to hand back."""

    def __init__(self, block: MoEBlock):
        super().__init__()
        self.block = block

    def forward(self, x):
        out = self.block(x)
        aux = self.block.aux_loss.to(torch.float32).reshape(())
        return out, aux, self.block.expert_counts.to(torch.float32)


class _OwnGradient(torch.autograd.Function):
    """The tensor itself, with a gradient of its own: torch's graphed callables hand back their own
    buffers, autograd takes such a buffer as p.grad without a copy, and the next replay overwrites it."""

    @staticmethod
    def forward(ctx, t):
        return t.view_as(t)

    @staticmethod
    def backward(ctx, grad):
        return grad.clone()


class GraphedMoEBlock(nn.Module):
    """`block(x)` replayed from CUDA graphs, one forward/backward pair per (input shape, dtype,
    training mode), captured on first use. Inputs the kernels decline (CPU tensors, other dtypes,
    exploration noise: anything `block._whole_block_ok` turns down) go through the block itself.

    The captured graphs hold the parameters by address: change them in place (an optimizer step
    does), do not replace them. The output, `aux_loss` and what the backward needs lie in the
    graphs' buffers: the next call of the same shape overwrites them. Gradients do not: any number
    of micro-steps may add up before they are cleared. A capture costs `warmup_iters` steps (at least
    one); do the first call of every shape outside any timed region."""

    def __init__(self, block: MoEBlock, warmup_iters: int = 3):
        super().__init__()
        self.block = block
        self.warmup_iters = warmup_iters
        self._pair = _BlockWithAux(block)
        self._graphed: Dict[Tuple, object] = {}

    # the attributes callers read after a forward (src/train/metrics.py:84-97)
    @property
    def aux_loss(self):
        return self.block.aux_loss

    @property
    def expert_counts(self):
        return self.block.expert_counts

    @property
    def dropped(self):
        return self.block.dropped

    @property
    def router(self):
        return self.block.router

    def _weights(self):
        b = self.block
        return b.router.W, b.W_in, b.W_out, b.W_sh_in, b.W_sh_out

    def _native_for(self, x2: torch.Tensor):
        """The native forward / backward graph pair (csrc/shim.cpp) for this input shape, or None
        where the block's weights or routing bias would have to be cast first."""
        b = self.block
        weights = self._weights()
        key = ("native", tuple(x2.shape), x2.dtype, x2.device, b.training, MK._atomic(b.combine_mode),
               b.router.logit_bias is None)
        g = self._graphed.get(key)
        if g is None:
            bias = b.router.logit_bias
            if (not all(w is None or (w.dtype == x2.dtype and w.is_contiguous()) for w in weights)
                    or not (bias is None or (bias.dtype == torch.float32 and bias.is_contiguous()))):
                return None
            rw, w_in, w_out, sh_in, sh_out = weights
            g = MK.K.shim().GraphedBlock(
                torch.randn_like(x2), rw, bias, w_in, w_out, sh_in, sh_out,
                b.router.top_k, bool(b.router.normalize_weights), b.router.wants_probs(),
                b.router.aux_loss_coef, MK._act_id(b._kernel_act), not MK._atomic(b.combine_mode),
                self.warmup_iters)
            self._graphed[key] = g
        return g

    def _callable_for(self, x: torch.Tensor):
        key = (tuple(x.shape), x.dtype, x.device, self.block.training, x.requires_grad)
        names, params = zip(*self._pair.named_parameters())
        fn = self._graphed.get(key)
        if fn is None:
            sample = torch.zeros_like(x).normal_().requires_grad_(x.requires_grad)

            def step(x, *weights):
                return torch.func.functional_call(self._pair, dict(zip(names, weights)), (x,))
            weights = (p.detach().requires_grad_(p.requires_grad) for p in params)
            fn = torch.cuda.make_graphed_callables(
                step, (sample, *weights), num_warmup_iters=self.warmup_iters,
                allow_unused_input=True)
            self._graphed[key] = fn
        return lambda x: fn(*(_OwnGradient.apply(t) if t.requires_grad else t
                              for t in (x, *params)))

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        b = self.block
        x2 = x.reshape(-1, x.shape[-1]) if x.dim() not in (1, 2) else x
        # (without autograd there is no backward to pair the forward with: the block's own
        # inference path is the lighter one then, and nanospeaker_b200.decode graphs it)
        if (not x.is_cuda or x2.shape[0] == 0 or x.shape[-1] != b.d_model
                or not torch.is_grad_enabled() or not b._whole_block_ok(x2)
                or (b.training and b.router.noise_std)):   # noise: fresh random numbers every call
            return b(x)
        if (x2.dim() == 2 and MK.native_ok(x2) and MK._aux_reduce is None
                and not MK._DEBUG_ONE_STREAM):
            g = self._native_for(x2)
            if g is not None:
                rw, w_in, w_out, sh_in, sh_out = self._weights()
                out, b.aux_loss, b.expert_counts = g.run(x2, rw, w_in, w_out, sh_in, sh_out)
                return out if x.dim() == 2 else out.view(x.shape)
        out, aux, counts = self._callable_for(x)(x)
        full = b.router.wants_probs()
        b.aux_loss = aux if full else torch.zeros((), device=x.device, dtype=x.dtype)
        b.expert_counts = counts.detach().to(torch.int32)
        return out
