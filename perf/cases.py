"""The work this package does for its users, as timed cases: one pass each through the public entry
points, over the range of batch sizes, options and directions that the block is called with.

Kinds of a case:
  decode    StackedMoEDecoder.step: a stack of blocks on one token per sequence (generation)
  infer     MoEBlock.forward without autograd: prompt prefill and evaluation
  train     MoEBlock.forward + backward, eager: the block inside a training step
  graphed   the same step through GraphedMoEBlock (a trainer with a fixed micro-batch shape)
  sublayer  MoEFFNSublayer forward + backward: x + ffn(rmsnorm(x)), one per layer of the model
  muon      Muon.step over the stacked expert weights of one block

Sizes: the model's block (d_model 576, 76 routed + 2 shared experts of hidden width 128, top-6) with
the batch sizes of the benchmark configurations (64, 2048, 16384, 131072 tokens) and ragged ones in
between; draws also take other widths, expert counts and top-k of the kernels' grid.
"""
import torch

from nanospeaker_b200 import GraphedMoEBlock, MoEBlock, MoEFFNSublayer, Muon
from nanospeaker_b200.decode import StackedMoEDecoder

D_HIDDEN = 128          # the expert width the kernels are built for
D_FF = 192              # -> GLU width 2 * 192 // 3 = 128
DEV = "cuda"
BF16 = torch.bfloat16


def _case(kind, tokens, **kw):
    """A case with the model's shape and default options; skew is the spread of the per-expert
    routing bias (0: uniform, 0.27: expert loads with CV ~ 1, 1.5: half of the experts idle)."""
    c = dict(kind=kind, tokens=tokens, d_model=576, experts=76, top_k=6, shared=2, layers=1,
             skew=0.0, activation="silu", bias=False, capacity=0.0, combine="default")
    c.update(kw)
    return c


def listed():
    return [
        # one sequence being generated: the smallest call there is, twenty layers of one token
        dict(name="decode 1 token x 20 layers", **_case("decode", 1, layers=20)),
        # a serving batch of 64 sequences
        dict(name="decode 64 tokens x 20 layers", **_case("decode", 64, layers=20)),
        # the prompt of one request, eager, of no particular length
        dict(name="infer 333 tokens", **_case("infer", 333)),
        # prefill of 16 long contexts in one call: the largest forward
        dict(name="infer 131072 tokens", **_case("infer", 131072)),
        # the training step of the benchmark: 8 sequences of 2048, uneven expert loads
        dict(name="train 16384 tokens", **_case("train", 16384, skew=0.27)),
        # another model's block: wider, fewer experts, no shared ones; a ragged batch whose router
        # has collapsed onto half of the experts
        dict(name="train 3001 tokens, wide", **_case("train", 3001, d_model=768, experts=64,
                                                      top_k=4, shared=0, skew=1.5)),
        # a training step that has to reproduce bit for bit
        dict(name="train 4096 tokens, store", **_case("train", 4096, skew=0.27, combine="store")),
        # one sequence per micro-batch, replayed from graphs
        dict(name="graphed 2048 tokens", **_case("graphed", 2048, skew=0.27)),
        # the sublayer as the model's Block has it, at the benchmark's batch
        dict(name="sublayer 16384 tokens", **_case("sublayer", 16384, skew=0.27)),
        # experts with biases and GELU gates
        dict(name="train 4096 tokens, biases", **_case("train", 4096, activation="gelu",
                                                        bias=True)),
        # a fixed expert capacity
        dict(name="train 8000 tokens, capacity", **_case("train", 8000, skew=0.27, capacity=1.25)),
        # the optimizer's step on the expert stacks
        dict(name="muon 76 experts", **_case("muon", 1)),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread evenly over the logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["decode", "decode", "infer", "infer", "train", "train", "train", "graphed",
                       "sublayer", "muon"])
    shape = {}
    if rng.random() < 0.3:      # another model's block
        experts = rng.choice([8, 16, 32, 64, 128])
        shape = dict(d_model=rng.choice([256, 384, 512, 768, 1024]), experts=experts,
                     top_k=rng.choice([1, 2, 4, 8]), shared=rng.choice([0, 1, 2]))
    skew = rng.choice([0.0, 0.27, 0.27, 1.5])
    if kind == "decode":
        return _case(kind, _log_int(rng, 1, 256), layers=rng.choice([4, 8, 12, 20]), **shape)
    if kind == "infer":
        return _case(kind, _log_int(rng, 16, 49152), skew=skew, **shape)
    if kind == "muon":
        e = _log_int(rng, 4, 128)
        return _case(kind, 1, experts=e, d_model=rng.choice([384, 512, 576, 768]),
                     top_k=1, shared=rng.choice([0, 1, 2]))
    tokens = _log_int(rng, 64, 12288)
    if kind == "train":
        how = rng.random()
        if how < 0.25:
            return _case(kind, tokens, skew=skew, bias=True,
                         activation=rng.choice(["silu", "gelu"]), **shape)
        if how < 0.45:
            return _case(kind, tokens, skew=skew, capacity=rng.choice([1.0, 1.25, 2.0]), **shape)
        return _case(kind, tokens, skew=skew, combine=rng.choice(["default", "default", "store"]),
                     **shape)
    return _case(kind, tokens, skew=skew, **shape)


# ------------------------------------------------------------------------------------- prepare
def _block(case, gen, expert_std=None):
    """A bf16 block with fresh weights: router N(0, 0.02), experts N(0, 1 / sqrt(fan_in)) (or
    expert_std), biases N(0, 0.02)."""
    d, e = case["d_model"], case["experts"]
    with torch.device(DEV):
        m = MoEBlock(d, e, d_ff=D_FF, top_k=case["top_k"], n_shared=case["shared"],
                     capacity_factor=case["capacity"] or None, activation=case["activation"],
                     bias=case["bias"]).to(BF16)
    with torch.no_grad():
        for name, p in m.named_parameters():
            std = {"W_in": d ** -0.5, "W_sh_in": d ** -0.5, "W_out": D_HIDDEN ** -0.5,
                   "W_sh_out": D_HIDDEN ** -0.5}.get(name, 0.02)
            if expert_std is not None and name.startswith("W_"):
                std = expert_std
            p.copy_(torch.randn(p.shape, generator=gen, device=DEV) * std)
    if case["skew"]:
        m.router.logit_bias = torch.randn(e, generator=gen, device=DEV) * case["skew"]
    if case["combine"] != "default":
        m.combine_mode = case["combine"]
    return m


def prepare(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    kind, t, d = case["kind"], case["tokens"], case["d_model"]
    rows = lambda: torch.randn(t, d, generator=gen, device=DEV).to(BF16)
    if kind == "decode":
        # freshly initialised blocks (the constructor's std, 0.02): the residual stream keeps its
        # scale down the stack, as it does behind the norms of a model
        stack = StackedMoEDecoder([_block(case, gen, 0.02) for _ in range(case["layers"])])
        x = rows()
        stack.step(x)           # a server captures its batch shape once, before it serves
        return dict(kind=kind, stack=stack, x=x)
    if kind == "infer":
        return dict(kind=kind, block=_block(case, gen).eval(), x=rows())
    if kind == "muon":
        block = _block(case, gen)
        params = [p for n, p in block.named_parameters() if n.startswith("W_")]
        opt = Muon(params)
        for p in params:
            p.grad = (torch.randn(p.shape, generator=gen, device=DEV) * 1e-3).to(BF16)
        return dict(kind=kind, opt=opt, params=params)
    block = _block(case, gen).train()
    call = block
    if kind == "graphed":
        call = GraphedMoEBlock(block)
    elif kind == "sublayer":
        with torch.device(DEV):
            call = MoEFFNSublayer(block).to(BF16)
        with torch.no_grad():
            call.norm_gamma.add_(0.1 * torch.randn(d, generator=gen, device=DEV))
    s = dict(kind=kind, block=block, call=call, x=rows().requires_grad_(True), dout=rows(),
             params=dict(call.named_parameters()), one=torch.ones((), device=DEV))
    if kind == "graphed":
        run(s)                  # the capture, outside the training loop's steps
    return s


# ----------------------------------------------------------------------------------------- run
def run(s):
    kind = s["kind"]
    if kind == "decode":
        return s["stack"].step(s["x"])
    if kind == "infer":
        with torch.no_grad():
            return s["block"](s["x"])
    if kind == "muon":
        s["opt"].step()
        state = s["opt"].state
        return [p.detach() for p in s["params"]], [state[p]["momentum"] for p in s["params"]]
    # one step of a training loop: the gradient of what follows the block arrives as `dout`, the
    # balance loss joins the total loss with weight one
    s["x"].grad = None
    for p in s["params"].values():
        p.grad = None
    block = s["block"]
    if kind == "sublayer":
        out, aux = s["call"](s["x"])
    else:
        out = s["call"](s["x"])
        aux = s["call"].aux_loss
    torch.autograd.backward([out, aux], [s["dout"], s["one"].to(aux.dtype)])
    return dict(out=out.detach(), aux=aux.detach(), counts=block.expert_counts, dx=s["x"].grad,
                grads={n: p.grad for n, p in s["params"].items()})


# ------------------------------------------------------------------------------------ the work
def _expert_params(case, n):
    """Values in the weights (and biases) of n experts."""
    d = case["d_model"]
    return n * (3 * d * D_HIDDEN + ((2 * D_HIDDEN + d) if case["bias"] else 0))


def work(case):
    kind, t, d = case["kind"], case["tokens"], case["d_model"]
    e, k, sh = case["experts"], case["top_k"], case["shared"]
    if kind == "muon":
        n = (e + sh) * 3 * d * D_HIDDEN
        flops = 0
        for small, large in ((min(2 * D_HIDDEN, d), max(2 * D_HIDDEN, d)),
                             (min(D_HIDDEN, d), max(D_HIDDEN, d))):
            flops += (e + sh) * 5 * (4 * small * small * large + 2 * small ** 3)
        # weights and momentum read and written, gradients read
        return {"bytes": 2 * 5 * n, "flops": flops}
    router = d * e
    pairs = t * (k + sh)
    if case["capacity"]:
        pairs = t * sh + min(t * k, int(case["capacity"] * t * k))
    fwd = 2 * t * router + pairs * 6 * d * D_HIDDEN
    # the experts that t tokens reach, when each picks k of e at random
    reached = e * (1 - (1 - k / e) ** t) + sh
    if kind in ("decode", "infer"):
        weights = _expert_params(case, reached) + router
        return {"bytes": case["layers"] * 2 * weights + 4 * t * d, "flops": case["layers"] * fwd}
    weights = _expert_params(case, e + sh) + router
    # x, dout and the weights read; out, dx and the weights' gradients written
    return {"bytes": 2 * (4 * t * d + 2 * weights), "flops": 3 * fwd}


def tolerance(case):
    # bf16 results of sums in another order; the router's selection works on bf16 logits and is the
    # same in any correct implementation that forms them with fp32 accumulation in k order
    return {"rel": 1e-2}
