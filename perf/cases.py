"""The work this package is asked to do, as cases that can be timed and compared.

Four kinds, each through the public entry points a training program calls:

``orthogonalise``  ``NewtonSchulz(...).local(G, 5)`` on one matrix: trainers that
                   drive their own update, tensor-parallel owners, diagnostics.
                   Gram form (fp16 products) and direct form (bf16).
``update``         gradients arrive from backward, optional global-norm clip,
                   ``Muon.step()``: what one rank of a data-parallel job does for
                   the matrices it owns.  Dense decoder layers, expert matrices,
                   vision blocks; fp32 or bf16 momentum.
``train``          forward, backward, clip and step of a decoder wrapped with
                   ``dedicate_params`` and FSDP2, bf16 compute, fp32 masters.
``evaluate``       forward of the decoder to its logits without gradients.

Sizes are those of this repository's model configurations, benchmarks and tests
(widths 128 ... 4096, hidden sizes up to 14336, vocabularies 512 ... 128256,
sequences 128 ... 8192) and what lies between them; every matrix dimension is a
multiple of 8, which is what the matrix kernels take.
"""
import functools
import gc
import math

import torch
import torch.distributed as dist
import torch.nn as nn
from torch.distributed.device_mesh import init_device_mesh
from torch.distributed.fsdp import MixedPrecisionPolicy, fully_shard

import dmuon_b200 as dmuon
from dmuon_b200.models.llama import LlamaConfig, LlamaModel

#: a learning rate of the middle of a run; the update's RMS is 0.2 times this
_LR = 2e-3
_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}


# ---------------------------------------------------------------------------- cases
def listed():
    return [
        # one small matrix (MLP of the 256-wide decoder): a call of a few microseconds of arithmetic
        _orthogonalise("ns_256x1024", 256, 1024, "bf16"),
        # vision MLP of the 1152-wide tower: no dimension is a multiple of a tile; fp32 gradient
        _orthogonalise("ns_1152x4304", 1152, 4304, "fp32"),
        # tall down/up projection of the 4096-wide decoder: the largest single matrix
        _orthogonalise("ns_14336x4096", 14336, 4096, "bf16"),
        # direct formulation (`ns_backend="direct"`) on the 3072-wide decoder's MLP
        _orthogonalise("ns_direct_3072x8192", 3072, 8192, "bf16", backend="direct"),
        # every matrix of the 4-layer, 256-wide decoder: launches and host time decide
        _update("update_256_wide", width=256, kv=256, hidden=1024, layers=4),
        # one mixture-of-experts layer: 24 expert matrices of two shapes and the attention
        _update("update_experts", width=1024, kv=256, hidden=1408, layers=1, experts=8, clip=1.0),
        # vision blocks with ragged sizes, bf16 momentum
        _update("update_vision", width=1152, kv=1152, hidden=4304, layers=4, gated=False, momentum="bf16"),
        # what one of eight ranks owns of the 32-layer, 4096-wide decoder, global-norm clip
        _update("update_4096_wide", width=4096, kv=1024, hidden=14336, layers=4, clip=1.0),
        # the 256-wide decoder as the smallest run there is: 4 x 128 tokens
        _train("train_256_wide", width=256, heads=4, kv_heads=4, hidden=1024, layers=4, vocab=1024, batch=4, seq=128,
               tied=True),
        # a 1024-wide decoder, 2 x 1024 tokens, clipped
        _train("train_1024_wide", width=1024, heads=8, kv_heads=4, hidden=4096, layers=4, vocab=32000, batch=2,
               seq=1024, clip=1.0),
        # two layers of the 4096-wide decoder with its embedding and loss, 8192 tokens, clipped
        _train("train_4096_wide", width=4096, heads=32, kv_heads=8, hidden=14336, layers=2, vocab=128256, batch=1,
               seq=8192, clip=1.0),
        # scoring: logits of a few layers of the 3072-wide decoder
        _evaluate("evaluate_3072_wide", width=3072, heads=24, kv_heads=8, hidden=8192, layers=4, vocab=128256,
                  batch=1, seq=2048),
    ]


def _orthogonalise(name, rows, cols, dtype, backend="gram"):
    return dict(name=name, kind="orthogonalise", rows=rows, cols=cols, dtype=dtype, backend=backend)


def _update(name, width, kv, hidden, layers, experts=0, gated=True, momentum="fp32", clip=0.0):
    return dict(name=name, kind="update", width=width, kv=kv, hidden=hidden, layers=layers, experts=experts,
                gated=gated, momentum=momentum, clip=clip)


def _train(name, width, heads, kv_heads, hidden, layers, vocab, batch, seq, tied=False, clip=0.0):
    return dict(name=name, kind="train", width=width, heads=heads, kv_heads=kv_heads, hidden=hidden, layers=layers,
                vocab=vocab, batch=batch, seq=seq, tied=tied, clip=clip)


def _evaluate(name, width, heads, kv_heads, hidden, layers, vocab, batch, seq):
    return dict(name=name, kind="evaluate", width=width, heads=heads, kv_heads=kv_heads, hidden=hidden, layers=layers,
                vocab=vocab, batch=batch, seq=seq)


def _spread(rng, lo, hi, step=8):
    """A multiple of ``step`` between ``lo`` and ``hi``, even over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def _decoder_sizes(rng, top_width):
    head_dim = rng.choice((64, 128)) if top_width > 512 else 64
    kv_heads = rng.choice((1, 2, 4, 8) if top_width > 512 else (1, 2, 4))
    width = _spread(rng, 128, top_width)
    heads = kv_heads * max(1, width // (head_dim * kv_heads))
    return dict(width=width, heads=heads, kv_heads=kv_heads, head_dim=head_dim,
                hidden=_spread(rng, 2 * width, min(14336, 4 * width)))


def draw(rng):
    kind = rng.choice(("orthogonalise", "orthogonalise", "update", "update", "train", "evaluate"))
    if kind == "orthogonalise":
        c = _orthogonalise("", _spread(rng, 128, 14336), _spread(rng, 128, 4096), rng.choice(("bf16", "fp32")),
                           rng.choice(("gram", "gram", "gram", "direct")))
        if rng.random() < 0.5:
            c["rows"], c["cols"] = c["cols"], c["rows"]
    elif kind == "update":
        width = _spread(rng, 128, 4096)
        layers = rng.randint(1, 4)
        experts = rng.choice((0, 0, 0, rng.randint(2, 8)))
        c = _update("", width, width // rng.choice((1, 2, 4)) // 8 * 8, _spread(rng, width, min(14336, 4 * width)),
                    1 if experts else layers, experts, experts > 0 or rng.random() < 0.7,
                    rng.choice(("fp32", "fp32", "bf16")), rng.choice((0.0, 1.0)))
    else:
        large = rng.random() < 0.6
        c = _decoder_sizes(rng, 3072 if large else 512)
        seq = _spread(rng, 128, 4096 if large else 512, 1)
        c.update(kind=kind, layers=rng.randint(2, 4), vocab=_spread(rng, 512, 64000 if large else 4096, rng.choice((1, 8, 64))),
                 seq=seq, batch=max(1, min(4, 4096 // seq)))
        if kind == "train":
            c.update(tied=rng.random() < 0.3, clip=rng.choice((0.0, 1.0)))
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _mesh():
    """A data-parallel mesh of this one GPU."""
    dev = torch.device("cuda", torch.cuda.current_device())
    if not dist.is_initialized():
        dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=dev)
    return init_device_mesh("cuda", (1,), mesh_dim_names=("dp",))


def _is_matrix(name, p):
    return "proj" in name and p.ndim == 2


def _gradient(shape, gen, dtype):
    """What a weight gradient looks like early in training: a few strong directions over a noise floor."""
    dev = gen.device
    rows, cols = shape
    r = min(16, rows, cols)
    strength = torch.logspace(0, -1.5, r, device=dev)
    g = torch.randn(rows, cols, generator=gen, device=dev)
    g.addmm_(torch.randn(rows, r, generator=gen, device=dev) * strength, torch.randn(r, cols, generator=gen, device=dev))
    return g.mul_(1e-3).to(dtype)


class _GivenGradients(torch.autograd.Function):
    """Backward hands every weight the gradient of this pass, without a forward of its own."""

    @staticmethod
    def forward(ctx, x, grads, *weights):
        ctx.grads = grads
        return x.clone()

    @staticmethod
    def backward(ctx, g):
        return (g, None, *ctx.grads)


class _Matrices(nn.Module):
    """The matrices of one layer under the names the models use."""

    def __init__(self, shapes):
        super().__init__()
        self.mats = nn.ModuleDict({n: nn.Linear(cols, rows, bias=False) for n, (rows, cols) in shapes.items()})

    def forward(self, x, grads):
        return _GivenGradients.apply(x, grads, *(m.weight for m in self.mats.values()))


class _Stack(nn.Module):
    def __init__(self, layers, shapes):
        super().__init__()
        self.layers = nn.ModuleList(_Matrices(shapes) for _ in range(layers))

    def forward(self, grads):
        x = torch.zeros((), device="cuda")
        for layer, g in zip(self.layers, grads):
            x = layer(x, g)
        return x


def _layer_shapes(c):
    w, kv, h = c["width"], c["kv"], c["hidden"]
    shapes = {"q_proj": (w, w), "k_proj": (kv, w), "v_proj": (kv, w), "o_proj": (w, w)}
    for e in range(max(1, c["experts"])):
        tag = "expert%d_" % e if c["experts"] else ""
        if c["gated"]:
            shapes[tag + "gate_proj"] = (h, w)
        shapes[tag + "up_proj"] = (h, w)
        shapes[tag + "down_proj"] = (w, h)
    return shapes


def _decoder(c):
    return LlamaConfig(
        vocab_size=c["vocab"], d_model=c["width"], n_layers=c["layers"], n_heads=c["heads"], n_kv_heads=c["kv_heads"],
        head_dim=c.get("head_dim", c["width"] // c["heads"]), ffn_hidden=c["hidden"], tie_embeddings=c.get("tied", False))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    if case["kind"] == "orthogonalise":
        return dict(kind=case["kind"], grad=_gradient((case["rows"], case["cols"]), gen, _DTYPES[case["dtype"]]),
                    ns=dmuon.NewtonSchulz(backend=case["backend"]))
    gc.collect()            # models of earlier cases are cycles of modules and hooks
    torch.manual_seed(seed)
    if case["kind"] == "update":
        shapes = _layer_shapes(case)
        with torch.device(dev):
            model = _Stack(case["layers"], shapes)
        with torch.no_grad():
            for p in model.parameters():
                p.normal_(0.0, 0.02, generator=gen)
        policy = None
        if case["momentum"] == "bf16":
            policy = {"defaults": {"param_dtype": "bf16", "optim_dtype": "bf16"}}
        dmuon.dedicate_params(model, _mesh(), _is_matrix, compute_dtype=None if policy else torch.bfloat16,
                              reshard_after_forward=False, param_policy=policy)
        grads = [[_gradient(s, gen, torch.bfloat16) for s in shapes.values()] for _ in range(case["layers"])]
        opt = dmuon.Muon(model, lr=_LR, weight_decay=0.1, first_step_progress_log=False)
        owned = dmuon.get_owned_params(model)
        return dict(kind=case["kind"], model=model, opt=opt, clip=case["clip"], grads=grads, owned=owned,
                    weights=[dp._owned_data for dp in owned])
    with torch.device(dev):
        model = LlamaModel(_decoder(case))
    ids = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), generator=gen, device=dev)
    if case["kind"] == "evaluate":
        return dict(kind=case["kind"], model=model.to(torch.bfloat16).eval(), ids=ids[:, :-1].contiguous())
    mesh, mp = _mesh(), MixedPrecisionPolicy(param_dtype=torch.bfloat16, reduce_dtype=torch.bfloat16)
    dmuon.dedicate_params(model, mesh, _is_matrix, compute_dtype=torch.bfloat16, reshard_after_forward=False)
    for layer in model.layers:
        fully_shard(layer, mesh=mesh, mp_policy=mp)
    fully_shard(model, mesh=mesh, mp_policy=mp)
    opt = dmuon.Muon(model, lr=_LR, adamw_lr=_LR, weight_decay=0.1, first_step_progress_log=False)
    weights = [dp._owned_data for dp in dmuon.get_owned_params(model)]
    weights += [p.detach().to_local() for p in model.parameters() if hasattr(p, "to_local")]
    return dict(kind=case["kind"], model=model, opt=opt, clip=case["clip"], ids=ids, weights=weights)


# ---------------------------------------------------------------------------- one pass
def run(state):
    if state["kind"] == "orthogonalise":
        return state["ns"].local(state["grad"], 5)
    if state["kind"] == "evaluate":
        with torch.no_grad():
            return state["model"](state["ids"])
    model, opt = state["model"], state["opt"]
    opt.zero_grad()
    if state["kind"] == "update":
        loss = model(state["grads"])
    else:
        ids = state["ids"]
        loss = model(ids[:, :-1], labels=ids[:, 1:])
    loss.backward()
    out = [loss.detach()] if state["kind"] == "train" else []
    if state["clip"] > 0:
        out.append(dmuon.clip_grad_norm_(opt, state["clip"]).total_norm)
    opt.step()
    if state["kind"] == "update":
        out += [opt.state[id(dp)]["momentum_buffer"] for dp in state["owned"]]
    return out + state["weights"]


# ---------------------------------------------------------------------------- the same results in 64 bits
#: step triples of the iteration (Polar Express, arXiv 2505.16932, with a safety factor of 1.05)
_TRIPLES = [(a / 1.05, b / 1.05**3, c / 1.05**5) for a, b, c in (
    (8.28721201814563, -23.595886519098837, 17.300387312530933),
    (4.107059111542203, -2.9478499167379106, 0.5448431082926601),
    (3.9486908534822946, -2.908902115962949, 0.5518191394370137),
    (3.3184196573706015, -2.488488024314874, 0.51004894012372),
    (2.300652019954817, -1.6689039845747493, 0.4188073119525673))]


def _exact_newton_schulz(g):
    x = g.double()
    tall = x.shape[0] > x.shape[1]
    x = x.T if tall else x
    x = x / (x.norm() + 1e-7)
    for a, b, c in _TRIPLES:
        r = x @ x.T
        x = a * x + (b * r + c * (r @ r)) @ x
    return x.T if tall else x


def _exact_muon(weight, grad):
    """First step: momentum 0.95 with Nesterov, decoupled decay 0.1, update RMS 0.2."""
    step = _exact_newton_schulz(1.95 * grad) * (_LR * 0.2 * math.sqrt(max(grad.shape)))
    return weight.double() * (1 - _LR * 0.1) - step


def _exact_adamw(weight, grad):
    """First step: the bias-corrected averages are the gradient and its square; decay 0.01."""
    return weight * (1 - _LR * 0.01) - _LR * grad / (grad.abs() + 1e-8)


def _exact_decoder(cfg, p, ids):
    """The decoder on a dictionary of parameters: pre-RMSNorm, rotate-half positions, grouped-query attention, SwiGLU."""
    def norm(x, w):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + cfg.norm_eps) * w

    b, s = ids.shape
    d, kv = cfg.head_dim, cfg.n_kv_heads
    inv = cfg.rope_theta ** (-torch.arange(0, d, 2, device=ids.device).double() / d)
    angle = torch.outer(torch.arange(s, device=ids.device).double(), inv)
    cos, sin = angle.cos(), angle.sin()
    later = torch.ones(s, s, dtype=torch.bool, device=ids.device).triu(1)

    def heads(x, rotate):
        x = x.view(b, s, -1, d).transpose(1, 2)
        if rotate:
            x1, x2 = x.chunk(2, -1)
            x = torch.cat((x1 * cos - x2 * sin, x2 * cos + x1 * sin), -1)
        return x

    x = p["embed_tokens.weight"][ids]
    for i in range(cfg.n_layers):
        w = {n: p["layers.%d.%s.weight" % (i, n)] for n in (
            "input_layernorm", "self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj",
            "post_attention_layernorm", "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj")}
        h = norm(x, w["input_layernorm"])
        q = heads(h @ w["self_attn.q_proj"].T, True)
        k = heads(h @ w["self_attn.k_proj"].T, True)
        v = heads(h @ w["self_attn.v_proj"].T, False)
        o = []
        for j in range(q.shape[1]):             # one head at a time: the scores are the large ones
            g = j // (q.shape[1] // kv)
            scores = (q[:, j] @ k[:, g].transpose(1, 2) / math.sqrt(d)).masked_fill(later, -math.inf)
            o.append(scores.softmax(-1) @ v[:, g])
        x = x + torch.cat(o, -1) @ w["self_attn.o_proj"].T
        h = norm(x, w["post_attention_layernorm"])
        x = x + (nn.functional.silu(h @ w["mlp.gate_proj"].T) * (h @ w["mlp.up_proj"].T)) @ w["mlp.down_proj"].T
    x = norm(x, p["norm.weight"])
    return x @ p.get("lm_head.weight", p["embed_tokens.weight"]).T


def exact(case, seed):
    tokens = case.get("batch", 0) * case.get("seq", 0)
    if case["kind"] == "train" and tokens * case["vocab"] > 1.4e8:
        return None                             # logits, their gradient and the scores of every layer at 8 bytes
    state = prepare(case, seed)
    if case["kind"] == "orthogonalise":
        return _exact_newton_schulz(state["grad"])
    if case["kind"] == "evaluate":
        weights = {n: w.detach().double() for n, w in state["model"].named_parameters()}
        with torch.no_grad():
            return _exact_decoder(_decoder(case), weights, state["ids"])
    if case["kind"] == "update":
        grads = {"layers.%d.mats.%s.weight" % (i, n): g for i, layer in enumerate(state["grads"])
                 for n, g in zip(_layer_shapes(case), layer)}
        order = [dp.fqn for dp in state["owned"]]
        plain, out = [], []
    else:
        owned = dmuon.get_owned_params(state["model"])
        order = [dp.fqn for dp in owned]
        plain = [n for n, p in state["model"].named_parameters() if hasattr(p, "to_local")]
        leaves = {n: w.double().view(dp._orig_size).requires_grad_() for n, dp, w in zip(order, owned, state["weights"])}
        leaves.update((n, w.double().requires_grad_()) for n, w in zip(plain, state["weights"][len(owned):]))
        ids = state["ids"]
        logits = _exact_decoder(_decoder(case), leaves, ids[:, :-1])
        loss = nn.functional.cross_entropy(logits.flatten(0, 1), ids[:, 1:].flatten())
        grads = dict(zip(leaves, torch.autograd.grad(loss, list(leaves.values()))))
        out = [loss.detach()]
    coef = 1.0
    if case["clip"] > 0:
        total = torch.stack([grads[n].double().norm() for n in order]).norm()
        coef = torch.clamp(case["clip"] / (total + 1e-6), max=1.0)
        out.append(total)
    with torch.no_grad():
        if case["kind"] == "update":
            out += [grads[n].double() * coef for n in order]        # momentum after its first step
        out += [_exact_muon(w.view(grads[n].shape), grads[n].double() * coef) for n, w in zip(order, state["weights"])]
        out += [_exact_adamw(w.double(), grads[n]) for n, w in zip(plain, state["weights"][len(order):])]
    return out


# ---------------------------------------------------------------------------- what a pass cannot do without
def _newton_schulz_flops(rows, cols, backend="gram"):
    """Five steps; a symmetric product counts half."""
    m, n = min(rows, cols), max(rows, cols)
    if backend == "direct":
        return 5.0 * (m * m * n + m**3 + 2.0 * m * m * n)
    return 14.0 * m**3 + 2 * (1.0 * m * m * n) + 2 * (2.0 * m * m * n)


def work(case):
    if case["kind"] == "orthogonalise":
        size = case["rows"] * case["cols"]
        return dict(bytes=2.0 * size * _DTYPES[case["dtype"]].itemsize,
                    flops=_newton_schulz_flops(case["rows"], case["cols"], case["backend"]))
    if case["kind"] == "update":
        shapes = list(_layer_shapes(case).values()) * case["layers"]
        size = float(sum(r * k for r, k in shapes))
        # gradient in; momentum and fp32 weight in and out; bf16 weight out
        return dict(bytes=size * (2 + 2 * _DTYPES[case["momentum"]].itemsize + 8 + 2),
                    flops=sum(_newton_schulz_flops(r, k) for r, k in shapes))
    cfg = _decoder(case)
    tokens, w = case["batch"] * case["seq"], case["width"]
    q, kv = cfg.n_heads * cfg.head_dim, cfg.n_kv_heads * cfg.head_dim
    shapes = [(q, w), (kv, w), (kv, w), (w, q), (case["hidden"], w), (case["hidden"], w), (w, case["hidden"])]
    matrices = float(cfg.n_layers * sum(r * k for r, k in shapes))
    table = float(case["vocab"] * w)
    attention = 2.0 * cfg.n_layers * q * case["seq"] * tokens          # two causal products
    forward = 2.0 * tokens * (matrices + table) + attention
    # between layers the residual stream and the gated product have to exist
    stream = 2.0 * tokens * cfg.n_layers * (4 * w + 2 * q + 2 * kv + 3 * case["hidden"])
    if case["kind"] == "evaluate":
        return dict(bytes=2.0 * (matrices + table) + stream + 2.0 * tokens * case["vocab"], flops=forward)
    tables = table if case["tied"] else 2 * table
    return dict(bytes=matrices * 20 + tables * 28 + 3 * stream + 6.0 * tokens * case["vocab"],
                flops=3.0 * forward + cfg.n_layers * sum(_newton_schulz_flops(r, k) for r, k in shapes))


def tolerance(case):
    """About four times the largest difference seen, over the listed cases and fourteen drawn ones, between the
    kernels and other correct forms of the same computation: the iteration in fp32 and with PyTorch's products, the
    models with plain PyTorch operators and with another attention kernel, one to three passes on one state."""
    if case["kind"] == "orthogonalise":
        # fp16 products: 0.0045 / 0.061; bf16 products: 0.0094 / 0.061
        return {"rel": 0.016, "max": 0.2} if case["backend"] == "gram" else {"rel": 0.03, "max": 0.25}
    if case["kind"] == "update":
        # 0.0032 / 0.025: one pass moves a weight by about 0.02 of its size
        return {"rel": 0.012, "max": 0.1}
    if case["kind"] == "evaluate":
        # 0.02 / 0.12: bf16 activations through up to four layers
        return {"rel": 0.03, "max": 0.4}
    # 0.01 / 0.59: AdamW turns the sign of a gradient near zero into a full-size step
    return {"rel": 0.03, "max": 0.9}
