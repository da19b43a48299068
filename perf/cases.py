"""The optimizer steps whose speed this repository watches.

A case is one `Adafactor8Bit.step()` over the parameters of a decoder-only transformer (or of one
matrix), resumed from a checkpoint, with the gradients of one backward pass in place.  Parameters,
gradients and each kind of state lie in one flat buffer per kind, as a data-parallel program keeps
them, and the tensors are views of these buffers on 512-byte boundaries, like allocations of their own.

Fields of a case:
  rule     adamw | rmsprop | adafactor | came | apollo
  hidden, mlp, kv, layers, vocab   sizes of the model; layers = 0: one mlp x hidden matrix
  experts  0, or the number of expert matrices stacked into each three-dimensional MLP tensor
  grad     f32 | bf16, dtype of the gradients
  param    f32 | bf16, dtype of the parameters; sr: bf16 parameters are rounded stochastically
  m, v     formats of the first and the second moment (m = none: the rule keeps no momentum)
  block    elements of a second-moment block
  limiter  the norm-growth limiter is on (full-rank and factored rules)
  rank     rank of the APOLLO projection, else 0
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "adafactor-8bit_b200"))

from adafactor8bit import Adafactor8Bit  # noqa: E402

_DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16}
_BYTES = {"f32": 4, "bf16": 2, "uf8": 1, "uf4": 0.5, "al8": 1, "al16": 2, "none": 0}
_ALIGN = 512
_MIN_QUANTISED = 4096          # tensors below this size keep binary32 states


def _case(rule, hidden, mlp, kv, layers, vocab=0, experts=0, grad="bf16", param="f32", sr=False, m="uf8", v="al8",
          block=2048, limiter=False, rank=0):
    return dict(rule=rule, hidden=hidden, mlp=mlp, kv=kv, layers=layers, vocab=vocab, experts=experts, grad=grad,
                param=param, sr=sr, m=m, v=v, block=block, limiter=limiter, rank=rank)


def listed():
    tiny = dict(hidden=2048, mlp=5632, kv=256)                       # the TinyLlama-1.1B layer
    return [
        # the smallest call: a toy model or a set of adapters, a hundred thousand parameters in 19 tensors
        dict(_case("adamw", 64, 176, 64, 2), name="adamw_toy"),
        # a small model of many small tensors with the rule that takes the most passes
        dict(_case("came", 512, 1376, 512, 8, vocab=8000, v="al16"), name="came_small"),
        # one large matrix, binary32 gradients: what a single weight costs
        dict(_case("adamw", 4096, 4096, 0, 0, grad="f32"), name="adamw_matrix"),
        # the headline step: TinyLlama-1.1B, AdamW UF8/AL8 with the limiter
        dict(_case("adamw", layers=22, vocab=32000, limiter=True, **tiny), name="adamw_fira_model"),
        # the same model trained in pure bf16 with stochastic rounding
        dict(_case("adamw", layers=22, vocab=32000, limiter=True, param="bf16", sr=True, **tiny), name="adamw_fira_bf16_sr"),
        # the other code widths: 4-bit momentum, 16-bit second moment
        dict(_case("adamw", layers=4, m="uf4", v="al16", **tiny), name="adamw_uf4_al16"),
        # no momentum, binary32 gradients (no autocast), a middle-sized model
        dict(_case("rmsprop", 1024, 2816, 1024, 6, vocab=16000, grad="f32", m="none"), name="rmsprop_f32"),
        # factored Adafactor with the constructor's defaults
        dict(_case("adafactor", layers=22, vocab=32000, m="none", block=256, **tiny), name="adafactor_model"),
        # the same with a momentum on a model whose sizes fit no tile
        dict(_case("adafactor", 1001, 2731, 1001, 4, vocab=5003, block=256), name="adafactor_ragged"),
        # mixture of experts: the MLP weights are stacks of matrices
        dict(_case("adafactor", 2048, 1408, 256, 2, experts=8, m="none", block=256), name="adafactor_experts"),
        # Llama-2-7B layers with CAME
        dict(_case("came", 4096, 11008, 4096, 4, v="al16"), name="came_layers"),
        # Llama-3-8B layers with APOLLO, vectors on the AdamW-style fallback
        dict(_case("apollo", 4096, 14336, 1024, 4, rank=256), name="apollo_layers"),
    ]


def draw(rng):
    """A case of the same ranges: models from a toy to 1.1 billion parameters."""
    while True:
        rule = rng.choice(("adamw", "adamw", "rmsprop", "adafactor", "adafactor", "came", "apollo"))
        low = 512 if rule == "apollo" else 64
        hidden = int(round(math.exp(rng.uniform(math.log(low), math.log(4096)))))
        mlp = int(hidden * rng.uniform(2.0, 3.6))
        step = 64 if rule == "apollo" else rng.choice((1, 8, 8, 64))      # odd sizes, rounded ones, tiles
        hidden, mlp = max(hidden // step, 1) * step, max(mlp // step, 1) * step
        kv = hidden // rng.choice((1, 4, 8)) if hidden % 64 == 0 else hidden
        layers = int(round(math.exp(rng.uniform(0.0, math.log(24)))))
        vocab = rng.choice((0, rng.randrange(1000, 32001)))
        c = _case(rule, hidden, mlp, kv, layers, vocab, grad=rng.choice(("bf16", "bf16", "f32")))
        if rule == "apollo":
            c["grad"] = "bf16"
            c["rank"] = rng.choice((64, 128, 256))
            if kv < c["rank"]:
                c["kv"] = hidden
        if rule in ("adafactor", "came"):
            c["experts"] = rng.choice((0, 0, rng.randrange(2, 17)))
        if rule in ("adamw", "adafactor") and rng.random() < 0.3:
            c["param"], c["grad"], c["sr"] = "bf16", "bf16", rng.random() < 0.5
        if rule == "adamw":
            c["m"] = rng.choice(("uf8", "uf8", "uf4"))
            c["limiter"] = rng.random() < 0.5
        elif rule == "rmsprop" or (rule == "adafactor" and rng.random() < 0.5):
            c["m"] = "none"
        if rule in ("adamw", "rmsprop", "came"):
            c["v"] = rng.choice(("al8", "al8", "al16"))
        if rule == "adafactor":
            c["block"] = rng.choice((256, 2048))
        n = sum(math.prod(s) for _, s in _shapes(c))
        if n <= (600_000_000 if rule in ("came", "apollo") else 1_000_000_000):
            return c


def _shapes(c):
    """(role, shape) of every parameter tensor."""
    h, mlp, kv, ex = c["hidden"], c["mlp"], c["kv"], c["experts"]
    if c["layers"] == 0:
        return [("matrix", (mlp, h))]
    stack = (ex,) if ex else ()
    out = [("embed", (c["vocab"], h))] if c["vocab"] else []
    for _ in range(c["layers"]):
        out += [("matrix", (h, h)), ("matrix", (kv, h)), ("matrix", (kv, h)), ("matrix", (h, h)),
                ("matrix", stack + (mlp, h)), ("matrix", stack + (mlp, h)), ("matrix", stack + (h, mlp)),
                ("norm", (h,)), ("norm", (h,))]
    out.append(("norm", (h,)))
    return out + ([("head", (c["vocab"], h))] if c["vocab"] else [])


def _options(c):
    plain = dict(beta2_decay=None, relative_step=False, scale_parameter=False, scale_weight_decay=False)
    o = dict(block_size=c["block"], v_quant_type=c["v"], enable_fira_for_adafactor=c["limiter"],
             stochastic_round_writeback=c["sr"])
    if c["m"] != "none":
        o.update(beta1=0.9, m_quant_type=c["m"], m_block_size=256)
    if c["rule"] == "adamw":
        o.update(plain, beta2=0.999, factored=False, d=0.0, eps=(1e-8, 1e-3), lr=1e-3, weight_decay=0.01)
    elif c["rule"] == "rmsprop":
        o.update(plain, beta2=0.99, factored=False, d=0.0, eps=(1e-8, 1e-3), lr=1e-3)
    elif c["rule"] == "came":
        o.update(plain, beta2=0.999, beta3=0.9999, factored=True, d=1.0, eps_came=1e-16, lr=1e-4, c_quant_type=c["v"])
    elif c["rule"] == "apollo":
        o.update(plain, beta2=0.999, factored=False, d=0.0, eps=(1e-6, 1e-3), lr=1e-3, weight_decay=0.01,
                 apollo_rank=c["rank"], apollo_update_proj_gap=200, apollo_eps=1e-6, apollo_cache_proj=True,
                 enable_fira_for_apollo=True)
    return o                                             # adafactor: the constructor's defaults


def _flat(shapes, dtype):
    """A zeroed buffer and a view of it for every shape."""
    per = _ALIGN // torch.empty(0, dtype=dtype).element_size()
    offs, total = [], 0
    for s in shapes:
        offs.append(total)
        total += -(-math.prod(s) // per) * per
    buf = torch.zeros(total, dtype=dtype, device="cuda")
    return buf, [buf[o:o + math.prod(s)].view(s) for o, s in zip(offs, shapes)]


def _fill_grads(views, gen):
    """Heavy-tailed gradients: N(0, 1e-3) with a lognormal scale per row, half a per cent exact zeros."""
    for v in views:
        g = torch.randn(v.shape, generator=gen, device="cuda") * 1e-3
        rows = torch.randn(v.shape[:-1] + (1,), generator=gen, device="cuda")
        g.mul_(rows.exp_())
        g.masked_fill_(torch.rand(v.shape, generator=gen, device="cuda") < 0.005, 0.0)
        v.copy_(g)


def _optimizer(c, roles, params):
    if c["rule"] != "apollo":
        return Adafactor8Bit(params, **_options(c))
    groups = [dict(params=[p for r, p in zip(roles, params) if r == "matrix"])]
    rest = [p for r, p in zip(roles, params) if r != "matrix"]
    return Adafactor8Bit(groups + ([dict(params=rest, apollo_rank=0)] if rest else []), **_options(c))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    roles = [r for r, _ in _shapes(case)]
    shapes = [s for _, s in _shapes(case)]
    flat_p, views = _flat(shapes, _DTYPE[case["param"]])
    for r, v in zip(roles, views):
        v.copy_(torch.randn(v.shape, generator=gen, device="cuda") * 0.02 + (1.0 if r == "norm" else 0.0))
    params = [torch.nn.Parameter(v) for v in views]
    _, grads = _flat(shapes, _DTYPE[case["grad"]])
    for p, g in zip(params, grads):
        p.grad_dtype = None                              # bf16 gradients on binary32 parameters
        p.grad = g
    _fill_grads(grads, gen)
    first = _optimizer(case, roles, params)
    first.step()
    # resume: every kind of state moves into a flat buffer of its own
    opt = _optimizer(case, roles, params)
    kinds = {}
    for p in params:
        for k, x in first.state[p].items():
            if isinstance(x, torch.Tensor):
                kinds.setdefault((k, x.dtype), []).append((p, x))
            else:
                opt.state[p][k] = x
    out = {"param": flat_p}
    for (k, dtype), owners in kinds.items():
        buf, state_views = _flat([tuple(x.shape) for _, x in owners], dtype)
        for (p, x), v in zip(owners, state_views):
            v.copy_(x)
            opt.state[p][k] = v
        if "proj" not in k:                              # (the projection matrix is an input of the step)
            out[k] = buf
    _fill_grads(grads, gen)
    opt.step()                                           # the program has been running
    _fill_grads(grads, gen)
    return {"opt": opt, "out": out}


def run(state):
    state["opt"].step()
    return state["out"]


def work(case):
    """Gradient read once, parameters and states read and written once; the projection's flops."""
    gb, pb = _BYTES[case["grad"]], _BYTES[case["param"]]
    mb, vb = _BYTES[case["m"]], _BYTES[case["v"]]
    total, flops = 0.0, 0.0
    for role, s in _shapes(case):
        n = math.prod(s)
        rows, cols = n // s[-1], s[-1]
        quant = n >= _MIN_QUANTISED
        m = 0 if case["m"] == "none" else (mb if quant else 4)
        v = vb if quant else 4
        total += n * (gb + 2 * pb)
        if case["rule"] == "apollo" and role == "matrix":
            total += 2 * max(s) * case["rank"] * (m + v) + 4 * case["rank"] * min(s)
            flops += 2.0 * case["rank"] * n
        elif case["rule"] in ("adafactor", "came") and len(s) >= 2:
            vectors = rows + (n // (s[-2] * cols)) * cols
            total += 2 * n * m + 2 * vectors * v * (2 if case["rule"] == "came" else 1)
        else:
            total += 2 * n * (m + v)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Codes come from binary32 arithmetic with one rounding per operation; another correct
    implementation may resolve a tie the other way on one element in 10^4 (in 10^3 for AL16, whose
    codes are 257 times finer).  A flipped momentum code moves u = m / sqrt(v) by up to 1/128 of the
    block's largest m (1/8 with UF4), so one parameter by lr * 0.03 = 3e-5 of a root mean square of
    2e-2 (5e-4 with UF4, whose ties are as rare); parameters differ by 1e-5 as a whole.  bf16 parameters:
    the neighbouring number, 2^-8, on such elements.
    The APOLLO projection is a sum of up to 14336 products in binary32, in any order: relative 2e-6
    of a typical element, so that a block's smallest square (a 2000th of that) carries 1e-2 and its
    logarithm, the block's min_log, 1e-4; the grid of codes moves with it."""
    if case["rule"] == "apollo":
        return {"rel": 3e-4, "max": 5e-2, "differ": 1e-2}
    t = {"rel": 1e-5, "max": 2e-3, "differ": 1e-4}
    if case["v"] == "al16":
        t["differ"] = 1e-3
    if case["m"] == "uf4":
        t["max"] = 3e-2
    if case["param"] == "bf16":
        t["rel"], t["max"] = 1e-4, 1e-2
    return t
