"""Second moments and gradients at the ends of binary32 in the specialised full-rank kernels."""
import numpy as np
import pytest
import torch

from oracle_runner import OracleRun
from test_fullrank_gpu import compare_state, make_optimizer, to_cuda_grad

pytestmark = pytest.mark.gpu

FORMATS = [(m, v) for m in ("uf8", "uf4", None) for v in ("al8", "al16")]


def options(m, v, **extra):
    hp = dict(beta1=0.9 if m else None, beta2=0.999, beta2_decay=None, factored=False, relative_step=False,
              scale_parameter=False, scale_weight_decay=False, d=0.0, lr=1e-3, weight_decay=0.01, block_size=2048,
              m_block_size=256, m_quant_type=m or "uf8", v_quant_type=v, min_8bit_size=1)
    hp.update(extra)
    return hp


@pytest.mark.parametrize("limiter", [False, True])
@pytest.mark.parametrize("m,v", FORMATS)
def test_subnormal_second_moments(m, v, limiter, oracle):
    """Gradients of 1e-22 .. 1e-16 with the constructor's eps of 1e-30: the new second moments are subnormal, and their
    square roots, not eps, are the denominators."""
    case = dict(shapes=[(5 * 2048 + 300,), (2049,)], steps=3, seed=67, hp=options(m, v, eps=(1e-30, 1e-3), enable_fira_for_adafactor=limiter),
                grad=dict(dist="normal", std=1e-3, zero_frac=0.0, dtype="f32"))
    run = OracleRun("subnormal", case=case)
    rng = np.random.default_rng(67)
    for t in range(1, case["steps"] + 1):
        run.grads[t] = [(10.0 ** rng.uniform(-22, -16, g.shape) * rng.choice((-1.0, 1.0), g.shape)).astype(np.float32)
                        for g in run.grads[t]]
    params, opt = make_optimizer(run)
    for t in range(1, case["steps"] + 1):
        for p, g in zip(params, run.grads[t]):
            p.grad = to_cuda_grad(g, p.shape)
        opt.step()
        run.step()
        torch.cuda.synchronize()
        for i, p in enumerate(params):
            compare_state(f"{m}/{v}", t, i, opt.state[p], run.states[i], p, run.params[i], strict=False)
            if limiter:
                a, b = float(opt.state[p]["fira_prev_norm"].item()), float(run.states[i]["fira_prev_norm"])
                assert abs(a - b) <= 2e-6 * abs(b), f"{m}/{v} t{t} p{i}: norm {a} against {b}"

KEYS = ("variance_q", "variance_scale", "variance_min_log", "m_q", "m_scale")


def bits(x):
    """The bytes of a tensor, every NaN as the same one."""
    a = x.detach().cpu().contiguous()
    if a.is_floating_point():
        a = torch.where(torch.isnan(a), torch.full_like(a, float("nan")), a)
        a = a.view(torch.int32 if a.element_size() == 4 else torch.int16)
    return a


def two_kernels(hp, shapes, steps, edit, seed=71):
    """Steps the same tensors twice, with gradients in binary32 (specialised kernels) and in fp16 (general kernel); edit(t, i, g)
    changes the fp16 gradient of tensor i in place.  -> ((parameters, optimizer), (parameters, optimizer))"""
    from adafactor8bit import Adafactor8Bit
    gen = torch.Generator().manual_seed(seed)
    start = [torch.randn(s, generator=gen) * 0.02 for s in shapes]
    grads = []
    for t in range(1, steps + 1):
        row = [(torch.randn(s, generator=gen) * 1e-2).half() for s in shapes]
        for i, g in enumerate(row):
            edit(t, i, g)
        grads.append(row)
    out = []
    for dtype in (torch.float32, torch.float16):
        params = [torch.nn.Parameter(x.clone().cuda()) for x in start]
        for p in params:
            p.grad_dtype = None
        opt = Adafactor8Bit(params, **hp)
        for row in grads:
            for p, g in zip(params, row):
                p.grad = g.cuda().to(dtype)
            opt.step()
        torch.cuda.synchronize()
        out.append((params, opt))
    return out


def assert_same_state(a, b, what):
    (pa, oa), (pb, ob) = a, b
    for i, (x, y) in enumerate(zip(pa, pb)):
        for key in KEYS:
            if key in ob.state[y]:
                s, r = bits(oa.state[x][key]), bits(ob.state[y][key])
                assert torch.equal(s, r), f"{what} p{i} {key}: {int((s != r).sum())} of {r.numel()} differ"


@pytest.mark.parametrize("limiter", [False, True])
@pytest.mark.parametrize("m,v", [f for f in FORMATS if f != ("uf8", "al8")])
def test_updates_are_the_general_kernels(m, v, limiter):
    """AL16, UF4 and momentum-free states: parameters and states bit for bit as the general kernel gives them.  With the limiter a
    tensor is one block with one gradient that is not zero, so that its norm is one element's update, whatever the order of the sum."""
    def edit(t, i, g):
        if limiter:
            keep = g[7 + i].clone()
            g.zero_()
            g[7 + i] = keep
    shapes = [(2048,)] * 6 if limiter else [(1 << 22,), (5 * 2048 + 300,), (2049,), (300,)]
    fast, general = two_kernels(options(m, v, eps=(1e-8, 1e-3), enable_fira_for_adafactor=limiter), shapes, 3, edit)
    assert_same_state(fast, general, f"{m}/{v}")
    for i, (x, y) in enumerate(zip(fast[0], general[0])):
        assert torch.equal(bits(x), bits(y)), f"{m}/{v} p{i}: {int((x != y).sum())} of {x.numel()} parameters differ"
        if limiter:
            assert torch.equal(fast[1].state[x]["fira_prev_norm"], general[1].state[y]["fira_prev_norm"])
@pytest.mark.parametrize("limiter", [False, True])
@pytest.mark.parametrize("m,v", [f for f in FORMATS if f != ("uf8", "al8")])
def test_infinities_and_nans(m, v, limiter):
    """Gradients with infinities and NaNs in whole blocks and tails: states as the general kernel leaves them."""
    def edit(t, i, g):
        if t == 2 and i < 3:
            g[5] = float("inf")
            g[300] = float("nan")
            g[-1] = -float("inf") if i == 0 else float("nan")
            if i == 1:
                g[2048:2048 + 2048] = float("inf")
            if i == 2:
                g[256:512] = float("nan")
    shapes = [(3 * 2048 + 300,), (3 * 2048 + 300,), (2048,), (2049,)]
    fast, general = two_kernels(options(m, v, eps=(1e-8, 1e-3), enable_fira_for_adafactor=limiter), shapes, 4, edit)
    assert_same_state(fast, general, f"{m}/{v}")
    for i, (x, y) in enumerate(zip(fast[0], general[0])):
        np.testing.assert_allclose(x.detach().cpu().numpy(), y.detach().cpu().numpy(), rtol=1e-5, atol=1e-8, equal_nan=True, err_msg=f"{m}/{v} p{i}")
        if limiter:
            a, b = float(fast[1].state[x]["fira_prev_norm"]), float(general[1].state[y]["fira_prev_norm"])
            # (binary32 sums of a block, at most 38 roundings deep on the two sides together, under a square root)
            assert abs(a - b) <= 19 * 2.0 ** -24 * abs(b), f"{m}/{v} p{i}: norm {a} against {b}"


@pytest.mark.parametrize("m,v", FORMATS)
def test_overflowing_second_moment(m, v, oracle):
    """A square beyond binary32 makes its block's scale infinite, so that the block decodes to NaN; the other blocks do not notice."""
    hp = options(m, v, eps=(1e-8, 1e-3))
    case = dict(shapes=[(3 * 2048,)], steps=2, seed=73, hp=hp, grad=dict(dist="normal", std=1e-3, zero_frac=0.0, dtype="f32"))
    run = OracleRun("overflow", case=case)
    run.grads[1][0][2048 + 9] = 1e25
    params, opt = make_optimizer(run)
    for t in (1, 2):
        params[0].grad = to_cuda_grad(run.grads[t][0], params[0].shape)
        opt.step()
        run.step()
        torch.cuda.synchronize()
        st = opt.state[params[0]]
        if t == 1:
            assert np.array_equal(st["variance_scale"].cpu().numpy(), run.states[0]["variance_scale"])
            assert np.isinf(run.states[0]["variance_scale"][1])
            assert (st["variance_q"][2048:4096] == 1).all()
    got, want = params[0].detach().cpu().numpy(), run.params[0]
    assert np.isnan(np.delete(want[2048:4096], 9)).all() and np.isfinite(want[:2048]).all()
    assert np.isnan(np.delete(got[2048:4096], 9)).all()
    np.testing.assert_allclose(np.delete(got, np.s_[2048:4096]), np.delete(want, np.s_[2048:4096]), rtol=1e-5, atol=1e-9)


def test_nan_in_a_tail_leaves_the_range(oracle):
    """UF8/AL8: the range of a tail block is that of the elements that are numbers."""
    hp = options("uf8", "al8", eps=(1e-8, 1e-3))
    case = dict(shapes=[(300,), (2048 + 300,)], steps=1, seed=79, hp=hp, grad=dict(dist="normal", std=1e-3, zero_frac=0.0, dtype="f32"))
    run = OracleRun("nan tail", case=case)
    for g in run.grads[1]:
        g[-5] = np.nan
    params, opt = make_optimizer(run)
    for p, g in zip(params, run.grads[1]):
        p.grad = to_cuda_grad(g, p.shape)
    opt.step()
    run.step()
    for p, st in zip(params, run.states):
        for key in ("variance_scale", "variance_min_log"):
            assert np.array_equal(opt.state[p][key].cpu().numpy(), st[key]), key


@pytest.mark.parametrize("m", ["uf8", "uf4", None])
def test_al16_codes_far_below_the_floor(m, oracle):
    """A block whose maximum lies just above the floor of 2^-126 and whose other values lie below it: hundreds of ranges below
    min_log, where the rounding constant no longer covers the quotient; their code is 1."""
    hp = options(m, "al16", eps=(1e-8, 1e-3))
    case = dict(shapes=[(2048,)], steps=1, seed=83, hp=hp, grad=dict(dist="normal", std=1e-3, zero_frac=0.0, dtype="f32"))
    run = OracleRun("below the floor", case=case)
    v = np.full(2048, 5e-39)
    v[::64] = 2.0 ** np.linspace(-126.2, -125.999, 32)
    run.grads[1][0][:] = np.sqrt(v / 0.001).astype(np.float32)
    params, opt = make_optimizer(run)
    params[0].grad = to_cuda_grad(run.grads[1][0], params[0].shape)
    opt.step()
    run.step()
    scale = float(run.states[0]["variance_scale"][0])
    assert 6e-4 < scale < 1.3e-3
    assert np.array_equal(opt.state[params[0]]["variance_q"].cpu().numpy().view(np.uint16), run.states[0]["variance_q"])
