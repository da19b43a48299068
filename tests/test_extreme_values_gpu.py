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
