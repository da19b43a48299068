"""The specialised full-rank kernels at the edges of their blocks: every pair of formats they cover (AL8 / AL16
second moments, UF8 / UF4 / no momentum), each type of parameter and gradient, tensors of one element, of one
element less and more than a momentum block and a second-moment block, and of several blocks with a tail."""
import numpy as np
import pytest
import torch

import parity
from oracle_runner import OracleRun
from test_fullrank_gpu import compare_state, state_np, to_cuda_grad

pytestmark = pytest.mark.gpu

SHAPES = [(1,), (255,), (257,), (2047,), (2048,), (2049,), (5 * 2048 + 300,), (33, 640)]
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}
# (momentum, second moment, parameter, gradient, stochastic rounding, what else)
FORMATS = [(m, v, "f32", g, False, {}) for m in ("uf8", "uf4", None) for v in ("al8", "al16") for g in ("f32", "bf16")]
FORMATS += [(m, v, "bf16", "bf16", sr, {}) for m, v in (("uf8", "al8"), ("uf4", "al16"), (None, "al8")) for sr in (False, True)]
# the general forms of the EMAs (weights of 0.5 and more), a negated gradient
FORMATS += [("uf8", "al8", "f32", "bf16", False, dict(beta1=0.4)), ("uf4", "al16", "f32", "f32", False, dict(beta2=0.45, maximize=True)),
            (None, "al8", "bf16", "bf16", True, dict(beta2=0.3)), ("uf8", "al16", "f32", "bf16", False, dict(maximize=True))]


@pytest.mark.parametrize("m,v,param,grad,sr,extra", FORMATS)
def test_block_edges_match_oracle(m, v, param, grad, sr, extra, oracle):
    from adafactor8bit import Adafactor8Bit
    hp = dict(beta1=0.9, beta2=0.999, beta2_decay=None, factored=False, relative_step=False, scale_parameter=False,
              scale_weight_decay=False, d=0.0, eps=(1e-8, 1e-3), lr=1e-3, weight_decay=0.01, block_size=2048, m_block_size=256,
              m_quant_type=m or "uf8", v_quant_type=v, min_8bit_size=1, enable_fira_for_adafactor=True,
              stochastic_round_writeback=sr)
    if m is None:
        hp["beta1"] = None
    hp.update(extra)
    case = dict(shapes=SHAPES, steps=3, seed=61, param_dtype=param, hp=hp,
                grad=dict(dist="rowscale", std=1e-3, zero_frac=0.01, dtype=grad, spike_step=2, spike_mult=100.0))
    run = OracleRun("block edges", case=case)
    params = [torch.nn.Parameter(torch.from_numpy(p.copy()).to(DTYPES[param]).cuda()) for p in run.params0]
    for p in params:
        p.grad_dtype = None
    opt = Adafactor8Bit(params, **hp)
    for t in range(1, case["steps"] + 1):
        for p, g in zip(params, run.grads[t]):
            p.grad = to_cuda_grad(g, p.shape)
        opt.step()
        run.step()
        torch.cuda.synchronize()
        for i, p in enumerate(params):
            what = f"{m}/{v} {param}/{grad} t{t} {tuple(p.shape)}"
            if param == "f32":
                compare_state(what, t, i, opt.state[p], run.states[i], p, run.params[i], strict=False)
            else:
                # u carries 3e-7 of itself from the hardware sqrt and reciprocal, so a parameter 3e-10: against a bf16 unit of
                # 2^-8 * 2e-2 = 8e-5 it lands on the neighbouring number on 4e-6 of the elements, at most 1e-4
                parity.assert_lowp_params(p.detach().float().cpu().numpy(), run.params[i], param, what, frac=1e-4)
                for key in ("variance_q", "m_q"):
                    if key in run.states[i]:
                        a, b = state_np(opt.state[p], key), np.asarray(run.states[i][key]).reshape(-1)
                        if key == "m_q" and m == "uf4":
                            a, b = parity.unpack_nibbles(a), parity.unpack_nibbles(b)
                        parity.assert_codes(a, b, what + " " + key, al16=b.dtype == np.uint16, zero_reserved=key != "m_q")
