"""Which launch tables the tensors of a group go to (no GPU needed)."""
import pytest
import torch

from adafactor8bit import Adafactor8Bit


def tensor(shape, shift=0):
    n = 1
    for s in shape:
        n *= s
    return torch.zeros(n + shift)[shift:].view(shape)


@pytest.mark.parametrize("batch,shift_p,shift_g,tables", [((4, 64, 64), 0, 0, 1), ((4, 64, 64), 1, 0, 2), ((4, 64, 64), 0, 1, 2),
                                                          ((4, 64, 60), 0, 0, 2), ((1, 64, 64), 0, 0, 2)])
def test_matrices_join_batches(batch, shift_p, shift_g, tables):
    """Momentum-free matrices share the table of batches that hold most of the elements, unless a batch lies off the 16-byte
    boundaries or some rows are no whole vectors."""
    opt = Adafactor8Bit([torch.nn.Parameter(tensor((96, 64)))])
    entries = [(0, tensor((96, 64)), tensor((96, 64)), {}), (1, tensor(batch, shift_p), tensor(batch, shift_g), {})]
    launches = opt._sort_group(opt.param_groups[0], entries)
    assert len(launches) == tables and sorted(e[0] for _, _, items in launches for e in items) == [0, 1]


@pytest.mark.parametrize("v,m,param,grad,mode,name", [
    ("al8", "uf8", "f32", "bf16", "apply", "fullrank_fast_apply"), ("al16", "uf4", "f32", "f32", "noclip", "fullrank_fast_noclip"),
    ("al8", None, "bf16", "bf16", "sumsq", "fullrank_stat"), ("al16", "uf8", "f32", "bf16", "lag", "fullrank_generic_lag"),
    ("al8", "d8", "f32", "bf16", "apply", "fullrank_generic_apply"), ("al8", "uf8", "f32", "f16", "apply", "fullrank_generic_apply"),
    ("fp32", "uf8", "f32", "f32", "sumsq", "fullrank_generic_sumsq")])
def test_kernel_names_follow_the_dispatch(v, m, param, grad, mode, name):
    from adafactor8bit import _engine as E, _native as N
    plan = object.__new__(E.FullrankPlan)
    plan.cfg = N.FullrankCfg(block=2048, m_block=256 if m else 0, v_fmt=N.V_FMT[v], m_fmt=N.M_FMT[m], use_adam_denom=1,
                             param_dtype=getattr(N, param.upper()), grad_dtype=getattr(N, grad.upper()))
    assert plan.kernel_name(getattr(N, "MODE_" + mode.upper())) == name


def test_scalars_of_a_launch_template_follow_every_step():
    """One value for the table, one per tensor, and the change from either to the other; unchanged values stay."""
    import numpy as np
    from adafactor8bit import _engine as E
    static, last = np.zeros((2, 3), dtype=[("alpha", np.float32), ("decay", np.float32)]), {}
    array = np.array([1.0, 2.0, 3.0], dtype=np.float32)
    for alpha, decay in [(0.5, array), (0.5, 0.25), (array, 0.25), (0.5, 0.25), (np.float32(0.1), float("nan")), (np.float32(0.1), 0.0), (0.0, array * 2)]:
        E._update_scalars(static, last, dict(alpha=alpha, decay=decay), ("alpha", "decay"))
        for k, v in (("alpha", alpha), ("decay", decay)):
            np.testing.assert_array_equal(static[k], np.broadcast_to(np.float32(v), (2, 3)), err_msg=k)
