"""Parity of the CUDA factored path (Adafactor, CAME) with the CPU oracle and the
reference's golden vectors, through the optimizer class."""
import numpy as np
import pytest
import torch

import cases
import parity
from oracle_runner import FACTORED_CASES, OracleRun, golden_entries, load_golden
from test_fullrank_gpu import make_optimizer, state_np, to_cuda_grad

pytestmark = pytest.mark.gpu

CODE_KEYS = ("row_var_q", "col_var_q", "conf_row_q", "conf_col_q", "variance_q", "m_q")
RANGE_KEYS = ("row_var_scale", "row_var_min_log", "col_var_scale", "col_var_min_log", "conf_row_scale",
              "conf_row_min_log", "conf_col_scale", "conf_col_min_log", "variance_scale", "variance_min_log", "m_scale")
F32_KEYS = ("row_var", "col_var", "conf_row", "conf_col", "variance", "m")


def compare(name, t, i, st_gpu, st_cpu, p_gpu, p_cpu, param_tol):
    for key in CODE_KEYS:
        if key in st_cpu:
            a, b = state_np(st_gpu, key), np.asarray(st_cpu[key]).reshape(-1)
            parity.assert_codes(a, b, f"{name} t{t} p{i} {key}", al16=(b.dtype == np.uint16),
                                zero_reserved=(key != "m_q"))
    for key in RANGE_KEYS:
        if key in st_cpu:
            parity.assert_ranges(state_np(st_gpu, key), st_cpu[key], f"{name} t{t} p{i} {key}", max_ulp=4)
    for key in F32_KEYS:
        if key in st_cpu:
            assert parity.rel_l2(state_np(st_gpu, key), st_cpu[key]) <= 1e-6, f"{name} t{t} p{i} {key}"
    parity.assert_params(p_gpu.detach().cpu().numpy(), p_cpu, f"{name} t{t} p{i} param", tol=param_tol)


# Cases without fixtures.  "odd": column counts that are not multiples of 8 take the
# element-wise kernels; "tiles": several statistic tiles per tensor with ragged edges and
# chunks that end inside a momentum block, through the 128-bit kernels.
EXTRA_CASES = {
    "adafactor_odd": dict(shapes=[(37, 131), (50, 100)], steps=3, seed=31, grad=cases.CASES["adafactor_factored"]["grad"],
                          hp=cases.CASES["adafactor_factored"]["hp"]),
    "adafactor_m_odd": dict(shapes=[(37, 131), (130, 273)], steps=3, seed=32, grad=cases.CASES["adafactor_factored_m"]["grad"],
                            hp=cases.CASES["adafactor_factored_m"]["hp"]),
    "came_odd": dict(shapes=[(33, 77), (129, 300)], steps=3, seed=33, grad=cases.CASES["came_al16"]["grad"],
                     hp=cases.CASES["came_al16"]["hp"]),
    "adafactor_tiles": dict(shapes=[(200, 520), (70, 264), (3, 8)], steps=3, seed=34,
                            grad=cases.CASES["adafactor_factored"]["grad"], hp=cases.CASES["adafactor_factored"]["hp"]),
    "adafactor_m_tiles": dict(shapes=[(200, 520), (70, 264), (3, 8)], steps=3, seed=35,
                              grad=cases.CASES["adafactor_factored_m"]["grad"], hp=cases.CASES["adafactor_factored_m"]["hp"]),
    "adafactor_m_uf4_tiles": dict(shapes=[(200, 520), (5, 24)], steps=3, seed=36,
                                  grad=cases.CASES["adafactor_factored_m"]["grad"],
                                  hp=dict(cases.CASES["adafactor_factored_m"]["hp"], m_quant_type="uf4")),
    "came_tiles": dict(shapes=[(200, 520), (70, 264), (3, 8)], steps=3, seed=37, grad=cases.CASES["came_al16"]["grad"],
                       hp=dict(cases.CASES["came_al16"]["hp"], block_size=256)),
}


# column counts that are multiples of 2048: the apply pass walks such tensors strip by strip
EXTRA_CASES.update({
    "adafactor_strips": dict(shapes=[(5, 2048), (70, 4096), (1, 2048), (33, 6144)], steps=3, seed=39,
                             grad=cases.CASES["adafactor_factored"]["grad"], hp=cases.CASES["adafactor_factored"]["hp"]),
    "adafactor_m_strips": dict(shapes=[(5, 2048), (70, 4096), (33, 6144)], steps=3, seed=40,
                               grad=cases.CASES["adafactor_factored_m"]["grad"], hp=cases.CASES["adafactor_factored_m"]["hp"]),
    "came_strips": dict(shapes=[(5, 2048), (70, 4096), (33, 6144)], steps=3, seed=41, grad=cases.CASES["came_al16"]["grad"],
                        hp=cases.CASES["came_al16"]["hp"]),
})

# rows of any length and batches of matrices through the 128-bit kernels: a row end inside a vector, the shortest
# rows (8, 9), a partial last vector, a partial last momentum block, several chunks, fp32 gradients, one matrix of the
# table with whole vectors; columns of a multiple of 256 in a batch (the write pass over the tiles).  (7, 5) and
# (3, 7): fewer than 8 columns take the whole table to the general kernels.
_ANY = [(9, 9), (5, 8), (131, 273), (700, 257), (64, 264)]
_ANY3 = [(3, 70, 40), (2, 33, 131), (2, 600, 72)]
_F32 = dict(cases.CASES["adafactor_factored"]["grad"], dtype="f32")
EXTRA_CASES.update({
    "adafactor_any": dict(shapes=_ANY, steps=3, seed=51, grad=cases.CASES["adafactor_factored"]["grad"],
                          hp=cases.CASES["adafactor_factored"]["hp"]),
    "adafactor_any_f32": dict(shapes=_ANY, steps=3, seed=52, grad=_F32, hp=cases.CASES["adafactor_factored"]["hp"]),
    "adafactor_m_any": dict(shapes=_ANY, steps=3, seed=53, grad=cases.CASES["adafactor_factored_m"]["grad"],
                            hp=cases.CASES["adafactor_factored_m"]["hp"]),
    "adafactor_mf32_any": dict(shapes=_ANY, steps=3, seed=54, grad=_F32,
                               hp=dict(cases.CASES["adafactor_factored_m"]["hp"], m_quant_type="fp32")),
    "adafactor_m_any_lag": dict(shapes=_ANY, steps=4, seed=55, grad=cases.CASES["adafactor_factored_m"]["grad"],
                                hp=dict(cases.CASES["adafactor_factored_m"]["hp"], lag_norm=True)),
    "came_any": dict(shapes=_ANY, steps=3, seed=56, grad=cases.CASES["came_al16"]["grad"], hp=cases.CASES["came_al16"]["hp"]),
    "adafactor_any_short": dict(shapes=[(7, 5), (3, 7), (40, 33)], steps=3, seed=57,
                                grad=cases.CASES["adafactor_factored"]["grad"], hp=cases.CASES["adafactor_factored"]["hp"]),
    "adafactor_any_3d": dict(shapes=_ANY3, steps=3, seed=58, grad=cases.CASES["adafactor_factored"]["grad"],
                             hp=cases.CASES["adafactor_factored"]["hp"]),
    "came_any_3d": dict(shapes=_ANY3, steps=3, seed=59, grad=cases.CASES["came_al16"]["grad"], hp=cases.CASES["came_al16"]["hp"]),
    # matrices that join the batches' table (no momentum, batches hold most elements), and a CAME table where only some
    # tensors have columns of a multiple of 256
    "adafactor_mixed_3d": dict(shapes=[(3, 70, 40), (64, 264), (2, 600, 72), (9, 8)], steps=3, seed=61,
                               grad=cases.CASES["adafactor_factored"]["grad"], hp=cases.CASES["adafactor_factored"]["hp"]),
    "came_mixed_cols": dict(shapes=[(70, 512), (37, 264), (530, 256), (5, 1376)], steps=3, seed=62,
                            grad=cases.CASES["came_al16"]["grad"], hp=cases.CASES["came_al16"]["hp"]),
    "adafactor_m_256_3d": dict(shapes=[(3, 40, 256), (2, 530, 512)], steps=3, seed=60,
                               grad=cases.CASES["adafactor_factored_m"]["grad"], hp=cases.CASES["adafactor_factored_m"]["hp"]),
})

# small states in blocks longer than what waits in shared memory, of either width, and norm vectors of the general kernel beside them
EXTRA_CASES["came_long_blocks"] = dict(shapes=[(5000, 16), (40, 9001), (4100,)], steps=3, seed=63, grad=cases.CASES["came_al16"]["grad"],
                                       hp=dict(cases.CASES["came_al16"]["hp"], block_size=4096))
EXTRA_CASES["adafactor_long_blocks"] = dict(shapes=[(5000, 16), (40, 9001)], steps=3, seed=64, grad=cases.CASES["adafactor_factored"]["grad"],
                                            hp=dict(cases.CASES["adafactor_factored"]["hp"], block_size=8192, v_quant_type="al8"))

# row slices through the warps' rings: binary32 gradients, momentum weights of 1/2 and more (the other form of lerp), a last unit
# of 16 bytes that belongs to one or to two slices of the last row, tiles that end within a group of four rows (with a momentum
# the sums take slices in large tables only, see below)
_SLICES = [(700, 257), (131, 273), (39, 264), (1030, 513), (67, 1001)]
EXTRA_CASES.update({
    "came_slices_f32": dict(shapes=_SLICES, steps=3, seed=65, grad=_F32, hp=cases.CASES["came_al16"]["hp"]),
    "came_slices_w": dict(shapes=_SLICES, steps=3, seed=66, grad=cases.CASES["came_al16"]["grad"], hp=dict(cases.CASES["came_al16"]["hp"], beta1=0.4)),
    "adafactor_m_slices": dict(shapes=_SLICES, steps=3, seed=67, grad=cases.CASES["adafactor_factored_m"]["grad"],
                               hp=cases.CASES["adafactor_factored_m"]["hp"]),
    "adafactor_m_slices_f32_w": dict(shapes=_SLICES, steps=3, seed=68, grad=_F32, hp=dict(cases.CASES["adafactor_factored_m"]["hp"], beta1=0.4)),
    "adafactor_m_slices_8": dict(shapes=[(39, 264), (520, 776), (1030, 520)], steps=3, seed=69, grad=cases.CASES["adafactor_factored_m"]["grad"],
                                 hp=dict(cases.CASES["adafactor_factored_m"]["hp"], maximize=True)),
    # tables of whole vectors without boxes: binary32 gradients, rows of which only some are multiples of 256
    "came_slices_8_f32_w": dict(shapes=[(700, 256), (131, 520), (1030, 512)], steps=3, seed=72, grad=_F32,
                                hp=dict(cases.CASES["came_al16"]["hp"], beta1=0.4)),
    "came_slices_8_w": dict(shapes=[(700, 256), (131, 520), (39, 264)], steps=3, seed=73, grad=cases.CASES["came_al16"]["grad"],
                            hp=dict(cases.CASES["came_al16"]["hp"], beta1=0.4)),
    # the write pass in flat order over whole vectors with that form of lerp; chunks that end a tensor; row ends in a third of the warps
    "came_flat_w": dict(shapes=[(200, 520), (70, 264), (9, 2056)], steps=3, seed=70, grad=cases.CASES["came_al16"]["grad"],
                        hp=dict(cases.CASES["came_al16"]["hp"], beta1=0.4)),
    "came_flat_any": dict(shapes=[(300, 747), (2, 70, 2051), (33, 4099)], steps=3, seed=71, grad=cases.CASES["came_al16"]["grad"],
                          hp=cases.CASES["came_al16"]["hp"]),
})

# the write pass without a momentum in units of 2048 elements: tensors that end a unit, just after it or far inside, units with no, one or
# many row ends, the shortest rows, rows longer than a unit, matrices of a batch that end in a unit (a CTA has one unit here at most;
# test_write_pass_of_many_units gives it several)
_WRITE = [(1, 8), (2, 1024), (1, 2056), (257, 8), (3, 2048), (5, 4104), (100, 24), (1000, 40), (1, 8), (300, 2040), (2, 8)]
EXTRA_CASES.update({
    "adafactor_write": dict(shapes=_WRITE, steps=2, seed=81, grad=cases.CASES["adafactor_factored"]["grad"], hp=cases.CASES["adafactor_factored"]["hp"]),
    "adafactor_write_f32": dict(shapes=_WRITE, steps=2, seed=82, grad=_F32, hp=dict(cases.CASES["adafactor_factored"]["hp"], maximize=True)),
    "adafactor_write_3d": dict(shapes=[(5, 9, 8), (2, 300, 2056), (7, 33, 64), (3, 1, 2048)], steps=2, seed=83,
                               grad=cases.CASES["adafactor_factored"]["grad"], hp=cases.CASES["adafactor_factored"]["hp"]),
})

# lag_norm=True (one pass with the previous step's norm; optimizer.py:1056-1071): the vector kernels, the
# element-wise kernels (odd column counts) and the limiter on top of the clip
EXTRA_CASES.update({
    "adafactor_lag": dict(cases.CASES["adafactor_factored"], steps=5,
                          hp=dict(cases.CASES["adafactor_factored"]["hp"], lag_norm=True)),
    "adafactor_m_lag_fira": dict(shapes=[(200, 520), (37, 131)], steps=5, seed=38,
                                 grad=dict(cases.CASES["adafactor_factored_m"]["grad"], spike_step=3, spike_mult=50.0),
                                 hp=dict(cases.CASES["adafactor_factored_m"]["hp"], lag_norm=True,
                                         enable_fira_for_adafactor=True)),
})


@pytest.mark.parametrize("name", FACTORED_CASES + cases.FACTORED_3D_CASES + sorted(EXTRA_CASES))
def test_factored_free_running_matches_oracle(name, oracle):
    run = OracleRun(name, EXTRA_CASES.get(name))
    params, opt = make_optimizer(run)
    steps = run.case["steps"]
    for t in range(1, steps + 1):
        for p, g in zip(params, run.grads[t]):
            p.grad = to_cuda_grad(g, p.shape)
        opt.step()
        run.step()
        torch.cuda.synchronize()
        for i, p in enumerate(params):
            compare(name, t, i, opt.state[p], run.states[i], p, run.params[i], param_tol=2e-6)
            for key in ("prev_update_norm", "lag_fira_scale"):
                if key in run.states[i]:
                    a, b = float(opt.state[p][key].item()), float(run.states[i][key])
                    assert abs(a - b) <= 2e-6 * max(abs(b), 1.0), f"{name} t{t} p{i} {key}: {a} vs {b}"
    if run.hp["lag_norm"]:
        assert all("prev_update_norm" in opt.state[p] for p in params if p.dim() == 2)
    from adafactor8bit import _native
    assert _native.device_status(torch.cuda.current_stream().cuda_stream) == 0


@pytest.mark.parametrize("name", ["adafactor_factored", "adafactor_factored_m"] + cases.FACTORED_3D_CASES)
def test_factored_matches_reference_golden(name, oracle):
    run = OracleRun(name)
    gold = load_golden(name)
    params, opt = make_optimizer(run)
    steps = run.case["steps"]
    for t in range(1, steps + 1):
        for p, g in zip(params, run.grads[t]):
            p.grad = to_cuda_grad(g, p.shape)
        opt.step()
    torch.cuda.synchronize()
    for i, p in enumerate(params):
        ref = golden_entries(gold, steps, i)
        # (CAME with the limiter: torch's float32 norm puts the reference's limiter state 2e-5 off the accurately
        # summed one, which the parameters then carry)
        parity.assert_params(p.detach().cpu().numpy(), ref["param"], f"{name} final p{i} vs reference",
                             tol=5e-5 if name == "came_3d" else 1e-6)
        for key in CODE_KEYS:
            if key in ref:
                parity.assert_codes(state_np(opt.state[p], key), ref[key], f"{name} final p{i} {key} vs reference",
                                    al16=(ref[key].dtype == np.uint16), zero_reserved=(key != "m_q"))


def test_a_matrix_beside_batches_is_the_same(oracle):
    """Momentum-free matrices share the launch table of batches that hold most of the elements: their norms, and so their clip
    divisors and parameters, are bit for bit those of a table of their own (the grouping differs between the ranks of a
    sharded step, and with the parameters that have a gradient)."""
    from adafactor8bit import Adafactor8Bit
    hp = dict(cases.CASES["adafactor_factored"]["hp"], enable_fira_for_adafactor=True)
    gen = torch.Generator().manual_seed(29)
    flats = [(3 + 7 * i % 40, 8 * (1 + i % 5)) for i in range(60)] + [(64, 264), (530, 1024), (700, 520), (33, 640), (48, 4096)]
    batch = (6, 600, 512)
    start = [torch.randn(s, generator=gen) * 0.02 for s in flats + [batch]]
    grads = [[(torch.randn(s, generator=gen) * torch.randn(s[:-1] + (1,), generator=gen).exp() * 1e-3).bfloat16() for s in flats + [batch]]
             for _ in range(3)]
    out = []
    for n in (len(flats), len(flats) + 1):
        params = [torch.nn.Parameter(x.clone().cuda()) for x in start[:n]]
        for p in params:
            p.grad_dtype = None
        opt = Adafactor8Bit(params, **hp)
        for row in grads:
            for p, g in zip(params, row):
                p.grad = g.cuda()
            opt.step()
        torch.cuda.synchronize()
        out.append([(p.detach().cpu(), float(opt.state[p]["fira_prev_norm"])) for p in params[:len(flats)]])
    apart = [(s, na, nb) for s, (a, na), (b, nb) in zip(flats, *out) if na != nb or not torch.equal(a, b)]
    assert not apart, f"{len(apart)} of {len(flats)} matrices differ: {apart[:3]}"


_UNITS = [(1, 8), (1500, 2048), (257, 8), (1, 2056)] + [(2, 24)] * 12 + [(700, 4104), (8, 8), (1000, 1000), (40, 40000)]


@pytest.mark.parametrize("param,grad,sr", [(torch.float32, torch.bfloat16, False), (torch.float32, torch.float32, False),
                                           (torch.bfloat16, torch.bfloat16, False), (torch.bfloat16, torch.bfloat16, True)])
@pytest.mark.parametrize("shapes", [_UNITS, [(600, 9, 8), (5, 900, 1032), (3, 1, 2048), (7, 33, 64), (2, 300, 2056), (2, 1000, 1000)]], ids=["matrices", "batches"])
def test_write_pass_of_many_units(param, grad, sr, shapes):
    """About 4000 units, four to seven for each resident CTA of the write pass without a momentum: units within a
    tensor and across tensors of a few elements, every stage of the ring used again.  From the same factors the general kernel writes the
    same bits."""
    from adafactor8bit import Adafactor8Bit, _engine, _native as N
    hp = dict(cases.CASES["adafactor_factored"]["hp"], min_8bit_size=1, weight_decay=0.01, stochastic_round_writeback=sr)
    gen = torch.Generator().manual_seed(91)
    params = [torch.nn.Parameter((torch.randn(s, generator=gen) * 0.02).to(param).cuda()) for s in shapes]
    for p in params:
        p.grad_dtype = None
        p.grad = (torch.randn(p.shape, generator=gen) * 1e-3).to(grad).cuda()
    opt = Adafactor8Bit(params, **hp)
    opt.step()
    plan = max((x for x in opt._plans.values() if isinstance(x, _engine.FactoredPlan)), key=lambda x: x.total_chunks)
    params, update, seen = plan.params, plan._update, []

    def both(mode, *args):
        if mode != N.FUPD_APPLY:
            return update(mode, *args)
        assert plan.cfg.aligned8 and plan.total_chunks > 3500 and len(params) > 4
        before, route = [p.detach().clone() for p in params], plan.cfg.aligned8
        for plan.cfg.aligned8 in (0, route):
            for p, b in zip(params, before):
                p.detach().copy_(b)
            update(mode, *args)
            seen.append([p.detach().clone() for p in params])
        assert not any(torch.equal(a, b) for a, b in zip(seen[0], before) if a.numel() >= 1000)

    plan._update = both
    opt.step()
    torch.cuda.synchronize()
    bits = torch.int32 if param == torch.float32 else torch.int16
    for a, b in zip(*seen):
        assert torch.equal(a.view(bits), b.view(bits)), (a.shape, int((a != b).sum()))


_ROWS8, _RAGGED = [(39, 264), (520, 776), (1030, 520)], [(700, 257), (131, 273), (39, 264), (1030, 513), (67, 1001)]


@pytest.mark.parametrize("grad,beta1,shapes,sliced", [
    (torch.bfloat16, 0.9, _ROWS8 + [(2552, 8184)], True), (torch.bfloat16, 0.4, _ROWS8 + [(2552, 8184)], True),
    (torch.float32, 0.9, _ROWS8 + [(4104, 16392)], True), (torch.float32, 0.4, _ROWS8 + [(4104, 16392)], True),
    (torch.bfloat16, 0.9, _RAGGED + [(4099, 2067)], True), (torch.bfloat16, 0.4, _RAGGED + [(4099, 2067)], True),
    (torch.float32, 0.9, _RAGGED + [(4099, 2067)], True), (torch.float32, 0.4, _RAGGED + [(4099, 2067)], True),
    (torch.bfloat16, 0.9, [(3, 70, 40), (2, 33, 131), (2, 2040, 2100)], True), (torch.float32, 0.9, [(2, 600, 72), (2, 2040, 2104)], True),
    (torch.bfloat16, 0.9, [(73000, 117)], False), (torch.bfloat16, 0.9, [(132000, 128)], False), (torch.bfloat16, 0.9, [(2040, 8200)], False),
    (torch.float32, 0.9, [(4088, 16392)], False), (torch.float32, 0.9, [(4000, 2067)], False)])
def test_sums_with_a_momentum_are_the_same_in_slices_and_flat(grad, beta1, shapes, sliced):
    """Sums of squares of Adafactor with a UF8 momentum: tables from 2^24 elements on (2^26 with binary32 gradients; 2^23 for rows
    that are not whole vectors and batches) that fill their tiles take them in row slices, the others in flat order.  The binary32 sums of eight
    squares are the same in both, so only the order of binary64 additions differs: 2^-53 of the sum for each of the 2^17 that
    pass through one accumulator at most, 1.5e-11."""
    from adafactor8bit import Adafactor8Bit, _engine
    hp = dict(cases.CASES["adafactor_factored_m"]["hp"], beta1=beta1, m_quant_type="uf8", m_block_size=256, min_8bit_size=1)
    totals = []
    for flat in (False, True):
        gen = torch.Generator(device="cuda").manual_seed(33)
        params = [torch.nn.Parameter(torch.randn(s, generator=gen, device="cuda") * 0.02) for s in shapes]
        opt = Adafactor8Bit(params, **hp)
        for t in (1, 2):
            for p in params:
                p.grad_dtype = None
                p.grad = (torch.randn(p.shape, generator=gen, device="cuda") * 1e-3).to(grad)
            if t == 2:
                plan, = [x for x in opt._plans.values() if isinstance(x, _engine.FactoredPlan)]
                assert plan.cfg.total_tiles > 0
                if flat:
                    plan.cfg.total_tiles = 0
            opt.step()
        sums = [plan.d_sumsq[int(f):int(f) + int(n)] for f, n in zip(plan.first_chunk, plan.nchunks)]
        assert bool((sums[-1][1:] == 0.0).all()) == (sliced and not flat)
        totals.append([float(x.sum()) for x in sums])
    for shape, a, b in zip(shapes, *totals):
        assert b > 0.0 and abs(a - b) <= 1.5e-11 * b, (shape, a, b)


@pytest.mark.parametrize("came", [False, True])
@pytest.mark.parametrize("shape", [(3, 40, 264), (3, 33, 131), (70, 1001), (3, 40, 256)])
def test_infinities_and_nans_in_rows_of_any_length(shape, came, oracle):
    """Batches and rows of any length with a UF8 momentum: momenta, ranges and parameters as the general kernels (fp16 gradients) leave them."""
    from adafactor8bit import Adafactor8Bit
    hp = dict(cases.CASES["came_al16" if came else "adafactor_factored_m"]["hp"], m_quant_type="uf8", m_block_size=256, min_8bit_size=1)
    gen = torch.Generator().manual_seed(31)
    start = torch.randn(shape, generator=gen) * 0.02
    grads = [(torch.randn(shape, generator=gen) * 1e-2).half() for _ in range(3)]
    flat = grads[1].view(-1)
    flat[7], flat[-1], flat[400] = float("inf"), float("nan"), -float("inf")
    out = []
    for dtype in (torch.float32, torch.float16):
        p = torch.nn.Parameter(start.clone().cuda())
        p.grad_dtype = None
        opt = Adafactor8Bit([p], **hp)
        for g in grads:
            p.grad = g.cuda().to(dtype)
            opt.step()
        torch.cuda.synchronize()
        out.append((p.detach().cpu(), {k: v.cpu() for k, v in opt.state[p].items() if isinstance(v, torch.Tensor)}))
    (p, st), (q, ref) = out
    np.testing.assert_allclose(st["m_scale"].numpy(), ref["m_scale"].numpy(), rtol=1e-5, equal_nan=True)
    parity.assert_codes(st["m_q"].numpy(), ref["m_q"].numpy(), f"{shape} m_q", zero_reserved=False)
    np.testing.assert_allclose(p.numpy(), q.numpy(), rtol=1e-4, atol=1e-7, equal_nan=True)
