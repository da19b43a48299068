"""Uploads of launch tables from any host memory, tensor maps that are written anew at every step, and calls that are captured into a graph."""
import ctypes

import numpy as np
import pytest
import torch

import cases

pytestmark = pytest.mark.gpu

SHAPES = [(70, 264), (4100,), (3, 2048), (40, 1000)]


def make():
    from adafactor8bit import Adafactor8Bit
    gen = torch.Generator().manual_seed(3)
    params = [torch.nn.Parameter((torch.randn(s, generator=gen) * 0.02).cuda()) for s in SHAPES]
    for p in params:
        p.grad = (torch.randn(p.shape, generator=gen) * 1e-3).cuda()
    opt = Adafactor8Bit(params, **dict(cases.CASES["adamw_uf8_al8"]["hp"], min_8bit_size=1))
    opt.step()
    plan, = opt._plans.values()
    ring = plan.h_table
    torch.cuda.synchronize()
    return params, opt, plan, np.array(ring.views[ring.i])       # (the launch table of that step)


def again(plan, address, stream):
    from adafactor8bit import _native as N
    N.check(N.lib().af8_fullrank_step(ctypes.byref(plan.cfg), address, plan.d_table.data_ptr(), plan.n, plan.total_blocks,
                                      plan.d_dyn.data_ptr(), None, stream.cuda_stream), "af8_fullrank_step")


def result(params, opt):
    torch.cuda.synchronize()
    return [p.detach().cpu().view(torch.int32) for p in params] + [opt.state[p][k].cpu() for p in params for k in ("m_q", "variance_q")]


def test_a_table_comes_from_any_host_memory():
    """The same second step from a pinned table (copied by a kernel), a pinned one off the 16-byte units, and a pageable one."""
    out = []
    for kind in ("pinned", "unaligned", "pageable"):
        params, opt, plan, table = make()
        plan.d_table.zero_()
        room = torch.empty(table.size + 64, dtype=torch.uint8, pin_memory=kind != "pageable")
        off = -room.data_ptr() % 16 + (8 if kind == "unaligned" else 0)
        room.numpy()[off:off + table.size] = table
        again(plan, room.data_ptr() + off, torch.cuda.current_stream())
        out.append(result(params, opt))
    for other in out[1:]:
        assert all(torch.equal(a, b) for a, b in zip(out[0], other))


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5])
def test_no_table_of_an_apollo_step_takes_the_copy_engine(n):
    """The write-back table has 104 bytes a tensor: odd numbers of tensors end in half a 16-byte unit."""
    from adafactor8bit import Adafactor8Bit
    gen = torch.Generator().manual_seed(n)
    params = [torch.nn.Parameter((torch.randn(256, 128 + 64 * i, generator=gen) * 0.02).cuda()) for i in range(n)]
    opt = Adafactor8Bit(params, **dict(cases.CASES["apollo_r32"]["hp"], apollo_update_proj_gap=100))
    for p in params:
        p.grad_dtype = None
        p.grad = (torch.randn(p.shape, generator=gen) * 1e-3).bfloat16().cuda()
    before = [p.detach().clone() for p in params]
    opt.step()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        opt.step()
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if e.device_type == torch.autograd.DeviceType.CUDA]
    assert any("apollo_write_kernel" in k for k in names) and not any("Memcpy HtoD" in k for k in names)
    assert all(bool((p != b).any(1).all()) for p, b in zip(params, before))


def test_a_captured_step_replays():
    """Two steps captured into a graph, upload included, are the two steps launched one by one."""
    out = []
    for graph in (False, True):
        params, opt, plan, table = make()
        room = torch.empty(table.size, dtype=torch.uint8, pin_memory=True)
        room.numpy()[:] = table
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            if graph:
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=stream):
                    again(plan, room.data_ptr(), stream)
                    again(plan, room.data_ptr(), stream)
                g.replay()
            else:
                again(plan, room.data_ptr(), stream)
                again(plan, room.data_ptr(), stream)
        out.append(result(params, opt))
    assert all(torch.equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("name", ["came_al16", "apollo_r32"])
def test_gradients_that_move(name):
    """The tensor maps of a step lie where those of the last step lay.  Gradients at another address at every step, the steps queued
    behind one another, against the same gradients copied to one place, step by step.  Sums by binary64 atomics differ in their order, so
    that a stored code may tip: a few elements off by 1e-2 of an update, 1e-6 of the norm.  One step with another step's gradients: 1e-3 and more."""
    from adafactor8bit import Adafactor8Bit
    shapes = [(512, 1024), (1024, 256), (768, 512)]
    hp = dict(cases.CASES[name]["hp"], min_8bit_size=1)
    out = []
    for moving in (False, True):
        gen = torch.Generator().manual_seed(11)
        torch.manual_seed(0)
        params = [torch.nn.Parameter((torch.randn(s, generator=gen) * 0.02).cuda()) for s in shapes]
        opt = Adafactor8Bit(params, **hp)
        grads = [[(torch.randn(s, generator=gen) * 1e-3 * 4.0 ** k).bfloat16().cuda() for s in shapes] for k in range(4)]
        home = [torch.empty_like(g) for g in grads[0]]
        for p in params:
            p.grad_dtype = None
        for k in range(8):
            for i, p in enumerate(params):
                p.grad = grads[k % 4][i] if moving else home[i].copy_(grads[k % 4][i])
            opt.step()
            if not moving:
                torch.cuda.synchronize()
        out.append([p.detach().clone() for p in params])
    for a, b in zip(*out):
        assert float((a - b).norm() / a.norm()) < 1e-4
