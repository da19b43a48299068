"""The step's own wrapper: hooks run, and a profiler sees the step, as with torch.optim's."""
import pytest
import torch
from torch.optim.optimizer import register_optimizer_step_post_hook, register_optimizer_step_pre_hook

from adafactor8bit import Adafactor8Bit


def make():
    return Adafactor8Bit([torch.nn.Parameter(torch.zeros(8))])


@pytest.mark.parametrize("kind", ["own", "global"])
def test_hooks_run_around_the_step(kind):
    opt, seen = make(), []

    def before(o, args, kwargs):
        seen.append(("before", o is opt, args[1:], kwargs))

    def after(o, args, kwargs):
        seen.append(("after", o is opt, args[1:], kwargs))

    if kind == "own":
        handles = [opt.register_step_pre_hook(before), opt.register_step_post_hook(after)]
    else:
        handles = [register_optimizer_step_pre_hook(before), register_optimizer_step_post_hook(after)]
    opt.step(grad_ready=[None])
    for h in handles:
        h.remove()
    opt.step()
    want = [("before", True, (), {"grad_ready": [None]}), ("after", True, (), {"grad_ready": [None]})]
    assert seen == want


def test_the_closure_and_the_profiler():
    opt = make()
    assert opt.step(lambda: 3.0) == 3.0
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        opt.step()
    assert any(e.name == "Optimizer.step#Adafactor8Bit.step" for e in prof.events())
