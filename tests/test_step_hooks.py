"""The step's own wrapper: hooks run, and a profiler sees the step, as with torch.optim's."""
import functools
import json

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


def subclass():
    class Scaled(Adafactor8Bit):
        def step(self, closure=None):
            return super().step(closure)
    return Scaled


def patched():
    """A class whose step another library has wrapped, after its first instance was made."""
    class Patched(Adafactor8Bit):
        pass
    Patched([torch.nn.Parameter(torch.zeros(8))])
    inner = Patched.step

    @functools.wraps(inner)
    def step(self, *args, **kwargs):
        return inner(self, *args, **kwargs)
    Patched.step = step
    return Patched


@pytest.mark.parametrize("kind", ["own", "global"])
@pytest.mark.parametrize("make_class", [subclass, patched])
def test_hooks_run_once_around_a_step_that_calls_the_base_step(kind, make_class):
    make()                                      # (torch.optim has wrapped the base class's step)
    opt, seen = make_class()([torch.nn.Parameter(torch.zeros(8))]), []
    pre, post = (lambda *a: seen.append("pre")), (lambda *a: seen.append("post"))
    handles = ([opt.register_step_pre_hook(pre), opt.register_step_post_hook(post)] if kind == "own" else
               [register_optimizer_step_pre_hook(pre), register_optimizer_step_post_hook(post)])
    for _ in range(2):
        opt.step()
    for h in handles:
        h.remove()
    assert seen == ["pre", "post"] * 2


def test_a_step_that_fails_leaves_the_hooks_in_place():
    opt, seen = make(), []
    opt.register_step_pre_hook(lambda *a: seen.append("pre"))
    with pytest.raises(ValueError):
        opt.step(grad_ready=[])
    opt.step()
    assert seen == ["pre"] * 2


def test_the_profiler_sees_one_range_of_a_subclass():
    opt = subclass()([torch.nn.Parameter(torch.zeros(8))])
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        opt.step()
    assert [e.name for e in prof.events()].count("Optimizer.step#Scaled.step") == 1


def test_an_execution_trace_without_a_profiler_sees_the_step(tmp_path):
    opt, path = make(), str(tmp_path / "trace.json")
    observer = torch.profiler.ExecutionTraceObserver().register_callback(path)
    observer.start()
    opt.step()
    observer.stop()
    observer.unregister_callback()
    with open(path) as f:
        names = [n["name"] for n in json.load(f)["nodes"]]
    assert names.count("Optimizer.step#Adafactor8Bit.step") == 1
