"""Calls made under a torch stream that is not the default one, which does not
wait for the default one: their device copies are ordered on that stream."""
import types

import numpy as np
import pytest


def test_device_copies_run_on_the_current_stream(monkeypatch):
    """memcpy_d2d issues its copy on torch's current stream and waits there;
    on the default stream cudaMemcpy is that copy.  The runtime's calls are
    recorded in place of a GPU."""
    import torch
    from pgrav import step
    calls = []

    def record(name):
        return lambda *a: calls.append((name,) + a) or (0,)

    fake = types.SimpleNamespace(
        cudaMemcpyKind=types.SimpleNamespace(cudaMemcpyDeviceToDevice=3),
        cudaMemcpy=record("cudaMemcpy"), cudaMemcpyAsync=record("cudaMemcpyAsync"),
        cudaStreamSynchronize=record("cudaStreamSynchronize"))
    monkeypatch.setattr(step, "_rt", lambda: fake)
    for stream in (77, 0):
        monkeypatch.setattr(torch.cuda, "current_stream",
                            lambda: types.SimpleNamespace(cuda_stream=stream))
        step.memcpy_d2d(16, 32, 64)
    assert calls == [("cudaMemcpyAsync", 16, 32, 64, 3, 77), ("cudaStreamSynchronize", 77),
                     ("cudaMemcpy", 16, 32, 64, 3)]


def test_bodies_are_complete_before_the_build(monkeypatch):
    """Plan.build waits for the stream that its bodies are written on, with the
    library's and torch's calls recorded in place of a GPU."""
    import torch
    from pgrav import gravcuda as gc
    calls = []
    monkeypatch.setattr(torch.cuda, "current_stream", lambda: types.SimpleNamespace(
        cuda_stream=77, synchronize=lambda: calls.append("wait")))
    monkeypatch.setattr(gc, "lib", lambda: types.SimpleNamespace(
        grav_plan_build_CUDA=lambda *a: calls.append("build") or 0, grav_plan_free=lambda h: None))
    gc.Plan.build(None, None, 1e-4, bodies=torch.zeros((8, 4)))
    assert calls == ["wait", "build"]


@pytest.mark.gpu
def test_stepper_on_a_side_stream():
    """A stepper made and rebuilt under a side stream that is held up before its
    bodies are written gives the default stream's states, bit for bit."""
    import torch
    from pgrav import ics
    from pgrav.step import Stepper
    p, m = ics.plummer(3000, seed=6)
    v = np.random.default_rng(6).normal(0, 0.1, p.shape)

    def go(hold):
        hold()
        s = Stepper(p, v, m, 1e-4, rebuild=2, tree_kw=dict(tol=1e-4))
        for _ in range(3):
            hold()
            s.run(2, 1e-3)
        out = s.state()
        s.free()
        return out

    want = go(lambda: None)
    with torch.cuda.stream(torch.cuda.Stream()):
        got = go(lambda: torch.cuda._sleep(20_000_000))
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.gpu
@pytest.mark.parametrize("box", [0.0, 1.0])
def test_gradient_on_a_side_stream(monkeypatch, box):
    """Forward and backward under a side stream, with the default stream held
    up after every build, give the default stream's forces and gradients."""
    import torch
    from pgrav import gravcuda as gc, ics
    from pgrav.autograd import gravity
    if box > 0:
        p, m = ics.grf_box(12, seed=5, rms_disp=0.25)
    else:
        p, m = ics.plummer(3000, seed=5)
    kw = dict(tol=1e-4, p2cut=7, p4cut=20)
    if box > 0:
        kw.update(box=box, ewald=True)
    g = torch.Generator(device="cuda").manual_seed(5)
    pos = torch.from_numpy(np.ascontiguousarray(p, np.float32)).cuda().requires_grad_(True)
    mass = torch.from_numpy(np.ascontiguousarray(m, np.float32)).cuda().requires_grad_(True)
    w = torch.randn(pos.shape, generator=g, device="cuda")
    u = torch.randn(len(pos), generator=g, device="cuda")

    def go():
        acc, phi = gravity(pos, mass, 1e-4, **kw)
        return (acc, phi) + torch.autograd.grad((w * acc).sum() + (u * phi).sum(), (pos, mass))

    want = [t.detach().clone() for t in go()]
    real = gc.Plan.build.__func__

    def held_up(cls, *a, **k):
        plan = real(cls, *a, **k)
        with torch.cuda.stream(torch.cuda.default_stream()):
            torch.cuda._sleep(20_000_000)  # about 10 ms
        return plan

    monkeypatch.setattr(gc.Plan, "build", classmethod(held_up))
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        got = [t.detach().clone() for t in go()]
    side.synchronize()
    # forces are the same bits; a gradient's FP64 atomic sums may round to the next float
    for k, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b) if k < 2 else (a - b).abs().max() <= 1e-6 * b.abs().max()
