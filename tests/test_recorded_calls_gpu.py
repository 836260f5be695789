"""Calls recorded into a caller's graph between ordinary steps: the host is not told when (or whether) a recording runs,
and the engine's steps before and after a replay, or without one, equal those of an engine that made the same calls
directly, bit for bit (the sort is stable, whichever way its histogram was made)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(gpe_mod, kind, cap=0):
    from gpe import scenes

    if kind == "reference":
        p = scenes.reference_pbf_params(2)
        p.flags |= gpe_mod.PBF_DYNAMIC_COUNT
        pos, vel, boxes = scenes.reference_pbf_block()
    else:  # (beyond 65,536 particles the histogram does not count the scan's tile totals)
        p = scenes.dam_params(iters=2)
        p.dt = 1.0 / 480.0
        side = 64 if kind == "dam" else 265
        pos, vel, boxes = scenes.dam_break(n_side=side, box=2 * side * 0.01)
    vel = np.random.default_rng(1).normal(0, 0.3, pos.shape).astype(np.float32)
    e = gpe_mod.Pbf(p, boxes, capacity=len(pos) + cap)
    e.set_state(pos, vel)
    return e, pos, vel


def _recorded(torch, calls):
    """A graph of what calls(stream) issues."""
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=torch.cuda.Stream()):
        calls(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return g


def _same(torch, a, b):
    torch.cuda.synchronize()
    assert a.status() == 0 and b.status() == 0
    (xa, va, _), (xb, vb, _) = a.get_state(), b.get_state()
    np.testing.assert_array_equal(xa, xb)
    np.testing.assert_array_equal(va, vb)


@pytest.mark.parametrize("kind", ["dam", "dam70k", "reference"])
@pytest.mark.parametrize("what", ["set_state", "enqueue", "both", "stages", "emit"])
def test_steps_around_recorded_calls(gpe_mod, cuda_ok, kind, what):
    torch = pytest.importorskip("torch")
    if what == "emit" and kind != "reference":
        pytest.skip("emitters need a device-resident count")
    (a, pos, vel), (b, _, _) = _engine(gpe_mod, kind, 4000), _engine(gpe_mod, kind, 4000)
    new = [torch.from_numpy(np.ascontiguousarray(q[::-1])).cuda() for q in (pos, vel)]
    # (32 particles: a warp's emission has one order, several warps' append in any)
    hose = gpe_mod.make_hose((50.0, 150.0), (1.0, -0.3), 8.0, 1.05, 0.02, 4)
    stages = [gpe_mod.PBF_STAGE_PREDICT_SORT] + 2 * [gpe_mod.PBF_STAGE_LAMBDA, gpe_mod.PBF_STAGE_DELTA_P] + [
        gpe_mod.PBF_STAGE_XSPH, gpe_mod.PBF_STAGE_FINISH]

    def calls(e, st):
        if what in ("set_state", "both"):
            e.set_state(*new, stream=st)
        if what in ("enqueue", "both"):
            e.enqueue(2, stream=st)
        if what == "emit":
            assert e.emit(hose, seed=9, stream=st) == 32
        if what == "stages":
            for s in stages:
                e.stage(s, stream=st)

    for e in (a, b):
        e.step(3)
    g = _recorded(torch, lambda st: calls(a, st))
    for e in (a, b):
        e.step(2)  # the recording has not run
    _same(torch, a, b)
    for steps in (1, 3):
        g.replay()
        torch.cuda.synchronize()
        calls(b, None)
        for e in (a, b):
            e.step(steps)
        _same(torch, a, b)


def test_device_state_is_read_and_written_in_a_recording(gpe_mod, cuda_ok):
    torch = pytest.importorskip("torch")
    (a, pos, vel), (b, _, _) = _engine(gpe_mod, "dam"), _engine(gpe_mod, "dam")
    new = [torch.from_numpy(q).cuda() for q in (pos, vel)]
    out = [torch.zeros_like(q) for q in new]

    def calls(st):
        a.set_state(*new, stream=st)
        a.enqueue(3, stream=st)
        a.get_state(*out, stream=st)

    g = _recorded(torch, calls)
    for r in range(2):
        new[1].mul_(0.5)
        g.replay()
        torch.cuda.synchronize()
        b.set_state(*new)
        b.step(3)
        x, v, _ = b.get_state()
        np.testing.assert_array_equal(out[0].cpu().numpy(), x)
        np.testing.assert_array_equal(out[1].cpu().numpy(), v)
