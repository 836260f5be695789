"""State in and out through device arrays: arrays that the engines' kernels read and write in place give what host
arrays give, and so do arrays at an odd offset, which go through copies. Counts around the launch's blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _on_device(a, offset):
    """a on the GPU, `offset` floats into its allocation (so aligned to 4 bytes only when the offset is odd)"""
    import torch

    flat = torch.empty(a.size + offset, dtype=torch.float32, device="cuda")
    flat[offset:] = torch.from_numpy(a.ravel()).cuda()
    return flat[offset:].view(a.shape)


@pytest.mark.parametrize("n", [1, 255, 257, 4099])
@pytest.mark.parametrize("offset", [0, 1])
def test_pbf_device_arrays(gpe_mod, cuda_ok, n, offset):
    from gpe import scenes

    g = np.random.default_rng(n)
    pos = g.uniform(0.0, 1.0, (n, 2)).astype(np.float32)
    vel = g.normal(0, 0.2, (n, 2)).astype(np.float32)
    p = scenes.dam_params(iters=2)
    p.dt = 1.0 / 480.0
    got = []
    for dev in (False, True):
        e = gpe_mod.Pbf(p, [(0.0, 0.0, 1.0, 1.0)], capacity=n + 3)
        for _ in range(2):  # the second state finds the histogram that the first one's last step left
            a, b = (_on_device(pos, offset), _on_device(vel, offset)) if dev else (pos, vel)
            e.set_state(a, b)
            e.step(2)
        if dev:
            x, v = _on_device(pos * 0, offset), _on_device(vel * 0, offset)
            e.get_state(x, v)
            got.append((x.cpu().numpy(), v.cpu().numpy()))
        else:
            got.append(e.get_state()[:2])
        assert e.status() == 0
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n", [1, 255, 4099])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("given", ["x", "all"])
def test_mpm_device_arrays(gpe_mod, cuda_ok, n, offset, given):
    """Before any step the state comes back as it was set, defaults included, in the caller's order after a sort."""
    from gpe import scenes

    g = np.random.default_rng(n)
    p = scenes.elastic_params(n, 64)
    want = [g.uniform(0.2, 0.8, (n, 2)), np.zeros((n, 2)), np.zeros((n, 4)), np.tile([1.0, 0, 0, 1], (n, 1)), np.ones(n)]
    if given == "all":
        want[1:] = [g.normal(0, 1, w.shape) for w in want[1:]]
    want = [w.astype(np.float32) for w in want]
    e = gpe_mod.Mpm(p, capacity=n)
    e.set_state(*[_on_device(w, offset) for w in (want if given == "all" else want[:1])])
    e.stage(gpe_mod.MPM_STAGE_SORT)
    out = [_on_device(w * 0, offset) for w in want]
    e.get_state_device(*out)
    for a, b in zip(out, want):
        np.testing.assert_array_equal(a.cpu().numpy(), b)
    host = e.get_state()
    for a, b in zip(host, want):
        np.testing.assert_array_equal(a, b)
