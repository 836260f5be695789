"""MLS-MPM calls of several steps (G2P and the next P2G in one launch) against the same steps one call at a time (the
separate kernels), over every material mode and the storage orders that the scatter's paths differ in: particles sorted
by base node, in lattice rows (many short runs on neighbouring nodes), at random, all on one node, and counts around a
warp's 64 particles. The two differ in the rounding of a few sums a step: 2e-5 of each field's largest magnitude over
four steps (C, a velocity difference over one cell, of |v| / dx at least)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _state(order, n, seed=3):
    g = np.random.default_rng(seed)
    if order == "rows":
        w = max(1, int(np.sqrt(n)))
        i = np.arange(n)
        x = 0.25 + np.stack([(i % w) * 0.45, (i // w) * 0.45], 1) / (2 * w)
    elif order == "one":
        x = np.full((n, 2), 0.5) + g.uniform(-1e-3, 1e-3, (n, 2))
    else:
        x = g.uniform(0.3, 0.7, (n, 2))
    v = g.normal(0, 0.3, (n, 2))
    return x.astype(np.float32), v.astype(np.float32)


@pytest.mark.parametrize("order", ["sorted", "rows", "random", "one"])
@pytest.mark.parametrize("n", [1, 2, 63, 65, 4097])
@pytest.mark.parametrize("material", [0, 1, 2, 3, 4, "mixed"])
def test_steps_of_one_call_match_single_steps(gpe_mod, cuda_ok, order, n, material):
    from gpe import scenes

    p = scenes.mixed_params(max(n, 1024), 64)
    mat = None
    if material == "mixed":
        mat = (np.arange(n) % 5).astype(np.int32)
    else:
        p.flags = 0
        p.material = material
    p.sort_interval = 100 if order == "sorted" else 0
    x, v = _state(order, n)
    got = []
    for calls in ([4], [1, 1, 1, 1]):
        e = gpe_mod.Mpm(p, capacity=n)
        e.set_state(x, v, material=mat)
        for c in calls:
            e.step(c)
        got.append(e.get_state())
        assert e.status() == 0
    for f, (a, b) in enumerate(zip(*got)):
        scale = max(np.abs(b).max(), np.abs(got[1][1]).max() / p.dx if f == 2 else 0.0)
        assert np.abs(a - b).max() <= 2e-5 * scale


def test_scenes_of_one_call_match_single_steps(gpe_mod, cuda_ok):
    from gpe import scenes

    p, sc, pos, mat, sid = scenes.mixed_batch(n_scenes=3, lo=3000, hi=9000, total_ref=65536)
    table = [gpe_mod.make_mpm_scene(*s) for s in sc]
    vel = np.random.default_rng(2).normal(0, 0.2, pos.shape).astype(np.float32)
    got = []
    for calls in ([4], [1, 1, 1, 1]):
        e = gpe_mod.Mpm(p, capacity=len(pos), scenes=table)
        e.set_state(pos, vel, material=mat, scene_id=sid)
        for c in calls:
            e.step(c)
        got.append(e.get_state())
    for f, (a, b) in enumerate(zip(*got)):
        scale = max(np.abs(b).max(), np.abs(got[1][1]).max() / p.dx if f == 2 else 0.0)
        assert np.abs(a - b).max() <= 2e-5 * scale
