"""Candidate lists where device memory is short: lists of 48, 32 and 16 candidates a particle and none at all give the
same state bit for bit, and an engine without lists says so. The memory is taken up by one allocation beside the engine."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CAP = 20_000_000
LISTS = 96 * CAP  # bytes of the full lists


def _scene(kind):
    from gpe import scenes

    p = scenes.dam_params(iters=3)
    p.dt = 1.0 / 480.0
    pos, _, boxes = scenes.dam_break(n_side=100)
    if kind == "crowded":  # 14 to 40 candidates a particle: lists of 16 and 32 hold some of them
        pos = (pos * np.float32(0.7)).astype(np.float32)
    if kind == "wide":
        boxes = [(0.0, 0.0, 4100 * p.h, 2.56)]
    return p, pos, np.random.default_rng(3).normal(0, 0.3, pos.shape).astype(np.float32), boxes


@pytest.mark.parametrize("kind", ["lattice", "crowded", "wide"])
def test_state_does_not_depend_on_the_room_for_lists(gpe_mod, cuda_ok, kind):
    torch = pytest.importorskip("torch")
    p, pos, vel, boxes = _scene(kind)
    torch.cuda.empty_cache()

    def engine():
        return gpe_mod.Pbf(p, boxes, capacity=CAP)

    def run(e):
        e.set_state(pos, vel)
        e.step(4)
        x, v, _ = e.get_state()
        assert e.status() == 0
        return x, v

    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    e = engine()
    whole = free - torch.cuda.mem_get_info()[0]  # the engine with its full lists
    lists = LISTS * (2 if kind == "wide" else 1)
    assert whole > lists
    want = run(e)
    assert e.tuning().skin == np.float32(0.075)
    e.close()
    for share in (5 / 6, 1 / 2, 1 / 6):  # room for 2/3 of the lists, for 1/3, for none
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ballast = torch.empty(free - (whole - lists) - int(share * lists), dtype=torch.uint8, device="cuda")
        try:
            e = engine()
            assert e.tuning().skin == (np.float32(0.075) if share > 0.2 else 0.0)
            got = run(e)
            if share < 0.2:
                assert e.autotune(2)[0].skin == 0.0
            e.close()
        finally:
            del ballast
            torch.cuda.empty_cache()
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
