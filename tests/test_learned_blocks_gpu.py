"""The network step, the step that starts its memory and the collection of training pairs run, with one result bit for
bit, at every block size that the tuning accepts."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind):
    from gpe import scenes

    p = scenes.dam_params(iters=2)
    p.dt = 1.0 / 480.0
    if kind == "dam":
        pos, _, boxes = scenes.dam_break(n_side=50)
        dom = None
    else:
        pos, _, dom, boxes = scenes.batched_scenes(n_scenes=4, seed=5, lo=300, hi=2000)
    return p, pos, np.random.default_rng(3).normal(0, 0.2, pos.shape).astype(np.float32), dom, boxes


@pytest.mark.parametrize("kind", ["dam", "scenes"])
@pytest.mark.parametrize("block", [128, 512])
@pytest.mark.parametrize("skin", [0.075, 0.0])
def test_learned_steps_and_collection_at_every_block_size(gpe_mod, cuda_ok, kind, block, skin):
    p, pos, vel, dom, boxes = _scene(kind)
    got = []
    for b in (256, block):
        e = gpe_mod.Pbf(p, boxes, capacity=len(pos))
        e.set_tuning(block=b, skin=skin)
        e.set_state(pos, vel, dom)
        net = gpe_mod.Mlp(max_pairs=3 * len(pos), seed=2)
        net.collect(e, n_steps=3, stride=1, seed=5)
        X, T, at = net.pairs()
        order = np.lexsort((T, at))
        e.set_warm_start(gpe_mod.WARM_MLP, net)
        e.set_state(pos, vel, dom)
        e.step(3)
        assert e.status() == 0
        got.append((X[order], T[order], at[order], *e.get_state()))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
