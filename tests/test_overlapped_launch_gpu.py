"""Kernels launched while the one before them ends (the graph of a step call, a frame's passes): steps of one call against
the same steps enqueued one by one, which keep full dependencies, and frames drawn in a row or replayed from a caller's
graph against frames with a synchronisation after every call. Everything is the same bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(gpe_mod, option, n=6000):
    from gpe import scenes

    p = scenes.dam_params(iters=3)
    p.dt = 1.0 / 480.0
    if option == "vorticity":
        p.vort_eps = 0.02
    if option == "ids":
        p.flags |= gpe_mod.PBF_PAIR_IDS | gpe_mod.PBF_SELF_GRAD
    size = 1.0 if n <= 6000 else 4.0
    boxes = [(0.0, 0.0, size, size)]
    g = np.random.default_rng(n)
    pos = g.uniform(0.0, size, (n, 2)).astype(np.float32)
    dom = None
    if option == "scenes":
        boxes = [(2.0 * size * d, 0.0, size, size) for d in range(3)]
        dom = np.sort(np.arange(n) % 3).astype(np.int32)
        pos[:, 0] += np.float32(2.0 * size) * dom
    e = gpe_mod.Pbf(p, boxes, capacity=n)
    e.set_state(pos, g.normal(0, 0.2, (n, 2)).astype(np.float32), domain=dom)
    return e


@pytest.mark.parametrize("option", ["plain", "vorticity", "ids", "scenes"])
@pytest.mark.parametrize("n", [1, 129, 6000, 65536, 65537])  # 65,536: the last whose histogram counts tile sums
def test_steps_of_one_call_equal_enqueued_steps(gpe_mod, cuda_ok, option, n):
    got = []
    for whole in (True, False):
        e = _engine(gpe_mod, option, n)
        for _ in range(2):
            if whole:
                e.step(5)
            else:
                for _ in range(5):
                    e.enqueue(1)
        assert e.status() == 0
        got.append(e.get_state()[:2])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)


def test_frames_in_a_row(gpe_mod, cuda_ok):
    torch = pytest.importorskip("torch")
    from test_render_gpu import _raster

    cx, cy, dim, cap, size = 4, 4, 0.25, 4096, 512
    out = []
    for how in ("synchronised", "in a row", "captured"):
        e = _engine(gpe_mod, "plain")
        vp = torch.zeros((cx * cy * cap, 2), dtype=torch.float32, device="cuda")
        vv, vc = torch.zeros_like(vp), torch.zeros(cx * cy, dtype=torch.int32, device="cuda")
        view = gpe_mod.View(vp.data_ptr(), vv.data_ptr(), vc.data_ptr(), cx, cy, dim, cap)
        r, img, _ = _raster(gpe_mod, torch, size, size, size, dim, pad=0)
        st = torch.cuda.Stream()
        torch.cuda.synchronize()
        sync = st.synchronize if how == "synchronised" else (lambda: None)

        def frame():
            e.publish(view, stream=st.cuda_stream)
            sync()
            gpe_mod.render_frame(r, view, stream=st.cuda_stream)
            sync()

        with torch.cuda.stream(st):
            if how == "captured":
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=st):
                    frame()
                frame = graph.replay
            images = []
            for _ in range(6):
                e.step(2, stream=st.cuda_stream)
                frame()
                images.append(img.clone())
        st.synchronize()
        assert e.status() == 0
        out.append(torch.stack(images).cpu().numpy())
    assert (out[0][0] != out[0][5]).any()
    np.testing.assert_array_equal(out[1], out[0])
    np.testing.assert_array_equal(out[2], out[0])
