"""Triangles find their draw among draws of one or two triangles and runs of empty draws: the
oracle's image, bit for bit, and no time for the draws that draw nothing."""
import numpy as np
import pytest

import cpu_oracle
import mopcuda
import scenes

pytestmark = pytest.mark.gpu


def _scene(empty, tiny):
    """A few meshes with `empty` draws of no triangles after two of them, where a warp's triangles
    straddle the run, and `tiny` draws of one or two triangles."""
    rng = np.random.default_rng(7)
    sc = scenes.small_scene(seed=3, width=96, height=72, n_meshes=5)
    v, i = scenes._quad(-0.2, -0.2, 0.2, 0.2, 0.0, (0.3, 0.7, 0.9, 1.0))

    def mesh(idx, oid):
        m = scenes.mat_trs(rng.uniform(-1.0, 1.0, 3), np.eye(3), (1.0, 1.0, 1.0))
        return scenes.Mesh(v, idx, oid, m)

    out = []
    for k, base in enumerate(sc.meshes):
        out.append(base)
        if k < 2:
            out.append(mesh(i, 500 + k))
            out += [mesh(i[:0], 600 + k)] * empty
    out += [mesh(i[:3 + 3 * (k % 2)], 1000 + k) for k in range(tiny)]
    sc.meshes[:] = out
    return sc


@pytest.mark.parametrize("empty,tiny", [(0, 0), (1, 3), (3, 31), (4, 33), (5, 65), (40, 7)])
def test_draws_found(cuda_device, empty, tiny):
    sc = _scene(empty, tiny)
    want = cpu_oracle.render(sc)
    r = mopcuda.SceneRenderer(cuda_device, sc)
    try:
        r.render()
        assert (r.object_id() == want["object_id"]).all()
        assert (r.depth().view(np.uint32) == want["depth"].view(np.uint32)).all()
        assert (r.color_full() == want["color_full"]).all()
    finally:
        r.close()


def test_empty_draws_cost_no_setup(cuda_device):
    """40,000 empty draws: a lane stepping over them takes about 0.2 us for each (8.8 ms); its
    search is 15 loads, tens of microseconds at most with the launches around it."""
    r = mopcuda.SceneRenderer(cuda_device, _scene(20000, 0))
    cuda_device.set_stage_timing(True)
    try:
        ms = []
        for _ in range(5):
            r.render()
            ms.append(cuda_device.stage_times()["setup_clip"])
        assert min(ms) < 1.0, ms
    finally:
        cuda_device.set_stage_timing(False)
        r.close()
