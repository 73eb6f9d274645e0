"""Wireframe frames whose samples receive line plots from many triangles:
the fold's three list sizes (a thread's list, a warp's list sorted in shared
memory, a longer one) at their borders, against the oracle, bit for bit."""
import dataclasses

import numpy as np
import pytest

import cpu_oracle
import mopcuda
import scenes

pytestmark = pytest.mark.gpu


# every layer draws the same quad: 2 plots per layer on its diagonal's samples, 1 on its
# sides', so lists of n and 2n fragments around 24 (a thread's) and 512 (a warp's sort)
@pytest.mark.parametrize("layers", [1, 12, 13, 24, 25, 255, 256, 257, 512, 513])
def test_stacked_wireframe_lists(cuda_device, layers):
    rng = np.random.default_rng(layers)
    sc = scenes.small_scene(seed=5, width=61, height=43, n_meshes=2)
    oid = 100
    for k in range(layers):
        v, i = scenes._quad(-1.1, -0.8, 1.2, 0.9, 0.0, (*rng.uniform(0, 1, 3), 1.0))
        m = scenes.mat_trs((0.0, 1.0, 1.0), np.eye(3), (1.0, 1.0, 1.0))
        sc.meshes.append(scenes.Mesh(v, i, oid + k, m))
    if layers % 2:  # a filled, blended mesh between the lines (ID 0 stays solid)
        v, i = scenes._quad(-0.9, -0.9, 0.9, 0.9, 0.1, (0.2, 0.9, 0.4, 1.0))
        sc.meshes.insert(3, scenes.Mesh(v, i, 0, scenes.mat_trs((0.0, 1.0, 1.2), np.eye(3),
                                                                (1.0, 1.0, 1.0)), opacity=0.6))
    sc = dataclasses.replace(sc, wireframe=True)
    want = cpu_oracle.render(sc)
    r = mopcuda.SceneRenderer(cuda_device, sc)
    try:
        r.render()
        assert (r.object_id() == want["object_id"]).all()
        assert (r.depth().view(np.uint32) == want["depth"].view(np.uint32)).all()
        assert (r.color_full() == want["color_full"]).all()
    finally:
        r.close()
