"""The server admits by its estimate of a request's device memory: what it estimates for one
request is what the slot that served it holds.

Every buffer is allocated with half its size and 4 KiB to spare, so a slot holds 1.5 times what
its launch asked for; the pools' spare entries (4,096 of each), the launch's tables and that
4 KiB per buffer come to less than 2 MiB."""
import dataclasses

import numpy as np
import pytest
import torch

import mopcuda
import scenes

pytestmark = pytest.mark.gpu


def _hidden(sc):
    """The scene with as many triangles again behind the camera: the pools are sized for half of
    a scene in view, and a launch that needs more runs again with larger ones."""
    eye, to = np.asarray(sc.eye), np.asarray(sc.target)
    tris = sum(m.indices.size for m in sc.meshes) // 3
    v, i = scenes.icosphere(5, 1.0, (0.5, 0.6, 0.7, 1.0))
    at = eye + 40.0 * (eye - to) / np.linalg.norm(eye - to)
    for k in range(tris // (i.size // 3) + 1):
        sc.meshes.append(scenes.Mesh(v, i, 5000 + k, scenes.mat_trs(at, np.eye(3), (1.0,) * 3)))
    return sc


def _scene(kind):
    if kind == "triangles":
        sc = scenes.config2(seed=2, width=64, height=64, ssaa=1, instances=0, tex_size=64)
        v, i = scenes.icosphere(5, 1.0, (0.5, 0.6, 0.7, 1.0))
        for k in range(40):
            m = scenes.mat_trs((float(k % 8) - 4.0, 1.0, float(k // 8) - 2.0), np.eye(3),
                               (0.4, 0.4, 0.4))
            sc.meshes.append(scenes.Mesh(v, i, 100 + k, m))
        return sc
    sc = scenes.config2(seed=2, width=1280, height=720, ssaa=2, instances=4, tex_size=64)
    if kind == "blended":
        sc.meshes[-1] = dataclasses.replace(sc.meshes[-1], opacity=0.5, blend_mode=1)
    return dataclasses.replace(sc, wireframe=kind == "wireframe")


@pytest.mark.parametrize("kind", ["plain", "triangles", "blended", "wireframe"])
def test_estimate_is_what_a_slot_holds(cuda_device, kind):
    sc = _hidden(_scene(kind))
    rs = mopcuda.ResidentScene(cuda_device, sc)
    srv = mopcuda.Server(cuda_device, hbm_budget=64 << 30, max_views=1, max_inflight=1)
    try:
        v = scenes.View(sc.width, sc.height, sc.ssaa, sc.eye, sc.target, fov_deg=sc.fov_deg,
                        near=sc.near, far=sc.far)
        # a page-locked destination: the copy needs no staging
        out = torch.empty((sc.height, sc.width, 4), dtype=torch.uint8, pin_memory=True).numpy()
        srv.wait(srv.submit_render(srv.add_scene(rs), v, out=out))
        srv.drain()
        st = srv.stats()
        assert st["reruns"] == 0 and st["failed"] == 0
        estimate, held = st["peak_inflight_bytes"], st["device_bytes"] / 1.5
        assert estimate > 32 << 20  # the fixed part is small beside it
        assert estimate <= held <= estimate + (2 << 20), (estimate, held)
    finally:
        srv.close()
        rs.close()
