"""Records above the small-record limits against the oracle, bit for bit: boxes around the widths
where the raster changes its shape (one chunk of 32 samples, 4 chunks, bands of 8 chunks by 8
rows), smooth and flat, and a stack of full-screen triangles that outgrows the chunk table."""
import dataclasses
import math

import numpy as np
import pytest

import cpu_oracle
import mopcuda
import scenes

pytestmark = pytest.mark.gpu

W, H, FOV, DIST = 333, 177, 50.0, 5.0


def _scene(rng, boxes, smooth):
    """One slanted triangle per (x, y, w, h) box in pixels, at slightly different depths."""
    sc = scenes.Scene("large", W, H, 1, eye=(0.0, 0.0, DIST), target=(0.0, 0.0, 0.0), fov_deg=FOV,
                      near=0.1, far=50.0, smooth=smooth)
    sc.lights.append(scenes.Light(scenes.LIGHT_DIRECTIONAL, direction=(-0.3, -0.6, -1.0)))
    sc.lights.append(scenes.Light(scenes.LIGHT_POINT, position=(1.0, 1.0, 3.0), intensity=6.0))
    u = 2.0 * DIST * math.tan(math.radians(FOV) / 2) / H  # world units of a pixel at z = 0
    for k, (x, y, w, h) in enumerate(boxes):
        a, b = rng.uniform(0.0, 1.0, 2)
        px = np.array([[x, y + a * h], [x + w, y], [x + b * w, y + h]]) + rng.uniform(-0.4, 0.4, 2)
        z = rng.uniform(-0.3, 0.3, 3)
        s = (DIST - z) / DIST
        pos = np.stack([(px[:, 0] - W / 2) * u * s, (H / 2 - px[:, 1]) * u * s, z], 1)
        nrm = np.tile(np.array([0.1, 0.2, 0.97]), (3, 1))
        col = np.c_[rng.uniform(0.1, 1.0, (3, 3)), np.ones(3)]
        v = scenes._pack(pos, nrm, col, np.zeros((3, 2)))
        sc.meshes.append(scenes.Mesh(v, np.array([0, 1, 2, 0, 2, 1], np.uint32), k + 1,
                                     scenes.mat_identity(), 0.3, 0.4))
    return sc


def _check(dev, sc):
    want = cpu_oracle.render(sc)
    r = mopcuda.SceneRenderer(dev, sc)
    try:
        r.render()
        assert (r.object_id() == want["object_id"]).all()
        assert (r.depth().view(np.uint32) == want["depth"].view(np.uint32)).all()
        assert (r.color_full() == want["color_full"]).all()
    finally:
        r.close()


@pytest.mark.parametrize("smooth", [True, False])
@pytest.mark.parametrize("w", [4, 31, 32, 33, 64, 127, 128, 129, 255, 256, 257, 320])
def test_large_record_widths(cuda_device, w, smooth):
    rng = np.random.default_rng(w)
    boxes = [(float(rng.uniform(-20, W - w + 20)), float(rng.uniform(-10, H - h + 10)), w, h)
             for h in (1, 7, 8, 9, 33, 64, 65, 150)]
    _check(cuda_device, _scene(rng, boxes, smooth))


@pytest.mark.parametrize("ssaa", [1, 2])
def test_chunk_table_runs_out(cuda_device, ssaa):
    rng = np.random.default_rng(ssaa)
    boxes = [(-40.0, -30.0, W + 80, H + 60)] * 24 + [(10.0 * k, 3.0, 60, 150) for k in range(20)]
    _check(cuda_device, dataclasses.replace(_scene(rng, boxes, True), ssaa=ssaa))
