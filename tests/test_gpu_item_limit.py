"""A frame whose large records have more rows than their numbering holds (2^32) is refused, and
none of its lists is walked: an offset past 2^32 carries into the slot count, so a slot may hold
what an earlier frame left there.  264,000 triangles from the bottom to the top of a column 40
samples wide and 16,384 high (the largest framebuffer) have 4.30e9 rows.  The next frame is the
oracle's."""
import dataclasses

import numpy as np
import pytest

import cpu_oracle
import mopcuda
import scenes

pytestmark = pytest.mark.gpu

TRIS, HEIGHT = 264000, 16384


def _column(opacity):
    sc = scenes.Scene("column", 40, HEIGHT, 1, eye=(0.0, 0.0, 5.0), target=(0.0, 0.0, 0.0),
                      fov_deg=50.0, near=0.1, far=50.0, smooth=False)
    sc.lights.append(scenes.Light(scenes.LIGHT_DIRECTIONAL, direction=(-0.3, -0.6, -1.0)))
    pos = np.array([[-0.002, -2.32, 0.0], [0.002, -2.32, 0.0], [0.0, 2.32, 0.0]])
    # 2 * 5 * tan(25 deg) is the frame's height at the triangles' distance
    assert TRIS * (HEIGHT * 4.64 / (10.0 * np.tan(np.radians(25.0))) - 2.0) > 2.0 ** 32
    v = scenes._pack(pos, np.tile([0.0, 0.0, 1.0], (3, 1)), np.ones((3, 4)), np.zeros((3, 2)))
    i = np.tile(np.array([0, 1, 2], np.uint32), TRIS)
    sc.meshes.append(scenes.Mesh(v, i, 1, scenes.mat_identity(), opacity=opacity))
    return sc


def _refused(e):
    """The code, and a text that names every list that can have outgrown its numbering."""
    assert e.value.code == mopcuda.EUNSUPPORTED
    assert all(w in str(e.value) for w in ("large", "blended", "wireframe")), str(e.value)


def _next_frame_is_right(dev):
    sc = scenes.small_scene(seed=5, width=61, height=43, n_meshes=4)
    want = cpu_oracle.render(sc)
    r = mopcuda.SceneRenderer(dev, sc)
    try:
        r.render()
        assert (r.object_id() == want["object_id"]).all()
        assert (r.color_full() == want["color_full"]).all()
    finally:
        r.close()


@pytest.mark.parametrize("opacity", [1.0, 0.5])
def test_frame_past_the_numbering(cuda_device, opacity):
    r = mopcuda.SceneRenderer(cuda_device, _column(opacity))
    try:
        with pytest.raises(mopcuda.MopCudaError) as e:
            r.render()
        _refused(e)
    finally:
        r.close()
    _next_frame_is_right(cuda_device)


def test_batch_past_the_numbering(cuda_device):
    sc = _column(1.0)
    v = scenes.View(sc.width, sc.height, 1, sc.eye, sc.target, fov_deg=sc.fov_deg, near=sc.near,
                    far=sc.far)
    small = dataclasses.replace(v, width=64, height=48)
    b = mopcuda.BatchRenderer(cuda_device, sc, [small, v])
    try:
        with pytest.raises(mopcuda.MopCudaError) as e:
            b.render()
        _refused(e)
    finally:
        b.close()
    _next_frame_is_right(cuda_device)
