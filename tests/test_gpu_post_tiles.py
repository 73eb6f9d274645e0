"""The post pass at the edges of its tiles (32 pixels wide, 8 or, at SSAA 1, 32 high) for every
SSAA factor, as a frame and in a batch, against the oracle: bit for bit without vignette (a byte
map or, with fog, a threshold search), within the colour contract's 1 LSB with it (powf)."""
import dataclasses

import numpy as np
import pytest

import cpu_oracle
import mopcuda
import scenes

pytestmark = pytest.mark.gpu

P = scenes
EFFECTS = {"plain": P.POST_GAMMA | P.POST_FXAA,
           "fog": P.POST_GAMMA | P.POST_FXAA | P.POST_FOG | P.POST_TONEMAP,
           "vignette": P.POST_GAMMA | P.POST_FXAA | P.POST_VIGNETTE,
           "fog_vignette": P.POST_GAMMA | P.POST_FXAA | P.POST_FOG | P.POST_VIGNETTE}


def _scene(w, h, ssaa, effects):
    sc = scenes.small_scene(seed=w + h, width=w, height=h, ssaa=ssaa, n_meshes=4)
    return dataclasses.replace(sc, post_effects=EFFECTS[effects],
                               fog=((0.5, 0.6, 0.8, 1.0), 0.9, 1.0))


def _same(got, want, effects):
    d = np.abs(got.astype(np.int32) - want.astype(np.int32))
    assert d.max() <= (1 if "vignette" in effects else 0), (int(d.max()), int((d > 0).sum()))


@pytest.mark.parametrize("effects", list(EFFECTS))
@pytest.mark.parametrize("ssaa", [1, 2, 3, 4])
@pytest.mark.parametrize("w,h", [(1, 1), (31, 33), (32, 32), (33, 31), (65, 8), (64, 9), (97, 65)])
def test_frame_post(cuda_device, w, h, ssaa, effects):
    sc = _scene(w, h, ssaa, effects)
    want = cpu_oracle.render(sc)
    r = mopcuda.SceneRenderer(cuda_device, sc)
    try:
        r.render()
        _same(r.color_full(), want["color_full"], effects)
        _same(r.color(), want["color"], effects)
    finally:
        r.close()


@pytest.mark.parametrize("effects", list(EFFECTS))
def test_batch_post(cuda_device, effects):
    sc = _scene(64, 48, 1, effects)
    views = [scenes.View(w, h, s, sc.eye, sc.target, fov_deg=sc.fov_deg, near=sc.near, far=sc.far)
             for w, h, s in ((31, 33, 1), (64, 32, 1), (33, 9, 2), (40, 25, 3), (16, 16, 4),
                             (65, 64, 1), (32, 8, 2))]
    b = mopcuda.BatchRenderer(cuda_device, sc, views)
    try:
        b.render()
        for i, v in enumerate(views):
            want = cpu_oracle.render(scenes.scene_for_view(sc, v))
            _same(b.read(i, mopcuda.BATCH_COLOR), want["color_full"], effects)
            _same(b.read(i, mopcuda.BATCH_PRESENTED), want["color"], effects)
    finally:
        b.close()
