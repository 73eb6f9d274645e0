"""Fog with vignette gives the bytes that the double-precision pow gives: the single-precision
one settles a byte only away from a rounding boundary.  The reference here is the same sequence
of float operations in numpy on the frame's own unprocessed colours and depths."""
import dataclasses

import numpy as np
import pytest

import mopcuda
import scenes

pytestmark = pytest.mark.gpu

F = np.float32
W, H = 1280, 720


def _frame(dev, sc):
    r = mopcuda.SceneRenderer(dev, sc)
    try:
        r.render()
        return r.color_full(), r.depth()
    finally:
        r.close()


def _post(raw, depth, effects, fog):
    colour, near, far = fog
    fog_range = F(far) - F(near)
    factor = np.clip((depth - F(near)) / fog_range, F(0), F(1))[..., None]
    v = raw[..., :3].astype(F) / F(255)
    v = v + (np.array(colour[:3], F) - v) * factor
    if effects & scenes.POST_TONEMAP:
        v = v / (v + F(1))
    x = np.maximum(v, F(0))
    p = (x.astype(np.float64) ** np.float64(F(1) / F(2.4))).astype(F)
    v = np.where(x <= F(0.0031308), x * F(12.92), F(1.055) * p - F(0.055))
    cx, cy = F(W) * F(0.5), F(H) * F(0.5)
    dx, dy = np.arange(W, dtype=F) - cx, (np.arange(H, dtype=F) - cy)[:, None]
    dist = np.sqrt(dx * dx + dy * dy) / np.sqrt(cx * cx + cy * cy)
    vg = np.maximum(F(1) - dist * dist * F(0.5), F(0))
    v = np.clip(v * vg[..., None], F(0), F(1))
    assert v.dtype == F
    return (v * F(255) + F(0.5)).astype(np.uint8)


@pytest.mark.parametrize("tonemap", [0, scenes.POST_TONEMAP])
@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_fog_vignette_bytes(cuda_device, seed, tonemap):
    rng = np.random.default_rng(seed)
    sc = scenes.config2(seed, W, H, 1, 24, tex_size=128, n_textures=2)
    raw, depth = _frame(cuda_device, dataclasses.replace(sc, post_effects=0))
    near = float(rng.uniform(0.9, 0.99))
    top = 4.0 if seed == 4 else 1.0  # fog brighter than white, cut back by the vignette
    fog = (tuple(rng.uniform(0.0, top, 3)) + (1.0,), near, float(rng.uniform(near + 0.005, 1.0)))
    effects = scenes.POST_GAMMA | scenes.POST_VIGNETTE | scenes.POST_FOG | tonemap
    got, same = _frame(cuda_device, dataclasses.replace(sc, post_effects=effects, fog=fog))
    assert (same == depth).all()
    want = _post(raw, depth, effects, fog)
    differ = got[..., :3] != want
    assert not differ.any(), (int(differ.sum()), np.argwhere(differ)[:4])
