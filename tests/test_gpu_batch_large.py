"""Large records in batches, at the widths where the raster changes its shape (one chunk of 32
samples, 4 chunks, bands of 8 chunks by 8 rows): views of several sizes, so that a warp's queue
goes from one view's chunks to another's, chunk tables behind odd-sized views, and views that
outgrow their table, each against the oracle's frame, bit for bit."""
import numpy as np
import pytest

import cpu_oracle
import mopcuda
import scenes
from test_gpu_large_raster import DIST, FOV, H, W, _scene

pytestmark = pytest.mark.gpu

SIZES = [(W, H, 1), (1, 1, 1), (33, 17, 1), (W, H, 2), (129, 64, 1), (257, 9, 1), (65, 63, 2),
         (320, 177, 1)]


def _check(dev, sc):
    views = [scenes.View(w, h, s, (0.02 * k, 0.0, DIST), (0.0, 0.0, 0.0), fov_deg=FOV, near=0.1,
                         far=50.0) for k, (w, h, s) in enumerate(SIZES)]
    b = mopcuda.BatchRenderer(dev, sc, views)
    try:
        b.render()
        for k, v in enumerate(views):
            want = cpu_oracle.render(scenes.scene_for_view(sc, v))
            assert (b.read(k, mopcuda.BATCH_IDS) == want["object_id"]).all(), SIZES[k]
            assert (b.read(k, mopcuda.BATCH_COLOR) == want["color_full"]).all(), SIZES[k]
    finally:
        b.close()


@pytest.mark.parametrize("smooth", [True, False])
@pytest.mark.parametrize("w", [31, 33, 64, 128, 129, 256, 257, 320])
def test_widths(cuda_device, w, smooth):
    rng = np.random.default_rng(w)
    boxes = [(float(rng.uniform(-20, W - w + 20)), float(rng.uniform(-10, H - h + 10)), w, h)
             for h in (1, 8, 9, 64, 65, 150)]
    _check(cuda_device, _scene(rng, boxes, smooth))


def test_full_tables(cuda_device):
    rng = np.random.default_rng(5)
    boxes = [(-40.0, -30.0, W + 80, H + 60)] * 24 + [(10.0 * k, 3.0, 60, 150) for k in range(20)]
    _check(cuda_device, _scene(rng, boxes, True))
