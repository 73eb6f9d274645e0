"""A device's first environment, which uploads the sample tables, gives the maps that a later
one gives: the same bytes from the tables already there."""
import numpy as np
import pytest

import mopcuda

pytestmark = pytest.mark.gpu


def _maps(dev, env):
    if env is None:
        dev.ibl_procedural_sky((0.3, 0.8, 0.4), 3.0, 0.3)
    else:
        dev.ibl_from_env(env)
    return dev.ibl_maps()


@pytest.mark.parametrize("kind", ["sky", "panorama"])
def test_first_environment_equals_the_second(kind):
    env = None
    if kind == "panorama":
        env = np.random.default_rng(3).uniform(0.0, 4.0, (64, 128, 4)).astype(np.float32)
    dev = mopcuda.Device(0)
    try:
        first, second = _maps(dev, env), _maps(dev, env)
        assert np.isfinite(first["irr"]).all() and first["irr"].any()
        for k in ("irr", "pf", "brdf"):
            assert (first[k].view(np.uint32) == second[k].view(np.uint32)).all(), k
    finally:
        dev.close()
