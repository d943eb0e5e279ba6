"""The regions the nearest-region cache takes beside exact distances change by at most
the distance moved: revolved eggs and onions of shapes, on the oracle's FP64 values at
random pairs of points and at pairs across the egg's arcs."""

import numpy as np
import pytest

from signedmcrt_b200 import presets as P, scene as S

OPT = S.mono(0.0, 0.0, 0.0, 1.0)


@pytest.mark.parametrize("name", ["preset", "flat_egg", "onions"])
def test_modified_regions_are_1_lipschitz(oracle, name):
    if name == "preset":
        arr = P.setup_egg()
    elif name == "flat_egg":
        arr = [S.revolution(S.egg(2.0, 1.9, 0.4, OPT, 1), 0.3), S.revolution(S.egg(1.0, 0.2, 1.5, OPT, 2), 0.0)]
    else:
        arr = [S.onion(S.torus(1.0, 0.3, OPT, 1), 0.1), S.onion(S.revolution(S.box((0.4, 1.0, 1.0), OPT, 2), 1.0), 0.05),
               S.revolution(S.onion(S.sphere(0.5, OPT, 3), 0.2), 0.7)]
    flat = S.FlatScene(arr)
    rng = np.random.default_rng(1)
    for scale in (1e-4, 1e-2, 0.3, 3.0):
        a = rng.uniform(-5, 5, (100000, 3))
        b = a + rng.normal(size=a.shape) * scale
        near = np.concatenate([a, a * (1.0, 1e-3, 1.0)])  # half of them beside the egg's y = 0
        far = np.concatenate([b, b * (1.0, 1e-3, 1.0)])
        d = np.abs(oracle.eval_sdf(flat, near, "fp64") - oracle.eval_sdf(flat, far, "fp64"))
        step = np.linalg.norm(near - far, axis=1)[:, None]
        assert np.all(d <= step * (1 + 1e-12) + 64 * 16 * 2.0 ** -53), (d - step).max()
