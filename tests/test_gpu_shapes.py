"""Plain shapes: a single box, sphere or capsule whose transform only translates is
evaluated without the affine map (RegionShape).  Its value is that of the general
path, bit for bit: the same primitive as both children of a union is folded by the
general path, and min(d, d) = d."""
import dataclasses

import numpy as np
import pytest

from signedmcrt_b200 import scene as S

pytestmark = pytest.mark.gpu
OPT = S.mono(0.0, 0.0, 0.0, 1.0)
SHAPES = {
    "box": lambda t: S.box((1.0, 0.5, 0.01), OPT, 1, transform=t),
    "sphere": lambda t: S.sphere(0.37, OPT, 1, transform=t),
    "capsule": lambda t: S.capsule((-0.9, 0.1, 0.2), (0.9, 0.1, -0.1), 0.05, OPT, 1, transform=t),
}


def points(q, t):
    """Random points, and points on and beside the faces, edges and corners q away from the centre."""
    rng = np.random.default_rng(3)
    u = np.concatenate([rng.uniform(-2, 2, (4000, 3)), rng.uniform(-0.1, 0.1, (1000, 3))])
    ax = [np.array([-h, -h - 1e-9, -h + 1e-9, 0.0, h, h + 1e-9, h - 1e-9, h + 0.3]) for h in q]
    g = np.stack(np.meshgrid(*ax, indexing="ij"), axis=-1).reshape(-1, 3)
    return np.concatenate([u, g]) + np.asarray(t)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("t", [(0.0, 0.0, 0.0), (0.25, -0.4, 0.111)])
@pytest.mark.parametrize("name", list(SHAPES))
def test_plain_shape_is_the_general_path_bit_for_bit(gpu, name, t, precision):
    prim = SHAPES[name](S.invert(S.translate(t)))
    q = (0.5, 0.25, 0.005) if name == "box" else (0.37, 0.37, 0.37) if name == "sphere" else (0.9, 0.05, 0.05)
    pts = points(q, t)
    out = gpu.eval_sdf(S.FlatScene([prim, S.model([prim, prim], S.union)]), pts, precision)
    assert np.array_equal(out[:, 0], out[:, 1])


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("name", list(SHAPES))
def test_non_finite_points_and_parameters_take_the_general_path(gpu, name, precision):
    nan, inf, ax = np.nan, np.inf, (-1.3, 0.0, 0.004, 1.3)
    pts = np.array([p for a in ax for b in ax for x in (nan, inf, -inf)
                    for p in ((x, a, b), (a, x, b), (a, b, x), (x, x, a))] + [(nan, nan, nan)])
    prim = SHAPES[name](S.invert(S.translate((0.1, 0.0, 0.0))))
    bad = [dataclasses.replace(prim, params=tuple(x if i == k else q for i, q in enumerate(prim.params)))
           for k in range(len(prim.params)) for x in (nan, inf)]
    for p, at in [(prim, pts)] + [(b, points((0.5, 0.25, 0.005), (0.1, 0.0, 0.0))) for b in bad]:
        out = gpu.eval_sdf(S.FlatScene([p, S.model([p, p], S.union)]), at, precision)
        assert np.array_equal(out[:, 0], out[:, 1], equal_nan=True)
