"""The render's tiles (regions left out where another is nearer over the whole tile, a
thread's column of voxels sharing its x and y terms): the image is that of every
region's value at every voxel, at the edges of tiles and for every kind of region
(plain shapes; rotated ones, folds and modifiers, which are never left out)."""
import math

import numpy as np
import pytest

from signedmcrt_b200 import presets as P, scene as S

pytestmark = pytest.mark.gpu
OPT = S.mono(0.0, 0.0, 0.0, 1.0)


def mixed():
    sph = S.sphere(0.3, OPT, 1, transform=S.invert(S.translate((0.4, -0.3, 0.2))))
    box = S.box((0.3, 0.2, 0.5), OPT, 2, transform=S.invert(S.rotate_y(30.0)) @ S.invert(S.translate((0.2, 0.0, 0.0))))
    fold = S.model([S.sphere(0.25, OPT, 3), S.box((0.3, 0.3, 0.3), OPT, 3)], S.smooth_union, 0.1)
    tw = S.twist(S.box((0.2, 0.3, 0.8), OPT, 4), 2.0)
    cap = S.capsule((-0.9, 0.5, 0.1), (0.9, 0.5, 0.2), 0.05, OPT, 5)
    return [sph, box, fold, tw, cap]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("samples", [(1, 1, 1), (16, 8, 16), (17, 9, 33), (15, 7, 1), (40, 23, 50), (1, 64, 5)])
@pytest.mark.parametrize("name", ["mixed", "layered", "sphere_water"])
def test_render_tiles_equal_the_point_values(gpu, name, samples, precision):
    arr = {"mixed": mixed, "layered": P.layered_vessels, "sphere_water": P.sphere_water}[name]()
    flat, ext = S.FlatScene(arr), (1.1, 0.9, 2.5)
    img = gpu.render(flat, samples, ext, precision)
    ax = [(np.arange(1, n + 1) - (n + 1) // 2) * (e / ((n + 1) // 2)) for n, e in zip(samples, ext)]
    pts = np.stack(np.meshgrid(*ax, indexing="ij"), axis=-1).reshape(-1, 3)
    want = gpu.eval_sdf(flat, pts, precision).min(axis=1).reshape(samples)
    # the point probe is built with FMA contraction: a few roundings of values up to ~4,
    # and 0.05 of slope for twist's trigonometric terms in FP32
    tol = 64 * 4 * (2.0 ** -24 if precision == "fp32" else 2.0 ** -53) + 2.0 ** -23 * np.abs(want)
    assert np.all(np.abs(img.astype(np.float64) - want) <= tol), np.abs(img - want).max()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_render_passes_over_a_nan_region(gpu, precision):
    """A degenerate cone's values are NaN everywhere; behind the first region they are
    no minimum, wherever the first region is left out."""
    far = S.sphere(0.1, OPT, 1, transform=S.invert(S.translate((-0.9, 0.0, 0.0))))
    near = S.sphere(0.2, OPT, 2, transform=S.invert(S.translate((0.8, 0.0, 0.0))))
    cone = S.cone((0.0, 0.0, 0.0), (0.0, 0.0, 0.0), 0.1, 0.1, OPT, 3)
    samples, ext = (64, 17, 33), (1.0, 1.0, 1.0)
    img = gpu.render(S.FlatScene([far, cone, near]), samples, ext, precision)
    assert np.array_equal(img, gpu.render(S.FlatScene([far, near]), samples, ext, precision))


# both sides of the rule that picks tiles or single voxels: whole and partial tiles,
# slices and rods, images with too few tiles
SIZES = [(96, 64, 160), (95, 63, 159), (16, 200, 256), (161, 8, 300), (33, 17, 700), (1, 300, 200), (300, 1, 200),
         (200, 300, 1), (5000, 1, 1), (64, 64, 64)]


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("samples", SIZES)
@pytest.mark.parametrize("name", ["mixed", "layered", "sphere_water"])
def test_render_of_any_shape_equals_the_point_values(gpu, name, samples, precision):
    test_render_tiles_equal_the_point_values(gpu, name, samples, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("samples", [(1, 1024, 1024), (1024, 1, 1024), (1024, 1024, 1)])
def test_a_slice_costs_less_than_a_slab(gpu, samples, precision):
    """A slice of 2^20 voxels costs well under a slab eight voxels thick: a slice computed
    in whole tiles (15 of 16 voxels padding) costs the same as the slab."""
    import torch
    flat, ext = S.FlatScene(P.layered_vessels()), (1.0, 1.0, 0.605)

    def us(n):
        img = torch.empty(int(np.prod(n)), dtype=torch.float32, device="cuda")
        s = torch.cuda.current_stream().cuda_stream
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t = []
        for _ in range(12):
            a.record()
            gpu.render_device(flat, n, ext, img.data_ptr(), precision=precision, stream=s)
            b.record()
            torch.cuda.synchronize()
            t.append(1e3 * a.elapsed_time(b))
        return sorted(t[3:])[4]

    slab = tuple(8 if k == 1 else k for k in samples)
    assert us(samples) < 0.7 * us(slab)
