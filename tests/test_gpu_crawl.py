"""Steps on the nearest-region cache taken in registers (crawls), and launches that
never fill a CTA: the histories are those of full sweeps.  The scene has shared and
close faces (a stack of boxes in a slightly larger box), so that the cache keeps one
region in some places and two in others, and a beam along the walls, so that packets
creep in steps of their distance to a wall."""
import numpy as np
import pytest

from signedmcrt_b200 import presets as P, scene as S
from tests.test_gpu_parity import COUNT_KEYS

pytestmark = pytest.mark.gpu


def stack(kind):
    opt = S.mono(2.0, 0.5, 0.8, 1.38)
    arr = [S.box((2.0, 2.0, 0.5), opt, 1 + k, transform=S.invert(S.translate((0.0, 0.0, 0.75 - 0.5 * k))))
           for k in range(4)]
    arr.insert(0, S.sphere(0.2, S.mono(5.0, 0.1, 0.9, 1.45), 1, transform=S.invert(S.translate((0.3, 0.1, 0.5)))))
    arr.append(S.box((2.002, 2.002, 2.002), P.AMBIENT, 6))
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 33, 20, 7
    if kind == "wall":  # 1e-4 from a wall, parallel to it
        st.source.position = (1.0 - 1e-4, 0.2, 1.0 - 1e-5)
    return st, arr


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("kind", ["axis", "wall"])
@pytest.mark.parametrize("n", [1, 33, 80, 81, 641, 1281, 20011])
def test_crawls_follow_the_histories_of_full_sweeps(gpu, n, kind, precision):
    st, arr = stack(kind)
    out = []
    for cache in (1, 2):
        with gpu.Transport(arr, st, precision=precision, nearest_cache=cache, timeout_ms=20000) as tr:
            out.append(tr.run(n, 5))
    on, off = out
    assert on.stats["packets"] == n
    for k in COUNT_KEYS:
        assert on.stats[k] == off.stats[k], (k, on.stats[k], off.stats[k])
    # the same segment lengths summed in another order: FP64 rounding of up to ~1e6 adds
    assert np.allclose(on.jmean, off.jmean, rtol=1e-9, atol=1e-12 * off.jmean.max())


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("x", [0.0, 1.3, 2.79])
def test_modified_regions_on_the_cache_follow_full_sweeps(gpu, x, precision):
    """Revolved eggs and onions are on the cache (values that change by at most the
    distance moved): the histories are those of full sweeps."""
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 41, 30, 17
    st.grid.xmax = st.grid.ymax = st.grid.zmax = 4.0
    st.source.position = (x, 0.2, 3.9)
    out = []
    for cache in (1, 2):
        with gpu.Transport(P.setup_egg(), st, precision=precision, nearest_cache=cache, timeout_ms=20000) as tr:
            out.append(tr.run(20000, 11))
    on, off = out
    for k in COUNT_KEYS:
        assert on.stats[k] == off.stats[k], (k, on.stats[k], off.stats[k])
    assert np.allclose(on.jmean, off.jmean, rtol=1e-9, atol=1e-12 * off.jmean.max())


@pytest.mark.parametrize("kind", ["axis", "wall"])
def test_crawls_match_the_oracle_in_fp64(gpu, oracle, kind):
    st, arr = stack(kind)
    with gpu.Transport(arr, st, precision="fp64") as tr:
        g = tr.run(3001, 7)
    o = oracle.run(arr, st, nphotons=3001, seed=7, policy=oracle.device_policy("fp64", st.grid_c()))
    diff = {k: (g.stats[k], o.stats[k]) for k in COUNT_KEYS if g.stats[k] != o.stats[k]}
    assert not diff, diff


# (cells along the beam, distance from the wall): steps that are no multiple of an ulp of
# the way to the voxel face (an FP32 position, a wall that is none), inside the band of
# FP64 sweeps, up to 1.3e6 of them in a voxel of 0.1 to 0.4 cm; the last ones outside it
WALLS = [(7, 3e-7), (5, 3e-7), (5, 3.1e-7), (20, 3e-7), (9, 1.7e-7), (20, 1.3e-6), (5, 1.02e-5), (20, 1.02e-5)]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("nz,d", WALLS)
def test_long_crawls_end_at_the_voxel_face(gpu, nz, d, precision):
    """A beam along a wall steps by its distance to it, all through a voxel: the lengths
    are those of full sweeps in every voxel.  (Each packet makes 1.3 voxels' worth of
    steps, then the step cap ends it.)"""
    x = float(np.float32(0.9))
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 5, 3, nz
    st.source.position = (x, 0.2, 1.0 - 1e-5)
    arr = [S.box((2.0 * (x + d), 2.0, 2.0), S.mono(0.0, 0.0, 0.0, 1.0), 1)]
    out = []
    for cache in (1, 2):
        with gpu.Transport(arr, st, precision=precision, nearest_cache=cache, timeout_ms=60000,
                           max_trace_steps=int(1.3 * (2.0 / nz) / d)) as tr:
            out.append(tr.run(2, 5))
    on, off = out
    for k in COUNT_KEYS:
        assert on.stats[k] == off.stats[k], (k, on.stats[k], off.stats[k])
    # the same lengths summed in another order: FP64 rounding of up to 3e6 adds
    assert np.allclose(on.jmean, off.jmean, rtol=1e-9, atol=1e-12 * off.jmean.max())


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("dirx", [-1.8e-16, 1.8e-16, -1e-12, -1e-9, 1e-6])
@pytest.mark.parametrize("x,nx", [(0.0, 4), (-1 / 3, 6), (-1 / 3 + 1e-12, 6)])
def test_crawls_along_a_voxel_face(gpu, x, nx, dirx, precision):
    """A beam on a voxel face, or a rounding beside it, turned from it by as little: the cells
    are those that every step's rounded position lies in."""
    y = float(np.float32(0.9))
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = nx, 3, 5
    st.source.position, st.source.direction = (x, y, 1.0 - 1e-5), (dirx, 0.0, -1.0)
    arr = [S.box((2.0, 2.0 * (y + 3e-5), 2.0), S.mono(0.0, 0.0, 0.0, 1.0), 1)]
    out = []
    for cache in (1, 2):
        with gpu.Transport(arr, st, precision=precision, nearest_cache=cache, timeout_ms=60000) as tr:
            out.append(tr.run(2, 5))
    on, off = out
    for k in COUNT_KEYS:
        assert on.stats[k] == off.stats[k], (k, on.stats[k], off.stats[k])
    assert np.allclose(on.jmean, off.jmean, rtol=1e-9, atol=1e-12 * off.jmean.max())


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("n", [1, 11000])
def test_time_limit_in_launches_of_few_packets(gpu, n, precision):
    """The time limit ends a launch whose packets (one to 75 a CTA, up to four a warp)
    run to their end in one go, more than once, and the device goes on."""
    from signedmcrt_b200._lib import SmcrtError
    x, d = float(np.float32(0.9)), 1.7e-7
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 5, 3, 4
    st.source.position = (x, 0.2, 1.0 - 1e-5)
    arr = [S.box((2.0 * (x + d), 2.0, 2.0), S.mono(0.0, 0.0, 0.0, 1.0), 1)]
    with gpu.Transport(arr, st, precision=precision, timeout_ms=10, max_trace_steps=2097151) as tr:
        for _ in range(2):
            with pytest.raises(SmcrtError, match="time limit"):
                tr.run(n, 5)
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 5, 3, 4
    with gpu.Transport(P.box_slab(), st, precision=precision, timeout_ms=1000) as tr:
        assert tr.run(n, 5).stats["packets"] == n


def egg_settings(x=0.3):
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 41, 30, 17
    st.grid.xmax = st.grid.ymax = st.grid.zmax = 4.0
    st.source.position = (x, 0.2, 3.9)
    return st


def rigid_scene():
    opt = S.mono(10.0, 0.1, 0.9, 1.38)
    t = S.invert(S.rotate_y(30.0)) @ S.invert(S.translate((0.1, 0.2, 0.3)))
    return [S.torus(0.3, 0.1, opt, 1, transform=t), S.cylinder((-.5, -.5, 0), (.5, -.5, .2), 0.1, opt, 2),
            S.segment((-.5, .7, 0), (.5, .7, .2), opt, 3), S.box((0.3, 0.2, 0.5), opt, 4, transform=t),
            S.box((2.0, 2.0, 2.0), S.mono(1.0, 0.1, 0.8, 1.33), 5), S.box((2.002, 2.002, 2.002), P.AMBIENT, 6)]


def scene_and_settings(name):
    if name == "egg":
        return P.setup_egg(), egg_settings()
    if name == "rigid":
        st = P.benchmark_settings("box_slab")
        st.grid.nxg, st.grid.nyg, st.grid.nzg = 30, 21, 17
        return rigid_scene(), st
    st = P.benchmark_settings(name)
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 40, 33, 50
    return P.setup_simulation(st), st


def same_histories(a, b):
    for k in COUNT_KEYS:
        assert a.stats[k] == b.stats[k], (k, a.stats[k], b.stats[k])
    # the same lengths summed in another order: FP64 rounding of up to ~1e6 adds
    assert np.allclose(a.jmean, b.jmean, rtol=1e-9, atol=1e-12 * b.jmean.max())


SCENES = ["egg", "rigid", "sphere_water", "layered_vessels"]


@pytest.mark.parametrize("kernel", ["pathlength", "weight", "test"])
@pytest.mark.parametrize("name", SCENES)
def test_fp32_histories_do_not_depend_on_where_the_scene_lies(gpu, name, kernel):
    """Parameter block and device memory, cache on and off: every inlined copy of a
    region's value rounds alike, so FP32 histories are the same."""
    arr, st = scene_and_settings(name)
    out = []
    for memory, cache in ((0, 1), (0, 2), (1, 1), (1, 2)):
        with gpu.Transport(arr, st, kernel=kernel, scene_memory=memory, nearest_cache=cache, timeout_ms=20000) as tr:
            out.append(tr.run(20000, 3))
    for r in out[1:]:
        same_histories(r, out[0])


@pytest.mark.parametrize("kernel", ["pathlength", "weight"])
@pytest.mark.parametrize("name", SCENES)
def test_second_moment_on_the_cache_follows_full_sweeps(gpu, name, kernel):
    arr, st = scene_and_settings(name)
    out = []
    for cache in (1, 2):
        with gpu.Transport(arr, st, kernel=kernel, nearest_cache=cache, variance=True, timeout_ms=20000) as tr:
            out.append(tr.run_moments(20000, 3))
    same_histories(*out)
    a, b = out[0].jmean2, out[1].jmean2
    # each packet adds its FP32 lengths in the order of its history, on and off the cache;
    # the squares are summed in FP64
    assert np.allclose(a, b, rtol=1e-9, atol=1e-12 * b.max())


@pytest.mark.parametrize("name", ["box_slab", "layered_vessels"])
def test_batch_follows_full_sweeps(gpu, name):
    arr, st = scene_and_settings(name)
    n, seeds = [9001, 300], [5, 6]
    flat = S.FlatScene(arr)
    optics = np.array([[(o.mus, o.mua, o.hgg, o.n) for o in flat.optics()]] * 2)
    optics[1, :, 0] *= 0.5
    with gpu.Batch(flat, st, 2, optics=optics) as b:
        jm, _, per, _ = b.run(n, seeds)
    for i in range(2):
        own = [e for e in arr]
        for e, o in zip(own, optics[i]):
            e.opt = S.mono(*o)
        with gpu.Transport(own, st, nearest_cache=2, timeout_ms=20000) as tr:
            r = tr.run(n[i], seeds[i])
        for k in ("packets", "rng_draws", "nscatt"):
            assert per[i][k] == r.stats[k], (i, k, per[i][k], r.stats[k])
        assert np.allclose(jm[i], r.jmean, rtol=1e-9, atol=1e-12 * r.jmean.max())


@pytest.mark.parametrize("name", ["egg", "sphere_water", "layered_vessels"])
def test_adjoint_on_the_cache_follows_full_sweeps(gpu, name):
    """Random voxel weights, so that a step weighted by another cell than its own shows."""
    import torch
    arr, st = scene_and_settings(name)
    nx, ny, nz = st.grid.nxg, st.grid.nyg, st.grid.nzg
    w = torch.rand(nx * ny * nz, generator=torch.Generator().manual_seed(1), dtype=torch.float32).cuda()
    groups = np.arange(len(arr)) % 4
    out = []
    for cache in (1, 2):
        with gpu.Transport(arr, st, nearest_cache=cache, timeout_ms=20000) as tr:
            out.append(tr.adjoint(20000, 3, w.data_ptr(), None, groups, 4))
    (ga, sa), (gb, sb) = out
    for k in COUNT_KEYS:
        assert sa[k] == sb[k], (k, sa[k], sb[k])
    # FP32 sums per thread of some hundred terms (2^-24 each), of both signs and up to a
    # hundred times their sum; the packets' places on the threads differ from run to run
    assert np.all(np.abs(ga - gb) <= 1e-3 * np.abs(gb).max(axis=1, keepdims=True)), (ga, gb)


def plateau_scene(kind):
    """Overlapping regions with a box revolved off its plane, whose values are one constant
    deep inside: a crossing resolved there has no normal (0 / 0)."""
    def at(*t):
        m = S.identity()
        m[3, :3] = t
        return m
    if kind == "beam at the rim":
        return [S.cylinder((0, 0, -.3), (0, .1, .4), .2, S.mono(.5, 0., .5, 1.5), 1, transform=at(.25, .25, .25)),
                S.box((.5, 1.25, .625), S.mono(.5, 1., .9, 1.33), 2,
                      transform=at(0.3140462012492589, -0.21184131052779065, -0.4987951372882876)),
                S.revolution(S.box((1.25, .875, .875), S.mono(20., 0., .9, 1.), 3,
                                   transform=at(-0.41726337545446734, -0.48435662718498895, -0.40519797866702933)), .3),
                S.box((1.8, 1.8, 1.8), S.mono(0., 0., .5, 1.33), 4)], (0.8397171426642697, 0.8266132134794663, 0.9)
    return [S.sphere(.4, S.mono(5., 1., 0., 1.5), 1, transform=at(.5, .5, 0.)),
            S.box((1.25, .75, .75), S.mono(5., 1., .5, 1.), 2, transform=at(-.5, -.25, -.5)),
            S.torus(.4, .15, S.mono(.5, 1., .9, 1.33), 3, transform=at(0., .25, .5)),
            S.revolution(S.box((1.25, 1.125, .875), S.mono(20., .05, .5, 1.33), 4, transform=at(.5, .25, -.25)), .3),
            S.box((2., 2., 2.), S.mono(5., 0., .5, 1.33), 5), S.box((2.002, 2.002, 2.002), P.AMBIENT, 6)], (0., 0., .5)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("memory", [0, 1])
@pytest.mark.parametrize("kernel", ["pathlength", "weight", "test"])
@pytest.mark.parametrize("kind", ["beam at the rim", "beam at the axis"])
def test_directions_that_are_not_numbers_leave_the_cache(gpu, kind, kernel, memory, precision):
    """A packet refracted at a normal of 0 / 0 has no position after its next step, and no
    bound of the cache holds there: full sweeps end it, with the cache on and off."""
    arr, pos = plateau_scene(kind)
    st = P.benchmark_settings("box_slab")
    st.grid.nxg, st.grid.nyg, st.grid.nzg = 15, 37, 17
    st.source.position = pos
    out = []
    for cache in (1, 2):
        with gpu.Transport(arr, st, kernel=kernel, precision=precision, scene_memory=memory, nearest_cache=cache,
                           max_trace_steps=20000, timeout_ms=20000) as tr:
            out.append(tr.run(700, 28377))
    on, off = out
    for k in COUNT_KEYS:
        assert on.stats[k] == off.stats[k], (k, on.stats[k], off.stats[k])
    assert on.stats["kills_error"] == off.stats["kills_error"]
    assert np.allclose(on.jmean, off.jmean, rtol=1e-9, atol=1e-12 * off.jmean.max())
