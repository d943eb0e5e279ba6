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
