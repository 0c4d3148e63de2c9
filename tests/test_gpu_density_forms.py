"""The launch geometry of the density pass on both sides of the particle count below which 64, 128
and 256 threads per block are one form: the bits of every geometry above it, what the tuner times
below it, and which contexts share a cached choice."""
import json
import os

import numpy as np
import pytest

import sph_b200
import sph_input

pytestmark = pytest.mark.gpu


def _box(workdir, N, precision, overlap=3.0, **over):
    p = os.path.join(workdir, "input_" + "x".join(map(str, N)))
    dx = 1.0 / N[0]
    sph_input.write_input(p, **dict(dict(N=N, L=tuple(n * dx for n in N), dim=len(N),
                                         overlap=overlap, dt=1e-6), **over))
    return sph_b200.System(p, precision=precision)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("N,overlap", [((352, 345), 4.0), ((52, 47, 52), 3.0)])
def test_geometries_give_identical_bits_in_large_contexts(workdir, N, overlap, precision):
    out = []
    for tpc, blk in [(32, 128), (16, 64), (32, 256), (16, 0)]:
        s = _box(workdir, N, precision, overlap, wall=1, Vwall_bottom=-0.3, Vwall_top=0.3)
        assert s.N > 113664  # 24 warps on each of 148 multiprocessors
        rng = np.random.default_rng(1)
        fluid = s.type() == 0
        for q in "xyz"[:len(N)]:
            s.set_field(q, s.field(q) + np.where(fluid, rng.uniform(-0.2, 0.2, s.N) / N[0], 0.0))
        s.set_tuning(tpc, blk)
        s.step(3)
        s.synchronize()
        out.append([s.field(f) for f in ("x", "vy", "fx", "fy", "dens", "press", "cxy")])
        s.close()
    for r in out[1:]:
        for a, b in zip(out[0], r):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("N,density_launches", [((250, 250), 2), ((265, 265), 4)])
def test_tuner_times_each_form_once(workdir, N, density_launches):
    """62,500 particles (FP64 line: 66,304): the tile pass and one per-particle form; 70,225: the
    tile pass and three block sizes.  Each is launched eleven times, as are the two list builds."""
    s = _box(workdir, N, "fp64")
    s.neighbours_search()
    s.synchronize()
    before = s.kernel_launches()
    choice = s.autotune()
    assert s.kernel_launches() - before == 11 * (2 + density_launches)
    assert density_launches == 4 or choice["density_block"] in (0, 128)
    s.close()


def test_cached_choices_are_shared_by_like_contexts_only(workdir):
    cache = os.path.join(workdir, "tune.json")
    keys = []
    for N, precision in [((250, 250), "fp64"), ((265, 265), "fp64"), ((250, 250), "mixed"),
                         ((265, 265), "mixed"), ((251, 249), "fp64")]:
        s = _box(workdir, N, precision)
        s.autotune(cache)
        s.close()
        keys.append(len(json.load(open(cache))))
    # one bucket of sizes; FP64 on both sides of its line, mixed on one side of its own
    assert keys == [1, 2, 3, 3, 3]
