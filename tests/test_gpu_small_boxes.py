"""Contexts of few particles take other forms of the list build (two warps per cell) and the density
pass (eight entries side by side) than large ones.  The sums are the same, term for term: a box alone gives the bits it gives among
enough copies of itself to take the forms for many particles."""
import os

import numpy as np
import pytest

import sph_b200
import sph_input

pytestmark = pytest.mark.gpu

BOXES = {
    # fluid only, periodic, with a body force
    "kolmogorov": dict(N=(64, 64), L=(1.0, 1.0), dim=2, overlap=4.0, ext_force_type=2,
                       ext_force=(1.0, 0.0), dt=5e-5),
    # walls and colloids: warps that mix the forms, ragged sides
    "channel": dict(N=(93, 67), L=(1.0, 67.0 / 93.0), dim=2, overlap=3.0, wall=1,
                    Vwall_bottom=-0.2, Vwall_top=0.2, dt=2e-5, N_colloids=2, coll_R=4.0 / 93,
                    coll_x=((0.3, 0.3), (0.7, 0.4)), coll_repulsion_cuton=0.2 / 93,
                    F0_repulsion=1e-3, tau_repulsion=3.0, cutoff_magnetic=20.0 / 93,
                    F0_magnetic=1e-4, omega_magnetic=6.28),
    # 3D, cells of 27 to 64 particles
    "couette3d": dict(N=(25, 19, 31), L=(25.0 / 31, 19.0 / 31, 1.0), dim=3, overlap=3.0, wall=1,
                      Vwall_bottom=-0.5, Vwall_top=0.5, dt=2e-5),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name,copies", [("kolmogorov", 30), ("channel", 20), ("couette3d", 16)])
def test_a_box_alone_and_among_many_gives_the_same_bits(workdir, name, copies, precision):
    p = sph_input.write_input(os.path.join(workdir, "input"), **BOXES[name])
    dim = BOXES[name]["dim"]
    alone = sph_b200.System(p, precision=precision)
    n = alone.N
    rng = np.random.default_rng(7)
    fluid = alone.type() == 0
    dx = BOXES[name]["L"][0] / BOXES[name]["N"][0]
    start = {q: alone.field(q) + np.where(fluid, rng.uniform(-0.2, 0.2, n) * dx, 0.0)
             for q in "xyz"[:dim]}
    start.update({"v" + q: np.where(fluid, rng.uniform(-0.5, 0.5, n), 0.0) for q in "xyz"[:dim]})
    many = sph_b200.System([p] * copies, precision=precision)
    for s, k in ((alone, 1), (many, copies)):
        for q, v in start.items():
            s.set_field(q, np.tile(v, k))
        s.initial_forces()
        s.step(4)
        s.synchronize()
    for q in list(start) + ["fx", "fy", "dens", "press", "cxx", "cxy", "dcdt_xy"]:
        a, b = alone.field(q), many.field(q)
        assert np.array_equal(a, b[:n]) and np.array_equal(a, b[-n:]), q
    alone.close()
    many.close()


def test_colloids_alone_and_beside_larger_ones_give_the_same_bits(workdir):
    """The colloid pass takes as many threads a block as the largest colloid of the context has
    particles, up to 256: about 28, 79 and 201 particles (64, 128 and 256 threads)."""
    paths, alone = [], []
    for k, R in enumerate((3.0, 5.0, 8.0)):
        spec = dict(N=(96, 80), L=(1.2, 1.0), dim=2, overlap=3.0, dt=2e-5, N_colloids=2,
                    coll_R=R / 80, coll_x=((0.3, 0.31), (0.8, 0.6)), coll_repulsion_cuton=0.2 / 80,
                    F0_repulsion=1e-3, tau_repulsion=10.0, cutoff_magnetic=8.0 / 80,
                    F0_magnetic=1e-4, omega_magnetic=6.28)
        paths.append(sph_input.write_input(os.path.join(workdir, "input%d" % k), **spec))

    def run(some):
        s = sph_b200.System(some)
        x, y, fluid = s.field("x"), s.field("y"), s.type() == 0
        s.set_field("vx", np.where(fluid, 0.5 * np.sin(9.0 * x + 14.0 * y), 0.0))
        s.set_field("vy", np.where(fluid, 0.5 * np.cos(11.0 * x - 8.0 * y), 0.0))
        s.initial_forces()
        s.step(3)
        s.synchronize()
        out = [s.colloid_field(q) for q in ("fx_colloid", "fy_colloid", "tz_colloid", "coll_x",
                                            "coll_vx", "coll_omegaz")]
        s.close()
        return np.stack(out)

    for n in (1, 2, 3):
        alone.append(run(paths[n - 1:n]))
        assert np.array_equal(run(paths[:n]), np.concatenate(alone, axis=1))
