"""Distances of zero in FP64: a fluid particle exactly in the centre of a colloid, and two fluid
particles whose distance squared is below the smallest normal number.  Both have finite values in
the reference's formulas (a fluid particle inside a colloid takes the plain velocity difference; the
kernel at zero distance is W(0)).

Against the FP64 oracle: forces within 1e-11 of the group's scale (some 30 pairs of a few dozen
rounded operations each, 1e-14, with a margin for the cancellation of the pressure terms, a factor
of 100 here), densities within 1e-13 (a few ulps a term)."""
import os

import numpy as np
import pytest

import oracle
import sph_b200
import sph_input
from conftest import GROUPS, group_error

pytestmark = pytest.mark.gpu

N = 24
BOXES = {2: dict(N=(N, N), L=(1.0, 1.0), dim=2, coll_x=((12.0 / N, 12.0 / N),)),
         3: dict(N=(N, N, N + 2), L=(1.0, 1.0, (N + 2.0) / N), dim=3,
                 coll_x=((12.0 / N, 12.0 / N, 13.0 / N),))}


def _pair(workdir, dim, precision="fp64"):
    p = sph_input.write_input(os.path.join(workdir, "input"), overlap=3.0, dt=1e-5, N_colloids=1,
                              coll_R=3.0 / N, coll_repulsion_cuton=0.2 / N, tau_repulsion=30.0,
                              cutoff_magnetic=0.2, F0_magnetic=1e-4, omega_magnetic=6.28, **BOXES[dim])
    e, o = sph_b200.System(p, precision=precision), oracle.Oracle(p)
    rng = np.random.default_rng(3)
    fluid = e.type() == 0
    for q in "xyz"[:dim]:
        v = np.where(fluid, rng.uniform(-0.5, 0.5, fluid.size), 0.0)
        for s in (e, o):
            s.set_field("v" + q, v)
    return e, o, np.flatnonzero(fluid)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("dim", [2, 3])
def test_fluid_particle_in_the_centre_of_a_colloid(workdir, dim, precision):
    e, o, fluid = _pair(workdir, dim, precision)
    for q in "xyz"[:dim]:
        x = e.field(q)
        x[fluid[5]] = e.colloid_field("coll_" + q)[0]
        for s in (e, o):
            s.set_field(q, x)
    e.neighbours_search()
    e.calculate_forces((0.0, 0.0, 0.0))
    o.neighbours_search()
    o.calculate_forces((0.0, 0.0, 0.0))
    for name in ("force", "dcdt"):
        fields = [f for f in GROUPS[name][0] if dim == 3 or "z" not in f]
        assert all(np.isfinite(o.field(f)).all() for f in fields)
        assert all(np.isfinite(e.field(f)).all() for f in fields), name
        if precision == "fp64":
            assert group_error(e.field, o.field, fields, "max", dim) <= 1e-11, name
    e.close()
    o.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_density_of_two_particles_at_one_point(workdir, dim):
    e, o, fluid = _pair(workdir, dim)
    a, b = fluid[3], fluid[40]
    for q in "xyz"[:dim]:
        x = e.field(q)
        x[a], x[b] = (0.0, 1e-160) if q == "x" else (2.3 / N, 2.3 / N)
        for s in (e, o):
            s.set_field(q, x)
    for s in (e, o):
        s.neighbours_search()
        s.calculate_density()
    want, got = o.field("dens"), e.field("dens")
    assert np.isfinite(want).all() and want[a] > 1.2 * np.median(want)
    assert np.abs(got - want).max() <= 1e-13 * want.max()
    e.close()
    o.close()
