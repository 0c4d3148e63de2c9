"""A particle so far out along x that its linear cell index still falls inside the grid, further
than a float16 holds in cutoffs: the list build reports it, lists nothing for it, and leaves the
other particles' lists alone."""
import os

import numpy as np
import pytest

import sph_b200
import sph_input

pytestmark = pytest.mark.gpu


def test_particle_beyond_the_float16_range_is_reported(workdir):
    n = 801  # 267 x 267 cells, 71,289 of them
    p = sph_input.write_input(os.path.join(workdir, "input"), N=(n, n), L=(1.0, 1.0), dim=2,
                              overlap=3.0, dt=1e-6)
    s = sph_b200.System(p)
    s.neighbours_search()
    s.calculate_density()
    x, want = s.field("x"), s.field("dens")
    far = x.copy()
    far[n] = 66000.5 * 3.0 / n  # row 0, cell 66,000: below 71,289, above 65,504
    s.set_field("x", far)
    with pytest.raises(sph_b200.SphError) as err:
        s.neighbours_search()
    assert err.value.status == "SPH_ERR_CELL_RANGE" and "global id %d)" % n in str(err.value)
    s.set_field("x", x)
    s.neighbours_search()
    s.calculate_density()
    assert np.array_equal(s.field("dens"), want)
    s.close()
