"""The list build where it can go wrong: cells of 0 (never filled), 1, 15 to 17, 31 to 33, 48 and
70 particles side by side, so that rows of neighbour cells end anywhere in a chunk of 32 and rounds
of particles are full, short or empty; three wide cells per axis, where a row wraps on both sides
and candidates lie furthest from the listing cell's centre; walls.  Densities against the FP64
oracle within 1e-12 of their scale: the terms agree to a few ulps and a sum has at most some
hundred of them, while a neighbour lost anywhere but at the very edge of the kernel, where its
weight is below that, or a neighbour counted twice, is far above it."""
import os

import numpy as np
import pytest

import oracle
import sph_b200
import sph_input

pytestmark = pytest.mark.gpu

COUNTS = {2: [0, 1, 15, 16, 17, 31, 32, 33, 0, 15], 3: [0, 1, 31, 32, 33, 0, 48, 70]}


@pytest.mark.parametrize("tpc", [32, 16])
@pytest.mark.parametrize("dim,N,overlap,wall", [
    (2, (40, 36), 4.0, 0), (2, (15, 15), 4.0, 0), (2, (41, 33), 4.0, 1),
    (3, (27, 24, 24), 3.0, 0), (3, (11, 11, 11), 3.0, 0), (3, (22, 19, 17), 3.0, 1)])
def test_densities_of_uneven_cells(workdir, dim, N, overlap, wall, tpc):
    dx = 1.0 / max(N)
    p = sph_input.write_input(os.path.join(workdir, "input"), N=N, L=tuple(n * dx for n in N),
                              dim=dim, overlap=overlap, wall=wall, dt=1e-5)
    e, o = sph_b200.System(p, precision="fp64"), oracle.Oracle(p)
    e.set_tuning(list_threads_per_cell=tpc, density_block=128)
    info = o.info()
    cells = [info["Ncells%d" % q] for q in range(dim)]
    rng = np.random.default_rng(11)
    fluid = np.flatnonzero(e.type() == 0)
    counts = rng.permutation(np.resize(COUNTS[dim], int(np.prod(cells))))
    where = np.repeat(np.arange(counts.size), counts)[:fluid.size]
    where = np.append(where, rng.choice(np.flatnonzero(counts > 0), fluid.size - where.size))
    for q in range(dim):
        at = (where // int(np.prod(cells[:q]))) % cells[q]
        v = (at + rng.uniform(0.001, 0.999, fluid.size)) * N[q] * dx / cells[q]
        if wall and q == 1:
            v = rng.uniform(0.01, 0.99, fluid.size) * N[1] * dx
        x = e.field("xyz"[q])
        x[fluid] = v
        e.set_field("xyz"[q], x)
        o.set_field("xyz"[q], x)
    for s in (e, o):
        s.neighbours_search()
        s.calculate_density()
    a, b = e.field("dens"), o.field("dens")
    assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
    e.close()
    o.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lists_without_a_spare_entry_and_lists_just_grown(workdir, precision):
    """A capacity of exactly the entries in use gives the same bits as a larger one; grown for
    headroom by synchronize(), the emptied lists are built again before they are read."""
    p = sph_input.write_input(os.path.join(workdir, "input"), N=(24, 20, 28),
                              L=(24 / 28.0, 20 / 28.0, 1.0), dim=3, overlap=3.0, dt=1e-5)
    wide = sph_b200.System(p, precision=precision)
    wide.neighbours_search()
    wide.calculate_density()
    used = wide.neighbour_lists()["max_used"]
    tight = sph_b200.System(p, precision=precision, nbr_capacity=used)
    tight.neighbours_search()
    tight.calculate_density()
    want = wide.field("dens")
    assert np.array_equal(tight.field("dens"), want)
    tight.synchronize()
    lists = tight.neighbour_lists()
    assert lists["grown"] == 1 and lists["capacity"] > used
    tight.calculate_density()
    assert np.array_equal(tight.field("dens"), want)
    wide.close()
    tight.close()
