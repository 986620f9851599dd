"""Positions at and next to the boundaries of the tiles.

The sort puts a particle into a tile, the push takes it from the tile that its
own decode names: both have to agree for every position, else the particle is
in no tile's list.  Tiles of nodes change at half cells, tiles of cells at
whole cells; the decode adds mem - 1 (and 1/2) to the position, which rounds,
so the doubles next to these points are where the two can part.  The
27-per-cell lattice of the loader has such coordinates in every box, e.g.
3.4999999999999996 with 10 cells.

One step of the loop, its push right after the sort, against the oracle at the
parity bounds of the other one-step tests: relative L2 1e-10 in FP64, 1e-5 in
FP32, every array and every particle.  (Not the push at t = 0, whose currents
the reference leaves unfolded: an FP32 context stores x = n as 0, where they
would sit at the other image.)
"""
import numpy as np
import pytest

import oracle as O
from parity import TOL_FP32, TOL_FP64, array_errors, particle_errors, periods

from pic3d_b200 import workloads as W


def lattice(n, per_cell):
    """the loader's coordinates (src/particle.cpp:58-75)"""
    num = int(n * np.cbrt(per_cell))
    norm = float(n) / num
    return np.arange(num) * norm + norm / 2.0


def edges(n, periodic):
    """every half and whole cell with both neighbours; x = n and the double
    below 0 (which wraps to n) only where the axis is periodic"""
    c = np.arange(2 * n + 1) * 0.5
    x = np.concatenate([c, np.nextafter(c, -1.0), np.nextafter(c, n + 1.0)])
    return x[(x <= n) if periodic else ((x >= 0) & (x < n))]


def particles(w, coords, count, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(count, dtype=W.PARTICLE_DTYPE)
    p["id"] = np.arange(count)
    for f, c in zip("xyz", coords):
        p[f] = c[np.arange(count) % len(c)] if f == "x" else rng.choice(c, count)
    for f in ("px", "py", "pz"):
        p[f] = 0.1 * rng.normal(size=count)
    p["gamma"] = np.sqrt(1.0 + p["px"] ** 2 + p["py"] ** 2 + p["pz"] ** 2)
    p["charge"], p["mass"], p["weight"] = -1.0, 1.0, 0.01
    return p


def test_the_lattice_has_positions_where_floor_and_rounding_differ():
    """(CPU) what the GPU cases below rest on: the coordinate is there, and
    the two ways to form a node name different tiles"""
    for n in range(10, 65):
        x = lattice(n, 27)
        for mem in (2, 4):
            by_floor = np.floor(x) + (x - np.floor(x) >= 0.5)
            by_decode = np.trunc((x - (1.0 - mem)) + 0.5) - (mem - 1)
            assert np.any(by_floor // 4 != by_decode // 4), (n, mem)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("tile", [0, 2], ids=["nodes", "cells"])
@pytest.mark.parametrize("period", [(1, 1, 1), (0, 1, 0)], ids=["periodic", "absorbing_xz"])
@pytest.mark.parametrize("where", ["edges", "lattice"])
def test_particles_at_tile_boundaries_are_pushed(where, period, tile, mem, precision):
    from pic3d_b200.simulation import Simulation
    n = (36, 12, 10)
    w = W.Workload(name=where, nx=n[0], ny=n[1], nz=n[2], mem=mem, period=period, ppc=(1, 0), u_th=(0.1, 0.0), steps=1)
    coords = [edges(n[d], period[d]) if where == "edges" else lattice(n[d], 27) for d in range(3)]
    parts = [particles(w, coords, 6000, seed=17), np.zeros(0, dtype=W.PARTICLE_DTYPE)]
    o = O.Oracle(w, parts)
    o.step(1)
    ref = o.state()
    sim = Simulation(w, precision=precision, tile=tile)
    sim.upload_particles(0, parts[0])
    sim.run_main_time_loop(1)
    got = sim.state()
    sim.close()
    tol, pos_tol = (TOL_FP64, 1e-11) if precision == "fp64" else (TOL_FP32, 2e-6)
    errs = array_errors(got, ref)
    assert max(errs.values()) < tol, errs
    perr, merr = particle_errors(got["particles"][0], ref["particles"][0], periods(w.params()))
    assert perr < pos_tol and merr < tol, (perr, merr)
