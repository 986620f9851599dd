"""Tiles with more particles than the reverse kernel's scratch holds.

The scratch holds 640 (FP64) or 1152 (FP32) particles; a fuller tile is taken
in rounds, each with its own scale and flush of the field adjoints.  One
particle per cell fits a tile of 4^3 easily, 11 and 24 per cell leave the
last round partly filled in one or both precisions.  The gradients equal those
of the unsorted global-memory kernels, with the bounds of the same comparison
at 2 per cell (test_adjoint.py).
"""
import dataclasses

import numpy as np
import pytest

from pic3d_b200.workloads import LAMBDA, Workload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mem", [2, 4], ids=["o2", "o4"])
@pytest.mark.parametrize("ppc", [1, 11, 24])
def test_rounds_of_a_tile_agree_with_the_global_adjoint(ppc, mem, precision):
    from pic3d_b200.adjoint import AdjointSpec, objective_and_grad
    w = Workload(name="adj_rounds", nx=24, ny=9, nz=10, mem=mem, period=(0, 0, 0), dx=LAMBDA / 16, dy=LAMBDA / 8,
                 dz=LAMBDA / 8, ppc=(ppc, 0), u_th=(0.02, 0.0), laser_amplitude=1.0, laser_pulse_duration=4.0,
                 waist=LAMBDA, laser_polarization=3, steps=20)
    spec = AdjointSpec(workload=w, n_knots=6, profile_n=4, window=(4.0, 20.0), ramp=4.0, segment=7, seed=77,
                       precision=precision)
    rng = np.random.default_rng(5)
    knots = 0.05 + 0.05 * rng.random(6)
    prof = 1.0 + 0.5 * rng.random((4, 4))
    lt, kt, pt, wt = objective_and_grad(spec, knots, prof)
    lg, kg, pg, wg = objective_and_grad(dataclasses.replace(spec, tile=-1), knots, prof)
    tol = 1e-9 if precision == "fp64" else 2e-4
    assert lt == pytest.approx(lg, rel=1e-12 if precision == "fp64" else 1e-6)
    for a, b in ((kt, kg), (pt, pg), (wt, wg)):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
