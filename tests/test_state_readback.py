"""Counts and diagnostics come back the same whether the context has no
staging buffers yet, small ones (a few particles uploaded) or has grown them
(an array downloaded)."""
import pytest

from pic3d_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_state_words_before_and_after_the_staging_buffers(precision):
    from pic3d_b200.simulation import Simulation
    w = W.Workload(name="state", nx=12, ny=10, nz=11, mem=2, period=(1, 1, 1), ppc=(3, 0), u_th=(0.1, 0.0), steps=2)
    parts = W.make_particles(w, seed=2)
    sim = Simulation(w, precision=precision)
    sim.generate_thermal(0, 3, 1.0, 0.1, 7)
    first = sim.diagnostics()
    assert sim.num_particles(0) == 3 * 12 * 10 * 11 and sim.num_particles(1) == 0
    assert first["kinetic0"] > 0.0 and first["kinetic1"] == 0.0
    sim.upload_particles(1, W.make_particles(w.with_(ppc=(0, 1), u_th=(0.0, 0.1)), seed=3)[1])
    small = sim.diagnostics()
    assert sim.num_particles(0) == 3 * 12 * 10 * 11 and sim.num_particles(1) == 12 * 10 * 11
    assert small["kinetic0"] == pytest.approx(first["kinetic0"], rel=1e-12) and small["kinetic1"] > 0.0
    sim.download_array("ex")
    grown = sim.diagnostics()
    assert sim.num_particles(0) == 3 * 12 * 10 * 11 and sim.num_particles(1) == 12 * 10 * 11
    for k in small:
        assert grown[k] == pytest.approx(small[k], rel=1e-12, abs=1e-300), k
    sim.upload_particles(0, parts[0])
    assert sim.num_particles(0) == len(parts[0])
    sim.close()
