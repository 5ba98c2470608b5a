"""A potential set with two different columns at the seam (0 and nnx-1) in the
precision form, whose tiles take one for the other: the solve leaves them for the
launches that read both, tuned in the middle of the run.  Only the potential
changes, and what follows equals the oracle to the bit."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncx,ncy", [(256, 1024), (300, 700), (128, 512), (48, 90)])
def test_two_seam_columns_change_the_potential_alone(gpu_lib, monkeypatch, ncx, ncy):
    for name in ("CTAS", "DEPTH", "TUNE"):
        monkeypatch.delenv("CUPIC_JACOBI_" + name, raising=False)
    p = cg.workload_params("tiny", ncx=ncx, ncy=ncy, n=2.0, refine_every=16, tol=1e-9, min_sweeps=16, max_sweeps=64,
                           init_tol=1e-9, init_min_sweeps=16, init_max_sweeps=64)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        sim.step(2)
        ora.step(2)
        field, particles, stats = sim.efield(), [sim.particles(s) for s in (0, 1)], sim.stats(2)
        phi = ora.phi()
        phi[1:-1, -1] += 0.125
        sim.set_phi(phi)
        ora.set_phi(phi)
        np.testing.assert_array_equal(sim.phi64(), phi)
        np.testing.assert_array_equal(sim.phi(), phi.astype(np.float32))
        for g, o in zip(sim.efield(), field):
            np.testing.assert_array_equal(g, o)
        for s in (0, 1):
            np.testing.assert_array_equal(sim.particles(s), particles[s])
        assert sim.stats(2) == stats and sim.flags() == 0
        sim.poisson_solver(1e-9, 16, 64, 16)
        ora.solve(1e-9, 16, 64, 16)
        np.testing.assert_array_equal(sim.phi64(), ora.phi())
        sim.step(2)
        ora.step(2)
        np.testing.assert_array_equal(sim.phi64(), ora.phi())
        for s in (0, 1):
            np.testing.assert_array_equal(sim.particles(s), ora.particles(s))
        g, o = sim.stats(1)[0], ora.stats()
        assert g["sweeps"] == o["sweeps"] and g["residual"] == o["residual"]
    ora.close()


def test_equal_seam_columns_bring_the_tiles_back(gpu_lib):
    p = cg.workload_params("tiny", ncx=96, ncy=200, n=2.0, refine_every=8, tol=1e-9, min_sweeps=8, max_sweeps=40,
                           init_tol=1e-9, init_min_sweeps=8, init_max_sweeps=40)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        plan = sim.solver_plan()
        for dphi in (0.125, 0.0, 0.25, None):
            if dphi is None:
                sim.init_plasma()
                ora.init_plasma()
            else:
                phi = ora.phi()
                phi[:, -1] = phi[:, 0]
                phi[1:-1, -1] += dphi
                sim.set_phi(phi)
                ora.set_phi(phi)
            if not dphi:
                assert sim.solver_plan() == plan
            sim.step(2)
            ora.step(2)
            np.testing.assert_array_equal(sim.phi64(), ora.phi())
            for s in (0, 1):
                np.testing.assert_array_equal(sim.particles(s), ora.particles(s))
    ora.close()
