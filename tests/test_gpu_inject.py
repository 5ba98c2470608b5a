"""Few injected particles a step: drawn beside the solve where it leaves two
SMs free (150 CTAs of 152 SMs and fewer), else beside the push; at a low and a
high flux.  Particles and reports equal the oracle's to the bit."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", (1, 150, 151, 152))
@pytest.mark.parametrize("dens", (4.0, 400.0))
def test_injection_beside_the_solve(gpu_lib, monkeypatch, ctas, dens):
    monkeypatch.setenv("CUPIC_JACOBI_CTAS", str(ctas))
    p = cg.workload_params("tiny", ncx=12, ncy=153 if ctas > 1 else 60, n=dens, max_sweeps=20)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        assert sim.solver_plan()[0] == ctas
        for _ in range(6):
            sim.step(3)
            ora.step(3)
            g, o = sim.stats(1)[0], ora.stats()
            for k in ("step", "absorbed", "removed", "injected", "live", "sweeps"):
                assert g[k] == o[k], k
        for sp in (0, 1):
            np.testing.assert_array_equal(sim.particles(sp), ora.particles(sp))
    ora.close()
