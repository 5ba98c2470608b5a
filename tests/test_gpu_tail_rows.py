"""The end of a step in one launch (k_tail, csrc/particles.cu) around its most
rows: 4085 is the most whose counts fit shared memory without an opt-in, 4096
the most that it takes, 4097 the first of the four launches.  Particles,
potential and reports equal the oracle's to the bit, also where rows run out of
room."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncy", (4085, 4086, 4096, 4097))
@pytest.mark.parametrize("slack", (0.5, 0.0))
def test_step_at_the_most_rows(gpu_lib, ncy, slack):
    p = cg.workload_params("tiny", ncx=3, ncy=ncy, n=100.0, max_sweeps=20, row_slack=slack)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        for _ in range(3):
            sim.step(4)
            ora.step(4)
            g, o = sim.stats(1)[0], ora.stats()
            for k in ("step", "absorbed", "removed", "injected", "live", "sweeps"):
                assert g[k] == o[k], k
        for sp in (0, 1):
            np.testing.assert_array_equal(sim.particles(sp), ora.particles(sp))
        np.testing.assert_array_equal(sim.phi().astype(np.float64), ora.phi())
    ora.close()


@pytest.mark.parametrize("ncx,ncy,n", [(2, 1500, 8000.0), (40, 600, 400.0)])
def test_runs_that_halt_again_and_again(gpu_lib, ncx, ncy, n):
    """Rows without room: steps halt in the check of the step's end, whose many CTAs
    see the flag at their start, in the check or not at all; no draw is appended
    twice and no step ends early."""
    p = cg.workload_params("tiny", ncx=ncx, ncy=ncy, n=n, max_sweeps=8, row_slack=0.0)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        most = 0
        for _ in range(4):
            sim.step(9)
            ora.step(9)
            most = max(most, int(sim.row_counts(0).max()), int(sim.row_counts(1).max()))
            g, o = sim.stats(1)[0], ora.stats()
            for k in ("step", "absorbed", "removed", "injected", "live", "sweeps"):
                assert g[k] == o[k], k
            np.testing.assert_array_equal(sim.rho_fixed(), ora.rho_fixed())
        assert most > p.ppr + 72  # rows start with room for ppr + 64 particles, rounded up to eights
        for sp in (0, 1):
            np.testing.assert_array_equal(sim.particles(sp), ora.particles(sp))
    ora.close()
