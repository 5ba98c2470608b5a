"""The initial plasma's draws in double-float arithmetic (csrc/draws.cuh)
against the oracle's FP64 draws, bit for bit: cell sizes that are no power of
two, rows on both sides of the 32768th (the FP64 path beyond it), and enough
particles that some fail the rounding test and take the FP64 path (about one
in 2000)."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [
    {"ncx": 3, "ncy": 33000, "n": 16.0},
    {"ncx": 37, "ncy": 61, "ds": 0.1, "n": 90000.0, "mi": 1836.0, "kti": 0.07},
    {"ncx": 300, "ncy": 64, "ds": 0.37, "n": 700.0, "seed": (1 << 63) + 12345},
])
def test_initial_draws_match_oracle(gpu_lib, over):
    p = cg.workload_params("tiny", max_sweeps=2, init_max_sweeps=2, **over)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        for sp in (0, 1):
            np.testing.assert_array_equal(sim.particles(sp), ora.particles(sp))
    ora.close()
