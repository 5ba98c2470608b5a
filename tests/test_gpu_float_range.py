"""Double-float arithmetic (csrc/draws.cuh) in place of FP64 where its low parts
would leave the normal floats: source terms of very small and very large
charge-to-potential factors, and initial velocities and places of very cold
species and of very small and very large cells.  FP64 decides there."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


# 2^-32 / (ds eps0): beside 2^-90 and 2^75 on both sides, far outside of them, and powers of two
@pytest.mark.parametrize("ds,eps0", [(0.37, 3e17), (0.37, 1e18), (0.37, 1e27), (0.25, 2.0 ** 88), (0.25, 2.0 ** 122),
                                     (0.37, 2.5e-32), (0.37, 1e-32)])
@pytest.mark.parametrize("ncx", (48, 150))
def test_sources_match_oracle(gpu_lib, ds, eps0, ncx):
    p = cg.workload_params("tiny", ncx=ncx, ncy=60, ds=ds, eps0=eps0, n=600.0, phi_p=0.0, max_sweeps=20,
                           init_max_sweeps=20, dt=1e-3)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        assert np.abs(ora.phi()).max() > 0 and np.isfinite(ora.phi()).all()
        np.testing.assert_array_equal(sim.rho_fixed(), ora.rho_fixed())
        # equal to the bit but for what the smallest float rounds: four times a
        # sweep on the tiles and once in the oracle, by half of 2^-149 each
        assert np.abs(sim.phi().astype(np.float64) - ora.phi()).max() <= 20 * 5 * 2.0 ** -150
    ora.close()


@pytest.mark.parametrize("over", [{"kti": 1e-28}, {"kti": 5.8e-70}, {"kte": 2.0 ** -200, "kti": 2.0 ** -81}, {"ds": 2.0 ** -43 * 1.1},
                                  {"ds": 2.0 ** -100 * 1.1}, {"ds": 2.0 ** 76 * 1.1}])
def test_initial_draws_match_oracle(gpu_lib, over):
    over = dict(over)
    if "ds" in over:
        over["n"] = 40.0 / over["ds"] ** 3
        over["eps0"] = over["n"]
    p = cg.workload_params("tiny", ncx=61, ncy=67, max_sweeps=0, init_max_sweeps=0, phi_p=0.0, **over)  # no field
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        for sp in (0, 1):
            assert len(ora.particles(sp)) > 10000
            np.testing.assert_array_equal(sim.particles(sp), ora.particles(sp))
    ora.close()
