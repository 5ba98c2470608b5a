"""Kernels whose dynamic shared memory fits 48 KB only without their static part:
the push of rows about 200 cells wide, and tiles of the solve just below
48 KB.  Each in a process of its own, where no wider mesh has raised the
kernels' limits before; results equal the oracle's to the bit."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUN = """
import sys
import numpy as np
import cupic_gb300 as cg
from oracle.oracle import Oracle
p = cg.workload_params("tiny", ncx=int(sys.argv[1]), ncy=int(sys.argv[2]), n=4.0, max_sweeps=40)
ora = Oracle(p, fp64=False)
ora.init_plasma()
with cg.Sim(p) as sim:
    sim.init_plasma()
    sim.step(3)
    ora.step(3)
    for sp in (0, 1):
        np.testing.assert_array_equal(sim.particles(sp), ora.particles(sp))
    np.testing.assert_array_equal(sim.phi().astype(np.float64), ora.phi())
"""


@pytest.mark.parametrize("ncx,ncy", [(196, 40), (197, 40), (200, 40), (204, 40), (205, 40), (32, 128), (46, 138)])
def test_meshes_at_the_default_limit_step(gpu_lib, ncx, ncy):
    env = {**os.environ, "PYTHONPATH": ROOT}
    subprocess.run([sys.executable, "-c", RUN, str(ncx), str(ncy)], check=True, cwd=ROOT, env=env, timeout=300)
