"""Ring layouts whose CTAs are one cluster and trade rows through shared memory
(csrc/tile.cuh): the smallest and largest cluster, one CTA more than a cluster
holds, blocks of exactly the depth (strips with rows from both neighbours),
ragged last lanes, stops inside and outside a block, and the precision form.
Every layout rounds as the oracle does, so all results are equal to the bit."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

# (cells in x, cells in y, CTAs, depth, sweeps per correction; 0: the FP32 solve)
LAYOUTS = [
    (32, 128, 2, 16, 0), (32, 128, 16, 7, 0), (32, 129, 17, 7, 0), (8, 33, 16, 2, 0), (128, 64, 8, 7, 0),
    (126, 49, 16, 3, 0), (5, 40, 13, 3, 0), (64, 97, 16, 6, 12), (61, 50, 7, 7, 9),
]


@pytest.mark.parametrize("ncx,ncy,ctas,depth,every", LAYOUTS)
def test_cluster_layouts_match_oracle(gpu_lib, monkeypatch, ncx, ncy, ctas, depth, every):
    monkeypatch.setenv("CUPIC_JACOBI_CTAS", str(ctas))
    monkeypatch.setenv("CUPIC_JACOBI_DEPTH", str(depth))
    p = cg.workload_params("tiny", ncx=ncx, ncy=ncy, refine_every=every, max_sweeps=60)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        assert sim.solver_plan()[0] == ctas and sim.solver_plan()[2] == depth
        step = max(every, 1)
        for tol, mn, mx in ((0.0, 50 * step, 50 * step), (0.3, step, 300), (0.03, 3 * step, 900)):
            sim.poisson_solver(tol, mn, mx, step)
            ora.solve(tol, mn, mx, step)
            np.testing.assert_array_equal(sim.phi64() if every else sim.phi().astype(np.float64), ora.phi())
        sim.step(3)
        ora.step(3)
        for g, o in zip(sim.efield(), ora.efield()):
            np.testing.assert_array_equal(g.astype(np.float64), o)
        st, so = sim.stats(1)[0], ora.stats()
        assert st["sweeps"] == so["sweeps"] and st["residual"] == so["residual"]
    ora.close()
