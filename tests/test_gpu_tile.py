"""The register-tile solve (csrc/tile.cuh) at the edges of its layouts: ring
tiles (a strip's lanes hold a whole mesh row) with full and ragged last lanes,
several strips per warp, halo tiles with odd widths and periodic images, one
block and many, depths that divide the sweep count and depths that do not,
fewer sweeps than the depth, and a stop in the first, the last and a middle
sweep of a block.  The tile kernels round every operation where the oracle
does, so potential, field, sweep count and residual are equal to the bit."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

# (cells in x, cells in y, CTAs, depth): CTAs and depth None -> the tuned layout
LAYOUTS = [
    (2, 2, None, None), (3, 5, None, None), (5, 9, 2, 3), (31, 40, 1, 1), (32, 129, 1, 1),
    (33, 64, 4, 5), (64, 257, 7, 4), (100, 33, 1, 1), (127, 130, 6, 16), (128, 128, 1, 1),
    (129, 70, 4, 4), (130, 96, 12, 8), (250, 60, 9, 4), (251, 61, 8, 8), (301, 40, None, None),
    (512, 100, 25, 4),
]


@pytest.mark.parametrize("ncx,ncy,ctas,depth", LAYOUTS)
def test_tile_layouts_match_oracle(gpu_lib, monkeypatch, ncx, ncy, ctas, depth):
    for name, v in (("CUPIC_JACOBI_CTAS", ctas), ("CUPIC_JACOBI_DEPTH", depth)):
        if v is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, str(v))
    p = cg.workload_params("tiny", ncx=ncx, ncy=ncy, max_sweeps=60)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    rng = np.random.default_rng(ncx * 1000 + ncy)
    with cg.Sim(p) as sim:
        sim.init_plasma()
        if ctas is not None:
            assert sim.solver_plan()[0] == ctas
        # the mirror column's own starting value is read by the first sweep
        phi0 = rng.standard_normal((p.nny, p.nnx)).astype(np.float32).astype(np.float64)
        for tol, mn, mx, chk in ((0.0, 1, 1, 1), (0.0, 3, 3, 3), (0.0, 37, 37, 37), (1e-30, 1, 48, 1),
                                 (0.35, 1, 200, 1), (0.2, 1, 200, 3), (0.05, 30, 400, 1), (0.02, 33, 400, 7)):
            sim.set_phi(phi0)
            ora.set_phi(phi0)
            sim.poisson_solver(tol, mn, mx, chk)
            ora.solve(tol, mn, mx, chk)
            sim.field_solver()
            ora.field()
            what = f"tol {tol}, {mn}..{mx} sweeps, check {chk}"
            np.testing.assert_array_equal(sim.phi().astype(np.float64), ora.phi(), err_msg=what)
            for g, o in zip(sim.efield(), ora.efield()):
                np.testing.assert_array_equal(g.astype(np.float64), o, err_msg=what)
        # the field of a step comes out of the solve itself
        sim.step(2)
        ora.step(2)
        for g, o in zip(sim.efield(), ora.efield()):
            np.testing.assert_array_equal(g.astype(np.float64), o)
        st, so = sim.stats(1)[0], ora.stats()
        assert st["sweeps"] == so["sweeps"] and st["residual"] == so["residual"]
    ora.close()


# precision form: (cells in x, cells in y, CTAs, depth, sweeps per correction)
REFINED = [(3, 5, None, None, 4), (32, 40, 1, 1, 8), (64, 90, 5, 4, 32), (67, 50, 4, 8, 5), (100, 40, 3, 16, 24),
           (140, 70, 6, 8, 10), (257, 60, 12, 4, 16), (300, 64, None, None, 32)]


@pytest.mark.parametrize("ncx,ncy,ctas,depth,every", REFINED)
def test_refining_tiles_match_oracle(gpu_lib, monkeypatch, ncx, ncy, ctas, depth, every):
    """The precision form in one launch: FP64 potential, field, sweep counts
    and residuals equal the oracle's, for stops by the sweep cap, by the
    tolerance and before the first correction, and for sweeps per correction
    that are no multiple of the depth."""
    for name, v in (("CUPIC_JACOBI_CTAS", ctas), ("CUPIC_JACOBI_DEPTH", depth)):
        if v is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, str(v))
    p = cg.workload_params("tiny", ncx=ncx, ncy=ncy, refine_every=every, tol=2e-3, min_sweeps=every, max_sweeps=60,
                           init_tol=1e-2, init_min_sweeps=every, init_max_sweeps=500)
    ora = Oracle(p, fp64=False)
    ora.init_plasma()
    with cg.Sim(p) as sim:
        sim.init_plasma()
        np.testing.assert_array_equal(sim.phi64(), ora.phi())
        for tol, mn, mx in ((0.0, 0, 0), (0.0, 7, 7), (1e9, 0, 50), (5e-2, 10, 300), (1e-3, 10, 97)):
            sim.poisson_solver(tol, mn, mx, 1)
            ora.solve(tol, mn, mx, 1)
            np.testing.assert_array_equal(sim.phi64(), ora.phi(), err_msg=f"tol {tol}, {mn}..{mx} sweeps")
        for _ in range(3):
            sim.step(1)
            ora.step(1)
            g, o = sim.stats(1)[0], ora.stats()
            assert g["sweeps"] == o["sweeps"] and g["residual"] == o["residual"] and g["flags"] == 0
        np.testing.assert_array_equal(sim.phi64(), ora.phi())
        for g, o in zip(sim.efield(), ora.efield()):
            np.testing.assert_array_equal(g.astype(np.float64), o)
        # a mirror column that differs keeps its own FP64 value (launches of jacobi.cu)
        phi = ora.phi()
        phi[1:-1, -1] += 1e-3
        sim.set_phi(phi)
        ora.set_phi(phi)
        sim.step(1)
        ora.step(1)
        for sp in (0, 1):
            np.testing.assert_array_equal(sim.particles(sp), ora.particles(sp))
    ora.close()
