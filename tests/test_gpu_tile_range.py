"""The register-tile solve (csrc/tile.cuh) at both ends of a float's range.  It
forms a node from quarters of its neighbours, so potentials up to the largest
float solve as in the oracle, to the bit, where the sums are finite; far below,
its four partial sums are each rounded to a multiple of 2^-149."""
import numpy as np
import pytest

import cupic_gb300 as cg
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu

MESHES = [(32, 129), (33, 64), (64, 20), (130, 96), (301, 75)]


@pytest.fixture
def pair(gpu_lib, monkeypatch):
    for name in ("CTAS", "DEPTH", "TUNE"):
        monkeypatch.delenv("CUPIC_JACOBI_" + name, raising=False)
    made = []

    def make(ncx, ncy):
        p = cg.workload_params("tiny", ncx=ncx, ncy=ncy, n=4.0, max_sweeps=20)
        sim, ora = cg.Sim(p), Oracle(p, fp64=False)
        made.extend((sim, ora))
        sim.init_plasma()
        ora.init_plasma()
        return p, sim, ora

    yield make
    for x in made:
        x.close()


@pytest.mark.parametrize("ncx,ncy", MESHES)
def test_large_potentials_match_oracle(pair, ncx, ncy):
    p, sim, ora = pair(ncx, ncy)
    rng = np.random.default_rng(ncx)
    phi = np.zeros((p.nny, p.nnx))
    # far enough apart, round the seam too, that no sum of four passes 2^128
    phi[2:-2:5, 1:-3:4] = rng.choice((-1.0, 1.0), phi[2:-2:5, 1:-3:4].shape) * 2.0 ** 127 * 1.5
    phi[0], phi[-1] = 2.0 ** 126 * 1.25, -2.0 ** 126 * 1.25
    phi[1:3], phi[-3:-1] = 0.0, 0.0
    phi[:, -1] = phi[:, 0]
    for tol, mn, mx in ((0.0, 1, 1), (0.0, 3, 3), (1e30, 1, 3)):
        sim.set_phi(phi)
        ora.set_phi(phi)
        sim.poisson_solver(tol, mn, mx, 1)
        ora.solve(tol, mn, mx, 1)
        assert np.isfinite(ora.phi()).all() and np.abs(ora.phi()).max() > 2.0 ** 125
        np.testing.assert_array_equal(sim.phi().astype(np.float64), ora.phi())
        sim.field_solver()
        ora.field()
        for g, o in zip(sim.efield(), ora.efield()):
            np.testing.assert_array_equal(g.astype(np.float64), o)


def test_small_potentials_round_to_the_smallest_float(pair):
    p, sim, ora = pair(32, 150)
    phi = np.zeros((p.nny, p.nnx))
    phi[0] = 1e-36
    sweeps = 60
    # no charge: the plasma is taken out
    for s in (0, 1):
        sim.load(s, np.empty((0, 4)))
        ora.load(s, np.empty((0, 4)))
    sim.set_phi(phi)
    ora.set_phi(phi)
    sim.poisson_solver(0.0, sweeps, sweeps, sweeps)
    ora.solve(0.0, sweeps, sweeps, sweeps)
    assert ((ora.phi() > 0) & (ora.phi() < 2.0 ** -126)).any()
    # four roundings a sweep here and one there, by half of 2^-149 each; the
    # average of four neighbours does not add to them
    assert np.abs(sim.phi().astype(np.float64) - ora.phi()).max() <= sweeps * 5 * 2.0 ** -150
