"""Runs around the length from which steps go several to a graph: one step
short of it, exactly it, and a rest of single steps; with rows that run out of
room on the way, so that the steps after the halt in the same graph are rerun.
Same particles, potential and step reports as the same steps one at a time."""
import numpy as np
import pytest

import cupic_gb300 as cg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", (63, 64, 77))
@pytest.mark.parametrize("slack", (None, 0.0))
def test_long_runs_match_single_steps(gpu_lib, steps, slack):
    p = cg.workload_params("tiny", **({} if slack is None else {"row_slack": slack}))
    with cg.Sim(p) as run, cg.Sim(p) as single:
        run.init_plasma()
        single.init_plasma()
        run.step(steps)
        for _ in range(steps):
            single.step(1)
        run.sync()
        single.sync()
        np.testing.assert_array_equal(run.phi(), single.phi())
        for sp in (0, 1):
            np.testing.assert_array_equal(run.particles(sp), single.particles(sp))
        assert run.stats(8) == single.stats(8)
        run.step(steps)  # the graph again
        for _ in range(steps):
            single.step(1)
        np.testing.assert_array_equal(run.phi(), single.phi())
