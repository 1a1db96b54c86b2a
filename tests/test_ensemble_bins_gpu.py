"""Overflow of the Q5.27 aggregate in a batch of systems: each system's bin
bounds are settled when an advance ends, for that system alone. A state whose
aggregate wraps raises S_overflow in its own system only, one whose bound
passes 2^32 without any total doing so raises nothing, and both equal the
returning scatter of the systems run alone; the bounds are clear again for the
next advance."""
import numpy as np
import pytest

import pfb200
from helpers2d import params
from test_scatter_bins_gpu import S_OVERFLOW, run_sim, stacked_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("steps", [1, 7])
def test_each_system_settles_its_own_bounds(steps):
    wraps, bound = stacked_state(False), stacked_state(True)
    plain = params(512, 12, seed=3)
    ps = [wraps[0], plain, bound[0]]
    cs = [pfb200.palmieri_centres(p.num_cells, p.L, p.target_radius, p.seed) for p in ps]
    ens = pfb200.Ensemble2D(ps, cs)
    for r, (_, cells, phi) in ((0, wraps), (2, bound)):
        ens.system(r).set_state(cells, phi, 0)
    ens.advance(steps)
    flags = [ens.system(r).flags() for r in range(3)]
    assert flags[0][S_OVERFLOW] and not flags[1][S_OVERFLOW]
    for r, (p, cells, phi) in ((0, wraps), (2, bound)):
        alone = run_sim(p, cells, phi, steps, 2)
        assert ens.system(r).phi().tobytes() == alone[1].tobytes()
        np.testing.assert_array_equal(flags[r], alone[3])
        assert ens.system(r).scatter_recounts() >= 1
    counts = ens.system(0).scatter_recounts(), ens.system(2).scatter_recounts()
    ens.system(2).set_state(bound[1], bound[2], steps)  # clears its bounds
    ens.advance(0)
    assert (ens.system(0).scatter_recounts(), ens.system(2).scatter_recounts()) == counts
    ens.close()
