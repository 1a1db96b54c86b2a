"""Overflow of the Q5.27 aggregate in a batch of systems: each system's bin
bounds are settled when an advance ends, for that system alone. A state whose
aggregate wraps raises S_overflow in its own system only, one whose bound
passes 2^32 without any total doing so raises nothing, and both equal the
returning scatter of the systems run alone; the bounds are clear again for the
next advance. A batch too small for the bounds to pay scatters with returns and
raises the same."""
import numpy as np
import pytest

import pfb200
from helpers2d import params
from test_scatter_bins_gpu import S_OVERFLOW, run_sim, stacked_state

pytestmark = pytest.mark.gpu


def batch(plain_side, plain_cells):
    """An ensemble of the wrapping state, an ordinary system and the state of
    which only a bound passes 2^32."""
    wraps, bound = stacked_state(False), stacked_state(True)
    ps = [wraps[0], params(plain_side, plain_cells, seed=3), bound[0]]
    cs = [pfb200.palmieri_centres(p.num_cells, p.L, p.target_radius, p.seed) for p in ps]
    ens = pfb200.Ensemble2D(ps, cs)
    for r, (_, cells, phi) in ((0, wraps), (2, bound)):
        ens.system(r).set_state(cells, phi, 0)
    return ens, wraps, bound


LARGE = (1024, 430)  # with the others 448 cells: one step of them scatters under bounds
SMALL = (512, 12)


def state(s):
    return s.cells().tobytes(), s.phi().tobytes(), s.S().tobytes(), s.flags().tobytes()


@pytest.mark.parametrize("plain", [LARGE, SMALL], ids=["bounds", "returns"])
@pytest.mark.parametrize("steps", [1, 7])
def test_each_system_settles_its_own_bounds(steps, plain):
    ens, wraps, bound = batch(*plain)
    ens.advance(steps)
    flags = [ens.system(r).flags() for r in range(3)]
    assert flags[0][S_OVERFLOW] and not flags[1][S_OVERFLOW] and not flags[2][S_OVERFLOW]
    for r, (p, cells, phi) in ((0, wraps), (2, bound)):
        alone = run_sim(p, cells, phi, steps, 2)
        assert ens.system(r).phi().tobytes() == alone[1].tobytes()
        np.testing.assert_array_equal(flags[r], alone[3])
        # a launch that settles nothing recounts nothing
        assert (ens.system(r).scatter_recounts() >= 1) == (plain is LARGE)
    p = ens.params[1]
    alone = pfb200.Sim2D(p, *pfb200.palmieri_centres(p.num_cells, p.L, p.target_radius, p.seed))
    alone.advance(steps)
    assert state(ens.system(1)) == state(alone)
    alone.close()
    ens.close()


@pytest.mark.parametrize("cut", [[1, 6], [3, 1, 3], [6, 1]])
def test_bounds_are_clear_after_an_advance(cut):
    """An advance that settles and one that goes on recount the same bins as
    often: no bound of the last launch is left for the next call."""
    a, b = batch(*LARGE)[0], batch(*LARGE)[0]
    a.advance(sum(cut))
    for n in cut:
        b.advance(n)
    for r in range(3):
        assert state(a.system(r)) == state(b.system(r))
        assert a.system(r).scatter_recounts() == b.system(r).scatter_recounts()
    assert a.system(2).scatter_recounts() >= 1
    a.close()
    b.close()


def test_serial_steps_between_advances():
    """One launch per system (returning) between two batch advances."""
    a, b = batch(*LARGE)[0], batch(*LARGE)[0]
    a.advance(5)
    b.advance(2)
    b.advance_serial(1)
    b.advance(2)
    for r in range(3):
        assert state(a.system(r)) == state(b.system(r))
    a.close()
    b.close()
