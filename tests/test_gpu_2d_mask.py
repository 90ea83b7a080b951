"""2D steps from states with content outside the alias mask, which the stepper carries
unmoved instead of combining: two steps in replay against the oracle, each from its own
set_state, and a direct right-hand side between them (it takes another stage input).
One step 1e-11 relative L2 of y, next h 1e-6, as the replay test of the 2D stepper."""
import numpy as np
import pytest

from hawassi_c_b200 import decks2d
from hawassi_c_b200.engine2d import Engine2D
from oracle_lib import Oracle2D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,model,bottom", [(64, 64, 2, "flat"), (128, 64, 3, "flat"),
                                                (64, 128, 2, "shoal"), (256, 64, 1, "flat")])
def test_steps_outside_the_mask(nx, ny, model, bottom):
    tb = decks2d.tables(nx=nx, ny=ny, Lx=0.9 * nx, Ly=0.9 * ny, depth=2.0, shallow=0.6, Hs=0.1, Tp=3.0, n_freq=24,
                        n_dir=6, t_end=6.0, dt=0.1, damp=6.0, x_line=10.0, nadj=1.0, seed=2, bathymetry=bottom,
                        ninterp=2, model=model)
    eng, ora = Engine2D(tb, 1e-8, 1e-6), Oracle2D(tb, 1e-8, 1e-6)
    rng = np.random.default_rng(4)
    n = nx * ny
    for t0 in (0.7, 2.1):
        y = 0.002 * rng.standard_normal(6 * n) * np.sqrt(n)
        yo, yg = y.copy(), y.copy()
        to, ho = ora.evolve_apply(t0, t0 + 0.5, 1e-3, yo)
        tg, hg = eng.evolve_apply(t0, t0 + 0.5, 1e-3, yg)
        assert abs(tg - to) < 1e-12 and abs(hg - ho) <= 1e-6 * abs(ho)
        assert np.linalg.norm(yg - yo) / np.linalg.norm(yo) < 1e-11
        out = np.tile(np.asarray(tb["aal"] if isinstance(tb, dict) else tb.aal).ravel() == 0.0, 6)
        assert np.any(out) and np.array_equal(yg[out], y[out])
        eng.rhs(t0, rng.standard_normal(6 * n))
    eng.close()
