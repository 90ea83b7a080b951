"""The 2D right-hand side's pass plans against the oracle where they differ: K
reference depths go through the passes two or four fields at a time (odd and even K,
one to four iterations), the damping travels in physical space, as one spectrum
(breaking) or as three (ChiAdj = 1), and every slice length has its own transform
plan, in rows and in columns.  One RHS 1e-11 relative L2, the bar of the other 2D
tests (FP64 on both sides, different transforms and the linear terms summed before
them)."""
import numpy as np
import pytest

from hawassi_c_b200 import decks2d
from hawassi_c_b200.engine2d import Engine2D
from oracle_lib import Oracle2D

pytestmark = pytest.mark.gpu


def deck(nx, ny, bottom, K, model, nadj, walls, breaking):
    tb = decks2d.tables(nx=nx, ny=ny, Lx=0.9 * nx, Ly=0.9 * ny, depth=2.0, shallow=0.6, Hs=0.1, Tp=3.0, n_freq=24,
                        n_dir=6, t_end=6.0, dt=0.1, damp=6.0, x_line=10.0, nadj=nadj, seed=2, bathymetry=bottom,
                        ninterp=3 if K == 3 else 2, model=model, breaking=breaking,
                        walls=((30.0, 20.0, 33.0, 45.0),) if walls else ())
    return decks2d.plain_k_operator(tb, K) if K > 3 else tb


@pytest.mark.parametrize("nx,ny,bottom,K,model,nadj,walls,breaking", [
    (64, 512, "flat", 0, 2, 1.0, False, True), (512, 64, "flat", 0, 3, 0.0, True, False),
    (256, 64, "flat", 0, 3, 1.0, False, True), (128, 256, "flat", 0, 1, 0.0, False, False),
    (512, 128, "shoal", 2, 2, 0.0, True, True), (64, 256, "shoal", 2, 1, 1.0, False, False),
    (128, 64, "shoal", 3, 3, 0.0, False, False), (64, 64, "shoal", 5, 2, 1.0, True, True),
    (256, 128, "shoal", 7, 3, 1.0, False, True), (64, 128, "shoal", 8, 2, 0.0, False, False),
    (128, 128, "shoal", 9, 3, 0.0, True, True), (64, 64, "shoal", 16, 1, 1.0, False, False),
    (1024, 64, "shoal", 6, 2, 1.0, False, True), (64, 1024, "shoal", 4, 3, 1.0, False, False)])
def test_pass_plans(nx, ny, bottom, K, model, nadj, walls, breaking):
    tb = deck(nx, ny, bottom, K, model, nadj, walls, breaking)
    eng, ora = Engine2D(tb, 1e-8, 1e-6), Oracle2D(tb, 1e-8, 1e-6)
    rng = np.random.default_rng(6)
    n = nx * ny
    # every wavenumber excited, the self-conjugate and Nyquist points too
    y = 0.01 * rng.standard_normal(6 * n) * np.sqrt(n)
    for t in (0.7, 3.35):
        if breaking:
            ora.set_tprev(t)   # no update of the breaking state: the RHS alone
            eng.set_state(t, 0.01, y)
        got, ref = eng.rhs(t, y), ora.rhs(t, y)
        assert np.linalg.norm(got - ref) / np.linalg.norm(ref) < 1e-11
