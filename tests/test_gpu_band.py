"""The flat HS2 right-hand side and the stepper around the alias band's edge: the
device forms nothing but the state outside the band, and pairs k with N - k, so bands
of several widths, slices and cluster sizes (with content outside the band, an influx
and breaking or not) against the oracle.  Tolerances are those of the parity tests:
one RHS 1e-12, one step in replay mode t 1e-13 and y 1e-12 (FP64, different FFTs)."""
import numpy as np
import pytest

import oracle_lib as ol
from decks_util import random_state, rel_l2, small_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,slice_,cutfrac,breaking", [
    (256, 256, "4", False), (512, 256, "3", False), (1024, 256, "5", True), (2048, 2048, "2", False),
    (4096, 256, "9", False), (4096, 2048, "7", True), (16384, 2048, "4", True)])
def test_band_edges(tmp_path, nx, slice_, cutfrac, breaking):
    import hawassi_c_b200 as hw
    deck = small_deck(tmp_path, "band", nx=nx, breaking=breaking, T_end=4.0, cutfrac=cutfrac)
    o = ol.Oracle(deck, eps_abs=1e-8, eps_rel=1e-6)
    e = hw.Engine(deck, eps_abs=1e-8, eps_rel=1e-6, slice=slice_, exact_sequence=True)
    y = random_state(nx, 5)
    ref, got = o.rhs(1.3, y), e.rhs(1.3, y)
    assert rel_l2(got, ref) < 1e-12
    assert np.array_equal(got == 0.0, ref == 0.0) or not np.any(got[ref == 0.0])
    ya, yb = y.copy(), y.copy()
    ta, _ = o.evolve_apply(1.0, 1.2, 1e-3, ya)
    tb, _ = e.evolve_apply(1.0, 1.2, 1e-3, yb)
    assert abs(ta - tb) < 1e-13 and rel_l2(yb, ya) < 1e-12
    e.close()
    o.close()
