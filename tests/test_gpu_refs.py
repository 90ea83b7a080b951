"""The varying-bottom sweeps for every shape of their plan: K reference depths fill the
iterations' four fields differently (the sum of the images goes back with the last of
them or in one more iteration), HS2 and HS3, one CTA to a cluster of 16, breaking or
not, against the oracle.  One RHS 1e-12, one step in replay mode t 1e-13 and y 1e-12, as
in the parity tests (FP64 on both sides, different FFTs)."""
import pytest

import oracle_lib as ol
from decks_util import random_state, rel_l2, small_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nref", [2, 3, 4, 5, 6, 7, 8, 9, 15, 16])
@pytest.mark.parametrize("model,nx,slice_,breaking", [
    ("HS2", 512, 512, False), ("HS3", 1024, 256, True), ("HS2", 4096, 256, True), ("HS3", 2048, 2048, False)])
def test_reference_depths(tmp_path, nref, model, nx, slice_, breaking):
    import hawassi_c_b200 as hw
    deck = small_deck(tmp_path, "refs", nx=nx, model=model, varying=True, breaking=breaking, T_end=4.0)
    kw = dict(eps_abs=1e-8, eps_rel=1e-6, nref=nref)
    o = ol.Oracle(deck, **kw)
    e = hw.Engine(deck, slice=slice_, exact_sequence=True, **kw)
    y = random_state(nx, 9)
    assert rel_l2(e.rhs(1.3, y), o.rhs(1.3, y)) < 1e-12
    ya, yb = y.copy(), y.copy()
    ta, _ = o.evolve_apply(1.0, 1.2, 1e-3, ya)
    tb, _ = e.evolve_apply(1.0, 1.2, 1e-3, yb)
    assert abs(ta - tb) < 1e-13 and rel_l2(yb, ya) < 1e-12
    e.close()
    o.close()
