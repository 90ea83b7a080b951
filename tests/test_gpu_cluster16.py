"""Members in clusters of sixteen CTAs, whose cross-CTA transform steps are shared by two
neighbouring lanes a position, against the oracle in every slice length and model: one
RHS 1e-12 and one replayed step (t 1e-13, y 1e-12), the bounds of the parity tests (FP64,
different FFTs)."""
import numpy as np
import pytest

import oracle_lib as ol
from decks_util import random_state, rel_l2, small_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,model,varying,breaking", [
    (4096, "HS2", False, True), (4096, "HS3", True, False), (8192, "HS1", False, False), (8192, "HS2", True, True),
    (16384, "HS2", False, False), (16384, "HS3", True, True), (32768, "HS2", False, True)])
def test_sixteen_ctas(tmp_path, nx, model, varying, breaking):
    import hawassi_c_b200 as hw
    deck = small_deck(tmp_path, "c16", nx=nx, model=model, varying=varying, breaking=breaking, T_end=4.0)
    o = ol.Oracle(deck, eps_abs=1e-8, eps_rel=1e-6)
    e = hw.Engine(deck, cluster=16, eps_abs=1e-8, eps_rel=1e-6, exact_sequence=True)
    y = random_state(nx, 5)
    assert rel_l2(e.rhs(1.3, y), o.rhs(1.3, y)) < 1e-12
    ya, yb = y.copy(), y.copy()
    ta, _ = o.evolve_apply(1.4, 1.6, 1e-3, ya)
    tb, _ = e.evolve_apply(1.4, 1.6, 1e-3, yb)
    assert abs(ta - tb) < 1e-13 and rel_l2(yb, ya) < 1e-12
    e.close()
    o.close()
