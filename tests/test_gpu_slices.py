"""Automatic slices: with none given, the members' CTAs are 512 points or more each, so
many that the GPU's 148 SMs are used and not one more.  Member counts on both sides of
the rule's lines and grids on both sides of its sizes, each against the oracle (one RHS
1e-12: FP64, different FFTs)."""
import numpy as np
import pytest

import oracle_lib as ol
from decks_util import random_state, rel_l2, small_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,count", [
    ((256,), 1), ((1024,), 2), ((2048,), 1), ((8192,), 1), ((16384,), 1),
    ((2048,), 37), ((2048,), 38), ((2048,), 74), ((2048,), 75), ((1024, 4096), 8), ((512, 2048, 8192), 16)])
def test_default_slices(tmp_path, sizes, count):
    import hawassi_c_b200 as hw
    decks = [small_deck(tmp_path, f"s{n}", nx=n, T_end=4.0, breaking=n == 2048) for n in sizes]
    e = hw.Engine(decks * count, eps_abs=1e-8, eps_rel=1e-6)
    for m, n in enumerate(sizes):
        o = ol.Oracle(decks[m], eps_abs=1e-8, eps_rel=1e-6)
        y = random_state(n, 5)
        ref = o.rhs(1.3, y)
        for i in (m, m + len(sizes) * (count - 1)):
            assert rel_l2(e.rhs(1.3, y, member=i), ref) < 1e-12
        o.close()
    e.close()
