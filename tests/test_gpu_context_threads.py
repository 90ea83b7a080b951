"""Contexts made, used for host calls and destroyed by several threads at once, of grids
whose buffers differ: every right-hand side and step is what one context gives alone, bit
for bit (one context of each grid first; the same kernels on the same inputs)."""
import threading

import numpy as np
import pytest

from decks_util import random_state, small_deck

pytestmark = pytest.mark.gpu


def calls(hw, deck, nx):
    with hw.Engine(deck, slice=512, exact_sequence=True) as e:
        y = random_state(nx, nx)
        dy = e.rhs(1.3, y)
        z = y.copy()
        t, h = e.evolve_apply(1.4, 1.6, 1e-3, z)
        return dy, z, t, h


def test_threads_make_and_destroy_contexts(tmp_path):
    import hawassi_c_b200 as hw
    grids = (512, 1024, 4096, 8192)
    decks = {n: small_deck(tmp_path, f"t{n}", nx=n, T_end=4.0) for n in grids}
    want = {n: calls(hw, decks[n], n) for n in grids}
    bad = []

    def work(k):
        try:
            for i in range(6):
                n = grids[(k + i) % len(grids)]
                got = calls(hw, decks[n], n)
                if not all(np.array_equal(a, b) for a, b in zip(got, want[n])):
                    bad.append((k, i, n))
        except Exception as x:
            bad.append((k, repr(x)))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad
