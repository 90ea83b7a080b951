"""The slices that a context took (Engine.slices) at member counts on both sides of the
rule's lines for the device's SMs, and one RHS of a member in each against the oracle
(1e-12: FP64, different FFTs)."""
import pytest

import oracle_lib as ol
from decks_util import random_state, rel_l2, small_deck

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", ["512", "1024 low", "1024 high", "2048"])
def test_counts_beside_the_lines(tmp_path, side):
    import torch
    import hawassi_c_b200 as hw
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    count, want = {"512": (sms // 4, 512), "1024 low": (sms // 4 + 1, 1024),
                   "1024 high": ((sms + sms // 4) // 2, 1024), "2048": ((sms + sms // 4) // 2 + 1, 2048)}[side]
    deck = small_deck(tmp_path, "s", nx=2048, T_end=4.0, breaking=True)
    e = hw.Engine([deck] * count, eps_abs=1e-8, eps_rel=1e-6)
    assert e.slices == [want] * count
    o = ol.Oracle(deck, eps_abs=1e-8, eps_rel=1e-6)
    y = random_state(2048, 5)
    assert rel_l2(e.rhs(1.3, y, member=count - 1), o.rhs(1.3, y)) < 1e-12
    e.close()
    o.close()


def test_named_and_single(tmp_path):
    import hawassi_c_b200 as hw
    a = small_deck(tmp_path, "a", nx=4096, T_end=4.0)
    b = small_deck(tmp_path, "b", nx=16384, T_end=4.0)
    for kw, want in (({}, [512, 1024]), ({"slice": 2048}, [2048, 2048]), ({"slices": {4096: 256}}, [256, 1024]),
                     ({"slices": [1024, 0], "slice": 2048}, [1024, 2048])):
        with hw.Engine([a, b], **kw) as e:
            assert e.slices == want, kw
    with hw.Engine(a, cluster=16) as e:
        assert e.slices == [256]
