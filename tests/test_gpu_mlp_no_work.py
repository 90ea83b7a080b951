"""Training calls without a step to take succeed, whatever their batch: the mean loss of
no records is NaN, the parameters stay.  A batch that could take no step is an error."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,epochs,batch,rc", [
    (0, 2, 64, 0), (0, 2, 0, 0), (0, 2, -1, 0), (8, 0, 4, 0), (8, 0, 0, 0), (8, -1, 0, 0), (8, 2, 0, 1), (8, 2, -4, 1),
    (-1, 2, 4, 1)])
def test_no_work(n, epochs, batch, rc):
    from hawassi_c_b200 import learned
    from hawassi_c_b200.engine import load_library
    mlp = learned.MLP(seed=1)
    p = mlp.params()
    rec = np.ones((8, 45), np.float32)
    losses = np.zeros(4, np.float32)
    fp = ctypes.POINTER(ctypes.c_float)
    got = load_library().hw_mlp_train(mlp._h, rec.ctypes.data_as(fp), n, epochs, batch, 1e-3, losses.ctypes.data_as(fp))
    assert got == rc
    if rc == 0:
        assert np.isnan(losses[:max(epochs, 0)]).all() and not losses[max(epochs, 0):].any()
    assert np.array_equal(mlp.params(), p)
