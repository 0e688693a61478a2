"""The MLP's update step: BF16 weight copies written by Adam, and gradients
added to an aligned or an unaligned buffer."""
import ctypes

import numpy as np
import pytest

from pylbm_gb300 import closure, runtime

pytestmark = pytest.mark.gpu


def _copies(mlp):
    out = np.empty(mlp.nweights, dtype=np.uint16)
    mlp.w.download(out)
    return out


def test_adam_writes_the_copies_that_sync_writes():
    rng = np.random.default_rng(5)
    mlp = closure.Mlp(seed=5)
    before = _copies(mlp)
    mlp.w.upload(np.full(mlp.nweights, 0x7FC0, dtype=np.uint16))   # every place has to be written
    mlp.set_grad(rng.normal(size=mlp.nparam))
    mlp.adam_step(1e-2)
    got = _copies(mlp)
    mlp.sync()
    ref = _copies(mlp)
    assert np.array_equal(got, ref) and not np.array_equal(got, before)
    assert not mlp.grad_host().any()


@pytest.mark.parametrize("n", [1, 129, 20000])
def test_gradients_to_an_unaligned_buffer(n):
    rng = np.random.default_rng(n)
    mlp = closure.Mlp(seed=1)
    dx, dt, _ = mlp._device_data(rng.normal(size=(n, closure.IN)), rng.normal(size=(n, closure.OUT)))
    grads = []
    for shift in (0, 4):
        g = runtime.DeviceBuffer(4 * mlp.nparam + 16)
        g.zero(None)
        runtime.check(mlp._core.lbm_mlp_gradients_tc(dx.handle, dt.handle, n, mlp.p.handle,
                                                     ctypes.c_void_p(g.ptr + shift), mlp.loss.handle, None))
        out = np.empty(mlp.nparam, dtype=np.float32)
        g.download(out, offset=shift)
        grads.append(out)
    # the same values added by up to 152 blocks in another order
    assert np.abs(grads[0]).max() > 0
    assert np.allclose(grads[0], grads[1], rtol=0, atol=152 * 2.0**-24 * np.abs(grads[0]).max())
