"""bgk_adjoint runs on states of its own: a context whose time loop failed still gives
gradients, and an adjoint that failed leaves the time loop's state valid."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _adjoint(box, n, steps=6):
    rng = np.random.default_rng(3)
    u = [np.ascontiguousarray(0.03 * rng.standard_normal((n, n, n))) for _ in range(6)]
    dp = C.POINTER(C.c_double)
    loss = C.c_double()
    rc = box._lib.bgk_adjoint(box._h, *(a.ctypes.data_as(dp) for a in u), steps, 3, C.byref(loss), None, None)
    return rc, loss.value


def test_adjoint_of_a_context_whose_step_failed(bgk):
    n = 24
    box = bgk.BGK3D(n, kernel=8)
    box.init()
    want = _adjoint(box, n)
    assert want[0] == 0
    assert box._lib.bgk_debug_stall_next_step(box._h) == 0
    box.run(1)
    with pytest.raises(bgk.BgkError):
        box.synchronize()
    assert _adjoint(box, n) == want
    with pytest.raises(bgk.BgkError):
        box.synchronize()
    box.close()


def test_state_of_a_context_whose_adjoint_failed(bgk):
    n = 128
    box = bgk.BGK3D(n, icheck=1)
    box.init()
    box.run(4)
    want, rec = box.populations(), box.diagnostic(4)
    good = _adjoint(box, n)
    assert box._lib.bgk_debug_stall_next_step(box._h) == 0
    assert _adjoint(box, n)[0] == bgk._abi.BGK_ERR_CUDA
    box.synchronize()
    assert box.diagnostic(4) == rec
    assert np.array_equal(box.populations().view(np.uint8), want.view(np.uint8))
    assert _adjoint(box, n) == good
    box.close()
