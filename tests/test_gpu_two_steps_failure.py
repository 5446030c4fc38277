"""The bounded wait of the kernel that takes two steps per launch: injected by a plane
that is never asked for, it abandons the pair, every call that looks at the state
reports it, and a new state makes the context whole again. No fault is involved."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [("fp64", 0.0, (128, 128, 128)), ("fp64", 0.17, (190, 177, 190)), ("fp32", 0.0, (224, 190, 180))]


@pytest.mark.parametrize("steps", [2, 7])
@pytest.mark.parametrize("form,les,shape", CASES)
def test_a_wait_that_runs_out_is_reported_and_the_context_recovers(bgk, form, les, shape, steps):
    nx, ny, nz = shape
    rng = np.random.default_rng(23)
    u = [0.04 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
    box = bgk.BGK3D(nx, ny, nz, svisc=0.03, precision=form, les_cs=les, icheck=1)
    ref = bgk.BGK3D(nx, ny, nz, svisc=0.03, precision=form, les_cs=les, kernel=1)
    for b in (box, ref):
        b.init_velocity(*u)
    start = box.populations()
    assert box._lib.bgk_debug_stall_next_step(box._h) == 0
    box.run(steps)
    for look in (box.synchronize, lambda: box.diagnostic(steps), box.populations):
        with pytest.raises(bgk.BgkError) as e:
            look()
        assert e.value.code == bgk._abi.BGK_ERR_CUDA and "gave up" in str(e.value)
    box.set_populations(start)
    for b in (box, ref):
        b.run(steps)
        b.synchronize()
    assert np.array_equal(box.populations().view(np.uint8), ref.populations().view(np.uint8))
    box.close()
    ref.close()


def test_adjoint_reports_a_wait_that_runs_out(bgk):
    n = 128
    rng = np.random.default_rng(3)
    u = [np.ascontiguousarray(0.03 * rng.standard_normal((n, n, n))) for _ in range(6)]
    dp = C.POINTER(C.c_double)
    box = bgk.BGK3D(n, svisc=0.03)
    loss = [C.c_double(), C.c_double()]

    def adjoint(out):
        return box._lib.bgk_adjoint(box._h, *(a.ctypes.data_as(dp) for a in u), 6, 3, C.byref(out), None, None)

    assert adjoint(loss[0]) == 0
    assert box._lib.bgk_debug_stall_next_step(box._h) == 0
    assert adjoint(C.c_double()) == bgk._abi.BGK_ERR_CUDA
    box.init()
    assert adjoint(loss[1]) == 0
    assert loss[0].value == loss[1].value
    box.close()


def test_stall_hook_is_refused_where_no_kernel_waits(bgk):
    for kw in (dict(kernel=1), dict(scheme="aa"), dict(mode="faithful"), dict(precision="fp16")):
        box = bgk.BGK3D(128, **kw)
        assert box._lib.bgk_debug_stall_next_step(box._h) == bgk._abi.BGK_ERR_INVALID
        box.close()
