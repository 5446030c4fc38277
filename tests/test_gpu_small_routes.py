"""Small boxes whose rows are no power of two run one cell per thread, in the adjoint's
steps and in z-slabs as in the time loop (below 2^17 cells the several-cells kernels
leave the chip idle). The results are the same bits either way, so the kernels' names
are looked at."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _kernels(work):
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.init()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        work()
        torch.cuda.synchronize()
    names = {e.key for e in prof.key_averages() if "bgk::" in e.key}
    if not names:
        pytest.skip("no kernel names from the profiler here")
    return names


@pytest.mark.parametrize("n,wide", [(33, False), (50, False), (66, True), (32, True), (64, True)])
def test_adjoint_steps(bgk, n, wide):
    rng = np.random.default_rng(3)
    u = [np.ascontiguousarray(0.03 * rng.standard_normal((n, n, n))) for _ in range(6)]
    dp = C.POINTER(C.c_double)
    box = bgk.BGK3D(n, precision="fp32")
    loss = C.c_double()

    def work():
        assert box._lib.bgk_adjoint(box._h, *(a.ctypes.data_as(dp) for a in u), 4, 2, C.byref(loss), None, None) == 0

    names = _kernels(work)
    assert any("k_two_f32v" in k for k in names) == wide, names
    assert any("k_two<" in k for k in names) != wide, names
    box.close()


@pytest.mark.parametrize("form,kernel", [("fp32", "k_two_f32v"), ("fp16", "k_two_f16v")])
@pytest.mark.parametrize("n,wide", [(34, False), (66, True), (32, True)])
def test_slab_interiors(bgk, form, kernel, n, wide):
    from bgk3d_hit_b200.slabs import LocalSlabs

    slabs = LocalSlabs(n, n, n * 2, 2, precision=form, fp16_scale=4096.0 if form == "fp16" else 0.0)
    slabs.init_velocity(*(np.zeros((2 * n, n, n)) for _ in range(3)))
    names = _kernels(lambda: slabs.step(1))
    assert any(kernel in k for k in names) == wide, names
    slabs.close()
