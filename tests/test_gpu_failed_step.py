"""A step that gave up (injected on the row-pipelined kernel: a wait that runs out, no
fault) is reported by every call that hands out fields of the invalid state."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(64, 16, 8), (256, 128, 96)])  # a chunk of planes, several
@pytest.mark.parametrize("look", ["velocity", "spectrum"])
def test_fields_of_a_failed_step_are_refused(bgk, look, shape):
    box = bgk.BGK3D(*shape, kernel=8)
    box.init()
    want = getattr(box, look)()
    assert box._lib.bgk_debug_stall_next_step(box._h) == 0
    box.run(1)
    with pytest.raises(bgk.BgkError) as e:
        getattr(box, look)()
    assert e.value.code == bgk._abi.BGK_ERR_CUDA and "gave up" in str(e.value)
    box.init()
    assert np.allclose(np.asarray(getattr(box, look)()), np.asarray(want), rtol=1e-12, atol=1e-30)
    box.close()
