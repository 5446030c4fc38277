"""Read-back of populations, deviations and velocity on a device that has little memory
left: the staging takes the size that can be had."""
import numpy as np
import pytest

from test_gpu_full_device import MB, Filled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp64", "fp32"])
def test_read_back_in_what_is_left(bgk, form):
    n = 60  # padded rows; 1.7 MB per population or component in double

    def look(b):
        return [b.populations(), b.deviations(), np.asarray(b.velocity())]

    ref, box = bgk.BGK3D(n, precision=form), bgk.BGK3D(n, precision=form)
    for b in (ref, box):
        b.init()
        b.run(3)
        b.synchronize()
    want = look(ref)
    pops = want[0]
    with Filled(4 * MB):
        box.set_populations(pops)
        got = look(box)
    for a, b in zip(got, want):
        assert np.array_equal(a.view(np.uint8), b.view(np.uint8))
    ref.close()
    box.close()
