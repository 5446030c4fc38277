"""Launches that overlap the end of the kernel before them, over runs of many steps on
boxes of several waves: the in-place AA steps, whose successor is resident while they
read and write the same lines, give the bits of the two-lattice scheme on the
one-cell-per-thread kernel, which is synchronised after every step.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("les", [0.0, 0.17])
@pytest.mark.parametrize("form", ["fp64", "fp32", "fp16"])
def test_long_aa_runs_match_separate_steps(bgk, form, les):
    rng = np.random.default_rng(17)
    for nx, ny, nz in ((256, 96, 96), (250, 90, 101)):
        u = [0.04 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
        ref = bgk.BGK3D(nx, ny, nz, svisc=0.02, precision=form, les_cs=les, kernel=1)
        boxes = [bgk.BGK3D(nx, ny, nz, svisc=0.02, precision=form, scheme="aa", les_cs=les, kernel=k) for k in (0, 1)]
        for b in [ref] + boxes:
            b.init_velocity(*u)
        for _ in range(61):
            ref.run(1)
            ref.synchronize()
        want = ref.populations().view(np.uint8)
        ref.close()
        for b in boxes:
            b.run(61)
            assert np.array_equal(b.populations().view(np.uint8), want), (nx, ny, nz)
            b.close()
