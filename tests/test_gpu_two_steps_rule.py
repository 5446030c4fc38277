"""Which boxes take two steps per launch: flat ones, whose walks are a few planes long
and which were up to 2.3 times slower that way, keep single steps; boxes that the rule
newly takes give the bits of single steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,les,shape", [
    ("fp64", 0.0, (512, 512, 8)), ("fp64", 0.0, (1024, 1024, 4)), ("fp64", 0.0, (1024, 512, 10)),
    ("fp64", 0.17, (512, 512, 8)), ("fp64", 0.17, (512, 512, 16)), ("fp64", 0.17, (1024, 1024, 16)),
    ("fp64", 0.17, (2000, 64, 24)), ("fp32", 0.0, (1024, 1024, 8))])
def test_flat_boxes_keep_single_steps(bgk, form, les, shape):
    box = bgk.BGK3D(*shape, precision=form, les_cs=les)
    box.init()
    l0 = box.launch_count
    box.run(4)
    assert box.launch_count - l0 == 4
    box.close()


@pytest.mark.parametrize("form,les,shape,pairs", [
    ("fp64", 0.0, (512, 512, 16), True), ("fp64", 0.0, (130, 130, 130), True), ("fp64", 0.17, (136, 136, 136), True),
    ("fp64", 0.17, (144, 144, 144), True), ("fp64", 0.17, (256, 256, 64), True), ("fp32", 0.0, (140, 140, 140), True),
    ("fp32", 0.0, (129, 200, 200), True), ("fp32", 0.0, (150, 150, 150), True), ("fp64", 0.0, (80, 80, 80), False),
    ("fp32", 0.0, (128, 128, 128), False)])
def test_boxes_near_the_line(bgk, form, les, shape, pairs):
    nx, ny, nz = shape
    rng = np.random.default_rng(29)
    u = [0.04 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
    ref, box = (bgk.BGK3D(nx, ny, nz, svisc=0.03, precision=form, les_cs=les, kernel=k) for k in (1, 0))
    for b in (ref, box):
        b.init_velocity(*u)
    l0 = box.launch_count
    for b in (ref, box):
        b.run(5)
    assert box.launch_count - l0 == (3 if pairs else 5)
    assert np.array_equal(ref.populations().view(np.uint8), box.populations().view(np.uint8))
    ref.close()
    box.close()
