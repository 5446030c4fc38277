"""Two steps per launch (bgk_run on two-lattice boxes) against single steps on the
one-cell-per-thread kernel, bit for bit: last tiles of every width and height, a
tile that ends one cell before a face, walks of uneven length, odd step counts,
single and fused steps mixed, and the places of the rest population after each.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COMMON = [(62, 514, 150), (190, 177, 190), (255, 127, 140), (257, 240, 190)]
SHAPES = {("fp64", 0.0): COMMON + [(128, 128, 128), (161, 121, 160), (97, 250, 200), (543, 66, 67), (96, 18, 2000)],
          ("fp64", 0.17): COMMON + [(128, 128, 128), (543, 66, 67), (96, 18, 2000)],
          ("fp32", 0.0): COMMON + [(543, 67, 100), (224, 190, 180)]}


def _pair(bgk, shape, form, les):
    nx, ny, nz = shape
    rng = np.random.default_rng(11)
    u = [0.04 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
    boxes = [bgk.BGK3D(nx, ny, nz, svisc=0.03, precision=form, les_cs=les, kernel=k) for k in (1, 0)]
    for b in boxes:
        b.init_velocity(*u)
    return boxes


def _same(a, b):
    return np.array_equal(a.populations().view(np.uint8), b.populations().view(np.uint8))


@pytest.mark.parametrize("form,les,shape", [(f, les, shape) for (f, les), v in SHAPES.items() for shape in v])
def test_two_steps_per_launch_match_single_steps(bgk, form, les, shape):
    ref, box = _pair(bgk, shape, form, les)
    l0 = box.launch_count
    ref.run(5)
    box.run(5)
    assert box.launch_count - l0 == 3  # two pairs and a single step
    assert box.step == 5
    assert _same(ref, box)
    ref.close()
    box.close()


@pytest.mark.parametrize("form,les,scheme,mode,shape", [
    ("fp16", 0.0, "two_lattice", "corrected", (128, 128, 128)), ("fp32", 0.17, "two_lattice", "corrected", (256, 128, 128)),
    ("fp64", 0.0, "aa", "corrected", (128, 128, 128)), ("fp64", 0.0, "two_lattice", "faithful", (128, 128, 128)),
    ("fp64", 0.0, "two_lattice", "corrected", (33, 400, 400)), ("fp64", 0.0, "two_lattice", "corrected", (400, 9, 400)),
    ("fp64", 0.0, "two_lattice", "corrected", (64, 64, 64))])
def test_other_boxes_keep_single_steps(bgk, form, les, scheme, mode, shape):
    box = bgk.BGK3D(*shape, precision=form, les_cs=les, scheme=scheme, mode=mode)
    box.init()
    box.run(1)
    l0, l1 = box.launch_count, None
    box.run(2)
    l1 = box.launch_count
    assert l1 - l0 == (4 if mode == "faithful" else 2)  # faithful mode also keeps the boundary planes
    box.close()


def test_fused_and_single_steps_mixed(bgk):
    ref, box = _pair(bgk, (160, 144, 128), "fp64", 0.0)
    l0 = box.launch_count
    for n in (1, 2, 3, 1, 4, 1):
        ref.run(n)
        if n == 1:
            box.col_MC(0)
        else:
            box.run(n)
        d, e = ref.diagnostic(0), box.diagnostic(0)
        assert d == e
        assert _same(ref, box)
    assert box.launch_count - l0 == 3 * 1 + 1 + 2 + 2 + 6 * 3  # singles, pairs (and one odd), diagnostics
    box.set_populations(ref.populations())
    ref.run(2)
    box.run(2)
    assert _same(ref, box)
    ref.close()
    box.close()


@pytest.mark.parametrize("steps", [4, 7])
def test_adjoint_forward_in_pairs(bgk, steps):
    """States that no checkpoint keeps are passed over two steps at a time; with a
    checkpoint at every step none are. The results are the same bits."""
    import ctypes as C

    nx, ny, nz = shape = (128, 128, 128)
    rng = np.random.default_rng(2)
    u = [np.ascontiguousarray(0.03 * rng.standard_normal((nz, ny, nx))) for _ in range(6)]
    dp = C.POINTER(C.c_double)
    box = bgk.BGK3D(*shape, svisc=0.03)
    got = []
    for every in (1, 3, 7):
        loss, gtau, grad = C.c_double(), C.c_double(), np.zeros((3, nz, ny, nx))
        rc = box._lib.bgk_adjoint(box._h, *(a.ctypes.data_as(dp) for a in u), steps, every, C.byref(loss),
                                  grad.ctypes.data_as(dp), C.byref(gtau))
        assert rc == 0
        got.append((loss.value, gtau.value, grad))
    for loss, gtau, grad in got[1:]:
        assert loss == got[0][0] and gtau == got[0][1]
        assert np.array_equal(grad, got[0][2])
    box.close()
