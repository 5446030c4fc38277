"""Rows of any length on the several-cells-per-thread kernels (FP32 and FP16,
both schemes, BGK and Smagorinsky) against the one-cell-per-thread kernels, bit
for bit: rows shorter than a chunk, last chunks of every size, row ends in the
middle of a warp, rows over several warps and blocks, planes that do not fill
their last block.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 5, 4), (2, 3, 3), (3, 7, 2), (5, 9, 3), (6, 4, 5), (7, 33, 3), (10, 13, 2), (11, 3, 4), (24, 5, 3),
          (40, 11, 2), (61, 6, 3), (66, 3, 3), (96, 5, 2), (130, 3, 2), (201, 4, 3), (264, 3, 2), (517, 3, 2),
          (1040, 2, 2)]


@pytest.mark.parametrize("les", [0.0, 0.17])
@pytest.mark.parametrize("scheme", ["two_lattice", "aa"])
@pytest.mark.parametrize("form", ["fp32", "fp16"])
def test_any_row_length_matches_the_one_cell_kernels(bgk, form, scheme, les):
    rng = np.random.default_rng(3)
    for nx, ny, nz in SHAPES:
        u = [0.05 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
        boxes = [bgk.BGK3D(nx, ny, nz, svisc=0.02, precision=form, scheme=scheme, les_cs=les, kernel=k)
                 for k in (1, 0, 4 if form == "fp16" else 2)]
        for b in boxes:
            b.init_velocity(*u)
        for step in range(4):
            for b in boxes:
                b.run(1)
            ref = boxes[0].populations().view(np.uint8)
            for b in boxes[1:]:
                assert np.array_equal(b.populations().view(np.uint8), ref), (nx, ny, nz, step)
        for b in boxes:
            b.close()


# boxes that the automatic choice runs on the widest kernels: aligned rows within
# a warp, of one warp, of several warps and blocks; rows of whole 16-byte chunks
# of no power of two; ragged ones
BIG = [(64, 64, 64), (256, 32, 32), (512, 32, 16), (1024, 16, 16), (24, 105, 105), (40, 82, 81), (264, 63, 16),
       (1040, 16, 16), (61, 66, 66), (90, 55, 54)]


@pytest.mark.parametrize("les", [0.0, 0.17])
@pytest.mark.parametrize("scheme", ["two_lattice", "aa"])
@pytest.mark.parametrize("form", ["fp64", "fp32", "fp16"])
def test_automatic_kernels_match_the_one_cell_kernels(bgk, form, scheme, les):
    rng = np.random.default_rng(5)
    for nx, ny, nz in BIG:
        u = [0.05 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
        ref, box = (bgk.BGK3D(nx, ny, nz, svisc=0.02, precision=form, scheme=scheme, les_cs=les, kernel=k)
                    for k in (1, 0))
        for b in (ref, box):
            b.init_velocity(*u)
            b.run(5)
        assert np.array_equal(box.populations().view(np.uint8), ref.populations().view(np.uint8)), (nx, ny, nz)
        ref.close()
        box.close()


@pytest.mark.parametrize("form", ["fp32", "fp16"])
def test_any_row_length_in_slabs(bgk, form):
    from bgk3d_hit_b200.slabs import LocalSlabs

    rng = np.random.default_rng(4)
    for nx, ny, nz in ((7, 5, 12), (66, 3, 8), (201, 4, 8)):
        u = [0.05 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
        one = bgk.BGK3D(nx, ny, nz, svisc=0.02, precision=form, kernel=1, fp16_scale=4096.0 if form == "fp16" else 0.0)
        one.init_velocity(*u)
        slabs = LocalSlabs(nx, ny, nz, 2, svisc=0.02, precision=form,
                           fp16_scale=4096.0 if form == "fp16" else 0.0)
        slabs.init_velocity(*u)
        one.run(3)
        for it in range(1, 4):
            slabs.step(it)
        assert np.array_equal(np.asarray(slabs.populations()).view(np.uint8), one.populations().view(np.uint8))
        one.close()
        slabs.close()
