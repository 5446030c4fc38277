"""Read-back paths on the GPU at the sizes where they change: shells of the
spectrum in tables and by atomics, velocity in one chunk and in several,
populations copied directly and through the export kernel, in either layout.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CX = np.array([1, 1, 1, 1, 1, 0, 0, 0, 0, -1, -1, -1, -1, -1, 0, 0, 0, 0, 0])
CY = np.array([-1, 0, 1, 0, 0, 0, 1, 1, 1, -1, 0, 1, 0, 0, 0, -1, -1, -1, 0])
CZ = np.array([0, -1, 0, 1, 0, 1, 1, 0, -1, 0, -1, 0, 1, 0, -1, -1, 0, 1, 0])


def _box(bgk, shape, form, scheme="two_lattice", seed=7, steps=3):
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    box = bgk.BGK3D(nx, ny, nz, svisc=0.05, u0=0.05, precision=form, scheme=scheme)
    box.init_velocity(*(0.02 * rng.standard_normal((nz, ny, nx)) for _ in range(3)))
    box.run(steps)
    return box


def _velocity_from(box):
    """Velocity from the box's deviations in 64 bits, and the rounding bound of
    the form's arithmetic: 10 additions, a reciprocal and a product."""
    d = box.deviations()
    rho = 1.0 + d.sum(0)
    eps = np.finfo(np.float64 if box.dtype == np.float64 else np.float32).eps
    out = []
    for c in (CX, CY, CZ):
        mag = np.abs(d[c != 0]).sum(0) + np.abs(d).sum(0) + 1.0
        out.append((np.tensordot(c.astype(float), d, 1) / rho, 16 * eps * (np.abs(d[c != 0]).sum(0) * mag)))
    return out


@pytest.mark.parametrize("form", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("shape", [(33, 20, 7), (32, 8, 4), (131, 129, 128), (64, 64, 513)])
def test_velocity_in_chunks(bgk, shape, form):
    """(131, 129, 128) and (64, 64, 513) take two chunks (the second of one plane)."""
    for scheme in ("two_lattice", "aa"):
        box = _box(bgk, shape, form, scheme)
        for got, (want, tol) in zip(box.velocity(), _velocity_from(box)):
            assert np.all(np.abs(got - want) <= tol + 1e-18)
        box.close()


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("shape", [(32, 32, 32), (33, 20, 7), (6, 5, 70), (1530, 4, 4), (1600, 4, 4), (20000, 2, 2)])
def test_spectrum_shells(bgk, shape, form):
    """Up to 768 shells in tables, (1600, 4, 4) and (20000, 2, 2) by atomics;
    also fewer bins asked for than there are shells."""
    nx, ny, nz = shape
    box = _box(bgk, shape, form, steps=1)
    k = [np.fft.fftfreq(n, 1.0 / n) for n in (nz, ny, nx)]
    k2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    shell = np.floor(np.sqrt(k2) + 0.5).astype(int).ravel()
    e = sum(np.abs(np.fft.fftn(c)) ** 2 for c in box.velocity()).ravel() * 0.5 / (nx * ny * nz) ** 2
    want = np.bincount(shell, e)
    for nb in (max(shape) // 2 + 1, 5, len(want) + 9):
        got = box.spectrum(nb)
        ref = np.zeros(nb)
        ref[:min(nb, len(want))] = want[:nb]
        # FFT rounding: log2(cells) stages of about one eps each, relative to the total energy
        eps = np.finfo(np.float64 if form == "fp64" else np.float32).eps
        assert np.allclose(got, ref, rtol=64 * eps * np.log2(nx * ny * nz), atol=8 * eps * e.sum())
    box.close()


@pytest.mark.parametrize("form", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("shape", [(32, 8, 4), (64, 5, 3), (33, 8, 4), (160, 160, 131)])
@pytest.mark.parametrize("steps", [3, 4])
def test_populations_round_trip(bgk, shape, form, steps):
    """Rows without padding go by plain copies (except in the AA layout between
    its two steps), the others through the kernels, in one piece or several;
    both schemes hold the same bits, and an upload is read back as it was."""
    a, b = _box(bgk, shape, form, "two_lattice", steps=steps), _box(bgk, shape, form, "aa", steps=steps)
    pa, pb = a.populations(), b.populations()
    assert np.array_equal(pa.view(np.uint8), pb.view(np.uint8))
    scale = a.scale
    assert np.array_equal(a.deviations(), pa.astype(np.float64) / scale)
    mark = (np.arange(pa.size) % 2039).reshape(pa.shape).astype(pa.dtype)
    for box in (a, b):
        box.set_populations(mark)
        assert np.array_equal(box.populations(), mark)
        box.close()
