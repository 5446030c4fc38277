"""Two steps per launch against the CPU oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form,les,shape", [("fp64", 0.0, (126, 121, 127)), ("fp64", 0.17, (136, 136, 136)),
                                            ("fp32", 0.0, (150, 145, 150))])
def test_pairs_and_an_odd_step_give_the_oracles_bits(bgk, oracle_mod, form, les, shape):
    nx, ny, nz = shape
    rng = np.random.default_rng(31)
    u = [0.04 * rng.standard_normal((nz, ny, nx)) for _ in range(3)]
    orc = oracle_mod.OracleLattice(nx, ny, nz, form="f64" if form == "fp64" else "f32")
    orc.init_velocity(*(x.ravel() for x in u), 1.0)
    if les:
        orc.set_les(les)
    box = bgk.BGK3D(nx, ny, nz, svisc=0.01, precision=form, les_cs=les)
    box.init_velocity(*u)
    l0 = box.launch_count
    box.run(5)
    assert box.launch_count - l0 == 3
    for _ in range(5):
        orc.step(0.01, periodic=True)
    assert np.array_equal(box.populations().view(np.uint8), orc.get_pops().view(np.uint8))
    box.close()
    orc.close()
