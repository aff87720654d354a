"""GPU test of the mixed form's triples, one at a time: near-equilateral triangles of carbon at distances where the
damping acts, with a steep exponent, against the FP64 form.  The pair values of a triple are rounded once each from
FP64; with the FP32 arithmetic of the triple some 40 roundings of at most 2^-24 / sqrt(3) (root mean square), so the
error over many triangles is below sqrt(40 / 3) x 2^-24 = 2.2e-7, twice that allowed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alp", [14.0, 60.0])
def test_triangles(alp):
    from dftd3.interface import BatchedDispersion, RationalDampingParam
    rng = np.random.default_rng(1)
    n = 2000
    r = rng.uniform(6.5, 8.5, size=(n, 1, 1))      # the ATM radius of two carbon atoms is 7.3 Bohr
    tri = np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [0.5, 0.75 ** 0.5, 0.0]]) * r + rng.uniform(-0.2, 0.2, size=(n, 3, 3))
    bat = BatchedDispersion([np.array([6, 6, 6])] * n, list(tri))
    param = RationalDampingParam(s6=0.0, s8=0.0, a1=0.4, a2=4.4, alp=alp, s9=1.0)
    res = {}
    for precision in ("fp64", "mixed"):
        bat.set_precision(precision)
        res[precision] = np.array(bat.get_dispersion(param, grad=True)["energy"])
    err = res["mixed"] / res["fp64"] - 1.0
    assert np.sqrt((err ** 2).mean()) <= 4.4e-7
