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


# a cluster per molecule; the sweeps of tiles; periodic.  50 and 51: the last exponent of the FP32 triples and the next
@pytest.mark.parametrize("natoms, periodic", [(40, False), (300, False), (45, True)])
@pytest.mark.parametrize("alp", [13.0, 50.0, 51.0, 100.0, 200.0])
def test_steep_damping(natoms, periodic, alp):
    """The three-body part within the mixed form's budget of 1e-7 of the total energy and 1e-7 Hartree/Bohr."""
    from dftd3 import synthetic as S
    from dftd3.interface import DispersionModel, RationalDampingParam
    rng = np.random.default_rng(natoms)
    num = rng.choice([1, 6, 7, 8], size=natoms).astype(np.int32)
    side = (natoms / 0.012) ** (1 / 3) + 1.0
    pos = S.pack_box(rng, natoms, 0.0, side, 1.4)
    pos[1] = pos[0] + [0.0, 0.0, 1.4]               # a bond of hydrogen
    num[:2] = 1
    model = DispersionModel(num, pos, np.eye(3) * (side + 2.0) if periodic else None,
                            np.ones(3, dtype=bool) if periodic else None)
    model.set_realspace_cutoff(20.0, 15.0, 15.0)
    res = {}
    for precision in ("fp64", "mixed"):
        model.set_precision(precision)
        for s9 in (0.0, 1.0):
            param = RationalDampingParam(**{k: S.PBE_BJ[k] for k in ("s6", "s8", "a1", "a2")}, alp=alp, s9=s9)
            res[precision, s9] = model.get_dispersion(param, grad=True)
            energy = float(model.get_dispersion(param, grad=False)["energy"])
            assert abs(energy - float(res[precision, s9]["energy"])) <= 1e-7 * abs(energy)
    part = {p: (float(res[p, 1.0]["energy"]) - float(res[p, 0.0]["energy"]),
                res[p, 1.0]["gradient"] - res[p, 0.0]["gradient"]) for p in ("fp64", "mixed")}
    total = abs(float(res["fp64", 1.0]["energy"]))
    assert abs(part["mixed"][0] - part["fp64"][0]) <= 1e-7 * total
    assert np.abs(part["mixed"][1] - part["fp64"][1]).max() <= 1e-7
