"""GPU tests of the three-body sums of primitive cells with large cutoffs, where all root contributions fall on one or
two atoms: the gradient vanishes by symmetry, and energy and virial are those of the conventional cell per atom (1e-12,
the bound of the other three-body tests; the oracle adds the 6e7 terms of such a cell one by one, to 1.4e-12 only).
Mixed form: a triple is a product of nine pair values, each within about two units of 2^-24, so two evaluations agree
within 2 x 9 x 2 x 2^-24, about 2e-6."""
import numpy as np
import pytest

from test_gpu_twobody import GTOL64, RTOL64

pytestmark = pytest.mark.gpu
TOL_MIXED = 2.0e-6


def _evaluate(z, pos, lat, cut, precision):
    from dftd3 import synthetic as S
    from dftd3.interface import DispersionModel, RationalDampingParam
    model = DispersionModel(np.full(len(pos), z), np.array(pos), lat, np.ones(3, dtype=bool))
    model.set_realspace_cutoff(*cut)
    model.set_precision(precision)
    param = RationalDampingParam(**{k: S.PBE_BJ[k] for k in ("s6", "s8", "a1", "a2", "alp")}, s9=1.0)
    return model.get_dispersion(param, grad=True)


@pytest.mark.parametrize("precision, etol, gtol", [("fp64", RTOL64, GTOL64), ("mixed", TOL_MIXED, TOL_MIXED)])
# fcc Cu and diamond; additions to one atom's sums: 3.0e7, 1.8e8 and 1.5e7
@pytest.mark.parametrize("z, a, disp3", [(29, 6.83, 60.0), (29, 6.83, 79.9), (6, 6.74, 50.0)])
def test_primitive_and_conventional_cell(z, a, disp3, precision, etol, gtol):
    cut = (30.0, disp3, 20.0, 0.0, 0.0)
    prim = 0.5 * a * np.array([[0.0, 1.0, 1.0], [1.0, 0.0, 1.0], [1.0, 1.0, 0.0]])
    basis = np.array([[0.0] * 3, [0.25 * a] * 3])[:2 if z == 6 else 1]
    corners = np.vstack([np.zeros(3), prim])
    one = _evaluate(z, basis, prim, cut, precision)
    four = _evaluate(z, (corners[:, None] + basis[None]).reshape(-1, 3), np.eye(3) * a, cut, precision)
    energy, virial = float(four["energy"]) / 4, four["virial"] / 4
    assert abs(float(one["energy"]) - energy) <= etol * abs(energy)
    scale = np.abs(virial).max()
    for res in (one, four):
        assert np.abs(res["gradient"]).max() <= gtol * scale
    assert np.abs(one["virial"] - virial).max() <= gtol * scale
