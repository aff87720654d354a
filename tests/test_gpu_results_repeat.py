"""GPU test of the two ways pair matrices and Hessians reach the host: the first request of a model is copied, later ones
are stored to a pinned buffer (up to 2^20 doubles, and again after a larger one), with the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(natoms, periodic=False):
    from dftd3 import synthetic as S
    from dftd3.interface import DispersionModel, RationalDampingParam
    rng = np.random.default_rng(natoms)
    edge = (natoms / 0.02) ** (1 / 3) + 2.0
    num = rng.choice([1, 6, 7, 8], size=natoms).astype(np.int32)
    pos = S.pack_cell(rng, natoms, edge * np.eye(3), 2.0)
    model = DispersionModel(num, pos, edge * np.eye(3) if periodic else None, np.ones(3, dtype=bool) if periodic else None)
    if periodic:
        model.set_realspace_cutoff(15.0, 9.0, 12.0)
    return model, RationalDampingParam(method="pbe", atm=True)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("natoms", [1, 5, 33, 341, 342])
def test_requests_in_turn(natoms, periodic):
    model, param = _model(natoms, periodic)
    first = model.get_pairwise_dispersion(param)
    hess = np.asarray(model.get_hessian(param)["hessian"])
    for _ in range(2):
        again = model.get_pairwise_dispersion(param)
        for key in first:
            assert np.array_equal(again[key], first[key]), key
        assert np.array_equal(np.asarray(model.get_hessian(param)["hessian"]), hess)
    other = _model(natoms, periodic)[0]
    assert np.array_equal(np.asarray(other.get_hessian(param)["hessian"]), hess)
    for key in first:
        assert np.array_equal(other.get_pairwise_dispersion(param)[key], first[key]), key
