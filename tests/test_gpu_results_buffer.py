"""GPU test of the two ways pair matrices and Hessians reach the host: stores to a
pinned buffer up to 2^20 doubles (Hessians of 341 atoms, matrices of 724) and copies
above.  Oracle sizes have their tests elsewhere; here the sums that the result obeys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _model(natoms):
    from dftd3 import synthetic as S
    from dftd3.interface import DispersionModel, RationalDampingParam
    rng = np.random.default_rng(natoms)
    edge = (natoms / 0.02) ** (1 / 3) + 2.0
    num = rng.choice([1, 6, 7, 8], size=natoms).astype(np.int32)
    pos = S.pack_cell(rng, natoms, edge * np.eye(3), 2.0)
    return rng, pos, DispersionModel(num, pos), RationalDampingParam(method="pbe", atm=True)


@pytest.mark.parametrize("natoms", [1, 5, 6, 341, 342])
def test_hessian_sizes(natoms):
    """Symmetric, zero under a translation (rounding of 3 n entries of TOL 1e-12 of the
    largest: 1e-11), and along a direction the fourth-order difference of the gradient
    (the second-order one is 2e-4 off at this step, so this one some 1e-7: bound 1e-4)."""
    rng, pos, model, param = _model(natoms)
    h = np.asarray(model.get_hessian(param)["hessian"])
    assert h.shape == (3 * natoms, 3 * natoms)
    scale = max(np.abs(h).max(), 1e-300)
    assert np.abs(h - h.T).max() <= 1e-12 * scale
    assert np.abs(h.reshape(3 * natoms, natoms, 3).sum(axis=1)).max() <= 1e-11 * scale
    v = rng.standard_normal(pos.shape)
    hv = h @ v.ravel()
    num = np.zeros_like(hv)
    for step, weight in ((1e-3, 8.0), (-1e-3, -8.0), (2e-3, -1.0), (-2e-3, 1.0)):
        model.update(pos + step * v)
        num += weight / 12e-3 * model.get_dispersion(param, grad=True)["gradient"].ravel()
    assert np.abs(num - hv).max() <= 1e-4 * np.abs(hv).max()


@pytest.mark.parametrize("natoms", [1, 2, 33, 724, 725])
def test_pairwise_sizes(natoms):
    """Symmetric matrices that sum to the energies of the two parts."""
    from dftd3.interface import RationalDampingParam
    _, _, model, param = _model(natoms)
    pw = model.get_pairwise_dispersion(param)
    e = model.get_dispersion(param, grad=False)["energy"]
    e2 = model.get_dispersion(RationalDampingParam(method="pbe", atm=False), grad=False)["energy"]
    for key, want in (("additive pairwise energy", e2), ("non-additive pairwise energy", e - e2)):
        m = np.asarray(pw[key])
        assert m.shape == (natoms, natoms)
        assert np.abs(m - m.T).max() <= 1e-12 * np.abs(m).max()
        assert abs(m.sum() - want) <= 1e-11 * abs(e)
