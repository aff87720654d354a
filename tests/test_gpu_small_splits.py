"""GPU test of the automatic split of the pair sweeps for systems with few tile
pairs (one to sixteen tiles, 32 to 8 parts of a tile), in the forms that take the
tile sweeps: other damping families, parameter derivatives and the mixed form,
against the FP64 oracle at the bounds of the two-body tests."""
import numpy as np
import pytest

import oracle_ref as O
from test_gpu_twobody import GTOL64, RTOL64

pytestmark = pytest.mark.gpu
MZERO = dict(damping="mzero", s6=1.0, s8=1.532981, rs6=1.338153, rs8=1.0, bet=0.013988, s9=0.0, alp=14.0)
CUT = (31.3, 13.7, 18.9, 0.0, 0.0)


@pytest.mark.parametrize("natoms,periodic", [(3, True), (32, True), (33, True), (130, True), (500, True), (33, False),
                                             (270, False)])
def test_few_tile_pairs(natoms, periodic):
    from dftd3 import synthetic as S
    from dftd3.interface import DispersionModel, ModifiedZeroDampingParam
    rng = np.random.default_rng(natoms)
    edge = (natoms / 0.02) ** (1 / 3) + 2.0
    lat = S.triclinic(edge, 1.03 * edge, 1.08 * edge, 88.0, 91.0, 92.0)
    num = rng.choice([1, 6, 7, 8], size=natoms).astype(np.int32)
    pos = S.pack_cell(rng, natoms, lat, 2.0)
    lat, per = (lat, [True] * 3) if periodic else (None, None)
    model = DispersionModel(num, pos, lat, None if per is None else np.array(per))
    model.set_realspace_cutoff(*CUT)
    keys = ("s6", "s8", "rs6", "rs8", "bet", "alp", "s9")
    res = model.get_dispersion(ModifiedZeroDampingParam(**{k: MZERO[k] for k in keys}), grad=True)
    ref = O.dispersion(num, pos, MZERO, lattice=lat, periodic=per, cutoff=CUT)
    assert abs(float(res["energy"]) - ref["energy"]) <= RTOL64 * abs(ref["energy"])
    for k in ("gradient", "virial"):
        assert np.abs(res[k] - ref[k]).max() <= GTOL64 * np.abs(ref[k]).max(), k


@pytest.mark.parametrize("precision,etol", [("fp64", 1e-12), ("mixed", 1e-7)])
@pytest.mark.parametrize("natoms", [40, 300])
def test_few_tile_pairs_parameter_derivatives(natoms, precision, etol):
    """Energies and gradients of a pass with parameter derivatives (FP64: 1e-12;
    mixed: the form's 1e-7 and 1e-7 Hartree/Bohr)."""
    import torch
    from dftd3 import synthetic as S
    from dftd3.torch_api import D3Batch
    rng = np.random.default_rng(7 * natoms)
    edge = (natoms / 0.02) ** (1 / 3)
    lat = np.diag(edge * np.array([1.0, 1.05, 1.1]))
    num = rng.choice([1, 6, 8], size=natoms).astype(np.int32)
    pos = S.pack_cell(rng, natoms, lat, 2.0)
    par = dict(S.PBE_BJ, damping="rational", s9=0.0)
    model = D3Batch([num], lattices=lat[None], periodic=np.ones((1, 3), dtype=bool), precision=precision, cutoffs=CUT)
    x = torch.tensor(pos, device="cuda", requires_grad=True)
    params = torch.tensor([1.0, par["s8"], par["a1"], par["a2"], 0.0], dtype=torch.float64, device="cuda",
                          requires_grad=True)
    e = model(x, params)
    e.sum().backward()
    ref = O.dispersion(num, pos, par, lattice=lat, periodic=[True] * 3, cutoff=CUT)
    assert abs(e.item() - ref["energy"]) <= etol * abs(ref["energy"])
    gtol = GTOL64 * np.abs(ref["gradient"]).max() if precision == "fp64" else 1e-7
    assert np.abs(x.grad.cpu().numpy() - ref["gradient"]).max() <= gtol


@pytest.mark.parametrize("split", [0, 1, 2, 4])
@pytest.mark.parametrize("natoms", [1, 33, 200])
def test_slot_sums_energy_only(natoms, split):
    """Energies of a pass without derivatives, whose gather reads two values per slot,
    against the pass with them (1e-14 of the energy: the same sums), for every way the
    tile pairs are cut."""
    from dftd3 import library as lib, synthetic as S
    from dftd3.interface import BatchedDispersion, ModifiedZeroDampingParam
    rng = np.random.default_rng(natoms)
    edge = (natoms / 0.02) ** (1 / 3) + 2.0
    num = rng.choice([1, 6, 7, 8], size=natoms).astype(np.int32)
    pos = S.pack_cell(rng, natoms, edge * np.eye(3), 2.0)
    keys = ("s6", "s8", "rs6", "rs8", "bet", "alp", "s9")
    param = ModifiedZeroDampingParam(**{k: MZERO[k] for k in keys})
    model = BatchedDispersion([num], [pos], edge * np.eye(3)[None], np.ones((1, 3), dtype=bool))
    lib.set_batch_tuning(model._batch, 0.0, split, 0)
    full = model.get_dispersion(param, grad=True)["energy"]
    only = model.get_dispersion(param, grad=False)["energy"]
    assert np.abs(np.asarray(only) - np.asarray(full)).max() <= 1e-14 * np.abs(full).max()
