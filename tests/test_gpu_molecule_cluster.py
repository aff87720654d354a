"""GPU tests of the small-molecule kernels (one cluster per system): sizes around
the warps, blocks and clusters of the kernels, every damping family, ghosts, smooth
cutoffs, several systems, host and device entries, against the FP64 oracle (1e-12)
or each other."""
import numpy as np
import pytest

import oracle_ref as O
from test_gpu_twobody import GTOL64, RTOL64

pytestmark = pytest.mark.gpu
PARAMS = {
    "rational": dict(s6=1.0, s8=0.7875, a1=0.4289, a2=4.4407),
    "zero": dict(s6=1.0, s8=0.722, rs6=1.217, rs8=1.0),
    "mzero": dict(s6=1.0, s8=1.532981, rs6=1.338153, rs8=1.0, bet=0.013988),
    "optimizedpower": dict(s6=1.0, s8=0.43185, a1=0.575, a2=3.0, bet=8.0),
    "cso": dict(s6=1.0, a1=0.86, a2=2.5, a3=0.0, a4=6.25),
    "z": dict(s6=1.0, s8=1.0, a1=200770.0),
}


def _param(damping, s9, alp=14.0):
    from dftd3 import interface as I
    cls = {"rational": I.RationalDampingParam, "zero": I.ZeroDampingParam, "mzero": I.ModifiedZeroDampingParam,
           "optimizedpower": I.OptimizedPowerDampingParam, "cso": I.CSODampingParam, "z": I.ZDampingParam}[damping]
    return cls(**PARAMS[damping], s9=s9, alp=alp), dict(PARAMS[damping], damping=damping, s9=s9, alp=alp)


def _molecule(natoms, seed=0):
    from dftd3 import synthetic as S
    rng = np.random.default_rng(1000 * seed + natoms)
    num = rng.choice([1, 6, 7, 8, 16], size=natoms).astype(np.int32)
    return num, S.pack_box(rng, natoms, 0.0, (natoms / 0.012) ** (1 / 3) + 1.0, 2.0)


def _check(res, ref):
    assert abs(float(res["energy"]) - ref["energy"]) <= RTOL64 * abs(ref["energy"])
    if "gradient" in res:
        for k in ("gradient", "virial"):
            assert np.abs(res[k] - ref[k]).max() <= GTOL64 * max(np.abs(ref[k]).max(), 1e-30), k


@pytest.mark.parametrize("s9", [0.0, 1.0])
@pytest.mark.parametrize("natoms", [1, 2, 15, 16, 17, 33, 64, 65, 129, 256, 257])
def test_sizes(natoms, s9):
    from dftd3.interface import DispersionModel
    num, pos = _molecule(natoms)
    param, par = _param("rational", s9)
    ref = O.dispersion(num, pos, par)
    model = DispersionModel(num, pos)
    for graph in (False, True):
        model.set_graph(graph)
        for grad in (True, False):
            _check(model.get_dispersion(param, grad=grad), ref)


@pytest.mark.parametrize("damping", sorted(PARAMS))
@pytest.mark.parametrize("alp", [14.0, 13.0])
def test_families_ghosts_smooth(damping, alp):
    from dftd3.interface import DispersionModel
    num, pos = _molecule(70, seed=1)
    cut = (30.0, 12.0, 25.0, 4.0, 3.0)
    ghost = [0, 9, 33, 69]
    for s9 in (0.0, 1.0):
        param, par = _param(damping, s9, alp)
        model = DispersionModel(num, pos)
        model.set_realspace_cutoff(*cut)
        model.set_ghost_atoms(ghost)
        _check(model.get_dispersion(param, grad=True), O.dispersion(num, pos, par, cutoff=cut, ghost=ghost))


@pytest.mark.parametrize("s9", [0.0, 1.0])
def test_batches_and_entries(s9):
    """Three systems of uneven size; the device entry, with and without the captured
    sequence, gives the same bits as the host entry."""
    import torch
    from dftd3 import library
    from dftd3.interface import BatchedDispersion
    mols = [_molecule(n, seed=2) for n in (5, 120, 38)]
    param, par = _param("zero", s9)
    bat = BatchedDispersion([m[0] for m in mols], [m[1] for m in mols])
    res = bat.get_dispersion(param, grad=True)
    for k, (num, pos) in enumerate(mols):
        _check({"energy": res["energy"][k], "gradient": res["gradient"][k], "virial": res["virial"][k]},
               O.dispersion(num, pos, par))
    x = torch.tensor(np.concatenate([m[1] for m in mols]), device="cuda")
    for graph in (False, True):
        library.set_batch_graph(bat._batch, graph)
        for _ in range(2):
            e = torch.zeros(3, dtype=torch.float64, device="cuda")
            g = torch.zeros_like(x)
            s = torch.zeros((3, 9), dtype=torch.float64, device="cuda")
            library.get_dispersion_device(bat._batch, param._param, x.data_ptr(), None, e.data_ptr(), g.data_ptr(),
                                          s.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
            assert np.array_equal(e.cpu().numpy(), res["energy"])
            assert np.array_equal(g.cpu().numpy(), np.concatenate(res["gradient"]))
            assert np.array_equal(s.cpu().numpy().reshape(3, 3, 3), res["virial"])
