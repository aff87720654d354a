"""GPU tests of the three-body pair blocks (tiles of 8 atoms): sizes around the
tile edges, periodic images of one and of several tiles, smooth cutoffs, and
batches whose blocks are kept for the tile pairs in reach only, against the
FP64 oracle or the same system evaluated alone.  FP64: 1e-12, the bound of the
other three-body tests.  Mixed: the three-body part (the difference of the
results with and without it; the two-body part repeats bit for bit) stays
within the form's budget of 1e-7 of the total energy and 1e-7 Hartree/Bohr."""
import numpy as np
import pytest

import oracle_ref as O
from test_gpu_twobody import GTOL64, RTOL64

pytestmark = pytest.mark.gpu
ETOL_MIXED = GTOL_MIXED = 1.0e-7
CUT = (25.3, 13.7, 18.9, 0.0, 0.0)


def _param(s9=1.0):
    from dftd3 import synthetic as S
    from dftd3.interface import RationalDampingParam
    par = dict(S.PBE_BJ, damping="rational", s9=s9)
    return par, RationalDampingParam(**{k: par[k] for k in ("s6", "s8", "a1", "a2", "alp", "s9")})


def _check(res, ref):
    assert abs(float(res["energy"]) - ref["energy"]) <= RTOL64 * abs(ref["energy"])
    for k in ("gradient", "virial"):
        assert np.abs(res[k] - ref[k]).max() <= GTOL64 * np.abs(ref[k]).max(), k


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("natoms", [2, 3, 8, 9, 16, 17, 31, 32, 33, 41, 264])
def test_tile_edges_molecule(natoms, precision):
    from dftd3 import synthetic as S
    from dftd3.interface import DispersionModel
    rng = np.random.default_rng(natoms)
    num = rng.choice([1, 6, 7, 8], size=natoms).astype(np.int32)
    pos = S.pack_box(rng, natoms, 0.0, (natoms / 0.012) ** (1 / 3) + 3.0, 2.0)
    par, param = _param()
    par0, param0 = _param(0.0)
    for cut in ((60.0, 40.0, 40.0, 0.0, 0.0), (40.0, 11.3, 25.0, 4.0, 3.0)):
        model = DispersionModel(num, pos)
        model.set_precision(precision)
        model.set_realspace_cutoff(*cut)
        res, ref = model.get_dispersion(param, grad=True), O.dispersion(num, pos, par, cutoff=cut)
        alone = float(model.get_dispersion(param, grad=False)["energy"])
        if precision == "fp64":
            _check(res, ref)
            assert abs(alone - ref["energy"]) <= RTOL64 * abs(ref["energy"])
            continue
        res0, ref0 = model.get_dispersion(param0, grad=True), O.dispersion(num, pos, par0, cutoff=cut)
        alone0 = float(model.get_dispersion(param0, grad=False)["energy"])
        e3 = ref["energy"] - ref0["energy"]
        assert abs(float(res["energy"]) - float(res0["energy"]) - e3) <= ETOL_MIXED * abs(ref["energy"])
        assert abs(alone - alone0 - e3) <= ETOL_MIXED * abs(ref["energy"])
        g3 = ref["gradient"] - ref0["gradient"]
        assert np.abs(res["gradient"] - res0["gradient"] - g3).max() <= GTOL_MIXED


@pytest.mark.parametrize("natoms,periodic", [(1, (1, 1, 1)), (3, (1, 1, 1)), (9, (1, 1, 0)), (17, (0, 0, 1)),
                                              (20, (1, 1, 1))])
def test_tile_edges_periodic(natoms, periodic):
    from dftd3 import synthetic as S
    from dftd3.interface import DispersionModel
    rng = np.random.default_rng(100 + natoms)
    edge = (natoms / 0.02) ** (1 / 3) + 2.0
    lat = S.triclinic(edge, 1.07 * edge, 1.13 * edge, 90.0, 90.0, 90.0)
    num = rng.choice([1, 6, 8], size=natoms).astype(np.int32)
    pos = S.pack_cell(rng, natoms, lat, 2.0)
    par, param = _param()
    per = np.array(periodic, dtype=bool)
    for cut in (CUT, CUT[:3] + (4.0, 3.0)):
        model = DispersionModel(num, pos, lat, per)
        model.set_realspace_cutoff(*cut)
        ref = O.dispersion(num, pos, par, lattice=lat, periodic=per, cutoff=cut)
        res = model.get_dispersion(param, grad=True)
        if natoms == 1:        # the gradient vanishes by symmetry
            assert np.abs(res["gradient"]).max() <= GTOL64 * np.abs(ref["virial"]).max()
            res["gradient"] = ref["gradient"]
        _check(res, ref)


def _crystals(rng, nsys):
    from dftd3 import synthetic as S
    nums, pos, lats = [], [], []
    for k in range(nsys):
        n = int(rng.integers(20, 57))
        lat = np.diag(rng.uniform(13.1, 13.9, size=3))
        nums.append(rng.choice([1, 6, 8], size=n).astype(np.int32))
        pos.append(S.pack_cell(rng, n, lat, 1.9))
        lats.append(lat)
    return nums, pos, np.array(lats)


def test_blocks_in_reach_match_single_systems():
    """A batch whose blocks exceed the dense limit, with and without the captured
    sequence, and a replay that needs more blocks than the capture reserved."""
    from dftd3.interface import BatchedDispersion
    nums, pos, lats = _crystals(np.random.default_rng(8), 260)
    _, param = _param()
    per = np.ones((len(nums), 3), dtype=bool)
    inner = [0.35 * p + 4.0 for p in pos]      # the same atoms in a third of the cell: fewer blocks in reach
    bat = BatchedDispersion(nums, inner, lats, per)
    bat.set_realspace_cutoff(25.3, 20.0, 18.9)
    bat.set_graph(True)
    bat.get_dispersion(param, grad=True)
    for where in (inner, pos, pos):
        bat.update(where)
        got = bat.get_dispersion(param, grad=True)
        for k in (0, 57, 259):
            one = BatchedDispersion([nums[k]], [where[k]], lats[k:k + 1], per[k:k + 1])
            one.set_realspace_cutoff(25.3, 20.0, 18.9)
            ref = one.get_dispersion(param, grad=True)
            # the same FP64 sums in another order of the tiles' roots
            assert abs(got["energy"][k] - ref["energy"][0]) <= RTOL64 * abs(ref["energy"][0])
            if where is inner:      # 0.7 Bohr between atoms: its pair terms cancel to the forces
                continue
            assert np.abs(got["gradient"][k] - ref["gradient"][0]).max() <= GTOL64 * np.abs(ref["gradient"][0]).max()
            assert np.abs(got["virial"][k] - ref["virial"][0]).max() <= GTOL64 * np.abs(ref["virial"][0]).max()
