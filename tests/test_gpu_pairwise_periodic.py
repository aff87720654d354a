"""GPU tests of the non-additive pair energies of periodic systems, whose triples read their pair factors from a table
over the translations: one to three periodic directions, skewed cells smaller and larger than the cutoff, fewer and
more atoms than a warp's lanes, against the FP64 oracle (1e-12 of the largest entry, the bound of the other pairwise
tests), and the table against the triples that compute the factors."""
import numpy as np
import pytest

import oracle_ref as O
from test_gpu_pairwise import FAMILIES, TOL, assert_pairs, assert_sums_to, gpu_pairwise

pytestmark = pytest.mark.gpu


def _cell(natoms, angles=(90.0, 90.0, 90.0)):
    from dftd3 import synthetic as S
    rng = np.random.default_rng(natoms)
    edge = (natoms / 0.02) ** (1 / 3) + 1.0
    lat = S.triclinic(0.9 * edge, 1.1 * edge, 1.05 * edge, *angles)
    return rng.choice([1, 6, 8], size=natoms).astype(np.int32), S.pack_cell(rng, natoms, lat, 1.9), lat


@pytest.mark.parametrize("natoms", [1, 3, 20, 33])
@pytest.mark.parametrize("periodic, angles", [((1, 1, 1), (60.0, 75.0, 110.0)), ((1, 1, 0), (90.0, 90.0, 70.0)),
                                              ((0, 0, 1), (90.0, 90.0, 90.0))])
def test_against_the_oracle(natoms, periodic, angles):
    num, pos, lat = _cell(natoms, angles)
    per = [bool(p) for p in periodic]
    for cut in ((15.0, 9.0, 12.0, 0.0, 0.0), (15.0, 14.3, 12.0, 3.0, 4.0)):
        pw, energy = gpu_pairwise(num, pos, FAMILIES["rational"], lattice=lat, periodic=per, cutoff=cut)
        assert_pairs(pw, O.pairwise_dispersion(num, pos, FAMILIES["rational"], lattice=lat, periodic=per, cutoff=cut))
        assert_sums_to(pw, energy)


def test_without_memory_for_the_table():
    import torch
    from test_gpu_twobody import _param_obj
    from dftd3.interface import DispersionModel
    num, pos, lat = _cell(400)                  # 400 x 400 pairs, 125 translations, 16 bytes: above 256 MB
    model = DispersionModel(num, pos, lat, np.ones(3, dtype=bool))
    model.set_realspace_cutoff(15.0, 30.0, 12.0)
    param = _param_obj(FAMILIES["rational"])
    want = model.get_pairwise_dispersion(param)
    torch.cuda.empty_cache()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (128 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = model.get_pairwise_dispersion(param)
    finally:
        del hold
        torch.cuda.empty_cache()
    for key in want:
        assert np.abs(got[key] - want[key]).max() <= TOL * np.abs(want[key]).max(), key
