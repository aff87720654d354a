"""GPU test of calls that find too little device memory: they fail with an error, and the same object evaluates again
once there is memory, with the results of a new one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _cells():
    from dftd3 import synthetic as S
    rng = np.random.default_rng(3)
    nums, pos, lats = [], [], []
    for _ in range(6):
        lat = np.diag(rng.uniform(24.0, 26.0, size=3))
        nums.append(rng.choice([1, 6, 8], size=300).astype(np.int32))
        pos.append(S.pack_cell(rng, 300, lat, 2.0))
        lats.append(lat)
    return nums, pos, np.array(lats)


def _batch():
    from dftd3.interface import BatchedDispersion
    nums, pos, lats = _cells()
    bat = BatchedDispersion(nums, pos, lats, np.ones((len(nums), 3), dtype=bool))
    bat.set_realspace_cutoff(20.0, 10.0, 10.0)
    return bat


# the buffer that does not fit: one of the first, the numbering's, the records, their CN derivatives
@pytest.mark.parametrize("left", [16 << 20, 64 << 20, 256 << 20, 400 << 20])
def test_evaluates_again(left):
    import torch
    from dftd3 import synthetic as S
    from dftd3.interface import RationalDampingParam
    plain, param = (RationalDampingParam(**{k: S.PBE_BJ[k] for k in ("s6", "s8", "a1", "a2", "alp")}, s9=s9)
                    for s9 in (0.0, 1.0))
    ref = _batch()
    ref.get_dispersion(param, grad=True)
    ref.set_realspace_cutoff(45.0, 40.0, 20.0)
    want = ref.get_dispersion(param, grad=True)      # loads every kernel, too
    del ref
    bat = _batch()
    bat.get_dispersion(plain, grad=True)             # no buffers of the three-body term yet
    bat.set_realspace_cutoff(45.0, 40.0, 20.0)
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    hold = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            with pytest.raises(RuntimeError, match="out of memory"):
                bat.get_dispersion(param, grad=True)
    finally:
        del hold
        torch.cuda.empty_cache()
    got = bat.get_dispersion(param, grad=True)
    assert np.array_equal(got["energy"], want["energy"])
    for a, b in zip(got["gradient"], want["gradient"]):
        assert np.array_equal(a, b)
