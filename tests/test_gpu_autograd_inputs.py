"""GPU test of the autograd wrapper's evaluation by which inputs require a
gradient: with and without a strain tensor and parameter derivatives, the
energies and the remaining gradients are the same (FP64, 1e-12: the passes with
parameter derivatives sum their pairs in another order)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s9", [0.0, 1.0])
@pytest.mark.parametrize("natoms", [5, 40])
def test_gradients_do_not_depend_on_the_other_inputs(natoms, s9):
    import torch
    from dftd3 import synthetic as S
    from dftd3.torch_api import D3Batch
    rng = np.random.default_rng(natoms)
    nums, pos, lats = [], [], []
    for n in (natoms, natoms + 3):
        lat = np.diag(rng.uniform(11.1, 11.9, size=3))
        nums.append(rng.choice([1, 6, 7, 8], size=n).astype(np.int32))
        pos.append(S.pack_cell(rng, n, lat, 1.9))
        lats.append(lat)
    model = D3Batch(nums, lattices=np.array(lats), periodic=np.ones((2, 3), dtype=bool), precision="fp64",
                    cutoffs=(20.0, 9.7, 14.3, 0.0, 0.0))
    weight = torch.tensor([1.0, -0.3], dtype=torch.float64, device="cuda")
    results = {}
    for with_strain in (False, True):
        for with_params in (False, True):
            x = torch.tensor(np.concatenate(pos), device="cuda", requires_grad=True)
            params = torch.tensor([1.0, 0.7875, 0.4289, 4.4407, s9], dtype=torch.float64, device="cuda",
                                  requires_grad=with_params)
            strain = torch.zeros((2, 3, 3), dtype=torch.float64, device="cuda", requires_grad=True) if with_strain else None
            e = model(x, params, strain)
            (e * weight).sum().backward()
            results[with_strain, with_params] = (e.detach(), x.grad, strain.grad if with_strain else None, params.grad)
    e0, g0, _, _ = results[False, False]
    for e, g, _, _ in results.values():
        assert (e - e0).abs().max() <= 1e-12 * e0.abs().max()
        assert (g - g0).abs().max() <= 1e-12 * g0.abs().max()
    s0, s1 = results[True, False][2], results[True, True][2]
    assert (s0 - s1).abs().max() <= 1e-12 * s1.abs().max()
    p0, p1 = results[False, True][3], results[True, True][3]
    assert (p0 - p1).abs().max() <= 1e-12 * p1.abs().max()
    assert results[False, False][3] is None and results[True, False][3] is None
