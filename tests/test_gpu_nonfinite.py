"""GPU test of positions that are not numbers, as a device entry may get them: the other
systems of the batch keep their results bit for bit, and so does the next evaluation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems(sizes, periodic):
    from dftd3 import synthetic as S
    rng = np.random.default_rng(sum(sizes))
    nums, pos, lats = [], [], []
    for n in sizes:
        side = (n / 0.012) ** (1 / 3) + 2.0
        nums.append(rng.choice([1, 6, 7, 8], size=n).astype(np.int32))
        pos.append(S.pack_box(rng, n, 0.0, side, 2.0))
        lats.append(np.eye(3) * (side + 2.0))
    return nums, pos, (np.array(lats) if periodic else None)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
# a cluster per system; tiles of 32 atoms; their last one, partly filled; periodic
@pytest.mark.parametrize("sizes, periodic", [((12, 40), False), ((300, 31), False), ((17, 270), False), ((12, 37), True)])
@pytest.mark.parametrize("where", [0, 11])
def test_other_systems_keep_their_bits(sizes, periodic, precision, where):
    import torch
    from dftd3.torch_api import D3Batch
    nums, pos, lats = _systems(sizes, periodic)
    model = D3Batch(nums, lattices=lats, periodic=np.ones((2, 3), dtype=bool) if periodic else None,
                    precision=precision, cutoffs=(20.0, 15.0, 15.0, 0.0, 0.0))
    params = torch.tensor([1.0, 0.7875, 0.4289, 4.4407, 1.0], dtype=torch.float64)

    def evaluate(x):
        x = x.clone().requires_grad_()
        e = model(x, params)
        e.sum().backward()
        return e.detach().cpu().numpy(), x.grad.cpu().numpy()

    x = torch.tensor(np.concatenate(pos), device="cuda")
    e0, g0 = evaluate(x)
    bad = x.clone()
    bad[where, 1] = float("nan")
    e1, g1 = evaluate(bad)
    assert e1[1] == e0[1] and np.array_equal(g1[sizes[0]:], g0[sizes[0]:])
    e2, g2 = evaluate(x)
    assert np.array_equal(e2, e0) and np.array_equal(g2, g0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sizes, periodic", [((12, 40), False), ((300, 31), False), ((17, 270), False), ((12, 37), True)])
@pytest.mark.parametrize("where, value", [(0, float("nan")), (11, float("nan")), (3, float("inf"))])
def test_three_body_term_is_nan(sizes, periodic, precision, where, value):
    """The three-body term alone: NaN for the system and for the atom, as any sum with a NaN, not the numbers its
    fixed-point form would have."""
    import torch
    from dftd3.torch_api import D3Batch
    nums, pos, lats = _systems(sizes, periodic)
    model = D3Batch(nums, lattices=lats, periodic=np.ones((2, 3), dtype=bool) if periodic else None,
                    precision=precision, cutoffs=(20.0, 15.0, 15.0, 0.0, 0.0))
    params = torch.tensor([0.0, 0.0, 0.4289, 4.4407, 1.0], dtype=torch.float64)
    x = torch.tensor(np.concatenate(pos), device="cuda")
    e0 = model(x.clone().requires_grad_(), params)      # the energies of the pass with gradients
    x[where, 2] = value
    x.requires_grad_()
    e1 = model(x, params)
    e1.sum().backward()
    assert torch.isnan(e1[0]) and e1[1] == e0[1]
    assert torch.isnan(x.grad[where]).all()
    assert torch.isfinite(x.grad[sizes[0]:]).all()
    assert torch.isnan(model(x.detach(), params)[0])
