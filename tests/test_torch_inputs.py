"""Inputs of the autograd wrapper, on the CPU with a stand-in for the library: the evaluation gets one row of three
doubles per atom, and positions of any other shape are refused before it."""
import ctypes

import numpy as np
import pytest
import torch

NATOMS = 5


@pytest.fixture
def model(monkeypatch):
    from dftd3 import library, torch_api
    seen = []

    def evaluate(batch, param, pos, lat, energies, grad, sigma, pgrad, stream):
        seen.append(np.array((ctypes.c_double * (3 * NATOMS)).from_address(pos)).reshape(NATOMS, 3))

    monkeypatch.setattr(library, "new_batch", lambda *a: None)
    monkeypatch.setattr(library, "set_batch_precision", lambda *a: None)
    monkeypatch.setattr(library, "new_rational_damping", lambda *a: None)
    monkeypatch.setattr(library, "get_dispersion_device", evaluate)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda dev: type("S", (), {"cuda_stream": 0}))
    m = torch_api.D3Batch([np.ones(3), np.ones(2)])
    m.seen = seen
    return m


PARAMS = torch.tensor([1.0, 0.8, 0.4, 4.4, 0.0], dtype=torch.float64)
# a long buffer behind every input, so that a wrong shape reads no foreign memory here
BUFFER = torch.arange(96, dtype=torch.float64)


@pytest.mark.parametrize("strained", [False, True])
@pytest.mark.parametrize("shape", [(NATOMS - 1, 3), (NATOMS + 1, 3), (3 * NATOMS,), (1, NATOMS, 3), (NATOMS, 2)])
def test_other_shapes_are_refused(model, shape, strained):
    x = BUFFER[:int(np.prod(shape))].view(shape)
    with pytest.raises((ValueError, RuntimeError)):
        model(x, PARAMS, torch.zeros((2, 3, 3), dtype=torch.float64) if strained else None)
    assert not model.seen


@pytest.mark.parametrize("strained", [False, True])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("form", ["rows", "transposed", "broadcast"])
def test_rows_of_doubles_arrive(model, form, dtype, strained):
    buf = BUFFER.to(dtype)
    x = {"rows": buf[:3 * NATOMS].view(NATOMS, 3), "transposed": buf[:3 * NATOMS].view(3, NATOMS).t(),
         "broadcast": buf[1:4].view(1, 3)}[form]
    model(x, PARAMS, torch.zeros((2, 3, 3), dtype=dtype) if strained else None)
    assert np.array_equal(model.seen[0], np.broadcast_to(x.double().numpy(), (NATOMS, 3)))
