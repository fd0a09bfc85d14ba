"""
Positions whose last dimension is not three coordinates are refused before
anything is launched, by every public call and also where the number of
entries would fill whole structures.
"""

from __future__ import annotations

from importlib import import_module

import pytest
import torch

from conftest import package

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}
SHAPES = [(2, 5, 2), (2, 5, 4), (1, 5, 1), (3, 4, 2), (2, 4, 6), (5, 2), (6, 6), (2, 3, 5, 4)]


@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_structures_takes_three_coordinates_only(shape):
    disp = import_module("tad-dftd4_gb300.disp")
    with pytest.raises(RuntimeError, match="three coordinates"):
        disp._structures(torch.zeros(shape), shape[-2])
    whole = disp._structures(torch.zeros(*shape[:-1], 3), shape[-2])
    assert whole.shape[1:] == (shape[-2], 3)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64], ids=str)
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_public_calls_refuse(shape, dtype):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    numbers = torch.full(shape[:-1], 6, device="cuda")
    positions = 4.0 * torch.arange(int(torch.tensor(shape).prod()), device="cuda",
                                   dtype=dtype).reshape(shape)
    for call in (d4.dftd4, d4.dispersion_energy_gradient, d4.hessian):
        for _ in range(2):  # (the second of a kept configuration)
            with pytest.raises(RuntimeError, match="three coordinates"):
                call(numbers, positions, 0.0, PARAM)
    with pytest.raises(RuntimeError, match="three coordinates"):
        d4.get_properties(numbers, positions)
