"""
The adjoint EEQ solves of the precision form under energy weights of any size:
all of the arithmetic scales with a power of two, so gradients do, to the order of
their sums (2e-6 of the largest entry; FP32 sums of a few hundred terms).  A
weight that is not finite gives a gradient that is not, and no error: a
training loop steps over such a batch.
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}


def _runner(sizes):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    width = max(sizes)
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    for b, n in enumerate(sizes):
        numbers[b, :n], positions[b, :n] = d4.workloads.structure(90 + n, n)
    dev = torch.device("cuda")
    nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
    charge = torch.zeros(len(sizes), dtype=torch.float64, device=dev)
    runner, _, _ = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                                 d4.Cutoff(disp2=30.0, disp3=8.0), None, None, None, "mixed")
    weights = 0.5 + torch.arange(numbers.size, device=dev, dtype=torch.float64) % 7 / 8.0
    return runner, pt, weights.reshape(numbers.shape)


@pytest.mark.parametrize("sizes", [(30, 200), (301,), (400, 33, 391), (997,), (5001,)], ids=str)
@pytest.mark.parametrize("power", [-50, -20, -10, 20, 50])
def test_gradient_scales_with_the_weights(sizes, power):
    runner, pt, weights = _runner(sizes)
    one = runner.run(pt, gradient=True, weights=weights)[1]
    got = runner.run(pt, gradient=True, weights=weights * 2.0 ** power)[1] * 2.0 ** -power
    assert (got - one).abs().max().item() <= 2e-6 * one.abs().max().item()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("sizes", [(301, 290), (5001,)], ids=str)
def test_weights_that_are_not_finite(sizes, value):
    runner, pt, weights = _runner(sizes)
    weights[0, 3] = value
    grad = runner.run(pt, gradient=True, weights=weights)[1]
    assert not torch.isfinite(grad[0]).all()
    assert torch.isfinite(grad[1:]).all()
