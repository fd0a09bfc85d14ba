"""
Residuals of the iterative EEQ solves (max |b - A x|).  A factorisation of
these matrices leaves 1.0e-11 to 1.6e-11 for the charges and up to 1.7e-13 for
the adjoint; the conjugate gradients aim at 1.2e-11 and 3e-13 and may miss that
by the last correction's rounding: 1.6e-11 and 5e-13.
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}


@pytest.mark.parametrize("sizes", [(300,), (423, 400, 391), (997,), (2000,), (5000,), (6001,),
                                   (4800, 4700)], ids=str)
def test_residuals_are_those_of_a_factorisation(sizes):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    width = max(sizes)
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    for b, n in enumerate(sizes):
        numbers[b, :n], positions[b, :n] = d4.workloads.structure(20 + n, n)
    dev = torch.device("cuda")
    nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
    charge = torch.zeros(len(sizes), dtype=torch.float64, device=dev)
    runner, _, _ = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                                 d4.Cutoff(disp2=30.0, disp3=15.0), None, None, None, "mixed")
    runner.run(pt, gradient=True)
    charges, adjoint = runner.eeq_residuals().amax(0).tolist()
    assert 0.0 < charges <= 1.6e-11 and 0.0 < adjoint <= 5e-13, (charges, adjoint)
