"""
The C6 adjoints of the FP64 method at the sizes where they change from a lane
per frequency to a lane per partner, against the oracle: whole and broken
blocks of 32 partners on both sides, one atom, padding between the atoms.

Tolerances as in test_gpu_parity.py: gradients 1e-10 relative, energies 1e-12.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from conftest import assert_close, package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}


@pytest.fixture(scope="module")
def d4():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return package()


@pytest.mark.parametrize("sizes,width", [
    ((1, 2, 31, 32, 33), 33), ((64, 65, 93, 94, 96), 98), ((116, 117, 128), 129),
    ((129, 139, 140), 141),
], ids=lambda v: str(v) if isinstance(v, int) else str(max(v)))
def test_forces_match_oracle(d4, sizes, width):
    wl = package().workloads
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(6)
    for b, n in enumerate(sizes):
        z, r = wl.structure(500 + n, n)
        at = np.sort(rng.permutation(width)[:n])
        numbers[b, at], positions[b, at] = z, r
    charge = torch.zeros(len(sizes), dtype=torch.float64)
    nt, pt = torch.from_numpy(numbers), torch.from_numpy(positions)
    e_ref, g_ref = oracle.dftd4_energy_and_grad(nt, pt, charge, PARAM)
    dev = torch.device("cuda")
    e, g = d4.dispersion_energy_gradient(nt.to(dev), pt.to(dev), charge.to(dev), PARAM)
    assert_close(e.cpu().numpy(), e_ref.numpy(), 1e-12, 1e-15, "energy")
    assert_close(g.cpu().numpy(), g_ref.numpy(), 1e-10, 1e-13, "gradient")
