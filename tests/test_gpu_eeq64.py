"""
The FP64 EEQ solve against the oracle at the sizes where its blocks can go
wrong: ends of the 32-column panels, the largest one-CTA size and the first
beyond it, padding between the atoms, structures much smaller than their
batch, and more structures than one panel launch gives a warp per CTA.

Tolerances as in test_gpu_parity.py: charges and gradients 1e-10 relative,
atom energies 1e-12 relative.
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


def _batch(sizes, width):
    wl = package().workloads
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(11)
    for b, n in enumerate(sizes):
        z, r = wl.structure(700 + n, n)
        at = np.sort(rng.permutation(width)[:n])
        numbers[b, at], positions[b, at] = z, r
    charge = np.array([(-1.0, 0.0, 1.0)[b % 3] for b in range(len(sizes))])
    return tuple(torch.from_numpy(x) for x in (numbers, positions, charge))


@pytest.mark.parametrize("sizes,width", [
    ((1, 2, 31, 32), 32), ((33, 63, 64, 5), 64), ((65, 95, 96, 1), 96), ((97, 33, 64, 2), 97),
    ((128, 129, 160), 161), ((290, 7), 301), (tuple(range(97, 137)) * 2, 140),
], ids=lambda v: str(v) if isinstance(v, int) else str(max(v)))
def test_charges_match_oracle(d4, sizes, width):
    numbers, positions, charge = _batch(sizes, width)
    q_ref = oracle.eeq_charges(numbers, positions, charge, oracle.load_tables())
    dev = torch.device("cuda")
    _, q, _, _ = d4.get_properties(numbers.to(dev), positions.to(dev), charge.to(dev))
    assert_close(q.cpu().numpy(), q_ref.numpy(), 1e-10, 1e-13, "charges")


@pytest.mark.parametrize("sizes,width", [((1, 31, 33), 34), ((96, 64), 96), ((97, 65, 2), 99),
                                         ((131,), 133)],
                         ids=lambda v: str(v) if isinstance(v, int) else str(max(v)))
def test_forces_match_oracle(d4, sizes, width):
    numbers, positions, charge = _batch(sizes, width)
    e_ref, g_ref = oracle.dftd4_energy_and_grad(numbers, positions, charge, PARAM)
    dev = torch.device("cuda")
    e, g = d4.dispersion_energy_gradient(numbers.to(dev), positions.to(dev), charge.to(dev),
                                         PARAM)
    assert_close(e.cpu().numpy(), e_ref.numpy(), 1e-12, 1e-15, "energy")
    assert_close(g.cpu().numpy(), g_ref.numpy(), 1e-10, 1e-13, "gradient")
