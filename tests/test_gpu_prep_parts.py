"""
Structures whose set-up is spread over several CTAs, against the same structure
with its padding atoms elsewhere: padding inside, at both ends and over whole
blocks of 32, an empty structure, a last CTA without whole blocks, both methods.

Tolerance: 1e-13 relative of the largest entry in FP64 (order of sums), 2e-6 in
the precision form (its own accuracy; positions are relative to the first atom).
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 0.0}


@pytest.fixture(scope="module")
def d4():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return package()


@pytest.mark.parametrize("model", ["d4", "d4s"])
@pytest.mark.parametrize("n,width", [(500, 513), (515, 1001), (700, 1600)])
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-13), (torch.float32, 2e-6)])
def test_padding_anywhere_gives_the_same(d4, n, width, model, dtype, tol):
    z, r = package().workloads.structure(n, n)
    rng = np.random.default_rng(n)
    slots = [np.arange(n), np.arange(width - n, width), np.sort(rng.permutation(width)[:n]),
             np.concatenate([np.arange(32), np.arange(width - n + 32, width)])]
    numbers = np.zeros((len(slots) + 1, width), dtype=np.int64)
    positions = np.zeros((len(slots) + 1, width, 3))
    for b, at in enumerate(slots):
        numbers[b, at], positions[b, at] = z, r
    dev = torch.device("cuda")
    nt = torch.from_numpy(numbers).to(dev)
    pt = torch.from_numpy(positions).to(dev, dtype)
    charge = torch.zeros(len(numbers), dtype=dtype, device=dev)
    e, g = d4.dispersion_energy_gradient(nt, pt, charge, PARAM, model=model)
    e, g = e.cpu().numpy(), g.cpu().numpy()
    assert not e[-1].any() and not g[-1].any()
    for b, at in enumerate(slots):
        pad = np.ones(width, dtype=bool)
        pad[at] = False
        assert not e[b, pad].any() and not g[b, pad].any()
        assert np.abs(e[b, at] - e[0, slots[0]]).max() <= tol * np.abs(e[0]).max()
        assert np.abs(g[b, at] - g[0, slots[0]]).max() <= tol * np.abs(g[0]).max()
