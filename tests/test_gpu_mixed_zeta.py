"""
The charge scaling of the precision form over its whole range, with given
charges, against the plain FP64 path: ordinary charges, charges near the
effective nuclear charge from either side (scaling exponents beyond 80, both
signs of q + zeff), several CTAs of atoms and D4S slots.

Tolerance: 1e-6 of the largest atom energy (FP32 pair arithmetic; an error of the
scaling itself would show undiminished).  Forces are not compared: the
cancellations of the CN derivatives at such charges, not the scaling, set theirs.
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}


@pytest.fixture(scope="module")
def d4():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return package()


@pytest.mark.parametrize("model", ["d4", "d4s"])
@pytest.mark.parametrize("n", [1, 127, 130, 257])
def test_given_charges_match_fp64(d4, n, model):
    disp = import_module("tad-dftd4_gb300.disp")
    wl = package().workloads
    z, r = wl.structure(21, n)
    q = np.random.default_rng(4).choice([-0.4, 0.0, 0.3, 2.0, -0.97, -0.999, -1.0, -1.2, 8.0], n)
    q = np.where(np.abs(q) >= 0.97, q * np.minimum(z, 8), q)
    dev = torch.device("cuda")
    nt, pt = torch.from_numpy(z[None]).to(dev), torch.from_numpy(r[None]).to(dev)
    qt = torch.from_numpy(q[None]).to(dev)
    charge = torch.zeros(1, dtype=torch.float64, device=dev)
    out = []
    for precision in ("mixed", "fp64"):
        runner, _, _ = disp._prepare(nt, pt, charge, PARAM, model, None, None, None, qt,
                                     d4.Cutoff(disp3=15.0), None, None, None, precision)
        out.append(runner.run(pt)[0])
    ref = out[1]
    assert torch.isfinite(ref).all()
    assert (out[0] - ref).abs().max().item() <= 1e-6 * max(ref.abs().max().item(), 1e-3)
