"""
Three-body damping exponents far from the method's 16 in the precision form,
over all triples and over neighbour triples: finite, and the FP64 path's
energies.  (R0/r)^(alp/3) is exp(alp/3 log(R0/r)) in FP32, so its relative error
is alp/3 log(R0/r) 6e-8, 5e-6 at alp = 150: a bar of 2e-5 on three-body energies.
"""

from __future__ import annotations

from importlib import import_module

import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,disp3", [(9, 40.0), (67, 40.0), (260, 40.0), (1000, 12.0)])
@pytest.mark.parametrize("alp", [0.0, 2.0, 47.0, 60.0, 150.0])
@pytest.mark.parametrize("gradient", [False, True])
def test_exponents_match_fp64(n, disp3, alp, gradient):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    param = {"s6": 0.0, "s8": 0.0, "a1": 0.4, "a2": 5.0, "s9": 1.0, "alp": alp}
    z, r = d4.workloads.structure(n, n)
    nt, pt = torch.from_numpy(z)[None].cuda(), torch.from_numpy(r)[None].cuda()
    charge = torch.zeros(1, dtype=torch.float64, device="cuda")
    mixed, plain = (disp._prepare(nt, pt, charge, param, "d4", None, None, None, None,
                                  d4.Cutoff(disp3=disp3), None, None, None, p)[0]
                    .run(pt, gradient=gradient) for p in ("mixed", "fp64"))
    scale = plain[0].abs().max().item()
    assert (mixed[0] - plain[0]).abs().max().item() <= 2e-5 * scale
    if gradient:
        assert torch.isfinite(mixed[1]).all()
