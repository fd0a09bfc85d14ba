"""
EEQ matrices that are not positive definite (hardnesses of a caller's tables below
the smallest eigenvalue of the rest) are refused by every solver, as by a
factorisation, by however little they miss.
"""

from __future__ import annotations

from importlib import import_module

import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}


def _smallest_eigenvalue(z, pos, tab):
    rad, eta = tab.tensors["eeq_rad"][z].double(), tab.tensors["eeq_eta"][z].double()
    r = torch.cdist(pos, pos, compute_mode="donot_use_mm_for_euclid_dist")
    r.fill_diagonal_(1.0)
    a = torch.erf(r / torch.sqrt(rad[:, None] ** 2 + rad[None] ** 2)) / r
    a.diagonal().copy_(eta + (2.0 / torch.pi) ** 0.5 / rad)
    return torch.linalg.eigvalsh(a)[0].item()


@pytest.mark.parametrize("precision,n", [("fp64", 60), ("fp64", 301), ("mixed", 200),
                                         ("mixed", 301), ("mixed", 1003), ("mixed", 2531),
                                         ("mixed", 5001)])
@pytest.mark.parametrize("below", [0.01, 0.1])
def test_not_positive_definite_is_refused(precision, n, below):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    z, r = d4.workloads.structure(n, n)
    nt, pt = torch.from_numpy(z)[None].cuda(), torch.from_numpy(r)[None].cuda()
    charge = torch.zeros(1, dtype=torch.float64, device="cuda")
    runner = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                           d4.Cutoff(disp2=30.0, disp3=8.0), None, None, None, precision)[0]
    eta = runner.tables.tensors["eeq_eta"]
    kept = eta.clone()
    smallest = _smallest_eigenvalue(nt[0], pt[0], runner.tables)
    try:
        eta.sub_(smallest - 0.01)  # still positive definite
        runner.run(pt, gradient=True)
        eta.sub_(0.01 + below)
        with pytest.raises(d4._lib.LibraryError, match="EEQ_SINGULAR"):
            runner.run(pt, gradient=True)
    finally:
        eta.copy_(kept)
    runner.run(pt, gradient=True)
