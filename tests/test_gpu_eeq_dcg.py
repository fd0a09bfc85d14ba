"""
The deflated conjugate-gradient EEQ solves of the precision form (one or two
large structures in spatial order) against the plain FP64 path: rows with and
without 16-byte alignment, sizes beside whole blocks and tiles, padding atoms,
two structures, one of them empty or within one block.

Tolerances: charges 1e-7, forces 1e-6 Eh/Bohr, final residuals below the
solver's 1e-10 (test_gpu_eeq_cg.py).
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


@pytest.mark.parametrize("sizes,width", [
    ((4737,), 4739), ((4800,), 4800), ((4865,), 4868), ((3393, 3400), 3400), ((3400, 0), 3401),
    ((50, 3329), 3400),
], ids=lambda v: str(v))
def test_charges_and_forces_match_fp64(d4, sizes, width):
    disp = import_module("tad-dftd4_gb300.disp")
    wl = package().workloads
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(5)
    for b, n in enumerate(sizes):
        if n:
            z, r = wl.structure(60 + b, n)
            at = np.sort(rng.permutation(width)[:n])
            numbers[b, at], positions[b, at] = z, r
    dev = torch.device("cuda")
    charge = torch.tensor([(-1.0, 1.0)[b] * (n > 0) for b, n in enumerate(sizes)],
                          dtype=torch.float64, device=dev)
    nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
    out = []
    for precision in ("mixed", "fp64"):
        runner, _, _ = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                                     d4.Cutoff(disp3=12.0), None, None, None, precision)
        out.append(runner.run(pt, gradient=True, charges_out=True))
        if precision == "mixed":
            assert runner.eeq_residuals().max().item() <= 1e-10
    mixed, plain = out
    assert (mixed[3] - plain[3]).abs().max().item() <= 1e-7
    assert (mixed[1] - plain[1]).abs().max().item() <= 1e-6
