"""
The D4S pair stages of the precision form, whose warps take partners grouped by
element slot, against the plain FP64 path: one slot, runs of whole and broken
groups of eight, more slots than eight warps have shared memory for, padding
atoms, structures beyond one list of 1024 atoms.

Tolerances: the precision form's 1e-7 Eh per structure and 1e-6 Eh/Bohr
(test_gpu_mixed.py); parameter gradients 1e-6 of the largest (test_gpu_atm32.py).
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}
MANY = tuple((z, 1.0 / 85) for z in range(1, 86))  # elements 1 .. 85


@pytest.fixture(scope="module")
def d4():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return package()


@pytest.mark.parametrize("sizes,width,table", [
    ((1, 2, 9, 33), 33, ((6, 1.0),)), ((16, 17, 64), 70, ((1, 0.5), (8, 0.5))),
    ((85, 200, 0, 150), 201, MANY), ((1023, 5), 1023, ((1, 0.5), (6, 0.3), (17, 0.2))),
    ((1061,), 1100, None),
], ids=["one", "two", "many", "full-list", "two-lists"])
@pytest.mark.parametrize("params", [False, True])
def test_matches_fp64(d4, sizes, width, table, params):
    disp = import_module("tad-dftd4_gb300.disp")
    wl = package().workloads
    table = wl.ELEMENTS_12 if table is None else table
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(9)
    for b, n in enumerate(sizes):
        if n:
            z, r = wl.structure(80 + b, n, table)
            at = np.sort(rng.permutation(width)[:n])
            numbers[b, at], positions[b, at] = z, r
    dev = torch.device("cuda")
    nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
    charge = torch.zeros(len(sizes), dtype=torch.float64, device=dev)
    out = []
    for precision in ("mixed", "fp64"):
        runner, _, _ = disp._prepare(nt, pt, charge, PARAM, "d4s", None, None, None, None,
                                     d4.Cutoff(disp3=15.0), None, None, None, precision)
        out.append(runner.run(pt, gradient=True, param_grad=params))
    mixed, plain = out
    assert (mixed[0].sum(-1) - plain[0].sum(-1)).abs().max().item() <= 1e-7
    assert (mixed[1] - plain[1]).abs().max().item() <= 1e-6
    if params:
        gm, gp = mixed[2][:, :7], plain[2][:, :7]
        assert (gm - gp).abs().max().item() <= 1e-6 * max(1.0, gp.abs().max().item())
