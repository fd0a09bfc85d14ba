"""
Structures that run in spatial order (padded to 960 atoms and more) take their
FP32 positions relative to the same atom as others, the input's first: what
FP32 leaves of an energy depends on that atom.

The same structures padded to 959 and to 960 atoms then differ by the order of
their sums only: 1e-7 of a pair's sum each, so about 1e-9 of a three-body energy
with its ten thousand near pairs.  The bar is 5e-9 (rms over the structures);
relative to another atom the two differ by 2e-8 and more.
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 0.0, "s8": 0.0, "a1": 0.4, "a2": 5.0, "s9": 1.0}


def test_energies_do_not_depend_on_the_order_taken():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    dev = torch.device("cuda")
    B = 8
    total = []
    for width in (959, 960):
        numbers = np.zeros((B, width), dtype=np.int64)
        positions = np.zeros((B, width, 3))
        for b in range(B):
            n = 900 + 7 * b
            z, r = d4.workloads.structure(500 + b, n)
            at = slice(b, b + n)  # (padding before the first atom, too)
            numbers[b, at], positions[b, at] = z, r
        nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
        charge = torch.zeros(B, dtype=torch.float64, device=dev)
        runner = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                               d4.Cutoff(disp3=25.0), None, None, None, "mixed")[0]
        total.append(runner.run(pt)[0].sum(-1))
    rel = (total[1] - total[0]) / total[0]
    assert rel.pow(2).mean().sqrt().item() <= 5e-9, rel.tolist()
