"""
The FP64 EEQ solves with their vectors in global memory: structures whose
vectors do not fit a CTA's shared memory (against the precision form's
charges), and small ones through the test flag (against the usual path, which
does the same arithmetic; 1e-12 is the bar of tests/test_gpu_eeq64.py).
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


def _runner(nt, pt, charge, precision):
    disp = import_module("tad-dftd4_gb300.disp")
    return disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None, None, None, None,
                         None, precision)[0]


@pytest.mark.parametrize("sizes,width", [((97,), 97), ((130, 0, 1, 33), 131), ((301, 290), 303)],
                         ids=str)
def test_vectors_in_global_memory(d4, sizes, width):
    wl = d4.workloads
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(5)
    for b, n in enumerate(sizes):
        if n:
            z, r = wl.structure(70 + n, n)
            at = np.sort(rng.permutation(width)[:n])
            numbers[b, at], positions[b, at] = z, r
    dev = torch.device("cuda")
    nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
    charge = torch.tensor([float(n > 1) for n in sizes], dtype=torch.float64, device=dev)
    runner = _runner(nt, pt, charge, "fp64")
    usual = runner.run(pt, gradient=True, charges_out=True)
    out = runner.run(pt, gradient=True, charges_out=True,
                     extra_flags=d4._lib.FLAG_TEST_FALLBACK)
    for k in (0, 1, 3):
        assert (out[k] - usual[k]).abs().max().item() <= 1e-12


def test_charges_beyond_shared_memory(d4):
    n = 14700
    z, r = d4.workloads.structure(9, n)
    dev = torch.device("cuda")
    nt = torch.from_numpy(np.asarray(z)[None]).to(dev)
    pt = torch.from_numpy(np.asarray(r)[None]).to(dev)
    charge = torch.zeros(1, dtype=torch.float64, device=dev)
    q = d4.get_properties(nt, pt, charge)[1]
    mixed = _runner(nt, pt, charge, "mixed").run(pt, charges_out=True)[3]
    # FP32 CN and matrix inputs of the precision form (tests/test_gpu_eeq_dcg.py)
    assert (q - mixed).abs().max().item() <= 1e-7
