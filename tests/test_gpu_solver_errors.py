"""
Errors out of the multi-CTA EEQ solvers: coincident atoms (the EEQ matrix has no
such entry) and positions that are not finite are reported from every solver, its
waits end, the other calls on the device are not affected, and structures of the
batch that have no fault solve as without the others.
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}
# (precision, sizes): one CTA and panels of FP64; one CTA, conjugate gradients with
# rows in shared memory and in L2, deflated, factorisation
CASES = [("fp64", (40, 33)), ("fp64", (131, 97)), ("fp64", (301, 290)),
         ("mixed", (200, 150)), ("mixed", (301, 290)), ("mixed", (1003, 990)),
         ("mixed", (2531, 2500)), ("mixed", (5001,)), ("mixed", (301,) * 80)]


def _inputs(sizes):
    wl = package().workloads
    width = max(sizes)
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    made = {}
    for b, n in enumerate(sizes):
        numbers[b, :n], positions[b, :n] = made.setdefault(n, wl.structure(800 + n, n))
    return torch.from_numpy(numbers).cuda(), torch.from_numpy(positions).cuda()


@pytest.mark.parametrize("precision,sizes", CASES, ids=lambda v: str(v)[:16])
@pytest.mark.parametrize("fault", ["coincident", "nan", "inf"])
def test_faults_are_reported(precision, sizes, fault):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    nt, pt = _inputs(sizes)
    charge = torch.zeros(len(sizes), dtype=torch.float64, device="cuda")

    def run(positions):
        runner = disp._prepare(nt, positions, charge, PARAM, "d4", None, None, None, None,
                               d4.Cutoff(disp2=30.0, disp3=8.0), None, None, None, precision)[0]
        return runner.run(positions, gradient=True, charges_out=True)

    want = run(pt)
    bad = pt.clone()
    if fault == "coincident":
        bad[0, 17] = bad[0, 5]
        with pytest.raises(d4._lib.LibraryError, match="EEQ_SINGULAR"):
            run(bad)
    else:
        bad[0, 17, 1] = float(fault)
        with pytest.raises(ValueError, match="non-finite"):
            run(bad)
    check, disp.CHECK_STATUS = disp.CHECK_STATUS, False
    try:
        got = run(bad)
    finally:
        disp.CHECK_STATUS = check
    bar = 1e-12 if precision == "fp64" else 1e-8
    for x, y in ((got[3], want[3]), (got[1], want[1])):
        assert len(sizes) == 1 or (x[1:] - y[1:]).abs().max().item() <= bar
    again = run(pt)
    assert (again[3] - want[3]).abs().max().item() <= bar
