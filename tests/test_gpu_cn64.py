"""
The FP64 coordination numbers, summed over unordered pairs, against the oracle:
one atom, broken and whole queues of 32 pairs, padding between the atoms, more
pairs than one launch of single rounds takes, cutoffs inside the structure, and
nearly isolated atoms (counts down to 1e-30).

Tolerance: 1e-12 relative (an erfc argument of up to 9 multiplies a rounding
error of the distance by 160), 1e-34 absolute (counts below 1e-36 are dropped).
"""

from __future__ import annotations

from importlib import import_module

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


def _run(d4, numbers, positions, cn, cn_eeq):
    disp = import_module("tad-dftd4_gb300.disp")
    dev = torch.device("cuda")
    nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
    charge = torch.zeros(len(numbers), dtype=torch.float64, device=dev)
    runner, _, _ = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                                 d4.Cutoff(cn=cn, cn_eeq=cn_eeq), None, None, None, "fp64")
    out = runner.run(pt, cn_out=True, cn_eeq_out=True)
    tables = oracle.load_tables()
    nc, pc = torch.from_numpy(numbers), torch.from_numpy(positions)
    # (the D4 count keeps its own cutoff, whatever Cutoff.cn says)
    assert_close(out[4].cpu().numpy(), oracle.cn_d4(nc, pc, tables).numpy(), 1e-12, 1e-34, "cn")
    assert_close(out[5].cpu().numpy(), oracle.cn_eeq(nc, pc, tables, cn_eeq).numpy(), 1e-12, 1e-34,
                 "cn_eeq")


@pytest.mark.parametrize("sizes,width", [
    ((1, 2, 8, 9), 12), ((33, 1, 0, 64), 65), (tuple(range(20, 84)), 90), ((130, 7), 133),
], ids=["9", "65", "64-structures", "133"])
@pytest.mark.parametrize("cut", [(30.0, 25.0), (6.0, 4.5)])
def test_matches_oracle(d4, sizes, width, cut):
    wl = package().workloads
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(2)
    for b, n in enumerate(sizes):
        if n:
            z, r = wl.structure(900 + n, n)
            at = np.sort(rng.permutation(width)[:n])
            numbers[b, at], positions[b, at] = z, r
    _run(d4, numbers, positions, *cut)


def test_nearly_isolated_atoms_match_oracle(d4):
    far = np.linspace(1.0, 9.0, 33)
    numbers = np.tile(np.array([[6, 17]]), (33, 1))
    positions = np.zeros((33, 2, 3))
    positions[:, 1, 0] = far
    _run(d4, numbers, positions, 30.0, 25.0)
