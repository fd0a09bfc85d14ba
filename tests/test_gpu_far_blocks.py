"""
Large structures in spatial order whose pair kernels pass over blocks of atoms
beyond the cutoffs, against the plain FP64 path (given charges): a bar with
padding atoms over neighbour triples, and two distant clusters over all triples,
with energies alone, energy weights and parameter gradients.

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


@pytest.fixture(scope="module")
def d4():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return package()


def _bar(wl):  # 5003 atoms, eight cubes in a row, three padding slots
    parts = [wl.structure(30 + k, 625 + 3 * (k == 0)) for k in range(8)]
    side = max(r.max() for _, r in parts) + 2.5
    z = np.concatenate([p[0] for p in parts])
    r = np.concatenate([p[1] + [k * side, 0.0, 0.0] for k, p in enumerate(parts)])
    numbers, positions = np.zeros((1, 5006), dtype=np.int64), np.zeros((1, 5006, 3))
    at = np.sort(np.random.default_rng(1).permutation(5006)[:5003])
    order = np.random.default_rng(2).permutation(5003)
    numbers[0, at], positions[0, at] = z[order], r[order]
    return numbers, positions


def _clusters(wl):  # 2700 and 2300 atoms, 300 Bohr apart
    (za, ra), (zb, rb) = wl.structure(40, 2700), wl.structure(41, 2300)
    return (np.concatenate([za, zb])[None], np.concatenate([ra, rb + 300.0])[None])


@pytest.mark.parametrize("make,disp2,disp3", [(_bar, 25.0, 8.0), (_clusters, 30.0, 60.0)],
                         ids=["bar", "clusters"])
def test_matches_fp64(d4, make, disp2, disp3):
    disp = import_module("tad-dftd4_gb300.disp")
    numbers, positions = make(package().workloads)
    dev = torch.device("cuda")
    nt, pt = torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev)
    g = torch.Generator().manual_seed(3)
    real = (nt != 0).cpu()
    q = ((torch.rand(real.shape, generator=g, dtype=torch.float64) - 0.5) * real).to(dev)
    weights = (torch.rand(real.shape, generator=g, dtype=torch.float64) * real).to(dev)
    charge = torch.zeros(1, dtype=torch.float64, device=dev)
    out = []
    for precision in ("mixed", "fp64"):
        runner, _, _ = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, q,
                                     d4.Cutoff(disp2=disp2, disp3=disp3), None, None, None,
                                     precision)
        junk = torch.full((1 << 26,), float("nan"), device=dev)  # nothing unwritten is read
        del junk
        out.append((runner.run(pt, gradient=True, param_grad=True), runner.run(pt)[0],
                    runner.run(pt, gradient=True, weights=weights)[1]))
    (mixed, me, mw), (plain, pe, pw) = out
    assert (mixed[0].sum() - plain[0].sum()).abs().item() <= 1e-7
    assert (me.sum() - pe.sum()).abs().item() <= 1e-7
    assert (mixed[1] - plain[1]).abs().max().item() <= 1e-6
    assert (mw - pw).abs().max().item() <= 1e-6
    gm, gp = mixed[2][:, :7], plain[2][:, :7]
    assert (gm - gp).abs().max().item() <= 1e-6 * max(1.0, gp.abs().max().item())
