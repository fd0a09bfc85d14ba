"""
The register-tiled ATM of the precision form against the plain FP64 path at
the sizes where its tasks can go wrong: fewer than three atoms, ends of the
tiles and of the 128-atom inner ranges, padding between the atoms, three-body
cutoffs that leave triples with two sides inside, structures beyond the
shared-memory kernels' sizes, more structures than one scan of the task plan.

Tolerances: the precision form's bar, 1e-7 Eh per atom and structure and 1e-6
Eh/Bohr; parameter gradients 1e-6 relative (test_gpu_mixed.py).
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 0.9}
E_TOL, F_TOL = 1e-7, 1e-6


@pytest.fixture(scope="module")
def d4():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return package()


def _batch(sizes, width, seed=900):
    wl = package().workloads
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(seed)
    for b, n in enumerate(sizes):
        z, r = wl.structure(seed + n, n)
        at = np.sort(rng.permutation(width)[:n])
        numbers[b, at], positions[b, at] = z, r
    dev = torch.device("cuda")
    return (torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev),
            torch.zeros(len(sizes), dtype=torch.float64, device=dev))


def _both(d4, batch, cut3, model="d4", **kw):
    disp = import_module("tad-dftd4_gb300.disp")
    out = []
    for precision in ("mixed", "fp64"):
        runner, _, _ = disp._prepare(*batch, PARAM, model, None, None, None, None,
                                     d4.Cutoff(disp3=cut3), None, None, None, precision)
        out.append([x.cpu().numpy() if x is not None else None
                    for x in runner.run(batch[1], **kw)])
    return out


@pytest.mark.parametrize("sizes,width", [
    ((1, 2, 3, 4, 5), 5), ((9, 10, 11, 17, 18), 18), ((34, 129, 130, 138), 140),
    ((250, 40), 250), (tuple(5 + k % 7 for k in range(1100)), 12),
], ids=["1-5", "9-18", "34-138", "250", "1100-structures"])
@pytest.mark.parametrize("gaps", [0, 3])
@pytest.mark.parametrize("cut3,model", [(40.0, "d4"), (9.0, "d4"), (12.0, "d4s")])
def test_matches_fp64(d4, sizes, width, gaps, cut3, model):
    batch = _batch(sizes, width + gaps)
    for gradient in (True, False):
        mixed, plain = _both(d4, batch, cut3, model, gradient=gradient)
        assert np.abs(mixed[0] - plain[0]).max() <= E_TOL
        assert np.abs(mixed[0].sum(-1) - plain[0].sum(-1)).max() <= E_TOL
        if gradient:
            assert np.abs(mixed[1] - plain[1]).max() <= F_TOL


@pytest.mark.parametrize("cut3", [40.0, 10.0])
@pytest.mark.parametrize("sizes,width", [((3, 12, 26), 30), ((137, 9), 140), ((240,), 240)],
                         ids=["26", "137", "240"])
def test_parameter_gradients_match_fp64(d4, sizes, width, cut3):
    mixed, plain = _both(d4, _batch(sizes, width), cut3, gradient=True, param_grad=True)
    assert np.abs(mixed[0] - plain[0]).max() <= E_TOL
    assert np.abs(mixed[1] - plain[1]).max() <= F_TOL
    gm, gp = mixed[2][:, :7], plain[2][:, :7]
    assert np.abs(gm - gp).max() <= 1e-6 * max(1.0, np.abs(gp).max())


@pytest.mark.parametrize("cut3", [12.0, 60.0])
def test_spatial_order_and_neighbour_triples_match_fp64(d4, cut3):
    """Structures that run in spatial order: every per-atom input and output
    (r4r2 and energy weights in; energies, forces, charges, both CNs out) keeps
    its atom; 12 Bohr takes the neighbour triples, 60 Bohr all triples."""
    disp = import_module("tad-dftd4_gb300.disp")
    batch = _batch((1536, 300), 1540)
    dev = batch[1].device
    g = torch.Generator().manual_seed(5)
    real = (batch[0] != 0).cpu()
    r4r2 = ((2.0 + 3.0 * torch.rand(real.shape, generator=g, dtype=torch.float64)) * real).to(dev)
    weights = (torch.rand(real.shape, generator=g, dtype=torch.float64) * real).to(dev)
    out = []
    for precision in ("mixed", "fp64"):
        runner, _, _ = disp._prepare(*batch, PARAM, "d4", None, r4r2, None, None,
                                     d4.Cutoff(disp3=cut3), None, None, None, precision)
        out.append((runner.run(batch[1], gradient=True, param_grad=True, charges_out=True,
                               cn_out=True, cn_eeq_out=True),
                    runner.run(batch[1], gradient=True, weights=weights)[1],
                    runner.run(batch[1])[0]))
    (mixed, mw, me), (plain, pw, pe) = out
    for k, tol in ((0, E_TOL), (1, F_TOL), (3, 1e-7), (4, 1e-6), (5, 1e-6)):
        assert (mixed[k] - plain[k]).abs().max().item() <= tol, k
    assert (mw - pw).abs().max().item() <= F_TOL
    assert (me - pe).abs().max().item() <= E_TOL
    gm, gp = mixed[2][:, :7].cpu().numpy(), plain[2][:, :7].cpu().numpy()
    assert np.abs(gm - gp).max() <= 1e-6 * max(1.0, np.abs(gp).max())
