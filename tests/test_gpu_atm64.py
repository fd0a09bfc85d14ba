"""
The register-tiled FP64 ATM against the oracle at the sizes where its tiles
can go wrong: fewer than three atoms, ends of the 8 x 8 tiles, ranges of the
inner atom cut short, padding between the atoms, three-body cutoffs that
leave triples with two sides inside, exponents on either side of the rule
that selects it.

Tolerances as in test_gpu_parity.py: atom energies 1e-12 relative, gradients
1e-10 relative.
"""

from __future__ import annotations

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


def _structures(sizes, gaps):
    """Structures of ``sizes`` atoms in one padded batch; ``gaps`` spreads padding among them."""
    wl = package().workloads
    made = [wl.structure(500 + n, n) for n in sizes]
    width = max(sizes) + (5 if gaps else 0)
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(7)
    for b, (z, r) in enumerate(made):
        at = np.sort(rng.permutation(width)[:len(z)]) if gaps else np.arange(len(z))
        numbers[b, at], positions[b, at] = z, r
    charge = np.array([(-1.0, 0.0, 1.0)[b % 3] for b in range(len(sizes))])
    return tuple(torch.from_numpy(x) for x in (numbers, positions, charge))


@pytest.mark.parametrize("sizes", [(1, 2, 3, 4, 5), (9, 10, 11, 17, 18), (34, 41), (67,)],
                         ids=lambda s: "-".join(map(str, s)))
@pytest.mark.parametrize("cut3,gaps,model", [(40.0, False, "d4"), (40.0, True, "d4"),
                                             (8.0, True, "d4"), (11.0, False, "d4s")])
def test_tiles_match_oracle(d4, sizes, cut3, gaps, model):
    numbers, positions, charge = _structures(sizes, gaps)
    e_ref, g_ref = oracle.dftd4_energy_and_grad(numbers, positions, charge, PARAM, model=model,
                                                cutoff={"disp3": cut3})
    dev = torch.device("cuda")
    args = (numbers.to(dev), positions.to(dev), charge.to(dev), PARAM)
    kw = {"model": model, "cutoff": d4.Cutoff(disp3=cut3)}
    e, g = d4.dispersion_energy_gradient(*args, **kw)
    alone = d4.dftd4(*args, **kw)
    assert_close(e.cpu().numpy(), e_ref.numpy(), 1e-12, 1e-15, "energy")
    assert_close(alone.cpu().numpy(), e_ref.numpy(), 1e-12, 1e-15, "energy without gradient")
    assert_close(g.cpu().numpy(), g_ref.numpy(), 1e-10, 1e-13, "gradient")


@pytest.mark.parametrize("cut3", [40.0, 9.0])
@pytest.mark.parametrize("alp", [14.0, 100.0, 101.0])
def test_parameter_gradients_match_oracle(d4, cut3, alp):
    numbers, positions, charge = _structures((3, 12, 26), True)
    keys = ("a1", "a2", "s9", "alp")
    ref = {**PARAM, "s9": 0.7, "alp": alp}
    ref = {k: torch.tensor(v, dtype=torch.float64, requires_grad=k in keys)
           for k, v in ref.items()}
    e_ref = oracle.dftd4(numbers, positions, charge, ref, cutoff={"disp3": cut3})
    g_ref = torch.autograd.grad(e_ref.sum(), [ref[k] for k in keys])
    dev = torch.device("cuda")
    par = {k: v.detach().to(dev).requires_grad_(k in keys) for k, v in ref.items()}
    e = d4.dftd4(numbers.to(dev), positions.to(dev), charge.to(dev), par,
                 cutoff=d4.Cutoff(disp3=cut3))
    got = torch.autograd.grad(e.sum(), [par[k] for k in keys])
    assert_close(e.detach().cpu().numpy(), e_ref.detach().numpy(), 1e-12, 1e-15, "energy")
    for k, a, r in zip(keys, got, g_ref):
        assert_close(a.cpu().numpy(), r.numpy(), 1e-10, 1e-13, k)
