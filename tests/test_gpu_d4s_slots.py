"""
D4S with more slots than elements: a caller of the C interface sizes them ahead of
its structures, and more of them than there are elements change nothing (FP32
atomics: 2e-6 of the largest gradient entry, 1e-9 Eh).
"""

from __future__ import annotations

from importlib import import_module

import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("slots", [12, 40, 128, 129, 400])
def test_slots_beyond_the_elements(slots, precision):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    wl = d4.workloads
    b = wl.batch_uniform(77, 3, 20, 70, wl.ELEMENTS_12, True, "slots", 70)
    nt, pt, ct = (torch.from_numpy(x).cuda() for x in (b.numbers, b.positions, b.charge))
    runner = disp._prepare(nt, pt, ct, PARAM, "d4s", None, None, None, None, None, None, None,
                           None, precision)[0]
    e, g = runner.run(pt, gradient=True)[:2]
    runner.n_slots = slots
    e2, g2 = runner.run(pt, gradient=True)[:2]
    assert (e2 - e).abs().max().item() <= 1e-9
    assert (g2 - g).abs().max().item() <= 2e-6 * g.abs().max().item()
