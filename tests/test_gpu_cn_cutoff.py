"""
A pair exactly at the cutoff of the EEQ coordination number counts (r <= cutoff,
with r the correctly rounded distance), in the counts and in their adjoint; one a
rounding step beyond does not.
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 0.0}


@pytest.mark.parametrize("seed", range(4))
def test_pairs_at_the_cutoff_count(seed):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    rng = np.random.default_rng(seed)
    numbers = torch.tensor([[6, 8]], device="cuda")
    charge = torch.zeros(1, dtype=torch.float64, device="cuda")
    for _ in range(40):
        d = rng.uniform(2.2, 3.0, 3)
        # FP64 r^2 as the kernels add it up (sums of products, either order, agree here)
        d[1:] = 0.0
        r = float(np.sqrt(d[0] * d[0]))
        pos = torch.zeros((1, 2, 3), dtype=torch.float64, device="cuda")
        pos[0, 1] = torch.from_numpy(d)

        def run(cut):
            runner = disp._prepare(numbers, pos, charge, PARAM, "d4", None, None, None, None,
                                   d4.Cutoff(cn_eeq=cut), None, None, None, "fp64")[0]
            return runner.run(pos, gradient=True, cn_eeq_out=True)

        at, above, below = run(r), run(np.nextafter(r, 9.0)), run(np.nextafter(r, 0.0))
        assert torch.equal(at[5], above[5]) and (at[5] > 0.0).all()
        assert (below[5] == 0.0).all()
        assert torch.equal(at[1], above[1]) and not torch.equal(at[1], below[1])
