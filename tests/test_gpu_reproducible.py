"""
The properties of the FP64 path repeat themselves to the last bit.
"""

from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2, 8, 9, 33), (64, 95, 96, 17), (97, 131, 40), (301, 300)],
                         ids=str)
def test_properties_repeat_exactly(sizes):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    width = max(sizes)
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    for b, n in enumerate(sizes):
        numbers[b, :n], positions[b, :n] = d4.workloads.structure(300 + n, n)
    nt, pt = torch.from_numpy(numbers).cuda(), torch.from_numpy(positions).cuda()
    first = d4.get_properties(nt, pt)
    for _ in range(10):
        assert all(torch.equal(x, y) for x, y in zip(first, d4.get_properties(nt, pt)))
