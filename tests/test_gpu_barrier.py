"""
The barrier between the CTAs of an EEQ solve gives up after its limit, in every
CTA, and reports it; launches after that are not affected.
"""

from __future__ import annotations

import time

import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu
LIMIT = 5_000_000  # ns


@pytest.mark.parametrize("ctas", [1, 2, 37, 64])
def test_barrier_gives_up_in_every_cta(ctas):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib = package()._lib.load()
    res = torch.full((2 + ctas,), -1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream

    def run(extra):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        assert lib.d4_selftest_barrier(res.data_ptr(), ctas, extra, LIMIT, stream) == 0
        out = res.tolist()
        return out[0], out[1], out[2:], time.perf_counter() - t0

    assert run(0)[:3] == (0, 2 * ctas, [2] * ctas)
    status, arrivals, passed, seconds = run(1)
    assert (status, arrivals, passed) == (8, 2 * ctas, [1] * ctas)
    assert 1e-9 * LIMIT <= seconds < 0.5
    assert run(0)[:3] == (0, 2 * ctas, [2] * ctas)


def test_argument_checks():
    lib = package()._lib.load()
    for bad in ((None, 2, 1, LIMIT), (8, 0, 1, LIMIT), (8, 65, 1, LIMIT), (8, 2, 2, LIMIT),
                (8, 2, 1, 2 * 10 ** 9)):
        assert lib.d4_selftest_barrier(*bad, None) == 1  # nothing launched
