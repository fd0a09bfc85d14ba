"""
A launch that the runtime refuses reaches the caller, whatever the library
sets up after it.
"""

from __future__ import annotations

import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu


def test_refused_launch_is_reported_every_time():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    torch.cuda.init()
    lib = package()._lib.load()
    stream = torch.cuda.current_stream().cuda_stream
    # the first call sets the second kernel up, later ones find it done
    assert [lib.d4_selftest_launch_error(stream) for _ in range(3)] == [3, 3, 3]
