"""
The library's own reciprocal, inverse square root (FP64) and exponential (FP32)
against values of more digits, over their whole ranges, and at their edges.

Bounds: a third-order step from 20 bits leaves 2^-60, so the reciprocal is within
0.5 ulp of its last rounding plus 0.01; the inverse root has the rounding of d y in
its residual on top, 1.01; the exponential is formed to 1e-10 relative (0.002 ulp
of FP32) and rounded once, 0.502.
"""

from __future__ import annotations

from fractions import Fraction
from math import isqrt

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu
INF = float("inf")


def _apply(which, x):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    lib = package()._lib.load()
    dx = torch.from_numpy(np.asarray(x, dtype=np.float64)).cuda()
    dy = torch.empty_like(dx)
    assert lib.d4_selftest_math(which, dx.data_ptr(), dy.data_ptr(), dx.numel(),
                                torch.cuda.current_stream().cuda_stream) == 0
    return dy.cpu().numpy()


def _arguments(lo, hi, n=20000):
    rng = np.random.default_rng(1)
    wide = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n))
    near = np.nextafter(np.ldexp(1.0, rng.integers(lo + 1, hi, 200)), rng.choice([0.0, INF], 200))
    return np.concatenate([wide, rng.uniform(1.0, 4.0, n), near, np.ldexp(1.0, np.arange(lo, hi, 7))])


def test_reciprocal():
    x = _arguments(-1021, 1021)
    got = _apply(0, x)
    worst = 0.0
    for a, y in zip(x.tolist(), got.tolist()):
        worst = max(worst, abs(float((Fraction(y) - 1 / Fraction(a)) / Fraction(np.spacing(y)))))
    assert worst <= 0.51, worst


def test_inverse_root():
    x = _arguments(-1021, 1023)
    got = _apply(1, x)
    worst = 0.0
    for a, y in zip(x.tolist(), got.tolist()):
        f = Fraction(a)
        # 1 / sqrt(f) to 200 bits and more below the result's last one
        shift = 600 + 2 * max(0, f.denominator.bit_length(), f.numerator.bit_length())
        root = Fraction(isqrt((f.denominator << (2 * shift)) // f.numerator), 1 << shift)
        worst = max(worst, abs(float((Fraction(y) - root) / Fraction(np.spacing(y)))))
    assert worst <= 1.01, worst


def test_exponential():
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-80.0, 80.0, 20000), rng.uniform(-3.0, 3.0, 20000),
                        rng.uniform(-1e-3, 1e-3, 2000), [0.0, 80.0, -80.0, 1e-30, -1e-30]])
    got = _apply(2, x)
    ulp = np.spacing(got.astype(np.float32)).astype(np.float64)
    worst = np.abs((got - np.exp(x)) / ulp).max()  # (FP64's exp: 2e-9 of such an ulp)
    assert worst <= 0.502, worst


def test_edges():
    tiny = 5e-324
    assert _apply(0, [INF, 0.0, tiny]).tolist() == [0.0, INF, INF]
    assert _apply(0, [2.0 ** 1023, 1.7e308]).tolist() == [0.0, 0.0]
    assert _apply(1, [INF, 0.0, tiny]).tolist() == [0.0, INF, INF]
    assert np.isnan(_apply(0, [np.nan])).all() and np.isnan(_apply(1, [np.nan])).all()


@pytest.mark.parametrize("gradient", [False, True])
def test_far_atom_without_cutoff(gradient):
    """r^8 of a pair beyond FP64's range: no energy, as of any pair that far."""
    d4 = package()
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    param = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 0.0}
    numbers = torch.tensor([[6, 8, 10]], device="cuda")
    pos = torch.zeros((1, 3, 3), dtype=torch.float64, device="cuda")
    pos[0, 1, 0], pos[0, 2, 0] = 2.3, 1e40
    call = d4.dispersion_energy_gradient if gradient else (lambda *a, **k: (d4.dftd4(*a, **k),))
    far = call(numbers, pos, 0.0, param, cutoff=d4.Cutoff(disp2=INF))
    near = call(numbers, pos, 0.0, param)
    for x, y in zip(far, near):
        assert torch.isfinite(x).all() and (x - y).abs().max().item() <= 1e-15
