"""
The multi-CTA factorisation of the precision form's EEQ matrices: the batches that
the conjugate gradients leave to it, and its part as their fallback where a
cooperative launch is refused (by the test flag: the matrix is rebuilt for it,
in the adjoint too).

Tolerances: residuals below the solvers' 1e-10; charges 1e-7 and forces 1e-6
against FP64 (FP32 CN and matrix inputs); 1e-8 and 1e-7 against the other
solver on the same inputs (residuals of 1e-10 times an inverse of norm ~10).
"""

from __future__ import annotations

from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}
ONE_CTA, CG, DEFLATED, FACTORISATION = range(4)


@pytest.fixture(scope="module")
def d4():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return package()


def _inputs(sizes, width):
    wl = package().workloads
    numbers = np.zeros((len(sizes), width), dtype=np.int64)
    positions = np.zeros((len(sizes), width, 3))
    rng = np.random.default_rng(17)
    made = {}
    for b, n in enumerate(sizes):
        if n:
            z, r = made.setdefault(n, wl.structure(60 + n, n))
            at = np.sort(rng.permutation(width)[:n])
            numbers[b, at], positions[b, at] = z, r
    dev = torch.device("cuda")
    charge = torch.tensor([(-1.0, 0.0, 1.0)[b % 3] * (n > 0) for b, n in enumerate(sizes)],
                          dtype=torch.float64, device=dev)
    return torch.from_numpy(numbers).to(dev), torch.from_numpy(positions).to(dev), charge


def _runner(nt, pt, charge, precision="mixed"):
    disp = import_module("tad-dftd4_gb300.disp")
    return disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                         package().Cutoff(disp2=30.0, disp3=12.0), None, None, None, precision)[0]


def test_which_solver_takes_a_batch(d4):
    solver = d4._lib.load().d4_eeq_solver
    assert [solver(*x) for x in ((1, 296), (1, 297), (1, 4000), (16, 512), (1, 5000), (1, 16384),
                                 (2, 4000))] == [ONE_CTA, CG, CG, CG, DEFLATED, DEFLATED, DEFLATED]
    assert {solver(*x) for x in ((80, 303), (12, 1003), (3, 5000), (1, 16385))} == {FACTORISATION}
    assert solver(0, 5) == -1 and solver(5, 0) == -1


@pytest.mark.parametrize("sizes,width", [(tuple(range(224, 304)), 303),
                                         ((1003, 960, 1001, 0, 40) + (1002,) * 7, 1003),
                                         ((1024,) * 12, 1024)], ids=lambda v: str(v)[:20])
def test_factorisation_matches_fp64(d4, sizes, width):
    nt, pt, charge = _inputs(sizes, width)
    assert d4._lib.load().d4_eeq_solver(*nt.shape) == FACTORISATION
    mixed = _runner(nt, pt, charge)
    out = mixed.run(pt, gradient=True, charges_out=True)
    assert mixed.eeq_residuals().max().item() <= 1e-10
    plain = _runner(nt, pt, charge, "fp64").run(pt, gradient=True, charges_out=True)
    assert (out[3] - plain[3]).abs().max().item() <= 1e-7
    assert (out[1] - plain[1]).abs().max().item() <= 1e-6


def test_host_wait_changes_nothing(d4):
    """From eight 512-row blocks the later corrections wait for the host to see the
    residuals, unless the call says otherwise."""
    nt, pt, charge = _inputs((5000, 4800, 4901), 5000)
    assert d4._lib.load().d4_eeq_solver(*nt.shape) == FACTORISATION
    runner = _runner(nt, pt, charge)
    out = runner.run(pt, gradient=True, charges_out=True)
    res = runner.eeq_residuals()
    again = runner.run(pt, gradient=True, charges_out=True,
                       extra_flags=d4._lib.FLAG_NO_HOST_WAIT)
    res2 = runner.eeq_residuals()
    assert torch.equal(out[3], again[3]) and torch.equal(res[:, 0], res2[:, 0])
    assert res.max().item() <= 1e-10 and res2.max().item() <= 1e-10


@pytest.mark.parametrize("flags", ["usual", "fallback"])
@pytest.mark.parametrize("B,n", [(80, 301), (1, 423)])
def test_graph_capture(d4, B, n, flags):
    disp = import_module("tad-dftd4_gb300.disp")
    nt, pt, charge = _inputs((n,) * B, n + 2)
    runner = _runner(nt, pt, charge)
    extra = d4._lib.FLAG_TEST_FALLBACK if flags == "fallback" else 0
    want = [x.clone() for x in runner.run(pt, gradient=True, extra_flags=extra)[:2]]
    torch.cuda.synchronize()
    check, disp.CHECK_STATUS = disp.CHECK_STATUS, False
    try:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side, capture_error_mode="relaxed"):
            out = runner.run(pt, gradient=True, extra_flags=extra)
        graph.replay()
        torch.cuda.synchronize()
    finally:
        disp.CHECK_STATUS = check
    assert (out[0].sum(-1) - want[0].sum(-1)).abs().max().item() <= 1e-9
    assert (out[1] - want[1]).abs().max().item() <= 1e-8


@pytest.mark.parametrize("sizes,width", [((301,), 301), ((400, 0, 391), 403), ((1000,), 1003),
                                         ((5001,), 5001), ((4600, 4700), 4703)], ids=str)
def test_fallback_of_the_conjugate_gradients(d4, sizes, width):
    nt, pt, charge = _inputs(sizes, width)
    assert d4._lib.load().d4_eeq_solver(*nt.shape) in (CG, DEFLATED)
    runner = _runner(nt, pt, charge)
    usual = runner.run(pt, gradient=True, charges_out=True)
    out = runner.run(pt, gradient=True, charges_out=True, extra_flags=d4._lib.FLAG_TEST_FALLBACK)
    res = runner.eeq_residuals()
    assert 0.0 < res[:, 0].max().item() <= 1e-10 and 0.0 < res[:, 1].max().item() <= 1e-10
    assert (out[3] - usual[3]).abs().max().item() <= 1e-8
    assert (out[1] - usual[1]).abs().max().item() <= 1e-7
