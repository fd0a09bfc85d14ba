"""
Calls on several streams and threads at once: the cooperative launches of the
iterative EEQ solves (which need all of their CTAs resident) beside each other
and beside ordinary kernels.  Every wait of theirs is bounded, so a launch that
did not get its CTAs would report status 8; results are those of calls one
after the other (charges 1e-8, forces 1e-7: order of FP32 sums).
"""

from __future__ import annotations

import threading
from importlib import import_module

import numpy as np
import pytest
import torch

from conftest import package

pytestmark = pytest.mark.gpu

PARAM = {"s6": 1.0, "s8": 1.2, "a1": 0.4, "a2": 5.0, "s9": 1.0}
# (structures, atoms, precision): conjugate gradients of one and of several groups,
# deflated, factorisation with its side stream, one CTA, FP64
BATCHES = [(1, 997, "mixed"), (16, 512, "mixed"), (1, 5001, "mixed"), (80, 301, "mixed"),
           (100, 60, "mixed"), (8, 131, "fp64")]


def test_concurrent_calls_match_sequential_ones():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    d4 = package()
    disp = import_module("tad-dftd4_gb300.disp")
    jobs = []
    for B, n, precision in BATCHES:
        z, r = d4.workloads.structure(n, n)
        nt = torch.from_numpy(np.tile(z, (B, 1))).cuda()
        pt = torch.from_numpy(np.tile(r, (B, 1, 1))).cuda()
        charge = torch.zeros(B, dtype=torch.float64, device="cuda")

        def make(nt=nt, pt=pt, charge=charge, precision=precision):
            runner = disp._prepare(nt, pt, charge, PARAM, "d4", None, None, None, None,
                                   d4.Cutoff(disp2=30.0, disp3=8.0), None, None, None,
                                   precision)[0]
            return runner.run(pt, gradient=True, charges_out=True)

        jobs.append((make, [x.clone() for x in (lambda o: (o[1], o[3]))(make())]))
    torch.cuda.synchronize()
    failures = []

    def work(first):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for k in range(18):
                    make, (g, q) = jobs[(first + k) % len(jobs)]
                    out = make()  # (reads its status word)
                    if (out[3] - q).abs().max().item() > 1e-8:
                        failures.append((first, k, "charges"))
                    if (out[1] - g).abs().max().item() > 1e-7:
                        failures.append((first, k, "gradient"))
        except Exception as exc:  # noqa: BLE001 (reported below)
            failures.append((first, repr(exc)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
