"""The library's streams are non-blocking: they do not wait for the legacy
stream, so every copy and every fill has to be queued on the stream of the
kernels that read it, and a call that promises its result has to wait for it."""
from __future__ import annotations

import re
import time
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tups_b200" / "csrc"


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh", ".h")))
def test_no_copy_or_fill_on_the_legacy_stream(source):
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    calls = re.findall(r"\b(cudaMemcpy|cudaMemset|cudaMemcpyToSymbol|cudaMemcpyFromSymbol|cudaMemcpy2D)\s*\(", text)
    assert not calls, calls


@pytest.mark.gpu
def test_crossing_tensor_calls_complete_before_they_return(gpu_lib):
    """13 form factors on 16x16 momenta: some milliseconds of device work per tensor, by the library's own events."""
    from tups_b200 import Params, Solver
    sol = Solver(Params(beta=2.0, U=2.0, nParticle=1.0, Nx=16, Nf=8, neighbours=4, ite_max=5))
    sol.calculate_expSqR()
    sol.calculate_expqSR()
    for name in ("phbar_to_ph", "pp_to_ph", "ph_to_pp", "phbar_to_pp"):
        calc = getattr(sol, "calc_M_" + name)
        calc()  # the first call makes the tables
        sol.synchronize()
        sol.record_event(0)
        t0 = time.perf_counter()
        calc()
        host_ms = 1e3 * (time.perf_counter() - t0)
        sol.record_event(1)
        device_ms = sol.event_elapsed_ms(0, 1)
        assert device_ms > 0.2  # against some 0.02 ms for a call that only queues its kernel
        assert host_ms >= 0.5 * device_ms, (name, host_ms, device_ms)
    sol.close()
