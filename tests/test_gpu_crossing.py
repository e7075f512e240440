"""The crossing on a B200 at sizes around its tiles: element lists and columns
that no tile divides, sums of one and several stages, the short-sum and the
long-sum tiles, both product forms, one form factor."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import tups_oracle as O
import parity

pytestmark = pytest.mark.gpu

# FP64 sums of a few hundred terms against the oracle's: 1e-12 of the largest
TOL = 1e-12


@pytest.mark.parametrize("products", [3, 4])
@pytest.mark.parametrize("case", [
    dict(Nx=4, Nf=6, neighbours=1),
    dict(Nx=4, Nf=18, neighbours=1),
    dict(Nx=4, Nf=6, neighbours=2),
    dict(Nx=6, Nf=14, neighbours=2),
    dict(Nx=4, Nf=10, neighbours=3),
], ids=["nl1_nf6", "nl1_nf18", "nl5_nf6", "nl5_nf14_nx6", "nl9_nf10"])
def test_crossing_at_tile_edges(gpu_lib, case, products):
    from tups_b200 import Solver
    p = O.Params(beta=3.0, U=2.0, nParticle=0.95, f_damping=0.5, ite_max=10, **case)
    st = O.initialize(p)
    sol = Solver(parity.to_solver_params(p))
    sol.set_crossing_products(products)
    rng = np.random.default_rng(case["Nf"] + products)
    shape = (sol.Nz, sol.Nz, sol.Nb)
    G = {r: rng.standard_normal(shape) + 1j * rng.standard_normal(shape) for r in "dmst"}
    sol.calculate_expSqR()
    sol.calculate_expqSR()
    for w in ("phbar_to_ph", "pp_to_ph", "ph_to_pp", "phbar_to_pp"):
        getattr(sol, "calc_M_" + w)()
    for r in "dmst":
        sol.set_vertex(r, 1, G[r])
    sol.calc_PhiR(0)
    sol.calculate_PAE()
    O.calculate_expSqR(st)
    O.calculate_expqSR(st)
    for r in "dmst":
        st.G[r] = G[r].copy()
    O.calc_PhiR(st)
    O.calc_M(st)
    O.calculate_PAE(st)
    for r in "dmst":
        assert parity.rel(sol.F(r), st.F[r]) <= TOL, r
    sol.close()


def test_crossing_takes_no_memory_of_its_own(gpu_lib):
    """The gathered operand (0.15 GB here) goes into the BSE's scratch: the first crossing of a context allocates its
    element lists and no more, so that what fits a card beside a context does not depend on it."""
    import torch
    from tups_b200 import Params, Solver
    sol = Solver(Params(beta=3.0, U=2.0, nParticle=0.95, Nx=8, Nf=32, neighbours=2, f_damping=0.5, ite_max=10))
    sol.set_autotune(False)
    sol.calculate_expSqR()
    sol.calculate_expqSR()
    for w in ("phbar_to_ph", "pp_to_ph", "ph_to_pp", "phbar_to_pp"):
        getattr(sol, "calc_M_" + w)()
    sol.calc_PhiR(0)
    free0 = torch.cuda.mem_get_info()[0]
    sol.calculate_PAE()
    assert free0 - torch.cuda.mem_get_info()[0] <= 16 << 20
    sol.close()


def test_crossing_leaves_the_bse_alone(gpu_lib):
    """The scratch is the BSE's again in the next iteration: three iterations, two in FP64 and one split, queued as
    one against the single calls, each of which waits."""
    from tups_b200 import Params, Solver
    p = Params(beta=3.0, U=2.0, nParticle=0.95, Nx=4, Nf=10, neighbours=3, f_damping=0.5, ite_max=10)
    a, b = Solver(p), Solver(p)
    for ite in range(3):
        if ite == 2:
            for s in (a, b):
                s.set_bse_precision(5)
        a.iteration(ite)
        b.calc_Gkw_Grt(ite)
        b.BSE(ite)
        if ite == 0:
            b.calculate_expSqR()
            b.calculate_expqSR()
            for w in ("phbar_to_ph", "pp_to_ph", "ph_to_pp", "phbar_to_pp"):
                getattr(b, "calc_M_" + w)()
        b.calc_PhiR(ite)
        b.calculate_PAE()
        b.calc_SDE(ite)
        b.conv()
        if ite % 5 == 0:
            b.output_block()
        b.vertex_update()
        assert np.array_equal(a.Sigma, b.Sigma)
        for r in "dmst":
            assert np.array_equal(a.F(r), b.F(r)) and np.array_equal(a.G(r), b.G(r))
    a.close()
    b.close()


@pytest.mark.parametrize("neighbours,ntasks", [(2, 30), (2, 15), (2, 10), (2, 6), (2, 5), (2, 3), (2, 2), (3, 30), (3, 10)])
def test_crossing_of_a_ranks_slots(gpu_lib, neighbours, ntasks):
    """One slot, some frequencies of a momentum, of two, whole momenta: the crossing of a rank's slots, by the form
    that gathers in the GEMM (up to 64 columns) or ahead of it, against the crossing of all slots."""
    import torch
    from tups_b200 import Params, Solver
    from tups_b200.sharded import _DeviceBuffer
    p = Params(beta=3.0, U=2.0, nParticle=0.95, Nx=4, Nf=10, neighbours=neighbours, f_damping=0.5, ite_max=10)
    full = Solver(p)
    rng = np.random.default_rng(ntasks)
    shape = (full.Nz, full.Nz, full.Nb)
    G = {r: rng.standard_normal(shape) + 1j * rng.standard_normal(shape) for r in "dmst"}
    phir = {}

    def whole_phir(what, ptr, count, op):
        t = torch.as_tensor(_DeviceBuffer(ptr, count), device="cuda:0")
        t.copy_(torch.from_numpy(phir["dmst"[what]]))
        torch.cuda.synchronize()

    def crossing(sol, slots):
        sol.calculate_expSqR()
        sol.calculate_expqSR()
        for w in ("phbar_to_ph", "pp_to_ph", "ph_to_pp", "phbar_to_pp"):
            getattr(sol, "calc_M_" + w)()
        for r in "dmst":
            sol.set_vertex(r, 1, np.asfortranarray(G[r][..., slots]))
        sol.calc_PhiR(0)

    crossing(full, slice(None))
    phir.update({r: np.ravel(full.PhiR(r), order="F").view(np.float64).copy() for r in "dmst"})
    want = {}
    for products in (3, 4):
        full.set_crossing_products(products)
        full.calculate_PAE()
        want[products] = {r: full.F(r).copy() for r in "dmst"}
    full.close()
    for rank in sorted({0, ntasks // 2, ntasks - 1}):
        sol = Solver(p, 0, rank, ntasks, whole_phir)
        slots = slice(sol.slot0, sol.slot0 + sol.Nb)
        crossing(sol, slots)
        for products in (3, 4):
            sol.set_crossing_products(products)
            sol.calculate_PAE()
            for r in "dmst":
                assert parity.rel(sol.F(r), want[products][r][..., slots]) <= TOL, (rank, products, r)
        sol.close()
