"""LU form of the BSE (F = (1 - c Gamma chi)^{-1} Gamma), batched over
instances of uneven size: CPU checks of the oracle and the workload
generator, GPU parity with LAPACK (scipy zgetrf/zgetrs)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import lu as LU


def test_lu_form_is_the_fixed_point_of_the_damped_update():
    """The reference's damped two-ordering BSE update, iterated with Gamma
    fixed, converges to the LU solution."""
    from tups_b200.bse_batched import make_instances
    inst = make_instances(n_q=2, n_w=1, nf=8, nff_choices=(1, 5), rho=0.6, seed=3)
    for g, c in zip(inst.gamma, inst.chi):
        F_lu = LU.bse_lu(g, c, 1.0)
        F_it = LU.damped_fixed_point(g, c, 1.0, f=0.5)
        assert np.abs(F_lu - F_it).max() <= 1e-12 * np.abs(F_lu).max()


def test_generator_is_seeded_and_scaled():
    from tups_b200.bse_batched import chi_dense, make_instances, spectral_radius
    a = make_instances(n_q=3, n_w=2, nf=8, seed=7)
    b = make_instances(n_q=3, n_w=2, nf=8, seed=7)
    assert np.array_equal(a.nl, b.nl)
    for x, y in zip(a.gamma, b.gamma):
        assert np.array_equal(x, y)
    for g, c in zip(a.gamma, a.chi):
        assert np.allclose(g, g.conj().T)
        assert np.max(np.abs(np.linalg.eigvals(g @ chi_dense(c)))) == pytest.approx(0.9, rel=1e-8)
    assert set(a.n.tolist()) <= {8, 40, 72, 104}


@pytest.mark.gpu
def test_batched_lu_matches_lapack(gpu_lib):
    from tups_b200.bse_batched import make_instances, solve
    inst = make_instances(n_q=6, n_w=4, nf=16, seed=11)  # n in {16, 80, 144, 208}
    assert len(set(inst.n.tolist())) >= 3
    F = solve(inst)
    for i, (g, c) in enumerate(zip(inst.gamma, inst.chi)):
        ref = LU.bse_lu(g, c, 1.0)
        err = np.abs(F[i] - ref).max() / np.abs(ref).max()
        assert err < 1e-12, (i, int(inst.n[i]), err)


@pytest.mark.gpu
def test_batched_lu_phi_and_scale(gpu_lib):
    from tups_b200.bse_batched import make_instances, solve
    inst = make_instances(n_q=2, n_w=3, nf=12, seed=5, rho=0.5)
    inst.scale = np.linspace(0.5, 1.5, len(inst.n))
    Phi = solve(inst, want_phi=True)
    for i, (g, c) in enumerate(zip(inst.gamma, inst.chi)):
        ref = LU.bse_lu(g, c, float(inst.scale[i])) - g
        assert np.abs(Phi[i] - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.gpu
def test_batched_lu_reports_singular_pivot(gpu_lib):
    """Gamma chi with an eigenvalue 1 makes A = I - Gamma chi singular; the
    status array reports the column instead of returning NaNs silently."""
    from tups_b200 import TupsError
    from tups_b200.bse_batched import Instances, solve
    n = 8
    chi = np.zeros((1, 1, n), dtype=np.complex128, order="F")
    chi[0, 0, :] = 1.0
    g = np.asfortranarray(np.eye(n, dtype=np.complex128))  # A = I - I = 0
    inst = Instances(n=np.array([n], dtype=np.int32), nl=np.array([1], dtype=np.int32), scale=np.ones(1),
                     gamma=[g], chi=[chi], q=np.zeros((1, 3), dtype=np.int32))
    with pytest.raises(TupsError, match="singular"):
        solve(inst)


@pytest.mark.gpu
@pytest.mark.parametrize("slices", [4, 5, 7])
def test_split_lu_with_refinement_matches_lapack(gpu_lib, slices):
    """Split-precision LU (int8 trailing and solve updates) refined in FP64
    to the LAPACK answer; sizes up to 2 blocks of 128 plus a ragged tail."""
    from tups_b200.bse_batched import make_instances, solve_split
    inst = make_instances(n_q=4, n_w=4, nf=48, seed=13, nff_choices=(1, 5, 9))  # n in {48, 240, 432}
    assert len(set(inst.n.tolist())) >= 2
    F, info = solve_split(inst, slices=slices, tol=1e-12, max_refine=8)
    assert np.all(info["residual"] <= 1e-12), info
    for i, (g, c) in enumerate(zip(inst.gamma, inst.chi)):
        ref = LU.bse_lu(g, c, 1.0)
        err = np.abs(F[i] - ref).max() / np.abs(ref).max()
        assert err < 1e-12, (i, int(inst.n[i]), slices, err)
    # the int8 factors alone are not FP64-accurate: at least one correction
    assert int(info["refinements"].max()) >= 1


@pytest.mark.gpu
def test_split_lu_phi_scale_and_unrefined_error(gpu_lib):
    """want_phi and per-instance scales; without refinement the error is the
    split GEMM's, after refinement the FP64 LU's."""
    from tups_b200.bse_batched import LuBatch, make_instances
    inst = make_instances(n_q=2, n_w=3, nf=40, seed=5, rho=0.5, nff_choices=(1, 5))
    inst.scale = np.linspace(0.5, 1.5, len(inst.n))
    b = LuBatch(inst)
    refs = [LU.bse_lu(g, c, float(inst.scale[i])) - g for i, (g, c) in enumerate(zip(inst.gamma, inst.chi))]
    errs = {}
    for steps in (0, 8):
        info = b.run_split(slices=3, tol=1e-12, max_refine=steps, want_phi=True)
        out = b.results()
        errs[steps] = max(np.abs(out[i] - refs[i]).max() / np.abs(refs[i]).max() for i in range(len(refs)))
    assert 1e-9 < errs[0] < 1e-2, errs
    assert errs[8] < 1e-12, errs


@pytest.mark.gpu
def test_batched_lu_at_block_edges(gpu_lib):
    """Sizes around the 32-column panels, the 64-column blocks, the 512 rows of
    one register row per thread and the 1024 rows past which a panel stays in
    global memory, each with rows that need interchanges, in one batch."""
    from tups_b200.bse_batched import Instances, solve
    sizes = [1, 7, 16, 31, 32, 33, 63, 64, 65, 96, 97, 128, 129, 513, 577, 1089]
    rng = np.random.default_rng(29)
    gam, chi, nls = [], [], []
    for n in sizes:
        nl = next(k for k in (9, 5, 3, 1) if n % k == 0)
        c = rng.standard_normal((nl, nl, n // nl)) + 1j * rng.standard_normal((nl, nl, n // nl))
        g = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        # |Gamma chi|_2 <= 0.9 (|g|_2 below 3 sqrt(n), blocks by their own norm) ...
        g *= 0.9 / (3.0 * np.sqrt(n) * max(np.linalg.norm(c[:, :, i], 2) for i in range(n // nl)))
        gam.append(np.asfortranarray(g))
        chi.append(np.asfortranarray(c))
        nls.append(nl)
    inst = Instances(n=np.array(sizes, dtype=np.int32), nl=np.array(nls, dtype=np.int32), scale=np.ones(len(sizes)),
                     gamma=gam, chi=chi, q=np.zeros((len(sizes), 3), dtype=np.int32))
    for i, (got, g, c) in enumerate(zip(solve(inst), gam, chi)):
        ref = LU.bse_lu(g, c, 1.0)
        # ... so cond(A) <= 1.9 / 0.1, and the forward error is at most about 4 n eps cond
        assert np.abs(got - ref).max() <= 4 * sizes[i] * 2.3e-16 * 19 * np.abs(ref).max(), sizes[i]
    # rows far from the diagonal as pivots: A = I - chi with chi cyclic shifts per frequency block
    n = 130
    g = np.zeros((n, n), dtype=np.complex128, order="F")
    g[np.arange(n), (np.arange(n) + 67) % n] = 5.0 + rng.uniform(0.0, 1.0, n)
    g += 0.01 * rng.standard_normal((n, n))
    inst = Instances(n=np.array([n], dtype=np.int32), nl=np.array([1], dtype=np.int32), scale=np.ones(1), gamma=[g],
                     chi=[np.ones((1, 1, n), dtype=np.complex128, order="F")], q=np.zeros((1, 3), dtype=np.int32))
    ref = LU.bse_lu(g, inst.chi[0], 1.0)
    cond = np.linalg.cond(np.eye(n) - g)
    assert np.abs(solve(inst)[0] - ref).max() <= 4 * n * 2.3e-16 * cond * np.abs(ref).max()


def _unit_chi_instances(mats):
    """A x = (I - A) for each matrix A: Gamma = I - A with one form factor and chi = 1."""
    from tups_b200.bse_batched import Instances
    n = np.array([a.shape[0] for a in mats], dtype=np.int32)
    return Instances(n=n, nl=np.ones(len(mats), dtype=np.int32), scale=np.ones(len(mats)),
                     gamma=[np.asfortranarray(np.eye(a.shape[0]) - a) for a in mats],
                     chi=[np.ones((1, 1, k), dtype=np.complex128, order="F") for k in n],
                     q=np.zeros((len(mats), 3), dtype=np.int32))


def _residual_over_factors(g, x):
    """max |Gamma - A X| / (|L| |U| |X|) with LAPACK's factors of A = 1 - Gamma."""
    import scipy.linalg as sl
    n = g.shape[0]
    a = np.eye(n) - g
    lu, piv = sl.lu_factor(a)
    p = np.arange(n)
    for i, k in enumerate(piv):
        p[[i, k]] = p[[k, i]]
    low, up = np.tril(lu, -1) + np.eye(n), np.triu(lu)
    r = np.abs(g.astype(np.clongdouble) - a.astype(np.clongdouble) @ x)[p].astype(float)
    return (r / np.maximum(np.abs(low) @ (np.abs(up) @ np.abs(x)), 1e-300)).max()


def _hard_matrices(n):
    rng = np.random.default_rng(n)
    z = lambda: rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    u, v = (np.linalg.qr(z())[0] for _ in range(2))
    s = np.logspace(6, -6, n)
    h = z()
    w, q = np.linalg.eigh(h + h.conj().T)
    w *= 0.9 / np.abs(w).max()
    w[-1] = 1.0 - 1e-8
    return [z(), z() * s[None, :], z() * s[:, None], z() * np.sqrt(s)[:, None] / np.sqrt(s)[None, :],
            (u * np.logspace(0, -6, n)) @ v, (u * np.logspace(0, -10, n)) @ v, np.eye(n) - (q * w) @ q.conj().T]


# The factorisation and the two triangular solves each leave a residual of sums of n complex products, 2 sqrt(2)
# units of rounding each, that add up as their square root: 3 x 2.83 sqrt(n) units of |L| |U| |X|
def _residual_bound(n):
    return 8.5 * np.sqrt(n) * 1.11e-16


@pytest.mark.gpu
@pytest.mark.parametrize("n", [50, 130, 300])
def test_batched_lu_is_backward_stable(gpu_lib, n):
    """Condition numbers of 1e6 and 1e10, rows and columns over twelve decades, 1 - Gamma chi next to singular: the
    residual stays that of substitution with the factors."""
    from tups_b200.bse_batched import solve
    inst = _unit_chi_instances(_hard_matrices(n))
    for i, x in enumerate(solve(inst)):
        r = _residual_over_factors(inst.gamma[i], x)
        assert r <= _residual_bound(n), (i, r)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [50, 128])
def test_unsplit_blocks_of_the_split_lu_are_backward_stable(gpu_lib, n):
    """Up to 128 columns nothing runs on int8 slices: the same bound without a correction."""
    from tups_b200.bse_batched import solve_split
    inst = _unit_chi_instances(_hard_matrices(n))
    for i, x in enumerate(solve_split(inst, slices=8, max_refine=0)[0]):
        r = _residual_over_factors(inst.gamma[i], x)
        assert r <= _residual_bound(n), (i, r)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 129, 300])
def test_batched_lu_keeps_small_imaginary_parts(gpu_lib, n):
    """A real to 1e-8: the imaginary part of the solution has the relative error of the real one (4 n eps cond,
    cond(A) of the real part), since every product of the imaginary parts' sums is small."""
    from tups_b200.bse_batched import solve
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1e-8j * rng.standard_normal((n, n))
    inst = _unit_chi_instances([a])
    g = inst.gamma[0]
    a = np.eye(n) - g
    ref = LU.bse_lu(g, inst.chi[0], 1.0).astype(np.clongdouble)
    for _ in range(3):
        r = g.astype(np.clongdouble) - a.astype(np.clongdouble) @ ref
        ref += np.linalg.solve(a, r.real.astype(float)) + 1j * np.linalg.solve(a, r.imag.astype(float))
    err = np.abs((solve(inst)[0] - ref).imag).max() / np.abs(ref.imag).max()
    assert err <= 4 * n * 2.3e-16 * np.linalg.cond(a), err


def _edge_instances(sizes, seed):
    """One form factor, chi diagonal in the frequency; |Gamma chi|_2 <= 0.9, so |A^-1|_2 <= 10."""
    from tups_b200.bse_batched import Instances
    rng = np.random.default_rng(seed)
    gam, chi = [], []
    for n in sizes:
        c = rng.standard_normal((1, 1, n)) + 1j * rng.standard_normal((1, 1, n))
        g = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        g *= 0.9 / (3.0 * np.sqrt(n) * np.abs(c).max())
        gam.append(np.asfortranarray(g))
        chi.append(np.asfortranarray(c))
    return Instances(n=np.array(sizes, dtype=np.int32), nl=np.ones(len(sizes), dtype=np.int32),
                     scale=np.ones(len(sizes)), gamma=gam, chi=chi, q=np.zeros((len(sizes), 3), dtype=np.int32))


@pytest.mark.gpu
def test_split_lu_at_block_edges(gpu_lib):
    """Remainders of 1, 63, 64, 65 and 127 in a block of 128, fewer than 64 rows, and the row counts past which a
    panel takes two rows per thread and past which it stays in global memory; two instances of some sizes."""
    from tups_b200.bse_batched import solve_split
    sizes = [1, 7, 33, 63, 64, 65, 65, 127, 128, 129, 129, 191, 192, 193, 255, 257, 513, 577, 1089]
    inst = _edge_instances(sizes, 31)
    tol = 1e-12
    out, info = solve_split(inst, slices=6, tol=tol, max_refine=8)
    assert np.all(info["residual"] <= tol)
    for i, x in enumerate(out):
        g = inst.gamma[i]
        ref = LU.bse_lu(g, inst.chi[i], 1.0)
        # a column of the residual is at most sqrt(n) tol max|Gamma|, and the oracle's own error is far below
        assert np.abs(x - ref).max() <= 11 * np.sqrt(sizes[i]) * tol * np.abs(g).max(), sizes[i]


@pytest.mark.gpu
@pytest.mark.parametrize("n", [130, 200, 600])
def test_split_lu_interchanges_far_from_the_diagonal(gpu_lib, n):
    """Every pivot far below its diagonal entry, by another distance in each of three instances of one group."""
    from tups_b200.bse_batched import solve_split
    rng = np.random.default_rng(n)
    mats = []
    for shift in (n // 2 + 2, 1, n - 70):
        a = 0.01 * (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
        a[(np.arange(n) + shift) % n, np.arange(n)] += 5.0 + rng.uniform(0.0, 1.0, n)
        mats.append(a)
    inst = _unit_chi_instances(mats)
    tol = 1e-12
    out, info = solve_split(inst, slices=6, tol=tol, max_refine=8)
    assert np.all(info["residual"] <= tol)
    for i, x in enumerate(out):
        g = inst.gamma[i]
        # |A^-1| is at most 1 / (5 - 0.02)
        assert np.abs(x - LU.bse_lu(g, inst.chi[i], 1.0)).max() <= 0.25 * np.sqrt(n) * tol * np.abs(g).max(), i


@pytest.mark.gpu
@pytest.mark.parametrize("t", [1e-40, 1e-158, 1e-250, 1e-300])
def test_pivots_of_any_magnitude(gpu_lib, t):
    """A = 1 - Gamma with pivots of t, whose square is far below the smallest double: the first columns hold nothing
    but -t, one row off the diagonal, and X = A^-1 Gamma comes out in closed form."""
    from tups_b200.bse_batched import solve, solve_split
    n, m = 70, 5
    a = 2.0 * np.eye(n, dtype=np.complex128)
    a[:m, :m] = -t * (1.0 + 0.5j) * np.roll(np.eye(m), 1, axis=0)
    inst = _unit_chi_instances([a])
    want = -0.5 * np.eye(n, dtype=np.complex128)
    want[:m, :m] = np.roll(np.eye(m), -1, axis=0) / (-t * (1.0 + 0.5j)) - np.eye(m)  # A^-1 - 1
    for got in (solve(inst)[0], solve_split(inst, slices=8, max_refine=0)[0][0]):
        big = np.abs(want) > 0.0
        assert np.all(got[~big] == 0.0)
        assert np.abs(got[big] / want[big] - 1.0).max() <= 8 * 2.3e-16


@pytest.mark.gpu
@pytest.mark.parametrize("split", [False, True])
def test_small_instances_are_solved_whole(gpu_lib, split):
    """Up to 32 rows an instance is one CTA's: the residual bound of the blocks, in a batch where larger instances
    stand before and between them."""
    from tups_b200.bse_batched import solve, solve_split
    mats = [m for n in (40, 32, 5, 31, 33, 2, 20) for m in _hard_matrices(n)] + [np.full((1, 1), 3.0 - 2.0j)]
    inst = _unit_chi_instances(mats)
    out = solve_split(inst, slices=8, max_refine=0)[0] if split else solve(inst)
    for i, x in enumerate(out):
        r = _residual_over_factors(inst.gamma[i], x)
        assert r <= _residual_bound(mats[i].shape[0]), (i, mats[i].shape[0], r)
