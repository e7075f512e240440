"""The warm start on a B200: MLP kernels vs the float64 oracle, the warm-start
entry point vs the oracle, checkpoint/restore, and the fallback."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import tups_oracle as O
from oracle import warmstart as OW
import parity

pytestmark = pytest.mark.gpu

# FP32 kernels against the float64 oracle: max-norm relative error
MLP_TOL = 1e-4


@pytest.mark.parametrize("shape", [(37, 64, 3, 11, 20), (964, 512, 3, 968, 32)], ids=["small", "config5"])
def test_mlp_forward_and_gradients_match_oracle(gpu_lib, shape):
    from tups_b200.warmstart import MLP
    n_in, hidden, layers, n_out, batch = shape
    net = MLP(n_in, n_out, hidden, layers, max_batch=64, seed=5)
    rng = np.random.default_rng(7)
    p = net.get_params() + rng.normal(0, 0.02, net.n_params).astype(np.float32)
    net.set_params(p)
    x = rng.normal(size=(batch, n_in)).astype(np.float32)
    t = rng.normal(size=(batch, n_out)).astype(np.float32)
    y = net.forward(x)
    y_ref, _ = OW.mlp_forward(p, net.widths, x)
    assert parity.rel(y, y_ref) <= MLP_TOL
    loss, g = net.gradients(x, t)
    loss_ref, g_ref = OW.mlp_loss_grad(p, net.widths, x, t)
    assert abs(loss - loss_ref) <= MLP_TOL * loss_ref
    layout, _ = OW.mlp_layout(net.widths)
    for wo, bo, fin, fout in layout:   # per weight matrix and bias vector
        assert parity.rel(g[wo:bo], g_ref[wo:bo]) <= MLP_TOL
        assert parity.rel(g[bo:bo + fout], g_ref[bo:bo + fout]) <= MLP_TOL
    assert net.kernel_launches > 0
    net.close()


def test_mlp_training_fits_a_smooth_map(gpu_lib):
    from tups_b200.warmstart import MLP
    rng = np.random.default_rng(11)
    x = rng.uniform(-1, 1, size=(160, 6))
    a = rng.normal(size=(6, 4))
    t = np.sin(x @ a) + 0.1 * (x @ a) ** 2
    net = MLP(6, 4, 128, 3, max_batch=256, seed=1)
    loss0, _ = net.gradients(x, t)
    hist = net.train(x, t, batch=32, epochs=400, lr=2e-3, seed=3)
    loss1, _ = net.gradients(x, t)
    assert loss1 < 0.02 * loss0, (loss0, loss1)
    assert hist[-1] < 0.05 * hist[0]
    # determinism: same seed, same parameters
    net2 = MLP(6, 4, 128, 3, max_batch=256, seed=1)
    net2.train(x, t, batch=32, epochs=400, lr=2e-3, seed=3)
    np.testing.assert_allclose(net2.get_params(), net.get_params(), rtol=0, atol=1e-5)
    net.close()
    net2.close()


def _case():
    return O.Params(beta=2.0, U=2.0, nParticle=0.9, Nx=4, Nf=8, neighbours=2, tprime=-0.1, f_damping=0.5,
                    ite_max=50)


def test_warm_start_matches_oracle(gpu_lib):
    from tups_b200 import Solver
    p = _case()
    st = O.initialize(p)
    O.iteration(st, 0)
    sol = Solver(parity.to_solver_params(p))
    sol.iteration(0)
    rng = np.random.default_rng(4)
    sigma = st.Sigma * (1.0 + 0.05 * rng.normal(size=st.Sigma.size))
    gam = np.array([2.1 + 0.02j, -1.8 - 0.01j, 3.9, 0.3j])
    OW.warm_start(st, sigma, gam)
    sol.warm_start(sigma, gam)
    assert abs(sol.mu - st.mu) <= 1e-12
    assert parity.rel(sol.Sigma, st.Sigma) == 0.0
    for i, r in enumerate("dmst"):
        assert parity.rel(sol.G(i), st.G[r]) == 0.0
        # LU with partial pivoting vs LAPACK's solve: <= 1e-12
        assert parity.rel(sol.F(i), st.F[r]) <= 1e-12, r
    # F is the fixed point of the library's own damped BSE update
    F = [sol.F(i) for i in range(4)]
    G = [sol.G(i) for i in range(4)]
    sol.calc_Gkw_Grt(1)
    sol.BSE(1)
    for i in range(4):
        assert parity.rel(sol.G(i), F[i] - G[i]) <= 1e-12
    # and the loop continues from it on both sides
    sol2 = Solver(parity.to_solver_params(p))
    sol2.iteration(0)
    sol2.warm_start(sigma, gam)
    for ite in range(1, 4):
        O.iteration(st, ite)
        sol2.iteration(ite)
    assert parity.rel(sol2.Sigma, st.Sigma) <= 1e-10
    sol.close()
    sol2.close()


def test_checkpoint_restore_replays_the_same_iterations(gpu_lib):
    from tups_b200 import Solver
    from tups_b200._lib import TupsError
    p = parity.to_solver_params(_case())
    sol = Solver(p)
    with pytest.raises(TupsError):
        sol.checkpoint(False)          # nothing stored yet
    for ite in range(2):
        sol.iteration(ite)
    sol.checkpoint(True)
    a = [sol.iteration(ite)["dsigma_inf"] for ite in range(2, 5)]
    sa, fa = sol.Sigma, sol.F(1)
    sol.checkpoint(False)
    b = [sol.iteration(ite)["dsigma_inf"] for ite in range(2, 5)]
    assert parity.rel(sol.Sigma, sa) <= 1e-14
    assert parity.rel(sol.F(1), fa) <= 1e-14
    np.testing.assert_allclose(a, b, rtol=1e-12)
    sol.close()


def test_run_warm_falls_back_on_a_bad_prediction(gpu_lib):
    from tups_b200 import warmstart as W
    p = parity.to_solver_params(_case())
    p.conv_abs = 1e-10
    cold = W.run_cold(p, max_iter=400)
    assert cold.converged

    def bad(params, sigma2):
        return sigma2 * 40.0, np.array([50.0, -50.0, 80.0, 9.0])

    def exact(params, sigma2):
        return cold.sigma, cold.gamma_l1

    fb = W.run_warm(p, bad, max_iter=400)
    assert fb.fallback and fb.converged
    assert fb.iterations <= cold.iterations + 1
    assert parity.rel(fb.sigma, cold.sigma) <= 1e-8
    # a kept warm start reaches the same fixed point
    kept = W.run_warm(p, exact, max_iter=400, accept=np.inf)
    assert kept.converged and not kept.fallback
    assert parity.rel(kept.sigma, cold.sigma) <= 1e-8


def test_sweep_trains_on_solver_runs_and_reports_the_gain(gpu_lib):
    """The whole learned warm start at a small size: seeded sweep, training by
    the library's kernels, warm vs cold on held-out runs.  Every warm run must
    reach the cold run's fixed point, and the fallback bounds the loss to one
    iteration per run on average."""
    from tups_b200 import Params
    from tups_b200 import warmstart as W
    base = Params(Nx=4, Nf=8, neighbours=1, f_damping=0.5, use_U2=True, ite_max=10 ** 6, conv_abs=1e-10)
    res = W.sweep(base, runs=36, n_train=28, seed=1, max_iter=1000, epochs=400, log=lambda *a: None)
    s = res["summary"]
    print("warm start sweep 4x4/Nl=1/Nf=8:", s)
    assert s["n_train"] >= 20 and s["n_test"] >= 6
    assert s["loss_last"] < 0.2 * s["loss_first"]
    assert s["all_warm_converged"]
    # the reference's mu bisection stops at |n - n0| < 1e-6 (parquet_chi.f90),
    # so two trajectories can settle on self-consistent mu values that differ
    # within that band: their fixed points agree to ~1e-6, not to 1e-10
    assert s["max_final_sigma_rel_diff"] <= 1e-4
    assert s["warm_iterations_mean"] <= s["cold_iterations_mean"] + 1.0


@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 1), (35, 33, 2, 17, 31), (260, 64, 1, 16, 33), (1030, 129, 2, 66, 65)],
                         ids=["one", "odd", "edge", "long"])
def test_mlp_layers_at_tile_edges(gpu_lib, shape):
    """Widths and batches around the 32 x 16 output tiles, the four k ranges of
    a cluster and its 256-wide k chunks, aligned and unaligned rows; one Adam
    step over a gathered minibatch against the float64 oracle."""
    from tups_b200.warmstart import MLP
    n_in, hidden, layers, n_out, batch = shape
    net = MLP(n_in, n_out, hidden, layers, max_batch=batch, seed=3)
    rng = np.random.default_rng(19)
    p = net.get_params()
    x = rng.normal(size=(batch, n_in)).astype(np.float32)
    t = rng.normal(size=(batch, n_out)).astype(np.float32)
    y_ref, _ = OW.mlp_forward(p, net.widths, x)
    # a sum of n FP32 products is off by at most about n eps of the sum of magnitudes
    tol = 4 * max(n_in, hidden) * 6e-8
    assert parity.rel(net.forward(x), y_ref) <= max(tol, 1e-6)
    loss, g = net.gradients(x, t)
    loss_ref, g_ref = OW.mlp_loss_grad(p, net.widths, x, t)
    assert abs(loss - loss_ref) <= MLP_TOL * loss_ref
    assert parity.rel(g, g_ref) <= MLP_TOL
    # the first Adam step moves a parameter by lr g / (|g| + eps): compared where |g| is far above rounding
    net.train(x, t, batch=batch, epochs=1, lr=1e-2, weight_decay=0.1, seed=5)
    layout, _ = OW.mlp_layout(net.widths)
    want = p.astype(np.float64)
    for wo, bo, fin, fout in layout:
        want[wo:bo] *= 1.0 - 1e-2 * 0.1
    want -= 1e-2 * g_ref / (np.abs(g_ref) + 1e-8)
    big = np.abs(g_ref) > 1e-3 * np.abs(g_ref).max()
    assert np.abs(net.get_params() - want)[big].max() <= 1e-2 * 2 * MLP_TOL / 1e-3
    net.close()


@pytest.mark.parametrize("shape", [(37, 65, 2, 66, 1023), (37, 65, 2, 66, 1024), (130, 64, 1, 3, 1089), (8, 129, 3, 64, 2047)],
                         ids=["below", "at", "narrow", "wide"])
def test_mlp_layers_of_large_batches(gpu_lib, shape):
    """Both sides of the row count from which a layer runs on whole 64 x 64 tiles, with remainders in rows, columns
    and depth: outputs, loss and gradients against the float64 oracle."""
    from tups_b200.warmstart import MLP
    n_in, hidden, layers, n_out, batch = shape
    net = MLP(n_in, n_out, hidden, layers, max_batch=batch, seed=4)
    rng = np.random.default_rng(23)
    p = net.get_params()
    x = rng.normal(size=(batch, n_in)).astype(np.float32)
    t = rng.normal(size=(batch, n_out)).astype(np.float32)
    y_ref, _ = OW.mlp_forward(p, net.widths, x)
    assert parity.rel(net.forward(x), y_ref) <= 4 * max(n_in, hidden) * 6e-8
    loss, g = net.gradients(x, t)
    loss_ref, g_ref = OW.mlp_loss_grad(p, net.widths, x, t)
    assert abs(loss - loss_ref) <= MLP_TOL * loss_ref
    assert parity.rel(g, g_ref) <= MLP_TOL
    # a training pass gathers its rows: one batch of all samples in some order
    hist = net.train(x, t, batch=batch, epochs=1, lr=1e-3, seed=5)
    assert abs(hist[0] - loss_ref) <= MLP_TOL * loss_ref
    net.close()


def test_mlp_batches_beyond_two_million_rows(gpu_lib):
    """More row tiles of 32 than the second grid dimension takes."""
    from tups_b200.warmstart import MLP
    batch = 32 * 65535 + 1
    net = MLP(1, 1, 1, 1, max_batch=batch, seed=4)
    x = np.linspace(-2.0, 2.0, batch, dtype=np.float32)[:, None]
    y_ref, _ = OW.mlp_forward(net.get_params(), net.widths, x)
    assert parity.rel(net.forward(x), y_ref) <= 1e-6
    net.close()


def test_mlp_training_with_a_nan_rate_shows(gpu_lib):
    """A NaN learning rate is not refused: the parameters turn NaN, they do not stay as if trained."""
    from tups_b200.warmstart import MLP
    net = MLP(3, 2, 4, 1, max_batch=8, seed=4)
    rng = np.random.default_rng(3)
    net.train(rng.normal(size=(8, 3)).astype(np.float32), rng.normal(size=(8, 2)).astype(np.float32), batch=8, epochs=1,
              lr=float("nan"))
    assert np.all(np.isnan(net.get_params()))
    net.close()


def test_mlp_adam_against_the_float64_steps(gpu_lib):
    """Three steps on one full batch against Adam in float64 with the oracle's gradients, weights and biases apart, a
    decay of 4 % per step on the weights alone.  Where |g| is within a factor 10 of its largest, a gradient is known
    to about 1e-5, so its step lr m / sqrt(v) to some 1e-4 of lr; a decay left out or laid on the biases would show
    as 400 times that."""
    from tups_b200.warmstart import MLP
    n_in, hidden, layers, n_out, batch, lr, wd = 20, 33, 2, 17, 32, 1e-2, 4.0
    net = MLP(n_in, n_out, hidden, layers, max_batch=batch, seed=6)
    rng = np.random.default_rng(29)
    layout, _ = OW.mlp_layout(net.widths)
    p = net.get_params()
    for _, bo, _, fout in layout:
        p[bo:bo + fout] = rng.normal(size=fout)
    net.set_params(p)
    p = p.astype(np.float64)
    x = rng.normal(size=(batch, n_in)).astype(np.float32)
    t = rng.normal(size=(batch, n_out)).astype(np.float32)
    weight = np.zeros(p.size, dtype=bool)
    for wo, bo, _, _ in layout:
        weight[wo:bo] = True
    b1, b2, eps, m, v = 0.9, 0.999, 1e-8, np.zeros_like(p), np.zeros_like(p)
    clear = np.ones(p.size, dtype=bool)
    for step in range(1, 4):
        _, g = OW.mlp_loss_grad(p, net.widths, x.astype(np.float64), t.astype(np.float64))
        for part in (weight, ~weight):
            clear &= ~part | (np.abs(g) > 0.1 * np.abs(g[part]).max())
        p[weight] *= 1.0 - lr * wd
        m, v = b1 * m + (1 - b1) * g, b2 * v + (1 - b2) * g * g
        p -= lr * (m / (1 - b1 ** step)) / (np.sqrt(v / (1 - b2 ** step)) + eps)
    net.train(x, t, batch=batch, epochs=3, lr=lr, weight_decay=wd, seed=5)
    got = net.get_params()
    for part in (weight, ~weight):
        assert np.count_nonzero(clear & part) >= 10
        assert np.abs(got - p)[clear & part].max() <= 3 * 1e-4 * lr + 6e-8 * np.abs(p).max()
    net.close()
