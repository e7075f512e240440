"""Workloads of the framework for timing: the parquet loop over its range of
lattices, form factors and frequencies, the stand-alone Bethe-Salpeter
solvers, the split-precision ZGEMM and the warm-start network, each through
the entry points a program calls.

``listed()`` gives the named cases, ``draw(rng)`` further ones of the same
ranges; ``prepare(case, seed)`` makes inputs and handles, ``run(state)`` is
one pass, ``work(case)`` its compulsory bytes and flops, ``exact(case, seed)``
the 64-bit value of its outputs where plain torch gives one.

The loop cases have no ``exact``: their only 64-bit value is the whole loop
restated (form-factor tables, crossing tensors, frequency maps, spline), so
their FP64 outputs are compared between two builds instead.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from tups_b200 import Params, Solver, _lib
from tups_b200.bse_batched import Instances, LuBatch
from tups_b200.parquet import host_tables
from tups_b200.warmstart import MLP

CHANNELS = "dmst"
_LOOP = ("Nx", "Nf", "neighbours", "beta", "U", "nParticle", "tprime", "f_range", "Ngrain")


def _loop_case(kind, Nx, Nf, neighbours, beta, U, nParticle=1.0, tprime=0.0, f_range=0, Ngrain=1, **more):
    return {"kind": kind, "Nx": Nx, "Nf": Nf, "neighbours": neighbours, "beta": beta, "U": U,
            "nParticle": nParticle, "tprime": tprime, "f_range": f_range, "Ngrain": Ngrain, **more}


def listed() -> list[dict]:
    return [
        # the smallest run, start to end: 10 iterations of execute_loop from a stored
        # starting state, then the vertices read back as the final vertex output does
        {"name": "execute_4x4_nl1_nf16", **_loop_case("execute", 4, 16, 1, 2.0, 2.0, iterations=10)},
        # a doped run with next-nearest hopping, an extended frequency box and a refined
        # momentum grid, on a lattice and a frequency count that no tile divides, launched
        # kernel by kernel as Solver.iteration does by default
        {"name": "loop_6x6_nl5_nf22_doped",
         **_loop_case("loop", 6, 22, 2, 2.0, 2.0, 0.9, -0.2, 1, 2, graph=False, slices=0)},
        # the ordinary production size, replayed from a CUDA graph
        {"name": "loop_8x8_nl5_nf32", **_loop_case("loop", 8, 32, 2, 5.0, 2.0, graph=True, slices=0)},
        # nine form factors with the split-precision BSE at the slice count of early iterations
        {"name": "loop_8x8_nl9_nf32_split3", **_loop_case("loop", 8, 32, 3, 4.0, 2.0, graph=True, slices=3)},
        # the largest lattice of which several states fit one card side by side
        {"name": "loop_12x12_nl9_nf48",
         **_loop_case("loop", 12, 48, 3, 4.0, 2.0, 0.9, -0.2, graph=True, slices=0)},
        # an output iteration: the iteration with chi0 and the susceptibilities
        {"name": "readout_8x8_nl5_nf32", **_loop_case("readout", 8, 32, 2, 4.0, 2.0, 0.9, -0.2)},
        # the split ZGEMM alone at the matrix size of 9 form factors x 64 frequencies
        {"name": "zgemm_split_576_s6", "kind": "zgemm", "batch": 32, "M": 576, "N": 576, "K": 576, "slices": 6},
        # the BSE update on buffers of a caller that owns all device memory: one channel of 8x8 / Nl = 5
        {"name": "bse_noalloc_160x240", "kind": "noalloc", "n_inst": 240, "Nf": 32, "Nl": 5},
        # the LU form over bosonic instances whose form-factor counts vary (n = 64 .. 832)
        {"name": "lu_batch_96_nf64", "kind": "lu", "n_inst": 96, "Nf": 64},
        # the same form in split precision with FP64 refinement
        {"name": "lu_split_32_nf64_s5", "kind": "lu_split", "n_inst": 32, "Nf": 64, "slices": 5},
        # training the warm-start network: 8x8 / Nf = 32 features, 160 runs, minibatches of 32
        {"name": "mlp_train_964_b32", "kind": "mlp_train", "n_in": 964, "n_out": 968, "samples": 160, "batch": 32,
         "epochs": 4, "weight_decay": 1e-4},
        # predicting the held-out runs
        {"name": "mlp_forward_964_b40", "kind": "mlp_forward", "n_in": 964, "n_out": 968, "samples": 40},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["loop", "loop", "loop", "execute", "readout", "zgemm", "noalloc", "lu", "lu_split",
                       "mlp_train", "mlp_forward"])
    if kind in ("loop", "execute", "readout"):
        doped = rng.random() < 0.5
        nb = rng.choice([1, 2, 3])
        Nx = rng.choice([4, 6] if kind == "execute" else [4, 6, 8, 10])
        Nf = 2 * _log_int(rng, 4, 10 if kind == "execute" else 20)
        c = _loop_case(kind, Nx, Nf, nb, round(rng.uniform(1.0, 4.0), 3), round(rng.uniform(0.8, 2.0), 3),
                       round(rng.uniform(0.85, 0.95), 3) if doped else 1.0,
                       round(rng.uniform(-0.3, 0.0), 3) if doped else 0.0,
                       rng.choice([0, 0, 1]), rng.choice([1, 1, 2]))
        if kind == "execute":
            c["iterations"] = rng.randint(3, 10)
        if kind == "loop":
            c["graph"] = rng.random() < 0.5
            c["slices"] = rng.choice([0, 0, 0, 3, 5])
        return c
    if kind == "zgemm":
        return {"kind": kind, "batch": _log_int(rng, 1, 32), "M": _log_int(rng, 24, 576), "N": _log_int(rng, 24, 576),
                "K": _log_int(rng, 24, 576), "slices": rng.randint(2, 8)}
    if kind == "noalloc":
        return {"kind": kind, "n_inst": _log_int(rng, 6, 240), "Nf": 2 * _log_int(rng, 4, 20),
                "Nl": rng.choice([1, 5, 9])}
    if kind == "lu":
        return {"kind": kind, "n_inst": _log_int(rng, 4, 96), "Nf": _log_int(rng, 12, 64)}
    if kind == "lu_split":
        return {"kind": kind, "n_inst": _log_int(rng, 4, 32), "Nf": _log_int(rng, 12, 64), "slices": rng.randint(4, 7)}
    n = 2 * _log_int(rng, 30, 480)
    if kind == "mlp_train":
        return {"kind": kind, "n_in": n + 4, "n_out": n + 8, "samples": _log_int(rng, 20, 160),
                "batch": rng.choice([16, 32, 32]), "epochs": rng.randint(1, 4), "weight_decay": 1e-4}
    return {"kind": kind, "n_in": n + 4, "n_out": n + 8, "samples": _log_int(rng, 1, 200)}


# ---- inputs -------------------------------------------------------------------
def _params(case) -> Params:
    return Params(ite_max=case.get("iterations", 10 ** 6), f_damping=0.5, use_U2=True,
                  **{k: case[k] for k in _LOOP})


def _start_sigma(case, rng) -> np.ndarray:
    """A self-energy as a neighbouring run leaves it: U^2/4 over the Matsubara frequency with a
    momentum dependence of the lattice's symmetry, index ((kx-1) Ny + ky-1) Nf + nu."""
    nx, nf = case["Nx"], case["Nf"]
    k = 2.0 * math.pi / nx * np.arange(nx)
    cx, cy = np.cos(k)[:, None], np.cos(k)[None, :]
    a = rng.uniform(-0.2, 0.2, size=3)
    form = 1.0 + a[0] + a[1] * (cx + cy) + a[2] * cx * cy
    nu = math.pi / case["beta"] * (2.0 * (np.arange(nf) - nf // 2) + 1.0)
    tail = nu / (nu * nu + rng.uniform(0.5, 1.5))
    return (-0.25j * case["U"] ** 2 * form[:, :, None] * tail[None, None, :]).reshape(-1)


def _complex(g, *shape) -> torch.Tensor:
    return torch.randn(*shape, dtype=torch.complex128, generator=g, device="cuda")


def _chi_blocks(g, nl: int, nf: int, n_inst: int) -> torch.Tensor:
    """nu-diagonal bubbles, summed over the momenta of an 8x8 lattice: (n_inst, nu, l2, l1), falling
    as 1/nu^2, near diagonal in the form factors."""
    nu = 2.0 * (torch.arange(nf, device="cuda", dtype=torch.float64) - nf // 2) + 1.0
    fall = -64.0 / (nu * nu + 9.0)
    eye = torch.eye(nl, device="cuda", dtype=torch.complex128)
    return (eye + 0.2 * _complex(g, n_inst, nf, nl, nl)) * fall[None, :, None, None]


def _lu_sizes(case, seed) -> np.ndarray:
    # the counts of one workload are fixed: every seed has the same work
    return np.random.default_rng(12345).permutation(np.resize([1, 5, 9, 13], case["n_inst"]))


def _lu_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nf = case["Nf"]
    gam, chi = [], []
    for nl in _lu_sizes(case, seed):
        n = int(nl) * nf
        a = _complex(g, n, n)
        herm = 0.5 * (a + a.mH)
        c = _chi_blocks(g, int(nl), nf, 1)[0]
        # |Gamma chi| <= |Gamma| max|chi block| <= 0.9, |Gamma| about sqrt(2 n) here
        top = float(torch.linalg.matrix_norm(c, 2).max())
        gam.append(herm * (0.9 / (math.sqrt(2.0 * n) * 1.1 * top)))
        chi.append(c)
    return gam, chi


def _noalloc_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    nz = case["Nl"] * case["Nf"]
    gam, f = _complex(g, case["n_inst"], nz, nz), _complex(g, case["n_inst"], nz, nz)
    return gam, f, _chi_blocks(g, case["Nl"], case["Nf"], case["n_inst"])


_NOALLOC_SCALE, _NOALLOC_DAMP = 0.5 * 0.5 / (5.0 * 64.0), 0.5


def _zgemm_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    # column-major matrices: (batch, K, M) and (batch, N, K) tensors, over four decades in K as vertex columns are
    w = torch.logspace(-2, 2, case["K"], dtype=torch.float64, device="cuda")
    a = _complex(g, case["batch"], case["K"], case["M"]) * w[None, :, None]
    return a, _complex(g, case["batch"], case["N"], case["K"])


def _mlp_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n_in, n_out, s = case["n_in"], case["n_out"], case["samples"]
    latent = rng.standard_normal((s, 5))  # the five swept parameters decide a run
    x = np.tanh(latent @ rng.standard_normal((5, n_in)) / 2.0) + 0.1 * rng.standard_normal((s, n_in))
    t = np.tanh(latent @ rng.standard_normal((5, n_out)) / 2.0)
    return x.astype(np.float32), t.astype(np.float32)


_MLP_LR = 1e-3


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("loop", "execute", "readout"):
        sol = Solver(_params(case))
        rng = np.random.default_rng(seed)
        sol.Sigma = _start_sigma(case, rng)
        pinned = torch.empty(sol.Nt, dtype=torch.complex128, pin_memory=True).numpy()
        s.update(sol=sol, sigma=pinned)
        if kind == "execute":
            sol.checkpoint(True)
        else:
            sol.iteration(0)  # builds the crossing tensors
            if kind == "loop":
                sol.set_bse_precision(case["slices"])
                sol.set_graph(case["graph"])
            sol.iteration(1)  # captures the graph
            s["ite"] = 2
    elif kind in ("lu", "lu_split"):
        gam, chi = _lu_inputs(case, seed)
        nl = _lu_sizes(case, seed).astype(np.int32)
        inst = Instances(n=nl * np.int32(case["Nf"]), nl=nl, scale=np.ones(len(nl)),
                         gamma=[np.asfortranarray(x.cpu().numpy()) for x in gam],
                         chi=[x.cpu().numpy().transpose(2, 1, 0) for x in chi], q=np.zeros((len(nl), 3), np.int32))
        s.update(batch=LuBatch(inst), slices=case.get("slices"))
    elif kind == "noalloc":
        # one stored matrix is column-major: the tensor holds its transpose, and so do Gamma and F alike
        gam, f, chi = _noalloc_inputs(case, seed)
        s.update(lib=_lib.load(), gam=gam, f=f, chi=chi, n=case["n_inst"], nl=case["Nl"], nf=case["Nf"])
    elif kind == "zgemm":
        a, b = _zgemm_inputs(case, seed)
        lib, c = _lib.load(), torch.empty(case["batch"], case["N"], case["M"], dtype=torch.complex128, device="cuda")
        need = lib.tups_zgemm_split_workspace(case["batch"], case["M"], case["N"], case["K"], case["slices"])
        s.update(lib=lib, a=a, b=b, c=c, work=torch.empty(need, dtype=torch.uint8, device="cuda"),
                 dims=(case["batch"], case["M"], case["N"], case["K"]), slices=case["slices"])
    else:
        x, t = _mlp_inputs(case, seed)
        s.update(net=MLP(case["n_in"], case["n_out"], seed=seed), x=x, t=t)
        if kind == "mlp_train":
            s.update(batch=case["batch"], epochs=case["epochs"], wd=case["weight_decay"])
    return s


def _loop_outputs(s, info) -> dict:
    s["sol"].get_sigma_into(s["sigma"])
    out = {"Sigma": s["sigma"], "mu": info["mu"], "rel_sig_max": info["rel_sig_max"],
           "converged": info["converged"]}
    out.update({f"F_{r}_max": info[f"F_{r}_max"] for r in CHANNELS})
    return out


def run(s):
    kind = s["kind"]
    if kind == "loop":
        info = s["sol"].iteration(s["ite"])
        s["ite"] += 1
        return _loop_outputs(s, info)
    if kind == "execute":
        sol = s["sol"]
        sol.checkpoint(False)
        ite, converged = sol.execute_loop()
        sol.get_sigma_into(s["sigma"])
        return {"iterations": ite, "converged": converged, "Sigma": s["sigma"], "F": [sol.F(r) for r in CHANNELS],
                "G": [sol.G(r) for r in CHANNELS]}
    if kind == "readout":
        sol = s["sol"]
        s["ite"] += -s["ite"] % 5  # the next output iteration
        out = _loop_outputs(s, sol.iteration(s["ite"], readout=True))
        s["ite"] += 1
        out["chi0"] = sol.chi0(bz=True)
        out["sus"] = [sol.sus(r, bz=True) for r in CHANNELS]
        return out
    if kind == "lu":
        s["batch"].run()
        return s["batch"].out
    if kind == "lu_split":
        info = s["batch"].run_split(slices=s["slices"])
        # the residual reached is rounding below its tolerance; the solution and the steps taken are the result
        return {"F": s["batch"].out, "refinements": info["refinements"]}
    if kind == "noalloc":
        p = [C.c_void_p(s[k].data_ptr()) for k in ("gam", "f", "chi")]
        rc = s["lib"].tups_bse_noalloc(s["n"], s["nl"] * s["nf"], s["nf"], s["nl"], *p, _NOALLOC_SCALE,
                                       _NOALLOC_DAMP, C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise _lib.TupsError(rc, "tups_bse_noalloc failed")
        return s["gam"]
    if kind == "zgemm":
        p = [C.c_void_p(s[k].data_ptr()) for k in ("a", "b", "c")]
        rc = s["lib"].tups_zgemm_split(*s["dims"], *p, s["slices"], C.c_void_p(s["work"].data_ptr()),
                                       s["work"].numel(), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise _lib.TupsError(rc, "tups_zgemm_split failed")
        return s["c"]
    if kind == "mlp_train":
        hist = s["net"].train(s["x"], s["t"], batch=s["batch"], epochs=s["epochs"], lr=_MLP_LR, weight_decay=s["wd"],
                              seed=7)
        # losses of an FP32 network
        return {"loss": hist.astype(np.float32), "params": s["net"].get_params()}
    return s["net"].forward(s["x"])


# ---- compulsory work --------------------------------------------------------------
def _loop_work(case):
    d = host_tables(_params(case))["dims"]
    nz, nl, nb, nf, nr = d["Nz"], d["Nl"], d["Nb"], d["Nf"], d["NR"]
    vert = 16.0 * nz * nz * nb
    flops = 4 * nb * (16.0 * nz ** 3 + 16.0 * nz * nz * nl)  # BSE: one GEMM of depth 2 Nz, two block-diagonal products
    flops += 16.0 * nl ** 4 * nr * 2.8 * nb * nf * nf        # crossing: 2.8 of the 4 contributions fall into the box
    flops += 8.0 * 4 * nz * nz * (nf // 2) * nr * d["Nc"]     # Phi(q) -> Phi(R)
    byts = 16.0 * vert + 2.0 * 16.0 * d["Nt"]                # four F and four Gamma, read and written
    return byts, flops


def _mlp_flops(case, rows):
    w = [case["n_in"], 512, 512, 512, case["n_out"]]
    n = sum(a * b + b for a, b in zip(w[:-1], w[1:]))
    return n, 2.0 * rows * n


def work(case):
    kind = case["kind"]
    if kind in ("loop", "readout"):
        byts, flops = _loop_work(case)
    elif kind == "execute":
        byts, flops = (x * case["iterations"] for x in _loop_work(case))
    elif kind in ("lu", "lu_split"):
        n = _lu_sizes(case, 0).astype(np.float64) * case["Nf"]
        byts, flops = float(np.sum(32.0 * n ** 2)), float(np.sum((8.0 / 3.0 + 8.0) * n ** 3))
    elif kind == "noalloc":
        nz = case["Nl"] * case["Nf"]
        byts = 16.0 * case["n_inst"] * (3.0 * nz * nz + case["Nl"] * nz)
        flops = 16.0 * case["n_inst"] * (nz ** 3 + nz * nz * case["Nl"])
    elif kind == "zgemm":
        b, m, n, k = (case[x] for x in ("batch", "M", "N", "K"))
        byts, flops = 16.0 * b * (m * k + k * n + m * n), 8.0 * b * m * n * k
    elif kind == "mlp_train":
        n, f = _mlp_flops(case, case["samples"] * case["epochs"])
        steps = case["epochs"] * math.ceil(case["samples"] / case["batch"])
        # forward, two backward products; parameters and both moments read and written in every step
        byts, flops = 24.0 * n * steps, 3.0 * f
    else:
        n, flops = _mlp_flops(case, case["samples"])
        byts = 4.0 * (n + case["samples"] * (case["n_in"] + case["n_out"]))
    return {"bytes": byts, "flops": flops}


# ---- 64-bit values ------------------------------------------------------------------
def _dense_chi(c: torch.Tensor) -> torch.Tensor:
    """(nu, l2, l1) blocks of column-major (l1, l2, nu) storage -> dense chi[(l1, nu), (l2, nu)]"""
    nf, nl, _ = c.shape
    d = torch.zeros(nl, nf, nl, nf, dtype=c.dtype, device=c.device)
    i = torch.arange(nf, device=c.device)
    d[:, i, :, i] = c.permute(0, 2, 1)
    return d.reshape(nl * nf, nl * nf)


def _mlp_layers(case, seed):
    """The start parameters as MLP makes them: uniform weights within 1/sqrt(fan in), zero biases."""
    rng = np.random.default_rng(seed)
    w = [case["n_in"], 512, 512, 512, case["n_out"]]
    layers = []
    for a, b in zip(w[:-1], w[1:]):
        lim = 1.0 / np.sqrt(a)
        layers.append((rng.uniform(-lim, lim, a * b).astype(np.float32).reshape(b, a), np.zeros(b, np.float32)))
    return [torch.from_numpy(x).cuda().double() for pair in layers for x in pair]


def _mlp_apply(p, x):
    for i in range(0, len(p), 2):
        x = x @ p[i].T + p[i + 1]
        if i + 2 < len(p):
            x = x * torch.sigmoid(x)
    return x


def _shuffles(n: int, epochs: int, seed: int):
    """splitmix64-driven Fisher-Yates permutations, one after the other from one stream"""
    mask, state = (1 << 64) - 1, seed
    for _ in range(epochs):
        perm = list(range(n))
        for i in range(n - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = state
            z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            perm[i], perm[j] = perm[j], perm[i]
        yield perm


def _train_exact(case, seed):
    x, t = (torch.from_numpy(a).cuda().double() for a in _mlp_inputs(case, seed))
    p = _mlp_layers(case, seed)
    m, v = [torch.zeros_like(a) for a in p], [torch.zeros_like(a) for a in p]
    lr, wd, step, hist = float(np.float32(_MLP_LR)), case["weight_decay"], 0, []
    b1, b2, eps = (float(np.float32(a)) for a in (0.9, 0.999, 1e-8))
    batch = min(case["batch"], case["samples"])
    for perm in _shuffles(case["samples"], case["epochs"], 7):
        losses = []
        for r0 in range(0, case["samples"], batch):
            rows = torch.tensor(perm[r0:r0 + batch], device="cuda")
            q = [a.clone().requires_grad_() for a in p]
            loss = ((_mlp_apply(q, x[rows]) - t[rows]) ** 2).mean()
            grads = torch.autograd.grad(loss, q)
            losses.append(float(loss))
            step += 1
            c1, c2 = 1.0 - b1 ** step, 1.0 - b2 ** step
            for i, g in enumerate(grads):
                if i % 2 == 0:
                    p[i] = p[i] * (1.0 - lr * wd)
                m[i] = b1 * m[i] + (1.0 - b1) * g
                v[i] = b2 * v[i] + (1.0 - b2) * g * g
                p[i] = p[i] - lr * (m[i] / c1) / ((v[i] / c2).sqrt() + eps)
        hist.append(sum(losses) / len(losses))
    return {"loss": np.array(hist), "params": torch.cat([a.reshape(-1) for a in p])}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("lu", "lu_split"):
        gam, chi = _lu_inputs(case, seed)
        out = []
        for x, c in zip(gam, chi):
            a = torch.eye(x.shape[0], dtype=x.dtype, device="cuda") - x @ _dense_chi(c)
            out.append(torch.linalg.solve(a, x).T.reshape(-1))
        flat = torch.cat(out)
        return flat if kind == "lu" else {"F": flat, "refinements": None}
    if kind == "noalloc":
        gam, f, chi = _noalloc_inputs(case, seed)
        for i in range(case["n_inst"]):
            x, y, c = gam[i].T, f[i].T, _dense_chi(chi[i])
            gam[i] = (_NOALLOC_SCALE * (x @ c @ y + y @ c @ x) + (1.0 - _NOALLOC_DAMP) * (y - x)).T.clone()
        return gam
    if kind == "zgemm":
        a, b = _zgemm_inputs(case, seed)
        return torch.matmul(b, a)  # C^T = B^T A^T
    if kind == "mlp_train":
        return _train_exact(case, seed)
    if kind == "mlp_forward":
        x, _ = _mlp_inputs(case, seed)
        return _mlp_apply(_mlp_layers(case, seed), torch.from_numpy(x).cuda().double())
    return None
