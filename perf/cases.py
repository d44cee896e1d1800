"""Performance cases of the batched TEMPO / PT-TEMPO engine and its surrogate.

Each case is one call sequence that a user's program makes through the
public entry points, on inputs drawn from a seed:

* ``backend``   one trajectory through the drop-in ``GpuTempoBackend``, step
                by step (what ``Tempo.compute`` does): latency of one instance.
* ``screen``    a parameter sweep of spin-boson trajectories in the mixed form
                with short memory, stored in single precision as the
                surrogate's training set stores it.
* ``tempo``     a ``TempoBatch`` advanced from its initial states and read
                back: either precision form, two- and three-level systems,
                memory longer than the run or shorter, tolerances of a
                converged calculation.
* ``pt``        process tensors built together (``PtBatch.build``) and the
                dynamics of a few Hamiltonians on each of them.
* ``sweep``     the dynamics of many systems on one process tensor that the
                program keeps (constant or time-dependent propagators).
* ``gradient``  forward and adjoint sweeps of the gradient on a kept process
                tensor.
* ``infer``     the surrogate network evaluated on a batch of points.
* ``train``     one optimiser step of the surrogate network.

The spin-boson distribution (alpha, omega_c, T, Omega, bias; sigma_z / 2
coupling; dt 0.05), the super-ohmic qutrit distribution, the process-tensor
model (omega_c 5, T 1, dt 0.02) and the network shape are those of the
benchmark and of the surrogate's defaults.  Below about 1e-10 relative
tolerance, a TEMPO step's result hardly depends on which vector of an exactly
degenerate pair a truncation keeps; at 1e-6 it does (by about that much), so
the sweeps at 1e-6 hand over single-precision trajectories.
"""

import math
import random

import numpy as np
import torch

from oqupy_gb300 import bath
from oqupy_gb300.pt import PtBatch
from oqupy_gb300.surrogate import BOX, KEYS, Mlp, tempo_bloch
from oqupy_gb300.tempo import GpuTempoBackend, TempoBatch

_SX = np.array([[0, 1], [1, 0]], dtype=complex)
_SZ = np.diag([1.0, -1.0]).astype(complex)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one trajectory at a converged tolerance, step by step
        dict(name="backend_c128", kind="backend", precision="complex128", dkmax=11, steps=10, epsrel=1e-11,
             chi_cap=160),
        # the surrogate's training data: a chunk of the parameter sweep
        dict(name="screen_mixed", kind="screen", n=253, dkmax=8, steps=40, epsrel=1e-6, chi_cap=64),
        # batches at converged tolerances: short memory, memory longer than the run
        dict(name="tempo_mixed", kind="tempo", precision="mixed", d=2, n=95, dkmax=20, steps=12, epsrel=1e-10,
             chi_cap=160),
        dict(name="tempo_c128", kind="tempo", precision="complex128", d=2, n=48, dkmax=8, steps=12, epsrel=1e-10,
             chi_cap=128),
        # three-level systems: 9 Liouville states, wide splits
        dict(name="tempo_qutrit", kind="tempo", precision="complex128", d=3, n=16, dkmax=6, steps=5, epsrel=1e-10,
             chi_cap=128),
        # process tensors: a batch in the mixed form, a few in complex128
        dict(name="pt_mixed", kind="pt", precision="mixed", n=24, dkmax=10, steps=24, epsrel=1e-6, chi_cap=96,
             systems=4),
        dict(name="pt_c128", kind="pt", precision="complex128", n=3, dkmax=8, steps=17, epsrel=1e-6, chi_cap=96,
             systems=3),
        # a few and many systems on one process tensor
        dict(name="sweep_few", kind="sweep", dkmax=8, steps=60, epsrel=1e-6, chi_cap=96, systems=8, per_step=False),
        dict(name="sweep_many", kind="sweep", dkmax=8, steps=60, epsrel=1e-6, chi_cap=96, systems=1024,
             per_step=False),
        # the gradient of driven systems: forward and adjoint sweeps, derivative cores
        dict(name="gradient", kind="gradient", dkmax=8, steps=60, epsrel=1e-6, chi_cap=96, systems=24, per_step=True),
        # the network on a large screening batch, and one training step
        dict(name="infer_large", kind="infer", batch=60001, hidden=512, layers=4, outputs=1500),
        dict(name="train_step", kind="train", batch=256, hidden=512, layers=4, outputs=1500),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["backend", "screen", "tempo", "tempo", "qutrit", "pt", "sweep", "gradient", "infer", "train"])
    if kind == "backend":
        return dict(kind="backend", precision=rng.choice(["complex128", "mixed"]), dkmax=rng.randint(4, 11),
                    steps=rng.randint(4, 10), epsrel=10.0 ** rng.uniform(-11.5, -10.7), chi_cap=160)
    if kind == "screen":
        return dict(kind="screen", n=_log_int(rng, 3, 256), dkmax=rng.randint(3, 8), steps=rng.randint(10, 40),
                    epsrel=10.0 ** rng.uniform(-7.0, -6.0), chi_cap=64)
    if kind == "tempo":
        return dict(kind="tempo", precision=rng.choice(["complex128", "mixed"]), d=2, n=_log_int(rng, 2, 48),
                    dkmax=rng.randint(4, 20), steps=rng.randint(6, 11), epsrel=10.0 ** rng.uniform(-11.0, -10.0),
                    chi_cap=128)
    if kind == "qutrit":
        return dict(kind="tempo", precision="complex128", d=3, n=_log_int(rng, 2, 16), dkmax=rng.randint(3, 6),
                    steps=rng.randint(3, 5), epsrel=10.0 ** rng.uniform(-10.5, -10.0), chi_cap=128)
    if kind == "pt":
        precision = rng.choice(["complex128", "mixed"])
        big = precision == "mixed"
        return dict(kind="pt", precision=precision, n=_log_int(rng, 1, 24 if big else 3),
                    dkmax=rng.randint(3, 10 if big else 8), steps=rng.randint(12, 24 if big else 17),
                    epsrel=10.0 ** rng.uniform(-6.0, -5.0), chi_cap=96, systems=rng.randint(1, 4))
    if kind in ("sweep", "gradient"):
        return dict(kind=kind, dkmax=rng.randint(3, 8), steps=rng.randint(20, 60), epsrel=10.0 ** rng.uniform(-6.0, -5.0),
                    chi_cap=96, systems=_log_int(rng, 1, 1024 if kind == "sweep" else 64),
                    per_step=rng.random() < 0.5)
    if kind == "infer":
        return dict(kind="infer", batch=_log_int(rng, 1, 60000), hidden=rng.choice([192, 256, 512, 500]),
                    layers=rng.randint(2, 4), outputs=rng.choice([150, 300, 750, 1500]))
    return dict(kind="train", batch=_log_int(rng, 32, 1024), hidden=rng.choice([192, 256, 512, 500]),
                layers=rng.randint(2, 4), outputs=rng.choice([150, 300, 750, 1500]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _box_points(n, seed):
    rng = np.random.default_rng(seed)
    return np.stack([rng.uniform(*BOX[k], size=n) for k in KEYS], axis=1)


def _spin_boson(n, seed, dkmax, epsrel):
    """Spin-boson instances as plain arrays (sigma_z / 2 coupling)."""
    out = []
    for a, wc, T, om, ep in _box_points(n, seed):
        infl, _ = bath.influences(a, 1.0, wc, "exponential", T, 0.05, dkmax, 0.5 * _SZ)
        p1, p2 = bath.half_step_propagators(0.5 * om * _SX + 0.5 * ep * _SZ, 0.05)
        out.append(dict(hs_dim=2, dkmax=dkmax, epsrel=epsrel, influences=infl, prop1=p1, prop2=p2,
                        rho0=np.diag([1.0, 0.0]).astype(complex)))
    return out


def _qutrits(n, seed, dkmax, epsrel):
    """Super-ohmic three-level instances with a seeded GUE Hamiltonian."""
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(n):
        a, T = rng.uniform(0.05, 0.2), rng.uniform(0.0, 2.0)
        g = rng.normal(size=(3, 3)) + 1j * rng.normal(size=(3, 3))
        h = 0.5 * (g + g.conj().T)
        h /= np.linalg.norm(h, 2)
        infl, _ = bath.influences(a, 3.0, 3.0, "exponential", T, 0.05, dkmax, np.diag([1.0, 0.0, -1.0]))
        p1, p2 = bath.half_step_propagators(h, 0.05)
        out.append(dict(hs_dim=3, dkmax=dkmax, epsrel=epsrel, influences=infl, prop1=p1, prop2=p2,
                        rho0=np.diag([1.0, 0.0, 0.0]).astype(complex)))
    return out


def _tempo_instances(case, seed):
    make = _spin_boson if case["d"] == 2 else _qutrits
    return make(case["n"], seed, case["dkmax"], case["epsrel"])


def _pt_instances(case, seed, n):
    """Process-tensor inputs: alpha ~ 0.1 U[0.8, 1], omega_c 5, T 1, dt 0.02."""
    rng = np.random.default_rng(seed)
    steps, dkmax = case["steps"], case["dkmax"]
    out = []
    for _ in range(n):
        infl, _ = bath.influences(0.1 * rng.uniform(0.8, 1.0), 1.0, 5.0, "exponential", 1.0, 0.02, dkmax, 0.5 * _SZ)
        out.append(dict(hs_dim=2, num_steps=steps, dkmax=dkmax, epsrel=case["epsrel"],
                        influences=infl[:min(steps, dkmax + 1)]))
    return out


def _pairs(n, seed):
    """Half-step propagator pairs ``[n, 2, 4, 4]`` of Hamiltonians a sx + b sz."""
    rng = np.random.default_rng(seed + 1)
    return np.array([bath.half_step_propagators(a * _SX + b * _SZ, 0.02)
                     for a, b in rng.uniform(-2.0, 2.0, size=(n, 2))])


def _up(n):
    return np.tile(np.array([1, 0, 0, 0], dtype=complex), (n, 1))


def _sweep_inputs(case, seed):
    """Propagator table, index ``[systems, steps]`` and initial states."""
    H, steps = case["systems"], case["steps"]
    pairs = _pairs(H, seed)
    if not case["per_step"]:
        index = np.repeat(np.arange(H, dtype=np.int32)[:, None], steps, axis=1)
    else:  # driven systems: every step takes another pair of the table
        index = np.random.default_rng(seed + 2).integers(0, H, size=(H, steps)).astype(np.int32)
    return pairs, index, _up(H)


def _targets(H, seed):
    rng = np.random.default_rng(seed + 3)
    return rng.normal(size=(H, 4)) + 1j * rng.normal(size=(H, 4))


def _sizes(case):
    return [5] + [case["hidden"]] * case["layers"] + [case["outputs"]]


def _net_inputs(case, seed, device):
    g = torch.Generator(device=device).manual_seed(seed + 1)
    X = 2.0 * torch.rand(case["batch"], 5, generator=g, device=device) - 1.0
    T = 0.3 * torch.randn(case["batch"], case["outputs"], generator=g, device=device) if case["kind"] == "train" else None
    return X, T


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": dict(case)}
    if kind == "backend":
        state["inst"] = _spin_boson(1, seed, case["dkmax"], case["epsrel"])[0]
    elif kind == "screen":
        state["points"] = _box_points(case["n"], seed)
    elif kind == "tempo":
        state["insts"] = _tempo_instances(case, seed)
    elif kind == "pt":
        state["insts"] = _pt_instances(case, seed, case["n"])
        state["pairs"] = _pairs(case["systems"], seed)
    elif kind in ("sweep", "gradient"):
        pt = PtBatch(_pt_instances(case, seed, 1), precision="mixed", chi_cap=case["chi_cap"])
        pt.build()
        state["pt"] = pt
        state["pairs"], state["index"], state["rho0"] = _sweep_inputs(case, seed)
        state["target"] = _targets(case["systems"], seed)
    else:
        state["net"] = Mlp(_sizes(case), seed=seed)
        state["X"], state["T"] = _net_inputs(case, seed, "cuda")
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "backend":
        inst = state["inst"]
        infl, D = inst["influences"], 4
        be = GpuTempoBackend(inst["rho0"], lambda dk: infl[dk] if 0 <= dk < len(infl) else None, np.identity(2),
                             lambda step: (inst["prop1"], inst["prop2"]), np.ones(D), np.ones(D), c["dkmax"],
                             c["epsrel"], config={"precision": c["precision"], "chi_cap": c["chi_cap"]})
        states = [be.initialize()[1]]
        for _ in range(c["steps"]):
            states.append(be.compute_step()[1])
        return np.array(states)
    if kind == "screen":
        traj, _ = tempo_bloch(state["points"], c["steps"], dkmax=c["dkmax"], epsrel=c["epsrel"], chi_cap=c["chi_cap"])
        return torch.tensor(traj.reshape(len(traj), -1), dtype=torch.float32, device="cuda")
    if kind == "tempo":
        batch = TempoBatch(state["insts"], precision=c["precision"], chi_cap=c["chi_cap"], out_cap=c["steps"] + 1)
        batch.advance(c["steps"])
        states = batch.states(0, c["steps"] + 1)
        batch.close()
        return states
    if kind == "pt":
        pt = PtBatch(state["insts"], precision=c["precision"], chi_cap=c["chi_cap"])
        pt.build()
        p, rho0 = state["pairs"], _up(c["systems"])
        states = [pt.dynamics(i, p[:, 0], p[:, 1], rho0) for i in range(c["n"])]
        pt.close()
        return np.array(states)
    if kind == "sweep":
        p = state["pairs"]
        if c["per_step"]:
            return state["pt"].dynamics_steps(0, p, state["index"], state["rho0"], c["steps"])
        return state["pt"].dynamics(0, p[:, 0], p[:, 1], state["rho0"])
    if kind == "gradient":
        states, cores = state["pt"].gradient_cores(0, state["pairs"], state["index"], state["rho0"], state["target"],
                                                   c["steps"])
        return {"states": states, "cores": cores}
    net = state["net"]
    if kind == "infer":
        return net.forward(state["X"])
    loss, gW, gb = net.loss_and_grads(state["X"], state["T"])
    net.step(gW, gb, lr=1e-3)
    return {"loss": loss, "gW": gW, "gb": gb, "W": net.W, "b": net.b}


# ---------------------------------------------------------------------------
# work and exact values
# ---------------------------------------------------------------------------

def _split_flops(R, N):
    """Real operations of a truncated complex SVD of R x N (Golub-Van Loan)."""
    return 4.0 * (6.0 * R * N * N + 20.0 * N ** 3)


def _bond(case):
    """Typical bond dimension of the case's chain, for the operation count."""
    digits = -math.log10(case["epsrel"])
    full = 4.0 if case.get("d", 2) == 3 else 2.4
    return min(full * digits, 0.5 * case["chi_cap"])


def work(case):
    kind = case["kind"]
    if kind in ("backend", "screen", "tempo"):
        n, D = case.get("n", 1), case.get("d", 2) ** 2
        steps, K = case["steps"], case["dkmax"] + 1
        sites = sum(min(s, K) for s in range(1, steps + 1))
        chi = _bond(case)
        # two splits per site and step: the zip-up's D chi x D chi / 2, the sweep's D chi x chi
        flops = n * sites * (_split_flops(D * chi, 0.5 * D * chi) + _split_flops(D * chi, chi) + 16.0 * (D * chi) ** 2 * chi)
        return {"bytes": n * 16.0 * (K * D * D + 2 * D * D + D * (steps + 2)), "flops": flops}
    if kind == "pt":
        n, D, steps = case["n"], 4, case["steps"]
        chi = _bond(case)
        splits = steps * (min(steps, case["dkmax"] + 1) + 0.5 * steps)
        return {"bytes": n * 16.0 * ((case["dkmax"] + 1) * D * D + (steps + 1) * case["systems"] * D),
                "flops": n * splits * (_split_flops(D * chi, chi) + 16.0 * D * chi ** 3)}
    if kind in ("sweep", "gradient"):
        H, steps, D = case["systems"], case["steps"], 4
        chi = _bond(case)
        flops = 8.0 * H * steps * (D * chi * chi + 2 * D * D * chi)
        moved = 16.0 * (steps * chi * chi * D + H * 2 * D * D + (steps + 1) * H * D)
        if kind == "gradient":
            flops = 2 * flops + 8.0 * H * steps * (D * D * chi * chi + D ** 3 * chi)
            moved += 16.0 * H * steps * D ** 3
        return {"bytes": moved, "flops": flops}
    sizes, B = _sizes(case), case["batch"]
    weights = sum(a * b for a, b in zip(sizes[:-1], sizes[1:]))
    if kind == "infer":
        return {"bytes": 2.0 * weights + 4.0 * B * (sizes[0] + sizes[-1]), "flops": 2.0 * B * weights}
    # forward, weight gradients, input gradients; master weights and moments read and written
    return {"bytes": 28.0 * weights + 4.0 * B * (sizes[0] + 2 * sizes[-1]),
            "flops": 2.0 * B * (3 * weights - sizes[0] * sizes[1])}


def _path_sum(infl, p1, p2, rho0, steps, device):
    """The trajectory without any truncation: the sum over all paths of the
    memory window, in complex128.  States ``[steps + 1, D]``."""
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.complex128, device=device)  # noqa: E731
    infl, p1, p2, v = t(infl), t(p1), t(p2), t(np.asarray(rho0).reshape(-1))
    D, window = v.numel(), infl.shape[0]
    between = p1 @ p2
    out = [v]
    A = (p1 @ v)[None, :]          # [older indices, newest index]
    K = 1
    for s in range(1, steps + 1):
        if s > 1:
            A = (A[:, :, None] * between.T[None]).reshape(-1, D)
            K += 1
            if K > min(s, window):
                A = A.reshape(D, -1, D).sum(0)
                K -= 1
        for k in range(K - 1):
            A = (A.reshape(D ** k, D, -1, D) * infl[K - 1 - k][None, :, None, :]).reshape(-1, D)
        A = A * torch.diagonal(infl[0])[None, :]
        out.append(p2 @ A.sum(0))
    return torch.stack(out)


def _driven_path_sum(infl, pairs, rho0, target, device):
    """The same for one propagator pair per step, ``pairs[n] = (P1, P2)``,
    and, with a target, the derivative of target . rho(N) with respect to
    every step's ``X[a, m, e] = P1[m, a] P2[e, m]``: ``(states, cores)``."""
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.complex128, device=device)  # noqa: E731
    infl, pairs, v = t(infl), t(pairs), t(np.asarray(rho0).reshape(-1))
    D, window = v.numel(), infl.shape[0]
    X = [(p[0].T[:, :, None] * p[1].T[None]).requires_grad_(target is not None) for p in pairs]
    out, K = [v], 0
    A = v[None, :]                 # [indices inside the memory, open leg]
    for x in X:
        if K == window:            # the oldest index leaves the memory
            A = A.reshape(D, -1, D).sum(0)
            K -= 1
        A = torch.einsum("ha,ame->hme", A, x)
        for k in range(K):
            A = (A.reshape(D ** k, D, -1, D, D) * infl[K - k][None, :, None, :, None]).reshape(-1, D, D)
        A = (A * torch.diagonal(infl[0])[None, :, None]).reshape(-1, D)
        K += 1
        out.append(A.sum(0))
    cores = None
    if target is not None:
        f = (t(target) * out[-1]).sum()
        cores = torch.stack([g.conj() for g in torch.autograd.grad(f.real, X)])
    return torch.stack(out).detach(), cores


def _exact_net(case, seed, device):
    sizes = _sizes(case)
    g = torch.Generator(device="cpu").manual_seed(seed)
    W = []
    for fin, fout in zip(sizes[:-1], sizes[1:]):
        w = torch.randn(fout, fin, generator=g) * (2.0 / fin) ** 0.5
        W.append(w.to(device).double())
    b = [torch.zeros(w.shape[0], dtype=torch.float64, device=device) for w in W]
    return W, b


def _forward(W, b, X):
    H = X
    for l, (w, c) in enumerate(zip(W, b)):
        H = H @ w.T + c
        if l < len(W) - 1:
            H = torch.nn.functional.gelu(H)
    return H


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind in ("backend", "screen", "tempo"):
        if kind == "tempo":
            insts = _tempo_instances(case, seed)
        elif kind == "backend":
            insts = _spin_boson(1, seed, case["dkmax"], case["epsrel"])
        else:
            insts = _spin_boson(case["n"], seed, case["dkmax"], case["epsrel"])
        states = torch.stack([_path_sum(i["influences"], i["prop1"], i["prop2"], i["rho0"], case["steps"], device)
                              for i in insts])
        if kind == "backend":
            return states[0].cpu().numpy()
        if kind == "tempo":
            return states.cpu().numpy()
        s = states[:, 1:]
        bloch = torch.stack([2 * s[..., 1].real, -2 * s[..., 1].imag, (s[..., 0] - s[..., 3]).real], dim=1)
        return bloch.reshape(len(insts), -1)
    if kind == "pt":
        pairs = _pairs(case["systems"], seed)
        up = _up(1)[0]
        return np.array([torch.stack([_path_sum(i["influences"], p[0], p[1], up, case["steps"], device)
                                      for p in pairs], dim=1).cpu().numpy() for i in _pt_instances(case, seed, case["n"])])
    if kind in ("sweep", "gradient"):
        infl = _pt_instances(case, seed, 1)[0]["influences"]
        pairs, index, rho0 = _sweep_inputs(case, seed)
        if kind == "sweep" and not case["per_step"]:
            return torch.stack([_path_sum(infl, p[0], p[1], r, case["steps"], device)
                                for p, r in zip(pairs, rho0)], dim=1).cpu().numpy()
        targets = _targets(case["systems"], seed) if kind == "gradient" else [None] * case["systems"]
        got = [_driven_path_sum(infl, pairs[i], r, t, device) for i, r, t in zip(index, rho0, targets)]
        states = torch.stack([g[0] for g in got], dim=1).cpu().numpy()
        if kind == "sweep":
            return states
        return {"states": states, "cores": torch.stack([g[1] for g in got]).cpu().numpy()}
    W, b = _exact_net(case, seed, device)
    X, T = _net_inputs(case, seed, device)
    X = X.double()
    if kind == "infer":
        return _forward(W, b, X)
    params = [p.requires_grad_(True) for p in W + b]
    err = _forward(W, b, X) - T.double()
    loss = (err * err).sum()
    grads = torch.autograd.grad(loss / err.numel(), params)
    n, lr = len(W), 1e-3
    new = [(p - lr * g / (g.abs() + 1e-8)).detach() for p, g in zip(params, grads)]   # AdamW's first step
    return {"loss": loss.detach()[None], "gW": list(grads[:n]), "gb": list(grads[n:]), "W": new[:n], "b": new[n:]}
