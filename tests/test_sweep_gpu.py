"""The whole-sweep kernel against the sweep's equations in numpy on the process
tensor's own tensors and caps (oqupy/system_dynamics.py:131-165, 631-700), at
every launch shape: clusters (few systems on a wide bond), one system per CTA,
several per CTA, columns staged in shared memory or read in place, constant and
per-step propagators, D = 4 and 9."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def build(d, alpha, dkmax, steps, chi_cap, zeta=1.0):
    from oqupy_gb300 import bath
    from oqupy_gb300.pt import PtBatch
    op = np.diag([0.5, -0.5]) if d == 2 else np.diag([1.0, 0.0, -1.0])
    infl, _ = bath.influences(alpha, zeta, 3.0, "exponential", 0.5, 0.1, dkmax, op)
    b = PtBatch([dict(hs_dim=d, num_steps=steps, dkmax=dkmax, epsrel=1e-7, influences=infl[:min(steps, dkmax + 1)])],
                precision="mixed", chi_cap=chi_cap)
    b.build()
    return b


def numpy_sweep(b, steps, pairs, index, rho0):
    tensors = [b.mpo_tensor(0, k) for k in range(steps)]
    caps = [b.cap(0, k) for k in range(steps + 1)]
    out = np.zeros((steps + 1,) + rho0.shape, dtype=complex)
    for h in range(len(rho0)):
        v = rho0[h][None, :]
        out[0, h] = caps[0] @ v
        for k in range(steps):
            p1, p2 = pairs[index[h, k]]
            w = np.einsum("la,lra->ra", v @ p1.T, tensors[k])
            v = w @ p2.T
            out[k + 1, h] = caps[k + 1] @ v
    return out


CASES = [(2, 0.3, 9, 14, 128), (2, 0.05, 3, 9, 16), (3, 0.1, 3, 6, 64)]


@pytest.fixture(scope="module")
def tensors():
    return {c: build(*c, zeta=1.0 if c[0] == 2 else 3.0) for c in CASES}


@pytest.mark.parametrize("case", CASES, ids=["wide", "narrow", "qutrit"])
@pytest.mark.parametrize("systems", [1, 7, 153, 310, 700])
@pytest.mark.parametrize("per_step", [False, True])
def test_sweep_matches_numpy(tensors, case, systems, per_step):
    """Sums of at most ~100 terms per step over 14 steps in FP64 on both
    sides, states of order one: 1e-12."""
    b = tensors[case]
    steps, D = case[3], case[0] ** 2
    rng = np.random.default_rng(systems)
    pairs = 0.4 * (rng.normal(size=(systems, 2, D, D)) + 1j * rng.normal(size=(systems, 2, D, D))) / np.sqrt(D) \
        + 0.8 * np.eye(D)
    index = np.repeat(np.arange(systems)[:, None], steps, axis=1)
    if per_step:
        index = rng.integers(0, systems, size=(systems, steps))
    rho0 = rng.normal(size=(systems, D)) + 1j * rng.normal(size=(systems, D))
    check = np.unique(np.concatenate([[0, systems - 1], rng.integers(0, systems, 3)]))
    if per_step:
        got = b.dynamics_steps(0, pairs, index, rho0, steps)
    else:
        got = b.dynamics(0, pairs[:, 0], pairs[:, 1], rho0)
    want = numpy_sweep(b, steps, pairs, index[check], rho0[check])
    np.testing.assert_allclose(got[:, check], want, rtol=0, atol=1e-12 * max(1.0, np.abs(want).max()))


def test_sweeps_from_threads(tensors):
    """The kept workspace serves one call at a time; a second thread's call
    allocates its own."""
    from concurrent.futures import ThreadPoolExecutor
    b = tensors[CASES[1]]
    rng = np.random.default_rng(0)
    jobs = [(np.tile(np.eye(4), (n, 1, 1)) + 0.1 * rng.normal(size=(n, 4, 4)), rng.normal(size=(n, 4)))
            for n in (3, 200, 17, 90)]
    want = [b.dynamics(0, p, p, r) for p, r in jobs]
    with ThreadPoolExecutor(4) as ex:
        for _ in range(5):
            for g, w in zip(ex.map(lambda j: b.dynamics(0, j[0], j[0], j[1]), jobs), want):
                np.testing.assert_array_equal(g, w)
