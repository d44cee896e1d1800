"""The gradient sweeps (forward states, adjoint vectors, derivative cores)
against the same equations in numpy on the process tensor's own tensors
(oqupy/gradient.py:323-437): D = 4 and 9, one and several systems, clusters and
one CTA per system, bonds wide enough for partial sums, per-step propagators."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tests.test_sweep_gpu import CASES, build, numpy_sweep  # noqa: E402


@pytest.fixture(scope="module")
def tensors():
    return {c: build(*c, zeta=1.0 if c[0] == 2 else 3.0) for c in CASES}


def numpy_cores(b, steps, pairs, index, rho0, target):
    """core_n[a][m][e] = sum_lr v_n[l][a] T_n[l][r][m] Y_{n+1}[r][e] with v_n the
    state before step n and Y_n = P1_n^T T_n^T P2_n^T Y_{n+1}, Y_N the target."""
    T = [b.mpo_tensor(0, k) for k in range(steps)]
    D = rho0.shape[1]
    out = np.zeros((len(rho0), steps, D, D, D), dtype=complex)
    for h in range(len(rho0)):
        Y = target[h][None, :]
        back = [Y]
        for k in reversed(range(steps)):
            p1, p2 = pairs[index[h, k]]
            Y = np.einsum("lrb,rb->lb", T[k], Y @ p2) @ p1
            back.append(Y)
        back.reverse()
        v = rho0[h][None, :]
        for k in range(steps):
            p1, p2 = pairs[index[h, k]]
            out[h, k] = np.einsum("la,lrm,re->ame", v, T[k], back[k + 1])
            v = np.einsum("la,lra->ra", v @ p1.T, T[k]) @ p2.T
    return out


@pytest.mark.parametrize("case", CASES, ids=["wide", "narrow", "qutrit"])
@pytest.mark.parametrize("systems", [1, 7, 77, 153, 229])
def test_gradient_matches_numpy(tensors, case, systems):
    """Sums of at most ~100 terms over 14 steps in FP64 on both sides: 1e-12 of
    the largest value."""
    b = tensors[case]
    steps, D = case[3], case[0] ** 2
    rng = np.random.default_rng(systems)
    pairs = 0.4 * (rng.normal(size=(systems, 2, D, D)) + 1j * rng.normal(size=(systems, 2, D, D))) / np.sqrt(D) \
        + 0.8 * np.eye(D)
    index = rng.integers(0, systems, size=(systems, steps))
    rho0, target = (rng.normal(size=(systems, D)) + 1j * rng.normal(size=(systems, D)) for _ in range(2))
    check = np.unique(np.concatenate([[0, systems - 1], rng.integers(0, systems, 2)]))
    states, cores = b.gradient_cores(0, pairs, index, rho0, target, steps)
    want = numpy_sweep(b, steps, pairs, index[check], rho0[check])
    np.testing.assert_allclose(states[:, check], want, rtol=0, atol=1e-12 * max(1.0, np.abs(want).max()))
    want = numpy_cores(b, steps, pairs, index[check], rho0[check], target[check])
    np.testing.assert_allclose(cores[check], want, rtol=0, atol=1e-12 * max(1.0, np.abs(want).max()))
