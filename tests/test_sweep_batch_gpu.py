"""A system's states and derivative cores are the same bits alone and in any
batch: the order of every sum follows from the process tensor's bonds only."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tests.test_sweep_gpu import CASES, build  # noqa: E402

IDS = ["wide", "narrow", "qutrit"]


@pytest.fixture(scope="module")
def tensors():
    return {c: build(*c, zeta=1.0 if c[0] == 2 else 3.0) for c in CASES}


def inputs(D, n, seed=3):
    rng = np.random.default_rng(seed)
    pairs = 0.4 * (rng.normal(size=(n, 2, D, D)) + 1j * rng.normal(size=(n, 2, D, D))) / np.sqrt(D) + 0.8 * np.eye(D)
    return pairs, rng.normal(size=(n, D)) + 1j * rng.normal(size=(n, D)), \
        rng.normal(size=(n, D)) + 1j * rng.normal(size=(n, D))


@pytest.mark.parametrize("case", CASES, ids=IDS)
@pytest.mark.parametrize("per_step", [False, True])
def test_states_do_not_depend_on_the_batch(tensors, case, per_step):
    b, steps, D = tensors[case], case[3], case[0] ** 2
    pairs, rho0, _ = inputs(D, 1024)

    def run(first, n):
        p, r = pairs[first:first + n], rho0[first:first + n]
        if per_step:
            return b.dynamics_steps(0, p, np.repeat(np.arange(n)[:, None], steps, axis=1), r, steps)
        return b.dynamics(0, p[:, 0], p[:, 1], r)
    ref = run(0, 1024)
    for first, n in [(0, 1), (0, 2), (1, 9), (0, 19), (0, 37), (0, 76), (5, 77), (0, 152), (0, 153), (100, 400),
                     (3, 1021)]:
        np.testing.assert_array_equal(run(first, n), ref[:, first:first + n])


@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_gradients_do_not_depend_on_the_batch(tensors, case):
    b, steps, D = tensors[case], case[3], case[0] ** 2
    pairs, rho0, target = inputs(D, 200)

    def run(first, n):
        s = slice(first, first + n)
        return b.gradient_cores(0, pairs[s], np.repeat(np.arange(n)[:, None], steps, axis=1), rho0[s], target[s], steps)
    states, cores = run(0, 200)
    for first, n in [(0, 1), (0, 19), (7, 38), (0, 77), (0, 153)]:
        s, c = run(first, n)
        np.testing.assert_array_equal(s, states[:, first:first + n])
        np.testing.assert_array_equal(c, cores[first:first + n])
