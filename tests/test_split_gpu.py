"""The truncated bond split on the GPU at the shapes where it can go wrong:
rank-deficient operands (a bath of zero coupling leaves product states, so
every split has exactly zero columns), operands from below the width at which
they are orthogonalised by products up to the widest register form, and rounding
that must not depend on the launch shape or on the rest of the batch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SX = np.array([[0, 1], [1, 0]], dtype=complex)
SZ = np.diag([1.0, -1.0]).astype(complex)


def spin_boson(alpha, dkmax, epsrel, omega=1.3, eps=0.4, T=0.7):
    from oqupy_gb300 import bath
    infl, _ = bath.influences(alpha, 1.0, 5.0, "exponential", T, 0.1, dkmax, 0.5 * SZ)
    p1, p2 = bath.half_step_propagators(0.5 * omega * SX + 0.5 * eps * SZ, 0.1)
    return dict(hs_dim=2, dkmax=dkmax, epsrel=epsrel, influences=infl, prop1=p1, prop2=p2,
                rho0=np.diag([1.0, 0.0]).astype(complex))


def states(insts, steps, precision, **kw):
    from oqupy_gb300.tempo import TempoBatch
    b = TempoBatch(insts, precision=precision, chi_cap=64, out_cap=steps + 1, **kw)
    b.advance(steps)
    s = b.states(0, steps + 1)
    b.close()
    return s


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
@pytest.mark.parametrize("dkmax", [1, 5, 9])
def test_zero_coupling_is_the_free_evolution(precision, dkmax):
    """alpha = 0: rank-one splits.  The free evolution is exact; the tolerance
    is 20 steps' rounding (2^-48 and 2^-53 per operation, ~100 operations)."""
    inst = spin_boson(0.0, dkmax, 1e-8)
    got = states([inst], 20, precision)[0]
    u = inst["prop2"] @ inst["prop1"]
    v = inst["rho0"].reshape(-1)
    want = [v]
    for _ in range(20):
        v = u @ v
        want.append(v)
    np.testing.assert_allclose(got, np.array(want), atol=1e-13 if precision == "complex128" else 1e-11)


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
def test_rounding_is_independent_of_launch_shape_and_batch(precision):
    insts = [spin_boson(a, d, 1e-6) for a, d in [(0.1, 6), (0.4, 12), (0.25, 3)]]
    ref = states(insts, 16, precision)
    for kw in (dict(block=256, smem_kb=100), dict(block=128, smem_kb=48), dict(block=512, smem_kb=1),
               dict(block=64, smem_kb=16, grid=1)):
        np.testing.assert_array_equal(states(insts, 16, precision, **kw), ref)
    for i in range(3):
        np.testing.assert_array_equal(states([insts[i]], 16, precision)[0], ref[i])


def qutrit(dkmax, epsrel):
    from oqupy_gb300 import bath
    infl, _ = bath.influences(0.15, 3.0, 3.0, "exponential", 1.0, 0.05, dkmax, np.diag([1.0, 0.0, -1.0]))
    rng = np.random.default_rng(5)
    g = rng.normal(size=(3, 3)) + 1j * rng.normal(size=(3, 3))
    h = 0.5 * (g + g.conj().T)
    p1, p2 = bath.half_step_propagators(h / np.linalg.norm(h, 2), 0.05)
    return dict(hs_dim=3, dkmax=dkmax, epsrel=epsrel, influences=infl, prop1=p1, prop2=p2,
                rho0=np.diag([1.0, 0.0, 0.0]).astype(complex))


def check_against_oracle(inst, steps, precision, atol, **shape):
    from oracle import tempo_oracle as to
    infl = inst["influences"]
    want, _ = to.tempo_dynamics(inst["rho0"].reshape(-1), lambda dk: infl[dk] if 0 <= dk < len(infl) else None,
                                np.eye(inst["hs_dim"]), lambda s: (inst["prop1"], inst["prop2"]),
                                inst["dkmax"], inst["epsrel"], steps)
    from oqupy_gb300.tempo import TempoBatch
    b = TempoBatch([inst], precision=precision, chi_cap=128, out_cap=steps + 1, **shape)
    b.advance(steps)
    got = b.states(0, steps + 1)[0]
    b.close()
    np.testing.assert_allclose(got, want, rtol=0, atol=atol)


@pytest.mark.parametrize("shape", [dict(), dict(block=512, smem_kb=200), dict(block=256, smem_kb=8)])
@pytest.mark.parametrize("make, steps", [(lambda: spin_boson(0.05, 2, 1e-12), 12),   # narrow: up to 12 columns
                                         (lambda: spin_boson(0.3, 7, 1e-12), 12),
                                         (lambda: spin_boson(0.3, 7, 1e-12, eps=0.0), 12),   # symmetric: equal pairs
                                         (lambda: qutrit(4, 1e-12), 5)])
def test_complex128_split_matches_the_oracle(make, steps, shape):
    """Operands on either side of the width for the product form, with working
    matrices in shared and in global memory.  Both sides drop at most
    epsrel s_0 = 1e-12 per split, at most 16 splits a step: 192 splits and a
    factor of 2 for the two sides give 4e-10."""
    check_against_oracle(make(), steps, "complex128", 4e-10, **shape)


@pytest.mark.parametrize("make, steps", [(lambda: spin_boson(0.3, 7, 1e-9), 12),
                                         (lambda: spin_boson(0.3, 7, 1e-9, eps=0.0), 12),
                                         (lambda: qutrit(4, 1e-9), 5)])
def test_mixed_split_matches_the_oracle(make, steps):
    """As above with epsrel 1e-9: 4e-7."""
    check_against_oracle(make(), steps, "mixed", 4e-7)
