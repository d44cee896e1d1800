"""One bond split against LAPACK, at the operands where it can go wrong: tied
singular values, columns far below the others, the ends of the FP64 range; and
the reciprocal square roots it is built on."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from tests import split_probe  # noqa: E402


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return split_probe.load(tmp_path_factory.mktemp("probe"))


def unitary(rng, n, k):
    q, _ = np.linalg.qr(rng.normal(size=(n, k)) + 1j * rng.normal(size=(n, k)))
    return q


EPS = {"complex128": 1.11e-16, "mixed": 3.6e-15}   # unit roundoff of the form


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
@pytest.mark.parametrize("decades", [0, 4, 8])
@pytest.mark.parametrize("R, N, rank", [(20, 8, 8), (20, 9, 9), (20, 10, 10), (24, 11, 11), (32, 12, 12), (30, 16, 16),
                                        (33, 32, 12), (60, 24, 24), (64, 40, 40), (90, 77, 30)])
def test_tied_pairs(lib, precision, decades, R, N, rank):
    """Exactly tied pairs of singular values, on both sides of the width from
    which complex128 rotations are applied as products, with and without the
    second QR.  Bound for singular values and for the reconstruction: 4 N^1.5
    unit roundoffs of the largest singular value (the Gram-Schmidt QR's
    backward error, which any later step may match: a small column is exact
    only to that already when the sweeps or products receive it)."""
    rng = np.random.default_rng(R * N + decades)
    s = 10.0 ** (-decades * (np.arange(rank) // 2) / max(1, rank // 2))
    A = (unitary(rng, R, rank) * s) @ unitary(rng, N, rank).conj().T
    want = np.linalg.svd(A, compute_uv=False)
    bound = 4 * N ** 1.5 * EPS[precision] * want[0]
    U, got, V, status = split_probe.split(lib, A, 1e-11, precision)
    assert status == 0 and len(got) == rank
    assert np.abs(got - want[:rank]).max() < bound
    assert np.linalg.norm(A - (U * got) @ V.conj().T, 2) < bound


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
@pytest.mark.parametrize("small", [1e-18, 1e-20, 3e-21, 1e-22, 1e-25])
@pytest.mark.parametrize("R, N, big", [(20, 9, 6), (24, 12, 8), (40, 24, 12), (40, 24, 21)])
def test_columns_whose_squares_leave_the_fp32_range(lib, precision, small, R, N, big):
    """A cut of the QR far below rounding keeps columns whose squared norms are
    denormal in FP32, where the hardware's estimates return infinity.  They
    may be kept or dropped; the others come out as if they were not there."""
    rng = np.random.default_rng(N)
    A = unitary(rng, R, N) * np.where(np.arange(N) < big, 1.0 + np.arange(N) / N, small)
    want = np.linalg.svd(A[:, :big], compute_uv=False)
    bound = 4 * N ** 1.5 * EPS[precision] * want[0]
    U, got, V, status = split_probe.split(lib, A, 1e-12, precision, qr_cut=1e-30)
    assert status == 0 and len(got) == big
    assert np.abs(got - want).max() < bound
    assert np.linalg.norm(A - (U * got) @ V.conj().T, 2) < bound


@pytest.mark.parametrize("N", [5, 12])
@pytest.mark.parametrize("scale", [1e-150, 1e150, 1.2e154])
def test_rank_decision_near_the_ends_of_the_fp64_range(lib, N, scale):
    """Squares of the single values fit in FP64, their sum need not."""
    rng = np.random.default_rng(N)
    s = np.where(np.arange(N) < N - 2, 1.0, 1e-6)
    A = (unitary(rng, 2 * N, N) * s) @ unitary(rng, N, N).conj().T * scale
    U, got, V, status = split_probe.split(lib, A, 1e-5)
    assert status == 0 and len(got) == N - 2
    np.testing.assert_allclose(got / scale, 1.0, rtol=0, atol=4 * N ** 1.5 * EPS["complex128"])


@pytest.mark.parametrize("N", [5, 12])
@pytest.mark.parametrize("value", [1e160, np.inf, np.nan])
def test_values_whose_squares_overflow_are_refused(lib, N, value):
    rng = np.random.default_rng(N)
    A = unitary(rng, 2 * N, N)
    A[3, 2] = value
    assert split_probe.split(lib, A, 1e-8)[3] == -6


def test_reciprocal_square_roots(lib):
    """Against 1 / sqrt in extended precision.  FP64: y + y (r / 2 + 3 r^2 / 8)
    with r = 1 - u y^2 for an FP32 estimate y (relative error below 2^-22,
    PTX's bound 2^-22.9 and the rounding of u): the terms left out are below
    5 r^3 / 16 < 2^-64, the correction's own roundings below 2^-73, and the
    final addition rounds once: 0.5 ulp + 2^-63, so 0.51 ulp.  Double-float: r
    from three FP32 roundings of at most 2^-46 each and the correction from
    four of 2^-24 of 2^-22: below 2^-44."""
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(1.0, 4.0, 200000), 2.0 ** rng.uniform(-80, 80, 200000),
                        1.0 + 2.0 ** -rng.uniform(1, 52, 50000)])
    d, f = split_probe.rsqrt(lib, x)
    want = 1 / np.sqrt(x.astype(np.longdouble))
    assert np.abs((d - want) / np.spacing(want.astype(np.float64))).max() < 0.51
    hi = x.astype(np.float32)
    ff = hi.astype(np.longdouble) + (x - hi).astype(np.float32)   # the double-float operand
    assert np.abs(f * np.sqrt(ff) - 1).max() < 2.0 ** -44
    # zero gives zero, NaN stays NaN; squares below the FP32 range keep FP64's accuracy
    d, f = split_probe.rsqrt(lib, np.array([0.0, np.nan]))
    assert d[0] == 0 and f[0] == 0 and np.isnan(d[1]) and np.isnan(f[1])
    t = 2.0 ** rng.uniform(-300, -126, 100000)
    d, _ = split_probe.rsqrt(lib, t)
    want = 1 / np.sqrt(t.astype(np.longdouble))
    assert np.abs((d - want) / np.spacing(want.astype(np.float64))).max() < 0.51
