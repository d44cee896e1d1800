"""The device memory that process tensors keep between sweeps is bounded over
all of them, and given back with them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_kept_workspace_is_bounded_over_handles():
    from tests.test_sweep_gpu import build
    n, steps = 600, 30
    eye = np.tile(np.eye(4, dtype=complex), (n, 2, 1, 1))
    index = np.repeat(np.arange(n)[:, None], steps, axis=1)
    rho0 = np.tile(np.array([1.0, 0, 0, 0], dtype=complex), (n, 1))
    handles = [build(2, 0.02, 3, steps, 64) for _ in range(5)]
    want = handles[0].gradient_cores(0, eye[:8], index[:8], rho0[:8], rho0[:8], steps)[1]
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for b in handles:      # about 170 MB of workspace each
        got = b.gradient_cores(0, eye, index, rho0, rho0, steps)[1]
        np.testing.assert_array_equal(got[:8], want)
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept <= 272 * MB, kept / MB
    for b in handles:
        b.close()
    assert before - torch.cuda.mem_get_info()[0] <= 16 * MB
    again = build(2, 0.02, 3, steps, 64)       # the room is there again
    before = torch.cuda.mem_get_info()[0]
    again.gradient_cores(0, eye, index, rho0, rho0, steps)
    kept = before - torch.cuda.mem_get_info()[0]
    assert 64 * MB < kept <= 272 * MB, kept / MB
    again.close()
