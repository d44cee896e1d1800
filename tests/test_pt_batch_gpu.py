"""Process-tensor builds of more instances than SMs: two CTAs share an SM, and an
instance's tensors are the same bits in a batch and alone."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def instances(n, dkmax, steps):
    from oqupy_gb300 import bath
    infl, _ = bath.influences(0.1, 1.0, 5.0, "exponential", 1.0, 0.02, dkmax, np.diag([0.5, -0.5]))
    return [dict(hs_dim=2, num_steps=steps, dkmax=dkmax, epsrel=1e-6, influences=infl[:dkmax + 1])] * n


def built(n, precision, dkmax=8, steps=16):
    """The built batch and its build time in ms."""
    from oqupy_gb300.pt import PtBatch
    b = PtBatch(instances(n, dkmax, steps), precision=precision, chi_cap=64)
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    start.record()
    b.advance(steps)
    stop.record()
    torch.cuda.synchronize()
    b.check_status()
    return b, start.elapsed_time(stop)


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
def test_two_builds_share_an_sm(precision):
    """One after the other, two equal builds on every SM would take twice as long
    as one."""
    def best(n):
        times = []
        for _ in range(4):
            b, ms = built(n, precision)
            b.close()
            times.append(ms)
        return min(times)
    one, two = best(sms()), best(2 * sms())
    assert two < 1.9 * one, (one, two)


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
def test_tensors_do_not_depend_on_the_batch(precision):
    alone, _ = built(1, precision)
    batch, _ = built(sms() + 1, precision)
    for i in (0, sms()):
        np.testing.assert_array_equal(batch.bond_dimensions(i), alone.bond_dimensions(0))
        for k in range(16):
            np.testing.assert_array_equal(batch.mpo_tensor(i, k), alone.mpo_tensor(0, k))
            np.testing.assert_array_equal(batch.cap(i, k), alone.cap(0, k))
    alone.close()
    batch.close()
