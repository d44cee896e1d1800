"""How many CTAs of the TEMPO kernel are resident: what the default launch
shapes say, read off the launch timeline (an instance's span is its CTA's)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SX = np.array([[0, 1], [1, 0]], dtype=complex)
SZ = np.diag([1.0, -1.0]).astype(complex)


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


def instance(dkmax=6):
    from oqupy_gb300 import bath
    infl, _ = bath.influences(0.2, 1.0, 5.0, "exponential", 0.7, 0.1, dkmax, 0.5 * SZ)
    p1, p2 = bath.half_step_propagators(0.65 * SX + 0.2 * SZ, 0.1)
    return dict(hs_dim=2, dkmax=dkmax, epsrel=1e-6, influences=infl, prop1=p1, prop2=p2,
                rho0=np.diag([1.0, 0.0]).astype(complex))


def resident(n, precision, launch=None, dkmax=6, **kw):
    """Largest number of instances in flight at one time."""
    from oqupy_gb300.tempo import TempoBatch
    b = TempoBatch([instance(dkmax)] * n, precision=precision, chi_cap=32, **kw)
    b.advance(8)
    if launch is not None:
        b.set_launch(**launch)
    b.advance(6)
    spans = b.timeline()
    b.check_status()
    b.close()
    events = sorted([(t, 1) for t in spans[:, 0]] + [(t, -1) for t in spans[:, 1]])
    return int(np.cumsum([e for _, e in events]).max())


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
def test_default_shape(precision):
    """One CTA per SM; two for more instances than SMs, all of short memory."""
    assert resident(3 * sms(), precision, dkmax=5) == 2 * sms()
    assert resident(3 * sms(), precision, dkmax=6) == sms()
    assert resident(sms(), precision, dkmax=5) == sms()


@pytest.mark.parametrize("precision", ["complex128", "mixed"])
@pytest.mark.parametrize("block, per_sm", [(128, 3), (160, 3), (192, 2), (256, 2), (288, 1), (512, 1)])
def test_default_grid_and_memory_of_a_given_block(precision, block, per_sm):
    """Without a grid or a shared-memory size, as many CTAs as fit, up to three."""
    n = 4 * sms()
    assert resident(n, precision, block=block) == per_sm * sms()
    assert resident(n, precision, launch=dict(block=block)) == per_sm * sms()


def test_given_sizes_are_kept():
    n = 4 * sms()
    assert resident(n, "mixed", block=256, smem_kb=56) == 2 * sms()
    assert resident(n, "mixed", block=256, smem_kb=200) == sms()
    assert resident(n, "mixed", block=128, smem_kb=48, grid=17) == 17
    assert resident(n, "mixed", launch=dict(block=128, smem_kb=48, grid=17)) == 17
