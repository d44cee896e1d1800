"""The network entry points on flat arrays (column sums, transposition,
conversion, mean-squared-error gradient, AdamW of one tensor) against torch in
64 bits on the same inputs."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture
def lib():
    from oqupy_gb300 import _native as nat
    return nat


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 5000])
def test_mse_gradient(lib, n):
    """d = y - t is one FP32 rounding of operands below 8, the gradient three
    (2^-24 each); the loss adds n squares in FP64."""
    gen = torch.Generator().manual_seed(n)
    y, t = (torch.randn(n, generator=gen).cuda() for _ in range(2))
    gf = torch.full((n + 8,), float("nan"), device="cuda")
    gb = torch.full((n + 8,), float("nan"), dtype=torch.bfloat16, device="cuda")
    loss = torch.full((1,), 3.0, dtype=torch.float64, device="cuda")
    lib.check(lib.lib().otb_mlp_mse_grad(y.data_ptr(), t.data_ptr(), gf.data_ptr(), gb.data_ptr(), n,
                                         loss.data_ptr(), None))
    d = y.double() - t.double()
    want = 2.0 * d / n
    assert float((gf[:n].double() - want).abs().max()) <= 3 * 2 ** -24 * float(want.abs().max())
    assert torch.equal(gb[:n], gf[:n].to(torch.bfloat16))
    assert torch.isnan(gf[n:]).all() and torch.isnan(gb[n:]).all()
    assert abs(float(loss) - 3.0 - float((d * d).sum())) <= 4 * 2 ** -24 * float((d * d).sum()) + 1e-14


@pytest.mark.parametrize("R, C", [(1, 1), (7, 33), (256, 1500)])
def test_colsum_transpose_conversion(lib, R, C):
    """The sums: R additions of order-one values in FP32; the others exact."""
    gen = torch.Generator().manual_seed(R + C)
    x = torch.randn(R, C, generator=gen).cuda()
    s = torch.empty(C, device="cuda")
    b = torch.empty(R, C, dtype=torch.bfloat16, device="cuda")
    bt = torch.empty(C, R, dtype=torch.bfloat16, device="cuda")
    L = lib.lib()
    lib.check(L.otb_mlp_colsum(x.data_ptr(), s.data_ptr(), R, C, None))
    lib.check(L.otb_mlp_f32_to_bf16(x.data_ptr(), b.data_ptr(), x.numel(), None))
    lib.check(L.otb_mlp_transpose_bf16(b.data_ptr(), bt.data_ptr(), R, C, None))
    assert float((s.double() - x.double().sum(0)).abs().max()) <= R * 2 ** -24 * float(x.double().abs().sum(0).max())
    assert torch.equal(b, x.to(torch.bfloat16))
    assert torch.equal(bt, b.T)


@pytest.mark.parametrize("n", [1, 257, 3000])
def test_adamw(lib, n):
    """Three steps against torch.optim.AdamW in float64 (FP32 updates: 1e-5)."""
    gen = torch.Generator().manual_seed(n)
    w, m, v = torch.randn(n, generator=gen).cuda(), torch.zeros(n, device="cuda"), torch.zeros(n, device="cuda")
    wb = torch.empty(n, dtype=torch.bfloat16, device="cuda")
    ref = w.double().clone().requires_grad_(True)
    opt = torch.optim.AdamW([ref], lr=1e-2, betas=(0.9, 0.999), eps=1e-8, weight_decay=0.1)
    for k in range(1, 4):
        g = torch.randn(n, generator=gen).cuda()
        ref.grad = g.double()
        opt.step()
        lib.check(lib.lib().otb_mlp_adamw(w.data_ptr(), g.data_ptr(), m.data_ptr(), v.data_ptr(), wb.data_ptr(), n,
                                          1e-2, 0.9, 0.999, 1e-8, 0.1, k, None))
    assert float((w.double() - ref.detach()).abs().max()) < 1e-5
    assert torch.equal(wb, w.to(torch.bfloat16))
