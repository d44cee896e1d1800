"""The strided tensor-core product in every operand layout and tile width, the
multi-matrix column sums and the one-launch AdamW, against float64 numpy /
torch on the same inputs."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def padded(rows, cols, gen, scale=1.0):
    """Random bf16 [rows][cols] with rows padded to 8 elements (the padding NaN)."""
    ld = (cols + 7) // 8 * 8
    m = torch.full((rows, ld), float("nan"), dtype=torch.bfloat16, device="cuda")
    m[:, :cols] = (scale * torch.randn(rows, cols, generator=gen)).to("cuda")
    return m[:, :cols]


# every tile width (64, 128, 256: tiles against 152 SMs), edges and remainders
SHAPES = [(1, 1, 1), (128, 64, 64), (129, 65, 7), (300, 1500, 130), (512, 512, 256), (1500, 512, 33),
          (5000, 500, 72), (20000, 515, 40), (19999, 513, 8)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_strided_product(M, N, K, ta, tb):
    """bf16 inputs, FP32 accumulation over K terms of order 1 / sqrt(K): 1e-4."""
    from oqupy_gb300 import _native as nat
    gen = torch.Generator().manual_seed(M + N + K)
    A = padded(K, M, gen) if ta else padded(M, K, gen)
    B = padded(K, N, gen, K ** -0.5) if tb else padded(N, K, gen, K ** -0.5)
    bias = torch.randn(N, generator=gen).cuda()
    outf = torch.zeros(M, N, device="cuda")
    outb = padded(M, N, gen)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.check(nat.lib().otb_mlp_gemm_strided(
        A.data_ptr(), A.stride(0), ta, B.data_ptr(), B.stride(0), tb, M, N, K, bias.data_ptr(), 0, None, None,
        outf.data_ptr(), outb.data_ptr(), outb.stride(0), err.data_ptr(), None))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    a, b = A.double(), B.double()
    want = (a.T if ta else a) @ (b if tb else b.T) + bias.double()
    assert float((outf.double() - want).abs().max()) < 1e-4
    assert float((outb.double() - want).abs().max()) < 1e-4 + 2 ** -8 * float(want.abs().max())


@pytest.mark.parametrize("rows", [1, 7, 256, 1000])
def test_colsums(rows):
    from oqupy_gb300 import _native as nat
    cols = [1, 31, 33, 512, 1500]
    mats = [torch.randn(rows, c, device="cuda") for c in cols]
    outs = [torch.empty(c, device="cuda") for c in cols]
    P = ctypes.c_void_p * len(cols)
    nat.check(nat.lib().otb_mlp_colsums(len(cols), P(*[m.data_ptr() for m in mats]), P(*[o.data_ptr() for o in outs]),
                                        rows, (ctypes.c_int32 * len(cols))(*cols), None))
    for m, o in zip(mats, outs):
        # rows FP32 additions of order-one values
        assert float((o.double() - m.double().sum(0)).abs().max()) < rows * 6e-8 * 4 * max(1.0, rows ** 0.5)


@pytest.mark.parametrize("sizes", [[5, 33, 7], [3, 64, 65, 150]])
def test_adamw_net_matches_torch(sizes):
    """Three steps against torch.optim.AdamW in float64 (FP32 updates: 1e-5)."""
    from oqupy_gb300.surrogate import Mlp
    net = Mlp(sizes, seed=3)
    ref = [p.double().clone().requires_grad_(True) for p in net.W + net.b]
    n = len(net.W)
    opt = torch.optim.AdamW([{"params": ref[:n], "weight_decay": 0.1}, {"params": ref[n:], "weight_decay": 0.0}],
                            lr=1e-2, betas=(0.9, 0.999), eps=1e-8)
    for k in range(3):
        g = [torch.randn_like(p) for p in net.W + net.b]
        for r, x in zip(ref, g):
            r.grad = x.double()
        opt.step()
        net.step(g[:n], g[n:], lr=1e-2, weight_decay=0.1)
    for p, r in zip(net.W + net.b, ref):
        assert float((p.double() - r.detach()).abs().max()) < 1e-5
    for l in range(n):
        assert torch.equal(net.Wb[l], net.W[l].to(torch.bfloat16))
        assert torch.equal(net.WbT[l], net.W[l].T.to(torch.bfloat16))
