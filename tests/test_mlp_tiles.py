"""Products of the network's kernels at the edges of their tiles of 64 rows (64 tiles or more) and of 32, of
their steps of 32 along K and of its eights, with row pitches, alpha and beta, and as layers.  Against 64 bits; a
sum of K FP32 products is off by at most (K + 3) 2^-24 sum |a b| (one rounding per addition and product)."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')


def need_gpu():
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')


@pytest.mark.gpu
@pytest.mark.parametrize('M,N,K', [(4096, 64, 8), (4097, 65, 9), (4033, 63, 33), (64 * 63, 64, 1), (1030, 260, 31),
                                   (513, 515, 64), (512, 512, 513), (70, 4100, 7), (2000, 64, 64), (33, 66, 40)])
@pytest.mark.parametrize('ta,tb', [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_products(M, N, K, ta, tb):
    need_gpu()
    from srw_b200 import capi
    L = capi.lib()
    g = torch.Generator(device='cuda').manual_seed(M * 7 + N * 3 + K)
    for alpha, beta, pad in ((1., 0., 0), (1., 0., 3), (-0.5, 2., 4)):
        A = torch.randn((K, M + pad) if ta else (M, K + pad), device='cuda', generator=g)
        B = torch.randn((N, K + pad) if tb else (K, N + pad), device='cuda', generator=g)
        C = torch.randn((M, N + pad), device='cuda', generator=g)
        C0 = C.double()
        a = (A[:, :M].t() if ta else A[:, :K]).double()
        b = (B[:, :K].t() if tb else B[:, :N]).double()
        r = L.srwgMlpGemm(M, N, K, A.data_ptr(), A.shape[1], ta, B.data_ptr(), B.shape[1], tb, C.data_ptr(), N + pad, alpha,
                          beta, torch.cuda.current_stream().cuda_stream)
        assert r == 0
        want = alpha * (a @ b) + beta * C0[:, :N]
        bound = (abs(alpha) * (a.abs() @ b.abs()) + abs(beta) * C0[:, :N].abs()) * (K + 3) * 2. ** -24
        assert bool(((C[:, :N].double() - want).abs() <= bound).all())
        assert torch.equal(C[:, N:].double(), C0[:, N:])


@pytest.mark.gpu
@pytest.mark.parametrize('B,n_in,n_out', [(4097, 65, 70), (1024, 256, 256), (8, 4109, 256)])
def test_layer_and_its_gradients(B, n_in, n_out):
    need_gpu()
    from srw_b200 import capi
    L = capi.lib()
    g = torch.Generator(device='cuda').manual_seed(B)
    new = lambda *s: torch.randn(s, device='cuda', generator=g)  # noqa: E731
    X, W, b, dZ, Zp = new(B, n_in), new(n_in, n_out), new(n_out), new(B, n_out), new(B, n_in)
    Z, Y, dW, db, dX = (torch.empty(s, device='cuda') for s in ((B, n_out), (B, n_out), (n_in, n_out), (n_out,), (B, n_in)))
    st = torch.cuda.current_stream().cuda_stream
    assert L.srwgMlpLinear(B, n_out, n_in, X.data_ptr(), W.data_ptr(), b.data_ptr(), Z.data_ptr(), Y.data_ptr(), 1, st) == 0
    assert L.srwgMlpLinearBackward(B, n_out, n_in, X.data_ptr(), W.data_ptr(), dZ.data_ptr(), dW.data_ptr(), db.data_ptr(),
                                   dX.data_ptr(), Zp.data_ptr(), st) == 0
    x, w, d, zp = X.double(), W.double(), dZ.double(), Zp.double().requires_grad_(True)
    u = 2. ** -24
    z = x @ w + b.double()
    assert bool(((Z.double() - z).abs() <= (x.abs() @ w.abs() + b.double().abs()) * (n_in + 3) * u).all())
    y = torch.nn.functional.gelu(Z.double(), approximate='tanh')
    # (GELU of the same Z: a dozen roundings of terms up to |z|)
    assert bool(((Y.double() - y).abs() <= 16 * u * (Z.double().abs() + 1.)).all())
    assert bool(((dW.double() - x.t() @ d).abs() <= (x.abs().t() @ d.abs()) * (B + 3) * u).all())
    assert bool(((db.double() - d.sum(0)).abs() <= d.abs().sum(0) * (B + 3) * u).all())
    torch.nn.functional.gelu(zp, approximate='tanh').sum().backward()
    want = (d @ w.t()) * zp.grad
    # (GELU' is at most 1.13: its own roundings, a dozen of terms up to |z| (1 + |z|^3) / 8, weigh with the sum)
    bound = (d.abs() @ w.abs().t()) * 1.13 * ((n_out + 3) * u + 32 * u * (1. + Zp.double().abs() ** 3))
    assert bool(((dX.double() - want).abs() <= bound).all())
