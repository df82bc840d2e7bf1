"""The network's layer kernels (product in pieces of K over a cluster, with bias, activation, activation
gradient and column sums behind it; Adam of several arrays) at the edges of their 32 x 64 tiles and of
their pieces, against FP64.  A product of FP32 values summed in any order is within K u (|A| |B|) of the
exact one, u = 2^-24 per operation."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip('torch')

U = 2. ** -24


def gelu(z):
    return 0.5 * z * (1. + np.tanh(0.7978845608028654 * (z + 0.044715 * z ** 3)))


def gelu_grad(z):
    u = 0.7978845608028654 * (z + 0.044715 * z ** 3)
    t = np.tanh(u)
    return 0.5 * (1. + t) + 0.5 * z * (1. - t * t) * 0.7978845608028654 * (1. + 3. * 0.044715 * z * z)


@pytest.mark.gpu
@pytest.mark.parametrize('M,N,K', [(1, 1, 1), (1, 256, 4109), (31, 63, 65), (33, 65, 127), (128, 256, 512), (32, 64, 1023),
                                   (7, 4, 256), (500, 130, 33)])
def test_layer_and_its_gradients(M, N, K):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200 import capi
    L = capi.lib()
    rng = np.random.default_rng(M * 7919 + N * 31 + K)
    X, W, dZ, Zp = (rng.standard_normal(s).astype(np.float32) for s in ((M, K), (K, N), (M, N), (M, K)))
    b = rng.standard_normal(N).astype(np.float32)
    d = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    tX, tW, tb, tdZ, tZp = d(X), d(W), d(b), d(dZ), d(Zp)
    Z, Y, dX = torch.empty((M, N), device='cuda'), torch.empty((M, N), device='cuda'), torch.empty((M, K), device='cuda')
    dW, db = torch.empty((K, N), device='cuda'), torch.empty(N, device='cuda')
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.srwgMlpLinear(M, N, K, tX.data_ptr(), tW.data_ptr(), tb.data_ptr(), Z.data_ptr(), Y.data_ptr(), 1, st) == 0
    assert L.srwgMlpLinearBackward(M, N, K, tX.data_ptr(), tW.data_ptr(), tdZ.data_ptr(), dW.data_ptr(), db.data_ptr(),
                                   dX.data_ptr(), tZp.data_ptr(), st) == 0
    torch.cuda.synchronize()
    X, W, b, dZ, Zp = (a.astype(np.float64) for a in (X, W, b, dZ, Zp))
    z = X @ W + b
    assert np.all(np.abs(Z.cpu().numpy() - z) <= 1.1 * (K + 2) * U * (np.abs(X) @ np.abs(W) + np.abs(b)) + 1e-30)
    # GELU of the kernel's own Z: a few roundings and tanhf (2 ulp)
    zk = Z.cpu().numpy().astype(np.float64)
    assert np.all(np.abs(Y.cpu().numpy() - gelu(zk)) <= 16. * U * (np.abs(zk) + 1.))
    assert np.all(np.abs(dW.cpu().numpy() - X.T @ dZ) <= 1.1 * (M + 1) * U * (np.abs(X).T @ np.abs(dZ)) + 1e-30)
    assert np.all(np.abs(db.cpu().numpy() - dZ.sum(0)) <= 1.1 * (M + 1) * U * np.abs(dZ).sum(0) + 1e-30)
    g = gelu_grad(Zp)
    lim = 1.1 * (N + 1) * U * (np.abs(dZ) @ np.abs(W).T) * np.abs(g) + 64. * U * np.abs(dZ @ W.T)
    assert np.all(np.abs(dX.cpu().numpy() - (dZ @ W.T) * g) <= lim + 1e-30)


@pytest.mark.gpu
@pytest.mark.parametrize('lens', [(1,), (255, 256, 257), tuple(range(1, 18))])
def test_adam_of_many_arrays_is_adam_of_each(lens):
    if not torch.cuda.is_available():
        pytest.skip('no CUDA device')
    from srw_b200 import capi
    L = capi.lib()
    g = torch.Generator(device='cuda').manual_seed(3)
    new = lambda n: torch.randn(n, device='cuda', generator=g)  # noqa: E731
    one = [[new(n), new(n), new(n), new(n).abs()] for n in lens]
    many = [[t.clone() for t in a] for a in one]
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for a in one:
        assert L.srwgMlpAdam(*[t.data_ptr() for t in a], a[0].numel(), 1e-3, 0.9, 0.999, 1e-8, 3, st) == 0
    n = len(lens)
    arr = [(C.c_void_p * n)(*[a[k].data_ptr() for a in many]) for k in range(4)]
    assert L.srwgMlpAdamMany(n, *arr, (C.c_longlong * n)(*lens), 1e-3, 0.9, 0.999, 1e-8, 3, st) == 0
    torch.cuda.synchronize()
    for a, b in zip(one, many):
        assert all(torch.equal(x, y) for x, y in zip(a, b))
