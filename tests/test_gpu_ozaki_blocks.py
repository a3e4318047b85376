"""The int8 products' tiles where their epilogue and their raster can go wrong
(csrc/ozaki.cu): columns one before, at and one past a strip of 16 column
tiles, with an old C and an odd leading dimension; the symmetric products with
two element-wise factors (the reverse chi0 sweep) at one tile, across the
diagonal and with ragged last tiles, against torch's autograd.

Tolerances: 8 digits carry each entry to K 2^-56 of its row and column maxima
(1e-13 of that scale as in the products' own test); the reverse sweep chains
three such products over K <= 321, held to 1e-11 of each result's scale."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import _lib                                      # noqa: E402
from mbptcode_b200._lib import check, lib, ptr                      # noqa: E402
from mbptcode_b200.adjoint import chi0_backward                     # noqa: E402


@pytest.mark.parametrize('m,n,k', [(1, 1023, 64), (130, 1024, 65), (257, 1025, 129),
                                   (40, 2113, 193), (1153, 33, 320)])
@pytest.mark.parametrize('beta', [0.0, -0.75])
def test_product_strips(m, n, k, beta):
    g = torch.Generator(device='cuda').manual_seed(m + n + k)
    A = torch.randn(m, k, generator=g, device='cuda', dtype=torch.float64)
    B = torch.randn(n, k, generator=g, device='cuda', dtype=torch.float64)
    C = torch.randn(m, n + 3, generator=g, device='cuda', dtype=torch.float64)
    ref = 1.5 * A @ B.T + beta * C[:, :n]
    pad = C[:, n:].clone()
    ws = torch.empty(lib().mbpt_dgemm_ozaki_workspace_bytes(m, n, k, 8), dtype=torch.uint8,
                     device='cuda')
    err = torch.zeros(1, dtype=torch.int32, device='cuda')
    check(lib().mbpt_dgemm_ozaki(0, 1, m, n, k, 1.5, ptr(A), k, ptr(B), k, beta, ptr(C), n + 3, 8,
                                 ptr(ws), ws.numel(), ptr(err), _lib.stream_ptr()),
          'mbpt_dgemm_ozaki')
    assert int(err.item()) == 0
    bound = 1.5 * k * A.abs().amax(1)[:, None] * B.abs().amax(1)[None, :] + 1.0
    assert float(((C[:, :n] - ref).abs() / bound).max()) < 1e-13
    assert torch.equal(C[:, n:], pad)


@pytest.mark.parametrize('M,n,nocc,naux,ntau', [(1, 2, 1, 1, 1), (33, 9, 4, 20, 2),
                                                (64, 12, 5, 64, 1), (65, 12, 5, 33, 2),
                                                (128, 20, 7, 66, 1), (190, 31, 6, 129, 3),
                                                (321, 40, 9, 200, 2)])
def test_reverse_sweep(M, n, nocc, naux, ntau):
    g = torch.Generator(device='cuda').manual_seed(M + n)
    X = torch.randn(M, n, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(n)
    D = torch.randn(M, naux, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(M)
    pb = torch.randn(ntau, naux, naux, generator=g, device='cuda', dtype=torch.float64)
    rng = np.random.default_rng(M)
    eps = np.concatenate([np.sort(rng.uniform(-1.5, -0.3, nocc)),
                          np.sort(rng.uniform(0.1, 3.0, n - nocc))])
    tau, mu = np.linspace(0.2, 2.0, ntau), -0.1
    got = chi0_backward(pb, X, D, eps, nocc, tau, mu, precision='fp64_int8')
    leaf = [torch.as_tensor(eps, device='cuda'), X.clone(), D.clone()]
    for t in leaf:
        t.requires_grad_(True)
    e, Xl, Dl = leaf
    total = 0.0
    for k, t in enumerate(tau):
        Go = (Xl[:, :nocc] * torch.exp(float(t) * (e[:nocc] - mu))) @ Xl[:, :nocc].T
        Gv = (Xl[:, nocc:] * torch.exp(-float(t) * (e[nocc:] - mu))) @ Xl[:, nocc:].T
        total = total + (pb[k] * (-2.0 * Dl.T @ ((Go * Gv) @ Dl))).sum()
    total.backward()
    for a, b in zip(got, leaf):
        assert float((a - b.grad).abs().max()) <= 1e-11 * max(float(b.grad.abs().max()), 1e-300)
