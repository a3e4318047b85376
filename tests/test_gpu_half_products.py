"""chi0 with Pi held by halves (csrc/dmma.cu, capi.cu half_pi) against plain FP64
torch: sizes on both sides of the rule's lines (M = 3/2 naux, M = 5/4 naux, one
round of CTAs), one row or column past a 64-wide tile, odd and even leading
dimensions, D^T Y cut along K into 2 to 8 parts with a ragged last one, and
orbital counts at, one past and one before a multiple of four (the steps of a
product's last K tile).

Tolerance: three FP64 sums in a row over K <= 1217 terms of one sign or with
cancellation of a factor 10: 1e-12 of the result's scale. The halves add S and
S^T, which is one rounding."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import space_time                                # noqa: E402


@pytest.mark.parametrize('M,n,nocc,naux,ntau', [
    (96, 9, 4, 64, 34), (97, 10, 5, 65, 34), (449, 21, 4, 130, 26), (449, 22, 5, 129, 26),
    (1217, 24, 8, 1, 32), (704, 40, 16, 449, 8), (705, 41, 17, 470, 12), (1100, 30, 3, 63, 34),
    (830, 20, 7, 664, 28), (831, 20, 7, 664, 29)])
def test_chi0_by_halves(M, n, nocc, naux, ntau):
    g = torch.Generator(device='cuda')
    g.manual_seed(M + naux)
    X = torch.randn(M, n, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(n)
    D = torch.randn(M, naux, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(M)
    rng = np.random.default_rng(M)
    eps = np.concatenate([np.sort(rng.uniform(-1.5, -0.3, nocc)),
                          np.sort(rng.uniform(0.1, 3.0, n - nocc))])
    tau = np.linspace(0.0, 2.0, ntau)
    cw = rng.uniform(0.1, 1.0, (3, ntau))
    chi0, proj = space_time.chi0_sweep(X, D, eps, nocc, tau, cw, mu=-0.1, want_proj=True,
                                       precision='fp64')
    e = torch.as_tensor(eps + 0.1, device='cuda')
    ref = []
    for t in tau:
        Go = (X[:, :nocc] * torch.exp(t * e[:nocc])) @ X[:, :nocc].T
        Gv = (X[:, nocc:] * torch.exp(-t * e[nocc:])) @ X[:, nocc:].T
        ref.append(-2.0 * D.T @ ((Go * Gv) @ D))
    ref = torch.stack(ref)
    assert float((proj - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
    ref = torch.einsum('fk,kab->fab', torch.as_tensor(cw, device='cuda'), ref)
    assert float((chi0 - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
