"""The FP64 sweeps' products (csrc/dmma.cu) against plain FP64 torch on the
same device: 64 x 64 tiles and 16-wide K steps, so sizes one below, at and
one above a tile and a step; odd leading dimensions (8-byte copies) and even
ones (16-byte); one occupied orbital; one state, the last narrow tile's 32 and
33; more tau points than one launch takes; a W(tau) that is not symmetric; W = I.

The int8-emulated mode shares the G products and the contraction with the
states: the same sizes at 1e-11, its products carrying 5e-15 of K times their
operands' row maxima (K <= 1100).

Tolerance: an FP64 sum of K terms is off by at most K eps of the sum of its
terms' magnitudes; three sums in a row over K <= 1100 give 1e-12 of the
result's scale with room for cancellation of a factor 10 (the largest branch
sums and chi0 are sums of one sign)."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import gw, space_time                            # noqa: E402

TOL = {'fp64': 1e-12, 'fp64_int8': 1e-11}


def _system(M, n, nocc, naux, seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    X = torch.randn(M, n, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(n)
    D = torch.randn(M, naux, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(M)
    rng = np.random.default_rng(seed)
    eps = np.concatenate([np.sort(rng.uniform(-1.5, -0.3, nocc)),
                          np.sort(rng.uniform(0.1, 3.0, n - nocc))])
    return X, D, eps


def _branches(X, eps, nocc, mu, tau):
    e = torch.as_tensor(eps - mu, device=X.device)
    Go = (X[:, :nocc] * torch.exp(tau * e[:nocc])) @ X[:, :nocc].T
    Gv = (X[:, nocc:] * torch.exp(-tau * e[nocc:])) @ X[:, nocc:].T
    return Go, Gv


def _close(got, ref, precision):
    return float((got - ref).abs().max()) <= TOL[precision] * float(ref.abs().max())


@pytest.mark.parametrize('precision', ['fp64', 'fp64_int8'])
@pytest.mark.parametrize('M,n,nocc,naux,ntau', [
    (1, 2, 1, 1, 1), (15, 3, 1, 17, 2), (63, 17, 1, 64, 3), (64, 18, 16, 66, 12),
    (65, 33, 15, 63, 24), (129, 40, 8, 128, 5), (200, 35, 17, 301, 20), (1100, 61, 6, 130, 34)])
def test_chi0_and_proj(M, n, nocc, naux, ntau, precision):
    X, D, eps = _system(M, n, nocc, naux, M + n)
    tau = np.linspace(0.0, 2.0, ntau)
    cw = np.random.default_rng(3).uniform(0.1, 1.0, (4, ntau))
    chi0, proj = space_time.chi0_sweep(X, D, eps, nocc, tau, cw, mu=-0.1, want_proj=True,
                                       precision=precision)
    ref = []
    for t in tau:
        Go, Gv = _branches(X, eps, nocc, -0.1, float(t))
        ref.append(-2.0 * D.T @ ((Go * Gv) @ D))
    ref = torch.stack(ref)
    assert _close(proj, ref, precision)
    assert _close(chi0, torch.einsum('fk,kab->fab', torch.as_tensor(cw, device='cuda'), ref),
                  precision)


@pytest.mark.parametrize('precision', ['fp64', 'fp64_int8'])
@pytest.mark.parametrize('M,n,nocc,naux,ntau,S,w', [
    (1, 2, 1, 1, 1, 1, 'any'), (63, 17, 1, 63, 3, 17, 'any'), (64, 40, 16, 64, 2, 32, 'sym'),
    (65, 40, 15, 66, 24, 33, 'any'), (129, 70, 8, 127, 37, 64, 'any'), (300, 70, 9, 100, 3, 70, None),
    (1100, 20, 6, 258, 5, 1, 'any')])
def test_branch_sums(M, n, nocc, naux, ntau, S, w, precision):
    if precision == 'fp64_int8' and w == 'any':
        w = 'sym'                            # that mode takes W(tau) as symmetric
    X, D, eps = _system(M, n, nocc, naux, M + n + 1)
    tau = np.linspace(0.0, 2.0, ntau)
    g = torch.Generator(device='cuda')
    g.manual_seed(5)
    Wt = None
    if w:
        Wt = torch.rand(ntau, naux, naux, generator=g, device='cuda', dtype=torch.float64)
        Wt.diagonal(dim1=-2, dim2=-1).add_(1.0)
        if w == 'sym':
            Wt = Wt + Wt.transpose(-1, -2)
    states = np.linspace(0, n - 1, S).astype(int)
    got = gw.sigma_branch_sums(X, D, Wt, eps, nocc, tau, states, -0.1, precision=precision)
    Xs = X[:, torch.as_tensor(states, device='cuda')]
    lo, hi = [], []
    scale = []
    for k, t in enumerate(tau):
        Z = D @ Wt[k] @ D.T if w else D @ D.T
        for out, G, s in zip((lo, hi), _branches(X, eps, nocc, -0.1, float(t)), (1.0, -1.0)):
            out.append(s * (Xs * ((G * Z) @ Xs)).sum(0))
            scale.append((Xs.abs() * ((G * Z).abs() @ Xs.abs())).sum(0).max())
    ref = torch.stack([torch.stack(lo), torch.stack(hi)])
    # random signs cancel here: against the sum of the terms' magnitudes
    assert float((got - ref).abs().max()) <= TOL[precision] * float(torch.stack(scale).max())
