"""Sweeps and Dyson steps that take several batches, the last one shorter: sizes
where the scratch caps (640 MB of FP64 arrays, 1 GB of TF32 pairs but four
matrices) leave 12 + 11, 8 + 8 + 7 and 6 + 6 + 6 + 5 tau points and 3 + 2
matrices, one of the last round's not positive definite. Against plain FP64
torch on the same device.

Tolerances: three FP64 sums in a row over K <= 2000 terms, 1e-12 of the
result's scale (the branch sums: of the sum of their terms' magnitudes);
condition numbers below 30, so 3e-12 n / 400 on the FP64 inverse and 5e-6 on
the mixed one, as in the step's own tests."""
import warnings

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import gw, space_time                            # noqa: E402
from mbptcode_b200.space_time import dyson_batch                    # noqa: E402


@pytest.mark.parametrize('naux', [1300, 2000])
def test_fp64_sweeps(naux):
    M, n, nocc, ntau = 2000, 30, 5, 23
    g = torch.Generator(device='cuda')
    g.manual_seed(naux)
    X = torch.randn(M, n, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(n)
    D = torch.randn(M, naux, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(M)
    rng = np.random.default_rng(naux)
    eps = np.concatenate([np.sort(rng.uniform(-1.5, -0.3, nocc)),
                          np.sort(rng.uniform(0.1, 3.0, n - nocc))])
    tau, cw = np.linspace(0.0, 2.0, ntau), rng.uniform(0.1, 1.0, (2, ntau))
    chi0, proj = space_time.chi0_sweep(X, D, eps, nocc, tau, cw, mu=-0.1, want_proj=True,
                                       precision='fp64')
    Wt = torch.rand(ntau, naux, naux, generator=g, device='cuda', dtype=torch.float64)
    states = np.array([0, nocc - 1, nocc, n - 1])
    branch = gw.sigma_branch_sums(X, D, Wt, eps, nocc, tau, states, -0.1, precision='fp64')
    e = torch.as_tensor(eps + 0.1, device='cuda')
    Xs = X[:, torch.as_tensor(states, device='cuda')]
    total = torch.zeros_like(chi0)
    for k, t in enumerate(tau):
        Go = (X[:, :nocc] * torch.exp(t * e[:nocc])) @ X[:, :nocc].T
        Gv = (X[:, nocc:] * torch.exp(-t * e[nocc:])) @ X[:, nocc:].T
        ref = -2.0 * D.T @ ((Go * Gv) @ D)
        assert float((proj[k] - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
        total += torch.as_tensor(cw[:, k], device='cuda')[:, None, None] * ref
        Z = D @ Wt[k] @ D.T
        for b, G, s in ((0, Go, 1.0), (1, Gv, -1.0)):
            ref = s * (Xs * ((G * Z) @ Xs)).sum(0)
            scale = float((Xs.abs() * ((G * Z).abs() @ Xs.abs())).sum(0).max())
            assert float((branch[b, k] - ref).abs().max()) <= 1e-12 * scale
    assert float((chi0 - total).abs().max()) <= 1e-12 * float(total.abs().max())


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_dyson_rounds(precision):
    n, nfreq, bad = 4100, 5, 4
    g = torch.Generator(device='cuda')
    g.manual_seed(n)
    chi0 = torch.empty(nfreq, n, n, device='cuda', dtype=torch.float64)
    for f in range(nfreq):
        A = torch.randn(n, n // 2, generator=g, device='cuda', dtype=torch.float64)
        chi0[f] = A @ A.T * (-(1.0 + f) / n)
    chi0[bad, 200, :] = 0.0
    chi0[bad, :, 200] = 0.0
    chi0[bad, 200, 200] = 1.5                # 1 - chi0 is -0.5 there
    W = chi0.clone()
    with warnings.catch_warnings():
        warnings.simplefilter('ignore')
        logdet, _, info, sign = dyson_batch(W, want_w=True, precision=precision)
    assert info[bad] == 201 and sign[bad] == -1 and np.count_nonzero(info) == 1
    eye = torch.eye(n, device='cuda', dtype=torch.float64)
    for f in range(nfreq):
        tol = 5e-6 if precision == 'mixed' and f != bad else 3e-12 * n / 400
        assert float((W[f] - (torch.linalg.inv(eye - chi0[f]) - eye)).abs().max()) < tol
        ld = torch.linalg.slogdet(eye - chi0[f])[1]
        assert abs(float(logdet[f]) - float(ld)) < 1e-12 * n
