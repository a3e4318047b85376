"""The mixed sweeps and the mixed Dyson step with several tau points or
frequencies in a launch against the same calls one point (four frequencies) at
a time: a batch member's tiles hold the same operands, so the results are equal
to the bit. Sizes where a member's last row tile has no partner and its 256-wide
column tiles hang over into the next member's rows (128-row tiles odd in
number), and where they do not."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import gw, space_time                            # noqa: E402


def _system(M, n, nocc, naux, seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    X = torch.randn(M, n, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(n)
    D = torch.randn(M, naux, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(M)
    rng = np.random.default_rng(seed)
    eps = np.concatenate([np.sort(rng.uniform(-1.5, -0.3, nocc)),
                          np.sort(rng.uniform(0.1, 3.0, n - nocc))])
    return X, D, eps


SIZES = [(100, 20, 3, 90, 3), (130, 70, 5, 129, 5), (256, 65, 64, 256, 2), (385, 40, 7, 300, 26),
         (700, 90, 9, 641, 7)]


@pytest.mark.parametrize('M,n,nocc,naux,ntau', SIZES)
def test_sweeps_of_many_tau_points(M, n, nocc, naux, ntau):
    X, D, eps = _system(M, n, nocc, naux, M)
    tau = np.linspace(0.1, 2.0, ntau)
    cw = np.ones((1, ntau))
    proj = space_time.chi0_sweep(X, D, eps, nocc, tau, cw, mu=-0.1, want_proj=True,
                                 precision='mixed')[1]
    Wt = torch.rand(ntau, naux, naux, device='cuda', dtype=torch.float64)
    Wt = Wt + Wt.transpose(-1, -2)
    states = np.arange(n)
    br = gw.sigma_branch_sums(X, D, Wt, eps, nocc, tau, states, -0.1, precision='mixed')
    bare = gw.sigma_branch_sums(X, D, None, eps, nocc, tau, states, -0.1, precision='mixed')
    for k in range(ntau):
        one = space_time.chi0_sweep(X, D, eps, nocc, tau[k:k + 1], cw[:, :1], mu=-0.1,
                                    want_proj=True, precision='mixed')[1]
        assert torch.equal(proj[k], one[0])
        # the branch sums add their row tiles atomically, in FP64: any order
        for got, w in ((br, Wt[k:k + 1].contiguous()), (bare, None)):
            ref = gw.sigma_branch_sums(X, D, w, eps, nocc, tau[k:k + 1], states, -0.1,
                                       precision='mixed')
            assert float((got[:, k] - ref[:, 0]).abs().max()) <= 1e-14 * float(ref.abs().max())


@pytest.mark.parametrize('n,nfreq', [(1, 5), (90, 12), (129, 9), (300, 34), (641, 8)])
def test_dyson_of_many_frequencies(n, nfreq):
    g = torch.Generator(device='cuda')
    g.manual_seed(n)
    A = torch.randn(nfreq, n, max(1, n // 2), generator=g, device='cuda', dtype=torch.float64)
    chi0 = -(A @ A.transpose(-1, -2)) / n
    chi0 = 0.5 * (chi0 + chi0.transpose(-1, -2))
    bad = nfreq // 2
    chi0[bad] = 0.0
    chi0[bad].diagonal()[n // 2] = 1.5           # not positive definite: the LU route
    whole = chi0.clone()
    ld, tr, info, sign = space_time.dyson_batch(whole, precision='mixed')
    assert info[bad] == n // 2 + 1 and sign[bad] == -1 and np.count_nonzero(info) == 1
    W = torch.linalg.inv(torch.eye(n, device='cuda', dtype=torch.float64) - chi0[bad])
    W.diagonal().sub_(1.0)
    assert float((whole[bad] - W).abs().max()) < 1e-12
    for f0 in range(0, nfreq - 3, 4):
        part = chi0[f0:f0 + 4].clone()
        ld4 = space_time.dyson_batch(part, precision='mixed')[0]
        assert torch.equal(part, whole[f0:f0 + 4]) and torch.equal(ld4, ld[f0:f0 + 4])
