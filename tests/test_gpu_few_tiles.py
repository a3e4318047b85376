"""chi0 of one to four tau points, whose products have fewer tiles than the GPU
has SMs and are cut along K (csrc/dmma.h cut_parts, square_parts), on scratch
that holds NaN bit patterns and against plain FP64 torch: sizes on both sides
of the rules' lines, ragged last parts, 2 to 8 of them, naux past M (nothing fits
where Pi was), odd and even leading dimensions, 32- and 64-wide tiles.

Tolerance: three FP64 sums in a row over K <= 2001 terms of one sign or with
cancellation of a factor 10: 1e-12 of the result's scale, as in the tests of
the uncut products."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import _lib, space_time                          # noqa: E402


@pytest.mark.parametrize('M,n,nocc,naux', [
    (130, 20, 4, 130), (255, 12, 3, 40), (300, 30, 5, 300), (301, 30, 5, 333), (444, 26, 5, 100),
    (449, 21, 4, 449), (600, 17, 3, 257), (771, 20, 4, 768), (888, 43, 5, 141), (889, 42, 5, 65),
    (1332, 58, 5, 236), (1333, 30, 5, 700), (2001, 40, 6, 300)])
def test_few_tau_points(M, n, nocc, naux):
    g = torch.Generator(device='cuda')
    g.manual_seed(M + naux)
    X = torch.randn(M, n, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(n)
    D = torch.randn(M, naux, generator=g, device='cuda', dtype=torch.float64) / np.sqrt(M)
    rng = np.random.default_rng(M)
    eps = np.concatenate([np.sort(rng.uniform(-1.5, -0.3, nocc)),
                          np.sort(rng.uniform(0.1, 3.0, n - nocc))])
    e = torch.as_tensor(eps + 0.1, device='cuda')
    for ntau in (1, 2, 4):
        tau = np.linspace(0.0, 2.0, ntau)
        cw = rng.uniform(0.1, 1.0, (2, ntau))
        ws = _lib.WORKSPACE.get(_lib.lib().mbpt_chi0_workspace_bytes(
            M, n, nocc, naux, ntau, space_time._mode('fp64')), X.device)
        ws.fill_(255)
        chi0, proj = space_time.chi0_sweep(X, D, eps, nocc, tau, cw, mu=-0.1, want_proj=True,
                                           precision='fp64')
        ref = []
        for t in tau:
            Go = (X[:, :nocc] * torch.exp(t * e[:nocc])) @ X[:, :nocc].T
            Gv = (X[:, nocc:] * torch.exp(-t * e[nocc:])) @ X[:, nocc:].T
            ref.append(-2.0 * D.T @ ((Go * Gv) @ D))
        ref = torch.stack(ref)
        assert float((proj - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
        ref = torch.einsum('fk,kab->fab', torch.as_tensor(cw, device='cuda'), ref)
        assert float((chi0 - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
