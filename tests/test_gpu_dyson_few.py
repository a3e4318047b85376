"""The Dyson step of one to three frequencies (one potrf each, their inverses
in shared launches) on scratch that holds NaN bit patterns, at sizes around the
inverse's 128-row blocks: against LAPACK, to the bit against the same
frequencies one at a time, and with one matrix that is not positive definite
(LU, or its info word where the host does not wait).

Tolerances: those of the batched step's tests at the same matrices (condition
numbers below 30): 5e-6 for the mixed inverse, 3e-12 in proportion to n past
400 for the FP64 modes, 1e-11 for the LU route."""
import warnings

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import _lib                                      # noqa: E402
from mbptcode_b200.space_time import _mode, dyson_batch             # noqa: E402


def _chi0(n, nfreq):
    rng = np.random.default_rng(n + nfreq)
    out = []
    for f in range(nfreq):
        A = rng.standard_normal((n, max(1, n // 2))) / np.sqrt(n)
        out.append(-(A @ A.T) * (1.0 + f))
    return np.stack(out)


def _run(chi0, precision, **kw):
    c = torch.as_tensor(chi0, device='cuda').clone()
    ws = _lib.WORKSPACE.get(_lib.lib().mbpt_dyson_workspace_bytes(
        c.shape[-1], c.shape[0], _mode(precision)), c.device)
    ws.fill_(255)
    with warnings.catch_warnings():
        warnings.simplefilter('ignore')
        return (c,) + dyson_batch(c, want_w=True, precision=precision, **kw)


@pytest.mark.parametrize('precision', ['fp64', 'fp64_int8', 'mixed'])
@pytest.mark.parametrize('n', [1, 33, 127, 128, 129, 257, 300, 641])
def test_few_frequencies(n, precision):
    tol = 5e-6 if precision == 'mixed' else 3e-12 * max(1.0, n / 400)
    for nfreq in (1, 2, 3):
        chi0 = _chi0(n, nfreq)
        W, logdet, trace, info, sign = _run(chi0, precision)
        assert not info.any() and (sign == 1).all()
        late, ld, _, info_d, _ = _run(chi0, precision, deferred=True)
        assert torch.equal(late, W) and torch.equal(ld, logdet) and not info_d.any()
        for f in range(nfreq):
            A = np.eye(n) - chi0[f]
            assert abs(float(logdet[f]) - np.linalg.slogdet(A)[1]) < 1e-13 * n
            assert np.abs(W[f].cpu().numpy() - (np.linalg.inv(A) - np.eye(n))).max() < tol
            assert torch.equal(_run(chi0[f:f + 1], precision)[0][0], W[f])


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
@pytest.mark.parametrize('n,nfreq,bad', [(40, 1, 0), (40, 2, 1), (300, 3, 0), (300, 3, 1),
                                         (300, 3, 2)])
def test_one_that_is_not_positive_definite(n, nfreq, bad, precision):
    chi0 = _chi0(n, nfreq)
    p = n // 2
    chi0[bad, p, :] = chi0[bad, :, p] = 0.0
    chi0[bad, p, p] = 1.5                    # 1 - chi0 is -0.5 there
    W, logdet, _, info, sign = _run(chi0, precision)
    assert info[bad] == p + 1 and sign[bad] == -1 and np.count_nonzero(info) == 1
    info_d = _run(chi0, precision, deferred=True)[3]
    assert np.array_equal(info_d.cpu().numpy(), info)
    for f in range(nfreq):
        A = np.eye(n) - chi0[f]
        tol = 1e-11 if f == bad or precision == 'fp64' else 5e-6
        assert abs(float(logdet[f]) - np.linalg.slogdet(A)[1]) < 1e-12 * n
        assert np.abs(W[f].cpu().numpy() - (np.linalg.inv(A) - np.eye(n))).max() < tol
