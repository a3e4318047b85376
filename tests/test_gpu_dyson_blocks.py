"""The batched Dyson step at the sizes where its blocking changes: matrices of
one row up to three 128-row blocks, with last blocks of 1, 31, 32, 33, 64, 97
rows (the factorisation works in 32-row sub-blocks, the inverse in 64-row tiles
and halves split at multiples of 128), four frequencies and five, against
LAPACK: log-determinants, traces and W - I in each mode, and where the first
bad pivot is of a matrix that is not positive definite.

Tolerances: A = 1 - chi0 has condition number below 30 here, so a backward
stable factorisation of n <= 400 rows moves W by less than 30 n eps = 3e-12
of its largest entry and log det by n eps relative to its scale n; the mixed
inverse's TF32x3 products carry 5e-6 (their own test's bar)."""
import warnings

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200.space_time import dyson_batch                    # noqa: E402


def _chi0(n, nfreq, seed):
    rng = np.random.default_rng(seed)
    out = []
    for f in range(nfreq):
        A = rng.standard_normal((n, max(1, n // 2))) / np.sqrt(n)
        out.append(-(A @ A.T) * (1.0 + f))
    return np.stack(out)


SIZES = [1, 2, 31, 32, 33, 63, 64, 65, 97, 127, 128, 129, 160, 192, 225, 255, 256, 257, 384, 400]


@pytest.mark.parametrize('precision', ['fp64', 'fp64_int8', 'mixed'])
@pytest.mark.parametrize('n', SIZES)
def test_batched_dyson_against_lapack(n, precision):
    nfreq = 4 + n % 2
    chi0 = _chi0(n, nfreq, n)
    c = torch.as_tensor(chi0, device='cuda').clone()
    logdet, trace, info, sign = dyson_batch(c, want_w=True, precision=precision)
    assert not info.any() and (sign == 1).all()
    got = c.cpu().numpy()
    for f in range(nfreq):
        A = np.eye(n) - chi0[f]
        ref = np.linalg.slogdet(A)[1]
        assert abs(float(logdet[f]) - ref) < 1e-13 * n
        assert abs(float(trace[f]) - np.trace(chi0[f])) < 1e-13 * n
        W = np.linalg.inv(A) - np.eye(n)
        assert np.abs(got[f] - W).max() < (5e-6 if precision == 'mixed' else 3e-12)
        if precision != 'mixed':  # there the diagonal tiles' hi lo and lo hi terms differ
            assert np.array_equal(got[f], got[f].T)


@pytest.mark.parametrize('n,p', [(1, 0), (40, 33), (129, 128), (300, 127), (300, 200)])
def test_first_bad_pivot_and_lu_fallback(n, p):
    chi0 = _chi0(n, 5, n + 1)
    chi0[2, p, :] = 0.0
    chi0[2, :, p] = 0.0
    chi0[2, p, p] = 1.5                      # 1 - chi0 is -0.5 there
    c = torch.as_tensor(chi0, device='cuda').clone()
    with warnings.catch_warnings():
        warnings.simplefilter('ignore')
        logdet, _, info, sign = dyson_batch(c, want_w=True, precision='fp64')
    assert info[2] == p + 1 and sign[2] == -1
    assert not np.delete(info, 2).any() and (np.delete(sign, 2) == 1).all()
    got = c.cpu().numpy()
    for f in range(5):
        A = np.eye(n) - chi0[f]
        assert abs(float(logdet[f]) - np.linalg.slogdet(A)[1]) < 1e-12 * n
        assert np.abs(got[f] - (np.linalg.inv(A) - np.eye(n))).max() < 1e-11
