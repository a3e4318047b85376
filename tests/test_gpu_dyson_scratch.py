"""The batched Dyson step on scratch that holds NaN bit patterns: everything it
reads it has written in the same call. Sizes around 128-row blocks, the
256-row tiles of the mixed inverse (odd and even numbers of blocks, halves
split at odd blocks) and the padding past n, against LAPACK in FP64 with the
bounds of the step's own test (the same matrices' condition numbers, below 30):
5e-6 for the mixed inverse, 3e-12 for the FP64 modes up to n = 400 and in
proportion to n past it."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import _lib                                      # noqa: E402
from mbptcode_b200.space_time import _mode, dyson_batch             # noqa: E402


@pytest.mark.parametrize('precision,n', [('mixed', n) for n in (
    1, 31, 127, 128, 129, 255, 256, 257, 383, 385, 500, 512, 640, 641, 700, 769, 897, 1153)] +
    [('fp64', 129), ('fp64', 641), ('fp64_int8', 129), ('fp64_int8', 700)])
def test_poisoned_scratch(precision, n):
    nfreq = 5
    rng = np.random.default_rng(n)
    chi0 = []
    for f in range(nfreq):
        A = rng.standard_normal((n, max(1, n // 2))) / np.sqrt(n)
        chi0.append(-(A @ A.T) * (1.0 + f))
    chi0 = np.stack(chi0)
    c = torch.as_tensor(chi0, device='cuda').clone()
    ws = _lib.WORKSPACE.get(_lib.lib().mbpt_dyson_workspace_bytes(n, nfreq, _mode(precision)),
                            c.device)
    ws.fill_(255)
    logdet, trace, info, sign = dyson_batch(c, want_w=True, precision=precision)
    assert not info.any() and (sign == 1).all()
    tol = 5e-6 if precision == 'mixed' else 3e-12 * max(1.0, n / 400)
    for f in range(nfreq):
        A = np.eye(n) - chi0[f]
        assert abs(float(logdet[f]) - np.linalg.slogdet(A)[1]) < 1e-13 * n
        assert np.abs(c[f].cpu().numpy() - (np.linalg.inv(A) - np.eye(n))).max() < tol
