"""The entry points under a CUDA default device, where torch's factory calls
that name no device give device tensors: staging blocks on the host stay there,
and the results are those without a default device."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import grids, gw, space_time                     # noqa: E402
from mbptcode_b200.synthetic import synthetic_system                # noqa: E402


@pytest.mark.parametrize('precision', ['fp64', 'mixed'])
def test_calls_under_a_default_device(precision):
    n, nocc, M = 40, 5, 200
    X, D, eps = synthetic_system(n, nocc, M, seed=1, variant='calibrated')
    axes = grids.space_time_axes(eps, nocc, ntau=20)
    states = np.arange(nocc - 4, nocc + 4)

    def calls():
        e = space_time.rpa_correlation_energy_space_time(X, D, eps, nocc, axes.grid,
                                                         precision=precision)
        r = gw.gw_sweep(X, D, eps, nocc, states=states, axes=axes, precision=precision)
        return e, float(r['e_c']), torch.as_tensor(r['roots']).cpu().numpy()

    ref = calls()
    with torch.device('cuda'):
        got = calls()
    # the sums over row tiles are added in any order: last bits of E_c and of
    # Sigma, which the root search's 1e-8 bisection does not resolve
    for a, b in zip(got[:2], ref[:2]):
        assert abs(a - b) <= 1e-12 * abs(b)
    assert np.abs(got[2] - ref[2]).max() <= 2e-8
