"""E_c on a stream of its own while other work is queued on the current one:
nothing of the call (the clearing of its outputs included) may run on the
current stream once the library call is under way, or the result is
overwritten or read too early. The work is queued between the call's input
copies and its outputs, where another thread's would fall."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import space_time                                # noqa: E402


@pytest.mark.parametrize('ntau', [2, 6])
def test_energy_with_a_busy_current_stream(monkeypatch, ntau):
    rng = np.random.default_rng(ntau)
    M, n, nocc, naux = 60, 12, 4, 40
    X = torch.as_tensor(rng.standard_normal((M, n)) / np.sqrt(n), device='cuda')
    D = torch.as_tensor(0.3 * rng.standard_normal((M, naux)) / np.sqrt(M), device='cuda')
    eps = np.concatenate([np.sort(rng.uniform(-1.5, -0.3, nocc)),
                          np.sort(rng.uniform(0.1, 3.0, n - nocc))])
    tau, cw, ow = np.linspace(0.1, 2.0, ntau), np.full((ntau, ntau), 0.2), np.ones(ntau)
    call = (X, D, eps, nocc, tau, cw, ow)
    ref, _, _ = space_time.rpa_energy_device(*call)
    assert float(ref) != 0.0
    big = torch.ones(4096, 4096, device='cuda', dtype=torch.float64)
    other = torch.empty_like(big)
    check = space_time.check_mixed_weights

    def queue_work(*a):
        check(*a)
        for _ in range(8):                   # about 30 ms
            torch.mm(big, big, out=other)

    monkeypatch.setattr(space_time, 'check_mixed_weights', queue_work)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    got, info, _ = space_time.rpa_energy_device(*call, stream=side)
    torch.cuda.synchronize()
    assert abs(float(got) - float(ref)) <= 1e-12 * abs(float(ref)) and not info.any()
