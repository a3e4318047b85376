"""The root search of one CTA per state against the oracle's serial one:
evaluation counts, quasiparticle flags and roots of pole-sum self-energies,
for the smallest and the largest fractions (npade 2, 3, 31, 32: the greedy
ordering is one warp), one state and many, the smooth Sigma of a sweep and one
of a few strong poles (several brackets per window, whole ranges of slow
cells, all three windows).

Tolerance: both sides bisect the same cells to 1e-8, so a midpoint whose sign
the last bits of Sigma decide moves a root by at most 2e-8; a state whose
oracle root (or count) itself changes when Sigma is perturbed by 1e-13 is
undecided by the input and only has to be finite where the oracle's is."""
import numpy as np
import pytest

torch = pytest.importorskip('torch')

from oracle import st_oracle as orc                                 # noqa: E402
from mbptcode_b200 import gw                                        # noqa: E402


def _case(npade, nstates, strong, seed):
    rng = np.random.default_rng(seed)
    nocc = max(1, nstates // 3)
    eps = np.sort(np.concatenate([rng.uniform(-4.5, -0.3, nocc),
                                  rng.uniform(0.1, 4.5, max(1, nstates - nocc))]))[:nstates]
    mu = -0.1
    if strong:
        poles = np.concatenate([rng.uniform(-6.0, -0.6, 5), rng.uniform(0.6, 6.0, 6)])
        amp = rng.uniform(0.02, 0.4, (nstates, poles.size))
    else:
        poles = np.concatenate([-rng.uniform(2.0, 40.0, 40), rng.uniform(2.0, 40.0, 60)])
        amp = rng.uniform(0.0, 0.02, (nstates, poles.size))
    freq = 0.3 * (np.arange(npade) + 0.5) ** 1.5
    z = mu + 1j * freq
    sigma = np.einsum('pk,kw->pw', amp, 1.0 / (z[None, :] - poles[:, None]))
    if npade >= 18:  # keeps the long fractions' coefficients well determined
        sigma *= 1.0 + 0.02 * (rng.standard_normal(sigma.shape)
                               + 1j * rng.standard_normal(sigma.shape))
    return eps, nocc, mu, freq, sigma


def _oracle(eps, nocc, mu, freq, sigma, greedy):
    roots, zs, qp, counts = [], [], [], []
    for p in range(len(eps)):
        z_fit = orc.imaginary_axis_sample_points(freq, nocc, p, mu)
        s = np.conj(sigma[p]) if p < nocc else sigma[p]
        fit = orc.PadeFit(z_fit, s, greedy=greedy)
        func = orc._Counted(lambda w: w - eps[p] - fit(np.array([w], dtype=complex))[0].real)
        root, z, ok = orc.solve_qp_equation_pole_strength(func, eps[p])
        roots.append(root)
        zs.append(z)
        qp.append(ok)
        counts.append(func.n)
    return np.array(roots), np.array(zs), np.array(qp), np.array(counts)


@pytest.mark.gpu
@pytest.mark.parametrize('npade,nstates,strong,greedy',
                         [(2, 5, False, True), (3, 1, True, True), (12, 14, True, True),
                          (12, 9, True, False), (18, 12, False, True), (31, 6, False, True),
                          (32, 6, True, True)])
def test_root_search_matches_the_serial_one(npade, nstates, strong, greedy):
    eps, nocc, mu, freq, sigma = _case(npade, nstates, strong, 7 * npade + nstates)
    with np.errstate(all='ignore'):
        root, zs, qp, count = _oracle(eps, nocc, mu, freq, sigma, greedy)
        rng = np.random.default_rng(1)
        bent = sigma * (1.0 + 1e-13 * rng.standard_normal(sigma.shape))
        root2, _, qp2, count2 = _oracle(eps, nocc, mu, freq, bent, greedy)
    settled = (np.abs(root - root2) < 2e-8) | (np.isnan(root) & np.isnan(root2))
    settled &= qp == qp2
    assert settled.mean() >= 0.5
    got = gw.qp_solve(torch.as_tensor(sigma, device='cuda'), freq, eps, np.arange(len(eps)),
                      nocc, mu, greedy=greedy)
    r, z, flags, evals = (t.cpu().numpy() for t in got)
    assert np.array_equal(np.isfinite(r), np.isfinite(root))
    assert np.array_equal((flags[settled] & 1) != 0, qp[settled])
    ok = settled & np.isfinite(root)
    assert np.abs(r[ok] - root[ok]).max(initial=0.0) < 2e-8
    fixed = settled & (count == count2)
    assert (evals[fixed] == count[fixed]).mean() > 0.9
