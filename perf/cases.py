"""The calls whose speed this repository looks after, as data and as code.

`listed()` names them, `draw(rng)` gives further ones of the same ranges,
`prepare(case, seed)` builds what a program holds before the call (factors,
spectrum, grids, on the GPU), `run(state)` makes ONE pass through the public
entry points, `work(case)` counts the bytes and operations such a pass cannot
do without, and `exact(case, seed)` computes the same outputs in plain FP64
torch.

Kinds:
  energy   rpa_correlation_energy_space_time: E_c of one geometry
  gw       gw_sweep: chi0, W, Sigma and the quasiparticle roots of the
           frontier orbitals
  chi0     chi0_sweep: chi0(i omega) of the interpolation points
  screen   proj(tau) -> chi0(i omega) -> W(i omega) - I -> W(tau): the two
           transforms around the Dyson step
  sigma    sigma_branch_sums + sigma_frequency: Sigma_pp(i omega)
  qp       qp_solve: Pade continuation and root search of every state
  adjoint  rpa_energy_and_adjoint: E_c and dE_c/d(eps, X, D)

The systems are the synthetic ISDF ones of `mbptcode_b200.synthetic`
(strongly coupled variant). A molecule's auxiliary basis is smaller than its
interpolation grid (naux < M); the benchmark configurations take naux = M.
Grids have 20 or more points, where the transforms are regularised and both
precisions are accepted.
"""
import math

import numpy as np
import torch

from mbptcode_b200 import adjoint, grids, gw, space_time
from mbptcode_b200.synthetic import EPS_OCC, EPS_VIRT, V_DECAY, V_SHIFT, synthetic_system_torch

F64 = torch.float64


def listed():
    return [
        # E_c of a water-sized molecule (10 electrons, a few hundred points per
        # atom): one point of a geometry scan, where launches count
        dict(name='energy_molecule', kind='energy', precision='fp64', n=43, nocc=5, M=888,
             naux=141, ntau=20),
        # the G0W0 frontier levels of the same size class, default precision
        dict(name='gw_molecule', kind='gw', precision='fp64', n=58, nocc=5, M=1332, naux=236,
             ntau=20),
        # one system of a learned warm start's training set or of an evGW loop
        # (n_orb in [100, 800], M = 6 n_orb, mixed precision, 24 points)
        dict(name='gw_small_mixed', kind='gw', precision='mixed', n=131, nocc=13, M=786,
             naux=786, ntau=24),
        # the mid-size configuration's layers in the default precision
        dict(name='chi0_mid', kind='chi0', precision='fp64', n=400, nocc=40, M=2400, naux=2400,
             ntau=20),
        dict(name='sigma_mid', kind='sigma', precision='fp64', n=400, nocc=40, M=2400,
             naux=2400, ntau=20, nstates=400),
        dict(name='screen_mid', kind='screen', precision='fp64', n=250, nocc=25, M=1500,
             naux=1500, ntau=20),
        # the benchmark configuration's layers in mixed precision, and a
        # ragged one below it
        dict(name='chi0_large', kind='chi0', precision='mixed', n=1200, nocc=120, M=7200,
             naux=7200, ntau=24),
        dict(name='screen_large', kind='screen', precision='mixed', n=900, nocc=90, M=5400,
             naux=5400, ntau=24),
        dict(name='sigma_ragged', kind='sigma', precision='mixed', n=701, nocc=67, M=4219,
             naux=3001, ntau=24, nstates=701),
        # the root search of every state of the benchmark configuration, and
        # of a molecule
        dict(name='qp_all_states', kind='qp', n=1200, nocc=120, npade=18),
        dict(name='qp_molecule', kind='qp', n=58, nocc=5, npade=18),
        # forward and backward: the gradient of E_c at the mid-size configuration
        dict(name='adjoint_mid', kind='adjoint', precision='default', n=400, nocc=40, M=2400,
             naux=2400, ntau=20),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['energy', 'gw', 'gw', 'chi0', 'chi0', 'screen', 'screen', 'sigma',
                       'sigma', 'qp', 'adjoint'])
    if kind == 'qp':
        n = _log(rng, 20, 1200)
        return dict(kind='qp', n=n, nocc=max(2, n // rng.randint(5, 12)),
                    npade=rng.choice([12, 16, 18, 24]))
    if kind in ('energy', 'adjoint'):
        precision = 'fp64' if kind == 'energy' else 'default'
        M = _log(rng, 192, 2400 if kind == 'energy' else 2000)
    else:
        precision = rng.choice(['fp64', 'mixed'])
        top = {('gw', 'fp64'): 1600, ('gw', 'mixed'): 3600, ('chi0', 'fp64'): 2400,
               ('chi0', 'mixed'): 7200, ('screen', 'fp64'): 1800, ('screen', 'mixed'): 5400,
               ('sigma', 'fp64'): 2400, ('sigma', 'mixed'): 4800}[kind, precision]
        M = _log(rng, 192 if precision == 'fp64' else 480, top)
    n = max(16, M // rng.randint(6, 20))
    nocc = max(2, n // rng.randint(5, 12))
    naux = M if rng.random() < 0.5 else max(64, int(M * rng.uniform(0.15, 0.9)))
    case = dict(kind=kind, precision=precision, n=n, nocc=nocc, M=M, naux=naux,
                ntau=rng.choice([20, 20, 22, 24, 24, 26]))
    if kind == 'sigma':
        case['nstates'] = n if rng.random() < 0.5 else max(1, int(n * rng.uniform(0.02, 0.9)))
    return case


# --------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed))
    return g


def _system(c, seed):
    """(X, D, eps host array): the synthetic system, D of naux columns."""
    n, nocc, M, naux = c['n'], c['nocc'], c['M'], c['naux']
    if naux == M:
        X, D, eps = synthetic_system_torch(n, nocc, M, seed=seed, variant='calibrated')
        return X, D, eps.cpu().numpy()
    g = _gen(seed)
    X = torch.linalg.qr(torch.randn(M, n, generator=g, device='cuda', dtype=F64))[0].contiguous()
    k = torch.arange(1, naux + 1, device='cuda', dtype=F64) ** V_DECAY
    D = torch.randn(M, naux, generator=g, device='cuda', dtype=F64) * k
    D += math.sqrt(V_SHIFT / naux) * torch.randn(M, naux, generator=g, device='cuda', dtype=F64)
    return X, D.contiguous(), _spectrum(n, nocc, seed)


def _spectrum(n, nocc, seed):
    rng = np.random.default_rng(seed)
    eo = np.sort(rng.uniform(*EPS_OCC, nocc))
    ev = np.sort(np.exp(rng.uniform(math.log(EPS_VIRT[0]), math.log(EPS_VIRT[1]), n - nocc)))
    return np.concatenate([eo, ev])


def _proj(X, D, eps, nocc, mu, taus):
    """proj(tau) = -2 D^T [G_occ o G_virt] D in plain FP64."""
    e = torch.as_tensor(eps - mu, device=X.device)
    out = torch.empty((len(taus), D.shape[1], D.shape[1]), dtype=F64, device=X.device)
    for k, t in enumerate(taus):
        Yo = X[:, :nocc] * torch.exp(0.5 * float(t) * e[:nocc])
        Yv = X[:, nocc:] * torch.exp(-0.5 * float(t) * e[nocc:])
        out[k] = -2.0 * (D.T @ (((Yo @ Yo.T) * (Yv @ Yv.T)) @ D))
    return out


def _screened_like(naux, taus, seed):
    """W(tau)-like stacks: symmetric, negative, dominated by a few hundred
    screened modes that decay in tau at their own rates."""
    g = _gen(seed + 77)
    r = min(naux, 384)
    Q = torch.randn(naux, r, generator=g, device='cuda', dtype=F64) / math.sqrt(naux)
    s = torch.arange(1, r + 1, device='cuda', dtype=F64)
    lam, rate = 0.5 * s ** -0.8, 0.3 + 2.0 * torch.rand(r, generator=g, device='cuda', dtype=F64)
    out = torch.empty((len(taus), naux, naux), dtype=F64, device='cuda')
    for k, t in enumerate(taus):
        torch.matmul(Q * (-lam * torch.exp(-rate * float(t))), Q.T, out=out[k])
    return out


def _sigma_model(c, seed):
    """Sigma_pp(i omega) of every state as a sum of poles at eps_i - Omega and
    eps_a + Omega, and the spectrum: what the root search reads. The plasmon
    energies Omega are log-uniform over [1, 80] Ha and a pole's weight grows
    with its Omega, which gives the sweeps' own Sigma (0.06 Ha at the lowest
    sample frequency, 0.005 at the highest), Z and scan lengths."""
    n, nocc = c['n'], c['nocc']
    eps = _spectrum(n, nocc, seed)
    mu = 0.5 * (eps[nocc - 1] + eps[nocc])
    om = np.exp(np.sort(np.random.default_rng(seed + 9).uniform(0.0, math.log(80.0), 6)))
    e, om = torch.as_tensor(eps, device='cuda'), torch.as_tensor(om, device='cuda')
    poles = torch.cat([(e[:nocc, None] - om).reshape(-1), (e[nocc:, None] + om).reshape(-1)])
    amp = torch.rand(n, poles.numel(), generator=_gen(seed + 5), device='cuda', dtype=F64)
    amp *= om.repeat(n) * (2.4 / (om.mean() * poles.numel()))
    freq = grids.pade_nodes(c['npade'])
    z = torch.as_tensor(mu + 1j * freq, device='cuda')
    sigma = amp.to(z.dtype) @ (1.0 / (z[None, :] - poles[:, None]))
    return eps, mu, freq, sigma


def _frontier(c):
    return np.arange(max(0, c['nocc'] - 10), min(c['n'], c['nocc'] + 10))


def prepare(case, seed):
    c = dict(case)
    s = dict(case=c)
    if c['kind'] == 'qp':
        eps, mu, freq, sigma = _sigma_model(c, seed)
        s.update(mu=mu, freq=freq, states=np.arange(c['n']), sigma=sigma,
                 eps=torch.as_tensor(eps, device='cuda'))
        return s
    if c['kind'] == 'energy' or c['kind'] == 'adjoint':
        X, D, eps = _system(c, seed)
        gap, span, mu = space_time.particle_hole_window(eps, c['nocc'])
        s.update(X=X, D=D, eps=eps, mu=mu,
                 grid=grids.TimeFrequencyGrid.minimax(c['ntau'], gap, span, with_sine=False))
        return s
    X, D, eps = _system(c, seed)
    axes = grids.space_time_axes(eps, c['nocc'], ntau=c['ntau'])
    s.update(axes=axes, eps=eps)
    if c['kind'] == 'screen':
        s['proj'] = _proj(X, D, eps, c['nocc'], axes.mu, axes.grid.tau_points)
        return s
    s.update(X=X, D=D)
    if c['kind'] == 'sigma':
        s['Wt'] = _screened_like(c['naux'], axes.tau_sigma, seed)
        s['states'] = np.linspace(0, c['n'] - 1, c['nstates']).astype(int)
    elif c['kind'] == 'gw':
        s['states'] = _frontier(c)
    return s


# ----------------------------------------------------------------------- pass

def run(s):
    c = s['case']
    kind = c['kind']
    if kind == 'energy':
        return space_time.rpa_correlation_energy_space_time(
            s['X'], s['D'], s['eps'], c['nocc'], s['grid'], precision=c['precision'])
    if kind == 'gw':
        r = gw.gw_sweep(s['X'], s['D'], s['eps'], c['nocc'], states=s['states'],
                        axes=s['axes'], precision=c['precision'])
        return {'roots': r['roots'], 'sigma': r['sigma'], 'e_c': r['e_c']}
    if kind == 'chi0':
        g = s['axes'].grid
        return space_time.chi0_sweep(s['X'], s['D'], s['eps'], c['nocc'], g.tau_points,
                                     g.cosft_wt, mu=s['axes'].mu, precision=c['precision'])[0]
    if kind == 'screen':
        chi0 = space_time.transform(s['proj'], s['axes'].grid.cosft_wt)
        logdet, trace, _, _ = space_time.dyson_batch(chi0, want_w=True,
                                                     precision=c['precision'])
        return {'Wt': gw.w_tau_from_frequencies(chi0, s['axes'].Ctw), 'logdet': logdet,
                'trace': trace}
    if kind == 'sigma':
        a = s['axes']
        branch = gw.sigma_branch_sums(s['X'], s['D'], s['Wt'], s['eps'], c['nocc'],
                                      a.tau_sigma, s['states'], a.mu,
                                      precision=c['precision'])
        return gw.sigma_frequency(branch, a.C, a.S)
    if kind == 'qp':
        return gw.qp_solve(s['sigma'], s['freq'], s['eps'], s['states'], c['nocc'], s['mu'])
    if kind == 'adjoint':
        return adjoint.rpa_energy_and_adjoint(s['X'], s['D'], s['eps'], c['nocc'],
                                              s['grid'])[:4]
    raise ValueError(kind)


# ----------------------------------------------------------------------- work

def work(case):
    """Multiply-adds (two operations each) with symmetric products formed on
    one side of the diagonal, and every input and output moved once."""
    c = case
    kind, n = c['kind'], c['n']
    if kind == 'qp':
        # the 150-point scan of one window, a continued fraction of npade
        # complex levels per evaluation
        return {'bytes': 16.0 * n * c['npade'] + 32.0 * n, 'flops': 150.0 * n * c['npade'] * 20}
    M, A, T = float(c['M']), float(c['naux']), c['ntau']
    inputs = 8 * (M * n + M * A + n)
    chi0 = T * (M * M * n + 2 * M * M * A + M * A * A) + 2 * T * T * A * A
    dyson = T * (A ** 3 / 3 + 2 * A ** 3 / 3)
    if kind == 'energy':
        return {'bytes': inputs, 'flops': chi0 + T * A ** 3 / 3}
    if kind == 'chi0':
        return {'bytes': inputs + 8 * T * A * A, 'flops': chi0}
    if kind == 'screen':
        return {'bytes': 16 * T * A * A, 'flops': dyson + 4 * T * T * A * A}
    ns = c.get('nstates', len(_frontier(c)))
    sigma = T * (2 * M * A * A + M * M * A + M * M * n + 2 * M * M * ns)
    if kind == 'sigma':
        return {'bytes': inputs + 8 * T * A * A, 'flops': sigma}
    if kind == 'gw':
        return {'bytes': inputs, 'flops': chi0 + dyson + 2 * T * T * A * A + sigma}
    if kind == 'adjoint':
        # the reverse sweep: E, D_bar, Pi_bar, the G branches again and their adjoints
        back = T * (2 * M * A * A + 2 * M * M * A + M * M * A + 3 * M * M * n)
        return {'bytes': 2 * inputs, 'flops': chi0 + dyson + back}
    raise ValueError(kind)


# ---------------------------------------------------------------------- exact

def _transform(w, stack):
    w = torch.as_tensor(np.asarray(w, float), device=stack.device)
    return (w @ stack.reshape(stack.shape[0], -1)).reshape((-1,) + tuple(stack.shape[1:]))


def _dyson(chi0):
    """(W - I, logdet, trace) per frequency."""
    eye = torch.eye(chi0.shape[-1], dtype=F64, device=chi0.device)
    W, ld = torch.empty_like(chi0), []
    for f in range(chi0.shape[0]):
        L = torch.linalg.cholesky(eye - 0.5 * (chi0[f] + chi0[f].T))
        ld.append(2.0 * torch.log(torch.diagonal(L)).sum())
        W[f] = torch.cholesky_inverse(L) - eye
    return W, torch.stack(ld), torch.diagonal(chi0, dim1=-2, dim2=-1).sum(-1)


def _sigma(X, D, Wt, eps, nocc, taus, states, mu, C, S):
    e = torch.as_tensor(eps - mu, device=X.device)
    Xs = X[:, torch.as_tensor(states, device=X.device)]
    lo, hi = [], []
    for k, t in enumerate(taus):
        Z = D @ Wt[k] @ D.T
        Go = (X[:, :nocc] * torch.exp(float(t) * e[:nocc])) @ X[:, :nocc].T
        lo.append((Xs * ((Go * Z) @ Xs)).sum(0))
        Gv = (X[:, nocc:] * torch.exp(-float(t) * e[nocc:])) @ X[:, nocc:].T
        hi.append(-(Xs * ((Gv * Z) @ Xs)).sum(0))
    lo, hi = torch.stack(lo), torch.stack(hi)
    C, S = (torch.as_tensor(np.asarray(m, float), device=X.device) for m in (C, S))
    return torch.complex(-0.5 * (C @ (hi + lo)), -0.5 * (S @ (hi - lo))).T.contiguous()


def _energy(logdet, trace, weights):
    w = torch.as_tensor(np.asarray(weights, float), device=logdet.device)
    return (w * (logdet + trace)).sum() / (2 * math.pi)


def _energy_of(eps, X, D, nocc, grid, mu):
    """Differentiable E_c, one tau point at a time under checkpointing."""
    from torch.utils.checkpoint import checkpoint

    def proj(eps, X, D, t):
        e = eps - mu
        Go = (X[:, :nocc] * torch.exp(t * e[:nocc])) @ X[:, :nocc].T
        Gv = (X[:, nocc:] * torch.exp(-t * e[nocc:])) @ X[:, nocc:].T
        return -2.0 * (D.T @ ((Go * Gv) @ D))

    p = torch.stack([checkpoint(proj, eps, X, D, float(t), use_reentrant=False)
                     for t in grid.tau_points])
    chi0 = _transform(grid.cosft_wt, p)
    eye = torch.eye(D.shape[1], dtype=F64, device=D.device)
    ld = [2.0 * torch.log(torch.diagonal(torch.linalg.cholesky(eye - 0.5 * (x + x.T)))).sum()
          for x in chi0]
    return _energy(torch.stack(ld), torch.diagonal(chi0, dim1=-2, dim2=-1).sum(-1),
                   grid.omega_weights)


def exact(case, seed):
    c = case
    kind = c['kind']
    if kind == 'qp':
        return None
    s = prepare(case, seed)
    if kind == 'adjoint':
        v = [torch.as_tensor(s['eps'], device='cuda').requires_grad_(True),
             s['X'].clone().requires_grad_(True), s['D'].clone().requires_grad_(True)]
        e = _energy_of(*v, c['nocc'], s['grid'], s['mu'])
        return (e.detach(),) + torch.autograd.grad(e, v)
    if kind == 'energy':
        p = _proj(s['X'], s['D'], s['eps'], c['nocc'], s['mu'], s['grid'].tau_points)
        _, ld, tr = _dyson(_transform(s['grid'].cosft_wt, p))
        return float(_energy(ld, tr, s['grid'].omega_weights))
    a = s['axes']
    if kind == 'screen':
        W, ld, tr = _dyson(_transform(a.grid.cosft_wt, s['proj']))
        return {'Wt': _transform(a.Ctw, W), 'logdet': ld, 'trace': tr}
    if kind == 'sigma':
        return _sigma(s['X'], s['D'], s['Wt'], s['eps'], c['nocc'], a.tau_sigma, s['states'],
                      a.mu, a.C, a.S)
    chi0 = _transform(a.grid.cosft_wt,
                      _proj(s['X'], s['D'], s['eps'], c['nocc'], a.mu, a.grid.tau_points))
    if kind == 'chi0':
        return chi0
    W, ld, tr = _dyson(chi0)
    return {'roots': None, 'e_c': _energy(ld, tr, a.grid.omega_weights),
            'sigma': _sigma(s['X'], s['D'], _transform(a.Ctw, W), s['eps'], c['nocc'],
                            a.tau_sigma, s['states'], a.mu, a.C, a.S)}
