"""The root search of one CTA per state against a serial search in plain
float64, to the bit: roots, Z, flags and evaluation counts. The kernel is
compiled without FMA contraction and the search below makes the same IEEE
operations one after another, so that nothing but the order of independent
evaluations differs.

Besides strong and smooth self-energies, ones for which w - eps - Re Sigma(w)
is rounding noise around zero: more sign changes in a window than the bracket
list holds (192, the cells are then taken again a few at a time), every cell
slow (the halving stacks at their fullest), more roots than are kept (96)."""
import math

import numpy as np
import pytest

torch = pytest.importorskip('torch')
pytestmark = pytest.mark.gpu

from mbptcode_b200 import gw                                        # noqa: E402

TIERS, HALF = (0.0, 1.5, 4.0), (0.5, 1.0, 2.0)


def cdiv(ar, ai, br, bi):
    """Smith's division on arrays."""
    with np.errstate(all='ignore'):
        big = np.abs(br) >= np.abs(bi)
        zero = big & (br == 0.0) & (bi == 0.0)
        rat = np.where(big, bi / br, br / bi)
        scl = 1.0 / np.where(big, br + bi * rat, bi + br * rat)
        re = np.where(big, (ar + ai * rat) * scl, (ar * rat + ai) * scl)
        im = np.where(big, (ai - ar * rat) * scl, (ai * rat - ar) * scl)
        return (np.where(zero, ar / np.abs(br), re), np.where(zero, ai / np.abs(bi), im))


class Serial:
    def __init__(self, z, sig, eps, xc, greedy):
        self.eps, self.xc, self.evals = eps, xc, 0
        self.ok, n = True, len(z)
        zr, zi, gr, gi = z.real.copy(), z.imag.copy(), sig.real.copy(), sig.imag.copy()
        open_ = np.ones(n, bool)
        self.z, self.a = [], []
        for m in range(n):
            if m:
                (pr, pi), (xr, xi) = self.z[-1], self.a[-1]
                dr, di = zr - pr, zi - pi
                with np.errstate(all='ignore'):
                    gr2, gi2 = cdiv(xr - gr, xi - gi, dr * gr - di * gi, dr * gi + di * gr)
                gr, gi = np.where(open_, gr2, gr), np.where(open_, gi2, gi)
            j = m
            if greedy:
                s = np.hypot(zr, zi) if m == 0 else np.hypot(gr, gi)
                s = np.where(open_ & np.isfinite(s), s, np.inf)
                if not np.isfinite(s).any():
                    if m:
                        self.ok = False
                        return
                    j = 0
                else:
                    j = int(np.argmin(s))
            self.z.append((zr[j], zi[j]))
            self.a.append((gr[j], gi[j]))
            open_[j] = False

    def f(self, w):
        """The residual at the points w, not counted."""
        w = np.atleast_1d(np.asarray(w, float))
        rr, ri = np.full(w.shape, self.a[-1][0]), np.full(w.shape, self.a[-1][1])
        with np.errstate(all='ignore'):
            for (zr, zi), (ar, ai) in zip(self.z[-2::-1], self.a[-2::-1]):
                dr, di = w - zr, np.float64(0.0) - zi
                tr, ti = dr * rr - di * ri, dr * ri + di * rr
                rr, ri = cdiv(ar, ai, 1.0 + tr, ti)
            return w - self.eps - self.xc - rr

    def bracket(self, l, r, fl, fr, found):
        a, b, fa = r, l, fr
        self.evals += 1
        for _ in range(100):
            c = 0.5 * (a + b)
            fc = self.f(c)[0]
            self.evals += 1
            if fa * fc <= 0.0:
                b = c
            else:
                a, fa = c, fc
            if abs(b - a) <= 1e-8:
                break
        w = 0.5 * (a + b)
        fw, up, down = self.f([w, w + 1e-3, w - 1e-3])
        self.evals += 1
        if not abs(fw) <= max(abs(fl), abs(fr)):
            return
        if len(found) >= 96:
            self.overflow = True
            return
        self.evals += 2
        d = (up - down) / (2.0 * 1e-3)
        found.append((w, math.nan if d == 0.0 or not np.isfinite(d) else 1.0 / d))

    def solve(self):
        """(root, Z, flags, evaluations, most brackets of a window)."""
        if not self.ok:
            return math.nan, math.nan, 8, 0, 0
        self.overflow, most = False, 0
        tier = max(k for k in range(3) if abs(self.eps) > TIERS[k] or k == 0)
        valid = lambda z, lo: np.isfinite(z) and lo < z <= 1.0
        for t in range(tier, 3):
            lo, hi = self.eps - HALF[t], self.eps + HALF[t]
            g = np.arange(150.0) * ((hi - lo) / 149) + lo
            g[0], g[-1] = lo, hi
            fg = self.f(g)
            self.evals += 150
            found, count = [], 0
            for c in range(149):
                stack = [(g[c], g[c + 1], fg[c], fg[c + 1], 6)]
                while stack:
                    l, r, fl, fr, depth = stack.pop()
                    if fl * fr < 0.0:
                        count += 1
                        self.bracket(l, r, fl, fr, found)
                    elif depth and fl != 0.0 and fr != 0.0 and fr - fl < 0.5 * (r - l):
                        m = 0.5 * (l + r)
                        fm = self.f(m)[0]
                        self.evals += 1
                        stack.append((m, r, fm, fr, depth - 1))
                        stack.append((l, m, fl, fm, depth - 1))
            most = max(most, count)
            best = None
            for k, (_, z) in enumerate(found):
                if valid(z, 0.0) and (best is None or z > found[best][1]):
                    best = k
            if best is not None and valid(found[best][1], 0.5):
                break
        else:
            t = None
        flags = 0 if t is None else 1
        root = z = math.nan
        if best is None and found:
            best = min(range(len(found)), key=lambda k: (abs(found[k][0] - self.eps), k))
        if best is None:
            flags |= 2
        else:
            root, z = found[best]
        if np.isfinite(root) and not (0.0 < z <= 1.0):
            flags |= 4
        return root, z, flags | (32 if self.overflow else 0), self.evals, most


def _states(kind, npade, seed):
    rng = np.random.default_rng(seed)
    nocc = 2
    eps = np.sort(np.concatenate([rng.uniform(-4.5, -0.3, nocc), rng.uniform(0.1, 4.5, 3)]))
    freq = 0.3 * (np.arange(npade) + 0.5) ** 1.5
    mu = -0.1
    z = mu + 1j * freq
    if kind == 'noise':
        # w - eps up to a slope of a few 1e-16 to 1e-13: rounding decides every sign
        slope = 1.0 + 10.0 ** rng.uniform(-16, -13, 5)
        sigma = slope[:, None] * z[None, :] - eps[:, None]
    else:
        amp = rng.uniform(0.02, 0.4, (5, 11)) if kind == 'strong' else rng.uniform(0, 0.02, (5, 11))
        poles = np.concatenate([rng.uniform(-6.0, -0.6, 5), rng.uniform(0.6, 6.0, 6)])
        sigma = np.einsum('pk,kw->pw', amp, 1.0 / (z[None, :] - poles[:, None]))
        sigma *= 1.0 + 0.02 * (rng.standard_normal(sigma.shape)
                               + 1j * rng.standard_normal(sigma.shape))
    return eps, nocc, mu, freq, sigma


@pytest.mark.parametrize('kind,npade,greedy,many', [
    ('smooth', 18, True, 0), ('strong', 2, True, 0), ('strong', 12, True, 0),
    ('strong', 12, False, 0), ('strong', 32, True, 0), ('noise', 2, True, 0),
    ('noise', 3, False, 193), ('noise', 3, True, 193)])
def test_bits_of_the_serial_search(kind, npade, greedy, many):
    eps, nocc, mu, freq, sigma = _states(kind, npade, npade)
    ref, most = [], 0
    for p in range(len(eps)):
        s = np.conj(sigma[p]) if p < nocc else sigma[p]
        z = mu + 1j * (-1.0 if p < nocc else 1.0) * freq
        r = Serial(z, s, eps[p], 0.0, greedy).solve()
        ref.append(r[:4])
        most = max(most, r[4])
    assert most >= many                      # the case takes the path it is here for
    got = gw.qp_solve(torch.as_tensor(sigma, device='cuda'), freq, eps, np.arange(len(eps)),
                      nocc, mu, greedy=greedy)
    roots, zs, flags, evals = (t.cpu().numpy() for t in got)
    for k, col in enumerate((roots, zs, flags, evals)):
        assert np.array_equal(col, np.array([r[k] for r in ref]), equal_nan=k < 2), k
