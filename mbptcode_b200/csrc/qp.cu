// Batched Thiele-Pade continuation and quasiparticle root search, one CTA of
// four warps per state, FP64. Compiled without FMA contraction so that each
// complex operation rounds as the plain expression does.
//
// Per state p (MBPTcode: GW/qp_solve.py:529-558, :575-695):
//   * sample points z = mu +/- i w (occupied states on the negative branch,
//     with Sigma conjugated, qp_solve.py:659, :698-703);
//   * greedy Thiele ordering (analytic_continuation.py:34-61): start at the
//     point nearest the origin, then repeatedly add the point whose next
//     reciprocal-difference coefficient is smallest in magnitude;
//   * root of f(w) = w - eps_p - xc_p - Re Sigma(w) (qp_equation.py:1353-1393):
//     150-point scan per window (tiers +-0.5/+-1/+-2 Ha by |eps_p|), slow cells
//     halved up to 6 times, bisection to 1e-8, Z from a central difference
//     (h = 1e-3), the root of largest valid Z; Z > 1/2 ends the search.
//   * optional warm start: safeguarded Newton on the analytic derivative of
//     the continued fraction from a predicted root, accepted only when it
//     converges inside the narrowest window with Z in (1/2, 1]; otherwise
//     the scan above runs as the fallback.
//
// What bounds it: latency. One evaluation of the fraction is a chain of npade
// complex divisions (~2 us); a state needs a few hundred of them, and all
// states together are ~1e-3 of what the FP64 units could do. So the
// evaluations a state's search would make one after another are made side by
// side wherever they do not depend on one another, with the operations of
// each, the decisions and the order of the roots as the serial search has
// them (the results are the same to the bit, the evaluation count is the
// serial one):
//   * greedy ordering: one lane per sample point, each carrying its own
//     reciprocal difference forward by one step per coefficient chosen;
//   * the 150 scan points: one thread each;
//   * halving: each warp takes every fourth cell, the slow intervals of a warp
//     on a stack in shared memory, 32 midpoints per pass;
//   * bisection: one warp per bracket, the 31 midpoints of the next five
//     levels at once, then the five decisions;
//   * the residual at the root and the two of its pole strength: three lanes.
// Measured (B200, npade 18, pole-sum Sigma, whole call): 1200 states 0.20 ms,
// 58 states 0.11 ms (16.2 and 13.9 ms with one thread per state, everything in
// sequence); the worst state's chain sets the time, so the count of states hardly
// matters. A warm start saves evaluations, not time: its Newton steps are a
// chain on one thread, and a state that it does not settle scans after it
// (400 states of a mixed sweep: 98 us, 134 us warm-started with 364 accepted).
#include <cmath>

#include "common.cuh"

namespace mbpt {
namespace {

constexpr int kMaxPade = 32;
constexpr int kMaxFound = 96;
constexpr int kNOmega = 150;
constexpr double kTol = 1e-8;
constexpr int kMaxBisect = 100;
constexpr double kZStep = 1e-3;
constexpr double kZMin = 0.5;
constexpr double kSecantMin = 0.5;
constexpr int kSplitDepth = 6;
__constant__ double kTierDepth[3] = {0.0, 1.5, 4.0};
__constant__ double kTierHalf[3] = {0.5, 1.0, 2.0};

struct cplx {
  double re, im;
};

__device__ __forceinline__ cplx cmul(cplx a, cplx b) {
  return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}

// Smith's algorithm (Comm. ACM 5, 435 (1962)) for a / b.
__device__ __forceinline__ cplx cdiv(cplx a, cplx b) {
  const double ar = fabs(b.re), ai = fabs(b.im);
  if (ar >= ai) {
    if (ar == 0.0 && ai == 0.0) return {a.re / ar, a.im / ai};
    const double rat = b.im / b.re;
    const double scl = 1.0 / (b.re + b.im * rat);
    return {(a.re + a.im * rat) * scl, (a.im - a.re * rat) * scl};
  }
  const double rat = b.re / b.im;
  const double scl = 1.0 / (b.im + b.re * rat);
  return {(a.re * rat + a.im) * scl, (a.im * rat - a.re) * scl};
}

__device__ __forceinline__ bool cfinite(cplx a) { return isfinite(a.re) && isfinite(a.im); }

// A state's continued fraction: nodes in greedy order and coefficients, in
// shared memory (every thread reads the same element: a broadcast).
struct Fit {
  cplx z[kMaxPade];
  cplx a[kMaxPade];
  double eps, xc;
  int n;
};

// Re of the continued fraction at real w
__device__ __forceinline__ double pade_re(const Fit &s, double w) {
  cplx r = s.a[s.n - 1];
  for (int i = s.n - 2; i >= 0; --i) {
    const cplx d = {w - s.z[i].re, 0.0 - s.z[i].im};
    const cplx t = cmul(d, r);
    r = cdiv(s.a[i], {1.0 + t.re, t.im});
  }
  return r.re;
}

// value and w-derivative of Re of the fraction (forward mode)
__device__ void pade_re_d(const Fit &s, double w, double &val, double &der) {
  cplx r = s.a[s.n - 1], dr = {0.0, 0.0};
  for (int i = s.n - 2; i >= 0; --i) {
    const cplx d = {w - s.z[i].re, 0.0 - s.z[i].im};
    const cplx t = cmul(d, r);
    const cplx den = {1.0 + t.re, t.im};
    const cplx nr = cdiv(s.a[i], den);
    // d/dw [a / (1 + d r)] = -a (r + d dr) / den^2
    const cplx inner = cmul(d, dr);
    const cplx num = {r.re + inner.re, r.im + inner.im};
    const cplx q = cdiv(cdiv(num, den), den);
    const cplx ndr = cmul({-s.a[i].re, -s.a[i].im}, q);
    r = nr;
    dr = ndr;
  }
  val = r.re;
  der = dr.re;
}

__device__ __noinline__ double residual(const Fit &s, double w) {
  return w - s.eps - s.xc - pade_re(s, w);
}

// Z from the residuals at w + kZStep and w - kZStep
__device__ __forceinline__ double pole_strength(double up, double down) {
  const double d = (up - down) / (2.0 * kZStep);
  if (d == 0.0 || !isfinite(d)) return NAN;
  return 1.0 / d;
}

__device__ __forceinline__ bool valid_z(double z, double zmin) {
  return isfinite(z) && zmin < z && z <= 1.0;
}

constexpr unsigned kAll = 0xffffffffu;

// The lane of the smallest v (the lowest such lane), NaN and infinite values
// never; -1 when there is none.
__device__ __forceinline__ int argmin_lane(double v, int lane) {
  int j = isfinite(v) ? lane : -1;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(kAll, v, o);
    const int oj = __shfl_xor_sync(kAll, j, o);
    if (oj >= 0 && (j < 0 || ov < v || (ov == v && oj < j))) {
      v = ov;
      j = oj;
    }
  }
  return j;
}

// Thiele coefficients of state i (sample points mu +/- i w, Sigma conjugated
// on the occupied branch) into s.z / s.a, greedily ordered unless greedy is
// 0, by one whole warp; false when the greedy ordering finds no finite next
// coefficient. Lane j carries the reciprocal difference of point j against
// the nodes chosen so far.
__device__ bool build_fit(Fit &s, const double *sigma, const double *pade_freq, int npade,
                          int i, int64_t p, int64_t nocc, double mu, int greedy, int lane) {
  const double sign = p < nocc ? -1.0 : 1.0;
  const bool conj = p < nocc;
  cplx zz = {mu, 0.0}, g = {0.0, 0.0};
  bool open = lane < npade;  // not a node yet
  if (open) {
    zz.im = sign * pade_freq[lane];
    const double re = sigma[2 * (static_cast<int64_t>(i) * npade + lane)];
    const double im = sigma[2 * (static_cast<int64_t>(i) * npade + lane) + 1];
    g = {re, conj ? -im : im};
  }
  if (lane == 0) s.n = npade;
  for (int m = 0; m < npade; ++m) {
    if (m > 0 && open) {
      const cplx zp = s.z[m - 1], ap = s.a[m - 1];
      const cplx dz = {zz.re - zp.re, zz.im - zp.im};
      const cplx num = {ap.re - g.re, ap.im - g.im};
      g = cdiv(num, cmul(dz, g));
    }
    int j = m;
    if (greedy) {
      // the first node: the point nearest the origin (point 0 if none is)
      const double score = m == 0 ? hypot(zz.re, zz.im) : hypot(g.re, g.im);
      j = argmin_lane(open ? score : INFINITY, lane);
      if (j < 0 && m > 0) return false;
      if (j < 0) j = 0;
    }
    if (lane == j) {
      s.z[m] = zz;
      s.a[m] = g;
      open = false;
    }
    __syncwarp();
  }
  return true;
}

constexpr int kWarps = 4;
constexpr int kThreads = 32 * kWarps;
constexpr int kLeaf = 1 << kSplitDepth;  // sub-intervals of a cell at the last halving
// A warp pops its 32 topmost intervals and pushes at most their 64 halves, the
// less halved ones lower on the stack: at most 32 stay behind per halving
// level and 64 at the last, so 192 slots hold any sequence.
constexpr int kStackCap = 192;
// brackets held at once; a range of cells with more is taken again kFewCells
// cells at a time, which always fit
constexpr int kBracketCap = 192;
constexpr int kFewCells = kBracketCap / kLeaf;

// A sub-interval of the scan: cell, position in units of the last halving and
// halvings left, in one word; keys order as positions on the axis do.
__device__ __forceinline__ int pack(int cell, int pos, int depth) {
  return ((cell * kLeaf + pos) << 3) | depth;
}

struct Scan {
  Fit fit;
  double lo, hi, step;
  double f[kNOmega];
  double sfl[kWarps][kStackCap], sfr[kWarps][kStackCap];
  int skey[kWarps][kStackCap];
  double bfl[kBracketCap], bfr[kBracketCap];  // after the bisection: root and Z
  int bkey[kBracketCap];
  unsigned char border[kBracketCap], bkeep[kBracketCap];
  int nb, splits, evals, flag;
  // the search so far (thread 0)
  int found, best, nearest;
  double best_w, best_z, near_w, near_z;
  bool overflow, done;
};

__device__ __forceinline__ double grid_point(const Scan &c, int q) {
  return q == 0 ? c.lo : (q == kNOmega - 1 ? c.hi : static_cast<double>(q) * c.step + c.lo);
}

// end points of an interval, by the halvings that led to it
__device__ __forceinline__ void ends_of(const Scan &c, int key, double &l, double &r) {
  const int depth = key & 7, at = key >> 3, cell = at / kLeaf, pos = at % kLeaf;
  l = grid_point(c, cell);
  r = grid_point(c, cell + 1);
  for (int d = kSplitDepth - 1; d >= depth; --d) {
    const double m = 0.5 * (l + r);
    if ((pos >> d) & 1)
      l = m;
    else
      r = m;
  }
}

enum Kind { kDrop, kBracket, kSlow };

// an interval with a sign change is a bracket; one whose secant slope is
// below 1/2 is halved while halvings are left
__device__ __forceinline__ Kind kind_of(double fl, double fr, double width, int depth) {
  if (fl * fr < 0.0) return kBracket;
  if (depth == 0 || fl == 0.0 || fr == 0.0 || !(fr - fl < kSecantMin * width)) return kDrop;
  return kSlow;
}

__device__ __forceinline__ void add_bracket(Scan &c, int key, double fl, double fr) {
  const int k = atomicAdd(&c.nb, 1);
  if (k < kBracketCap) {
    c.bkey[k] = key;
    c.bfl[k] = fl;
    c.bfr[k] = fr;
  }
}

// This warp's share of the cells [c0, c1): every kWarps-th one. Brackets go to
// the list of the CTA (in no order), c.splits counts the midpoints.
__device__ void warp_cells(Scan &c, int c0, int c1, int warp, int lane) {
  double *sfl = c.sfl[warp], *sfr = c.sfr[warp];
  int *skey = c.skey[warp];
  const unsigned below = (1u << lane) - 1u;
  int splits = 0;
  for (int first = c0 + warp; first < c1; first += 32 * kWarps) {
    const int cell = first + kWarps * lane;
    Kind k = kDrop;
    double fl = 0.0, fr = 0.0;
    if (cell < c1) {
      fl = c.f[cell];
      fr = c.f[cell + 1];
      k = kind_of(fl, fr, grid_point(c, cell + 1) - grid_point(c, cell), kSplitDepth);
      if (k == kBracket) add_bracket(c, pack(cell, 0, kSplitDepth), fl, fr);
    }
    const unsigned slow = __ballot_sync(kAll, k == kSlow);
    if (k == kSlow) {
      const int at = __popc(slow & below);
      sfl[at] = fl;
      sfr[at] = fr;
      skey[at] = pack(cell, 0, kSplitDepth);
    }
    int cnt = __popc(slow);
    __syncwarp();
    while (cnt > 0) {
      const int k32 = min(cnt, 32);
      cnt -= k32;
      const bool live = lane < k32;
      Kind kl = kDrop, kr = kDrop;
      double fm = 0.0, ifl = 0.0, ifr = 0.0;
      int lkey = 0, rkey = 0;
      if (live) {
        ifl = sfl[cnt + lane];
        ifr = sfr[cnt + lane];
        const int key = skey[cnt + lane];
        const int depth = (key & 7) - 1;  // of the halves
        double l, r;
        ends_of(c, key, l, r);
        const double m = 0.5 * (l + r);
        fm = residual(c.fit, m);
        lkey = ((key >> 3) << 3) | depth;
        rkey = (((key >> 3) + (1 << depth)) << 3) | depth;
        kl = kind_of(ifl, fm, m - l, depth);
        kr = kind_of(fm, ifr, r - m, depth);
        if (kl == kBracket) add_bracket(c, lkey, ifl, fm);
        if (kr == kBracket) add_bracket(c, rkey, fm, ifr);
      }
      splits += k32;
      __syncwarp();  // every pop before the pushes
      const unsigned ml = __ballot_sync(kAll, kl == kSlow), mr = __ballot_sync(kAll, kr == kSlow);
      int at = cnt + __popc(ml & below) + __popc(mr & below);
      if (kl == kSlow) {
        sfl[at] = ifl;
        sfr[at] = fm;
        skey[at] = lkey;
        ++at;
      }
      if (kr == kSlow) {
        sfl[at] = fm;
        sfr[at] = ifr;
        skey[at] = rkey;
      }
      cnt += __popc(ml) + __popc(mr);
      __syncwarp();
    }
  }
  if (lane == 0) atomicAdd(&c.splits, splits);
}

// Bracket k by one warp: bisection from its right end a as the reference
// refines a bracket, five levels of midpoints at a time (lane t holds node t
// of the binary tree below (a, b): bit by bit from its leading one, 0 moves b
// to the midpoint, 1 moves a). Leaves the root, Z and whether it is one (a
// pole's residual grows); returns the residuals a serial search evaluates.
__device__ int solve_bracket(Scan &c, int k, int lane) {
  double l, r;
  ends_of(c, c.bkey[k], l, r);
  const double fl = c.bfl[k], fr = c.bfr[k];
  __syncwarp();
  double w = l;
  int evals = 0;
  if (l != r) {
    double a = r, b = l, fa = fr;
    evals = 1;  // fa
    int it = 0;
    bool stop = false;
    while (!stop) {
      double ta = a, tb = b;
      for (int lev = 30 - __clz(lane | 1); lev >= 0; --lev) {
        const double m = 0.5 * (ta + tb);
        if ((lane >> lev) & 1)
          ta = m;
        else
          tb = m;
      }
      const double f = residual(c.fit, 0.5 * (ta + tb));
      int node = 1;
#pragma unroll 1
      for (int lev = 0; lev < 5 && !stop; ++lev) {
        const double mid = 0.5 * (a + b);
        const double fc = __shfl_sync(kAll, f, node);
        ++evals;
        if (fa * fc <= 0.0) {
          b = mid;
          node = 2 * node;
        } else {
          a = mid;
          fa = fc;
          node = 2 * node + 1;
        }
        stop = fabs(b - a) <= kTol || ++it >= kMaxBisect;
      }
    }
    w = 0.5 * (a + b);
  }
  // lane 1: the residual at the root, lanes 2 and 3: its two neighbours
  const double f = residual(c.fit, lane == 2 ? w + kZStep : (lane == 3 ? w - kZStep : w));
  const double fw = __shfl_sync(kAll, f, 1);
  const double up = __shfl_sync(kAll, f, 2), down = __shfl_sync(kAll, f, 3);
  bool keep = true;
  if (l != r) {
    ++evals;  // fw
    keep = fabs(fw) <= fmax(fabs(fl), fabs(fr));
  }
  if (lane == 0) {
    c.bfl[k] = w;
    c.bfr[k] = pole_strength(up, down);
    c.bkeep[k] = keep;
  }
  return evals;
}

// flags: 1 quasiparticle, 2 no root, 4 Z outside (0,1], 8 Pade failed,
//        16 warm start accepted, 32 bracket list overflow
__global__ void __launch_bounds__(kThreads) pade_qp_kernel(
    const double *sigma, const double *pade_freq, int npade, const double *eps_anchor,
    const double *xc, const int64_t *states, int nstates, int64_t nocc, double mu, int greedy,
    const double *warm, double *roots, double *zout, int *flags, int *evals) {
  __shared__ Scan c;
  const int i = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t p = states[i];
  if (warp == 0) {
    const bool ok = build_fit(c.fit, sigma, pade_freq, npade, i, p, nocc, mu, greedy, lane);
    if (lane == 0) {
      c.fit.eps = eps_anchor[p];
      c.fit.xc = xc ? xc[i] : 0.0;
      c.evals = 0;
      c.flag = ok ? 0 : 8;
    }
  }
  __syncthreads();
  if (c.flag & 8) {
    if (tid == 0) {
      roots[i] = NAN;
      zout[i] = NAN;
      flags[i] = 8;
      evals[i] = 0;
    }
    return;
  }
  const Fit &s = c.fit;
  const double a = s.eps;
  int tier = 0;
  for (int k = 0; k < 3; ++k)
    if (fabs(a) > kTierDepth[k]) tier = k;

  // ---- warm start: safeguarded Newton inside the narrowest window ----
  if (warm) {
    if (tid == 0) {
      const double lo = a - kTierHalf[tier], hi = a + kTierHalf[tier];
      double w = warm[i];
      bool conv = false;
      if (isfinite(w) && w > lo && w < hi) {
        for (int it = 0; it < 30; ++it) {
          double pv, pd;
          pade_re_d(s, w, pv, pd);
          c.evals++;
          const double f = w - s.eps - s.xc - pv;
          const double fp = 1.0 - pd;
          if (!(fp > 0.0) || !isfinite(f)) break;
          double step = f / fp;
          if (fabs(step) > 0.1) step = copysign(0.1, step);
          w -= step;
          if (!(w > lo && w < hi)) break;
          if (fabs(step) < 1e-12 * fmax(1.0, fabs(w))) {
            conv = true;
            break;
          }
        }
      }
      if (conv) {
        const double up = residual(s, w + kZStep);
        const double z = pole_strength(up, residual(s, w - kZStep));
        c.evals += 2;
        if (valid_z(z, kZMin)) {
          roots[i] = w;
          zout[i] = z;
          flags[i] = 1 | 16;
          evals[i] = c.evals;
          c.flag = 16;
        }
      }
    }
    __syncthreads();
    if (c.flag & 16) return;
  }

  // ---- graphical scan ----
  if (tid == 0) {
    c.overflow = false;
    c.done = false;
  }
  for (int t = tier; t < 3; ++t) {
    if (tid == 0) {
      c.lo = a - kTierHalf[t];
      c.hi = a + kTierHalf[t];
      c.step = (c.hi - c.lo) / (kNOmega - 1);
      c.found = 0;
      c.best = c.nearest = -1;
      c.evals += kNOmega;
    }
    __syncthreads();
    for (int q = tid; q < kNOmega; q += kThreads) c.f[q] = residual(s, grid_point(c, q));
    int span = kNOmega - 1;
    for (int c0 = 0; c0 < kNOmega - 1;) {
      const int c1 = min(c0 + span, kNOmega - 1);
      if (tid == 0) c.nb = c.splits = 0;
      __syncthreads();
      warp_cells(c, c0, c1, warp, lane);
      __syncthreads();
      const int nb = c.nb;
      if (nb > kBracketCap) {  // uniform; kFewCells cells cannot get here
        span = kFewCells;
        __syncthreads();
        continue;
      }
      // places of the brackets along the axis
      for (int k = tid; k < nb; k += kThreads) {
        int at = 0;
        for (int q = 0; q < nb; ++q) at += c.bkey[q] < c.bkey[k];
        c.border[at] = static_cast<unsigned char>(k);
      }
      int ev = 0;
      for (int k = warp; k < nb; k += kWarps) ev += solve_bracket(c, k, lane);
      if (lane == 0 && ev) atomicAdd(&c.evals, ev);
      __syncthreads();
      if (tid == 0) {
        c.evals += c.splits;
        for (int q = 0; q < nb; ++q) {
          const int k = c.border[q];
          if (!c.bkeep[k]) continue;
          if (c.found >= kMaxFound) {
            c.overflow = true;
            continue;
          }
          c.evals += 2;  // its pole strength
          const double w = c.bfl[k], z = c.bfr[k];
          if (valid_z(z, 0.0) && (c.best < 0 || z > c.best_z)) {
            c.best = c.found;
            c.best_w = w;
            c.best_z = z;
          }
          if (c.nearest < 0 || fabs(w - a) < fabs(c.near_w - a)) {
            c.nearest = c.found;
            c.near_w = w;
            c.near_z = z;
          }
          c.found++;
        }
      }
      c0 = c1;
    }
    if (tid == 0 && c.best >= 0 && valid_z(c.best_z, kZMin)) c.done = true;
    __syncthreads();
    if (c.done) break;
  }
  if (tid == 0) {
    int fl = 0;
    double root = NAN, zr = NAN;
    if (c.done) fl |= 1;
    if (c.best >= 0) {
      root = c.best_w;
      zr = c.best_z;
    } else if (c.found > 0) {
      root = c.near_w;
      zr = c.near_z;
    } else {
      fl |= 2;
    }
    if (isfinite(root) && !(0.0 < zr && zr <= 1.0)) fl |= 4;
    if (c.overflow) fl |= 32;
    roots[i] = root;
    zout[i] = zr;
    flags[i] = fl;
    evals[i] = c.evals;
  }
}

// out[i, q] = Re Sigma_c(query[i, q]) of state i's continuation (NaN when its
// Pade construction failed); one CTA per state, its queries over the threads
__global__ void __launch_bounds__(kThreads) pade_eval_kernel(
    const double *sigma, const double *pade_freq, int npade, const int64_t *states, int nstates,
    int64_t nocc, double mu, int greedy, const double *query, int nq, double *out) {
  __shared__ Fit s;
  __shared__ bool ok;
  const int i = blockIdx.x, lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    const bool built =
        build_fit(s, sigma, pade_freq, npade, i, states[i], nocc, mu, greedy, lane);
    if (lane == 0) ok = built;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nq; q += kThreads) {
    const int64_t o = static_cast<int64_t>(i) * nq + q;
    out[o] = ok ? pade_re(s, query[o]) : NAN;
  }
}

}  // namespace

int launch_pade_eval(const double *sigma, const double *pade_freq, int npade,
                     const int64_t *states, int nstates, int64_t nocc, double mu, int greedy,
                     const double *query, int nq, double *out, cudaStream_t st) {
  if (npade < 2 || npade > kMaxPade || nstates < 0 || nq < 1) return MBPT_ERR_SHAPE;
  if (nstates == 0) return MBPT_OK;
  count_launch();
  pade_eval_kernel<<<nstates, kThreads, 0, st>>>(sigma, pade_freq, npade, states, nstates, nocc,
                                                 mu, greedy, query, nq, out);
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

int launch_pade_qp(const double *sigma, const double *pade_freq, int npade,
                   const double *eps_anchor, const double *xc, const int64_t *states,
                   int nstates, int64_t nocc, double mu, int greedy, const double *warm,
                   double *roots, double *z, int *flags, int *evals, cudaStream_t st) {
  if (npade < 2 || npade > kMaxPade || nstates < 0) return MBPT_ERR_SHAPE;
  if (nstates == 0) return MBPT_OK;
  count_launch();
  pade_qp_kernel<<<nstates, kThreads, 0, st>>>(sigma, pade_freq, npade, eps_anchor, xc, states,
                                               nstates, nocc, mu, greedy, warm, roots, z, flags,
                                               evals);
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

}  // namespace mbpt
