// Small FP64 kernels of the adjoint and of the Dyson step (its triangular
// inverse and the FP64 <-> TF32-pair conversions of its tensor-core products).
#include <cmath>

#include "internal.h"

namespace mbpt {
namespace {

inline int blocks(int64_t n) {
  int64_t b = (n + 255) / 256;
  return static_cast<int>(b > 148 * 32 ? 148 * 32 : (b < 1 ? 1 : b));
}

// a_f <- -(w_f / 2pi) a_f^T for each W - I slice: chi0_bar of the dRPA energy
// (W - I is symmetric here, the mirrored output of the Dyson step).
__global__ void chi0_bar_seed_kernel(double *a, int64_t n, const double *w) {
  double *m = a + static_cast<int64_t>(blockIdx.y) * n * n;
  const double s = -w[blockIdx.y] / (2.0 * 3.14159265358979323846);
  const int64_t total = n * n;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    m[i] *= s;
}

// a[i] = the sum of a[i + p n] over the parts p, i < n
__global__ void sum_parts_kernel(double *a, int64_t n, int parts) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double s = a[i];
#pragma unroll 4
    for (int p = 1; p < parts; ++p) s += a[i + p * n];
    a[i] = s;
  }
}

// out = (in + in^T) / 2 for each n x n slice, `in` the sum of `parts` arrays
// part_stride apart: one 32 x 32 tile and its mirror per block, both halves
// through shared memory so that every access runs along rows
__global__ void sym_half_kernel(const double *__restrict__ in, double *__restrict__ out,
                                int64_t n, int parts, int64_t part_stride) {
  __shared__ double lo[32][33], up[32][33];
  if (blockIdx.x < blockIdx.y) return;
  const int64_t base = static_cast<int64_t>(blockIdx.z) * n * n;
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * 32, c0 = static_cast<int64_t>(blockIdx.x) * 32;
  const int x = threadIdx.x;
  // eight loads in flight per thread (one row of both tiles at a time: 31 us
  // for one slice of n = 2400, now 24)
  double u[4] = {}, l[4] = {};
  auto add = [&](const double *a) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = threadIdx.y + 8 * q;
      if (r0 + k < n && c0 + x < n) u[q] += a[(r0 + k) * n + c0 + x];
      if (c0 + k < n && r0 + x < n) l[q] += a[(c0 + k) * n + r0 + x];
    }
  };
  add(in + base);
#pragma unroll 2
  for (int p = 1; p < parts; ++p) add(in + p * part_stride + base);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    up[threadIdx.y + 8 * q][x] = u[q];
    lo[threadIdx.y + 8 * q][x] = l[q];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    if (r0 + k < n && c0 + x < n)
      out[base + (r0 + k) * n + c0 + x] = 0.5 * (up[k][x] + lo[x][k]);
    if (r0 != c0 && c0 + k < n && r0 + x < n)
      out[base + (c0 + k) * n + r0 + x] = 0.5 * (lo[k][x] + up[x][k]);
  }
}

// X_bar[:, occ] += 2 GoX w, X_bar[:, virt] += 2 GvX u;
// eps_bar[i] += tau w_i sum_b X[b,i] GoX[b,i], eps_bar[a] -= tau u_a sum_b X[b,a] GvX[b,a]
__global__ void xbar_kernel(const double *GoX, const double *GvX, const double *X, int64_t M,
                            int64_t n, int64_t nocc, const double *eps, double mu, double tau,
                            double *X_bar, double *eps_bar) {
  const int64_t c = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;
  __shared__ double part[8][33];
  const int64_t nv = n - nocc;
  double s = 0.0;
  double f = 0.0;
  if (c < n) {
    const bool occ = c < nocc;
    f = occ ? exp((eps[c] - mu) * tau) : exp(-(eps[c] - mu) * tau);
    const int64_t r0 = static_cast<int64_t>(blockIdx.y) * 256;
    const int64_t r1 = min(r0 + 256, M);
    for (int64_t r = r0 + threadIdx.y; r < r1; r += 8) {
      const double g = occ ? GoX[r * nocc + c] : GvX[r * nv + (c - nocc)];
      X_bar[r * n + c] += 2.0 * g * f;
      s += X[r * n + c] * g;
    }
  }
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < n) {
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += part[k][threadIdx.x];
    const double sign = c < nocc ? 1.0 : -1.0;
    atomicAdd(eps_bar + c, sign * tau * f * t);
  }
}

// restore a symmetric matrix from its row-major lower triangle
__global__ void mirror_kernel(double *a, int64_t n) {
  const int64_t total = n * n;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / n, c = i % n;
    if (r < c) a[i] = a[c * n + r];
  }
}

// log|det| and sign from an LU factor with 1-based pivots (column-major view)
__global__ void lu_logdet_kernel(const double *LU, const int *piv, int64_t n, double *logdet,
                                 int *sign) {
  __shared__ double part[256];
  __shared__ int neg[256];
  double s = 0.0;
  int ng = 0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double d = LU[i * n + i];
    s += log(fabs(d));
    if (d < 0.0) ng ^= 1;
    if (piv[i] != i + 1) ng ^= 1;
  }
  part[threadIdx.x] = s;
  neg[threadIdx.x] = ng;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      part[threadIdx.x] += part[threadIdx.x + w];
      neg[threadIdx.x] ^= neg[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *logdet = part[0];
    *sign = neg[0] ? -1 : 1;
  }
}

// diag[f * n + i] <-> a_f[i, i]
__global__ void diag_kernel(double *a, int64_t n, double *diag, bool save) {
  double *m = a + static_cast<int64_t>(blockIdx.y) * n * n;
  double *d = diag + static_cast<int64_t>(blockIdx.y) * n;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    if (save)
      d[i] = m[i * n + i];
    else
      m[i * n + i] = d[i];
  }
}

// Inverts the nb x nb diagonal blocks of column-major lower-triangular n x n
// matrices (blockIdx.y, one after the other; the pair arrays ldp^2 apart) in
// place, one CTA per block: the block is staged row-major in shared
// memory and inverted row by row (forward substitution against the rows
// already inverted), so the block never leaves the SM until it is done.
// With c_hi set, the inverted blocks go out as TF32 pairs instead, in two
// layouts of the padded (ldp) pair arrays: rows of L^-1 (r_*) and columns of
// L^-1 as rows (c_*), zeros above the diagonal included; A keeps the factor.
// The row recursion's dot products are split over kDiagParts threads per
// column (partial sums combined by warp shuffles), and the block is stored
// with a padded row stride so the parts' reads fall in different banks.
constexpr int kDiagParts = 4;

__global__ void trtri_diag_blocks_kernel(double *A, int64_t n, int nb, float *c_hi, float *c_lo,
                                         float *r_hi, float *r_lo, int64_t ldp) {
  extern __shared__ double s[];  // m x m row-major block (stride m + 1), then one row of L
  const int64_t lda = n, pairs = blockIdx.y * ldp * ldp;
  A += blockIdx.y * n * n;
  const int64_t off = static_cast<int64_t>(blockIdx.x) * nb;
  const int m = static_cast<int>(min(static_cast<int64_t>(nb), n - off));
  const int ls = m + 1;
  double *row = s + m * ls;
  for (int idx = threadIdx.x; idx < m * m; idx += blockDim.x) {
    const int r = idx / m, c = idx % m;
    s[r * ls + c] = r >= c ? A[(off + c) * lda + off + r] : 0.0;
  }
  __syncthreads();
  const int j = threadIdx.x / kDiagParts, part = threadIdx.x % kDiagParts;
  for (int i = 0; i < m; ++i) {
    for (int k = threadIdx.x; k <= i; k += blockDim.x) row[k] = s[i * ls + k];
    __syncthreads();
    const double inv = 1.0 / row[i];
    // row i of L^-1: (L^-1)_ij = -(sum_{j<=k<i} L_ik (L^-1)_kj) / L_ii
    double acc = 0.0;
    if (j < i)
      for (int k = j + part; k < i; k += kDiagParts) acc = fma(row[k], s[k * ls + j], acc);
#pragma unroll
    for (int d = 1; d < kDiagParts; d <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if (part == 0 && j <= i) s[i * ls + j] = j == i ? inv : -acc * inv;
    __syncthreads();
  }
  if (c_hi) {
    for (int idx = threadIdx.x; idx < m * m; idx += blockDim.x) {
      const int r = idx / m, c = idx % m;
      const double x = s[r * ls + c];
      const float h = to_tf32(static_cast<float>(x));
      const float l = to_tf32(static_cast<float>(x - static_cast<double>(h)));
      r_hi[pairs + (off + r) * ldp + off + c] = h;
      r_lo[pairs + (off + r) * ldp + off + c] = l;
      c_hi[pairs + (off + c) * ldp + off + r] = h;
      c_lo[pairs + (off + c) * ldp + off + r] = l;
    }
    return;
  }
  for (int idx = threadIdx.x; idx < m * m; idx += blockDim.x) {
    const int r = idx / m, c = idx % m;
    if (r >= c) A[(off + c) * lda + off + r] = s[r * ls + c];
  }
}

// dst (rows_p x k_p row-major TF32 hi/lo pairs, zero padded) of the logical
// rows x k FP64 matrix X(r, c) = src[r * rs + c * cs], through a 32 x 33
// shared tile so that the global reads run along whichever stride is 1.
// The pair is split from the FP64 value: hi = tf32(x), lo = tf32(x - hi).
// Matrices over blockIdx.z (src and pairs src_stride and rows_p k_p apart);
// lower: only the 32 x 32 tiles on and below the diagonal.
__global__ void strided_to_tf32_kernel(const double *__restrict__ src, int64_t rows, int64_t k,
                                       int64_t rs, int64_t cs, int64_t src_stride, float *hi,
                                       float *lo, int64_t rows_p, int64_t k_p, bool lower) {
  __shared__ double tile[32][33];
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * 32;
  const int64_t c0 = static_cast<int64_t>(blockIdx.x) * 32;
  if (lower && c0 > r0) return;
  src += blockIdx.z * src_stride;
  hi += blockIdx.z * rows_p * k_p;
  lo += blockIdx.z * rows_p * k_p;
  const bool col_unit = cs == 1;
  for (int a = threadIdx.y; a < 32; a += blockDim.y) {
    const int64_t r = col_unit ? r0 + a : r0 + threadIdx.x;
    const int64_t c = col_unit ? c0 + threadIdx.x : c0 + a;
    const double v = (r < rows && c < k) ? src[r * rs + c * cs] : 0.0;
    if (col_unit)
      tile[a][threadIdx.x] = v;
    else
      tile[threadIdx.x][a] = v;
  }
  __syncthreads();
  for (int a = threadIdx.y; a < 32; a += blockDim.y) {
    const int64_t r = r0 + a, c = c0 + threadIdx.x;
    if (r < rows_p && c < k_p) {
      const double x = tile[a][threadIdx.x];
      const float h = to_tf32(static_cast<float>(x));
      hi[r * k_p + c] = h;
      lo[r * k_p + c] = to_tf32(static_cast<float>(x - static_cast<double>(h)));
    }
  }
}

__global__ void identity_kernel(double *a, int64_t n, double diag_shift, bool set) {
  const int64_t total = n * n;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / n, c = i % n;
    if (set)
      a[i] = (r == c) ? 1.0 : 0.0;
    else if (r == c)
      a[i] += diag_shift;
  }
}

// ---------------------------------------------------------- self-energy adjoint
// Xs[r, s] = X[r, states[s]] scaled by the branch adjoints of one tau point:
// Xl = Xs diag(sl), Xg = Xs diag(sg) (MBPTcode gradients/rpa/space_time_adjoint.py:846-853,
// there as the weights c of the bra slice)
__global__ void sigma_back_gather_kernel(const double *__restrict__ X, int64_t M, int64_t n,
                                         const int64_t *__restrict__ states, int64_t S,
                                         const double *__restrict__ sl,
                                         const double *__restrict__ sg, double *Xs, double *Xl,
                                         double *Xg) {
  const int64_t total = M * S;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / S, c = i % S;
    const double x = X[r * n + states[c]];
    Xs[i] = x;
    Xl[i] = x * sl[c];
    Xg[i] = x * sg[c];
  }
}

// The elementwise reverse of Sigma^<_s = x_s^T (Go o Zt) x_s and
// Sigma^>_s = -x_s^T (Gv o Zt) x_s with Al = sum_s sl_s x_s x_s^T and
// Ag = sum_s sg_s x_s x_s^T, in place:
//   zt <- Zt_bar = go al - gv ag,  al <- Go_bar = zt al,  ag <- Gv_bar = -zt ag,
//   go <- L = go zt,               gv <- H = gv zt
__global__ void sigma_back_hadamard_kernel(double *go, double *gv, double *zt, double *al,
                                           double *ag, int64_t total) {
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double o = go[i], v = gv[i], z = zt[i], a = al[i], g = ag[i];
    zt[i] = o * a - v * g;
    al[i] = z * a;
    ag[i] = -z * g;
    go[i] = o * z;
    gv[i] = v * z;
  }
}

// X_bar[r, states[s]] += scale * T[r, s] (a state listed twice adds twice)
__global__ void scatter_cols_kernel(const double *__restrict__ T, int64_t M, int64_t S,
                                    const int64_t *__restrict__ states, double scale,
                                    double *X_bar, int64_t n) {
  const int64_t total = M * S;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / S, c = i % S;
    atomicAdd(X_bar + r * n + states[c], scale * T[i]);
  }
}

// ------------------------------------------------ batched blocked Cholesky
// One 128-column step of the left-looking Cholesky of a batch of column-major
// n x n matrices (the lower factor, as cuSOLVER's lower-fill potrf leaves it;
// the strict upper triangle is never written).
constexpr int kCholNb = 128;
constexpr int kCholStride = kCholNb + 4;

// One CTA (512 threads) per matrix: the updated diagonal block (the top nbj
// rows of P_f, padded to whole sub-blocks with the identity) is factorised and
// inverted in shared memory, by 32-column sub-blocks k:
//  A. warp 0 factorises the 32 x 32 diagonal sub-block in registers (lane r
//     holds row r) as U D^-1 U^T without square roots, so that the chain from
//     pivot to pivot is one reciprocal, two shuffles and two FP64 operations;
//     the rows' entries below a pivot are read back from shared memory as
//     broadcasts; L_kk = U D^-1/2. Warp 1 follows it eight pivots behind
//     with the inverse X_kk (lane c holds column c). Meanwhile the other warps
//     of its schedulers finish the previous step: the rank-32 update of the
//     columns past this sub-block, T_ki = sum_{i <= j < k} L_kj X_ji for
//     every i < k, and the stores of what is final (in step 0, the loads of
//     the later columns);
//  B. L_ik = A_ik X_kk^T for the rows below, X_ki = -X_kk T_ki beside it;
//  C. the update of the next sub-block's 32 columns.
// B, C and the work beside A run as FP64 tensor-core products (m8n8k4) of 8-row
// strips, one strip a warp.
// The lower factor goes into A_f's diagonal block (lower triangle and
// diagonal only), X = L^-1 into Linv_f (column-major, ld kCholNb, zeros above
// the diagonal). The diagonal is sqrt(pivot), the scaling of the column below
// it rsqrt(pivot) (within an ulp of LAPACK's 1 / sqrt). A pivot that is not
// positive records info_f = its global column + 1 (the first one only), as
// potrf does; the factor of that matrix is then not meaningful.
// What bounds it: latency, 128 dependent pivots of about 230 cycles each.
// Measured (B200, 20 matrices, time of the launch): 128 columns 36.9 us, 64
// columns 18.4 us, 13 columns 11.0 us; 90, 84 and 80 us with the square root
// on the pivots' chain, 4 x 4 register tiles for the block products (34 000
// of 170 000 cycles in X alone) and every block padded to 128.
// Shared memory: s (128 x kCholStride: L in the lower triangle, the
// off-diagonal blocks of X transposed in the upper one, X[r][c] at s[c][r]),
// the diagonals of L and of X, the four X_kk dense, the sub-block's U by
// columns, and T. All strides are 4 modulo 16, which keeps a fragment load's
// half warp (four rows, four k) in sixteen different 8-byte banks whichever
// index runs along memory.
constexpr int kCholSub = 32;
constexpr int kCholXStride = kCholSub + 4;
constexpr int kCholSmemDoubles = kCholNb * kCholStride + 3 * kCholNb +
                                 (kCholNb / kCholSub) * kCholSub * kCholXStride +
                                 kCholSub * kCholXStride + 3 * kCholSub * kCholXStride;

// acc (8 x 32, four 8 x 8 blocks) += A B^T over 4 ksteps K columns: A(r, k) at
// a[r ar + k ak], B(c, k) at b[c br + k bk]; blocks from nblk on are left out
__device__ __forceinline__ void strip_product(double (&acc)[4][2], const double *a, int ar, int ak,
                                              const double *b, int br, int bk, int ksteps,
                                              int nblk, int lane) {
  const double *pa = a + (lane >> 2) * ar + (lane & 3) * ak;
  const double *pb = b + (lane >> 2) * br + (lane & 3) * bk;
#pragma unroll 2
  for (int q = 0; q < ksteps; ++q) {
    const double x = pa[4 * q * ak];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < nblk) {
        const double y = pb[8 * j * br + 4 * q * bk];
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(acc[j][0]), "+d"(acc[j][1])
            : "d"(x), "d"(y));
      }
  }
}

__global__ void __launch_bounds__(512) chol_diag_block_kernel(
    const double *__restrict__ P, int64_t m, int nbj, double *A, int64_t n, int64_t j0,
    double *__restrict__ Linv, int *info) {
  extern __shared__ __align__(16) double sm[];
  constexpr int ST = kCholStride, XS = kCholXStride, NB = kCholNb, SB = kCholSub;
  double *s = sm;
  double *diag = s + NB * ST;                 // L_cc
  double *xdiag = diag + NB;                  // X_cc = rsqrt(pivot)
  double *pinv = xdiag + NB;                  // 1 / pivot
  double *xd = pinv + NB;                     // X_kk dense, [k][r][c]
  double *ut = xd + (NB / SB) * SB * XS;      // U of the sub-block by columns, [c][r]
  double *tb = ut + SB * XS;                  // T_ki, [i][r][c]
  __shared__ double rsx[SB];
  __shared__ int bad;
  const int f = blockIdx.x, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int nsub = (nbj + SB - 1) / SB, nr = nsub * SB;
  const double *p = P + static_cast<int64_t>(f) * m * nbj;
  double *a = A + static_cast<int64_t>(f) * n * n;
  if (tid == 0) bad = -1;
  // columns [c0, c1) of the tile padded with the identity, zeros above the
  // diagonal, by `count` threads (this one the id-th); eight independent loads
  // in flight per thread before any store
  auto load_columns = [&](int c0, int c1, int id, int count) {
    for (int i0 = c0 * NB + id; i0 < c1 * NB; i0 += 8 * count) {
      double v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + u * count;
        const int c = i / NB, r = i % NB;
        v[u] = 0.0;
        if (c < c1 && r >= c)
          v[u] = (r < nbj && c < nbj) ? p[static_cast<int64_t>(c) * m + r] : (r == c ? 1.0 : 0.0);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + u * count;
        if (i < c1 * NB) s[(i % NB) * ST + i / NB] = v[u];
      }
    }
  };
  // L's column block k and X's row block k, by `count` warps (this one the
  // id-th)
  double *ld = Linv + static_cast<int64_t>(f) * NB * NB;
  auto store_block = [&](int k, int id, int count) {
    for (int c = k * SB + id; c < min(nbj, (k + 1) * SB); c += count)
      for (int r = k * SB + lane; r < nbj; r += 32)
        if (r >= c) a[(j0 + c) * n + j0 + r] = r == c ? diag[c] : s[r * ST + c];
    const int r = k * SB + lane;
    if (r < nbj)
      for (int c = id; c < nbj; c += count) {
        double x = 0.0;
        if (r == c)
          x = xdiag[c];
        else if (r > c)
          x = c / SB == k ? xd[(k * SB + lane) * XS + c % SB] : s[c * ST + r];
        ld[c * NB + r] = x;
      }
  };
  load_columns(0, SB, tid, 512);
  __syncthreads();
  // rows [r0, r0 + 8) of the trailing triangle, 32 columns from c0, minus the
  // panel in columns [b, b + 32)
  auto update = [&](int r0, int c0, int b) {
    const int nblk = min(4, (r0 - c0) / 8 + 1);  // blocks on and below the diagonal
    double acc[4][2] = {};
    strip_product(acc, s + r0 * ST + b, ST, 1, s + c0 * ST + b, ST, 1, SB / 4, nblk, lane);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < nblk) {
        double *at = s + (r0 + g) * ST + c0 + 8 * j + 2 * t;
        at[0] -= acc[j][0];
        at[1] -= acc[j][1];
      }
  };
  // rows [8 q, 8 q + 8) of T_ki (k the current sub-block)
  auto t_strip = [&](int k, int i, int q) {
    double acc[4][2] = {};
    for (int j = i; j < k; ++j) {
      const double *l = s + (k * SB + 8 * q) * ST + j * SB;
      if (j == i)
        strip_product(acc, l, ST, 1, xd + i * SB * XS, 1, XS, SB / 4, 4, lane);
      else
        strip_product(acc, l, ST, 1, s + i * SB * ST + j * SB, ST, 1, SB / 4, 4, lane);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      double *at = tb + (i * SB + 8 * q + g) * XS + 8 * j + 2 * t;
      at[0] = acc[j][0];
      at[1] = acc[j][1];
    }
  };
  for (int k = 0; k < nsub; ++k) {
    const int b = k * SB;
    double *xk = xd + k * SB * XS;
    if (warp == 0) {
      double v[SB];
#pragma unroll
      for (int j = 0; j < SB; ++j) v[j] = s[(b + lane) * ST + b + j];
      // right-looking in registers: entries of a lane above the diagonal
      // are never read by another lane
      double piv = 0.0;
#pragma unroll
      for (int c = 0; c < SB; ++c) {
        const double u = v[c];
        ut[c * XS + lane] = u;
        const double d = __shfl_sync(0xffffffffu, u, c);
        const double nxt = c + 1 < SB ? __shfl_sync(0xffffffffu, u, c + 1 < SB ? c + 1 : c) : 0.0;
        const double inv = 1.0 / d;
        if (lane == c) {
          piv = d;
          diag[b + c] = d;
          pinv[b + c] = inv;
        }
        const double w = -u * inv;
        if (c + 1 < SB) v[c + 1 < SB ? c + 1 : c] = fma(w, nxt, v[c + 1 < SB ? c + 1 : c]);
        __syncwarp();
#pragma unroll
        for (int j = c + 2; j < SB; ++j) v[j] = fma(w, ut[c * XS + j], v[j]);
        // eight more columns for warp 1 (a barrier of these two warps)
        if (c % 8 == 7) asm volatile("bar.arrive %0, 64;" ::"r"(1 + c / 8) : "memory");
      }
      const double rs = rsqrt(piv);
      xdiag[b + lane] = rs;
      const unsigned wrong = __ballot_sync(0xffffffffu, !(piv > 0.0) && b + lane < nbj);
      if (lane == 0 && wrong && bad < 0) bad = b + __ffs(wrong) - 1;
      __syncwarp();
#pragma unroll
      for (int c = 0; c < SB; ++c)
        if (c < lane) s[(b + lane) * ST + b + c] = ut[c * XS + lane] * xdiag[b + c];
    } else if (warp == 1) {
      // X_kk column `lane` by forward substitution on U, the sums carried
      // forward: t_i = e_i - sum_{j < i} U_ij t_j / d_j, x_i = t_i rsqrt(d_i)
      double x[SB];
#pragma unroll
      for (int r = 0; r < SB; ++r) x[r] = r == lane ? 1.0 : 0.0;
#pragma unroll
      for (int i = 0; i < SB; ++i) {
        if (i % 8 == 0) asm volatile("bar.sync %0, 64;" ::"r"(1 + i / 8) : "memory");
        const double y = -x[i] * pinv[b + i];
#pragma unroll
        for (int r = i + 1; r < SB; ++r) x[r] = fma(ut[i * XS + r], y, x[r]);
      }
      rsx[lane] = rsqrt(diag[b + lane]);
      __syncwarp();
      diag[b + lane] = sqrt(diag[b + lane]);
#pragma unroll
      for (int r = 0; r < SB; ++r) xk[r * XS + lane] = x[r] * rsx[r];
    } else if (warp % 4 != 0) {
      // the other warps of schedulers 1 to 3: the rest of the previous step's
      // update (columns past this sub-block), T, and what is final
      const int w = warp - 2 - warp / 4;  // 0 ... 10
      if (k == 0) {
        load_columns(SB, nr, w * 32 + lane, 11 * 32);
      } else {
        int item = w;
        for (int c0 = b + SB; c0 < nr; c0 += SB) {
          const int strips = (nr - c0) / 8;
          for (; item < strips; item += 11) update(c0 + 8 * item, c0, b - SB);
          item -= strips;
        }
        for (; item < 4 * k; item += 11) t_strip(k, item / 4, item % 4);
        store_block(k - 1, w, 11);
      }
    }
    __syncthreads();
    // B: panel strips below, then X strips of this block row
    const int below = (nr - b - SB) / 8;
    for (int item = warp; item < below + 4 * k; item += 16) {
      double acc[4][2] = {};
      if (item < below) {
        const int r0 = b + SB + 8 * item;
        strip_product(acc, s + r0 * ST + b, ST, 1, xk, XS, 1, SB / 4, 4, lane);
        __syncwarp();  // the strip is read before it is overwritten
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          double *at = s + (r0 + g) * ST + b + 8 * j + 2 * t;
          at[0] = acc[j][0];
          at[1] = acc[j][1];
        }
      } else {
        const int i = (item - below) / 4, q = (item - below) % 4;
        strip_product(acc, xk + 8 * q * XS, XS, 1, tb + i * SB * XS, 1, XS, 2 * (q + 1), 4, lane);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          double *at = s + (i * SB + 8 * j + 2 * t) * ST + b + 8 * q + g;
          at[0] = -acc[j][0];
          at[ST] = -acc[j][1];
        }
      }
    }
    __syncthreads();
    if (k + 1 == nsub) break;
    // C: the next sub-block's columns
    for (int item = warp; item < below; item += 16) update(b + SB + 8 * item, b + SB, b);
    __syncthreads();
  }
  store_block(nsub - 1, warp, 16);
  if (tid == 0 && bad >= 0 && info[f] == 0) info[f] = static_cast<int>(j0) + bad + 1;
}

// out[r, c] = X[r, p] X[r, c]: the collocation of state p times every
// orbital's, the grid side of the three-index slice B_p = D^T out
__global__ void row_scaled_copy_kernel(const double *__restrict__ X, int64_t M, int64_t n,
                                       int64_t p, double *__restrict__ out) {
  const int64_t total = M * n;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / n;
    out[i] = X[r * n + p] * X[i];
  }
}

// out[p] = sum_P X[P, p] R[P, p] with R in FP32 (a split product's output)
// and X in FP64: the screening contraction's column dots
__global__ void rowdot_f32_kernel(const float *__restrict__ R, int64_t ld_r,
                                  const double *__restrict__ X, int64_t ld_x, int64_t M,
                                  int64_t S, double *out) {
  __shared__ double part[8][33];
  const int64_t p = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;
  const int64_t r0 = static_cast<int64_t>(blockIdx.y) * 256;
  double s = 0.0;
  if (p < S) {
    const int64_t r1 = min(r0 + 256, M);
    for (int64_t r = r0 + threadIdx.y; r < r1; r += 8)
      s += X[r * ld_x + p] * static_cast<double>(R[r * ld_r + p]);
  }
  part[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && p < S) {
    double t = 0.0;
    for (int k = 0; k < 8; ++k) t += part[k][threadIdx.x];
    atomicAdd(out + p, t);
  }
}

// out[P, j] = s (C[P, j0 + j] f[j0 + j]) for an nr x nc block of the
// particle-hole columns of C (leading dimension ldc): the explicit response's
// scaled factor, one column chunk at a time
__global__ void cols_scaled_copy_kernel(const double *__restrict__ C, int64_t ldc, int64_t j0,
                                        const double *__restrict__ f, double s, int64_t nr,
                                        int64_t nc, double *__restrict__ out) {
  const int64_t total = nr * nc;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / nc, j = i % nc;
    out[i] = s * (C[r * ldc + j0 + j] * f[j0 + j]);
  }
}

// out[P, q] (+)= factor Y[P, q] v[q] over an nr x nc row-major block
__global__ void col_scale_kernel(const double *__restrict__ Y, const double *__restrict__ v,
                                 int64_t nr, int64_t nc, double factor, double *out,
                                 bool accumulate) {
  const int64_t total = nr * nc;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double x = factor * Y[i] * v[i % nc];
    out[i] = accumulate ? out[i] + x : x;
  }
}

// out[r, c] += a[r * lda + p] b[r, c]: row r scaled by a's column p
__global__ void row_scale_acc_kernel(const double *__restrict__ a, int64_t lda, int64_t p,
                                     const double *__restrict__ b, int64_t nr, int64_t nc,
                                     double *out) {
  const int64_t total = nr * nc;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x)
    out[i] += a[(i / nc) * lda + p] * b[i];
}

// out[r * ldo + p] += sum_c G[r, c] X[r, c]: one warp per row
__global__ void row_dot_into_col_kernel(const double *__restrict__ G,
                                        const double *__restrict__ X, int64_t nr, int64_t nc,
                                        double *out, int64_t ldo, int64_t p) {
  const int64_t r = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (r >= nr) return;
  double s = 0.0;
  for (int64_t c = lane; c < nc; c += 32) s += G[r * nc + c] * X[r * nc + c];
  for (int d = 16; d; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (lane == 0) out[r * ldo + p] += s;
}

// The inverted diagonal blocks of nmat factors (block j of matrix f at
// src + f sf + j sj, element (r, c) of L^-1 at c ld + r) into the diagonal
// blocks of the row-major V = L^-T (n x ldv each), zeros below the diagonal
__global__ void inverse_blocks_kernel(const double *__restrict__ src, int64_t sf, int64_t sj,
                                      int64_t ld, int64_t n, double *__restrict__ V,
                                      int64_t ldv) {
  const int64_t off = static_cast<int64_t>(blockIdx.x) * kCholNb;
  const int m = static_cast<int>(min(static_cast<int64_t>(kCholNb), n - off));
  const double *x = src + blockIdx.y * sf + blockIdx.x * sj;
  double *v = V + blockIdx.y * n * ldv + off * ldv + off;
  const int lane = threadIdx.x & 31;
  for (int c = threadIdx.x >> 5; c < m; c += blockDim.x >> 5)
#pragma unroll
    for (int q = 0; q < kCholNb / 32; ++q) {
      const int r = lane + 32 * q;
      if (r < m) v[c * ldv + r] = r >= c ? x[c * ld + r] : 0.0;
    }
}

// The batched Cholesky's inverted diagonal blocks (block j of matrix f at
// Linv + j step_stride + f kCholNb^2, column-major, ld kCholNb) as TF32 pairs in
// the two layouts of the triangular-inverse recursion: rows of L^-1 (r_*) and
// columns of L^-1 as rows (c_*), zeros above the diagonal and past row n
// included; the matrices' pair arrays ldp^2 apart. The recursion and the product
// after it start (end) K at the first row (last row) of a tile of up to 256, so
// beside the blocks they write they read one block on the zero side of the
// diagonal: that one is zeroed here too, c_* left of each block but the first
// and r_* right of each but the last, and nothing else has to be (clearing the
// four arrays took 57 of 2220 us in G0W0 at naux = 786, 330 of 40600 at 5400).
// One 32 x 32 tile of a block per CTA, transposed through shared memory (one
// CTA per block, strided 4-byte stores: 54 us at 7 blocks).
__global__ void linv_blocks_to_pairs_kernel(const double *__restrict__ Linv,
                                            int64_t step_stride, int64_t n, float *c_hi,
                                            float *c_lo, float *r_hi, float *r_lo, int64_t ldp) {
  __shared__ float th[32][33], tl[32][33];
  const int64_t off = static_cast<int64_t>(blockIdx.y) * kCholNb;
  const int m = static_cast<int>(min(static_cast<int64_t>(kCholNb), n - off));
  const int r0 = (blockIdx.x & 3) * 32, c0 = (blockIdx.x >> 2) * 32;
  const double *X = Linv + blockIdx.y * step_stride + blockIdx.z * int64_t{kCholNb * kCholNb};
  const int64_t base = blockIdx.z * ldp * ldp;
  const int x = threadIdx.x;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int r = r0 + x, c = c0 + k;
    const double v = r < m && c < m ? X[c * kCholNb + r] : 0.0;
    const float h = to_tf32(static_cast<float>(v));
    const float l = to_tf32(static_cast<float>(v - static_cast<double>(h)));
    float *at = c_hi + base + (off + c) * ldp + off + r;
    float *al = c_lo + base + (off + c) * ldp + off + r;
    *at = h;
    *al = l;
    if (off > 0) at[-kCholNb] = al[-kCholNb] = 0.f;
    th[k][x] = h;
    tl[k][x] = l;
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    float *at = r_hi + base + (off + r0 + k) * ldp + off + c0 + x;
    float *al = r_lo + base + (off + r0 + k) * ldp + off + c0 + x;
    *at = th[x][k];
    *al = tl[x][k];
    if (off + kCholNb < n) at[kCholNb] = al[kCholNb] = 0.f;
  }
}

}  // namespace

void launch_chi0_bar_seed(double *a, int64_t n, int nfreq, const double *w, cudaStream_t st) {
  dim3 grid(static_cast<unsigned>(blocks(n * n) / 8 + 1), nfreq);
  count_launch(); chi0_bar_seed_kernel<<<grid, 256, 0, st>>>(a, n, w);
}

void launch_sym_half(const double *in, double *out, int64_t n, int batch, cudaStream_t st,
                     int parts) {
  const unsigned t = static_cast<unsigned>((n + 31) / 32);
  count_launch();
  sym_half_kernel<<<dim3(t, t, batch), dim3(32, 8), 0, st>>>(in, out, n, parts, batch * n * n);
}

void launch_sum_parts(double *a, int64_t n, int parts, cudaStream_t st) {
  count_launch();
  sum_parts_kernel<<<blocks(n), 256, 0, st>>>(a, n, parts);
}

void launch_xbar_update(const double *GoX, const double *GvX, const double *X, int64_t M,
                        int64_t n, int64_t nocc, const double *eps, double mu, double tau,
                        double *X_bar, double *eps_bar, cudaStream_t st) {
  dim3 grid(static_cast<unsigned>((n + 31) / 32), static_cast<unsigned>((M + 255) / 256));
  count_launch(); xbar_kernel<<<grid, dim3(32, 8), 0, st>>>(GoX, GvX, X, M, n, nocc, eps, mu, tau, X_bar,
                                            eps_bar);
}

void launch_mirror_lower_to_upper(double *a, int64_t n, cudaStream_t st) {
  count_launch(); mirror_kernel<<<blocks(n * n), 256, 0, st>>>(a, n);
}

void launch_lu_logdet(const double *LU, const int *piv, int64_t n, double *logdet, int *sign,
                      cudaStream_t st) {
  count_launch(); lu_logdet_kernel<<<1, 256, 0, st>>>(LU, piv, n, logdet, sign);
}

void launch_diag(double *a, int64_t n, int nmat, double *diag, bool save, cudaStream_t st) {
  dim3 grid(static_cast<unsigned>((n + 255) / 256), nmat);
  count_launch(); diag_kernel<<<grid, 256, 0, st>>>(a, n, diag, save);
}

void launch_inverse_blocks(const double *src, int64_t sf, int64_t sj, int64_t ld, int64_t n,
                           int nmat, double *V, int64_t ldv, cudaStream_t st) {
  count_launch();
  inverse_blocks_kernel<<<dim3(static_cast<unsigned>((n + kCholNb - 1) / kCholNb), nmat), 256, 0,
                          st>>>(src, sf, sj, ld, n, V, ldv);
}

int launch_trtri_diag_blocks(double *A, int64_t n, int nmat, int nb, cudaStream_t st,
                             float *c_hi, float *c_lo, float *r_hi, float *r_lo, int64_t ldp) {
  if (nb < 1 || nb > 128) return MBPT_ERR_SHAPE;  // one thread group of kDiagParts per column
  const size_t smem = sizeof(double) * (static_cast<size_t>(nb) * (nb + 1) + nb);
  // the attribute is per device, so it is set on every call (a host-side write)
  if (cudaFuncSetAttribute(trtri_diag_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(smem)) != cudaSuccess)
    return MBPT_ERR_CUDA;
  count_launch();
  trtri_diag_blocks_kernel<<<dim3(static_cast<unsigned>((n + nb - 1) / nb), nmat),
                             nb * kDiagParts, smem, st>>>(A, n, nb, c_hi, c_lo, r_hi, r_lo, ldp);
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

void launch_strided_to_tf32(const double *src, int64_t rows, int64_t k, int64_t rs, int64_t cs,
                            int64_t src_stride, float *hi, float *lo, int64_t rows_p,
                            int64_t k_p, bool lower, int batch, cudaStream_t st) {
  count_launch();
  dim3 grid(static_cast<unsigned>((k_p + 31) / 32), static_cast<unsigned>((rows_p + 31) / 32),
            static_cast<unsigned>(batch));
  strided_to_tf32_kernel<<<grid, dim3(32, 8), 0, st>>>(src, rows, k, rs, cs, src_stride, hi, lo,
                                                       rows_p, k_p, lower);
}

void launch_identity(double *a, int64_t n, cudaStream_t st) {
  count_launch(); identity_kernel<<<blocks(n * n), 256, 0, st>>>(a, n, 0.0, true);
}

void launch_minus_identity(double *a, int64_t n, cudaStream_t st) {
  count_launch(); identity_kernel<<<blocks(n * n), 256, 0, st>>>(a, n, -1.0, false);
}

void launch_sigma_back_gather(const double *X, int64_t M, int64_t n, const int64_t *states,
                              int64_t S, const double *sl, const double *sg, double *Xs,
                              double *Xl, double *Xg, cudaStream_t st) {
  count_launch();
  sigma_back_gather_kernel<<<blocks(M * S), 256, 0, st>>>(X, M, n, states, S, sl, sg, Xs, Xl,
                                                          Xg);
}

void launch_sigma_back_hadamard(double *go, double *gv, double *zt, double *al, double *ag,
                                int64_t total, cudaStream_t st) {
  count_launch();
  sigma_back_hadamard_kernel<<<blocks(total), 256, 0, st>>>(go, gv, zt, al, ag, total);
}

void launch_scatter_cols(const double *T, int64_t M, int64_t S, const int64_t *states,
                         double scale, double *X_bar, int64_t n, cudaStream_t st) {
  count_launch();
  scatter_cols_kernel<<<blocks(M * S), 256, 0, st>>>(T, M, S, states, scale, X_bar, n);
}

int launch_chol_diag_block(const double *P, int64_t m, int nbj, double *A, int64_t n,
                           int64_t j0, int nmat, double *Linv, int *info, cudaStream_t st) {
  if (nbj < 1 || nbj > kCholNb) return MBPT_ERR_SHAPE;
  const size_t smem = sizeof(double) * kCholSmemDoubles;
  if (cudaFuncSetAttribute(chol_diag_block_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(smem)) != cudaSuccess)
    return MBPT_ERR_CUDA;
  count_launch();
  chol_diag_block_kernel<<<nmat, 512, smem, st>>>(P, m, nbj, A, n, j0, Linv, info);
  return MBPT_OK;
}

void launch_row_scaled_copy(const double *X, int64_t M, int64_t n, int64_t p, double *out,
                            cudaStream_t st) {
  count_launch();
  row_scaled_copy_kernel<<<blocks(M * n), 256, 0, st>>>(X, M, n, p, out);
}

void launch_rowdot_f32(const float *R, int64_t ld_r, const double *X, int64_t ld_x, int64_t M,
                       int64_t S, double *out, cudaStream_t st) {
  dim3 grid(static_cast<unsigned>((S + 31) / 32), static_cast<unsigned>((M + 255) / 256));
  count_launch();
  rowdot_f32_kernel<<<grid, dim3(32, 8), 0, st>>>(R, ld_r, X, ld_x, M, S, out);
}

void launch_cols_scaled_copy(const double *C, int64_t ldc, int64_t j0, const double *f,
                             double s, int64_t nr, int64_t nc, double *out, cudaStream_t st) {
  count_launch();
  cols_scaled_copy_kernel<<<blocks(nr * nc), 256, 0, st>>>(C, ldc, j0, f, s, nr, nc, out);
}

void launch_col_scale(const double *Y, const double *v, int64_t nr, int64_t nc, double factor,
                      double *out, bool accumulate, cudaStream_t st) {
  count_launch();
  col_scale_kernel<<<blocks(nr * nc), 256, 0, st>>>(Y, v, nr, nc, factor, out, accumulate);
}

void launch_row_scale_acc(const double *a, int64_t lda, int64_t p, const double *b, int64_t nr,
                          int64_t nc, double *out, cudaStream_t st) {
  count_launch();
  row_scale_acc_kernel<<<blocks(nr * nc), 256, 0, st>>>(a, lda, p, b, nr, nc, out);
}

void launch_row_dot_into_col(const double *G, const double *X, int64_t nr, int64_t nc,
                             double *out, int64_t ldo, int64_t p, cudaStream_t st) {
  count_launch();
  row_dot_into_col_kernel<<<static_cast<unsigned>((nr + 7) / 8), 256, 0, st>>>(G, X, nr, nc,
                                                                              out, ldo, p);
}

void launch_linv_blocks_to_pairs(const double *Linv, int64_t step_stride, int64_t n, int batch,
                                 float *c_hi, float *c_lo, float *r_hi, float *r_lo,
                                 int64_t ldp, cudaStream_t st) {
  constexpr unsigned kTiles = (kCholNb / 32) * (kCholNb / 32);
  count_launch();
  linv_blocks_to_pairs_kernel<<<dim3(kTiles, static_cast<unsigned>((n + kCholNb - 1) / kCholNb),
                                     static_cast<unsigned>(batch)),
                                dim3(32, 8), 0, st>>>(Linv, step_stride, n, c_hi, c_lo, r_hi,
                                                      r_lo, ldp);
}

}  // namespace mbpt
