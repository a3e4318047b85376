// FP64 products of the sweeps on the FP64 tensor pipe (mma.sync m8n8k4 f64):
// the N^3 products of MBPT_MODE_FP64, many tau points per launch, only the
// tiles on and above the diagonal of a symmetric result, and the element-wise
// and contraction steps that follow in the same kernel. Every multiply and
// add is FP64, as in a library DGEMM.
//
// What bounds it: the FP64 pipe (64 FMA per clock and SM, 37 TFLOP/s; cuBLAS
// DGEMM reaches 35.7 here). A library product cannot leave out the half of a
// symmetric result that the other half determines, writes G_occ, G_virt and
// Zt to memory for a pass of their own, and takes a launch per product and
// tau point, which at M = 888 is most of the time.
//
// Layout: a CTA of four warps owns a 64 x BN tile (BN = 64, or 32 for few
// columns), each warp 32 x BN/2 of it in registers. The operands come through a
// three-stage cp.async ring of 16 K columns per stage. An operand tile lies in
// shared memory as in global memory, [row][k] with a row stride of 20 doubles
// or [k][row] with a stride of rows + 4: both strides are 4 modulo 16, so the
// sixteen lanes of a fragment load's half warp (four rows, four k) fall into
// sixteen different 8-byte banks. 128 threads and 61 KB: three CTAs per SM,
// one's epilogue under the others' products. Rows of odd length or
// odd origin are copied 8 bytes at a time, the others 16.
// Measured (B200): 34.3 TFLOP/s on Pi D at M = naux = 2400, five tau points a
// launch (cuBLAS 34.1, one point a launch); smaller warp tiles (32 x 16, more
// warps) 32.8, two CTAs per SM with a deeper ring 32.1. The sweep with it
// (n = 400, M = naux = 2400, 20 points): chi0 36.9 -> 27.2 ms, Sigma of 400
// states 45.0 -> 31.1 ms; E_c at M = 888, naux = 141: 1.51 -> 0.49 ms.
// What small sizes took beyond that (20 points): Pi by halves, the product with
// it reading K from each row tile's first row, every member's longest sums
// first (179 -> 103 us at M = 888, naux = 141); D^T Y cut along K where its
// CTAs are few (72 -> 49 us there); no DMMAs on the padding of a product's
// last K tile and 16-byte stores (Pi of 5 + 38 orbitals at M = 888: 65 -> 46
// us); both branches' contractions with the states in one launch, the longest
// sums first (58 states at M = 1332: 157 -> 87 us). E_c of the first case
// 0.58 -> 0.49 ms, G0W0 of the last 2.07 -> 1.67 ms. A product of one or two
// points that leaves SMs without a CTA is cut along K, its parts added by a
// pass of their own (chi0 of one point at M = 1332, naux = 236: 265 -> 181 us).
//
// The Dyson step's FP64 products run on the same kernel, all frequencies (and
// all halvings of one depth of the triangular inverse) in one launch: the
// Cholesky's block-column updates and panels, V = U^-1 by halves and W = V V^T
// over the K columns where V is not zero. One frequency at a time the library
// took 1200 launches of small products at naux = 1500, 20 frequencies: 16.1
// ms, now 3.85.
#include <algorithm>
#include <vector>

#include "dmma.h"

namespace mbpt {
namespace dmma {
namespace {

// a halving of the triangular inverse: rows [o, o + n1) and the n2 after them
struct Node {
  int o, n1, n2;
};
constexpr int kMaxNodes = 32;

constexpr int BM = 64, BK = 16, kStages = 3, kThreads = 128;
constexpr int kKStride = BK + 4;  // [row][k] tiles

template <bool KC, int R>
struct Tile {
  static constexpr int kStride = KC ? kKStride : R + 4;
  static constexpr int kDoubles = KC ? R * kKStride : BK * (R + 4);
  __device__ static __forceinline__ int at(int r, int k) {
    return KC ? r * kStride + k : k * kStride + r;
  }
};

template <int BN, bool AK, bool BKC>
struct Smem {
  static constexpr int kA = Tile<AK, BM>::kDoubles, kB = Tile<BKC, BN>::kDoubles;
  static constexpr int kStage = kA + kB;
  static constexpr int kBytes = kStages * kStage * 8;
};

__device__ __forceinline__ void cp16(void *dst, const void *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp8(void *dst, const void *src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N));
}

// One operand's stream of tiles: rows [r0, r0 + R), K columns from k0 on, BK at
// a time, zeros past `rows` and `kend`. The copies of a tile that lies inside
// the matrix cost one pointer addition each (with the bounds worked out per
// copy, integer instructions outnumbered the DMMAs five to one and the FP64
// pipe was 85 % busy).
template <bool KC, int R>
struct Stream {
  using T = Tile<KC, R>;
  const double *base, *p;  // the operand; this thread's first copy of the next tile
  int64_t ld;
  int r0, rows, k0, kend;
  bool wide;

  __device__ __forceinline__ void start(const double *g, int64_t ld_, int r0_, int rows_,
                                        int k0_, int kend_, bool wide_) {
    base = g;
    ld = ld_;
    r0 = r0_;
    rows = rows_;
    k0 = k0_;
    kend = kend_;
    wide = wide_;
    const int tid = threadIdx.x, w = wide ? 2 : 1;
    const int r = KC ? tid / (BK / w) : tid % (R / w) * w;
    const int k = KC ? tid % (BK / w) * w : tid / (R / w);
    p = g + (KC ? static_cast<int64_t>(r0 + r) * ld + k0 + k
                : static_cast<int64_t>(k0 + k) * ld + r0 + r);
  }

  template <int W>
  __device__ __forceinline__ void tile(double *s) {
    constexpr int kCopies = R * BK / W / kThreads;
    constexpr int kRows = KC ? kThreads / (BK / W) : kThreads / (R / W);  // a copy's step
    const int tid = threadIdx.x;
    const int r = KC ? tid / (BK / W) : tid % (R / W) * W;
    const int k = KC ? tid % (BK / W) * W : tid / (R / W);
    double *dst = s + T::at(r, k);
    constexpr int kDst = kRows * T::kStride;
    const int64_t step = kRows * ld;
    if (r0 + R <= rows && k0 + BK <= kend) {
      const double *src = p;
#pragma unroll
      for (int i = 0; i < kCopies; ++i, src += step) {
        if constexpr (W == 2)
          cp16(dst + i * kDst, src, 16);
        else
          cp8(dst + i * kDst, src, 8);
      }
    } else {
#pragma unroll
      for (int i = 0; i < kCopies; ++i) {
        const int ri = r0 + r + (KC ? i * kRows : 0), ki = k0 + k + (KC ? 0 : i * kRows);
        const int in = KC ? (ri < rows ? min(max(kend - ki, 0), W) : 0)
                          : (ki < kend ? min(max(rows - ri, 0), W) : 0);
        const double *src = in ? p + i * step : base;
        if constexpr (W == 2)
          cp16(dst + i * kDst, src, 8 * in);
        else
          cp8(dst + i * kDst, src, 8 * in);
      }
    }
  }

  __device__ __forceinline__ void load(double *s) {
    if (wide)
      tile<2>(s);
    else
      tile<1>(s);
    k0 += BK;
    p += KC ? BK : BK * ld;
  }
};

__device__ __forceinline__ void mma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// tile `idx` of the upper triangle of nt x nt tiles, row by row
__device__ __forceinline__ void upper_tile(int idx, int nt, int &ti, int &tj) {
  const double q = 2.0 * nt + 1.0;
  int i = static_cast<int>(0.5 * (q - sqrt(q * q - 8.0 * idx)));
  i = max(0, min(i, nt - 1));
  auto first = [nt](int r) { return r * nt - r * (r - 1) / 2; };
  while (i > 0 && first(i) > idx) --i;
  while (i + 1 < nt && first(i + 1) <= idx) ++i;
  ti = i;
  tj = i + idx - first(i);
}

struct Args {
  Operand a[3], b[3];
  int k[3];
  bool wa[3], wb[3];  // 16-byte copies
  int m, n, tiles_m, tiles_n;
  bool upper;
  bool half;       // PRODUCT: upper tiles only, the diagonal ones halved; STORE: A is such a half
  bool pairs;      // 16-byte stores
  int members;     // half, ROWDOT: the batch, all in one grid dimension
  int ksplit;      // STORE: K in so many parts, each with a result of its own
  int64_t s_part;
  double alpha, beta;
  double *c0, *c1, *c2;  // PRODUCT: c1, c2 the factors themselves (null: not kept)
  int64_t ldc, sc;
  const double *zt;    // SIGMA: Zt as stored (ld m) instead of the first product
  const double *xs;    // row contraction
  int64_t ld_xs;
  double *out, *out2;
  int64_t s_out;
  // Dyson step
  const double *src;   // CHOL: the matrices whose identity complement is factorised
  int64_t ld_src, s_src;
  const int *info;     // matrices whose word is not zero are left alone (null: none)
  int nnodes;
  Node node[kMaxNodes];
};

// the K columns of one of `parts` parts of k: whole tiles
__host__ __device__ constexpr int round_to(int k, int parts) {
  return ((k + parts - 1) / parts + BK - 1) / BK * BK;
}

enum Epi : int {
  STORE = 0,     // C = alpha acc + beta C (upper: and its mirror; half: K from the tile's first row)
  PRODUCT = 1,   // C = acc0 o acc1, mirrored (half: as SIGMA's)
  SIGMA = 2,     // c0 = acc1 o acc0, c1 = acc2 o acc0: upper tiles, the diagonal ones halved
  ROWDOT = 3,    // out[p] += 2 sum_r xs[r, p] acc[r, p], K from the tile's first row; the
                 // second half of the members a[1]'s, out2[p] -= ...
  CHOL = 4,      // C = I - src - acc, on and above the diagonal
  NODE_T = 5,    // per node: T^T = U12^T V11^T, K from the tile's first column
  NODE_V = 6,    // per node: V12 = -T V22, K up to the tile's last column
  INVERSE = 7,   // C = -I + V V^T, mirrored, K from the tile's first column
};

template <int BN, bool AK, bool BKC, int EPI>
__global__ void __launch_bounds__(kThreads, BN == 32 ? 4 : 3) dmma_kernel(const __grid_constant__ Args p) {
  using S = Smem<BN, AK, BKC>;
  constexpr int NS = EPI == SIGMA ? 3 : (EPI == PRODUCT ? 2 : 1);
  constexpr int MI = 4, NJ = BN / 16;  // 8 x 8 blocks of a warp's 32 x BN/2
  extern __shared__ __align__(16) double sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * (BN / 2);
  int ti, tj;
  int rows_m = p.m, rows_n = p.n, k_end0 = p.k[0];
  int64_t z = blockIdx.z, off_a = 0, off_b = 0, off_c = 0;
  unsigned tile = blockIdx.x;
  int k_begin = 0;
  [[maybe_unused]] bool second = false;
  if constexpr (EPI == NODE_T || EPI == NODE_V) {
    const Node &q = p.node[z % p.nnodes];
    z /= p.nnodes;
    const int64_t o1 = q.o, o2 = q.o + q.n1;
    rows_m = EPI == NODE_T ? q.n2 : q.n1;
    rows_n = EPI == NODE_T ? q.n1 : q.n2;
    k_end0 = rows_n;
    off_a = EPI == NODE_T ? o1 * p.a[0].ld + o2 : o2 * p.a[0].ld + o1;
    off_b = EPI == NODE_T ? o1 * p.b[0].ld + o1 : o2 * p.b[0].ld + o2;
    off_c = EPI == NODE_T ? o2 * p.ldc + o1 : o1 * p.ldc + o2;
    const int tn = (rows_n + BN - 1) / BN;
    ti = tile / tn;
    tj = tile % tn;
    if (ti * BM >= rows_m) return;
  } else if (p.upper) {
    upper_tile(tile, p.tiles_m, ti, tj);
  } else {
    if constexpr (EPI == ROWDOT) {  // the longest sums of all members first
      z = tile % p.members;
      tile /= p.members;
      second = 2 * z >= p.members;
      if (second) z -= p.members / 2;
    }
    if constexpr (EPI == STORE) {
      if (p.half) {
        z = tile % p.members;
        tile /= p.members;
      } else if (p.ksplit > 1) {
        const int part = z % p.ksplit, per = round_to(p.k[0], p.ksplit);
        k_begin = part * per;
        k_end0 = min(k_end0, k_begin + per);
        off_c = part * p.s_part;
        z /= p.ksplit;
      }
    }
    // eight row tiles sweep the column tiles together (L2 reuse)
    const int per = 8 * p.tiles_n, grp = tile / per, first = grp * 8;
    const int rows = min(8, p.tiles_m - first), in = tile % per;
    ti = first + in % rows;
    tj = in / rows;
  }
  const int m0 = ti * BM, n0 = tj * BN;
  if constexpr (EPI >= CHOL) {
    if (p.info && p.info[z] != 0) return;
  }
  if (EPI == CHOL && n0 + BN <= m0) return;
  const int k_first = EPI == ROWDOT || (EPI == STORE && p.half)
                          ? m0
                          : (EPI == INVERSE || EPI == NODE_T ? n0 : k_begin);
  if (EPI == NODE_V) k_end0 = min(k_end0, n0 + BN);
  // a product's K columns and tiles
  auto depth = [&](int s) { return (s == 0 ? k_end0 : p.k[s]) - k_first; };
  auto tiles = [&](int s) { return (depth(s) + BK - 1) / BK; };
  int total = 0;
#pragma unroll
  for (int s = 0; s < NS; ++s) total += tiles(s);
  // the tiles of the products, one product after the other
  Stream<AK, BM> fa;
  Stream<BKC, BN> fb;
  int fseg = EPI == SIGMA && k_end0 == 0 ? 1 : 0, fleft = tiles(fseg), fstage = 0;
  auto open = [&](int s) {
    const int ke = s == 0 ? k_end0 : p.k[s];
    const Operand &oa = p.a[EPI == ROWDOT && second ? 1 : s];
    fa.start(oa.p + z * oa.stride + off_a, oa.ld, m0, rows_m, k_first, ke, p.wa[s]);
    fb.start(p.b[s].p + z * p.b[s].stride + off_b, p.b[s].ld, n0, rows_n, k_first, ke, p.wb[s]);
  };
  open(fseg);
  auto fetch = [&] {
    double *st = sm + fstage * S::kStage;
    fa.load(st);
    fb.load(st + S::kA);
    fstage = fstage + 1 == kStages ? 0 : fstage + 1;
    if (NS > 1 && --fleft == 0 && fseg + 1 < NS) {
      ++fseg;
      fleft = tiles(fseg < NS ? fseg : 0);
      open(fseg < NS ? fseg : 0);
    }
  };
  double acc[MI][NJ][2];
  double keep[NS > 1 ? MI : 1][NS > 1 ? NJ : 1][2];
  auto clear = [&] {
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  };
  // an element-wise result: the tile and, above the diagonal, its mirror
  auto store = [&](double *c, auto value, bool mirror) {
#pragma unroll
    for (int i = 0; i < MI; ++i) {
      const int r = m0 + wm + 8 * i + g;
      if (r >= rows_m) continue;
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int col = n0 + wn + 8 * j + 2 * t;
        if (col >= rows_n) continue;
        double *at = c + z * p.sc + off_c + static_cast<int64_t>(r) * p.ldc + col;
        const bool two = col + 1 < rows_n;
        const double v0 = value(i, j, 0, at), v1 = two ? value(i, j, 1, at + 1) : 0.0;
        if (two && p.pairs) {
          *reinterpret_cast<double2 *>(at) = make_double2(v0, v1);
        } else {
          at[0] = v0;
          if (two) at[1] = v1;
        }
        if (mirror) {
          double *tr = c + z * p.sc + static_cast<int64_t>(col) * p.ldc + r;
          tr[0] = v0;
          if (two) tr[p.ldc] = v1;
        }
      }
    }
  };
  clear();
  if constexpr (EPI == INVERSE) {
    // the sums start from -I: a diagonal entry's first term cancels it, and the
    // small ones that follow are not rounded at the size of 1 (W - I of the
    // mid-size test 3x nearer its value than with I taken off at the end)
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          if (m0 + wm + 8 * i + g == n0 + wn + 8 * j + 2 * t + e) acc[i][j][e] = -1.0;
  }
  int seg_end = tiles(0);
  [[maybe_unused]] int seg = 0;
  if constexpr (EPI == SIGMA) {
    if (p.zt) {
      seg = 1;
      seg_end = tiles(1);
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int r = m0 + wm + 8 * i + g, col = n0 + wn + 8 * j + 2 * t + e;
            keep[i][j][e] = r < p.m && col < p.n ? p.zt[static_cast<int64_t>(r) * p.ldc + col] : 0.0;
          }
    }
  }
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < total) fetch();
    cp_commit();
  }
  int stage = 0;
  for (int it = 0; it < total; ++it) {
    cp_wait<kStages - 2>();
    __syncthreads();
    if (it + kStages - 1 < total) fetch();
    cp_commit();
    const double *sa = sm + stage * S::kStage, *sb = sa + S::kA;
    stage = stage + 1 == kStages ? 0 : stage + 1;
    auto step = [&](int kk) {
      double a[MI], b[NJ];
#pragma unroll
      for (int i = 0; i < MI; ++i) a[i] = sa[Tile<AK, BM>::at(wm + 8 * i + g, kk + t)];
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[j] = sb[Tile<BKC, BN>::at(wn + 8 * j + g, kk + t)];
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) mma(acc[i][j], a[i], b[j]);
    };
    // a product's last tile takes the steps that it has columns for (5 occupied
    // and 53 virtual orbitals: 16 steps instead of 20)
    if (it + 1 == seg_end) {
      const int left = (depth(seg) - 1) % BK;
#pragma unroll 1
      for (int kk = 0; kk <= left; kk += 4) step(kk);
    } else {
#pragma unroll
      for (int kk = 0; kk < BK; kk += 4) step(kk);
    }
    if constexpr (NS > 1) {
      if (it + 1 == seg_end && seg + 1 < NS) {
        if (seg == 0) {
#pragma unroll
          for (int i = 0; i < MI; ++i)
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
              keep[i][j][0] = acc[i][j][0];
              keep[i][j][1] = acc[i][j][1];
            }
        } else {
          const double f = ti == tj ? 0.5 : 1.0;
          store(p.c0, [&](int i, int j, int e, double *) { return acc[i][j][e] * keep[i][j][e] * f; },
                false);
        }
        clear();
        ++seg;
        seg_end += tiles(seg < NS ? seg : 0);
      }
    }
  }
  if constexpr (EPI == CHOL) {
    const double *src = p.src + z * p.s_src;
    store(p.c0,
          [&](int i, int j, int e, double *) {
            const int r = m0 + wm + 8 * i + g, col = n0 + wn + 8 * j + 2 * t + e;
            return (r == col ? 1.0 : 0.0) - src[static_cast<int64_t>(r) * p.ld_src + col] -
                   acc[i][j][e];
          },
          false);
  } else if constexpr (EPI == NODE_T || EPI == NODE_V) {
    store(p.c0, [&](int i, int j, int e, double *) { return EPI == NODE_T ? acc[i][j][e] : -acc[i][j][e]; },
          false);
  } else if constexpr (EPI == INVERSE) {
    store(p.c0, [&](int i, int j, int e, double *) { return acc[i][j][e]; }, tj > ti);
  } else if constexpr (EPI == STORE) {
    const double alpha = p.alpha, beta = p.beta;
    store(p.c0,
          [&](int i, int j, int e, const double *at) {
            const double v = alpha * acc[i][j][e];
            return beta == 0.0 ? v : v + beta * *at;
          },
          p.upper && tj > ti);
  } else if constexpr (EPI == PRODUCT) {
    const double f = p.half && ti == tj ? 0.5 : 1.0;
    store(p.c0, [&](int i, int j, int e, double *) { return acc[i][j][e] * keep[i][j][e] * f; },
          !p.half && tj > ti);
    if (p.c1) {
      store(p.c1, [&](int i, int j, int e, double *) { return keep[i][j][e]; }, tj > ti);
      store(p.c2, [&](int i, int j, int e, double *) { return acc[i][j][e]; }, tj > ti);
    }
  } else if constexpr (EPI == SIGMA) {
    const double f = ti == tj ? 0.5 : 1.0;
    store(p.c1, [&](int i, int j, int e, double *) { return acc[i][j][e] * keep[i][j][e] * f; },
          false);
  } else {
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = n0 + wn + 8 * j + 2 * t + e;
        double s = 0.0;
#pragma unroll
        for (int i = 0; i < MI; ++i) {
          const int r = m0 + wm + 8 * i + g;
          if (r < p.m && col < p.n) s = fma(p.xs[static_cast<int64_t>(r) * p.ld_xs + col],
                                            acc[i][j][e], s);
        }
#pragma unroll
        for (int d = 4; d < 32; d <<= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (g == 0 && col < p.n)
          atomicAdd((second ? p.out2 : p.out) + z * p.s_out + col, (second ? -2.0 : 2.0) * s);
      }
  }
}

bool wide(const Operand &o, int64_t batch) {
  return (reinterpret_cast<uintptr_t>(o.p) & 15) == 0 && o.ld % 2 == 0 &&
         (batch <= 1 || o.stride % 2 == 0);
}

template <int BN, bool AK, bool BKC, int EPI>
int launch(Args &p, int batch, cudaStream_t st) {
  constexpr int NS = EPI == SIGMA ? 3 : (EPI == PRODUCT ? 2 : 1);
  using S = Smem<BN, AK, BKC>;
  if (p.m < 1 || p.n < 1 || batch < 1 || batch > 65535) return MBPT_ERR_SHAPE;
  for (int s = 0; s < NS; ++s) {
    const bool none = (EPI == SIGMA && s == 0 && p.zt) || EPI == CHOL;
    if (p.k[s] < (none ? 0 : 1)) return MBPT_ERR_SHAPE;
    p.wa[s] = wide(p.a[s], batch);
    p.wb[s] = wide(p.b[s], batch);
  }
  // the second and third results lie as the first
  p.pairs = p.ldc % 2 == 0 && (batch <= 1 || p.sc % 2 == 0) && p.s_part % 2 == 0 &&
            ((reinterpret_cast<uintptr_t>(p.c0) | reinterpret_cast<uintptr_t>(p.c1) |
              reinterpret_cast<uintptr_t>(p.c2)) & 15) == 0;
  p.tiles_m = (p.m + BM - 1) / BM;
  p.tiles_n = (p.n + BN - 1) / BN;
  if (p.upper && (BN != BM || p.m != p.n)) return MBPT_ERR_SHAPE;
  if (EPI >= CHOL && p.nnodes == 0) p.nnodes = 1;
  if ((EPI == NODE_T || EPI == NODE_V) && static_cast<int64_t>(batch) * p.nnodes > 65535)
    return MBPT_ERR_SHAPE;
  if (EPI == NODE_T || EPI == NODE_V) batch *= p.nnodes;
  int64_t grid = p.upper ? static_cast<int64_t>(p.tiles_m) * (p.tiles_m + 1) / 2
                         : static_cast<int64_t>(p.tiles_m) * p.tiles_n;
  if (grid > (int64_t{1} << 30)) return MBPT_ERR_SHAPE;
  if (EPI == ROWDOT) {
    p.wa[0] = p.wa[0] && wide(p.a[1], batch);
    batch *= 2;
  }
  if (EPI == ROWDOT || (EPI == STORE && p.half)) {
    p.members = batch;
    if (grid * batch > (int64_t{1} << 30)) return MBPT_ERR_SHAPE;
    grid *= batch;
    batch = 1;
  } else if (EPI == STORE && p.ksplit > 1) {
    // every part has a first column
    if (round_to(p.k[0], p.ksplit) * (p.ksplit - 1) >= p.k[0] ||
        static_cast<int64_t>(batch) * p.ksplit > 65535 || p.upper)
      return MBPT_ERR_SHAPE;
    batch *= p.ksplit;
  }
  auto kern = dmma_kernel<BN, AK, BKC, EPI>;
  static std::atomic<uint64_t> attr{0};
  if (!allow_smem(reinterpret_cast<const void *>(kern), S::kBytes, attr)) return MBPT_ERR_CUDA;
  count_launch();
  kern<<<dim3(static_cast<unsigned>(grid), 1, static_cast<unsigned>(batch)), kThreads, S::kBytes,
         st>>>(p);
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

// Whether 32-wide tiles pad n columns so much less than 64-wide ones that
// their lower rate pays (33.9 against 34.3 TFLOP/s at n = 2400, where both pad
// alike; 24.7 against 21.1 at n = 141, 160 columns against 192).
bool narrow(int64_t n) { return round_up(n, 64) * 20 >= round_up(n, 32) * 21; }

// A product with fewer CTAs than four per SM is cut along K.
constexpr int64_t kFewCtas = 4 * 148;

// Whether 64-wide tiles leave SMs without a CTA: 32-wide ones then take 0.6 us
// per 16 K columns instead of 0.93 (Pi D at 200 x 60: 14.2 -> 9.7 us).
bool lone(int64_t m, int64_t n, int batch) {
  return ((m + BM - 1) / BM) * ((n + 63) / 64) * batch <= 148;
}

// What a K tile of `ctas` CTAs takes, in units of an SM's time for one at its
// full rate (0.55 us): one CTA per SM 1.7, two 2.2, three 3, then the rest.
double rounds(int64_t ctas) {
  const double busy[4] = {0.0, 1.7, 2.2, 3.0};
  return 3.0 * (ctas / 444) + busy[(ctas % 444 + 147) / 148];
}

// Parts that K is cut into so that `ctas` CTAs fill the GPU: four K tiles each
// at least, the last one not empty.
int fill_parts(int64_t ctas, int64_t k) {
  auto ok = [k](int p) { return k >= 4 * BK * p && round_to(static_cast<int>(k), p) * (p - 1) < k; };
  int parts = 1;
  while (parts < kMaxParts && ctas * parts < kFewCtas && ok(parts + 1)) ++parts;
  return parts;
}

bool fits(int64_t v) { return v > 0 && v <= (int64_t{1} << 30); }

}  // namespace

int gemm(const Operand &a, bool a_k, const Operand &b, bool b_k, int64_t m, int64_t n, int64_t k,
         double alpha, double beta, double *c, int64_t ldc, int64_t sc, int batch, bool upper,
         cudaStream_t st, bool half) {
  if (half && (!a_k || m != k)) return MBPT_ERR_SHAPE;
  if (!fits(m) || !fits(n) || !fits(k)) return MBPT_ERR_SHAPE;
  Args p{};
  p.a[0] = a;
  p.b[0] = b;
  p.k[0] = static_cast<int>(k);
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(n);
  p.alpha = alpha;
  p.beta = beta;
  p.c0 = c;
  p.ldc = ldc;
  p.sc = sc;
  p.upper = upper;
  p.half = half;
  if (a_k && b_k) return launch<64, true, true, STORE>(p, batch, st);
  if (a_k && (narrow(n) || lone(m, n, batch))) return launch<32, true, false, STORE>(p, batch, st);
  if (a_k) return launch<64, true, false, STORE>(p, batch, st);
  if (!b_k) return launch<64, false, false, STORE>(p, batch, st);
  return MBPT_ERR_UNSUPPORTED;
}

int product_parts(int64_t m, int64_t n, int64_t k, int batch) {
  const int64_t ctas = ((m + BM - 1) / BM) * ((n + 63) / 64) * batch;
  int parts = 1;
  while (parts < kMaxParts && ctas * parts < kFewCtas && k >= 128 * (parts + 1)) ++parts;
  return parts;
}

int cut_parts(int64_t m, int64_t n, int64_t k, int batch) {
  const int64_t ctas = ((m + BM - 1) / BM) * ((n + 63) / 64) * batch;
  return (rounds(ctas) - ctas / 148.0) * k > 44.0 * BK ? fill_parts(ctas, k) : 1;
}

int square_parts(int64_t n, int64_t k, int batch) {
  const int64_t t = (n + BM - 1) / BM, whole = t * t * batch, upper = t * (t + 1) / 2 * batch;
  return (rounds(upper) - whole / 148.0) * k > 30.0 * BK ? fill_parts(whole, k) : 1;
}

int gemm_parts(const Operand &a, bool a_k, const Operand &b, int64_t m, int64_t n, int64_t k,
               double alpha, double *c, int64_t ldc, int64_t sc, int batch, int parts,
               cudaStream_t st) {
  if (!fits(m) || !fits(n) || !fits(k)) return MBPT_ERR_SHAPE;
  Args p{};
  p.a[0] = a;
  p.b[0] = b;
  p.k[0] = static_cast<int>(k);
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(n);
  p.alpha = alpha;
  p.c0 = c;
  p.ldc = ldc;
  p.sc = sc;
  p.ksplit = parts;
  p.s_part = sc * batch;
  if (a_k && (narrow(n) || lone(m, n, batch))) return launch<32, true, false, STORE>(p, batch, st);
  if (a_k) return launch<64, true, false, STORE>(p, batch, st);
  return launch<64, false, false, STORE>(p, batch, st);
}

int hadamard_product(const Operand &a0, const Operand &b0, int64_t k0, const Operand &a1,
                     const Operand &b1, int64_t k1, int64_t m, double *c, int64_t ldc,
                     int64_t sc, int batch, cudaStream_t st, double *g0, double *g1,
                     bool half) {
  if (!fits(m) || !fits(k0) || !fits(k1)) return MBPT_ERR_SHAPE;
  Args p{};
  p.a[0] = a0;
  p.b[0] = b0;
  p.a[1] = a1;
  p.b[1] = b1;
  p.k[0] = static_cast<int>(k0);
  p.k[1] = static_cast<int>(k1);
  p.m = p.n = static_cast<int>(m);
  p.c0 = c;
  p.c1 = g0;
  p.c2 = g1;
  p.ldc = ldc;
  p.sc = sc;
  p.upper = true;
  p.half = half;
  return launch<64, true, true, PRODUCT>(p, batch, st);
}

int sigma_h(const double *zt, const Operand &u, const Operand &d, int64_t naux,
            const Operand &xo_s, const Operand &xo, int64_t nocc, const Operand &xv_s,
            const Operand &xv, int64_t nv, int64_t m, double *hl, double *hg, int64_t sh,
            int batch, cudaStream_t st) {
  if (!fits(m) || !fits(naux) || !fits(nocc) || !fits(nv)) return MBPT_ERR_SHAPE;
  Args p{};
  p.zt = zt;
  const Operand *as[3] = {&u, &xo_s, &xv_s}, *bs[3] = {&d, &xo, &xv};
  const int64_t ks[3] = {zt ? 0 : naux, nocc, nv};
  for (int s = 0; s < 3; ++s) {
    p.a[s] = *as[s];
    p.b[s] = *bs[s];
    p.k[s] = static_cast<int>(ks[s]);
  }
  p.m = p.n = static_cast<int>(m);
  p.c0 = hl;
  p.c1 = hg;
  p.ldc = m;
  p.sc = sh;
  p.upper = true;
  return launch<64, true, true, SIGMA>(p, batch, st);
}

int half_quadratic(const double *hl, const double *hg, int64_t sh, int64_t m, const double *xs,
                   int64_t ns, double *out_l, double *out_g, int64_t s_out, int batch,
                   cudaStream_t st) {
  if (!fits(m) || !fits(ns)) return MBPT_ERR_SHAPE;
  Args p{};
  p.a[0] = {hl, m, sh};
  p.a[1] = {hg, m, sh};
  p.b[0] = {xs, ns, 0};
  p.k[0] = static_cast<int>(m);
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(ns);
  p.xs = xs;
  p.ld_xs = ns;
  p.out = out_l;
  p.out2 = out_g;
  p.s_out = s_out;
  if (narrow(ns)) return launch<32, true, false, ROWDOT>(p, batch, st);
  return launch<64, true, false, ROWDOT>(p, batch, st);
}

int chol_update(const double *chi0, int64_t n, int64_t j0, int nbj, double *P, int batch,
                cudaStream_t st) {
  const int64_t m = n - j0;
  if (!fits(m) || nbj < 1 || nbj > m || j0 < 0) return MBPT_ERR_SHAPE;
  Args p{};
  p.a[0] = p.b[0] = {chi0 + j0, n, n * n};
  p.k[0] = static_cast<int>(j0);
  p.m = nbj;
  p.n = static_cast<int>(m);
  p.src = chi0 + j0 * n + j0;
  p.ld_src = n;
  p.s_src = n * n;
  p.c0 = P;
  p.ldc = m;
  p.sc = m * nbj;
  return launch<64, false, false, CHOL>(p, batch, st);
}

int spd_inverse(double *chi0, int64_t n, double *V, int64_t ldv, const int *info, int batch,
                cudaStream_t st) {
  if (!fits(n)) return MBPT_ERR_SHAPE;
  std::vector<std::vector<Node>> levels;
  struct Split {
    static void add(int64_t o, int64_t len, size_t depth, std::vector<std::vector<Node>> &lv) {
      if (len <= kInverseLeaf) return;
      if (lv.size() <= depth) lv.resize(depth + 1);
      const int64_t n1 = round_up(len / 2, kInverseLeaf);
      lv[depth].push_back({static_cast<int>(o), static_cast<int>(n1), static_cast<int>(len - n1)});
      add(o, n1, depth + 1, lv);
      add(o + n1, len - n1, depth + 1, lv);
    }
  };
  Split::add(0, n, 0, levels);
  const int64_t sv = n * ldv;
  for (size_t d = levels.size(); d-- > 0;)
    for (size_t first = 0; first < levels[d].size(); first += kMaxNodes) {
      Args p{};
      p.nnodes = static_cast<int>(std::min<size_t>(kMaxNodes, levels[d].size() - first));
      for (int i = 0; i < p.nnodes; ++i) {
        p.node[i] = levels[d][first + i];
        p.m = std::max(p.m, std::max(p.node[i].n1, p.node[i].n2));
      }
      p.n = p.m;
      p.k[0] = p.m;
      p.info = info;
      p.c0 = V;
      p.ldc = ldv;
      p.sc = sv;
      Args q = p;
      p.a[0] = {chi0, n, n * n};
      p.b[0] = {V, ldv, sv};
      int rc = launch<64, false, true, NODE_T>(p, batch, st);
      if (rc) return rc;
      q.a[0] = q.b[0] = {V, ldv, sv};
      rc = launch<64, false, false, NODE_V>(q, batch, st);
      if (rc) return rc;
    }
  Args p{};
  p.a[0] = p.b[0] = {V, ldv, sv};
  p.k[0] = p.m = p.n = static_cast<int>(n);
  p.info = info;
  p.c0 = chi0;
  p.ldc = n;
  p.sc = n * n;
  p.upper = true;
  return launch<64, true, true, INVERSE>(p, batch, st);
}

}  // namespace dmma
}  // namespace mbpt
