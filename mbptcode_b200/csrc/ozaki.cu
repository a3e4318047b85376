// FP64-accurate trailing updates of the batched Cholesky on the int8 tensor
// cores (tcgen05.mma kind::i8, exact int32 accumulation): the Ozaki scheme.
//
// Digit widths: S = 7 and 8 cut signed 7-bit digits (d_s in [-64, 64], base
// 128, as below); S = 6 cuts signed 8-bit digits of base 254 (x = L_rk / 2^e_r,
// t = 127 x, d_1 = rint(t), then t <- 254 (t - d); d_s in [-127, 127], 47 bits
// in all, against 49 for S = 7), whose levels 2..7 take 21 digit products per
// K step instead of 28. Level l weighs 127^-2 254^-(l-2), exact to one
// rounding in FP64; its int32 sums stay exact for K below 2^31 / (6 127^2).
//
// Each row r of the factor L is scaled by 2^-e_r, with 2^e_r >= sqrt(A_rr)
// (|L_rk| <= sqrt(A_rr) for a positive definite A), and cut into S signed
// digits: x = L_rk 2^-e_r, |x| <= 1, x = sum_s d_s 2^-(7s-1) + O(2^-7S),
// d_s in [-64, 64]. A block column of L is cut once, when it is final, into S
// int8 planes (row r, K = column k contiguous). The update of step j,
// P -= L[j0:, :j0] L[j0:j0+nb, :j0]^T, is then
//   sum over levels l = s + t (2 <= l <= S + 1) of 2^(2 - 7l) sum_(s+t=l) D_s D_t^T,
// each level one int32 TMEM accumulator fed by exact 8-bit products (|sum| <=
// S 64^2 K < 2^31 for K below 65 536), combined in FP64 in the epilogue and
// scaled by 2^(e_r + e_c). The terms dropped (s + t > S + 1) have no sign
// preference off the diagonal; on it (a row against itself) their squares
// are all positive, so each step's diagonal entries are taken from an exact
// FP64 row norm instead, which the slicing of each block column accumulates.
//
// Kernel layout: 128 x 64 output tiles (rows r of the panel, 64 of its
// columns), warp 0 the TMA producer (64-byte swizzled boxes of 64 K), warp 1
// the TMEM owner and MMA issuer (the S(S+1)/2 products of a 32-wide K step
// as one MMA per A plane and group of up to four B planes), warps
// 2-9 the epilogue; two pipeline stages of S A-planes and S B-planes; every
// mbarrier wait bounded, as in the split engine.
#include <algorithm>

#include "internal.h"

namespace mbpt {
namespace ozaki {

using umma::mbar_expect_tx;
using umma::mbar_init;
using umma::mbar_wait;
using umma::mma_commit;
using umma::smem_u32;
using umma::tc_fence_after;
using umma::tc_fence_before;

constexpr int BM = 128;   // panel rows per tile
constexpr int BN = 64;    // panel columns per tile
constexpr int BKB = 64;   // K bytes (int8 elements) per stage: two MMA K steps
// (32-byte steps with four stages in the same shared memory measured slower:
// 64.9 against 70.1 TFLOP/s FP64-equivalent at 4096^3)
// the K-major operand layout of a stage's rows: BKB-byte rows swizzled by
// BKB bytes, in 8-row groups of 8 * BKB bytes
constexpr int kSwizzleBytes = BKB;
constexpr CUtensorMapSwizzle kTmaSwizzle =
    kSwizzleBytes == 32 ? CU_TENSOR_MAP_SWIZZLE_32B : CU_TENSOR_MAP_SWIZZLE_64B;
constexpr int kStackPlanes = 4;  // B planes per MMA: N = 4 x 64 = 256, the largest

template <int S>
struct Layout {
  static constexpr int kAPlane = BM * BKB;   // 8 KB
  static constexpr int kBPlane = BN * BKB;   // 4 KB
  static constexpr int kStageBytes = S * (kAPlane + kBPlane);
  // as many stages as 196 KB hold: 2 for S = 7 and 8 (84 and 96 KB each)
  static constexpr int kStages = (196 * 1024) / kStageBytes < 8 ? (196 * 1024) / kStageBytes : 8;
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024 + 512;
  static constexpr int kLevels = S;
  static constexpr int kTmemCols = 512;
  static_assert(kLevels * BN <= 512, "levels exceed TMEM");
  static_assert(kStages * kStageBytes >= 16 * 32 * 33 * 8, "the epilogue's blocks");
};

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *tm, int x, int y,
                                            int z, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// K-major operand with kSwizzleBytes-byte rows and swizzle: 8-row groups
// 8 * kSwizzleBytes bytes apart (layout type 6 = 32-byte swizzle, 4 = 64-byte).
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t saddr) {
  static_assert(kSwizzleBytes == 32 || kSwizzleBytes == 64, "32- or 64-byte swizzle");
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>((8 * kSwizzleBytes) >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(kSwizzleBytes == 32 ? 6 : 4) << 61;
  return d;
}

// Instruction descriptor: s8 x s8 -> s32, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t idesc_s8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_s8(uint32_t tmem_d, uint64_t da, uint64_t db,
                                       uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void tmem_ld32_s32(uint32_t addr, int (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
        "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
        "=r"(v[31])
      : "r"(addr)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16_s32(uint32_t addr, int (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
        "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr)
      : "memory");
}

// Shared tile of the cutting kernels, 32 rows x 128 columns: one double of
// padding per 16 columns and a row stride of 137, so that a half warp hits 16
// different 8-byte banks when it writes 16 columns or 16 rows, and 15 when it
// reads two rows at eight 16-column groups (8 lanes in one bank without).
constexpr int kCutStride = 137;
__device__ __forceinline__ int cut_at(int r, int c) { return r * kCutStride + c + (c >> 4); }

// The next digit of t (|t| <= 127): adding 1.5 2^52 leaves rint(t), ties to
// even, in the low word, so a digit costs FP64 additions instead of the
// conversion unit's two instructions (16 lanes per clock and SM; the cutting
// kernels ran at its rate: 60 us for two 2400 x 2400 operands, 8 digits; now
// 36 us). t
// becomes the exact remainder times the base. A t that is not finite gives
// some byte and stays not finite.
__device__ __forceinline__ int8_t next_digit(double &t, double base) {
  constexpr double kMagic = 6755399441055744.0;  // 1.5 2^52
  const double r = t + kMagic;
  t = (t - (r - kMagic)) * base;
  return static_cast<int8_t>(__double2loint(r));
}

// An int32 as a double by one FP64 addition (the conversion unit takes 16 lanes
// per clock and SM, a quarter of the FP64 pipe's rate)
__device__ __forceinline__ double exact_double(int v) {
  return __hiloint2double(0x43300000, v ^ static_cast<int>(0x80000000u)) - 4503601774854144.0;
}

enum Epi : int {
  EPI_CHOL = 0,  // the Cholesky panel: P = I - chi0 - product, column-major, exact diagonal
  EPI_GEMM = 1,  // C = alpha product + beta C, row-major
};

struct UpdateArgs {
  CUtensorMap tm_a;    // A digit planes (K, rows, planes), box 64 x 128
  CUtensorMap tm_b;    // B digit planes, box 64 x 64 (the Cholesky: the same array)
  int64_t n;           // matrix size (Cholesky)
  int j0, nb;          // the step's first column and width (<= 128) (Cholesky)
  int k_tiles;         // K / BKB
  int nmat;            // planes per digit level (matrices of a batch)
  int a_row0, b_row0;  // first plane rows of the A and B operands
  int tiles_n;         // 64-column tiles per row of tiles
  const double *A0;    // Cholesky: nmat n x n chi0, I - chi0 being factorised
  double *P;           // nmat panels, column-major m x nb (ld m), m = n - j0
  int64_t p_stride;    // elements between panels
  const double *scale; // Cholesky: nmat x n, 2^e_r; GEMM: the rows of A
  const double *scale_b;  // GEMM: the rows of B
  const double *rowsq; // nmat x n: sum_(k < j0) L_(r, k)^2 of each row, exact
  double *C;           // GEMM output, row-major m_rows x n_cols, ld ldc
  int64_t ldc;
  double alpha, beta;
  int m_rows, n_cols;
  int tiles_m;
  int sym;             // GEMM: symmetric product, upper tiles formed and mirrored
  const double *H1, *H2;  // GEMM: element-wise factors of C and C2 (null: none)
  double *C2;
  int *err;
};

// Weights of the levels: 2^(2 - 7 l), and 127^-2 254^-(l - 2) for the 8-bit
// digits (the powers of 254 are exact, so each is one rounding), l = 2 on.
__constant__ double kLevel7[8] = {0x1p-12, 0x1p-19, 0x1p-26, 0x1p-33,
                                  0x1p-40, 0x1p-47, 0x1p-54, 0x1p-61};
__constant__ double kLevel6[6] = {1.0 / 16129.0,
                                  1.0 / (16129.0 * 254.0),
                                  1.0 / (16129.0 * 254.0 * 254.0),
                                  1.0 / (16129.0 * 254.0 * 254.0 * 254.0),
                                  1.0 / (16129.0 * 254.0 * 254.0 * 254.0 * 254.0),
                                  1.0 / (16129.0 * 254.0 * 254.0 * 254.0 * 254.0 * 254.0)};
constexpr int kThreads = 320;

// The N columns at taddr of all levels, combined: smallest levels first.
template <int S, int N>
__device__ __forceinline__ void levels(uint32_t taddr, double (&acc)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) acc[i] = 0.0;
#pragma unroll 1
  for (int lev = S - 1; lev >= 0; --lev) {
    int v[N];
    if constexpr (N == 16)
      tmem_ld16_s32(taddr + static_cast<uint32_t>(lev * BN), v);
    else
      tmem_ld32_s32(taddr + static_cast<uint32_t>(lev * BN), v);
    const double w = S == 6 ? kLevel6[lev] : kLevel7[lev];
#pragma unroll
    for (int i = 0; i < N; ++i) acc[i] += exact_double(v[i]) * w;
  }
}

// What the epilogue takes matters as much as the products' rate: combining
// eight levels costs 1.6e5 FP64 operations a tile, and a tile's products last
// 57 us at K = 2400. With four warps that loaded and stored 64 columns of
// their own rows in eight round trips it was 16 us on top (the tensor pipe
// idle); eight warps, blocks turned in shared memory and the Cholesky's
// chi0 entries fetched while the products run: 3.3 us. Measured: products of
// 1000, 2400 and 4096 with their operand cutting 70, 467 and 1890 -> 57, 402
// and 1690 us, the factor of 24 x 5400 (six digits) 19.3 -> 17.1 ms, of 24 x
// 2400 3.35 -> 2.90. What is left is the products' operand traffic: a stage
// (two K steps) of S = 8 reads 96 KB of A and 144 KB of B from shared memory
// and has 96 KB written to it, 2690 clocks at 128 bytes a clock where its MMAs
// take 2300; 2684 measured.
template <int S, int EPI>
__global__ void __launch_bounds__(kThreads, 1) chol_update_kernel(const __grid_constant__ UpdateArgs p) {
  static_assert(S != 6 || EPI == EPI_CHOL, "8-bit digits: the Cholesky's planes only");
  using L = Layout<S>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  // A stage is filled and freed in G chunks of C A planes: full[0] covers the
  // first chunk and all B planes, full[g] chunk g; empty[g] the A planes of
  // chunk g and the B planes that no later step reads. One barrier per stage
  // refills it only once all of its products are done, and the next stage's
  // products are short cover for that on a few K steps: the Cholesky's factor
  // of 24 x 5400 21.2 -> 19.3 ms with chunks of two, 2400 3.55 -> 3.35 (one
  // plane a chunk: 20.9 and 3.51); a product at 3100 1.01 -> 0.99 ms with four.
  constexpr int C = EPI == EPI_CHOL ? 2 : 4, G = (S + C - 1) / C;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::kStages * L::kStageBytes);
  uint64_t *empty = full + L::kStages * G;
  uint64_t *accum = empty + L::kStages * G;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(accum + 1);
  int *fail = reinterpret_cast<int *>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int f = blockIdx.y;
  int tm = blockIdx.x / p.tiles_n, tn = blockIdx.x % p.tiles_n;
  if (EPI == EPI_GEMM) {
    // down strips of 16 column tiles: the CTAs in flight read 9 rows of A
    // tiles and 16 of B instead of 3 and all of them (from memory once the
    // planes outgrow L2: 3100 0.99 -> 0.97 ms, 4096 1.90 -> 1.88)
    const int per = 16 * p.tiles_m, first = blockIdx.x / per * 16, in = blockIdx.x % per;
    const int cols = min(16, p.tiles_n - first);
    tm = in / cols;
    tn = first + in % cols;
  }
  const int r0 = tm * BM;       // tile row (Cholesky: matrix row j0 + r0)
  const int c0 = tn * BN;       // tile column
  // uniform: the second half of a narrow last panel, a tile below the
  // diagonal of a symmetric product
  if (EPI == EPI_CHOL && c0 >= p.nb) return;
  if (EPI == EPI_GEMM && p.sym && c0 + BN <= r0) return;
  const int m = static_cast<int>(p.n - p.j0);

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * L::kStages * G; ++s) mbar_init(&full[s], 1);
    mbar_init(accum, 1);
    *fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(L::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      int it = 0;
      for (int kt = 0; kt < p.k_tiles && ok; ++kt, ++it) {
        const int s = it % L::kStages;
        const uint32_t ph = (it / L::kStages) & 1;
        uint8_t *st = smem + s * L::kStageBytes;
        uint64_t *fs = full + s * G, *es = empty + s * G;
        const int kx = kt * BKB;
#pragma unroll
        for (int g = 0; g < G; ++g) {
          if (!mbar_wait(&es[g], ph ^ 1)) { ok = false; break; }
          const int q1 = (g + 1) * C < S ? (g + 1) * C : S;
          mbar_expect_tx(&fs[g], (q1 - g * C) * L::kAPlane + (g == 0 ? S * L::kBPlane : 0));
#pragma unroll
          for (int q = g * C; q < q1; ++q) {
            const int t = S - 1 - q;
            tma_load_3d(st + q * L::kAPlane, &p.tm_a, kx, p.a_row0 + r0, q * p.nmat + f, &fs[g]);
            tma_load_3d(st + S * L::kAPlane + t * L::kBPlane, &p.tm_b, kx, p.b_row0 + c0,
                        t * p.nmat + f, &fs[0]);
          }
        }
      }
      if (!ok) {
        atomicExch(fail, 1);
        DevErr{p.err}.set(MBPT_ERR_TIMEOUT);
      }
      for (int k = max(0, it - L::kStages); k < it; ++k)
        for (int g = 0; g < G; ++g)
          mbar_wait(&full[k % L::kStages * G + g], (k / L::kStages) & 1);
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      bool ok = true;
      for (int kt = 0; kt < p.k_tiles && ok; ++kt) {
        const int s = kt % L::kStages;
        const uint32_t ph = (kt / L::kStages) & 1;
        const uint32_t st = smem_u32(smem + s * L::kStageBytes);
        // A plane sa against the B planes 1 .. S + 1 - sa stacked as one
        // operand (they lie back to back, 64 rows each): product (sa, t)
        // lands in column block sa + t - 2, its level's accumulator, so one
        // MMA of up to 256 columns serves four levels and A is read from
        // shared memory once per four products. Plane 1 covers every
        // level, so its MMAs open the accumulators. After step sa its A plane
        // and B plane S + 1 - sa are not read again.
#pragma unroll
        for (int sa = 1; sa <= S; ++sa) {
          if ((sa - 1) % C == 0) {
            if (!mbar_wait(&full[s * G + (sa - 1) / C], ph) ||
                *reinterpret_cast<volatile int *>(fail)) {
              ok = false;
              break;
            }
            tc_fence_after();
          }
#pragma unroll
          for (int kk = 0; kk < BKB / 32; ++kk) {
            const uint64_t adv = static_cast<uint64_t>(kk * 2);  // 32 bytes >> 4
            const bool first = kt == 0 && kk == 0;
            const uint64_t da = kmajor_desc(st + (sa - 1) * L::kAPlane) + adv;
#pragma unroll
            for (int t0 = 1; t0 <= S + 1 - sa; t0 += kStackPlanes) {
              const int cnt = S + 1 - sa - t0 + 1 < kStackPlanes ? S + 1 - sa - t0 + 1
                                                                  : kStackPlanes;
              const uint32_t d = tmem + static_cast<uint32_t>((sa - 1 + t0 - 1) * BN);
              const uint64_t db =
                  kmajor_desc(st + S * L::kAPlane + (t0 - 1) * L::kBPlane) + adv;
              mma_s8(d, da, db, idesc_s8(cnt * BN), (first && sa == 1) ? 0u : 1u);
            }
          }
          if (sa % C == 0 || sa == S) mma_commit(&empty[s * G + (sa - 1) / C]);
        }
      }
      if (!ok) {
        atomicExch(fail, 1);
        DevErr{p.err}.set(MBPT_ERR_TIMEOUT);
      }
      mma_commit(accum);
      mbar_wait(accum, 0);  // no MMA may still write TMEM when it is freed
    }
    __syncwarp();
  } else {
    // eight warps: rows by the TMEM lanes a warp reaches, columns by halves
    const int sp = warp & 3, ch = (warp - 2) >> 2;
    const uint32_t taddr = tmem + (static_cast<uint32_t>(sp * 32) << 16) + ch * 32;
    const int pr = r0 + sp * 32 + lane;             // tile row of this thread
    const int cb = c0 + ch * 32;                    // the warp's first column
    double old[EPI == EPI_CHOL ? 32 : 1], scol = 0.0, srow = 0.0, diag = 0.0;
    const bool live = EPI == EPI_CHOL && pr < m;
    if constexpr (EPI == EPI_CHOL) {
      // what the result takes from memory, while the products run
      const double *sc = p.scale + static_cast<int64_t>(f) * p.n + p.j0;
      const double *Arow = p.A0 + f * p.n * p.n + p.j0 * (p.n + 1) + pr;
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const int pc = cb + i;  // panel column
        old[i] = (pr == pc ? 1.0 : 0.0) - (live && pc < p.nb ? Arow[pc * p.n] : 0.0);
      }
      srow = live ? sc[pr] : 0.0;
      scol = cb + lane < p.nb ? sc[cb + lane] : 0.0;
      // the diagonal entry comes from the exact running row norm
      if (pr >= cb && pr < cb + 32 && pr < p.nb)
        diag = p.rowsq[static_cast<int64_t>(f) * p.n + p.j0 + pr];
    } else {
      srow = pr < p.m_rows ? p.alpha * p.scale[pr] : 0.0;
      scol = cb + lane < p.n_cols ? p.scale_b[cb + lane] : 0.0;
    }
    const bool ok = mbar_wait(accum, 0) && !*reinterpret_cast<volatile int *>(fail);
    __syncwarp();
    if (!ok) {
      if (lane == 0) DevErr{p.err}.set(MBPT_ERR_TIMEOUT);
    } else {
      tc_fence_after();
      if constexpr (EPI == EPI_CHOL) {
        double *Prow = p.P + static_cast<int64_t>(f) * p.p_stride + pr;
#pragma unroll
        for (int h = 0; h < 32; h += 16) {
          double acc[16];
          levels<S>(taddr + h, acc);
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int pc = cb + h + i;
            const double s = __shfl_sync(0xffffffffu, scol, h + i);
            if (live && pc < p.nb)
              Prow[static_cast<int64_t>(pc) * m] = pr == pc ? old[h + i] - diag
                                                            : old[h + i] - acc[i] * srow * s;
          }
        }
      } else {
        double acc[32];
        levels<S>(taddr, acc);
        // the warp's 32 x 32 block through shared memory (the ring is free), so
        // that rows are read and written 256 bytes at a time
        constexpr int kRow = 33;
        double *blk = reinterpret_cast<double *>(smem) + (warp - 2) * 32 * kRow;
#pragma unroll
        for (int i = 0; i < 32; ++i) blk[lane * kRow + i] = srow * acc[i];
        __syncwarp();
        const int col = cb + lane, rb = r0 + sp * 32;
        double *b2 = reinterpret_cast<double *>(smem) + (8 + warp - 2) * 32 * kRow;
        const bool two = p.H1 && p.H2;
        // this column's rows that are stored end here
        const int last = col < p.n_cols ? (p.sym ? min(p.m_rows, col + 1) : p.m_rows) - rb : 0;
#pragma unroll 1
        for (int h = 0; h < 32; h += 16) {
          double *c = p.C + static_cast<int64_t>(rb + h) * p.ldc + col;
          const int n_in = last - h;
          double v[16], g[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) v[i] = blk[(h + i) * kRow + lane] * scol;
          if (two) {
            const double *h2 = p.H2 + (c - p.C);
            double *c2 = p.C2 + (c - p.C);
#pragma unroll
            for (int i = 0; i < 16; ++i) g[i] = i < n_in ? h2[i * p.ldc] : 0.0;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              g[i] *= v[i];
              if (i < n_in) c2[i * p.ldc] = g[i];
              if (p.sym) b2[(h + i) * kRow + lane] = g[i];
            }
          }
          if (p.H1) {
            const double *h1 = p.H1 + (c - p.C);
#pragma unroll
            for (int i = 0; i < 16; ++i) g[i] = i < n_in ? h1[i * p.ldc] : 0.0;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] *= g[i];
          } else if (p.beta != 0.0) {
#pragma unroll
            for (int i = 0; i < 16; ++i) g[i] = i < n_in ? c[i * p.ldc] : 0.0;
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = v[i] + p.beta * g[i];
          }
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i < n_in) c[i * p.ldc] = v[i];
          if (p.sym) {
#pragma unroll
            for (int i = 0; i < 16; ++i) blk[(h + i) * kRow + lane] = v[i];
          }
        }
        if (p.sym && cb + 31 > rb) {
          // each entry above the diagonal also at its mirror
          __syncwarp();
#pragma unroll 8
          for (int i = 0; i < 32; ++i) {
            const int c = cb + i;
            if (pr < p.m_rows && c < p.n_cols && c > pr) {
              const int64_t mo = static_cast<int64_t>(c) * p.ldc + pr;
              p.C[mo] = blk[lane * kRow + i];
              if (two) p.C2[mo] = b2[lane * kRow + i];
            }
          }
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(L::kTmemCols)
                 : "memory");
  }
}

// scale[f][r] = 2^e_r with e_r = ceil(log2(sqrt((I - A_f)_rr))) (A column-major, ld n);
// 1 for a diagonal that is not positive and finite (that matrix fails its
// factorisation and is redone by LU; its digits only need to stay in range).
__global__ void chol_scale_kernel(const double *A, int64_t n, int64_t mat_stride, int nmat,
                                  double *scale) {
  const int64_t total = n * nmat;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t f = i / n, r = i % n;
    const double a = 1.0 - A[f * mat_stride + r * n + r];
    double s = 1.0;
    if (a > 0.0 && a < 1e300) {
      int e;
      frexp(sqrt(a), &e);          // sqrt(a) = m 2^e, m in [0.5, 1): 2^e >= sqrt(a)
      s = ldexp(1.0, e);
    }
    scale[i] = s;
  }
}

// Digits of block column [j0, j0 + nb) of L (column-major in A, ld n, rows
// j0..n-1): plane q of matrix f, row r, K = column c, at
// D[((q * nmat + f) * npad + r) * npad + c]. Rows are read contiguously through
// shared memory and written 16 columns per thread.
template <int S>
__global__ void __launch_bounds__(256) chol_slice_kernel(const double *A, int64_t n, int64_t mat_stride, int nmat,
                                  int j0, int nb, const double *scale, int8_t *D,
                                  int64_t npad, double *rownorm) {
  __shared__ double tile[32 * kCutStride];
  const int f = blockIdx.y;
  const int64_t rbase = j0 + static_cast<int64_t>(blockIdx.x) * 32;
  const double *Af = A + f * mat_stride;
  // load 32 rows x nb columns: threads walk rows fastest (column-major source),
  // 16 loads each in flight (one after the other they were half of the 12 us
  // that a step took at n = 786)
  const int lr = threadIdx.x & 31, lc = threadIdx.x >> 5;
  const int64_t gr = rbase + lr;
  double v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int cc = lc + 8 * i;
    // the factor is lower triangular: above the block's diagonal A still holds
    // 1 - chi0, which is not part of L
    v[i] = gr < n && cc < nb && gr >= j0 + cc ? Af[static_cast<int64_t>(j0 + cc) * n + gr] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < 16; ++i) tile[cut_at(lr, lc + 8 * i)] = v[i];
  __syncthreads();
  // each thread: one row, 16 consecutive columns, all S planes
  const int rr = threadIdx.x >> 3, cg = (threadIdx.x & 7) * 16;
  const int64_t r = rbase + rr;
  // the rows' running FP64 norms over the columns cut so far (the exact
  // diagonal of the later updates), summed over the 8 threads of a row in a
  // fixed order
  double sq = 0.0;
#pragma unroll
  for (int i = 0; i < 16; ++i) sq = fma(tile[cut_at(rr, cg + i)], tile[cut_at(rr, cg + i)], sq);
  sq += __shfl_xor_sync(0xffffffffu, sq, 1);
  sq += __shfl_xor_sync(0xffffffffu, sq, 2);
  sq += __shfl_xor_sync(0xffffffffu, sq, 4);
  if (r >= n) return;
  if (cg == 0) rownorm[static_cast<int64_t>(f) * n + r] += sq;
  // 7-bit digits: |t| <= 64, base 128; 8-bit (S = 6): |t| <= 127, base 254
  constexpr double kTop = S == 6 ? 127.0 : 64.0, kBase = S == 6 ? 254.0 : 128.0;
  const double inv = kTop / scale[static_cast<int64_t>(f) * n + r];
  __align__(16) int8_t out[S][16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    double t = tile[cut_at(rr, cg + i)] * inv;   // |t| <= kTop
#pragma unroll
    for (int q = 0; q < S; ++q) out[q][i] = next_digit(t, kBase);
  }
  if (cg >= nb) return;
#pragma unroll
  for (int q = 0; q < S; ++q) {
    int8_t *dst = D + ((static_cast<int64_t>(q) * nmat + f) * npad + r) * npad + j0 + cg;
    *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(out[q]);
  }
}


// An operand as the digit cutting reads it: x(i, k) = src[i ld + k], or
// src[k ld + i] with trans. rowmax (rows, zeroed by the caller) receives the
// bits of max_k |x(i, k)|, planes and scale the result.
struct Source {
  const double *src;
  int64_t rows, kdim, ld;
  int trans;
  unsigned long long *rowmax;
  double *scale;
  int8_t *planes;
  int64_t rows_pad, k_pad;
};
struct Sources {
  Source s[2];
};

// The row maxima of one or two operands (blockIdx.z). Two passes over memory
// (this and the cutting, the second mostly from L2) are what the scheme needs;
// a block takes 32 rows x 256 K columns, so that both layouts are read along
// their contiguous index with eight loads in flight per thread (32 where K runs
// along memory) and K is spread
// over blocks: with one thread per row of a transposed operand, walking all
// of K, a 2400 x 2400 operand took 200 us of latency; now 7 us. The maximum
// of non-negative doubles is that of their bits; NaN counts as nothing.
constexpr int kMaxRows = 32, kMaxK = 256;

__global__ void __launch_bounds__(256) row_max_kernel(const __grid_constant__ Sources p) {
  const Source &s = p.s[blockIdx.z];
  const int64_t i0 = static_cast<int64_t>(blockIdx.y) * kMaxRows;
  const int64_t k0 = static_cast<int64_t>(blockIdx.x) * kMaxK;
  if (i0 >= s.rows || k0 >= s.kdim) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (s.trans) {
    // lanes on rows, each warp 32 of the K columns
    __shared__ double part[8][32];
    const int64_t i = i0 + lane;
    double mx = 0.0;
    if (i < s.rows) {
#pragma unroll 8
      for (int q = 0; q < kMaxK / 8; ++q) {
        const int64_t k = k0 + warp + 8 * q;
        if (k < s.kdim) mx = fmax(mx, fabs(s.src[k * s.ld + i]));
      }
    }
    part[warp][lane] = mx;
    __syncthreads();
    if (warp == 0 && i < s.rows) {
#pragma unroll
      for (int w = 1; w < 8; ++w) mx = fmax(mx, part[w][lane]);
      if (mx > 0.0) atomicMax(s.rowmax + i, __double_as_longlong(mx));
    }
  } else {
    // each warp four rows, lanes on K
#pragma unroll
    for (int r = 0; r < kMaxRows / 8; ++r) {
      const int64_t i = i0 + warp * (kMaxRows / 8) + r;
      if (i >= s.rows) break;
      double mx = 0.0;
#pragma unroll
      for (int q = 0; q < kMaxK / 32; ++q) {
        const int64_t k = k0 + lane + 32 * q;
        if (k < s.kdim) mx = fmax(mx, fabs(s.src[i * s.ld + k]));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      if (lane == 0 && mx > 0.0) atomicMax(s.rowmax + i, __double_as_longlong(mx));
    }
  }
}

// 2^e >= the row's largest magnitude (1 for a row of zeros or with an
// infinite entry)
__device__ __forceinline__ double scale_of(unsigned long long max_bits) {
  const double mx = __longlong_as_double(static_cast<long long>(max_bits));
  int e = 0;
  frexp(mx, &e);
  return (mx > 0.0 && mx < 1e300) ? ldexp(1.0, e) : 1.0;
}

// Digit planes of one or two operands (blockIdx.z; rows x kdim, row maxima in
// rowmax): plane q, row i, column k at planes[(q rows_pad + i) k_pad + k],
// zeros beyond rows and kdim up to rows_pad and k_pad, and the rows' scales.
// One block per 32 rows x 128 columns, through shared memory so that both
// layouts of the source are read along their contiguous index.
template <int S>
__global__ void __launch_bounds__(256) operand_slice_kernel(const __grid_constant__ Sources p) {
  __shared__ double tile[32 * kCutStride];
  const Source &s = p.s[blockIdx.z];
  const int64_t i0 = static_cast<int64_t>(blockIdx.y) * 32;
  const int64_t k0 = static_cast<int64_t>(blockIdx.x) * 128;
  if (i0 >= s.rows_pad || k0 >= s.k_pad) return;
#pragma unroll 8
  for (int q = 0; q < 32 * 128 / 256; ++q) {
    const int t = threadIdx.x + 256 * q;
    const int rr = s.trans ? t & 31 : t >> 7, kk = s.trans ? t >> 5 : t & 127;
    const int64_t i = i0 + rr, k = k0 + kk;
    double v = 0.0;
    if (i < s.rows && k < s.kdim) v = s.trans ? s.src[k * s.ld + i] : s.src[i * s.ld + k];
    tile[cut_at(rr, kk)] = v;
  }
  __syncthreads();
  const int rr = threadIdx.x >> 3, cg = (threadIdx.x & 7) * 16;
  const int64_t i = i0 + rr;
  if (i >= s.rows_pad) return;
  double inv = 0.0;
  if (i < s.rows) {
    const double sc = scale_of(s.rowmax[i]);
    inv = 64.0 / sc;
    if (blockIdx.x == 0 && cg == 0) s.scale[i] = sc;
  }
  __align__(16) int8_t out[S][16];
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    double t = tile[cut_at(rr, cg + c)] * inv;     // |t| <= 64
#pragma unroll
    for (int q = 0; q < S; ++q) out[q][c] = next_digit(t, 128.0);
  }
#pragma unroll
  for (int q = 0; q < S; ++q) {
    int8_t *dst = s.planes + (static_cast<int64_t>(q) * s.rows_pad + i) * s.k_pad + k0 + cg;
    *reinterpret_cast<uint4 *>(dst) = *reinterpret_cast<const uint4 *>(out[q]);
  }
}

bool make_operand_map(CUtensorMap *m, const int8_t *planes, int64_t k_pad, int64_t rows_pad,
                      int64_t nplanes, int box_rows) {
  auto fn = encode_fn();
  if (!fn || (reinterpret_cast<uintptr_t>(planes) & 15) || k_pad % 128) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(k_pad), static_cast<cuuint64_t>(rows_pad),
                        static_cast<cuuint64_t>(nplanes)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(k_pad),
                           static_cast<cuuint64_t>(k_pad * rows_pad)};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(BKB), static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t es[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t *>(planes), dims, strides,
            box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, kTmaSwizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool make_plane_map(CUtensorMap *m, const int8_t *D, int64_t npad, int64_t planes,
                    int box_rows) {
  auto fn = encode_fn();
  if (!fn || (reinterpret_cast<uintptr_t>(D) & 15) || npad % 128) return false;
  cuuint64_t dims[3] = {static_cast<cuuint64_t>(npad), static_cast<cuuint64_t>(npad),
                        static_cast<cuuint64_t>(planes)};
  cuuint64_t strides[2] = {static_cast<cuuint64_t>(npad),
                           static_cast<cuuint64_t>(npad * npad)};
  cuuint32_t box[3] = {static_cast<cuuint32_t>(BKB), static_cast<cuuint32_t>(box_rows), 1};
  cuuint32_t es[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t *>(D), dims, strides, box,
            es, CU_TENSOR_MAP_INTERLEAVE_NONE, kTmaSwizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline int grid_blocks(int64_t n) {
  int64_t b = (n + 255) / 256;
  return static_cast<int>(b > 148 * 32 ? 148 * 32 : (b < 1 ? 1 : b));
}

}  // namespace ozaki

size_t ozaki_planes_bytes(int64_t n, int nmat, int slices) {
  const int64_t npad = round_up(n, 128);
  return static_cast<size_t>(slices) * nmat * npad * npad;
}

int ozaki_chol_scales(const double *A, int64_t n, int nmat, double *scale, double *rownorm,
                      cudaStream_t st) {
  if (cudaMemsetAsync(rownorm, 0, sizeof(double) * n * nmat, st) != cudaSuccess)
    return MBPT_ERR_CUDA;
  count_launch();
  ozaki::chol_scale_kernel<<<ozaki::grid_blocks(n * nmat), 256, 0, st>>>(A, n, n * n, nmat,
                                                                         scale);
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

int ozaki_chol_slice(const double *A, int64_t n, int nmat, int64_t j0, int nb,
                     const double *scale, int8_t *planes, int slices, double *rownorm,
                     cudaStream_t st) {
  const int64_t npad = round_up(n, 128);
  dim3 grid(static_cast<unsigned>((n - j0 + 31) / 32), nmat);
  count_launch();
  if (slices == 8)
    ozaki::chol_slice_kernel<8><<<grid, 256, 0, st>>>(A, n, n * n, nmat, static_cast<int>(j0),
                                                      nb, scale, planes, npad, rownorm);
  else if (slices == 6)
    ozaki::chol_slice_kernel<6><<<grid, 256, 0, st>>>(A, n, n * n, nmat, static_cast<int>(j0),
                                                      nb, scale, planes, npad, rownorm);
  else if (slices == 7)
    ozaki::chol_slice_kernel<7><<<grid, 256, 0, st>>>(A, n, n * n, nmat, static_cast<int>(j0),
                                                      nb, scale, planes, npad, rownorm);
  else
    return MBPT_ERR_SHAPE;
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

int ozaki_chol_update(const double *A, int64_t n, int nmat, int64_t j0, int nb, double *P,
                      const double *scale, const int8_t *planes, int slices, double *rowsq,
                      int *err, cudaStream_t st) {
  if (j0 <= 0) return MBPT_OK;
  if (j0 % ozaki::BKB || nb < 1 || nb > 128 || j0 >= 65536 ||
      (slices == 6 && j0 > kOzakiEightBitMaxK))
    return MBPT_ERR_SHAPE;
  const int64_t npad = round_up(n, 128);
  ozaki::UpdateArgs p{};
  if (!ozaki::make_plane_map(&p.tm_a, planes, npad, static_cast<int64_t>(slices) * nmat,
                             ozaki::BM) ||
      !ozaki::make_plane_map(&p.tm_b, planes, npad, static_cast<int64_t>(slices) * nmat,
                             ozaki::BN))
    return MBPT_ERR_SHAPE;
  const int64_t m = n - j0;
  p.n = n;
  p.j0 = static_cast<int>(j0);
  p.nb = nb;
  p.k_tiles = static_cast<int>(j0 / ozaki::BKB);
  p.nmat = nmat;
  p.A0 = A;
  p.P = P;
  p.p_stride = m * nb;
  p.scale = scale;
  p.rowsq = rowsq;
  p.tiles_m = static_cast<int>((m + ozaki::BM - 1) / ozaki::BM);
  p.a_row0 = p.b_row0 = static_cast<int>(j0);
  p.tiles_n = 2;
  p.scale_b = nullptr;
  p.C = nullptr;
  p.ldc = 0;
  p.alpha = p.beta = 0.0;
  p.m_rows = p.n_cols = 0;
  p.err = err;
  const dim3 grid(static_cast<unsigned>(p.tiles_m * 2), nmat);
  static std::atomic<uint64_t> attr8{0}, attr7{0}, attr6{0};
  if (slices == 6) {
    auto kern = ozaki::chol_update_kernel<6, ozaki::EPI_CHOL>;
    const int smem = ozaki::Layout<6>::kSmemBytes;
    if (!allow_smem(reinterpret_cast<const void *>(kern), smem, attr6)) return MBPT_ERR_CUDA;
    count_launch();
    kern<<<grid, ozaki::kThreads, smem, st>>>(p);
  } else if (slices == 8) {
    auto kern = ozaki::chol_update_kernel<8, ozaki::EPI_CHOL>;
    const int smem = ozaki::Layout<8>::kSmemBytes;
    if (!allow_smem(reinterpret_cast<const void *>(kern), smem, attr8)) return MBPT_ERR_CUDA;
    count_launch();
    kern<<<grid, ozaki::kThreads, smem, st>>>(p);
  } else if (slices == 7) {
    auto kern = ozaki::chol_update_kernel<7, ozaki::EPI_CHOL>;
    const int smem = ozaki::Layout<7>::kSmemBytes;
    if (!allow_smem(reinterpret_cast<const void *>(kern), smem, attr7)) return MBPT_ERR_CUDA;
    count_launch();
    kern<<<grid, ozaki::kThreads, smem, st>>>(p);
  } else {
    return MBPT_ERR_SHAPE;
  }
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

// ---- the general FP64-accurate GEMM ------------------------------------------
// Largest K of one product pass: S 64^2 K must stay below 2^31 (S <= 8).

size_t ozaki_gemm_scratch_bytes(int64_t m, int64_t n, int64_t k, int slices) {
  const int64_t kc = std::min<int64_t>(round_up(k, 128), kOzakiKChunk);
  const int64_t mp = round_up(m, 128), np = round_up(n, 128);
  return static_cast<size_t>(slices) * (mp + np) * kc + 16 * (mp + np) + 4096;
}

// The row maxima and digit planes of `count` operands (their rowmax words
// zeroed by the caller).
static int cut_operands(const ozaki::Sources &src, int count, int slices, cudaStream_t st) {
  if (count == 0) return MBPT_OK;
  int64_t rmax = 0, kmax = 0, kpmax = 0;
  for (int i = 0; i < count; ++i) {
    rmax = std::max(rmax, src.s[i].rows_pad);
    kmax = std::max(kmax, src.s[i].kdim);
    kpmax = std::max(kpmax, src.s[i].k_pad);
  }
  const dim3 gm(static_cast<unsigned>((kmax + ozaki::kMaxK - 1) / ozaki::kMaxK),
                static_cast<unsigned>(rmax / ozaki::kMaxRows), count);
  const dim3 gs(static_cast<unsigned>(kpmax / 128), static_cast<unsigned>(rmax / 32), count);
  count_launch(2);
  ozaki::row_max_kernel<<<gm, 256, 0, st>>>(src);
  if (slices == 8)
    ozaki::operand_slice_kernel<8><<<gs, 256, 0, st>>>(src);
  else
    ozaki::operand_slice_kernel<7><<<gs, 256, 0, st>>>(src);
  return cudaGetLastError() == cudaSuccess ? MBPT_OK : MBPT_ERR_CUDA;
}

size_t ozaki_operand_bytes(int64_t rows, int64_t k) {
  const int64_t rp = round_up(rows, 128);
  return static_cast<size_t>(8) * rp * round_up(k, 128) + 16 * rp + 1024;
}

int ozaki_cut(const double *src, int64_t rows, int64_t k, int64_t ld, bool trans, void *buf,
              OzakiOperand *op, cudaStream_t st) {
  *op = OzakiOperand();
  if (k > kOzakiKChunk || k < 1 || rows < 1) return MBPT_OK;  // cut chunk by chunk instead
  const int64_t rp = round_up(rows, 128), kp = round_up(k, 128);
  int8_t *planes = static_cast<int8_t *>(buf);
  double *scale = reinterpret_cast<double *>(planes + 8 * rp * kp);
  unsigned long long *rowmax = reinterpret_cast<unsigned long long *>(scale + rp);
  if (cudaMemsetAsync(rowmax, 0, sizeof(unsigned long long) * rp, st) != cudaSuccess)
    return MBPT_ERR_CUDA;
  ozaki::Sources s{};
  s.s[0] = {src, rows, k, ld, trans ? 1 : 0, rowmax, scale, planes, rp, kp};
  *op = {planes, scale, rows, k};
  return cut_operands(s, 1, 8, st);
}

int ozaki_dgemm(bool ta, bool tb, int64_t m, int64_t n, int64_t k, double alpha,
                const double *A, int64_t lda, const double *B, int64_t ldb, double beta,
                double *C, int64_t ldc, int slices, void *scratch, size_t scratch_bytes,
                int *err, cudaStream_t st, const OzakiEpi *epi) {
  if (m < 1 || n < 1 || k < 1) return MBPT_ERR_SHAPE;
  if (slices != 7 && slices != 8) return MBPT_ERR_SHAPE;
  const OzakiEpi none;
  const OzakiEpi &x = epi ? *epi : none;
  if (x.sym && m != n) return MBPT_ERR_SHAPE;
  if (x.h1 && (beta != 0.0 || k > kOzakiKChunk || (x.h2 && !x.c2))) return MBPT_ERR_SHAPE;
  if (scratch_bytes < ozaki_gemm_scratch_bytes(m, n, k, slices)) return MBPT_ERR_WORKSPACE;
  // operands cut beforehand (one pass, 8 digits)
  const bool one = k <= kOzakiKChunk && slices == 8;
  const OzakiOperand *ca = one && x.a && x.a->planes ? x.a : nullptr;
  const OzakiOperand *cb = one && x.b && x.b->planes ? x.b : nullptr;
  if ((ca && (ca->rows != m || ca->k != k)) || (cb && (cb->rows != n || cb->k != k)))
    return MBPT_ERR_SHAPE;
  const int64_t mp = round_up(m, 128), np = round_up(n, 128);
  static std::atomic<uint64_t> attr8{0}, attr7{0};
  for (int64_t kb = 0; kb < k; kb += kOzakiKChunk) {
    const int64_t kc = std::min<int64_t>(kOzakiKChunk, k - kb);
    const int64_t kp = round_up(kc, 128);
    uint8_t *base = static_cast<uint8_t *>(scratch);
    int8_t *pa = reinterpret_cast<int8_t *>(base);
    int8_t *pb = pa + static_cast<int64_t>(slices) * mp * kp;
    double *sa = reinterpret_cast<double *>(
        (reinterpret_cast<uintptr_t>(pb + static_cast<int64_t>(slices) * np * kp) + 255) &
        ~static_cast<uintptr_t>(255));
    double *sb = sa + mp;
    unsigned long long *ma = reinterpret_cast<unsigned long long *>(sb + np), *mb = ma + mp;
    // op(A) rows are K-contiguous unless ta; op(B) = B^T rows unless tb
    ozaki::Sources src{};
    int count = 0;
    if (!ca)
      src.s[count++] = {ta ? A + kb * lda : A + kb, m, kc, lda, ta ? 1 : 0, ma, sa, pa, mp, kp};
    if (!cb)
      src.s[count++] = {tb ? B + kb : B + kb * ldb, n, kc, ldb, tb ? 0 : 1, mb, sb, pb, np, kp};
    if (count && cudaMemsetAsync(ma, 0, sizeof(unsigned long long) * (mp + np), st) != cudaSuccess)
      return MBPT_ERR_CUDA;
    const int rc = cut_operands(src, count, slices, st);
    if (rc) return rc;
    if (ca) {
      pa = ca->planes;
      sa = ca->scale;
    }
    if (cb) {
      pb = cb->planes;
      sb = cb->scale;
    }
    ozaki::UpdateArgs p{};
    if (!ozaki::make_operand_map(&p.tm_a, pa, kp, mp, slices, ozaki::BM) ||
        !ozaki::make_operand_map(&p.tm_b, pb, kp, np, slices, ozaki::BN))
      return MBPT_ERR_SHAPE;
    p.n = 0;
    p.j0 = 0;
    p.nb = 0;
    p.k_tiles = static_cast<int>(kp / ozaki::BKB);
    p.nmat = 1;
    p.a_row0 = p.b_row0 = 0;
    p.tiles_m = static_cast<int>(mp / ozaki::BM);
    p.tiles_n = static_cast<int>((n + ozaki::BN - 1) / ozaki::BN);
    p.P = nullptr;
    p.p_stride = 0;
    p.scale = sa;
    p.scale_b = sb;
    p.rowsq = nullptr;
    p.C = C;
    p.ldc = ldc;
    p.alpha = alpha;
    p.beta = kb == 0 ? beta : 1.0;
    p.m_rows = static_cast<int>(m);
    p.n_cols = static_cast<int>(n);
    p.sym = x.sym ? 1 : 0;
    p.H1 = x.h1;
    p.H2 = x.h1 ? x.h2 : nullptr;
    p.C2 = x.c2;
    p.err = err;
    const dim3 grid(static_cast<unsigned>(p.tiles_m * p.tiles_n), 1);
    count_launch();
    if (slices == 8) {
      auto kern = ozaki::chol_update_kernel<8, ozaki::EPI_GEMM>;
      const int smem = ozaki::Layout<8>::kSmemBytes;
      if (!allow_smem(reinterpret_cast<const void *>(kern), smem, attr8)) return MBPT_ERR_CUDA;
      kern<<<grid, ozaki::kThreads, smem, st>>>(p);
    } else {
      auto kern = ozaki::chol_update_kernel<7, ozaki::EPI_GEMM>;
      const int smem = ozaki::Layout<7>::kSmemBytes;
      if (!allow_smem(reinterpret_cast<const void *>(kern), smem, attr7)) return MBPT_ERR_CUDA;
      kern<<<grid, ozaki::kThreads, smem, st>>>(p);
    }
    if (cudaGetLastError() != cudaSuccess) return MBPT_ERR_CUDA;
  }
  return MBPT_OK;
}

}  // namespace mbpt
