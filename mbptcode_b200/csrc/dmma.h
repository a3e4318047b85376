// FP64 products on the FP64 tensor pipe (dmma.cu), batched over tau points.
#pragma once
#include "internal.h"

namespace mbpt {
namespace dmma {

// An FP64 operand: element (r, k) at p[r ld + k] (K contiguous) or
// p[k ld + r] (rows contiguous), `stride` doubles between batch members
// (0: the same for all).
struct Operand {
  const double *p = nullptr;
  int64_t ld = 0, stride = 0;
};

// C (m x n, row-major, ldc) = alpha A B^T + beta C per batch member, A (m x k)
// and B (n x k) K-contiguous (a_k, b_k) or row-contiguous (not A
// row-contiguous with B K-contiguous). upper: the product is symmetric (m ==
// n): the tiles on and above the diagonal are formed and mirrored. half: A
// (m x m, K-contiguous) is held by halves (below): of each row tile, K runs
// from the tile's first row on.
int gemm(const Operand &a, bool a_k, const Operand &b, bool b_k, int64_t m, int64_t n, int64_t k,
         double alpha, double beta, double *c, int64_t ldc, int64_t sc, int batch, bool upper,
         cudaStream_t st, bool half = false);

// C_0 + ... + C_{parts-1} = alpha A B^T, A K-contiguous (a_k) or row-contiguous,
// B row-contiguous: each part sums its own range of K and lies batch sc doubles
// after the one before.
// product_parts: the number of parts that fills the GPU (1 to kMaxParts).
// cut_parts: 1 unless the time that uneven rounds of CTAs cost (0.55 us per 16
// columns of K and round) is well above that of a pass that adds the parts, 24
// us. square_parts: the same for a symmetric n x n product, all of it in parts
// against its upper tiles in one piece, 16 us. chi0 of one tau point, in one
// piece, cut, and by the library's products (M x naux, us): 444 x 100 164, 132
// and 133; 888 x 141 193, 147 and 150; 1332 x 236 265, 181 and 187; 1332 x 700
// 303, 281 and 298; 2000 x 300 402, 272 and 289; of two points 2000 x 300 504,
// 393 and 484. Not worth it, in one piece and cut: 444 x 300 of four points 163
// and 170, 444 x 100 of twenty 188 and 196.
constexpr int kMaxParts = 8;
int product_parts(int64_t m, int64_t n, int64_t k, int batch);
int cut_parts(int64_t m, int64_t n, int64_t k, int batch);
int square_parts(int64_t n, int64_t k, int batch);
int gemm_parts(const Operand &a, bool a_k, const Operand &b, int64_t m, int64_t n, int64_t k,
               double alpha, double *c, int64_t ldc, int64_t sc, int batch, int parts,
               cudaStream_t st);

// C (m x m) = (A0 B0^T) o (A1 B1^T), both symmetric: Pi = G_occ o G_virt.
// All operands K-contiguous. g0, g1: the two factors as well, laid out as C
// (both or neither). half: C is held by halves, the 64 x 64 tiles on and above
// the diagonal only, the diagonal ones times 1/2, so that C = T + T^T for the
// T that is stored.
int hadamard_product(const Operand &a0, const Operand &b0, int64_t k0, const Operand &a1,
                     const Operand &b1, int64_t k1, int64_t m, double *c, int64_t ldc,
                     int64_t sc, int batch, cudaStream_t st, double *g0 = nullptr,
                     double *g1 = nullptr, bool half = false);

// Zt = U D^T, hl = (Xo_s Xo^T) o Zt and hg = (Xv_s Xv^T) o Zt (all symmetric,
// K-contiguous operands), leading dimension m, as `half_quadratic` reads
// them: the 64 x 64 tiles on and above the diagonal only, the diagonal ones
// times 1/2. zt not null: Zt (m x m, its upper triangle, the same for the
// whole batch) is read instead of formed from u and d.
int sigma_h(const double *zt, const Operand &u, const Operand &d, int64_t naux,
            const Operand &xo_s, const Operand &xo, int64_t nocc, const Operand &xv_s,
            const Operand &xv, int64_t nv, int64_t m, double *hl, double *hg, int64_t sh,
            int batch, cudaStream_t st);

// out_l[p] += x_p^T Hl x_p and out_g[p] -= x_p^T Hg x_p for the ns columns x_p
// of xs (m x ns) and the symmetric Hl and Hg held as sigma_h leaves them: twice
// the sum over their tiles.
int half_quadratic(const double *hl, const double *hg, int64_t sh, int64_t m, const double *xs,
                   int64_t ns, double *out_l, double *out_g, int64_t s_out, int batch,
                   cudaStream_t st);

// One step of the left-looking Cholesky of I - chi0 for `batch` row-major
// n x n matrices whose rows above j0 hold the factor U (I - chi0 = U^T U):
// P (nbj x (n - j0)) = (I - chi0)[j0:j0+nbj, j0:] - U[:j0, j0:j0+nbj]^T U[:j0, j0:],
// on and above the diagonal.
int chol_update(const double *chi0, int64_t n, int64_t j0, int nbj, double *P, int batch,
                cudaStream_t st);

// The triangular inverse halves down to diagonal blocks of this many rows.
constexpr int64_t kInverseLeaf = 128;

// chi0 <- U^-1 U^-T - I for `batch` factors U (the upper triangles of the
// row-major n x n chi0; the strict lower ones are not read), symmetric to the
// bit. V: batch x n x ldv doubles of scratch (ldv >= n) whose kInverseLeaf
// diagonal blocks hold the inverses of U's, zeros below the diagonal. Where a
// matrix's info word is not zero nothing is written.
int spd_inverse(double *chi0, int64_t n, double *V, int64_t ldv, const int *info, int batch,
                cudaStream_t st);

}  // namespace dmma
}  // namespace mbpt
