// Dense FP64 complex helpers for the GCG eigensolver (see k_dense.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace ncgm {

// C (p x q, ld ldc) = A^H B; partials: >= maxChunks * p * q double2.
void gram(const double2 *A, size_t lda, int p, const double2 *B, size_t ldb,
          int q, size_t N, double2 *C, int ldc, double2 *partials,
          int maxChunks, cudaStream_t s);
int gramMaxChunks();
// C = A^H B on the tensor cores (tcgen05 kind::tf32, split TF32 products,
// FP32 accumulation over row chunks, FP64 chunk sums; k_tcgram.cu). part:
// tcGramPartialFloats(N, p, q) floats.
void gramTC(const double2 *A, size_t lda, int p, const double2 *B, size_t ldb,
            int q, size_t N, double2 *C, int ldc, float *part,
            cudaStream_t s);
size_t tcGramPartialFloats(size_t N, int p, int q);
int *tcGramErrWord();
// C = A^H B on the tensor cores: error-free splitting into 6 (~1e-13 relative)
// or 8 (FP64 accuracy) BF16 integer digits (digitised once per operand),
// exact FP32 level sums, exact integer combination (k_tcgram_exact.cu).
// scratch: exactGramScratchDoubles(N, p, q, digits) doubles, 16-byte aligned.
// 8 digits: operands with infinities, NaNs or extreme magnitudes take a plain
// FP64 sum on the device. err (device): set to 1 when a bounded wait gives up.
void gramTCExact(const double2 *A, size_t lda, int p, const double2 *B,
                 size_t ldb, int q, size_t N, double2 *C, int ldc,
                 double *scratch, cudaStream_t s, int digits, int *err);
// self: for Grams of a block with itself alone (half of the images)
size_t exactGramScratchDoubles(size_t N, int p, int q, int digits,
                               bool self = false);
// Y = V C on the tensor cores with the exact digit products of gramTCExact
// (6 digits: ~1e-12 relative of the column maxima; 8: FP64 accuracy;
// k_tcgram_exact.cu). scratch: exactVCScratchBytes(N, m, k, digits) bytes,
// 16-byte aligned.
void gemmVCExact(const double2 *V, size_t ldv, int m, const double2 *C,
                 int ldc, int k, double2 *Y, size_t ldy, size_t N,
                 void *scratch, cudaStream_t s, bool accum, int digits,
                 int *err);
size_t exactVCScratchBytes(size_t N, int m, int k, int digits);
// Y = V C + beta Y (V: N x m with m <= 1600, C: m x k; C is staged in
// shared memory in blocks of columns).
void gemmVC(const double2 *V, size_t ldv, int m, const double2 *C, int ldc,
            int k, double2 *Y, size_t ldy, size_t N, double beta,
            cudaStream_t s);
// Whether the 8-digit tensor-core products beat the plain FP64 kernels for
// C (p x q) = A^H B and Y (N x k) = V (N x m) C.
bool digitsPayGram(size_t N, int p, int q);
bool digitsPayVC(size_t N, int m, int k);
// The products of tall blocks in one of three forms: 6 digits (tensor-core
// precision form), 8 digits (FP64 accuracy on the tensor cores, where
// digitsPay) or the plain FP64 kernels (no scratch, or small blocks).
struct BlockProducts {
  int digits = 8;
  double *gramScr = nullptr; // exactGramScratchDoubles
  void *vcScr = nullptr;     // exactVCScratchBytes (may be the same memory)
  int *err = nullptr;        // the context's error word (with scratch)
  double2 *partials = nullptr; // plain Gram: maxChunks p q
  int maxChunks = 1;
  // C = A^H B
  void gram(const double2 *A, size_t lda, int p, const double2 *B, size_t ldb,
            int q, size_t N, double2 *C, int ldc, cudaStream_t s) const;
  // Y = V C (accum: Y += V C)
  void vc(const double2 *V, size_t ldv, int m, const double2 *C, int ldc,
          int k, double2 *Y, size_t ldy, size_t N, cudaStream_t s,
          bool accum = false) const;
};
// Cholesky of Gram G with MGS-equivalent drop; T = R^{-1}; keep flags.
// fast: the FP32 forms' variant (double-float pivot roots and reciprocals).
void cholDrop(const double2 *G, int ldg, int m, double dropTol, double2 *R,
              double2 *T, int *keep, cudaStream_t s, bool fast = false);
// Multi-kernel Hermitian eigensolver for m > 80 (k_heig_large.cu): Householder
// tridiagonalisation, bisection, inverse iteration, back-transformation.
void heigLarge(const double2 *A, int lda, int m, double2 *V, double *w,
               int *perm, int *status, void *scratch, cudaStream_t s);
size_t heigLargeScratchBytes(int m);
// The same method with the tridiagonalisation in one CTA and the matrix in
// shared memory, for m <= heigMidMax() (k_heig_large.cu).
void heigMid(const double2 *A, int lda, int m, double2 *V, double *w,
             int *perm, int *status, void *scratch, cudaStream_t s);
size_t heigMidScratchBytes(int m);
int heigMidMax();
// FP64 solver for the sizes that heigRefinedTakes: heigMid and one step of FP64
// refinement (k_heig_refine.cu). *status = 1: it gave up, solve again.
bool heigRefinedTakes(int m);
size_t heigRefinedScratchBytes(int m);
void heigRefined(const double2 *A, int lda, int m, double2 *V, double *w,
                 int *perm, int *status, void *scratch, cudaStream_t s);
// Hermitian eigensolver (lower triangle): w ascending, V eigenvectors (m x m).
// fast (the FP32 precision forms): for m <= heigMidMax(), the one-CTA
// double-float Householder method (heigMid; with NCGM_HEIG_MID=0 the
// double-float Jacobi up to m = 80); otherwise the FP64 Jacobi below
// m = 48, the refined method up to m = 80 and the multi-kernel Householder
// method above it. Degenerate eigenvectors
// may come out rotated within their eigenspace between the methods.
// scratch (optional, heigScratchBytes(m) bytes): the Householder methods'
// workspace; without it they take stream-ordered allocations per call.
void heig(const double2 *A, int lda, int m, double2 *work, double2 *V,
          double *w, int *perm, int *status, cudaStream_t s,
          bool fast = false, void *scratch = nullptr,
          size_t scratchBytes = 0);
size_t heigScratchBytes(int m);

} // namespace ncgm
