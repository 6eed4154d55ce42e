// FP64 Hermitian eigensolver for 48 <= m <= 80: the double-float Householder
// method (heigMid) gives eigenvectors with residuals of about 1e-13, and FP64
// refinement brings them to the rounding of two FP64 products.
//
// Its inverse iteration leaves vectors of close eigenvalues orthogonal to 1e-5
// only: two Newton-Schulz steps X (I + R / 2) first, each squaring R.
// With X the approximate eigenvectors, R = I - X^H X and S = X^H A X, the
// correction E of X (I + E) is (Ogita and Aishima, Iterative refinement for
// symmetric eigenvalue decomposition, 2018)
//   E_ij = (S_ij + l_j R_ij) / (l_j - l_i),  E_ij = R_ij / 2 on the diagonal
// and for close eigenvalues, l_i = S_ii / (1 - R_ii). The first form is
// quadratic in its own size, so it is taken where it is below 3e-9; pairs that
// it leaves out (clusters, such as the twofold levels of time-reversal
// symmetry) keep a residual of X's size and are resolved by Jacobi rotations
// of S = X^H A X that skip every pair already at rounding level.
//
// A cyclic Jacobi from the start is bound by the FP64 pipe of one SM: about
// ten sweeps of m^2 / 2 rotations, all of them full. m = 60: 5100 -> 1250 us,
// m = 80 (occupations, most of them near 0 or 1): 19300 -> 2900 us.
#include "k_dense.cuh"

#include <cuda_runtime.h>

#include <algorithm>

namespace ncgm {

namespace {

constexpr int kRefMin = 48, kRefMax = 80;
constexpr int kJacobiT = 512;
constexpr int kMaxSweeps = 30;

struct RefState {
  double scale; // A = scale * (the scaled copy)
  int bad;      // the method gives up: not finite, or X too far off
  int pad;
};

// Full Hermitian copy of A (lower triangle read), divided by the power of two
// of its largest entry: the double-float stage has the exponent range of FP32.
__global__ void __launch_bounds__(kJacobiT)
    refPrepKernel(const double2 *A, int lda, int m, double2 *As, RefState *st) {
  __shared__ int top;
  if (threadIdx.x == 0) top = 0;
  __syncthreads();
  int e = 0;
  for (int q = threadIdx.x; q < m * m; q += kJacobiT) {
    const int i = q % m, j = q / m;
    if (i < j) continue;
    const double2 v = A[(size_t)j * lda + i];
    e = max(e, (__double2hiint(v.x) >> 20) & 0x7FF);
    if (i > j) e = max(e, (__double2hiint(v.y) >> 20) & 0x7FF);
  }
  e = __reduce_max_sync(0xffffffffu, e);
  if (threadIdx.x % 32 == 0) atomicMax(&top, e);
  __syncthreads();
  const int big = top;
  const bool bad = big == 0x7FF;
  const int ex = big == 0 ? 0 : max(-1000, min(1000, big - 1023));
  const double down = ldexp(1.0, -ex);
  if (threadIdx.x == 0) *st = {ldexp(1.0, ex), bad, 0};
  for (int q = threadIdx.x; q < m * m; q += kJacobiT) {
    const int i = q % m, j = q / m;
    double2 v = i >= j ? A[(size_t)j * lda + i] : A[(size_t)i * lda + j];
    if (i < j) v.y = -v.y;
    if (i == j) v.y = 0.0;
    As[q] = bad ? make_double2(i == j ? 1.0 : 0.0, 0.0)
                : make_double2(v.x * down, v.y * down);
  }
}

// C = op(A) B (+ D), m x m: op(A) = A^H or A. A block makes 8 x 8 elements, so
// that m = 60 fills 64 SMs; an element's four real sums are independent chains.
struct Product {
  const double2 *A, *B, *D;
  double2 *C;
};
constexpr int kTileO = 8, kTileK = 16;
template <bool kConj>
__global__ void __launch_bounds__(kTileO *kTileO)
    refMulKernel(Product p0, Product p1, int m) {
  __shared__ double2 a[kTileK][kTileO + 1], b[kTileK][kTileO + 1];
  const Product p = blockIdx.z ? p1 : p0;
  const int i0 = blockIdx.x * kTileO, j0 = blockIdx.y * kTileO;
  const int ti = threadIdx.x % kTileO, tj = threadIdx.x / kTileO;
  const double2 zero = make_double2(0.0, 0.0);
  double xx = 0, yy = 0, xy = 0, yx = 0;
  for (int k0 = 0; k0 < m; k0 += kTileK) {
    for (int e = threadIdx.x; e < kTileO * kTileK; e += kTileO * kTileO) {
      // neighbouring threads read along the contiguous index
      const int k = e % kTileK, o = e / kTileK;
      const int kk = k0 + k;
      if (kConj)
        a[k][o] = kk < m && i0 + o < m ? p.A[(size_t)(i0 + o) * m + kk] : zero;
      b[k][o] = kk < m && j0 + o < m ? p.B[(size_t)(j0 + o) * m + kk] : zero;
      if (!kConj) {
        const int i = i0 + e % kTileO, q = k0 + e / kTileO;
        a[e / kTileO][e % kTileO] =
            q < m && i < m ? p.A[(size_t)q * m + i] : zero;
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kTileK; ++k) {
      const double2 u = a[k][ti], v = b[k][tj];
      xx = fma(u.x, v.x, xx);
      yy = fma(u.y, v.y, yy);
      xy = fma(u.x, v.y, xy);
      yx = fma(u.y, v.x, yx);
    }
    __syncthreads();
  }
  const int i = i0 + ti, j = j0 + tj;
  if (i >= m || j >= m) return;
  double2 c = kConj ? make_double2(xx + yy, xy - yx)
                    : make_double2(xx - yy, xy + yx);
  if (p.D) {
    const double2 d = p.D[(size_t)j * m + i];
    c.x += d.x;
    c.y += d.y;
  }
  p.C[(size_t)j * m + i] = c;
}

// E from G = X^H X and S = X^H A X (without S: the Newton-Schulz step R / 2)
__global__ void refCorrectionKernel(const double2 *G, const double2 *S, int m,
                                    double limit, double2 *E, RefState *st) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= m * m) return;
  const int i = q % m, j = q / m;
  const double2 g = G[q];
  const double2 r = make_double2((i == j ? 1.0 : 0.0) - g.x, -g.y);
  double2 e = make_double2(0.5 * r.x, 0.5 * r.y);
  // what X (I + E) leaves is of the order of R^2: above the limit (1e-2 before
  // the two Newton-Schulz steps, 3e-9 after them) the method gives up. The
  // comparison fails for NaN.
  if (!(fabs(r.x) + fabs(r.y) < limit)) st->bad = 1;
  if (S && i != j) {
    // the Hermitian part of S: its rounding over a small gap would otherwise
    // enter the lengths and angles of the new vectors
    const double2 up = S[q], lo = S[(size_t)i * m + j];
    const double2 s = make_double2(0.5 * (up.x + lo.x), 0.5 * (up.y - lo.y));
    const double li = S[(size_t)i * m + i].x / G[(size_t)i * m + i].x,
                 lj = S[(size_t)j * m + j].x / G[(size_t)j * m + j].x;
    const double gap = lj - li;
    // |S_ij| + |l| |R_ij| bounds the numerators of E_ij and E_ji alike
    const double num = fabs(s.x) + fabs(s.y) +
                       fmax(fabs(li), fabs(lj)) * (fabs(r.x) + fabs(r.y));
    if (num < 3e-9 * fabs(gap)) {
      // E_ij = R_ij / 2 + K_ij with K_ji = -conj(K_ij)
      const double inv = 1.0 / gap, mean = 0.5 * (li + lj);
      e.x += (s.x + mean * r.x) * inv;
      e.y += (s.y + mean * r.y) * inv;
    }
  }
  E[q] = e;
}

// Jacobi rotations of S = X^H A X in one CTA, on the pairs whose element is
// above the rounding of S, applied to the columns of X; then the eigenvalues
// in ascending order and the columns in the same order.
__global__ void __launch_bounds__(kJacobiT)
    refJacobiKernel(const double2 *S, int m, double2 *X, double2 *V, double *w,
                    int *perm, int *status, const RefState *st) {
  extern __shared__ double2 As[];
  __shared__ int P[kRefMax / 2], Q[kRefMax / 2], nact;
  __shared__ double C[kRefMax / 2], Sn[kRefMax / 2], red[kJacobiT / 32];
  __shared__ double2 E[kRefMax / 2];
  __shared__ double ev[kRefMax];
  const int tid = threadIdx.x;
  if (st->bad) {
    if (tid == 0) *status = 1;
    return;
  }
  double big = 0.0;
  for (int q = tid; q < m * m; q += kJacobiT) {
    As[q] = S[q];
    if (q % m == q / m) big = fmax(big, fabs(S[q].x));
  }
  for (int o = 16; o > 0; o >>= 1)
    big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
  if (tid % 32 == 0) red[tid / 32] = big;
  __syncthreads();
  for (int k = 0; k < kJacobiT / 32; ++k) big = fmax(big, red[k]);
  // four roundings of the largest eigenvalue: below the error of S itself
  const double tol = 4.4e-16 * big;
  const int mp = m + m % 2, npairs = mp / 2;
  bool clean = false;
  for (int sweep = 0; sweep < kMaxSweeps && !clean; ++sweep) {
    clean = true;
    for (int r = 0; r < mp - 1; ++r) {
      // round-robin: pair k of round r
      int p = 0, q = 0;
      double2 apq = make_double2(0.0, 0.0);
      bool act = false;
      if (tid < npairs) {
        const int a = tid == 0 ? mp - 1 : (r + tid) % (mp - 1);
        const int b = tid == 0 ? r : (r - tid + (mp - 1)) % (mp - 1);
        p = min(a, b);
        q = max(a, b);
        if (q < m) {
          apq = As[(size_t)q * m + p];
          act = fmax(fabs(apq.x), fabs(apq.y)) > tol;
        }
      }
      if (tid == 0) nact = 0;
      if (!__syncthreads_or(act)) continue;
      clean = false;
      if (act) {
        const double mag = sqrt(apq.x * apq.x + apq.y * apq.y);
        const double app = As[(size_t)p * m + p].x,
                     aqq = As[(size_t)q * m + q].x;
        const double tau = (aqq - app) / (2.0 * mag);
        const double t =
            (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
        const double c = 1.0 / sqrt(1.0 + t * t);
        // the pairs of a round are disjoint: their order is immaterial
        const int k = atomicAdd(&nact, 1);
        P[k] = p;
        Q[k] = q;
        C[k] = c;
        Sn[k] = t * c;
        E[k] = make_double2(apq.x / mag, apq.y / mag);
      }
      __syncthreads();
      const int n = nact;
      // S <- S U and X <- X U
      for (int e = tid; e < 2 * m * n; e += kJacobiT) {
        const int row = e % m, k = e / m % n;
        double2 *M = e < m * n ? As : X;
        double2 &x = M[(size_t)P[k] * m + row], &y = M[(size_t)Q[k] * m + row];
        const double c = C[k], s = Sn[k];
        const double2 u = E[k], xv = x, yv = y;
        const double2 t = make_double2(u.x * yv.x + u.y * yv.y,
                                       u.x * yv.y - u.y * yv.x); // conj(u) y
        x = make_double2(c * xv.x - s * t.x, c * xv.y - s * t.y);
        y = make_double2(s * xv.x + c * t.x, s * xv.y + c * t.y);
      }
      __syncthreads();
      // S <- U^H S
      for (int e = tid; e < m * n; e += kJacobiT) {
        const int col = e % m, k = e / m;
        double2 &x = As[(size_t)col * m + P[k]], &y = As[(size_t)col * m + Q[k]];
        const double c = C[k], s = Sn[k];
        const double2 u = E[k], xv = x, yv = y;
        const double2 t = make_double2(u.x * yv.x - u.y * yv.y,
                                       u.x * yv.y + u.y * yv.x); // u y
        x = make_double2(c * xv.x - s * t.x, c * xv.y - s * t.y);
        y = make_double2(s * xv.x + c * t.x, s * xv.y + c * t.y);
      }
      __syncthreads();
      if (tid < n) {
        const int a = P[tid], b = Q[tid];
        As[(size_t)b * m + a] = make_double2(0.0, 0.0);
        As[(size_t)a * m + b] = make_double2(0.0, 0.0);
        As[(size_t)a * m + a].y = 0.0;
        As[(size_t)b * m + b].y = 0.0;
      }
      __syncthreads();
    }
  }
  if (tid < m) ev[tid] = As[(size_t)tid * m + tid].x;
  __syncthreads();
  __shared__ int rank[kRefMax];
  if (tid < m) {
    const double x = ev[tid];
    int k = 0;
    for (int j = 0; j < m; ++j) k += ev[j] < x || (ev[j] == x && j < tid);
    rank[tid] = k;
    w[k] = x * st->scale;
    perm[k] = k;
  }
  if (tid == 0) *status = clean ? 0 : 1;
  __syncthreads();
  for (int q = tid; q < m * m; q += kJacobiT)
    V[(size_t)rank[q / m] * m + q % m] = X[q];
}

} // namespace

bool heigRefinedTakes(int m) { return m >= kRefMin && m <= kRefMax; }

size_t heigRefinedScratchBytes(int m) {
  return heigMidScratchBytes(m) + 256 + // heigMid's, and its alignment
         6 * ((size_t)m * m * sizeof(double2) + 256) + 512;
}

// *status = 0: V and w hold the result; 1: the method gave up (V, w undefined)
void heigRefined(const double2 *A, int lda, int m, double2 *V, double *w,
                 int *perm, int *status, void *scratch, cudaStream_t s) {
  const size_t mm = (size_t)m * m;
  char *p = static_cast<char *>(scratch);
  auto take = [&](size_t bytes) {
    char *r = p;
    p += (bytes + 255) & ~(size_t)255;
    return r;
  };
  double2 *M[6];
  for (auto &x : M) x = reinterpret_cast<double2 *>(take(mm * sizeof(double2)));
  auto *st = reinterpret_cast<RefState *>(take(sizeof(RefState)));
  double2 *As = M[0], *G = M[1], *S = M[2], *B = M[3], *E = M[4], *X = M[5];
  const int smem = kRefMax * kRefMax * (int)sizeof(double2);
  // a per-device attribute: set on every call
  cudaFuncSetAttribute(refJacobiKernel,
                       cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  refPrepKernel<<<1, kJacobiT, 0, s>>>(A, lda, m, As, st);
  heigMid(As, m, m, V, w, perm, status, p, s);
  const unsigned t = (unsigned)((m + kTileO - 1) / kTileO);
  const dim3 one(t, t, 1), two(t, t, 2);
  const Product none{};
  const int thr = kTileO * kTileO;
  const unsigned ge = (unsigned)((mm + 127) / 128);
  auto schulz = [&](const double2 *from, double2 *to) {
    refMulKernel<true><<<one, thr, 0, s>>>({from, from, nullptr, G}, none, m);
    refCorrectionKernel<<<ge, 128, 0, s>>>(G, nullptr, m, 1e-2, E, st);
    refMulKernel<false><<<one, thr, 0, s>>>({from, E, from, to}, none, m);
  };
  schulz(V, X);
  schulz(X, V);
  refMulKernel<true><<<two, thr, 0, s>>>({As, V, nullptr, B},
                                         {V, V, nullptr, G}, m);
  refMulKernel<true><<<one, thr, 0, s>>>({V, B, nullptr, S}, none, m);
  refCorrectionKernel<<<ge, 128, 0, s>>>(G, S, m, 3e-9, E, st);
  refMulKernel<false><<<one, thr, 0, s>>>({V, E, V, X}, none, m);
  refMulKernel<true><<<one, thr, 0, s>>>({As, X, nullptr, B}, none, m);
  refMulKernel<true><<<one, thr, 0, s>>>({X, B, nullptr, S}, none, m);
  refJacobiKernel<<<1, kJacobiT, mm * sizeof(double2), s>>>(S, m, X, V, w, perm,
                                                            status, st);
}

} // namespace ncgm
