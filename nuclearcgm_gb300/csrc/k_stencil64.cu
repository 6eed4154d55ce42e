// FP64 Hamiltonian product Y = (H + shift) X in integer arithmetic.
//
// GB300's FP64 pipe retires two operations per clock per SM, its integer
// pipes 64 to 128, and H at one lattice point and column takes 144 FP64
// operations, so an FP64 kernel is bound by that pipe: one thread per point and
// column took 0.76 ms for 36^3 x 60 columns and 1.11 ms for 40^3 x 64, where
// the bytes take 0.03 ms. This kernel takes 0.21 and 0.27 ms, bound by
// instruction latency (14 warps per SM, 36 % of the issue slots). Here the
// operator is evaluated exactly, or to more bits than FP64 keeps, on the
// integer pipes.
//  * A block owns a tile of lattice points and walks over columns. It copies
//    the tile with its two-point face halos into shared memory (cp.async, the
//    next column's copy in flight while this one is computed), takes the
//    largest exponent e of the tile and rounds every value to an integer of 57
//    bits below 2^e, held as two 32-bit limbs X = Xh 2^29 + Xl. The scale is
//    the tile's own, so the tails of an orbital keep their digits.
//  * Neighbour sums S1 (distance 1), S2 (distance 2) and the differences E_a =
//    (p1 - m1) - (p2 - m2)/8 along each axis are formed limb by limb, without
//    carries (the /8 rounds down by one unit of a term that is ~60 times
//    smaller).
//  * Coefficients are 58-bit integers (intCoefKernel), scaled so that no sum
//    of |coefficient| |X| can overflow, C = Ch 2^27 + Cl. A product takes three
//    32 x 32 -> 64 bit multiply-adds; Xl Cl is left out (2^-60 of the largest
//    value the operator can give in the tile). The 12 products of one output
//    component add up in three 64-bit integers, which become one double at
//    the end.
// Errors: 2^-58 of the tile's largest |x| in X and 2^-59 of the largest
// possible |Y| in the products, against ~2^-53 per operation in FP64.
// A tile that holds an infinity, a NaN or numbers outside 2^-900 .. 2^900, and
// fields or shifts outside the format, are computed in FP64 by the same block.
#include "ncgm_internal.cuh"
#include "stencil_core.cuh"

#include <algorithm>

namespace ncgm {

int smCount();

namespace {

constexpr int kCoefs = 9; // d, alpha1, alpha2, 8 g_x..z, 8 w_x..z
constexpr int kThreadsMax = 256;
constexpr int kIterMax = 5; // copied points per thread
constexpr int kXBits = 57, kXLow = 29, kCBits = 57, kCLow = 27;
constexpr int kSmemMax = 110 * 1024;

__device__ __forceinline__ uint32_t sAddr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void copy16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src)
               : "memory");
}

// sum of |coefficient| times the largest |X|-combination it multiplies, in
// units of the tile's largest |x|
__device__ double rowBound(const double *c) {
  double r = fabs(c[0]) + 6.0 * (4.0 / 3.0 + 1.0 / 12.0) * fabs(c[1]);
  for (int a = 0; a < 3; ++a) r += 18.0 * (fabs(c[2 + a]) + 2 * fabs(c[5 + a]));
  return r;
}
// the largest bound of the lattice, as IEEE bits (a NaN is largest)
__global__ void rowBoundKernel(const double *coef, size_t ns,
                               unsigned long long *rmax) {
  __shared__ unsigned long long sh[256];
  unsigned long long m = 0;
  for (size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x; p < ns;
       p += (size_t)gridDim.x * blockDim.x)
    m = max(m, (unsigned long long)(__double_as_longlong(
                                        rowBound(coef + 8 * p)) &
                                    0x7FFFFFFFFFFFFFFFll));
  sh[threadIdx.x] = m;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      sh[threadIdx.x] = max(sh[threadIdx.x], sh[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicMax(rmax, sh[0]);
}

// exponent ec with R < 2^ec, or false when the fields are outside the format
__device__ __forceinline__ bool coefExp(const unsigned long long *rmax,
                                        int &ec) {
  const int f = (int)(*rmax >> 52);
  ec = f - 1022;
  return f > 1023 - 400 && f < 1023 + 400;
}

// C = Ch 2^27 + Cl, |Cl| <= 2^26
__device__ __forceinline__ int2 splitCoef(long long C) {
  const int lo = ((int)(C + (1 << (kCLow - 1))) & ((1 << kCLow) - 1)) -
                 (1 << (kCLow - 1));
  return make_int2((int)((C - lo) >> kCLow), lo);
}

// out: kCoefs arrays of ns int2
__global__ void intCoefKernel(const double *coef, size_t ns,
                              const unsigned long long *rmax, int2 *out) {
  const size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (p >= ns) return;
  int ec;
  const bool ok = coefExp(rmax, ec);
  const double *c = coef + 8 * p;
  const double v[kCoefs] = {c[0],       -(4.0 / 3.0) * c[1], c[1] / 12.0,
                            8.0 * c[2], 8.0 * c[3],          8.0 * c[4],
                            8.0 * c[5], 8.0 * c[6],          8.0 * c[7]};
  for (int q = 0; q < kCoefs; ++q)
    out[q * ns + p] =
        splitCoef(ok ? __double2ll_rn(scalbn(v[q], kCBits - ec)) : 0ll);
}

// |x| < 2^e rounded to an integer of kXBits bits in two limbs Xh 2^29 + Xl,
// |Xl| <= 2^28; f = 1027 + e. Zeros and numbers below 2^-1022 shift out.
__device__ __forceinline__ int2 toLimbs(int lo, int hi, int f) {
  const unsigned long long m =
      (((unsigned long long)((hi & 0xFFFFF) | 0x100000) << 32) | (unsigned)lo)
      << 10;
  const int s = min(f - ((hi >> 20) & 0x7FF), 63);
  const long long w = (long long)(m >> s); // in half units
  const long long g = hi >> 31;
  const long long u = (w ^ g) + 1; // |x| rounded half up
  return make_int2((int)((u + (1 << kXLow)) >> (kXLow + 1)),
                   (int)((unsigned)u << (31 - kXLow)) >> (32 - kXLow));
}

struct Acc {
  long long hh, mx, mc; // weights 2^56, 2^29, 2^27
  // C X, x = limbs (h, l)
  __device__ __forceinline__ void add(int2 c, int2 x) {
    hh += (long long)c.x * x.x;
    mx += (long long)c.y * x.x;
    mc += (long long)c.x * x.y;
  }
  // in units of 2^53: |sum| < 2^115, so below 2^62
  __device__ __forceinline__ long long value() const {
    return hh * 8 + ((mx * 4 + mc) >> 26);
  }
};
__device__ __forceinline__ int2 neg(int2 v) { return make_int2(-v.x, -v.y); }
__device__ __forceinline__ int2 sum2(int2 a, int2 b) {
  return make_int2(a.x + b.x, a.y + b.y);
}
// (p1 - m1) - (p2 - m2) / 8
__device__ __forceinline__ int2 diff(int2 p1, int2 m1, int2 p2, int2 m2) {
  const int bh = p2.x - m2.x, bl = p2.y - m2.y;
  return make_int2((p1.x - m1.x) - (bh >> 3),
                   (p1.y - m1.y) - (bl >> 3) - ((bh & 7) << (kXLow - 3)));
}
__device__ __forceinline__ double pow2(int e) { // normal range
  return __hiloint2double((e + 1023) << 20, 0);
}

// Tile tx x ty x tz, nx x ny x nz of them; the box in shared memory has row
// pitch px and plane pitch pz (points), P points in all; `points` of them are
// copied, `iters` per thread.
struct Tiling {
  int tx, ty, tz, nx, ny, nz, threads, px, pz, P, points, iters;
};

// One output point in FP64 (tiles outside the integer format)
__device__ __noinline__ void fp64Point(const double2 *x, const double *coef,
                                       int n, int i, int j, int k,
                                       double shift, double2 *y) {
  const size_t p = i + (size_t)n * (j + (size_t)n * k);
  auto at = [&](int di, int dj, int dk) -> Spinor<double> {
    const int ii = i + di, jj = j + dj, kk = k + dk;
    if (ii < 0 || ii >= n || jj < 0 || jj >= n || kk < 0 || kk >= n)
      return {0.0, 0.0, 0.0, 0.0};
    const size_t q = ii + (size_t)n * (jj + (size_t)n * kk);
    const double2 u = x[2 * q], d = x[2 * q + 1];
    return {u.x, u.y, d.x, d.y};
  };
  double c[8];
  for (int q = 0; q < 8; ++q) c[q] = coef[8 * p + q];
  const Spinor<double> o = pointH<double>(
      c, shift, at(0, 0, 0), at(1, 0, 0), at(-1, 0, 0), at(2, 0, 0),
      at(-2, 0, 0), at(0, 1, 0), at(0, -1, 0), at(0, 2, 0), at(0, -2, 0),
      at(0, 0, 1), at(0, 0, -1), at(0, 0, 2), at(0, 0, -2));
  y[2 * p] = make_double2(o.r0, o.i0);
  y[2 * p + 1] = make_double2(o.r1, o.i1);
}

__global__ void __launch_bounds__(kThreadsMax, 2)
    stencilInt(const double2 *__restrict__ X, double2 *__restrict__ Y,
               const int2 *__restrict__ CI, const double *__restrict__ coef,
               const unsigned long long *__restrict__ rmax, int n, int cols,
               int group, double shift, Tiling T) {
  extern __shared__ __align__(16) int4 box[]; // [buffer][spin][point]
  __shared__ int wmax[2][kThreadsMax / 32];
  const size_t ns = (size_t)n * n * n;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int x0 = ((int)blockIdx.x % T.nx) * T.tx,
            y0 = ((int)blockIdx.x / T.nx % T.ny) * T.ty,
            z0 = ((int)blockIdx.x / (T.nx * T.ny)) * T.tz;
  const int c0 = blockIdx.y * group, c1 = min(cols, c0 + group);
  // the points that this thread copies: place in the box and lattice index
  // (-1: outside the lattice, stays zero in both buffers; place -1: none).
  // The tile comes first, then its x, y and z halos.
  int off[kIterMax], at[kIterMax];
#pragma unroll
  for (int it = 0; it < kIterMax; ++it) {
    off[it] = at[it] = -1;
    int b = tid + it * nthr;
    if (b >= T.points) continue;
    int i, j, k;
    const int pts = T.tx * T.ty * T.tz, hx = 4 * T.ty * T.tz,
              hy = 4 * T.tx * T.tz;
    // halo layer h = 0 .. 3 -> coordinate -2, -1, t, t + 1
    const auto layer = [](int h, int t) { return h < 2 ? h - 2 : t + h - 2; };
    if (b < pts) {
      i = b % T.tx, j = b / T.tx % T.ty, k = b / (T.tx * T.ty);
    } else if ((b -= pts) < hx) {
      i = layer(b & 3, T.tx), j = (b >> 2) % T.ty, k = (b >> 2) / T.ty;
    } else if ((b -= hx) < hy) {
      i = b % T.tx, j = layer(b / T.tx & 3, T.ty), k = b / (4 * T.tx);
    } else {
      b -= hy;
      i = b % T.tx, j = b / T.tx % T.ty, k = layer(b / (T.tx * T.ty), T.tz);
    }
    at[it] = i + 2 + T.px * (j + 2) + T.pz * (k + 2);
    const int gx = x0 + i, gy = y0 + j, gz = z0 + k;
    if (gx >= 0 && gx < n && gy >= 0 && gy < n && gz >= 0 && gz < n)
      off[it] = gx + n * (gy + n * gz);
    else
#pragma unroll
      for (int q = 0; q < 4; ++q)
        box[q * T.P + at[it]] = make_int4(0, 0, 0, 0);
  }
  auto fetch = [&](int col, int buf) {
    const double2 *x = X + (size_t)col * 2 * ns;
    const uint32_t d = sAddr(box + 2 * buf * T.P);
#pragma unroll
    for (int it = 0; it < kIterMax; ++it)
      if (off[it] >= 0) {
        copy16(d + 16u * at[it], x + 2 * (size_t)off[it]);
        copy16(d + 16u * (T.P + at[it]), x + 2 * (size_t)off[it] + 1);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(c0, 0);
  // this thread's output point and its coefficients
  const int i = tid % T.tx, j = tid / T.tx % T.ty, k = tid / (T.tx * T.ty);
  const int gi = x0 + i, gj = y0 + j, gk = z0 + k;
  const bool active = k < T.tz && gi < n && gj < n && gk < n;
  const size_t p = gi + (size_t)n * (gj + (size_t)n * gk);
  const int pb = i + 2 + T.px * (j + 2) + T.pz * (k + 2);
  int ec;
  bool fields = coefExp(rmax, ec);
  int2 cd = {}, ca1 = {}, ca2 = {}, cg[3] = {}, cw[3] = {};
  if (active && fields) {
    cd = CI[p];
    ca1 = CI[ns + p];
    ca2 = CI[2 * ns + p];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      cg[a] = CI[(3 + a) * ns + p];
      cw[a] = CI[(6 + a) * ns + p];
    }
  }
  if (shift != 0.0 && fields) {
    const double sI = scalbn(shift, kCBits - ec);
    if (fabs(sI) < 0.85 * (double)(1ll << kCBits))
      cd = splitCoef(((long long)cd.x << kCLow) + cd.y + __double2ll_rn(sI));
    else
      fields = false; // NaN too
  }
  unsigned long long bad = 0; // columns left to FP64 (bit c - c0)
  // the coefficients wait in shared memory between their uses (each thread
  // reads back its own): held in registers they made the loop spill (244 us
  // against 213 us for 36^3 x 60)
  int2 *ct = reinterpret_cast<int2 *>(box + 4 * T.P) + tid;
  ct[0] = cd;
  ct[nthr] = ca1;
  ct[2 * nthr] = ca2;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    ct[(3 + a) * nthr] = cg[a];
    ct[(6 + a) * nthr] = cw[a];
  }
  for (int c = c0; c < c1; ++c) {
    const int buf = (c - c0) & 1;
    int4 *B = box + 2 * buf * T.P;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // largest high word of the tile; a value with only low bits counts as 1
    int m = 0;
#pragma unroll
    for (int it = 0; it < kIterMax; ++it)
      if (off[it] >= 0)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int4 v = B[q * T.P + at[it]];
          m = max(m, max((v.y & 0x7FFFFFFF) | (v.x != 0),
                         (v.w & 0x7FFFFFFF) | (v.z != 0)));
        }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((tid & 31) == 0) wmax[buf][tid >> 5] = m;
    __syncthreads();
    // every thread has left column c - 1: its buffer takes column c + 1
    if (c + 1 < c1) fetch(c + 1, buf ^ 1);
    m = wmax[buf][0];
    for (int w = 1; w < (nthr >> 5); ++w) m = max(m, wmax[buf][w]);
    const int f = m >> 20; // exponent field of the largest value
    const bool ok =
        fields && (m == 0 || (f > 1023 - 900 && f < 1023 + 900));
    const int e = m ? f - 1022 : 0; // all |x| < 2^e
    if (ok) {
#pragma unroll
      for (int it = 0; it < kIterMax; ++it)
        if (off[it] >= 0)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            int4 &v = B[q * T.P + at[it]];
            const int2 re = toLimbs(v.x, v.y, 1027 + e),
                       im = toLimbs(v.z, v.w, 1027 + e);
            v = make_int4(re.x, re.y, im.x, im.y);
          }
    } else {
      bad |= 1ull << (c - c0);
    }
    __syncthreads();
    if (ok && active) {
      double2 *y = Y + (size_t)c * 2 * ns;
      Acc o[4] = {}; // Re, Im of the upper and the lower component
      int2 s1[4], s2[4];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int4 v = B[q * T.P + pb];
        o[2 * q].add(ct[0], make_int2(v.x, v.y));
        o[2 * q + 1].add(ct[0], make_int2(v.z, v.w));
        s1[2 * q] = s1[2 * q + 1] = make_int2(0, 0);
        s2[2 * q] = s2[2 * q + 1] = make_int2(0, 0);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int st = a == 0 ? 1 : (a == 1 ? T.px : T.pz);
        int2 E[4];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int4 *b = B + q * T.P + pb;
          const int4 p1 = b[st], m1 = b[-st], p2 = b[2 * st], m2 = b[-2 * st];
          const int2 p1r = {p1.x, p1.y}, p1i = {p1.z, p1.w};
          const int2 m1r = {m1.x, m1.y}, m1i = {m1.z, m1.w};
          const int2 p2r = {p2.x, p2.y}, p2i = {p2.z, p2.w};
          const int2 m2r = {m2.x, m2.y}, m2i = {m2.z, m2.w};
          s1[2 * q] = sum2(s1[2 * q], sum2(p1r, m1r));
          s1[2 * q + 1] = sum2(s1[2 * q + 1], sum2(p1i, m1i));
          s2[2 * q] = sum2(s2[2 * q], sum2(p2r, m2r));
          s2[2 * q + 1] = sum2(s2[2 * q + 1], sum2(p2i, m2i));
          E[2 * q] = diff(p1r, m1r, p2r, m2r);
          E[2 * q + 1] = diff(p1i, m1i, p2i, m2i);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q].add(ct[(3 + a) * nthr], E[q]);
        // spin-orbit, -i (sigma x W)_a E_a (see pointH)
        if (a == 0) { // [[i Wy, -Wz], [Wz, -i Wy]]
          const int2 wy = ct[7 * nthr], wz = ct[8 * nthr];
          const int2 ny = neg(wy), nz = neg(wz);
          o[0].add(ny, E[1]), o[0].add(nz, E[2]);
          o[1].add(wy, E[0]), o[1].add(nz, E[3]);
          o[2].add(wz, E[0]), o[2].add(wy, E[3]);
          o[3].add(wz, E[1]), o[3].add(ny, E[2]);
        } else if (a == 1) { // [[-i Wx, i Wz], [i Wz, i Wx]]
          const int2 wx = ct[6 * nthr], wz = ct[8 * nthr];
          const int2 nx = neg(wx), nz = neg(wz);
          o[0].add(wx, E[1]), o[0].add(nz, E[3]);
          o[1].add(nx, E[0]), o[1].add(wz, E[2]);
          o[2].add(nz, E[1]), o[2].add(nx, E[3]);
          o[3].add(wz, E[0]), o[3].add(wx, E[2]);
        } else { // [[0, Wx - i Wy], [-Wx - i Wy, 0]]
          const int2 wx = ct[6 * nthr], wy = ct[7 * nthr];
          const int2 nx = neg(wx), ny = neg(wy);
          o[0].add(wx, E[2]), o[0].add(wy, E[3]);
          o[1].add(wx, E[3]), o[1].add(ny, E[2]);
          o[2].add(nx, E[0]), o[2].add(wy, E[1]);
          o[3].add(nx, E[1]), o[3].add(ny, E[0]);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        o[q].add(ct[nthr], s1[q]);
        o[q].add(ct[2 * nthr], s2[q]);
      }
      // units: 2^(e - kXBits) 2^(ec - kCBits) 2^53; |e| <= 901, |ec| <= 401:
      // in two factors
      const double u1 = pow2(e);
      const double u2 = pow2(ec + 53 - kXBits - kCBits);
      y[2 * p] = make_double2((double)o[0].value() * u2 * u1,
                              (double)o[1].value() * u2 * u1);
      y[2 * p + 1] = make_double2((double)o[2].value() * u2 * u1,
                                  (double)o[3].value() * u2 * u1);
    }
  }
  if (active)
    for (; bad; bad &= bad - 1) {
      const size_t o = (size_t)(c0 + __ffsll((long long)bad) - 1) * 2 * ns;
      fp64Point(X + o, coef, n, gi, gj, gk, shift, Y + o);
    }
}

// two boxes of two spins, and the coefficients
size_t smemBytes(const Tiling &t) {
  return (size_t)t.P * 4 * sizeof(int4) +
         (size_t)kCoefs * t.threads * sizeof(int2);
}

// Tile of an n^3 lattice: 256 threads at most, one point each, two boxes in
// shared memory for two blocks per SM. The cost of a tile is what its threads
// compute plus what they convert (the tile and its six face halos), so tiles
// that divide the lattice and are close to cubes win. Rows are padded so that
// eight consecutive points, also over the end of a row or a plane, lie in
// different 16-byte bank groups.
Tiling chooseTiling(int n) {
  Tiling best{};
  double bestCost = 1e300;
  for (int tx = 1; tx <= std::min(n, 16); ++tx)
    for (int ty = 1; ty <= std::min(n, 16); ++ty)
      for (int tz = 1; tz <= std::min(n, 16); ++tz) {
        const int pts = tx * ty * tz;
        if (pts > kThreadsMax) continue;
        Tiling t{};
        t.tx = tx, t.ty = ty, t.tz = tz;
        t.nx = (n + tx - 1) / tx;
        t.ny = (n + ty - 1) / ty;
        t.nz = (n + tz - 1) / tz;
        t.threads = (pts + 31) / 32 * 32;
        t.px = tx % 8 ? tx + 8 : tx + 4;
        t.pz = t.px * (ty + 4) + (t.px % 2 ? 4 : 0);
        t.P = t.pz * (tz + 4);
        t.points = pts + 4 * (ty * tz + tx * tz + tx * ty);
        t.iters = (t.points + t.threads - 1) / t.threads;
        if (t.iters > kIterMax || smemBytes(t) > kSmemMax) continue;
        const double cost =
            (double)t.nx * t.ny * t.nz * t.threads * (4.4 + t.iters);
        if (cost < bestCost) {
          bestCost = cost;
          best = t;
        }
      }
  return best;
}

} // namespace

size_t intCoefBytes(size_t ns) { return kCoefs * ns * sizeof(int2) + 256; }

// the integer coefficients of a species' table: the row bound in the first
// 8 bytes of buf, the table from byte 256 on
void buildIntCoefficients(const double *coef64, size_t ns, void *buf,
                          cudaStream_t s) {
  auto *rmax = static_cast<unsigned long long *>(buf);
  auto *tab = reinterpret_cast<int2 *>(static_cast<char *>(buf) + 256);
  cudaMemsetAsync(rmax, 0, sizeof(*rmax), s);
  rowBoundKernel<<<(unsigned)std::min<size_t>(256, (ns + 255) / 256), 256, 0,
                   s>>>(coef64, ns, rmax);
  intCoefKernel<<<(unsigned)((ns + 255) / 256), 256, 0, s>>>(coef64, ns, rmax,
                                                             tab);
}

void applyHInt(const double2 *X, double2 *Y, const double *coef64,
               const void *intCoef, int n, int ncols, double shift,
               cudaStream_t s) {
  static const bool attr = [] {
    cudaFuncSetAttribute(stencilInt,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kSmemMax);
    return true;
  }();
  (void)attr;
  thread_local int lastN = 0;
  thread_local Tiling T{};
  if (lastN != n) {
    T = chooseTiling(n);
    lastN = n;
  }
  const long long tiles = (long long)T.nx * T.ny * T.nz;
  // columns per block: the fewest waves of two blocks per SM, counting a
  // block's set-up as a column and a half
  const long long slots = 2ll * smCount();
  int group = 1;
  double best = 1e300;
  for (int g = 1; g <= std::min(ncols, 64); ++g) { // 64: the bits of `bad`
    const long long blocks = tiles * ((ncols + g - 1) / g);
    const double cost = (double)((blocks + slots - 1) / slots) * (g + 1.5);
    if (cost < best) {
      best = cost;
      group = g;
    }
  }
  stencilInt<<<dim3((unsigned)tiles, (ncols + group - 1) / group), T.threads,
               smemBytes(T), s>>>(
      X, Y,
      reinterpret_cast<const int2 *>(static_cast<const char *>(intCoef) + 256),
      coef64, static_cast<const unsigned long long *>(intCoef), n, ncols,
      group, shift, T);
}

} // namespace ncgm
