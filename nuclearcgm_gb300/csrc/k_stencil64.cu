// FP64 Hamiltonian product Y = (H + shift) X in integer arithmetic.
//
// GB300's FP64 pipe retires two operations per clock per SM, its integer
// pipes 64 to 128, and H at one lattice point and column takes 144 FP64
// operations, so an FP64 kernel is bound by that pipe: one thread per point and
// column took 758 us for 36^3 x 60 columns and 1108 us for 40^3 x 64, where
// the bytes take 30 us. Here the products run on the integer pipes, with more
// bits than FP64 keeps, in 243 and 302 us, bound by instruction issue and
// latency: 43 and 47 % of the slots with 13 and 15 warps per SM (128
// registers, two blocks of 224 or 256 threads per SM). One scale per tile, 57
// bits below its largest value, took 210 and 266 us, but an orbital falls by
// more than the spare bits inside a tile.
//  * A block owns a tile of lattice points and walks over columns. It copies
//    the tile with its two-point face halos into shared memory (cp.async, the
//    next column's copy in flight while this one is computed). The thread
//    that copied a point replaces its four real values by integers of 57 bits
//    below 2^e, e the exponent of the point's largest value, and stores e.
//  * An output point takes the largest exponent of the 13 points that it
//    reads, shifts their integers right to it, and forms the centre, the
//    neighbour sums S1 (distance 1), S2 (distance 2) and the differences E_a =
//    8 (p1 - m1) - (p2 - m2), the first three times 8, in 64 bits, S = Sh 2^32
//    + Sl. So the scale of every output is the one of its own stencil, as far
//    as an orbital may fall inside the tile.
//  * Coefficients are integers of 58 bits (intCoefKernel), scaled for every
//    lattice point by the
//    largest |Y| / max|X| that its row can give, C = Ch 2^28 + Cl. A product
//    takes three 32 x 32 -> 64 bit multiply-adds; Sl Cl is left out. The 12
//    products of one output component add up in three 64-bit integers, which
//    become one double at the end.
//  * What is cut off is rounded to odd, which treats x and -x alike, and sums
//    of integers do not depend on their order: a block with the mirror
//    symmetries of the lattice keeps them to the bit, as in FP64 arithmetic (a
//    nucleus would drift otherwise: its centre of mass is a near-zero mode).
// Errors, in units of the largest |x| of the point's stencil times the row sum
// R of its |coefficients|: 2^-57 per value of X, 2^-59 per coefficient, 2^-60
// per product for the part left out, and one rounding to FP64 at the end,
// where an FP64 sum rounds every product and partial sum to 2^-53 of itself.
// The unit is the stencil's: a component that is 2^-s of the largest one of
// its stencil keeps 57 - s bits.
// A point that reads an infinity, a NaN or numbers outside 2^-500 .. 2^500, and
// points whose fields or shift are outside the format, are computed in FP64
// (fp64Point).
#include "ncgm_internal.cuh"
#include "stencil_core.cuh"

#include <algorithm>

namespace ncgm {

int smCount();

namespace {

constexpr int kCoefs = 9; // d, alpha1, alpha2, 8 g_x..z, 8 w_x..z
constexpr int kThreadsMax = 256;
constexpr int kIterMax = 5; // copied points per thread
// bits of X, of the neighbour sums' unit (they are multiples of X / 8) and of C
constexpr int kXBits = 57, kSBits = kXBits + 3, kCBits = 58, kCLow = 28;
// exponent fields of the format: 2^-500 .. 2^500, and the mark of a point
// outside it
constexpr int kExpLo = 1023 - 500, kExpHi = 1023 + 500, kExpBad = 4095;
constexpr int kSmemMax = 113 * 1024; // two blocks per SM

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
// C = Ch 2^28 + Cl, |Cl| <= 2^27
__device__ __forceinline__ int2 splitCoef(long long C) {
  const int lo = ((int)(C + (1 << (kCLow - 1))) & ((1 << kCLow) - 1)) -
                 (1 << (kCLow - 1));
  return make_int2((int)((C - lo) >> kCLow), lo);
}

// out: kCoefs arrays of ns int2, then the exponents ec (the row's bound is
// below 2^ec; kExpBad for fields outside the format)
__global__ void intCoefKernel(const double *coef, size_t ns, int2 *out,
                              int *exps) {
  const size_t p = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (p >= ns) return;
  const double *c = coef + 8 * p;
  const double v[kCoefs] = {c[0],       -(4.0 / 3.0) * c[1], c[1] / 12.0,
                            8.0 * c[2], 8.0 * c[3],          8.0 * c[4],
                            8.0 * c[5], 8.0 * c[6],          8.0 * c[7]};
  // exponent field of the bound (2047: a NaN or an infinity)
  const int f = (__double2hiint(rowBound(c)) >> 20) & 0x7FF;
  const bool ok = f > 1023 - 400 && f < 1023 + 400;
  const int ec = f - 1022;
  exps[p] = ok ? ec : kExpBad;
  for (int q = 0; q < kCoefs; ++q)
    out[q * ns + p] =
        splitCoef(ok ? __double2ll_rn(scalbn(v[q], kCBits - ec)) : 0ll);
}

// |x| < 2^e as an integer of kXBits bits, f = e + 1022 the largest exponent
// field of the point. It is rounded to odd: the lowest bit of every value but
// zero is set, also where nothing is cut off, and stays set when the integer is
// shifted further (shifted), so that -x gives the negative integer throughout.
// Zeros and numbers below 2^-1022 give 0.
__device__ __forceinline__ long long toFixed(int lo, int hi, int f) {
  const unsigned long long m =
      (((unsigned long long)((hi & 0xFFFFF) | 0x100000) << 32) | (unsigned)lo)
      << (kXBits - 53);
  const int fx = (hi >> 20) & 0x7FF;
  const long long w =
      (long long)((m >> min(f - fx, 63)) | (unsigned)min(fx, 1));
  const long long g = hi >> 31;
  return (w ^ g) - g;
}
__device__ __forceinline__ int2 pair(long long v) {
  return make_int2((int)v, (int)(v >> 32));
}
// the 64-bit integer (lo, hi) 2^-s rounded to odd (zero: 0)
__device__ __forceinline__ long long shifted(int lo, int hi, int s) {
  long long v = (long long)(((unsigned long long)(unsigned)hi << 32) |
                            (unsigned)lo);
  asm("shr.s64 %0, %0, %1;" : "+l"(v) : "r"(s)); // clamps s
  return v | (unsigned)(lo & 1);
}

// One output component: the sum of C S in integers. With the row bound and the
// shift the sum of |C| |S| stays below 1.85 2^118, that of |Ch| below 2^31,
// and that of |Sh| below 34 2^28.
struct Acc {
  long long hh, mx, mc; // Ch Sh, Cl Sh, Ch Sl: weights 2^60, 2^32, 2^28
  __device__ __forceinline__ void add(int2 c, int2 s) { // (h, l)
    hh += (long long)c.x * s.x;
    mx += (long long)c.y * s.x;
    mc += (long long)c.x * s.y;
  }
  // in units of 2^56, rounded to odd, so that the double made of it is the
  // sum's nearest one
  __device__ __forceinline__ long long value() const {
    const long long t = mx + (mc >> 4);
    const unsigned cut = ((unsigned)t & 0xFFFFFFu) | ((unsigned)mc & 15u);
    return (hh * 16 + (t >> 24)) | min(cut, 1u);
  }
};
__device__ __forceinline__ int2 neg(int2 v) { return make_int2(-v.x, -v.y); }
// v = h 2^32 + l with a signed l
__device__ __forceinline__ int2 limbs(long long v) {
  const int l = (int)v;
  return make_int2((int)(v >> 32) + (int)((unsigned)l >> 31), l);
}
__device__ __forceinline__ double pow2(int e) { // normal range
  return __hiloint2double((e + 1023) << 20, 0);
}

// Tile tx x ty x tz, nx x ny x nz of them; the box in shared memory has row
// pitch px and plane pitch pz (points): point (i, j, k) of the tile at i + px j
// + pz (k + 2), halos at -2, -1, t, t + 1 of one axis each, so P points from the
// first to the last; `points` of them are copied, `iters` per thread.
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
               const int2 *__restrict__ CI, const int *__restrict__ EC,
               const double *__restrict__ coef, int n, int cols, int group,
               double shift, Tiling T) {
  // [buffer][spin][point], the coefficients, the exponents [buffer][point]
  extern __shared__ __align__(16) int4 box[];
  const size_t ns = (size_t)n * n * n;
  const int tid = threadIdx.x, nthr = blockDim.x;
  int2 *ct = reinterpret_cast<int2 *>(box + 4 * T.P) + tid;
  short *ex = reinterpret_cast<short *>(ct - tid + kCoefs * nthr);
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
    at[it] = i + T.px * j + T.pz * (k + 2);
    const int gx = x0 + i, gy = y0 + j, gz = z0 + k;
    if (gx >= 0 && gx < n && gy >= 0 && gy < n && gz >= 0 && gz < n) {
      off[it] = gx + n * (gy + n * gz);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        box[q * T.P + at[it]] = make_int4(0, 0, 0, 0);
      ex[at[it]] = ex[T.P + at[it]] = 0;
    }
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
  const int pb = i + T.px * j + T.pz * (k + 2);
  // the coefficients wait in shared memory between their uses (each thread
  // reads back its own): held in registers they made the loop spill
  int ec = kExpBad;
  if (active) {
    ec = EC[p];
#pragma unroll
    for (int q = 0; q < kCoefs; ++q) ct[q * nthr] = CI[q * ns + p];
    if (shift != 0.0 && ec != kExpBad) {
      const double sI = scalbn(shift, kCBits - ec);
      if (fabs(sI) < 0.85 * (double)(1ll << kCBits)) {
        const int2 d = ct[0];
        ct[0] =
            splitCoef(((long long)d.x << kCLow) + d.y + __double2ll_rn(sI));
      } else {
        ec = kExpBad; // NaN too
      }
    }
  }
  unsigned long long bad = 0; // columns left to FP64 (bit c - c0)
  for (int c = c0; c < c1; ++c) {
    const int buf = (c - c0) & 1;
    int4 *B = box + 2 * buf * T.P;
    short *eb = ex + buf * T.P;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // each thread replaces the points that it copied
#pragma unroll
    for (int it = 0; it < kIterMax; ++it)
      if (off[it] >= 0) {
        int4 &u = B[at[it]], &d = B[T.P + at[it]];
        // largest high word; a value with only low bits counts as 1
        const int m = max(max((u.y & 0x7FFFFFFF) | (u.x != 0),
                              (u.w & 0x7FFFFFFF) | (u.z != 0)),
                          max((d.y & 0x7FFFFFFF) | (d.x != 0),
                              (d.w & 0x7FFFFFFF) | (d.z != 0)));
        // (a point of zeros: an exponent that shifts their implicit bit out)
        const int f = max(m >> 20, 64);
        eb[at[it]] = (short)(m == 0                       ? 0
                             : f > kExpLo && f < kExpHi ? f
                                                        : kExpBad);
        const int2 ur = pair(toFixed(u.x, u.y, f)),
                   ui = pair(toFixed(u.z, u.w, f)),
                   dr = pair(toFixed(d.x, d.y, f)),
                   di = pair(toFixed(d.z, d.w, f));
        u = make_int4(ur.x, ur.y, ui.x, ui.y);
        d = make_int4(dr.x, dr.y, di.x, di.y);
      }
    __syncthreads();
    // every thread has left column c - 1: its buffer takes column c + 1
    if (c + 1 < c1) fetch(c + 1, buf ^ 1);
    if (!active) continue;
    // the scale of this stencil
    int sh[3][4]; // p1, m1, p2, m2 per axis
    int top = eb[pb], sc = top;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int st = a == 0 ? 1 : (a == 1 ? T.px : T.pz);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        sh[a][q] = eb[pb + (q < 2 ? st : 2 * st) * (q & 1 ? -1 : 1)];
        top = max(top, sh[a][q]);
      }
    }
    if (top == kExpBad || ec == kExpBad) {
      bad |= 1ull << (c - c0);
      continue;
    }
    sc = top - sc;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int q = 0; q < 4; ++q) sh[a][q] = top - sh[a][q];
    Acc o[4] = {}; // Re, Im of the upper and the lower component
#pragma unroll
    for (int q = 0; q < 2; ++q) { // spin of the input
      const int4 *b = B + q * T.P + pb;
      long long s1[2] = {0, 0}, s2[2] = {0, 0};
      int2 E[3][2]; // [axis][Re, Im]
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const int st = a == 0 ? 1 : (a == 1 ? T.px : T.pz);
        const int4 p1 = b[st], m1 = b[-st], p2 = b[2 * st], m2 = b[-2 * st];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const auto at = [&](const int4 &v, int s) {
            return shifted(r ? v.z : v.x, r ? v.w : v.y, s);
          };
          const long long xp1 = at(p1, sh[a][0]), xm1 = at(m1, sh[a][1]),
                          xp2 = at(p2, sh[a][2]), xm2 = at(m2, sh[a][3]);
          s1[r] += xp1 + xm1;
          s2[r] += xp2 + xm2;
          E[a][r] = limbs(((xp1 - xm1) << 3) - (xp2 - xm2));
        }
      }
      const int4 v = b[0];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        Acc &s = o[2 * q + r];
        s.add(ct[0], limbs(shifted(r ? v.z : v.x, r ? v.w : v.y, sc) << 3));
        s.add(ct[nthr], limbs(s1[r] << 3));
        s.add(ct[2 * nthr], limbs(s2[r] << 3));
#pragma unroll
        for (int a = 0; a < 3; ++a) s.add(ct[(3 + a) * nthr], E[a][r]);
      }
      // spin-orbit, -i (sigma x W)_a E_a (see pointH): what this spin adds to
      // itself (0, 1) and to the other one (2, 3)
      const int2 wx = ct[6 * nthr], wy = ct[7 * nthr], wz = ct[8 * nthr];
      Acc &o0 = o[2 * q], &o1 = o[2 * q + 1], &o2 = o[2 - 2 * q],
          &o3 = o[3 - 2 * q];
      const int2 ny = neg(wy), nx = neg(wx), nz = neg(wz);
      if (q == 0) {
        o0.add(ny, E[0][1]), o0.add(wx, E[1][1]);
        o1.add(wy, E[0][0]), o1.add(nx, E[1][0]);
        o2.add(wz, E[0][0]), o2.add(nx, E[2][0]);
        o2.add(nz, E[1][1]), o2.add(wy, E[2][1]);
        o3.add(wz, E[0][1]), o3.add(nx, E[2][1]);
        o3.add(wz, E[1][0]), o3.add(ny, E[2][0]);
      } else {
        o0.add(wy, E[0][1]), o0.add(nx, E[1][1]);
        o1.add(ny, E[0][0]), o1.add(wx, E[1][0]);
        o2.add(nz, E[0][0]), o2.add(wx, E[2][0]);
        o2.add(nz, E[1][1]), o2.add(wy, E[2][1]);
        o3.add(nz, E[0][1]), o3.add(wx, E[2][1]);
        o3.add(wz, E[1][0]), o3.add(ny, E[2][0]);
      }
    }
    // units: 2^(e - kSBits) 2^(ec - kCBits) 2^56, e = top - 1022
    const double u = pow2(max(top, kExpLo) - 1022 + ec + 56 - kSBits - kCBits);
    double2 *y = Y + (size_t)c * 2 * ns + 2 * p;
    y[0] = make_double2((double)o[0].value() * u, (double)o[1].value() * u);
    y[1] = make_double2((double)o[2].value() * u, (double)o[3].value() * u);
  }
  for (; bad; bad &= bad - 1) {
    const size_t o = (size_t)(c0 + __ffsll((long long)bad) - 1) * 2 * ns;
    fp64Point(X + o, coef, n, gi, gj, gk, shift, Y + o);
  }
}

// two boxes of two spins, the coefficients, two boxes of exponents
size_t smemBytes(const Tiling &t) {
  return (size_t)t.P * (4 * sizeof(int4) + 2 * sizeof(short)) +
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
        t.P = tx + t.px * (ty - 1) + t.pz * (tz + 3);
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

size_t intCoefBytes(size_t ns) {
  return ns * (kCoefs * sizeof(int2) + sizeof(int));
}

// the integer coefficients of a species' table and their exponents
void buildIntCoefficients(const double *coef64, size_t ns, void *buf,
                          cudaStream_t s) {
  auto *tab = static_cast<int2 *>(buf);
  intCoefKernel<<<(unsigned)((ns + 255) / 256), 256, 0, s>>>(
      coef64, ns, tab, reinterpret_cast<int *>(tab + kCoefs * ns));
}

void applyHInt(const double2 *X, double2 *Y, const double *coef64,
               const void *intCoef, int n, int ncols, double shift,
               cudaStream_t s) {
  // a per-device attribute: set on every call
  cudaFuncSetAttribute(stencilInt, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       kSmemMax);
  thread_local int lastN = 0;
  thread_local Tiling T{};
  if (lastN != n) {
    T = chooseTiling(n);
    lastN = n;
  }
  const size_t ns = (size_t)n * n * n;
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
  const auto *tab = static_cast<const int2 *>(intCoef);
  stencilInt<<<dim3((unsigned)tiles, (ncols + group - 1) / group), T.threads,
               smemBytes(T), s>>>(
      X, Y, tab, reinterpret_cast<const int *>(tab + kCoefs * ns), coef64, n,
      ncols, group, shift, T);
}

} // namespace ncgm
