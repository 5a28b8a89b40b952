// Coefficient solve of 3D tables stored in FP32 or 16 bits: the same three
// FP64 line solves (x, y, z) as solve.cu's k_sweep, whose result is rounded
// once on store, in fewer FP64 operations and fewer passes over memory.
//
// FP64 tables keep the reference's operations one by one (k_sweep: 12 FP64
// operations a coefficient and axis), because their bits are the
// reference's.  Here the result is rounded to at most 24 bits, so only the
// FP64 accuracy has to stay, and GB300's FP64 pipe (2 operations a clock
// and SM, 1/64 of FP32) is what bounds the solve.  So:
//  * cyclic axes: the circulant band (1, 4, 1)/6 factors as
//      -(1 - z q^-1)(1 - z q) / (6 z),  z = sqrt(3) - 2,
//    with q the shift: one forward and one backward recurrence of one FMA
//    each from zero, then the wrap-around as two geometric terms alpha z^r
//    and beta z^(M-r).  A term below a quarter ulp of the value it is added
//    to (read off the exponents with integer instructions) cannot change it
//    and is left out, so usually one FMA a coefficient remains.  The gain
//    -6 z of all cyclic axes is applied once, as the data is read.
//  * other axes: the recorded elimination with reciprocals: two operations
//    forward, one back.
// Three FP64 operations a coefficient and axis, every rounding error at
// most a few ulps of FP64, as in the elimination.
//
// A thread solves one line, which stays in shared memory between its forward
// and backward recurrence: each axis is one read and one write of the work
// array (the x solve reads the caller's data and transposes it, the z solve
// of an FP32 table writes the table), 40 bytes a coefficient in all where the
// sweeps moved 120.
//
// Measured on GB300, 64^3 x 512 FP32, set + flush: 3.00 ms (the sweeps, with a
// staging copy for each spline: 12.35); about 2.2 of them are the FP64 pipe's.
#include <math.h>
#include <string.h>

#include <algorithm>

#include "eg_internal.h"

namespace eg {

namespace {

// Line factors of one axis: this header, then for cyclic axes z^r
// (r = 0..M), for the others 1/P, L/P and U (M + 2 each).
struct FastFactors {
  int M, cyclic, anti, pad_;
  double z, k1, k2, k4, k5;          // cyclic: see solve_line_fast
  double iQ, R0, R1, U0a, U0b;       // boundary rows
};
constexpr int kFastHead = sizeof(FastFactors) / sizeof(double);

// Conversions in integer instructions: F2F between FP32 and FP64 runs on the
// FP64 pipe.  The calls keep the rare forms out of line, so that a warp
// without one issues nothing to that pipe.
__device__ __noinline__ double scaled_slow(float f, double g) { return g * (double)f; }
__device__ __noinline__ float rounded_slow(double v) { return __double2float_rn(v); }

// g * f for a normal f, g = G * 2^(ge - 63) with bit 63 of G set: the 24-bit
// significand times 64 bits of g, rounded to 53 bits.
__device__ __forceinline__ double scaled(float f, double g, uint64_t G, int ge) {
  const unsigned w = __float_as_uint(f), e = (w >> 23) & 0xFFu;
  if (e - 1u >= 254u) return scaled_slow(f, g);
  const uint64_t h = __umul64hi((uint64_t)((w & 0x7FFFFFu) | 0x800000u) << 40, G);  // in [2^62, 2^64 - 2^40)
  const int sh = 10 + (int)(h >> 63);
  const uint64_t m = (h + (1ull << (sh - 1))) >> sh;  // [2^52, 2^53]
  const uint64_t bits = m + ((uint64_t)(unsigned)(sh + (int)e + ge + 885) << 52);
  return __longlong_as_double((long long)(bits | (uint64_t)(w & 0x80000000u) << 32));
}

// v rounded to nearest even, as __double2float_rn, for results that are
// normal floats.
__device__ __forceinline__ float rounded(double v) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  const unsigned e = (hi >> 20) & 0x7FFu;
  if (e - 897u >= 253u) return rounded_slow(v);
  const unsigned f = __funnelshift_l(lo, (hi & 0x7FFFFFFFu) - (896u << 20), 3);
  const uint64_t x = ((uint64_t)f << 32 | (lo << 3)) + 0x7FFFFFFFu + (f & 1u);
  return __uint_as_float((unsigned)(x >> 32) | (hi & 0x80000000u));
}

__device__ __forceinline__ int exponent(double v) { return (__double2hiint(v) >> 20) & 0x7FF; }

// False when t * p cannot change any FP64 value of exponent field eu or more
// it is added to: its magnitude, below 2^(e(t) + e(p) + 2), does not reach a
// quarter ulp.
__device__ __forceinline__ bool counts(double t, double p, int eu) {
  return exponent(t) + exponent(p) - 1023 + 2 > eu - 54;
}

// Solves one line.  in(r): data r (r < M), read once each in order; s: the
// line's M doubles of shared memory, st apart (in(r) may read s[r * st]);
// out(r, c): coefficient r, every r < M + 3 (cyclic) or M + 2 once.
template <typename In, typename Out>
__device__ __forceinline__ void solve_line_fast(const double *__restrict__ pk, In in, double *s, int st, double lval,
                                                double rval, Out out) {
  const FastFactors &h = *reinterpret_cast<const FastFactors *>(pk);
  const int M = h.M;
  if (h.cyclic) {
    const double z = h.z;
    const double *zp = pk + kFastHead;
    double v = 0.0;
    int r = 0;
    for (; r + 8 <= M; r += 8) {
      double y[8];
#pragma unroll
      for (int q = 0; q < 8; q++) y[q] = in(r + q);
#pragma unroll
      for (int q = 0; q < 8; q++) {
        v = fma(z, v, y[q]);
        s[(r + q) * st] = v;
      }
    }
    for (; r < M; r++) {
      v = fma(z, v, in(r));
      s[r * st] = v;
    }
    const double A = h.k1 * v;  // the forward recurrence's true value before row 0
    double b = 0.0;
#pragma unroll 4
    for (r = M - 1; r >= 0; r--) {
      b = fma(z, b, s[r * st]);
      s[r * st] = b;
    }
    const double U = h.k1 * fma(h.k2, A, b);  // the value past the last row
    const double al = h.k4 * A, be = fma(-h.k5, A, U);
    double u0 = 0.0, u1 = 0.0, u = 0.0;
    // eight rows a step, so that a term that counts for none is branched over
    for (r = 0; r < M; r += 8) {
      double w[8];
      int eu = 0x7FF;
#pragma unroll
      for (int q = 0; q < 8; q++) {
        w[q] = r + q < M ? s[(r + q) * st] : 0.0;
        if (r + q < M) eu = min(eu, exponent(w[q]));
      }
      if (counts(al, zp[r], eu)) {
#pragma unroll
        for (int q = 0; q < 8; q++) w[q] = fma(al, zp[min(r + q, M)], w[q]);
      }
      if (counts(be, zp[max(M - r - 7, 1)], eu)) {
#pragma unroll
        for (int q = 0; q < 8; q++) w[q] = fma(be, zp[max(M - r - q, 1)], w[q]);
      }
      if (r == 0) { u0 = w[0]; u1 = w[1]; }
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (r + q < M) {
          u = w[q];
          out(r + q + 1, u);
        }
    }
    out(0, h.anti ? -u : u);
    out(M + 1, h.anti ? -u0 : u0);
    out(M + 2, h.anti ? -u1 : u1);
  } else {
    const double *iP = pk + kFastHead, *LP = iP + M + 2, *U = LP + M + 2;
    const double d0 = lval * iP[0];
    double prev = d0, prev2 = 0.0;
    int r = 1;
    for (; r + 4 <= M + 1; r += 4) {
      double y[4];
#pragma unroll
      for (int q = 0; q < 4; q++) y[q] = in(r - 1 + q);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        prev2 = prev;
        prev = fma(-LP[r + q], prev, y[q] * iP[r + q]);
        s[(r - 1 + q) * st] = prev;
      }
    }
    for (; r <= M; r++) {
      prev2 = prev;
      prev = fma(-LP[r], prev, in(r - 1) * iP[r]);
      s[(r - 1) * st] = prev;
    }
    double c = fma(-h.R1, prev, fma(-h.R0, prev2, rval)) * h.iQ;
    out(M + 1, c);
    double c2 = 0.0;
#pragma unroll 4
    for (r = M; r > 0; r--) {
      c = fma(-U[r], c, s[(r - 1) * st]);
      if (r == 2) c2 = c;
      out(r, c);
    }
    out(0, fma(-h.U0b, c2, fma(-h.U0a, c, d0)));
  }
}

struct FastArgs {
  const double *fac;
  double *W;                   // work array [Nx][Ny][Nz][ncw]
  int64_t wx, wy;              // its strides (the z stride is ncw)
  int ncw, ncomp;
  int Mx, My, Mz, Ny, Nz;
  double lval[2], rval[2];
  // x solve
  const float *stg;            // queued data [n][Mx][My][Mz][ncomp]
  double gain;                 // the cyclic axes' gains, also as gain_m * 2^(gain_e - 63)
  uint64_t gain_m;
  int gain_e;
  int cw_log, yz_log;          // tile: 2^cw_log columns x 2^yz_log (y, z) lines
  // z solve
  int64_t nlines;              // Nx * Ny
  float *table;                // FP32 table, or null: back into W, with the columns' largest magnitudes
  int64_t zs;
  const int *slot_spline;
  unsigned *colmax;
};

// x lines: a block takes a tile of 8 columns x 8 neighbouring (y, z) lines
// (fewer columns and more lines for narrow batches, fewer lines for long
// ones).  The caller's data is spline-major, so it is read 8 neighbours at
// a time (32 bytes) per spline and x and lands transposed in shared memory,
// rows one double longer than the columns so that neither side's accesses
// collide on a bank; W is written 8 columns (64 bytes) at a time.
constexpr int kLoads = 16;  // reads in flight a thread
template <int NC>
__global__ void __launch_bounds__(64) k_solve_x(const FastArgs a) {
  extern __shared__ double line[];
  const int CW = 1 << a.cw_log, YZ = 1 << a.yz_log, CS = CW | 1;
  const int ctiles = (a.ncw + CW - 1) / CW;
  const int64_t ntot = (int64_t)a.My * a.Mz, yz0 = (int64_t)(blockIdx.x / ctiles) * YZ;
  const int c0 = (int)(blockIdx.x % ctiles) * CW;
  const int T = CW * YZ, st = YZ * CS;
  const int slots = CW / NC, n = a.ncw / NC, s0 = c0 / NC;
  const int run = YZ * NC;                        // consecutive input reals per (spline, x)
  const int run_log = a.yz_log + NC - 1, slots_log = a.cw_log - (NC - 1);
  const int left = (int)min((int64_t)run, (ntot - yz0) * NC);
  for (int i0 = threadIdx.x; i0 < a.Mx * T; i0 += kLoads * T) {
    float f[kLoads];
#pragma unroll
    for (int q = 0; q < kLoads; q++) {
      const int idx = i0 + q * T, e = idx & (run - 1), rest = idx >> run_log;
      const int sl = rest & (slots - 1), x = rest >> slots_log;
      f[q] = 0.f;
      if (x < a.Mx && s0 + sl < n && e < left)
        f[q] = __ldcs(a.stg + ((int64_t)(s0 + sl) * a.Mx + x) * ntot * NC + yz0 * NC + e);
    }
#pragma unroll
    for (int q = 0; q < kLoads; q++) {
      const int idx = i0 + q * T, e = idx & (run - 1), rest = idx >> run_log;
      const int sl = rest & (slots - 1), x = rest >> slots_log;
      if (x < a.Mx) line[(x * YZ + e / NC) * CS + sl * NC + e % NC] = scaled(f[q], a.gain, a.gain_m, a.gain_e);
    }
  }
  __syncthreads();
  const int t = threadIdx.x, cl = t & (CW - 1), yl = t >> a.cw_log, c = c0 + cl;
  const int64_t yz = yz0 + yl;
  if (c >= a.ncw || yz >= ntot) return;
  double *s = line + yl * CS + cl;
  double *w = a.W + (yz / a.Mz) * a.wy + (yz % a.Mz) * a.ncw + c;
  const int p = NC == 1 ? 0 : c & 1;
  solve_line_fast(a.fac, [&](int r) { return s[r * st]; }, s, st, a.lval[p], a.rval[p],
                  [&](int r, double v) { w[(int64_t)r * a.wx] = v; });
}

// y lines, in place on W: the z and column axes are one contiguous run, so
// neighbouring threads hold neighbouring doubles whatever the batch's width.
__global__ void __launch_bounds__(32) k_solve_y(const FastArgs a) {
  extern __shared__ double line[];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)a.Mz * a.ncw) return;
  double *w = a.W + blockIdx.y * a.wx + i;
  const int p = a.ncomp == 1 ? 0 : (int)(i % a.ncw) & 1;
  solve_line_fast(a.fac, [&](int r) { return w[(int64_t)r * a.wy]; }, line + threadIdx.x, blockDim.x, a.lval[p],
                  a.rval[p], [&](int r, double v) { w[(int64_t)r * a.wy] = v; });
}

// z lines: into the FP32 table, or back into W with the columns' largest
// magnitudes for the 16-bit tables' factors.
__global__ void __launch_bounds__(32) k_solve_z(const FastArgs a) {
  extern __shared__ double line[];
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nlines * a.ncw) return;
  const int64_t xy = i / a.ncw;
  const int c = (int)(i - xy * a.ncw), p = a.ncomp == 1 ? 0 : c & 1;
  double *w = a.W + xy * a.wy + c;
  auto in = [&](int r) { return w[(int64_t)r * a.ncw]; };
  double *s = line + threadIdx.x;
  if (a.table) {
    float *o = a.table + xy * a.Nz * a.zs + (int64_t)a.slot_spline[c / a.ncomp] * a.ncomp + p;
    solve_line_fast(a.fac, in, s, blockDim.x, a.lval[p], a.rval[p],
                    [&](int r, double v) { o[(int64_t)r * a.zs] = rounded(v); });
  } else {
    float m = 0.f;
    solve_line_fast(a.fac, in, s, blockDim.x, a.lval[p], a.rval[p], [&](int r, double v) {
      w[(int64_t)r * a.ncw] = v;
      m = fmaxf(m, rounded(fabs(v)));
    });
    atomicMax(a.colmax + c, __float_as_uint(m));
  }
}

// Lines a block of the y and z solves: one warp, so that 13 blocks of
// 64-row lines share an SM's shared memory.
constexpr int kLines = 32;

}  // namespace

void pack_fast_factors(const LineFactors &f, std::vector<double> &out) {
  const int M = f.M, n = M + 2;
  FastFactors h;
  memset(&h, 0, sizeof(h));
  h.M = M; h.cyclic = f.cyclic; h.anti = f.anti;
  out.assign(kFastHead + (f.cyclic ? (size_t)M + 1 : 3 * (size_t)n), 0.0);
  double *p = out.data() + kFastHead;
  if (f.cyclic) {
    const double z = sqrt(3.0) - 2.0, s = f.anti ? -1.0 : 1.0;
    for (int r = 0; r <= M; r++) p[r] = pow(z, r);
    const double zM = pow(z, M), z2 = 1.0 - z * z;
    // with v and b the zero-started recurrences: the forward recurrence's
    // true value before row 0 is A = k1 v[M-1]; the solution past the last
    // row is U = k1 (b[0] + k2 A); and u[r] = b[r] + k4 A z^r + (U - k5 A) z^(M-r)
    h.z = z;
    h.k1 = s / (1.0 - s * zM);
    h.k2 = z * (1.0 - zM * zM) / z2;
    h.k4 = z / z2;
    h.k5 = zM * z / z2;
  } else {
    h.iQ = 1.0 / f.Q; h.R0 = f.R0; h.R1 = f.R1; h.U0a = f.U0a; h.U0b = f.U0b;
    for (int r = 0; r <= M; r++) {
      p[r] = 1.0 / f.P[r];
      p[n + r] = f.L[r] / f.P[r];
      p[2 * n + r] = f.U[r];
    }
  }
  memcpy(out.data(), &h, sizeof(h));
}

bool fast_solve_fits(const Table *t) {
  return t->dims == 3 && t->storage != ST_F64 && std::max(t->M[0], std::max(t->M[1], t->M[2])) <= kFastMaxLine;
}

int solve_fast(Table *t, int n, cudaStream_t s) {
  FastArgs a;
  memset(&a, 0, sizeof(a));
  const int nc = t->ncomp, ncw = n * nc;
  const int Nx = t->Nc[0], Ny = t->Nc[1], Nz = t->Nc[2];
  a.W = t->work_w;
  a.ncw = ncw;
  a.ncomp = nc;
  a.Mx = t->M[0]; a.My = t->M[1]; a.Mz = t->M[2];
  a.Ny = Ny; a.Nz = Nz;
  a.wy = (int64_t)Nz * ncw;
  a.wx = (int64_t)Ny * a.wy;
  // the gains of the cyclic axes, all applied to the data; the boundary
  // values of an axis see those of the cyclic axes still to come
  const double gz = -6.0 * (sqrt(3.0) - 2.0);
  double after[3], g = 1.0;
  for (int ax = 2; ax >= 0; ax--) {
    after[ax] = g;
    if (t->lcode[ax] == PERIODIC || t->lcode[ax] == ANTIPERIODIC) g *= gz;
  }
  a.gain = g;
  int ge;
  a.gain_m = (uint64_t)ldexp(frexp(g, &ge), 64);
  a.gain_e = ge - 1;
  auto axis = [&](int ax) {
    a.fac = t->factors_d + t->fast_off[ax];
    for (int p = 0; p < 2; p++) {
      a.lval[p] = t->lval[ax][p] * after[ax];
      a.rval[p] = t->rval[ax][p] * after[ax];
    }
  };
  // x
  axis(0);
  a.stg = (const float *)t->staging;
  const int T = a.Mx <= 144 ? 64 : 32;
  a.cw_log = nc == 2 ? 1 : 0;
  while (a.cw_log < 3 && (1 << a.cw_log) < ncw) a.cw_log++;
  while ((2 << a.yz_log << a.cw_log) <= T) a.yz_log++;
  const int CW = 1 << a.cw_log, YZ = 1 << a.yz_log;
  size_t sm = (size_t)a.Mx * YZ * (CW | 1) * sizeof(double);
  const int64_t yzt = ((int64_t)a.My * a.Mz + YZ - 1) / YZ;
  const unsigned gx = (unsigned)(yzt * ((ncw + CW - 1) / CW));
  const void *fx = nc == 1 ? (const void *)k_solve_x<1> : (const void *)k_solve_x<2>;
  void *args[] = {&a};
  if (int r = allow_smem(fx, sm)) return r;
  EG_CUDA(cudaLaunchKernel(fx, dim3(gx), dim3(CW * YZ), args, sm, s));
  // y
  axis(1);
  sm = (size_t)kLines * a.My * sizeof(double);
  if (int r = allow_smem((const void *)k_solve_y, sm)) return r;
  k_solve_y<<<dim3((unsigned)(((int64_t)a.Mz * ncw + kLines - 1) / kLines), (unsigned)Nx), kLines, sm, s>>>(a);
  EG_CUDA(cudaGetLastError());
  // z
  axis(2);
  sm = (size_t)kLines * a.Mz * sizeof(double);
  a.nlines = (int64_t)Nx * Ny;
  a.table = t->storage == ST_F32 ? (float *)t->coefs : nullptr;
  a.zs = t->zs;
  a.slot_spline = t->slot_spline_d;
  a.colmax = (unsigned *)t->colmax;
  if (!a.table) EG_CUDA(cudaMemsetAsync(t->colmax, 0, ncw * sizeof(unsigned), s));
  if (int r = allow_smem((const void *)k_solve_z, sm)) return r;
  k_solve_z<<<(unsigned)((a.nlines * ncw + kLines - 1) / kLines), kLines, sm, s>>>(a);
  EG_CUDA(cudaGetLastError());
  count_launch(3);
  return 0;
}

}  // namespace eg
