// Fused QMC determinant step: orbital evaluation + Slater-determinant ratio,
// and the Sherman-Morrison update of the inverse after an accepted move.
//
// The reference's QMC prototype (src/cuda_walker.cu) moves electron k of
// every walker, evaluates the N orbitals at the new positions into a row
// buffer (calc_new_row, :69-88, eval_multi_multi_UBspline_3d_s_cuda), dots
// that row with column k of each walker's inverse Slater matrix (calc_ratios,
// :171-201) and, for accepted walkers, updates the inverse in two kernels
// (update_inverse_cuda1/2, src/determinant_update.h:9-111, launched at
// src/cuda_walker.cu:92-136).
//
// k_det_ratio fuses the first two: a block of 4 warps gathers the stencil
// of all N orbitals with the evaluation kernels' separable reduction and
// contracts value, gradient and Laplacian with the inverse column in
// registers, so the per-orbital outputs never reach HBM (only the value row,
// on request, for the update).  Block sums use a fixed shuffle tree: results
// are deterministic.  k_det_tc does the same for F16 and BF16 tables on the
// tensor cores (their default load mode 5).
//
// The update (k_det_update; matrices above kUpMax by separate kernels, one
// a pass) is two passes over each accepted walker's inverse:
//   pass 1: x = delta^T Ainv (delta = u - A[k,:]) and colk = Ainv[:,k];
//   pass 2: Ainv += (-1 / (1 + x[k])) colk x^T, A[k,:] = u.
// Unlike the reference's kernel 1, where every block of a walker writes the
// new row into A while other blocks still read the old one, A is only read in
// pass 1 and written in pass 2.
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "eval_core.h"

namespace eg {

struct DetArgs {
  EvalArgs e;                  // geometry, storage scale, positions, rule
  const float *const *ainv;    // per walker
  float *const *amat;          // update: per walker A (row k replaced)
  const float *const *urow;    // update: per walker new row u
  float *const *row_out;       // ratio: optional value row per walker
  float *ratio, *grad, *lapl;  // ratio outputs (grad, lapl optional)
  float *work;                 // update scratch: [walker][2][n] (x, colk)
  const int64_t *refused;      // update: a walker index was out of range, nothing is updated (or null)
  int n, k, ld, trans;
};

constexpr int kDetThreads = 128;
// Copy-pipeline depth: two stages keep a block at ~70 KB of shared memory so
// three blocks (12 warps) share an SM; the register cap of the kernel
// (launch bounds) matches.
constexpr int kDetStages = 2;
constexpr int kDetBlocksPerSM = 3;

// Inverse entry (orbital j, electron c).
__device__ __forceinline__ float ainv_at(const float *m, int j, int c, int ld, int trans) {
  return trans ? m[(int64_t)c * ld + j] : m[(int64_t)j * ld + c];
}

// Shared memory of k_det_ratio: the evaluation prologue's weights, cells and
// sources for pb walkers, the copy pipeline, and per-warp partial sums.
__host__ __device__ __forceinline__ size_t det_pipe_off(int pb) { return align_up(smem_total(pb, 4), 16); }
__host__ __device__ __forceinline__ size_t det_red_off(int pb, int rb) {
  return det_pipe_off(pb) + pipe_bytes(kDetThreads, rb, kDetStages);
}
__host__ __device__ __forceinline__ size_t det_ptr_off(int pb, int rb) {
  return align_up(det_red_off(pb, rb) + (size_t)pb * (kDetThreads / 32) * 5 * sizeof(float), 16);
}
__host__ __device__ __forceinline__ size_t det_av_off(int pb, int rb) {
  return align_up(det_ptr_off(pb, rb) + (size_t)pb * sizeof(void *), 16);
}
__host__ __device__ __forceinline__ size_t det_smem(int pb, int rb) {
  return det_av_off(pb, rb) + (size_t)kDetThreads * 8 * sizeof(float);
}

// A block takes pb walkers and all N orbitals, in column groups of
// kDetThreads * VW.  A pipeline stage is one x-plane (16 stencil rows) of one
// column group of one walker; as in k_eval_pipe each thread copies its own
// columns of the rows of stage s+2 into shared memory while it reduces stage
// s, and reads back only what it copied.  At the end of a walker's planes the
// thread dots its columns' value, gradient and Laplacian with the inverse
// column (loaded when the walker's first plane starts, so its latency hides
// behind the reduction); at the end of the walker each warp folds its lanes
// with a fixed shuffle tree into shared memory, and after the loop one thread
// per walker adds the warps in order.  WIDE (16-bit tables): 8 columns and
// one 16-byte copy per thread and row.
template <int ST, bool GL, bool WIDE>
__global__ void __launch_bounds__(kDetThreads, kDetBlocksPerSM) k_det_ratio(const DetArgs d) {
  using Raw = typename CT<ST>::Raw;
  static_assert(sizeof(typename CT<ST>::A) == 4, "determinant step: real float tables only");
  constexpr int VW = WIDE ? 2 * CT<ST>::VW : CT<ST>::VW;
  constexpr int RB = WIDE ? 2 * (int)sizeof(Raw) : (int)sizeof(Raw);
  constexpr int NW = kDetThreads / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  const EvalArgs &a = d.e;
  const int64_t p0 = (int64_t)blockIdx.x * a.pb;
  const int pn = eval_prologue<float>(a, smem, p0, a.pb, threadIdx.x, kDetThreads);
  const float **sptr = reinterpret_cast<const float **>(smem + det_ptr_off(a.pb, RB));
  for (int q = threadIdx.x; q < pn; q += kDetThreads) sptr[q] = d.ainv[p0 + q];
  __syncthreads();
  const float *sw = reinterpret_cast<const float *>(smem);
  const int *sidx = reinterpret_cast<const int *>(smem + smem_w_bytes(a.pb, 4));
  const int64_t *ssrc = reinterpret_cast<const int64_t *>(smem + smem_w_bytes(a.pb, 4) + align_up((size_t)a.pb * 12, 8));
  unsigned char *pipe = smem + det_pipe_off(a.pb);
  float *red = reinterpret_cast<float *>(smem + det_red_off(a.pb, RB));
  // the thread's inverse-column entries of the walker in flight: copied with
  // the walker's first plane, read when that plane is reduced (the next
  // first plane is four stages later, after the pipeline's depth)
  float *avbuf = reinterpret_cast<float *>(smem + det_av_off(a.pb, RB)) + threadIdx.x * VW;

  constexpr int GC = kDetThreads * VW;  // columns per group
  const int G = (d.n + GC - 1) / GC;
  const int64_t xsb = a.xs * CT<ST>::BYTES, ysb = a.ys * CT<ST>::BYTES, zsb = a.zs * CT<ST>::BYTES;
  const char *cbase = reinterpret_cast<const char *>(a.coefs) + (int64_t)threadIdx.x * VW * CT<ST>::BYTES;
  const unsigned my = (unsigned)__cvta_generic_to_shared(pipe + (size_t)threadIdx.x * RB);
  constexpr unsigned row_step = (unsigned)(kDetThreads * RB), slot_step = 16u * row_step;
  const int S = pn * G * 4;
  auto issue = [&](int st) {
    const int i = st & 3, rest = st >> 2, g = rest % G, pp = rest / G;
    if ((g * kDetThreads + (int)threadIdx.x) * VW >= d.n) return;
    const char *plane = cbase + (int64_t)g * GC * CT<ST>::BYTES + (sidx[3 * pp] + i) * xsb +
                        sidx[3 * pp + 1] * ysb + sidx[3 * pp + 2] * zsb;
    const unsigned dst = my + (unsigned)(st % kDetStages) * slot_step;
#pragma unroll
    for (int r = 0; r < 16; r++) cp_async<RB>(dst + r * row_step, plane + (r >> 2) * ysb + (r & 3) * zsb);
    if (i == 0) {
      const int col0 = (g * kDetThreads + (int)threadIdx.x) * VW;
      const float *src = d.trans ? sptr[pp] + (int64_t)d.k * d.ld + col0 : sptr[pp] + (int64_t)col0 * d.ld + d.k;
      const unsigned av = (unsigned)__cvta_generic_to_shared(avbuf);
      if (d.trans && col0 + VW <= d.n && al16(src)) {
#pragma unroll
        for (int e = 0; e < VW; e += 4) cp_async<16>(av + 4 * e, reinterpret_cast<const char *>(src + e));
      } else {
        const int64_t step = d.trans ? 1 : d.ld;
#pragma unroll
        for (int e = 0; e < VW; e++)
          if (col0 + e < d.n) cp_async<4>(av + 4 * e, reinterpret_cast<const char *>(src + e * step));
      }
    }
  };
#pragma unroll
  for (int st = 0; st < kDetStages - 1; st++) {
    if (st < S) issue(st);
    cp_async_commit();
  }
  float o[10][VW];  // assigned by each point's plane 0
  float wz[3][4];
  float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  float av[VW];
  for (int st = 0; st < S; st++) {
    if (st + kDetStages - 1 < S) issue(st + kDetStages - 1);
    cp_async_commit();
    cp_async_wait<kDetStages - 1>();
    const int i = st & 3, rest = st >> 2, g = rest % G, pp = rest / G;
    const int col0 = (g * kDetThreads + (int)threadIdx.x) * VW;
    const bool live = col0 < d.n;
    const float *w = sw + pp * 36;
    if (i == 0) {
      z_weights<float>(w, wz);
      if (live) {
#pragma unroll
        for (int e = 0; e < VW; e++) av[e] = col0 + e < d.n ? avbuf[e] : 0.f;
      }
    }
    if (live) {
      const unsigned char *slot = pipe + (size_t)(st % kDetStages) * slot_step + (size_t)threadIdx.x * RB;
      reduce_plane<float, VW, GL>(
          i, w, wz,
          [&](int j, int k, float(&c)[VW]) {
            const Raw *rp = reinterpret_cast<const Raw *>(slot + (j * 4 + k) * row_step);
            if (WIDE) {
              float lo[CT<ST>::VW], hi[CT<ST>::VW];
              CT<ST>::decode(rp[0], lo);
              CT<ST>::decode(rp[1], hi);
#pragma unroll
              for (int e = 0; e < CT<ST>::VW; e++) { c[e] = lo[e]; c[CT<ST>::VW + e] = hi[e]; }
            } else {
              CT<ST>::decode(rp[0], *reinterpret_cast<float(*)[CT<ST>::VW]>(&c[0]));
            }
          },
          o);
    }
    if (i == 3) {
      if (live) {
        if (a.scale) {
#pragma unroll
          for (int e = 0; e < VW; e++) {
            const float sc = a.scale[col0 + e];
#pragma unroll
            for (int q = 0; q < (GL ? 10 : 1); q++) o[q][e] *= sc;
          }
        }
        float *row = d.row_out ? d.row_out[ssrc[pp]] : nullptr;
#pragma unroll
        for (int e = 0; e < VW; e++) {
          acc[0] = fmaf(o[0][e], av[e], acc[0]);
          if (GL) {
            acc[1] = fmaf(o[1][e], av[e], acc[1]);
            acc[2] = fmaf(o[2][e], av[e], acc[2]);
            acc[3] = fmaf(o[3][e], av[e], acc[3]);
            acc[4] = fmaf((o[4][e] + o[7][e]) + o[9][e], av[e], acc[4]);
          }
          if (row && col0 + e < d.n) row[col0 + e] = o[0][e];
        }
      }
      if (g == G - 1) {
#pragma unroll
        for (int q = 0; q < 5; q++) {
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], off);
          if ((threadIdx.x & 31) == 0) red[(pp * NW + (threadIdx.x >> 5)) * 5 + q] = acc[q];
          acc[q] = 0.f;
        }
      }
    }
  }
  __syncthreads();
  if ((int)threadIdx.x < pn) {
    const int pp = threadIdx.x;
    float s[5];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      s[q] = red[pp * NW * 5 + q];
#pragma unroll
      for (int r = 1; r < NW; r++) s[q] += red[(pp * NW + r) * 5 + q];
    }
    const int64_t wk = ssrc[pp];
    d.ratio[wk] = s[0];
    if (GL) {
      const float inv = 1.0f / s[0];
      if (d.grad) {
        d.grad[3 * wk] = s[1] * inv;
        d.grad[3 * wk + 1] = s[2] * inv;
        d.grad[3 * wk + 2] = s[3] * inv;
      }
      if (d.lapl) d.lapl[wk] = s[4] * inv;
    }
  }
}

// ------------------------------------------------------------ tensor cores
// k_det_tc: the ratio of F16 and BF16 tables in their default load mode 5,
// with the evaluation kernel's tensor-core contraction (k_eval_tc, eval.cu):
// per walker and tile of 128 orbitals, D[128 orbitals x NC] = A[128 x 64] *
// B[64 x NC] in four tcgen05.mma (K = 16, one per x-plane), A the stencil as
// a TMA box copies it (128-byte swizzle), B the walker's weights of seven
// outputs (value, gradient, the Hessian's diagonal) split into the table
// type's parts, each part in its own column.  Instead of storing the
// outputs, the epilogue dots them with the inverse column.
//
// A block takes pb walkers and all N orbitals: unit u = p * TT + t is tile
// t of walker p.  Warp 0 (one lane) keeps kDtStages stencil copies in
// flight, one unit a stage; warp 1 (one lane) issues a unit's MMAs into
// one of the block's accumulator slots (unit u into slot u modulo their
// number) once its stencil, the walker's weights and the slot are there,
// and commits the unit to the barriers that free its
// stage and fill its slot; warps 2-5 (one orbital of each tile a thread)
// read a slot, free it, add the weight parts, scale, and accumulate the
// products with the thread's inverse entries; at a walker's last tile (its
// MMAs then all complete) they build the weights of the walker two ahead in
// its buffer and fold their five sums with a fixed shuffle tree into shared
// memory, which one thread per walker adds up in order after the loop, so
// the results are deterministic.  The value row, on request, equals the
// flat evaluation's mode-5 values bit for bit.  Every wait is bounded, as
// in k_eval_tc.
//
// Two stencil stages and five blocks an SM: more walkers in flight than four
// stages and three blocks (2,048 walkers: 0.047 against 0.052 ms; 16,384:
// 0.285 against 0.298 ms).
constexpr int kDtStages = 2, kDtSlots = 4, kDtMaxWalkers = 7, kDtBlocksPerSM = 5, kDtUnits = 8;
__host__ __device__ __forceinline__ size_t dt_ptr_off(int pb) { return align_up(smem_total(pb, 4), 16); }
__host__ __device__ __forceinline__ size_t dt_red_off(int pb) { return dt_ptr_off(pb) + (size_t)pb * 8; }
__host__ __device__ __forceinline__ size_t dt_head(int pb) { return dt_red_off(pb) + (size_t)pb * 4 * 5 * 4; }
// the head, slack to align the operand area to 1024 bytes, the stages, two
// weight buffers, the mbarriers and the TMEM address / abort flag / count;
// at kDtMaxWalkers walkers kDtBlocksPerSM blocks share an SM
__host__ __device__ __forceinline__ size_t dt_smem(int pb) {
  return dt_head(pb) + 1024 + (size_t)kDtStages * 16384 + 2 * 4096 + 8 * (2 * kDtStages + 2 + 2 * kDtSlots) + 16;
}

template <int ST, bool GL>
__global__ void __launch_bounds__(kTcThreads, kDtBlocksPerSM) k_det_tc(const __grid_constant__ DetArgs d) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int NS = kDtStages, NP = TcCfg<ST>::parts, NQ = GL ? 7 : 1;
  constexpr int NC = NQ * NP <= 16 ? 16 : 32;  // accumulator columns a unit (the MMA's N)
  // accumulator slots: 64 TMEM columns a block, so five blocks hold 320 of 512
  constexpr int RA = NC == 16 ? kDtSlots : kDtSlots / 2;
  constexpr unsigned kB = 4096u, kStage = 16384u;
  constexpr int NW = 4;  // output warps
  const EvalArgs &a = d.e;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t p0 = (int64_t)blockIdx.x * a.pb;
  const int pn = (int)min((int64_t)a.pb, a.npts - p0);
  const int TT = (d.n + 127) >> 7;
  float *sw = reinterpret_cast<float *>(smem);
  int *sidx = reinterpret_cast<int *>(smem + smem_w_bytes(a.pb, 4));
  int64_t *ssrc = reinterpret_cast<int64_t *>(smem + smem_w_bytes(a.pb, 4) + align_up((size_t)a.pb * 12, 8));
  const float **sptr = reinterpret_cast<const float **>(smem + dt_ptr_off(a.pb));
  float *red = reinterpret_cast<float *>(smem + dt_red_off(a.pb));
  // cells and the unscaled basis weights (delta_inv applied in the epilogue)
  for (int q = tid; q < pn * 3; q += kTcThreads) {
    const int pp = q / 3, ax = q - 3 * pp;
    const int64_t src = p0 + pp;
    const double xd = a.pos_f64 ? reinterpret_cast<const double *>(a.pos)[3 * src + ax]
                                : (double)reinterpret_cast<const float *>(a.pos)[3 * src + ax];
    int idx;
    float t;
    cell(a, ax, xd, idx, t);
    bspline_weights<float>(t, sw + pp * 36 + ax * 12, 1.0f);
    sidx[pp * 3 + ax] = idx;
    if (ax == 0) ssrc[pp] = src;
  }
  for (int q = tid; q < pn; q += kTcThreads) sptr[q] = d.ainv[p0 + q];
  const unsigned base_s = (unsigned)__cvta_generic_to_shared(smem);
  const unsigned a_s = (base_s + (unsigned)dt_head(a.pb) + 1023u) & ~1023u;
  const unsigned b_s = a_s + NS * kStage;
  const unsigned full_s = b_s + 2 * kB, empty_s = full_s + 8 * NS, bfull_s = empty_s + 8 * NS;
  const unsigned tfull_s = bfull_s + 16, tempty_s = tfull_s + 8 * RA, slot_s = tempty_s + 8 * RA;
  unsigned char *bgen = smem + (b_s - base_s);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + (slot_s + 4 - base_s));
  volatile int *consumed = reinterpret_cast<volatile int *>(smem + (slot_s + 8 - base_s));
  // weight columns past the outputs' parts stay zero
  for (int e = tid; e < 2 * (int)kB / 16; e += kTcThreads) reinterpret_cast<uint4 *>(bgen)[e] = make_uint4(0, 0, 0, 0);
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot_s), "n"(RA * NC)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 32) {
#pragma unroll
    for (int s = 0; s < NS; s++) {
      mbar_init(full_s + 8 * s, 1);
      mbar_init(empty_s + 8 * s, 1);
    }
#pragma unroll
    for (int b = 0; b < 2; b++) mbar_init(bfull_s + 8 * b, 128);
#pragma unroll
    for (int r = 0; r < RA; r++) {
      mbar_init(tfull_s + 8 * r, 1);
      mbar_init(tempty_s + 8 * r, 128);
    }
    *abort_flag = 0;
    *consumed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = *reinterpret_cast<volatile unsigned *>(smem + (slot_s - base_s));
  const unsigned long long lim = a.wait_ns ? a.wait_ns : kWaitNs;
  auto wait = [&](unsigned bar, unsigned parity) -> bool {
    if (*abort_flag) return false;
    if (mbar_wait(bar, parity, lim)) return true;
    *abort_flag = 1;
    return false;
  };
  const int U = pn * TT;
  int issued = 0, skipped = -1, last_commit = -1;
  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_map(&a.tmap);
      for (int u = 0; u < U; u++) {
        const int s = u % NS, p = u / TT, t = u - p * TT;
        if (u >= NS && !wait(empty_s + 8 * s, (unsigned)((u / NS - 1) & 1))) break;
        issued = u + 1;
        // test hook: no copy for this walker, so its wait runs out
        if (a.test_skip == p + 1 && blockIdx.x == 0) { skipped = p; continue; }
        mbar_arrive_expect_tx(full_s + 8 * s, kStage);
#pragma unroll
        for (int mg = 0; mg < 2; mg++)
          tma_load_4d(a_s + s * kStage + mg * 8192u, &a.tmap, full_s + 8 * s, 128 * t + 64 * mg, sidx[3 * p + 2],
                      sidx[3 * p + 1], sidx[3 * p]);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_16(128, NC, TcCfg<ST>::fmt);
      bool go = true;
      for (int p = 0; p < pn && go; p++) {
        const int bb = p & 1;
        if (!wait(bfull_s + 8 * bb, (unsigned)((p >> 1) & 1))) break;
        for (int t = 0; t < TT; t++) {
          const int u = p * TT + t, s = u % NS, r = u % RA;
          if (u >= RA && !wait(tempty_s + 8 * r, (unsigned)((u / RA - 1) & 1))) { go = false; break; }
          if (!wait(full_s + 8 * s, (unsigned)((u / NS) & 1))) { go = false; break; }
          *consumed = u + 1;
          tc_fence_after();
#pragma unroll
          for (int i = 0; i < 4; i++)
            umma_f16(tmem + r * NC, umma_desc(a_s + s * kStage + i * 2048u, 8192u, 1024u, 2),
                     umma_desc(b_s + bb * kB + i * 1024u, 128u, 256u, 0), idesc, i > 0);
          umma_commit(empty_s + 8 * s);
          umma_commit(tfull_s + 8 * r);
          last_commit = u;
        }
      }
    }
  } else {
    const int et = tid - 64;
    const int colr = (warp & 3) * 32 + lane;  // this thread's orbital (TMEM lane) in every tile
    // this thread's share of a weight matrix: stencil row k, outputs 0-3
    // (even threads) or 4-6 (odd threads)
    const int k = et >> 1;
    const int ki = k >> 4, kj = (k >> 2) & 3, km = k & 3, kk = k & 15;
    const unsigned boff = ki * 1024 + (kk >> 3) * 128 + (kk & 7) * 2;
    // derivative orders in x, y, z of each output (v, gx, gy, gz, hxx, hyy, hzz)
    static constexpr int OA[7] = {0, 1, 0, 0, 2, 0, 0};
    static constexpr int OB[7] = {0, 0, 1, 0, 0, 2, 0};
    static constexpr int OC[7] = {0, 0, 0, 1, 0, 0, 2};
    auto build_b = [&](int p) {
      const float *w = sw + p * 36;
      unsigned char *bm = bgen + (p & 1) * kB + boff;
      float wx[3], wy[3], wz[3];
#pragma unroll
      for (int dd = 0; dd < 3; dd++) {
        wx[dd] = w[4 * dd + ki];
        wy[dd] = w[12 + 4 * dd + kj];
        wz[dd] = w[24 + 4 * dd + km];
      }
      auto put = [&](auto qc) {
        constexpr int q = decltype(qc)::value;
        const float wq = wx[OA[q]] * wy[OB[q]] * wz[OC[q]];
        auto at = [&](int n) { return bm + (n >> 3) * 256 + (n & 7) * 16; };
        if constexpr (ST == ST_BF16) {
          const __nv_bfloat16 hi = __float2bfloat16_rn(wq);
          const float r1 = wq - __bfloat162float(hi);
          const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
          const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
          *reinterpret_cast<__nv_bfloat16 *>(at(3 * q)) = hi;
          *reinterpret_cast<__nv_bfloat16 *>(at(3 * q + 1)) = mid;
          *reinterpret_cast<__nv_bfloat16 *>(at(3 * q + 2)) = lo;
        } else {
          const __half hi = __float2half_rn(wq);
          const __half lo = __float2half_rn(wq - __half2float(hi));
          *reinterpret_cast<__half *>(at(2 * q)) = hi;
          *reinterpret_cast<__half *>(at(2 * q + 1)) = lo;
        }
      };
      if (!(et & 1)) {
        put(std::integral_constant<int, 0>());
        if constexpr (GL) {
          put(std::integral_constant<int, 1>());
          put(std::integral_constant<int, 2>());
          put(std::integral_constant<int, 3>());
        }
      } else if constexpr (GL) {
        put(std::integral_constant<int, 4>());
        put(std::integral_constant<int, 5>());
        put(std::integral_constant<int, 6>());
      }
      fence_proxy_async();
      mbar_arrive(bfull_s + 8 * (p & 1));
    };
    const float dx = a.dinvf[0], dy = a.dinvf[1], dz = a.dinvf[2];
    float acc[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    build_b(0);
    if (pn > 1) build_b(1);
    // the inverse entry and the spline's factor of unit u, loaded during
    // unit u - 1 (the reference layout's entries are scattered 4-byte reads)
    auto load_av = [&](int u, float &av, float &sc) {
      const int p = u / TT, col = (u - p * TT) * 128 + colr;
      av = 0.f;
      sc = 1.f;
      if (u < U && col < d.n) {
        av = d.trans ? sptr[p][(int64_t)d.k * d.ld + col] : sptr[p][(int64_t)col * d.ld + d.k];
        if (a.scale) sc = a.scale[col];
      }
    };
    float av_n, sc_n;
    load_av(0, av_n, sc_n);
    for (int u = 0; u < U; u++) {
      const int p = u / TT, t = u - p * TT, r = u % RA;
      const int col = t * 128 + colr;
      const bool live = col < d.n;
      const float av = av_n, sc = sc_n;
      load_av(u + 1, av_n, sc_n);
      if (!wait(tfull_s + 8 * r, (unsigned)((u / RA) & 1))) break;
      // walker p's MMAs are all complete after its last tile: its weight
      // buffer takes walker p + 2's weights
      if (t == TT - 1 && p + 2 < pn) build_b(p + 2);
      tc_fence_after();
      uint32_t rr[32];
      if constexpr (NC == 16) tmem_ld16(tmem + ((unsigned)((warp & 3) * 32) << 16) + r * NC, rr);
      else tmem_ld32(tmem + ((unsigned)((warp & 3) * 32) << 16) + r * NC, rr);
      tc_fence_before();
      mbar_arrive(tempty_s + 8 * r);
      float o[NQ];
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        float v = __uint_as_float(rr[NP * q]);
#pragma unroll
        for (int h = 1; h < NP; h++) v += __uint_as_float(rr[NP * q + h]);
        o[q] = v;
      }
      if (live) {
        const float v = o[0] * (sc * 1.f);  // as the flat kernel's value: (sum of parts) x (factor x 1)
        acc[0] = fmaf(v, av, acc[0]);
        if constexpr (GL) {
          acc[1] = fmaf(o[1] * (sc * dx), av, acc[1]);
          acc[2] = fmaf(o[2] * (sc * dy), av, acc[2]);
          acc[3] = fmaf(o[3] * (sc * dz), av, acc[3]);
          const float lap = (o[4] * (sc * (dx * dx)) + o[5] * (sc * (dy * dy))) + o[6] * (sc * (dz * dz));
          acc[4] = fmaf(lap, av, acc[4]);
        }
        if (d.row_out) d.row_out[ssrc[p]][col] = v;
      }
      if (t == TT - 1) {
#pragma unroll
        for (int q = 0; q < 5; q++) {
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], off);
          if (lane == 0) red[(p * NW + (warp - 2)) * 5 + q] = acc[q];
          acc[q] = 0.f;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out: report it, and let no copy or MMA outlive the block
    if (tid == 0) {
      if (a.wait_err) {
        *(volatile int *)a.wait_err = 1;
        __threadfence_system();
      }
      for (int u = *consumed; u < issued; u++)
        if (u / TT != skipped) mbar_wait(full_s + 8 * (u % NS), (unsigned)((u / NS) & 1), lim);
    }
    if (tid == 32 && last_commit >= 0) {
      const int u = *consumed - 1;
      mbar_wait(empty_s + 8 * (u % NS), (unsigned)((u / NS) & 1), lim);
    }
  } else if (tid < pn) {
    const int pp = tid;
    float s[5];
#pragma unroll
    for (int q = 0; q < 5; q++) {
      s[q] = red[pp * NW * 5 + q];
#pragma unroll
      for (int w = 1; w < NW; w++) s[q] += red[(pp * NW + w) * 5 + q];
    }
    const int64_t wk = ssrc[pp];
    d.ratio[wk] = s[0];
    if (GL) {
      const float inv = 1.0f / s[0];
      if (d.grad) {
        d.grad[3 * wk] = s[1] * inv;
        d.grad[3 * wk + 1] = s[2] * inv;
        d.grad[3 * wk + 2] = s[3] * inv;
      }
      if (d.lapl) d.lapl[wk] = s[4] * inv;
    }
  }
  __syncthreads();
  tc_fence_after();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(RA * NC) : "memory");
}

// ------------------------------------------------------------ fused update
// Accepted walkers' updates, each by one thread-block cluster: the CTAs
// split the stored rows of the inverse, read them for x and column k, exchange
// over distributed shared memory, and read them again for the rank-1
// correction while they are still in L2.  The two passes below move 3 N^2
// floats a walker through DRAM, this 2 N^2.  Clusters stay and take walker
// after walker.
//
// The rows stream through a ring of kUpDepth 16-byte asynchronous copies a
// thread, in order: a walker's rows, the same rows again, the next walker's.
// A thread reads back only what it copied itself, so the stream needs no
// barrier, and the copies in flight (64 KB for 512 threads) keep DRAM busy
// while the cluster exchanges.  Bound by DRAM: 768 x 768, 512 walkers: 488 us
// (two passes 1098 us), 2.78 GB at 5.8 TB/s, of which 0.4 GB are rows that
// had left L2; launch shapes and figures at update_shape.
//
// Reference layout (TRANS 0, rows are orbitals): every CTA sums its rows'
// share of x for all columns, and every CTA adds all shares in rank order.
// A thread owns a unit of 4 columns and every G-th row of its CTA.
// Transposed layout (rows are electrons): x[c] is the dot product of row c
// with delta, found and used by the same CTA; column k is stored row k, which
// every CTA reads before its owner changes it.  2^lpr_log lanes share a row.
//
// Sums run in a fixed order: results do not vary from run to run.
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// The float at shared-memory address a (of this CTA) in CTA `rank` of the cluster.
__device__ __forceinline__ float ld_cluster(unsigned a, unsigned rank) {
  float v;
  asm volatile(
      "{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.f32 %0, [ra];\n\t}"
      : "=f"(v)
      : "r"(a), "r"(rank)
      : "memory");
  return v;
}

constexpr int kUpVec = 4;    // entries of a walker's vectors a thread: n <= kUpVec * THREADS
constexpr int kUpDepth = 8;  // items in flight a thread

// Shared memory: the ring, then floats -- the new row's own entries; TRANS 0:
// the own rows' delta and column k, this CTA's share of x, x, partial sums of
// the row groups; TRANS 1: delta, column k, the own rows' x.
__host__ __device__ __forceinline__ int up4(int n) { return (n + 3) & ~3; }
__host__ __device__ __forceinline__ size_t up_smem(int n, int cs, int trans, int threads) {
  const size_t n4 = up4(n), own = up4((n + cs - 1) / cs);
  const size_t part = n4 > (size_t)(4 * threads) ? n4 : 4 * threads;
  return (size_t)kUpDepth * threads * 16 + 4 * (trans ? 2 * n4 + 2 * own : 3 * own + 2 * n4 + part);
}

template <int TRANS, int THREADS>
__global__ void __launch_bounds__(THREADS) k_det_update(const DetArgs d, int cs, int naccept, int lpr_log) {
  if (d.refused && *d.refused) return;  // the same on every block
  extern __shared__ __align__(16) unsigned char up_raw[];
  constexpr int D = kUpDepth;
  constexpr unsigned kSlot = THREADS * 16;
  float *up = reinterpret_cast<float *>(up_raw + D * kSlot);
  const int n = d.n, tid = threadIdx.x;
  const int U = (n + 3) >> 2, n4 = up4(n), own = (n + cs - 1) / cs, ownp = up4(own);
  const unsigned rank = cluster_rank();
  const int step = gridDim.x / cs;
  const int r0 = (int)((int64_t)n * rank / cs), r1 = (int)((int64_t)n * (rank + 1) / cs);
  // A pass over the own rows takes QN x R items a thread, the same for every
  // thread, in whole rounds of D; this one has NQ x NR of them (TRANS 0: R
  // rows of one unit; TRANS 1: QN rows of R units).
  const int LPR = 1 << lpr_log;
  const int G = TRANS ? THREADS >> lpr_log : THREADS / U;
  const int g = TRANS ? tid >> lpr_log : tid / U;
  const int q0 = TRANS ? tid & (LPR - 1) : tid % U;
  const int QN = TRANS ? (own + G - 1) / G : 1;
  const int R = TRANS ? (U + LPR - 1) >> lpr_log : (own + G - 1) / G;
  const int rounds = (QN * R + D - 1) / D;
  const int rows = g < G && r0 + g < r1 ? (r1 - r0 - g + G - 1) / G : 0;
  const int NQ = TRANS ? rows : 1, NR = TRANS ? (U - q0 + LPR - 1) >> lpr_log : rows;
  const int64_t first = (int64_t)(r0 + g) * d.ld + 4 * q0;      // the first item's place in the matrix
  const int64_t inner = TRANS ? 4 * LPR : (int64_t)G * d.ld;    // from item to item
  const int64_t outer = TRANS ? (int64_t)G * d.ld - (int64_t)R * inner : 0;  // further after R items (TRANS 1)
  const int tail = n & 3;                                       // columns of the last unit, when not 4
  const bool rows16 = (d.ld & 3) == 0;                          // every row as aligned as the first

  // the stream's issue side: the next round's walker, pass and items
  const float *ibase = nullptr, *inext = nullptr, *isrc = nullptr;
  int iw = blockIdx.x / cs, iround = 0, iq = 0, ir = 0, ipass = 0;
  bool ivec = false;
  auto enter_walker = [&](const float *base) {
    ibase = base;
    ivec = rows16 && al16(base);
    isrc = base + first;
    if (iw + step < naccept) inext = d.ainv[iw + step];
  };
  if (iw < naccept) enter_walker(d.ainv[iw]);
  else ir = NR;  // nothing to copy
  const unsigned ring = (unsigned)__cvta_generic_to_shared(up_raw) + tid * 16;
  auto issue = [&](int q) {  // one item into slot q
    if (TRANS ? ir < NR && iq < NQ : ir < NR) {
      const unsigned dst = ring + q * kSlot;
      if (ivec) {  // a last unit of fewer columns reads on into its row's padding
        cp_async<16>(dst, reinterpret_cast<const char *>(isrc));
      } else {
        const int e1 = tail && q0 + (TRANS ? ir << lpr_log : 0) == U - 1 ? tail : 4;
        for (int e = 0; e < e1; e++) cp_async<4>(dst + 4 * e, reinterpret_cast<const char *>(isrc + e));
      }
    }
    cp_async_commit();
    isrc += inner;
    ir++;
    if (TRANS && ir == R) {
      ir = 0;
      iq++;
      isrc += outer;
    }
  };
  auto next_round = [&]() {
    if (++iround < rounds) return;
    iround = iq = ir = 0;
    if ((ipass ^= 1) == 0) {
      iw += step;
      if (iw < naccept) enter_walker(inext);
    }
    if (iw < naccept) isrc = ibase + first;
    else { ir = NR; iq = NQ; }
  };
#pragma unroll
  for (int q = 0; q < D; q++) issue(q);
  next_round();
  // the item in slot q, the oldest in flight
  auto take = [&](int q) {
    cp_async_wait<D - 1>();
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(ring + q * kSlot)
                 : "memory");
    return v;
  };

  float *unew = up, *delta = up + ownp, *ck = delta + (TRANS ? n4 : ownp), *sx = ck + (TRANS ? n4 : ownp);
  float *xf = sx + n4, *part = xf + n4;  // TRANS 0
  // The vectors a walker needs beside its rows (u and A's row k -- the own
  // entries, or for TRANS all of them and stored row k) are read into
  // registers a walker ahead, so that no wait for them is exposed.
  const int v0 = TRANS ? 0 : r0, v1 = TRANS ? n : r1;
  float vu[kUpVec], va[kUpVec], vk[TRANS ? kUpVec : 1];
  int w = blockIdx.x / cs;
  const float *pu = nullptr, *pa = nullptr, *pm = nullptr;
  auto addresses = [&](int wk) {
    if (wk < naccept) { pu = d.urow[wk]; pa = d.amat[wk]; pm = d.ainv[wk]; }
  };
  auto read_vectors = [&]() {
#pragma unroll
    for (int i = 0; i < kUpVec; i++) {
      const int j = v0 + tid + i * THREADS;
      if (j < v1) {
        vu[i] = pu[j];
        va[i] = pa[(int64_t)d.k * d.ld + j];
        if (TRANS) vk[TRANS ? i : 0] = pm[(int64_t)d.k * d.ld + j];
      }
    }
  };
  addresses(w);
  if (w < naccept) read_vectors();
  const unsigned sxa = (unsigned)__cvta_generic_to_shared(sx);
  const int kc = !TRANS && q0 == d.k >> 2 ? d.k & 3 : -1;  // the component of this thread's unit in column k
  for (; w < naccept; w += step) {
    float *m = const_cast<float *>(pm), *arow = const_cast<float *>(pa) + (int64_t)d.k * d.ld;
    const bool vec = rows16 && al16(m);
    __syncthreads();  // the last walker's vectors are no longer read
#pragma unroll
    for (int i = 0; i < kUpVec; i++) {
      const int j = v0 + tid + i * THREADS;
      if (j < v1) {
        delta[j - v0] = vu[i] - va[i];
        if (TRANS) ck[j] = vk[TRANS ? i : 0];
        if (!TRANS || (j >= r0 && j < r1)) unew[j - r0] = vu[i];
      } else if (TRANS && j < n4) {
        delta[j] = ck[j] = 0.f;
      }
    }
    addresses(w + step);
    __syncthreads();
    // pass 1: x
    if constexpr (TRANS) {
      int qi = 0, ri = 0;
      float s = 0.f;
      for (int c = 0; c < rounds; c++) {
#pragma unroll
        for (int q = 0; q < D; q++) {
          float4 v = take(q);
          if (ri < NR && qi < NQ) {
            const int unit = q0 + (ri << lpr_log);
            if (tail && unit == U - 1) {  // what lies past the row's end does not count, not even as 0 * NaN
              v.w = 0.f;
              if (tail < 3) v.z = 0.f;
              if (tail < 2) v.y = 0.f;
            }
            const float4 de = *reinterpret_cast<const float4 *>(delta + 4 * unit);
            s = fmaf(v.x, de.x, s); s = fmaf(v.y, de.y, s);
            s = fmaf(v.z, de.z, s); s = fmaf(v.w, de.w, s);
          }
          issue(q);
          if (++ri == R) {
            for (int off = LPR >> 1; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
            if (q0 == 0 && qi < NQ) sx[g + qi * G] = s;
            s = 0.f;
            ri = 0;
            qi++;
          }
        }
        next_round();
      }
    } else {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      const float *de = delta + g;
      float *cp = ck + g;
      int left = NR;
      for (int c = 0; c < rounds; c++, left -= D) {
#pragma unroll
        for (int q = 0; q < D; q++, de += G, cp += G) {
          const float4 v = take(q);
          if (q < left) {
            const float x = *de;
            if (kc >= 0) *cp = kc == 0 ? v.x : kc == 1 ? v.y : kc == 2 ? v.z : v.w;
            acc.x = fmaf(v.x, x, acc.x); acc.y = fmaf(v.y, x, acc.y);
            acc.z = fmaf(v.z, x, acc.z); acc.w = fmaf(v.w, x, acc.w);
          }
          issue(q);
        }
        next_round();
      }
      if (g < G) *reinterpret_cast<float4 *>(part + g * n4 + 4 * q0) = acc;
    }
    __syncthreads();
    if (!TRANS) {
      for (int c = tid; c < n; c += THREADS) {
        float s = part[c];
        for (int i = 1; i < G; i++) s += part[i * n4 + c];
        sx[c] = s;
      }
    }
    // the shares of x are ready; A's row k and stored row k have been read
    cluster_arrive();
    cluster_wait();
    if (TRANS) {
      const int kown = (int)((((int64_t)d.k + 1) * cs - 1) / n);  // the CTA that holds row k
      const float p = -1.0f / (1.0f + ld_cluster(sxa + 4 * (d.k - (int)((int64_t)n * kown / cs)), kown));
      for (int j = tid; j < n; j += THREADS) ck[j] *= p;
    } else {
      for (int c = tid; c < n4; c += THREADS) {
        float s = 0.f;
        if (c < n) {
          float t[8];  // clusters of at most 8: all reads in flight at once
#pragma unroll
          for (int i = 0; i < 8; i++) t[i] = i < cs ? ld_cluster(sxa + 4 * c, i) : 0.f;
#pragma unroll
          for (int i = 0; i < 8; i++) s += t[i];
        }
        xf[c] = s;
      }
    }
    cluster_arrive();  // this CTA is done with the others' shared memory
    for (int j = r0 + tid; j < r1; j += THREADS) arow[j] = unew[j - r0];
    __syncthreads();
    if (w + step < naccept) read_vectors();
    // pass 2: the correction
    float *dst = m + first;
    auto put = [&](float4 v, int unit) {
      const bool whole = tail == 0 || unit != U - 1;
      if (vec && whole) {
        __stcs(reinterpret_cast<float4 *>(dst), v);
      } else {
        dst[0] = v.x;
        if (whole || tail > 1) dst[1] = v.y;
        if (whole || tail > 2) dst[2] = v.z;
        if (whole) dst[3] = v.w;
      }
    };
    if constexpr (TRANS) {
      int qi = 0, ri = 0;
      float xr = NQ > 0 ? sx[g] : 0.f;
      for (int c = 0; c < rounds; c++) {
#pragma unroll
        for (int q = 0; q < D; q++) {
          float4 v = take(q);
          if (ri < NR && qi < NQ) {
            const int unit = q0 + (ri << lpr_log);
            const float4 c4 = *reinterpret_cast<const float4 *>(ck + 4 * unit);
            v.x = fmaf(xr, c4.x, v.x); v.y = fmaf(xr, c4.y, v.y);
            v.z = fmaf(xr, c4.z, v.z); v.w = fmaf(xr, c4.w, v.w);
            put(v, unit);
          }
          issue(q);
          dst += inner;
          if (++ri == R) {
            ri = 0;
            qi++;
            dst += outer;
            if (qi < NQ) xr = sx[g + qi * G];
          }
        }
        next_round();
      }
    } else {
      const float p = -1.0f / (1.0f + xf[d.k]);
      const float4 x = *reinterpret_cast<const float4 *>(xf + 4 * q0);
      const float *cp = ck + g;
      int left = NR;
      for (int c = 0; c < rounds; c++, left -= D) {
#pragma unroll
        for (int q = 0; q < D; q++, cp += G, dst += inner) {
          float4 v = take(q);
          if (q < left) {
            const float rs = p * *cp;
            v.x = fmaf(x.x, rs, v.x); v.y = fmaf(x.y, rs, v.y);
            v.z = fmaf(x.z, rs, v.z); v.w = fmaf(x.w, rs, v.w);
            put(v, q0);
          }
          issue(q);
        }
        next_round();
      }
    }
    cluster_wait();
  }
  cp_async_wait<0>();
}

// Pass 1, reference layout (Ainv[j][c] row-major): thread per column c,
// rows streamed in order with delta staged in shared memory; the thread that
// owns column k also copies that column out.
__global__ void __launch_bounds__(256) k_det_update1_rows(const DetArgs d) {
  __shared__ float sdelta[256];
  if (d.refused && *d.refused) return;
  const int w = blockIdx.y;
  const int c = blockIdx.x * 256 + threadIdx.x;
  const float *ainv = d.ainv[w];
  const float *u = d.urow[w];
  const float *ak = d.amat[w] + (int64_t)d.k * d.ld;
  float *x = d.work + (int64_t)w * 2 * d.n, *colk = x + d.n;
  float acc = 0.f;
  for (int j0 = 0; j0 < d.n; j0 += 256) {
    const int jn = min(256, d.n - j0);
    __syncthreads();
    if (threadIdx.x < jn) sdelta[threadIdx.x] = u[j0 + threadIdx.x] - ak[j0 + threadIdx.x];
    __syncthreads();
    if (c < d.n) {
      for (int i = 0; i < jn; i++) {
        const float v = ainv[(int64_t)(j0 + i) * d.ld + c];
        if (c == d.k) colk[j0 + i] = v;
        acc = fmaf(v, sdelta[i], acc);
      }
    }
  }
  if (c < d.n) x[c] = acc;
}

// Pass 1, transposed layout (AinvT[c][j]): warp per row c, a dot product
// with delta (16-byte loads when the rows allow); the warp on row k also
// copies that row (column k of Ainv).
__global__ void __launch_bounds__(256) k_det_update1_trans(const DetArgs d) {
  const int w = blockIdx.y;
  const int c = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (c >= d.n || (d.refused && *d.refused)) return;
  const float *ainvr = d.ainv[w] + (int64_t)c * d.ld;
  const float *u = d.urow[w];
  const float *ak = d.amat[w] + (int64_t)d.k * d.ld;
  float *x = d.work + (int64_t)w * 2 * d.n, *colk = x + d.n;
  const bool copy = c == d.k;
  float acc = 0.f;
  int j0 = 0;
  if (al16(ainvr) && al16(u) && al16(ak) && (!copy || al16(colk))) {
    const int n4 = d.n >> 2;
    for (int q = lane; q < n4; q += 32) {
      const float4 v = reinterpret_cast<const float4 *>(ainvr)[q];
      const float4 uu = reinterpret_cast<const float4 *>(u)[q];
      const float4 aa = reinterpret_cast<const float4 *>(ak)[q];
      if (copy) reinterpret_cast<float4 *>(colk)[q] = v;
      acc = fmaf(v.x, uu.x - aa.x, acc);
      acc = fmaf(v.y, uu.y - aa.y, acc);
      acc = fmaf(v.z, uu.z - aa.z, acc);
      acc = fmaf(v.w, uu.w - aa.w, acc);
    }
    j0 = n4 << 2;
  }
  for (int j = j0 + lane; j < d.n; j += 32) {
    const float v = ainvr[j];
    if (copy) colk[j] = v;
    acc = fmaf(v, u[j] - ak[j], acc);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane == 0) x[c] = acc;
}

// Pass 2: rank-1 correction of every entry and the new row of A; warp per
// stored row, 16-byte accesses when the row allows.  Entry (orbital j,
// electron c) becomes Ainv + x[c] * (p * colk[j]) in both layouts (the
// reference's kernel 2 expression, src/determinant_update.h:104-106).
__global__ void __launch_bounds__(256) k_det_update2(const DetArgs d) {
  const int w = blockIdx.y;
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (r >= d.n || (d.refused && *d.refused)) return;
  const float *x = d.work + (int64_t)w * 2 * d.n, *colk = x + d.n;
  const float p = -1.0f / (1.0f + x[d.k]);
  float *m = const_cast<float *>(d.ainv[w]) + (int64_t)r * d.ld;
  // reference layout: row r is orbital j = r, columns are electrons c;
  // transposed: row r is electron c = r, columns are orbitals j
  const float *vec = d.trans ? colk : x;
  const float rs = d.trans ? x[r] : p * colk[r];
  int i0 = 0;
  if (al16(m) && al16(vec)) {
    const int n4 = d.n >> 2;
    for (int q = lane; q < n4; q += 32) {
      float4 mv = reinterpret_cast<float4 *>(m)[q];
      const float4 v = reinterpret_cast<const float4 *>(vec)[q];
      if (d.trans) {
        mv.x = fmaf(rs, p * v.x, mv.x); mv.y = fmaf(rs, p * v.y, mv.y);
        mv.z = fmaf(rs, p * v.z, mv.z); mv.w = fmaf(rs, p * v.w, mv.w);
      } else {
        mv.x = fmaf(v.x, rs, mv.x); mv.y = fmaf(v.y, rs, mv.y);
        mv.z = fmaf(v.z, rs, mv.z); mv.w = fmaf(v.w, rs, mv.w);
      }
      reinterpret_cast<float4 *>(m)[q] = mv;
    }
    i0 = n4 << 2;
  }
  for (int i = i0 + lane; i < d.n; i += 32) m[i] = d.trans ? fmaf(rs, p * vec[i], m[i]) : fmaf(vec[i], rs, m[i]);
  if (r == d.k) {
    float *ak = d.amat[w] + (int64_t)d.k * d.ld;
    const float *u = d.urow[w];
    for (int j = lane; j < d.n; j += 32) ak[j] = u[j];
  }
}

// Addresses of the accepted walkers' matrices, inverses and new rows: one
// block, so that it can tell whether every index is in range before any
// inverse changes.  A negative index counts from the end.
// It stands for three gathers of pointer tables by index: 25 walkers of 39
// electrons, a call of Determinants.update 74 -> 30 us; 512 of 768 488 -> 463.
struct PickArgs {
  const int64_t *accepted;
  char *base[3];
  int64_t step[3], count[3];
  int64_t *out;  // [3][naccept], then the refusal
  int *status, mark;
  int naccept;
};
__global__ void __launch_bounds__(1024) k_det_pick(const PickArgs a) {
  bool bad = false;
  for (int i = threadIdx.x; i < a.naccept; i += blockDim.x) {
    const int64_t w = a.accepted[i];
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const int64_t v = w < 0 ? w + a.count[q] : w;
      bad |= v < 0 || v >= a.count[q];
      a.out[(int64_t)q * a.naccept + i] = (int64_t)(a.base[q] + v * a.step[q]);
    }
  }
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    a.out[3 * (int64_t)a.naccept] = bad;
    if (bad && a.status) {
      // an earlier owner's late refusal (a smaller mark) leaves this one's
      if (a.mark) atomicMax_system(a.status, a.mark);
      else *(volatile int *)a.status = 1;
      __threadfence_system();
    }
  }
}

}  // namespace eg

using namespace eg;

namespace {

int num_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    cudaGetLastError();
    return 152;
  }
  return n;
}

// The fused update's launch, by the matrix size.  Larger clusters keep fewer
// matrices in flight, so that a walker's rows are still in L2 when they are
// read again (measured: all of them up to 45 MB in flight, two thirds at
// 85 MB); smaller blocks and clusters spend less on each walker's
// exchange, which is what bounds small matrices.  us an update of about 1 GB
// of inverses (16000 walkers for n = 64, 0.26 GB), reference / transposed
// layout, the line's own shape in brackets, and the two passes:
//          1 x 128    2 x 128    2 x 256    8 x 128    8 x 256    8 x 512   passes
//   n 64  [125/144]   166/222    281/402                                   484/453
//    160   396/402   [318/412]   322/--                                    850/768
//    200    --/499    430/435   [357/480]   456/530                        965/850
//    256                         --         [378/400]              696/1035 877/710
//    384              561/560    508/570     446/456   [400/452]   528/669  913/643
//    512                         --          533/533    417/455   [413/448] 843/616
//    768                                                           [498/506] 1097/665
//   2048                                                           [517/515] 1260/557
// Beyond kUpMax a matrix no longer fits the vectors' registers.
struct UpdateShape {
  int cs, threads;
};
constexpr int kUpMax = 2048;
UpdateShape update_shape(int n) {
  if (n <= 100) return {1, 128};
  if (n <= 160) return {2, 128};
  if (n <= 240) return {2, 256};
  if (n <= 360) return {8, 128};
  if (n <= 500) return {8, 256};
  return {8, 512};
}

template <int THREADS>
const void *update_kernel(int trans) {
  return trans ? (const void *)k_det_update<1, THREADS> : (const void *)k_det_update<0, THREADS>;
}

cudaLaunchConfig_t cluster_config(int blocks, int cs, int threads, size_t smem, cudaStream_t s,
                                  cudaLaunchAttribute *at) {
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3((unsigned)blocks);
  lc.blockDim = dim3((unsigned)threads);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = (unsigned)cs;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  return lc;
}

// Clusters of a kernel that the current device holds at once (0: none, or
// the query failed), looked up once per kernel, shape and device.
int resident_clusters(const void *func, int cs, int threads, size_t smem) {
  struct Key {
    const void *f;
    int cs, threads, dev;
    size_t smem;
    bool operator<(const Key &o) const {
      return std::tie(f, cs, threads, dev, smem) < std::tie(o.f, o.cs, o.threads, o.dev, o.smem);
    }
  };
  static std::mutex mu;
  static std::map<Key, int> cache;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return 0; }
  const Key k{func, cs, threads, dev, smem};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(k);
  if (it != cache.end()) return it->second;
  int fit = 0;
  cudaLaunchAttribute at;
  const cudaLaunchConfig_t lc = cluster_config(cs, cs, threads, smem, nullptr, &at);
  if (allow_smem(func, smem)) return 0;
  if (cudaOccupancyMaxActiveClusters(&fit, func, &lc) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return cache[k] = fit;
}

int check_det_opts(const einspline_gb300_det_opts *o, const char *fn) {
  if (!o) return fail(EINSPLINE_GB300_EINVAL, "%s: NULL options", fn);
  if (o->nelec <= 0) return fail(EINSPLINE_GB300_EINVAL, "%s: nelec must be positive", fn);
  if (o->k < 0 || o->k >= o->nelec) return fail(EINSPLINE_GB300_EINVAL, "%s: k out of [0, nelec)", fn);
  if (o->ld < o->nelec) return fail(EINSPLINE_GB300_EINVAL, "%s: ld < nelec", fn);
  if (o->ainv_trans != 0 && o->ainv_trans != 1) return fail(EINSPLINE_GB300_EINVAL, "%s: ainv_trans must be 0 or 1", fn);
  if (o->rule != 0 && o->rule != 1) return fail(EINSPLINE_GB300_EINVAL, "%s: rule must be 0 or 1", fn);
  return 0;
}

template <int ST, bool GL>
cudaError_t launch_ratio_k(const DetArgs &d, unsigned grid, cudaStream_t s) {
  constexpr bool WIDE = ST != ST_F32;
  constexpr int RB = WIDE ? 16 : (int)sizeof(typename CT<ST>::Raw);
  const size_t sm = det_smem(d.e.pb, RB);
  const void *f = (const void *)k_det_ratio<ST, GL, WIDE>;
  if (allow_smem(f, sm)) return cudaErrorInvalidValue;
  k_det_ratio<ST, GL, WIDE><<<grid, kDetThreads, sm, s>>>(d);
  return cudaGetLastError();
}

template <int ST>
cudaError_t launch_ratio(const DetArgs &d, bool gl, unsigned grid, cudaStream_t s) {
  return gl ? launch_ratio_k<ST, true>(d, grid, s) : launch_ratio_k<ST, false>(d, grid, s);
}

template <int ST, bool GL>
cudaError_t launch_det_tc_k(const DetArgs &d, unsigned grid, cudaStream_t s) {
  const size_t sm = dt_smem(d.e.pb);
  const void *f = (const void *)k_det_tc<ST, GL>;
  if (allow_smem(f, sm)) return cudaErrorInvalidValue;
  k_det_tc<ST, GL><<<grid, kTcThreads, sm, s>>>(d);
  return cudaGetLastError();
}

template <int ST>
cudaError_t launch_det_tc(const DetArgs &d, bool gl, unsigned grid, cudaStream_t s) {
  return gl ? launch_det_tc_k<ST, true>(d, grid, s) : launch_det_tc_k<ST, false>(d, grid, s);
}

}  // namespace

extern "C" {

int einspline_gb300_det_ratio(einspline_gb300_table *t, const einspline_gb300_det_opts *o, int nwalkers,
                              const void *pos_d, const float *const *ainv_d, float *ratio_d, float *grad_d,
                              float *lapl_d, float *const *row_d, void *stream) {
  static const char *fn = "einspline_gb300_det_ratio";
  clear();
  if (!table3_ok(t)) return fail(EINSPLINE_GB300_EINVAL, "%s: bad table handle", fn);
  if (int r = check_det_opts(o, fn)) return r;
  if (t->ncomp != 1 || t->storage == ST_F64)
    return fail(EINSPLINE_GB300_EINVAL, "%s: real float tables only (s kind, any float/16-bit storage)", fn);
  if (o->nelec > t->num_splines) return fail(EINSPLINE_GB300_EINVAL, "%s: nelec exceeds the table's splines", fn);
  if (nwalkers < 0) return fail(EINSPLINE_GB300_EINVAL, "%s: nwalkers < 0", fn);
  if (nwalkers == 0) return 0;
  if (!pos_d || !ainv_d || !ratio_d) return fail(EINSPLINE_GB300_EINVAL, "%s: NULL buffer", fn);
  if (int r = table_flush(t)) return r;
  DetArgs d;
  memset(&d, 0, sizeof(d));
  fill_eval_geometry(t, d.e);
  d.e.pos = pos_d;
  d.e.pos_f64 = o->pos_f64 ? 1 : 0;
  d.e.rule = o->rule;
  d.e.npts = nwalkers;
  d.ainv = ainv_d;
  d.row_out = row_d;
  d.ratio = ratio_d;
  d.grad = grad_d;
  d.lapl = lapl_d;
  d.n = o->nelec;
  d.k = o->k;
  d.ld = o->ld;
  d.trans = o->ainv_trans;
  const bool gl = grad_d || lapl_d;
  cudaStream_t s = stream ? (cudaStream_t)stream : cudaStreamLegacy;
  if ((t->storage == ST_F16 || t->storage == ST_BF16) && pick_mode(t, true) == 5) {
    // tensor cores, as the table's vgh evaluation
    if (int r = tc_table_map(t, d.e)) return r;
    d.e.wait_err = t->wait_err_d;
    if (t->test_skip.load(std::memory_order_relaxed)) {
      d.e.test_skip = t->test_skip.exchange(0);
      d.e.wait_ns = t->test_wait_ns;
    }
    // Blocks of about kDtUnits tiles: long enough for the copies to run ahead
    // of a block's set-up, short enough for the last wave to end evenly;
    // beyond four waves of them, longer ones.  us
    // a ratio with gradient and laplacian, walkers spread over whole waves
    // of at most 7 a block (before) / this: N = 1024, 2048 walkers 99.4 / 95.6
    // (transposed inverse 49.5 / 47.6), 4096 walkers 186 / 179 (88.5 /
    // 85.1); N = 256, 4096 walkers 52 / 50 (26.8 / 24.7).  Bound by DRAM's
    // random reads: the stencils and, in the reference's layout, 128 bytes
    // for each inverse entry.
    const int tiles = (d.n + 127) / 128;
    const int64_t wave = kDtBlocksPerSM * (int64_t)num_sms();
    // Few walkers spread over the SMs, three blocks each, before blocks get
    // longer: N = 128, 4 to 48 walkers 8.8 / 4.4, 200 walkers 9.0 / 5.6.
    int64_t units = std::max(1, kDtUnits / tiles);
    if (nwalkers <= 2 * wave) units = std::min<int64_t>(units, (nwalkers + 3 * num_sms() - 1) / (3 * num_sms()));
    const int pb = (int)std::min<int64_t>(kDtMaxWalkers, std::max<int64_t>(units, nwalkers / (4 * wave)));
    d.e.pb = pb;
    const unsigned grid = (unsigned)((nwalkers + pb - 1) / pb);
    EG_CUDA(t->storage == ST_F16 ? launch_det_tc<ST_F16>(d, gl, grid, s) : launch_det_tc<ST_BF16>(d, gl, grid, s));
    count_launch();
    return 0;
  }
  // kDetBlocksPerSM blocks fit on an SM.  The walkers are spread evenly
  // over at most one wave of such blocks, so each block runs one long
  // pipeline over its walkers (no per-block fill and drain for every walker,
  // no partial last wave); beyond 32 walkers per block the grid grows
  // instead.
  const int slots = kDetBlocksPerSM * num_sms();
  int pb = (nwalkers + slots - 1) / slots;
  pb = pb < 1 ? 1 : (pb > 32 ? 32 : pb);
  d.e.pb = pb;
  const unsigned grid = (unsigned)((nwalkers + pb - 1) / pb);
  cudaError_t e;
  switch (t->storage) {
    case ST_F32: e = launch_ratio<ST_F32>(d, gl, grid, s); break;
    case ST_F16: e = launch_ratio<ST_F16>(d, gl, grid, s); break;
    case ST_BF16: e = launch_ratio<ST_BF16>(d, gl, grid, s); break;
    default: e = launch_ratio<ST_I16>(d, gl, grid, s); break;
  }
  EG_CUDA(e);
  count_launch();
  return 0;
}

static int update_walkers(const DetArgs &d, int naccept, cudaStream_t s) {
  if (d.n <= kUpMax) {
    const UpdateShape sh = update_shape(d.n);
    const void *f = sh.threads == 128 ? update_kernel<128>(d.trans)
                  : sh.threads == 256 ? update_kernel<256>(d.trans) : update_kernel<512>(d.trans);
    const size_t sm = up_smem(d.n, sh.cs, d.trans, sh.threads);
    const int fit = resident_clusters(f, sh.cs, sh.threads, sm);
    if (fit > 0) {
      const int clusters = std::min(naccept, fit);
      int lpr_log = 0;
      while (lpr_log < 5 && (1 << lpr_log) < (d.n + 3) / 4) lpr_log++;
      int cs = sh.cs;
      void *args[] = {const_cast<DetArgs *>(&d), &cs, &naccept, &lpr_log};
      cudaLaunchAttribute at;
      const cudaLaunchConfig_t lc = cluster_config(clusters * cs, cs, sh.threads, sm, s, &at);
      EG_CUDA(cudaLaunchKernelExC(&lc, f, args));
      count_launch();
      return 0;
    }
  }
  if (!d.trans) k_det_update1_rows<<<dim3((d.n + 255) / 256, naccept), 256, 0, s>>>(d);
  else k_det_update1_trans<<<dim3((d.n + 7) / 8, naccept), 256, 0, s>>>(d);
  EG_CUDA(cudaGetLastError());
  k_det_update2<<<dim3((d.n + 7) / 8, naccept), 256, 0, s>>>(d);
  EG_CUDA(cudaGetLastError());
  count_launch(2);
  return 0;
}

int einspline_gb300_det_update(const einspline_gb300_det_opts *o, int naccept, float *const *a_d,
                               float *const *ainv_d, const float *const *row_d, float *work_d, void *stream) {
  static const char *fn = "einspline_gb300_det_update";
  clear();
  if (int r = check_det_opts(o, fn)) return r;
  if (naccept < 0) return fail(EINSPLINE_GB300_EINVAL, "%s: naccept < 0", fn);
  if (naccept == 0) return 0;
  if (naccept > 65535) return fail(EINSPLINE_GB300_ESIZE, "%s: at most 65535 walkers per call", fn);
  if (!a_d || !ainv_d || !row_d || !work_d) return fail(EINSPLINE_GB300_EINVAL, "%s: NULL buffer", fn);
  DetArgs d;
  memset(&d, 0, sizeof(d));
  d.ainv = ainv_d;
  d.amat = a_d;
  d.urow = row_d;
  d.work = work_d;
  d.n = o->nelec;
  d.k = o->k;
  d.ld = o->ld;
  d.trans = o->ainv_trans;
  return update_walkers(d, naccept, stream ? (cudaStream_t)stream : cudaStreamLegacy);
}

static int update_accepted(const char *fn, const einspline_gb300_det_opts *o, int naccept, const int64_t *accepted_d,
                           const einspline_gb300_det_batch *b, float *work_d, int64_t *ptrs_d, int *status, int mark,
                           void *stream) {
  clear();
  if (int r = check_det_opts(o, fn)) return r;
  if (naccept < 0) return fail(EINSPLINE_GB300_EINVAL, "%s: naccept < 0", fn);
  if (naccept == 0) return 0;
  if (naccept > 65535) return fail(EINSPLINE_GB300_ESIZE, "%s: at most 65535 walkers per call", fn);
  if (!accepted_d || !b || !b->a || !b->ainv || !b->rows || !work_d || !ptrs_d)
    return fail(EINSPLINE_GB300_EINVAL, "%s: NULL buffer", fn);
  cudaStream_t s = stream ? (cudaStream_t)stream : cudaStreamLegacy;
  PickArgs p;
  p.accepted = accepted_d;
  p.base[0] = (char *)b->a; p.base[1] = (char *)b->ainv; p.base[2] = (char *)const_cast<float *>(b->rows);
  p.step[0] = b->a_step; p.step[1] = b->ainv_step; p.step[2] = b->row_step;
  p.count[0] = b->a_count; p.count[1] = b->ainv_count; p.count[2] = b->row_count;
  p.out = ptrs_d;
  p.status = status;
  p.mark = mark;
  p.naccept = naccept;
  k_det_pick<<<1, naccept >= 1024 ? 1024 : (naccept + 31) / 32 * 32, 0, s>>>(p);
  EG_CUDA(cudaGetLastError());
  count_launch();
  DetArgs d;
  memset(&d, 0, sizeof(d));
  d.amat = reinterpret_cast<float *const *>(ptrs_d);
  d.ainv = reinterpret_cast<const float *const *>(ptrs_d + naccept);
  d.urow = reinterpret_cast<const float *const *>(ptrs_d + 2 * (int64_t)naccept);
  d.refused = ptrs_d + 3 * (int64_t)naccept;
  d.work = work_d;
  d.n = o->nelec;
  d.k = o->k;
  d.ld = o->ld;
  d.trans = o->ainv_trans;
  return update_walkers(d, naccept, s);
}

int einspline_gb300_det_update_accepted(const einspline_gb300_det_opts *o, int naccept, const int64_t *accepted_d,
                                        const einspline_gb300_det_batch *b, float *work_d, int64_t *ptrs_d,
                                        int *status, void *stream) {
  return update_accepted("einspline_gb300_det_update_accepted", o, naccept, accepted_d, b, work_d, ptrs_d, status, 0,
                         stream);
}

int einspline_gb300_det_update_accepted_mark(const einspline_gb300_det_opts *o, int naccept, const int64_t *accepted_d,
                                             const einspline_gb300_det_batch *b, float *work_d, int64_t *ptrs_d,
                                             int *status, int mark, void *stream) {
  static const char *fn = "einspline_gb300_det_update_accepted_mark";
  clear();
  if (mark < 1) return fail(EINSPLINE_GB300_EINVAL, "%s: mark must be positive", fn);
  return update_accepted(fn, o, naccept, accepted_d, b, work_d, ptrs_d, status, mark, stream);
}

}  // extern "C"
