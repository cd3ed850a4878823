// sinkhorn_resident.cu -- a whole Sinkhorn solve, vanilla or log-stabilised,
// with or without its gradient, in one cooperative launch, for problems whose
// kernel matrix fits on the chip (up to 4096 rows and about 29 MB).
//
// Both methods run in scaling form on K = exp(-C/eps):
//   u_1 = a / (K 1),   v = b / (K^T u),   u = a / (K v)
// (Sinkhorn::_fwd_vanilla, src/sinkhorn_impl_vanilla.cpp:93-166; the log form's
// updates, src/sinkhorn_impl_log.cpp:327-375, are the same with f = eps log u,
// g = eps log v), with each method's own stopping error, and the plan, loss and
// marginals from C at the end.  Zero masses need no packing: their scalings are
// zero and drop out of every sum.  The solve is given up (status kResUnsafe,
// and the general drivers in sinkhorn_log.cu start again from scratch) when a
// mass is negative or not finite, when K has subnormal entries (log method), or
// when a sum or a scaling leaves the safe range.
//
// The gradient with respect to a (Sinkhorn::_bwd_vanilla :169-213, _bwd_log
// :379-520: one function, so one gradient) is unrolled in the same launch from
// the scalings of every iteration.  With pb = (C + eps log P) o P,
//   step L:  col = (pb^T 1) v / b,      ubar = (pb 1) / u - K col,
//   step l:  col = (K^T x) v_l^2 / b,   ubar = K col,
//   each:    grad_a += ubar u_l / a,    x = ubar u_l^2 / a.
// So every iteration, forward or backward, is the same sweep over K.
//
// What bounds it: at these sizes neither memory nor arithmetic but the latency
// of one iteration, two exchanges between CTAs plus the sweep's own barriers.
// The general path's two grid barriers (arrive, poll), the partials read after
// the first and the totals after the second took 13 us per iteration at every
// size up to 2048^2.  Here:
//   * each CTA keeps its strip of K in shared memory (its last two columns, if
//     need be, in registers);
//   * partial sums and totals travel as 16-byte packets (value, tag), written
//     and read by single 128-bit accesses: a reader polls the data itself, so
//     an exchange costs one trip through L2 instead of a fence, a counter and a
//     second trip.  A tag holds the launch's number and the round, so packets
//     need no reset; a round's packets are overwritten only after every reader
//     has sent what it computed from them;
//   * small problems use few CTAs, and each adds all partials itself (one
//     exchange per iteration); larger ones split the rows, one warp per row;
//   * the stopping test runs beside the next sweep's sums.
// Measured (B200, whole calls): see the table beside launch_resident.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "engine.h"
#include "sk_host.h"

namespace rwig {
namespace skres {

constexpr int NTT = 512, NW = NTT / 32;
constexpr int kMaxRows = 4096;
constexpr int kMaxG = 160;       // CTAs (five packets per lane of a merging warp)
constexpr int kRowsPerWarp = 2;  // merged rows per warp: M <= 32 G
constexpr int kRegCols = 2;      // columns of a strip that may live in registers
constexpr double kLo = 1e-250, kHi = 1e250;

struct alignas(16) Packet {
  unsigned long long v, tag;
};

struct Args {
  const double* a;
  const double* b;
  const double* C;  // M x N, leading dimension M
  double* P;        // optional
  double* f;        // optional: f / u
  double* g;        // optional: g / v
  double* grad;     // optional (with uh, vh)
  double* uh;       // u_l at uh[l M] (l = 1..L; redundant: a copy per CTA), gradient only
  double* vh;       // v_l at vh[l N]
  const double* info;  // masses_kernel: support sizes, bad masses
  int M, N, G, R, lds, ncmax, nsm;
  int vanilla, redundant, max_iter;
  double eps, tol;
  Packet* part;  // redundant: [2][G][M] by the tag's parity; split: [merger][G][R]
  Packet* up;    // [M]
  Packet* cer;   // [2][G]
  Packet* fin;   // [G][6]
  unsigned long long epoch;  // launch number << 32
  double* res;               // host-mapped results (kRes*)
  unsigned* err;
};

__device__ __forceinline__ void put(Packet* p, double v, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ bool get(const Packet* p, unsigned long long tag, double& v) {
  unsigned long long x, t;
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(x), "=l"(t)
               : "l"(p)
               : "memory");
  v = __longlong_as_double((long long)x);
  return t == tag;
}

// Polls NP packets at(k), k < n, until all carry the tag; bounded (2 s, or an
// error elsewhere).
template <int NP, class At>
__device__ __forceinline__ bool poll(int n, At at, unsigned long long tag, double (&v)[NP], unsigned* err) {
  unsigned pend = 0;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    v[k] = 0.0;
    if (k < n) pend |= 1u << k;
  }
  unsigned long long t0 = 0;
  for (unsigned spin = 1; pend; ++spin) {
#pragma unroll
    for (int k = 0; k < NP; ++k)
      if (pend >> k & 1u) {
        double x;
        if (get(at(k), tag, x)) {
          v[k] = x;
          pend &= ~(1u << k);
        }
      }
    if ((spin & 255u) == 0u) {
      if (*(volatile unsigned*)err != 0u) return false;
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > kWaitLimitNs) {
        atomicOr(err, KERR_BARRIER_TIMEOUT);
        return false;
      }
    }
  }
  return true;
}

// Partial sums of 8 NQ columns from c0 over row pairs [p0, p1): 8 column lanes
// x 4 row lanes, NQ columns per lane, so that one load of u serves NQ of K (a
// broadcast 16-byte load takes the shared-memory pipe as long as a full one).
template <int NQ>
__device__ __forceinline__ void sum_block(const double* K, int lds, int nc, int c0, int p0, int p1, const double* su,
                                          double* out) {
  const int lane = threadIdx.x & 31, cl = lane & 7, rl = lane >> 3;
  const double* col[NQ];
  double x[NQ], y[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    const int c = c0 + 8 * q + cl;
    col[q] = K + (size_t)(c < nc ? c : 0) * lds;
    x[q] = y[q] = 0.0;
  }
#pragma unroll 4
  for (int p = p0 + rl; p < p1; p += 4) {
    const double2 uu = *reinterpret_cast<const double2*>(su + 2 * p);
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const double2 kk = *reinterpret_cast<const double2*>(col[q] + 2 * p);
      x[q] = fma(kk.x, uu.x, x[q]);
      y[q] = fma(kk.y, uu.y, y[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    double t = x[q] + y[q];
    t += __shfl_xor_sync(0xffffffffu, t, 8);
    t += __shfl_xor_sync(0xffffffffu, t, 16);
    const int c = c0 + 8 * q + cl;
    if (rl == 0 && c < nc) out[c] = t;
  }
}

// Column sums of the strip's nc shared columns with su: the 16 warps form
// blocks of 32 columns and row chunks; red[chunk * ld + c].  Returns the chunks.
__device__ __forceinline__ int sum_columns(const double* K, int lds, int M, int nc, int ld, const double* su, double* red) {
  const int w = threadIdx.x >> 5;
  const int nblk = (nc + 31) >> 5;
  const int lg = nblk > 8 ? 4 : nblk > 4 ? 3 : nblk > 2 ? 2 : nblk > 1 ? 1 : 0;
  const int nrc = NW >> lg, rc = w & (nrc - 1);
  const int pairs = (M + 1) >> 1;
  const int p0 = rc * pairs / nrc, p1 = (rc + 1) * pairs / nrc;
  for (int blk = w >> (4 - lg); blk < nblk; blk += 1 << lg) {
    const int c0 = 32 * blk, nq = (min(32, nc - c0) + 7) >> 3;
    double* out = red + rc * ld;
    if (nq == 4) sum_block<4>(K, lds, nc, c0, p0, p1, su, out);
    else if (nq == 3) sum_block<3>(K, lds, nc, c0, p0, p1, su, out);
    else if (nq == 2) sum_block<2>(K, lds, nc, c0, p0, p1, su, out);
    else sum_block<1>(K, lds, nc, c0, p0, p1, su, out);
  }
  return nrc;
}

// Shared memory (doubles): strip [nsm][lds], su [lds], red, vs, vn, cb [ncmax]
// each, es [4][NW], with the gradient red2 [NW][ncmax].
__host__ __device__ constexpr int red_doubles(int ncmax) { return NW * ncmax > 1024 ? NW * ncmax : 1024; }
__host__ __device__ constexpr size_t smem_doubles(int lds, int nsm, int ncmax, bool grad) {
  return (size_t)nsm * lds + lds + red_doubles(ncmax) + 3 * (size_t)ncmax + 4 * NW + (grad ? NW * (size_t)ncmax : 0);
}

// Host-mapped results.
constexpr double kResRunning = 0.0, kResFinished = 1.0, kResUnsafe = 2.0;
enum { kResIter = 0, kResErr, kResStatus, kResLoss, kResL1Row, kResL1Col, kResL2Row, kResL2Col, kResSupM, kResSupN,
       kResKerr, kResGradNs, kResWords };

// RPT rows per thread: 2 up to 1024 rows, 4 up to 2048, 8 up to 4096.  Row sets
// of a thread: pairs 2 (lt + tg k) of the sweep's second half, and (polling u,
// building K, the final pass) rows tid + 512 j.
template <int RPT, bool GRAD>
__global__ void __launch_bounds__(NTT, 1) resident_kernel(Args p) {
  extern __shared__ __align__(128) double sm[];
  constexpr int KP = RPT / 2;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, cta = blockIdx.x;
  const int M = p.M, N = p.N, G = p.G, lds = p.lds;
  const double eps = p.eps, inv_eps = 1.0 / p.eps;
  const int c0 = (int)(((long long)cta * N) / G), ncols = (int)(((long long)(cta + 1) * N) / G) - c0;
  const int nc = min(ncols, p.nsm), nreg = ncols - nc;  // columns in shared memory, in registers
  const int ld = p.ncmax;
  double* const K = sm;
  double* const su = K + (size_t)p.nsm * lds;
  double* const red = su + lds;
  double* const vs = red + red_doubles(ld);  // v of the last completed sweep
  double* const vn = vs + ld;                // factors of the running sweep's second half
  double* const cb = vn + ld;                // b
  double* const es = cb + ld;                // [4][NW]
  double* const red2 = es + 4 * NW;          // GRAD
  double* const uh = GRAD ? p.uh + (p.redundant ? (size_t)cta * (p.max_iter + 2) * M : 0) : nullptr;

  if (p.info[2] != 0.0) {  // a mass the scaling form does not take, or no support
    if (cta == 0 && tid == 0) p.res[kResStatus] = kResUnsafe;
    return;
  }
  // second half: column groups for few rows
  const int ncg = RPT > 2 ? 1 : M <= 64 ? 16 : M <= 128 ? 8 : M <= 256 ? 4 : M <= 512 ? 2 : 1;
  const int tg = NTT / ncg, cg = tid / tg, r0 = 2 * (tid - cg * tg);
  int nk = 0;
#pragma unroll
  for (int k = 0; k < KP; ++k) nk += r0 + 2 * NTT * k < M;

  // ---- K, b and the row sums of K over the support
  double ra[RPT], uo[RPT], un[RPT];  // a, current and next u of rows tid + 512 j
  double kr[kRegCols][RPT];          // register columns, this thread's pairs
  bool bad = false;
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int i = tid + j * NTT;
    ra[j] = i < M ? p.a[i] : 0.0;
    uo[j] = un[j] = 0.0;
  }
  for (int c = tid; c < ncols; c += NTT) cb[c] = p.b[c0 + c];
  auto kernel_entry = [&](double c) {
    const double x = exp(-c / eps);
    if (!p.vanilla && !(x >= 2.2250738585072014e-308 && x <= 1.79e308)) bad = true;
    return x;
  };
#pragma unroll 2
  for (int c = 0; c < nc; ++c) {
    const double* Cc = p.C + (size_t)(c0 + c) * M;
    double* Kc = K + (size_t)c * lds;
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int i = tid + j * NTT;
      if (i < M) Kc[i] = kernel_entry(Cc[i]);
    }
  }
  for (int c = tid; c < nc; c += NTT)
    for (int i = M; i < lds; ++i) K[(size_t)c * lds + i] = 0.0;
#pragma unroll
  for (int q = 0; q < kRegCols; ++q)
#pragma unroll
    for (int t = 0; t < RPT; ++t) {
      const int i = r0 + 2 * NTT * (t >> 1) + (t & 1);
      kr[q][t] = q < nreg && i < M ? kernel_entry(p.C[(size_t)(c0 + nc + q) * M + i]) : 0.0;
    }
  for (int i = M + tid; i < lds; i += NTT) su[i] = 0.0;
  __syncthreads();
  for (int c = tid; c < ncols; c += NTT) vn[c] = cb[c] != 0.0 ? 1.0 : 0.0;
  __syncthreads();

  // ---------------------------------------------------------------- exchange
  int row_q[RPT];  // split: packet of row r0.. in its merger's block
  if (!p.redundant) {
#pragma unroll
    for (int t = 0; t < RPT; ++t) {
      const int i = ncg > 1 ? tid : r0 + 2 * NTT * (t >> 1) + (t & 1);
      row_q[t] = i < M ? (i / p.R * G + cta) * p.R + i % p.R : 0;
    }
  }
  // A tag's partials.  Redundant merges keep two rounds: a CTA may send the next
  // round's while another still reads this one's (of the round after that it
  // may not: it needs that other's next partials first).  Split merges keep
  // one: a CTA sends only after it has every row's total, and so after every
  // merger has read its partials.
  auto part_at = [&](unsigned long long t) { return p.part + (p.redundant && (t & 1) ? (size_t)G * M : 0); };
  auto cer_at = [&](unsigned long long t) { return p.cer + (t & 1) * G; };
  // The sweep's second half, r = K vn over this thread's pairs, sent as this
  // CTA's partials of the round; extra[t] is added for the pairs (ncg = 1) or
  // for row tid (ncg > 1, extra[0]).
  auto send_rows = [&](unsigned long long tag, const double* extra) {
    double r[RPT];
#pragma unroll
    for (int t = 0; t < RPT; ++t) r[t] = 0.0;
    const double* col = K + (size_t)cg * lds + r0;
    const int step = ncg * lds;
    if (nk == KP) {
#pragma unroll 4
      for (int c = cg; c < nc; c += ncg, col += step) {
        const double v = vn[c];
#pragma unroll
        for (int k = 0; k < KP; ++k) {
          const double2 kk = *reinterpret_cast<const double2*>(col + 2 * NTT * k);
          r[2 * k] = fma(kk.x, v, r[2 * k]);
          r[2 * k + 1] = fma(kk.y, v, r[2 * k + 1]);
        }
      }
    } else {
      for (int c = cg; c < nc; c += ncg, col += step) {
        const double v = vn[c];
#pragma unroll
        for (int k = 0; k < KP - 1; ++k)
          if (k < nk) {
            const double2 kk = *reinterpret_cast<const double2*>(col + 2 * NTT * k);
            r[2 * k] = fma(kk.x, v, r[2 * k]);
            r[2 * k + 1] = fma(kk.y, v, r[2 * k + 1]);
          }
      }
    }
    if (cg == 0)
#pragma unroll
      for (int q = 0; q < kRegCols; ++q)
        if (q < nreg)
#pragma unroll
          for (int t = 0; t < RPT; ++t) r[t] = fma(kr[q][t], vn[nc + q], r[t]);
    if (ncg > 1) {  // the groups' sums in group order, then one row per thread
      __syncthreads();
      if (r0 < M) red[cg * M + r0] = r[0];
      if (r0 + 1 < M) red[cg * M + r0 + 1] = r[1];
      __syncthreads();
      if (tid < M) {
        double s = 0.0;
        for (int q = 0; q < ncg; ++q) s += red[q * M + tid];
        if (extra) s = extra[0] - s;
        put(p.redundant ? part_at(tag) + (size_t)cta * M + tid : p.part + row_q[0], s, tag);
      }
    } else {
#pragma unroll
      for (int t = 0; t < RPT; ++t) {
        const int i = r0 + 2 * NTT * (t >> 1) + (t & 1);
        if (i < M) put(p.redundant ? part_at(tag) + (size_t)cta * M + i : p.part + row_q[t], extra ? extra[t] - r[t] : r[t], tag);
      }
    }
  };
  // Totals of the round's partials -> x_i = fn(i, j, total) for rows tid + 512 j
  // into `out` (every CTA gets all rows).  fn runs once per row and CTA
  // (redundant; j: its index here) or once per row on its merger (j = -1, slot
  // = the merger's row of this warp).
  const int q0 = cta * p.R, q1 = min(M, q0 + p.R);  // split: this CTA's rows
  auto totals = [&](unsigned long long tag, double (&out)[RPT], auto fn) -> bool {
    bool ok = true;
    if (p.redundant) {
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        const int i = tid + j * NTT;
        if (i >= M) continue;
        double acc = 0.0;
        for (int k = 0; k < G && ok; k += 8) {
          double x[8];
          ok = poll<8>(min(8, G - k), [&](int e) { return part_at(tag) + (size_t)(k + e) * M + i; }, tag, x, p.err);
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (k + e < G) acc += x[e];
        }
        out[j] = fn(i, j, acc);
      }
      return ok;
    }
#pragma unroll
    for (int s = 0; s < kRowsPerWarp; ++s) {
      const int i = q0 + w + NW * s;
      if (i < q1) {  // warp-uniform
        constexpr int NP = kMaxG / 32;
        double x[NP];
        const Packet* base = p.part + (size_t)cta * G * p.R + (i - q0);
        const int n = (G - lane + 31) >> 5;
        ok = poll<NP>(n, [&](int e) { return base + (size_t)(lane + 32 * e) * p.R; }, tag, x, p.err) && ok;
        double t = 0.0;
#pragma unroll
        for (int e = 0; e < NP; ++e) t += x[e];
        t = warp_sum(t);
        if (lane == 0) put(p.up + i, fn(i, -1 - s, t), tag);
      }
    }
    double x[RPT];
    const int n = tid < M ? (M - tid + NTT - 1) / NTT : 0;
    ok = poll<RPT>(n, [&](int j) { return p.up + tid + j * NTT; }, tag, x, p.err) && ok;
#pragma unroll
    for (int j = 0; j < RPT; ++j) out[j] = x[j];
    return ok;
  };
  auto store_su = [&](const double (&x)[RPT]) {
#pragma unroll
    for (int j = 0; j < RPT; ++j)
      if (tid + j * NTT < M) su[tid + j * NTT] = x[j];
  };
  // Column sums of the whole strip with su: red[chunk * ld + c], chunks returned
  // (register columns: NW warps' partials).
  auto sums = [&]() {
    const int n = sum_columns(K, lds, M, nc, ld, su, red);
    if (nreg > 0) {
      double u[RPT];
#pragma unroll
      for (int t = 0; t < RPT; ++t) {
        const int i = r0 + 2 * NTT * (t >> 1) + (t & 1);
        u[t] = i < M ? su[i] : 0.0;
      }
#pragma unroll
      for (int q = 0; q < kRegCols; ++q)
        if (q < nreg) {
          double x = 0.0;
#pragma unroll
          for (int t = 0; t < RPT; ++t) x = fma(kr[q][t], u[t], x);
          x = warp_sum(cg == 0 ? x : 0.0);
          if (lane == 0) red[w * ld + nc + q] = x;
        }
    }
    return n;
  };
  auto col_total = [&](int c, int n) {
    double x[NW];
    const int m = c < nc ? n : NW;
#pragma unroll
    for (int q = 0; q < NW; ++q) x[q] = q < m ? red[q * ld + c] : 0.0;
#pragma unroll
    for (int h = NW / 2; h >= 1; h >>= 1)
#pragma unroll
      for (int q = 0; q < h; ++q) x[q] += x[q + h];
    return x[0];
  };
  auto sum_es = [&](int k) {
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < NW; ++q) t += es[k * NW + q];
    return t;
  };
  auto in_range = [](double x) { return x >= kLo && x <= kHi; };
  // u_{l} = a / total
  double ga[RPT];        // gradient (redundant: rows tid + 512 j; split: [s] the merger's rows, lane 0)
#pragma unroll
  for (int j = 0; j < RPT; ++j) ga[j] = 0.0;
  auto next_u = [&](int l) {
    return [&, l](int i, int j, double t) {
      const double a = j >= 0 ? ra[j >= 0 ? j : 0] : p.a[i];
      // a total outside the safe range ends the solve (its u is checked by every CTA)
      const double u = a == 0.0 ? 0.0 : in_range(t) ? a / t : INFINITY;
      if (GRAD) uh[(size_t)l * M + i] = u;
      return u;
    };
  };
  // ---------------------------------------------------------------- forward
  unsigned long long tag = p.epoch + 1;
  {
    const double nb = __syncthreads_or(bad) ? INFINITY : 0.0;
    if (tid == 0) put(cer_at(tag) + cta, nb, tag);
  }
  send_rows(tag, nullptr);
  int iter = 0;
  double status = kResRunning;
  double err = 1000.0;
  bool ok = true;
  while (true) {
    // u of the next iteration, and (beside its sums) the error of the last one
    ok = totals(tag, un, next_u(iter + 1));
    store_su(un);
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    const int n = sums();
    {
      double e = 0.0;
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        if (tid + j * NTT >= M || ra[j] == 0.0) continue;
        if (!in_range(un[j])) e = INFINITY;
        else if (iter > 0) {
          const double q = uo[j] / un[j];  // u_i (K v)_i / a_i
          const double d = p.vanilla ? ra[j] * (q - 1.0) : log(q);
          e = fma(d, d, e);
        }
      }
      e = warp_sum(e);
      if (lane == 0) es[w] = e;
      if (w == NW - 1) {
        double x[kMaxG / 32], t = 0.0;
        ok = poll<kMaxG / 32>((G - lane + 31) >> 5, [&](int k) { return cer_at(tag) + lane + 32 * k; }, tag, x, p.err);
#pragma unroll
        for (int k = 0; k < kMaxG / 32; ++k) t += x[k];
        t = warp_sum(t);
        if (lane == 0) es[NW] = t;
      }
    }
    if (__syncthreads_or(!ok)) {
      ok = false;
      break;
    }
    const double er = sum_es(0), ec = es[NW];
    if (!(er + ec <= 1e300)) {
      status = kResUnsafe;
      break;
    }
    if (iter > 0) {
      err = sqrt(er) + sqrt(ec);
      if (!(iter < p.max_iter && err >= p.tol)) break;
    }
    ++iter;
    ++tag;
    // v = b / (K^T u)
    double e = 0.0;
    for (int c = tid; c < ncols; c += NTT) {
      const double b = cb[c], s = col_total(c, n);
      const double v = b / s;
      vn[c] = b == 0.0 ? 0.0 : v;
      vs[c] = vn[c];
      if (GRAD) p.vh[(size_t)iter * N + c0 + c] = vn[c];
      if (b != 0.0) {
        const double d = p.vanilla ? fma(v, s, -b) : fma(v, s, -b) / b;  // log(v s / b) to first order
        e = in_range(s) && in_range(v) ? fma(d, d, e) : INFINITY;
      }
    }
    e = warp_sum(e);
    if (lane == 0) es[2 * NW + w] = e;
#pragma unroll
    for (int j = 0; j < RPT; ++j) uo[j] = un[j];
    __syncthreads();
    if (tid == 0) put(cer_at(tag) + cta, sum_es(2), tag);
    send_rows(tag, nullptr);
  }
  if (!ok || status == kResUnsafe) {
    if (cta == 0 && tid == 0) {
      p.res[kResKerr] = ok ? 0.0 : 1.0;
      p.res[kResStatus] = kResUnsafe;
    }
    return;
  }

  // ---------------------------------------------------------------- plan, loss, marginals
  ++tag;
  double f[RPT], pr[RPT], rp[RPT];  // f, row sums of P and of pb, rows tid + 512 j
  double l1 = 0.0, l2 = 0.0, cl1 = 0.0, cl2 = 0.0;
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int i = tid + j * NTT;
    f[j] = eps * log(uo[j]);
    pr[j] = rp[j] = 0.0;
    if (cta == 0 && i < M && p.f) p.f[i] = p.vanilla ? uo[j] : f[j];
  }
  __syncthreads();  // vn, red are free
  for (int c = tid; c < ncols; c += NTT) {
    const double gj = eps * log(vs[c]);
    vn[c] = gj;
    if (p.g) p.g[c0 + c] = p.vanilla ? vs[c] : gj;
  }
  __syncthreads();
  bool zero_plan = false;
  for (int cc = 0; cc < ncols; cc += 4) {
    double cs[4], cp[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      cs[q] = cp[q] = 0.0;
      const int c = cc + q;
      if (c >= ncols) continue;
      const bool live = cb[c] != 0.0;
      const double gj = vn[c];
      const double* Cc = p.C + (size_t)(c0 + c) * M;
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        const int i = tid + j * NTT;
        if (i >= M) continue;
        double pv = 0.0;
        if (live && ra[j] != 0.0) {
          const double cij = Cc[i];
          pv = exp(-((cij - f[j]) - gj) * inv_eps);
          const double lp = log(pv);
          l1 += cij * pv;
          l2 += pv * (lp - 1.0);
          pr[j] += pv;
          cs[q] += pv;
          if (GRAD) {
            const double pb = (cij + eps * lp) * pv;
            rp[j] += pb;
            cp[q] += pb;
            zero_plan |= !(pv > 0.0);
          }
        }
        if (p.P) p.P[(size_t)(c0 + c) * M + i] = pv;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (cc + q >= ncols) continue;
      double t = warp_sum(cs[q]);
      if (lane == 0) red[w * ld + cc + q] = t;
      if (GRAD) {
        t = warp_sum(cp[q]);
        if (lane == 0) red2[w * ld + cc + q] = t;
      }
    }
  }
  __syncthreads();
  for (int c = tid; c < ncols; c += NTT) {
    double t = 0.0;
    for (int q = 0; q < NW; ++q) t += red[q * ld + c];
    if (cb[c] != 0.0) {
      cl1 += fabs(t - cb[c]);
      cl2 += (t - cb[c]) * (t - cb[c]);
    }
    if (GRAD) {  // col of step L
      t = 0.0;
      for (int q = 0; q < NW; ++q) t += red2[q * ld + c];
      vn[c] = cb[c] != 0.0 ? t * vs[c] / cb[c] : 0.0;
    }
  }
  // row sums of P to their mergers (redundant: to CTA 0)
#pragma unroll
  for (int j = 0; j < RPT; ++j) {
    const int i = tid + j * NTT;
    if (i < M) put(part_at(tag) + (p.redundant ? (size_t)cta * M + i : (size_t)(i / p.R * G + cta) * p.R + i % p.R), pr[j], tag);
  }
  double a1 = 0.0, a2 = 0.0;
  auto row_marginal = [&](int i, double t) {
    const double a = p.a[i];
    if (a != 0.0) {
      a1 += fabs(t - a);
      a2 += (t - a) * (t - a);
    }
  };
  if (p.redundant) {
    if (cta == 0)
#pragma unroll
      for (int j = 0; j < RPT; ++j) {
        const int i = tid + j * NTT;
        if (i >= M) continue;
        double acc = 0.0;
        for (int k = 0; k < G && ok; ++k) {
          double x[1];
          ok = poll<1>(1, [&](int) { return part_at(tag) + (size_t)k * M + i; }, tag, x, p.err);
          acc += x[0];
        }
        row_marginal(i, acc);
      }
  } else {
#pragma unroll
    for (int s = 0; s < kRowsPerWarp; ++s) {
      const int i = q0 + w + NW * s;
      if (i < q1) {
        constexpr int NP = kMaxG / 32;
        double x[NP], t = 0.0;
        const Packet* base = p.part + (size_t)cta * G * p.R + (i - q0);
        ok = poll<NP>((G - lane + 31) >> 5, [&](int e) { return base + (size_t)(lane + 32 * e) * p.R; }, tag, x, p.err) && ok;
#pragma unroll
        for (int e = 0; e < NP; ++e) t += x[e];
        t = warp_sum(t);
        if (lane == 0) row_marginal(i, t);
      }
    }
  }
  // block sums of the six scalars, sent to CTA 0
  {
    double v[6] = {l1, l2, cl1, cl2, a1, a2};
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const double x = warp_sum(v[t]);
      if (lane == 0) red[t * NW + w] = x;
    }
    const bool zp = __syncthreads_or(zero_plan);
    if (tid < 6) {
      double t = 0.0;
      for (int q = 0; q < NW; ++q) t += red[tid * NW + q];
      put(p.fin + cta * 6 + tid, t, tag);
    }
    if (GRAD && tid == 0) put(cer_at(tag) + cta, zp ? INFINITY : 0.0, tag);  // (its row marginals are merged)
  }
  if (cta == 0) {
    if (w < 6) {
      double x[kMaxG / 32], t = 0.0;
      ok = poll<kMaxG / 32>((G - lane + 31) >> 5, [&](int k) { return p.fin + (lane + 32 * k) * 6 + w; }, tag, x, p.err) && ok;
#pragma unroll
      for (int k = 0; k < kMaxG / 32; ++k) t += x[k];
      t = warp_sum(t);
      if (lane == 0) es[w] = t;
    }
    ok = !__syncthreads_or(!ok);
    if (tid == 0) {
      p.res[kResIter] = iter;
      p.res[kResErr] = err;
      p.res[kResLoss] = es[0] + eps * es[1];
      p.res[kResL1Row] = es[4];
      p.res[kResL1Col] = es[2];
      p.res[kResL2Row] = sqrt(es[5]);
      p.res[kResL2Col] = sqrt(es[3]);
      p.res[kResSupM] = p.info[0];
      p.res[kResSupN] = p.info[1];
      p.res[kResGradNs] = 0.0;
      p.res[kResKerr] = ok ? 0.0 : 1.0;
      if (!GRAD || !ok) p.res[kResStatus] = ok ? kResFinished : kResUnsafe;
    }
  }
  if constexpr (GRAD) {
    // -------------------------------------------------------------- backward
    const unsigned long long t_b = globaltimer_ns();
    // a plan entry that underflowed: the reference's sums turn NaN or infinite
    // there, which the general path reproduces
    if (w == 0) {
      double x[kMaxG / 32], t = 0.0;
      ok = poll<kMaxG / 32>((G - lane + 31) >> 5, [&](int k) { return cer_at(tag) + lane + 32 * k; }, tag, x, p.err) && ok;
#pragma unroll
      for (int k = 0; k < kMaxG / 32; ++k) t += x[k];
      t = warp_sum(t);
      if (lane == 0) es[3 * NW] = t;
    }
    ok = !__syncthreads_or(!ok);
    if (!ok || !(es[3 * NW] <= 1e300)) {
      if (cta == 0 && tid == 0) {
        p.res[kResKerr] = ok ? 0.0 : 1.0;
        p.res[kResStatus] = kResUnsafe;
      }
      return;
    }
    // step L: this CTA's share of (pb 1) / u rides along
#pragma unroll
    for (int j = 0; j < RPT; ++j) {
      const int i = tid + j * NTT;
      if (i < M) su[i] = ra[j] != 0.0 ? rp[j] / uo[j] : 0.0;
    }
    __syncthreads();
    double ex[RPT];
#pragma unroll
    for (int t = 0; t < RPT; ++t) {
      const int i = ncg > 1 ? tid : r0 + 2 * NTT * (t >> 1) + (t & 1);
      ex[t] = i < M ? su[i] : 0.0;
    }
    ++tag;
    send_rows(tag, ex);
    double x[RPT];
    for (int l = iter;; --l) {
      // x = ubar u_l^2 / a, grad += ubar u_l / a
      ok = totals(tag, x, [&](int i, int j, double t) {
        const double a = j >= 0 ? ra[j >= 0 ? j : 0] : p.a[i];
        if (a == 0.0) return 0.0;
        const double u = uh[(size_t)l * M + i];  // written by this thread
        const double q = t * u / a;
        if (j >= 0) ga[j >= 0 ? j : 0] += q;
        else ga[j < 0 ? -1 - j : 0] += q;
        return q * u;
      });
      if (l == 1) {
        ok = !__syncthreads_or(!ok);
        break;
      }
      store_su(x);
      double vl = 0.0;
      if (tid < ncols) vl = __ldcg(p.vh + (size_t)(l - 1) * N + c0 + tid);
      if (__syncthreads_or(!ok)) {
        ok = false;
        break;
      }
      const int n = sums();
      __syncthreads();
      for (int c = tid; c < ncols; c += NTT) {
        const double v = c < NTT ? vl : __ldcg(p.vh + (size_t)(l - 1) * N + c0 + c);
        vn[c] = cb[c] != 0.0 ? col_total(c, n) * (v * v) / cb[c] : 0.0;
      }
      __syncthreads();
      ++tag;
      send_rows(tag, nullptr);
    }
    if (p.redundant) {
      if (cta == 0)
#pragma unroll
        for (int j = 0; j < RPT; ++j)
          if (tid + j * NTT < M) p.grad[tid + j * NTT] = ga[j];
    } else {
#pragma unroll
      for (int s = 0; s < kRowsPerWarp; ++s) {
        const int i = q0 + w + NW * s;
        if (i < q1 && lane == 0) p.grad[i] = ga[s];
      }
    }
    if (cta == 0 && tid == 0) {
      p.res[kResGradNs] = (double)(globaltimer_ns() - t_b);
      p.res[kResKerr] = ok ? 0.0 : 1.0;
      p.res[kResStatus] = ok ? kResFinished : kResUnsafe;
    }
  }
}

// Support sizes (non-zero masses) and whether a mass is one the scaling form
// does not take (negative or not finite) or a side has none; clears *err.
__global__ void __launch_bounds__(NTT) masses_kernel(const double* a, const double* b, int M, int N, double* info,
                                                     unsigned* err) {
  __shared__ int cnt[2];
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  int ca = 0, cbn = 0, bad = 0;
  for (int i = threadIdx.x; i < M; i += NTT) {
    const double x = a[i];
    ca += x != 0.0;
    bad |= !(x >= 0.0 && x <= 1e300);
  }
  for (int j = threadIdx.x; j < N; j += NTT) {
    const double x = b[j];
    cbn += x != 0.0;
    bad |= !(x >= 0.0 && x <= 1e300);
  }
  if (ca) atomicAdd(cnt, ca);
  if (cbn) atomicAdd(cnt + 1, cbn);
  bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    info[0] = cnt[0];
    info[1] = cnt[1];
    info[2] = bad || cnt[0] == 0 || cnt[1] == 0 ? 1.0 : 0.0;
    *err = 0u;
  }
}

// Leading dimension of a shared strip: ldk / 2 odd, so that the 16-byte loads
// of eight neighbouring columns hit all banks.
int strip_ld(int M) {
  const int e = (M + 1) & ~1;
  return (e >> 1) & 1 ? e : e + 2;
}

struct Shape {
  int G, R, lds, ncmax, nsm, redundant;
  size_t smem;
};

// The launch of an M x N problem; false when it does not fit.
//
// G: 8192 elements (64 KB) of K per CTA, up to every SM: below that a sweep
// takes about 1 us, no longer than the exchange that more CTAs would lengthen.
// Redundant merges while a CTA adds at most 4096 partials (8 per thread).
bool shape(const Context* ctx, int M, int N, bool grad, Shape* s) {
  if (M > kMaxRows || ctx->sm_count > kMaxG) return false;
  const int gmax = std::min(N, ctx->sm_count);
  const long long el = (long long)M * N;
  int G = (int)std::min<long long>(gmax, std::max<long long>(1, (el + 8191) / 8192));
  s->lds = strip_ld(M);
  for (; G <= gmax; ++G) {
    s->ncmax = (N + G - 1) / G;
    const size_t fixed = smem_doubles(s->lds, 0, s->ncmax, grad) * 8;
    if (fixed >= (size_t)ctx->smem_optin) continue;
    const int room = (int)(((size_t)ctx->smem_optin - fixed) / (8 * (size_t)s->lds));
    s->nsm = std::min(s->ncmax, room);
    if (s->nsm < 1 || s->ncmax - s->nsm > kRegCols) continue;
    s->R = (M + G - 1) / G;
    s->redundant = (long long)G * M <= 4096;
    if (!s->redundant && s->R > NW * kRowsPerWarp) {  // more rows than a merger's warps take
      if (M <= NW * kRowsPerWarp * gmax || (long long)G * M > 65536) continue;
      s->redundant = 1;
    }
    s->G = G;
    s->smem = smem_doubles(s->lds, s->nsm, s->ncmax, grad) * 8;
    return true;
  }
  return false;
}

template <int RPT, bool GRAD>
int launch(Args& p, const Shape& s, cudaStream_t st) {
  auto kern = resident_kernel<RPT, GRAD>;
  static size_t attr = 0;  // callers hold the context lock
  if (attr < s.smem) {
    RWIG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem));
    attr = s.smem;
  }
  void* args[] = {&p};
  RWIG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)kern, dim3(s.G), dim3(NTT), args, s.smem, st));
  return 0;
}

enum { SRS_PACKETS = 250, SRS_INFO, SRS_UH, SRS_VH };

}  // namespace skres

int sinkhorn_resident(Context* ctx, cudaStream_t st, bool vanilla, double* P, double* grad_a, double* f, double* g,
                      double* loss, int* iter, double* err, const double* a, const double* b, const double* C, int M,
                      int N, double reg, int max_iter, double zero_tol, int* status_out) {
  using namespace skres;
  const bool grad = grad_a != nullptr;
  Shape s;
  if (max_iter < 1 || !(zero_tol <= 999.0) || !shape(ctx, M, N, grad, &s)) return 0;
  const size_t L2 = (size_t)max_iter + 2;
  const size_t hist = grad ? 8 * L2 * ((size_t)M * (s.redundant ? s.G : 1) + N) : 0;
  if (hist > (size_t(32) << 30)) return 0;
  if (!ctx->resident_res) {
    void* h = nullptr;
    RWIG_CUDA_TRY(cudaHostAlloc(&h, sizeof(double) * kResWords, cudaHostAllocMapped));
    ctx->resident_res = (double*)h;
  }
  double* dres = nullptr;
  RWIG_CUDA_TRY(cudaHostGetDevicePointer((void**)&dres, ctx->resident_res, 0));
  const size_t npart = s.redundant ? 2 * (size_t)s.G * M : (size_t)s.G * s.G * s.R;
  const size_t bytes = sizeof(Packet) * (npart + M + 8 * (size_t)s.G);
  const bool fresh = (int)ctx->slots.size() <= SRS_PACKETS || ctx->slot_bytes[SRS_PACKETS] < bytes;
  Packet* pk = (Packet*)scratch(ctx, SRS_PACKETS, bytes);
  double* info = (double*)scratch(ctx, SRS_INFO, sizeof(double) * 4);
  double* uh = grad ? (double*)scratch(ctx, SRS_UH, 8 * L2 * M * (s.redundant ? s.G : 1)) : nullptr;
  double* vh = grad ? (double*)scratch(ctx, SRS_VH, 8 * L2 * N) : nullptr;
  if (!pk || !info || (grad && (!uh || !vh))) return RWIG_E_NOMEM;
  if (fresh)  // no packet of an earlier life of this memory may carry a tag to come
    RWIG_CUDA_TRY(cudaMemsetAsync(pk, 0, ctx->slot_bytes[SRS_PACKETS], st));
  Args p{};
  p.a = a;
  p.b = b;
  p.C = C;
  p.P = P;
  p.f = f;
  p.g = g;
  p.grad = grad_a;
  p.uh = uh;
  p.vh = vh;
  p.info = info;
  p.M = M;
  p.N = N;
  p.G = s.G;
  p.R = s.R;
  p.lds = s.lds;
  p.ncmax = s.ncmax;
  p.nsm = s.nsm;
  p.vanilla = vanilla;
  p.redundant = s.redundant;
  p.max_iter = max_iter;
  p.eps = reg;
  p.tol = zero_tol;
  p.part = pk;
  p.up = pk + npart;
  p.cer = p.up + M;
  p.fin = p.cer + 2 * s.G;
  p.epoch = ++ctx->resident_epoch << 32;
  p.res = dres;
  p.err = (unsigned*)(info + 3);
  double* res = ctx->resident_res;
  res[kResStatus] = kResRunning;
  res[kResKerr] = 0.0;
  RWIG_CUDA_TRY(cudaEventRecord(ctx->ev0, st));
  masses_kernel<<<1, NTT, 0, st>>>(a, b, M, N, info, p.err);
  int rc;
  if (grad) rc = M <= 1024 ? launch<2, true>(p, s, st) : M <= 2048 ? launch<4, true>(p, s, st) : launch<8, true>(p, s, st);
  else rc = M <= 1024 ? launch<2, false>(p, s, st) : M <= 2048 ? launch<4, false>(p, s, st) : launch<8, false>(p, s, st);
  if (rc) return rc;
  RWIG_CUDA_TRY(cudaEventRecord(ctx->ev1, st));
  RWIG_CUDA_TRY(cudaEventSynchronize(ctx->ev1));
  if (res[kResKerr] != 0.0) return set_error(RWIG_E_TIMEOUT, "Sinkhorn kernel stopped by a bounded wait");
  if (res[kResStatus] != kResFinished) return 0;  // not in the scaling form's range
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  const int it = (int)res[kResIter];
  const double e = res[kResErr];
  if (loss) *loss = res[kResLoss];
  if (iter) *iter = it;
  if (err) *err = e;
  *status_out = (e <= zero_tol) ? 0 : (it == max_iter ? 1 : 2);
  rwig_report& R = report();
  R.iter = it;
  R.status = *status_out;
  R.err = e;
  R.marg_l1_row = res[kResL1Row];
  R.marg_l1_col = res[kResL1Col];
  R.marg_l2_row = res[kResL2Row];
  R.marg_l2_col = res[kResL2Col];
  R.device_ms = ms;
  R.kernel_ms = ms;
  R.grad_ms = res[kResGradNs] * 1e-6;
  R.sweep_ms = ms - R.grad_ms;
  R.sweep_iters = it;
  R.kernel_launches = 2;
  R.support_m = (int)res[kResSupM];
  R.support_n = (int)res[kResSupN];
  return 1;
}

}  // namespace rwig
