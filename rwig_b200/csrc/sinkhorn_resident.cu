// sinkhorn_resident.cu -- a whole Sinkhorn solve, vanilla or log-stabilised,
// with or without its gradient, in one cooperative launch, for problems whose
// kernel matrix fits on the chip (about 4 million elements).
//
// Both methods run in scaling form on K = exp(-C/eps):
//   u_1 = a / (K 1),   v = b / (K^T u),   u = a / (K v)
// (Sinkhorn::_fwd_vanilla, src/sinkhorn_impl_vanilla.cpp:93-166; the log form's
// updates, src/sinkhorn_impl_log.cpp:327-375, are the same with f = eps log u,
// g = eps log v), with each method's own stopping error, and the plan, loss and
// marginals from C at the end.  Zero masses need no packing: their scalings are
// zero and drop out of every sum.  The solve is given up (status kResUnsafe,
// and the general drivers in sinkhorn_log.cu start again from scratch) when a
// mass is negative or not finite, when K has subnormal entries (log method),
// when a sum or a scaling leaves the safe range or, with a gradient, when a plan
// entry underflows or the gradient is not finite.  K and the first u are judged
// within the first iteration: 20 log iterations that are given up there take 485
// us at 701 x 513, 470 in the general drivers alone.  A scaling that leaves the
// range later (only with max C / eps above 575) costs the iterations up to there.
//
// The gradient with respect to a (Sinkhorn::_bwd_vanilla :169-213, _bwd_log
// :379-520: one function, so one gradient) is unrolled in the same launch from
// the scalings of every iteration.  With pb = (C + eps log P) o P,
//   step L:  col = (pb^T 1) v / b,      ubar = (pb 1) / u - K col,
//   step l:  col = (K^T x) v_l^2 / b,   ubar = K col,
//   each:    grad_a += ubar u_l / a,    x = ubar u_l^2 / a.
// So every iteration, forward or backward, is the same two passes over K.
//
// What bounds it: at these sizes neither memory nor arithmetic but the latency
// of one iteration.  With column strips, two grid barriers (arrive, poll),
// partials read after the first and totals after the second, an iteration took
// 13 us at every size up to 2048^2.  Here:
//   * K is cut into gr x gc blocks, one per CTA, kept in shared memory (a few
//     columns in registers when a block is a little too large).  A CTA needs u
//     of its block's rows and v of its columns only, and the partial sums of a
//     pass go to the CTAs of one block row or column: 270 numbers per CTA at
//     1777 x 1501 where a column strip sends and receives 1777 each;
//   * every CTA of a block row (column) adds that row's (column's) partials
//     itself, in the same order, so totals need no second trip;
//   * partials travel as 16-byte packets (value, tag), written and read by
//     single 128-bit accesses: a reader polls the data itself, one trip through
//     L2 instead of a fence, a counter and a second trip.  A tag holds the
//     launch's number and the round, so packets need no reset;
//   * 15 warps iterate; the last one only forms, exchanges and judges the
//     stopping error, two iterations behind (what was computed since is thrown
//     away when it stops);
//   * a gradient's scalings are stored once, by the first CTA of each block row
//     and column, and read back from L2 behind one fence.
// Whole solves through the C entry against the general drivers (us): 256 x 256
// vanilla, 19 iterations 134 (430); 1777 x 1501 log, 31 iterations 324 (723);
// with gradient 701 x 513 vanilla, 11 iterations 192 (482); 2048 x 2048 log,
// 100 iterations 1929 (5332), 9.3 us per iteration in each direction: of about
// 17500 clocks the two passes take 6600, the exchanges 4000-5000 each.
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "engine.h"
#include "resident_words.h"
#include "sk_host.h"

namespace rwig {
namespace skres {

constexpr int NW = 15, NTT = 32 * NW;  // the iterating warps
constexpr int kThreads = NTT + 32;     // and the error warp
constexpr int kMaxSide = NTT;          // rows and columns of a block: one of each per thread
constexpr int kMaxG = 160;     // CTAs (five error packets per lane)
constexpr int kPoll = 6;       // packets a thread loads at once
constexpr int kRegCols = 4;    // REG: columns in registers per column group of the row pass

// Barriers: 1 of the iterating warps; 2 and 3 hand su, suo, sd to the error
// warp and its verdict back.
__device__ __forceinline__ void sync() { asm volatile("bar.sync 1, 480;" ::: "memory"); }
__device__ __forceinline__ bool sync_or(bool x) {
  int r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.or.pred q, 1, 480, p;\n\tselp.s32 %0, 1, 0, "
      "q;\n\t}"
      : "=r"(r)
      : "r"((int)x)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void errors_in() { asm volatile("bar.arrive 2, 512;" ::: "memory"); }
__device__ __forceinline__ void errors_wait() { asm volatile("bar.sync 2, 512;" ::: "memory"); }
__device__ __forceinline__ void verdict_out() { asm volatile("bar.arrive 3, 512;" ::: "memory"); }
__device__ __forceinline__ void verdict_wait() { asm volatile("bar.sync 3, 512;" ::: "memory"); }
static_assert(kThreads == 512 && NTT == 480, "thread counts of the barriers");

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
  double* grad;     // gradient: M
  double* uh;       // gradient: u_l at [l][M], stored by the first CTA of each block row
  double* vh;       // gradient: v_l at [l][N], stored by the first CTA of each block column
  const double* info;  // masses_kernel: support sizes, bad masses
  int M, N, gr, gc, lds, vanilla, ldn, nsm, chunks, max_iter;
  double eps, tol;
  // packets, two exchanges of each kind by the tag's parity: a CTA may send the
  // next one's while a peer still reads this one's, but not the one after that,
  // for which it needs that peer's part in the next one first
  Packet* cpart;  // [2][gr][N] column partials
  Packet* rpart;  // [2][gc][M] row partials
  Packet* epart;  // [4][G][2]  error shares: rows, columns (four: read one iteration after they are sent)
  Packet* fin;    // [G][6]
  unsigned long long epoch;  // launch number << 32
  double* res;               // host-mapped results (kRes*)
  unsigned* err;
};

__device__ __forceinline__ void put(Packet* p, double v, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(v)), "l"(tag)
               : "memory");
}
__device__ __forceinline__ void get(const Packet* p, unsigned long long& v, unsigned long long& tag) {
  asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
               : "=l"(v), "=l"(tag)
               : "l"(p)
               : "memory");
}

// 8 bytes to shared memory, no register held meanwhile; the thread waits for its own.
__device__ __forceinline__ void copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Polls NP packets at(k), k < n, until all carry the tag (n <= 0: none);
// bounded (2 s, or an error elsewhere).  All loads of a try are issued before
// the first is looked at: a test after each load would cost a round trip to L2
// per packet (7000-10000 clocks for a dozen, against 2000).
template <int NP, class At>
__device__ __forceinline__ bool poll(int n, At at, unsigned long long tag, double (&v)[NP], unsigned* err) {
#pragma unroll
  for (int k = 0; k < NP; ++k) v[k] = 0.0;
  if (n <= 0) return true;
  unsigned long long t0 = 0;
  for (unsigned spin = 1;; ++spin) {
    unsigned long long x[NP], t[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) get(at(k < n ? k : n - 1), x[k], t[k]);
    bool all = true;
#pragma unroll
    for (int k = 0; k < NP; ++k) all = all && t[k] == tag;
    if (all) {
#pragma unroll
      for (int k = 0; k < NP; ++k) v[k] = k < n ? __longlong_as_double((long long)x[k]) : 0.0;
      return true;
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

// Shared memory (doubles): block [nsm][lds], su, suo, sa [lds], sv, sd, sb
// [ldn], colp [chunks][ldn], rowp [1024], es [8].
__host__ __device__ constexpr size_t smem_doubles(int lds, int ldn, int nsm, int chunks) {
  return (size_t)nsm * lds + 3 * (size_t)lds + 3 * (size_t)ldn + (size_t)chunks * ldn + 1024 + 6 * NW + 8;
}

// REG: the last kRegCols columns per column group of the row pass are held in
// registers (nsm of the block's columns in shared memory).
template <bool GRAD, bool REG>
__global__ void __launch_bounds__(kThreads, 1) resident_kernel(Args p) {
  extern __shared__ __align__(128) double sm[];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, cta = blockIdx.x;
  const int M = p.M, N = p.N, gr = p.gr, gc = p.gc, G = gr * gc, lds = p.lds, ldn = p.ldn;
  const int ri = cta / gc, ci = cta - ri * gc;
  const double eps = p.eps, inv_eps = 1.0 / p.eps;
  const int m0 = (int)((long long)ri * M / gr), mr = (int)((long long)(ri + 1) * M / gr) - m0;
  const int n0 = (int)((long long)ci * N / gc), nr = (int)((long long)(ci + 1) * N / gc) - n0;
  const int ns = REG ? min(nr, p.nsm) : nr;  // columns in shared memory
  double* const K = sm;
  double* const su = K + (size_t)p.nsm * lds;
  double* const suo = su + lds;  // u of the iteration before
  double* const sa = suo + lds;
  double* const sv = sa + lds;   // v, or the factors of the row pass
  double* const sd = sv + ldn;   // columns' error terms
  double* const sb = sd + ldn;
  double* const colp = sb + ldn;
  double* const rowp = colp + (size_t)p.chunks * ldn;
  double* const es = rowp + 1024;

  if (cta == 0 && tid == 0) {
    p.res[kResSupM] = p.info[0];
    p.res[kResSupN] = p.info[1];
  }
  if (p.info[2] != 0.0) {  // a mass the scaling form does not take, or no support
    if (cta == 0 && tid == 0) p.res[kResStatus] = kResUnsafe;
    return;
  }
  // row pass: nrw warps cover the rows' pairs, ngrp groups of them the columns
  const int nrw = (mr + 63) >> 6, ngrp = NW / nrw;
  const int rw = w % nrw, grp = w / nrw;
  const bool in_pass = grp < ngrp;
  const int r0 = 64 * rw + 2 * lane;  // first row of this thread's pair
  const bool row_ok = in_pass && r0 < mr;
  double2 kr[REG ? kRegCols : 1];     // its register columns ns + grp kRegCols + q
  const double a_i = tid < mr ? p.a[m0 + tid] : 0.0;
  const double b_j = tid < nr ? p.b[n0 + tid] : 0.0;
  const double rb_j = b_j != 0.0 ? 1.0 / b_j : 0.0;
  if (tid < mr) sa[tid] = a_i;
  if (tid < nr) sb[tid] = b_j;
  for (int i = mr + tid; i < lds; i += NTT) su[i] = 0.0;
  for (int c = tid; c < ns; c += NTT)
    for (int i = mr; i < lds; ++i) K[(size_t)c * lds + i] = 0.0;
  bool bad = false, ok = true;
  // tags: the launch and the number of the exchange, counted for each kind apart
  unsigned long long ct = p.epoch, rt = p.epoch;

  // fn(C_ij, i, j) for the block's elements in shared memory, spread over the
  // threads, four loads at a time
  auto each = [&](auto fn) {
    const int dc = NTT / mr, di = NTT - dc * mr;
    int c = tid / mr, i = tid - c * mr;
    const double* const Cb = p.C + (size_t)n0 * M + m0;
    while (c < ns && !bad) {  // (what a thread that found K out of range leaves out is not used)
      double x[4];
      int cc[4], ii[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        cc[k] = c;
        ii[k] = i;
        x[k] = c < ns ? Cb[(size_t)c * M + i] : 0.0;
        c += dc;
        i += di;
        if (i >= mr) {
          i -= mr;
          ++c;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (cc[k] < ns) fn(x[k], ii[k], cc[k]);
    }
  };
  // What stands in the block's place: K = exp(-C/eps) (kind 0), the plan P (1),
  // or pb = (C + eps log P) o P (2); su, sd hold f, g for the latter two.
  double l1 = 0.0, l2 = 0.0;
  bool zero_plan = false;
  auto fill = [&](int kind) {
    auto entry = [&](double c, int i, int j) {
      if (kind == 0) {
        const double x = exp(-c / eps);
        if (!p.vanilla && !(x >= 2.2250738585072014e-308 && x <= 1.79e308)) bad = true;
        if (GRAD) zero_plan |= x < 1e-250;
        return x;
      }
      if (sa[i] == 0.0 || sb[j] == 0.0) return 0.0;
      const double x = -((c - su[i]) - sd[j]) * inv_eps;
      const double pv = exp(x);
      // log P: x itself, from which the logarithm of the rounded P differs by
      // less than one unit of the last place of 1; minus infinity where P underflowed
      const double lp = pv > 0.0 ? x : -INFINITY;
      if (kind == 2) return (c + eps * lp) * pv;
      l1 += c * pv;
      l2 += pv * (lp - 1.0);
      zero_plan |= !(pv > 0.0);
      return pv;
    };
    double* const Pb = kind == 1 && p.P ? p.P + (size_t)n0 * M + m0 : nullptr;
    each([&](double cij, int i, int c) {
      const double x = entry(cij, i, c);
      K[(size_t)c * lds + i] = x;
      if (Pb) Pb[(size_t)c * M + i] = x;
    });
    if constexpr (REG) {
      const double* const Cb = p.C + (size_t)n0 * M + m0;
#pragma unroll
      for (int q = 0; q < kRegCols; ++q) {
        const int c = ns + grp * kRegCols + q;
        const size_t at = (size_t)c * M + r0;
        const bool in = row_ok && c < nr, in1 = in && r0 + 1 < mr;
        kr[q].x = in ? entry(Cb[at], r0, c) : 0.0;
        kr[q].y = in1 ? entry(Cb[at + 1], r0 + 1, c) : 0.0;
        if (Pb && in) Pb[at] = kr[q].x;
        if (Pb && in1) Pb[at + 1] = kr[q].y;
      }
    }
  };
  // Row pass: partial sums over the block's columns of K sv -> rowp[grp][mr].
  auto row_pass = [&]() {
    double x = 0.0, y = 0.0;
    if (row_ok) {
      const double* col = K + (size_t)grp * lds + r0;
      const int step = ngrp * lds;
#pragma unroll 8
      for (int c = grp; c < ns; c += ngrp, col += step) {
        const double2 kk = *reinterpret_cast<const double2*>(col);
        const double v = sv[c];
        x = fma(kk.x, v, x);
        y = fma(kk.y, v, y);
      }
      if constexpr (REG) {
#pragma unroll
        for (int q = 0; q < kRegCols; ++q) {
          const int c = ns + grp * kRegCols + q;
          const double v = c < nr ? sv[c] : 0.0;
          x = fma(kr[q].x, v, x);
          y = fma(kr[q].y, v, y);
        }
      }
      rowp[grp * mr + r0] = x;
      if (r0 + 1 < mr) rowp[grp * mr + r0 + 1] = y;
    }
    sync();
  };
  // Sends this thread's partial t (mine: it has one) as sender `me` of n and adds
  // all n in order.  Whole warps; packets of sender e at base + e ld + tid.
  auto exchange = [&](Packet* base, int ld, int n, int me, bool mine, double t, unsigned long long tag) {
    Packet* const q = base + tid;
    if (mine) put(q + (size_t)me * ld, t, tag);
    t = 0.0;
    if (mine)
      for (int k = 0; k < n && ok; k += kPoll) {
        double x[kPoll];
        ok = poll<kPoll>(min(kPoll, n - k), [&](int e) { return q + (size_t)(k + e) * ld; }, tag, x, p.err);
#pragma unroll
        for (int e = 0; e < kPoll; ++e) t += x[e];
      }
    return t;
  };
  // The rows' totals over the block row (thread tid < mr: row m0 + tid): this
  // CTA's partial (rest: `extra` minus it) sent and all gc added in order.
  auto row_total = [&](bool rest, double extra) {
    double t = 0.0;
    const unsigned long long tag = ++rt;
    if (tid < mr) {
      for (int q = 0; q < ngrp; ++q) t += rowp[q * mr + tid];
      if (rest) t = extra - t;
    }
    if (gc > 1 && 32 * w < mr) t = exchange(p.rpart + (tag & 1) * (size_t)gc * M + m0, M, gc, ci, tid < mr, t, tag);
    return t;
  };
  // Column pass: partial sums over the block's rows of K^T su -> colp[chunk][ldn];
  // returns the chunks (register columns: nrw).
  const int nblk = (p.nsm + 31) >> 5;  // (the same in every CTA: it sizes colp)
  const int nrc = NW / nblk;           // row chunks: nblk x nrc warps
  const int blk = w / nrc, chunk = w - blk * nrc;
  const int pairs = (mr + 1) >> 1;
  const int p0 = chunk * pairs / nrc, p1 = (chunk + 1) * pairs / nrc;
  auto col_pass = [&]() {
    const int c0 = 32 * blk;
    double* out = colp + chunk * ldn;
    if (c0 + 16 < ns) sum_block<4>(K, lds, ns, c0, p0, p1, su, out);
    else if (c0 < ns) sum_block<2>(K, lds, ns, c0, p0, p1, su, out);
    if constexpr (REG) {
      const double u0 = row_ok ? su[r0] : 0.0, u1 = row_ok ? su[r0 + 1] : 0.0;
#pragma unroll
      for (int q = 0; q < kRegCols; ++q) {
        const double x = warp_sum(fma(kr[q].x, u0, kr[q].y * u1));
        const int c = ns + grp * kRegCols + q;
        if (lane == 0 && in_pass && c < nr) colp[rw * ldn + c] = x;
      }
    }
    sync();
  };
  // The columns' totals over the block column (thread tid < nr: column n0 + tid).
  auto col_total = [&]() {
    double t = 0.0;
    const unsigned long long tag = ++ct;
    if (tid < nr) {
      const int n = REG && tid >= ns ? nrw : nrc;
      for (int q = 0; q < n; ++q) t += colp[q * ldn + tid];
    }
    if (gr > 1 && 32 * w < nr) t = exchange(p.cpart + (tag & 1) * (size_t)gr * N + n0, N, gr, ri, tid < nr, t, tag);
    return t;
  };
  auto in_range = [](double x) { return x >= kLo && x <= kHi; };
  double* const uh = GRAD ? p.uh + m0 : nullptr;
  double* const vh = GRAD ? p.vh + n0 : nullptr;
  // Packets of exchange e: each CTA's shares of the row and the column error.
  auto error_at = [&](unsigned long long e) { return p.epart + (e & 3) * 2 * G; };

  // ---------------------------------------------------------------- error warp
  if (w == NW) {
    // Gradient: whether an entry of the plan u_i K_ij v_j of its block is below half
    // of the smallest subnormal number.  A plan with such an entry has no finite
    // gradient and the call is the general drivers' (which repeat the reference's
    // NaN).  The plan itself is the test that counts, but finding it there costs the
    // whole forward: 1270 us of the general drivers became 1617 at 701 x 513, 50
    // iterations; found after two iterations, on blocks with entries of K below
    // 1e-250, 1293.
    auto underflows = [&]() {
      auto ex = [](double x) { return __double2hiint(x) >> 20; };  // (biased)
      int low = 0;
      for (int i = lane; i < mr; i += 32) {
        const int eu = su[i] != 0.0 ? ex(su[i]) - 3 * 1023 : 0x10000;
#pragma unroll 8
        for (int c = 0; c < ns; ++c) {
          const double x = K[(size_t)c * lds + i];
          const int ev = ex(sv[c]);
          low = min(low, eu + (x != 0.0 ? ex(x) : -1076 + 1023) + (ev ? ev : 0x10000));
        }
      }
      return __any_sync(0xffffffffu, low < -1077);
    };
    // this CTA's share: rows and columns of its block's row and column
    const int ea = ci * mr / gc, eb = (ci + 1) * mr / gc, ec0 = ri * nr / gr, ec1 = (ri + 1) * nr / gr;
    for (int k = 1;; ++k) {  // loop k: u_k is in su, u_{k-1} in suo, the terms of v_{k-1} in sd
      errors_wait();
      if (es[2] != 0.0) return;
      const unsigned long long now = p.epoch + k, from = k == 1 ? now : now - 1;
      double e = 0.0, ec = 0.0;
      for (int i = ea + lane; i < eb; i += 32) {
        const double a = sa[i], x = su[i];
        if (a == 0.0) continue;
        if (!in_range(x)) e = INFINITY;
        else if (k > 1) {
          const double q = suo[i] / x;  // u_i (K v)_i / a_i
          const double d = p.vanilla ? a * (q - 1.0) : log(q);
          e = fma(d, d, e);
        }
      }
      for (int c = ec0 + lane; c < ec1; c += 32) ec += sd[c];
      e = warp_sum(e);
      ec = warp_sum(ec);
      if (k == 1 && es[3] != 0.0) e = INFINITY;  // K has subnormal entries
      if (GRAD && k == 3 && es[4] != 0.0 && underflows()) e = INFINITY;  // (of u_3, v_2)
      if (lane < 2) put(error_at(now) + 2 * cta + lane, lane ? ec : e, now);
      double verdict = 0.0, er = 0.0;
      // loop 1 waits for its own exchange (the checks of K and of the first u, so
      // that a problem out of range leaves early), loop k > 2 judges iteration k - 2
      if (k != 2) {
        constexpr int NP = 2 * kMaxG / 32;
        double x[NP], t[2] = {0.0, 0.0};
        const int n = (G - lane + 31) >> 5;
        const bool ok = poll<NP>(2 * n, [&](int q) { return error_at(from) + 2 * (lane + 32 * (q >> 1)) + (q & 1); }, from, x, p.err);
#pragma unroll
        for (int q = 0; q < NP; ++q) t[q & 1] += x[q];
        const double e0 = warp_sum(t[0]), e1 = warp_sum(t[1]);
        er = sqrt(e0) + sqrt(e1);
        verdict = __any_sync(0xffffffffu, !ok) ? 3.0 : !(e0 + e1 <= 1e300) ? 2.0
                  : k > 2 && !(k - 2 < p.max_iter && er >= p.tol) ? 1.0 : 0.0;
      }
      if (lane == 0) {
        es[0] = er;
        es[1] = verdict;
      }
      __syncwarp();
      verdict_out();
      if (verdict != 0.0) return;
    }
  }

  // ---------------------------------------------------------------- iterating warps
  // One loop runs every stage of the solve, so that the passes and exchanges
  // are in the code once (inlined per stage, the loop outgrew the instruction
  // cache: 16000 clocks for an exchange of the backward steps).
  enum { kInit, kForward, kMargins, kMargins2, kBackward0, kBackward };
  int stage = kInit, kind = 0;
  int k = 0, l = 0, iter = 0;
  double err = 0.0;
  double u = 0.0, u1 = 0.0, u2 = 0.0, v = 0.0, v1 = 0.0, v2 = 0.0;  // of this and the last two iterations
  double s = 0.0, t = 0.0;      // column and row totals
  double fi = 0.0, ex = 0.0, ga = 0.0, ul = 0.0, vl = 0.0;
  unsigned long long et = 0, t_b = 0;
  while (true) {
    if (kind >= 0) {  // (synchronised before)
      fill(kind);
      const bool any = sync_or(bad);
      if (stage == kInit) {
        const bool look = GRAD && sync_or(zero_plan);
        zero_plan = false;
        if (tid < nr) {
          sv[tid] = b_j != 0.0 ? 1.0 : 0.0;  // K 1 over the support
          sd[tid] = 0.0;
        }
        if (tid == 0) {
          es[1] = es[2] = 0.0;
          es[3] = any ? 1.0 : 0.0;
          es[4] = look ? 1.0 : 0.0;
        }
      } else if (stage == kBackward0) {
        if (tid < nr) sv[tid] = b_j != 0.0 ? s * v * rb_j : 0.0;
      } else {
        if (tid < mr) su[tid] = 1.0;
        if (tid < nr) sv[tid] = 1.0;
      }
      kind = -1;
      sync();
    }
    if (stage != kInit && stage != kBackward0) {
      col_pass();
      s = col_total();
    }
    if (stage == kForward) {
      v2 = v1;
      v1 = v;
      v = b_j == 0.0 ? 0.0 : b_j / s;
      verdict_wait();  // (and everyone is done with sv and sd)
      if (es[1] != 0.0) {
        // iteration k - 2 is the last: its potentials, then the plan
        iter = k - 2;
        err = es[0];
        u = u2;
        v = v2;
        fi = eps * log(u);
        const double gj = eps * log(v);
        if (es[1] != 1.0) break;
        // the histories, stored by one CTA of each block row and column, are out
        // before this thread's next packets, which the same thread of every
        // other CTA there waits for (in kMargins) before it reads them
        if (GRAD) __threadfence();
        sync();
        if (tid < mr) {
          su[tid] = fi;
          if (ci == 0 && p.f) p.f[m0 + tid] = p.vanilla ? u : fi;
        }
        if (tid < nr) {
          sd[tid] = gj;
          if (ri == 0 && p.g) p.g[n0 + tid] = p.vanilla ? v : gj;
        }
        et = p.epoch + k + 1;
        stage = kMargins;
        kind = 1;
        sync();
        continue;
      }
      if (tid < nr) {
        sv[tid] = v;
        const double d = p.vanilla ? fma(v, s, -b_j) : fma(v, s, -b_j) * rb_j;  // log(v s / b) to first order
        sd[tid] = b_j == 0.0 ? 0.0 : in_range(s) && in_range(v) ? d * d : INFINITY;
        if (GRAD && ri == 0) vh[(size_t)k * N + tid] = v;
      }
    } else if (GRAD && stage == kBackward) {
      // one factor at a time: v_l^2 alone overflows from 1e154 on, v_l (K^T x)_j is
      // of the size of the gradient's terms
      if constexpr (REG) copies_wait();
      if (tid < nr) {
        if constexpr (REG) vl = sd[tid];
        sv[tid] = s * vl * rb_j * vl;
      }
    }
    if (sync_or(!ok)) {
      ok = false;
      break;
    }
    row_pass();
    t = row_total(GRAD && stage == kBackward0, ex);

    if (stage <= kForward) {  // iteration k: u_k from the totals of K v_{k-1}
      stage = kForward;
      ++k;
      u2 = u1;
      u1 = u;
      u = a_i == 0.0 ? 0.0 : in_range(t) ? a_i / t : INFINITY;  // (an infinite u fails the error warp's check)
      if (tid < mr) {
        suo[tid] = u1;
        su[tid] = u;
        if (GRAD && ci == 0) uh[(size_t)k * M + tid] = u;
      }
      if (sync_or(!ok)) {
        ok = false;
        break;
      }
      errors_in();
    } else if (stage == kMargins) {
      // loss and marginals to CTA 0
      const bool ra = ci == 0 && tid < mr && a_i != 0.0, cb = ri == 0 && tid < nr && b_j != 0.0;
      const double dr = ra ? t - a_i : 0.0, dc = cb ? s - b_j : 0.0;
      const double t6[6] = {l1, l2, fabs(dc), dc * dc, fabs(dr), dr * dr};
      sync();
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const double x = warp_sum(t6[q]);
        if (lane == 0) rowp[q * NW + w] = x;
      }
      const bool zp = sync_or(zero_plan);
      if (tid < 6) {
        double x = 0.0;
        for (int q = 0; q < NW; ++q) x += rowp[tid * NW + q];
        put(p.fin + cta * 6 + tid, x, p.epoch);
      }
      if (GRAD && tid == 0) put(error_at(et) + 2 * cta, zp ? INFINITY : 0.0, et);
      if (cta == 0) {
        if (w < 6) {
          double x[kMaxG / 32], y = 0.0;
          ok = poll<kMaxG / 32>((G - lane + 31) >> 5, [&](int q) { return p.fin + (lane + 32 * q) * 6 + w; }, p.epoch, x, p.err) && ok;
#pragma unroll
          for (int q = 0; q < kMaxG / 32; ++q) y += x[q];
          y = warp_sum(y);
          if (lane == 0) es[2 + w] = y;
        }
        sync();
        if (tid == 0) {
          p.res[kResIter] = iter;
          p.res[kResErr] = err;
          p.res[kResLoss] = es[2] + eps * es[3];
          p.res[kResL1Row] = es[6];
          p.res[kResL1Col] = es[4];
          p.res[kResL2Row] = sqrt(es[7]);
          p.res[kResL2Col] = sqrt(es[5]);
          p.res[kResGradNs] = 0.0;
        }
      }
      if (!GRAD) break;
      __threadfence();  // (after the packets of the CTAs that stored the histories)
      t_b = globaltimer_ns();
      // a plan entry that underflowed: the reference's sums turn NaN or infinite
      // there, which the general path reproduces
      if (w == 0) {
        double x[kMaxG / 32], y = 0.0;
        ok = poll<kMaxG / 32>((G - lane + 31) >> 5, [&](int q) { return error_at(et) + 2 * (lane + 32 * q); }, et, x, p.err) && ok;
#pragma unroll
        for (int q = 0; q < kMaxG / 32; ++q) y += x[q];
        y = warp_sum(y);
        if (lane == 0) es[1] = y <= 1e300 ? 1.0 : 2.0;
      }
      if (tid < mr) su[tid] = fi;
      stage = kMargins2;
      kind = 2;
      if (sync_or(!ok)) {
        ok = false;
        break;
      }
      if (es[1] != 1.0) break;
    } else if (stage == kMargins2) {
      // (pb 1) / u: the whole row total, so one CTA of the block row brings it in
      ex = ci == 0 && a_i != 0.0 ? t / u : 0.0;
      stage = kBackward0;
      kind = 0;
      l = iter;
      if constexpr (!REG) ul = u;
      else if (tid < mr) suo[tid] = u;
      sync();
    } else {  // step l: x = ubar u_l^2 / a, grad += ubar u_l / a
      if constexpr (REG) ul = tid < mr ? suo[tid] : 0.0;
      const double q = a_i != 0.0 ? t * ul / a_i : 0.0;
      ga += q;
      --l;
      if (l == 0) break;
      if (tid < mr) su[tid] = q * ul;
      // u_l and v_l from L2 (plain loads of lines that other CTAs share cost 0.8% of a
      // call), into registers or, where columns of K take those, into suo and sd, which
      // are free by now: 2048 x 2048, 100 iterations, takes 1944 us on the device so and
      // 1973 with registers; 701 x 513, which has registers left, 181-197 us a call with
      // them and 201-204 without
      if constexpr (REG) {
        if (tid < mr) copy8(suo + tid, uh + (size_t)l * M + tid);
        if (tid < nr) copy8(sd + tid, vh + (size_t)l * N + tid);
      } else {
        ul = tid < mr && a_i != 0.0 ? __ldcg(uh + (size_t)l * M + tid) : 0.0;
        vl = tid < nr ? __ldcg(vh + (size_t)l * N + tid) : 0.0;
      }
      stage = kBackward;
      if (sync_or(!ok)) {
        ok = false;
        break;
      }
    }
  }
  ok = !sync_or(!ok || *(volatile unsigned*)p.err != 0u);
  if (es[1] == 0.0) {  // left before a verdict: let the error warp go
    if (tid == 0) es[2] = 1.0;
    errors_in();
  }
  const bool done = ok && es[1] == 1.0;
  if (GRAD && done && ci == 0 && tid < mr) {
    p.grad[m0 + tid] = ga;
    if (!isfinite(ga)) p.res[kResGradBad] = 1.0;
  }
  if (tid == 0) {
    if (GRAD && done && cta == 0) p.res[kResGradNs] = (double)(globaltimer_ns() - t_b);
    words_leave(p.res, cta, ok && es[1] != 3.0, done);
  }
}

// Support sizes (non-zero masses) and whether a mass is one the scaling form
// does not take (negative or not finite) or a side has none; clears *err.
__global__ void __launch_bounds__(kThreads) masses_kernel(const double* a, const double* b, int M, int N, double* info,
                                                     unsigned* err) {
  __shared__ int cnt[2];
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  int ca = 0, cbn = 0, bad = 0;
  for (int i = threadIdx.x; i < M; i += kThreads) {
    const double x = a[i];
    ca += x != 0.0;
    bad |= !(x >= 0.0 && x <= 1e300);
  }
  for (int j = threadIdx.x; j < N; j += kThreads) {
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

struct Shape {
  int gr, gc, lds, ldm, ldn, nsm, chunks, reg;
  size_t smem;
};

// Leading dimension of a block: lds / 2 odd, so that the 16-byte loads of eight
// neighbouring columns hit all banks.
int block_ld(int m) {
  const int e = (m + 1) & ~1;
  return (e >> 1) & 1 ? e : e + 2;
}

// The grid of an M x N problem; false when no grid of one block per SM holds it.
// The cost of an iteration in clocks, as measured: about 0.17 per element of a
// block (two passes, 16 bytes of shared memory each, at 100 B per clock) and
// 2200 + 40 g for an exchange among g CTAs, none when a block spans the side.
// A problem that fits on the chip always goes here: from 120 x 95 (one CTA: 237
// us a call against 571) to 2048^2 (1929 against 5332) the general drivers lost.
bool shape(const Context* ctx, int M, int N, Shape* best) {
  if (ctx->sm_count > kMaxG || M > 8192) return false;  // (the general drivers refuse more rows of support)
  double cost = 0.0;
  bool found = false;
  for (int gr = (M + kMaxSide - 1) / kMaxSide; gr <= std::min(M, ctx->sm_count); ++gr)
    for (int gc = (N + kMaxSide - 1) / kMaxSide; gc <= std::min(N, ctx->sm_count / gr); ++gc) {
      Shape s{};
      s.gr = gr;
      s.gc = gc;
      s.ldm = (M + gr - 1) / gr;
      s.ldn = (N + gc - 1) / gc;
      const double t = 0.17 * s.ldm * s.ldn + (gr > 1 ? 2200.0 + 40.0 * gr : 0.0) + (gc > 1 ? 2200.0 + 40.0 * gc : 0.0);
      if (found && t >= cost) continue;
      s.lds = block_ld(s.ldm);
      const int nrw = (s.ldm + 63) / 64;
      s.nsm = s.ldn;
      s.chunks = 1;
      for (int q = 0; q < 2; ++q) {  // all columns in shared memory, else some in registers
        s.chunks = std::max(NW / ((s.nsm + 31) / 32), q ? nrw : 1);
        s.smem = sizeof(double) * smem_doubles(s.lds, s.ldn, s.nsm, s.chunks);
        if (s.smem <= (size_t)ctx->smem_optin) break;
        s.nsm = s.ldn - kRegCols * (NW / nrw);
        s.reg = 1;
        if (s.nsm < 1) break;
      }
      if (s.nsm < 1 || s.smem > (size_t)ctx->smem_optin) continue;
      *best = s;
      cost = t;
      found = true;
    }
  return found;
}

template <bool GRAD, bool REG>
int launch(Context* ctx, Args& p, const Shape& s, cudaStream_t st) {
  auto kern = resident_kernel<GRAD, REG>;
  static const KernelSlot slot;
  if (int rc = raise_smem(ctx, slot, (const void*)kern, s.smem)) return rc;
  void* args[] = {&p};
  RWIG_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)kern, dim3(s.gr * s.gc), dim3(kThreads), args, s.smem, st));
  return 0;
}

enum { SRS_PACKETS = 250, SRS_INFO };

}  // namespace skres

int sinkhorn_resident(Context* ctx, cudaStream_t st, bool vanilla, double* P, double* grad_a, double* f, double* g,
                      double* loss, int* iter, double* err, const double* a, const double* b, const double* C, int M,
                      int N, double reg, int max_iter, double zero_tol, ResidentTry* out) {
  using namespace skres;
  const bool grad = grad_a != nullptr;
  Shape s;
  if (max_iter < 1 || !(zero_tol <= 999.0) || !shape(ctx, M, N, &s)) return 0;
  const size_t G = (size_t)s.gr * s.gc, L2 = (size_t)max_iter + 4;
  // the scalings of every iteration, in the general drivers' own slots: they are
  // of the same size, so what cannot be had here is refused there
  const size_t bytes_u = 8 * L2 * (size_t)M, bytes_v = 8 * L2 * (size_t)N;
  if (grad && bytes_u + bytes_v > kMaxHistoryBytes) return 0;
  if (!ctx->resident_res) {
    void* h = nullptr;
    RWIG_CUDA_TRY(cudaHostAlloc(&h, sizeof(double) * kResWords, cudaHostAllocMapped));
    ctx->resident_res = (double*)h;
  }
  double* dres = nullptr;
  RWIG_CUDA_TRY(cudaHostGetDevicePointer((void**)&dres, ctx->resident_res, 0));
  const size_t nc = 2 * (size_t)s.gr * N, nrp = 2 * (size_t)s.gc * M;
  const size_t bytes = sizeof(Packet) * (nc + nrp + 14 * G);
  const bool fresh = (int)ctx->slots.size() <= SRS_PACKETS || ctx->slot_bytes[SRS_PACKETS] < bytes;
  Packet* pk = (Packet*)scratch(ctx, SRS_PACKETS, bytes);
  double* info = (double*)scratch(ctx, SRS_INFO, sizeof(double) * 4);
  double* uh = grad ? (double*)scratch(ctx, kSlotHistoryF, bytes_u) : nullptr;
  double* vh = grad ? (double*)scratch(ctx, kSlotHistoryG, bytes_v) : nullptr;
  if (!pk || !info || (grad && (!uh || !vh))) return 0;
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
  p.gr = s.gr;
  p.gc = s.gc;
  p.lds = s.lds;
  p.ldn = s.ldn;
  p.nsm = s.nsm;
  p.chunks = s.chunks;
  p.vanilla = vanilla;
  p.max_iter = max_iter;
  p.eps = reg;
  p.tol = zero_tol;
  p.cpart = pk;
  p.rpart = p.cpart + nc;
  p.epart = p.rpart + nrp;
  p.fin = p.epart + 8 * G;
  p.epoch = ++ctx->resident_epoch << 32;
  p.res = dres;
  p.err = (unsigned*)(info + 3);
  double* res = ctx->resident_res;
  words_clear(res);
  RWIG_CUDA_TRY(cudaEventRecord(ctx->ev0, st));
  masses_kernel<<<1, kThreads, 0, st>>>(a, b, M, N, info, p.err);
  int rc;
  if (grad) rc = s.reg ? launch<true, true>(ctx, p, s, st) : launch<true, false>(ctx, p, s, st);
  else rc = s.reg ? launch<false, true>(ctx, p, s, st) : launch<false, false>(ctx, p, s, st);
  if (rc) return rc;
  out->launches = 2;
  RWIG_CUDA_TRY(cudaEventRecord(ctx->ev1, st));
  RWIG_CUDA_TRY(cudaEventSynchronize(ctx->ev1));
  const int outcome = words_outcome(res);
  if (outcome < 0) return set_error(RWIG_E_TIMEOUT, "Sinkhorn kernel stopped by a bounded wait");
  out->support_m = (int)res[kResSupM];
  out->support_n = (int)res[kResSupN];
  if (outcome == 0) return 0;
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  const int it = (int)res[kResIter];
  const double e = res[kResErr];
  if (loss) *loss = res[kResLoss];
  if (iter) *iter = it;
  if (err) *err = e;
  out->status = (e <= zero_tol) ? 0 : (it == max_iter ? 1 : 2);
  rwig_report& R = report();
  R.iter = it;
  R.status = out->status;
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
  R.kernel_launches = out->launches;
  R.support_m = out->support_m;
  R.support_n = out->support_n;
  return 1;
}

}  // namespace rwig
