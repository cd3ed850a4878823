// barycenter_log.cu -- the log barycenter in the log domain: the reference's
// own updates (Barycenter::_fwd_log, src/barycenter_impl_log.cpp:189-272, and
// _bwd_log, :275-382) with no Gibbs kernel K anywhere, for the regimes where
// the scaling form of barycenter.cu would leave the range of doubles (max
// C / eps above ~700, or scalings beyond 1e+-290).  barycenter.cu runs the
// scaling form first and hands the problem here when its range certificate
// fails (or always, with the option "barycenter.log_path" = 1).
//
// Every sweep is a soft-min over one axis of C minus a potential,
//   column pass  m_js = softmin_i (C_ij - F_is),   row pass  r_is = softmin_j (C_ij - G_js),
// softmin_k(x_k) = -eps log sum_k exp(-x_k / eps), evaluated with the running
// maximum of each tile as the shift (one exponential per element).  With
// R_s = C - F_s 1^T - 1 G_s^T one forward iteration l is
//   F_l      = F_{l-1} + (eps log A + KV_{l-1}),   KV_{l-1} = r_{l-1} - F_{l-1}   (:231)
//   m_l      = column pass over C - F_l,   KTU = m_l - G_{l-1}                   (:238)
//   logb_l   = -(sum_s w_s m_l,s) / eps,   G_l = eps logb_l + m_l                (:239, :245)
//   r_l      = row pass over C - G_l,      KV_l = r_l - F_l                      (:251)
//   err      = || -KV_l / eps - log A ||_2 (spectral norm, :252)
// and the adjoint step l reads the row- and column-softmax weights of the
// reference (:306-346) with their normalisers from the forward:
//   X_ij = exp((r_l,is + G_l,js - C_ij) / eps)    (row softmax at F_l, G_l)
//   W_ij = exp((m_l,js + F_l,is - C_ij) / eps)    (column softmax at F_l, G_{l-1})
//   Gbar_js = -sum_i X_ij Fbar_is,  logbbar_j = eps sum_s Gbar_js  (l < L)
//   y_js = (w_s / eps) logbbar_j - Gbar_js,  Fbar_is = sum_j W_ij y_js
//   grad_A += Fbar / A,  grad_w -= m_l^T logbbar,  then grad_A *= eps, grad_w /= eps.
// The histories F_l, G_l, m_l, r_l (l = 0..L) stay on the device.
//
// Pass kernel: a CTA owns one output and all its histograms; lanes run along
// the reduction axis, which is the contiguous one of C or, for the row passes,
// of a transposed copy made once per call.  So a sum is complete in its CTA,
// which carries the elementwise updates above as well: two launches per
// iteration in each direction, nothing merged between CTAs, every sum in a
// fixed order (results are bitwise repeatable).  The exponential is the table
// method of fastexp.cuh.  Large problems are bound by instruction issue (about
// 26 of them per exponential, 14 in FP64): 2048 x 2048 x 32 takes 355 us a pass.
// Small ones are bound by one CTA's chain (two loads from L2, the exponentials,
// two warp reductions, log: 3 us) and the launch: programmatic launches let the
// next pass's CTAs stand by.  360 x 360 x 5, 20 iterations with gradient: 650 us
// a call, 7.5 us a pass; with 64 x 16 output tiles and slices of the reduction
// axis merged by another kernel, 18 CTAs in all there, it took 6047 us, and 8039
// against 7144 us for 5 iterations of 2048 x 2048 x 32.
#include <algorithm>
#include <cmath>
#include <vector>

#include "barycenter.h"
#include "common.cuh"
#include "dgemm.cuh"
#include "engine.h"
#include "fastexp.cuh"

namespace rwig {
namespace barylog {

constexpr int kMaxWarps = 16;  // per CTA
constexpr int kChunk = 4;      // reduction elements a lane holds at once
constexpr int kSpread = 4;     // replicas of the exponential's table
// Where a maximum starts.  Finite, so that a lane or a warp whose every term is
// exp(-inf) (zero masses, infinite costs) keeps a sum of zero, which adds nothing
// to the others' (from -inf on it is 0 * exp(-inf + inf) = NaN).
constexpr double kNoTerm = -1.7976931348623157e308;

enum Mode { kColFwd, kRowFwd, kColBwd, kRowBwd };

// One pass over the outputs o < O, histograms s < S, k < K, with C(k,o) at
// C[k + o K]:
//   forward   t_os = -eps log sum_k exp((P_ks - C(k,o)) / eps),
//   backward  t_os = sum_k exp((P_ks + Q_os - C(k,o)) / eps) Y_ks,
// then the mode's updates (kColFwd: o = j, the new m, logb, G; kRowFwd: o = i,
// r = t, KV = r - F, the next F and, when D is given, the residual; kColBwd:
// Gbar = -t and the row step's right-hand side; kRowBwd: Fbar = t, grad_A).
struct Pass {
  const double* C;
  int K, O, S;
  int sw, kw;  // warps along the histograms and along k
  double eps, inv_eps;
  const double* P;   // K x S
  const double* Q;   // O x S (backward)
  const double* Y;   // K x S (backward)
  const double* w;   // S
  double* out;       // O x S: m, r, y, Fbar
  const double* in;  // O x S: -, F, m, A
  double* x1;        // O x S: G, the next F, gwp (S x O), grad_A
  double* logb;      // O (kColFwd)
  const double* logA;  // O x S (kRowFwd)
  double* D;           // (kRowFwd)
  long long ldd;
};

// exp(x) by the table method for x <= 709, 0 below -708 and for NaN: what the
// method makes of those is thrown away, which takes a third of the
// instructions of clamping them first.
__device__ __forceinline__ double expz(double x, const double* tbl) {
  const double e = exp_tbl<kSpread, false>(x, tbl);
  return x >= -708.0 ? e : 0.0;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double x = __shfl_xor_sync(0xffffffffu, v, o);
    v = x > v ? x : v;
  }
  return v;
}

// SQ histograms per warp share each load of C.
template <int MODE, int SQ>
__global__ void __launch_bounds__(32 * kMaxWarps, 2) pass_kernel(Pass a) {
  constexpr bool FWD = MODE == kColFwd || MODE == kRowFwd;
  constexpr int CH = kChunk;
  extern __shared__ double part[];  // [kw][S] sums, then (forward) [kw][S] maxima
  __shared__ double tbl_all[64 * kSpread];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int S = a.S, K = a.K, O = a.O;
  for (int i = tid; i < 64 * kSpread; i += blockDim.x) tbl_all[i] = __longlong_as_double((long long)kExp2J64[i / kSpread]);
  const double* tbl = tbl_all + (tid & (kSpread - 1));
  const double ie = a.inv_eps;
  const int si = wid % a.sw, ki = wid / a.sw, step = 32 * a.kw;
  asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the kernel before has ended
  for (int o = blockIdx.x; o < O; o += gridDim.x) {
    __syncthreads();  // the table is loaded; the last output's partials are read
    const double* Co = a.C + (size_t)o * K;
    // what the updates of histogram tid need, on its way meanwhile
    double in0 = 0.0, la0 = 0.0;
    if (MODE != kColFwd && tid < S) {
      in0 = a.in[o + (size_t)tid * O];
      if (MODE == kRowFwd) la0 = a.logA[o + (size_t)tid * O];
    }
    for (int s0 = si * SQ; s0 < S; s0 += a.sw * SQ) {
      double mx[SQ], sm[SQ], qv[SQ];
      const double* P[SQ];
      const double* Y[SQ];
#pragma unroll
      for (int q = 0; q < SQ; ++q) {
        const int s = min(s0 + q, S - 1);
        P[q] = a.P + (size_t)s * K;
        Y[q] = FWD ? nullptr : a.Y + (size_t)s * K;
        qv[q] = FWD ? 0.0 : a.Q[o + (size_t)s * O] * ie;
        mx[q] = kNoTerm;
        sm[q] = 0.0;
      }
      for (int kb = 32 * ki; kb < K; kb += CH * step) {
        // elements beyond K: C = inf, which contributes nothing; whole warps
        // beyond it are skipped
        double x[SQ][CH], y[FWD ? 1 : SQ][CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
          const int k = kb + i * step + lane;
          const bool in = k < K;
          const double c = in ? Co[k] : INFINITY;
#pragma unroll
          for (int q = 0; q < SQ; ++q) {
            x[q][i] = ((in ? P[q][k] : 0.0) - c) * ie;
            if (!FWD) y[q][i] = in ? Y[q][k] : 0.0;
          }
        }
#pragma unroll
        for (int q = 0; q < SQ; ++q) {
          if (FWD) {
            double tm = mx[q];
#pragma unroll
            for (int i = 0; i < CH; ++i) tm = x[q][i] > tm ? x[q][i] : tm;
            if (tm > mx[q]) {
              if (kb >= CH * step) sm[q] *= expz(mx[q] - tm, tbl);
              mx[q] = tm;
            }
          }
#pragma unroll
          for (int i = 0; i < CH; ++i)
            if (kb + i * step < K) {
              if (FWD) {
                sm[q] += expz(x[q][i] - mx[q], tbl);
              } else {
                const double z = x[q][i] + qv[q];
                sm[q] = fma(expz(z > 709.0 ? 709.0 : z, tbl), y[q][i], sm[q]);
              }
            }
        }
      }
#pragma unroll
      for (int q = 0; q < SQ; ++q) {
        double m = 0.0, t = sm[q];
        if (FWD) {
          m = warp_max(mx[q]);
          t *= exp(mx[q] - m);
        }
        t = warp_sum(t);
        if (lane == 0 && s0 + q < S) {
          part[ki * S + s0 + q] = t;
          if (FWD) part[(a.kw + ki) * S + s0 + q] = m;
        }
      }
    }
    __syncthreads();
    // totals over the k warps, and the updates; threads s < S (one warp for the
    // column modes, which also sum over s)
    constexpr bool COL = MODE == kColFwd || MODE == kColBwd;
    double acc = 0.0;
    const int ns = COL ? 32 : (int)blockDim.x;
    if (tid < ns)
      for (int s = tid; s < S; s += ns) {
        double t = 0.0;
        if (FWD) {
          double m = kNoTerm;
          for (int z = 0; z < a.kw; ++z) m = fmax(m, part[(a.kw + z) * S + s]);
          if (a.kw == 1) t = part[s];
          else
            for (int z = 0; z < a.kw; ++z) t += part[z * S + s] * exp(part[(a.kw + z) * S + s] - m);
          t = -a.eps * (m + log(t == 0.0 ? NAN : t));  // (an output without a finite term)
        } else {
          for (int z = 0; z < a.kw; ++z) t += part[z * S + s];
        }
        const size_t e = o + (size_t)s * O;
        if (MODE == kColFwd) {
          a.out[e] = t;
          part[s] = t;  // (this thread alone reads column s of the partials)
          acc += t * a.w[s];
        } else if (MODE == kRowFwd) {
          const double f = s == tid ? in0 : a.in[e], kv = t - f, la = s == tid ? la0 : a.logA[e];
          a.out[e] = t;
          a.x1[e] = f + (a.eps * la + kv);                                   // :231
          if (a.D) a.D[o + (long long)s * a.ldd] = -kv / a.eps - la;         // :252
        } else if (MODE == kColBwd) {
          part[s] = -t;
          acc -= t;
        } else {
          a.out[e] = t;
          a.x1[e] += t / (s == tid ? in0 : a.in[e]);
        }
      }
    if (COL && tid < 32) {
      acc = warp_sum(acc);
      if (MODE == kColFwd) {
        const double lb = -acc / a.eps;  // barycenter_impl_log.cpp:239
        if (lane == 0) a.logb[o] = lb;
        for (int s = lane; s < S; s += 32) a.x1[o + (size_t)s * O] = a.eps * lb + part[s];  // :245
      } else {
        const double lbb = a.eps * acc;
        for (int s = lane; s < S; s += 32) {
          a.out[o + (size_t)s * O] = (a.w[s] / a.eps) * lbb - part[s];
          a.x1[(size_t)o * S + s] -= (s == tid ? in0 : a.in[o + (size_t)s * O]) * lbb;  // :368-372
        }
      }
    }
  }
}

// Adjoint seed (thread per support point j): logbbar = 2 (b - b_ext) o b with
// the normalised b (:324), Gbar = 0, y = (w / eps) logbbar, gwp[j S + s] =
// -m_L,js logbbar_j.
__global__ void seed_bwd(int N, int S, double eps, const double* bn, const double* bext, const double* w,
                         const double* Ml, double* Yv, double* gwp) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < N; j += gridDim.x * blockDim.x) {
    const double lbb = 2.0 * (bn[j] - bext[j]) * bn[j];
    for (int s = 0; s < S; ++s) {
      Yv[j + (long long)s * N] = (w[s] / eps) * lbb;
      gwp[(long long)j * S + s] -= Ml[j + (long long)s * N] * lbb;
    }
  }
}

// Ct (N x M) = the transpose of C (M x N), 32 x 32 tiles.
__global__ void __launch_bounds__(256) transpose_kernel(const double* C, int M, int N, double* Ct) {
  __shared__ double t[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int tm = (M + 31) / 32;
  const long long tiles = (long long)tm * ((N + 31) / 32);
  for (long long b = blockIdx.x; b < tiles; b += gridDim.x) {
    const int m0 = (int)(b % tm) * 32, n0 = (int)(b / tm) * 32;
    __syncthreads();
    for (int r = ty; r < 32; r += 8)
      if (m0 + tx < M && n0 + r < N) t[r][tx] = C[(size_t)(n0 + r) * M + m0 + tx];
    __syncthreads();
    for (int r = ty; r < 32; r += 8)
      if (n0 + tx < N && m0 + r < M) Ct[(size_t)(m0 + r) * N + n0 + tx] = t[tx][r];
  }
}

__global__ void axpby_kernel(double* x, long long n, double a) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    x[k] *= a;
}

__global__ void zero_kernel(double* x, long long n) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    x[k] = 0.0;
}

__global__ void log_kernel(const double* x, long long n, double* out) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    out[k] = log(x[k]);
}

// grad_w[s] = (sum_j gwp[j S + s]) / eps, one block per s, fixed order.
__global__ void reduce_gw_eps(const double* gwp, int N, int S, double eps, double* gw) {
  __shared__ double sh[256];
  const int s = blockIdx.x;
  double v = 0.0;
  for (int j = threadIdx.x; j < N; j += blockDim.x) v += gwp[(long long)j * S + s];
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) gw[s] = sh[0] / eps;  // :377
}

// One block: b = exp(logb) / sum, loss = sum (b - b_ext)^2 when b_ext (:268-271).
__global__ void finish_b(const double* logb, int N, const double* bext, double* bn, double* out2) {
  __shared__ double sh[1024];
  double acc = 0.0;
  for (int j = threadIdx.x; j < N; j += blockDim.x) acc += exp(logb[j]);
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  const double tot = sh[0];
  __syncthreads();
  double l = 0.0;
  for (int j = threadIdx.x; j < N; j += blockDim.x) {
    const double v = exp(logb[j]) / tot;
    bn[j] = v;
    if (bext) {
      const double d = v - bext[j];
      l += d * d;
    }
  }
  sh[threadIdx.x] = l;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out2[0] = tot;
    out2[1] = sh[0];
  }
}

enum {
  SL_FH = 300, SL_GH, SL_MH, SL_RH, SL_LB, SL_LOGA, SL_D, SL_GRAM, SL_CT, SL_FBAR, SL_Y, SL_GA,
  SL_GWP, SL_GW, SL_BN, SL_SCAL
};

int grid1(const Context* ctx, long long n) {
  return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 8LL * ctx->sm_count));
}

// Launch of a pass.  Histograms per warp: one up to 8 of them (more warps),
// else two, which read C half as often (2048 x 2048 x 32: 1421 us per iteration
// and its backward step against 1607 with one and 1460 with four, which need
// 128 registers).  Warps along k: until the chip has 16 warps per SM or a lane
// has one chunk (360 x 360 x 5: 838 us a call against 922 with 8 warps per SM).
template <int MODE>
void launch_pass(const Context* ctx, Pass a, cudaStream_t st) {
  const int sq = a.S <= 8 ? 1 : 2;
  a.sw = std::min(8, (a.S + sq - 1) / sq);
  a.kw = 1;
  while (2 * a.kw * a.sw <= kMaxWarps && 32LL * kChunk * a.kw < a.K &&
         (long long)a.O * a.sw * a.kw < 16LL * ctx->sm_count)
    a.kw *= 2;
  const int threads = 32 * a.sw * a.kw;
  const int grid = (int)std::min<long long>(a.O, (long long)ctx->sm_count * (2048 / threads));
  const size_t smem = sizeof(double) * 2 * (size_t)a.kw * a.S;  // at most 16 KB (64 histograms)
  // the next pass may take its place while this one drains (it waits for its
  // end before it reads anything)
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, sq == 1 ? pass_kernel<MODE, 1> : pass_kernel<MODE, 2>, a);  // (errors: at the next check)
}

}  // namespace barylog

namespace bary {

using namespace barylog;

// The log barycenter in the log domain; arguments and outputs as run()
// (barycenter.h).  *launches is increased by the kernels launched.
int run_log(Context* ctx, cudaStream_t st, double* X1, double* X2, double* b, double* gradA, double* gradw,
            double* loss, int* iter_out, double* err_out, const double* A, const double* w, const double* C,
            const double* bext, int M, int N, int S, double reg, int withgrad, int max_iter, double tol,
            int* launches) {
  const int L = std::max(0, max_iter);
  const size_t MS = (size_t)M * S, NS = (size_t)N * S;
  const long long ldd = ((M + 1) / 2) * 2;
  const int H = withgrad ? L + 2 : 2;  // slots of F (l = 0..L+1) and of G, m, r
  const bool fixed = !(tol > 0.0);
  double* Fh = (double*)scratch(ctx, SL_FH, sizeof(double) * MS * H);
  double* Gh = (double*)scratch(ctx, SL_GH, sizeof(double) * NS * H);
  double* Mh = (double*)scratch(ctx, SL_MH, sizeof(double) * NS * H);
  double* Rh = (double*)scratch(ctx, SL_RH, sizeof(double) * MS * H);
  double* lb = (double*)scratch(ctx, SL_LB, sizeof(double) * N);
  double* logA = (double*)scratch(ctx, SL_LOGA, sizeof(double) * MS);
  double* D = (double*)scratch(ctx, SL_D, sizeof(double) * ldd * S);
  double* gram = (double*)scratch(ctx, SL_GRAM, sizeof(double) * S * S);
  double* Ct = (double*)scratch(ctx, SL_CT, sizeof(double) * (size_t)M * N);
  double* bn = (double*)scratch(ctx, SL_BN, sizeof(double) * N);
  double* scal = (double*)scratch(ctx, SL_SCAL, sizeof(double) * 8);
  if (!Fh || !Gh || !Mh || !Rh || !lb || !logA || !D || !gram || !Ct || !bn || !scal) return RWIG_E_NOMEM;
  double *Fbar = nullptr, *Yv = nullptr, *gA = nullptr, *gwp = nullptr, *gw = nullptr;
  if (withgrad) {
    Fbar = (double*)scratch(ctx, SL_FBAR, sizeof(double) * MS);
    Yv = (double*)scratch(ctx, SL_Y, sizeof(double) * NS);
    gA = (double*)scratch(ctx, SL_GA, sizeof(double) * MS);
    gwp = (double*)scratch(ctx, SL_GWP, sizeof(double) * NS);
    gw = (double*)scratch(ctx, SL_GW, sizeof(double) * S);
    if (!Fbar || !Yv || !gA || !gwp || !gw) return RWIG_E_NOMEM;
  }
  auto slot = [&](double* base, size_t sz, int l) { return base + sz * (size_t)(withgrad ? l : (l & 1)); };
  const double inv_eps = 1.0 / reg;
  int nl = 0;
  // passes over the columns (o = j, k = i) and the rows (o = i, k = j) of C
  Pass col{}, row{};
  col.C = C;
  col.K = row.O = M;
  col.O = row.K = N;
  row.C = Ct;
  col.S = row.S = S;
  col.eps = row.eps = reg;
  col.inv_eps = row.inv_eps = inv_eps;
  col.w = w;
  col.logb = lb;
  row.logA = logA;
  row.ldd = ldd;
  auto row_fwd = [&](int l, double* d) {  // r_l, F_{l+1}
    row.P = slot(Gh, NS, l);
    row.in = slot(Fh, MS, l);
    row.out = slot(Rh, MS, l);
    row.x1 = slot(Fh, MS, l + 1);
    row.D = d;
    launch_pass<kRowFwd>(ctx, row, st);
    ++nl;
  };

  // F_0 = G_0 = 0, log A; the initial row soft-min at (0, 0) gives F_1 (:221, :231)
  zero_kernel<<<grid1(ctx, MS), 256, 0, st>>>(slot(Fh, MS, 0), (long long)MS);
  zero_kernel<<<grid1(ctx, NS), 256, 0, st>>>(slot(Gh, NS, 0), (long long)NS);
  zero_kernel<<<grid1(ctx, N), 256, 0, st>>>(lb, N);
  log_kernel<<<grid1(ctx, MS), 256, 0, st>>>(A, (long long)MS, logA);
  nl += 4;
  transpose_kernel<<<std::min(16 * ctx->sm_count, ((M + 31) / 32) * ((N + 31) / 32)), 256, 0, st>>>(C, M, N, Ct);
  ++nl;
  row_fwd(0, nullptr);
  int iter = 0;
  double err = 1000.0;
  while (iter < L && err >= tol) {
    ++iter;
    const int l = iter;
    col.P = slot(Fh, MS, l);
    col.out = slot(Mh, NS, l);
    col.x1 = slot(Gh, NS, l);
    launch_pass<kColFwd>(ctx, col, st);
    ++nl;
    const bool need_err = !fixed || iter == L;
    row_fwd(l, need_err ? D : nullptr);
    RWIG_CUDA_TRY(cudaGetLastError());
    if (need_err) {
      int gl = 0;
      if (int rc = dg::gemm<1>(ctx, dg::GemmArgs{D, ldd, S, M, S, D, ldd, 0}, dg::EpiStore{gram, S, S}, st, 0, &gl))
        return rc;
      nl += gl;
      std::vector<double> G((size_t)S * S);
      RWIG_CUDA_TRY(cudaMemcpyAsync(G.data(), gram, sizeof(double) * S * S, cudaMemcpyDeviceToHost, st));
      RWIG_CUDA_TRY(cudaStreamSynchronize(st));
      err = std::sqrt(lambda_max(G, S));  // Armadillo norm(X, 2) of a matrix: the spectral norm
    }
  }
  // normalised barycenter and loss (:268-271)
  finish_b<<<1, 1024, 0, st>>>(lb, N, withgrad ? bext : nullptr, bn, scal);
  ++nl;

  if (withgrad && iter > 0) {
    RWIG_CUDA_TRY(cudaMemsetAsync(gA, 0, sizeof(double) * MS, st));
    RWIG_CUDA_TRY(cudaMemsetAsync(gwp, 0, sizeof(double) * NS, st));
    for (int l = iter; l >= 1; --l) {
      if (l == iter) {
        seed_bwd<<<grid1(ctx, N), 256, 0, st>>>(N, S, reg, bn, bext, w, slot(Mh, NS, l), Yv, gwp);
      } else {
        // Gbar: column pass weighted by the row softmax at (F_l, G_l) (:306-320)
        col.P = slot(Rh, MS, l);
        col.Q = slot(Gh, NS, l);
        col.Y = Fbar;
        col.out = Yv;
        col.in = slot(Mh, NS, l);
        col.x1 = gwp;
        launch_pass<kColBwd>(ctx, col, st);
      }
      // Fbar: row pass weighted by the column softmax at (F_l, G_{l-1}) (:330-346)
      row.P = slot(Mh, NS, l);
      row.Q = slot(Fh, MS, l);
      row.Y = Yv;
      row.out = Fbar;
      row.in = A;
      row.x1 = gA;
      launch_pass<kRowBwd>(ctx, row, st);
      nl += 2;
    }
    axpby_kernel<<<grid1(ctx, MS), 256, 0, st>>>(gA, (long long)MS, reg);  // :376
    reduce_gw_eps<<<S, 256, 0, st>>>(gwp, N, S, reg, gw);                 // :377
    nl += 2;
    if (gradA) RWIG_CUDA_TRY(cudaMemcpyAsync(gradA, gA, sizeof(double) * MS, cudaMemcpyDeviceToDevice, st));
    if (gradw) RWIG_CUDA_TRY(cudaMemcpyAsync(gradw, gw, sizeof(double) * S, cudaMemcpyDeviceToDevice, st));
  } else if (withgrad) {  // nothing to unroll
    if (gradA) RWIG_CUDA_TRY(cudaMemsetAsync(gradA, 0, sizeof(double) * MS, st));
    if (gradw) RWIG_CUDA_TRY(cudaMemsetAsync(gradw, 0, sizeof(double) * S, st));
  }
  // outputs F_L, G_L (the reference keeps them as U, V: :386-387); b
  if (X1) RWIG_CUDA_TRY(cudaMemcpyAsync(X1, slot(Fh, MS, iter), sizeof(double) * MS, cudaMemcpyDeviceToDevice, st));
  if (X2) RWIG_CUDA_TRY(cudaMemcpyAsync(X2, slot(Gh, NS, iter), sizeof(double) * NS, cudaMemcpyDeviceToDevice, st));
  if (b) RWIG_CUDA_TRY(cudaMemcpyAsync(b, bn, sizeof(double) * N, cudaMemcpyDeviceToDevice, st));
  double sc[2] = {0.0, 0.0};
  RWIG_CUDA_TRY(cudaMemcpyAsync(sc, scal, sizeof(sc), cudaMemcpyDeviceToHost, st));
  RWIG_CUDA_TRY(cudaStreamSynchronize(st));
  RWIG_CUDA_TRY(cudaGetLastError());
  if (loss) *loss = withgrad ? sc[1] : 0.0;
  if (iter_out) *iter_out = iter;
  if (err_out) *err_out = err;
  if (launches) *launches += nl;
  report().bary_norm = sc[0];
  return (err <= tol) ? 0 : (iter == L ? 1 : 2);
}

}  // namespace bary
}  // namespace rwig
