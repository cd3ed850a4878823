// resident_words.h -- the host-mapped words through which a resident Sinkhorn
// solve (sinkhorn_resident.cu) reports, what its CTAs leave in them and what the
// host makes of them.
#pragma once

#ifdef __CUDACC__
#define RWIG_HD __host__ __device__ __forceinline__
#else
#define RWIG_HD inline
#endif

namespace rwig {
namespace skres {

constexpr double kResRunning = 0.0, kResFinished = 1.0, kResUnsafe = 2.0;
enum { kResIter = 0, kResErr, kResStatus, kResLoss, kResL1Row, kResL1Col, kResL2Row, kResL2Col, kResSupM, kResSupN,
       kResKerr, kResGradNs, kResGradBad, kResWords };

// Before the launch.
inline void words_clear(double* res) {
  res[kResStatus] = kResRunning;
  res[kResKerr] = res[kResGradBad] = 0.0;
}

// A CTA's end: `waits` none of its waits ran out and it saw no other's run out,
// `done` its share of the outputs is written.  The status is CTA 0's, but a wait
// can run out anywhere, also after CTA 0 has left (the last exchange of a
// gradient is among one block row only), so any CTA reports that and none
// takes it back.
RWIG_HD void words_leave(volatile double* res, int cta, bool waits, bool done) {
  if (!waits) res[kResKerr] = 1.0;
  if (cta == 0) res[kResStatus] = done ? kResFinished : kResUnsafe;
}

// After the launch: 1 finished, 0 not in the scaling form's range (the general
// drivers start again), -1 a bounded wait ran out.
inline int words_outcome(const double* res) {
  if (res[kResKerr] != 0.0) return -1;
  return res[kResStatus] == kResFinished && res[kResGradBad] == 0.0 ? 1 : 0;
}

}  // namespace skres
}  // namespace rwig
