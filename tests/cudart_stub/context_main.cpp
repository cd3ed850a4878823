// The engine's per-device contexts (rwig_b200/csrc/context.cu, compiled as C++)
// on a stand-in CUDA runtime with two devices, which records the kernels'
// shared-memory limits per device as the real one does.  Exits 0 when all holds.
#include <cstdio>
#include <map>
#include <utility>

#include "../../rwig_b200/csrc/engine.h"

static int g_current = 0, g_calls = 0;
static std::map<std::pair<int, const void*>, int> g_limit;

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { *n = 2; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { g_current = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = g_current; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  *p = cudaDeviceProp{};
  p->major = 10;
  p->multiProcessorCount = 148;
  p->sharedMemPerBlockOptin = 232448;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
  ++g_calls;
  g_limit[{g_current, f}] = v;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return ""; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void**, size_t, unsigned) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}

#define CHECK(x)                                        \
  do {                                                  \
    if (!(x)) {                                         \
      std::printf("line %d: %s\n", __LINE__, #x);       \
      return 1;                                         \
    }                                                   \
  } while (0)

int main() {
  static int kern, other;
  static const rwig::KernelSlot ks, os;
  rwig::Context* ctx[2];
  for (int d = 0; d < 2; ++d) {
    CHECK(rwig_init(d) == 0);
    ctx[d] = rwig::get_context();
    CHECK(ctx[d] && ctx[d]->device == d);
  }
  CHECK(ctx[0] != ctx[1]);
  for (int d = 0; d < 2; ++d) {  // the same kernel on either device, small launches after large ones
    cudaSetDevice(d);
    CHECK(rwig::raise_smem(ctx[d], ks, &kern, 200000) == 0 && g_limit[std::make_pair(d, &kern)] == 200000);
    CHECK(rwig::raise_smem(ctx[d], ks, &kern, 60000) == 0 && g_limit[std::make_pair(d, &kern)] == 200000);
    CHECK(rwig::raise_smem(ctx[d], os, &other, 60000) == 0 && g_limit[std::make_pair(d, &other)] == 60000);
    CHECK(g_calls == 2 * (d + 1));
  }
  CHECK(rwig::raise_smem(ctx[1], ks, &kern, 210000) == 0 && g_limit[std::make_pair(1, &kern)] == 210000 && g_calls == 5);
  rwig_shutdown();
  return 0;
}
