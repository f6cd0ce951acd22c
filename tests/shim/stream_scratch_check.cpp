// The scratch of stream_scratch.cu over a runtime of its own: what consecutive calls of a capture are given when some of them
// may overlap the call before them, some may not and some fail.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../qw38_b200/csrc/stream_scratch.h"

namespace {
bool g_capturing = false;
unsigned long long g_capture = 1;
std::vector<std::pair<void (*)(void*), void*>> g_objects;  // of the live graph
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); return cudaSuccess; }
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus* st, unsigned long long* id, cudaGraph_t* graph,
                                     const cudaGraphNode_t**, size_t*) {
  *st = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  *id = g_capture;
  *graph = nullptr;
  return cudaSuccess;
}
cudaError_t cudaUserObjectCreate(cudaUserObject_t* o, void* p, cudaHostFn_t f, unsigned, unsigned) {
  *o = nullptr;
  g_objects.emplace_back(f, p);
  return cudaSuccess;
}
cudaError_t cudaGraphRetainUserObject(cudaGraph_t, cudaUserObject_t, unsigned, unsigned) { return cudaSuccess; }
}

int main() {
  uint32_t state = 7;
  auto rnd = [&](uint32_t n) { state = state * 1664525u + 1013904223u; return (state >> 8) % n; };
  int overlapped = 0;
  for (int round = 0; round < 400; ++round) {
    g_capturing = round % 8 != 7;
    uintptr_t begin = 0, end = 0;  // of the last call that was launched
    for (int call = 0; call < 40; ++call) {
      uint64_t const bytes = 256 + rnd(rnd(4) ? 1u << 20 : 9u << 20);
      bool const alternate = rnd(3) != 0, fails = rnd(8) == 0;
      q4k::StreamScratch s;
      if (s.acquire(nullptr, bytes, alternate) != cudaSuccess) return std::puts("acquire failed"), 1;
      uintptr_t const b = reinterpret_cast<uintptr_t>(s.p()), e = b + bytes;
      if (b % 256 && g_capturing) return std::puts("misaligned"), 1;
      for (uintptr_t i = b; i < e; i += 4096) *reinterpret_cast<volatile char*>(i) = 1;
      if (s.alternates()) {
        ++overlapped;
        if (!g_capturing || !alternate) return std::puts("alternates without being asked, or eagerly"), 1;
        if (begin < e && b < end) return std::printf("round %d call %d: shares scratch with the call before it\n", round, call), 1;
      }
      if (fails) continue;  // the launch failed: no release()
      if (s.release() != cudaSuccess) return std::puts("release failed"), 1;
      begin = b;
      end = e;
    }
    for (auto const& o : g_objects) o.first(o.second);  // the graph is gone
    g_objects.clear();
    ++g_capture;
  }
  if (overlapped < 1000) return std::printf("only %d calls alternated\n", overlapped), 1;
  return std::puts("stream scratch ok"), 0;
}
