// Per-call scratch.
//
//   * Eager calls: stream-ordered allocation from a memory pool of the library.  The driver hands a block freed on a stream
//     to the next call of that stream without any wait, keeps at most kKeep bytes between calls and gives the rest back at
//     the next synchronisation; two streams or threads never share a block.
//   * Captured calls: one block per capture and stream, because an allocation recorded as a graph node would separate
//     kernels that may overlap.  The graph owns the block through a user object; when the graph and its executables are
//     gone it serves the next capture (or goes back to the pool, beyond kMaxFree idle blocks).  Calls that may overlap the
//     one before them take the two halves of the block in turn; the block remembers whether its last call did, because one
//     that did not (launch overlap was off, or it failed) may lie across both halves.
#include "stream_scratch.h"

#include <mutex>
#include <vector>

namespace q4k {

struct CapturedBlock {
  void* p = nullptr;
  uint64_t bytes = 0;
  int device = 0;
  unsigned long long capture = 0;  // 0 = idle
  cudaStream_t stream = nullptr;
  uint32_t turn = 0;
  bool alternating = true;  // its last call took a half and has been launched; also before the first one
};

namespace {

constexpr uint64_t kKeep = 192ull << 20;
constexpr size_t kMaxFree = 4;

struct Pool {
  cudaMemPool_t eager = nullptr, captured = nullptr;  // apart, so that blocks graphs hold do not count against what is kept
  cudaStream_t helper = nullptr;  // allocations of captured blocks are ordered on it
};

std::mutex g_mutex;
Pool g_pools[64];
std::vector<CapturedBlock*> g_blocks;

// While any stream of the process is being captured, allocation calls are refused unless the thread says that it knows.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};

cudaError_t pool_of(int device, Pool** out) {  // g_mutex held
  if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
  Pool& p = g_pools[device];
  if (!p.captured) {
    RelaxedCapture relaxed;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaError_t st = cudaSuccess;
    if (!p.helper) st = cudaStreamCreateWithFlags(&p.helper, cudaStreamNonBlocking);
    if (st == cudaSuccess && !p.eager) {
      uint64_t keep = kKeep;
      st = cudaMemPoolCreate(&p.eager, &props);
      if (st == cudaSuccess) st = cudaMemPoolSetAttribute(p.eager, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    if (st == cudaSuccess) st = cudaMemPoolCreate(&p.captured, &props);
    if (st != cudaSuccess) return st;
  }
  *out = &p;
  return cudaSuccess;
}

// The last graph that used the block is gone (no CUDA call may be made here).
void CUDART_CB retire_captured(void* data) {
  std::lock_guard<std::mutex> lock(g_mutex);
  static_cast<CapturedBlock*>(data)->capture = 0;
}

cudaError_t captured_block(cudaStream_t stream, cudaGraph_t graph, unsigned long long capture, int device, uint64_t bytes, bool alternate, CapturedBlock** block, void** out,
                           bool* alternates) {
  uint64_t const half = (bytes + 255) / 256 * 256;
  if (alternate) bytes = 2 * half;
  auto take = [&](CapturedBlock* b) {  // halves are half the block's size, whatever the call needs
    *out = static_cast<uint8_t*>(b->p) + (alternate ? (b->turn++ & 1) * (b->bytes / 512 * 256) : 0);
    *alternates = alternate && b->alternating;
    b->alternating = false;  // until release()
    *block = b;
  };
  std::lock_guard<std::mutex> lock(g_mutex);
  CapturedBlock* idle = nullptr;
  size_t idle_count = 0;
  for (CapturedBlock* b : g_blocks) {
    if (b->device != device) continue;
    if (b->capture == capture && b->stream == stream && b->bytes >= bytes) {
      take(b);
      return cudaSuccess;
    }
    if (b->capture == 0) {
      ++idle_count;
      if (b->bytes >= bytes && (!idle || b->bytes < idle->bytes)) idle = b;
    }
  }
  RelaxedCapture relaxed;
  Pool* pool = nullptr;
  cudaError_t st = pool_of(device, &pool);
  if (st != cudaSuccess) return st;
  if (!idle) {
    for (size_t i = g_blocks.size(); i-- > 0 && idle_count > kMaxFree;)
      if (g_blocks[i]->device == device && g_blocks[i]->capture == 0) {
        (void)cudaFreeAsync(g_blocks[i]->p, pool->helper);
        delete g_blocks[i];
        g_blocks.erase(g_blocks.begin() + long(i));
        --idle_count;
      }
    idle = new CapturedBlock;
    idle->device = device;
    idle->bytes = (bytes + (4ull << 20) - 1) / (4ull << 20) * (4ull << 20);
    st = cudaMallocFromPoolAsync(&idle->p, idle->bytes, pool->captured, pool->helper);
    if (st == cudaSuccess) st = cudaStreamSynchronize(pool->helper);
    if (st != cudaSuccess) {
      delete idle;
      return st;
    }
    g_blocks.push_back(idle);
  }
  cudaUserObject_t object = nullptr;
  if ((st = cudaUserObjectCreate(&object, idle, retire_captured, 1, cudaUserObjectNoDestructorSync)) != cudaSuccess) return st;
  idle->capture = capture;
  idle->stream = stream;
  idle->alternating = true;
  if ((st = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove)) != cudaSuccess) {
    idle->capture = ~0ull;  // the object still refers to it: not reused
    return st;
  }
  take(idle);
  return cudaSuccess;
}

}  // namespace

cudaError_t StreamScratch::acquire(cudaStream_t stream, uint64_t bytes, bool alternate) {
  int device = 0;
  cudaError_t st = cudaGetDevice(&device);
  if (st != cudaSuccess) return st;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long capture = 0;
  cudaGraph_t graph = nullptr;
  if ((st = cudaStreamGetCaptureInfo(stream, &status, &capture, &graph)) != cudaSuccess) return st;
  if (status == cudaStreamCaptureStatusActive) {
    alternate_ = alternate;
    return captured_block(stream, graph, capture + 1, device, bytes, alternate, &block_, &p_, &alternates_);
  }
  Pool* pool = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    if ((st = pool_of(device, &pool)) != cudaSuccess) return st;
  }
  if ((st = cudaMallocFromPoolAsync(&p_, bytes, pool->eager, stream)) != cudaSuccess) {
    p_ = nullptr;
    return st;
  }
  stream_ = stream;
  owned_ = true;
  return cudaSuccess;
}

cudaError_t StreamScratch::release() {
  if (block_) {
    std::lock_guard<std::mutex> lock(g_mutex);
    block_->alternating = alternate_;
    block_ = nullptr;
  }
  return give_back();
}

cudaError_t StreamScratch::give_back() {
  if (!owned_) return cudaSuccess;
  owned_ = false;
  return cudaFreeAsync(p_, stream_);
}

}  // namespace q4k
