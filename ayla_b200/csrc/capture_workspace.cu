// Workspaces of launches that are captured into CUDA graphs.
//
// A captured launch keeps its workspace pointer for as long as its graph lives, and a graph may be replayed beside
// eager launches and other graphs, so it can share theirs with neither: each capture gets memory of its own, which the
// graph (and every executable made from it) holds through a user object.  Launches captured on one stream follow one
// another and leave the arrival counters at zero, so they share a block.
#include "capture_workspace.h"

#include <mutex>
#include <new>

namespace ayla_b200 {
namespace {

struct Block {
  void* ptr = nullptr;
  size_t bytes = 0;
  int device = 0;
  bool held = false;  // by a graph, or about to be
  unsigned long long capture = 0;
  cudaGraph_t graph = nullptr;
  cudaStream_t stream = nullptr;
  Block* next = nullptr;
};

std::mutex g_mutex;
Block* g_blocks = nullptr;

// The graph and its executables are gone and none of their launches is running.  Runs on a thread of the driver, which
// must not call CUDA: the memory is given back by the next capture.
void CUDART_CB let_go(void* block) {
  std::lock_guard<std::mutex> lock(g_mutex);
  static_cast<Block*>(block)->held = false;
}

// Allocating, clearing and waiting on a stream of our own, while this or another thread captures.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// Memory whose first `zero_bytes` are zero; gives `idle` back first.
cudaError_t cleared(void** ptr, size_t bytes, size_t zero_bytes, Block* idle) {
  RelaxedCapture relaxed;
  cudaStream_t stream = nullptr;
  cudaError_t err = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
  if (err != cudaSuccess) {
    std::lock_guard<std::mutex> lock(g_mutex);
    while (idle != nullptr) {
      Block* next = idle->next;
      idle->next = g_blocks;
      g_blocks = idle;
      idle = next;
    }
    return err;
  }
  while (idle != nullptr) {
    Block* next = idle->next;
    cudaFreeAsync(idle->ptr, stream);
    delete idle;
    idle = next;
  }
  err = cudaMallocAsync(ptr, bytes, stream);
  if (err == cudaSuccess) {
    err = cudaMemsetAsync(*ptr, 0, zero_bytes, stream);
    if (err != cudaSuccess) cudaFreeAsync(*ptr, stream);
  }
  const cudaError_t synced = cudaStreamSynchronize(stream);
  if (err == cudaSuccess && synced != cudaSuccess) {
    err = synced;
    cudaFreeAsync(*ptr, stream);
  }
  cudaStreamDestroy(stream);
  return err;
}

}  // namespace

cudaError_t capture_workspace(cudaStream_t stream, size_t bytes, size_t zero_bytes, void** workspace) {
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long capture = 0;
  cudaGraph_t graph = nullptr;
  err = cudaStreamGetCaptureInfo_v2(stream, &status, &capture, &graph, nullptr, nullptr);
  if (err != cudaSuccess) return err;
  if (status != cudaStreamCaptureStatusActive || graph == nullptr) return cudaErrorIllegalState;

  Block* idle = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    for (Block* b = g_blocks; b != nullptr; b = b->next) {
      if (b->device == device && b->held && b->capture == capture && b->graph == graph && b->stream == stream &&
          b->bytes >= bytes) {
        *workspace = b->ptr;
        return cudaSuccess;
      }
    }
    for (Block** at = &g_blocks; *at != nullptr;) {
      Block* b = *at;
      if (b->device == device && !b->held) {
        *at = b->next;
        b->next = idle;
        idle = b;
      } else {
        at = &b->next;
      }
    }
  }
  Block* block = new (std::nothrow) Block;
  if (block == nullptr) return cudaErrorMemoryAllocation;
  err = cleared(&block->ptr, bytes, zero_bytes, idle);
  if (err != cudaSuccess) {
    delete block;
    return err;
  }
  block->bytes = bytes;
  block->device = device;
  block->stream = stream;
  cudaUserObject_t object = nullptr;
  err = cudaUserObjectCreate(&object, block, let_go, 1, cudaUserObjectNoDestructorSync);
  const bool made = err == cudaSuccess;
  if (made) {
    block->held = true;
    err = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
  }
  if (err == cudaSuccess) {
    block->capture = capture;
    block->graph = graph;
    *workspace = block->ptr;
  }
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    block->next = g_blocks;
    g_blocks = block;
  }
  if (made && err != cudaSuccess) cudaUserObjectRelease(object, 1);  // lets go of the block
  return err;
}

}  // namespace ayla_b200
