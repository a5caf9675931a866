// Pools of the process: idle device blocks and idle stream sets (internal to libgbx_eri).  Host
// code on the CUDA runtime alone, so that it also runs against a fake runtime.
#pragma once
#include <cuda_runtime_api.h>

#include <cstddef>
#include <memory>
#include <vector>

namespace gbx {

constexpr int kStageBuffers = 3;  // host-output staging slabs in flight

// Streams and events of one basis or batch: the class blocks' auxiliary streams, their join and fork
// events, and the host-output copy stream with the staging slabs' events.  Sets live in a pool per
// device (streams_take / streams_give): creating and destroying 7 streams and 13 events took 2 of
// the 2.9 ms of a 20-function host call.  A set has one owner at a time.
struct StreamSet {
  int device = 0;
  std::vector<cudaStream_t> aux;
  std::vector<cudaEvent_t> join;
  cudaEvent_t fork = nullptr, in = nullptr, out = nullptr;
  cudaStream_t copy = nullptr;
  cudaEvent_t stage_ready[kStageBuffers] = {};
  cudaEvent_t stage_free[kStageBuffers] = {};
  int ensure_aux(int n);  // at least n auxiliary streams
  ~StreamSet();
};
// A set for the current device (from the pool, or a new one).
int streams_take(int device, std::unique_ptr<StreamSet>* out);
// Back to the pool, or destroyed when the pool is full; the caller has made sure that no work is
// queued on its streams (idle), else the set is destroyed.
void streams_give(std::unique_ptr<StreamSet> set, bool idle);
// Device blocks of the process's block cache (release_pools empties it).
int block_alloc(int device, void** p, size_t bytes, size_t* got, const char* what);
void block_give(int device, void* p, size_t bytes);  // no work on the device still uses p
void release_pools();  // frees the idle blocks and destroys the idle stream sets

}  // namespace gbx
