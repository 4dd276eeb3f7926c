// The pool that batches take their device memory from.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <mutex>

namespace dense_b200 {

// Device memory kept for the next batch.  cudaMalloc and cudaFree of more
// than the driver's 2 MB chunks map and unmap memory: 0.3-1 ms and 0.3-3 ms
// here (1 MB to 256 MB), as much as a small batch's run, and a search makes
// and drops a batch per generation.  Allocations of up to kPoolKeep come
// from a stream-ordered pool of the device that keeps at most kPoolKeep
// (0.3 % of the GPU's memory) mapped once they are freed (1 us each then);
// larger ones, and any the pool cannot serve, are plain cudaMalloc, for which
// the pool gives back what it keeps when the device has no room.  The
// pool is the driver's own object: calls from several threads are safe, and
// an allocation is freed only after the device has been synchronised, so no
// stream can still use it.
//
// A program may load a library per model; they share one pool per device.
// The table below is a static of an inline function of default visibility,
// which the compiler emits as a unique symbol: the dynamic linker keeps one
// copy for all libraries of a process, locally loaded ones included.  (Its
// name carries a version: raise it when the table's layout changes.)
constexpr size_t kPoolKeep = size_t(512) << 20;

struct __attribute__((visibility("default"))) DevicePool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;  // orders the pool's allocations and frees
};

struct __attribute__((visibility("default"))) PoolTable {
  static constexpr int kDevices = 64;
  std::mutex mu;
  DevicePool pools[kDevices];
  bool tried[kDevices] = {};
};

__attribute__((visibility("default"))) inline PoolTable& pool_table_v1() {
  static PoolTable table;
  return table;
}

// The device's pool; without one (pool null) where the driver makes none.
inline DevicePool device_pool(int device) {
  PoolTable& t = pool_table_v1();
  if (device < 0 || device >= PoolTable::kDevices) return {};
  std::lock_guard<std::mutex> lock(t.mu);
  if (!t.tried[device]) {
    t.tried[device] = true;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    DevicePool made;
    uint64_t keep = kPoolKeep;
    if (cudaMemPoolCreate(&made.pool, &props) == cudaSuccess &&
        cudaMemPoolSetAttribute(made.pool, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess &&
        cudaStreamCreateWithFlags(&made.stream, cudaStreamNonBlocking) == cudaSuccess)
      t.pools[device] = made;
    else
      cudaGetLastError();
  }
  return t.pools[device];
}

}  // namespace dense_b200
