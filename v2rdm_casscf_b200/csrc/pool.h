// Device and pinned host memory of the solver's calls.
//
// Every v2g_update_xz, solve and block product allocates its workspaces and
// gives them back at its end.  With cudaMalloc / cudaFree and cudaMallocHost /
// cudaFreeHost that was most of a short call (a projection of ten orbitals on a
// B200: 0.5 ms of kernels in a 10 ms call; a block product of 19 x 800: 0.25 in
// 1.8 to 12 ms), so both come from pools of the library's own, bounded by what
// they may hold while unused.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace v2g {

// Unused bytes the pools keep while a PoolOwner lives: device memory per device
// beyond which it goes back to the system at the next synchronisation, pinned
// memory in all.
constexpr size_t kPoolKeep = size_t(1) << 30;
constexpr size_t kPinnedKeep = size_t(16) << 20;

// Device memory on the current device, ordered by the legacy default stream:
// streams created without cudaStreamNonBlocking may use it right away and
// need not be drained before it is freed; for the others synchronise the
// default stream after the allocation and the stream before the free.
cudaError_t pool_alloc(void** p, size_t bytes);
void pool_free(void* p, int device);  // device: where it was allocated

// Device memory outside the pool, for what a caller's streams may still read when
// its owner goes: device_free waits for the device, whatever the stream.
cudaError_t device_alloc(void** p, size_t bytes);
void device_free(void* p, int device);

// Device memory that the pool holds unused: it serves the pool's next allocations,
// beside what the device has free.
size_t pool_idle(int device);

// Handles and networks own one each; when the last goes, the pools give back all
// that they hold unused.
struct PoolOwner {
    PoolOwner();
    ~PoolOwner();
    PoolOwner(const PoolOwner&) = delete;
    PoolOwner& operator=(const PoolOwner&) = delete;
};

// Page-locked host memory, in powers of two.  Give back only what no copy in
// flight uses.
cudaError_t pinned_alloc(void** p, size_t bytes);
void pinned_free(void* p, size_t bytes);

}  // namespace v2g
