// lm_launch.cu -- what a launch needs of the driver beforehand: the kernel's
// limit of dynamic shared memory and its occupancy.  Host code alone.
#include <map>
#include <mutex>
#include <utility>

#include "lm_internal.h"

namespace lm {

cudaError_t grow_smem_limit(const void *kern, size_t smem) {
  // (compared and set under the lock: a thread that asks for less may not
  // come between another's call and its launch)
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, size_t> limits;
  // the 48 KB that need no attribute hold the static shared memory too (16 KB
  // of row offsets at most)
  if (smem < 32 * 1024) return cudaSuccess;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  size_t &limit = limits[{kern, dev}];
  if (limit >= smem) return cudaSuccess;
  const cudaError_t err = cudaFuncSetAttribute(
      kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (err == cudaSuccess)
    limit = smem;
  else
    cudaGetLastError();  // (not for the check after a later launch to find)
  return err;
}

int prepare_launch(const void *kern, LaunchCache &c, size_t smem, int threads,
                   cudaError_t *err) {
  *err = cudaSuccess;
  int dev = 0;
  cudaGetDevice(&dev);
  const int d = dev & 63;
  const int need = (int)smem + 1;
  if (c.smem_set[d].load(std::memory_order_acquire) < need) {
    if ((*err = grow_smem_limit(kern, smem)) != cudaSuccess) return 0;
    int cur = c.smem_set[d].load();
    while (cur < need && !c.smem_set[d].compare_exchange_weak(cur, need)) {
    }
  }
  const uint64_t key = c.occ_key[d].load(std::memory_order_acquire);
  if (key && (key >> 16) == (uint64_t)smem) return (int)(key & 0xffff);
  int occ = 0;
  if ((*err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, threads,
                                                            smem)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  c.occ_key[d].store(((uint64_t)smem << 16) | (uint64_t)(occ & 0xffff),
                     std::memory_order_release);
  return occ;
}

}  // namespace lm
