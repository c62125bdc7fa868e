// Library-wide helpers: status strings, ABI version, device SM count.
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "qsgb_common.cuh"

namespace qsgb {

int sm_count() {
  static int cache[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return kNumSMs;
  if (cache[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = kNumSMs;
    cache[dev] = n;
  }
  return cache[dev];
}

int allow_dynamic_smem(const void* func, int bytes) {
  if (bytes <= 48 * 1024) return QSGB_OK;
  struct Entry {
    const void* func;
    int dev, bytes;
  };
  static std::mutex mu;
  static std::vector<Entry> table;
  int dev = 0;
  QSGB_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  for (Entry& e : table) {
    if (e.func == func && e.dev == dev) {
      if (bytes <= e.bytes) return QSGB_OK;
      QSGB_CUDA_TRY(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
      e.bytes = bytes;
      return QSGB_OK;
    }
  }
  QSGB_CUDA_TRY(cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  table.push_back({func, dev, bytes});
  return QSGB_OK;
}

int resident_blocks(const void* func, int threads, size_t smem) {
  static std::mutex mu;
  static std::map<std::tuple<const void*, int, int, size_t>, int> known;
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const auto key = std::make_tuple(func, dev, threads, smem);
  std::lock_guard<std::mutex> lock(mu);
  const auto it = known.find(key);
  if (it != known.end()) return it->second;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, func, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;  // asked again next time
  }
  known.emplace(key, n);  // as many as there are kernels
  return n;
}

// A grid that takes more than half of the device's resident blocks, but not all,
// is placed badly while its predecessor of the same kind still holds its share:
// the first SMs to become free are filled, the last get few, and a pass takes as
// long as a full SM.  Measured on GB300, chains of one kernel in a graph, us a
// pass overlapped / not, by blocks per SM: one-qubit FP64 PTM (10 resident) 5:
// 3.2 / 3.6, 6: 4.7 / 3.9, 8: 4.8 / 4.5, 9: 4.5 / 4.9, 16: 6.9 / 7.3; noisy CZ
// with rotations (3 resident) 1: 4.0 / 4.4, 2: 9.1 / 6.8, 4: 11.5 / 11.7; two
// layers of 10 qubits 147 / 126.
static bool placed_well(const void* func, dim3 grid, dim3 block, size_t smem) {
  const uint64_t blocks = (uint64_t)grid.x * grid.y * grid.z, sms = (uint64_t)sm_count();
  if (blocks <= sms || blocks >= 32 * sms) return true;  // no look-up for the smallest calls
  const uint64_t full = sms * (uint64_t)resident_blocks(func, (int)(block.x * block.y * block.z), smem);
  return 2 * blocks <= full || blocks >= full;
}

int launch_pdl(const void* func, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, void** args, bool overlap) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap && placed_well(func, grid, block, smem) ? 1 : 0;
  QSGB_CUDA_TRY(cudaLaunchKernelExC(&cfg, func, args));
  return QSGB_OK;
}

int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? QSGB_OK : QSGB_ERR_CUDA;
}

}  // namespace qsgb

extern "C" int qsgb_abi_version(void) { return 2; }

extern "C" const char* qsgb_status_string(int status) {
  switch (status) {
    case QSGB_OK:
      return "ok";
    case QSGB_ERR_INVALID:
      return "invalid argument";
    case QSGB_ERR_CUDA:
      return "CUDA runtime error";
    case QSGB_ERR_UNSUPPORTED:
      return "unsupported shape or configuration";
    case QSGB_ERR_SCRATCH:
      return "scratch buffer too small";
    default:
      return "unknown status";
  }
}
