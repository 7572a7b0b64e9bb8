// Instantiates the tensor-core packed GEMM for one stream width; included by packed_gemm_tc_k<K>.cu with HTR_INST_K set.
#include <map>
#include <mutex>
#include <tuple>

#include "packed_gemm_tc.cuh"

namespace htr {
namespace {

// the grouped form's stages all fit at its 16 rows and two planes, whatever the width
static_assert(gemm_smem_bytes(kGroupRows, 2, kGemmMaxStages, GemmRing<HTR_INST_K>::bytes) <= kGemmGroupSmem, "grouped GEMM: rings beyond the opt-in");

// shared memory beyond 48 KB: opted in once per device (the 227 KB limit includes the static part)
int allow_smem(int dev) {
  static bool allowed[64] = {false};
  if (dev >= 0 && dev < 64 && allowed[dev]) return 0;
  const cudaError_t e = cudaFuncSetAttribute(packed_gemm_tc_kernel<HTR_INST_K, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmSmem);
  if (e != cudaSuccess) return (int)e;
  const cudaError_t e2 = cudaFuncSetAttribute(packed_gemm_tc_kernel<HTR_INST_K, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmGroupSmem);
  if (e2 != cudaSuccess) return (int)e2;
  const cudaError_t e3 = cudaFuncSetAttribute(packed_gemm_tc_kernel<HTR_INST_K, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);   // up to 16
  if (e3 != cudaSuccess) return (int)e3;
  if (dev >= 0 && dev < 64) allowed[dev] = true;
  return 0;
}

}  // namespace

template <>
int packed_gemm_tc_clusters<HTR_INST_K>(int smem, int split) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  // the query costs tens of microseconds on the host: remember the answer
  static std::mutex mu;
  static std::map<std::tuple<int, int, int>, int> seen;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(dev, smem, split);
  const auto it = seen.find(key);
  if (it != seen.end()) return it->second;
  int clusters = 0;
  if (allow_smem(dev) == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)split);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)split;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&clusters, packed_gemm_tc_kernel<HTR_INST_K, false>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      clusters = 0;
    }
  }
  seen[key] = clusters;
  return clusters;
}

template <>
int launch_packed_gemm_tc<HTR_INST_K>(const GemmParams& p, int grid, int smem, cudaStream_t st) {
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return (int)e;
  if (const int e = allow_smem(dev)) return e;
  // programmatic stream serialisation: the kernel may start while the activation transform before it still runs; it
  // fetches packed words at once and waits (griddepcontrol.wait) before it touches anything that kernel writes
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (p.split > 1) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)p.split;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
  }
  GemmParams q = p;
  void* args[1] = {&q};
  return (int)cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(p.plan ? packed_gemm_tc_kernel<HTR_INST_K, true> : packed_gemm_tc_kernel<HTR_INST_K, false>), args);
}

}  // namespace htr
