// Instantiates the packed GEMV for one stream width; included by packed_gemv_k<K>.cu with HTR_INST_K set.
#include "packed_gemv.cuh"
#include "packed_gemv1.cuh"

namespace htr {

// dynamic shared memory beyond 48 KB needs an opt-in, done once per device and instantiation
template <int K, int MT, bool DEP>
static int allow_smem() {
  static bool done[64] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev >= 0 && dev < 64 && done[dev]) return 0;
  e = cudaFuncSetAttribute(packed_gemv_kernel<K, MT, DEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemv_smem_bytes<K, MT>());
  if (e != cudaSuccess) return (int)e;
  if (dev >= 0 && dev < 64) done[dev] = true;
  return 0;
}

template <int K, int MT, bool DEP>
static int launch_one(const GemvParams& p, int grid, cudaStream_t stream) {
  if (const int e = allow_smem<K, MT, DEP>()) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = p.split > 0 ? dim3(p.split, grid / p.split) : dim3(grid);   // split form: (parts of a row block, row blocks)
  cfg.blockDim = dim3(kGemvThreads);
  cfg.dynamicSmemBytes = gemv_smem_bytes<K, MT>();
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = gemv_overlap_enabled() ? 1 : 0;
  GemvParams q = p;
  if (p.split == 0) set_flat_runs(q, grid);
  return (int)cudaLaunchKernelEx(&cfg, packed_gemv_kernel<K, MT, DEP>, q);
}

template <int K, int MT>
static int occupancy_one() {
  int ctas = 0;
  if (allow_smem<K, MT, false>()) return -1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, packed_gemv_kernel<K, MT, false>, kGemvThreads, gemv_smem_bytes<K, MT>()) != cudaSuccess)
    return -1;
  return ctas;
}

template <>
int launch_packed_gemv<HTR_INST_K>(const GemvParams& p, int mt_rows, int grid, cudaStream_t stream) {
  switch (mt_rows) {
    case 1:
      return p.group == 0 && !p.independent ? launch_one<HTR_INST_K, 1, true>(p, grid, stream) : launch_one<HTR_INST_K, 1, false>(p, grid, stream);
    case 2: return launch_one<HTR_INST_K, 2, false>(p, grid, stream);
    case 4: return launch_one<HTR_INST_K, 4, false>(p, grid, stream);
    case 8: return launch_one<HTR_INST_K, 8, false>(p, grid, stream);
  }
  return (int)cudaErrorInvalidValue;
}

template <int HELD>
static int launch_gemv1(const GemvParams& p, int grid, cudaStream_t stream) {
  static bool allowed[64] = {false};                      // shared memory beyond 48 KB: opted in once per device
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return (int)e;
  if (dev < 0 || dev >= 64 || !allowed[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(packed_gemv1_kernel<HTR_INST_K, HELD>, cudaFuncAttributeMaxDynamicSharedMemorySize, gemv1_smem_bytes<HTR_INST_K>(kG1MaxCols));
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) allowed[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kG1Threads);
  cfg.dynamicSmemBytes = (size_t)gemv1_smem_bytes<HTR_INST_K>(p.nt * 16);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = gemv_overlap_enabled() ? 1 : 0;
  GemvParams q = p;
  const int hb = p.nt >> 3, units = (p.mt >> 3) * hb;
  q.run_q = units / grid;
  q.run_rem = units % grid;
  q.hb_magic = reciprocal(hb);
  return (int)cudaLaunchKernelEx(&cfg, packed_gemv1_kernel<HTR_INST_K, HELD>, q);
}

template <>
int launch_packed_gemv1<HTR_INST_K>(const GemvParams& p, int grid, cudaStream_t stream) {
  constexpr int kColsOfOne = kG1Warps * 128;
  const int n = p.nt * 16;
  if (n <= kColsOfOne) return launch_gemv1<1>(p, grid, stream);
  if (n <= 2 * kColsOfOne) return launch_gemv1<2>(p, grid, stream);
  if (n <= 5 * kColsOfOne) return launch_gemv1<5>(p, grid, stream);
  return launch_gemv1<(kG1MaxCols + kColsOfOne - 1) / kColsOfOne>(p, grid, stream);
}

template <>
int packed_gemv_ctas_per_sm<HTR_INST_K>(int mt_rows) {
  switch (mt_rows) {
    case 1: return occupancy_one<HTR_INST_K, 1>();
    case 2: return occupancy_one<HTR_INST_K, 2>();
    case 4: return occupancy_one<HTR_INST_K, 4>();
    case 8: return occupancy_one<HTR_INST_K, 8>();
  }
  return -1;
}

}  // namespace htr

