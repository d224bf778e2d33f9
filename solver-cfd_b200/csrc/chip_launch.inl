// chip_launch.inl -- launcher of k_chip, included by chip_fast.cu and chip_exact.cu inside namespace acs
// after `PT` (the arithmetic), CHIP_LAUNCH and CHIP_RESIDENT (the functions' names) are set.
namespace {

template <bool PHYS, bool QUICK>
cudaError_t chip_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, int cluster, int nclusters, size_t smem,
                        cudaStream_t s) {
  auto kern = k_chip<PT, PHYS, QUICK>;
  // attributes belong to the kernel, for every thread of the process: the same values at each launch
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CHIP_MAX_SMEM);
  if (e != cudaSuccess) return e;
  cfg = {};
  cfg.gridDim = dim3(cluster * nclusters);
  cfg.blockDim = dim3(CHIP_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaSuccess;
}

template <bool PHYS, bool QUICK>
cudaError_t launch_t(const ChipArgs& a, int cluster, int nclusters, size_t smem, cudaStream_t s) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  cudaError_t e = chip_config<PHYS, QUICK>(cfg, attr, cluster, nclusters, smem, s);
  return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, k_chip<PT, PHYS, QUICK>, a) : e;
}

}  // namespace

cudaError_t CHIP_LAUNCH(const ChipArgs& a, int cluster, int nclusters, bool phys, bool quick, size_t smem, cudaStream_t s) {
  if (quick) return phys ? launch_t<true, true>(a, cluster, nclusters, smem, s) : launch_t<false, true>(a, cluster, nclusters, smem, s);
  return phys ? launch_t<true, false>(a, cluster, nclusters, smem, s) : launch_t<false, false>(a, cluster, nclusters, smem, s);
}

int CHIP_RESIDENT(int cluster) {
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int n = 0;
  if (chip_config<false, true>(cfg, attr, cluster, 1, CHIP_MAX_SMEM, nullptr) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, k_chip<PT, false, true>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}
