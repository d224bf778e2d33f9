// chip_engine.h -- host side of the on-chip engine (chip_engine.cuh).
#pragma once
#include <cuda_runtime.h>

#include "acs_dev.cuh"

namespace acs {

// 256 threads: with 512 the 128 registers a thread spill (64 cases at 153 x 153, FAST: 310 us per
// pseudo-iteration against 273; 8 such cases, EXACT: 114 against 98; 51 x 51: 6.3 against 5.6)
constexpr int CHIP_THREADS = 256;
constexpr int CHIP_MAX_SMEM = 227 * 1024 - 2048;  // dynamic shared memory (the rest: static words)

// Modelled time of one pseudo-iteration (us): a constant and a slope per node of the largest strip.
// Measured, full equation set: FAST 102 x 102 in 15 CTAs (714 nodes) 15.6, 101 x 147 in 16 (1010 nodes)
// 18.7; EXACT 51 x 84 in 16 (306 nodes) 17.7, 153 x 153 in 16 (1530 nodes) 49.
constexpr double CHIP_T0_FAST = 9.0, CHIP_T1_FAST = 0.0095;
constexpr double CHIP_T0_EXACT = 10.0, CHIP_T1_EXACT = 0.025;

struct ChipArgs {
  const CaseDev* cs;
  CaseCtl* ctl;
  const int* cases;  // case id per cluster
  int* iters;        // [case * n_steps + step]
  double* err;
  int corner_role;   // role of the vm buffer whose history gives vm(imax, jmax+1) (see k_chip)
  bool tc_of_failed;  // a failed case's T and C n_tau arrays get the failing iteration's values (tile engine)
};

// Shared-memory layout of one CTA, offsets in doubles, the same in every CTA of a cluster: strips of
// at most `rows` node rows.
struct ChipLayout {
  int rows, uv_size, p_size, tc_size, own_size;
  int u, v, p, t, c, phys, w, met, mask, total;
};

__host__ __device__ inline ChipLayout chip_layout(int nx, int ny, int pitch, int K, bool scal, bool phys) {
  ChipLayout L;
  L.rows = (ny + 1 + K - 1) / K;
  L.uv_size = (L.rows + 4) * pitch;
  L.p_size = (L.rows + 1) * pitch;
  L.tc_size = (L.rows + 2) * pitch;
  L.own_size = L.rows * pitch;
  int o = 0;
  L.u = o; o += 3 * L.uv_size;
  L.v = o; o += 3 * L.uv_size;
  L.p = o; o += 2 * L.p_size;
  L.t = o; if (scal) o += 3 * L.tc_size;
  L.c = o; if (scal) o += 3 * L.tc_size;
  L.phys = o; if (phys) o += (scal ? 4 : 2) * L.own_size;
  L.w = o; if (phys) o += L.own_size;
  L.met = o;
  o += 4 * (nx + 2) + 4 * (L.rows + 2);  // four components per column 0..nx+1 and row r0-1..r1
  L.mask = o; o += (L.own_size + 7) / 8;
  L.total = o;
  return L;
}

// Launch `nclusters` clusters of `cluster` CTAs; cluster c handles case a.cases[c].  phys: the
// physical-step arrays lie in shared memory too; quick: CaseDev::scheme is 0.
cudaError_t launch_chip_exact(const ChipArgs& a, int cluster, int nclusters, bool phys, bool quick, size_t smem,
                              cudaStream_t s);
cudaError_t launch_chip_fast(const ChipArgs& a, int cluster, int nclusters, bool phys, bool quick, size_t smem,
                             cudaStream_t s);
// Clusters of this size that the device holds at once with one CTA per SM (0: none).
int chip_resident_exact(int cluster);
int chip_resident_fast(int cluster);

}  // namespace acs
