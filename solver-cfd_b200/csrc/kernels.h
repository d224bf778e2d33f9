// kernels.h -- kernel declarations shared between the kernel sources and the host launcher.
#pragma once
#include <cuda_runtime.h>
#include "acs_dev.cuh"

namespace acs {

// exact-arithmetic path (kernels_exact.cu); launchers so no kernel template crosses units.
// stage = 1..3; `is_c` selects solve_C (true) or solve_Z (false).
void launch_u_stage_exact(int stage, const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
void launch_v_stage_exact(int stage, const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
void launch_s_stage_exact(bool is_c, int stage, const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
void launch_p_exact(const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
// FAST-arithmetic per-stage kernels (kernels_fast.cu), same launch structure
void launch_u_stage_fast(int stage, const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
void launch_v_stage_fast(int stage, const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
void launch_s_stage_fast(bool is_c, int stage, const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
void launch_p_fast(const CaseDev*, CaseCtl*, const Tile*, int ntiles, cudaStream_t);
// boundary passes, one block per case (see kernels_exact.cu for `which`)
void launch_bc_uv(const CaseDev*, const CaseCtl*, int ncases, int which, cudaStream_t);
void launch_bc_cell(const CaseDev*, const CaseCtl*, int ncases, int which, cudaStream_t);

// cell-centred u, v (comp_mean) and |U| of one case (output.cu)
cudaError_t launch_cell_fields(const double* um, const double* vm, int nx, int ny, int pitch, double* u, double* v,
                               double* mag, cudaStream_t s);

// loop control (control.cu)
enum LoopMode { LOOP_COND = 1, LOOP_FLAG = 2 };
struct LoopEnd {
  int mode;                           // what the last block does with the number of active cases
  int tau_bc;                         // 1: apply the first iteration's side effects on um_tau, vm_tau
  cudaGraphConditionalHandle handle;  // LOOP_COND
  long long max_iters;
  long long* iter_count;
  int* ticket;                        // blocks done (0 between launches)
  int* host_flag;                     // LOOP_FLAG
};
__global__ void k_control(const CaseDev*, CaseCtl*, int* iters, double* err, int* n_active, LoopEnd end);

}  // namespace acs
