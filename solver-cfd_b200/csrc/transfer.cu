// transfer.cu -- field transfers between contiguous host arrays and the pitched case buffers.
//
// A 2-D copy of a field whose row length differs from the pitch runs row by row (a 153 x 153 field took
// about 20 us to the device and 40 back, synchronisation included).  Fields instead cross PCIe as they are
// on the host, one contiguous copy each or one for all, and a kernel moves the rows of all of them
// between the contiguous staging buffer and the pitched buffers.
#include <cuda_runtime.h>

#include "transfer.h"

namespace acs {

namespace {

template <bool TO_CASE>
__global__ void k_move(MoveList m, double* __restrict__ stage, CaseCtl* ctl, CaseCtl value) {
  const FieldMove& f = m.f[blockIdx.y];
  const int n = f.w * f.h;
  double* s = stage + f.off;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    double* d = f.dev + (q % f.w) + (long long)(q / f.w) * m.pitch;
    if (TO_CASE) *d = s[q];
    else s[q] = *d;
  }
  if (ctl && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    if (TO_CASE) {
      *ctl = value;
    } else {  // the residuals behind the fields; the case leaves the launch
      unsigned long long* r = reinterpret_cast<unsigned long long*>(stage + m.total);
      r[0] = ctl->res_u;
      r[1] = ctl->res_v;
      r[2] = ctl->res_p;
      ctl->active = 0;
    }
  }
}

dim3 move_grid(const MoveList& m) {
  int n = 0;
  for (int q = 0; q < m.n; ++q) n = m.f[q].w * m.f[q].h > n ? m.f[q].w * m.f[q].h : n;
  const int b = (n + 255) / 256;
  return dim3((unsigned)(b < 296 ? b : 296), (unsigned)m.n);
}

}  // namespace

void move_to_case(const MoveList& m, double* stage, CaseCtl* ctl, const CaseCtl& value, cudaStream_t s) {
  k_move<true><<<move_grid(m), 256, 0, s>>>(m, stage, ctl, value);
}
void move_from_case(const MoveList& m, double* stage, CaseCtl* ctl, cudaStream_t s) {
  k_move<false><<<move_grid(m), 256, 0, s>>>(m, stage, ctl, CaseCtl{});
}

}  // namespace acs
