// transfer.h -- field transfers through a contiguous staging buffer (transfer.cu).
#pragma once
#include <cuda_runtime.h>

#include "acs_dev.cuh"

namespace acs {

constexpr int MOVE_MAX = 14;

struct FieldMove {
  double* dev;    // first node of the field in the case's buffer
  long long off;  // of the contiguous field in the staging buffer (doubles)
  int w, h;
};
struct MoveList {
  FieldMove f[MOVE_MAX];
  int n, pitch;
  long long total;  // doubles of all fields
};

// Staging buffer -> case buffers; *ctl = value where ctl is given.
void move_to_case(const MoveList& m, double* stage, CaseCtl* ctl, const CaseCtl& value, cudaStream_t s);
// Case buffers -> staging buffer; where ctl is given its three residuals follow the fields (m.total) and
// the case is marked inactive.
void move_from_case(const MoveList& m, double* stage, CaseCtl* ctl, cudaStream_t s);

}  // namespace acs
