// unet_gemm.cu -- host launcher of the tcgen05 GEMM (gemm_tc.cuh) behind the C ABI in unet.h.
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include "../../../include/unet.h"
#include "conv_tc.cuh"
#include "gemm_tc.cuh"

namespace unet {
namespace {

template <int BN, int EPI, bool CONV = false>
cudaError_t go(const GemmArgs& a, int splits, cudaStream_t s) {
  constexpr int smem = TC_STAGES * (TC_BM * TC_BK * 2 + BN * TC_BK * 2) + 64;
  auto k = k_gemm_tc<BN, EPI, CONV>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  dim3 grid((a.M + TC_BM - 1) / TC_BM, (a.N + BN - 1) / BN, splits);
  k<<<grid, TC_THREADS, smem, s>>>(a);
  return cudaGetLastError();
}

template <int EPI, bool CONV = false>
cudaError_t by_bn(const GemmArgs& a, int bn, int splits, cudaStream_t s) {
  switch (bn) {
    case 16: return go<16, EPI, CONV>(a, splits, s);
    case 32: return go<32, EPI, CONV>(a, splits, s);
    case 64: return go<64, EPI, CONV>(a, splits, s);
    case 128: return go<128, EPI, CONV>(a, splits, s);
    default: return go<256, EPI, CONV>(a, splits, s);
  }
}

constexpr int kConvSmem = 226 * 1024;  // dynamic shared memory of a convolution CTA

// Tensor map of the weights [N][ldw] (K of a row used): boxes of 64 k x bn rows in the 128-byte swizzle, zero
// outside.
bool weight_map(CUtensorMap* m, const void* Wt, int N, int K, int ldw, int bn) {
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q{};
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn ||
      q != cudaDriverEntryPointSuccess)
    return false;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
  const cuuint64_t strides[1] = {(cuuint64_t)ldw * 2};
  const cuuint32_t box[2] = {TC_BK, (cuuint32_t)bn}, estr[2] = {1, 1};
  return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn)(
             m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(Wt), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct ConvCall {
  ConvArgs a;
  const void* Wt;
  int ldw, batch;
  cudaStream_t s;
};

// Shared memory: alignment, the weight ring (bn: output channels of a CTA) and the window's planes.
int conv_smem(int C, int bn, int mt) { return 1024 + cv_stages(bn) * bn * TC_BK * 2 + (C >> 3) * cv_plane(mt); }
// the same for the gathering variant: planes of col(X), the window as it is
constexpr int kGatherPlane = (TC_BM | 1) * 16;
int gather_smem(int C, int K, int bn) {
  return 1024 + cv_stages(bn) * bn * TC_BK * 2 + (K + 15) / 16 * 2 * kGatherPlane + cv_pixels(1) * C * 2;
}

template <int BN, int MT, int EPI, bool GATHER>
cudaError_t conv_go(const ConvCall& c) {
  ConvArgs a = c.a;
  a.plane = GATHER ? kGatherPlane : cv_plane(MT);
  a.tx = (a.W + CV_W - 1) / CV_W;
  a.ty = (a.H + CV_H * MT - 1) / (CV_H * MT);
  const int smem = GATHER ? gather_smem(a.C, a.K, BN) : conv_smem(a.C, BN, MT);
  auto k = k_conv3x3<BN, MT, EPI, GATHER>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  CUtensorMap map;
  if (!weight_map(&map, c.Wt, a.N, a.K, c.ldw, BN)) return cudaErrorInvalidValue;
  k<<<dim3((unsigned)(c.batch * a.ty * a.tx)), TC_THREADS, smem, c.s>>>(map, a);
  return cudaGetLastError();
}

// Two tiles per CTA share the weight slabs and the window's border where two such CTAs still fit on an SM
// and there are enough of them to fill the device four times; else one.
template <int BN, int EPI>
cudaError_t conv_mt(const ConvCall& c) {
  const ConvArgs& a = c.a;
  const long long ctas2 = (long long)c.batch * ((a.H + 2 * CV_H - 1) / (2 * CV_H)) * ((a.W + CV_W - 1) / CV_W);
  if (BN <= 128 && conv_smem(a.C, BN, 2) <= kConvSmem / 2 && ctas2 >= 4 * 148) return conv_go<BN, BN <= 128 ? 2 : 1, EPI, false>(c);
  return conv_go<BN, 1, EPI, false>(c);
}

template <int EPI>
cudaError_t conv_bn(const ConvCall& c, int bn) {
  switch (bn) {
    case 16: return conv_mt<16, EPI>(c);
    case 32: return conv_mt<32, EPI>(c);
    case 64: return conv_mt<64, EPI>(c);
    case 128: return conv_mt<128, EPI>(c);
    default: return conv_mt<256, EPI>(c);
  }
}

ConvArgs conv_args(const void* X, int H, int W, int C, int K, int Cout, float* Cf, void* Y, int ldc, const float* bias,
                   int relu, int* err) {
  ConvArgs c{};
  c.X = static_cast<const __nv_bfloat16*>(X);
  c.H = H; c.W = W; c.C = C; c.N = Cout; c.K = K;
  c.Cf = Cf; c.Y = static_cast<__nv_bfloat16*>(Y); c.ldc = ldc; c.bias = bias; c.relu = relu; c.err = err;
  return c;
}

}  // namespace
}  // namespace unet

extern "C" int unet_gemm(const void* A, int lda, const void* B, int ldb, int M, int N, int K, int epilogue,
                         float* C, void* Y, int ldc, const float* bias, int relu, int splits, int* err,
                         void* stream) {
  using namespace unet;
  if (!A || !B || M <= 0 || N <= 0 || K <= 0 || (K & 7) || (lda & 7) || (ldb & 7) || lda < K || ldb < K)
    return 1;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return 1;
  if (epilogue < 0 || epilogue > 3 || splits < 1) return 1;
  if ((epilogue == EPI_BIAS_BF16 && !Y) || (epilogue != EPI_BIAS_BF16 && !C)) return 1;
  int bn = 16;
  while (bn < N && bn < 256) bn *= 2;
  const int kt = (K + TC_BK - 1) / TC_BK;
  if (splits > kt) splits = kt;
  GemmArgs a;
  a.A = static_cast<const __nv_bfloat16*>(A);
  a.B = static_cast<const __nv_bfloat16*>(B);
  a.M = M; a.N = N; a.K = K; a.lda = lda; a.ldb = ldb;
  a.C = C; a.Y = static_cast<__nv_bfloat16*>(Y); a.ldc = ldc; a.bias = bias; a.relu = relu;
  a.k_tiles_per_split = (kt + splits - 1) / splits;
  a.cH = a.cW = a.cC = 0;
  splits = (kt + a.k_tiles_per_split - 1) / a.k_tiles_per_split;
  a.err = err;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  switch (epilogue) {
    case EPI_STORE_F32: e = by_bn<EPI_STORE_F32>(a, bn, splits, s); break;
    case EPI_ATOMIC_F32: e = by_bn<EPI_ATOMIC_F32>(a, bn, splits, s); break;
    case EPI_BIAS_BF16: e = by_bn<EPI_BIAS_BF16>(a, bn, splits, s); break;
    default: e = by_bn<EPI_BIAS_F32>(a, bn, splits, s); break;
  }
  return e == cudaSuccess ? 0 : 3;
}

extern "C" int unet_conv3x3(const void* X, int B, int H, int W, int C, const void* Wt, int ldw, int Cout, int epilogue,
                            float* Cf, void* Y, int ldc, const float* bias, int relu, int* err, void* stream) {
  using namespace unet;
  if (!X || !Wt || B <= 0 || H <= 0 || W <= 0 || C <= 0 || (C & 7) || Cout <= 0 || (ldw & 7) || ldw < 9 * C)
    return 1;
  if ((reinterpret_cast<uintptr_t>(X) & 15) || (reinterpret_cast<uintptr_t>(Wt) & 15)) return 1;
  if (epilogue != EPI_STORE_F32 && epilogue != EPI_BIAS_BF16 && epilogue != EPI_BIAS_F32) return 1;
  if ((epilogue == EPI_BIAS_BF16 && !Y) || (epilogue != EPI_BIAS_BF16 && !Cf)) return 1;
  const long long M = (long long)B * H * W;
  if (M > 0x7fffffffLL) return 1;
  int bn = 16;
  while (bn < Cout && bn < 256) bn *= 2;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e;
  // The window kernel takes whole K steps of one tap (C a multiple of 16), one column of CTAs (Cout up
  // to 256) and a window that fits in shared memory; the rest goes through the gathering GEMM.
  if (C % 16 == 0 && Cout <= 256 && conv_smem(C, bn, 1) <= kConvSmem) {
    ConvCall c{conv_args(X, H, W, C, 9 * C, Cout, Cf, Y, ldc, bias, relu, err), Wt, ldw, B, s};
    switch (epilogue) {
      case EPI_STORE_F32: e = conv_bn<EPI_STORE_F32>(c, bn); break;
      case EPI_BIAS_BF16: e = conv_bn<EPI_BIAS_BF16>(c, bn); break;
      default: e = conv_bn<EPI_BIAS_F32>(c, bn); break;
    }
    return e == cudaSuccess ? 0 : 3;
  }
  GemmArgs a;
  a.A = static_cast<const __nv_bfloat16*>(X);
  a.B = static_cast<const __nv_bfloat16*>(Wt);
  a.M = (int)M; a.N = Cout; a.K = 9 * C; a.lda = C; a.ldb = ldw;
  a.C = Cf; a.Y = static_cast<__nv_bfloat16*>(Y); a.ldc = ldc; a.bias = bias; a.relu = relu;
  a.k_tiles_per_split = (a.K + TC_BK - 1) / TC_BK;
  a.err = err;
  a.cH = H; a.cW = W; a.cC = C;
  switch (epilogue) {
    case EPI_STORE_F32: e = by_bn<EPI_STORE_F32, true>(a, bn, 1, s); break;
    case EPI_BIAS_BF16: e = by_bn<EPI_BIAS_BF16, true>(a, bn, 1, s); break;
    default: e = by_bn<EPI_BIAS_F32, true>(a, bn, 1, s); break;
  }
  return e == cudaSuccess ? 0 : 3;
}

extern "C" int unet_conv3x3_gather(const void* X, int B, int H, int W, int C, const void* Wt, int ldw, int Kp, int Cout,
                                   void* Y, int ldc, const float* bias, int relu, int* err, void* stream) {
  using namespace unet;
  if (!X || !Wt || !Y || B <= 0 || H <= 0 || W <= 0 || C <= 0 || Cout <= 0 || Cout > 64 || (ldw & 7) || ldw < Kp ||
      Kp != (9 * C + 7) / 8 * 8 || (reinterpret_cast<uintptr_t>(Wt) & 15) || (long long)B * H * W > 0x7fffffffLL)
    return 1;
  const int bn = Cout <= 32 ? 32 : 64;
  if (gather_smem(C, Kp, bn) > kConvSmem) return 1;
  ConvCall c{conv_args(X, H, W, C, Kp, Cout, nullptr, Y, ldc, bias, relu, err), Wt, ldw, B, static_cast<cudaStream_t>(stream)};
  const cudaError_t e = bn == 32 ? conv_go<32, 1, EPI_BIAS_BF16, true>(c) : conv_go<64, 1, EPI_BIAS_BF16, true>(c);
  return e == cudaSuccess ? 0 : 3;
}
