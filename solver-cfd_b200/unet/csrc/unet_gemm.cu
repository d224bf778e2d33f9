// unet_gemm.cu -- host launcher of the tcgen05 GEMM (gemm_tc.cuh) behind the C ABI in unet.h.
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include "../../../include/unet.h"
#include "conv_grad_tc.cuh"
#include "conv_tc.cuh"
#include "gemm_tc.cuh"

namespace unet {
// Measured on one B200 (64 canvases of 160 x 160, 4 levels, 32 base channels; us per layer, gathering
// GEMM -> k_conv3x3): level 0, 32 -> 32: 651 -> 104, 96 -> 32: 1729 -> 367; level 1, 64 -> 64: 324 -> 100,
// 192 -> 64: 916 -> 279; level 2, 128 -> 128: 251 -> 87, 384 -> 128: 721 -> 301; level 3, 256 -> 256: 326 -> 107;
// input layer 11 -> 32 (im2col + GEMM before): 1720 -> 304.  Without its MMAs the 384 -> 128 layer takes 142,
// without its window copies 260, without its stores 264: the parts overlap only across the one to four
// CTAs of an SM.
// Gradients of 16 canvases, all layers (us): dW with im2col, transposes and split-K GEMM 6600 -> k_conv_dw
// 1540; dX with the FP32 product and col2im 4950 -> k_conv_dx 1140.
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
  // (the same limit at each launch: it belongs to the kernel, for every thread of the process)
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmem);
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

template <int BN>
cudaError_t dw_go(DwArgs a, cudaStream_t s) {
  const int smem = 2 * dw_stage<BN>();
  auto k = a.W % CV_W ? k_conv_dw<BN, true> : k_conv_dw<BN, false>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  a.nco = (a.N + BN - 1) / BN;
  k<<<dim3((unsigned)((a.tiles + DW_TILES - 1) / DW_TILES), (unsigned)(3 * a.nco * ((a.C + 127) / 128))), TC_THREADS, smem, s>>>(a);
  return cudaGetLastError();
}

int dx_smem(int N, int bn) {
  const int kpad = (N + 15) / 16 * 16;
  return (kpad >> 3) * cv_plane(1) + DX_RING * bn * kpad * 2;
}
// Input channels of a CTA: all of them up to 96, else blocks of 64.
int dx_bn(int C) { return C <= 32 ? 32 : C <= 64 ? 64 : C <= 96 ? 96 : 64; }

template <int BN>
cudaError_t dx_go(const DxArgs& a, int batch, cudaStream_t s) {
  const int smem = dx_smem(a.N, BN);
  auto k = k_conv_dx<BN>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmem);
  if (e != cudaSuccess) return e;
  k<<<dim3((unsigned)(batch * a.ty * a.tx), (unsigned)((a.C + BN - 1) / BN)), TC_THREADS, smem, s>>>(a);
  return cudaGetLastError();
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

extern "C" int unet_conv3x3_dw(const void* X, const void* dZ, int B, int H, int W, int C, int Cout, float* gW, int* err,
                               void* stream) {
  using namespace unet;
  if (!X || !dZ || !gW || B <= 0 || H <= 0 || W <= 0 || C <= 0 || Cout <= 0 || (Cout & 7) ||
      (long long)B * H * W > 0x7fffffffLL)
    return 1;
  if ((reinterpret_cast<uintptr_t>(dZ) & 15) || (reinterpret_cast<uintptr_t>(gW) & 15) ||
      ((C & 7) == 0 && (reinterpret_cast<uintptr_t>(X) & 15)))
    return 1;
  DwArgs a{};
  a.X = static_cast<const __nv_bfloat16*>(X);
  a.dZ = static_cast<const __nv_bfloat16*>(dZ);
  a.batch = B; a.H = H; a.W = W; a.C = C; a.N = Cout;
  a.tx = (W + CV_W - 1) / CV_W;
  a.ty = (H + CV_H - 1) / CV_H;
  a.tiles = B * a.tx * a.ty;
  a.gW = gW;
  a.err = err;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const cudaError_t e = Cout <= 16 ? dw_go<16>(a, s) : Cout <= 32 ? dw_go<32>(a, s) : Cout <= 64 ? dw_go<64>(a, s) : dw_go<128>(a, s);
  return e == cudaSuccess ? 0 : 3;
}

extern "C" int unet_conv3x3_dx_fits(int C, int Cout) {
  return C > 0 && Cout > 0 && (Cout & 7) == 0 && unet::dx_smem(Cout, unet::dx_bn(C)) <= unet::kConvSmem;
}

extern "C" int unet_conv3x3_dx(const void* dZ, const void* Wt, int B, int H, int W, int C, int Cout, float* dX, int* err,
                               void* stream) {
  using namespace unet;
  if (!dZ || !Wt || !dX || B <= 0 || H <= 0 || W <= 0 || !unet_conv3x3_dx_fits(C, Cout) || (long long)B * H * W > 0x7fffffffLL)
    return 1;
  if ((reinterpret_cast<uintptr_t>(dZ) & 15) || (reinterpret_cast<uintptr_t>(Wt) & 15) || (reinterpret_cast<uintptr_t>(dX) & 15))
    return 1;
  DxArgs a{};
  a.dZ = static_cast<const __nv_bfloat16*>(dZ);
  a.Wt = static_cast<const __nv_bfloat16*>(Wt);
  a.H = H; a.W = W; a.C = C; a.N = Cout;
  a.tx = (W + CV_W - 1) / CV_W;
  a.ty = (H + CV_H - 1) / CV_H;
  a.plane = cv_plane(1);
  a.kpad = (Cout + 15) / 16 * 16;
  a.dX = dX;
  a.err = err;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int bn = dx_bn(C);
  const cudaError_t e = bn == 32 ? dx_go<32>(a, B, s) : bn == 96 ? dx_go<96>(a, B, s) : dx_go<64>(a, B, s);
  return e == cudaSuccess ? 0 : 3;
}
