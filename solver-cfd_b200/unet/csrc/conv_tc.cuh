// conv_tc.cuh -- 3x3 "same" convolutions of the U-Net on tcgen05 without a gathered operand per tap.
//
//   k_conv3x3:  Y[p][n] = sum_tap sum_c X[p + tap][c] * W[n][tap*C + c]     (forward, BF16 x BF16 -> FP32)
//
// One CTA computes MT tiles of 128 pixels -- 8 columns x 16 rows each, one below the other -- for up to 256
// output channels.  The pixels of the tiles with their one-pixel border are copied to shared memory once
// (cp.async, 16-byte chunks, zero outside the canvas) as planes of 8 channels: chunk c of pixel q at
// plane c, 16 bytes * q.  That is the canonical K-major no-swizzle UMMA layout (a core matrix is 8 pixels
// of a row = 128 contiguous bytes) for every tap at once: tap (ky, kx) only moves the start address by
// (ky * (8 + 2) + kx) * 16 bytes, the stride between 8-pixel groups is one row of the window and the
// stride between the two K chunks of a step one plane.  The implicit GEMM that gathered its A operand
// for each tap read every pixel nine times through L1/L2 and spent its time on the index arithmetic of
// those copies.  The weights stream through a ring of 64-wide K slabs.  K runs tap by tap, channels
// fastest, in steps of 16, as in col(X) W^T, so results are bit-identical to the GEMM's.
//
// Bound: for few output channels the copies (each pixel is read 1.33 to 1.41 times), for many the tensor
// pipe.  Measured: see unet_gemm.cu.
#pragma once
#include "gemm_tc.cuh"

namespace unet {

constexpr int CV_W = 8, CV_H = 16;     // pixels of a tile
constexpr int CV_STAGES = 3;

struct ConvArgs {
  const __nv_bfloat16* X;   // [batch][H][W][C]
  const __nv_bfloat16* Wt;  // [N][ldw], K = tap*C + c
  int H, W, C, N, ldw;
  int tx, ty;               // tiles per row, tile groups (MT * 16 rows) per column
  int plane;                // bytes of a plane (pixels of the window * 16, an odd multiple of 16)
  float* Cf;
  __nv_bfloat16* Y;
  int ldc;
  const float* bias;
  int relu;
  int* err;
};

// Window pixels of MT tiles, and a plane of them: an odd number of 16-byte words, so the eight planes
// that eight neighbouring threads write fall into different banks.
__host__ __device__ constexpr int cv_pixels(int mt) { return (CV_W + 2) * (CV_H * mt + 2); }
__host__ __device__ constexpr int cv_plane(int mt) { return (cv_pixels(mt) | 1) * 16; }

// One row of 16 accumulator columns to global memory (see k_gemm_tc's epilogue).
template <int EPI>
__device__ __forceinline__ void store16(const uint32_t* r, int nb, int N, long long o0, const float* bias, int relu, float* C,
                                        __nv_bfloat16* Y, int ldc) {
  if (EPI == EPI_BIAS_BF16 && nb + 16 <= N && (ldc & 7) == 0 && !(reinterpret_cast<uintptr_t>(Y) & 15)) {
    uint32_t pk[8];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      float v0 = __uint_as_float(r[j]) + (bias ? __ldg(bias + nb + j) : 0.f);
      float v1 = __uint_as_float(r[j + 1]) + (bias ? __ldg(bias + nb + j + 1) : 0.f);
      if (relu) { v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); }
      const __nv_bfloat162 h = __floats2bfloat162_rn(v0, v1);
      pk[j >> 1] = *reinterpret_cast<const uint32_t*>(&h);
    }
    uint4* dst = reinterpret_cast<uint4*>(Y + o0);
    dst[0] = make_uint4(pk[0], pk[1], pk[2], pk[3]);
    dst[1] = make_uint4(pk[4], pk[5], pk[6], pk[7]);
    return;
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const int n = nb + j;
    if (n >= N) break;
    float v = __uint_as_float(r[j]);
    if (EPI == EPI_STORE_F32) C[o0 + j] = v;
    else if (EPI == EPI_BIAS_F32) C[o0 + j] = v + (bias ? __ldg(bias + n) : 0.f);
    else {
      v += bias ? __ldg(bias + n) : 0.f;
      if (relu) v = fmaxf(v, 0.f);
      Y[o0 + j] = __float2bfloat16_rn(v);
    }
  }
}

__device__ __forceinline__ void tmem_ld16(uint32_t* r, uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ void mma_f16(uint32_t tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(tmem), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(0), "r"(0), "r"(0), "r"(0));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Copies the window of `rows` x (8 + 2) pixels whose top-left pixel is (y0 - 1, x0 - 1) of image b: C / 8
// chunks per pixel, chunk fastest so that neighbouring threads read neighbouring addresses.
__device__ __forceinline__ void load_window(uint32_t sx, int plane, const __nv_bfloat16* X, int b, int H, int W, int C, int y0,
                                            int x0, int rows) {
  const int c8 = C >> 3, total = (CV_W + 2) * rows * c8;
  int q = threadIdx.x / c8, c = threadIdx.x - q * c8;       // pixel of the window, chunk
  const int dq = blockDim.x / c8, dc = blockDim.x - dq * c8;
  const long long img = (long long)b * H * W;
  for (int v = threadIdx.x; v < total; v += blockDim.x) {
    const int wy = q / (CV_W + 2), wx = q - wy * (CV_W + 2);
    const int y = y0 - 1 + wy, x = x0 - 1 + wx;
    const bool ok = y >= 0 && y < H && x >= 0 && x < W;
    const __nv_bfloat16* src = ok ? X + (img + (long long)y * W + x) * C + 8 * c : X;
    cp_async16(sx + (uint32_t)(c * plane + q * 16), src, ok);
    q += dq;
    c += dc;
    if (c >= c8) { c -= c8; q += 1; }
  }
}

template <int BN, int MT, int EPI>
__global__ void __launch_bounds__(TC_THREADS) k_conv3x3(ConvArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int S = CV_STAGES;
  constexpr int B_BYTES = BN * TC_BK * 2;
  constexpr int TMEM_COLS = BN * MT < 32 ? 32 : BN * MT;
  // [window planes][S weight slabs]; the barriers and the TMEM address are static
  __shared__ unsigned long long bars[S];
  __shared__ uint32_t tmem_holder;
  __shared__ int wait_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int K = 9 * a.C, nk = (K + TC_BK - 1) / TC_BK;
  int t = blockIdx.x;
  const int txi = t % a.tx;
  t /= a.tx;
  const int tyi = t % a.ty, b = t / a.ty;
  const int x0 = txi * CV_W, y0 = tyi * CV_H * MT;
  const uint32_t sx = smem_u32(smem), sw = sx + (uint32_t)((a.C >> 3) * a.plane);

  if (threadIdx.x == 0) {
    for (int q = 0; q < S; ++q) mbar_init(smem_u32(&bars[q]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  load_window(sx, a.plane, a.X, b, a.H, a.W, a.C, y0, x0, CV_H * MT + 2);
  auto load_w = [&](int s) { load_slab(sw + (uint32_t)((s % S) * B_BYTES), a.Wt, a.ldw, 0, a.N, s * TC_BK, K, BN); };
  for (int s = 0; s < S - 1; ++s) {  // the first group also holds the window
    if (s < nk) load_w(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_holder;
  constexpr uint32_t idesc = umma_idesc(TC_BM, BN);
  bool ok = true;
  uint32_t phase = 0u;
  int last_commit = -1;
  int tap = 0, c0 = 0;  // of the next K step (thread 0)
  for (int i = 0; i < nk; ++i) {
    const int st = i % S;
    asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t sb = sw + (uint32_t)(st * B_BYTES);
#pragma unroll
      for (int ks = 0; ks < TC_BK / 16; ++ks) {
        if (i * TC_BK + ks * 16 < K) {
          // channels c0..c0+15 of tap (ky, kx); with 8 channels the second chunk of a step is the next tap's
          const uint64_t db = umma_desc(sb + ks * 2 * BN * 16, BN * 16, 128);
          const int ky = tap / 3, kx = tap - 3 * ky;
          const uint32_t sa = sx + (uint32_t)((c0 >> 3) * a.plane + (ky * (CV_W + 2) + kx) * 16);
#pragma unroll
          for (int m = 0; m < MT; ++m)
            mma_f16(tmem + m * BN, umma_desc(sa + m * CV_H * (CV_W + 2) * 16, a.plane, (CV_W + 2) * 16), db, idesc,
                    i > 0 || ks > 0 ? 1u : 0u);
          c0 += 16;
          if (c0 == a.C) {
            c0 = 0;
            ++tap;
          }
        }
      }
      mma_commit(smem_u32(&bars[st]));
    }
    last_commit = i;
    const int j = i + S - 1;
    if (j < nk) {
      if (i >= 1) {
        const int sp = (i - 1) % S;
        ok = cta_wait(smem_u32(&bars[sp]), (phase >> sp) & 1u, &wait_flag);
        phase ^= 1u << sp;
        if (!ok) break;
      }
      load_w(j);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  for (int s = nk > S ? nk - S : 0; ok && s < nk; ++s) {
    const int sp = s % S;
    ok = cta_wait(smem_u32(&bars[sp]), (phase >> sp) & 1u, &wait_flag);
    phase ^= 1u << sp;
  }
  if (!ok && last_commit >= 0)  // one more bounded wait drains the MMAs issued (see k_gemm_tc)
    cta_wait(smem_u32(&bars[last_commit % S]), (uint32_t)((last_commit / S) & 1), &wait_flag);
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (!ok) {
    if (threadIdx.x == 0 && a.err) atomicExch(a.err, 1);
  } else {
    const int m = warp * 32 + lane;  // pixel of the tile
    const int x = x0 + (m & 7);
#pragma unroll 1
    for (int q = 0; q < MT; ++q) {
      const int y = y0 + q * CV_H + (m >> 3);
      const long long row = ((long long)b * a.H + y) * a.W + x;
#pragma unroll 1
      for (int n = 0; n < BN; n += 16) {
        uint32_t r[16];
        tmem_ld16(r, tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(q * BN + n));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (x < a.W && y < a.H && n < a.N) store16<EPI>(r, n, a.N, row * a.ldc + n, a.bias, a.relu, a.Cf, a.Y, a.ldc);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
}

}  // namespace unet
