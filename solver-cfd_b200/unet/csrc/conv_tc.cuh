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
// those copies.  The weights arrive by TMA, 64-wide K slabs in the 128-byte swizzle, through a ring with
// full / empty mbarriers: one thread loads, one issues the MMAs, nothing in the K loop synchronises the
// CTA.  K runs tap by tap, channels fastest, in steps of 16, as in col(X) W^T, so results are
// bit-identical to the GEMM's.
//   GATHER: channel counts whose steps of 16 cross taps (the network's 11-channel input).  The window
// arrives element by element and the CTA builds the rows of col(X) from it, as K-major planes.
//
// Bound: for few output channels the copies (each pixel is read 1.33 to 1.41 times) and the epilogue's
// stores, for many the tensor pipe.  Measured: see unet_gemm.cu.
#pragma once
#include <cuda.h>

#include "gemm_tc.cuh"

namespace unet {

constexpr int CV_W = 8, CV_H = 16;     // pixels of a tile
__host__ __device__ constexpr int cv_stages(int bn) { return bn > 128 ? 3 : 4; }

struct ConvArgs {
  const __nv_bfloat16* X;   // [batch][H][W][C]
  int H, W, C, N, K;        // K = 9C (GATHER: rounded up to 8)
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

// Shared-memory descriptor of a K-major operand in the 128-byte swizzle: rows of 128 bytes, 8-row groups
// 1024 bytes apart (layout type 2); a K step of 16 moves the start address by 32 bytes.
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
  uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// The 64 x BN slab of the weights at column k (a multiple of 64 elements: 16-byte aligned).
__device__ __forceinline__ void tma_weights(uint32_t dst, const CUtensorMap* map, int k, int n, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(k), "r"(n), "r"(bar)
      : "memory");
}

// GATHER: the window's elements to shared memory as they are ([pixel][C]), then row m of col(X) as planes of
// 8 k (chunk c of row m at plane c, 16 bytes * m; zero from K on).
__device__ __forceinline__ void gather_rows(unsigned char* smem, uint32_t sx, int plane, int raw, const ConvArgs& a, int b,
                                            int y0, int x0) {
  unsigned short* w = reinterpret_cast<unsigned short*>(smem + raw);
  const unsigned short* X = reinterpret_cast<const unsigned short*>(a.X);
  const int row = (CV_W + 2) * a.C, n = row * (CV_H + 2);
  for (int v = threadIdx.x; v < n; v += blockDim.x) {
    const int wy = v / row, e = v - wy * row;  // element e of window row wy
    const int y = y0 - 1 + wy, first = (x0 - 1) * a.C + e;
    const bool ok = y >= 0 && y < a.H && first >= 0 && first < a.W * a.C;
    w[v] = ok ? __ldg(X + ((long long)b * a.H + y) * a.W * a.C + first) : (unsigned short)0;
  }
  __syncthreads();
  const int m = threadIdx.x;  // 128 threads, 128 rows
  const unsigned short* p = w + ((m >> 3) * (CV_W + 2) + (m & 7)) * a.C;
  int tap = 0, c = 0;
  const unsigned short* src = p;
  const int chunks = (a.K + 15) / 16 * 2;
  for (int q = 0; q < chunks; ++q) {
    unsigned short v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] = tap < 9 ? src[c] : (unsigned short)0;
      if (++c == a.C) {
        c = 0;
        ++tap;
        src = p + (tap / 3 * (CV_W + 2) + tap % 3) * a.C;
      }
    }
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sx + (uint32_t)(q * plane + m * 16)),
                 "r"(v[0] | (unsigned)v[1] << 16), "r"(v[2] | (unsigned)v[3] << 16), "r"(v[4] | (unsigned)v[5] << 16),
                 "r"(v[6] | (unsigned)v[7] << 16)
                 : "memory");
  }
}

// Shared memory: [S weight slabs, 1024-byte aligned][planes][GATHER: raw window].
template <int BN, int MT, int EPI, bool GATHER>
__global__ void __launch_bounds__(TC_THREADS) k_conv3x3(const __grid_constant__ CUtensorMap wmap, ConvArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  constexpr int S = cv_stages(BN);
  constexpr uint32_t B_BYTES = BN * TC_BK * 2;
  constexpr int TMEM_COLS = BN * MT < 32 ? 32 : BN * MT;
  __shared__ unsigned long long full[S], empty[S], done;
  __shared__ uint32_t tmem_holder;
  __shared__ int failed;
  const uint32_t pad = (1024u - (smem_u32(smem_raw) & 1023u)) & 1023u;
  unsigned char* smem = smem_raw + pad;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = (a.K + TC_BK - 1) / TC_BK;
  int t = blockIdx.x;
  const int txi = t % a.tx;
  t /= a.tx;
  const int tyi = t % a.ty, b = t / a.ty;
  const int x0 = txi * CV_W, y0 = tyi * CV_H * MT;
  const uint32_t sw = smem_u32(smem), sx = sw + S * B_BYTES;

  if (threadIdx.x == 32) {  // weights: barriers, then the first slabs at once
    for (int q = 0; q < S; ++q) {
      mbar_init(smem_u32(&full[q]), 1);
      mbar_init(smem_u32(&empty[q]), 1);
    }
    mbar_init(smem_u32(&done), 1);
    failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int i = 0; i < S && i < nk; ++i) {
      mbar_expect_tx(smem_u32(&full[i]), B_BYTES);
      tma_weights(sw + i * B_BYTES, &wmap, i * TC_BK, 0, smem_u32(&full[i]));
    }
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  __syncwarp();
  if (GATHER) {
    gather_rows(smem, sx, a.plane, (int)(sx - sw) + (a.K + 15) / 16 * 2 * a.plane, a, b, y0, x0);
  } else {
    load_window(sx, a.plane, a.X, b, a.H, a.W, a.C, y0, x0, CV_H * MT + 2);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_holder;
  constexpr uint32_t idesc = umma_idesc(TC_BM, BN);
  if (threadIdx.x == 0) {
    // MMA issue.  Every wait is bounded; after a timeout nothing more is issued, and the commit below
    // still arrives once the MMAs issued so far have finished.
    bool ok = true;
    int tap = 0, c0 = 0;
    for (int i = 0; i < nk; ++i) {
      const int st = i % S;
      ok = mbar_wait(smem_u32(&full[st]), (uint32_t)(i / S) & 1u);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      const uint32_t sb = sw + st * B_BYTES;
#pragma unroll
      for (int ks = 0; ks < TC_BK / 16; ++ks) {
        if (i * TC_BK + ks * 16 < a.K) {
          const uint64_t db = umma_desc_sw128(sb + ks * 32);
          const uint32_t acc = i > 0 || ks > 0 ? 1u : 0u;
          if (GATHER) {
            mma_f16(tmem, umma_desc(sx + (uint32_t)((i * (TC_BK / 8) + 2 * ks) * a.plane), a.plane, 128), db, idesc, acc);
          } else {
            // channels c0..c0+15 of tap (ky, kx)
            const int ky = tap / 3, kx = tap - 3 * ky;
            const uint32_t sa = sx + (uint32_t)((c0 >> 3) * a.plane + (ky * (CV_W + 2) + kx) * 16);
#pragma unroll
            for (int m = 0; m < MT; ++m)
              mma_f16(tmem + m * BN, umma_desc(sa + m * CV_H * (CV_W + 2) * 16, a.plane, (CV_W + 2) * 16), db, idesc, acc);
            c0 += 16;
            if (c0 == a.C) {
              c0 = 0;
              ++tap;
            }
          }
        }
      }
      mma_commit(smem_u32(&empty[st]));
    }
    mma_commit(smem_u32(&done));
    if (!mbar_wait(smem_u32(&done), 0) || !ok) failed = 1;
  } else if (threadIdx.x == 32) {
    bool ok = true;
    int i = S;
    for (; i < nk && ok; ++i) {
      const int st = i % S;
      ok = mbar_wait(smem_u32(&empty[st]), (uint32_t)(i / S - 1) & 1u);
      if (!ok) break;
      mbar_expect_tx(smem_u32(&full[st]), B_BYTES);
      tma_weights(sw + st * B_BYTES, &wmap, i * TC_BK, 0, smem_u32(&full[st]));
    }
    if (!ok) {  // no copy may land after the CTA has left: wait (bounded) for those issued
      failed = 1;
      for (int q = i > S ? i - S : 0; q < i && q < nk; ++q) mbar_wait(smem_u32(&full[q % S]), (uint32_t)(q / S) & 1u);
    }
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (failed) {
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
