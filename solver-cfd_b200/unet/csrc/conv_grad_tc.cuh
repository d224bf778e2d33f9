// conv_grad_tc.cuh -- gradients of the 3x3 convolutions on tcgen05, straight from the activations.
//
//   k_conv_dw:  dW[tap][ci][co] += sum_p X[p + tap][ci] * dZ[p][co]
//   k_conv_dx:  dX[p][ci]        = sum_tap sum_co dZ[p - tap][co] * W[tap][ci][co]
//
// The former route went through global matrices nine times the activations' size: im2col, its transpose
// and the transpose of dZ for dW, an FP32 product of the same width and col2im for dX.
//
// k_conv_dw: the reduction runs over pixels, so both operands are MN-major: a core matrix is 8 pixels of 8
// channels, which is what channel planes with 16 bytes per pixel hold (conv_tc.cuh).  A CTA takes the three
// taps of one ky, 128 input channels (missing ones are zero planes), up to 128 output channels and a
// range of 8 x 16-pixel tiles; tap kx moves A's start address by 16 bytes.  The three accumulators stay in
// tensor memory over the range, the next tile's copies (cp.async) run during the MMAs of this one, and
// the result is added to the gradient with vector atomics.  A range has at most DW_TILES tiles, so a sum
// in tensor memory is no longer than about the split-K GEMM's were and the rest is summed in FP32 atomics.
// Where a tile reaches over the canvas's right edge, tap kx = 0 would multiply the last column of X with the
// zeros of dZ beyond the edge; that column is cleared before the tap's MMAs, so an infinity or NaN there stays
// out of a sum that it does not belong to.
//
// k_conv_dx: a CTA takes one tile and up to 96 input channels.  Each tap is its own product over the output
// channels, into one of two accumulators in turn, and is added to the thread's registers while the next
// tap's MMAs run: the same products and the same order of FP32 additions as the GEMM followed by col2im,
// so results are bit-identical.  A tap whose pixel lies outside the canvas is not added.
//
// Bound: latency of the short K loops (copies, commits and tensor-memory loads per tap or tile) at two to
// four CTAs per SM.  Measured: see unet_gemm.cu.
#pragma once
#include <type_traits>

#include "conv_tc.cuh"

namespace unet {

constexpr int DW_TILES = 12;
constexpr int DW_XPLANE = ((CV_W + 2) * CV_H | 1) * 16;  // window rows of one ky: 16 x 10 pixels
constexpr int DW_ZPLANE = (TC_BM | 1) * 16;

// Instruction descriptor with both operands MN-major.
__host__ __device__ constexpr uint32_t umma_idesc_mn(int M, int N) { return umma_idesc(M, N) | (1u << 15) | (1u << 16); }

struct DwArgs {
  const __nv_bfloat16* X;   // [batch][H][W][C]
  const __nv_bfloat16* dZ;  // [batch][H][W][N]
  int batch, H, W, C, N;
  int tx, ty, tiles;        // tiles per row, per column, in all
  int nco;                  // blocks of BN output channels
  float* gW;                // [9*C][N]
  int* err;
};

template <int BN>
__host__ __device__ constexpr int dw_stage() { return 16 * DW_XPLANE + (BN < 16 ? 16 : BN) / 8 * DW_ZPLANE; }

// EDGE: some tiles reach over the right edge (W is not a multiple of CV_W).
template <int BN, bool EDGE>
__global__ void __launch_bounds__(TC_THREADS) k_conv_dw(DwArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int STAGE = dw_stage<BN>();
  constexpr int COLS = 3 * BN <= 32 ? 32 : 3 * BN <= 64 ? 64 : 3 * BN <= 128 ? 128 : 3 * BN <= 256 ? 256 : 512;
  __shared__ unsigned long long bar[2], edge_bar;
  __shared__ uint32_t tmem_holder;
  __shared__ int wait_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ky = blockIdx.y % 3, rest = blockIdx.y / 3;
  const int co0 = rest % a.nco * BN, ci0 = rest / a.nco * 128;
  const int t0 = blockIdx.x * DW_TILES, t1 = min(a.tiles, t0 + DW_TILES);
  const uint32_t s0 = smem_u32(smem);
  const int cn = min(128, a.C - ci0), nn = min(BN, a.N - co0);

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar[0]), 1);
    mbar_init(smem_u32(&bar[1]), 1);
    mbar_init(smem_u32(&edge_bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                 "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  // channels that do not exist stay zero in both stages
  for (int q = threadIdx.x; q < 2 * STAGE / 16; q += TC_THREADS) reinterpret_cast<uint4*>(smem)[q] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();

  auto load = [&](int t, int st) {
    const int x0 = t % a.tx * CV_W;
    t /= a.tx;
    const int y0 = t % a.ty * CV_H;
    const long long img = (long long)(t / a.ty) * a.H * a.W;
    const uint32_t sx = s0 + st * STAGE, sz = sx + 16 * DW_XPLANE;
    if ((a.C & 7) == 0) {
      const int c8 = cn >> 3, total = (CV_W + 2) * CV_H * c8;
      for (int v = threadIdx.x; v < total; v += TC_THREADS) {
        const int q = v / c8, c = v - q * c8, wy = q / (CV_W + 2);
        const int y = y0 + wy + ky - 1, x = x0 - 1 + q - wy * (CV_W + 2);
        const bool ok = y >= 0 && y < a.H && x >= 0 && x < a.W && y0 + wy < a.H;
        cp_async16(sx + (uint32_t)(c * DW_XPLANE + q * 16), ok ? a.X + (img + (long long)y * a.W + x) * a.C + ci0 + 8 * c : a.X, ok);
      }
    } else {
      const unsigned short* X = reinterpret_cast<const unsigned short*>(a.X);
      unsigned short* w = reinterpret_cast<unsigned short*>(smem + st * STAGE);
      for (int v = threadIdx.x; v < (CV_W + 2) * CV_H * cn; v += TC_THREADS) {
        const int q = v / cn, c = v - q * cn, wy = q / (CV_W + 2);
        const int y = y0 + wy + ky - 1, x = x0 - 1 + q - wy * (CV_W + 2);
        const bool ok = y >= 0 && y < a.H && x >= 0 && x < a.W && y0 + wy < a.H;
        w[(c >> 3) * (DW_XPLANE / 2) + q * 8 + (c & 7)] =
            ok ? __ldg(X + (img + (long long)y * a.W + x) * a.C + ci0 + c) : (unsigned short)0;
      }
    }
    const int n8 = nn >> 3;
    for (int v = threadIdx.x; v < TC_BM * n8; v += TC_THREADS) {
      const int q = v / n8, c = v - q * n8, y = y0 + (q >> 3), x = x0 + (q & 7);
      const bool ok = y < a.H && x < a.W;
      cp_async16(sz + (uint32_t)(c * DW_ZPLANE + q * 16), ok ? a.dZ + (img + (long long)y * a.W + x) * a.N + co0 + 8 * c : a.dZ, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load(t0, 0);
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_holder;
  constexpr uint32_t idesc = umma_idesc_mn(TC_BM, BN);
  bool ok = true;
  int last = -1;
  uint32_t edges = 0;  // tiles at the right edge so far
  for (int t = t0; t < t1; ++t) {
    const int i = t - t0, st = i & 1;
    if (t + 1 < t1) {
      // the other stage is free once the MMAs of the tile before this one are done
      if (i >= 1) {
        ok = cta_wait(smem_u32(&bar[st ^ 1]), (uint32_t)((i - 1) >> 1) & 1u, &wait_flag);
        if (!ok) break;
      }
      load(t + 1, st ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    const uint32_t sx = s0 + st * STAGE, sz = sx + 16 * DW_XPLANE;
    const int edge = a.W - t % a.tx * CV_W;  // columns of the canvas from the tile's first on
    auto issue = [&](auto first, auto end) {  // taps kx from first up to end, by one thread
      asm volatile("tcgen05.fence::after_thread_sync;");
      for (int k = 0; k < TC_BM / 16; ++k) {  // two rows of 8 pixels per step
        const uint64_t db = umma_desc(sz + k * 256, 128, DW_ZPLANE);
#pragma unroll
        for (int kx = first.value; kx < end.value; ++kx)
          mma_f16(tmem + kx * BN, umma_desc(sx + (uint32_t)(2 * k * (CV_W + 2) + kx) * 16, (CV_W + 2) * 16, DW_XPLANE), db, idesc,
                  i > 0 || k > 0 ? 1u : 0u);
      }
    };
    constexpr std::integral_constant<int, 0> tap0{};
    constexpr std::integral_constant<int, 1> tap1{};
    constexpr std::integral_constant<int, 3> tap3{};
    if (EDGE && edge < CV_W) {
      if (threadIdx.x == 0) {
        issue(tap1, tap3);
        mma_commit(smem_u32(&edge_bar));
      }
      ok = cta_wait(smem_u32(&edge_bar), edges & 1u, &wait_flag);
      ++edges;
      if (!ok) break;
      for (int q = threadIdx.x; q < 16 * CV_H; q += TC_THREADS) {  // window column of the canvas's last
        const int plane = q / CV_H, row = q - plane * CV_H;
        asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(sx + (uint32_t)(plane * DW_XPLANE + (row * (CV_W + 2) + edge) * 16)),
                     "r"(0)
                     : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (threadIdx.x == 0) {
        issue(tap0, tap1);
        mma_commit(smem_u32(&bar[st]));
      }
    } else if (threadIdx.x == 0) {
      issue(tap0, tap3);
      mma_commit(smem_u32(&bar[st]));
    }
    last = i;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (last >= 0) {  // the last commit covers every MMA issued before it
    const bool fin = cta_wait(smem_u32(&bar[last & 1]), (uint32_t)(last >> 1) & 1u, &wait_flag);
    ok = ok && fin;
  }
  if (EDGE && !ok && edges) cta_wait(smem_u32(&edge_bar), (edges - 1) & 1u, &wait_flag);  // (drains them if it timed out)
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (!ok) {
    if (threadIdx.x == 0 && a.err) atomicExch(a.err, 1);
  } else {
    const int ci = warp * 32 + lane;
#pragma unroll 1
    for (int kx = 0; kx < 3; ++kx) {
      float* g = a.gW + ((long long)(ky * 3 + kx) * a.C + ci0 + ci) * a.N + co0;
#pragma unroll 1
      for (int n = 0; n < nn; n += 16) {
        uint32_t r[16];
        tmem_ld16(r, tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(kx * BN + n));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (ci < cn) {
#pragma unroll
          for (int j = 0; j < 16; j += 4)
            if (n + j < nn)
              atomicAdd(reinterpret_cast<float4*>(g + n + j),
                        make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                                    __uint_as_float(r[j + 3])));
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
}

struct DxArgs {
  const __nv_bfloat16* dZ;  // [batch][H][W][N]
  const __nv_bfloat16* Wt;  // [9*C][N], row tap*C + ci
  int H, W, C, N;
  int tx, ty;
  int plane, kpad;          // bytes of a window plane; N rounded up to 16
  float* dX;                // [batch][H][W][C]
  int* err;
};

constexpr int DX_RING = 3;  // taps whose weights are in flight

// Shared memory: [window planes of dZ (kpad / 8)][DX_RING taps' weights: BN rows x kpad, K-major planes].
template <int BN>
__global__ void __launch_bounds__(TC_THREADS) k_conv_dx(DxArgs a) {
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int COLS = 2 * BN <= 64 ? 64 : 2 * BN <= 128 ? 128 : 256;
  __shared__ unsigned long long bar[2];
  __shared__ uint32_t tmem_holder;
  __shared__ int wait_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int t = blockIdx.x;
  const int x0 = t % a.tx * CV_W;
  t /= a.tx;
  const int y0 = t % a.ty * CV_H, b = t / a.ty;
  const int ci0 = blockIdx.y * BN, k8 = a.kpad >> 3;
  const uint32_t sx = smem_u32(smem), sw = sx + (uint32_t)(k8 * a.plane), wbytes = (uint32_t)(BN * a.kpad * 2);

  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&bar[0]), 1);
    mbar_init(smem_u32(&bar[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                 "r"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  load_window(sx, a.plane, a.dZ, b, a.H, a.W, a.N, y0, x0, CV_H + 2);
  if (a.kpad > a.N)  // 8 output channels: the second half of the K step is zero
    for (int q = threadIdx.x; q < cv_pixels(1); q += TC_THREADS)
      asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(sx + (uint32_t)((k8 - 1) * a.plane + q * 16)), "r"(0) : "memory");
  auto load_w = [&](int tap) {  // rows ci0.. of the tap, chunk c of row n at plane c (BN * 16 bytes)
    const uint32_t dst = sw + (uint32_t)(tap % DX_RING) * wbytes;
    for (int v = threadIdx.x; v < BN * k8; v += TC_THREADS) {
      const int n = v / k8, c = v - n * k8;
      const bool ok = ci0 + n < a.C && 8 * c < a.N;
      cp_async16(dst + (uint32_t)(c * BN * 16 + n * 16), ok ? a.Wt + ((long long)tap * a.C + ci0 + n) * a.N + 8 * c : a.Wt, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int q = 0; q < DX_RING; ++q) load_w(q);  // the first group also holds the window
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_holder;
  constexpr uint32_t idesc = umma_idesc(TC_BM, BN);
  float s[BN];
#pragma unroll
  for (int j = 0; j < BN; ++j) s[j] = 0.f;
  const int m = warp * 32 + lane, mx = x0 + (m & 7), my = y0 + (m >> 3);  // this thread's pixel
  bool ok = true;
  int last = -1;
  // tap's product, once its weights are there (up to `newer` younger copy groups may be in flight)
  auto issue = [&](int tap, int newer) {
    if (newer == 2) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (newer == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;");
      const int ky = tap / 3, kx = tap - 3 * ky;
      // output pixel p - tap: row y - ky + 1, column x - kx + 1, i.e. window offset (2 - ky, 2 - kx)
      const uint32_t sa = sx + (uint32_t)((2 - ky) * (CV_W + 2) + 2 - kx) * 16, sb = sw + (uint32_t)(tap % DX_RING) * wbytes;
      for (int k = 0; k < a.kpad / 16; ++k)
        mma_f16(tmem + (tap & 1) * BN, umma_desc(sa + (uint32_t)(2 * k * a.plane), a.plane, (CV_W + 2) * 16),
                umma_desc(sb + (uint32_t)(2 * k * BN * 16), BN * 16, 128), idesc, k > 0 ? 1u : 0u);
      mma_commit(smem_u32(&bar[tap & 1]));
    }
    last = tap;
  };
  issue(0, 2);
  auto add_taps = [&](auto edge) {
    for (int tap = 0; tap < 9; ++tap) {
      // the next tap's MMAs run while this one's accumulator is read; its TMEM half was read two taps ago
      if (tap + 1 < 9) issue(tap + 1, tap + 2 < 9 ? 1 : 0);
      ok = cta_wait(smem_u32(&bar[tap & 1]), (uint32_t)(tap >> 1) & 1u, &wait_flag);
      if (!ok) break;
      if (tap + DX_RING < 9) load_w(tap + DX_RING);
      const int ty = my + 1 - tap / 3, tx = mx + 1 - tap % 3;  // the pixel of dZ
      const bool in = !edge.value || (ty >= 0 && ty < a.H && tx >= 0 && tx < a.W);
      asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
      for (int n = 0; n < BN; n += 16) {
        uint32_t r[16];
        tmem_ld16(r, tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)((tap & 1) * BN + n));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; ++j) s[n + j] = in ? s[n + j] + __uint_as_float(r[j]) : s[n + j];
      }
    }
  };
  if (x0 > 0 && y0 > 0 && x0 + CV_W < a.W && y0 + CV_H < a.H) add_taps(std::false_type{});
  else add_taps(std::true_type{});
  asm volatile("cp.async.wait_all;" ::: "memory");
  if (!ok) {  // one more bounded wait drains the MMAs issued (see k_gemm_tc)
    cta_wait(smem_u32(&bar[last & 1]), (uint32_t)(last >> 1) & 1u, &wait_flag);
    if (threadIdx.x == 0 && a.err) atomicExch(a.err, 1);
  } else {
    if (mx < a.W && my < a.H) {
      float* d = a.dX + (((long long)b * a.H + my) * a.W + mx) * a.C + ci0;
      const int n1 = a.C - ci0;
      if ((a.C & 3) == 0) {
#pragma unroll
        for (int n = 0; n < BN; n += 4)
          if (n < n1) *reinterpret_cast<float4*>(d + n) = make_float4(s[n], s[n + 1], s[n + 2], s[n + 3]);
      } else {
#pragma unroll
        for (int n = 0; n < BN; ++n)
          if (n < n1) d[n] = s[n];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLS));
}

}  // namespace unet
