// chip_engine.cuh -- the on-chip engine: a case's whole pseudo-time state stays in the shared
// memory of one thread-block cluster for a whole launch (many physical steps of main.f90:116-186).
//
// Split: as in engine.cuh, K <= 16 CTAs each own a horizontal strip of node rows.  Here every array
// that is read with a stencil (u, v: tau and two stage arrays each, both pressures, T, C: tau and
// two stage arrays each) is a window of the strip plus its halo rows (two for u and v, one for T and
// C, one below for p) in the CTA's shared memory.  A node computed in a row that a neighbour holds as
// halo is also stored into that neighbour's window through distributed shared memory, so after the
// cluster barrier that ends a phase every CTA reads shared memory only.  What is read at its own node
// only (the physical-step u, v, T, C and the buoyancy term) sits in shared memory too where that fits
// (PHYS), else in global memory, written and read by the same CTA.
//
// Schedule: the four phases per pseudo-iteration of engine.cuh (U and V stages 1..3 with T, C stages
// 2 and 3 of the previous iteration in the first two, then P with T, C stage 1), one cluster barrier
// each.  Every CTA writes its residual maximum into every CTA's shared memory before the last
// barrier, so the exit decision needs no memory traffic and no further barrier.
//
// Bound: latency.  Four empty phases take 2.3 us of a pseudo-iteration (a cluster barrier alone 0.22 us
// with 256 threads), a node's loads, address arithmetic and dependence chain most of the rest; the FP64
// pipe (one warp instruction per two clocks and SM quarter) is busy for a fifth to a third of the time.
// Measured on one B200, us per pseudo-iteration, cluster engine -> this engine: 51 x 84 EXACT 208 -> 16.6,
// 51 x 51 upwind FAST 34 -> 5.4, 102 x 102 full FAST 64 -> 14.7, 8 cases of 153 x 153 EXACT 394 -> 99.
//
// Termination: as in engine.cuh -- identical decisions from identical residuals in every CTA, at most
// itc_max iterations per step.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "acs_dev.cuh"
#include "chip_engine.h"

namespace acs {
namespace cg = cooperative_groups;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// The shared::cluster address of `addr` in CTA `rank`.
__device__ __forceinline__ uint32_t map_cluster(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Stores v at a shared::cluster address.
__device__ __forceinline__ void st_cluster(uint32_t addr, double v) {
  // no memory clobber: the store never touches this CTA's memory, and the cluster barrier orders it
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v));
}

// Maximum over the warp of the bit patterns of non-negative doubles (NaN bits are above infinity's).
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v) {
  const unsigned hi = (unsigned)(v >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned lo = hi == mh ? (unsigned)v : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
  return ((unsigned long long)mh << 32) | ml;
}

// Metric differences of a column (d = x(i)-x(i-1), dm = xm(i+1)-xm(i)) or row and their reciprocals.
struct Half { double d, rd; };

// What a node's arithmetic reads besides the fields: the case, its constants (PT::constants) and the
// metrics in shared memory as 16-byte pairs {difference, reciprocal}: xd, xm by column, yd, ym by row.
struct ChipCtx {
  const CaseDev& d;
  const double* k;
  const Half* xd;
  const Half* xm;
  const Half* yd;
  const Half* ym;
  int P;
};

// Column metrics of a node (xe = xd(i+1), xw = xm(i-1)), and the node: its row metrics (yn = yd(j+1),
// ys = ym(j-1)) beside them.
struct ChipCol {
  Half xd, xm, xe, xw;
  __device__ __forceinline__ ChipCol(const ChipCtx& x, int i) : xd(x.xd[i]), xm(x.xm[i]), xe(x.xd[i + 1]), xw(x.xm[i - 1]) {}
};
struct ChipNode : ChipCol {
  Half yd, ym, yn, ys;
  int i, j;
  bool por;
  __device__ __forceinline__ ChipNode(const ChipCtx& x, const ChipCol& c, int i_, int j_, bool por_)
      : ChipCol(c), yd(x.yd[j_]), ym(x.ym[j_]), yn(x.yd[j_ + 1]), ys(x.ym[j_ - 1]), i(i_), j(j_), por(por_) {}
};

// Where node (i, j) of window k lies: x + k * xs + (i-1) + (j-1) * pitch (in doubles).  In shared memory:
// the compiler would otherwise derive these from the layout again in every phase.
struct ChipWin { int u, us, v, p, ps, t, c, ts, e, es, w; };

struct ChipRoles { int ru[3], rv[3], rt[3], rc[3]; };

template <class PT, bool PHYS, bool QUICK>
__global__ void __launch_bounds__(CHIP_THREADS, 1) k_chip(ChipArgs a) {
  constexpr int NT = CHIP_THREADS;
  extern __shared__ __align__(16) double sm[];
  __shared__ CaseDev d_sh;
  __shared__ ChipRoles g;
  __shared__ ChipWin W;
  __shared__ unsigned long long red[2][16];            // residual maxima by iteration parity and CTA
  __shared__ double kc[12];                            // constants of the case
  __shared__ unsigned long long wred[NT / 32];
  cg::cluster_group cl = cg::this_cluster();
  const int K = (int)cl.num_blocks();
  const int rank = (int)cl.block_rank();
  const int c = a.cases[blockIdx.x / K];
  const int tid = threadIdx.x;
  CaseCtl* gk = a.ctl + c;
  if (!gk->active) return;  // the whole cluster

  static_assert(sizeof(CaseDev) % 8 == 0, "case descriptor size");
  #pragma unroll 1
  for (int q = tid; q < (int)(sizeof(CaseDev) / 8); q += NT)
    reinterpret_cast<unsigned long long*>(&d_sh)[q] = reinterpret_cast<const unsigned long long*>(a.cs + c)[q];
  if (tid == 0) {
    for (int r = 0; r < 3; ++r) { g.ru[r] = gk->ru[r]; g.rv[r] = gk->rv[r]; g.rt[r] = gk->rt[r]; g.rc[r] = gk->rc[r]; }
  }
  __syncthreads();
  const CaseDev& d = d_sh;
  const int nx = d.nx, ny = d.ny, P = d.pitch;
  const int R = ny + 1;
  const int r0 = 1 + (rank * R) / K, r1 = 1 + ((rank + 1) * R) / K;
  const bool scal = gk->scalars && d.solve_scalars;
  const bool buoy = (d.flags & F_BUOY) != 0;
  // control word (the same values in every thread of the cluster)
  int itc = gk->itc, step = gk->step, n_steps = gk->n_steps, kk = gk->k, status = gk->status;
  int rp0 = gk->rp[0], rp1 = gk->rp[1], rp_read = gk->rp_read, ntau_alias = gk->ntau_alias;
  bool dirty = gk->tau_dirty != 0;
  long long total = gk->total_iters;

  // ---- shared-memory windows; w[lin(i, j)] is node (i, j) for the rows of the window ----
  const ChipLayout L = chip_layout(nx, ny, P, K, scal, PHYS);
  auto bias = [&](int off, int halo) { return off - (r0 - halo - 1) * P; };
  if (tid == 0)
    W = {bias(L.u, 2), L.uv_size, bias(L.v, 2), bias(L.p, 1), L.p_size, bias(L.t, 1), bias(L.c, 1), L.tc_size,
         bias(L.phys, 0), L.own_size, bias(L.w, 0)};
  auto U = [&](int k) { return sm + (W.u + k * W.us); };
  auto V = [&](int k) { return sm + (W.v + k * W.us); };
  auto Pw = [&](int k) { return sm + (W.p + k * W.ps); };
  auto Tw = [&](int k) { return sm + (W.t + k * W.ts); };
  auto Cw = [&](int k) { return sm + (W.c + k * W.ts); };
  unsigned char* por = reinterpret_cast<unsigned char*>(sm + L.mask) - (r0 - 1) * P;
  #pragma unroll 1
  for (int q = tid; q < L.total; q += NT) sm[q] = 0.0;
  __syncthreads();
  // rows [ja, jb) of a case array into a window (whole pitch), clipped to the array's rows 1..R
  auto load = [&](double* w, const double* src, int ja, int jb) {
    ja = ja < 1 ? 1 : ja;
    jb = jb > R + 1 ? R + 1 : jb;
    #pragma unroll 1
    for (int q = (ja - 1) * P + tid; q < (jb - 1) * P; q += NT) w[q] = src[q];
  };
  load(U(0), d.U[g.ru[R_TAU]], r0 - 2, r1 + 2);
  load(V(0), d.V[g.rv[R_TAU]], r0 - 2, r1 + 2);
  load(Pw(0), d.P[0], r0 - 1, r1);
  load(Pw(1), d.P[1], r0 - 1, r1);
  if (scal) {
    load(Tw(0), d.T[g.rt[R_TAU]], r0 - 1, r1 + 1);
    load(Cw(0), d.C[g.rc[R_TAU]], r0 - 1, r1 + 1);
  }
  #pragma unroll 1
  for (int q = (r0 - 1) * P + tid; q < (r1 - 1) * P; q += NT) por[q] = d.mask[q];
  // metrics of the columns 0..nx+1 and of the rows r0-1..r1 (0 where a neighbour does not exist)
  Half* mx = reinterpret_cast<Half*>(sm + L.met);
  Half* my = mx + 2 * (nx + 2);
  const int sy = L.rows + 2;
  const ChipCtx x{d, kc, mx, mx + nx + 2, my - (r0 - 1), my + sy - (r0 - 1), P};
  if (tid == 0) PT::constants(d, kc);
  auto metrics = [&](Half* td, Half* tm, int n, int k0, const double* f, const double* m, int kmax) {
    #pragma unroll 1
    for (int q = tid; q < n; q += NT) {
      const int k = k0 + q;
      if (k >= 2 && k <= kmax) { td[q].d = f[k] - f[k - 1]; td[q].rd = 1.0 / td[q].d; }
      if (k >= 1 && k <= kmax) { tm[q].d = m[k + 1] - m[k]; tm[q].rd = 1.0 / tm[q].d; }
    }
  };
  metrics(mx, mx + nx + 2, nx + 2, 0, d.x, d.xm, nx);
  metrics(my, my + sy, sy, r0 - 1, d.y, d.ym, ny);
  // physical-step arrays and the buoyancy term (own rows)
  double* pu = nullptr;
  double* pv = nullptr;
  double* pt = nullptr;
  double* pc = nullptr;
  double* bw = PHYS ? sm + W.w : d.S2[3];
  auto phys_pointers = [&]() {
    if constexpr (PHYS) {
      pu = sm + W.e;
      pv = sm + (W.e + W.es);
      pt = sm + (W.e + 2 * W.es);
      pc = sm + (W.e + 3 * W.es);
    } else {
      pu = d.U[g.ru[R_PHYS]];
      pv = d.V[g.rv[R_PHYS]];
      pt = d.T[g.rt[R_PHYS]];
      pc = d.C[g.rc[R_PHYS]];
    }
  };
  phys_pointers();
  if constexpr (PHYS) {
    load(pu, d.U[g.ru[R_PHYS]], r0, r1);
    load(pv, d.V[g.rv[R_PHYS]], r0, r1);
    if (scal) {
      load(pt, d.T[g.rt[R_PHYS]], r0, r1);
      load(pc, d.C[g.rc[R_PHYS]], r0, r1);
    }
  }
  const int ja = r0 > 2 ? r0 : 2, jb = r1 - 1 < ny - 1 ? r1 - 1 : ny - 1;  // rows with interior nodes
  const int wi = nx - 2;
  const int cells = jb >= ja ? wi * (jb - ja + 1) : 0;
  // the buoyancy term of the physical-step temperature at the v nodes (T: a window with its lower
  // halo row, or the case array)
  auto set_buoy = [&](const double* T) {
    #pragma unroll 1
    for (int q = tid; q < cells; q += NT) {
      const int i = 2 + q % wi, j = ja + q / wi;
      const int o = (i - 1) + (j - 1) * P;
      bw[o] = PT::buoy(x, T[o], T[o - P]);
    }
  };
  if (buoy) set_buoy(d.T[g.rt[R_PHYS]]);
  else if (!PHYS)
    #pragma unroll 1
    for (int q = (r0 - 1) * P + tid; q < (r1 - 1) * P; q += NT) bw[q] = 0.0;

  // ---- stores with the neighbours' halo copies ----
  // (distance from a word here to its copy in the neighbour's window, as shared::cluster addresses)
  const uint32_t s0 = smem_addr(sm);
  const uint32_t dlo = rank > 0 ? map_cluster(s0, rank - 1) - s0 + (r0 - (1 + ((rank - 1) * R) / K)) * P * 8 : 0u;
  const uint32_t dup = rank < K - 1 ? map_cluster(s0, rank + 1) - s0 + (r0 - r1) * P * 8 : 0u;
  const int jlo2 = rank > 0 ? r0 + 2 : 0, jlo1 = rank > 0 ? r0 + 1 : 0;          // rows below: pushed down
  const int jup2 = rank < K - 1 ? r1 - 2 : 1 << 30, jup1 = rank < K - 1 ? r1 - 1 : 1 << 30;  // rows from: pushed up
  auto put = [&](double* a, double v, int j, int lo, int up) {
    *a = v;
    if (j < lo) st_cluster(smem_addr(a) + dlo, v);
    if (j >= up) st_cluster(smem_addr(a) + dup, v);
  };
  // ---- boundary passes (boundary.f90:1-159; channel variant as in bc_exact.cuh) ----
  // A boundary value that copies or negates one interior node is stored by that node's thread with the
  // node itself (image_u, image_v, image_c); constant ones are set once (set_constants); the scalars'
  // extrapolated side is never stored inside the loop, the one node that reads it extrapolates itself
  // (edge_e, edge_n); the pressure's boundary is not read by the loop at all.  So a phase needs no pass
  // of its own and no CTA barrier, except for the outflow rows of v in the reference variant, which
  // extrapolate two rows (top_v, last strip only).  finish_c completes a scalar or pressure window
  // before it leaves the chip.  Neighbours read no boundary node of a halo row but u(imax, j).
  const bool ch = d.bc != 0;
  const bool bottom = r0 == 1, top = r1 == R + 1;
  auto at = [&](int i, int j) { return (i - 1) + (j - 1) * P; };
  const int edge_i = ch ? nx - 1 : 0, edge_j = ch ? 0 : ny - 1;  // nodes that extrapolate z(i+1, j) or z(i, j+1)
  auto image_u = [&](double* w, int i, int j, int o, double v) {  // node (i, j) was stored at w[o]
    if (ch && i == nx - 1) {
      put(w + o + 1, v, j, jlo2, jup2);
      w[o + 2] = v;
    }
    if (j == 2 && ch) {
      w[o - P] = -v;
      if (i == nx - 1) w[o - P + 1] = w[o - P + 2] = -v;
    }
    if (j == ny - 1) {
      w[o + P] = ch ? -v : v;
      if (ch && i == nx - 1) w[o + P + 1] = w[o + P + 2] = -v;
    }
  };
  auto image_v = [&](double* w, int i, int j, int o, double v) {
    const double l = ch ? -v : v;  // column 1; column imax holds v
    if (i == 2) w[o - 1] = l;
    if (i == nx - 1) w[o + 1] = v;
    if (ch && j == 3) {
      w[o - 2 * P] = -v;
      if (i == 2) w[o - 2 * P - 1] = -l;
      if (i == nx - 1) w[o - 2 * P + 1] = -v;
    }
    if (ch && j == ny - 1) {
      w[o + 2 * P] = -v;
      if (i == 2) w[o + 2 * P - 1] = -l;
      if (i == nx - 1) w[o + 2 * P + 1] = -v;
    }
  };
  auto image_c = [&](double* w, int i, int j, int o, double v) {
    if (ch) {
      if (j == 2) w[o - P] = v;
      if (j == ny - 1) w[o + P] = v;
    } else {
      if (i == 2) w[o - 1] = v;
      if (i == nx - 1) w[o + 1] = v;
    }
  };
  auto top_v = [&](double* v) {  // rows imax, jmax+1 of the reference variant
    #pragma unroll 1
    for (int i = 2 + tid; i <= nx - 1; i += NT) {
      const double b = v[at(i, ny - 1)], n = 2.0 * v[at(i, ny - 2)] - b, m = 2.0 * b - n;
      v[at(i, ny)] = n;
      v[at(i, ny + 1)] = m;
      if (i == 2) { v[at(1, ny)] = n; v[at(1, ny + 1)] = m; }
      if (i == nx - 1) v[at(nx, ny)] = n;
    }
  };
  auto set_constants_c = [&](double* t, double* s) {
    if (ch) {
      #pragma unroll 1
      for (int j = r0 + tid; j <= ny && j < r1; j += NT) {
        t[at(1, j)] = d.T_in;
        s[at(1, j)] = d.C_in;
      }
    } else if (bottom) {
      #pragma unroll 1
      for (int i = 1 + tid; i <= nx; i += NT) {
        t[at(i, 1)] = d.T_in;
        s[at(i, 1)] = d.C_in;
      }
    }
  };
  auto set_constants = [&](double* u, double* v) {
    #pragma unroll 1
    for (int j = (r0 - 2 < 1 ? 1 : r0 - 2) + tid; j <= ny && j < r1 + 2; j += NT) {
      const bool w = j == 1 || j == ny;
      u[at(1, j)] = u[at(2, j)] = ch ? (w ? -d.v_in : d.v_in) : 0.0;
      if (!ch) u[at(nx, j)] = u[at(nx + 1, j)] = 0.0;
    }
    #pragma unroll 1
    for (int i = 1 + tid; i <= nx; i += NT) {
      if (bottom) {
        v[at(i, 2)] = ch ? 0.0 : d.v_in;
        if (!ch) {
          v[at(i, 1)] = d.v_in;
          u[at(i, 1)] = 0.0;
        }
      }
      if (top && ch) v[at(i, ny)] = 0.0;
    }
  };
  // bcP (neumann: the inflow side copies its neighbour), bcZ or bcC (inflow value zin) on the own rows
  const int ju = r1 - 1 < ny ? r1 - 1 : ny;
  auto finish_c = [&](double* z, bool neumann, double zin) {
    auto sides = [&]() {
      #pragma unroll 1
      for (int j = r0 + tid; j <= ju; j += NT) {
        const double b = z[at(nx - 1, j)];
        z[at(1, j)] = ch && !neumann ? zin : z[at(2, j)];
        z[at(nx, j)] = ch ? b + 1.0 * (b - z[at(nx - 2, j)]) : b;
      }
    };
    __syncthreads();
    if (ch) sides();
    __syncthreads();
    #pragma unroll 1
    for (int i = 1 + tid; i <= nx; i += NT) {
      if (bottom) z[at(i, 1)] = ch || neumann ? z[at(i, 2)] : zin;
      if (top) {
        const double b = z[at(i, ny - 1)];
        z[at(i, ny)] = ch ? b : b + 1.0 * (b - z[at(i, ny - 2)]);
      }
    }
    __syncthreads();
    if (!ch) sides();
    __syncthreads();
  };
  // bcUV's pass over a whole tau array, on the rows of the window (halo rows included: side columns are
  // row-local, and no halo row is a wall row)
  auto full_bc = [&](double* u, double* v) {
    const int a0 = r0 - 2 < 1 ? 1 : r0 - 2, a1 = r1 + 1 < R ? r1 + 1 : R;
    auto sides = [&]() {
      #pragma unroll 1
      for (int j = a0 + tid; j <= a1; j += NT) {
        if (u && j <= ny) {
          const double r = ch ? u[at(nx - 1, j)] : 0.0;
          u[at(1, j)] = u[at(2, j)] = ch ? d.v_in : 0.0;
          u[at(nx, j)] = u[at(nx + 1, j)] = r;
        }
        if (v) {
          v[at(1, j)] = ch ? -v[at(2, j)] : v[at(2, j)];
          if (ch || (j >= 2 && j <= ny)) v[at(nx, j)] = v[at(nx - 1, j)];
        }
      }
    };
    if (ch) sides();
    __syncthreads();
    #pragma unroll 1
    for (int i = 1 + tid; i <= nx + 1; i += NT) {
      if (u && bottom) {
        if (ch) u[at(i, 1)] = -u[at(i, 2)];
        else if (i >= 2 && i <= nx) u[at(i, 1)] = 0.0;
      }
      if (u && top) {
        if (ch) u[at(i, ny)] = -u[at(i, ny - 1)];
        else if (i >= 2 && i <= nx) u[at(i, ny)] = u[at(i, ny - 1)];
      }
      if (v && i <= nx) {
        if (bottom && ch) { v[at(i, 2)] = 0.0; v[at(i, 1)] = -v[at(i, 3)]; }
        if (bottom && !ch) { v[at(i, 1)] = d.v_in; v[at(i, 2)] = d.v_in; }
        if (top && ch) { v[at(i, ny)] = 0.0; v[at(i, ny + 1)] = -v[at(i, ny - 1)]; }
        if (top && !ch && i >= 2) {
          const double b = v[at(i, ny - 1)], n = 2.0 * v[at(i, ny - 2)] - b;
          v[at(i, ny)] = n;
          v[at(i, ny + 1)] = 2.0 * b - n;
        }
      }
    }
    __syncthreads();
    if (!ch) sides();
  };

  // ---- node work ----
  double res = 0.0;  // this thread's residual maximum of the iteration (NaN wins)
  auto residual = [&](double r) {
    const double ar = fabs(r);
    res = (ar > res || ar != ar) ? ar : res;
  };
  // window indices of the tau array and the two stage arrays (the last also the n_tau array)
  int ut = 0, ua = 1, ub = 2, tt = 0, ta = 1, tb = 2;
  bool pend = false;

  // Runge-Kutta stage: ca * tau + cb * (in + r), with in = tau, ca = 0, cb = 1 in stage 1
  auto coef = [&](int st, double& ca, double& cb) {
    ca = st == 1 ? 0.0 : st == 2 ? 0.75 : 1.0 / 3.0;
    cb = st == 1 ? 1.0 : st == 2 ? 0.25 : 2.0 / 3.0;
  };
  // this thread's nodes, columns fastest: whole rows of threads (a fixed column per thread, whose
  // metrics then stay in registers) where that needs no more rounds than a stride of NT nodes
  const int nrow = jb - ja + 1, grp = NT / wi;
  const bool fixed = grp > 0 && (nrow + grp - 1) / grp <= (cells + NT - 1) / NT;
  const int stride = fixed ? grp * wi : NT;
  const int i0 = 2 + tid % wi, j0 = tid < stride ? ja + tid / wi : jb + 1, di = stride % wi, dj = stride / wi;
  const bool has = j0 <= jb;
  // U and V of a stage at this thread's nodes.  Both residuals are computed at every node of the strip
  // (the windows hold every neighbour), so their chains overlap; each is kept where its unknown is
  // updated.  What lies in global memory (PHYS = false) is loaded one node ahead.
  auto uv_stage = [&](int st, bool doU, bool doV, const double* uin, const double* vin, double* uo, double* vo,
                      const double* utau, const double* vtau, const double* pn) {
    double ca, cb;
    coef(st, ca, cb);
    const double dt = d.dt, dtau = d.dtau;
    int i = i0, j = j0;
    ChipCol col(x, i);
    double gu = 0.0, gv = 0.0, gw = 0.0;
    if (!PHYS) {
      const int o = at(i, j);
      gu = pu[o];
      gv = pv[o];
      gw = bw[o];
    }
    #pragma unroll 1
    do {
      const int o = at(i, j), io = i, jo = j;
      const double fu = PHYS ? pu[o] : gu, fv = PHYS ? pv[o] : gv, w = PHYS ? bw[o] : gw;
      const ChipNode n(x, col, i, j, por[o] != 0);
      i += di;
      j += dj;
      if (di) {
        if (i > nx - 1) { i -= wi; j += 1; }
        if (j <= jb) col = ChipCol(x, i);
      }
      if (!PHYS && j <= jb) {
        const int o2 = at(i, j);
        gu = pu[o2];
        gv = pv[o2];
        gw = bw[o2];
      }
      double Ru, Rv;
      PT::template uv<QUICK>(x, n, uin + o, vin + o, utau + o, vtau + o, pn + o, w, Ru, Rv);
      const double tu = utau[o], tv = vtau[o];
      const double ru = ((fu - tu) + Ru * dt) * dtau, rv = ((fv - tv) + Rv * dt) * dtau;
      const double nu = ca * tu + cb * (uin[o] + ru), nv = ca * tv + cb * (vin[o] + rv);
      const bool edge = io == 2 || io == nx - 1 || jo <= 3 || jo == ny - 1;
      if (doU && io >= 3) {
        put(uo + o, nu, jo, jlo2, jup2);
        if (edge) image_u(uo, io, jo, o, nu);
        if (st == 3) residual(ru);
      }
      if (doV && jo >= 3) {
        put(vo + o, nv, jo, jlo2, jup2);
        if (edge) image_v(vo, io, jo, o, nv);
        if (st == 3) residual(rv);
      }
    } while (j <= jb);
  };
  // T and C of a stage at this thread's nodes; with p1 also P (p0 -> p1).  ext: the stage input's
  // boundary is the loop's (an uploaded array is read as it is)
  auto tc_stage = [&](int st, bool ext, const double* un, const double* vn, const double* ti, const double* ci, double* to, double* co,
                      const double* ttau, const double* ctau, const double* p0, double* p1) {
    double ca, cb;
    coef(st, ca, cb);
    const double dt = d.dt, dtau = d.dtau;
    int i = i0, j = j0;
    ChipCol col(x, i);
    double gt = 0.0, gc = 0.0;
    if (!PHYS && scal) {
      const int o = at(i, j);
      gt = pt[o];
      gc = pc[o];
    }
    #pragma unroll 1
    do {
      const int o = at(i, j), io = i, jo = j;
      const ChipNode n(x, col, i, j, por[o] != 0);
      double ft = gt, fc = gc;
      if (PHYS && scal) {
        ft = pt[o];
        fc = pc[o];
      }
      i += di;
      j += dj;
      if (di) {
        if (i > nx - 1) { i -= wi; j += 1; }
        if (j <= jb) col = ChipCol(x, i);
      }
      if (!PHYS && scal && j <= jb) {
        const int o2 = at(i, j);
        gt = pt[o2];
        gc = pc[o2];
      }
      if (p1) {
        double r;
        const double v = PT::p_update(x, n, p0[o], un + o, vn + o, &r);
        put(p1 + o, v, jo, 0, jup1);
        residual(r);
      }
      if (scal) {
        double Rt, Rc;
        PT::tc(x, n, ext && io == edge_i, ext && jo == edge_j, un + o, vn + o, ti + o, ci + o, Rt, Rc);
        const double a = ttau[o], b = ctau[o];
        const double nt = ca * a + cb * (ti[o] + ((ft - a) + Rt * dt) * dtau);
        const double nc = ca * b + cb * (ci[o] + ((fc - b) + Rc * dt) * dtau);
        put(to + o, nt, jo, jlo1, jup1);
        put(co + o, nc, jo, jlo1, jup1);
        if (io == 2 || io == nx - 1 || jo == 2 || jo == ny - 1) {
          image_c(to, io, jo, o, nt);
          image_c(co, io, jo, o, nc);
        }
      }
    } while (j <= jb);
  };
  // own rows of a window into a case array (and into the physical-step window)
  auto store_rows = [&](double* dst, const double* w) {
    #pragma unroll 1
    for (int q = (r0 - 1) * P + tid; q < (r1 - 1) * P; q += NT) dst[q] = w[q];
  };
  // vm(imax, jmax+1) of the reference variant: bcUV's row pass computes it from what the n_tau
  // array holds in column imax before its column pass, i.e. from that array's previous contents
  // (the loop never reads it).  The stage windows rotate differently from the case's buffers, so
  // that history is kept here: nodes (imax, jmax-1) and (imax, jmax-2) of the buffer in each role.  (The tile
  // engine's n_tau tile holds the physical-step array before its passes; a batch that runs here in its
  // place gets the value from that one.)
  const bool corner = d.bc == 0 && r1 == R + 1 && tid == 0;
  double h1[3] = {0, 0, 0}, h2[3] = {0, 0, 0};
  if (corner)
    for (int r = 0; r < 3; ++r) {
      h1[r] = d.V[g.rv[r]][at(nx, ny - 1)];
      h2[r] = d.V[g.rv[r]][at(nx, ny - 2)];
    }

  // ---- the loop, one phase per trip (one copy of each stage's code) ----
  // 1..3: U and V stage, with the pending T, C stage phase + 1 in phases 1 and 2; 4: P and T, C stage 1,
  // then the control decision; 5, 6: the pending T, C stages 2 and 3 on their own before a step ends;
  // 7: the boundary pass on the other velocity's tau array that follows each U or V stage of an
  // iteration with CaseCtl::tau_dirty, which runs U (pass 0) and V (pass 1) one after the other
  // (bcUV(u_stage, vm_tau), bcUV(um_tau, v_stage)).
  enum { GO = 0, EXIT = 1, CAP = 2, FAILED = 3 };
  int ph = 1, st7 = 0, pass = 0, par = 0, fin = GO;
  int p_made = 0;       // pressure windows that the loop has written
  bool t_made = false;  // the T, C tau windows come from the loop
  double e = 0.0;
  bool active = true;
  bool tc_const = false;  // all three T, C windows hold the constant boundary
  auto swap_tc = [&]() {
    const int s = tt; tt = ta; ta = s;
    if (!tc_const) set_constants_c(Tw(ta), Cw(ta));
    tc_const = true;
  };
  // (the tau windows hold uploaded arrays or the loop's: those of u and v get their boundary in phase 7
  // or have it, those of T and C when they become stage windows)
  for (int k = 1; k < 3; ++k) {
    set_constants(U(k), V(k));
    if (scal) set_constants_c(Tw(k), Cw(k));
  }
  cl.sync();  // every window is loaded before a neighbour stores into it
  while (active) {
    const bool uvp = ph <= 3;
    const bool doU = uvp && (!dirty || pass == 0), doV = uvp && (!dirty || pass == 1);
    // T, C stage of this phase (0: none) and its windows
    const int z = ph == 4 ? (scal ? 1 : 0) : ph == 5 || ph == 6 ? ph - 3 : pend && ph <= 2 ? ph + 1 : 0;
    const int zi = z == 1 ? tt : z == 2 ? ta : tb, zo = z == 2 ? tb : ta;
    const int out = ph == 2 ? ub : ua;
    double* pn = Pw(rp1);
    if (uvp && has) {
      const int in = ph == 1 ? ut : ph == 2 ? ua : ub;
      uv_stage(ph, doU, doV, U(in), V(in), U(out), V(out), U(ut), V(ut), Pw(rp_read));
    }
    if ((z || ph == 4) && has) {
      const int nu = ph == 4 || fin == EXIT || fin == FAILED ? ua : ut;  // the velocities of the iteration that T, C belong to
      tc_stage(z, z != 1 || t_made, U(nu), V(nu), Tw(zi), Cw(zi), Tw(zo), Cw(zo), Tw(tt), Cw(tt), Pw(rp0), ph == 4 ? pn : nullptr);
    }
    if (ph == 4) {
      const unsigned long long m = warp_max_bits((unsigned long long)__double_as_longlong(res));
      if ((tid & 31) == 0) wred[tid >> 5] = m;
      res = 0.0;
    }
    if (ph == 7) full_bc(pass == 1 ? U(ut) : nullptr, pass == 0 ? V(ut) : nullptr);
    if (ph == 4 || (uvp && doV && top && !ch)) {
      __syncthreads();
      if (uvp) top_v(V(out));
    }
    if (ph == 4 && tid >= NT - 32) {  // the CTA's maximum to every CTA
      const int lane = tid & 31;
      const unsigned long long b = warp_max_bits(lane < NT / 32 ? wred[lane] : 0ull);
      if (lane < K) st_cluster(map_cluster(smem_addr(&red[par][rank]), lane), __longlong_as_double((long long)b));
    }
    cl.sync();

    if (ph <= 3 || ph == 7) {
      if (ph == 2 && z) {
        pend = false;
        swap_tc();  // T_n_tau becomes T_tau
      }
      if (dirty && ph != 7) {
        st7 = ph;
        ph = 7;
        continue;
      }
      const int st = ph == 7 ? st7 : ph;
      if (st < 3) {
        ph = st + 1;
      } else if (dirty && pass == 0) {
        pass = 1;
        ph = 1;
      } else {
        if (corner) {
          // (imax, jmax+1) of vm_n_tau from the buffers' history, then the n_tau buffer's update
          if (dirty) {
            h1[R_TAU] = V(ut)[at(nx, ny - 1)];
            h2[R_TAU] = V(ut)[at(nx, ny - 2)];
          }
          double* vn = V(ua);
          const double c1 = h1[a.corner_role], c2 = h2[a.corner_role], n = 2.0 * c2 - c1;
          vn[at(nx, ny + 1)] = 2.0 * c1 - n;
          h1[R_NTAU] = vn[at(nx, ny - 1)];
          h2[R_NTAU] = vn[at(nx, ny - 2)];
        }
        pass = 0;
        ph = 4;
      }
      continue;
    }
    if (ph == 5) {
      ph = 6;
      continue;
    }
    if (ph == 4) {
      // ---- control (main.f90:139-157), identical in every thread of the cluster ----
      const int lane = tid & 31;
      e = __longlong_as_double((long long)warp_max_bits(lane < K ? red[par][lane] : 0ull));
      par ^= 1;
      pend = scal;
      p_made |= 1 << rp1;
      kk += 1;
      total += 1;
      if (e != e || e > 1.0e300) {
        fin = FAILED;
        pend = scal && a.tc_of_failed;
      } else if (itc != 1 && e < d.eps) {
        fin = EXIT;
      } else {
        // um_tau = um_n_tau, p = pn, ...: the windows change roles
        const int s = ut; ut = ua; ua = s;
        if (corner) {
          double y = h1[R_TAU]; h1[R_TAU] = h1[R_NTAU]; h1[R_NTAU] = y;
          y = h2[R_TAU]; h2[R_TAU] = h2[R_NTAU]; h2[R_NTAU] = y;
        }
        const int q = rp0; rp0 = rp1; rp1 = q;
        rp_read = rp0;
        ntau_alias = 2;
        t_made = scal;
        dirty = false;
        itc += 1;
        fin = itc >= d.itc_max ? CAP : GO;
      }
      if (fin == GO) {
        ph = 1;
        continue;
      }
      if (pend) {
        ph = 5;
        continue;
      }
    }
    // ---- a physical step ends (ph is 4 or 6) ----
    if (ph == 6 && fin == CAP) swap_tc();
    pend = false;
    if (fin == FAILED) {
      status = 2;
      active = false;
      store_rows(d.U[g.ru[R_NTAU]], U(ua));
      store_rows(d.V[g.rv[R_NTAU]], V(ua));
      if (ph == 6) {
        finish_c(Tw(ta), false, d.T_in);
        finish_c(Cw(ta), false, d.C_in);
        store_rows(d.T[g.rt[R_NTAU]], Tw(ta));
        store_rows(d.C[g.rc[R_NTAU]], Cw(ta));
      }
    } else {
      // EXIT: the tau copies are skipped and the new iterate becomes the physical-step state (its buffer
      // and n_tau's change roles); CAP: the loop condition failed after the copies, phys = latest iterate
      // (main.f90:142-157)
      const int iu = fin == EXIT ? ua : ut, iz = fin == EXIT ? ta : tt;
      __syncthreads();
      if (fin == EXIT) {
        if (tid == 0) {
          int s;
          s = g.ru[R_PHYS]; g.ru[R_PHYS] = g.ru[R_NTAU]; g.ru[R_NTAU] = s;
          s = g.rv[R_PHYS]; g.rv[R_PHYS] = g.rv[R_NTAU]; g.rv[R_NTAU] = s;
          if (d.solve_scalars) {
            s = g.rt[R_PHYS]; g.rt[R_PHYS] = g.rt[R_NTAU]; g.rt[R_NTAU] = s;
            s = g.rc[R_PHYS]; g.rc[R_PHYS] = g.rc[R_NTAU]; g.rc[R_NTAU] = s;
          }
        }
        if (corner) {
          const double y = h1[R_PHYS], q = h2[R_PHYS];
          h1[R_PHYS] = h1[R_NTAU]; h1[R_NTAU] = y;
          h2[R_PHYS] = h2[R_NTAU]; h2[R_NTAU] = q;
        }
        rp_read = rp1;
        ntau_alias = 1;
      } else if (corner) {
        h1[R_PHYS] = h1[R_TAU];
        h2[R_PHYS] = h2[R_TAU];
      }
      __syncthreads();
      phys_pointers();
      if (scal) {
        finish_c(Tw(iz), false, d.T_in);
        finish_c(Cw(iz), false, d.C_in);
      }
      store_rows(d.U[g.ru[R_PHYS]], U(iu));
      store_rows(d.V[g.rv[R_PHYS]], V(iu));
      if (scal) {
        store_rows(d.T[g.rt[R_PHYS]], Tw(iz));
        store_rows(d.C[g.rc[R_PHYS]], Cw(iz));
      }
      if constexpr (PHYS) {
        store_rows(pu, U(iu));
        store_rows(pv, V(iu));
        if (scal) {
          store_rows(pt, Tw(iz));
          store_rows(pc, Cw(iz));
        }
      }
      if (buoy && scal) set_buoy(Tw(iz));
      __syncthreads();
    }
    if (rank == 0 && tid == 0 && step < n_steps) {
      if (a.iters) a.iters[(long long)c * n_steps + step] = kk;
      if (a.err) a.err[(long long)c * n_steps + step] = e;
    }
    if (status != 2) {
      step += 1;
      itc = 0;
      kk = 0;
      if (step >= n_steps) { active = false; status = 1; }
    }
    fin = GO;
    ph = 1;
  }
  // ---- the state goes back to the case's buffers ----
  for (int k = 0; k < 2; ++k)
    if (p_made >> k & 1) finish_c(Pw(k), true, 0.0);
  if (t_made) {
    finish_c(Tw(tt), false, d.T_in);
    finish_c(Cw(tt), false, d.C_in);
  }
  __syncthreads();
  store_rows(d.U[g.ru[R_TAU]], U(ut));
  store_rows(d.V[g.rv[R_TAU]], V(ut));
  store_rows(d.P[0], Pw(0));
  store_rows(d.P[1], Pw(1));
  if (scal) {
    store_rows(d.T[g.rt[R_TAU]], Tw(tt));
    store_rows(d.C[g.rc[R_TAU]], Cw(tt));
  }
  if (rank == 0 && tid == 0) {
    for (int r = 0; r < 3; ++r) { gk->ru[r] = g.ru[r]; gk->rv[r] = g.rv[r]; gk->rt[r] = g.rt[r]; gk->rc[r] = g.rc[r]; }
    gk->rp[0] = rp0;
    gk->rp[1] = rp1;
    gk->rp_read = rp_read; gk->ntau_alias = ntau_alias; gk->itc = itc; gk->step = step;
    gk->k = kk; gk->active = 0; gk->status = status; gk->tau_dirty = dirty ? 1 : 0;
    gk->total_iters = total;
  }
  cl.sync();  // no CTA leaves while another may still store into its windows or read the control word
}

}  // namespace acs
