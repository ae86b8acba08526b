// Tiled kernels of the inert metric / face-boundary step, 2D in both precisions
// and 3D in single precision: the CFL rate, and one SSPRK2 stage in a single
// pass over the state.
//
// The separate kernels (tfv_metric.cuh; the other sessions keep them) write the
// primitives, the geometric source and every face flux of a stage to HBM and
// read them back, about 150 B per cell and stage in single precision.  Here a
// CTA owns a block of cells of the plane normal to the last axis and marches
// along that axis through a chunk of planes: the primitives of the current
// plane (with a two-cell halo) live in shared memory, the face fluxes of the
// plane too, the marching-axis neighbours and the marching faces in registers,
// and a stage reads the state once and writes it once.
//
// Work split.  Thread (a, b) of a BX x BY block forms its cell's limited slopes
// once, leaves the cell's upper x and y face states in shared memory and then
// forms the cell's low x and low y face from its own lower states and the
// neighbours' upper ones; the last column and row of threads only form faces,
// so a block updates (BX - 1) x (BY - 1) cells, every thread does the same two
// faces, and no warp takes a remainder of high-edge faces while the others
// wait.  In 3D one warp adds the upper states of the column and row before the
// block; in 2D the first thread stands on that column (BX - 2 cells a block), as
// a second round of slopes by one warp of a 32-thread block would cost as much
// as the first.  Two barriers per plane.
//
// Measured, 256 x 192 x 192 single precision: the two stages 571 and 611 us, the
// rate 130 us, a step 1330; the separate kernels took 837 us a stage (march and
// update 385, x faces 179, y faces 163, primitives 110) and 174 for the rate, a
// step 2020 with its reductions and host looks.  Bound by instruction issue and
// latency: 1261 instructions a cell, issue slots 51 to 56% busy from 16 warps per
// SM.
// Variants: three CTAs per SM (84 registers) spill, a step 1650 us; high-edge
// faces by the column of threads itself (no redundant slopes, one more barrier)
// 621 and 698 us.
//
// Values are those of the separate kernels: in double precision bit for bit
// (the same expressions in the same order), in single precision with
// reciprocals shared and the limiters of the Cartesian step but VanLeer
// (tile_slope).
//
// Reference: python/cfdSolver/torchFiniteVolume.py:16-276.
#pragma once

#include "tfv_metric.cuh"

namespace tfv {

constexpr int kMPlanes = 65;  // longest chunk of planes plus one

// In-plane block: BX x BY threads (2D: one row of BX).
template <int DIM>
struct MBlock {
  static constexpr int kThreads = DIM == 3 ? 256 : 128;
  static constexpr int kFirst = DIM == 3 ? 0 : 1;  // thread of the block's first cell along x
};

// dt of the stage: given by the host, or CFL / rate limited by the remaining
// time (torchSession.py:533-536), with the rate maximum still on the device.
template <typename R>
__device__ __forceinline__ double stage_dt(const MArgs<R>& A) {
  if (!A.dt_from_rate) return A.dt;
  const unsigned long long bits = *A.rate_max;
  const double rate = sizeof(R) == 8 ? __longlong_as_double((long long)bits)
                                     : (double)__uint_as_float((unsigned)bits);
  const double dt = soft_div(A.cfl, rate);
  return soft_lt(A.remaining, dt) ? A.remaining : dt;  // std::min(dt, remaining)
}

template <typename R, int NV>
__device__ __forceinline__ void prim_from(const R* u, R g, R* p) {
  if constexpr (Exact<R>::value) {
    primitive_of<R, NV>(u, g, p);
  } else {
    R s = u[1] * u[1];
#pragma unroll
    for (int c = 2; c < NV - 1; ++c) s = s + u[c] * u[c];
    const R ir = rcp(u[0]);
    p[0] = u[0];
#pragma unroll
    for (int c = 1; c < NV - 1; ++c) p[c] = u[c] * ir;
    p[NV - 1] = (g - R(1)) * (u[NV - 1] - R(0.5) * s * ir);
  }
}

// Component v of a state array at cell offset `at`: the component's base is
// uniform over the grid and the offset 32 bits (a component stays below 2^31
// cells), which spares the 64-bit address arithmetic of every access.  An
// ordinary load: a launch of these kernels may begin before the kernel that
// writes this state has ended, so the state is not read-only for the kernel's
// lifetime as a non-coherent load (ro) asks, and pdl_wait orders ordinary loads
// only.  ro is for the geometry factors, written once at bind.
template <typename R>
__device__ __forceinline__ R row(const R* base, int64_t nc, int v, uint32_t at) {
  return base[v * nc + at];
}

// Limited slope of one component (metric_limited).  Single-precision VanLeer,
// 2 minus plus / (minus + plus), takes the quotient first: the Cartesian step's
// product of the differences overflows where both exceed 1.8e19 (pressures in
// small units), and the infinite slope would cost the step its second order.
template <typename R, int LIM>
__device__ __forceinline__ R tile_slope(R m, R c, R p) {
  if constexpr (!Exact<R>::value && LIM == 0) {
    const R minus = c - m, plus = p - c;
    const R mp = minus * plus;  // its sign, and NaN for NaN
    const R v = (minus + minus) * (plus * rcp(minus + plus));
    return mp > R(0) ? v : (mp == mp ? R(0) : mp);
  }
  return limited_slope<R, 3, LIM>(m, c, p);
}

// Half slopes of a cell from its neighbours' primitives (cell_slope, halved).
template <typename R, int NV, int LIM>
__device__ __forceinline__ void half_slopes(const R* m, const R* c, const R* p, R* h) {
  R s0 = R(0), s1 = R(0);
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const R s = tile_slope<R, LIM>(m[v], c[v], p[v]);
    h[v] = hf(s);
    if (v == 0) s0 = h[v];
    if (v == NV - 1) s1 = h[v];
  }
  const bool bad = le_(c[0] - R(fabs(s0)), R(1e-12)) | le_(c[NV - 1] - R(fabs(s1)), R(1e-12));
  if (__any_sync(__activemask(), bad)) {  // rare: one vote instead of a select per row
    const R keep = bad ? R(0) : R(1);
#pragma unroll
    for (int v = 0; v < NV; ++v) h[v] = h[v] * keep;
  }
}

// Area-weighted Rusanov flux along D between reconstructed primitive states,
// mirrored at walls (face_flux without fractions, constant gamma).
template <typename R, int DIM, int D>
__device__ __forceinline__ void rusanov_states(const MArgs<R>& A, R* left, R* right, bool edge,
                                               bool wall_lo, bool wall_hi, R ar, R* W) {
  constexpr int NV = DIM + 2;
  constexpr int E = NV - 1;
  if (edge) {  // uniform: the tile touches a domain face of this direction
    if (wall_lo) {
#pragma unroll
      for (int v = 0; v < NV; ++v) left[v] = v == D + 1 ? -right[v] : right[v];
    }
    if (wall_hi) {
#pragma unroll
      for (int v = 0; v < NV; ++v) right[v] = v == D + 1 ? -left[v] : left[v];
    }
  }
  R ul[NV], ur[NV], fl[NV], fr[NV];
  R cl, cr;
  if constexpr (Exact<R>::value) {
    conservative_of<R, NV>(left, A.gam, ul);
    conservative_of<R, NV>(right, A.gam, ur);
    cl = rt(qd(A.gam * left[E], left[0]));
    cr = rt(qd(A.gam * right[E], right[0]));
  } else {
    R sl = left[1] * left[1], sr = right[1] * right[1];
#pragma unroll
    for (int v = 2; v < E; ++v) {
      sl = sl + left[v] * left[v];
      sr = sr + right[v] * right[v];
    }
#pragma unroll
    for (int v = 0; v < E; ++v) {
      ul[v] = v == 0 ? left[0] : left[v] * left[0];
      ur[v] = v == 0 ? right[0] : right[v] * right[0];
    }
    ul[E] = left[E] * A.igm1 + R(0.5) * left[0] * sl;
    ur[E] = right[E] * A.igm1 + R(0.5) * right[0] * sr;
    cl = rt(A.gam * left[E] * rcp(left[0]));
    cr = rt(A.gam * right[E] * rcp(right[0]));
  }
  const R vl = left[D + 1], vr = right[D + 1];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    fl[v] = ul[v] * vl;
    fr[v] = ur[v] * vr;
  }
  fl[D + 1] = fl[D + 1] + left[E];
  fr[D + 1] = fr[D + 1] + right[E];
  fl[E] = fl[E] + vl * left[E];
  fr[E] = fr[E] + vr * right[E];
  const R speed = np_max(R(fabs(vl)) + cl, R(fabs(vr)) + cr);
  if constexpr (Exact<R>::value) {
#pragma unroll
    for (int v = 0; v < NV; ++v) W[v] = hf((fl[v] + fr[v]) - (ur[v] - ul[v]) * speed) * ar;
  } else {
    const R ha = hf(ar);
#pragma unroll
    for (int v = 0; v < NV; ++v) W[v] = ((fl[v] + fr[v]) - (ur[v] - ul[v]) * speed) * ha;
  }
}

// What a thread stages: the cell at in-plane position (gx, gy) of the padded
// plane.  kind 0: nothing; 1: a cell of the domain (or its periodic image);
// 2 + 2 d + (side > 0): the ghost beyond face `side` of direction d.
struct MItem {
  int off;
  int kind;
};
template <typename R, int DIM>
__device__ __forceinline__ MItem stage_item(const MArgs<R>& A, int gx, int gy) {
  const int nx = A.n[0], ny = DIM == 3 ? A.n[1] : 1;
  MItem it;
  it.off = 0;
  it.kind = 1;
  const bool ox = gx < 0 || gx >= nx, oy = gy < 0 || gy >= ny;
  if (ox && oy) {
    it.kind = 0;
    return it;
  }
  if (ox) {
    if (A.periodic[0]) {
      gx = gx < 0 ? gx + nx : gx - nx;
      if (gx < 0 || gx >= nx) it.kind = 0;  // beyond the second halo cell
    } else if (gx == -1 || gx == nx) {
      it.kind = gx < 0 ? 2 : 3;
      gx = gx < 0 ? 0 : nx - 1;
    } else {
      it.kind = 0;
    }
  }
  if (oy) {
    if (A.periodic[1]) {
      gy = gy < 0 ? gy + ny : gy - ny;
      if (gy < 0 || gy >= ny) it.kind = 0;
    } else if (gy == -1 || gy == ny) {
      it.kind = gy < 0 ? 4 : 5;
      gy = gy < 0 ? 0 : ny - 1;
    } else {
      it.kind = 0;
    }
  }
  if (it.kind) it.off = gy * nx + gx;
  return it;
}

// Source plane of padded plane k along the marching axis (n planes), and the
// side of the ghost it stands for (0: a cell of the domain or periodic image).
__device__ __forceinline__ int march_plane(int k, int n, bool periodic, int& side) {
  side = 0;
  if (k >= 0 && k < n) return k;
  if (periodic) return k < 0 ? k + n : k - n;
  side = k < 0 ? -1 : 1;
  return k < 0 ? 0 : n - 1;
}

template <typename R, int NV>
__device__ __forceinline__ int ghost_prim(const MArgs<R>& A, int d, int side, R* p) {
  MCell<R, NV> c;
#pragma unroll
  for (int v = 0; v < NV; ++v) c.p[v] = p[v];
  c.g = A.gam;
  c.q[0] = c.q[1] = R(0);
  const int err = ghost_state<R, NV>(A, A.face[2 * d + (side > 0)], d, side, c);
#pragma unroll
  for (int v = 0; v < NV; ++v) p[v] = c.p[v];
  return err;
}

// Primitives of a staged item from its conserved state u.
template <typename R, int NV>
__device__ __forceinline__ int item_prim(const MArgs<R>& A, int kind, const R* u, R* p) {
  prim_from<R, NV>(u, A.gam, p);
  return kind > 1 ? ghost_prim<R, NV>(A, (kind - 2) >> 1, (kind & 1) ? 1 : -1, p) : 0;
}

// Tile coordinates of block t: x fastest, then y, then the chunk.
template <typename R, int DIM>
struct MTile {
  int x0, y0, p0, p1;
  __device__ __forceinline__ MTile(const MArgs<R>& A, int t, int bx, int by) {
    const int tx = t % A.ntx, r = t / A.ntx;
    const int ty = DIM == 3 ? r % A.nty : 0, ch = DIM == 3 ? r / A.nty : r;
    x0 = tx * (bx - 1 - MBlock<DIM>::kFirst);
    y0 = DIM == 3 ? ty * (by - 1) : 0;
    p0 = ch * A.chunk;
    p1 = min(p0 + A.chunk, A.n[DIM - 1]);
  }
};

// -- one SSPRK2 stage -------------------------------------------------------------
// stage 1: Uout = U + dt K; stage 2: Uout = 0.5 (U0 + U + dt K)
// (torchFiniteVolume.py:234-276).  Block partials of the source and of the
// outward boundary fluxes go to tpart[tile][16] (source rows 0.., outward rows
// 8..).
template <typename R, int DIM, int LIM, int BX, int BY>
__global__ void __launch_bounds__(MBlock<DIM>::kThreads, TFV_STAGE_MIN_BLOCKS)
    metric_stage_kernel(MArgs<R> A, int stage) {
  constexpr int NV = DIM + 2;
  constexpr int MD = DIM - 1;
  constexpr int O = MBlock<DIM>::kFirst;
  constexpr int W = BX + 3;                     // staged columns -2 - O .. BX - O
  constexpr int NP = W * (DIM == 3 ? BY + 3 : 1);  // staged cells of a plane
  constexpr int NB = BX * BY;
  extern __shared__ __align__(16) unsigned char mstage_smem[];
  double* bs = reinterpret_cast<double*>(mstage_smem);  // edge-face sums [2][BY][NV], [2][BX][NV], [2][NV]
  constexpr int kXs = 2 * BY * NV, kYs = DIM == 3 ? 2 * BX * NV : 0;
  double* red = bs + kXs + kYs + 2 * NV;
  R* pl = reinterpret_cast<R*>(red + 40);  // primitives of the plane [NV][NP]
  R* ux = pl + NV * NP;                    // upper x states of columns -1 .. BX - 1 [NV][BY][BX + 1]
  constexpr int NX = BY * (BX + 1);
  R* uy = ux + NV * NX;                    // upper y states of rows -1 .. BY - 1 [NV][BY + 1][BX]
  constexpr int NY = DIM == 3 ? (BY + 1) * BX : 0;
  R* fxp = uy + NV * NY;                   // low face fluxes [MD][NV][NB]
  R* pf = fxp + MD * NV * NB;              // marching-axis factors of the chunk [4][kMPlanes]
  __shared__ double sh_dt;
  const int tid = threadIdx.x;
  pdl_wait();
  if (tid == 0) sh_dt = stage_dt(A);
  for (int e = tid; e < kXs + kYs + 2 * NV; e += NB) bs[e] = 0.0;
  // cells that no thread stages (corners, beyond a ghost) hold ones: their
  // slopes are formed and dropped
  for (int e = tid; e < NV * NP; e += NB) pl[e] = R(1);
  const MTile<R, DIM> T(A, blockIdx.x, BX, BY);
  const int np = A.n[MD];
  for (int e = tid; e <= T.p1 - T.p0; e += NB) {
    const int k = T.p0 + e;
    if (k < np) {
      pf[e] = ro(&A.ff[0][MD][k]);
      pf[kMPlanes + e] = DIM == 3 ? ro(&A.ff[1][MD][k]) : R(0);
      pf[2 * kMPlanes + e] = ro(&A.vf[MD][k]);
    }
    pf[3 * kMPlanes + e] = ro(&A.ff[MD][MD][k]);
  }
  __syncthreads();
  const R dt = R(sh_dt);
  const int nx = A.n[0], ny = DIM == 3 ? A.n[1] : 1;
  const int ps = nx * ny;
  const int a = tid % BX - O, b = DIM == 3 ? tid / BX : 0;  // cell of the block
  const int gx = T.x0 + a, gy = T.y0 + b;
  const bool col = gx < nx && a >= 0 && a < BX - 1 - O;
  const bool rowok = DIM == 2 || (gy < ny && b < BY - 1);
  const bool owner = col && rowok;
  const bool fx_on = gx <= nx && a >= 0 && rowok;                // low x face of (gx, gy)
  const bool fy_on = DIM == 3 && gy <= ny && col;                // low y face
  const bool perx = A.periodic[0], pery = DIM == 3 && A.periodic[1], perz = A.periodic[MD];
  const bool fo = A.first_order != 0;
  // own cell and at most one halo cell per thread
  const int nhalo = DIM == 3 ? 3 * BY + 3 * BX : 2;
  int ha = 0, hb = 0;
  if (DIM == 2) {
    ha = tid == 0 ? -2 : BX - 1;
  } else if (tid < 3 * BY) {
    const int k = tid / BY;
    ha = k == 2 ? BX : k - 2;
    hb = tid % BY;
  } else {
    const int r = tid - 3 * BY, k = r / BX;
    hb = k == 2 ? BY : k - 2;
    ha = r % BX;
  }
  const MItem own = stage_item<R, DIM>(A, gx, gy);
  MItem halo;
  halo.off = halo.kind = 0;
  if (tid < nhalo) halo = stage_item<R, DIM>(A, T.x0 + ha, T.y0 + hb);
  const int own_at = (DIM == 3 ? (b + 2) * W : 0) + a + 2;
  const int halo_at = (DIM == 3 ? (hb + 2) * W : 0) + ha + 2;
  int err = 0;
  // geometry: products of the x and y factors of this column
  R ax_lo = R(0), ax_hi = R(0), ay_lo = R(0), ay_hi = R(0), az = R(0), vxy = R(0);
  if (fx_on) ax_lo = DIM == 3 ? ro(&A.ff[0][0][gx]) * ro(&A.ff[0][1][gy]) : ro(&A.ff[0][0][gx]);
  if (owner) {
    ax_hi = DIM == 3 ? ro(&A.ff[0][0][gx + 1]) * ro(&A.ff[0][1][gy]) : ro(&A.ff[0][0][gx + 1]);
    az = DIM == 3 ? ro(&A.ff[2][0][gx]) * ro(&A.ff[2][1][gy]) : ro(&A.ff[1][0][gx]);
    vxy = DIM == 3 ? ro(&A.vf[0][gx]) * ro(&A.vf[1][gy]) : ro(&A.vf[0][gx]);
    if (DIM == 3) ay_hi = ro(&A.ff[1][0][gx]) * ro(&A.ff[1][1][gy + 1]);
  }
  if (fy_on) ay_lo = ro(&A.ff[1][0][gx]) * ro(&A.ff[1][1][gy]);
  const bool wx_lo = gx == 0 && A.face[0].type == kFaceWall;
  const bool wx_hi = gx == nx && A.face[1].type == kFaceWall;
  const bool wy_lo = DIM == 3 && gy == 0 && A.face[2].type == kFaceWall;
  const bool wy_hi = DIM == 3 && gy == ny && A.face[3].type == kFaceWall;
  const bool edge_x = T.x0 == 0 || nx - T.x0 <= BX - 1 - O;
  const bool edge_y = DIM == 3 && (T.y0 == 0 || ny - T.y0 <= BY - 1);
  const bool wz_lo = A.face[2 * MD].type == kFaceWall, wz_hi = A.face[2 * MD + 1].type == kFaceWall;

  auto load = [&](int k, int off, R* u) {
    int side;
    const uint32_t at = (uint32_t)(march_plane(k, np, perz, side) * ps + off);
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = row(A.U, A.nc, v, at);
  };
  // this column's primitives at plane k (ghost planes by the boundary rules)
  auto column = [&](int k, const R* u, R* p) {
    err |= item_prim<R, NV>(A, own.kind, u, p);
    if (!perz && owner && (k == -1 || k == np)) err |= ghost_prim<R, NV>(A, MD, k < 0 ? -1 : 1, p);
  };

  R pm[NV], pc[NV], top[NV], fprev[NV], part[NV];
  R un[NV], uh[NV];  // conserved states of the plane being staged
#pragma unroll
  for (int v = 0; v < NV; ++v) pm[v] = pc[v] = top[v] = fprev[v] = part[v] = uh[v] = R(0);
  const bool active = own.kind != 0;
  if (active) {
    // planes p0 - 2, p0 - 1, p0 of the column: the upper face state of p0 - 1
    R u[NV], p2[NV], h[NV];
    if (T.p0 >= 2 || perz) {
      load(T.p0 - 2, own.off, u);
      column(T.p0 - 2, u, p2);
    } else {
#pragma unroll
      for (int v = 0; v < NV; ++v) p2[v] = R(1);
    }
    load(T.p0 - 1, own.off, u);
    column(T.p0 - 1, u, pm);
    load(T.p0, own.off, u);
    column(T.p0, u, pc);
#pragma unroll
    for (int v = 0; v < NV; ++v) h[v] = R(0);
    // at p0 == 1 the plane below p0 - 1 is the ghost plane, loaded above only
    // when periodic
    if (T.p0 == 1 && !perz) {
      load(-1, own.off, u);
      column(-1, u, p2);
    }
    if (!fo && (T.p0 >= 1 || perz)) half_slopes<R, NV, LIM>(p2, pm, pc, h);
#pragma unroll
    for (int v = 0; v < NV; ++v) top[v] = pm[v] + h[v];
#pragma unroll
    for (int v = 0; v < NV; ++v) pl[v * NP + own_at] = pc[v];
    load(T.p0 + 1, own.off, un);
  } else {
#pragma unroll
    for (int v = 0; v < NV; ++v) un[v] = R(1);
  }
  if (halo.kind) {
    R u[NV], p[NV];
    load(T.p0, halo.off, u);
    err |= item_prim<R, NV>(A, halo.kind, u, p);
#pragma unroll
    for (int v = 0; v < NV; ++v) pl[v * NP + halo_at] = p[v];
    if (T.p0 + 1 < T.p1) load(T.p0 + 1, halo.off, uh);
  }
  // source sums of this column: rows 1 .. DIM (the others are zero)
  double src[DIM];
  R ks[DIM], kc[DIM];
#pragma unroll
  for (int v = 0; v < DIM; ++v) {
    src[v] = 0.0;
    ks[v] = kc[v] = R(0);
  }
  __syncthreads();

  // the slope of a cell counts unless the cell is a ghost (or the step is first
  // order); periodic images keep theirs
  const bool keep_x = !fo && (perx || (gx >= 0 && gx < nx));
  const bool keep_y = !fo && DIM == 3 && (pery || gy < ny);
  // cells before the block whose upper states one warp adds: column -1 (lanes
  // 0 .. BY - 1) and row -1 (the next BX lanes)
  const bool edge_lane = DIM == 3 && tid < BY + BX;
  const bool lane_x = tid < BY;
  const int lane_at = lane_x ? (tid + 2) * W + 1 : W + (tid - BY) + 2;
  const int lane_d = lane_x ? 1 : W;
  const bool lane_keep = !fo && (lane_x ? (perx || T.x0 > 0) : (pery || T.y0 > 0));
  const int lane_to = lane_x ? tid * (BX + 1) : tid - BY;

  for (int it = T.p0; it <= T.p1; ++it) {
    const bool full = it < T.p1;
    // 1. slopes of plane it, upper states of its cells
    R lx[NV], ly[NV];
    if (full) {
      R h[NV], n0[NV], n1[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        n0[v] = pl[v * NP + own_at - 1];
        n1[v] = pl[v * NP + own_at + 1];
      }
      half_slopes<R, NV, LIM>(n0, pc, n1, h);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (!keep_x) h[v] = R(0);
        lx[v] = pc[v] - h[v];
        ux[v * NX + (DIM == 3 ? b * (BX + 1) : 0) + a + 1] = pc[v] + h[v];
      }
      if (DIM == 3) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          n0[v] = pl[v * NP + own_at - W];
          n1[v] = pl[v * NP + own_at + W];
        }
        half_slopes<R, NV, LIM>(n0, pc, n1, h);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          if (!keep_y) h[v] = R(0);
          ly[v] = pc[v] - h[v];
          uy[v * NY + (b + 1) * BX + a] = pc[v] + h[v];
        }
      }
      if (DIM == 3 && edge_lane) {
        R c[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          n0[v] = pl[v * NP + lane_at - lane_d];
          c[v] = pl[v * NP + lane_at];
          n1[v] = pl[v * NP + lane_at + lane_d];
        }
        half_slopes<R, NV, LIM>(n0, c, n1, h);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const R u = lane_keep ? c[v] + h[v] : c[v];
          if (lane_x) ux[v * NX + lane_to] = u;
          else uy[v * NY + lane_to] = u;
        }
      }
    }
    // conserved states of the cell that this plane's marching face completes,
    // loaded ahead of their use
    R ue[NV], u0e[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) ue[v] = u0e[v] = R(0);
    if (owner && it > T.p0) {
      const uint32_t off = (uint32_t)((it - 1) * ps + own.off);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        ue[v] = row(A.U, A.nc, v, off);
        if (stage == 2) u0e[v] = row(A.U0, A.nc, v, off);
      }
    }
    __syncthreads();  // upper states complete, plane it read
    // 2. stage plane it + 1, start loading it + 2
    R pp[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) pp[v] = R(1);
    if (active) {
      column(it + 1, un, pp);
      if (full) {
#pragma unroll
        for (int v = 0; v < NV; ++v) pl[v * NP + own_at] = pp[v];
        load(it + 2, own.off, un);
      }
    }
    if (halo.kind && it + 1 < T.p1) {
      R p[NV];
      err |= item_prim<R, NV>(A, halo.kind, uh, p);
#pragma unroll
      for (int v = 0; v < NV; ++v) pl[v * NP + halo_at] = p[v];
      if (it + 2 < T.p1) load(it + 2, halo.off, uh);
    }
    // low x and low y faces of plane it
    if (full && fx_on) {
      R left[NV], F[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) left[v] = ux[v * NX + (DIM == 3 ? b * (BX + 1) : 0) + a];
      const R ar = ax_lo * pf[it - T.p0];
      rusanov_states<R, DIM, 0>(A, left, lx, edge_x, wx_lo, wx_hi, ar, F);
#pragma unroll
      for (int v = 0; v < NV; ++v) fxp[v * NB + tid] = F[v];
    }
    if (DIM == 3 && full && fy_on) {
      R left[NV], F[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) left[v] = uy[v * NY + b * BX + a];
      const R ar = ay_lo * pf[kMPlanes + it - T.p0];
      rusanov_states<R, DIM, 1>(A, left, ly, edge_y, wy_lo, wy_hi, ar, F);
#pragma unroll
      for (int v = 0; v < NV; ++v) fxp[(NV + v) * NB + tid] = F[v];
    }
    // 3. marching face below plane it; cell it - 1 is complete
    R fz[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) fz[v] = R(0);
    if (owner) {
      R h[NV], low[NV], tl[NV];
      half_slopes<R, NV, LIM>(pm, pc, pp, h);
      const bool keep_z = !fo && (perz || it < np);  // plane np is a ghost
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        if (!keep_z) h[v] = R(0);
        low[v] = pc[v] - h[v];
        tl[v] = top[v];
        top[v] = pc[v] + h[v];
      }
      const R ar = az * pf[3 * kMPlanes + it - T.p0];
      rusanov_states<R, DIM, MD>(A, tl, low, it == 0 || it == np, it == 0 && wz_lo,
                                 it == np && wz_hi, ar, fz);
      if (it > T.p0) {
        const int k = it - 1;
        const uint32_t off = (uint32_t)(k * ps + own.off);
        R out[NV];
        const R vol = vxy * pf[2 * kMPlanes + k - T.p0];
        const Divisor<R> dv_(vol);
        const R iv = Exact<R>::value ? R(0) : rcp(vol);
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const R df = fz[v] - fprev[v];
          const R kk = part[v] - (Exact<R>::value ? qd(df, dv_) : df * iv);
          if (stage == 1)
            out[v] = ue[v] + dt * kk;
          else
            out[v] = hf((u0e[v] + ue[v]) + dt * kk);
        }
        if (!physical_cell<R, NV>(out)) err |= kMErrNonphysical;
#pragma unroll
        for (int v = 0; v < NV; ++v) (A.Uout + v * A.nc)[off] = out[v];
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) fprev[v] = fz[v];
    }
    if (it == 0 || it == np) {  // marching-axis boundary faces (uniform)
      FaceFlux<R, NV> ff;
#pragma unroll
      for (int v = 0; v < NV; ++v) ff.v[v] = fz[v];
      march_boundary_sum<R, NV>(ff, red, bs + kXs + kYs + (it == 0 ? 0 : NV));
    }
    if (!full) break;
    __syncthreads();  // fluxes of plane it and primitives of plane it + 1 complete
    // 4. source and in-plane divergence of cell it
    if (owner) {
      const R fv = pf[2 * kMPlanes + it - T.p0];
      const R vol = vxy * fv;
      const Divisor<R> dv_(vol);
      const R iv = Exact<R>::value ? R(0) : rcp(vol);
      auto pv = [&](R x) { return Exact<R>::value ? qd(x, dv_) : x * iv; };
      R s[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) s[v] = R(0);
      if (A.geometry != kGeoCartesian) {  // torchGeometry.py:177-204
        const R f0 = pf[it - T.p0];
        const R rho = pc[0], pr = pc[NV - 1];
        const R radial = pv(ax_hi * f0 - ax_lo * f0);
        s[1] = pr * radial;
        if (A.geometry == kGeoSpherical) {
          const R invr = hf(radial);
          R sq = pc[2] * pc[2];
          if (DIM == 3) sq = sq + pc[DIM] * pc[DIM];
          s[1] = s[1] + (rho * sq) * invr;
          R cot;
          if (DIM == 3) {
            const R f1 = pf[kMPlanes + it - T.p0];
            cot = pv(ay_hi * f1 - ay_lo * f1);
          } else {
            const R g0 = ro(&A.ff[1][0][gx]);
            cot = pv(g0 * ro(&A.ff[1][1][it + 1]) - g0 * ro(&A.ff[1][1][it]));
          }
          s[2] = pr * cot - ((rho * pc[1]) * pc[2]) * invr;
          if (DIM == 3) {
            s[2] = s[2] + (rho * (pc[DIM] * pc[DIM])) * cot;
            s[DIM] = ((-rho) * pc[DIM]) * (pc[1] * invr + pc[2] * cot);
          }
        } else if (!(A.geometry == kGeoCylindrical && DIM == 2)) {
          s[1] = s[1] + (rho * (pc[2] * pc[2])) * radial;
          s[2] = (((-rho) * pc[1]) * pc[2]) * radial;
        }
#pragma unroll
        for (int v = 0; v < DIM; ++v) {
          if constexpr (Exact<R>::value) {
            src[v] += s[v + 1] * vol;
          } else {
            const R y = s[v + 1] * vol - kc[v];
            const R t = ks[v] + y;
            kc[v] = (t - ks[v]) - y;
            ks[v] = t;
          }
        }
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        part[v] = s[v] - pv(fxp[v * NB + tid + 1] - fxp[v * NB + tid]);
        if (DIM == 3) part[v] = part[v] - pv(fxp[(NV + v) * NB + tid + BX] - fxp[(NV + v) * NB + tid]);
      }
    }
    // FP64 sums of the domain-boundary in-plane faces (tiles at an edge)
    const int ex = nx - T.x0, ey = ny - T.y0;  // local index of the last face
    if (edge_x || edge_y) {
      for (int e = tid; e < kXs + kYs; e += NB) {
        if (e < kXs) {
          const int side = e / (BY * NV), j = (e / NV) % BY, v = e % NV;
          const bool in = DIM == 2 || (j < BY - 1 && T.y0 + j < ny);
          if (in && (side ? ex <= BX - 1 - O : T.x0 == 0))
            bs[e] += (double)fxp[v * NB + j * BX + (side ? ex : 0) + O];
        } else {
          const int q = e - kXs;
          const int side = q / (BX * NV), i = (q / NV) % BX, v = q % NV;
          if (i < BX - 1 && T.x0 + i < nx && (side ? ey <= BY - 1 : T.y0 == 0))
            bs[e] += (double)fxp[(NV + v) * NB + (side ? ey : 0) * BX + i];
        }
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      pm[v] = pc[v];
      pc[v] = pp[v];
    }
  }
  if (err) atomicOr(A.err, err);
  // tile record: source rows, then the outward sums of the boundary faces
  double* out = A.tpart + (size_t)blockIdx.x * 16;
#pragma unroll
  for (int v = 0; v < DIM; ++v) {
    if constexpr (!Exact<R>::value) src[v] = (double)ks[v] - (double)kc[v];
    const double t = block_sum(src[v], red);  // barriers: bs complete too
    if (tid == 0) out[1 + v] = t;
  }
  if (tid < NV) {
    double t = 0.0;
    for (int j = 0; j < BY; ++j) t += bs[(BY + j) * NV + tid] - bs[j * NV + tid];
    if (DIM == 3)
      for (int i = 0; i < BX; ++i) t += bs[kXs + (BX + i) * NV + tid] - bs[kXs + i * NV + tid];
    t += bs[kXs + kYs + NV + tid] - bs[kXs + kYs + tid];
    out[8 + tid] = t;
    if (tid == 0) out[0] = 0.0;
    if (tid == NV - 1) out[tid] = 0.0;
  }
}

// -- CFL rate ------------------------------------------------------------------------
// Sum over directions of max(area * face speed) / volume, maximum over the
// cells (torchFiniteVolume.py:74-102), from the state itself: |u_d| + a of a
// plane in shared memory, of the marching neighbours in registers (256 x 192 x
// 192, FP32: 283 us for the separate primitive and rate passes).  A variant
// without shared memory (30 cells and four rows a warp, shuffles along x) ran
// 226 us: its few boundary warps form each row's boundary state in turn.
template <typename R, int DIM, int BX, int BY>
__global__ void __launch_bounds__(MBlock<DIM>::kThreads, sizeof(R) == 4 ? 4 : 2)
    metric_rate_tile_kernel(MArgs<R> A) {
  constexpr int NV = DIM + 2;
  constexpr int MD = DIM - 1;
  constexpr int NB = BX * BY;
  constexpr int O = MBlock<DIM>::kFirst;
  constexpr int W = BX + 1;                        // columns -1 - O .. BX - 1 - O
  constexpr int NP = W * (DIM == 3 ? BY + 1 : 1);
  __shared__ R sp[2][MD][NP];  // |u_x| + a, |u_y| + a
  __shared__ R pf[4 * kMPlanes];
  __shared__ double red[40];
  pdl_wait();
  const int tid = threadIdx.x;
  const MTile<R, DIM> T(A, blockIdx.x, BX, BY);
  const int nx = A.n[0], ny = DIM == 3 ? A.n[1] : 1, np = A.n[MD];
  const int ps = nx * ny;
  for (int e = tid; e <= T.p1 - T.p0; e += NB) {
    const int k = T.p0 + e;
    if (k < np) {
      pf[e] = ro(&A.ff[0][MD][k]);
      pf[kMPlanes + e] = DIM == 3 ? ro(&A.ff[1][MD][k]) : R(0);
      pf[2 * kMPlanes + e] = ro(&A.vf[MD][k]);
    }
    pf[3 * kMPlanes + e] = ro(&A.ff[MD][MD][k]);
  }
  const int a = tid % BX - O, b = DIM == 3 ? tid / BX : 0;
  const int gx = T.x0 + a, gy = T.y0 + b;
  const bool owner = gx < nx && a >= 0 && a < BX - 1 - O && (DIM == 2 || (gy < ny && b < BY - 1));
  const bool perz = A.periodic[MD];
  // the column and row before the block (the ones after it are threads' own)
  const int nhalo = DIM == 3 ? BY + BX : 0;  // 2D: the first thread's own
  const int ha = tid < BY ? -1 : tid - BY;
  const int hb = tid < BY ? tid : -1;
  const MItem own = stage_item<R, DIM>(A, gx, gy);
  MItem halo;
  halo.off = halo.kind = 0;
  if (tid < nhalo) halo = stage_item<R, DIM>(A, T.x0 + ha, T.y0 + hb);
  const int own_at = (DIM == 3 ? (b + 1) * W : 0) + a + 1;
  const int halo_at = DIM == 3 ? (hb + 1) * W + ha + 1 : 0;
  int err = 0;
  auto load = [&](int k, int off, R* u) {
    int side;
    const uint32_t at = (uint32_t)(march_plane(k, np, perz, side) * ps + off);
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = row(A.U, A.nc, v, at);
  };
  auto speeds = [&](int k, int kind, const R* u, R* s, bool column) {
    R p[NV];
    err |= item_prim<R, NV>(A, kind, u, p);
    if (column && !perz && (k == -1 || k == np))
      err |= ghost_prim<R, NV>(A, MD, k < 0 ? -1 : 1, p);
    const R c = Exact<R>::value ? rt(qd(A.gam * p[NV - 1], p[0])) : rt(A.gam * p[NV - 1] * rcp(p[0]));
#pragma unroll
    for (int d = 0; d < DIM; ++d) s[d] = R(fabs(p[d + 1])) + c;
  };
  R ax_lo = R(0), ax_hi = R(0), ay_lo = R(0), ay_hi = R(0), az = R(0), vxy = R(0);
  if (owner) {
    const R f1 = DIM == 3 ? ro(&A.ff[0][1][gy]) : R(1);
    ax_lo = DIM == 3 ? ro(&A.ff[0][0][gx]) * f1 : ro(&A.ff[0][0][gx]);
    ax_hi = DIM == 3 ? ro(&A.ff[0][0][gx + 1]) * f1 : ro(&A.ff[0][0][gx + 1]);
    az = DIM == 3 ? ro(&A.ff[MD][0][gx]) * ro(&A.ff[MD][1][gy]) : ro(&A.ff[MD][0][gx]);
    vxy = DIM == 3 ? ro(&A.vf[0][gx]) * ro(&A.vf[1][gy]) : ro(&A.vf[0][gx]);
    if (DIM == 3) {
      ay_lo = ro(&A.ff[1][0][gx]) * ro(&A.ff[1][1][gy]);
      ay_hi = ro(&A.ff[1][0][gx]) * ro(&A.ff[1][1][gy + 1]);
    }
  }
  const bool active = own.kind != 0;
  R sc[DIM], sm = R(0), un[NV], uh[NV];
#pragma unroll
  for (int d = 0; d < DIM; ++d) sc[d] = R(0);
#pragma unroll
  for (int v = 0; v < NV; ++v) un[v] = uh[v] = R(1);
  if (active) {
    R u[NV], s[DIM];
    load(T.p0 - 1, own.off, u);
    speeds(T.p0 - 1, own.kind, u, s, owner);
    sm = s[MD];
    load(T.p0, own.off, u);
    speeds(T.p0, own.kind, u, sc, owner);
#pragma unroll
    for (int d = 0; d < MD; ++d) sp[0][d][own_at] = sc[d];
    load(T.p0 + 1, own.off, un);
  }
  if (halo.kind) {
    R u[NV], s[DIM];
    load(T.p0, halo.off, u);
    speeds(T.p0, halo.kind, u, s, false);
#pragma unroll
    for (int d = 0; d < MD; ++d) sp[0][d][halo_at] = s[d];
    if (T.p0 + 1 < T.p1) load(T.p0 + 1, halo.off, uh);
  }
  __syncthreads();
  R best = R(0);
  for (int it = T.p0; it < T.p1; ++it) {
    const int cur = (it - T.p0) & 1, e = it - T.p0;
    R sn[DIM];
#pragma unroll
    for (int d = 0; d < DIM; ++d) sn[d] = R(0);
    if (active) {
      speeds(it + 1, own.kind, un, sn, owner);
#pragma unroll
      for (int d = 0; d < MD; ++d) sp[cur ^ 1][d][own_at] = sn[d];
      if (it + 1 < T.p1) load(it + 2, own.off, un);
    }
    if (halo.kind && it + 1 < T.p1) {
      R s[DIM];
      speeds(it + 1, halo.kind, uh, s, false);
#pragma unroll
      for (int d = 0; d < MD; ++d) sp[cur ^ 1][d][halo_at] = s[d];
      if (it + 2 < T.p1) load(it + 2, halo.off, uh);
    }
    if (owner) {
      const R f0 = pf[e], vol = vxy * pf[2 * kMPlanes + e];
      const R mx = np_max((ax_lo * f0) * np_max(sp[cur][0][own_at - 1], sc[0]),
                          (ax_hi * f0) * np_max(sc[0], sp[cur][0][own_at + 1]));
      R my = R(0);
      if (DIM == 3) {
        const R f1 = pf[kMPlanes + e];
        my = np_max((ay_lo * f1) * np_max(sp[cur][MD - 1][own_at - W], sc[1]),
                    (ay_hi * f1) * np_max(sc[1], sp[cur][MD - 1][own_at + W]));
      }
      const R z0 = az * pf[3 * kMPlanes + e], z1 = az * pf[3 * kMPlanes + e + 1];
      const R mz = np_max(z0 * np_max(sm, sc[MD]), z1 * np_max(sc[MD], sn[MD]));
      R rate;
      if constexpr (Exact<R>::value) {
        const Divisor<R> dv_(vol);
        rate = qd(mx, dv_);
        if (DIM == 3) rate = rate + qd(my, dv_);
        rate = rate + qd(mz, dv_);
      } else {
        rate = ((mx + my) + mz) * rcp(vol);
      }
      if (!finite_(rate)) err |= kMErrRate;
      best = np_max(best, rate);
      sm = sc[MD];
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) sc[d] = sn[d];
    __syncthreads();
  }
  const R top = block_max(best, red);
  if (tid == 0 && top > R(0)) {
    if constexpr (Exact<R>::value)
      atomicMax(A.rate_max, (unsigned long long)__double_as_longlong(top));
    else
      atomicMax(A.rate_max, (unsigned long long)__float_as_uint(top));
  }
  if (err) atomicOr(A.err, err);
}

}  // namespace tfv
