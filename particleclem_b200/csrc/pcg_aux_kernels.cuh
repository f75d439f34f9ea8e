// pcg_aux_kernels.cuh -- the steps either side of the advance: the CFL timestep
// reduction, the state update with the temperature Newton solve, and the single-level
// ghost fill. All FP64.
#pragma once

#include <cooperative_groups.h>

#include "pcg_kernels.cuh"

namespace PCG_TU {

enum { AUX_ESTDT = 0, AUX_ESTDT_FINAL, AUX_UPDATE, AUX_FILL, AUX_FILL_BOXES, AUX_ESTDT_BOXES, AUX_COPY };

__device__ __forceinline__ bool aux_item(const pcg::AuxArgs& a, const pcg::AuxBox*& bx, int& i, int& j, int& k) {
  const pcg::Seg s = find_seg(a.few, a.segs, a.nseg, a.overlap);
  const unsigned local = unsigned(int(blockIdx.x) - (int)s.blk0) * blockDim.x + threadIdx.x;
  if (local >= (unsigned)s.count) return false;
  const unsigned n0 = s.n[0], n1 = s.n[1];
  const unsigned t = local / n0;
  i = s.lo[0] + (int)(local - t * n0);
  j = s.lo[1] + (int)(t % n1);
  k = s.lo[2] + (int)(t / n1);
  bx = a.boxes + s.region;
  return true;
}

// Block minimum with warp shuffles (blockDim.x == 128).
__device__ __forceinline__ double block_min(double v) {
  __shared__ double sh[4];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = dmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = (threadIdx.x < 4) ? sh[threadIdx.x] : DBL_MAX;
#pragma unroll
    for (int o = 2; o > 0; o >>= 1) v = dmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  return v;
}

// Source/Timestep.H:51-88 (pc_estdt_hydro) for one cell of state s:
// min over d of dx_d / (c + |u_d|), c from the stored temperature.
__device__ __forceinline__ double cfl_of(const double* s, const double* dx, double rhoInv, double c) {
  double dt = DBL_MAX;
  const double ux = s[pcg::UMX] * rhoInv;
  dt = dmin(dt, dx[0] / (c + fabs(ux)));
  const double uy = s[pcg::UMY] * rhoInv;
  dt = dmin(dt, dx[1] / (c + fabs(uy)));
  const double uz = s[pcg::UMZ] * rhoInv;
  dt = dmin(dt, dx[2] / (c + fabs(uz)));
  return dt;
}
template <int NS, bool MIX>
__device__ __forceinline__ double cfl_dt(const double* s, const double* dx) {
  using E = Eos<NS, MIX, double>;
  const double rho = s[pcg::URHO];
  const double rhoInv = 1.0 / rho;
  double y[NS];
#pragma unroll
  for (int n = 0; n < NS; ++n) y[n] = s[pcg::UFS + n] * rhoInv;
  return cfl_of(s, dx, rhoInv, E::rty2cs(rho, s[pcg::UTEMP], y));
}

// Per-cell CFL constraints of every valid cell, block minima.
template <int NS, bool MIX>
__global__ void __launch_bounds__(128) k_estdt(const __grid_constant__ pcg::AuxArgs a) {
  const pcg::AuxBox* bx;
  int i, j, k;
  double dt = DBL_MAX;
  if (aux_item(a, bx, i, j, k)) {
    const V4<const double> u = v4<const double>(bx->uin);
    double s[pcg::nvar(NS)];
#pragma unroll
    for (int n = 0; n < pcg::nvar(NS); ++n) s[n] = u(i, j, k, n);
    dt = cfl_dt<NS, MIX>(s, bx->dx);
  }
  dt = block_min(dt);
  if (threadIdx.x == 0) a.partial[blockIdx.x] = dt;
}

// Final reduction of the block minima, then estdt_hydro *= cfl (Source/PeleC.cpp:930), by one
// cluster of up to 8 blocks of 1024 threads (host: one block per 4096 minima), four loads in
// flight per thread; block 0 gathers the blocks' minima from their shared memory. The
// launch is a chain of load latencies, not bandwidth: one block of 128 threads took 21 us
// for the 16384 minima of a 128^3 level, as many loads in turn as this takes passes.
constexpr int kFinalThreads = 1024, kFinalLoads = 4, kFinalBlocks = 8;
__global__ void __launch_bounds__(kFinalThreads) k_estdt_final(const __grid_constant__ pcg::AuxArgs a) {
  namespace cg = cooperative_groups;
  __shared__ double sh[kFinalThreads / 32], part;
  const cg::cluster_group cl = cg::this_cluster();
  const int64_t stride = int64_t(gridDim.x) * kFinalThreads;
  await_previous(a.overlap);
  double v = DBL_MAX;
  for (int64_t b = int64_t(blockIdx.x) * kFinalThreads + threadIdx.x; b < a.npartial; b += kFinalLoads * stride) {
    double w[kFinalLoads];
#pragma unroll
    for (int m = 0; m < kFinalLoads; ++m) w[m] = b + m * stride < a.npartial ? a.partial[b + m * stride] : DBL_MAX;
#pragma unroll
    for (int m = 0; m < kFinalLoads; ++m) v = dmin(v, w[m]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = dmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (threadIdx.x % 32 == 0) sh[threadIdx.x / 32] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = sh[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = dmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (threadIdx.x == 0) part = v;
  }
  cl.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (unsigned r = 1; r < cl.num_blocks(); ++r) v = dmin(v, *cl.map_shared_rank(&part, r));
    *a.dt_out = v * a.cfl;
  }
  cl.sync();  // the minima stay readable until block 0 is done
}

// The energy step of pc_rst_int_e (default branch, PeleCUtilities.H:227-235) on a state s that
// already holds S_old + dt * hydro source: the internal energy into s, the mass fractions into
// y; returns the specific internal energy.
template <int NS>
__device__ __forceinline__ double energy_cell(double* s, double* y) {
  const double rho = s[pcg::URHO];
  const double rhoInv = 1.0 / rho;
  const double Up = s[pcg::UMX] * rhoInv;
  const double Vp = s[pcg::UMY] * rhoInv;
  const double Wp = s[pcg::UMZ] * rhoInv;
  const double ke = 0.5 * (Up * Up + Vp * Vp + Wp * Wp) - 0.5 * 0.0 * 0.0 * 0.0 * 0.0;
  s[pcg::UEINT] = s[pcg::UEDEN] - rho * ke;
  const double rhoInv2 = 1.0 / s[pcg::URHO];
  const double e = s[pcg::UEINT] * rhoInv2;
#pragma unroll
  for (int n = 0; n < NS; ++n) y[n] = s[pcg::UFS + n] * rhoInv2;
  return e;
}
// pc_rst_int_e and computeTemp (pc_cmpTemp, PeleCUtilities.H:70-84) on such a state.
template <int NS, bool MIX>
__device__ __forceinline__ void finish_cell(double* s) {
  using E = Eos<NS, MIX, double>;
  double y[NS];
  const double e = energy_cell<NS>(s, y);
  s[pcg::UTEMP] = E::rey2t(e, y, s[pcg::UTEMP]);
}
// finish_cell and the CFL constraint of the result. With one range switch temperature the
// reduced forms solve for T on the mixture polynomial and take the sound speed from it: the
// values of finish_cell and cfl_dt but for FP64 rounding. The reference-order form and tables with
// several switch temperatures call the two.
template <int NS, bool MIX>
__device__ __forceinline__ double finish_cfl(double* s, const double* dx) {
  if (MIX && !kExact && EosC<double, MIX>::uniform_tmid()) {
    double y[NS];
    const double e = energy_cell<NS>(s, y);
    const double rm = Eos<NS, MIX, double>::rmix(y);
    MixPoly<NS> mp;
    const double T = mp.temperature(e, y, s[pcg::UTEMP]);
    s[pcg::UTEMP] = T;
    const double rho = s[pcg::URHO], cv = mp.cv(T), p = rho * rm * T, g = (cv + rm) / cv;
    return cfl_of(s, dx, 1.0 / rho, sqrt(g * p / rho));
  }
  finish_cell<NS, MIX>(s);
  return cfl_dt<NS, MIX>(s, dx);
}

// Source/Advance.cpp:397-417 (construct_Snew, hydro only) then Source/PeleC.cpp:2289-2305
// (computeTemp) on one cell: s holds S_old on entry and S_new on exit.
template <int NS, bool MIX>
__device__ __forceinline__ void update_cell(double* s, const double* hsrc, double dt) {
#pragma unroll
  for (int n = 0; n < pcg::nvar(NS); ++n) s[n] += dt * hsrc[n];
  finish_cell<NS, MIX>(s);
}

template <int NS, bool MIX>
__global__ void __launch_bounds__(128) k_update(const __grid_constant__ pcg::AuxArgs a) {
  const pcg::AuxBox* bx;
  int i, j, k;
  if (!aux_item(a, bx, i, j, k)) return;
  const double dt = a.dt_in ? *a.dt_in : bx->dt;
  const V4<const double> so = v4<const double>(bx->uin);
  const V4<const double> hs = v4<const double>(bx->uout);
  const V4<double> sn = v4<double>(bx->snew);
  double s[pcg::nvar(NS)], h[pcg::nvar(NS)];
#pragma unroll
  for (int n = 0; n < pcg::nvar(NS); ++n) {
    s[n] = so(i, j, k, n);
    h[n] = hs(i, j, k, n);
  }
  update_cell<NS, MIX>(s, h, dt);
#pragma unroll
  for (int n = 0; n < pcg::nvar(NS); ++n) sn(i, j, k, n) = s[n];
}

// The tail of a level step in one pass over the cells of each region: the flux
// divergence of pc_consup (kept in registers, the hydro source array is not
// written), S_new = S_old + dt * hydro_source with computeTemp written over the state in
// place, and the CFL constraint of S_new for the next step (block minima; the final
// minimum is k_estdt_final). In place: a thread reads and writes the state of its own cell
// only. The step is the unfused one's (k_consup, k_update, k_estdt): bit for bit in the
// reference-order form; in the reduced forms temperature and timestep differ by FP64 rounding
// (finish_cfl).
template <int NS, bool MIX, int MINB>
__global__ void __launch_bounds__(128, MINB) k_advance(const __grid_constant__ pcg::StageArgs a) {
  Item it;
  double dtc = DBL_MAX;
  if (item_of(a, it)) {
    const pcg::Region& rg = *it.rg;
    double s[pcg::nvar(NS)];
    const CellPtr<double> u = at(v4<double>(rg.uin), it.i, it.j, it.k);
    const double dt = dt_of(a, rg);
    // S_old + dt * hydro source, each component as its source is formed (the source
    // itself is never held whole). UEINT is left out: finish_cfl forms it from the total
    // energy. The p div u term it would carry adds the region's pressure offset (p0_of), a read of
    // another cell of the state this launch is replacing.
    const auto add = [&](int n, double hn) { s[n] = u[n] + dt * hn; };
    if (rg.ff_single)
      consup_each<NS, float, true, false>(rg, it.i, it.j, it.k, 0.0, add);
    else
      consup_each<NS, double, false, false>(rg, it.i, it.j, it.k, 0.0, add);
    dtc = finish_cfl<NS, MIX>(s, rg.dx);
#pragma unroll
    for (int n = 0; n < pcg::nvar(NS); ++n) u[n] = s[n];
  }
  dtc = block_min(dtc);
  if (threadIdx.x == 0) a.partial[blockIdx.x] = dtc;
}

// Single-level FillBoundary of a domain FAB that covers grow(domain, ng), every ghost
// cell in one pass. Filling the directions x, y, z in turn, each over the full extent of
// the others (periodic wrap or foextrap, the zero-gradient copy of the nearest valid
// layer), leaves in ghost cell (i, j, k) the valid cell (m_x(i), m_y(j), m_z(k)), with m_d
// the wrap or clamp of direction d and the identity on valid indices; each thread copies
// that cell directly. Threads cover the z ghost slabs (full x, y extent), then the y ghost
// slabs of the valid k, then the x ghost slabs of the valid (j, k), i fastest.
__device__ __forceinline__ int ghost_src(int c, int lo, int hi, bool periodic) {
  const int n = hi - lo + 1;
  if (c < lo) return periodic ? c + n : lo;
  if (c > hi) return periodic ? c - n : hi;
  return c;
}
// Ghost cell number t of the domain [dlo, dhi] grown by ng (t < the ghost-cell count) gets
// its value from the valid cell the fill maps it to; a t past the last ghost cell does nothing.
// Eight components are loaded before any is stored (no ghost cell is a source): copied one by
// one, each component waits out the load before it, 16 of them 30 us on a 128^3 level.
// A view spans fewer than 2^31 elements, so the cell numbers are 32-bit.
__device__ __forceinline__ void fill_ghost(unsigned t, const int* dlo, const int* dhi, int ng, int periodic,
                                           const pcg::View& state, int ncomp) {
  const unsigned n0 = dhi[0] - dlo[0] + 1, n1 = dhi[1] - dlo[1] + 1, n2 = dhi[2] - dlo[2] + 1;
  const unsigned g2 = 2 * ng, e0 = n0 + g2, e1 = n1 + g2;
  const unsigned cz = e0 * e1 * g2, cy = e0 * g2 * n2, cx = g2 * n1 * n2;
  int c[3];
  if (t < cz) {  // z ghost slabs: (i, j) over the grown extent, 2 ng layers
    const unsigned r = t / e0;
    const int g = (int)(r / e1);
    c[0] = (int)(t - r * e0) + dlo[0] - ng;
    c[1] = (int)(r % e1) + dlo[1] - ng;
    c[2] = (g < ng) ? dlo[2] - ng + g : dhi[2] + 1 + (g - ng);
  } else if (t < cz + cy) {  // y ghost slabs of the valid k
    const unsigned u = t - cz, r = u / e0;
    const int g = (int)(r % g2);
    c[0] = (int)(u - r * e0) + dlo[0] - ng;
    c[1] = (g < ng) ? dlo[1] - ng + g : dhi[1] + 1 + (g - ng);
    c[2] = (int)(r / g2) + dlo[2];
  } else if (t < cz + cy + cx) {  // x ghost slabs of the valid (j, k)
    const unsigned u = t - cz - cy, r = u / g2;
    const int g = (int)(u - r * g2);
    c[0] = (g < ng) ? dlo[0] - ng + g : dhi[0] + 1 + (g - ng);
    c[1] = (int)(r % n1) + dlo[1];
    c[2] = (int)(r / n1) + dlo[2];
  } else {
    return;
  }
  int src[3];
  for (int d = 0; d < 3; ++d) src[d] = ghost_src(c[d], dlo[d], dhi[d], (periodic >> d) & 1);
  const V4<double> s = v4<double>(state);
  const double* from = &s(src[0], src[1], src[2], 0);
  double* to = &s(c[0], c[1], c[2], 0);
  constexpr int B = 8;
  for (int comp = 0; comp < ncomp; comp += B) {
    double v[B];
#pragma unroll
    for (int m = 0; m < B; ++m)
      if (comp + m < ncomp) v[m] = from[(comp + m) * s.ns];
#pragma unroll
    for (int m = 0; m < B; ++m)
      if (comp + m < ncomp) to[(comp + m) * s.ns] = v[m];
  }
}

// The ghost cells of many independent boxes (each its own domain) in one launch: the
// block finds its box by binary search over the boxes' first blocks.
__global__ void __launch_bounds__(128) k_fill_boxes(const __grid_constant__ pcg::AuxArgs a) {
  await_previous(a.overlap);
  const int64_t blk = blockIdx.x;
  int lo = 0, hi = a.nfill - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (a.fills[mid].blk0 <= blk) lo = mid; else hi = mid - 1;
  }
  const pcg::FillBox& f = a.fills[lo];
  const unsigned t = unsigned(blk - f.blk0) * blockDim.x + threadIdx.x;
  if (t >= (unsigned)f.count) return;
  fill_ghost(t, f.dlo, f.dhi, a.ng, f.periodic, f.state, a.ncomp);
}

// The next timestep of every box of a batched step: block b reduces the CFL minima the
// fused tail left for region b (the blocks of its advance segment), times cfl, into
// dt_boxes[b].
__global__ void __launch_bounds__(128) k_estdt_boxes(const __grid_constant__ pcg::AuxArgs a) {
  await_previous(a.overlap);
  const pcg::Seg& sg = a.bsegs[blockIdx.x];
  const int64_t nb = (sg.count + 127) / 128;
  double v = DBL_MAX;
  for (int64_t b = threadIdx.x; b < nb; b += blockDim.x) v = dmin(v, a.partial[sg.blk0 + b]);
  v = block_min(v);
  if (threadIdx.x == 0) a.dt_boxes[blockIdx.x] = v * a.cfl;
}

// Copy of the cells [dlo, dhi] of every component from one device FAB (state) to another
// (dst), FP64: the packing and unpacking of halo planes. One thread per cell and component.
__global__ void __launch_bounds__(128) k_copy_box(const __grid_constant__ pcg::AuxArgs a) {
  await_previous(a.overlap);
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n0 = a.dhi[0] - a.dlo[0] + 1, n1 = a.dhi[1] - a.dlo[1] + 1, n2 = a.dhi[2] - a.dlo[2] + 1;
  const int64_t cells = n0 * n1 * n2;
  if (t >= cells * a.ncomp) return;
  const int comp = (int)(t / cells);
  const int64_t c = t - comp * cells;
  const int i = a.dlo[0] + (int)(c % n0), j = a.dlo[1] + (int)((c / n0) % n1), k = a.dlo[2] + (int)(c / (n0 * n1));
  v4<double>(a.dst)(i, j, k, comp) = v4<const double>(a.state)(i, j, k, comp);
}

__global__ void __launch_bounds__(128) k_fill(const __grid_constant__ pcg::AuxArgs a) {
  await_previous(a.overlap);
  fill_ghost(blockIdx.x * blockDim.x + threadIdx.x, a.dlo, a.dhi, a.ng, a.periodic, a.state, a.ncomp);
}

static cudaError_t launch_estdt_final(const pcg::AuxArgs& a, cudaStream_t s) {
  const int64_t want = (a.npartial + kFinalThreads * kFinalLoads - 1) / (kFinalThreads * kFinalLoads);
  const unsigned nb = unsigned(want < 1 ? 1 : want > kFinalBlocks ? kFinalBlocks : want);
  return launch_kernel(k_estdt_final, nb, kFinalThreads, nb, a, s);
}

template <int NS, bool MIX>
static cudaError_t launch_advance_t(const pcg::StageArgs& a, int64_t nblocks, int variant, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)nblocks;
  switch (variant) {
    case 0: return launch_kernel(k_advance<NS, MIX, min_blocks<NS>(K_CONSUP, 0)>, grid, a, s);
    case 1: return launch_kernel(k_advance<NS, MIX, min_blocks<NS>(K_CONSUP, 1)>, grid, a, s);
    case 2: return launch_kernel(k_advance<NS, MIX, min_blocks<NS>(K_CONSUP, 2)>, grid, a, s);
    default: return cudaErrorInvalidValue;
  }
}

template <int NS, bool MIX>
static cudaError_t launch_aux_t(int which, const pcg::AuxArgs& a, int64_t nblocks, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)nblocks;
  switch (which) {
    case AUX_ESTDT: return launch_kernel(k_estdt<NS, MIX>, grid, a, s);
    case AUX_ESTDT_FINAL: return launch_estdt_final(a, s);
    case AUX_UPDATE: return launch_kernel(k_update<NS, MIX>, grid, a, s);
    case AUX_FILL: return launch_kernel(k_fill, grid, a, s);
    case AUX_FILL_BOXES: return launch_kernel(k_fill_boxes, grid, a, s);
    case AUX_ESTDT_BOXES: return launch_kernel(k_estdt_boxes, grid, a, s);
    case AUX_COPY: return launch_kernel(k_copy_box, grid, a, s);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace PCG_TU
