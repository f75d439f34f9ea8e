// The per-cell code of the step tail (csrc/pcg_aux_kernels.cuh) compiled for and run on the
// host, one thread at a time, where a stray read can be made to fail.
//
//   tail_host_test cells   the fused tail on FP32 and FP64 fluxes, every cell but those of the
//                          first row, whose state lies on pages that cannot be read: a tail
//                          that reads another cell's state, which its own thread may be
//                          replacing meanwhile, ends with SIGSEGV
//   tail_host_test energy FILE   FILE: an EOS table (mw, switch temperatures, low and high
//                          coefficients of 9 species), int32 n, n states [e, T guess, Y]; prints
//                          per state T of the fused tail and of the update, then the CFL bound of
//                          the fused tail and of estdt
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <type_traits>
#include <vector>

#include "pcg_types.h"

// What the device code takes from the compiler on a GPU: built-in variables, intrinsics, one
// thread's view of the warp and block primitives. Inline PTX vanishes.
static uint3 host_block, host_thread;
static dim3 host_block_dim(128), host_grid_dim(1);
#define blockIdx host_block
#define threadIdx host_thread
#define blockDim host_block_dim
#define gridDim host_grid_dim
static int __double2hiint(double x) { int64_t b; std::memcpy(&b, &x, 8); return int(b >> 32); }
static int __double2loint(double x) { int64_t b; std::memcpy(&b, &x, 8); return int(b); }
static double __hiloint2double(int h, int l) {
  const int64_t b = (int64_t(h) << 32) | uint32_t(l);
  double x;
  std::memcpy(&x, &b, 8);
  return x;
}
static float2 __fadd2_rn(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
static float2 __fmul2_rn(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
static float2 __ffma2_rn(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }
static float __fdividef(float a, float b) { return a / b; }
static double __shfl_xor_sync(unsigned, double v, int) { return v; }
static void __syncthreads() {}
static void __syncwarp() {}
static int __syncthreads_or(int v) { return v; }
static int atomicOr(int* p, int v) { const int o = *p; *p |= v; return o; }
static size_t __cvta_generic_to_shared(const void* p) { return reinterpret_cast<size_t>(p); }
namespace cooperative_groups {
struct cluster_group {
  void sync() const {}
  unsigned num_blocks() const { return 1; }
  template <class T> T* map_shared_rank(T* p, unsigned) const { return p; }
};
static cluster_group this_cluster() { return {}; }
}  // namespace cooperative_groups
using std::max;
using std::min;
#undef __launch_bounds__
#undef __grid_constant__
#define __launch_bounds__(...)
#define __grid_constant__
#define asm
#define volatile(...)

#define PCG_TU host_tail
namespace PCG_TU {
template <class A> static cudaError_t launch_kernel(void (*)(A), unsigned, unsigned, unsigned, const A&, cudaStream_t) { return cudaSuccess; }
template <class A> static cudaError_t launch_kernel(void (*)(A), unsigned, const A&, cudaStream_t) { return cudaSuccess; }
}  // namespace PCG_TU
#include "pcg_aux_kernels.cuh"
#undef asm
#undef volatile

using namespace host_tail;

namespace {

constexpr int NS = 9, NV = pcg::nvar(NS);

void constant_cv_table(pcg::EosConst& c) {
  c.kind = 1;
  c.nspec = NS;
  c.uniform_tmid = 1;
  for (int k = 0; k < NS; ++k) {
    c.imw[k] = 1.0 / (2.0 + 3.0 * k);
    c.tmid[k] = 1000.0;
    for (int r = 0; r < 2; ++r) c.cvc[k][r][0] = c.ec[k][r][1] = 2.5 * pcg::RU * c.imw[k];
  }
}

template <class F>
int run_cells() {
  constexpr int nx = 4, ny = 3, nz = 2, page = 512;  // a row of the state per page
  const size_t rows = size_t(NV) * ny * nz;
  auto* u = static_cast<double*>(mmap(nullptr, rows * page * 8, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
  if (u == MAP_FAILED) return 1;
  for (int n = 0; n < NV; ++n)
    for (int t = 0; t < nx * ny * nz; ++t) {
      const double rho = 1e-3, T = 300.0 + t;
      double cv = 0.0;
      for (int k = 0; k < NS; ++k) cv += c_eos[1].cvc[k][0][0] / NS;
      const double e = rho * cv * T;
      u[(size_t(n) * ny * nz + t / nx) * page + t % nx] =
        n == pcg::URHO ? rho : n <= pcg::UMZ ? 0.0 : n == pcg::UEDEN || n == pcg::UEINT ? e : n == pcg::UTEMP ? T : rho / NS;
    }
  constexpr int fx = nx + 1, fy = ny + 1, fz = nz + 1, cells = (fx * fy * fz + 31) / 32 * 32;
  constexpr bool single = sizeof(F) == 4;
  std::vector<F> ff(size_t(cells) * NV, F(0)), qe(size_t(cells) * 2, F(1));
  std::vector<double> out(size_t(cells) * NV, 0.0), partial(1);
  const auto view = [&](void* p, int nc) {
    pcg::View v{};
    v.p = p;
    v.js = fx;
    v.ks = fx * fy;
    v.ns = single ? 32 * nc : cells;
    return v;
  };
  pcg::Region rg{};
  const int hi[3] = {nx - 1, ny - 1, nz - 1};
  for (int d = 0; d < 3; ++d) {
    rg.hi[d] = hi[d];
    rg.dx[d] = rg.area_u[d] = 1.0;
    rg.ff[d] = view(ff.data(), NV);
    rg.qec[d] = view(qe.data(), 2);
  }
  rg.vol_u = 1.0;
  rg.dt = 1e-9;
  rg.zero_uout = 1;
  rg.ff_single = single;
  rg.uin.p = u;
  rg.uin.js = page;
  rg.uin.ks = page * ny;
  rg.uin.ns = page * ny * nz;
  rg.uout.p = out.data();
  rg.uout.js = nx;
  rg.uout.ks = nx * ny;
  rg.uout.ns = nx * ny * nz;
  pcg::StageArgs a{};
  a.regions = &rg;
  a.nseg = 1;
  pcg::Seg& s = a.few[0];
  s.n[0] = nx;
  s.n[1] = ny;
  s.n[2] = nz;
  s.count = nx * ny * nz;
  a.partial = partial.data();
  for (int n = 0; n < NV; ++n)
    if (mprotect(u + size_t(n) * ny * nz * page, page * 8, PROT_NONE)) return 1;
  for (int t = nx; t < nx * ny * nz; ++t) {
    host_thread.x = t;
    k_advance<NS, true, 1>(a);
    const double T = u[(size_t(pcg::UTEMP) * ny * nz + t / nx) * page + t % nx];
    if (!(std::fabs(T - (300.0 + t)) < 1e-6)) return 2;
  }
  munmap(u, rows * page * 8);
  return 0;
}

int run_energy(const char* path) {
  FILE* f = std::fopen(path, "rb");
  if (!f) return 1;
  pcg::EosConst& c = c_eos[1];
  c = pcg::EosConst{};
  c.kind = 1;
  c.nspec = NS;
  double mw[NS], tmid[NS], al[2][NS][7];
  size_t got = std::fread(mw, 8, NS, f) + std::fread(tmid, 8, NS, f) + std::fread(al, 8, 2 * NS * 7, f);
  int32_t n = 0;
  got += std::fread(&n, 4, 1, f);
  if (got != size_t(2 * NS + 14 * NS + 1)) return 1;
  c.uniform_tmid = 1;
  for (int k = 0; k < NS; ++k) {
    const double rw = pcg::RU / mw[k];
    c.imw[k] = 1.0 / mw[k];
    c.tmid[k] = tmid[k];
    if (tmid[k] != tmid[0]) c.uniform_tmid = 0;
    for (int r = 0; r < 2; ++r) {
      const double* a = al[r][k];
      for (int i = 0; i < 5; ++i) c.cvc[k][r][i] = rw * (a[i] - (i == 0));
      c.ec[k][r][0] = rw * a[5];
      for (int i = 0; i < 5; ++i) c.ec[k][r][i + 1] = rw * ((a[i] - (i == 0)) / (i + 1));
    }
  }
  const double dx[3] = {1.0, 1.5, 2.0};
  for (int m = 0; m < n; ++m) {
    double in[2 + NS], s[2][NV];
    if (std::fread(in, 8, 2 + NS, f) != size_t(2 + NS)) return 1;
    const double rho = 1.3e-3, v[3] = {2e3, -1e3, 5e2};
    for (auto& q : s) {
      q[pcg::URHO] = rho;
      double ke = 0.0;
      for (int d = 0; d < 3; ++d) q[pcg::UMX + d] = rho * v[d], ke += 0.5 * v[d] * v[d];
      q[pcg::UEDEN] = rho * (in[0] + ke);
      q[pcg::UEINT] = 0.0;
      q[pcg::UTEMP] = in[1];
      for (int k = 0; k < NS; ++k) q[pcg::UFS + k] = rho * in[2 + k];
    }
    const double fused = finish_cfl<NS, true>(s[0], dx);
    finish_cell<NS, true>(s[1]);
    std::printf("%.17g %.17g %.17g %.17g\n", s[0][pcg::UTEMP], s[1][pcg::UTEMP], fused, cfl_dt<NS, true>(s[1], dx));
  }
  std::fclose(f);
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "cells")) {
    constant_cv_table(c_eos[1]);
    const int a = run_cells<float>();
    return a ? a : run_cells<double>();
  }
  if (argc == 3 && !std::strcmp(argv[1], "energy")) return run_energy(argv[2]);
  return 64;
}
