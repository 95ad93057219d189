// engine.cuh - the Lagrangian-remap timestep on the device.
//
// Each routine below corresponds to a routine of the reference (file:line
// cited) and launches one kernel per reference loop nest over exactly the
// same index box, with the same left-to-right expression order.  Compiled
// with --fmad=false for FP64 (engine_f64.cu) the arithmetic is then
// bit-for-bit that of a gfortran -O3 x86-64 build of the reference, which
// emits no FMA.  Conduction is the exception: it forms T^2.5 and T^1.5 as
// T*T*sqrt(T) and T*sqrt(T) where the reference calls pow(), so its results
// differ in the last bits.  engine_f32.cu instantiates the same code in FP32
// (the FP32 form).
//
// All routines are free functions over Run<R>&; kernels capture only local
// copies of array handles and scalars (a capture of `run` itself fails to
// compile under -Werror cross-execution-space-call because Run owns a
// std::string).
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <map>
#include <string>
#include <utility>
#include <vector>

#include "../../include/lare_gpu.h"
#include "common.cuh"
#include "tma.cuh"

LARE_BEGIN

struct Par {
  double gamma, visc1, visc2, eta_background, eta0, j_max, kappa_0, flux_limiter;
  double ionise_pot, xi_n, va_max, dt_multiplier, dt_from_restart, kappa_perp_ratio;
  int resistive_mhd, conduction, heat_flux_limiter, use_viscous_damping, boris, restart;
  int eos_number, cowling_resistivity;                 // neutral.f90 (eos_number 0 read as EOS_IDEAL)
  double f_bar, t_bar, r_bar, tr, eta_bar;
  int radiation;                                       // radiative.f90
  int rke;                                             // the remap's kinetic-energy correction
  int cooling_term;                                    // lagran.F90:464, :1290
  double alpha_av;
  int coronal_heating;                                 // lagran.F90:127
  double temp_norm, time_norm, rho_norm, mf;
  int bc[3][2];   // [dim][0=min,1=max]
  bool per[3];    // periodic communicator in this dimension (mpi_routines.F90:195-210)
};

template <class R>
struct Arrays {
  // persistent
  A3<R> rho, energy, temperature, eta, cv, cv1, p_visc, visc_dep, ohmic_dep, gamma_boris;
  A3<R> vx, vy, vz, vx1, vy1, vz1, visc3, bx, by, bz;
  // lagran.F90 temporaries
  A3<R> bx0, by0, bz0, bx1, by1, bz1, alpha1, alpha2, alpha3, visc_heat, pressure, rho_v, cv_v;
  A3<R> flux_x, flux_y, flux_z, curlb, fx_visc, fy_visc, fz_visc, qx, qy, qz, energy0, cs, cs_v;
  // [xyz]remap.f90 temporaries (rho_alt, flux: second buffers of density and energy)
  A3<R> dm, cv2, flux, rho_alt;
  // conduct.f90 temporaries
  A3<R> larsen, Y1, Y2, Y3, Lc_Y0;  // RKL2 (Y0 is read from energy itself)
  A3<R> kf[9];                        // stage-invariant face coefficients, 3 per face direction
  // neutral.f90 (allocated only for a partially ionised run)
  A3<R> xi, eta_perp;
  // the energy after rad_losses (radiative.f90), allocated with radiation on
  A3<R> erad;
  // rke: the remap's kinetic-energy defect (shared_data.F90:108), the three
  // momentum fluxes before their product with dm, and what the split momentum
  // kernels read: the moved widths and the vertex averages
  A3<R> delta_ke, rke_f[3], rke_dk[3];
  A3<R> db1, dc1, r_rho_v, r_rho_v1, cv1v, cv2v, dmv;
  // cooling_term: moving averages of the viscous and ohmic heating
  // (shared_data.F90:109), persistent across steps
  A3<R> cool_term_v, cool_term_b;
  // coronal_heating: the user's heating rate (user_defined_heating's heat_in)
  A3<R> heat_in;
  // 1-D metrics (pointers at Fortran index 0)
  A1<R> dxb, dxc, dyb, dyc, dzb, dzc, grav;
  // reciprocals for conduction: 1/dxb, 1/dxc, 1/(dxc(i) + dxc(i-1)), per axis
  A1<R> rdb[3], rdc[3], rdc2[3];
};

enum Stag { ST_C = 0, ST_N = 1, ST_F = 2 };

// Per-launch-site timing (instrumentation, off by default).  A site is a
// launch statement (function, line); `words` is the number of distinct 3-D
// arrays it reads plus writes, so bytes = words * points * sizeof(R).
struct ProfSite {
  const char* func;
  int line;
  int words;
  long long count = 0;
  double ms = 0.0, bytes = 0.0;
};
struct Prof {
  bool on = false;
  std::vector<cudaEvent_t> ev;
  size_t used = 0;
  std::vector<int> ev_site;          // per event pair
  std::vector<double> ev_bytes;
  std::map<std::pair<std::string, int>, int> index;  // by name and line (the same name in several template instances is one site)
  std::vector<ProfSite> sites;
};

template <class R>
struct Run {
  Par p;
  int n[3];
  int sx, sxy, ntot;    // padded box
  size_t elems;         // elements per array
  Arrays<R> a;
  double* sc = nullptr;             // device scalar slots (Slot)
  unsigned long long* us = nullptr; // device min-reduction slots (USlot)
  double* partial = nullptr;        // block partial sums
  size_t partial_cap = 0;
  double* host_sc = nullptr;        // pinned mirror of sc
  cudaStream_t s = nullptr;
  long long launches = 0;
  std::vector<void*> allocations;
  bool visc2_norm_set = false;      // lagran.F90:539 first_call (SAVE)
  bool set_dt_first = true;         // lagran.F90:1078 first (SAVE)
  bool gamma_boris_one = true;      // gamma_boris holds 1 everywhere
  bool any_open = false;            // some side has BC_OPEN (boundary.f90:35-38)
  bool pip = false;                 // eos_number /= EOS_IDEAL: xi_n is the per-cell array a.xi
  bool cowling = false;             // cowling_resistivity: eta_perp in set_dt and rkstep
  int cur_step = 0;
  int peak_substeps = 0, last_substeps = 0, steps_taken = 0, n_s_stages = 0;
  int blk_x = 32, blk_y = 4;            // block shape of the point kernels (measured best at 256^3)
  bool capturing = false;               // recording a CUDA graph of whole steps
  PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;  // tma_encoder(), set by init
  bool launch_error = false;            // a tensor map could not be made: no kernel that copies by one is launched
  cudaStream_t s_body = nullptr;        // captures the body of the resistive sub-cycle loop
  GSpec g_cell, g_node, g_bx, g_by, g_bz, g_cell_mpi, g_cell_user, g_dm[3];
  Prof prof;
  std::string err;

  // Bracket one launch with events when profiling.
  int prof_begin(const char* func, int line, int words, double points) {
    if (!prof.on) return -1;
    auto key = std::make_pair(std::string(func), line);
    auto it = prof.index.find(key);
    int site;
    if (it == prof.index.end()) {
      site = (int)prof.sites.size();
      prof.index[key] = site;
      ProfSite ps;
      ps.func = func;
      ps.line = line;
      ps.words = words;
      prof.sites.push_back(ps);
    } else {
      site = it->second;
    }
    size_t k = prof.used;
    while (prof.ev.size() < 2 * (k + 1)) {
      cudaEvent_t e;
      cudaEventCreate(&e);
      prof.ev.push_back(e);
    }
    prof.ev_site.resize(k + 1);
    prof.ev_bytes.resize(k + 1);
    prof.ev_site[k] = site;
    prof.ev_bytes[k] = (double)words * points * (double)sizeof(R);
    cudaEventRecord(prof.ev[2 * k], s);
    return (int)k;
  }
  void prof_end(int k) {
    if (k < 0) return;
    cudaEventRecord(prof.ev[2 * k + 1], s);
    prof.used = k + 1;
  }
  // Fold recorded events into the per-site totals.
  void prof_collect() {
    cudaStreamSynchronize(s);
    for (size_t k = 0; k < prof.used; ++k) {
      float ms = 0.f;
      cudaEventElapsedTime(&ms, prof.ev[2 * k], prof.ev[2 * k + 1]);
      ProfSite& ps = prof.sites[prof.ev_site[k]];
      ps.ms += ms;
      ps.count += 1;
      ps.bytes += prof.ev_bytes[k];
    }
    prof.used = 0;
  }
};

// ---------------------------------------------------------------------
// Launch shorthands
template <int MINB64 = 0, int ZP32 = 1, class R, class Fn>
inline void rbox(Run<R>& run, const char* func, int line, int words, int i0, int i1, int j0, int j1, int k0, int k1,
                 Fn fn) {
  double pts = (double)(i1 - i0 + 1) * (double)(j1 - j0 + 1) * (double)(k1 - k0 + 1);
  int k = run.prof_begin(func, line, words, pts);
  launch_box<sizeof(R) == 8 ? MINB64 : 0, sizeof(R) == 4 ? ZP32 : 1>(run.s, run.launches, i0, i1, j0, j1, k0, k1, fn, run.blk_x, run.blk_y);
  run.prof_end(k);
}
// LARE_BOX: one kernel over an inclusive Fortran index box.  LARE_BOXW also
// states the kernel's algorithmic word count per point (arrays read +
// written), used for the roofline of profiled launches.  LARE_BOXWB adds an
// occupancy hint for the FP64 build (k_box_mb's MINB): latency-bound stencils
// with many live values run faster with a register cap that lets more
// blocks share an SM (measured per kernel at 256^3; FP32 keeps the default).
#define LARE_BOX(run, i0, i1, j0, j1, k0, k1, ...) \
  rbox((run), __func__, __LINE__, 0, (i0), (i1), (j0), (j1), (k0), (k1), __VA_ARGS__)
#define LARE_BOXW(run, words, i0, i1, j0, j1, k0, k1, ...) \
  rbox((run), __func__, __LINE__, (words), (i0), (i1), (j0), (j1), (k0), (k1), __VA_ARGS__)
#define LARE_BOXWB(run, minb, words, i0, i1, j0, j1, k0, k1, ...) \
  rbox<minb>((run), __func__, __LINE__, (words), (i0), (i1), (j0), (j1), (k0), (k1), __VA_ARGS__)
// LARE_BOXWH: both hints, the FP64 occupancy hint and the FP32 planes per
// thread (k_box_z's ZP), each measured per kernel at 256^3.
#define LARE_BOXWH(run, minb64, zp32, words, i0, i1, j0, j1, k0, k1, ...) \
  rbox<minb64, zp32>((run), __func__, __LINE__, (words), (i0), (i1), (j0), (j1), (k0), (k1), __VA_ARGS__)

// Some kernels write an array's new values into a second buffer that is
// then swapped in, covering only the points the reference updates (which it
// does in place, so every other point keeps its old value).  Periodic and
// BC_USER ghost fills rewrite every ghost right after; an open side is never
// refilled, so with an open side every point of the array's bounds [lo, hi]
// outside the updated box [a, b] is carried from the old buffer.
// The shell [lo, hi] minus [a, b] as six disjoint slabs (x below and above
// over the whole y, z range, then y below and above within a's x range,
// then z below and above within a's x and y ranges), walked by one flat
// index; up to three arrays share the walk.
template <class R>
struct CarryArgs {
  R* dst[3];
  const R* src[3];
  int narr, sx, sxy;
  int box[6][6];         // i0, i1, j0, j1, k0, k1 per slab
  long long start[7];    // first flat index of each slab; start[6] = total
};

template <class R>
__global__ void __launch_bounds__(256) k_carry(CarryArgs<R> g) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.start[6]) return;
  int s = 0;
  while (t >= g.start[s + 1]) ++s;  // at most five steps
  const int* q = g.box[s];
  const long long r = t - g.start[s];
  const long long e0 = q[1] - q[0] + 1, e1 = q[3] - q[2] + 1;
  const int i = q[0] + (int)(r % e0);
  const int j = q[2] + (int)((r / e0) % e1);
  const int k = q[4] + (int)(r / (e0 * e1));
  const int c = i + g.sx * j + g.sxy * k;
  for (int m = 0; m < g.narr; ++m) g.dst[m][c] = g.src[m][c];
}

template <class R>
inline void carry_outside_n(Run<R>& run, int narr, R* const* dst, const R* const* src, const int lo[3],
                            const int hi[3], const int a[3], const int b[3]) {
  if (!run.any_open) return;
  CarryArgs<R> g;
  g.narr = narr;
  g.sx = run.sx;
  g.sxy = run.sxy;
  for (int m = 0; m < 3; ++m) {
    g.dst[m] = m < narr ? dst[m] : nullptr;
    g.src[m] = m < narr ? src[m] : nullptr;
  }
  const int slab[6][6] = {
      {lo[0], a[0] - 1, lo[1], hi[1], lo[2], hi[2]}, {b[0] + 1, hi[0], lo[1], hi[1], lo[2], hi[2]},
      {a[0], b[0], lo[1], a[1] - 1, lo[2], hi[2]},   {a[0], b[0], b[1] + 1, hi[1], lo[2], hi[2]},
      {a[0], b[0], a[1], b[1], lo[2], a[2] - 1},     {a[0], b[0], a[1], b[1], b[2] + 1, hi[2]}};
  long long tot = 0;
  for (int s = 0; s < 6; ++s) {
    for (int d = 0; d < 6; ++d) g.box[s][d] = slab[s][d];
    g.start[s] = tot;
    const long long n0 = slab[s][1] - slab[s][0] + 1, n1 = slab[s][3] - slab[s][2] + 1,
                    n2 = slab[s][5] - slab[s][4] + 1;
    if (n0 > 0 && n1 > 0 && n2 > 0) tot += n0 * n1 * n2;
  }
  g.start[6] = tot;
  if (tot == 0) return;
  const int k = run.prof_begin("carry_outside", 0, 2 * narr, (double)tot);
  k_carry<R><<<(unsigned)((tot + 255) / 256), 256, 0, run.s>>>(g);
  run.prof_end(k);
  ++run.launches;
}

template <class R>
inline void carry_outside(Run<R>& run, R* dst, const R* src, const int lo[3], const int hi[3], const int a[3],
                          const int b[3]) {
  R* const d[1] = {dst};
  const R* const s[1] = {src};
  carry_outside_n(run, 1, d, s, lo, hi, a, b);
}

// the three velocity components after an update of the nodes 0:n
template <class R>
inline void carry_velocity(Run<R>& run, R* const nv[3], R* const ov[3]) {
  const int lo[3] = {-2, -2, -2}, hi[3] = {run.n[0] + 2, run.n[1] + 2, run.n[2] + 2};
  const int a[3] = {0, 0, 0}, b[3] = {run.n[0], run.n[1], run.n[2]};
  const R* const src[3] = {ov[0], ov[1], ov[2]};
  carry_outside_n(run, 3, nv, src, lo, hi, a, b);
}

template <class R>
inline void ghost(Run<R>& run, const GSpec& g, A3<R> a, A3<R>* b = nullptr, A3<R>* c = nullptr) {
  long long tot = g.c0 + g.c1 + g.c2;
  if (tot <= 0) return;
  int blocks = (int)((tot + 255) / 256);
  int narr = 1 + (b ? 1 : 0) + (c ? 1 : 0);
  int k = run.prof_begin("ghost", 0, 2 * narr, (double)tot);
  k_ghost<R><<<blocks, 256, 0, run.s>>>(g, a.p, b ? b->p : nullptr, c ? c->p : nullptr, run.sx, run.sxy);
  run.prof_end(k);
  ++run.launches;
}

// Deterministic sum of NV values over a box, into sc[slot..] (+=).
// site names the launch in the profile; words: the algorithmic words per
// point the kernel moves.  Planes per block: few enough blocks (4096) that
// the last one adds their partials in a few microseconds, which at 256^3 took
// 35 us for the 21,000 blocks of 4 planes.
template <int NV, class R, class Fn>
inline void box_sum(Run<R>& run, const char* site, int i0, int i1, int j0, int j1, int k0, int k1, Fn fn, int slot,
                    bool acc, int words = 0) {
  int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
  dim3 blk(64, 4, 1);
  dim3 grd((ni + 63) / 64, (nj + 3) / 4, 1);
  int planes = kSumPlanes;
  while (planes < 32 && (long long)grd.x * grd.y * ((nk + planes - 1) / planes) > 4096) planes *= 2;
  grd.z = (nk + planes - 1) / planes;
  int k = run.prof_begin(site, 0, words, (double)ni * nj * nk);
  k_box_sum<NV><<<grd, blk, 0, run.s>>>(i0, j0, k0, ni, nj, nk, planes, fn, run.partial, run.sc + slot, acc ? 1 : 0,
                                        (unsigned*)(run.us + U_DONE));
  run.prof_end(k);
  ++run.launches;
}

template <int NV, class R, class Fn>
inline void box_min(Run<R>& run, const char* site, int i0, int i1, int j0, int j1, int k0, int k1, Fn fn, int uslot,
                    int words = 0) {
  int ni = i1 - i0 + 1, nj = j1 - j0 + 1, nk = k1 - k0 + 1;
  // planes per block: fewer blocks contend for the atomic, and later blocks
  // find lower minima recorded (set_dt leaves out most cells by them), but a
  // thread takes its planes one after another, so a grid that has less than
  // five blocks an SM takes fewer.  set_dt in FP64 with 1, 2, 4 and 8 planes:
  // 12^3 8.6, 10, 13 and 17 us; 64^3 21, 18, 17 and 21; 96^3 42, 37, 39 and
  // 44; 128^3 87, 74, 70 and 69; 256^3 507, 417, 373 and 353.
  dim3 blk(64, 4, 1);
  dim3 grd((ni + 63) / 64, (nj + 3) / 4, 1);
  int planes = 8;
  while (planes > 1 && (long long)grd.x * grd.y * ((nk + planes - 1) / planes) < 5 * 148) planes /= 2;
  grd.z = (nk + planes - 1) / planes;
  int k = run.prof_begin(site, 0, words, (double)ni * nj * nk);
  k_box_min<NV><<<grd, blk, 0, run.s>>>(i0, j0, k0, ni, nj, nk, planes, fn, run.us + uslot);
  run.prof_end(k);
  ++run.launches;
}

// The map of array a (from its first element) with boxes of bx x by x bz, for a
// kernel that copies by it.  Where it cannot be made run.launch_error stays
// set, and the launcher returns without launching: a kernel given an unset map
// copies from whatever the map's bytes say.
template <class R>
inline void make_map(Run<R>& run, CUtensorMap* m, const R* first, int bx, int by, int bz) {
  if (!tma_map(run.encode, m, first, run.n, run.sx, run.sxy, bx, by, bz)) run.launch_error = true;
}

// ---------------------------------------------------------------------
// boundary.f90 fills, batched: every group of fills the reference performs
// back to back goes out as one launch (one job per array kind).
template <class R>
struct GhostBatch {
  GJobs<R> J;
  long long maxtot = 0;
  GhostBatch() { J.n = 0; }
  void add(const GSpec& g, R* p0, R* p1 = nullptr, R* p2 = nullptr) {
    J.s[J.n] = g;
    J.p[J.n][0] = p0;
    J.p[J.n][1] = p1;
    J.p[J.n][2] = p2;
    long long t = g.c0 + g.c1 + g.c2;
    if (t > maxtot) maxtot = t;
    ++J.n;
  }
};
template <class R>
inline void ghost_flush(Run<R>& run, GhostBatch<R>& b) {
  if (b.J.n == 0 || b.maxtot == 0) return;
  dim3 grd((unsigned)((b.maxtot + 255) / 256), (unsigned)b.J.n);
  int k = run.prof_begin("ghost", 0, 0, (double)b.maxtot * b.J.n);
  k_ghost_multi<R><<<grd, 256, 0, run.s>>>(b.J, run.sx, run.sxy);
  run.prof_end(k);
  ++run.launches;
}
template <class R> inline void energy_bcs(Run<R>& r) { GhostBatch<R> b; b.add(r.g_cell, r.a.energy.p); ghost_flush(r, b); }
template <class R> inline void density_bcs(Run<R>& r) { GhostBatch<R> b; b.add(r.g_cell, r.a.rho.p); ghost_flush(r, b); }
template <class R> inline void velocity_bcs(Run<R>& r) {
  GhostBatch<R> b;
  b.add(r.g_node, r.a.vx.p, r.a.vy.p, r.a.vz.p);
  ghost_flush(r, b);
}
template <class R> inline void remap_v_bcs(Run<R>& r) {
  GhostBatch<R> b;
  b.add(r.g_node, r.a.vx1.p, r.a.vy1.p, r.a.vz1.p);
  ghost_flush(r, b);
}
template <class R> inline void bfield_bcs(Run<R>& r) {
  GhostBatch<R> b;
  b.add(r.g_bx, r.a.bx.p);
  b.add(r.g_by, r.a.by.p);
  b.add(r.g_bz, r.a.bz.p);
  ghost_flush(r, b);
}
// boundary.f90:212 temperature_bcs exchanges rho (:214), then mirrors T.
template <class R> inline void temperature_bcs(Run<R>& r) {
  GhostBatch<R> b;
  b.add(r.g_cell_mpi, r.a.rho.p);
  b.add(r.g_cell_user, r.a.temperature.p);
  ghost_flush(r, b);
}
// boundary.f90:48-55 boundary_conditions
template <class R> inline void boundary_conditions(Run<R>& r) {
  GhostBatch<R> b;
  b.add(r.g_bx, r.a.bx.p);
  b.add(r.g_by, r.a.by.p);
  b.add(r.g_bz, r.a.bz.p);
  b.add(r.g_cell, r.a.energy.p, r.a.rho.p);
  b.add(r.g_node, r.a.vx.p, r.a.vy.p, r.a.vz.p);
  ghost_flush(r, b);
}
// energy_bcs + density_bcs at the end of lagrangian_step (lagran.F90:196-197),
// with the velocity_bcs after the corrector's new velocity (:409): nothing in
// between reads the velocity's ghosts unless a side is open.
template <class R> inline void end_of_step_bcs(Run<R>& r) {
  GhostBatch<R> b;
  b.add(r.g_cell, r.a.energy.p, r.a.rho.p);
  if (!r.any_open) b.add(r.g_node, r.a.vx.p, r.a.vy.p, r.a.vz.p);
  ghost_flush(r, b);
}
// bfield_bcs + energy_bcs at the end of a resistive sub-cycle
template <class R> inline void resistive_bcs(Run<R>& r) {
  GhostBatch<R> b;
  b.add(r.g_bx, r.a.bx.p);
  b.add(r.g_by, r.a.by.p);
  b.add(r.g_bz, r.a.bz.p);
  b.add(r.g_cell, r.a.energy.p);
  ghost_flush(r, b);
}

// Blocks of kernel K (threads a block, dynamic shared memory smem) that fit
// on the GPU at once.
template <auto K>
inline int resident_blocks(int threads, size_t smem = 0) {
  static const int n = [&] {
    int b = 0, dev = 0, sms = 148;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, K, threads, smem);
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (b > 0 ? b : 1) * sms;
  }();
  return n;
}
// Points of a marched axis of length len that one block of a marching kernel
// walks, for a launch of `tiles` blocks across it, `resident` of which fit on
// the GPU at once: the number of chunks that makes the fewest steps, a wave of
// blocks taking a chunk's points and about kMarchStart steps to fill its
// windows.  So a large grid gets long chunks (up to cap), a small one as many
// as run at once, down to 3 or 4 points, and no last wave is left nearly empty.
// With fixed chunks of 16 and 32 a 64^3 grid left most SMs idle (the march of
// eta_calc took 52 us on 96 x 80 x 121 with 8 % of the resident blocks).
constexpr int kMarchStart = 4;
inline int march_chunk(int len, int tiles, int cap, int resident) {
  const int n0 = (len + cap - 1) / cap, n1 = (len + 3) / 4;
  int best = n0;
  long long least = LLONG_MAX;
  for (int n = n0; n <= n1; ++n) {
    const long long waves = ((long long)tiles * n + resident - 1) / resident;
    const long long steps = waves * ((len + n - 1) / n + kMarchStart);
    if (steps < least) {
      least = steps;
      best = n;
    }
  }
  return (len + best - 1) / best;
}

// Full-array elementwise helpers (Fortran whole-array statements).
template <class R, class Fn>
inline void whole(Run<R>& r, Fn fn) {
  LARE_BOX(r, -2, r.n[0] + 2, -2, r.n[1] + 2, -2, r.n[2] + 2, fn);
}

// ---------------------------------------------------------------------
// lagran.F90:483-524 viscous_damping
template <class R>
void viscous_damping(Run<R>& run) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  auto vx = run.a.vx, vy = run.a.vy, vz = run.a.vz, visc3 = run.a.visc3;
  auto qx = run.a.qx, qy = run.a.qy, qz = run.a.qz;
  auto dxb = run.a.dxb, dyb = run.a.dyb, dzb = run.a.dzb, dxc = run.a.dxc, dyc = run.a.dyc, dzc = run.a.dzc;
  const double* sc = run.sc;
  LARE_BOXW(run, 7, 0, nx, 0, ny, 0, nz, [=] __device__(int ix, int iy, int iz) {
    int ixp = ix + 1, ixm = ix - 1, iyp = iy + 1, iym = iy - 1, izp = iz + 1, izm = iz - 1;
    A3<R> vv[3] = {vx, vy, vz};
    A3<R> qq[3] = {qx, qy, qz};
    for (int c = 0; c < 3; ++c) {
      A3<R> v = vv[c];
      qq[c](ix, iy, iz) = visc3(ix, iy, iz) *
          (((v(ixp, iy, iz) - v(ix, iy, iz)) / dxb(ixp) - (v(ix, iy, iz) - v(ixm, iy, iz)) / dxb(ix)) / dxc(ix) +
           ((v(ix, iyp, iz) - v(ix, iy, iz)) / dyb(iyp) - (v(ix, iy, iz) - v(ix, iym, iz)) / dyb(iy)) / dyc(iy) +
           ((v(ix, iy, izp) - v(ix, iy, iz)) / dzb(izp) - (v(ix, iy, iz) - v(ix, iy, izm)) / dzb(iz)) / dzc(iz));
    }
  });
  LARE_BOXW(run, 9, 0, nx, 0, ny, 0, nz, [=] __device__(int ix, int iy, int iz) {
    const R dt = (R)sc[SC_DT];
    vx(ix, iy, iz) = vx(ix, iy, iz) + dt * qx(ix, iy, iz);
    vy(ix, iy, iz) = vy(ix, iy, iz) + dt * qy(ix, iy, iz);
    vz(ix, iy, iz) = vz(ix, iy, iz) + dt * qz(ix, iy, iz);
  });
}

// ---------------------------------------------------------------------
// lagran.F90:795-855 edge_viscosity with the default DEFINES (psi = 0).
template <class R>
__device__ __forceinline__ R edge_viscosity(R dvdots, R r1, R r2, R c1, R c2, R dvx, R dvy, R dvz, R dx, R dt,
                                            R visc1, R visc2_norm) {
  dvdots = -fabs(dvdots);
  R rho_edge = qdiv(R(2) * r1 * r2, r1 + r2);
  R cs_edge = fmin(c1, c2);
  R dv2 = dvx * dvx + dvy * dvy + dvz * dvz;
  R dv = sqrt(dv2);
  R psi = R(0);
  if (qdiv(dv * dt, dx) < R(1.e-14)) dvdots = R(0);
  else dvdots = qdiv(dvdots, dv);
  R vc = visc1 * cs_edge;
  R q_k_bar = rho_edge * (visc2_norm * dv + sqrt(visc2_norm * visc2_norm * dv2 + vc * vc));
  return q_k_bar * (R(1) - psi) * dvdots;
}

// ---------------------------------------------------------------------
// x^2.5 and x^1.5 as x*x*sqrt(x) and x*sqrt(x): within an ulp or two of
// pow() and several times cheaper (the reference calls pow, so conduction is
// compared with the oracle at a 1e-12 relative tolerance, not bitwise).
template <class R>
__device__ __forceinline__ R pow25(R x) { return x * x * sqrt(x); }
template <class R>
__device__ __forceinline__ R pow15(R x) { return x * sqrt(x); }

// conduct.f90:56-143 calc_s_stages.  Produces larsen_factor and the stage
// count in sc[SC_STAGES] from the dt in sc[dt_slot].
template <class R>
void calc_s_stages(Run<R>& run, int dt_slot) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  auto temperature = run.a.temperature, energy = run.a.energy, rho = run.a.rho, larsen = run.a.larsen;
  auto dxb = run.a.dxb, dyb = run.a.dyb, dzb = run.a.dzb;
  const R g = (R)run.p.gamma, xi = (R)run.p.xi_n, ip = (R)run.p.ionise_pot, k0 = (R)run.p.kappa_0;
  const R fl = (R)run.p.flux_limiter;
  const bool limiter = run.p.heat_flux_limiter != 0;
  const bool pip = run.pip;
  auto xia = run.a.xi;  // per-cell xi_n when partially ionised
  unsigned long long* us = run.us;
  const R tc = (g - R(1)) / (R(2) - xi), te0 = (R(1) - xi) * ip;
  const A1<R> rdx = run.a.rdb[0], rdy = run.a.rdb[1], rdz = run.a.rdb[2];
  // one pass: the temperature over the whole cell box, the Larsen factor over
  // 0:n and the explicit limit over 1:n (three passes took 0.236 against
  // 0.199 ms at 256^3 in FP32)
  box_min<1>(run, "parabolic_dt_min", -1, nx + 2, -1, ny + 2, -1, nz + 2, [=] __device__(int ix, int iy, int iz, double* v, const double*) {
    // FP32 keeps the reference's grouping (kRegroup): a rounding here is the
    // same one at every cell of a uniform grid
    auto temp_at = [&](int i, int j, int k) {
      if (kRegroup<R> && !pip) return tc * (energy(i, j, k) - te0);
      const R x = pip ? xia(i, j, k) : xi;
      return (g - R(1)) / (R(2) - x) * (energy(i, j, k) - (R(1) - x) * ip);
    };
    const R T = temp_at(ix, iy, iz);
    temperature(ix, iy, iz) = T;
    if (ix < 0 || ix > nx || iy < 0 || iy > ny || iz < 0 || iz > nz) return;
    const R tp = pow25(T), r = rho(ix, iy, iz);
    R lf = R(1);
    if (limiter) {
      R q_fs = fl * R(42.85) * r * pow15(T);
      R q_fs2 = q_fs * q_fs;
      const R dTx = temp_at(ix + 1, iy, iz) - temp_at(ix - 1, iy, iz);
      const R dTy = temp_at(ix, iy + 1, iz) - temp_at(ix, iy - 1, iz);
      const R dTz = temp_at(ix, iy, iz + 1) - temp_at(ix, iy, iz - 1);
      if (kRegroup<R>) {
        const R kt = -k0 * tp * R(0.5);
        const R q_spx = kt * dTx * rdx(ix), q_spy = kt * dTy * rdy(iy), q_spz = kt * dTz * rdz(iz);
        lf = qdiv(q_fs, sqrt(q_fs2 + (q_spx * q_spx + q_spy * q_spy + q_spz * q_spz)));
      } else {
        R q_spx = -k0 * tp * dTx * R(0.5) / dxb(ix);
        R q_spy = -k0 * tp * dTy * R(0.5) / dyb(iy);
        R q_spz = -k0 * tp * dTz * R(0.5) / dzb(iz);
        R q_sp2 = q_spx * q_spx + q_spy * q_spy + q_spz * q_spz;
        lf = q_fs / sqrt(q_fs2 + q_sp2);
      }
    }
    larsen(ix, iy, iz) = lf;
    if (ix < 1 || iy < 1 || iz < 1) return;
    const R kappa1 = k0 * lf;
    // the least of rho d^2 / (2 kappa T^5/2) over the axes is that of the least d
    const R d = fmin(fmin(dxb(ix), dyb(iy)), dzb(iz));
    const R top = r * (d * d), bottom = R(2) * kappa1 * tp;
    v[0] = (double)(kRegroup<R> ? qdiv(top, bottom) : top / bottom);
  }, U_DTPARAB, 4);
  double* sc = run.sc;
  const double mult = run.p.dt_multiplier;
  const bool f32 = sizeof(R) == 4;
  launch_scalar(run.s, run.launches, [=] __device__() {
    double dtp_min = __longlong_as_double((long long)us[U_DTPARAB]);
    us[U_DTPARAB] = kMinReset;
    double dt = sc[dt_slot];
    double stages, dt_parab;
    if (f32) {
      // The FP32 form keeps this recurrence in FP64 but starts from the
      // FP32 minimum, as the field arithmetic produced it.
      dt_parab = mult * fmin(dtp_min, 1.e10) / sqrt(3.0);
    } else {
      dt_parab = mult * fmin(dtp_min, 1.e10) / sqrt(3.0);
    }
    stages = 0.5 * (sqrt(9.0 + 16.0 * (dt / dt_parab)) - 1.0);
    int ns = (int)ceil(stages);
    if (ns % 2 == 0) ns = ns + 1;
    sc[SC_STAGES] = (double)ns;
    sc[SC_DTPARAB] = dt_parab;
  });
}

// Temperature of an energy-like array, conduct.f90:68 and :371-374,
// evaluated where it is needed instead of stored.
template <class R>
struct TempOf {
  A3<R> y;
  R c, e0;  // (gamma - 1)/(2 - xi_n), (1 - xi_n)*ionise_pot
  __device__ __forceinline__ R operator()(int i, int j, int k) const { return c * (y(i, j, k) - e0); }
};

template <class R>
void temperature_from(Run<R>& run, A3<R> e) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  auto temperature = run.a.temperature;
  const R g = (R)run.p.gamma, xi = (R)run.p.xi_n, ip = (R)run.p.ionise_pot;
  const bool pip = run.pip;
  auto xia = run.a.xi;
  LARE_BOXW(run, 2, -1, nx + 2, -1, ny + 2, -1, nz + 2, [=] __device__(int ix, int iy, int iz) {
    const R x = pip ? xia(ix, iy, iz) : xi;
    temperature(ix, iy, iz) = (g - R(1)) / (R(2) - x) * (e(ix, iy, iz) - (R(1) - x) * ip);
  });
}

// Copy between whole arrays (Fortran whole-array assignment).
template <class R>
void copy_whole(Run<R>& run, A3<R> dst, A3<R> src) {
  int k = run.prof_begin("copy_whole", 0, 2, (double)run.elems);
  cudaMemcpyAsync(dst.p - (2 + 2 * run.sx + 2 * run.sxy), src.p - (2 + 2 * run.sx + 2 * run.sxy),
                  run.elems * sizeof(R), cudaMemcpyDeviceToDevice, run.s);
  run.prof_end(k);
}

LARE_END  // namespace lare

#include "neutral.cuh"
#include "radiative.cuh"
#include "conduct.cuh"

LARE_BEGIN

// conduct.f90:299-416 heat_conduct_sts2, dt from sc[dt_slot]; the stage
// count s must already be known on the host (run.n_s_stages).
//
// The reference keeps Y(0:3) and copies whole arrays between stages
// (Y1 = Y2; energy = Y3; energy_bcs; Y2 = energy).  Here the stages rotate
// three buffers instead, with Y0 read straight from `energy` (untouched
// until the end), and the temperature of Y2 is formed where the flux needs
// it.  The values are the same as the reference's, including its boundary
// detail: the temperature ghosts of stage 2 in MPI/periodic directions come
// from Y2's ghost cells, which still hold the energy's (temperature_bcs
// refreshes only BC_USER faces), so Y2 starts as a whole copy of energy and
// gets only the BC_USER fill before stage 2; from stage 3 on, Y2 is the
// previous Y3 after the full energy boundary fill.
template <class R>
void heat_conduct_sts2(Run<R>& run, int dt_slot) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  const int s = run.n_s_stages;
  std::vector<double> a(s + 1), b(s + 1), mu_tilde(s + 1), mu(s + 1), nu(s + 1), gamma_tilde(s + 1);
  double ds = (double)s;
  double omega_1 = 4.0 / (ds * ds + ds - 2.0);
  for (int j = 0; j <= (s < 2 ? s : 2); ++j) b[j] = 1.0 / 3.0;
  for (int j = 3; j <= s; ++j) {
    double dj = (double)j;
    b[j] = (dj * dj + dj - 2.0) / (2.0 * dj * (dj + 1.0));
  }
  for (int j = 0; j <= s; ++j) a[j] = 1.0 - b[j];
  mu_tilde[1] = omega_1 / 3.0;
  for (int j = 2; j <= s; ++j) {
    double dj = (double)j;
    mu_tilde[j] = ((2.0 * dj - 1.0) / dj) * omega_1 * (b[j] / b[j - 1]);
    mu[j] = ((2.0 * dj - 1.0) / dj) * (b[j] / b[j - 1]);
    nu[j] = -1.0 * ((dj - 1.0) / dj) * (b[j] / b[j - 2]);
    gamma_tilde[j] = -1.0 * a[j - 1] * mu_tilde[j];
  }
  Arrays<R>& A = run.a;
  auto energy = A.energy;
  const R g = (R)run.p.gamma, xi = (R)run.p.xi_n, ip = (R)run.p.ionise_pot;
  const R tc = (g - R(1)) / (R(2) - xi), te0 = (R(1) - xi) * ip;
  // With a per-cell xi_n (partially ionised) the temperature changes with
  // xi_n between stages, so each stage forms it into the temperature array
  // exactly as conduct.f90:346-376 does, and the stage reads it back
  // through 1 * (T - 0) = T.
  const bool pip = run.pip;
  auto temp = [&](A3<R> y) { return pip ? TempOf<R>{A.temperature, R(1), R(0)} : TempOf<R>{y, tc, te0}; };
  if (s < 2) {
    // The stage loop is empty and energy(1:n) = Y(3)(1:n) = energy: the
    // reference leaves the energy unchanged (conduct.f90:409).
    energy_bcs(run);
    return;
  }
  // rotating buffers: Y0 = energy (read only), Y1 = energy for stage 2
  A3<R> bufs[3] = {A.Y1, A.Y2, A.Y3};
  A3<R> Y1 = energy, Y2 = bufs[0], Y3 = bufs[1];
  int next_free = 2;
  copy_whole(run, Y2, energy);
  if (run.any_open) {
    // The reference's Y(3) keeps the energy's ghosts throughout (only
    // 1:n is written), and energy_bcs leaves an open side's ghosts alone:
    // every stage buffer starts as the energy so that those ghosts match.
    copy_whole(run, bufs[1], energy);
    copy_whole(run, bufs[2], energy);
  }
  face_coefficients(run);
  if (pip) temperature_from(run, energy);
  rkl2_stage<R, true>(run, __LINE__, temp(energy), energy, energy, energy, Y2, dt_slot, (R)mu_tilde[1], R(0), R(0),
                      R(0), R(0));
  ghost(run, run.g_cell_user, Y2);
  {
    GhostBatch<R> bb;
    bb.add(run.g_cell_mpi, A.rho.p);  // density_mpi of temperature_bcs (a no-op on a consistent rho)
    ghost_flush(run, bb);
  }
  for (int j = 2; j <= s; ++j) {
    const R gt = (R)gamma_tilde[j], mtj = (R)mu_tilde[j], mj = (R)mu[j], nj = (R)nu[j];
    const R omn_r = R(1) - mj - nj;
    if (pip) {
      temperature_from(run, Y2);
      temperature_bcs(run);
    }
    // The last stage writes the energy in place (conduct.f90:409): Y0 is read
    // at a cell only by the thread that writes it.
    if (j == s) Y3 = energy;
    rkl2_stage<R, false>(run, __LINE__, temp(Y2), Y2, Y1, energy, Y3, dt_slot, mtj, mj, nj, omn_r, gt);
    if (j < s) {
      GhostBatch<R> bb;
      bb.add(run.g_cell, Y3.p);  // energy_bcs on the copy of Y3
      ghost_flush(run, bb);
      if (pip) neutral_fraction(run, Y3);  // conduct.f90:404
      A3<R> freed = Y1;
      Y1 = Y2;
      Y2 = Y3;
      if (freed.p == energy.p) {
        Y3 = bufs[next_free];
      } else {
        Y3 = freed;
      }
    }
  }
  // The reference leaves temperature = T(Y2 of the last stage) after
  // temperature_bcs; keep that, then energy_bcs.
  {
    auto temperature = A.temperature;
    A3<R> y2 = Y2;
    if (!pip) {  // (a partially ionised run formed it for the last stage)
      LARE_BOXW(run, 2, -1, nx + 2, -1, ny + 2, -1, nz + 2, [=] __device__(int ix, int iy, int iz) {
        temperature(ix, iy, iz) = tc * (y2(ix, iy, iz) - te0);
      });
      GhostBatch<R> bb;
      bb.add(run.g_cell_user, temperature.p);
      ghost_flush(run, bb);
    }
  }
  energy_bcs(run);
}

// ---------------------------------------------------------------------
// Limited Van Leer flux shared by the *_flux routines of [xyz]remap.f90.
//
// Divisors arrive in carried form (dv_of): the value itself in the exact
// builds, its reciprocal in the product build, so a kernel that moves along
// a line forms each reciprocal once per point.  The exact builds evaluate
// the reference's expressions unchanged; the product build takes the upwind
// divisors by selection (vad_p is exactly 0 or 1, so the reference's
// weighted sums dxcm*vad_p + dxcp*vad_m equal one of the two) and multiplies.
template <class R>
struct LimOut {
  R sign_v, vad_p, vad_m, fu, Di, dxbu, phi;
};
template <class R>
__device__ __forceinline__ LimOut<R> limiter_dv(R v_advect, R fm, R fi, R fp, R fp2, R dvci, R dvcm, R dvcp,
                                                R dxbi, R dxbp, R dvu_p, R dvu_m, R dt, bool phi_from_dxu) {
  LimOut<R> L;
  R dfm = fi - fm, dfi = fp - fi, dfp = fp2 - fp;
  L.sign_v = copysign(R(1), v_advect);
  L.vad_p = (L.sign_v + R(1)) * R(0.5);
  L.vad_m = R(1) - L.vad_p;
  L.fu = fi * L.vad_p + fp * L.vad_m;
  R dfu = dfm * L.vad_p + dfp * L.vad_m;
  L.dxbu = dxbi * L.vad_p + dxbp * L.vad_m;
#if LARE_FAST
  const bool up = !signbit(v_advect);
  const R dvcu = up ? dvcm : dvcp;
  if (phi_from_dxu) {
    L.phi = fabs(v_advect) * dt * (up ? dvu_p : dvu_m);
  } else {
    L.phi = fabs(v_advect) * dt * fast_rcp(L.dxbu);
  }
#else
  R dvcu = dvcm * L.vad_p + dvcp * L.vad_m;
  if (phi_from_dxu) {
    R dxu = dvu_p * L.vad_p + dvu_m * L.vad_m;
    L.phi = fabs(v_advect) * dt / dxu;
  } else {
    L.phi = fabs(v_advect) * dt / L.dxbu;
  }
#endif
  R Da = dv_div((R(2) - L.phi) * fabs(dfi), dvci) + dv_div((R(1) + L.phi) * fabs(dfu), dvcu);
  Da = Da * (R(1) / R(6));
  R ss = R(0.5) * (copysign(R(1), dfi) + copysign(R(1), dfu));
  L.Di = L.sign_v * ss * fmin(fmin(fabs(Da) * L.dxbu, fabs(dfi)), fabs(dfu));
  return L;
}
// The product build's limited flux per unit mass or area moved, in terms of
// the faces' differences d and slopes s = |d| / dxc (faces below, at and
// above c): the reference's expressions regrouped, with the upwind choices
// (whose weights are exactly 0 or 1) and the product of signs taken by
// selection.  phi = |v dt| * rxu; the result is (f_u + D (1 - phi)) v dt.
// (kRegroup only, so in FP64.)
template <class R>
__device__ __forceinline__ R lesser(R a, R b) {
  return a < b ? a : b;
}
// copies +-m: zero unless a and b have the same sign, else m with the sign of a * s
__device__ __forceinline__ double signed_min(double m, double a, double b, double s) {
  const int ha = __double2hiint(a);
  const bool same = (ha ^ __double2hiint(b)) >= 0;
  const int h = __double2hiint(m) | ((ha ^ __double2hiint(s)) & 0x80000000);
  return same ? __hiloint2double(h, __double2loint(m)) : 0.0;
}
template <class R>
__device__ __forceinline__ R van_leer(R v, R vdt, R f0, R fp, R dm, R d0, R dp, R sm, R s0, R sp, R db0, R dbp, R r0,
                                      R rp) {
  const bool up = !signbit(v);
  const R phi = fabs(vdt) * (up ? r0 : rp);
  const R du = up ? dm : dp;
  const R da = (R(2) - phi) * s0 + (R(1) + phi) * (up ? sm : sp);
  const R m = lesser(lesser(fabs(da) * ((up ? db0 : dbp) * (R(1) / R(6))), R(fabs(d0))), R(fabs(du)));
  const R D = signed_min(m, d0, du, v);
  return ((up ? f0 : fp) + D * (R(1) - phi)) * vdt;
}
// The same with plain divisors.
template <class R>
__device__ __forceinline__ LimOut<R> limiter(R v_advect, R fm, R fi, R fp, R fp2, R dxci, R dxcm, R dxcp, R dxbi,
                                             R dxbp, R dxu_p, R dxu_m, R dt, bool phi_from_dxu) {
  return limiter_dv(v_advect, fm, fi, fp, fp2, dv_of(dxci), dv_of(dxcm), dv_of(dxcp), dxbi, dxbp,
                    phi_from_dxu ? dv_of(dxu_p) : dxu_p, phi_from_dxu ? dv_of(dxu_m) : dxu_m, dt, phi_from_dxu);
}

LARE_END  // namespace lare

#include "remap.cuh"

LARE_BEGIN

// The axes of a step's three sweeps in order (remap.f90:71-99).
inline const int* sweep_order(int step) {
  static const int order[6][3] = {{0, 1, 2}, {1, 2, 0}, {2, 0, 1}, {0, 2, 1}, {2, 1, 0}, {1, 0, 2}};
  return order[((step % 6) + 6) % 6];
}

// remap.f90:33-131 eulerian_remap (the corrector's full remap; the
// predictor's B-only remap is predictor_remap in lagran.cuh).
template <class R>
void eulerian_remap(Run<R>& run, int step) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  const int sx = run.sx, sxy = run.sxy;
  int pass[3] = {1, 1, 1};
  if (run.p.rke) {  // remap.f90:38
    R* const dke = run.a.delta_ke.p;
    LARE_BOXW(run, 1, 1, nx, 1, ny, 1, nz, [=] __device__(int ix, int iy, int iz) { dke[ix + sx * iy + sxy * iz] = R(0); });
  }
  // B -> flux form (remap.f90:43-69) and back (:101-127) are done by the
  // first and last sweeps' B kernels on the way (remap_sweep's bmode).
  const int* const order = sweep_order(step);
  for (int s = 0; s < 3; ++s) {
    const int bmode = s == 0 ? 1 : (s == 2 ? 2 : 0);
    switch (order[s]) {
      case 0: remap_sweep<0>(run, SC_DT, pass, bmode); break;
      case 1: remap_sweep<1>(run, SC_DT, pass, bmode); break;
      default: remap_sweep<2>(run, SC_DT, pass, bmode); break;
    }
  }
  // (the last sweep's boundary_conditions already filled the converted B:
  // bfield_bcs at remap.f90:128 would write the same values again)
}

// LARE_ECUDA, with its message, where the scalar slots on the host say that a
// kernel's tile copy was lost: what it computed is not to be used.
template <class R>
int lost_copy(Run<R>& run) {
  if (run.host_sc[SC_LOST] == 0.0) return LARE_OK;
  run.err = "a tile copy never arrived";
  return LARE_ECUDA;
}
// Pull the scalar slots to the host (one sync).
template <class R>
int pull_scalars(Run<R>& run) {
  cudaMemcpyAsync(run.host_sc, run.sc, SC_NSLOTS * sizeof(double), cudaMemcpyDeviceToHost, run.s);
  const cudaError_t e = cudaStreamSynchronize(run.s);
  if (e == cudaSuccess) return lost_copy(run);
  run.err = std::string("sync failed: ") + cudaGetErrorString(e);
  return LARE_ECUDA;
}

// ---------------------------------------------------------------------
// diagnostics.F90:517-609 energy_account into sc[SC_EN_B..SC_EN_INT], in one
// pass over the vertices 0:n, the cells among them.  A thread walks `planes`
// planes of its column and carries the lower quad of the vertex' eight cells
// (mass and volume): 17 loads a point instead of 30,
// 0.27 against 0.38 ms at 256^3 (FP64) for the two point kernels it replaces.
template <class R>
struct EnergyArgs {
  const R *bx, *by, *bz, *cv, *energy, *rho, *vx, *vy, *vz;
  double *partial, *out;
  unsigned* done;
  int nx, ny, nz, sx, sxy, planes;
};

template <class R>
__global__ void __launch_bounds__(256) k_energy_account(EnergyArgs<R> g) {
  const int ix = (int)(blockIdx.x * blockDim.x + threadIdx.x), iy = (int)(blockIdx.y * blockDim.y + threadIdx.y);
  const int z0 = (int)blockIdx.z * g.planes, z1 = min(z0 + g.planes - 1, g.nz);
  double v[3] = {0.0, 0.0, 0.0};
  if (ix <= g.nx && iy <= g.ny) {
    const int sx = g.sx;
    int c = ix + sx * iy + g.sxy * z0;
    // a plane's quad around the vertex: its sums, and the cell itself
    struct Quad {
      double r, w, r0, w0;
    };
    auto quad = [&](int q, double r, double w) {  // added to the sums r and w
      const int o[4] = {0, 1, sx, 1 + sx};
      Quad t{r, w, 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double cw = g.cv[q + o[k]], rw = (double)g.rho[q + o[k]] * cw;
        t.r += rw;
        t.w += cw;
        if (k == 0) {
          t.r0 = rw;
          t.w0 = cw;
        }
      }
      return t;
    };
    auto both = [&](int q, double r, double w, Quad& own) {  // a quad alone, and added to the sums below it
      const int o[4] = {0, 1, sx, 1 + sx};
      Quad t{r, w, 0.0, 0.0};
      own = Quad{0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const double cw = g.cv[q + o[k]], rw = (double)g.rho[q + o[k]] * cw;
        t.r += rw;
        t.w += cw;
        own.r = k == 0 ? rw : own.r + rw;
        own.w = k == 0 ? cw : own.w + cw;
        if (k == 0) {
          own.r0 = rw;
          own.w0 = cw;
        }
      }
      return t;
    };
    Quad lo = quad(c, 0.0, 0.0);
    double dlo = z0 >= 1 ? (double)g.bz[c - g.sxy] : 0.0;
    const double ex = ix == 0 || ix == g.nx ? 0.5 : 1.0, ey = iy == 0 || iy == g.ny ? 0.5 : 1.0;
    for (int iz = z0; iz <= z1; ++iz, c += g.sxy) {
      Quad up;
      const Quad t = both(c + g.sxy, lo.r, lo.w, up);
      const double d0 = g.bz[c];
      if (ix >= 1 && iy >= 1 && iz >= 1) {
        const double b0 = g.bx[c], b1 = g.bx[c - 1], c0 = g.by[c], c1 = g.by[c - sx];
        double w1 = (b0 * b0 + b1 * b1) * 0.5;
        const double w2 = (c0 * c0 + c1 * c1) * 0.5, w3 = (d0 * d0 + dlo * dlo) * 0.5;
        w1 = (w1 + w2 + w3) * 0.5;
        v[0] += w1 * lo.w0;
        v[2] += (double)g.energy[c] * lo.r0;
      }
      const double ux = g.vx[c], uy = g.vy[c], uz = g.vz[c];
      // rho_v cv_v = (sum rho cv / sum cv) (sum cv / 8)
      double w1 = t.r / t.w * (t.w * 0.125) * (ux * ux + uy * uy + uz * uz);
      w1 = w1 * ex * ey;
      if (iz == 0 || iz == g.nz) w1 = w1 * 0.5;
      v[1] += w1 * 0.5;
      lo = up;
      dlo = d0;
    }
  }
  const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  block_sum_write<3>(v, g.partial, bid);
  last_block_sum<3>(g.partial, (int)(gridDim.x * gridDim.y * gridDim.z), g.out, 0, g.done);
}

template <class R>
void energy_account(Run<R>& run) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  Arrays<R>& A = run.a;
  dim3 grd((nx + 1 + 63) / 64, (ny + 1 + 3) / 4, 1);
  int planes = march_chunk(nz + 1, grd.x * grd.y, 32, resident_blocks<k_energy_account<R>>(256));
  // few enough partials for the last block (box_sum), and room for them
  while (planes < 64 && (long long)grd.x * grd.y * ((nz + planes) / planes) > 4096) planes *= 2;
  grd.z = (nz + planes) / planes;
  const EnergyArgs<R> g{A.bx.p,      A.by.p, A.bz.p, A.cv.p, A.energy.p, A.rho.p, A.vx.p, A.vy.p, A.vz.p, run.partial,
                        run.sc + SC_EN_B, (unsigned*)(run.us + U_DONE), nx, ny, nz, run.sx, run.sxy, planes};
  const int k = run.prof_begin("energy_account", 0, 9, (double)(nx + 1) * (ny + 1) * (nz + 1));
  k_energy_account<R><<<grd, dim3(64, 4, 1), 0, run.s>>>(g);
  run.prof_end(k);
  ++run.launches;
}

LARE_END  // namespace lare

LARE_BEGIN

// diagnostics.F90:613-629 energy_correction, after eulerian_remap when rke
// is on (lare3d.f90:86): the kinetic energy the remap lost, where it lost
// some, goes into the internal energy of cells 1:n; then energy_bcs.
template <class R>
void energy_correction(Run<R>& run) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  auto dke = run.a.delta_ke, rho = run.a.rho, cv = run.a.cv, energy = run.a.energy;
  LARE_BOXW(run, 5, 1, nx, 1, ny, 1, nz, [=] __device__(int ix, int iy, int iz) {
    R d = -dke(ix, iy, iz);
    if (d < R(0)) d = R(0);
    d = d / (rho(ix, iy, iz) * cv(ix, iy, iz));
    dke(ix, iy, iz) = d;
    energy(ix, iy, iz) = energy(ix, iy, iz) + d;
  });
  energy_bcs(run);
}

LARE_END  // namespace lare

#include "openbc.cuh"

LARE_BEGIN

template <int F, class R>
inline void open_face(Run<R>& run, const OpenArgs<R>& g) {
  if (run.p.bc[F / 2][F & 1] != LARE_BC_OPEN) return;
  const int nu = F / 2 == 0 ? run.n[1] : run.n[0], nw = F / 2 == 2 ? run.n[1] : run.n[2];
  dim3 blk(32, 4, 1);
  dim3 grd((nu + 2 + 31) / 32, (nw + 2 + 3) / 4, 1);
  const int k = run.prof_begin("open_bcs", F, 0, (double)(nu + 2) * (nw + 2));
  k_open_face<F, R><<<grd, blk, 0, run.s>>>(g);
  run.prof_end(k);
  ++run.launches;
}

// openboundary.f90:30-324 open_bcs: the open faces in the reference's order.
template <class R>
void open_bcs(Run<R>& run) {
  OpenArgs<R> g;
  g.vx = run.a.vx.p;
  g.vy = run.a.vy.p;
  g.vz = run.a.vz.p;
  g.bx = run.a.bx.p;
  g.by = run.a.by.p;
  g.bz = run.a.bz.p;
  g.rho = run.a.rho.p;
  g.energy = run.a.energy.p;
  g.g = (R)run.p.gamma;
  g.nx = run.n[0];
  g.ny = run.n[1];
  g.nz = run.n[2];
  g.sx = run.sx;
  g.sxy = run.sxy;
  open_face<0>(run, g);
  open_face<1>(run, g);
  open_face<2>(run, g);
  open_face<3>(run, g);
  open_face<4>(run, g);
  open_face<5>(run, g);
}

LARE_END  // namespace lare

#include "lagran.cuh"
