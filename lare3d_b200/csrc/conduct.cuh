// conduct.cuh - the heat flux of conduct.f90:152-291 and the RKL2 stage of
// conduct.f90:299-416 as tiled kernels.
//
// Face flux (conduct.f90:170-275), x face between cells ix and ix+1:
//   q = -L k0 T_f^{5/2} (b0 (b0 g_x + by_f g_y + bz_f g_z) + min_b g_x) / |B|^2
// with T_f the face-mean temperature, g the temperature gradient at the
// face (the transverse parts from the face-mean temperatures of the two
// neighbouring rows), L the Larsen factor of cell ix and |B|^2 = b0^2 +
// by_f^2 + bz_f^2 + min_b.  heat_flux scatters q / dxb(ix) into the two
// cells.  Everything but T is fixed during a conduction step, so
// face_coefficients forms, once per step, three coefficients per face
//   k_n = L (b0^2 + min_b) / |B|^2 / dxc(ix) / dxb(ix)
//   k_1 = L b0 by_f / |B|^2 / (2 (dyc(iy) + dyc(iy-1))) / dxb(ix)
//   k_2 = L b0 bz_f / |B|^2 / (2 (dzc(iz) + dzc(iz-1))) / dxb(ix)
// and the stage kernel evaluates q / dxb = -k0 T_f^{5/2} (k_n dT_n + k_1 dS_1
// + k_2 dS_2) with dT_n = T(ix+1) - T(ix) and dS the differences of the
// two-point temperature sums of the neighbouring rows.  The same algebra,
// regrouped (and T^{5/2} = T^2 sqrt(T)), agrees with the reference to
// rounding (relative 1e-12 in FP64).
//
// Stage kernel: each face flux is formed once; a cell adds its six scaled face
// fluxes in the order in which the reference's scatter delivers them:
//   +Fz(c-ez), +Fy(c-ey), +Fx(c-ex), -Fx(c), -Fy(c), -Fz(c).
#pragma once

LARE_BEGIN

constexpr int kCTY = 8, kCZ = 32;             // rows of a CTA tile, largest chunk of z (march_chunk)
// Coefficients of every face of cells 0..n (conduct.f90:170-275 regrouped).
template <class R>
void face_coefficients(Run<R>& run) {
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  Arrays<R>& A = run.a;
  auto bx = A.bx, by = A.by, bz = A.bz, larsen = A.larsen;
  const A1<R> rdb0 = A.rdb[0], rdb1 = A.rdb[1], rdb2 = A.rdb[2];
  const A1<R> rdc0 = A.rdc[0], rdc1 = A.rdc[1], rdc2 = A.rdc[2];
  const A1<R> rs0 = A.rdc2[0], rs1 = A.rdc2[1], rs2 = A.rdc2[2];
  A3<R> k[9];
  for (int q = 0; q < 9; ++q) k[q] = A.kf[q];
  const A3<R> k0 = k[0], k1 = k[1], k2 = k[2], k3 = k[3], k4 = k[4], k5 = k[5], k6 = k[6], k7 = k[7], k8 = k[8];
  // Extension, not in the reference: kappa_perp = rp kappa_par adds
  // rp (g_n - b_n (b . g) / |B|^2) to the bracket, i.e. rp (|B|^2 - b0^2)
  // to the normal coefficient's numerator and a factor (1 - rp) to the
  // transverse ones; rp = 0 is the reference's flux.
  const R rp = (R)run.p.kappa_perp_ratio, orp = R(1) - rp;
  LARE_BOXW(run, 13, 0, nx, 0, ny, 0, nz, [=] __device__(int ix, int iy, int iz) {
    const R min_b = R(1.0e-10);  // conduct.f90:28
    const R half = R(0.5), q4 = R(0.25);
    const int ixp = ix + 1, ixm = ix - 1, iyp = iy + 1, iym = iy - 1, izp = iz + 1, izm = iz - 1;
    const R lf = larsen(ix, iy, iz);
    {  // x face
      const R byf = q4 * (by(ix, iy, iz) + by(ixp, iy, iz) + by(ix, iym, iz) + by(ixp, iym, iz));
      const R bzf = q4 * (bz(ix, iy, iz) + bz(ixp, iy, iz) + bz(ix, iy, izm) + bz(ixp, iy, izm));
      const R b0 = bx(ix, iy, iz);
      const R modb = b0 * b0 + byf * byf + bzf * bzf + min_b;
      const R w = lf / modb * rdb0(ix);
      k0(ix, iy, iz) = w * ((b0 * b0 + min_b) + rp * (modb - b0 * b0)) * rdc0(ix);
      k1(ix, iy, iz) = w * b0 * byf * orp * half * rs1(iy);
      k2(ix, iy, iz) = w * b0 * bzf * orp * half * rs2(iz);
    }
    {  // y face
      const R bxf = q4 * (bx(ix, iy, iz) + bx(ix, iyp, iz) + bx(ixm, iy, iz) + bx(ixm, iyp, iz));
      const R bzf = q4 * (bz(ix, iy, iz) + bz(ix, iyp, iz) + bz(ix, iy, izm) + bz(ix, iyp, izm));
      const R b0 = by(ix, iy, iz);
      const R modb = bxf * bxf + b0 * b0 + bzf * bzf + min_b;
      const R w = lf / modb * rdb1(iy);
      k3(ix, iy, iz) = w * ((b0 * b0 + min_b) + rp * (modb - b0 * b0)) * rdc1(iy);
      k4(ix, iy, iz) = w * b0 * bxf * orp * half * rs0(ix);
      k5(ix, iy, iz) = w * b0 * bzf * orp * half * rs2(iz);
    }
    {  // z face
      const R bxf = q4 * (bx(ix, iy, iz) + bx(ix, iy, izp) + bx(ixm, iy, iz) + bx(ixm, iy, izp));
      const R byf = q4 * (by(ix, iy, iz) + by(ix, iy, izp) + by(ix, iym, iz) + by(ix, iym, izp));
      const R b0 = bz(ix, iy, iz);
      const R modb = bxf * bxf + byf * byf + b0 * b0 + min_b;
      const R w = lf / modb * rdb2(iz);
      k6(ix, iy, iz) = w * ((b0 * b0 + min_b) + rp * (modb - b0 * b0)) * rdc2(iz);
      k7(ix, iy, iz) = w * b0 * bxf * orp * half * rs0(ix);
      k8(ix, iy, iz) = w * b0 * byf * orp * half * rs1(iy);
    }
  });
}

template <class R>
struct StageArgs {
  R* lc0;                           // Lc_Y0: written by stage 1
  R* out;
  const R* kz[3];                   // the z faces' coefficients
  const R* y2;                      // the stage input where the temperature is an array of its own, else null
  double* sc;
  R tc, te0;                        // temperature of the input: tc * (y - te0)
  R k0, mt, mu, nu, omn, gt;
  int dt_slot, nx, ny, nz, sx, sxy;
  int chunk;
};
struct StageMaps {
  CUtensorMap T, k[9], rho, y0, y1, lc0;
};

template <class R>
__device__ __forceinline__ R face_q(R k0, R T0, R T1, R kn, R k1, R s1, R k2, R s2) {
  R tb = (T1 + T0) * R(0.5);
  tb = tb > R(0) ? tb : R(0);
  return -k0 * pow25(tb) * (kn * (T1 - T0) + k1 * s1 + k2 * s2);
}

// Stage kernel.  A CTA of 32 x 8 threads owns a tile of 31 x 8 cells and
// walks a chunk of z.  Each thread forms the x face flux on the low side of
// its cell; lane 31's cell belongs to the next tile and only hands its low
// face to lane 30 (the high face of every cell comes from the lane above by
// a shuffle, so no lane forms a face twice).  Each thread also forms the y
// face flux on the low side of its cell into shared memory, where the row
// below reads it as its high face; the top row forms its high face itself.
// The z face flux on the high side is carried to the next plane.
//
// The planes arrive by TMA two steps ahead: the stage input with a one-cell x/y
// halo in a ring of four slots, of which three are read, and the nine face
// coefficients, rho, Y0, Y1 and Lc_Y0 of the plane itself in a ring of two.
// The input becomes the temperature in place a step before it is read (its
// value at the thread's own cell stays in a register).  One barrier a step
// orders that, the y faces and the reuse of slots.  With each array loaded by each thread a plane
// ahead a stage took 0.30 ms at 256^3 in FP32 and 0.136 ms on 160 x 129 x 177
// in FP64 (400 and 530 instructions a point, 118 registers in FP64); now 0.20
// and 0.116 ms.  Its floor is 15 words, 0.155 and 0.067 ms; bound by
// instruction issue and, in FP64, by 16 warps an SM.  (Rings of six and three
// slots left one CTA an SM in FP64: 0.183 ms.)
constexpr int kSTX = 31;  // cells per tile along x (a warp of 32 lanes)
constexpr int kStT = 4, kStD = 2;  // slots of the two rings
template <class R>
struct StageTile {
  static constexpr int W = sizeof(R) == 8 ? 36 : 40;  // 34 elements from the aligned start
  static constexpr int t = (W * (kCTY + 2) * (int)sizeof(R) + 127) / 128 * 128;
  static constexpr int h = (W * (kCTY + 1) * (int)sizeof(R) + 127) / 128 * 128;  // y coefficients: a row below
  static constexpr int c = (W * kCTY * (int)sizeof(R) + 127) / 128 * 128;
  static constexpr int kx = 0, kz = 3 * c, rho = 6 * c, y0 = 7 * c, y1 = 8 * c, lc = 9 * c, ky = 10 * c;
  static constexpr int slot = 10 * c + 3 * h;
  static constexpr unsigned sent_t = W * sizeof(R) * (kCTY + 2);
  static constexpr unsigned sent = W * sizeof(R) * (10 * kCTY + 3 * (kCTY + 1));
  static constexpr unsigned sent1 = sent - W * sizeof(R) * 2 * kCTY;             // stage 1: no Y1, no Lc_Y0
  static constexpr size_t smem = 128 + (size_t)kStT * t + (size_t)kStD * slot;
};

// FIRST: stage 1 (Y0 the input): Lc_Y0 = flux / rho and
//        out = Y0 + mt * dt * Lc_Y0.
// else:  stage j: out = mu Y2 + nu Y1 + (1 - mu - nu) Y0 + mt dt Lc + gt dt Lc_Y0
//        with Lc the flux of T(Y2) / rho.
template <class R, bool FIRST>
__global__ void __launch_bounds__(32 * kCTY, sizeof(R) == 4 ? 5 : 2)
    k_rkl2_stage(const __grid_constant__ StageMaps maps, StageArgs<R> a) {
  using L = StageTile<R>;
  extern __shared__ unsigned char st_smem[];
  __shared__ R fy[2][kCTY + 1][32];
  __shared__ __align__(8) unsigned long long bars[kStT];
  constexpr int W = L::W;
  const int nx = a.nx, ny = a.ny, nz = a.nz;
  const int lane = threadIdx.x, ty = threadIdx.y;
  const int ix0 = 1 + (int)blockIdx.x * kSTX, iy0 = 1 + (int)blockIdx.y * kCTY;
  const int iz0 = 1 + (int)blockIdx.z * a.chunk;
  const int iz1 = min(nz, iz0 + a.chunk - 1);
  const int ix = ix0 + lane, iy = iy0 + ty;
  const bool active = lane < kSTX && ix <= nx && iy <= ny;    // cells this tile updates
  const bool top = ty == kCTY - 1;                            // the top row also forms its high y face
  unsigned char* const buf = st_smem + ((128u - (smem_addr(st_smem) & 127u)) & 127u);
  unsigned char* const dat = buf + kStT * L::t;
  const uint32_t buf_s = smem_addr(buf), dat_s = buf_s + kStT * L::t, bar_s = smem_addr(bars);
  const int e0 = ix0 + 1, ea = e0 & ~(kTmaAlign<R> - 1);      // element of ix0 - 1, counted from x = -2
  // step s: the input's plane iz0 + s + 1 and the other arrays' plane iz0 + s;
  // steps -2 and -1 bring the input's planes iz0 - 1 and iz0
  auto issue = [&](int s) {
    const int q = s + 2, p = iz0 + s + 2;
    const uint32_t bar = bar_s + 8 * (q % kStT);
    mbar_expect(bar, s < 0 ? L::sent_t : L::sent_t + (FIRST ? L::sent1 : L::sent));
    tma_load_3d(buf_s + (q % kStT) * L::t, &maps.T, ea, iy0 + 1, p + 1, bar);
    if (s < 0) return;
    const uint32_t d = dat_s + (s % kStD) * L::slot;
    const int r = iy0 + 2;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      tma_load_3d(d + L::kx + m * L::c, &maps.k[m], ea, r, p, bar);
      tma_load_3d(d + L::ky + m * L::h, &maps.k[3 + m], ea, r - 1, p, bar);
      tma_load_3d(d + L::kz + m * L::c, &maps.k[6 + m], ea, r, p, bar);
    }
    tma_load_3d(d + L::rho, &maps.rho, ea, r, p, bar);
    tma_load_3d(d + L::y0, &maps.y0, ea, r, p, bar);
    if (!FIRST) {
      tma_load_3d(d + L::y1, &maps.y1, ea, r, p, bar);
      tma_load_3d(d + L::lc, &maps.lc0, ea, r, p, bar);
    }
  };
  const int steps = iz1 - iz0 + 1;
  const bool boss = lane == 0 && ty == 0;
  if (boss) {
    for (int q = 0; q < kStT; ++q) mbar_init(bar_s + 8 * q, 1);
    mbar_init_fence();
    for (int s = -2; s < 2 && s < steps; ++s) issue(s);
  }
  int dead = 0;
  auto await = [&](int s) {
    const int q = s + 2;
    tile_wait(bar_s + 8 * (q % kStT), (uint32_t)(q / kStT) & 1u, dead, a.sc);
  };
  const R tc = a.tc, te0 = a.te0, k0 = a.k0;
  const R dt = (R)a.sc[a.dt_slot];
  // this thread's cell in a plane of the input and in the other tiles, and the
  // halo element that it turns into a temperature (84 of them)
  const int ec = (ty + 1) * W + (e0 - ea) + lane + 1, cc = ty * W + (e0 - ea) + lane + 1;
  const int tid = ty * 32 + lane;
  const int eh = (e0 - ea) + (tid < 68 ? (tid < 34 ? tid : (kCTY + 1) * W + tid - 34)
                                       : ((tid - 68) / 2 + 1) * W + (tid & 1) * 33);
  auto plane = [&](int s) { return reinterpret_cast<R*>(buf + ((s + 2) % kStT) * L::t); };
  auto convert = [&](int s) {
    await(s);
    R* const p = plane(s);
    const R own = p[ec];
    p[ec] = tc * (own - te0);
    if (tid < 84) p[eh] = tc * (p[eh] - te0);
    return own;
  };
  // z face above the cell of planes lo (lower) and hi
  auto zface = [&](const R* lo, const R* hi, R k6, R k7, R k8) {
    return face_q(k0, lo[0], hi[0], k6, k7, (hi[1] + lo[1]) - (hi[-1] + lo[-1]), k8,
                  (hi[W] + lo[W]) - (hi[-W] + lo[-W]));
  };
  // y face between the cells at e - W and e of planes Pm, P0, Pp
  auto yface = [&](const R* Pm, const R* P0, const R* Pp, R k3, R k4, R k5) {
    return face_q(k0, P0[-W], P0[0], k3, k4, (P0[-W + 1] + P0[1]) - (P0[-W - 1] + P0[-1]), k5,
                  (Pp[-W] + Pp[0]) - (Pm[-W] + Pm[0]));
  };
  __syncthreads();  // the barriers are set up
  convert(-2);
  R own0 = convert(-1), own1 = convert(0);  // the input at this cell, planes iz and iz + 1
  __syncthreads();
  R fz_m = R(0);
  {
    // the z face below the chunk
    const int c = min(ix, nx + 2) + a.sx * min(iy, ny + 2) + a.sxy * (iz0 - 1);
    fz_m = zface(plane(-2) + ec, plane(-1) + ec, a.kz[0][c], a.kz[1][c], a.kz[2][c]);
  }
  for (int s = 0; s < steps; ++s) {
    const R* const Pm = plane(s - 2) + ec;
    const R* const P0 = plane(s - 1) + ec;
    const R* const Pp = plane(s) + ec;
    const unsigned char* const sl = dat + (s % kStD) * L::slot;
    auto at = [&](int off) { return reinterpret_cast<const R*>(sl + off)[cc]; };
    // x face between cells ix - 1 and ix
    const R* const kx = reinterpret_cast<const R*>(sl + L::kx) + cc - 1;
    const R fx_lo = face_q(k0, P0[-1], P0[0], kx[0], kx[L::c / (int)sizeof(R)],
                           (P0[W] + P0[W - 1]) - (P0[-W] + P0[-W - 1]), kx[2 * L::c / (int)sizeof(R)],
                           (Pp[0] + Pp[-1]) - (Pm[0] + Pm[-1]));
    const R fx_hi = __shfl_down_sync(0xffffffffu, fx_lo, 1);
    // (the y coefficients' tile starts a row lower, so cc is the row below)
    const R* const ky = reinterpret_cast<const R*>(sl + L::ky) + cc;
    R(*const f)[32] = fy[s & 1];
    f[ty][lane] = yface(Pm, P0, Pp, ky[0], ky[L::h / (int)sizeof(R)], ky[2 * L::h / (int)sizeof(R)]);
    if (top)
      f[kCTY][lane] = yface(Pm + W, P0 + W, Pp + W, ky[W], ky[W + L::h / (int)sizeof(R)],
                            ky[W + 2 * L::h / (int)sizeof(R)]);
    const R fz_p = zface(P0, Pp, at(L::kz), at(L::kz + L::c), at(L::kz + 2 * L::c));
    const R rr = R(1) / at(L::rho), v0 = at(L::y0);
    const R v1 = FIRST ? R(0) : at(L::y1), l0 = FIRST ? R(0) : at(L::lc), v2 = own0;
    own0 = own1;
    if (s + 1 < steps) own1 = convert(s + 1);
    __syncthreads();
    // every thread is past the last step: its slots are free
    if (boss && !dead && s + 2 < steps) {
      // the copy overwrites a plane that threads wrote (converted) before the barrier
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue(s + 2);
    }
    if (active) {
      R g = fz_m;
      g = g + f[ty][lane];
      g = g + fx_lo;
      g = g - fx_hi;
      g = g - f[ty + 1][lane];
      g = g - fz_p;
      const int c = ix + a.sx * iy + a.sxy * (iz0 + s);
      const R Lc = rr * g;
      if (FIRST) {
        a.lc0[c] = Lc;
        a.out[c] = v0 + a.mt * dt * Lc;
      } else {
        const R c0 = a.gt * dt * l0;
        const R c1 = a.mt * dt * Lc;
        const R yy = a.y2 ? a.y2[c] : v2;
#if LARE_FAST
        // the order of the fused operations is written out: 1 - mu - nu is held in omn, and on a
        // uniform energy another order rounds the same way in every cell of a stage (1.8e-8 of a
        // walls deck's internal energy in FP32)
        const R v = fma(a.omn, v0, fma(a.mu, yy, a.nu * v1));
#else
        const R v = a.mu * yy + a.nu * v1 + a.omn * v0;
#endif
        a.out[c] = v + c1 + c0;
      }
    }
    fz_m = fz_p;
  }
}

// Dynamic shared memory beyond the default 48 KiB, once per context.
template <class R>
inline cudaError_t stage_attributes() {
  cudaError_t e = cudaFuncSetAttribute(k_rkl2_stage<R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)StageTile<R>::smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_rkl2_stage<R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)StageTile<R>::smem);
  return e;
}

template <class R, bool FIRST>
void rkl2_stage(Run<R>& run, int line, const TempOf<R>& T, A3<R> y2, A3<R> y1, A3<R> y0, A3<R> out, int dt_slot,
                R mt, R mu, R nu, R omn, R gt) {
  using L = StageTile<R>;
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  StageArgs<R> a;
  a.lc0 = run.a.Lc_Y0.p;
  a.out = out.p;
  for (int q = 0; q < 3; ++q) a.kz[q] = run.a.kf[6 + q].p;
  a.y2 = T.y.p == y2.p ? nullptr : y2.p;
  a.sc = run.sc;
  a.tc = T.c;
  a.te0 = T.e0;
  a.k0 = (R)run.p.kappa_0;
  a.mt = mt;
  a.mu = mu;
  a.nu = nu;
  a.omn = omn;
  a.gt = gt;
  a.dt_slot = dt_slot;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.sx = run.sx;
  a.sxy = run.sxy;
  StageMaps maps;
  const long long f = 2 + 2LL * run.sx + 2LL * run.sxy;
  const auto map = [&](CUtensorMap* m, const A3<R>& x, int rows) {
    make_map(run, m, (const R*)x.p - f, L::W, rows, 1);
  };
  map(&maps.T, T.y, kCTY + 2);
  for (int q = 0; q < 9; ++q) map(&maps.k[q], run.a.kf[q], q / 3 == 1 ? kCTY + 1 : kCTY);
  map(&maps.rho, run.a.rho, kCTY);
  map(&maps.y0, y0, kCTY);
  map(&maps.y1, y1, kCTY);
  map(&maps.lc0, run.a.Lc_Y0, kCTY);
  if (run.launch_error) return;
  dim3 grid((nx + kSTX - 1) / kSTX, (ny + kCTY - 1) / kCTY, 1);
  a.chunk = march_chunk(nz, grid.x * grid.y, kCZ, resident_blocks<k_rkl2_stage<R, FIRST>>(32 * kCTY, L::smem));
  grid.z = (nz + a.chunk - 1) / a.chunk;
  // words per point: T stencil input, 9 coefficients, rho, Lc_Y0, output (+ Y1, Y0 after stage 1)
  const int k = run.prof_begin("rkl2_stage", line, FIRST ? 13 : 15, (double)nx * ny * nz);
  k_rkl2_stage<R, FIRST><<<grid, dim3(32, kCTY, 1), L::smem, run.s>>>(maps, a);
  run.prof_end(k);
  ++run.launches;
}

LARE_END  // namespace lare
