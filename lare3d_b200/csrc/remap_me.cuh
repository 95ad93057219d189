// remap_me.cuh - volumes, mass and energy of one directional remap sweep as
// one kernel: cv1 and cv2 (xremap.f90:57-86), the mass flux dm (:474-533) over
// the whole cell box with dm_[xyz]_bcs (:899-917) folded in, the new density
// (:174-182), the energy flux (:539-601) and the new energy (:187-196), with
// the mirrors of yremap.f90 and zremap.f90.
//
// The moved widths db1 and dc1 along the sweep axis come from the face
// velocity that the mass flux reads anyway, and cv1 and cv2 from the face
// velocities of the other axes, so no geometry array is read: the three
// velocity components, rho, energy and cv are read and dm, rho, energy, cv1
// and cv2 written (11 words a point in the first sweep), where a geometry
// kernel and this one moved 18.  An axis already swept drops out of the
// volumes (its pass flag is 0: 0 * dv / dx = 0), so a sweep reads only the
// components still to come (SWEPT: how many of the two other axes are done;
// the third sweep's cv2 is cv itself and is not written).
//
// At 256^3 a sweep takes 0.30 to 0.37 (y, z) and 0.40 ms (x) in FP64 with the
// components still to come, 0.24 ms in FP32, where the geometry kernel and this
// one took 0.59 and 0.67, 0.35 and 0.41 ms; its floor is 0.23 ms (11 words, FP64).
// Bound by instruction issue (55 % of slots) and FP64 latency at 16 warps an SM.  With plain loads a step ahead instead of
// the ring: 0.54 and 0.53 ms (168 registers, waiting on memory).
//
// The fluxes of the point below are carried, so neither flux but dm reaches
// memory.  The new density and energy go to second buffers: neighbouring
// threads' limiters still read the old values.  Every value is the
// reference's expression over the same operands in the same order.
#pragma once

LARE_BEGIN

constexpr int kMeXOut = 27;        // x sweep: lanes 3..29 write (stencils and left fluxes by shuffles)
constexpr int kMeXFirst = 3;

template <class R>
struct MEArgs {
  const R* v[3];                   // v1 along x, y, z
  const R* rho;                    // old density (rho1)
  R* rho_new;
  const R* energy;                 // old energy
  R* energy_new;
  R* dm;
  const R* cv;
  R* cv1;
  R* cv2;                          // not written where both other axes are swept
  R* db1;                          // rke only: the moved widths, for the split momentum kernels
  R* dc1;
  A1<R> m[3], r[3];                // cell widths and their reciprocals
  double* sc;
  int dt_slot, nx, ny, nz, sx, sxy;
  int chunk;
  int pass[3];
  bool per;                        // periodic along the sweep axis
};

// The mass flux at index s along the sweep axis, everything loaded from
// memory (dm's ghost values, taken at their source index).
template <int A, class R>
__device__ __forceinline__ R me_mass_flux(const MEArgs<R>& g, int c, int s, int S1, int S2, int SA, R dt, R area) {
  const R* __restrict__ va = g.v[A];
  auto vface = [&](int q) { return (va[q] + va[q - S1] + va[q - S2] + va[q - S1 - S2]) * R(0.25); };
  const R fmm = vface(c - 2 * SA), fm = vface(c - SA), f0 = vface(c), fp = vface(c + SA);
  const R fp2 = vface(c + 2 * SA);  // s + 2 <= n + 2 for every source index
  const A1<R> w = g.m[A];
  const R dbm = w(s - 1) + (fm - fmm) * dt, db0 = w(s) + (f0 - fm) * dt, dbp = w(s + 1) + (fp - f0) * dt;
  const R dbp2 = w(s + 2) + (fp2 - fp) * dt;
  const R dcm = R(0.5) * (dbm + db0), dc0 = R(0.5) * (db0 + dbp), dcp = R(0.5) * (dbp + dbp2);
  const LimOut<R> L = limiter<R>(f0, g.rho[c - SA], g.rho[c], g.rho[c + SA], g.rho[c + 2 * SA], dc0, dcm, dcp, db0,
                                 dbp, R(0), R(0), dt, false);
  return (L.fu + L.Di * (R(1) - L.phi)) * f0 * dt * area;
}

// Where dm at index ia along the axis comes from: ia itself, or dm_[xyz]_bcs'
// source index; NONE: zero.
__device__ __forceinline__ int me_source(int ia, int n, bool per, bool& none) {
  none = false;
  if (per) {
    if (ia == n + 1) return 1;
    if (ia == n + 2) return 2;
    if (ia == -1) return n - 1;
    if (ia == 0) return n;
  } else {
    if (ia == n + 1) return n;
    if (ia == -1) return 0;
    if (ia == n + 2) none = true;
  }
  return ia;
}

// The volumes after the sweep along A and before it (the reference's
// xpass/ypass/zpass terms), from the face velocity differences; H1, H2: the
// transverse axes still to be swept.
template <int A, bool H1, bool H2, class R>
__device__ __forceinline__ void me_volumes(const MEArgs<R>& g, const R (&dv)[3], int ix, int iy, int iz, R dt, R cv,
                                           R& c1, R& c2) {
  constexpr int T1 = A == 0 ? 1 : 0, T2 = A == 2 ? 1 : 2;
  const int pp[3] = {ix, iy, iz};
#if LARE_FAST
  auto quot = [&](R a, int d) { return a * g.r[d](pp[d]); };
#else
  auto quot = [&](R a, int d) { return div_rcp(a, g.m[d](pp[d]), g.r[d](pp[d])); };
#endif
  const R t1 = H1 ? quot(dv[T1], T1) : R(0), t2 = H2 ? quot(dv[T2], T2) : R(0);
  const R t12 = t1 + t2;
  c1 = cv * (R(1) + (t12 + quot(dv[A], A)) * dt);
  c2 = cv * (R(1) + t12 * dt);
}

// What the x and t faces of a y or z sweep need of one plane of v_x and v_t:
// the point, its neighbour below along the face's own axis, and both one down
// along the other transverse axis.
template <class R>
struct Tr2 {
  R x0, xm, x0t, xmt;  // v_x at x, x - 1, and both at t - 1
  R t0, tm, t0x, tmx;  // v_t at t, t - 1, and both at x - 1
  __device__ __forceinline__ void load_x(const R* p, int st) {
    x0 = p[0];
    xm = p[-1];
    x0t = p[-st];
    xmt = p[-st - 1];
  }
  __device__ __forceinline__ void load_t(const R* p, int st) {
    t0 = p[0];
    tm = p[-st];
    t0x = p[-1];
    tmx = p[-st - 1];
  }
  // face velocity differences from this plane and the one below (m), summed
  // in the reference's order: the lower transverse axis first (xremap.f90:64-86)
  template <int A>
  __device__ __forceinline__ R diff_x(const Tr2& m) const {
    const R q = R(0.25);
    if (A == 1) return (x0 + m.x0 + x0t + m.x0t) * q - (xm + m.xm + xmt + m.xmt) * q;
    return (x0 + x0t + m.x0 + m.x0t) * q - (xm + xmt + m.xm + m.xmt) * q;
  }
  template <int A>
  __device__ __forceinline__ R diff_t(const Tr2& m) const {
    const R q = R(0.25);
    return (t0 + t0x + m.t0 + m.t0x) * q - (tm + tmx + m.tm + m.tmx) * q;
  }
};

// The mass and energy fluxes of one point: rho or energy at -1..2, the
// carried divisors dc1 at -1..1, db1 at 0 and 1, the face velocity.  In the
// product build what the two share (the upwind choice, phi and the upwind
// widths) is formed once.
template <class R>
struct MEFace {
  R vf, dt, area;
  bool up;
  R phi, dxb, dxb6, vd0, vdu;  // kRegroup
  R vdc[3], db0, dbp;          // else
  __device__ __forceinline__ MEFace(const R (&vdc_)[3], R db0_, R dbp_, R vf_, R dt_, R area_)
      : vf(vf_), dt(dt_), area(area_) {
    if constexpr (kRegroup<R>) {
      up = !signbit(vf);
      dxb = up ? db0_ : dbp_;
      phi = fabs(vf) * dt * fast_rcp(dxb);
      dxb6 = dxb * (R(1) / R(6));
      vd0 = vdc_[1];
      vdu = up ? vdc_[0] : vdc_[2];
    } else {
      db0 = db0_;
      dbp = dbp_;
      vdc[0] = vdc_[0];
      vdc[1] = vdc_[1];
      vdc[2] = vdc_[2];
    }
  }
  // upwind value and limited difference
  __device__ __forceinline__ R limited(const R (&f)[4], R& fu) const {
    const R dm = f[1] - f[0], d0 = f[2] - f[1], dp = f[3] - f[2];
    const R du = up ? dm : dp;
    fu = up ? f[1] : f[2];
    const R da = (R(2) - phi) * (fabs(d0) * vd0) + (R(1) + phi) * (fabs(du) * vdu);
    return signed_min(lesser(lesser(R(fabs(da) * dxb6), R(fabs(d0))), R(fabs(du))), d0, du, vf);
  }
  __device__ __forceinline__ LimOut<R> plain(const R (&f)[4]) const {
    return limiter_dv<R>(vf, f[0], f[1], f[2], f[3], vdc[1], vdc[0], vdc[2], db0, dbp, R(0), R(0), dt, false);
  }
  __device__ __forceinline__ R mass(const R (&r)[4]) const {
    if constexpr (kRegroup<R>) {
      R fu;
      const R D = limited(r, fu);
      return (fu + D * (R(1) - phi)) * vf * dt * area;
    } else {
      const LimOut<R> L = plain(r);
      return (L.fu + L.Di * (R(1) - L.phi)) * vf * dt * area;
    }
  }
  __device__ __forceinline__ R energy(const R (&e)[4], R r0, R rp, R dm) const {
    if constexpr (kRegroup<R>) {
      R fu;
      const R D = limited(e, fu);
      const R dmu = fabs(dm) * fast_rcp(area * dxb * (up ? r0 : rp));
      return (fu + D * (R(1) - dmu)) * dm;
    } else {
      const LimOut<R> L = plain(e);
      const R rhou = r0 * L.vad_p + rp * L.vad_m;
#if LARE_FAST
      const R dmu = fabs(dm) * fast_rcp(area * L.dxbu * rhou);
#else
      const R dmu = fabs(dm) / area / L.dxbu / rhou;
#endif
      return (L.fu + L.Di * (R(1) - dmu)) * dm;
    }
  }
};

// The y and z sweeps.  A block of 32 x kMeY threads owns a tile of lines along
// A, x along the lanes and the third axis t along the rows (the cell box
// -1..n+2), and walks a chunk of it.  Each step's values arrive in a ring of
// shared-memory slots by TMA, two steps ahead: rho, energy and the velocity
// along A of the plane that enters the windows (two points on), and the other
// velocity components and cv of the point itself; the plane below's are still
// in the previous slot.  HX, HT: whether the x and t axes are still to be
// swept, so that their velocities enter the volumes.
constexpr int kMeY = 8, kMeSlots = 4;
template <bool HX, bool HT, class R>
struct METile {
  static constexpr int W = 36;                                                    // 33 elements, to 16 bytes
  static constexpr int h = (W * (kMeY + 1) * (int)sizeof(R) + 127) / 128 * 128;   // with a halo row
  static constexpr int c = (W * kMeY * (int)sizeof(R) + 127) / 128 * 128;
  static constexpr int oe = h + c, oc = h + 2 * c, ox = h + 3 * c, ot = ox + (HX ? h : 0);
  static constexpr int slot = ot + (HT ? h : 0);
  static constexpr unsigned sent = W * sizeof(R) * ((kMeY + 1) * (1 + (HX ? 1 : 0) + (HT ? 1 : 0)) + 3 * kMeY);
  static constexpr size_t smem = 128 + (size_t)kMeSlots * slot;
};
struct MEMaps {
  CUtensorMap va, rho, energy, cv, vx, vt;
};

template <int A, bool HX, bool HT, class R>
__global__ void __launch_bounds__(32 * kMeY, sizeof(R) == 8 ? 2 : 4)
    k_me_march(const __grid_constant__ MEMaps maps, MEArgs<R> g) {
  using L = METile<HX, HT, R>;
  extern __shared__ unsigned char me_smem[];
  __shared__ __align__(8) unsigned long long bars[2 * kMeSlots];
  constexpr int T = 3 - A;
  const int lane = threadIdx.x, ty = threadIdx.y;
  const int x0 = -1 + 32 * (int)blockIdx.x, t0 = -1 + kMeY * (int)blockIdx.y;
  const int x = x0 + lane, t = t0 + ty;
  const int nT = A == 1 ? g.nz : g.ny, na = A == 1 ? g.ny : g.nz;
  const int SA = A == 1 ? g.sx : g.sxy, S2 = A == 1 ? g.sxy : g.sx;
  const int ia0 = -1 + g.chunk * (int)blockIdx.z, ia1 = min(ia0 + g.chunk - 1, na + 2);
  // the first point computed: the one below the chunk, whose fluxes the first
  // update reads, where it has any
  const int first = ia0 >= 1 ? ia0 - 1 : ia0;
  unsigned char* const buf = me_smem + ((128u - (smem_addr(me_smem) & 127u)) & 127u);
  TileRing<kMeSlots> ring;
  ring.full = smem_addr(bars);
  ring.empty = ring.full + 8 * kMeSlots;
  ring.base = smem_addr(buf);
  ring.sc = g.sc;
  auto issue = [&](int ia, int slot) {
    const uint32_t d = ring.base + slot * L::slot, bar = ring.full + 8 * slot;
    mbar_expect(bar, L::sent);
    const int e = x0 + 1, r = t0 + 2, far = ia + 4, near = ia + 2;  // elements count from -2; x0 - 1 is e
    auto load = [&](int off, const CUtensorMap* m, int row, int p) {
      tma_load_3d(d + off, m, e, A == 1 ? p : row, A == 1 ? row : p, bar);
    };
    load(0, &maps.va, r - 1, far);
    load(L::h, &maps.rho, r, far);
    load(L::oe, &maps.energy, r, far);
    load(L::oc, &maps.cv, r, near);
    if (HX) load(L::ox, &maps.vx, r - 1, near);
    if (HT) load(L::ot, &maps.vt, r - 1, near);
  };
  const bool boss = lane == 0 && ty == 0;
  if (boss) {
    ring.init(kMeY);
    for (int s = 0; s < kMeSlots && first + s <= ia1; ++s) issue(first + s, s);
  }
  const bool inside_t = x >= 0 && x <= g.nx + 1 && t >= 0 && t <= nT + 1;  // dm's transverse range
  const bool line0 = x >= 0 && x <= g.nx && t >= 0 && t <= nT;             // the energy flux's
  const bool line1 = line0 && x >= 1 && t >= 1;                            // the updates'
  const bool own = x <= g.nx + 2 && t <= nT + 2;
  const R dt = (R)g.sc[g.dt_slot];
  const R area = inside_t ? g.m[0](x) * g.m[T](t) : R(0);
  const A1<R> w = g.m[A];
  const R q4 = R(0.25);
  const int base = min(x, g.nx + 2) + min(t, nT + 2) * S2;
  auto at = [&](int ia) { return base + min(ia, na + 2) * SA; };
  // windows of the first point: rho and energy at -1..1, the face velocity
  // along A and db1 to 1
  R r0, r1, r2, e0, e1, e2, vd0, vd1, db0, dbp, vfm, vf, vfp;
  Tr2<R> tm{};
  {
    const R* __restrict__ va = g.v[A];
    auto vface = [&](int q) { return (va[q] + va[q - 1] + va[q - S2] + va[q - 1 - S2]) * q4; };
    vfm = vface(at(first) - SA);
    vf = vface(at(first));
    vfp = vface(at(first + 1));
    db0 = w(first) + (vf - vfm) * dt;
    dbp = w(min(first + 1, na + 2)) + (vfp - vf) * dt;
    // (at -1 it is not used: dm there is a ghost value)
    const R dbm = first > -1 ? w(first - 1) + (vfm - vface(at(first) - 2 * SA)) * dt : db0;
    r0 = g.rho[at(first - 1)];
    r1 = g.rho[at(first)];
    r2 = g.rho[at(first + 1)];
    e0 = g.energy[at(first - 1)];
    e1 = g.energy[at(first)];
    e2 = g.energy[at(first + 1)];
    vd0 = dv_of(R(0.5) * (dbm + db0));
    vd1 = dv_of(R(0.5) * (db0 + dbp));
    const int q = at(first) - SA;
    if (HX) tm.load_x(g.v[0] + q, S2);
    if (HT) tm.load_t(g.v[T] + q, S2);
  }
  R dm_prev = R(0), ef_prev = R(0);
  __syncthreads();  // the barriers are set up
  // this thread's elements of a tile (past the grid, a neighbour's: zeros would
  // send the exact builds' divisions down their slow path)
  const int lx = min(x, g.nx + 2) - x0, lt = min(t, nT + 2) - t0;
  const int ch = (lt + 1) * L::W + lx + 1, cc = lt * L::W + lx + 1;
  int slot = 0;
  uint32_t ph = 0;
  for (int ia = first; ia <= ia1; ++ia) {
    ring.wait_full(slot, ph);
    const unsigned char* const sl = buf + slot * L::slot;
    const R* const v = reinterpret_cast<const R*>(sl) + ch;
    const R vf2 = (v[0] + v[-1] + v[-L::W] + v[-L::W - 1]) * q4;
    const R r3 = reinterpret_cast<const R*>(sl + L::h)[cc], e3 = reinterpret_cast<const R*>(sl + L::oe)[cc];
    const R cvc = reinterpret_cast<const R*>(sl + L::oc)[cc];
    Tr2<R> tc{};
    if (HX) tc.load_x(reinterpret_cast<const R*>(sl + L::ox) + ch, L::W);
    if (HT) tc.load_t(reinterpret_cast<const R*>(sl + L::ot) + ch, L::W);
    ring.release(slot);
    // (past n + 2 the plane is zeros and what comes of it is not used)
    const R dbp2 = w(min(ia + 2, na + 2)) + (vf2 - vfp) * dt;
    const R vdc[3] = {vd0, vd1, dv_of(R(0.5) * (dbp + dbp2))};
    const R r[4] = {r0, r1, r2, r3}, e[4] = {e0, e1, e2, e3};
    const MEFace<R> face(vdc, db0, dbp, vf, dt, area);
    R dmc = R(0);
    if (inside_t) {
      bool none;
      const int s = me_source(ia, na, g.per, none);
      if (none) {
        dmc = R(0);
      } else if (s != ia) {
        dmc = me_mass_flux<A, R>(g, base + s * SA, s, 1, S2, SA, dt, area);
      } else {
        dmc = face.mass(r);
      }
    }
    R ef = R(0);
    if (line0 && ia >= 0 && ia <= na) ef = face.energy(e, r1, r2, dmc);
    if (ia >= ia0 && own) {
      const int c = at(ia);
      R dv[3] = {R(0), R(0), R(0)};
      if (HX) dv[0] = tc.template diff_x<A>(tm);
      if (HT) dv[T] = tc.template diff_t<A>(tm);
      dv[A] = vf - vfm;
      R c1, c2;
      me_volumes<A, HX, HT>(g, dv, x, A == 1 ? ia : t, A == 1 ? t : ia, dt, cvc, c1, c2);
      g.dm[c] = dmc;
      g.cv1[c] = c1;
      if (HX || HT) g.cv2[c] = c2;
      if (g.db1) {
        g.db1[c] = db0;
        g.dc1[c] = R(0.5) * (db0 + (ia < na + 2 ? dbp : db0));
      }
      R rn = r1, en = e1;
      if (line1 && ia >= 1 && ia <= na) {
        rn = qdiv(r1 * c1 + dm_prev - dmc, c2);
        en = qdiv(e1 * c1 * r1 + ef_prev - ef, c2 * rn);
      }
      g.rho_new[c] = rn;
      g.energy_new[c] = en;
    }
    dm_prev = dmc;
    ef_prev = ef;
    r0 = r1; r1 = r2; r2 = r3;
    e0 = e1; e1 = e2; e2 = e3;
    db0 = dbp;
    dbp = dbp2;
    vfm = vf;
    vf = vfp;
    vfp = vf2;
    vd0 = vd1;
    vd1 = vdc[2];
    tm = tc;
    // the slot of the last step but one is refilled once every warp has left it
    if (boss && ia > first && ia - 1 + kMeSlots <= ia1) {
      const int ps = slot == 0 ? kMeSlots - 1 : slot - 1;
      ring.wait(ring.empty + 8 * ps, slot == 0 ? ph ^ 1u : ph);
      if (!ring.dead) issue(ia - 1 + kMeSlots, ps);
    }
    if (++slot == kMeSlots) {
      slot = 0;
      ph ^= 1u;
    }
  }
}

// dm's ghost values of a periodic x sweep, at their source index, before the
// sweep reads them: in the sweep itself the two lanes that need them would
// hold up every step of their warps for a chain of loads (0.132 against
// 0.068 ms at 128^3, 0.50 against 0.36 ms at 256^3, FP64).
template <class R>
__global__ void __launch_bounds__(128) k_me_ghost_x(MEArgs<R> g) {
  const int q = (int)(blockIdx.x * blockDim.x + threadIdx.x);      // 4 ghosts a row
  const int iy = q >> 2, iz = (int)blockIdx.y;
  if (iy > g.ny + 1) return;
  const int k = q & 3, ix = k < 2 ? k - 1 : g.nx + k - 1;          // -1, 0, n+1, n+2
  const int s = k < 2 ? ix + g.nx : ix - g.nx;
  const int row = g.sx * iy + g.sxy * iz;
  const R dt = (R)g.sc[g.dt_slot];
  g.dm[ix + row] = me_mass_flux<0, R>(g, s + row, s, g.sx, g.sxy, 1, dt, g.m[1](iy) * g.m[2](iz));
}

// The x sweep.  The lanes of a warp hold consecutive x positions and take
// their stencil neighbours and the fluxes to their left by shuffles; a block
// of 32 x kMeY threads holds kMeY rows of y and walks a chunk of z, its planes
// in the same kind of ring, carrying the velocities of the plane below that
// the face velocities need.  HY, HZ as above.
template <bool HY, bool HZ, class R>
__global__ void __launch_bounds__(32 * kMeY, sizeof(R) == 8 ? 2 : 4)
    k_me_x(const __grid_constant__ MEMaps maps, MEArgs<R> g) {
  using L = METile<HY, HZ, R>;  // (x and t of the tile: y and z here)
  extern __shared__ unsigned char me_smem[];
  __shared__ __align__(8) unsigned long long bars[2 * kMeSlots];
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x, ty = threadIdx.y;
  const int x0 = -1 - kMeXFirst + kMeXOut * (int)blockIdx.x, y0 = -1 + kMeY * (int)blockIdx.y;
  const int ix = x0 + lane;                                        // lane kMeXFirst holds the first output
  const int iy = min(y0 + ty, g.ny + 2);
  const int iz0 = -1 + g.chunk * (int)blockIdx.z, iz1 = min(iz0 + g.chunk - 1, g.nz + 2);
  const int sx = g.sx, sxy = g.sxy, na = g.nx;
  const int xl = min(max(ix, -2), g.nx + 2);                       // in-box load position
  const int e0 = x0 + 2, ea = e0 & ~(kTmaAlign<R> - 1);            // element of x0, counted from x = -2
  unsigned char* const buf = me_smem + ((128u - (smem_addr(me_smem) & 127u)) & 127u);
  TileRing<kMeSlots> ring;
  ring.full = smem_addr(bars);
  ring.empty = ring.full + 8 * kMeSlots;
  ring.base = smem_addr(buf);
  ring.sc = g.sc;
  auto issue = [&](int iz, int slot) {
    const uint32_t d = ring.base + slot * L::slot, bar = ring.full + 8 * slot;
    mbar_expect(bar, L::sent);
    const int r = y0 + 2, p = iz + 2;
    tma_load_3d(d, &maps.va, ea, r - 1, p, bar);
    tma_load_3d(d + L::h, &maps.rho, ea, r, p, bar);
    tma_load_3d(d + L::oe, &maps.energy, ea, r, p, bar);
    tma_load_3d(d + L::oc, &maps.cv, ea, r, p, bar);
    if (HY) tma_load_3d(d + L::ox, &maps.vx, ea, r - 1, p, bar);
    if (HZ) tma_load_3d(d + L::ot, &maps.vt, ea, r - 1, p, bar);
  };
  const bool boss = lane == 0 && ty == 0;
  if (boss) {
    ring.init(kMeY);
    for (int s = 0; s < kMeSlots && iz0 + s <= iz1; ++s) issue(iz0 + s, s);
  }
  const bool in_y = iy >= 0 && iy <= g.ny + 1;
  const bool out = lane >= kMeXFirst && lane < kMeXFirst + kMeXOut && ix <= na + 2 && y0 + ty <= g.ny + 2;
  const R dt = (R)g.sc[g.dt_slot];
  const R wx = g.m[0](max(xl, -1)), wy = g.m[1](iy);
  const R q4 = R(0.25);
  const int base = xl + sx * iy;
  // one plane's values: v_x and v_y at y and y - 1, v_z's face
  struct Pl {
    R x0, xm, y0, ym, zf;
  };
  auto zface = [&](R z0, R zm) {  // q, -x, -y, -x-y
    return (z0 + __shfl_up_sync(all, z0, 1) + zm + __shfl_up_sync(all, zm, 1)) * q4;
  };
  Pl pm;
  {
    const int c = base + sxy * (iz0 - 1);
    pm.x0 = g.v[0][c];
    pm.xm = g.v[0][c - sx];
    pm.y0 = HY ? g.v[1][c] : R(0);
    pm.ym = HY ? g.v[1][c - sx] : R(0);
    pm.zf = HZ ? zface(g.v[2][c], g.v[2][c - sx]) : R(0);
  }
  __syncthreads();  // the barriers are set up
  // this thread's elements of a tile (outside the box the nearest inside it)
  const int lx = (e0 - ea) + xl - x0, ly = iy - y0;
  const int ch = (ly + 1) * L::W + lx, cc = ly * L::W + lx;
  int slot = 0;
  uint32_t ph = 0;
  for (int iz = iz0; iz <= iz1; ++iz) {
    const int c = base + sxy * iz;
    ring.wait_full(slot, ph);
    const unsigned char* const sl = buf + slot * L::slot;
    auto tile = [&](int off) { return reinterpret_cast<const R*>(sl + off); };
    Pl pc{tile(0)[ch], tile(0)[ch - L::W], R(0), R(0), R(0)};
    if (HY) {
      pc.y0 = tile(L::ox)[ch];
      pc.ym = tile(L::ox)[ch - L::W];
    }
    if (HZ) pc.zf = zface(tile(L::ot)[ch], tile(L::ot)[ch - L::W]);
    const R r0 = tile(L::h)[cc], en0 = tile(L::oe)[cc], cvc = tile(L::oc)[cc];
    ring.release(slot);
    const bool inside_t = in_y && iz >= 0 && iz <= g.nz + 1;
    const bool ghost = inside_t && (ix <= 0 || ix >= na + 1);
    R dmg = R(0);
    if (g.per && ghost && ix >= -1 && ix <= na + 2) dmg = g.dm[c];
    const bool line0 = iy >= 0 && iy <= g.ny && iz >= 0 && iz <= g.nz;
    const bool line1 = line0 && iy >= 1 && iz >= 1;
    const R area = inside_t ? wy * g.m[2](iz) : R(0);
    const R vf = (pc.x0 + pc.xm + pm.x0 + pm.xm) * q4;             // q, -y, -z, -y-z
    const R dva = vf - __shfl_up_sync(all, vf, 1);
    const R db = wx + dva * dt;
    const R dbp = __shfl_down_sync(all, db, 1);
    const R dc = R(0.5) * (db + (ix < na + 2 ? dbp : db));
    const R dvc = dv_of(dc);
    const R r[4] = {__shfl_up_sync(all, r0, 1), r0, __shfl_down_sync(all, r0, 1), __shfl_down_sync(all, r0, 2)};
    const R e[4] = {__shfl_up_sync(all, en0, 1), en0, __shfl_down_sync(all, en0, 1), __shfl_down_sync(all, en0, 2)};
    const R vdc[3] = {__shfl_up_sync(all, dvc, 1), dvc, __shfl_down_sync(all, dvc, 1)};
    const MEFace<R> face(vdc, db, dbp, vf, dt, area);
    // dm at ix; a ghost's comes from the array (periodic, loaded above), from
    // the real point beside it, or is zero (dm_x_bcs)
    R dmc = R(0);
    if (inside_t && lane >= 2 && lane <= 29 && ix >= 0 && ix <= na) dmc = face.mass(r);
    if (g.per) {
      if (ghost) dmc = dmg;
    } else {
      const R up = __shfl_up_sync(all, dmc, 1), down = __shfl_down_sync(all, dmc, 1);
      if (ix == -1) dmc = down;
      if (ix == na + 1) dmc = up;
    }
    R ef = R(0);
    if (line0 && ix >= 0 && ix <= na && lane >= 2 && lane <= 29) ef = face.energy(e, r0, r[2], dmc);
    const R dm_prev = __shfl_up_sync(all, dmc, 1), ef_prev = __shfl_up_sync(all, ef, 1);
    R dv[3] = {dva, R(0), R(0)};
    if (HY) {  // v_y faces: q, -x, -z, -x-z at y and y - 1
      const R y0x = __shfl_up_sync(all, pc.y0, 1), ymx = __shfl_up_sync(all, pc.ym, 1);
      const R y0xm = __shfl_up_sync(all, pm.y0, 1), ymxm = __shfl_up_sync(all, pm.ym, 1);
      dv[1] = (pc.y0 + y0x + pm.y0 + y0xm) * q4 - (pc.ym + ymx + pm.ym + ymxm) * q4;
    }
    if (HZ) dv[2] = pc.zf - pm.zf;
    if (out) {
      R c1, c2;
      me_volumes<0, HY, HZ>(g, dv, ix, iy, iz, dt, cvc, c1, c2);
      g.dm[c] = dmc;
      g.cv1[c] = c1;
      if (HY || HZ) g.cv2[c] = c2;
      if (g.db1) {
        g.db1[c] = db;
        g.dc1[c] = dc;
      }
      R rn = r0, e1 = en0;
      if (line1 && ix >= 1 && ix <= na) {
        rn = qdiv(r0 * c1 + dm_prev - dmc, c2);
        e1 = qdiv(en0 * c1 * r0 + ef_prev - ef, c2 * rn);
      }
      g.rho_new[c] = rn;
      g.energy_new[c] = e1;
    }
    pm = pc;
    // the last step's slot is refilled once every warp has left it
    if (boss && iz > iz0 && iz - 1 + kMeSlots <= iz1) {
      const int ps = slot == 0 ? kMeSlots - 1 : slot - 1;
      ring.wait(ring.empty + 8 * ps, slot == 0 ? ph ^ 1u : ph);
      if (!ring.dead) issue(iz - 1 + kMeSlots, ps);
    }
    if (++slot == kMeSlots) {
      slot = 0;
      ph ^= 1u;
    }
  }
}

template <int A, bool HX, bool HT, class R>
inline void me_launch(Run<R>& run, MEArgs<R>& g, int words) {
  using L = METile<HX, HT, R>;
  constexpr int T1 = A == 0 ? 1 : 0, T2 = A == 2 ? 1 : 2;
  MEMaps maps;
  const long long f = 2 + 2LL * run.sx + 2LL * run.sxy;
  const auto map = [&](CUtensorMap* m, const R* p, int rows) {
    make_map(run, m, p - f, L::W, A == 1 ? 1 : rows, A == 1 ? rows : 1);
  };
  map(&maps.va, g.v[A], kMeY + 1);
  map(&maps.vx, g.v[T1], kMeY + 1);
  map(&maps.vt, g.v[T2], kMeY + 1);
  map(&maps.rho, g.rho, kMeY);
  map(&maps.energy, g.energy, kMeY);
  map(&maps.cv, g.cv, kMeY);
  if (run.launch_error) return;
  const int rows = (A == 1 ? g.nz : g.ny) + 4, len = (A == 1 ? g.ny : g.nz) + 4;
  const int xout = A == 0 ? kMeXOut : 32;
  dim3 grd((g.nx + 4 + xout - 1) / xout, (rows + kMeY - 1) / kMeY, 1);
  const dim3 blk(32, kMeY, 1);
  const int k = run.prof_begin(A == 0 ? "remap_sweep_mass_energy_x" : "remap_sweep_mass_energy_march", 0, words,
                               (double)(g.nx + 4) * (g.ny + 4) * (g.nz + 4));
  if constexpr (A == 0) {
    if (g.per) {
      k_me_ghost_x<R><<<dim3((4 * (g.ny + 2) + 127) / 128, g.nz + 2), 128, 0, run.s>>>(g);
      ++run.launches;
    }
    g.chunk = march_chunk(len, grd.x * grd.y, 32, resident_blocks<k_me_x<HX, HT, R>>(32 * kMeY, L::smem));
    grd.z = (len + g.chunk - 1) / g.chunk;
    k_me_x<HX, HT, R><<<grd, blk, L::smem, run.s>>>(maps, g);
  } else {
    g.chunk = march_chunk(len, grd.x * grd.y, 32, resident_blocks<k_me_march<A, HX, HT, R>>(32 * kMeY, L::smem));
    grd.z = (len + g.chunk - 1) / g.chunk;
    k_me_march<A, HX, HT, R><<<grd, blk, L::smem, run.s>>>(maps, g);
  }
  run.prof_end(k);
  ++run.launches;
}

// Dynamic shared memory beyond the default 48 KiB, once per context.
template <class R>
inline cudaError_t me_attributes() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* k, size_t bytes) {
    const cudaError_t q = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e == cudaSuccess) e = q;
  };
  set(k_me_x<true, true, R>, METile<true, true, R>::smem);
  set(k_me_x<true, false, R>, METile<true, false, R>::smem);
  set(k_me_x<false, true, R>, METile<false, true, R>::smem);
  set(k_me_x<false, false, R>, METile<false, false, R>::smem);
  set(k_me_march<1, true, true, R>, METile<true, true, R>::smem);
  set(k_me_march<1, true, false, R>, METile<true, false, R>::smem);
  set(k_me_march<1, false, true, R>, METile<false, true, R>::smem);
  set(k_me_march<1, false, false, R>, METile<false, false, R>::smem);
  set(k_me_march<2, true, true, R>, METile<true, true, R>::smem);
  set(k_me_march<2, true, false, R>, METile<true, false, R>::smem);
  set(k_me_march<2, false, true, R>, METile<false, true, R>::smem);
  set(k_me_march<2, false, false, R>, METile<false, false, R>::smem);
  return e;
}

// One sweep's volumes, mass and energy along axis A.
template <int A, class R>
void mass_energy_sweep(Run<R>& run, MEArgs<R> g, int swept) {
  constexpr int T1 = A == 0 ? 1 : 0, T2 = A == 2 ? 1 : 2;
  // words: rho, energy, cv and the velocity components still to come read;
  // dm, rho, energy, cv1 and (but in the third sweep) cv2 written
  const int words = swept == 0 ? 11 : (swept == 1 ? 10 : 8);
  if (g.pass[T1] && g.pass[T2])
    me_launch<A, true, true>(run, g, words);
  else if (g.pass[T1])
    me_launch<A, true, false>(run, g, words);
  else if (g.pass[T2])
    me_launch<A, false, true>(run, g, words);
  else
    me_launch<A, false, false>(run, g, words);
}

LARE_END  // namespace lare
