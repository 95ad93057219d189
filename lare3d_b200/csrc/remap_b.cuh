// remap_b.cuh - the magnetic part of one directional remap sweep as one
// kernel: the geometry it needs (xremap.f90:57-115), both constrained-
// transport edge fluxes (:340-470) and the four flux-difference updates
// (:121-157), with the mirrors of yremap.f90 and zremap.f90, and B's
// conversion to flux form before a remap's first sweep (remap.f90:43-69)
// and back after its last (:101-127).
//
// The moved cell width db1 and centre distance dc1 follow from the face-
// averaged velocity along the sweep axis alone (db1(c) = db(a) + (vf(c) -
// vf(c - e_A)) dt, dc1(c) = (db1(c) + db1(c + e_A)) / 2), so they are formed
// on the way and neither they nor the two fluxes reach memory: the velocity
// component along the axis and B are read and B is written, 7 words a point
// where separate geometry, flux and update kernels moved 23 (8 + 7 + 8).
// The new B goes to a second set of arrays: neighbouring tiles still read
// the old one.
//
// Every value is the reference's expression over the same operands in the
// same order, so the exact build stays bit for bit.
//
// At 256^3 a sweep takes 0.29 ms (y, z) and 0.30 ms (x) in FP64 and 0.20 to 0.24
// ms in FP32, against 0.70 and 0.44 ms for the three kernels; the floor is its 7
// words, 0.15 ms in FP64.  Bound by instruction issue (57 to 61 % of slots with
// the 16 warps an SM that the windows' registers allow; about 80 % in FP32) and
// by the halo, 15 (y, z) to 26 % (x) of the tiles' lanes.  Measured and not kept: planes prefetched into registers
// instead of the ring (0.50 ms: too little in flight for the DRAM latency), one
// component a thread on 512-thread blocks (0.37 ms: the barrier and the
// geometry formed twice), tiles of 4, 12 and 16 rows (0.31, 0.34, 0.31 ms).
//
// MODE 1, a remap's first sweep: B is read as stored and put in flux form.
// MODE 2, its last: the updated B is put back.  MODE 0 between.  Every point
// of the arrays' box -2..n+2 is written; the update covers 0..n+1.
#pragma once

LARE_BEGIN

constexpr int kBsY = 8;            // rows of a tile; its first row only hands on its fluxes
constexpr int kBsOut = 31;         // y/z sweeps: cells a warp updates (lane 0 only hands on its flux)
constexpr int kBsXFirst = 3;       // x sweep: first lane that updates a cell
constexpr int kBsXOut = 27;        // x sweep: lanes that do (stencil -2..+2 and the flux below by shuffles)

template <class R>
struct BSArgs {
  // arrays from their first element (elem_at)
  const R* va;                     // velocity component along the sweep axis (v1 of the reference)
  const R* in[3];                  // B along x, y, z
  R* out[3];
  A1<R> m[3], r[3];                // cell widths and their reciprocals
  double* sc;
  int dt_slot, nx, ny, nz, sx, sxy;
  int chunk;                       // points marched per block
};

// One transported component's four-point window along the sweep axis:
// B / dbv and dbv (in the carried divisor form) at c, c + e_A, c + 2 e_A, and
// what the limiter takes of the faces below, at and above c: B / dbv at
// c - e_A and dc1, for the reference's expressions, or (kRegroup) each face's
// difference and its slope |d| / dc1, formed once when the face enters the
// window instead of once for each of the three fluxes that read it.
template <class R>
struct BWin {
  R q0, qp, qp2, v0, vp, vp2;
  R dm, d0, dp, sm, s0, sp;  // kRegroup
  R qm, dcm, dc0, dcp;       // else
  // the points c - e_A (or c where the stencil is clamped) and c, and dc1 below c
  __device__ __forceinline__ void start(R qm_, R q0_, R v0_, R dcm_) {
    q0 = q0_;
    v0 = v0_;
    if constexpr (kRegroup<R>) {
      dm = q0_ - qm_;
      sm = fabs(dm) * fast_rcp(dcm_);
    } else {
      qm = qm_;
      dcm = dv_of(dcm_);
    }
  }
  // the point c + e_A, and dc1 at c
  __device__ __forceinline__ void next(R q, R v, R dc) {
    qp = q;
    vp = v;
    if constexpr (kRegroup<R>) {
      d0 = q - q0;
      s0 = fabs(d0) * fast_rcp(dc);
    } else {
      dc0 = dv_of(dc);
    }
  }
  // the point c + 2 e_A, and dc1 at c + e_A (in the carried divisor form)
  __device__ __forceinline__ void top(R q, R v, R dc) {
    qp2 = q;
    vp2 = v;
    if constexpr (kRegroup<R>) {
      dp = q - qp;
      sp = fabs(dp) * dc;
    } else {
      dcp = dc;
    }
  }
  __device__ __forceinline__ void shift() {
    if constexpr (kRegroup<R>) {
      dm = d0;
      d0 = dp;
      sm = s0;
      s0 = sp;
    } else {
      qm = q0;
      dcm = dc0;
      dc0 = dcp;
    }
    q0 = qp;
    qp = qp2;
    v0 = vp;
    vp = vp2;
  }
  // the flux at c: db1 at c and c + e_A
  __device__ __forceinline__ R flux(R v_advect, R db0, R dbp, R dt) const {
    if constexpr (kRegroup<R>) {
      return van_leer(v_advect, v_advect * dt, q0, qp, dm, d0, dp, sm, s0, sp, db0, dbp, v0, vp);
    } else {
      const LimOut<R> L = limiter_dv<R>(v_advect, qm, q0, qp, qp2, dc0, dcm, dcp, db0, dbp, v0, vp, dt, true);
      return (L.fu + L.Di * (R(1) - L.phi)) * v_advect * dt;
    }
  }
};

// B component J at (ix, iy, iz) to and from flux form, its two face widths
// given (or with their reciprocals), w1 along the lower axis.  The reference
// converts where both coordinates are at least -1.
template <class R>
__device__ __forceinline__ R bs_form(R b, R w1, R w2, bool ok) {
  return ok ? b * w1 * w2 : b;
}
template <class R>
__device__ __forceinline__ R bs_unform(R b, R w1, R r1, R w2, R r2, bool ok) {
  return ok ? div_rcp(div_rcp(b, w1, r1), w2, r2) : b;
}

// The y and z sweeps (A = 1, 2).  A block of 32 x kBsY threads owns a tile
// of columns across the sweep axis, x along the lanes and the third axis
// along the rows, and walks a chunk of the axis with the four-point windows
// of both components in registers.  The planes of the velocity component
// along the axis (with a one-point halo) and of B arrive in a ring of
// kBsStages shared-memory slots by TMA, three steps before they enter the
// windows, and stay until the point they belong to is updated.  db1 at the
// neighbouring columns (x + 1 and t + 1, for dbv) is formed from the face
// velocity there; the first flux of the lane below arrives by a shuffle, the
// second flux of the row below through shared memory.  One barrier a step
// orders both that exchange and the reuse of slots.
constexpr int kBsStages = 6;
template <class R>
struct BSTile {
  // row length: 34 elements from the aligned start, rounded up to 16 bytes
  static constexpr int W = sizeof(R) == 8 ? 36 : 40;
  static constexpr int va = (W * (kBsY + 2) * (int)sizeof(R) + 127) / 128 * 128;  // bytes
  static constexpr int b = (W * kBsY * (int)sizeof(R) + 127) / 128 * 128;
  static constexpr int slot = va + 3 * b;
  static constexpr unsigned sent = W * (4 * kBsY + 2) * sizeof(R);                // bytes a plane brings
  static constexpr size_t smem = 128 + (size_t)kBsStages * slot;
};
struct BSMaps {
  CUtensorMap va, b[3];  // b: components 0, T, A (x sweep: 0, 1, 2)
};

template <int A, int MODE, class R>
__global__ void __launch_bounds__(32 * kBsY, sizeof(R) == 8 ? 2 : 3) k_bsweep_march(const __grid_constant__ BSMaps maps,
                                                                              BSArgs<R> g) {
  using L = BSTile<R>;
  extern __shared__ unsigned char bs_smem[];
  __shared__ R f2s[2][kBsY][32];
  __shared__ __align__(8) unsigned long long bars[kBsStages];
  constexpr int T = 3 - A;                                   // the third axis
  const int lane = threadIdx.x, ty = threadIdx.y;
  const bool boss = lane == 0 && ty == 0;
  const int nT = A == 1 ? g.nz : g.ny, nA = A == 1 ? g.ny : g.nz;
  const int SA = A == 1 ? g.sx : g.sxy, ST = A == 1 ? g.sxy : g.sx;
  const int x0 = -3 + kBsOut * (int)blockIdx.x, t0 = -3 + (kBsY - 1) * (int)blockIdx.y;
  const int x = x0 + lane, t = t0 + ty;
  const bool wr = lane >= 1 && ty >= 1 && x <= g.nx + 2 && t <= nT + 2;
  const int xo = min(max(x, -2), g.nx + 2), to = min(max(t, -2), nT + 2);
  const int o0 = -2 + g.chunk * (int)blockIdx.z, o1 = min(o0 + g.chunk - 1, nA + 2);
  const int fs = max(o0 - 1, -1), fe = min(o1, nA + 1);
  // the ring: planes p0..pe in order, from the aligned element below x0 - 1
  const int p0 = max(fs - 1, -1) - 1, pe = min(fe + 2, nA + 2);
  const int e0 = x0 + 1, ea = e0 & ~(kTmaAlign<R> - 1);      // element of x0 - 1, counted from x = -2
  unsigned char* const ring = bs_smem + ((128u - (smem_addr(bs_smem) & 127u)) & 127u);
  const uint32_t ring_s = smem_addr(ring), bar_s = smem_addr(bars);
  auto issue = [&](int p, int slot) {
    const uint32_t d = ring_s + slot * L::slot, bar = bar_s + 8 * slot;
    mbar_expect(bar, L::sent);
    const int r = t0 + 2, q = p + 2;
    tma_load_3d(d, &maps.va, ea, A == 1 ? q : r - 1, A == 1 ? r - 1 : q, bar);
#pragma unroll
    for (int m = 0; m < 3; ++m)
      tma_load_3d(d + L::va + m * L::b, &maps.b[m], ea, A == 1 ? q : r, A == 1 ? r : q, bar);
  };
  if (boss) {
    for (int s = 0; s < kBsStages; ++s) mbar_init(bar_s + 8 * s, 1);
    mbar_init_fence();
    for (int s = 0; s < kBsStages && p0 + s <= pe; ++s) issue(p0 + s, s);
  }
  int next = p0 + kBsStages;                                 // the next plane to ask for
  const R dt = (R)g.sc[g.dt_slot];
  const R* __restrict__ mA = g.m[A].p;
  const R* __restrict__ rA = g.r[A].p;
  // face widths of the column (fluxes are used at -1..n+1 only)
  const bool okX = xo >= -1, okT = to >= -1;
  const R oX = g.m[0](xo), oT = g.m[T](to);
  const R orX = MODE == 2 ? g.r[0](xo) : R(0), orT = MODE == 2 ? g.r[T](to) : R(0);
  const unsigned uA = (unsigned)SA * sizeof(R), co = elem_off<R>(xo, 1, to, ST);
  // component 0 has its faces across y and z, component T across x and A
  auto form1 = [&](R b, R wa, R wt, bool ok) { return A == 1 ? bs_form(b, wa, wt, ok) : bs_form(b, wt, wa, ok); };
  auto form2 = [&](R b, R wa, R wx, bool ok) { return bs_form(b, wx, wa, ok); };
  const bool in_xt = x >= 0 && x <= g.nx + 1 && t >= 0 && t <= nT + 1;  // the update's columns
  // second flux into the component along A (yremap.f90:142-158)
  const bool r2x = A != 1 || (x >= 1 && x <= g.nx && t >= 1 && t <= g.nz);
  auto emit = [&](int ia, R b1, R bA, R b2) {
    if constexpr (MODE == 2) {
      const R w = mA[max(ia, -1)], r = rA[max(ia, -1)];
      const bool oka = ia >= -1;
      b1 = A == 1 ? bs_unform(b1, w, r, oT, orT, oka && okT) : bs_unform(b1, oT, orT, w, r, oka && okT);
      b2 = bs_unform(b2, oX, orX, w, r, oka && okX);
      bA = bs_unform(bA, oX, orX, oT, orT, okX && okT);
    }
    const unsigned c = co + uA * (unsigned)(ia + 2);
    elem_ref(g.out[0], c) = b1;
    elem_ref(g.out[T], c) = b2;
    elem_ref(g.out[A], c) = bA;
  };
  // the planes -2 and n+2 along A are outside every update: B as it is
  auto carry = [&](int ia) {
    const unsigned c = co + uA * (unsigned)(ia + 2);
    R b1 = elem_at(g.in[0], c), bA = elem_at(g.in[A], c), b2 = elem_at(g.in[T], c);
    if constexpr (MODE == 1) {
      const R w = mA[max(ia, -1)];
      b1 = form1(b1, w, oT, ia >= -1 && okT);
      b2 = form2(b2, w, oX, ia >= -1 && okX);
      bA = bs_form(bA, oX, oT, okX && okT);
    }
    emit(ia, b1, bA, b2);
  };
  if (wr && o0 == -2) carry(-2);
  if (wr && o1 == nA + 2) carry(nA + 2);
  // this thread's elements of a slot: of B for the update, and of the column
  // whose fluxes it forms (outside their range -1..n+1 the nearest one inside:
  // the fluxes are not used, and the zeros there would send the exact builds'
  // divisions down their slow path)
  const int lx = min(max(x, -1), g.nx + 1) - x0, lt = min(max(t, -1), nT + 1) - t0;
  const int cb = ty * L::W + (e0 - ea) + lane + 1;
  const int cv_ = (lt + 1) * L::W + (e0 - ea) + lx + 1, cbf = lt * L::W + (e0 - ea) + lx + 1;
  const R fX = g.m[0](x0 + lx), fT = g.m[T](t0 + lt);
  const R q4 = R(0.25);
  R vo, vx, vt;  // face velocity along A at the column, at x + 1 and at t + 1, last plane
  // one plane: db1 there, the two quotients and their divisors
  struct Pt {
    R db, q1, v1, q2, v2;
  };
  auto faces = [&](const R* v, R& o, R& ox, R& ot) {
    const R v00 = v[0], vm0 = v[-1], vp0 = v[1], v0m = v[-L::W], vmm = v[-L::W - 1], vpm = v[-L::W + 1];
    const R v0p = v[L::W], vmp = v[L::W - 1];
    o = (v00 + vm0 + v0m + vmm) * q4;
    ox = (vp0 + v00 + vpm + v0m) * q4;
    ot = (v0p + vmp + v00 + vm0) * q4;
  };
  auto plane = [&](int slot, int ia) {
    const R* const v = reinterpret_cast<const R*>(ring + slot * L::slot) + cv_;
    const R* const b = reinterpret_cast<const R*>(ring + slot * L::slot + L::va) + cbf;
    Pt p;
    R no, nx_, nt, b1 = b[0], b2 = b[L::b / (int)sizeof(R)];
    faces(v, no, nx_, nt);
    const R w = mA[ia];
    if constexpr (MODE == 1) {
      b1 = form1(b1, w, fT, true);
      b2 = form2(b2, w, fX, true);
    }
    p.db = w + (no - vo) * dt;
    const R dbx = w + (nx_ - vx) * dt, dbt = w + (nt - vt) * dt;
    vo = no;
    vx = nx_;
    vt = nt;
    p.v1 = dv_of((p.db + dbx) * R(0.5));
    p.q1 = dv_div(b1, p.v1);
    p.v2 = dv_of((p.db + dbt) * R(0.5));
    p.q2 = dv_div(b2, p.v2);
    return p;
  };
  BWin<R> w1, w2;
  R db0, dbp;
  int dead = 0;
  auto await = [&](int slot, uint32_t parity) { tile_wait(bar_s + 8 * slot, parity, dead, g.sc); };
  __syncthreads();  // the barriers are set up
  {
    // windows of the first flux; the stencil is clamped as MAX(ia-1, -1)
    const int pm = p0 + 1;
    await(0, 0);
    faces(reinterpret_cast<const R*>(ring) + cv_, vo, vx, vt);
    await(1, 0);
    const Pt m = plane(1, pm);
    Pt c = m;
    if (pm < fs) {
      await(2, 0);
      c = plane(2, fs);
    }
    await(fs + 1 - p0, 0);
    const Pt p = plane(fs + 1 - p0, fs + 1);
    db0 = c.db;
    dbp = p.db;
    const R dc0 = R(0.5) * (db0 + dbp), dcm = pm < fs ? R(0.5) * (m.db + db0) : dc0;
    w1.start(m.q1, c.q1, c.v1, dcm);
    w2.start(m.q2, c.q2, c.v2, dcm);
    w1.next(p.q1, p.v1, dc0);
    w2.next(p.q2, p.v2, dc0);
  }
  R f1a = R(0), f2a = R(0);
  int s0 = fs - p0, s2 = s0 + 2;  // slots of planes ia and ia + 2 (s2 <= 4 < kBsStages)
  uint32_t ph = 0;                // parity of plane ia + 2's slot
#pragma unroll 2
  for (int ia = fs; ia <= fe; ++ia) {
    // the point c + 2 e_A enters; MIN(ia+2, n+2): at the end it is c + e_A
    R dbp2 = dbp;
    if (ia + 2 <= nA + 2) {
      await(s2, ph);
      const Pt p = plane(s2, ia + 2);
      dbp2 = p.db;
      const R dc = dv_of(R(0.5) * (dbp + dbp2));
      w1.top(p.q1, p.v1, dc);
      w2.top(p.q2, p.v2, dc);
    } else {
      const R dc = dv_of(dbp);
      w1.top(w1.qp, w1.vp, dc);
      w2.top(w2.qp, w2.vp, dc);
    }
    const R* const v = reinterpret_cast<const R*>(ring + s0 * L::slot) + cv_;
    const R* const b = reinterpret_cast<const R*>(ring + s0 * L::slot + L::va) + cb;
    const R f1 = w1.flux((v[0] + v[-L::W]) * R(0.5), db0, dbp, dt);
    const R f2 = w2.flux((v[0] + v[-1]) * R(0.5), db0, dbp, dt);
    f2s[ia & 1][ty][lane] = f2;
    const R f1b = __shfl_up_sync(0xffffffffu, f1, 1);
    __syncthreads();
    // every thread is past the last step: the slots of the planes below ia are free
    if (boss && !dead)
      for (; next <= pe && next < ia + kBsStages; ++next) issue(next, (next - p0) % kBsStages);
    if (wr && ia >= o0) {
      R b1 = b[0], b2 = b[L::b / (int)sizeof(R)], bA = b[2 * L::b / (int)sizeof(R)];
      if constexpr (MODE == 1) {
        const R w = mA[ia];
        b1 = form1(b1, w, oT, okT);
        b2 = form2(b2, w, oX, okX);
        bA = bs_form(bA, oX, oT, okX && okT);
      }
      if (in_xt && ia >= 0) {
        const R f2b = f2s[ia & 1][ty - 1][lane];
        b1 = b1 - f1 + f1a;
        bA = bA + f1 - f1b;
        b2 = b2 - f2 + f2a;
        if (A != 1 || (r2x && ia <= nA)) bA = bA + f2 - f2b;
      }
      emit(ia, b1, bA, b2);
    }
    f1a = f1;
    f2a = f2;
    w1.shift();
    w2.shift();
    db0 = dbp;
    dbp = dbp2;
    s0 = s0 + 1 == kBsStages ? 0 : s0 + 1;
    if (++s2 == kBsStages) {
      s2 = 0;
      ph ^= 1u;
    }
  }
}

// The x sweep.  The lanes of a warp hold consecutive x positions and take
// their stencil neighbours by shuffles; a block of 32 x kBsY threads holds
// kBsY rows of y and walks a chunk of z, its planes in the same ring: the
// first flux of the row below comes through shared memory, the second flux of
// the plane below and db1 of the plane above (for the second dbv) stay in
// registers.
template <int MODE, class R>
__global__ void __launch_bounds__(32 * kBsY, sizeof(R) == 8 ? 2 : 4) k_bsweep_x(const __grid_constant__ BSMaps maps, BSArgs<R> g) {
  using L = BSTile<R>;
  extern __shared__ unsigned char bs_smem[];
  __shared__ R f1s[2][kBsY][32];
  __shared__ __align__(8) unsigned long long bars[kBsStages];
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x, ty = threadIdx.y;
  const bool boss = lane == 0 && ty == 0;
  const int x0 = -2 - kBsXFirst + kBsXOut * (int)blockIdx.x, y0 = -3 + (kBsY - 1) * (int)blockIdx.y;
  const int x = x0 + lane, y = y0 + ty;
  const int xf = min(max(x, -2), g.nx + 2), yo = min(max(y, -2), g.ny + 2);
  const bool wr = lane >= kBsXFirst && lane < kBsXFirst + kBsXOut && ty >= 1 && x <= g.nx + 2 && y <= g.ny + 2;
  const int o0 = -2 + g.chunk * (int)blockIdx.z, o1 = min(o0 + g.chunk - 1, g.nz + 2);
  const int fs = max(o0 - 1, -1), fe = min(o1, g.nz + 1);
  // the ring: planes p0..pe in order, from the aligned element below x0
  const int p0 = fs - 1, pe = fe + 1;
  const int e0 = x0 + 2, ea = e0 & ~(kTmaAlign<R> - 1);      // element of x0, counted from x = -2
  unsigned char* const ring = bs_smem + ((128u - (smem_addr(bs_smem) & 127u)) & 127u);
  const uint32_t ring_s = smem_addr(ring), bar_s = smem_addr(bars);
  auto issue = [&](int p, int slot) {
    const uint32_t d = ring_s + slot * L::slot, bar = bar_s + 8 * slot;
    mbar_expect(bar, L::sent);
    tma_load_3d(d, &maps.va, ea, y0 + 1, p + 2, bar);
#pragma unroll
    for (int m = 0; m < 3; ++m) tma_load_3d(d + L::va + m * L::b, &maps.b[m], ea, y0 + 2, p + 2, bar);
  };
  if (boss) {
    for (int s = 0; s < kBsStages; ++s) mbar_init(bar_s + 8 * s, 1);
    mbar_init_fence();
    for (int s = 0; s < kBsStages && p0 + s <= pe; ++s) issue(p0 + s, s);
  }
  int next = p0 + kBsStages;                                 // the next plane to ask for
  const R dt = (R)g.sc[g.dt_slot];
  const R mx = g.m[0](max(xf, -1)), oY = g.m[1](yo);
  const R rx = MODE == 2 ? g.r[0](max(xf, -1)) : R(0), rY = MODE == 2 ? g.r[1](yo) : R(0);
  const bool okX = xf >= -1, okY = yo >= -1;
  const unsigned uz = (unsigned)g.sxy * sizeof(R), co = elem_off<R>(xf, 1, yo, g.sx);
  const bool in_xy = x >= 0 && x <= g.nx + 1 && y >= 0 && y <= g.ny + 1;
  // second flux (xremap.f90:141-157)
  const bool r2a = x >= 1 && x <= g.nx && y >= 1 && y <= g.ny, r2b = x <= g.nx;
  const bool left = x > -1, right = x + 2 <= g.nx + 2;  // cm = MAX(ix-1, -1), cp2 = MIN(ix+2, n+2)
  auto emit = [&](int iz, R bx, R by, R bz) {
    if constexpr (MODE == 2) {
      const R w = g.m[2](max(iz, -1)), r = g.r[2](max(iz, -1));
      bx = bs_unform(bx, oY, rY, w, r, okY && iz >= -1);
      by = bs_unform(by, mx, rx, w, r, okX && iz >= -1);
      bz = bs_unform(bz, mx, rx, oY, rY, okX && okY);
    }
    const unsigned c = co + uz * (unsigned)(iz + 2);
    elem_ref(g.out[0], c) = bx;
    elem_ref(g.out[1], c) = by;
    elem_ref(g.out[2], c) = bz;
  };
  // B at (x, y, iz) in flux form, as the update reads it
  auto formed = [&](int iz, R& bx, R& by, R& bz) {
    if constexpr (MODE == 1) {
      const R w = g.m[2](max(iz, -1));
      bx = bs_form(bx, oY, w, okY && iz >= -1);
      by = bs_form(by, mx, w, okX && iz >= -1);
      bz = bs_form(bz, mx, oY, okX && okY);
    }
  };
  // the planes -2 and n+2 are outside every update: B as it is
  auto carry = [&](int iz) {
    const unsigned c = co + uz * (unsigned)(iz + 2);
    R bx = elem_at(g.in[0], c), by = elem_at(g.in[1], c), bz = elem_at(g.in[2], c);
    formed(iz, bx, by, bz);
    emit(iz, bx, by, bz);
  };
  if (wr && o0 == -2) carry(-2);
  if (wr && o1 == g.nz + 2) carry(g.nz + 2);
  // this thread's elements of a slot: of B for the update, and of the row whose
  // fluxes it forms (outside the box the nearest inside it, as above)
  const int lx = xf - x0, ly = min(max(y, -1), g.ny + 1) - y0;
  const int cb = ty * L::W + (e0 - ea) + lane;
  const int cv_ = (ly + 1) * L::W + (e0 - ea) + lx, cbf = ly * L::W + (e0 - ea) + lx;
  const R fY = g.m[1](y0 + ly);
  const R q4 = R(0.25);
  // v at rows y-1, y, y+1 of one plane
  struct Col {
    R m, c, p;
  };
  auto load_v = [&](int slot) {
    const R* const v = reinterpret_cast<const R*>(ring + slot * L::slot) + cv_;
    return Col{v[-L::W], v[0], v[L::W]};
  };
  // db1 from the face velocity of this lane's x and the one below
  auto width = [&](R vf) { return mx + (vf - __shfl_up_sync(all, vf, 1)) * dt; };
  auto face = [&](R a, R b, R c, R d) { return (a + b + c + d) * q4; };
  int dead = 0;
  auto await = [&](int slot, uint32_t parity) { tile_wait(bar_s + 8 * slot, parity, dead, g.sc); };
  __syncthreads();  // the barriers are set up
  await(0, 0);
  await(1, 0);
  Col vm = load_v(0), v0 = load_v(1);
  R db = width(face(v0.c, v0.m, vm.c, vm.m));  // db1 at (x, y, fs)
  R f2a = R(0);
  int s0 = 1, s1 = 2;  // slots of planes iz and iz + 1
  uint32_t ph = 0;     // parity of plane iz + 1's slot
#pragma unroll 2
  for (int iz = fs; iz <= fe; ++iz) {
    await(s1, ph);
    const Col vp = load_v(s1);
    const R* const bf = reinterpret_cast<const R*>(ring + s0 * L::slot + L::va) + cbf;
    R qy = bf[L::b / (int)sizeof(R)], qz = bf[2 * L::b / (int)sizeof(R)];
    if constexpr (MODE == 1) {
      qy = bs_form(qy, mx, g.m[2](iz), true);
      qz = bs_form(qz, mx, fY, true);
    }
    const R dby = width(face(v0.p, v0.c, vm.p, vm.c));  // at (x, y + 1, z)
    const R dbz = width(face(vp.c, vp.m, v0.c, v0.m));  // at (x, y, z + 1)
    const R d1 = dv_of((db + dby) * R(0.5)), d2 = dv_of((db + dbz) * R(0.5));
    const R q1 = dv_div(qy, d1), q2 = dv_div(qz, d2);
    const R dbp = __shfl_down_sync(all, db, 1);
    const R dc = dv_of(x < g.nx + 2 ? R(0.5) * (db + dbp) : db);
    R dcm = __shfl_up_sync(all, dc, 1);
    const R dcp = __shfl_down_sync(all, dc, 1);
    dcm = left ? dcm : dc;
    auto flux = [&](R v, R q, R d) {
      R qm = __shfl_up_sync(all, q, 1), qp2 = __shfl_down_sync(all, q, 2);
      const R qp = __shfl_down_sync(all, q, 1), dd = __shfl_down_sync(all, d, 1);
      qm = left ? qm : q;
      qp2 = right ? qp2 : qp;
      if constexpr (kRegroup<R>) {
        const R em = q - qm, e0_ = qp - q, ep = qp2 - qp;
        return van_leer(v, v * dt, q, qp, em, e0_, ep, R(fabs(em) * dcm), R(fabs(e0_) * dc), R(fabs(ep) * dcp), db,
                        dbp, d, dd);
      } else {
        const LimOut<R> M = limiter_dv<R>(v, qm, q, qp, qp2, dc, dcm, dcp, db, dbp, d, dd, dt, true);
        return (M.fu + M.Di * (R(1) - M.phi)) * v * dt;
      }
    };
    const R f1 = flux((v0.c + vm.c) * R(0.5), q1, d1);
    f1s[iz & 1][ty][lane] = f1;
    const R f2 = flux((v0.c + v0.m) * R(0.5), q2, d2);
    const R f1l = __shfl_up_sync(all, f1, 1), f2l = __shfl_up_sync(all, f2, 1);
    __syncthreads();
    // every thread is past the last step: the slots of the planes below iz are free
    if (boss && !dead)
      for (; next <= pe && next < iz + kBsStages; ++next) issue(next, (next - p0) % kBsStages);
    if (wr && iz >= o0) {
      const R* const b = reinterpret_cast<const R*>(ring + s0 * L::slot + L::va) + cb;
      R bx = b[0], by = b[L::b / (int)sizeof(R)], bz = b[2 * L::b / (int)sizeof(R)];
      formed(iz, bx, by, bz);
      if (in_xy && iz >= 0) {
        const R f1b = f1s[iz & 1][ty - 1][lane];
        by = by - f1 + f1l;
        bx = bx + f1 - f1b;
        if (r2a && iz <= g.nz) bz = bz - f2 + f2l;
        if (r2b) bx = bx + f2 - f2a;
      }
      emit(iz, bx, by, bz);
    }
    f2a = f2;
    db = dbz;
    vm = v0;
    v0 = vp;
    s0 = s1;
    if (++s1 == kBsStages) {
      s1 = 0;
      ph ^= 1u;
    }
  }
}

template <int A, int MODE, class R>
inline void bs_launch(const dim3& grd, cudaStream_t s, const BSMaps& maps, const BSArgs<R>& g) {
  const dim3 blk(32, kBsY, 1);
  if constexpr (A == 0) {
    k_bsweep_x<MODE, R><<<grd, blk, BSTile<R>::smem, s>>>(maps, g);
  } else {
    k_bsweep_march<A, MODE, R><<<grd, blk, BSTile<R>::smem, s>>>(maps, g);
  }
}

// Dynamic shared memory beyond the default 48 KiB, once per context.
template <class R>
inline cudaError_t bs_attributes() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* k) {
    const cudaError_t q = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)BSTile<R>::smem);
    if (e == cudaSuccess) e = q;
  };
  set(k_bsweep_x<0, R>);
  set(k_bsweep_x<1, R>);
  set(k_bsweep_x<2, R>);
  set(k_bsweep_march<1, 0, R>);
  set(k_bsweep_march<1, 1, R>);
  set(k_bsweep_march<1, 2, R>);
  set(k_bsweep_march<2, 0, R>);
  set(k_bsweep_march<2, 1, R>);
  set(k_bsweep_march<2, 2, R>);
  return e;
}

template <int A, class R>
inline int bs_resident() {
  if constexpr (A == 0)
    return resident_blocks<k_bsweep_x<0, R>>(32 * kBsY, BSTile<R>::smem);
  else
    return resident_blocks<k_bsweep_march<A, 0, R>>(32 * kBsY, BSTile<R>::smem);
}

// One sweep's B along axis A: reads the set `in`, writes the set `out`.
template <int A, class R>
void bsweep(Run<R>& run, R* const va, R* const (&in)[3], R* const (&out)[3], int dt_slot, int bmode) {
  BSArgs<R> g;
  const long long first = 2 + 2LL * run.sx + 2LL * run.sxy;
  g.va = va - first;
  for (int d = 0; d < 3; ++d) {
    g.in[d] = in[d] - first;
    g.out[d] = out[d] - first;
    g.r[d] = run.a.rdb[d];
  }
  g.m[0] = run.a.dxb;
  g.m[1] = run.a.dyb;
  g.m[2] = run.a.dzb;
  g.sc = run.sc;
  g.dt_slot = dt_slot;
  g.nx = run.n[0];
  g.ny = run.n[1];
  g.nz = run.n[2];
  g.sx = run.sx;
  g.sxy = run.sxy;
  BSMaps maps;
  const auto map = [&](CUtensorMap* m, const R* first, int rows) {
    make_map(run, m, first, BSTile<R>::W, A == 1 ? 1 : rows, A == 1 ? rows : 1);
  };
  map(&maps.va, g.va, kBsY + 2);
  map(&maps.b[0], g.in[0], kBsY);
  map(&maps.b[1], g.in[A == 0 ? 1 : 3 - A], kBsY);
  map(&maps.b[2], g.in[A == 0 ? 2 : A], kBsY);
  if (run.launch_error) return;
  const int nt = (A == 1 ? g.nz : g.ny) + 5;                   // rows: y, or z for the y sweep
  const int nm = (A == 1 ? g.ny : g.nz) + 5;                   // marched axis
  const int xout = A == 0 ? kBsXOut : kBsOut;
  dim3 grd((g.nx + 5 + xout - 1) / xout, (nt + kBsY - 2) / (kBsY - 1), 1);
  g.chunk = march_chunk(nm, grd.x * grd.y, 64, bs_resident<A, R>());
  grd.z = (nm + g.chunk - 1) / g.chunk;
  const double pts = (double)(g.nx + 5) * (g.ny + 5) * (g.nz + 5);
  // words: va and B (3) read, B (3) written.  The sweep that finishes a
  // remap's B (and puts it back from flux form) is a site of its own.
  const char* site = bmode == 2 ? "remap_sweep_bupd" : (A == 0 ? "remap_sweep_bflux_x" : "remap_sweep_bflux_march");
  const int k = run.prof_begin(site, 0, 7, pts);
  if (bmode == 1)
    bs_launch<A, 1, R>(grd, run.s, maps, g);
  else if (bmode == 2)
    bs_launch<A, 2, R>(grd, run.s, maps, g);
  else
    bs_launch<A, 0, R>(grd, run.s, maps, g);
  run.prof_end(k);
  ++run.launches;
}

LARE_END  // namespace lare
