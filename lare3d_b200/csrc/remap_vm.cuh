// remap_vm.cuh - vertex averages fused into the momentum kernels (rke off).
//
// K7 of a sweep (xremap.f90:201-290 and the y/z mirrors) forms at each
// vertex the eight-cell sums of rho cv1, cv1, cv2 and dm, and from them
// rho_v = sum(rho cv1) / sum(cv1), cv1_v = sum(cv1) / 8, cv2_v = sum(cv2) / 8,
// dm_v = sum(dm) / 8 and rho_v1 = (rho_v cv1_v + dm_m - dm_v) / cv2_v, where
// dm_m, the dm average around the vertex below along the sweep axis, is that
// vertex's dm_v: its eight cells are summed in the same order.  K8 + K9
// read these back.  Here the momentum kernel forms them on the way, and the
// moved widths db1 and dc1 from the face velocity, so no vertex or geometry
// array reaches memory (11 words per point instead of 9 + 14).  At 256^3 a
// sweep takes 0.34 ms (y, z) and 0.37 ms (x) in FP64 and 0.26 and 0.25 ms in
// FP32; reading db1 and dc1 with plain loads it took 0.46 and 0.36, 0.30 and
// 0.32 ms.  The floor is 0.23 ms (FP64); bound by issue at 16 warps an SM.
//
// Every sum keeps the reference's order: the four cells of the z-plane quad
// (x, y), (x+1, y), (x, y+1), (x+1, y+1) at z, then the same at z + 1, added
// left to right.  The eight cells of vertex ia are the 2 x 2 transverse
// cells of two neighbouring slices along the sweep axis, and each sweep
// interleaves the slices differently:
//   z sweep: slice z, then slice z + 1 (its running sum is carried);
//   y sweep: two cells of slice y, two of y + 1, two of y, two of y + 1 (the
//            first pair's sum and the last pair of slice y are carried);
//   x sweep: alternately slice x and slice x + 1 (the next lane's cells).
// The results are the split kernels' bit for bit.  The FP64 product build,
// not bound to the reference's rounding, sums each slice's four cells first
// and adds the two slice sums (kReassoc): fewer live values and shorter
// chains.
// With rke on, the kinetic-energy defect reads the vertex arrays, and the
// split kernels run instead.
#pragma once

LARE_BEGIN

// The product build's association of the eight-cell sums (two slice sums).
template <class R>
constexpr bool kReassoc = LARE_FAST && sizeof(R) == 8;

template <class R>
struct VMArgs {
  MomArgs<R> m;  // the momentum kernel's operands; rv, dmv, cv1v, cv2v, rv1 unused
  A1<R> dba;     // cell widths along the sweep axis
  const R* rho;  // rho1 (the density before this sweep)
  const R* cv1;
  const R* cv2;
  const R* dm;
};

// The four cells of a slice at cell index b (offsets o[0..3]) for the four
// summed quantities.
template <class R>
struct SliceCells {
  R p[4], w[4], w2[4], d[4];  // rho cv1, cv1, cv2, dm
};

template <class R>
__device__ __forceinline__ SliceCells<R> slice_cells(const VMArgs<R>& g, int b, const int (&o)[4]) {
  SliceCells<R> s;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    s.w[q] = g.cv1[b + o[q]];
    s.p[q] = g.rho[b + o[q]] * s.w[q];
    s.w2[q] = g.cv2[b + o[q]];
    s.d[q] = g.dm[b + o[q]];
  }
  return s;
}

// The eight-cell sums of one vertex.
template <class R>
struct VertexSums {
  R p, w, w2, d;
};

// What a march carries of the slice below the new one: the z sweep its
// running sum (four cells), the y sweep the sum of its first pair
// (x, z), (x+1, z) and its last pair (x, z+1), (x+1, z+1).
template <class R>
struct Carry {
  R h, e2, e3;
};

template <int A, class R>
__device__ __forceinline__ Carry<R> carry_of(const R (&v)[4]) {
  Carry<R> c;
  if (A == 2 || kReassoc<R>) {
    c.h = v[0] + v[1] + v[2] + v[3];
    c.e2 = c.e3 = R(0);
  } else {
    c.h = v[0] + v[1];
    c.e2 = v[2];
    c.e3 = v[3];
  }
  return c;
}

// The vertex sum from the carried lower slice and the upper slice's cells.
// z sweep: (x,y),(x+1,y),(x,y+1),(x+1,y+1) of z, then of z+1.  y sweep
// (slice offsets 0, 1 at z, 2, 3 at z+1): (x,y,z),(x+1,y,z) of the lower
// slice, (x,y+1,z),(x+1,y+1,z) of the upper, (x,y,z+1),(x+1,y,z+1) of the
// lower, (x,y+1,z+1),(x+1,y+1,z+1) of the upper.
template <int A, class R>
__device__ __forceinline__ R vertex_sum(const Carry<R>& lo, const R (&up)[4]) {
  if (kReassoc<R>) return lo.h + (up[0] + up[1] + up[2] + up[3]);
  if (A == 2) return lo.h + up[0] + up[1] + up[2] + up[3];
  return lo.h + up[0] + up[1] + lo.e2 + lo.e3 + up[2] + up[3];
}

template <int A, class R>
__device__ __forceinline__ VertexSums<R> advance(Carry<R> (&cr)[4], const SliceCells<R>& s) {
  VertexSums<R> v;
  v.p = vertex_sum<A>(cr[0], s.p);
  v.w = vertex_sum<A>(cr[1], s.w);
  v.w2 = vertex_sum<A>(cr[2], s.w2);
  v.d = vertex_sum<A>(cr[3], s.d);
  cr[0] = carry_of<A>(s.p);
  cr[1] = carry_of<A>(s.w);
  cr[2] = carry_of<A>(s.w2);
  cr[3] = carry_of<A>(s.d);
  return v;
}

// The y and z sweeps.  A block of 32 x kVmY threads owns a tile of vertex
// lines along A, x along the lanes and the third axis t along the rows, and
// walks a chunk of it.  The plane two points on, which enters the windows,
// arrives in a ring of shared-memory slots by TMA, two steps ahead: rho, cv1,
// cv2 and dm with the row and column above (a slice of the eight-cell sums),
// the three velocity components, and v1 along A with the row and column below
// (the face velocity, from which the moved widths follow).
constexpr int kVmY = 8, kVmSlots = 4;
template <class R>
struct VMTile {
  static constexpr int W = 36;                                                    // 35 elements, to 16 bytes
  static constexpr int h = (W * (kVmY + 1) * (int)sizeof(R) + 127) / 128 * 128;   // with a halo row
  static constexpr int c = (W * kVmY * (int)sizeof(R) + 127) / 128 * 128;
  static constexpr int va = 4 * h, v = 5 * h, slot = 5 * h + 3 * c;
  static constexpr unsigned sent = W * sizeof(R) * (5 * (kVmY + 1) + 3 * kVmY);
  static constexpr size_t smem = 128 + (size_t)kVmSlots * slot;
};
struct VMMaps {
  CUtensorMap s[4], va, v[3];  // s: rho, cv1, cv2, dm
};

template <int A, class R>
__global__ void __launch_bounds__(32 * kVmY, sizeof(R) == 8 ? 2 : 3)
    k_vm_march(const __grid_constant__ VMMaps maps, VMArgs<R> a) {
  using L = VMTile<R>;
  extern __shared__ unsigned char vm_smem[];
  __shared__ __align__(8) unsigned long long bars[2 * kVmSlots];
  const MomArgs<R>& g = a.m;
  const int lane = threadIdx.x, ty = threadIdx.y;
  const int x0 = 32 * (int)blockIdx.x, u0 = kVmY * (int)blockIdx.y;
  const int t0 = min(x0 + lane, g.nx), t1 = min(u0 + ty, g.n3);  // x and the third axis, from 0
  const bool own = x0 + lane <= g.nx && u0 + ty <= g.n3;
  const int ia0 = (int)blockIdx.z * g.chunk;
  const int ia1 = min(ia0 + g.chunk - 1, g.na);
  unsigned char* const buf = vm_smem + ((128u - (smem_addr(vm_smem) & 127u)) & 127u);
  TileRing<kVmSlots> ring;
  ring.full = smem_addr(bars);
  ring.empty = ring.full + 8 * kVmSlots;
  ring.base = smem_addr(buf);
  ring.sc = g.sc;
  auto issue = [&](int ia, int slot) {
    const uint32_t d = ring.base + slot * L::slot, bar = ring.full + 8 * slot;
    mbar_expect(bar, L::sent);
    const int e = x0, r = u0 + 2, p = ia + 4;  // elements count from -2: x0 - 2 is e
    auto load = [&](int off, const CUtensorMap* m, int row) {
      tma_load_3d(d + off, m, e, A == 1 ? p : row, A == 1 ? row : p, bar);
    };
#pragma unroll
    for (int q = 0; q < 4; ++q) load(q * L::h, &maps.s[q], r);
    load(L::va, &maps.va, r - 1);
#pragma unroll
    for (int q = 0; q < 3; ++q) load(L::v + q * L::c, &maps.v[q], r);
  };
  const bool boss = lane == 0 && ty == 0;
  if (boss) {
    ring.init(kVmY);
    for (int s = 0; s < kVmSlots && ia0 + s <= ia1; ++s) issue(ia0 + s, s);
  }
  const R dt = (R)g.sc[g.dt_slot];
  const int SA = g.SA, S3 = g.S3;
  const int o[4] = {0, 1, S3, 1 + S3};
  const R area = g.dct1(t0) * g.dct2(t1);
  const R eighth = R(0.125);
  int c = t0 + t1 * S3 + (ia0 - 1) * SA;  // vertex (and cell) index of face ia0 - 1
  // slices ia0 - 1, ia0, ia0 + 1: the sums of vertices ia0 - 1 (vlo) and
  // ia0 (vc), and slice ia0 + 1 carried
  Carry<R> cr[4];
  {
    const SliceCells<R> s = slice_cells(a, c, o);
    cr[0] = carry_of<A>(s.p);
    cr[1] = carry_of<A>(s.w);
    cr[2] = carry_of<A>(s.w2);
    cr[3] = carry_of<A>(s.d);
  }
  VertexSums<R> vlo = advance<A>(cr, slice_cells(a, c + SA, o));
  VertexSums<R> vc = advance<A>(cr, slice_cells(a, c + 2 * SA, o));
  R w[3][4];
#pragma unroll
  for (int comp = 0; comp < 3; ++comp)
#pragma unroll
    for (int q = 0; q < 4; ++q) w[comp][q] = g.v[comp][c + (q - 1) * SA];
  // the moved widths db1 and dc1 of the column (xremap.f90:57-115) from its
  // face velocities: db1(p) = db(p) + (vf(p) - vf(p - 1)) dt
  struct Va {
    R v, f;  // v along A at the vertex, face velocity of the cell column
  };
  auto vface = [&](int q) {
    const R v = g.va[q];
    return Va{v, (v + g.va[q - 1] + g.va[q - S3] + g.va[q - 1 - S3]) * R(0.25)};
  };
  const Va vm = vface(c - SA), vq0 = vface(c), vq1 = vface(c + SA);
  Va vq2 = vface(c + 2 * SA);
  R va0 = vq0.v, va1 = vq1.v;
  R dbw0 = a.dba(ia0 - 1) + (vq0.f - vm.f) * dt, dbw1 = a.dba(ia0) + (vq1.f - vq0.f) * dt;
  R dbw2 = a.dba(ia0 + 1) + (vq2.f - vq1.f) * dt;
  R dcw0 = R(0.5) * (dbw0 + dbw1), dcw1 = R(0.5) * (dbw1 + dbw2);
  // face ia0 - 1: rho_v at its two vertices, dm_v at the lower one
  R rvc = qdiv(vlo.p, vlo.w);
  R rvn = qdiv(vc.p, vc.w);
  R Fm[3], fpre[3];
  mom_flux_vals<R, false>(area, va0, va1, rvc, rvn, vlo.d * eighth, dbw0, dbw1, dbw2, dcw0, dcw1, w, dt, Fm, fpre);
  __syncthreads();  // the barriers are set up
  // this thread's element of a tile (past the grid, a neighbour's: zeros would
  // send the exact builds' divisions down their slow path)
  const int e = (t1 - u0) * L::W + t0 - x0 + 2;
  int slot = 0;
  uint32_t ph = 0;
  for (int ia = ia0; ia <= ia1; ++ia) {
    c += SA;
    ring.wait_full(slot, ph);
    const unsigned char* const sl = buf + slot * L::slot;
    // slice ia + 2 gives vertex ia + 1's sums
    SliceCells<R> s;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int b = e + (q & 1) + (q >> 1) * L::W;
      s.w[q] = reinterpret_cast<const R*>(sl + L::h)[b];
      s.p[q] = reinterpret_cast<const R*>(sl)[b] * s.w[q];
      s.w2[q] = reinterpret_cast<const R*>(sl + 2 * L::h)[b];
      s.d[q] = reinterpret_cast<const R*>(sl + 3 * L::h)[b];
    }
    const R* const pv = reinterpret_cast<const R*>(sl + L::va) + e + L::W;
    const Va nva{pv[0], (pv[0] + pv[-1] + pv[-L::W] + pv[-L::W - 1]) * R(0.25)};
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      w[comp][0] = w[comp][1];
      w[comp][1] = w[comp][2];
      w[comp][2] = w[comp][3];
      w[comp][3] = reinterpret_cast<const R*>(sl + L::v + comp * L::c)[e];
    }
    ring.release(slot);
    const VertexSums<R> vn = advance<A>(cr, s);
    va0 = va1;
    va1 = vq2.v;
    dbw0 = dbw1;
    dbw1 = dbw2;
    dbw2 = a.dba(ia + 2) + (nva.f - vq2.f) * dt;
    vq2 = nva;
    dcw0 = dcw1;
    dcw1 = R(0.5) * (dbw1 + dbw2);
    // vertex ia
    rvc = rvn;
    rvn = qdiv(vn.p, vn.w);
    const R dmv = vc.d * eighth;
    const R cc1 = vc.w * eighth, cc2 = vc.w2 * eighth;
    const R dmm = vlo.d * eighth;
    const R rv1 = qdiv(rvc * cc1 + dmm - dmv, cc2);
    R F[3];
    mom_flux_vals<R, false>(area, va0, va1, rvc, rvn, dmv, dbw0, dbw1, dbw2, dcw0, dcw1, w, dt, F, fpre);
    const R den = dv_of(cc2 * rv1);
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      if (own) g.vn[comp][c] = dv_div(rvc * w[comp][1] * cc1 + Fm[comp] - F[comp], den);
      Fm[comp] = F[comp];
    }
    vlo = vc;
    vc = vn;
    // the last step's slot is refilled once every warp has left it
    if (boss && ia > ia0 && ia - 1 + kVmSlots <= ia1) {
      const int ps = slot == 0 ? kVmSlots - 1 : slot - 1;
      ring.wait(ring.empty + 8 * ps, slot == 0 ? ph ^ 1u : ph);
      if (!ring.dead) issue(ia - 1 + kVmSlots, ps);
    }
    if (++slot == kVmSlots) {
      slot = 0;
      ph ^= 1u;
    }
  }
}

// The x sweep.  The lanes of a warp hold consecutive x positions; a block of
// 32 x kVmY threads holds kVmY rows of y and walks a chunk of z, its planes in
// the same kind of ring (a slice's upper cells are one plane ahead of the
// velocities).  Each lane holds the slice of cells at its x (y, y+1 at z, then
// at z+1) and takes the next lane's by shuffles, alternating the two in the
// reference's order; dm_m is the dm average of the lane below and rho_v of the
// next vertex is the next lane's.  A lane's face flux needs the two lanes above
// it, its moved width the lane below's face velocity, and its update the flux
// of the lane below, so a warp updates the kVMXOut = 28 vertices of lanes 2..29.
constexpr int kVMXOut = 28;
template <class R>
struct VXTile {
  static constexpr int W = sizeof(R) == 8 ? 36 : 40;  // 35 elements from the aligned start
  static constexpr int h = (W * (kVmY + 1) * (int)sizeof(R) + 127) / 128 * 128;
  static constexpr int c = (W * kVmY * (int)sizeof(R) + 127) / 128 * 128;
  static constexpr int va = 4 * h, v = 5 * h, slot = 5 * h + 3 * c;
  static constexpr unsigned sent = W * sizeof(R) * (5 * (kVmY + 1) + 3 * kVmY);
  static constexpr size_t smem = 128 + (size_t)kVmSlots * slot;
};

template <class R>
__global__ void __launch_bounds__(32 * kVmY, sizeof(R) == 8 ? 2 : 3)
    k_vm_x(const __grid_constant__ VMMaps maps, VMArgs<R> a) {
  using L = VXTile<R>;
  extern __shared__ unsigned char vm_smem[];
  __shared__ __align__(8) unsigned long long bars[2 * kVmSlots];
  const MomArgs<R>& g = a.m;
  const int lane = threadIdx.x, ty = threadIdx.y;
  const int x0 = -2 + kVMXOut * (int)blockIdx.x, y0 = kVmY * (int)blockIdx.y;
  const int ix = x0 + lane, iy = min(y0 + ty, g.ny);            // vertex / face x position, row
  const int xl = min(ix, g.nx + 2);
  const int iz0 = (int)blockIdx.z * g.chunk, iz1 = min(iz0 + g.chunk - 1, g.nz);
  const int e0 = x0 + 1, ea = e0 & ~(kTmaAlign<R> - 1);         // element of x0 - 1, counted from x = -2
  unsigned char* const buf = vm_smem + ((128u - (smem_addr(vm_smem) & 127u)) & 127u);
  TileRing<kVmSlots> ring;
  ring.full = smem_addr(bars);
  ring.empty = ring.full + 8 * kVmSlots;
  ring.base = smem_addr(buf);
  ring.sc = g.sc;
  auto issue = [&](int iz, int slot) {
    const uint32_t d = ring.base + slot * L::slot, bar = ring.full + 8 * slot;
    mbar_expect(bar, L::sent);
    const int r = y0 + 2, p = iz + 2;
#pragma unroll
    for (int q = 0; q < 4; ++q) tma_load_3d(d + q * L::h, &maps.s[q], ea, r, p + 1, bar);
    tma_load_3d(d + L::va, &maps.va, ea, r - 1, p, bar);
#pragma unroll
    for (int q = 0; q < 3; ++q) tma_load_3d(d + L::v + q * L::c, &maps.v[q], ea, r, p, bar);
  };
  const bool boss = lane == 0 && ty == 0;
  if (boss) {
    ring.init(kVmY);
    for (int s = 0; s < kVmSlots && iz0 + s <= iz1; ++s) issue(iz0 + s, s);
  }
  const int sx = g.sx, sxy = g.sxy;
  const bool own = lane >= 2 && lane <= kVMXOut + 1 && ix <= g.nx && y0 + ty <= g.ny;
  const R dt = (R)g.sc[g.dt_slot];
  const R eighth = R(0.125);
  const unsigned all = 0xffffffffu;
  const R wx = a.dba(max(xl, -1)), wt = g.dct1(iy);
  int c = xl + sx * iy + sxy * iz0;
  // the slice's cells (x, y) and (x, y+1) of plane iz0, and v1's face pair of
  // plane iz0 - 1
  SliceCells<R> s;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int b = c + q * sx;
    s.w[q] = a.cv1[b];
    s.p[q] = a.rho[b] * s.w[q];
    s.w2[q] = a.cv2[b];
    s.d[q] = a.dm[b];
  }
  R vz0 = g.va[c - sxy], vzm = g.va[c - sxy - sx];
  __syncthreads();  // the barriers are set up
  // this thread's element of a tile (past the grid, a neighbour's)
  const int e = (iy - y0) * L::W + (e0 - ea) + xl - x0 + 1;
  // vertex x: (x,y,z),(x+1,y,z),(x,y+1,z),(x+1,y+1,z), then the same at z+1
  // (the product build: this slice's sum plus the next lane's)
  auto vsum = [&](const R (&v)[4]) {
    if (kReassoc<R>) {
      const R t = v[0] + v[1] + v[2] + v[3];
      return t + __shfl_down_sync(all, t, 1);
    }
    R t = v[0];
    t = t + __shfl_down_sync(all, v[0], 1);
    t = t + v[1];
    t = t + __shfl_down_sync(all, v[1], 1);
    t = t + v[2];
    t = t + __shfl_down_sync(all, v[2], 1);
    t = t + v[3];
    return t + __shfl_down_sync(all, v[3], 1);
  };
  int slot = 0;
  uint32_t ph = 0;
  for (int iz = iz0; iz <= iz1; ++iz, c += sxy) {
    ring.wait_full(slot, ph);
    const unsigned char* const sl = buf + slot * L::slot;
    auto tile = [&](int off) { return reinterpret_cast<const R*>(sl + off); };
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int b = e + q * L::W;
      s.w[2 + q] = tile(L::h)[b];
      s.p[2 + q] = tile(0)[b] * s.w[2 + q];
      s.w2[2 + q] = tile(2 * L::h)[b];
      s.d[2 + q] = tile(3 * L::h)[b];
    }
    R w[3][4];
#pragma unroll
    for (int comp = 0; comp < 3; ++comp)
#pragma unroll
      for (int q = 0; q < 4; ++q) w[comp][q] = tile(L::v + comp * L::c)[e + q - 1];
    const R va0 = tile(L::va)[e + L::W], vam = tile(L::va)[e];
    ring.release(slot);
    const R sp = vsum(s.p), sw = vsum(s.w), sw2 = vsum(s.w2), sd = vsum(s.d);
    const R rvc = qdiv(sp, sw);                                 // vertex x
    const R rvn = __shfl_down_sync(all, rvc, 1);                // vertex x + 1
    const R dmv = sd * eighth;
    const R dmm = __shfl_up_sync(all, dmv, 1);                  // vertex x - 1
    // the moved widths of the cells x, x + 1 and x + 2 (xremap.f90:57-115)
    const R vf = (va0 + vam + vz0 + vzm) * R(0.25);
    const R db0 = wx + (vf - __shfl_up_sync(all, vf, 1)) * dt;
    const R db1 = __shfl_down_sync(all, db0, 1), db2 = __shfl_down_sync(all, db0, 2);
    // the face flux between vertices x and x + 1 (faces -1..n)
    R F[3], fpre[3];
    mom_flux_vals<R, false>(wt * g.dct2(iz), va0, __shfl_down_sync(all, va0, 1), rvc, rvn, dmv, db0, db1, db2,
                            R(0.5) * (db0 + db1), R(0.5) * (db1 + db2), w, dt, F, fpre);
    R Fm[3];
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) Fm[comp] = __shfl_up_sync(all, F[comp], 1);
    if (own) {
      const R cc1 = sw * eighth, cc2 = sw2 * eighth;
      const R rv1 = qdiv(rvc * cc1 + dmm - dmv, cc2);
      const R den = dv_of(cc2 * rv1);
#pragma unroll
      for (int comp = 0; comp < 3; ++comp)
        g.vn[comp][c] = dv_div(rvc * w[comp][1] * cc1 + Fm[comp] - F[comp], den);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      s.p[q] = s.p[2 + q];
      s.w[q] = s.w[2 + q];
      s.w2[q] = s.w2[2 + q];
      s.d[q] = s.d[2 + q];
    }
    vz0 = va0;
    vzm = vam;
    // the last step's slot is refilled once every warp has left it
    if (boss && iz > iz0 && iz - 1 + kVmSlots <= iz1) {
      const int ps = slot == 0 ? kVmSlots - 1 : slot - 1;
      ring.wait(ring.empty + 8 * ps, slot == 0 ? ph ^ 1u : ph);
      if (!ring.dead) issue(iz - 1 + kVmSlots, ps);
    }
    if (++slot == kVmSlots) {
      slot = 0;
      ph ^= 1u;
    }
  }
}

// Dynamic shared memory beyond the default 48 KiB, once per context.
template <class R>
inline cudaError_t vm_attributes() {
  cudaError_t e = cudaFuncSetAttribute(k_vm_march<1, R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)VMTile<R>::smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_vm_march<2, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VMTile<R>::smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_vm_x<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)VXTile<R>::smem);
  return e;
}

template <int A, class R>
inline void vm_launch(Run<R>& run, VMArgs<R>& vm) {
  MomArgs<R>& g = vm.m;
  constexpr int W = A == 0 ? VXTile<R>::W : VMTile<R>::W;
  VMMaps maps;
  const long long f = 2 + 2LL * run.sx + 2LL * run.sxy;
  const auto map = [&](CUtensorMap* m, const R* p, int rows) {
    make_map(run, m, p - f, W, A == 1 ? 1 : rows, A == 1 ? rows : 1);
  };
  const R* const cells[4] = {vm.rho, vm.cv1, vm.cv2, vm.dm};
  for (int q = 0; q < 4; ++q) map(&maps.s[q], cells[q], kVmY + 1);
  map(&maps.va, g.va, kVmY + 1);
  for (int q = 0; q < 3; ++q) map(&maps.v[q], g.v[q], kVmY);
  if (run.launch_error) return;
  const dim3 blk(32, kVmY, 1);
  // words: v (3), v1, rho, cv1, cv2, dm read and the new v (3) written
  const int k = run.prof_begin(A == 0 ? "remap_sweep_vert_mom_x" : "remap_sweep_vert_mom_march", 0, 11,
                               (double)(g.nx + 1) * (g.ny + 1) * (g.nz + 1));
  if constexpr (A == 0) {
    constexpr size_t smem = VXTile<R>::smem;
    dim3 grd((g.nx + 1 + kVMXOut - 1) / kVMXOut, (g.ny + 1 + kVmY - 1) / kVmY, 1);
    g.chunk = march_chunk(g.nz + 1, grd.x * grd.y, kMomA, resident_blocks<k_vm_x<R>>(32 * kVmY, smem));
    grd.z = (g.nz + 1 + g.chunk - 1) / g.chunk;
    k_vm_x<R><<<grd, blk, smem, run.s>>>(maps, vm);
  } else {
    constexpr size_t smem = VMTile<R>::smem;
    dim3 grd((g.nx + 1 + 31) / 32, (g.n3 + 1 + kVmY - 1) / kVmY, 1);
    g.chunk = march_chunk(g.na + 1, grd.x * grd.y, kMomA, resident_blocks<k_vm_march<A, R>>(32 * kVmY, smem));
    grd.z = (g.na + 1 + g.chunk - 1) / g.chunk;
    k_vm_march<A, R><<<grd, blk, smem, run.s>>>(maps, vm);
  }
  run.prof_end(k);
  ++run.launches;
}

LARE_END  // namespace lare
