// remap.cuh - one directional Van Leer remap sweep, fused.
//
// xremap.f90:37-336 remap_x and its mirrors yremap.f90:37-337 and
// zremap.f90:37-336, for a sweep along axis A (0 = x, 1 = y, 2 = z).  The
// reference runs about 25 loop nests per sweep; here they are grouped into
// a few kernels.  Every element is still computed by exactly the reference's
// expression over exactly the same inputs, so the results are unchanged bit
// for bit; what changes is where intermediates live:
//
//   K1 B          both constrained-transport edge fluxes (:340-470) and the
//                 four flux-difference updates (:121-157) with the geometry
//                 they need (remap_b.cuh), into a second set of B arrays.
//   K2 mass,      cv1 and cv2 (:57-86), dm (:474-533) over the whole cell box
//   energy        with dm_x_bcs (:899-917) folded in, the new rho (:174-182)
//                 into a second buffer (old rho stays readable as rho1), the
//                 energy flux (:539-601) and the new energy (:187-196)
//                 (remap_me.cuh).
//   K7 vertex     vertex rho_v, cv1, cv2, dm averages and rho_v1 (:201-290),
//   K8 momentum   the three momentum fluxes (:605-895), each times dm, and
//   K9 velocity   the three velocity updates (:292-329), one kernel that
//                 writes the new velocities to second buffers (remap_vm.cuh);
//                 with rke on K7 is a kernel of its own (below).
// The face-averaged vx1 written back at :265 is only read again as
// REAL(xpass)*(...) with xpass = 0, so it is formed in K8 and not stored.
// The predictor's sweeps (predictor_step = .TRUE.) are K1 alone.
//
// Indexing is linear: c = ix + sx*iy + sxy*iz, neighbours by constant
// offsets, with the axis a compile-time parameter.
#pragma once

#include <utility>

#include "remap_b.cuh"
#include "remap_me.cuh"

LARE_BEGIN

// K7 as a z-marching kernel: a thread owns an (x, y) column of vertices and
// walks a chunk of z.  The eight cells around vertex (x, y, z) are the
// (x..x+1, y..y+1) quads of planes z and z+1, summed lower quad first in
// the reference's order, so each step loads the upper quad of each input
// and carries it down as the next vertex's lower quad: 18 to 20 loads per
// vertex instead of 40, the same sums in the same order, the same results
// bit for bit.  dm around c - e_A needs the quads of planes z-1 and z (A = z,
// one more plane carried) or the quads shifted by one cell in x or y (two
// more loads per plane).
constexpr int kVertZ = 16;

template <class R>
struct VertArgs {
  const R* rho;
  const R* cv1;
  const R* cv2;
  const R* dm;
  R* rv;
  R* rv1;
  R* cv1v;
  R* cv2v;
  R* dmv;
  int lo[3], hi[3];
  int na, sx, sxy;
};

template <int A, class R>
__global__ void __launch_bounds__(128) k_vert_march(VertArgs<R> g) {
  const int ix = g.lo[0] + (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int iy = g.lo[1] + (int)(blockIdx.y * blockDim.y + threadIdx.y);
  if (ix > g.hi[0] || iy > g.hi[1]) return;
  const int z0 = g.lo[2] + (int)blockIdx.z * kVertZ;
  const int z1 = min(z0 + kVertZ - 1, g.hi[2]);
  const int sx = g.sx, sxy = g.sxy, na = g.na;
  const int q1 = 1, q2 = sx, q3 = 1 + sx;                     // quad offsets after 0
  const int e0 = A == 0 ? -1 : -sx, e1 = A == 0 ? -1 + sx : 1 - sx;  // shifted-quad cells not in the quad
  int c = ix + sx * iy + sxy * z0;
  // lower quads (plane z0)
  R pr[4], c1[4], c2[4], d[4], dx[2], dz[4];
  auto load = [&](int b, R (&p)[4], R (&w1)[4], R (&w2)[4], R (&m)[4], R (&mx)[2]) {
    const int o[4] = {0, q1, q2, q3};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      w1[q] = g.cv1[b + o[q]];
      p[q] = g.rho[b + o[q]] * w1[q];
      w2[q] = g.cv2[b + o[q]];
      m[q] = g.dm[b + o[q]];
    }
    if (A != 2) {
      mx[0] = g.dm[b + e0];
      mx[1] = g.dm[b + e1];
    }
  };
  load(c, pr, c1, c2, d, dx);
  if (A == 2) {
    const int b = c - sxy;
    dz[0] = g.dm[b];
    dz[1] = g.dm[b + q1];
    dz[2] = g.dm[b + q2];
    dz[3] = g.dm[b + q3];
  }
  for (int iz = z0; iz <= z1; ++iz, c += sxy) {
    R pu[4], cu1[4], cu2[4], du[4], dxu[2];
    load(c + sxy, pu, cu1, cu2, du, dxu);
    const int ia = A == 0 ? ix : (A == 1 ? iy : iz);
    R s = pr[0], w = c1[0];
#pragma unroll
    for (int q = 1; q < 4; ++q) {
      s = s + pr[q];
      w = w + c1[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      s = s + pu[q];
      w = w + cu1[q];
    }
    const R rvc = qdiv(s, w);
    g.rv[c] = rvc;
    R tp = d[0];
#pragma unroll
    for (int q = 1; q < 4; ++q) tp = tp + d[q];
#pragma unroll
    for (int q = 0; q < 4; ++q) tp = tp + du[q];
    if (ia <= na) g.dmv[c] = tp * R(0.125);
    if (ia >= 0 && ia <= na) {
      R w2 = c2[0];
#pragma unroll
      for (int q = 1; q < 4; ++q) w2 = w2 + c2[q];
#pragma unroll
      for (int q = 0; q < 4; ++q) w2 = w2 + cu2[q];
      const R cc1 = w * R(0.125), cc2 = w2 * R(0.125);
      g.cv1v[c] = cc1;
      g.cv2v[c] = cc2;
      // dm summed over the cells around c - e_A, lower quad first
      R tm;
      if (A == 2) {
        tm = dz[0] + dz[1] + dz[2] + dz[3] + d[0] + d[1] + d[2] + d[3];
      } else if (A == 0) {  // quad cells (x-1, y), (x, y), (x-1, y+1), (x, y+1)
        tm = dx[0] + d[0] + dx[1] + d[2] + dxu[0] + du[0] + dxu[1] + du[2];
      } else {              // quad cells (x, y-1), (x+1, y-1), (x, y), (x+1, y)
        tm = dx[0] + dx[1] + d[0] + d[1] + dxu[0] + dxu[1] + du[0] + du[1];
      }
      const R dmm = tm * R(0.125);
      const R dmp = tp * R(0.125);
      g.rv1[c] = qdiv(rvc * cc1 + dmm - dmp, cc2);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (A == 2) dz[q] = d[q];
      pr[q] = pu[q];
      c1[q] = cu1[q];
      c2[q] = cu2[q];
      d[q] = du[q];
    }
    if (A != 2) {
      dx[0] = dxu[0];
      dx[1] = dxu[1];
    }
  }
}

// K8 + K9 fused: the momentum fluxes (xremap.f90:605-895, each times dm)
// and the velocity updates that consume them (:292-329).  K9 updates v in
// place while K8's stencil reads v around each face, so the fused kernel
// writes the new velocities to a second set of buffers (swapped in by the
// caller; their ghosts are refilled by boundary_conditions right after) and
// never stores the fluxes: the update at c needs the fluxes at faces c-e_A
// and c.  x sweep: the lanes of a warp hold consecutive faces and pass the
// flux one lane up (31 updates per 32 lanes).  y and z sweeps: a thread
// walks kMomA faces along A, carrying the stencil windows (one new point
// per step) and the flux of the face behind; its register cap (launch
// bounds) is the measured best per precision.  Every flux and update is the
// reference's expression over the same operands, so the results are
// identical bit for bit.
constexpr int kMomA = 32;  // largest chunk (march_chunk)

template <class R>
struct MomArgs {
  const R* va;  // v1 along A
  const R* rv;
  const R* dmv;
  const R* db1;
  const R* dc1;
  const R* v[3];
  R* vn[3];
  const R* cv1v;
  const R* cv2v;
  const R* rv1;
  R* fp[3];  // rke: the fluxes before their product with dm
  A1<R> dct1, dct2;
  double* sc;
  int dt_slot, nx, ny, nz, na, n3, sx, sxy, SA, S3;
  int chunk;
};

// the three momentum fluxes through a face (K8's body) from its stencil
// values: w[comp] = v at c-e_A, c, c+e_A, c+2e_A; db1 at c, c+e_A, c+2e_A;
// dc1 at c, c+e_A; v1 (va), rho_v (rv) at c, c+e_A; dm at c
// BOTH: fpre[comp] also receives the flux before its product with dm (what
// rke's kinetic-energy terms use, xremap.f90:664-695).
template <class R, bool BOTH = false>
__device__ __forceinline__ void mom_flux_vals(R area, R va0, R va1, R rvc, R rvp, R dmc, R db0, R db1, R db2, R dc0,
                                              R dc1, const R (&w)[3][4], R dt, R (&F)[3], R* fpre = nullptr) {
  const R v_advect = (va0 + va1) * R(0.5);  // the face-averaged v1 of xremap.f90:257-265
  // The upwind choice, phi and dmu depend only on v_advect and the
  // geometry, so they are formed once for the three components (the same
  // expressions the limiter evaluates per component).
  const R dxci = db1, dxcm = db0, dxcp = db2, dxbi = dc0, dxbp = dc1;
  const R sign_v = copysign(R(1), v_advect);
  const R vad_p = (sign_v + R(1)) * R(0.5);
  const R vad_m = R(1) - vad_p;
  const R dxbu = dxbi * vad_p + dxbp * vad_m;
  const R rhou = rvc * vad_p + rvp * vad_m;
#if LARE_FAST
  // product build: the upwind widths by selection (vad_p is 0 or 1) and one
  // reciprocal per divisor, shared by the three components
  const R rci = fast_rcp(dxci), rcu = fast_rcp(signbit(v_advect) ? dxcp : dxcm), rbu = fast_rcp(dxbu);
  const R phi = fabs(v_advect) * dt * rbu;
  const R dmu = fabs(dmc) * rbu * fast_rcp(area * rhou);
#else
  const R dxcu = dxcm * vad_p + dxcp * vad_m;
  const R phi = fabs(v_advect) * dt / dxbu;
  const R dmu = fabs(dmc) / area / dxbu / rhou;
#endif
  // kRegroup: the slopes' factors, the widths and the 1/6 in, also shared
  const bool up = !signbit(v_advect);
  R k0 = R(0), ku = R(0), omd = R(0);
#if LARE_FAST
  if constexpr (kRegroup<R>) {
    const R dxb6 = dxbu * (R(1) / R(6));
    k0 = (R(2) - phi) * rci * dxb6;
    ku = (R(1) + phi) * rcu * dxb6;
    omd = R(1) - dmu;
  }
#endif
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) {
    const R fm = w[comp][0], fi = w[comp][1], fp = w[comp][2], fp2 = w[comp][3];
    const R dfm = fi - fm, dfi = fp - fi, dfp = fp2 - fp;
    R f;
    if constexpr (kRegroup<R>) {
      const R dfu = up ? dfm : dfp;
      const R da = k0 * fabs(dfi) + ku * fabs(dfu);
      const R Di = signed_min(lesser(lesser(R(fabs(da)), R(fabs(dfi))), R(fabs(dfu))), dfi, dfu, v_advect);
      f = (up ? fi : fp) + Di * omd;
    } else {
      const R fu = fi * vad_p + fp * vad_m;
      const R dfu = dfm * vad_p + dfp * vad_m;
#if LARE_FAST
      R Da = (R(2) - phi) * fabs(dfi) * rci + (R(1) + phi) * fabs(dfu) * rcu;
#else
      R Da = (R(2) - phi) * fabs(dfi) / dxci + (R(1) + phi) * fabs(dfu) / dxcu;
#endif
      Da = Da * (R(1) / R(6));
      const R ss = R(0.5) * (copysign(R(1), dfi) + copysign(R(1), dfu));
      const R Di = sign_v * ss * fmin(fmin(fabs(Da) * dxbu, fabs(dfi)), fabs(dfu));
      f = fu + Di * (R(1) - dmu);
    }
    if constexpr (BOTH) fpre[comp] = f;
    F[comp] = f * dmc;
  }
}

// the same, loading the stencil of face c and storing the fluxes before their
// product with dm in g.fp
template <class R>
__device__ __forceinline__ void mom_flux(const MomArgs<R>& g, int c, int i1, int i2, R dt, R (&F)[3]) {
  const int SA = g.SA;
  R w[3][4];
#pragma unroll
  for (int comp = 0; comp < 3; ++comp)
#pragma unroll
    for (int q = 0; q < 4; ++q) w[comp][q] = g.v[comp][c + (q - 1) * SA];
  R fpre[3];
  mom_flux_vals<R, true>(g.dct1(i1) * g.dct2(i2), g.va[c], g.va[c + SA], g.rv[c], g.rv[c + SA], g.dmv[c],
                         g.db1[c], g.db1[c + SA], g.db1[c + 2 * SA], g.dc1[c], g.dc1[c + SA], w, dt, F, fpre);
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) g.fp[comp][c] = fpre[comp];
}

// rke's kinetic-energy defect of one component through the vertex pair
// (c, c + e_A) (xremap.f90:664-695 and its eight siblings in [xyz]remap.f90,
// all of one form): f the flux before the product with dm, v the velocity
// before the update.
template <class R>
__device__ __forceinline__ R rke_dk(const R* v, const R* f, const R* dmv, const R* rv1, const R* cv2v, int c,
                                    int SA) {
  const R v0 = v[c], v1 = v[c + SA];
  const R fm = f[c - SA], f0 = f[c], fp = f[c + SA];
  const R dmm = dmv[c - SA], dm0 = dmv[c], dmp = dmv[c + SA];
  const R m = rv1[c] * cv2v[c], mp = rv1[c + SA] * cv2v[c + SA];
  const R ai = (v0 - fm) * dmm / m - (v0 - f0) * dm0 / m;
  const R aip = (v1 - f0) * dm0 / mp - (v1 - fp) * dmp / mp;
  R dk = (v1 - v0) * (f0 - R(0.5) * (v1 + v0)) - R(0.5) * ai * (v0 - f0) + R(0.5) * aip * (v1 - f0);
  return dk * dm0 * R(0.5);
}

// K9's update at c from the fluxes at faces c - e_A (Fm) and c (F)
template <class R>
__device__ __forceinline__ void mom_update(const MomArgs<R>& g, int c, const R (&Fm)[3], const R (&F)[3]) {
  const R rvc = g.rv[c], c1 = g.cv1v[c], den = dv_of(g.cv2v[c] * g.rv1[c]);
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) g.vn[comp][c] = dv_div(rvc * g.v[comp][c] * c1 + Fm[comp] - F[comp], den);
}

template <class R>
__global__ void __launch_bounds__(128) k_mom_x(MomArgs<R> g) {
  const int lane = (int)threadIdx.x;                        // blockDim.x == 32: one warp per row
  const int ix = -1 + (int)blockIdx.x * 31 + lane;          // face / vertex x position
  const int iy = (int)(blockIdx.y * blockDim.y + threadIdx.y);
  const int iz = (int)blockIdx.z;
  if (iy > g.ny) return;                                    // uniform over the warp
  const R dt = (R)g.sc[g.dt_slot];
  const int c = ix + g.sx * iy + g.sxy * iz;
  R F[3] = {R(0), R(0), R(0)};
  if (ix <= g.nx) mom_flux<R>(g, c, iy, iz, dt, F);    // faces -1..n
  R Fm[3];
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) Fm[comp] = __shfl_up_sync(0xffffffffu, F[comp], 1);
  if (lane >= 1 && ix >= 0 && ix <= g.nx) mom_update(g, c, Fm, F);
}

template <class R>
__global__ void __launch_bounds__(128, sizeof(R) == 8 ? 4 : 8) k_mom_march(MomArgs<R> g) {
  const int t0 = (int)(blockIdx.x * blockDim.x + threadIdx.x);  // x, 0..nx
  const int t1 = (int)(blockIdx.y * blockDim.y + threadIdx.y);  // the third axis, 0..n3
  if (t0 > g.nx || t1 > g.n3) return;
  const int ia0 = (int)blockIdx.z * g.chunk;
  const int ia1 = min(ia0 + g.chunk - 1, g.na);
  const R dt = (R)g.sc[g.dt_slot];
  const int SA = g.SA;
  const R area = g.dct1(t0) * g.dct2(t1);
  // stencil window of face ia0 - 1; each step shifts it by one and loads
  // the new far point
  int c = t0 + t1 * g.S3 + (ia0 - 1) * SA;
  R w[3][4];
#pragma unroll
  for (int comp = 0; comp < 3; ++comp)
#pragma unroll
    for (int q = 0; q < 4; ++q) w[comp][q] = g.v[comp][c + (q - 1) * SA];
  R va0 = g.va[c], va1 = g.va[c + SA], rvc = g.rv[c], rvn = g.rv[c + SA];
  R dbw0 = g.db1[c], dbw1 = g.db1[c + SA], dbw2 = g.db1[c + 2 * SA], dcw0 = g.dc1[c], dcw1 = g.dc1[c + SA];
  R Fm[3], fpre[3];
  mom_flux_vals<R, true>(area, va0, va1, rvc, rvn, g.dmv[c], dbw0, dbw1, dbw2, dcw0, dcw1, w, dt, Fm, fpre);
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) g.fp[comp][c] = fpre[comp];
  // the loads of face c + SA are issued one step ahead (a face's own values
  // and the new far points of the windows), so each step's arithmetic waits
  // on loads issued a step earlier
  struct Next {
    R w[3], va, rv, db, dc, dm, c1, c2, r1;
  };
  auto fetch = [&](int q) {
    Next n;
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) n.w[comp] = g.v[comp][q + 2 * SA];
    n.va = g.va[q + SA];
    n.rv = g.rv[q + SA];
    n.db = g.db1[q + 2 * SA];
    n.dc = g.dc1[q + SA];
    n.dm = g.dmv[q];
    n.c1 = g.cv1v[q];
    n.c2 = g.cv2v[q];
    n.r1 = g.rv1[q];
    return n;
  };
  Next nx = fetch(c + SA);
  for (int ia = ia0; ia <= ia1; ++ia) {
    c += SA;
    const Next cur = nx;
    if (ia < ia1) nx = fetch(c + SA);
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      w[comp][0] = w[comp][1];
      w[comp][1] = w[comp][2];
      w[comp][2] = w[comp][3];
      w[comp][3] = cur.w[comp];
    }
    va0 = va1;
    va1 = cur.va;
    rvc = rvn;
    rvn = cur.rv;
    dbw0 = dbw1;
    dbw1 = dbw2;
    dbw2 = cur.db;
    dcw0 = dcw1;
    dcw1 = cur.dc;
    R F[3];
    mom_flux_vals<R, true>(area, va0, va1, rvc, rvn, cur.dm, dbw0, dbw1, dbw2, dcw0, dcw1, w, dt, F, fpre);
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) g.fp[comp][c] = fpre[comp];
    // K9's update at c: fluxes at faces c - e_A and c
    const R c1 = cur.c1, den = dv_of(cur.c2 * cur.r1);
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      g.vn[comp][c] = dv_div(rvc * w[comp][1] * c1 + Fm[comp] - F[comp], den);
      Fm[comp] = F[comp];
    }
  }
}

LARE_END  // namespace lare

#include "remap_vm.cuh"

LARE_BEGIN

// bmode: 1 for the first sweep of a remap (B read as stored, put in flux
// form on the way), 2 for the last (B put back from flux form), 0 between.
template <int A, class R>
void remap_sweep(Run<R>& run, int dt_slot, int pass[3], int bmode) {
  constexpr int T1 = A == 0 ? 1 : 0, T2 = A == 2 ? 1 : 2;  // transverse axes, T1 < T2
  const int nx = run.n[0], ny = run.n[1], nz = run.n[2];
  const int nn[3] = {nx, ny, nz};
  const int na = nn[A];
  const int sx = run.sx, sxy = run.sxy;
  const int SA = A == 0 ? 1 : (A == 1 ? sx : sxy);
  const int S1 = T1 == 0 ? 1 : (T1 == 1 ? sx : sxy);
  const int S2 = T2 == 0 ? 1 : (T2 == 1 ? sx : sxy);
  Arrays<R>& Ar = run.a;
  R* const vx1 = Ar.vx1.p;
  R* const vy1 = Ar.vy1.p;
  R* const vz1 = Ar.vz1.p;
  R* const V1[3] = {vx1, vy1, vz1};
  R* const va = V1[A];
  R* const cv1 = Ar.cv1.p;
  R* const db1 = Ar.db1.p;
  R* const dc1 = Ar.dc1.p;
  const A1<R> dbm[3] = {Ar.dxb, Ar.dyb, Ar.dzb};
  const A1<R> dcm[3] = {Ar.dxc, Ar.dyc, Ar.dzc};
  const A1<R> dct1 = dcm[T1], dct2 = dcm[T2];

  // ---- K1: B, into the arrays of the Lagrangian step's B0, whose work is done
  // (bx1, by1, bz1 are named fields: the B before the last resistive sub-cycle)
  {
    R* const in[3] = {Ar.bx.p, Ar.by.p, Ar.bz.p};
    R* const out[3] = {Ar.bx0.p, Ar.by0.p, Ar.bz0.p};
    bsweep<A>(run, va, in, out, dt_slot, bmode);
    std::swap(Ar.bx.p, Ar.bx0.p);
    std::swap(Ar.by.p, Ar.by0.p);
    std::swap(Ar.bz.p, Ar.bz0.p);
  }

  R* const rho = Ar.rho.p;        // rho1 of the reference from here on
  R* const dm = Ar.dm.p;
  const int swept = 3 - pass[0] - pass[1] - pass[2];
  const R* const cv2 = swept == 2 ? Ar.cv.p : Ar.cv2.p;  // the third sweep ends at the grid itself
  {
    MEArgs<R> me;
    for (int d = 0; d < 3; ++d) {
      me.v[d] = V1[d];
      me.m[d] = dbm[d];
      me.r[d] = Ar.rdb[d];
      me.pass[d] = pass[d];
    }
    me.rho = rho;
    me.rho_new = Ar.rho_alt.p;
    me.energy = Ar.energy.p;
    me.energy_new = Ar.flux.p;  // swapped in below
    me.dm = dm;
    me.cv = Ar.cv.p;
    me.cv1 = cv1;
    me.cv2 = Ar.cv2.p;
    me.db1 = run.p.rke ? db1 : nullptr;
    me.dc1 = dc1;
    me.sc = run.sc;
    me.dt_slot = dt_slot;
    me.nx = nx;
    me.ny = ny;
    me.nz = nz;
    me.sx = sx;
    me.sxy = sxy;
    me.per = run.p.per[A];
    mass_energy_sweep<A>(run, me, swept);
    std::swap(Ar.energy.p, Ar.flux.p);
  }

  // ---- K7: vertex quantities.  rho_v over a -1:n+1, the rest over 0:n;
  // dm vertex averages over a -1:n.
  R* const rv = Ar.r_rho_v.p;
  R* const rv1 = Ar.r_rho_v1.p;
  R* const cv1v = Ar.cv1v.p;
  R* const cv2v = Ar.cv2v.p;
  R* const dmv = Ar.dmv.p;
  // rke off: the vertex averages are formed inside the momentum kernel, in
  // the reference's summation order (remap_vm.cuh)
  const bool fused_vm = !run.p.rke;
  if (!fused_vm) {
    int lo[3] = {0, 0, 0}, hi[3] = {nx, ny, nz};
    lo[A] = -1;
    hi[A] = na + 1;
    VertArgs<R> va7;
    va7.rho = rho;
    va7.cv1 = cv1;
    va7.cv2 = cv2;
    va7.dm = dm;
    va7.rv = rv;
    va7.rv1 = rv1;
    va7.cv1v = cv1v;
    va7.cv2v = cv2v;
    va7.dmv = dmv;
    for (int d = 0; d < 3; ++d) {
      va7.lo[d] = lo[d];
      va7.hi[d] = hi[d];
    }
    va7.na = na;
    va7.sx = sx;
    va7.sxy = sxy;
    dim3 blk(32, 4, 1);
    dim3 grd((hi[0] - lo[0] + 32) / 32, (hi[1] - lo[1] + 4) / 4, (hi[2] - lo[2] + kVertZ) / kVertZ);
    const int k = run.prof_begin("remap_sweep_vert", 0, 9,
                                 (double)(hi[0] - lo[0] + 1) * (hi[1] - lo[1] + 1) * (hi[2] - lo[2] + 1));
    k_vert_march<A, R><<<grd, blk, 0, run.s>>>(va7);
    run.prof_end(k);
    ++run.launches;
  }

  // ---- K8 + K9: momentum fluxes (faces a -1:n, transverse 0:n) and the
  // velocity updates (0:n) in one kernel, new velocities into the q buffers
  {
    MomArgs<R> gm;
    gm.va = va;
    gm.rv = rv;
    gm.dmv = dmv;
    gm.db1 = db1;
    gm.dc1 = dc1;
    gm.v[0] = Ar.vx.p;
    gm.v[1] = Ar.vy.p;
    gm.v[2] = Ar.vz.p;
    gm.vn[0] = Ar.qx.p;
    gm.vn[1] = Ar.qy.p;
    gm.vn[2] = Ar.qz.p;
    gm.cv1v = cv1v;
    gm.cv2v = cv2v;
    gm.rv1 = rv1;
    gm.dct1 = dct1;
    gm.dct2 = dct2;
    gm.sc = run.sc;
    gm.dt_slot = dt_slot;
    gm.nx = nx;
    gm.ny = ny;
    gm.nz = nz;
    gm.na = na;
    gm.n3 = A == 1 ? nz : ny;
    gm.sx = sx;
    gm.sxy = sxy;
    gm.SA = SA;
    gm.S3 = A == 1 ? sxy : sx;
    for (int q = 0; q < 3; ++q) gm.fp[q] = Ar.rke_f[q].p;
    if (fused_vm) {
      VMArgs<R> vm;
      vm.m = gm;
      vm.dba = dbm[A];
      vm.rho = rho;
      vm.cv1 = cv1;
      vm.cv2 = cv2;
      vm.dm = dm;
      vm_launch<A>(run, vm);
    } else {
      const int k = run.prof_begin(A == 0 ? "remap_sweep_mom_x" : "remap_sweep_mom_march", 0, 17,
                                   (double)(nx + 1) * (ny + 1) * (nz + 1));
      if (A == 0) {
        dim3 grd((nx + 1 + 30) / 31, (ny + 1 + 3) / 4, nz + 1);
        k_mom_x<R><<<grd, dim3(32, 4, 1), 0, run.s>>>(gm);
      } else {
        dim3 grd((nx + 1 + 31) / 32, (gm.n3 + 1 + 3) / 4, 1);
        gm.chunk = march_chunk(na + 1, grd.x * grd.y, kMomA, resident_blocks<k_mom_march<R>>(128));
        grd.z = (na + 1 + gm.chunk - 1) / gm.chunk;
        k_mom_march<R><<<grd, dim3(32, 4, 1), 0, run.s>>>(gm);
      }
      run.prof_end(k);
      ++run.launches;
    }
  }
  if (run.p.rke) {
    // rke (xremap.f90:664-695 and siblings): the old velocities are still
    // in v (the new ones went to the q buffers), and the momentum kernel
    // above stored the three fluxes before their product with dm (faces
    // -1:n along A).  R2 forms each vertex's defect dk per component; R3
    // adds, per cell 1:n, the dk of each vertex whose update scatters into
    // it, for the components in file order and the vertices in the
    // reference's loop order, so the sums are the reference's bit for bit.
    const R* const rf0 = Ar.rke_f[0].p;
    const R* const rf1 = Ar.rke_f[1].p;
    const R* const rf2 = Ar.rke_f[2].p;
    int lo[3] = {0, 0, 0}, hi[3] = {nx, ny, nz};
    R* const dke = Ar.delta_ke.p;
    const R* const vv0 = Ar.vx.p;
    const R* const vv1 = Ar.vy.p;
    const R* const vv2 = Ar.vz.p;
    R* const dk0 = Ar.rke_dk[0].p;
    R* const dk1 = Ar.rke_dk[1].p;
    R* const dk2 = Ar.rke_dk[2].p;
    // R2: each vertex's defect once (vertices 0:n-1 along A, 0:n across)
    lo[A] = 0;
    hi[A] = na - 1;
    LARE_BOXW(run, 15, lo[0], hi[0], lo[1], hi[1], lo[2], hi[2], [=] __device__(int ix, int iy, int iz) {
      const int c = ix + sx * iy + sxy * iz;
      dk0[c] = rke_dk(vv0, rf0, dmv, rv1, cv2v, c, SA);
      dk1[c] = rke_dk(vv1, rf1, dmv, rv1, cv2v, c, SA);
      dk2[c] = rke_dk(vv2, rf2, dmv, rv1, cv2v, c, SA);
    });
    // R3: the gather
    LARE_BOXW(run, 14, 1, nx, 1, ny, 1, nz, [=] __device__(int ix, int iy, int iz) {
      const int c = ix + sx * iy + sxy * iz;
      const int b = c - SA;  // the vertex below along A; its transverse neighbours below
      const int vtx[4] = {b - S1 - S2, b - S2, b - S1, b};
      const R* const dq[3] = {dk0, dk1, dk2};
      R d = dke[c];
#pragma unroll
      for (int comp = 0; comp < 3; ++comp)
#pragma unroll
        for (int q = 0; q < 4; ++q) d = d + dq[comp][vtx[q]];
      dke[c] = d;
    });
  }
  std::swap(Ar.vx.p, Ar.qx.p);
  std::swap(Ar.vy.p, Ar.qy.p);
  std::swap(Ar.vz.p, Ar.qz.p);
  {
    R* const nv[3] = {Ar.vx.p, Ar.vy.p, Ar.vz.p};
    R* const ov[3] = {Ar.qx.p, Ar.qy.p, Ar.qz.p};
    carry_velocity(run, nv, ov);
  }

  // The new density becomes rho; the old buffer is scratch again.
  std::swap(Ar.rho.p, Ar.rho_alt.p);
  boundary_conditions(run);
  pass[A] = 0;
}

LARE_END  // namespace lare
