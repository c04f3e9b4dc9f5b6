// fdtd_kernels.cu -- the fused staggered-grid FDTD step for sm_100a.
//
// One launch advances every active solve of a batch by one time step
// (forward_onestep!, src/kernels/forward.jl:13-139).  The step reads field
// buffer `rb` and writes buffer `wb`, so the pressure update, the q-channel
// injection/recording, the three velocity updates, the f-channel
// injection/recording and the rigid mirrors all happen in a single pass over
// HBM: 16 B read + 16 B written per cell, plus the CPML memory on the slabs
// and half a byte of mask per cell.
//
// Work decomposition (2.5D): a CTA owns a tile of 7 rows x 64 cells of one
// solve and a run of planes; each warp holds 16 cells of all the tile's rows
// (plus the halo row), its lanes 4-cell quads, and the CTA walks the planes
// in z keeping the z-neighbours in registers.  The new P of a plane goes
// through shared memory for the x-1 / y-1 neighbours of the velocity update;
// the halo row and column are recomputed, not exchanged.  Five such CTAs per
// SM keep HBM busy while a plane's chain (stage loads, Float64 arithmetic,
// exchange of the new P, Float64 arithmetic) runs in each; what bounds them is
// that chain and the instructions around it, not HBM.  The stage is read through
// shared-space addresses, on different banks, and the entries' code is out of the
// plane loop.  A launch of 8 x 256^3 takes 0.75 ms without boundaries and, with
// 10-cell CPML, a sphere and 2048 receivers, 1.21 ms in short runs and 1.25 over 2000
// steps (under the power cap).  The plane loop's code has to stay small: a masked form
// of the plain update made the second 2 % slower, one with the x slab's memory 6 %.
//
// Arithmetic: Arith<double> reproduces Julia's promotion (Float32 storage,
// Float64 Domain scalars, src/kernels/updates.jl) with explicit round-to-
// nearest intrinsics so that nothing is contracted; the one deliberate
// difference is x*(1/dx) in place of x/dx.  Arith<float> is the all-Float32
// variant.  Injection/recording (derivatives.jl:30-60) is pure Float32 with
// separate multiply and add, as the reference computes it.
#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "adf_internal.h"
#include "ptx_util.h"
#include "slab_index.h"

namespace adf {


// ---------------------------------------------------------------------------
// Arithmetic policies
// ---------------------------------------------------------------------------
template <typename R>
struct Arith;
template <>
struct Arith<double> {
  static __device__ __forceinline__ double cv(float x) { return (double)x; }
  static __device__ __forceinline__ float rn(double x) { return __double2float_rn(x); }
  static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
  static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
  static __device__ __forceinline__ double fq(const SolveDev& s) { return s.fq; }
  static __device__ __forceinline__ double fv(const SolveDev& s) { return s.fv; }
  static __device__ __forceinline__ double rdx(const SolveDev& s) { return s.rdx; }
  static __device__ __forceinline__ double rdy(const SolveDev& s) { return s.rdy; }
  static __device__ __forceinline__ double rdz(const SolveDev& s) { return s.rdz; }
};
template <>
struct Arith<float> {
  static __device__ __forceinline__ float cv(float x) { return x; }
  static __device__ __forceinline__ float rn(float x) { return x; }
  static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
  static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
  static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
  static __device__ __forceinline__ float fq(const SolveDev& s) { return s.fqf; }
  static __device__ __forceinline__ float fv(const SolveDev& s) { return s.fvf; }
  static __device__ __forceinline__ float rdx(const SolveDev& s) { return s.rdxf; }
  static __device__ __forceinline__ float rdy(const SolveDev& s) { return s.rdyf; }
  static __device__ __forceinline__ float rdz(const SolveDev& s) { return s.rdzf; }
};

// CPML memory update m = b*m + a*d; d += m  (updates.jl:46-61): b*m is a
// Float32 product, a*d is promoted, the sum is rounded to Float32 on store
// and re-added.  `m` is updated in place; the caller stores it.
template <typename R>
__device__ __forceinline__ void cpml_apply(R& dv, float& m, float a, float b) {
  using A = Arith<R>;
  const float bm = __fmul_rn(b, m);
  m = A::rn(A::add(A::cv(bm), A::mul(A::cv(a), dv)));
  dv = A::add(dv, A::cv(m));
}


__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
// (The kernels of a step start while their predecessors run, so the read-only path,
// __ldg, is for what the set-up wrote alone: what a predecessor still writes has to be
// read with ordinary loads, after the wait.)
// field stores: evict-first (the next step reads them back from HBM, and the
// halo rows that neighbouring tiles re-read are loads, which keep normal
// priority)
__device__ __forceinline__ void stcs4(float* p, float4 v) { __stcs(reinterpret_cast<float4*>(p), v); }
__device__ __forceinline__ float4 neg4(float4 v) { return make_float4(-v.x, -v.y, -v.z, -v.w); }

template <typename R>
struct Sc {  // per-solve update scalars
  R fq, fv, rdx, rdy, rdz;
};

// What the CPML updates of a work item need, in shared memory: per array (p x,
// y, z, v x, y, z) the buffer read, the one written and, for the x and y slabs,
// the plane stride; the coefficients of the tile's columns ([3] is the halo
// column's), rows and planes; and where the z slabs' layers lie (kNoSlab: none).
// Places are counted in quads (slab_index.h), which hold any buffer in 32 bits; in
// floats x-slab memory passes 2^31 at 128 x 4100 x 4100 cells and 63 layers.  A
// boundary warp's length sets its CTA's pace, so what does not change from plane
// to plane is worked out once per item.
struct PmlTab {
  const float4* rd[6];
  float4* wr[6];
  uint32_t stride[6];
  uint32_t hx;  // the halo column's cell, the last of its quad, in row 0 of the p side; or kNoSlab
  alignas(16) float xpa[68];  // (read four at a time)
  alignas(16) float xpb[68];
  alignas(16) float xva[68];
  alignas(16) float xvb[68];
  float ypa[8], ypb[8], yva[8], yvb[8];
  float zpa[kMaxZc + 1], zpb[kMaxZc + 1], zva[kMaxZc + 1], zvb[kMaxZc + 1];
  uint32_t zp[kMaxZc + 1], zv[kMaxZc + 1];
};

static_assert(offsetof(PmlTab, xpa) % 16 == 0 && offsetof(PmlTab, xpb) % 16 == 0 &&
                  offsetof(PmlTab, xva) % 16 == 0 && offsetof(PmlTab, xvb) % 16 == 0,
              "a quad's coefficients are one aligned float4");

// A thread's quad, for the planes of an item.
struct Quad {
  // cell e: bit e P updated (x <= nx-2), 4+e Vx updated (1 <= x < nx), 8+e in the
  // grid (x < nx), 12+e P has x-slab memory, 16+e Vx has; bit 20: cells in both x
  // slabs (narrow grids); 21 the quad lies in the grid, 22 and is stored by the thread
  uint32_t bits;
  int j, x0, r;
  uint32_t px, vx;  // x-slab memory of plane 0 (quads, as in PmlTab)
  uint32_t py, vy;  // y-slab memory of plane 0, kNoSlab: none
};

// Cell e of a quad of slab memory.
__device__ __forceinline__ const float* slab_cell(const float4* base, uint32_t quad, int e) {
  return reinterpret_cast<const float*>(base + quad) + e;
}

// Memory of cells that are not updated stays as it was read.
__device__ __forceinline__ void keep_rest(float (&m)[4], float4 t, uint32_t upd) {
  if (!(upd & 1u)) m[0] = t.x;
  if (!(upd & 2u)) m[1] = t.y;
  if (!(upd & 4u)) m[2] = t.z;
  if (!(upd & 8u)) m[3] = t.w;
}

// x-slab memory of a quad with cells in both slabs: cell by cell.
template <typename R>
__device__ __forceinline__ void x_slabs_narrow(R (&d)[4], const PmlTab& Q, int arr, int pitch,
                                               long long side, int xs1, int first1, int row, int x0,
                                               uint32_t in, bool store, const float* a,
                                               const float* b) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (!((in >> e) & 1u)) continue;
    const int right = x0 + e >= first1;
    const uint32_t o = slab_quad(side, right, row, pitch, right ? x0 - xs1 : x0);
    float m = *slab_cell(Q.rd[arr], o, e);
    cpml_apply<R>(d[e], m, a[e], b[e]);
    if (store) reinterpret_cast<float*>(Q.wr[arr] + o)[e] = m;
  }
}

// ---------------------------------------------------------------------------
// Pressure update of a quad of plane k (update_p_cpml!, update_p_mask!,
// update_p! on the rigid planes; updates.jl:21-136), u = k - kfirst.  Inputs are
// the plane's P, Vx (x0..x0+4), Vy (rows j, j+1) and Vz (planes k, k+1) from the
// input buffer.  Row- and plane-wide conditions (rigid planes, y/z slabs) are
// warp-uniform or nearly so; the x slab is a block taken only by quads that
// touch it.  `owned` stores the new CPML memory; recomputed halo cells and the
// prologue plane leave it alone.
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ float4 p_update_quad(const SolveDev& S, const PmlTab& Q, const Quad& q,
                                                const Sc<R>& g, bool pcpml, int k, int u, bool owned,
                                                float4 P4, float4 X4, float X5, float4 Y0, float4 Y1,
                                                float4 Z0, float4 Z1, uint32_t nib, float4 mx) {
  using A = Arith<R>;
  const bool rigid_y = q.j == S.ny - 1, rigid_z = k == S.nz - 1;
  // rigid planes use update_p! (-2V/d at the wall, no CPML, no mask); the
  // (ny, nz) corner is not updated at all
  if (rigid_y) Y1 = neg4(Y0);
  if (rigid_z) Z1 = neg4(Z0);
  if (rigid_y || rigid_z) nib = 0xFFFFu;
  uint32_t up = q.bits & 15u;
  if (rigid_y && rigid_z) up = 0;
  R dx[4] = {A::mul(A::cv(__fsub_rn(X4.y, X4.x)), g.rdx), A::mul(A::cv(__fsub_rn(X4.z, X4.y)), g.rdx),
             A::mul(A::cv(__fsub_rn(X4.w, X4.z)), g.rdx), A::mul(A::cv(__fsub_rn(X5, X4.w)), g.rdx)};
  R dy[4] = {A::mul(A::cv(__fsub_rn(Y1.x, Y0.x)), g.rdy), A::mul(A::cv(__fsub_rn(Y1.y, Y0.y)), g.rdy),
             A::mul(A::cv(__fsub_rn(Y1.z, Y0.z)), g.rdy), A::mul(A::cv(__fsub_rn(Y1.w, Y0.w)), g.rdy)};
  R dz[4] = {A::mul(A::cv(__fsub_rn(Z1.x, Z0.x)), g.rdz), A::mul(A::cv(__fsub_rn(Z1.y, Z0.y)), g.rdz),
             A::mul(A::cv(__fsub_rn(Z1.z, Z0.z)), g.rdz), A::mul(A::cv(__fsub_rn(Z1.w, Z0.w)), g.rdz)};
  if (pcpml && !rigid_y && !rigid_z) {
    if (q.bits & 0xF000u) {
      const float4 a4 = ld4(Q.xpa + 4 + 4 * (q.x0 / 4 % 16)), b4 = ld4(Q.xpb + 4 + 4 * (q.x0 / 4 % 16));
      const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
      if (q.bits & (1u << 20)) {
        x_slabs_narrow<R>(dx, Q, 0, S.npp, S.psi_p_side[0], S.xs1p, S.npml, k * S.ny + q.j, q.x0,
                          q.bits >> 12, owned, a, b);
      } else {
        const uint32_t o = q.px + k * Q.stride[0];
        const float4 t = mx;
        float m[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if ((q.bits >> (12 + e)) & 1u) cpml_apply<R>(dx[e], m[e], a[e], b[e]);
        // cells outside the slab or not updated write back what they read
        if (owned) Q.wr[0][o] = make_float4(m[0], m[1], m[2], m[3]);
      }
    }
    if (q.py != kNoSlab) {  // y slab: the whole quad, cells that are not updated keep their memory
      const uint32_t o = q.py + k * Q.stride[1];
      const float4 t = Q.rd[1][o];
      float m[4] = {t.x, t.y, t.z, t.w};
      const float a = Q.ypa[q.r], b = Q.ypb[q.r];
#pragma unroll
      for (int e = 0; e < 4; ++e) cpml_apply<R>(dy[e], m[e], a, b);
      if (up != 15u) keep_rest(m, t, up);
      if (owned) Q.wr[1][o] = make_float4(m[0], m[1], m[2], m[3]);
    }
    if (Q.zp[u] != kNoSlab && (q.bits & (1u << 21))) {
      const uint32_t o = Q.zp[u] + ((uint32_t)(q.j * S.nxp + q.x0) >> 2);
      const float4 t = Q.rd[2][o];
      float m[4] = {t.x, t.y, t.z, t.w};
      const float a = Q.zpa[u], b = Q.zpb[u];
#pragma unroll
      for (int e = 0; e < 4; ++e) cpml_apply<R>(dz[e], m[e], a, b);
      if (up != 15u) keep_rest(m, t, up);
      if (owned) Q.wr[2][o] = make_float4(m[0], m[1], m[2], m[3]);
    }
  }
  const float Pv[4] = {P4.x, P4.y, P4.z, P4.w};
  float o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float n = A::rn(A::sub(A::cv(Pv[e]), A::mul(g.fq, A::add(A::add(dx[e], dy[e]), dz[e]))));
    o[e] = ((up >> e) & (nib >> (4 * e)) & 1u) ? n : Pv[e];
  }
  return make_float4(o[0], o[1], o[2], o[3]);
}

// The same update for the cell before a tile's first quad q (the halo column
// x = xb-1 of an x tile), from the staged plane `st` (P, Vx, Vy of plane k; `c` the
// cell's offset in a channel, `cst` the channel stride) and Vz of planes k and k+1
// (Z0, Z1).  Its y and z slab memory lies one float before the quad's.
template <typename R>
__device__ __forceinline__ float p_update_cell(const SolveDev& S, const PmlTab& Q, const Quad& q,
                                               const Sc<R>& g, bool pcpml, const float* st, float Z0,
                                               float Z1, int c, int cst, int k, int u, bool masked) {
  using A = Arith<R>;
  const int nx = S.nx, ny = S.ny, nz = S.nz, x = q.x0 - 1, j = q.j, r = q.r;
  const bool rigid_y = j == ny - 1, rigid_z = k == nz - 1;
  const bool plain_rigid = rigid_y || rigid_z;
  const bool upd = x <= nx - 2 && !(rigid_y && rigid_z);
  const float P = st[c];
  if (!upd) return P;
  const float X0 = st[cst + c], X1 = st[cst + c + 1];
  const float Y0 = st[2 * cst + c];
  const float dy = rigid_y ? __fmul_rn(-2.0f, Y0) : __fsub_rn(st[2 * cst + c + kStageW], Y0);
  const float dz = rigid_z ? __fmul_rn(-2.0f, Z0) : __fsub_rn(Z1, Z0);
  R dvx = A::mul(A::cv(__fsub_rn(X1, X0)), g.rdx);
  R dvy = A::mul(A::cv(dy), g.rdy);
  R dvz = A::mul(A::cv(dz), g.rdz);
  bool open = true;
  if (!plain_rigid) {
    if (masked) open = (S.mask_bits[((long long)k * ny + j) * S.mw + (x >> 3)] >> (4 * (x & 7))) & 1u;
    if (pcpml) {
      if (Q.hx != kNoSlab) {
        float m = *slab_cell(Q.rd[0], Q.hx + slab_quad(0, 0, k * ny + j, S.npp, 0), 3);
        cpml_apply<R>(dvx, m, Q.xpa[3], Q.xpb[3]);
      }
      if (q.py != kNoSlab) {
        float m = *slab_cell(Q.rd[1], q.py + k * Q.stride[1], -1);
        cpml_apply<R>(dvy, m, Q.ypa[r], Q.ypb[r]);
      }
      if (Q.zp[u] != kNoSlab) {
        float m = *slab_cell(Q.rd[2], Q.zp[u] + ((uint32_t)(j * S.nxp + q.x0) >> 2), -1);
        cpml_apply<R>(dvz, m, Q.zpa[u], Q.zpb[u]);
      }
    }
  }
  const float n = A::rn(A::sub(A::cv(P), A::mul(g.fq, A::add(A::add(dvx, dvy), dvz))));
  return open ? n : P;
}

// ---------------------------------------------------------------------------
// Velocity updates of the quad (update_vx!/vy!/vz! and their masked forms,
// updates.jl:192-274, 380-500): Vx over x >= 1, Vy over j >= 1, Vz over k >= 1,
// x < nx; CPML with the half-grid coefficients (npml+1 layers).
// ---------------------------------------------------------------------------
template <typename R>
__device__ __forceinline__ void v_update_quad(const SolveDev& S, const PmlTab& Q, const Quad& q,
                                              const Sc<R>& g, bool vcpml, int k, int u, float4 Pc,
                                              float Pxm, float4 Pym, float4 Pzm, float4 VX, float4 VY,
                                              float4 VZ, uint32_t nib, float4 mx, float4& vxo, float4& vyo,
                                              float4& vzo) {
  using A = Arith<R>;
  const uint32_t in = (q.bits >> 8) & 15u;
  R dx[4] = {A::mul(A::cv(__fsub_rn(Pc.x, Pxm)), g.rdx), A::mul(A::cv(__fsub_rn(Pc.y, Pc.x)), g.rdx),
             A::mul(A::cv(__fsub_rn(Pc.z, Pc.y)), g.rdx), A::mul(A::cv(__fsub_rn(Pc.w, Pc.z)), g.rdx)};
  R dy[4] = {A::mul(A::cv(__fsub_rn(Pc.x, Pym.x)), g.rdy), A::mul(A::cv(__fsub_rn(Pc.y, Pym.y)), g.rdy),
             A::mul(A::cv(__fsub_rn(Pc.z, Pym.z)), g.rdy), A::mul(A::cv(__fsub_rn(Pc.w, Pym.w)), g.rdy)};
  R dz[4] = {A::mul(A::cv(__fsub_rn(Pc.x, Pzm.x)), g.rdz), A::mul(A::cv(__fsub_rn(Pc.y, Pzm.y)), g.rdz),
             A::mul(A::cv(__fsub_rn(Pc.z, Pzm.z)), g.rdz), A::mul(A::cv(__fsub_rn(Pc.w, Pzm.w)), g.rdz)};
  if (vcpml) {
    if (q.bits & 0xF0000u) {
      const float4 a4 = ld4(Q.xva + 4 + 4 * (q.x0 / 4 % 16)), b4 = ld4(Q.xvb + 4 + 4 * (q.x0 / 4 % 16));
      const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
      if (q.bits & (1u << 20)) {
        x_slabs_narrow<R>(dx, Q, 3, S.nvp, S.psi_v_side[0], S.xs1v, S.npml + 1, k * S.ny + q.j, q.x0,
                          q.bits >> 16, true, a, b);
      } else {
        const uint32_t o = q.vx + k * Q.stride[3];
        const float4 t = mx;
        float m[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if ((q.bits >> (16 + e)) & 1u) cpml_apply<R>(dx[e], m[e], a[e], b[e]);
        Q.wr[3][o] = make_float4(m[0], m[1], m[2], m[3]);
      }
    }
    if (q.vy != kNoSlab) {
      const uint32_t o = q.vy + k * Q.stride[4];
      const float4 t = Q.rd[4][o];
      float m[4] = {t.x, t.y, t.z, t.w};
      const float a = Q.yva[q.r], b = Q.yvb[q.r];
#pragma unroll
      for (int e = 0; e < 4; ++e) cpml_apply<R>(dy[e], m[e], a, b);
      if (in != 15u) keep_rest(m, t, in);
      Q.wr[4][o] = make_float4(m[0], m[1], m[2], m[3]);
    }
    if (Q.zv[u] != kNoSlab && (q.bits & (1u << 22))) {
      const uint32_t o = Q.zv[u] + ((uint32_t)(q.j * S.nxp + q.x0) >> 2);
      const float4 t = Q.rd[5][o];
      float m[4] = {t.x, t.y, t.z, t.w};
      const float a = Q.zva[u], b = Q.zvb[u];
#pragma unroll
      for (int e = 0; e < 4; ++e) cpml_apply<R>(dz[e], m[e], a, b);
      if (in != 15u) keep_rest(m, t, in);
      Q.wr[5][o] = make_float4(m[0], m[1], m[2], m[3]);
    }
  }
  const uint32_t ux = (q.bits >> 4) & 15u, uy = q.j >= 1 ? in : 0u, uz = k >= 1 ? in : 0u;
  const float Vx[4] = {VX.x, VX.y, VX.z, VX.w}, Vy[4] = {VY.x, VY.y, VY.z, VY.w},
              Vz[4] = {VZ.x, VZ.y, VZ.z, VZ.w};
  float ox[4], oy[4], oz[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float nxv = A::rn(A::sub(A::cv(Vx[e]), A::mul(g.fv, dx[e])));
    const float nyv = A::rn(A::sub(A::cv(Vy[e]), A::mul(g.fv, dy[e])));
    const float nzv = A::rn(A::sub(A::cv(Vz[e]), A::mul(g.fv, dz[e])));
    ox[e] = ((ux >> e) & (nib >> (4 * e + 1)) & 1u) ? nxv : Vx[e];
    oy[e] = ((uy >> e) & (nib >> (4 * e + 2)) & 1u) ? nyv : Vy[e];
    oz[e] = ((uz >> e) & (nib >> (4 * e + 3)) & 1u) ? nzv : Vz[e];
  }
  vxo = make_float4(ox[0], ox[1], ox[2], ox[3]);
  vyo = make_float4(oy[0], oy[1], oy[2], oy[3]);
  vzo = make_float4(oz[0], oz[1], oz[2], oz[3]);
}

// ---------------------------------------------------------------------------
// interp_trilinear! entries of one (y tile, plane, channel) bucket
// (derivatives.jl:30-60).  Segments are cells {x | row << 9 | n << 16};
// inside a cell the entries are in transceiver order: rec += w*f (stored per
// entry, summed by the epilogue in corner order), then f += w*src[it].  The
// CTA handles the cells of its x range [x_lo, x_hi) and records only those
// it owns (row >= 1, x >= xb; the P bucket also carries the tile's halo row
// with slot -1).  Cell (row, x) is base[row * pitch + x] in shared memory.
// Out of line: few planes carry entries, and inlined its address arithmetic
// is hoisted into every plane of the step loop.
// ---------------------------------------------------------------------------
__device__ __noinline__ void apply_entries(const SolveDev& S, int T, int k, int chan, int x_lo,
                                           int x_hi, int xb, bool records, int it, float* base,
                                           int pitch) {
  const int* tp = S.tp_off + ((long long)T * S.nz + k) * 4 + chan;
  const int b = __ldg(tp), e = __ldg(tp + 1);
  const int tid = threadIdx.y * 32 + threadIdx.x, nthr = blockDim.x * blockDim.y;
  const float* src = S.src[chan] + (long long)(it - 1) * S.src_ntx;
  for (int si = b + tid; si < e; si += nthr) {
    const int4 sg = __ldg(S.seg + si);
    const int x = sg.x & 0x1FF, r = (sg.x >> 9) & 0x7F, cnt = (int)((unsigned)sg.x >> 16);
    if (x < x_lo || x >= x_hi) continue;
    const bool rec = records && r >= 1 && x >= xb;
    float* c = base + r * pitch + x;
    float v = *c;
    if (cnt == 1) {
      const float w = __int_as_float(sg.y);
      if (rec && sg.z >= 0) S.contrib[sg.z] = __fmul_rn(w, v);
      if (sg.w >= 0) v = __fadd_rn(v, __fmul_rn(w, src[sg.w]));
    } else {
      for (int kk = sg.y; kk < sg.y + cnt; ++kk) {
        const float w = __ldg(S.ent_w + kk);
        const int slot = __ldg(S.ent_slot + kk);
        if (rec && slot >= 0) S.contrib[slot] = __fmul_rn(w, v);
        const int col = __ldg(S.ent_tx + kk);
        if (col >= 0) v = __fadd_rn(v, __fmul_rn(w, src[col]));  // receivers: src == 0
      }
    }
    *c = v;
  }
}

// ---- plain quads: every cell interior for its update (no rigid plane, no
// CPML slab, no grid edge); the same arithmetic as the general functions
// for such cells, without their conditions.
template <typename R>
__device__ __forceinline__ float p_plain(float P, float dx, float dy, float dz, const Sc<R>& g) {
  using A = Arith<R>;
  const R s = A::add(A::add(A::mul(A::cv(dx), g.rdx), A::mul(A::cv(dy), g.rdy)),
                     A::mul(A::cv(dz), g.rdz));
  return A::rn(A::sub(A::cv(P), A::mul(g.fq, s)));
}
template <typename R>
__device__ __forceinline__ float v_plain(float V, float dp, R rd, const Sc<R>& g) {
  using A = Arith<R>;
  return A::rn(A::sub(A::cv(V), A::mul(g.fv, A::mul(A::cv(dp), rd))));
}
template <typename R>
__device__ __forceinline__ float4 p_plain_quad(const Sc<R>& g, float4 P4, float4 X4, float X5,
                                               float4 Y0, float4 Y1, float4 Z0, float4 Z1) {
  float4 n;
  n.x = p_plain<R>(P4.x, __fsub_rn(X4.y, X4.x), __fsub_rn(Y1.x, Y0.x), __fsub_rn(Z1.x, Z0.x), g);
  n.y = p_plain<R>(P4.y, __fsub_rn(X4.z, X4.y), __fsub_rn(Y1.y, Y0.y), __fsub_rn(Z1.y, Z0.y), g);
  n.z = p_plain<R>(P4.z, __fsub_rn(X4.w, X4.z), __fsub_rn(Y1.z, Y0.z), __fsub_rn(Z1.z, Z0.z), g);
  n.w = p_plain<R>(P4.w, __fsub_rn(X5, X4.w), __fsub_rn(Y1.w, Y0.w), __fsub_rn(Z1.w, Z0.w), g);
  return n;
}
template <typename R>
__device__ __forceinline__ void v_plain_quad(const Sc<R>& g, float4 Pc, float Pxm, float4 Pym,
                                             float4 Pzm, float4 VX, float4 VY, float4 VZ,
                                             float4& vx, float4& vy, float4& vz) {
  vx.x = v_plain<R>(VX.x, __fsub_rn(Pc.x, Pxm), g.rdx, g);
  vx.y = v_plain<R>(VX.y, __fsub_rn(Pc.y, Pc.x), g.rdx, g);
  vx.z = v_plain<R>(VX.z, __fsub_rn(Pc.z, Pc.y), g.rdx, g);
  vx.w = v_plain<R>(VX.w, __fsub_rn(Pc.w, Pc.z), g.rdx, g);
  vy.x = v_plain<R>(VY.x, __fsub_rn(Pc.x, Pym.x), g.rdy, g);
  vy.y = v_plain<R>(VY.y, __fsub_rn(Pc.y, Pym.y), g.rdy, g);
  vy.z = v_plain<R>(VY.z, __fsub_rn(Pc.z, Pym.z), g.rdy, g);
  vy.w = v_plain<R>(VY.w, __fsub_rn(Pc.w, Pym.w), g.rdy, g);
  vz.x = v_plain<R>(VZ.x, __fsub_rn(Pc.x, Pzm.x), g.rdz, g);
  vz.y = v_plain<R>(VZ.y, __fsub_rn(Pc.y, Pzm.y), g.rdz, g);
  vz.z = v_plain<R>(VZ.z, __fsub_rn(Pc.z, Pzm.z), g.rdz, g);
  vz.w = v_plain<R>(VZ.w, __fsub_rn(Pc.w, Pzm.w), g.rdz, g);
}

// ---------------------------------------------------------------------------
// The step kernel.  One CTA per work item {solve, y tile | x tile << 16, z0,
// z1}: a tile of ty <= 7 rows j0..j0+ty-1 and the kXT = 64 cells
// xb..xb+63 of one solve, and the planes z0..z1-1.  blockDim = (32, 4): warp
// w holds the 4 quads 4w..4w+3 (16 cells) of all 8 tile rows
// r = j - j0 + 1 = 0..7 (lane = 4r + quad).  Row r = 0 is the halo row
// j0-1, whose new P the Vy update of row j0 needs: it is recomputed, not
// exchanged.  The lanes of quad 0 also recompute the halo column x = xb-1
// (for Vx at xb).  With this shape the x-slab quads of a grid sit in one
// warp of each x-edge tile and the tiles between hold none, so few warps
// take the CPML branch and few CTAs wait for such a warp at their barrier.
// Per plane, after a prologue plane z0-1 (new P only, for Vz at z0) when
// z0 > 0:
//   loads  : P, Vx, Vy of plane k and Vz of plane k+1 (Vz of plane k and the
//            new P of plane k-1 are carried in registers), 128-bit, coalesced;
//   P      : new P into a double-buffered shared plane; barrier;
//   q      : injection/recording on P (only planes with entries; barrier);
//   V      : Vx/Vy/Vz from the new P (x-1 and y-1 neighbours from shared
//            memory);
//   f      : injection/recording on V (only planes with entries: staged in
//            shared memory between two barriers);
//   stores : 128-bit stores of the four channels and the rigid mirrors.
// A warp whose quads are all plain for this plane (the bulk of the grid)
// takes the plain functions (warp-uniform branch); the rest the general
// ones.  Several CTAs per SM keep enough independent warps in flight to
// cover the latency of the float/double chains and of HBM.
// ---------------------------------------------------------------------------
constexpr int kMaxTy = 7;           // rows per tile (plus the halo row: 8 per warp)
constexpr int kXT = 64;             // cells per x tile (4 warps)
constexpr int kPnPitch = kStageW;   // shared new-P row: [3] = halo column, [4..] = cells
constexpr int kStepThreads = 32 * kXT / 16;  // warps of 4 quads x 8 rows

// One stage: P, Vx, Vy of a plane ([3][kMaxTy+2][kStageW]) and, from the next
// 128-B boundary on (TMA destinations must be 128-B aligned), Vz of the next
// plane ([kMaxTy+2][kStageW]).  The rows are those of the tallest tile, so that
// every offset in a stage is a constant.
constexpr int kStageChan = (kMaxTy + 2) * kStageW;
constexpr int kStageVz = (3 * kStageChan + 31) / 32 * 32;
constexpr int kStageFloats = (kStageVz + kStageChan + 31) / 32 * 32;
// Polls of a staged plane's bounded wait: a plane lands within microseconds,
// so a limit far below kWaitLimit keeps a lost copy from stalling the GPU
constexpr uint32_t kStepWaitLimit = 1u << 20;
static_assert((kStageFloats * 4) % 128 == 0, "stages stay 128-B aligned");

// Fetches plane k's slab memory of the item into L2, a warp to a plane (slab_piece says
// what each lane takes).  A boundary warp waits for reads of slab
// memory that nothing has touched since the last step, and its length sets its CTA's
// pace.  Launches in us, without this, with the y and z slabs, with the x slabs too:
//   8 x 256^3, CPML 1109 1064 1040; and a sphere 1259 1224 1209; 2 x 256^3 334 325 321;
//   256^3 168 164 162; 512^3 1009 976 965; 224^3 135 132 131; 192^3 94.4 92.6 92.4
// A small solve alone keeps its memory in L2 and loses (128^3 37.0 and 38.3, 96^3 26.9
// and 27.4, y and z slabs), so it is for solves of 2^22 cells and more, the x slabs,
// which are read a phase ahead anyway, for 2^24.  The line looks at one solve, not at
// the launch: batches of small solves lie on its wrong side (8 x 128^3 195 and 190,
// 30 x 96^3 398 and 381, 4 x 160^3 194 and 188).  Out of line, as apply_entries is.
constexpr long long kFetchCells = 1 << 22, kFetchXCells = 1 << 24;
__device__ __noinline__ void fetch_slabs(const SolveDev& S, const PmlTab& Q, int4 item, int kfirst,
                                         int k) {
  if (k >= item.w) return;
  const SlabPiece f = slab_piece(S, item.y >> 16, item.y & 0xFFFF, kXT, threadIdx.x, k,
                                 S.chan_stride >= kFetchXCells, Q.zp[k - kfirst], Q.zv[k - kfirst]);
  const float* p = slab_cell(Q.rd[f.array], f.quad, 0);
#pragma unroll 2
  for (int i = 0; i < f.floats; i += 32) prefetch_l2(p + i);  // a line each
}

// One thread: the copies of plane k's stage into a free slot.
__device__ __forceinline__ void stage_plane(const char* maps, float* slot, uint64_t* bar, int xb,
                                            int j0, int k, int nz) {
  const uint32_t b = smem_u32(bar);
  const bool vz = k + 1 < nz;
  mbar_expect_tx(b, (uint32_t)((vz ? 16 : 12) * kStageChan));
  tma_load_4d(smem_u32(slot), maps, xb - 4, j0 - 1, k, 0, b);
  if (vz) tma_load_4d(smem_u32(slot + kStageVz), maps + 128, xb - 4, j0 - 1, k + 1, 3, b);
}

template <typename R>
__device__ __forceinline__ void step_item(const SolveDev& S, const PmlTab& Q, int4 item, int it,
                                          float* sPn, float* sV, float* ring,
                                          const unsigned char* s_fl, uint64_t* rbar) {
  const int lane = threadIdx.x, wid = threadIdx.y;
  const int tid = wid * 32 + lane;
  const int nx = S.nx, ny = S.ny, nz = S.nz, nxp = S.nxp, ty = S.ty, npml = S.npml;
  const int T = item.y & 0xFFFF, X = item.y >> 16;
  const int j0 = T * ty, xb = X * kXT;
  // this thread's tile row r (0 = halo row) and quad qx; its warp's quads
  // (rows in the order 0 2 1 3 4 6 5 7: the eight quads of a 128-bit access are
  // two rows 144 floats apart, which lie on different banks)
  const int rq = lane >> 2;
  const int qx = 4 * wid + (lane & 3), r = (rq & 4) | ((rq & 1) << 1) | ((rq >> 1) & 1);
  const int wq0 = 4 * wid, wnq = 4, wr0 = 0, wnr = kMaxTy + 1;
  const int j = j0 - 1 + r, x0 = xb + 4 * qx;
  const bool row_ok = r <= ty && j >= 0 && j < ny;
  // this thread's quad lies in the grid; the others compute on the stage's zeros
  // (every shared address is valid) and touch no global memory
  const bool act = row_ok && x0 < nxp;
  const bool vrow = act && r >= 1;      // ... and owns it (velocity update, stores)
  const int rb = (it - S.it_first) & 1, wb = rb ^ 1;
  const long long cs = S.chan_stride;
  const int plane = ny * nxp;
  float* fout = S.field + wb * S.buf_stride;
  const bool pcp = (S.flags & SF_PCPML) != 0, vcp = (S.flags & SF_VCPML) != 0;
  Quad q;
  q.j = j;
  q.x0 = x0;
  q.r = r;
  q.bits = 0;
  q.px = q.vx = 0;
  q.py = q.vy = kNoSlab;
  {
    int seen = 0;  // x slabs that the quad's cells lie in: 1 left, 2 right
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int x = x0 + e;
      if (x <= nx - 2) q.bits |= 1u << e;
      if (x >= 1 && x < nx) q.bits |= 16u << e;
      if (x < nx) q.bits |= 256u << e;
      if (act && pcp && x <= nx - 2 && (x < npml || x >= nx - npml)) {
        q.bits |= 4096u << e;
        seen |= x < npml ? 1 : 2;
      }
      if (vrow && vcp && x >= 1 && x < nx && (x <= npml || x >= nx - npml - 1)) {
        q.bits |= 65536u << e;
        seen |= x <= npml ? 4 : 8;
      }
    }
    if ((seen & 3) == 3 || (seen & 12) == 12) q.bits |= 1u << 20;
    if (act) q.bits |= 1u << 21;
    if (vrow) q.bits |= 1u << 22;
    if (act && pcp) {
      const int right = !(seen & 1);
      q.px = slab_quad(S.psi_p_side[0], right, j, S.npp, right ? x0 - S.xs1p : x0);
      const int ys = j < npml ? 0 : (j >= ny - npml ? 1 : -1);
      if (ys >= 0) q.py = slab_quad(S.psi_p_side[1], ys, ys == 0 ? j : j - (ny - npml), nxp, x0);
    }
    if (vrow && vcp) {
      const int right = !(seen & 4);
      q.vx = slab_quad(S.psi_v_side[0], right, j, S.nvp, right ? x0 - S.xs1v : x0);
      const int ys = j < 1 ? -1 : (j <= npml ? 0 : (j >= ny - npml - 1 ? 1 : -1));
      if (ys >= 0) q.vy = slab_quad(S.psi_v_side[1], ys, ys == 0 ? j : j - (ny - npml - 1), nxp, x0);
    }
  }
  // warp-uniform: do all of the warp's rows and x cells take the plain P
  // (and, rows >= 1, V) updates?  The plane is checked per plane below.
  bool wplain_rx, hplain_x;
  {
    const int wj0 = j0 - 1 + wr0, wj1 = wj0 + wnr - 1;  // rows: P on all, V from wj0 + 1
    const int wx0 = xb + 4 * wq0, wx1 = wx0 + 4 * wnq - 1;
    const int p_xmin = pcp ? npml : 0, p_xmax = pcp ? min(nx - 2, nx - npml - 1) : nx - 2;
    const int v_xmin = vcp ? npml + 1 : 1, v_xmax = vcp ? nx - npml - 2 : nx - 1;
    bool ok = wr0 + wnr - 1 <= ty && wj0 >= 0 && wx1 < nxp;
    ok = ok && wj1 < ny - 1 && (!pcp || (wj0 >= npml && wj1 < ny - npml));
    ok = ok && wx0 >= p_xmin && wx1 <= p_xmax;
    ok = ok && wj0 + 1 >= 1 && (!vcp || (wj0 + 1 > npml && wj1 < ny - npml - 1));
    ok = ok && wx0 >= v_xmin && wx1 <= v_xmax;
    wplain_rx = ok;
    hplain_x = xb - 1 >= p_xmin && xb - 1 <= p_xmax;  // the halo column's cells
  }
  const int rowoff = (row_ok ? j : 0) * nxp + x0;
  const int pq = r * kPnPitch + 4 + 4 * qx;  // this quad in a shared new-P plane
  const int z0 = item.z, z1 = item.w;
  const int kfirst = z0 > 0 ? z0 - 1 : z0;
  // The stage of plane k, staged by TMA into a ring of kStepRing slots, holds
  // P, Vx, Vy of plane k and Vz of plane k+1 (channel slot 3; not loaded for
  // k = nz-1, whose update does not read it), rows j0-1 .. j0+kMaxTy,
  // x = xb-4 .. xb+67, zero outside the grid.  Vz of plane k is carried in
  // registers from the previous stage.
  // (The kernel has issued the item's first planes.)
  constexpr int cst = kStageChan, vzo = kStageVz;
  const int so = r * kStageW + 4 + 4 * qx;    // this quad in a stage channel
  const char* maps = static_cast<const char*>(S.fmap) + rb * 256;  // {P,Vx,Vy box; Vz box}
  auto slot_of = [&](int k) { return (k - kfirst) % kStepRing; };
  auto issue = [&](int k) {  // one thread
    const int sl = slot_of(k);
    fence_proxy_async_smem();  // the slot was last read through the generic proxy
    stage_plane(maps, ring + sl * kStageFloats, rbar + sl, xb, j0, k, nz);
  };
  auto wait = [&](int k) {
    const int u = k - kfirst;
    if (!mbar_wait(smem_u32(rbar + u % kStepRing), (uint32_t)(u / kStepRing) & 1u, kStepWaitLimit))
      atomicOr(S.err, 4);  // reported as ADF_E_TIMEOUT; the values read are wrong
  };
  // Vz of plane kfirst (the stages carry the next plane's), and of the halo
  // column for its single-cell update
  float4 Z0 = make_float4(0.f, 0.f, 0.f, 0.f), Pzm = Z0;
  const bool hcol = qx == 0 && r >= 1 && row_ok && xb > 0;
  float Zh = 0.f;
  {
    const float* vz0 = S.field + rb * S.buf_stride + 3 * cs + (long long)kfirst * plane + rowoff;
    if (act) Z0 = ld4(vz0);
    if (hcol) Zh = vz0[-1];
  }
  // The x-slab memory of a quad is read ahead of its use: the p side's of plane
  // k+1 during the velocity update of plane k, the v side's of plane k during its
  // pressure update.  One warp of every x-end tile would otherwise wait for two
  // more reads of global memory per plane than the other three: without this
  // 8 x 256^3 with CPML and a sphere takes 1241 us (1209), 8 x 96^3 137 (125),
  // 192^3 100 (93); 8 x 256^3 without CPML is 2 % faster (735, 748).
  const bool pxm = (q.bits & 0xF000u) && !(q.bits & (1u << 20));
  const bool vxm = (q.bits & 0xF0000u) && !(q.bits & (1u << 20));
  float4 mpx = make_float4(0.f, 0.f, 0.f, 0.f), mvx = mpx;
  if (pxm) mpx = Q.rd[0][q.px + kfirst * Q.stride[0]];
  for (int k = kfirst; k < z1; ++k) {
    const bool prologue = k < z0;
    if (vxm) mvx = Q.rd[3][q.vx + k * Q.stride[3]];
    const int u = k - kfirst;
    float* pn = sPn + (k & 1) * (kMaxTy + 1) * kPnPitch;
    const float* st = ring + slot_of(k) * kStageFloats;
    if (!mbar_try_wait(smem_u32(rbar + (uint32_t)u % kStepRing), (uint32_t)u / kStepRing & 1u)) wait(k);
    const int fl = s_fl[u];
    const bool has_mask = (fl & 4) != 0;  // elsewhere every cell of the tile's plane is open
    const bool wplain = wplain_rx && (fl & 12) == 8;
    uint32_t nib = 0xFFFFu;
    Sc<R> g;  // (read again in each phase: registers are what the loop is short of)
    g.fq = Arith<R>::fq(S);
    g.fv = Arith<R>::fv(S);
    g.rdx = Arith<R>::rdx(S);
    g.rdy = Arith<R>::rdy(S);
    g.rdz = Arith<R>::rdz(S);
    const float4 P4 = ld4(st + so);
    const float4 X4 = ld4(st + cst + so);
    const float4 Y0 = ld4(st + 2 * cst + so);
    const float X5 = st[cst + so + 4];
    const float4 Y1 = ld4(st + 2 * cst + so + kStageW);
    const float4 Z1 = ld4(st + vzo + so);
    if (has_mask && act)
      nib = (__ldg(S.mask_bits + ((long long)k * ny + j) * S.mw + (x0 >> 3)) >> ((x0 & 4) * 4)) &
            0xFFFFu;
    float4 Pn;
    if (wplain)
      Pn = p_plain_quad<R>(g, P4, X4, X5, Y0, Y1, Z0, Z1);
    else
      Pn = p_update_quad<R>(S, Q, q, g, pcp, k, u, vrow && !prologue, P4, X4, X5, Y0, Y1, Z0, Z1, nib,
                            mpx);
    st4(pn + pq, Pn);
    if (hcol) {
      const float Zh1 = st[vzo + so - 1];
      if (wplain && hplain_x)
        pn[pq - 1] = p_plain<R>(st[so - 1], __fsub_rn(X4.x, st[cst + so - 1]),
                                __fsub_rn(st[2 * cst + so - 1 + kStageW], st[2 * cst + so - 1]),
                                __fsub_rn(Zh1, Zh), g);
      else
        pn[pq - 1] = p_update_cell<R>(S, Q, q, g, pcp, st, Zh, Zh1, so - 1, cst, k, u, has_mask);
      Zh = Zh1;
    }
    __syncthreads();
    if (pxm && k + 1 < z1) mpx = Q.rd[0][q.px + (k + 1) * Q.stride[0]];
    // every read of plane k's stage is done: refill its slot
    if (tid == 0 && k + kStepRing < z1) issue(k + kStepRing);
    // ---- q channel: inject/record on the new P (forward.jl:92) ----
    if (fl & 1) {
      apply_entries(S, T, k, 0, xb - 1, xb + kXT, xb, !prologue, it, pn + 4 - xb, kPnPitch);
      __syncthreads();
      Pn = ld4(pn + pq);
    }
    if (!prologue) {
      float4 vx, vy, vz;
      Sc<R> g;
      g.fq = Arith<R>::fq(S);
      g.fv = Arith<R>::fv(S);
      g.rdx = Arith<R>::rdx(S);
      g.rdy = Arith<R>::rdy(S);
      g.rdz = Arith<R>::rdz(S);
      const float Pxm = pn[pq - 1];
      const float4 Pym = ld4(pn + pq - kPnPitch);
      if (wplain)
        v_plain_quad<R>(g, Pn, Pxm, Pym, Pzm, X4, Y0, Z0, vx, vy, vz);
      else
        v_update_quad<R>(S, Q, q, g, vcp, k, u, Pn, Pxm, Pym, Pzm, X4, Y0, Z0, nib, mvx, vx, vy, vz);
      // ---- f channel: inject/record on the new V (forward.jl:111-115) ----
      if (fl & 2) {
        float* sVx = sV;
        float* sVy = sV + kMaxTy * kXT;
        float* sVz = sV + 2 * kMaxTy * kXT;
        const int so = (r - 1) * kXT + 4 * qx;
        if (vrow) {
          st4(sVx + so, vx);
          st4(sVy + so, vy);
          st4(sVz + so, vz);
        }
        __syncthreads();
        for (int c = 1; c <= 3; ++c)
          apply_entries(S, T, k, c, xb, xb + kXT, xb, true, it,
                        sV + (c - 1) * kMaxTy * kXT - kXT - xb, kXT);
        __syncthreads();
        if (vrow) {
          vx = ld4(sVx + so);
          vy = ld4(sVy + so);
          vz = ld4(sVz + so);
        }
      }
      if (vrow) {
        float* o = fout + ((long long)k * plane + rowoff);
        stcs4(o, Pn);
        stcs4(o + cs, vx);
        if (wplain) {
          stcs4(o + 2 * cs, vy);
          stcs4(o + 3 * cs, vz);
        } else {
          // rigid mirrors (forward.jl:134-137): Vy[:,1,:] = -Vy[:,2,:], Vz[:,:,1] = -Vz[:,:,2]
          if (j != 0) stcs4(o + 2 * cs, vy);
          if (j == 1) st4(o + 2 * cs - nxp, neg4(vy));
          if (k != 0) stcs4(o + 3 * cs, vz);
          if (k == 1) st4(o + 3 * cs - plane, neg4(vz));
        }
      }
    }
    if (fl & 16) fetch_slabs(S, Q, item, kfirst, k + 1 + wid);
    Pzm = Pn;
    Z0 = Z1;
  }
}

// Fills the item's table: coefficients of cells in no slab are never read.
__device__ __forceinline__ void pml_table(const SolveDev& G, PmlTab& Q, int4 item, int it, int kfirst,
                                          int tid, int nthr) {
  const int n = G.npml, nb = 4 * n + 2;
  if (n == 0) {
    for (int u = tid; u < item.w - kfirst; u += nthr) Q.zp[u] = Q.zv[u] = kNoSlab;
    return;
  }
  const float* co = G.coef;
  if (tid < 6) {
    const int a = tid % 3, rb = (it - G.it_first) & 1;
    const bool v = tid >= 3;
    float* base = v ? G.psi_v[a] : G.psi_p[a];
    const long long buf = v ? G.psi_v_buf[a] : G.psi_p_buf[a];
    Q.rd[tid] = reinterpret_cast<const float4*>(base + rb * buf);
    Q.wr[tid] = reinterpret_cast<float4*>(base + (rb ^ 1) * buf);
    Q.stride[tid] = a == 0 ? slab_quad(0, 0, G.ny, v ? G.nvp : G.npp, 0)
                           : slab_quad(0, 0, n + (v ? 1 : 0), G.nxp, 0);
  }
  if (tid == 6) {
    const int x = (item.y >> 16) * kXT - 1, right = x >= n;
    Q.hx = x < 0 || (right && x < G.nx - n) ? kNoSlab
                                            : slab_quad(G.psi_p_side[0], right, 0, G.npp,
                                                        right ? x - G.xs1p : x);
  }
  // index of the coefficient of cell x of an axis of m cells, -1: no slab
  auto cp = [&](int x, int m) { return x < 0 || x >= m ? -1 : x < n ? x : (x >= m - n ? n + x - (m - n) : -1); };
  auto cv = [&](int x, int m) {
    return x < 0 || x >= m ? -1 : x <= n ? 2 * n + x : (x >= m - n - 1 ? 3 * n + 1 + x - (m - n - 1) : -1);
  };
  // the halo column's and the tile's 65 columns, 8 rows and the item's planes, one to
  // a thread, so that their reads go out together
  const int xb = (item.y >> 16) * kXT, j0 = (item.y & 0xFFFF) * G.ty, np = item.w - kfirst;
  for (int i = tid; i < 73 + np; i += nthr) {
    int x, m, e;
    float *pa, *pb, *va, *vb;
    if (i < 65) {
      x = xb - 1 + i, m = G.nx, e = 3 + i;
      pa = Q.xpa, pb = Q.xpb, va = Q.xva, vb = Q.xvb;
    } else if (i < 73) {
      e = i - 65, x = j0 - 1 + e, m = G.ny;
      pa = Q.ypa, pb = Q.ypb, va = Q.yva, vb = Q.yvb;
    } else {
      e = i - 73, x = kfirst + e, m = G.nz;
      pa = Q.zpa, pb = Q.zpb, va = Q.zva, vb = Q.zvb;
    }
    const int c = cp(x, m), v = i >= 73 && x < 1 ? -1 : cv(x, m);
    const int c0 = max(c, 0), v0 = max(v, 0);
    const float ca = co[c0], cb = co[nb + c0], wa = co[v0], wb = co[nb + v0];
    if (i >= 73) {
      const int top = c >= n, vtop = v >= 3 * n + 1;
      Q.zp[e] = c < 0 ? kNoSlab
                      : slab_quad(G.psi_p_side[2], top, (top ? c - n : c) * G.ny, G.nxp, 0);
      Q.zv[e] = v < 0 ? kNoSlab
                      : slab_quad(G.psi_v_side[2], vtop, (vtop ? v - 3 * n - 1 : v - 2 * n) * G.ny,
                                  G.nxp, 0);
    }
    pa[e] = ca, pb[e] = cb, va[e] = wa, vb[e] = wb;
  }
}

// Shared memory: the staged-plane ring (dynamic, kStepRing * kStageFloats
// floats) plus the new-P planes, the f-channel staging and the descriptor:
// 34.3 KB per CTA; five CTAs per SM (the register budget: 102 per thread,
// no spills; six CTAs at 80 registers spill and measured slower).
#ifndef ADF_STEP_CTAS_PER_SM
#define ADF_STEP_CTAS_PER_SM 5
#endif
constexpr int kStepCtasPerSm = ADF_STEP_CTAS_PER_SM;  // register budget: 65536 / (128 x this)
// (+128 B so that the ring can start on a 128-B boundary, as TMA destinations must)
constexpr size_t kStepDynSmem = sizeof(float) * kStepRing * kStageFloats + 128;

__global__ void __launch_bounds__(kStepThreads, kStepCtasPerSm) adf_fdtd_step_kernel(const StepParams p) {
  extern __shared__ __align__(128) float dyn_smem[];
  // (an index, not a rounded pointer, so that the compiler keeps shared-space accesses)
  float* ring = dyn_smem + ((0u - smem_u32(dyn_smem)) & 127u) / 4u;
  __shared__ __align__(8) uint64_t rbar[kStepRing];
  __shared__ __align__(16) float sPn[(2 * (kMaxTy + 1) + 1) * kPnPitch];  // (a row before the first)
  __shared__ __align__(16) float sV[3 * kMaxTy * kXT];
  __shared__ __align__(16) PmlTab Q;
  __shared__ unsigned char s_fl[kMaxZc + 1];  // planes kfirst ..: 1 q, 2 f entries, 4 closed cells, 8 plain, 16 fetch_slabs
  __shared__ __align__(16) SolveDev S;  // the solve descriptor, read in the hot loop
  const int4 item = p.items[blockIdx.x];
  const SolveDev& G = p.solves[item.x];
  const int it = G.it_base + p.step;
  if (it > G.it_stop) {
    pdl_wait();  // this kernel is not over before those it depends on
    return;
  }
  // The first warp's first thread starts the copies of the item's first planes as soon
  // as it has their place; the other warps read the item's tables meanwhile.
  const int tid = threadIdx.y * 32 + threadIdx.x, kfirst = item.z > 0 ? item.z - 1 : 0;
  if (tid == 0) {
    for (int q = 0; q < kStepRing; ++q) mbar_init(smem_u32(rbar + q), 1);
    fence_mbar_init();
    const char* maps = static_cast<const char*>(G.fmap) + ((it - G.it_first) & 1) * 256;
    prefetch_tensormap(maps);
    prefetch_tensormap(maps + 128);
    const int j0 = (item.y & 0xFFFF) * G.ty, nz = G.nz;
    pdl_wait();
    for (int k = kfirst; k < min(item.w, kfirst + kStepRing); ++k)
      stage_plane(maps, ring + (k - kfirst) * kStageFloats, rbar + (k - kfirst), (item.y >> 16) * kXT,
                  j0, k, nz);
  } else if (tid >= 32) {
    const int t = tid - 32, nthr = kStepThreads - 32;
    const int* src = reinterpret_cast<const int*>(&G);
    int* dst = reinterpret_cast<int*>(&S);
    for (int w = t; w < (int)(sizeof(SolveDev) / 4); w += nthr) dst[w] = src[w];
    if (t < item.w - kfirst) {
      const int* tp = G.tp_off + ((long long)(item.y & 0xFFFF) * G.nz + kfirst + t) * 4;
      int f = (tp[0] < tp[1] ? 1 : 0) | (tp[1] < tp[4] ? 2 : 0);
      if (G.closed &&
          G.closed[((long long)(item.y >> 16) * G.nty + (item.y & 0xFFFF)) * G.nz + kfirst + t])
        f |= 4;
      // planes without z-slab memory, mirror or rigid wall
      const int zm = (G.flags & (SF_PCPML | SF_VCPML)) ? G.npml + 1 : 1, k = kfirst + t;
      if (k >= max(zm, 2) && k < G.nz - zm) f |= 8;
      // every fourth plane: do the next four have slab memory to fetch?
      if ((t & 3) == 0 && G.npml > 0 && G.chan_stride >= kFetchCells) {
        const int X = item.y >> 16, j0 = (item.y & 0xFFFF) * G.ty;
        if (j0 - 1 < zm || j0 + G.ty > G.ny - zm || k + 1 < zm || k + 4 >= G.nz - zm ||
            (G.chan_stride >= kFetchXCells && (X == 0 || (X + 1) * kXT >= G.nxp)))
          f |= 16;
      }
      s_fl[t] = (unsigned char)f;
    }
    pml_table(G, Q, item, it, kfirst, t, nthr);
  }
  // Up to the wait only the descriptors and tables of the set-up are read.  The field,
  // the sources and the records belong to the kernels before.
  pdl_wait();
  pdl_trigger();  // after the wait: one step's kernels start ahead, not a chain of them
  __syncthreads();
  if (S.flags & SF_FP32)
    step_item<float>(S, Q, item, it, sPn + kPnPitch, sV, ring, s_fl, rbar);
  else
    step_item<double>(S, Q, item, it, sPn + kPnPitch, sV, ring, s_fl, rbar);
}

// closed[x tile][y tile][plane] = 1 where a cell of the tile's plane, its halo
// row and column included, has a closed mask bit (set-up, once per mask): the
// step kernel reads the mask on those planes of a tile only, so that the rest
// of the grid has neither the load in the plane's chain nor the selects (read
// everywhere, 512^3 with an ellipsoid takes 1272 us a launch, 8 x 256^3 with a
// sphere 1411; so 965 and 1209).  One warp per (x, y, plane).
__global__ void adf_mask_tiles_kernel(const uint32_t* bits, int nx, int ny, int nz, int mw, int ty,
                                      int nty, int nxt, unsigned char* closed) {
  const long long t = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  if (t >= (long long)nxt * nty * nz) return;
  const int k = (int)(t % nz), T = (int)(t / nz % nty), X = (int)(t / nz / nty);
  const int lane = threadIdx.x & 31;
  bool shut = false;
  for (int r = lane >> 2; r <= ty; r += 8) {
    const int j = T * ty - 1 + r;
    if (j < 0 || j >= ny) continue;
    // words of cells xb-8 .. xb+63; nibbles past nx are zero in the mask and not cells
    for (int i = (X * kXT >> 3) - 1 + (lane & 3); i < (X + 1) * kXT >> 3; i += 4) {
      const int n = nx - 8 * i;  // cells of the word inside the grid
      if (i < 0 || n <= 0) continue;
      const uint32_t full = n >= 8 ? 0xFFFFFFFFu : (1u << (4 * n)) - 1u;
      shut = shut || (bits[((long long)k * ny + j) * mw + i] & full) != full;
    }
  }
  shut = __any_sync(0xffffffffu, shut);
  if (lane == 0) closed[t] = shut ? 1 : 0;
}

cudaError_t launch_mask_tiles(const SolveDev& d, unsigned char* closed, cudaStream_t s) {
  const int nxt = (d.nxp + kXT - 1) / kXT;
  const long long warps = (long long)nxt * d.nty * d.nz;
  adf_mask_tiles_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, s>>>(d.mask_bits, d.nx, d.ny, d.nz,
                                                                    d.mw, d.ty, d.nty, nxt, closed);
  return cudaGetLastError();
}

// Per-step trace assembly (derivatives.jl:51-56 record sums in corner order,
// v2vn! :85-90, vn2v! :92-97 into row it+1).  Four lanes per transceiver, one per
// channel: the kernel does next to nothing and its time is the chain of its reads
// (a thread per transceiver, through the descriptor in global memory and corner by
// corner, took 9.9 us cold between a step and the next, this 5.4).  Places are looked up
// before the wait for the step kernel; after it, one round of reads is left.
constexpr int kEpiThreads = 128;
__global__ void __launch_bounds__(kEpiThreads) adf_fdtd_epilogue_kernel(const EpiParams p) {
  pdl_trigger();
  const SolveDev& S = p.solves[blockIdx.y];
  const int c = threadIdx.x & 3, tx = (int)(blockIdx.x * kEpiThreads + threadIdx.x) >> 2;
  const int ntx = S.ntx, nt = S.nt, stop = S.it_stop;
  const bool on = tx < ntx;
  float* const rec = S.rec[c];
  float* const vn_rec = S.vn_rec;
  const float* const vn_src = S.vn_src;
  float* const src = S.src[c];
  const float4* const cb = reinterpret_cast<const float4*>(S.contrib + ((long long)c * ntx + tx) * 8);
  const bool inb = on && S.inb[c * ntx + tx];
  const float d = on ? S.dir[4 * tx + c] : 0.0f;
  // vn2v into row it+1; a GF solve's driven columns get it when the
  // extrapolation has written their vn_src (gf_finish)
  const bool v2 = on && c > 0 && vn_src && (!(S.flags & SF_GF) || S.gf_col[tx] == 0);
  pdl_wait();
  const int it = S.it_base + p.step;
  if (it > stop) return;
  const long long row = (long long)(it - 1) * ntx + tx;
  // a record buffer that is not kept starts every row at zero, as the
  // reference's freshly packed rec (= src*0) does
  float r = on && rec ? rec[row] : 0.0f;
  float vs = 0.0f, sv = 0.0f;
  if (v2 && it < nt) {
    vs = vn_src[row + ntx];
    sv = src[row + ntx];
  }
  if (inb) {
    const float4 lo = cb[0], hi = cb[1];
    r = __fadd_rn(r, lo.x);
    r = __fadd_rn(r, lo.y);
    r = __fadd_rn(r, lo.z);
    r = __fadd_rn(r, lo.w);
    r = __fadd_rn(r, hi.x);
    r = __fadd_rn(r, hi.y);
    r = __fadd_rn(r, hi.z);
    r = __fadd_rn(r, hi.w);
    if (rec) rec[row] = r;
  }
  // vn = rec1 d1 + rec2 d2 + rec3 d3, in that order
  const float m = __fmul_rn(r, d);
  const float m1 = __shfl_sync(0xffffffffu, m, (threadIdx.x & 28) + 1);
  const float m2 = __shfl_sync(0xffffffffu, m, (threadIdx.x & 28) + 2);
  const float m3 = __shfl_sync(0xffffffffu, m, (threadIdx.x & 28) + 3);
  if (on && c == 0) vn_rec[row] = __fadd_rn(__fadd_rn(m1, m2), m3);
  if (v2 && it < nt) src[row + ntx] = __fadd_rn(sv, __fmul_rn(vs, d));
}

// Advances it_base of every solve by `by` steps: the last node of a captured
// chunk of steps, so replaying the graph continues where it stopped.
// Completes source o of step it from its summed lags: adds the far lags
// summed at the block's start (block-causal kinds), writes the p_src and
// vn_src samples of row it+1 (extrapolation.jl:215-216, 228-229, 246-247)
// and applies vn2v! to the column.
__device__ __forceinline__ void gf_finish(const SolveDev& S, int o, int it, int step, double sa,
                                          double sb) {
  if (S.gf_rs > 0) {
    const double* pp = S.gf_far + ((long long)o * S.gf_rs * kGfBlock + step % kGfBlock) * 2;
    sa = __dadd_rn(sa, pp[0]);
    sb = __dadd_rn(sb, pp[1]);
  }
  const int col = S.gf_isrc[o];
  float ps, vs;
  if (S.gf_kind == ADF_GF_P_FROM_PIN_) {
    const float pos = (float)sa, neg = (float)sb;
    ps = (float)((double)__fadd_rn(pos, neg) / S.gf_z0);  // vn_src
    vs = __fsub_rn(pos, neg);                              // p_src
  } else {
    ps = (float)sa;  // vn_src <- p_pin / (pv, pp)-derived
    vs = (float)sb;  // p_src  <- v_pin / (vv, vp)-derived
  }
  S.src[0][(long long)it * S.src_ntx + col] = vs;
  S.vn_src[(long long)it * S.ntx + col] = ps;
  if (S.gf_col[col] == o + 1) {  // vn2v! of the column (derivatives.jl:92-97), once
    const long long nr = (long long)it * S.ntx + col;
    const float* d = S.dir + 4 * col;
#pragma unroll
    for (int c = 1; c <= 3; ++c) S.src[c][nr] = __fadd_rn(S.src[c][nr], __fmul_rn(ps, d[c]));
  }
}

// In-loop GF extrapolation, extrapolate! (src/kernels/extrapolation.jl:204-249)
// after v2vn! of step it < nt, for every driven source o:
//   PVFromPin (:139-170): pin[t, r] = (p_rec - z0 vn_rec)/2 (Float64);
//     ps/vs = sum_r sum_tt p_pin/v_pin[T-tt+1, o, r] * pin[it-T+tt, r];
//     p_src[it+1, iSrc[o]] = vs, vn_src[it+1, iSrc[o]] = ps.
//   PFromPin (:172-193, 237-249): pos/neg[o] = sums of pos/neg[., r, o] * pin,
//     rounded to Float32; p_src = pos - neg, vn_src = (pos + neg) / z0.
//   PVFromPV (:91-137, 204-218): ps += pv*p + pp*vn, vs += vv*p + vp*vn over
//     the recorded p / v_n of the iRec columns (Float32 terms).
// Sums are accumulated in Float64 (the Float32 zero of the reference is
// promoted by the first Float64 add for the *FromPin kinds).  The receiver
// range of each source is split over gf_ks blocks (blockIdx.x = o*ks + part)
// whose partial sums the reduce kernel adds in a fixed order; with one block
// per source (ks = 1) that block completes the source itself.  Rows before
// `it` of pin come from gf_pin; row `it` is formed here and block 0 files it.
__global__ void __launch_bounds__(256, 4) adf_gf_extrapolate_kernel(const EpiParams p) {
  pdl_trigger();
  pdl_wait();
  const SolveDev& S = p.solves[blockIdx.y];
  const int it = S.it_base + p.step;
  if (it > S.it_stop || it >= S.nt || !(S.flags & SF_GF)) return;
  const int ks = S.gf_ks;
  const int o = blockIdx.x / ks, part = blockIdx.x - (blockIdx.x / ks) * ks;
  if (o >= S.gf_nout) return;
  const int nt = S.nt, ntx = S.ntx, ngf = S.gf_nt, n1 = S.gf_n1, nin = S.gf_nin;
  const int kind = S.gf_kind;
  // lags 0..T-1 (T = min(it, ngf)); with blocking only 0..b, b = this step's place
  // in its sub-block, the older lags coming from adf_gf_mid_kernel and
  // adf_gf_far_kernel
  const int T = S.gf_rs > 0 ? min(min(it, ngf), p.step % kGfSub + 1) : min(it, ngf);
  const int t0 = it - T;  // 0-based row of tt = 1
  const long long cur = (long long)(it - 1) * ntx;
  auto pin_now = [&](int r) {
    const int col = S.gf_irec[r];
    return ((double)S.rec[0][cur + col] - (double)S.vn_rec[cur + col] * S.gf_z0) / 2.0;
  };
  double a = 0.0, b = 0.0;
  if (S.gf_near) {
    // blocked kinds (one block per source): lags 0..T-1 <= b from the
    // near-lag copy and the history ring, both receiver-major, so every lag
    // is one coalesced row of each; thread t sums receivers t, t+256, ...
    // Block 0 files row it-1 into the history and the ring; the other rows
    // come from earlier launches.
    const int nl = S.gf_nl;
    const float* g0 = S.gf_near + (long long)o * nl * nin;
    const float* g1 = g0 + (long long)S.gf_nout * nl * nin;
    for (int r = threadIdx.x; r < nin; r += blockDim.x) {
      const double h0 = pin_now(r);
      if (blockIdx.x == 0) {
        S.gf_pin[(long long)r * nt + (it - 1)] = h0;
        S.gf_ring[(long long)((it - 1) % kGfRing) * nin + r] = h0;
      }
      a = __fma_rn((double)g0[r], h0, a);
      b = __fma_rn((double)g1[r], h0, b);
#pragma unroll 4
      for (int lag = 1; lag < T; ++lag) {
        const double h = S.gf_ring[(long long)((it - 1 - lag) % kGfRing) * nin + r];
        a = __fma_rn((double)g0[(long long)lag * nin + r], h, a);
        b = __fma_rn((double)g1[(long long)lag * nin + r], h, b);
      }
    }
  } else {
  if (blockIdx.x == 0 && kind != ADF_GF_PV_FROM_PV_)
    for (int r = threadIdx.x; r < nin; r += blockDim.x)
      S.gf_pin[(long long)r * nt + (it - 1)] = pin_now(r);
  const int rb = (int)((long long)nin * part / ks), re = (int)((long long)nin * (part + 1) / ks);
  // (r, tt) walk over this block's receivers, tt fastest: contiguous tensor
  // and pin reads, the index stepped instead of divided.  GF_U elements per
  // round: all their loads are issued before the first is accumulated, so
  // each thread keeps GF_U loads in flight; the accumulation order of a
  // thread is the walk order either way.
  constexpr int GF_U = 4;
  int r = rb + (int)threadIdx.x / T, tt = (int)threadIdx.x - ((int)threadIdx.x / T) * T;
  const int step_r = (int)blockDim.x / T, step_t = (int)blockDim.x - step_r * T;
  const long long so = kind == ADF_GF_PV_FROM_PIN_ ? (long long)ngf * o : (long long)ngf * n1 * o;
  const long long sr = kind == ADF_GF_PV_FROM_PIN_ ? (long long)ngf * n1 : (long long)ngf;
  while (r < re) {
    int ru[GF_U], tu[GF_U];
#pragma unroll
    for (int u = 0; u < GF_U; ++u) {
      ru[u] = r;
      tu[u] = tt;
      r += step_r;
      tt += step_t;
      if (tt >= T) {
        tt -= T;
        ++r;
      }
    }
    if (kind == ADF_GF_PV_FROM_PV_) {
      float g0[GF_U], g1[GF_U], g2[GF_U], g3[GF_U], pt[GF_U], vt[GF_U];
#pragma unroll
      for (int u = 0; u < GF_U; ++u) {
        if (ru[u] < re) {
          // tensor element [T-tt, ., .] (1-based lag) for this receiver and output
          const long long g = (long long)(T - 1 - tu[u]) + so + sr * ru[u];
          const int col = S.gf_irec[ru[u]];
          const long long e = (long long)(t0 + tu[u]) * ntx + col;
          g0[u] = S.gf_t[0][g];
          g1[u] = S.gf_t[1][g];
          g2[u] = S.gf_t[2][g];
          g3[u] = S.gf_t[3][g];
          pt[u] = S.rec[0][e];
          vt[u] = S.vn_rec[e];
        }
      }
#pragma unroll
      for (int u = 0; u < GF_U; ++u) {
        if (ru[u] < re) {
          const float ps = __fadd_rn(__fmul_rn(g1[u], pt[u]), __fmul_rn(g0[u], vt[u]));
          const float vs = __fadd_rn(__fmul_rn(g3[u], pt[u]), __fmul_rn(g2[u], vt[u]));
          a = __dadd_rn(a, (double)ps);
          b = __dadd_rn(b, (double)vs);
        }
      }
    } else {
      float g0[GF_U], g1[GF_U];
      double pin[GF_U];
#pragma unroll
      for (int u = 0; u < GF_U; ++u) {
        if (ru[u] < re) {
          const long long g = (long long)(T - 1 - tu[u]) + so + sr * ru[u];
          const int row = t0 + tu[u];
          g0[u] = S.gf_t[0][g];
          g1[u] = S.gf_t[1][g];
          pin[u] = row == it - 1 ? pin_now(ru[u]) : S.gf_pin[(long long)ru[u] * nt + row];
        }
      }
#pragma unroll
      for (int u = 0; u < GF_U; ++u) {
        if (ru[u] < re) {
          a = __dadd_rn(a, __dmul_rn((double)g0[u], pin[u]));
          b = __dadd_rn(b, __dmul_rn((double)g1[u], pin[u]));
        }
      }
    }
  }
  }
  __shared__ double red[2][8];
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    a = __dadd_rn(a, __shfl_down_sync(0xffffffffu, a, w));
    b = __dadd_rn(b, __shfl_down_sync(0xffffffffu, b, w));
  }
  const int wi = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    red[0][wi] = a;
    red[1][wi] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double sa = 0.0, sb = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) {
      sa = __dadd_rn(sa, red[0][k]);
      sb = __dadd_rn(sb, red[1][k]);
    }
    if (ks == 1) {
      gf_finish(S, o, it, p.step, sa, sb);
    } else {
      double* pp = S.gf_part + ((long long)o * ks + part) * 2;
      pp[0] = sa;
      pp[1] = sb;
    }
  }
}

// The same split inside a block: at the first step it0 of a sub-block of kGfSub steps
// (not the block's first), the sb rows that the block has filed so far, for the
// sub-block's steps it0 .. it0+kGfSub-1.  Step it0+q reads row it0-1-i with lag q+i,
// i = 1 .. sb; lags 0..q stay in adf_gf_extrapolate_kernel.  The sums go on top of the
// far lags' (gf_finish adds them).  One block per source, threads over receivers; each
// walks the rows from the newest back, the 8 steps' tensor values one window that moves
// by a lag per row, so a lag is read once for 8 steps and not at each: the near-lag
// copy, up to 58 MB of a 512 x 448 map, is what a step's sum is bound by (L2).
// With all 32 lags in the step's sum it took 11.4 us on a 256 x 256 map and 17.3 on a
// 512 x 448 one, cold, now 9.3 and 12.2, plus 17 and 32 every 8 steps here.
constexpr int kGfMidThreads = 128;
__global__ void __launch_bounds__(kGfMidThreads) adf_gf_mid_kernel(const EpiParams p) {
  pdl_trigger();
  pdl_wait();
  const SolveDev& S = p.solves[blockIdx.y];
  const int it0 = S.it_base + p.step, o = blockIdx.x;
  if (S.gf_rs <= 0 || it0 > S.it_stop || it0 >= S.nt || !(S.flags & SF_GF) || o >= S.gf_nout) return;
  const int sb = p.step % kGfBlock, nl = S.gf_nl, nin = S.gf_nin;
  const float* const g0 = S.gf_near + (long long)o * nl * nin;
  const float* const g1 = g0 + (long long)S.gf_nout * nl * nin;
  double acc[2][kGfSub];
#pragma unroll
  for (int q = 0; q < kGfSub; ++q) acc[0][q] = acc[1][q] = 0.0;
  for (int r = threadIdx.x; r < nin; r += kGfMidThreads) {
    float w0[kGfSub], w1[kGfSub];  // lags i .. i+7 at row i; past the map unused
#pragma unroll
    for (int q = 0; q < kGfSub - 1; ++q) {
      const bool in = q + 1 < nl;
      w0[q + 1] = in ? g0[(long long)(q + 1) * nin + r] : 0.f;
      w1[q + 1] = in ? g1[(long long)(q + 1) * nin + r] : 0.f;
    }
    auto rows = [&](auto checked) {
#pragma unroll 4
      for (int i = 1; i <= sb; ++i) {
        const double h = S.gf_ring[(long long)((it0 - 1 - i) % kGfRing) * nin + r];
#pragma unroll
        for (int q = 0; q < kGfSub - 1; ++q) w0[q] = w0[q + 1], w1[q] = w1[q + 1];
        const int lag = i + kGfSub - 1;
        if (!decltype(checked)::value || lag < nl) {
          w0[kGfSub - 1] = g0[(long long)lag * nin + r];
          w1[kGfSub - 1] = g1[(long long)lag * nin + r];
        }
#pragma unroll
        for (int q = 0; q < kGfSub; ++q)
          if (!decltype(checked)::value || i + q < nl) {
            acc[0][q] = __fma_rn((double)w0[q], h, acc[0][q]);
            acc[1][q] = __fma_rn((double)w1[q], h, acc[1][q]);
          }
      }
    };
    if (sb + kGfSub <= nl)
      rows(std::false_type());
    else
      rows(std::true_type());
  }
  __shared__ double red[2][kGfSub][kGfMidThreads / 32];
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int q = 0; q < kGfSub; ++q) {
      double a = acc[t][q];
#pragma unroll
      for (int w = 16; w > 0; w >>= 1) a = __dadd_rn(a, __shfl_down_sync(0xffffffffu, a, w));
      if ((threadIdx.x & 31) == 0) red[t][q][threadIdx.x >> 5] = a;
    }
  __syncthreads();
  if (threadIdx.x >= 2 * kGfSub) return;
  const int t = threadIdx.x & 1, q = threadIdx.x >> 1;
  double a = 0.0;
  for (int w = 0; w < kGfMidThreads / 32; ++w) a = __dadd_rn(a, red[t][q][w]);
  double* pp = S.gf_far + ((long long)o * S.gf_rs * kGfBlock + sb + q) * 2 + t;
  *pp = __dadd_rn(*pp, a);
}

// Far-lag part of the in-loop GF extrapolation (extrapolation.jl:139-170),
// block-causal form.  For the block of kGfBlock steps it0 .. it0+B-1 that
// starts at this launch-step, step it0+b needs lags 0 .. T_b-1 of the map
// (T_b = min(it0+b, ngf)).  Lags b+1 .. T_b-1 read input-history rows
// it0-1+b-lag <= it0-2, all complete before the block starts, so they are
// summed here once for the whole block: a contraction over (receiver, lag)
// of the block's 32 steps x 64 sources, which reads each tensor slice once
// per block instead of once per step.  Lags 0..b, whose rows appear during
// the block, stay in the kernels above.  FP64 fused multiply-adds;
// one partial per (source, receiver split, step), added in split order by
// adf_gf_far_combine_kernel.  Input-history kinds only.
//
// Block: 64 sources; two groups of four warps, each with half of the block's
// receivers.  A thread holds 2 sources x 8 steps x 2 tensors, so
// that one staged lag costs it 4 tensor values and one new history value for 32
// FMAs (the 8 steps' history values are one window that moves by a row per lag):
// with 4 steps a thread the shared loads, not the FP64 pipe, were the bound, and
// nothing read the next chunk while one was summed.  256 x 256 x 256 map, lags to
// 255, cold: 245 us a block before, 128 here, 64 at the FP64 pipe's rate.
constexpr int kGfLC = 32;  // lags per staged chunk
constexpr int kGfOT = 64;  // sources per tile (two per thread)
constexpr int kGfGroup = 128;
struct GfFarStage {  // a chunk of one receiver
  float g[2][kGfLC][kGfOT + 1];  // the two tensors, lag-major, padded against conflicts
  double h[kGfLC + kGfBlock];    // history rows
};
// asynchronous copies of 4 and 8 bytes, zeros where !in
__device__ __forceinline__ void copy4(void* dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src),
               "r"(in ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void copy8(void* dst, const void* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src),
               "r"(in ? 8 : 0)
               : "memory");
}
constexpr size_t kGfFarSmem = 4 * sizeof(GfFarStage);  // two groups, two buffers each
static_assert(kGfFarSmem >= 32 * kGfGroup * sizeof(double), "the groups' exchange");
static_assert(sizeof(GfFarStage) % 16 == 0 && offsetof(GfFarStage, h) % 8 == 0, "aligned copies");
__global__ void __launch_bounds__(2 * kGfGroup, 2) adf_gf_far_kernel(const EpiParams p) {
  const SolveDev& S = p.solves[blockIdx.y];
  const int it0 = S.it_base + p.step;
  if (S.gf_rs <= 0 || it0 > S.it_stop || it0 >= S.nt || !(S.flags & SF_GF) || (S.flags & SF_GF_TC))
    return;  // (tensor-core solves: adf_gf_far_tc_kernel)
  const int rsn = S.gf_rs, nout = S.gf_nout;
  const int ot = blockIdx.x / rsn, rsi = blockIdx.x - ot * rsn;
  if (ot * kGfOT >= nout) return;
  const int nt = S.nt, ngf = S.gf_nt, n1 = S.gf_n1, nin = S.gf_nin;
  const bool pv = S.gf_kind == ADF_GF_PV_FROM_PIN_;
  const int grp = (int)threadIdx.x / kGfGroup, tid = (int)threadIdx.x % kGfGroup;
  // this group's half of the block's receivers
  const int r0 = (int)((long long)nin * (2 * rsi + grp) / (2 * rsn));
  const int r1 = (int)((long long)nin * (2 * rsi + grp + 1) / (2 * rsn));
  const int ol = tid & 31, b0 = 8 * (tid >> 5);  // sources ol and ol+32, steps b0 .. b0+7
  extern __shared__ __align__(16) unsigned char gf_smem[];
  GfFarStage* const stage = reinterpret_cast<GfFarStage*>(gf_smem) + 2 * grp;  // [buffer]
  double acc[2][2][8];  // tensor, source, step
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[t][h][q] = 0.0;
  const int lag_hi = min(it0 + kGfBlock - 1, ngf) - 1;  // largest lag any step of the block uses
  const int nch = (lag_hi + kGfLC - 1) / kGfLC;         // chunks of lags 1 .. lag_hi
  const int total = (r1 - r0) * nch;
  // chunk i: receiver r0 + i / nch, lags 1 + 32 (i % nch) ..; copied a chunk ahead,
  // the lane the lag, so that a source's 32 values are one coalesced row
  const int ll = tid & 31, ow = tid >> 5;
  auto fetch = [&](int i) {
    GfFarStage& d = stage[i & 1];
    const int r = r0 + i / nch, l0 = 1 + (i % nch) * kGfLC, lag = l0 + ll;
    const long long step = 4ll * (pv ? (long long)ngf : (long long)ngf * n1);
    long long g = lag + (pv ? (long long)ngf * (ot * kGfOT + ow + (long long)n1 * r)
                            : (long long)ngf * (r + (long long)n1 * (ot * kGfOT + ow)));
#pragma unroll 4
    for (int s = 0; s < kGfOT / 4; ++s, g += step) {
      const bool in = lag <= lag_hi && ot * kGfOT + ow + 4 * s < nout;
      copy4(&d.g[0][ll][ow + 4 * s], S.gf_t[0] + (in ? g : 0), in);
      copy4(&d.g[1][ll][ow + 4 * s], S.gf_t[1] + (in ? g : 0), in);
    }
    // rows it0-1+b-lag of this chunk lie in [it0 - l0 - kGfLC, + kGfLC + kGfBlock - 2]
    if (tid < kGfLC + kGfBlock) {
      const int row = it0 - l0 - kGfLC + tid;
      const bool in = row >= 0 && row < nt;
      copy8(&d.h[tid], S.gf_pin + (in ? (long long)r * nt + row : 0), in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the groups' barriers are their own: their halves may differ by a receiver
  auto sync = [&] { asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(kGfGroup) : "memory"); };
  if (total > 0) fetch(0);
  for (int i = 0; i < total; ++i) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    sync();  // chunk i has landed for all, chunk i-1 has been used by all
    if (i + 1 < total) fetch(i + 1);
    const GfFarStage& d = stage[i & 1];
    const int l0 = 1 + (i % nch) * kGfLC;
    // past every step of the block and below every step's T, or checked
    const bool full = l0 >= kGfBlock && l0 + kGfLC <= min(it0, ngf);
    double h[8];  // rows of steps b0 .. b0+7 at the current lag
#pragma unroll
    for (int q = 0; q < 8; ++q) h[q] = d.h[b0 + q + kGfLC - 1];
    auto lags = [&](auto checked) {
#pragma unroll 8
      for (int k = 0; k < kGfLC; ++k) {
        const double a0 = d.g[0][k][ol], a1 = d.g[0][k][ol + 32], c0 = d.g[1][k][ol],
                     c1 = d.g[1][k][ol + 32];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int lag = l0 + k, b = b0 + q;
          if (!decltype(checked)::value || (lag > b && lag < min(it0 + b, ngf))) {
            acc[0][0][q] = __fma_rn(a0, h[q], acc[0][0][q]);
            acc[0][1][q] = __fma_rn(a1, h[q], acc[0][1][q]);
            acc[1][0][q] = __fma_rn(c0, h[q], acc[1][0][q]);
            acc[1][1][q] = __fma_rn(c1, h[q], acc[1][1][q]);
          }
        }
#pragma unroll
        for (int q = 7; q > 0; --q) h[q] = h[q - 1];
        h[0] = d.h[max(b0 + kGfLC - 2 - k, 0)];
      }
    };
    if (full)
      lags(std::false_type());
    else
      lags(std::true_type());
  }
  // the second group's sums are added to the first's
  __syncthreads();  // every group is done with its stages
  double* const other = reinterpret_cast<double*>(gf_smem) + tid;  // [32][kGfGroup]
  if (grp == 1) {
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 8; ++q) other[((t * 2 + h) * 8 + q) * kGfGroup] = acc[t][h][q];
  }
  __syncthreads();
  if (grp == 1) return;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int o = ot * kGfOT + ol + 32 * h;
    if (o >= nout) continue;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      double* pp = S.gf_far + (((long long)o * rsn + rsi) * kGfBlock + b0 + q) * 2;
      pp[0] = __dadd_rn(acc[0][h][q], other[(h * 8 + q) * kGfGroup]);
      pp[1] = __dadd_rn(acc[1][h][q], other[((2 + h) * 8 + q) * kGfGroup]);
    }
  }
}

// Sums the far-lag partials of each (source, step of the block) over the
// receiver splits, in split order, into split 0's slot.  Eight splits' loads in
// flight and small blocks: a chain of dependent adds over strided reads, 18.7 us for
// 256 sources of 64 splits (20.4 for 74, one load at a time in 256-thread blocks).
__global__ void adf_gf_far_combine_kernel(const EpiParams p) {
  const SolveDev& S = p.solves[blockIdx.y];
  const int it0 = S.it_base + p.step;
  if (S.gf_rs <= 0 || it0 > S.it_stop || it0 >= S.nt || !(S.flags & SF_GF)) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // (source, step of the block)
  if (i >= S.gf_nout * kGfBlock) return;
  const int o = i / kGfBlock, b = i - o * kGfBlock;
  double sa = 0.0, sb = 0.0;
#pragma unroll 8
  for (int k = 0; k < S.gf_rs; ++k) {
    const double* pp = S.gf_far + (((long long)o * S.gf_rs + k) * kGfBlock + b) * 2;
    sa = __dadd_rn(sa, pp[0]);
    sb = __dadd_rn(sb, pp[1]);
  }
  double* out = S.gf_far + ((long long)o * S.gf_rs * kGfBlock + b) * 2;
  out[0] = sa;
  out[1] = sb;
}

// Adds each source's partial sums in split order and writes its p_src and
// vn_src samples of row it+1 (solves with more than one block per source).
__global__ void adf_gf_reduce_kernel(const EpiParams p) {
  const SolveDev& S = p.solves[blockIdx.y];
  const int it = S.it_base + p.step;
  if (it > S.it_stop || it >= S.nt || !(S.flags & SF_GF) || S.gf_ks == 1) return;
  const int o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= S.gf_nout) return;
  double sa = 0.0, sb = 0.0;
  for (int k = 0; k < S.gf_ks; ++k) {
    const double* pp = S.gf_part + ((long long)o * S.gf_ks + k) * 2;
    sa = __dadd_rn(sa, pp[0]);
    sb = __dadd_rn(sb, pp[1]);
  }
  gf_finish(S, o, it, p.step, sa, sb);
}

__global__ void adf_advance_kernel(SolveDev* solves, int n, int by) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) solves[i].it_base += by;
}

cudaError_t launch_advance(SolveDev* solves, int n, int by, cudaStream_t s) {
  adf_advance_kernel<<<(n + 127) / 128, 128, 0, s>>>(solves, n, by);
  return cudaGetLastError();
}

// A launch that may overlap the end of the kernel before it: the launch latency
// and, in the step kernel, the reading of descriptors and tables go on while that
// one finishes.
template <typename P>
static cudaError_t launch_overlapped(void (*kernel)(P), dim3 grid, dim3 block, size_t smem,
                                     bool overlap, cudaStream_t s, P p) {
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute a = {};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, p);
}

cudaError_t launch_step(const StepParams& p, int grid, int max_ty, bool overlap, cudaStream_t s) {
  (void)max_ty;  // the block always holds kMaxTy rows; shorter tiles idle the rest
  return launch_overlapped(adf_fdtd_step_kernel, dim3(grid), dim3(32, kXT / 16), kStepDynSmem,
                           overlap, s, p);
}

int step_max_ty() { return kMaxTy; }
cudaError_t step_ctas_per_sm(int* n) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, adf_fdtd_step_kernel, kStepThreads,
                                                       kStepDynSmem);
}
int step_x_tile() { return kXT; }

cudaError_t launch_gf_extrapolate(const EpiParams& p, int max_blocks, int max_nsrc, bool reduce,
                                  bool overlap, cudaStream_t s) {
  // (source, receiver split) blocks of the largest map in the batch, then,
  // when some solve splits its receivers, the fixed-order reduction
  cudaError_t e = launch_overlapped(adf_gf_extrapolate_kernel,
                                    dim3(max_blocks > 0 ? max_blocks : 1, p.n_solves), dim3(256), 0,
                                    overlap, s, p);
  if (e != cudaSuccess || !reduce) return e;
  adf_gf_reduce_kernel<<<dim3((max_nsrc + 127) / 128, p.n_solves), 128, 0, s>>>(p);
  return cudaGetLastError();
}

// Copies lags 0..nl-1 of the two tensors of an input-history map into the
// receiver-major near-lag layout [2][n_out][nl][n_in] (set-up, once per map).
__global__ void adf_gf_near_pack_kernel(const float* t0, const float* t1, float* near, int kind,
                                        int ngf, int n1, int nout, int nin, int nl) {
  const long long per = (long long)nout * nl * nin;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < 2 * per;
       i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i / per);
    long long q = i - k * per;
    const int r = (int)(q % nin);
    q /= nin;
    const int lag = (int)(q % nl);
    const int o = (int)(q / nl);
    const long long g = kind == ADF_GF_PV_FROM_PIN_
                            ? lag + (long long)ngf * (o + (long long)n1 * r)
                            : lag + (long long)ngf * (r + (long long)n1 * o);
    near[i] = (k == 0 ? t0 : t1)[g];
  }
}

cudaError_t launch_gf_near_pack(const SolveDev& d, float* near, cudaStream_t s) {
  adf_gf_near_pack_kernel<<<4 * 148, 256, 0, s>>>(d.gf_t[0], d.gf_t[1], near, d.gf_kind, d.gf_nt,
                                                  d.gf_n1, d.gf_nout, d.gf_nin, d.gf_nl);
  return cudaGetLastError();
}

cudaError_t launch_gf_far(const EpiParams& p, int max_blocks, int max_nsrc, cudaStream_t s) {
  if (max_blocks > 0) {  // 0: every blocked solve of the batch is on the tensor cores
    cudaError_t e = cudaFuncSetAttribute((const void*)adf_gf_far_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGfFarSmem);
    if (e != cudaSuccess) return e;
    adf_gf_far_kernel<<<dim3(max_blocks, p.n_solves), 2 * kGfGroup, kGfFarSmem, s>>>(p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  adf_gf_far_combine_kernel<<<dim3((max_nsrc * kGfBlock + 63) / 64, p.n_solves), 64, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_gf_mid(const EpiParams& p, int max_nsrc, bool overlap, cudaStream_t s) {
  return launch_overlapped(adf_gf_mid_kernel, dim3(max_nsrc, p.n_solves), dim3(kGfMidThreads), 0,
                           overlap, s, p);
}

cudaError_t launch_epilogue(const EpiParams& p, int max_ntx, bool overlap, cudaStream_t s) {
  const int gx = std::max(1, (4 * max_ntx + kEpiThreads - 1) / kEpiThreads);
  return launch_overlapped(adf_fdtd_epilogue_kernel, dim3(gx, p.n_solves), dim3(kEpiThreads), 0,
                           overlap, s, p);
}

}  // namespace adf
