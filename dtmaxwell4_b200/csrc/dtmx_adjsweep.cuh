// dtmx_adjsweep.cuh -- one adjoint time step in one sweep over the grid.
//
// The adjoint step is the forward step's mirror image.  With
//   U = lam_E / eps  (per node and component)  and  G = -lam_H
// the transposed update without an absorber is the forward update itself:
//   G' = G - dt curl U,   U' = U + dt/eps curl G'.
// So it takes the single-sweep engine's walk (dtmx_fused.cuh): two sets of
// arrays, the old values read once by TMA and the new ones written once, the
// new G of the tile's halo recomputed, one CTA barrier a plane.  The kernels
// it replaces (adj_w_kernel, adj_curl_kernel: w of both curl terms to memory
// and back, twice a step) move 168 bytes a cell, this one 48 and the absorber's
// auxiliaries; on a 192x160x128 grid they took 187 us a step, this one takes 86
// (94 in pieces of equal length, plan_work).
//
// The absorber does differ: the transposed CPML stretches a value before the
// difference is taken.  For a derivative along axis a a tap reads
//   S_a x = (1/kappa + a) x + a psi   (old psi; x itself outside the slab),
// and psi <- b (x + psi).  A tap may lie in a neighbouring tile, which needs
// that node's old psi, so psi of both fields is kept twice as well.
//
// A dispersive node (none lies in a slab) holds in the
// U array the value its taps read (kE2 mu, written before the sweep by
// adj_ade_sweep_kernel) and gets curl G' alone from the sweep; its lam_E is kept
// with its ADE state.
//
// Order 2, box geometry, CPML or no absorber, no gyrotropic material and no
// dispersive node inside a slab; everything else takes the two-pass kernels.
#pragma once
#include "dtmx_fused.cuh"
#include "dtmx_adjoint.cuh"

namespace dtmx {

struct AdjSweepArgs {
  float* dst[6];             // set B: U (0-2), G (3-5)
  const float* psrc[3][4];   // psi of set A per axis: slots 0, 1 of U's components, 2, 3 of G's
  float* pdst[3][4];
};

// stretch coefficients of four nodes / one node along an axis, from the staged
// table (b, a, 1/kappa + a); off the slab a = 0 and the factor is 1
struct Str4 { float b[4], a[4], g[4]; };

// S_a of four nodes (psi 0 where a node lies outside the slab)
__device__ __forceinline__ Q4 stretch4(const Q4& x, const Q4& psi, const Str4& c) {
  Q4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) r.v[e] = __fmaf_rn(c.g[e], x.v[e], __fmul_rn(c.a[e], psi.v[e]));
  return r;
}
__device__ __forceinline__ Q4 psi4(const Q4& x, const Q4& psi, const Str4& c) {
  Q4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) r.v[e] = __fmul_rn(c.b[e], __fadd_rn(x.v[e], psi.v[e]));
  return r;
}
__device__ __forceinline__ float stretch1(float x, float psi, const float* c, int s) { return __fmaf_rn(c[2 * s], x, __fmul_rn(c[s], psi)); }
__device__ __forceinline__ Str4 str_same(const float* c) {
  Str4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) { r.b[e] = c[0]; r.a[e] = c[1]; r.g[e] = c[2]; }
  return r;
}

// Coefficient tables: x planes x0-1 .. x0+FX_MAX, rows j0-1 .. j0+TY, columns
// k0-1 .. k0+32 (the columns start at entry 3, so that k0 is 16-byte aligned).
template <int TY>
struct AL {
  static constexpr int X = 0, Y = (FX_MAX + 2) * 6, Z = (Y + (TY + 2) * 6 + 3) / 4 * 4, N = Z + 6 * 40;
  static constexpr int ZS = 40;                      // pitch of a column coefficient
  static constexpr size_t SMEM = (size_t)(F_NST * FL<TY>::STAGE + 2 * FL<TY>::HN + f_up32(N)) * 4 + MAXMAT * 3 * 4 + F_NST * 8 + 128;
};

// What a thread knows about the slab neighbours of its row and columns.
struct AdjNode {
  int ysm, ysp;              // slab coordinates of rows j-1 and j+1 (-1 outside the slab or the grid)
  int zsm, zsp;              // of columns k-1 and k+4
  bool first, last;          // first / last group of its row: the column neighbour belongs to another tile
};

template <int TY>
__device__ __forceinline__ const float* cfx(const float* fco, int row, int O) { return fco + AL<TY>::X + row * 6 + O; }
template <int TY>
__device__ __forceinline__ const float* cfy(const float* fco, int y, int O) { return fco + AL<TY>::Y + (y + 1) * 6 + O; }
template <int TY>
__device__ __forceinline__ const float* cfz(const float* fco, int z, int O) { return fco + AL<TY>::Z + O * AL<TY>::ZS + z + 4; }

__device__ __forceinline__ Str4 str_cols(const float* c, int pitch) {
  Str4 r;
  const Q4 b = ld4(c), a = ld4(c + pitch), g = ld4(c + 2 * pitch);
#pragma unroll
  for (int e = 0; e < 4; e++) { r.b[e] = b.v[e]; r.a[e] = a.v[e]; r.g[e] = g.v[e]; }
  return r;
}

// old psi of four nodes of one axis and slot; zero outside the slab
__device__ __forceinline__ Q4 psi_old(const Params& p, const float* q, int a, int i, int j, int k, int s, bool vec, unsigned m) {
  return aux4<true>(q + slab_at(p, a, i, j, k, s), vec, m);
}

// The old psi of the thread's nodes: what the G update of plane i reads (U's
// slots on all axes, own nodes; the row below) and what the U update of plane i
// reads (G's slots along y and z), requested before the stage wait.
struct AdjPsi {
  Q4 g[3][2], gm[2], u[2][2];
};
__device__ __forceinline__ void adj_psi_g(const Params& p, const AdjSweepArgs& fa, const FNode& f, const AdjNode& an, int i, int xs, AdjPsi& o) {
  const unsigned nm = (1u << f.nv) - 1u;
  if (f.nv > 0) {
    if (xs >= 0)
#pragma unroll
      for (int q = 0; q < 2; q++) o.g[0][q] = psi_old(p, fa.psrc[0][q], 0, i, f.j, f.k, xs, f.vxy, nm);
    if (f.ys >= 0)
#pragma unroll
      for (int q = 0; q < 2; q++) o.g[1][q] = psi_old(p, fa.psrc[1][q], 1, i, f.j, f.k, f.ys, f.vxy, nm);
    if (f.zm)
#pragma unroll
      for (int q = 0; q < 2; q++) o.g[2][q] = psi_old(p, fa.psrc[2][q], 2, i, f.j, f.k, f.zs, f.vz, f.zm);
  }
  const unsigned cm = (1u << min(4, max(0, p.g.n[2] - f.k))) - 1u;   // columns inside the grid, whatever the row
  if (an.ysm >= 0 && cm)
#pragma unroll
    for (int q = 0; q < 2; q++) o.gm[q] = psi_old(p, fa.psrc[1][q], 1, i, f.j - 1, f.k, an.ysm, f.vxy, cm);
}
__device__ __forceinline__ void adj_psi_u(const Params& p, const AdjSweepArgs& fa, const FNode& f, int i, AdjPsi& o) {
  if (f.nv == 0) return;
  const unsigned nm = (1u << f.nv) - 1u;
  if (f.ys >= 0)
#pragma unroll
    for (int q = 0; q < 2; q++) o.u[0][q] = psi_old(p, fa.psrc[1][2 + q], 1, i, f.j, f.k, f.ys, f.vxy, nm);
  if (f.zm)
#pragma unroll
    for (int q = 0; q < 2; q++) o.u[1][q] = psi_old(p, fa.psrc[2][2 + q], 2, i, f.j, f.k, f.zs, f.vz, f.zm);
}

// New G of plane i on the thread's nodes; ec gets the old U, ux the stretched
// old Uy, Uz of this plane (x taps of the next one; in: those of plane i - 1), hcx
// the stretched new Gy, Gz (x taps of the U update).
template <int TY, bool ABS>
__device__ __forceinline__ void adj_g_own(const Params& p, const AdjSweepArgs& fa, const float* st, float* hn, const FNode& f,
                                          const AdjNode& an, int i, bool store, Q4 (&ux)[2], Q4 (&hc)[3], Q4 (&hcx)[2], Q4 (&ec)[3],
                                          const float* fco, int xrow, int xs, const AdjPsi& ps) {
  const float cx = p.cdt[0], cy = p.cdt[1], cz = p.cdt[2];
  const Q4 ex = ld4(fE<TY>(st, 0, f.y, f.z)), ey = ld4(fE<TY>(st, 1, f.y, f.z)), ez = ld4(fE<TY>(st, 2, f.y, f.z));
  ec[0] = ex; ec[1] = ey; ec[2] = ez;
  const Q4 exm = ld4(fE<TY>(st, 0, f.y - 1, f.z)), ezm = ld4(fE<TY>(st, 2, f.y - 1, f.z));
  const float exl = *fE<TY>(st, 0, f.y, f.z - 1), eyl = *fE<TY>(st, 1, f.y, f.z - 1);
  Q4 d01, d02, d10, d12, d20, d21;
  const unsigned nm = (1u << f.nv) - 1u;
  if (!ABS) {
    d01 = diff4(-cy, ez, ezm); d02 = diff4(cz, ey, below4(eyl, ey));
    d10 = diff4(cx, ez, ux[1]); d12 = diff4(-cz, ex, below4(exl, ex));
    d20 = diff4(-cx, ey, ux[0]); d21 = diff4(cy, ex, exm);
    ux[0] = ey; ux[1] = ez;
  } else {
    // x: Uy (slot 0), Uz (slot 1)
    Q4 xy = ey, xz = ez;
    if (xs >= 0 && f.nv > 0) {
      const Str4 c = str_same(cfx<TY>(fco, xrow, 3));
      const Q4 p0 = ps.g[0][0], p1 = ps.g[0][1];
      xy = stretch4(ey, p0, c); xz = stretch4(ez, p1, c);
      if (store) {
        const int s = slab_at(p, 0, i, f.j, f.k, xs);
        put4(fa.pdst[0][0] + s, f.vxy, nm, psi4(ey, p0, c));
        put4(fa.pdst[0][1] + s, f.vxy, nm, psi4(ez, p1, c));
      }
    }
    d10 = diff4(cx, xz, ux[1]); d20 = diff4(-cx, xy, ux[0]);
    ux[0] = xy; ux[1] = xz;
    // y: Ux (slot 0), Uz (slot 1), own row and the one below
    Q4 yx = ex, yz = ez, yxm = exm, yzm = ezm;
    const unsigned cm = (1u << min(4, max(0, p.g.n[2] - f.k))) - 1u;   // columns inside the grid, whatever the row
    if (f.ys >= 0 && f.nv > 0) {
      const Str4 c = str_same(cfy<TY>(fco, f.y, 3));
      const Q4 p0 = ps.g[1][0], p1 = ps.g[1][1];
      yx = stretch4(ex, p0, c); yz = stretch4(ez, p1, c);
      if (store) {
        const int s = slab_at(p, 1, i, f.j, f.k, f.ys);
        put4(fa.pdst[1][0] + s, f.vxy, nm, psi4(ex, p0, c));
        put4(fa.pdst[1][1] + s, f.vxy, nm, psi4(ez, p1, c));
      }
    }
    if (an.ysm >= 0 && cm) {
      const Str4 c = str_same(cfy<TY>(fco, f.y - 1, 3));
      yxm = stretch4(exm, ps.gm[0], c);
      yzm = stretch4(ezm, ps.gm[1], c);
    }
    d01 = diff4(-cy, yz, yzm); d21 = diff4(cy, yx, yxm);
    // z: Ux (slot 0), Uy (slot 1), own columns and the one below
    Q4 zx = ex, zy = ey;
    if (f.zm) {
      const Str4 c = str_cols(cfz<TY>(fco, f.z, 3), AL<TY>::ZS);
      const Q4 p0 = ps.g[2][0], p1 = ps.g[2][1];
      zx = stretch4(ex, p0, c); zy = stretch4(ey, p1, c);
      if (store) {
        const int s = slab_at(p, 2, i, f.j, f.k, f.zs);
        put4(fa.pdst[2][0] + s, f.vz, f.zm, psi4(ex, p0, c));
        put4(fa.pdst[2][1] + s, f.vz, f.zm, psi4(ey, p1, c));
      }
    }
    float lx = __shfl_up_sync(0xffffffffu, zx.v[3], 1), ly = __shfl_up_sync(0xffffffffu, zy.v[3], 1);
    if (an.first) {
      lx = exl; ly = eyl;
      if (an.zsm >= 0 && f.nv > 0) {
        const float* c = cfz<TY>(fco, f.z - 1, 3);
        const int s = slab_at(p, 2, i, f.j, f.k - 1, an.zsm);
        lx = stretch1(exl, __ldg(fa.psrc[2][0] + s), c, AL<TY>::ZS);
        ly = stretch1(eyl, __ldg(fa.psrc[2][1] + s), c, AL<TY>::ZS);
      }
    }
    d02 = diff4(cz, zy, below4(ly, zy)); d12 = diff4(-cz, zx, below4(lx, zx));
  }
  hc[0] = add4(ld4(fHx<TY>(st, f.y, f.z)), add4(d01, d02));
  hc[1] = add4(ld4(fHy<TY>(st, f.y, f.z)), add4(d10, d12));
  hc[2] = add4(ld4(fHz<TY>(st, f.y, f.z)), add4(d20, d21));
  if (f.nv < 4) {
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
      for (int e = 0; e < 4; e++)
        if (e >= f.nv) hc[c].v[e] = 0.f;
  }
#pragma unroll
  for (int c = 0; c < 3; c++) st4(fN<TY>(hn, c, f.y, f.z), hc[c]);
  if (store && f.nv > 0) {
    const long long off = (long long)i * p.g.sx + (long long)f.j * p.g.sy + f.k;
#pragma unroll
    for (int c = 0; c < 3; c++) st4(fa.dst[3 + c] + off, hc[c]);
  }
  hcx[0] = hc[1]; hcx[1] = hc[2];
  if (ABS && xs >= 0 && f.nv > 0) {
    // x: Gy (slot 2), Gz (slot 3)
    const Str4 c = str_same(cfx<TY>(fco, xrow, 0));
    const Q4 p0 = psi_old(p, fa.psrc[0][2], 0, i, f.j, f.k, xs, f.vxy, nm), p1 = psi_old(p, fa.psrc[0][3], 0, i, f.j, f.k, xs, f.vxy, nm);
    hcx[0] = stretch4(hc[1], p0, c); hcx[1] = stretch4(hc[2], p1, c);
    if (store) {
      const int s = slab_at(p, 0, i, f.j, f.k, xs);
      put4(fa.pdst[0][2] + s, f.vxy, nm, psi4(hc[1], p0, c));
      put4(fa.pdst[0][3] + s, f.vxy, nm, psi4(hc[2], p1, c));
    }
  }
}

// stretched old U of the halo tasks: component c at tile-local (y, z) along axis a
template <int TY>
__device__ __forceinline__ float adj_tap(const Params& p, const AdjSweepArgs& fa, const float* st, const float* fco, int c, int a, int slot,
                                         int y, int z, int i, int xrow, int j0, int k0, int xs) {
  const float v = *fE<TY>(st, c, y, z);
  const int j = j0 + y, k = k0 + z;
  if (j < 0 || j >= p.g.n[1] || k < 0 || k >= p.g.n[2]) return v;
  const int s = a == 0 ? xs : slab_cs(p, a, a == 1 ? j : k);
  if (s < 0) return v;
  const float* cf = a == 0 ? cfx<TY>(fco, xrow, 3) : a == 1 ? cfy<TY>(fco, y, 3) : cfz<TY>(fco, z, 3);
  return stretch1(v, __ldg(fa.psrc[a][slot] + slab_at(p, a, i, j, k, s)), cf, a == 2 ? AL<TY>::ZS : 1);
}
// new G on the halo (tasks as in fused_h_halo); xe: stretched old U of the previous plane at the node
template <int TY, bool ABS>
__device__ __forceinline__ void adj_g_halo(const Params& p, const AdjSweepArgs& fa, const float* st, float* hn, int task, const FHalo& h,
                                           float& xe, const float* fco, int i, int xrow, int j0, int k0, int xs) {
  if (!h.on) return;
  const float cx = p.cdt[0], cy = p.cdt[1], cz = p.cdt[2];
  auto tap = [&](int c, int a, int slot, int dy, int dz) {
    return ABS ? adj_tap<TY>(p, fa, st, fco, c, a, slot, h.y + dy, h.z + dz, i, xrow, j0, k0, xs) : *fE<TY>(st, c, h.y + dy, h.z + dz);
  };
  float d0, d1, old;
  if (task == 0) {
    const float x = tap(1, 0, 0, 0, 0);
    d0 = __fmul_rn(-cx, __fsub_rn(x, xe));
    d1 = __fmul_rn(cy, __fsub_rn(tap(0, 1, 0, 0, 0), tap(0, 1, 0, -1, 0)));
    old = *fHz<TY>(st, h.y, h.z);
    xe = x;
  } else if (task == 2) {
    const float x = tap(2, 0, 1, 0, 0);
    d0 = __fmul_rn(cx, __fsub_rn(x, xe));
    d1 = __fmul_rn(-cz, __fsub_rn(tap(0, 2, 0, 0, 0), tap(0, 2, 0, 0, -1)));
    old = *fHy<TY>(st, h.y, h.z);
    xe = x;
  } else {
    d0 = __fmul_rn(-cy, __fsub_rn(tap(2, 1, 1, 0, 0), tap(2, 1, 1, -1, 0)));
    d1 = __fmul_rn(cz, __fsub_rn(tap(1, 2, 1, 0, 0), tap(1, 2, 1, 0, -1)));
    old = *fHx<TY>(st, h.y, h.z);
  }
  *fN<TY>(hn, task == 0 ? 2 : task == 2 ? 1 : 0, h.y, h.z) = h.ok ? __fadd_rn(old, __fadd_rn(d0, d1)) : 0.f;
}

// New U of plane i on the own nodes: ep old U, hpx / hcx the stretched new Gy,
// Gz of planes i and i + 1.  MODE as in fused_e_own.
template <int TY, int MODE, bool ABS>
__device__ __forceinline__ void adj_u_own(const Params& p, const AdjSweepArgs& fa, const float* st, const float* hn, const float* ies, int um,
                                          const FNode& f, const AdjNode& an, int i, const Q4 (&ep)[3], const Q4 (&hpx)[2],
                                          const Q4 (&hcx)[2], const float* fco, const AdjPsi& ps) {
  const float cx = p.cdt[0], cy = p.cdt[1], cz = p.cdt[2];
  const Q4 hx = ld4(fN<TY>(hn, 0, f.y, f.z)), hy = ld4(fN<TY>(hn, 1, f.y, f.z)), hz = ld4(fN<TY>(hn, 2, f.y, f.z));
  const Q4 hxp = ld4(fN<TY>(hn, 0, f.y + 1, f.z)), hzp = ld4(fN<TY>(hn, 2, f.y + 1, f.z));
  const float hxr = *fN<TY>(hn, 0, f.y, f.z + 4), hyr = *fN<TY>(hn, 1, f.y, f.z + 4);
  const Q4 d10 = diff4(-cx, hcx[1], hpx[1]), d20 = diff4(cx, hcx[0], hpx[0]);
  Q4 d01, d02, d12, d21;
  if (!ABS) {
    d01 = diff4(cy, hzp, hz); d21 = diff4(-cy, hxp, hx);
    d02 = diff4(-cz, above4(hy, hyr), hy); d12 = diff4(cz, above4(hx, hxr), hx);
  } else {
    const unsigned nm = (1u << f.nv) - 1u;
    // y: Gx (slot 2), Gz (slot 3), own row and the one above
    Q4 yx = hx, yz = hz, yxp = hxp, yzp = hzp;
    if (f.ys >= 0 && f.nv > 0) {
      const Str4 c = str_same(cfy<TY>(fco, f.y, 0));
      const Q4 p0 = ps.u[0][0], p1 = ps.u[0][1];
      yx = stretch4(hx, p0, c); yz = stretch4(hz, p1, c);
      const int s = slab_at(p, 1, i, f.j, f.k, f.ys);
      put4(fa.pdst[1][2] + s, f.vxy, nm, psi4(hx, p0, c));
      put4(fa.pdst[1][3] + s, f.vxy, nm, psi4(hz, p1, c));
    }
    if (an.ysp >= 0 && f.nv > 0) {
      const Str4 c = str_same(cfy<TY>(fco, f.y + 1, 0));
      yxp = stretch4(hxp, psi_old(p, fa.psrc[1][2], 1, i, f.j + 1, f.k, an.ysp, f.vxy, nm), c);
      yzp = stretch4(hzp, psi_old(p, fa.psrc[1][3], 1, i, f.j + 1, f.k, an.ysp, f.vxy, nm), c);
    }
    d01 = diff4(cy, yzp, yz); d21 = diff4(-cy, yxp, yx);
    // z: Gx (slot 2), Gy (slot 3), own columns and the one above
    Q4 zx = hx, zy = hy;
    if (f.zm) {
      const Str4 c = str_cols(cfz<TY>(fco, f.z, 0), AL<TY>::ZS);
      const Q4 p0 = ps.u[1][0], p1 = ps.u[1][1];
      zx = stretch4(hx, p0, c); zy = stretch4(hy, p1, c);
      const int s = slab_at(p, 2, i, f.j, f.k, f.zs);
      put4(fa.pdst[2][2] + s, f.vz, f.zm, psi4(hx, p0, c));
      put4(fa.pdst[2][3] + s, f.vz, f.zm, psi4(hy, p1, c));
    }
    float rx = __shfl_down_sync(0xffffffffu, zx.v[0], 1), ry = __shfl_down_sync(0xffffffffu, zy.v[0], 1);
    if (an.last) {
      rx = hxr; ry = hyr;
      if (an.zsp >= 0 && f.nv > 0) {
        const float* c = cfz<TY>(fco, f.z + 4, 0);
        const int s = slab_at(p, 2, i, f.j, f.k + 4, an.zsp);
        rx = stretch1(hxr, __ldg(fa.psrc[2][2] + s), c, AL<TY>::ZS);
        ry = stretch1(hyr, __ldg(fa.psrc[2][3] + s), c, AL<TY>::ZS);
      }
    }
    d02 = diff4(-cz, above4(zy, ry), zy); d12 = diff4(cz, above4(zx, rx), zx);
  }
  if (f.nv == 0) return;
  Q4 inc[3] = {add4(d01, d02), add4(d10, d12), add4(d20, d21)};
  Q4 out[3];
  if (MODE == 0) {
    const unsigned* mt = reinterpret_cast<const unsigned*>(st + FL<TY>::OFF_M);
    unsigned m[3];
#pragma unroll
    for (int c = 0; c < 3; c++) m[c] = mt[(c * F_MROWS * TZ + f.y * TZ + f.z) / 4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const long long di = p.des_on ? design_index(p, i, f.j, f.k + e) : -1;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        float ie = ies[((m[c] >> (8 * e)) & 255u) * 3 + c];
        if (di >= 0 && !is_dispersive(ie)) ie = __ldg(p.des_ie[c] + di);
        // (a dispersive node: curl G' alone)
        out[c].v[e] = is_dispersive(ie) ? inc[c].v[e] : __fmaf_rn(ie, inc[c].v[e], ep[c].v[e]);
      }
    }
  } else {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const float ie = MODE == 1 ? ies[um * 3 + c] : 1.f;
#pragma unroll
      for (int e = 0; e < 4; e++) out[c].v[e] = MODE == 1 ? __fmaf_rn(ie, inc[c].v[e], ep[c].v[e]) : __fadd_rn(ep[c].v[e], inc[c].v[e]);
    }
  }
  const long long off = (long long)i * p.g.sx + (long long)f.j * p.g.sy + f.k;
#pragma unroll
  for (int c = 0; c < 3; c++) st4(fa.dst[c] + off, out[c]);
}

template <int TY, bool TAB>
__global__ void __launch_bounds__(FL<TY>::NT, 3)
    adj_sweep_kernel(const __grid_constant__ Params p, const __grid_constant__ AdjSweepArgs fa, const __grid_constant__ FusedMaps m,
                     const __grid_constant__ Work<TAB> work) {
  using L = FL<TY>;
  extern __shared__ __align__(128) float fsm[];
  float* hnb = fsm + F_NST * L::STAGE;                           // two new-G planes
  float* fco = hnb + 2 * L::HN;
  float* ies = fco + f_up32(AL<TY>::N);                          // 1/eps of the material table
  uint64_t* bars = reinterpret_cast<uint64_t*>(ies + MAXMAT * 3);
  __shared__ signed char umc[FX_MAX];
  __shared__ int gave_up;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int4 job = cta_job<TAB>(p, work);
  const int k0 = job.x * TZ, j0 = job.y * TY;
  const int x0 = job.z, len = job.w - job.z;
  const int slast = len + 1;                               // stages 0 .. len + 1: planes x0 - 1 .. x1
  const bool cpml = p.ab.kind == 1;
  auto issue = [&](int s, bool want_mat) {
    fused_issue<TY>(m, fsm + (s % F_NST) * L::STAGE, &bars[s % F_NST], x0 - 1 + s, j0, k0, want_mat);
  };
  int issued = -1;
  if (tid == 0) {
    for (int q = 0; q < F_NST; q++) mbar_init(&bars[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    gave_up = 0;
    // the first two stages hold no material tile: they need not wait for the tables below
    pdl_wait();
    for (int s = 0; s < 2; s++) { issue(s, false); issued = s; }
  }
  for (int q = tid; q < MAXMAT * 3; q += L::NT) ies[q] = __ldg(&p.mt->inv_eps[0][0] + q);
  for (int q = tid; q < len; q += L::NT)
    umc[q] = __ldg(p.umat + ((long long)(x0 + q) * p.nty + j0 / F_MROWS) * p.ntz + job.x);
  if (cpml) {
    // coefficient row q: x plane x0 - 1 + q, then y row j0 - 1 + ..., then z column k0 - 1 + ...
    constexpr int RX = FX_MAX + 2, RY_ = TY + 2, RZ = TZ + 2;
    for (int q = tid; q < RX + RY_ + RZ; q += L::NT) {
      const int a = q < RX ? 0 : q < RX + RY_ ? 1 : 2;
      const int v0 = a == 0 ? q : a == 1 ? q - RX : q - RX - RY_;
      const int v = v0 - 1 + (a == 0 ? x0 : a == 1 ? j0 : k0);
      if (a == 0 && v0 > len + 1) continue;
#pragma unroll
      for (int o = 0; o < 2; o++) {
        const int h = 2 * v + o;
        const bool in = h >= 0 && h < 2 * p.g.n[a] + 2;
        const float cb = in ? __ldg(p.ab.c0[a] + h) : 1.f, ca = in ? __ldg(p.ab.c1[a] + h) : 0.f;
        const float cg = in ? __fadd_rn(__ldg(p.ab.c2[a] + h), ca) : 1.f;
        float* d = a == 2 ? fco + AL<TY>::Z + 3 * o * AL<TY>::ZS + v0 + 3 : fco + (a == 0 ? AL<TY>::X : AL<TY>::Y) + v0 * 6 + 3 * o;
        const int s = a == 2 ? AL<TY>::ZS : 1;
        d[0] = cb; d[s] = ca; d[2 * s] = cg;
      }
    }
  }
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  // stage s: plane x0 - 1 + s, with the materials of the plane before it (s >= 2)
  if (tid == 0 && slast >= 2) { issue(2, umc[0] < 0); issued = 2; }
  FNode f;
  f.y = tid >> 3; f.z = 4 * (tid & 7);
  f.j = j0 + f.y; f.k = k0 + f.z;
  f.nv = f.j < p.g.n[1] ? min(4, max(0, p.g.n[2] - f.k)) : 0;
  f.ys = cpml && f.nv > 0 ? slab_cs(p, 1, f.j) : -1;
  f.zs = 0; f.zm = 0;
  AdjNode an;
  an.ysm = cpml && f.j - 1 >= 0 && f.j - 1 < p.g.n[1] ? slab_cs(p, 1, f.j - 1) : -1;
  an.ysp = cpml && f.j + 1 < p.g.n[1] ? slab_cs(p, 1, f.j + 1) : -1;
  an.zsm = cpml && f.k - 1 >= 0 && f.k - 1 < p.g.n[2] ? slab_cs(p, 2, f.k - 1) : -1;
  an.zsp = cpml && f.k + 4 < p.g.n[2] ? slab_cs(p, 2, f.k + 4) : -1;
  an.first = (tid & 7) == 0; an.last = (tid & 7) == 7;
  if (cpml) {
    const int lo = p.ab.L[2][0], hi = p.g.n[2] - p.ab.L[2][1];
    f.zs = f.k < lo ? f.k : f.k + lo - hi;
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (e < f.nv && (f.k + e < lo || f.k + e >= hi)) f.zm |= 1u << e;
  }
  f.vxy = (p.g.n[2] & 3) == 0;
  f.vz = f.zm == 15u && ((p.ab.L[2][0] + p.ab.L[2][1]) & 3) == 0 && (f.zs & 3) == 0;
  FHalo hl[L::TASKS];
  float xe[L::TASKS];
#pragma unroll
  for (int q = 0; q < L::TASKS; q++) {
    const int task = w + q * L::NW;
    const bool row = task < 2;
    hl[q].y = row ? TY : lane; hl[q].z = row ? lane : TZ;
    hl[q].j = j0 + hl[q].y; hl[q].k = k0 + hl[q].z;
    hl[q].on = task < 4 && (row || lane < TY);
    hl[q].ok = hl[q].on && hl[q].j < p.g.n[1] && hl[q].k < p.g.n[2];
    hl[q].ysh = hl[q].zsh = -1;
    xe[q] = 0.f;
  }
  // does the tile, with one node around it, meet a y or z slab?
  const bool ab_yz = cpml && (j0 - 1 < p.ab.L[1][0] || j0 + TY + 1 > p.g.n[1] - p.ab.L[1][1] || k0 - 1 < p.ab.L[2][0] ||
                              k0 + TZ + 1 > p.g.n[2] - p.ab.L[2][1]);
  Q4 ep[3], hc[3], ec[3], ux[2], hpx[2], hcx[2];
  AdjPsi ps;
  // stage 0 (plane x0 - 1): the stretched old Uy, Uz of the own nodes and of the halo nodes (x taps)
  if (tid == 0 && !mbar_wait(&bars[0], 0u, p.err, p.wait_limit)) gave_up = 1;
  __syncthreads();
  int t = 0, swait = 0;                                    // swait: the stage waited for last
  if (!gave_up) {
    {
      const int xs = cpml && x0 >= 1 ? slab_cs(p, 0, x0 - 1) : -1;
      ux[0] = ld4(fE<TY>(fsm, 1, f.y, f.z)); ux[1] = ld4(fE<TY>(fsm, 2, f.y, f.z));
      if (xs >= 0 && f.nv > 0) {
        const Str4 c = str_same(cfx<TY>(fco, 0, 3));
        const unsigned nm = (1u << f.nv) - 1u;
        ux[0] = stretch4(ux[0], psi_old(p, fa.psrc[0][0], 0, x0 - 1, f.j, f.k, xs, f.vxy, nm), c);
        ux[1] = stretch4(ux[1], psi_old(p, fa.psrc[0][1], 0, x0 - 1, f.j, f.k, xs, f.vxy, nm), c);
      }
#pragma unroll
      for (int q = 0; q < L::TASKS; q++) {
        const int task = w + q * L::NW;
        if (hl[q].on && !(task & 1))
          xe[q] = adj_tap<TY>(p, fa, fsm, fco, task == 0 ? 1 : 2, 0, task == 0 ? 0 : 1, hl[q].y, hl[q].z, x0 - 1, 0, j0, k0, xs);
      }
#pragma unroll
      for (int c = 0; c < 3; c++) ep[c] = Q4{{0.f, 0.f, 0.f, 0.f}};
      hpx[0] = hpx[1] = ep[0];
    }
    for (; t <= len; t++) {
      const int s = t + 1, pc = x0 + t, pe = pc - 1;
      const int xs = cpml && pc < p.g.n[0] ? slab_cs(p, 0, pc) : -1;
      const bool ab = ab_yz || xs >= 0;
      if (ab && pc < p.g.n[0]) adj_psi_g(p, fa, f, an, pc, xs, ps);
      if (ab_yz && t >= 1) adj_psi_u(p, fa, f, pe, ps);
      swait = s;
      if (tid == 0 && !mbar_wait(&bars[s % F_NST], (unsigned)((s / F_NST) & 1), p.err, p.wait_limit)) gave_up = 1;
      // every thread is past iteration t - 1: the slot of stage t and the new-G
      // plane written two iterations ago are free
      __syncthreads();
      if (gave_up) break;
      if (tid == 0 && t + F_NST <= slast) { issue(t + F_NST, umc[t + F_NST - 2] < 0); issued = t + F_NST; }
      const float* st = fsm + (s % F_NST) * L::STAGE;
      float* hn1 = hnb + (t & 1) * L::HN;                        // new G of plane pc
      const float* hn0 = hnb + ((t + 1) & 1) * L::HN;            // new G of plane pc - 1
      if (pc < p.g.n[0]) {
        if (ab) adj_g_own<TY, true>(p, fa, st, hn1, f, an, pc, t < len, ux, hc, hcx, ec, fco, t + 1, xs, ps);
        else adj_g_own<TY, false>(p, fa, st, hn1, f, an, pc, t < len, ux, hc, hcx, ec, fco, t + 1, xs, ps);
#pragma unroll
        for (int q = 0; q < L::TASKS; q++) {
          const int task = w + q * L::NW;
          if (ab) adj_g_halo<TY, true>(p, fa, st, hn1, task, hl[q], xe[q], fco, pc, t + 1, j0, k0, xs);
          else adj_g_halo<TY, false>(p, fa, st, hn1, task, hl[q], xe[q], fco, pc, t + 1, j0, k0, xs);
        }
      } else {
        // beyond the last plane of the grid: G is zero there
#pragma unroll
        for (int c = 0; c < 3; c++) ec[c] = Q4{{0.f, 0.f, 0.f, 0.f}};
        hcx[0] = hcx[1] = ec[0];
      }
      if (t >= 1) {
        const int um = umc[pe - x0];
        const bool vac = um >= 0 && ies[um * 3] == 1.f && ies[um * 3 + 1] == 1.f && ies[um * 3 + 2] == 1.f;
        switch ((vac ? 4 : um >= 0 ? 2 : 0) + (ab_yz ? 1 : 0)) {
          case 5: adj_u_own<TY, 2, true>(p, fa, st, hn0, ies, um, f, an, pe, ep, hpx, hcx, fco, ps); break;
          case 4: adj_u_own<TY, 2, false>(p, fa, st, hn0, ies, um, f, an, pe, ep, hpx, hcx, fco, ps); break;
          case 3: adj_u_own<TY, 1, true>(p, fa, st, hn0, ies, um, f, an, pe, ep, hpx, hcx, fco, ps); break;
          case 2: adj_u_own<TY, 1, false>(p, fa, st, hn0, ies, um, f, an, pe, ep, hpx, hcx, fco, ps); break;
          case 1: adj_u_own<TY, 0, true>(p, fa, st, hn0, ies, um, f, an, pe, ep, hpx, hcx, fco, ps); break;
          default: adj_u_own<TY, 0, false>(p, fa, st, hn0, ies, um, f, an, pe, ep, hpx, hcx, fco, ps); break;
        }
      }
#pragma unroll
      for (int c = 0; c < 3; c++) ep[c] = ec[c];
      hpx[0] = hcx[0]; hpx[1] = hcx[1];
    }
  }
  if (gave_up && tid == 0) {
    // a wait gave up: no further copies were issued; wait (bounded) for those in flight, then leave
    for (int s = swait; s <= issued; s++) mbar_wait(&bars[s % F_NST], (unsigned)((s / F_NST) & 1), nullptr, DRAIN_POLLS);
  }
}

// Before the sweep of a step, in one launch: the objective's sources of step s
// on the plane x = X (blocks [0, ns): adj_source_kernel in U and G; 1/eps of the
// node scales U's) and the gradient of history slots st, st - 1 (the blocks
// after them: adj_grad_kernel with lam_E = U / (1/eps)).  The plane and the
// design region share no node in one launch: the gradient reads U after the sources.
__global__ void __launch_bounds__(256) adj_pre_kernel(const __grid_constant__ Params p, const __grid_constant__ AdjDev A, const double* F,
                                                      long long s, int X, double omega, double dt, int ns, int st) {
  pdl_wait();
  pdl_trigger();
  if ((int)blockIdx.x < ns) {
    __shared__ double ph[4];
    if (threadIdx.x < 2) {
      double sn, cs;
      sincos(omega * ((double)s - 0.5 * threadIdx.x) * dt, &sn, &cs);
      ph[2 * threadIdx.x] = cs * dt;
      ph[2 * threadIdx.x + 1] = -sn * dt;
    }
    __syncthreads();
    const int npl = p.g.n[1] * p.g.n[2], u = blockIdx.x * 256 + threadIdx.x;
    if (u >= npl) return;
    const double2* Fd = reinterpret_cast<const double2*>(F);
    const double2 ey = Fd[u], ez = Fd[npl + u], hy = Fd[2 * (long long)npl + u], hz = Fd[3 * (long long)npl + u];
    const int j = u / p.g.n[2], k = u - j * p.g.n[2];
    const long long id = (long long)X * p.g.sx + (long long)j * p.g.sy + k;
    const long long di = design_index(p, X, j, k);
    float ie[3];
#pragma unroll
    for (int c = 1; c < 3; c++) {
      const int mat = p.mat[c] ? (int)__ldg(p.mat[c] + id) : 0;
      ie[c] = __ldg(&p.mt->inv_eps[mat][c]);
      if (__ldg(&p.mt->npoles[mat]) > 0) ie[c] = 1.f;  // dispersive node: lam_E itself
      else if (di >= 0) ie[c] = __ldg(p.des_ie[c] + di);
    }
    A.lam[1][id] += (float)((ph[0] * hz.x + ph[1] * hz.y) * (double)ie[1]);
    A.lam[2][id] -= (float)((ph[0] * hy.x + ph[1] * hy.y) * (double)ie[2]);
    A.lam[5][id] -= (float)(ey.x * ph[2] + ey.y * ph[3]);
    A.lam[4][id] += (float)(ez.x * ph[2] + ez.y * ph[3]);
    return;
  }
  const int nd = A.nd, q = ((int)blockIdx.x - ns) * 256 + threadIdx.x;
  if (q >= 3 * nd) return;
  const int c = q / nd, di = q - c * nd;
  const int i = p.des_lo[0] + di / (p.des_n[1] * p.des_n[2]);
  const int j = p.des_lo[1] + (di / p.des_n[2]) % p.des_n[1];
  const int k = p.des_lo[2] + di % p.des_n[2];
  const long long id = (long long)i * p.g.sx + (long long)j * p.g.sy + k;
  if (p.mat[c] && __ldg(&p.mt->npoles[__ldg(p.mat[c] + id)]) > 0) return;
  const double dE = (double)A.hist[((long long)st * 3 + c) * nd + di] - (double)A.hist[((long long)(st - 1) * 3 + c) * nd + di];
  const double ie = (double)p.des_ie[c][di];
  A.grad[q] += (double)A.lam[c][id] * dE / (ie * ie);
}

// Transposed ADE recursion before the sweep (the recursion of adj_ade_kernel):
// the sweep left curl G' in the U array of a dispersive node, lE holds the rest of
// its lam_E; writes kE2 mu for the node's taps.
__global__ void __launch_bounds__(256) adj_ade_sweep_kernel(const __grid_constant__ Params p, const __grid_constant__ AdjDev A) {
  pdl_wait();
  pdl_trigger();
  const MatTable& mt = *p.mt;
  int bi, bj, bk;
  long long q;
  if (!ade_cell(p, bi, bj, bk, q)) return;
  const int i = p.ade.lo[0] + bi, j = p.ade.lo[1] + bj, k = p.ade.lo[2] + bk;
  const long long id = (long long)i * p.g.sx + (long long)j * p.g.sy + k;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int m = p.mat[c] ? (int)__ldg(p.mat[c] + id) : 0;
    const int np = __ldg(&mt.npoles[m]);
    if (np <= 0) continue;
    float mu = __fadd_rn(A.lE[c][q], A.lam[c][id]);
    for (int r = 0; r < np; r++) mu = __fmaf_rn(__ldg(&mt.kJ[m][c][r][2]), A.lJp[c][r][q], mu);
    A.lam[c][id] = __fmul_rn(__ldg(&mt.kE[m][c][2]), mu);
    float nE = __fmaf_rn(__ldg(&mt.kE[m][c][1]), mu, A.lEm[c][q]);
    float nEm = __fmul_rn(__ldg(&mt.kE[m][c][0]), mu);
    for (int r = 0; r < np; r++) {
      const float lp = A.lJp[c][r][q], lm = A.lJm[c][r][q];
      nE = __fmaf_rn(__ldg(&mt.kJ[m][c][r][4]), lp, nE);
      nEm = __fmaf_rn(__ldg(&mt.kJ[m][c][r][3]), lp, nEm);
      A.lJp[c][r][q] = __fmaf_rn(__ldg(&mt.kJ[m][c][r][0]), lp, __fmaf_rn(-__ldg(&mt.kEJ[m][c][r][0]), mu, lm));
      A.lJm[c][r][q] = __fmaf_rn(__ldg(&mt.kJ[m][c][r][1]), lp, -__fmul_rn(__ldg(&mt.kEJ[m][c][r][1]), mu));
    }
    A.lE[c][q] = nE;
    A.lEm[c][q] = nEm;
  }
}

}  // namespace dtmx
