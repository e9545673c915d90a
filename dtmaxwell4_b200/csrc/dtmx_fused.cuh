// dtmx_fused.cuh -- single-sweep engine: one launch per time step advances H
// and then E, plane by plane, reading the old fields once and writing the new
// ones once.
//
// The fields are kept twice (A, B).  A step reads A and writes B, and the next
// step the other way round, so no CTA can see a value that another CTA of the
// same launch has already advanced.  That lets a CTA recompute, redundantly,
// the new H on the one-node halo its E update needs (the row above the tile
// and the column beyond it) instead of waiting for the neighbour that owns
// those nodes.  The per-step engine makes two passes over the grid per step
// (H, then E), each reading the field the other one writes; this engine makes
// one.
//
// Tile: 32 (z) x 16 or 8 (y) nodes, eight threads a row with four consecutive z
// nodes each, walked upwards along an x chunk.  Iteration t of the walk
// consumes the stage of plane pc = x0 + t and
//   * computes the new H of plane pc on the own nodes (and the halo, one task a
//     warp: Hz and Hx of the row above, Hy and Hx of column 32) from the old
//     E of planes pc (staged) and pc - 1 (registers) and the old H of plane pc
//     (staged); the own values go to B and, with the halo, to a shared-memory
//     plane buffer;
//   * computes the new E of plane pc - 1 on the own nodes from its old E
//     (registers), the new H of plane pc - 1 (the other shared-memory plane
//     buffer) and of plane pc (registers).
// Each old value is therefore read from HBM once per step (the halo rows and
// columns of the TMA boxes come from L2), and every plane costs one CTA
// barrier.  One elected thread issues the TMA copies (cp.async.bulk.tensor,
// no multicast) of a plane's E box (TY + 2 rows x 40 floats per component),
// old-H boxes and, when the E update of the previous plane needs them, that
// plane's material tiles, into a 3-stage ring (two planes in flight).
// Everything outside the grid reads as zero (TMA fill; new H forced to zero
// outside), which is the box geometry; other geometries use the per-step
// engine.
//
// Why four nodes a thread: the sweep was bound by instructions, not by memory
// or the loads' latency (a CTA alone on its SM took 4600 cycles for an
// absorber plane, and loading the absorber's auxiliaries earlier made it
// slower).  With 16-byte shared and global accesses a row of four nodes costs
// 10 shared loads instead of 48 and a quarter of the address arithmetic and
// stores, and the 4 warps of a 16-row tile have one halo task each, where 8
// warps left the upper four waiting at the barrier.  Measured against two nodes
// a thread (32 lanes along z, two rows): 384^3 with a 12-cell CPML 739 -> 592 us
// a step (algorithmic bytes at 5.4 TB/s), without absorber 508 -> 454 us (6.0
// TB/s), 128^3 with a 10-cell CPML 57 -> 40 us.
//
// The node updates are the expressions of stream_body (dtmx_stream.cuh), in
// the same order with the same explicitly rounded operations (sums with an
// exact zero and products with an exact one left out), so without a TF/SF
// source this engine's fields equal the per-step engine's.  With one, the H
// correction is added to the old H before the sweep (the update is linear in
// it), which rounds differently at the box faces.
#pragma once
#include "dtmx_stream.cuh"

namespace dtmx {

constexpr int FE_W = 40;                     // E box: z in [k0-4, k0+36) (16-byte aligned start)
constexpr int FHX_W = 36, FHY_W = 36, FHZ_W = 32;
constexpr int F_NST = 3;
constexpr int HN_P = 36;                     // new-H plane buffer: z in [k0, k0+33), rows 16-byte aligned
constexpr int FX_MAX = 64;                   // longest x chunk
constexpr int F_MROWS = 16;                  // material tiles: the per-step kernels' 32 x 16 boxes
__host__ __device__ constexpr int f_up32(int v) { return (v + 31) / 32 * 32; }

// Shared-memory layout of a tile of TY rows, in floats.
template <int TY>
struct FL {
  static constexpr int NT = 8 * TY;                  // threads: eight a row
  static constexpr int NW = NT / 32;
  static constexpr int TASKS = NW >= 4 ? 1 : 4 / NW; // halo tasks of a warp (4 in all)
  static constexpr int FE_R = TY + 2;                // E box rows: y in [j0-1, j0+TY+1)
  static constexpr int FE_N = f_up32(FE_R * FE_W);
  static constexpr int FHX_R = TY + 1, FHY_R = TY, FHZ_R = TY + 1;   // old-H boxes
  static constexpr int OFF_HX = 3 * FE_N;
  static constexpr int OFF_HY = OFF_HX + f_up32(FHX_W * FHX_R);
  static constexpr int OFF_HZ = OFF_HY + f_up32(FHY_W * FHY_R);
  static constexpr int OFF_M = OFF_HZ + f_up32(FHZ_W * FHZ_R);
  static constexpr int STAGE = OFF_M + 3 * F_MROWS * TZ / 4;
  static constexpr unsigned BYTES = (3 * FE_W * FE_R + FHX_W * FHX_R + FHY_W * FHY_R + FHZ_W * FHZ_R) * 4;
  static constexpr unsigned BYTES_MAT = 3 * F_MROWS * TZ;
  static constexpr int HN_N = (TY + 1) * HN_P;       // new-H plane, per component: y in [j0, j0+TY+1)
  static constexpr int HN = f_up32(3 * HN_N);
  // CPML coefficients (absorber runs): per x plane x0-1 .. x0+FX_MAX and per row
  // j0 .. j0+TY six floats (b, a, 1/kappa - 1 at the half-coordinate 2v of the H
  // components' derivatives, then at 2v + 1 of the E components'); per z
  // column k0 .. k0+32 the same six as arrays of 36
  static constexpr int FCO_X = 0, FCO_Y = (FX_MAX + 2) * 6, FCO_Z = (FCO_Y + (TY + 1) * 6 + 3) / 4 * 4, FCO_N = FCO_Z + 6 * 36;
  static constexpr size_t SMEM = (size_t)(F_NST * STAGE + 2 * HN + f_up32(FCO_N)) * 4 + MAXMAT * 3 * 4 + F_NST * 8 + 128;
};
static_assert(FL<16>::STAGE == 4352 && FL<16>::OFF_HX == 2208, "16-row layout");

// TMA descriptors of one buffer set for one tile height
struct FusedMaps {
  CUtensorMap e[3];                          // 40 x (TY+2) E boxes
  CUtensorMap hx, hy, hz;                    // old-H boxes
  CUtensorMap mat[3];                        // 32 x 16 material tiles (the per-step kernels' maps)
};

// Per-launch arguments beyond Params (which describes the source buffer A)
struct FusedArgs {
  float* dst[6];                             // buffer B
  float* hsrc[3][2];                         // CPML auxiliaries of H (slots 2, 3) in A
  float* hdst[3][2];                         // ... and in B
};

// staged-tile addresses (tile-local y, z)
template <int TY> __device__ __forceinline__ const float* fE(const float* st, int c, int y, int z) { return st + c * FL<TY>::FE_N + (y + 1) * FE_W + z + 4; }
template <int TY> __device__ __forceinline__ const float* fHx(const float* st, int y, int z) { return st + FL<TY>::OFF_HX + y * FHX_W + z; }
template <int TY> __device__ __forceinline__ const float* fHy(const float* st, int y, int z) { return st + FL<TY>::OFF_HY + y * FHY_W + z; }
template <int TY> __device__ __forceinline__ const float* fHz(const float* st, int y, int z) { return st + FL<TY>::OFF_HZ + y * FHZ_W + z; }
template <int TY> __device__ __forceinline__ float* fN(float* hn, int q, int y, int z) { return hn + q * FL<TY>::HN_N + y * HN_P + z; }
template <int TY> __device__ __forceinline__ const float* fN(const float* hn, int q, int y, int z) { return hn + q * FL<TY>::HN_N + y * HN_P + z; }

// The old auxiliaries of the thread's nodes in plane i, all axes: requested
// before the stage wait, used after it.  H reads set A, E its own in place.
template <bool ISH>
__device__ __forceinline__ void fused_aux_load(const Params& p, const FusedArgs& fa, const FNode& f, int i, int xs, Q4 (&o)[3][2]) {
  if (f.nv == 0) return;
  const unsigned nm = (1u << f.nv) - 1u;
  if (xs >= 0) {
    const int s = slab_at(p, 0, i, f.j, f.k, xs);
#pragma unroll
    for (int q = 0; q < 2; q++) o[0][q] = aux4<ISH>((ISH ? fa.hsrc[0][q] : p.ab.aux[0][q]) + s, f.vxy, nm);
  }
  if (f.ys >= 0) {
    const int s = slab_at(p, 1, i, f.j, f.k, f.ys);
#pragma unroll
    for (int q = 0; q < 2; q++) o[1][q] = aux4<ISH>((ISH ? fa.hsrc[1][q] : p.ab.aux[1][q]) + s, f.vxy, nm);
  }
  if (f.zm) {
    const int s = slab_at(p, 2, i, f.j, f.k, f.zs);
#pragma unroll
    for (int q = 0; q < 2; q++) o[2][q] = aux4<ISH>((ISH ? fa.hsrc[2][q] : p.ab.aux[2][q]) + s, f.vz, f.zm);
  }
}

// one axis' term of four nodes of one component: psi <- b psi + a d, corr += (1/kappa - 1) d + psi
__device__ __forceinline__ void cpml4(const Q4& d, const float (&b)[4], const float (&a)[4], const float (&c)[4], unsigned m, bool vec,
                                      bool store, const Q4& old, float* mem, Q4& corr) {
  Q4 nv;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    nv.v[e] = __fmaf_rn(b[e], old.v[e], __fmul_rn(a[e], d.v[e]));
    const float t = __fmaf_rn(c[e], d.v[e], nv.v[e]);
    corr.v[e] = __fadd_rn(corr.v[e], (m >> e) & 1 ? t : 0.f);
  }
  if (store) put4(mem, vec, m, nv);
}

// CPML corrections of four nodes (the arithmetic of absorb4) from their
// scaled derivative terms dxy etc. (component, axis); inc += sum over the axes.
template <int TY, bool ISH>
__device__ __forceinline__ void fused_cpml(const Params& p, const FusedArgs& fa, const FNode& f, int i, int xs, const float* fco, int xrow,
                                           const Q4 (&o)[3][2], bool store, const Q4& d01, const Q4& d02, const Q4& d10, const Q4& d12,
                                           const Q4& d20, const Q4& d21, Q4 (&inc)[3]) {
  if (f.nv == 0 || (xs < 0 && f.ys < 0 && f.zm == 0)) return;
  constexpr int O = ISH ? 0 : 3;
  const unsigned nm = (1u << f.nv) - 1u;
  Q4 corr[3];
#pragma unroll
  for (int c = 0; c < 3; c++) corr[c] = Q4{{0.f, 0.f, 0.f, 0.f}};
  auto same = [](float v, float (&r)[4]) { r[0] = r[1] = r[2] = r[3] = v; };
  float b[4], a[4], c[4];
  if (xs >= 0) {
    const float* cf = fco + FL<TY>::FCO_X + xrow * 6 + O;
    same(cf[0], b); same(cf[1], a); same(cf[2], c);
    const int s = slab_at(p, 0, i, f.j, f.k, xs);
    cpml4(d10, b, a, c, nm, f.vxy, store, o[0][0], (ISH ? fa.hdst[0][0] : p.ab.aux[0][0]) + s, corr[1]);
    cpml4(d20, b, a, c, nm, f.vxy, store, o[0][1], (ISH ? fa.hdst[0][1] : p.ab.aux[0][1]) + s, corr[2]);
  }
  if (f.ys >= 0) {
    const float* cf = fco + FL<TY>::FCO_Y + f.y * 6 + O;
    same(cf[0], b); same(cf[1], a); same(cf[2], c);
    const int s = slab_at(p, 1, i, f.j, f.k, f.ys);
    cpml4(d01, b, a, c, nm, f.vxy, store, o[1][0], (ISH ? fa.hdst[1][0] : p.ab.aux[1][0]) + s, corr[0]);
    cpml4(d21, b, a, c, nm, f.vxy, store, o[1][1], (ISH ? fa.hdst[1][1] : p.ab.aux[1][1]) + s, corr[2]);
  }
  if (f.zm) {
    const float* cf = fco + FL<TY>::FCO_Z + O * 36 + f.z;
    const Q4 tb = ld4(cf), ta = ld4(cf + 36), tc = ld4(cf + 72);
    const int s = slab_at(p, 2, i, f.j, f.k, f.zs);
    cpml4(d02, tb.v, ta.v, tc.v, f.zm, f.vz, store, o[2][0], (ISH ? fa.hdst[2][0] : p.ab.aux[2][0]) + s, corr[0]);
    cpml4(d12, tb.v, ta.v, tc.v, f.zm, f.vz, store, o[2][1], (ISH ? fa.hdst[2][1] : p.ab.aux[2][1]) + s, corr[1]);
  }
#pragma unroll
  for (int q = 0; q < 3; q++)
#pragma unroll
    for (int e = 0; e < 4; e++) inc[q].v[e] = __fadd_rn(inc[q].v[e], corr[q].v[e]);
}

// New H of plane i on the thread's nodes: hc (registers), hn (shared plane
// buffer), B (when the chunk owns plane i).  ec gets the old E of the own nodes
// (the next plane's x taps and its E update); ep holds those of plane i - 1.
template <int TY, bool ABS>
__device__ __forceinline__ void fused_h_own(const Params& p, const FusedArgs& fa, const float* st, float* hn, const FNode& f, int i,
                                            bool store, const Q4 (&ep)[3], Q4 (&hc)[3], Q4 (&ec)[3], const float* fco, int xrow, int xs,
                                            const Q4 (&o)[3][2]) {
  const float cx = p.cdt[0], cy = p.cdt[1], cz = p.cdt[2];
  const Q4 ex = ld4(fE<TY>(st, 0, f.y, f.z)), ey = ld4(fE<TY>(st, 1, f.y, f.z)), ez = ld4(fE<TY>(st, 2, f.y, f.z));
  const Q4 exm = ld4(fE<TY>(st, 0, f.y - 1, f.z)), ezm = ld4(fE<TY>(st, 2, f.y - 1, f.z));
  const float exl = *fE<TY>(st, 0, f.y, f.z - 1), eyl = *fE<TY>(st, 1, f.y, f.z - 1);
  // Hx -= dt(dy Ez - dz Ey); Hy -= dt(dz Ex - dx Ez); Hz -= dt(dx Ey - dy Ex)
  const Q4 d01 = diff4(-cy, ez, ezm), d02 = diff4(cz, ey, below4(eyl, ey));
  const Q4 d10 = diff4(cx, ez, ep[2]), d12 = diff4(-cz, ex, below4(exl, ex));
  const Q4 d20 = diff4(-cx, ey, ep[1]), d21 = diff4(cy, ex, exm);
  ec[0] = ex; ec[1] = ey; ec[2] = ez;
  Q4 inc[3] = {add4(d01, d02), add4(d10, d12), add4(d20, d21)};
  if (ABS) fused_cpml<TY, true>(p, fa, f, i, xs, fco, xrow, o, store, d01, d02, d10, d12, d20, d21, inc);
  hc[0] = add4(ld4(fHx<TY>(st, f.y, f.z)), inc[0]);
  hc[1] = add4(ld4(fHy<TY>(st, f.y, f.z)), inc[1]);
  hc[2] = add4(ld4(fHz<TY>(st, f.y, f.z)), inc[2]);
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
}

// The halo of the new-H plane buffer (values the E update of the tile reads
// beyond its own nodes), one component per task, one node per lane:
//   task 0: Hz of row TY      task 1: Hx of row TY
//   task 2: Hy of column 32   task 3: Hx of column 32 (lanes below TY)
// Each component has two derivative axes, a0 < a1.
struct FHalo {
  int y, z, j, k;
  int ysh, zsh;              // slab coordinates of the node's row and column (-1 outside)
  bool on, ok;               // the lane has a node / it lies in the grid
};
__device__ __forceinline__ int halo_a0(int task) { return task & 1; }
__device__ __forceinline__ int halo_a1(int task) { return task == 0 ? 1 : 2; }
// old auxiliaries of both axes (slots: Hz 1 and 1; Hx 0 and 0; Hy 0 on x, 1 on z), read only
__device__ __forceinline__ void fused_halo_load(const Params& p, const FusedArgs& fa, int task, const FHalo& h, int i, int xs, float (&q)[2]) {
  q[0] = q[1] = 0.f;
  if (!h.ok) return;
  const int s0 = task & 1 ? h.ysh : xs, s1 = task == 0 ? h.ysh : h.zsh;
  if (s0 >= 0) q[0] = __ldg((task == 0 ? fa.hsrc[0][1] : task == 2 ? fa.hsrc[0][0] : fa.hsrc[1][0]) + slab_at(p, halo_a0(task), i, h.j, h.k, s0));
  if (s1 >= 0) q[1] = __ldg((task == 0 ? fa.hsrc[1][1] : task == 2 ? fa.hsrc[2][1] : fa.hsrc[2][0]) + slab_at(p, halo_a1(task), i, h.j, h.k, s1));
}
// xe: the old E of the previous plane at the halo node (x tap), updated
template <int TY, bool ABS>
__device__ __forceinline__ void fused_h_halo(const Params& p, const float* st, float* hn, int task, const FHalo& h, float& xe,
                                             const float* fco, int xrow, int xs, const float (&q)[2]) {
  if (!h.on) return;
  const float cx = p.cdt[0], cy = p.cdt[1], cz = p.cdt[2];
  float d0, d1, old;
  if (task == 0) {
    const float ey = *fE<TY>(st, 1, h.y, h.z);
    d0 = __fmul_rn(-cx, __fsub_rn(ey, xe));
    d1 = __fmul_rn(cy, __fsub_rn(*fE<TY>(st, 0, h.y, h.z), *fE<TY>(st, 0, h.y - 1, h.z)));
    old = *fHz<TY>(st, h.y, h.z);
    xe = ey;
  } else if (task == 2) {
    const float ez = *fE<TY>(st, 2, h.y, h.z);
    d0 = __fmul_rn(cx, __fsub_rn(ez, xe));
    d1 = __fmul_rn(-cz, __fsub_rn(*fE<TY>(st, 0, h.y, h.z), *fE<TY>(st, 0, h.y, h.z - 1)));
    old = *fHy<TY>(st, h.y, h.z);
    xe = ez;
  } else {
    d0 = __fmul_rn(-cy, __fsub_rn(*fE<TY>(st, 2, h.y, h.z), *fE<TY>(st, 2, h.y - 1, h.z)));
    d1 = __fmul_rn(cz, __fsub_rn(*fE<TY>(st, 1, h.y, h.z), *fE<TY>(st, 1, h.y, h.z - 1)));
    old = *fHx<TY>(st, h.y, h.z);
  }
  float inc = __fadd_rn(d0, d1);
  if (ABS) {
    float corr = 0.f;
    if ((task & 1 ? h.ysh : xs) >= 0) {
      const float* c = fco + (task & 1 ? FL<TY>::FCO_Y + h.y * 6 : FL<TY>::FCO_X + xrow * 6);
      corr = __fmaf_rn(c[2], d0, __fmaf_rn(c[0], q[0], __fmul_rn(c[1], d0)));
    }
    if ((task == 0 ? h.ysh : h.zsh) >= 0) {
      const float* c = fco + (task == 0 ? FL<TY>::FCO_Y + h.y * 6 : FL<TY>::FCO_Z + h.z);
      const int s = task == 0 ? 1 : 36;
      corr = __fadd_rn(corr, __fmaf_rn(c[2 * s], d1, __fmaf_rn(c[0], q[1], __fmul_rn(c[s], d1))));
    }
    inc = __fadd_rn(inc, corr);
  }
  *fN<TY>(hn, task == 0 ? 2 : task == 2 ? 1 : 0, h.y, h.z) = h.ok ? __fadd_rn(old, inc) : 0.f;
}

// New E of plane i on the own nodes.  ep: old E (registers), hn: new H of
// plane i (shared), hc: new H of plane i + 1 (own nodes).
//   MODE 2: vacuum; MODE 1: uniform non-dispersive material um;
//   MODE 0: general (mixed materials, design region).  A dispersive node's table
//           entry is -0, so it keeps its old E here and the ADE pass writes it
//           (its absorber auxiliaries, if it has any, stay 0).
template <int TY, int MODE, bool ABS>
__device__ __forceinline__ void fused_e_own(const Params& p, const FusedArgs& fa, const float* st, const float* hn, const float* ies, int um,
                                            const FNode& f, int i, const Q4 (&ep)[3], const Q4 (&hc)[3], const float* fco, int xrow, int xs,
                                            const Q4 (&o)[3][2]) {
  if (f.nv == 0) return;
  const float cx = p.cdt[0], cy = p.cdt[1], cz = p.cdt[2];
  const Q4 hx = ld4(fN<TY>(hn, 0, f.y, f.z)), hy = ld4(fN<TY>(hn, 1, f.y, f.z)), hz = ld4(fN<TY>(hn, 2, f.y, f.z));
  const Q4 hxp = ld4(fN<TY>(hn, 0, f.y + 1, f.z)), hzp = ld4(fN<TY>(hn, 2, f.y + 1, f.z));
  const float hxr = *fN<TY>(hn, 0, f.y, f.z + 4), hyr = *fN<TY>(hn, 1, f.y, f.z + 4);
  // Ex += dt/eps(dy Hz - dz Hy); Ey += dt/eps(dz Hx - dx Hz); Ez += dt/eps(dx Hy - dy Hx)
  Q4 d01 = diff4(cy, hzp, hz), d02 = diff4(-cz, above4(hy, hyr), hy);
  Q4 d10 = diff4(-cx, hc[2], hz), d12 = diff4(cz, above4(hx, hxr), hx);
  Q4 d20 = diff4(cx, hc[1], hy), d21 = diff4(-cy, hxp, hx);
  if (MODE == 1) {
    const float i0 = ies[um * 3], i1 = ies[um * 3 + 1], i2 = ies[um * 3 + 2];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      d01.v[e] = __fmul_rn(d01.v[e], i0); d02.v[e] = __fmul_rn(d02.v[e], i0);
      d10.v[e] = __fmul_rn(d10.v[e], i1); d12.v[e] = __fmul_rn(d12.v[e], i1);
      d20.v[e] = __fmul_rn(d20.v[e], i2); d21.v[e] = __fmul_rn(d21.v[e], i2);
    }
  }
  if (MODE == 0) {
    const unsigned* mt = reinterpret_cast<const unsigned*>(st + FL<TY>::OFF_M);
    unsigned m[3];
#pragma unroll
    for (int c = 0; c < 3; c++) m[c] = mt[(c * F_MROWS * TZ + f.y * TZ + f.z) / 4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      float ie[3];
#pragma unroll
      for (int c = 0; c < 3; c++) ie[c] = ies[((m[c] >> (8 * e)) & 255u) * 3 + c];
      if (p.des_on) {
        const long long di = design_index(p, i, f.j, f.k + e);
        if (di >= 0) {
#pragma unroll
          for (int c = 0; c < 3; c++)
            if (!is_dispersive(ie[c])) ie[c] = p.des_ie[c][di];     // (a dispersive design node keeps its ADE update)
        }
      }
      d01.v[e] = __fmul_rn(d01.v[e], ie[0]); d02.v[e] = __fmul_rn(d02.v[e], ie[0]);
      d10.v[e] = __fmul_rn(d10.v[e], ie[1]); d12.v[e] = __fmul_rn(d12.v[e], ie[1]);
      d20.v[e] = __fmul_rn(d20.v[e], ie[2]); d21.v[e] = __fmul_rn(d21.v[e], ie[2]);
    }
  }
  Q4 inc[3] = {add4(d01, d02), add4(d10, d12), add4(d20, d21)};
  if (ABS) fused_cpml<TY, false>(p, fa, f, i, xs, fco, xrow, o, true, d01, d02, d10, d12, d20, d21, inc);
  const long long off = (long long)i * p.g.sx + (long long)f.j * p.g.sy + f.k;
#pragma unroll
  for (int c = 0; c < 3; c++) st4(fa.dst[c] + off, add4(ep[c], inc[c]));
}

// Issue the copies of stage s (plane x0 - 1 + s; the material tiles of the
// plane before it, whose E update runs while this stage is current).
template <int TY>
__device__ __forceinline__ void fused_issue(const FusedMaps& m, float* st, uint64_t* bar, int ip, int j0, int k0,
                                            bool want_mat) {
  mbar_arrive_expect_tx(bar, FL<TY>::BYTES + (want_mat ? FL<TY>::BYTES_MAT : 0u));
#pragma unroll
  for (int c = 0; c < 3; c++) tma_load_3d(st + c * FL<TY>::FE_N, &m.e[c], k0 - 4, j0 - 1, ip, bar);
  tma_load_3d(st + FL<TY>::OFF_HX, &m.hx, k0, j0, ip, bar);
  tma_load_3d(st + FL<TY>::OFF_HY, &m.hy, k0, j0, ip, bar);
  tma_load_3d(st + FL<TY>::OFF_HZ, &m.hz, k0, j0, ip, bar);
  if (want_mat)
#pragma unroll
    for (int c = 0; c < 3; c++)
      tma_load_3d(reinterpret_cast<uint8_t*>(st + FL<TY>::OFF_M) + c * F_MROWS * TZ, &m.mat[c], k0, j0, ip - 1, bar);
}

// 16 rows: 3 CTAs per SM, what shared memory allows (a 3-stage ring and two
// new-H planes); 8 rows: 5
template <int TY, bool TAB>
__global__ void __launch_bounds__(FL<TY>::NT, TY == 16 ? 3 : 5)
    fused_kernel(const __grid_constant__ Params p, const __grid_constant__ FusedArgs fa,
                 const __grid_constant__ FusedMaps m, const __grid_constant__ Work<TAB> work) {
  using L = FL<TY>;
  extern __shared__ __align__(128) float fsm[];
  float* hnb = fsm + F_NST * L::STAGE;                           // two new-H planes
  float* fco = hnb + 2 * L::HN;
  float* ies = fco + f_up32(L::FCO_N);                           // 1/eps of the material table
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
    // coefficient row q: x plane x0 - 1 + q, then y row j0 + ..., then z column k0 + ...
    constexpr int RX = FX_MAX + 2, RY_ = TY + 1, RZ = TZ + 1;
    for (int q = tid; q < RX + RY_ + RZ; q += L::NT) {
      const int a = q < RX ? 0 : q < RX + RY_ ? 1 : 2;
      const int v0 = a == 0 ? q : a == 1 ? q - RX : q - RX - RY_;
      const int v = v0 + (a == 0 ? x0 - 1 : a == 1 ? j0 : k0);
      if (a == 0 && v0 > len + 1) continue;
#pragma unroll
      for (int o = 0; o < 2; o++) {
        const int h = 2 * v + o;
        const bool in = h >= 0 && h < 2 * p.g.n[a] + 2;
        const float cb = in ? __ldg(p.ab.c0[a] + h) : 1.f, ca = in ? __ldg(p.ab.c1[a] + h) : 0.f;
        const float cc = in ? __fsub_rn(__ldg(p.ab.c2[a] + h), 1.f) : 0.f;
        float* d = a == 2 ? fco + L::FCO_Z + 3 * o * 36 + v0 : fco + (a == 0 ? L::FCO_X : L::FCO_Y) + v0 * 6 + 3 * o;
        const int s = a == 2 ? 36 : 1;
        d[0] = cb; d[s] = ca; d[2 * s] = cc;
      }
    }
  }
  pdl_wait();
  pdl_trigger();
  __syncthreads();
  // stage s: plane x0 - 1 + s, with the materials of the plane before it (s >= 2)
  if (tid == 0 && slast >= 2) { issue(2, umc[0] < 0); issued = 2; }
  // per-thread constants of the walk
  FNode f;
  f.y = tid >> 3; f.z = 4 * (tid & 7);
  f.j = j0 + f.y; f.k = k0 + f.z;
  f.nv = f.j < p.g.n[1] ? min(4, max(0, p.g.n[2] - f.k)) : 0;
  f.ys = cpml ? slab_cs(p, 1, f.j) : -1;
  f.zs = 0; f.zm = 0;
  if (cpml) {
    // (the grid is at least four cells wider than both slabs, so four nodes meet one of them at most)
    const int lo = p.ab.L[2][0], hi = p.g.n[2] - p.ab.L[2][1];
    f.zs = f.k < lo ? f.k : f.k + lo - hi;
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (e < f.nv && (f.k + e < lo || f.k + e >= hi)) f.zm |= 1u << e;
  }
  f.vxy = (p.g.n[2] & 3) == 0;
  f.vz = f.zm == 15u && ((p.ab.L[2][0] + p.ab.L[2][1]) & 3) == 0 && (f.zs & 3) == 0;
  FHalo hl[L::TASKS];
  float xe[L::TASKS], hq[L::TASKS][2];
#pragma unroll
  for (int q = 0; q < L::TASKS; q++) {
    const int task = w + q * L::NW;
    const bool row = task < 2;
    hl[q].y = row ? TY : lane; hl[q].z = row ? lane : TZ;
    hl[q].j = j0 + hl[q].y; hl[q].k = k0 + hl[q].z;
    hl[q].on = task < 4 && (row || lane < TY);
    hl[q].ok = hl[q].on && hl[q].j < p.g.n[1] && hl[q].k < p.g.n[2];
    hl[q].ysh = cpml ? slab_cs(p, 1, hl[q].j) : -1;
    hl[q].zsh = cpml ? slab_cs(p, 2, hl[q].k) : -1;
    xe[q] = 0.f; hq[q][0] = hq[q][1] = 0.f;
  }
  // does the tile (own nodes, then with the halo) meet a y or z slab?
  const bool own_yz = cpml && (j0 < p.ab.L[1][0] || j0 + TY > p.g.n[1] - p.ab.L[1][1] || k0 < p.ab.L[2][0] ||
                               k0 + TZ > p.g.n[2] - p.ab.L[2][1]);
  const bool halo_yz = cpml && (own_yz || j0 + TY + 1 > p.g.n[1] - p.ab.L[1][1] || k0 + TZ + 1 > p.g.n[2] - p.ab.L[2][1]);
  Q4 ep[3], hc[3], ec[3], oh[3][2], oe[3][2];
  // stage 0 (plane x0 - 1): the old E of the own nodes and of the halo nodes (x taps)
  if (tid == 0 && !mbar_wait(&bars[0], 0u, p.err, p.wait_limit)) gave_up = 1;
  __syncthreads();
  int t = 0, swait = 0;                                    // swait: the stage waited for last
  if (!gave_up) {
#pragma unroll
    for (int c = 0; c < 3; c++) ep[c] = ld4(fE<TY>(fsm, c, f.y, f.z));
#pragma unroll
    for (int q = 0; q < L::TASKS; q++) {
      const int task = w + q * L::NW;
      if (hl[q].on && !(task & 1)) xe[q] = *fE<TY>(fsm, task == 0 ? 1 : 2, hl[q].y, hl[q].z);
    }
    for (; t <= len; t++) {
      const int s = t + 1, pc = x0 + t, pe = pc - 1;
      const int xs = cpml ? slab_cs(p, 0, pc) : -1, xse = cpml ? slab_cs(p, 0, pe) : -1;
      const bool abh = own_yz || xs >= 0, abe = own_yz || xse >= 0, abl = halo_yz || xs >= 0;
      // absorber tile-planes: the old auxiliaries, requested before the stage wait
      if (pc < p.g.n[0]) {
        if (abh) fused_aux_load<true>(p, fa, f, pc, xs, oh);
        if (abl)
#pragma unroll
          for (int q = 0; q < L::TASKS; q++) fused_halo_load(p, fa, w + q * L::NW, hl[q], pc, xs, hq[q]);
      }
      if (t >= 1 && abe) fused_aux_load<false>(p, fa, f, pe, xse, oe);
      swait = s;
      if (tid == 0 && !mbar_wait(&bars[s % F_NST], (unsigned)((s / F_NST) & 1), p.err, p.wait_limit)) gave_up = 1;
      // every thread is past iteration t - 1: the slot of stage t and the new-H
      // plane written two iterations ago are free
      __syncthreads();
      if (gave_up) break;
      if (tid == 0 && t + F_NST <= slast) { issue(t + F_NST, umc[t + F_NST - 2] < 0); issued = t + F_NST; }
      const float* st = fsm + (s % F_NST) * L::STAGE;
      float* hn1 = hnb + (t & 1) * L::HN;                        // new H of plane pc
      const float* hn0 = hnb + ((t + 1) & 1) * L::HN;            // new H of plane pc - 1
      if (pc < p.g.n[0]) {
        if (abh) fused_h_own<TY, true>(p, fa, st, hn1, f, pc, t < len, ep, hc, ec, fco, t + 1, xs, oh);
        else fused_h_own<TY, false>(p, fa, st, hn1, f, pc, t < len, ep, hc, ec, fco, t + 1, xs, oh);
#pragma unroll
        for (int q = 0; q < L::TASKS; q++) {
          const int task = w + q * L::NW;
          if (abl) fused_h_halo<TY, true>(p, st, hn1, task, hl[q], xe[q], fco, t + 1, xs, hq[q]);
          else fused_h_halo<TY, false>(p, st, hn1, task, hl[q], xe[q], fco, t + 1, xs, hq[q]);
        }
      } else {
        // beyond the last plane of the grid: H is zero there
#pragma unroll
        for (int c = 0; c < 3; c++) { hc[c] = Q4{{0.f, 0.f, 0.f, 0.f}}; ec[c] = hc[c]; }
      }
      if (t >= 1) {
        const int um = umc[pe - x0];
        const bool vac = um >= 0 && ies[um * 3] == 1.f && ies[um * 3 + 1] == 1.f && ies[um * 3 + 2] == 1.f;
        switch ((vac ? 4 : um >= 0 ? 2 : 0) + (abe ? 1 : 0)) {
          case 5: fused_e_own<TY, 2, true>(p, fa, st, hn0, ies, um, f, pe, ep, hc, fco, t, xse, oe); break;
          case 4: fused_e_own<TY, 2, false>(p, fa, st, hn0, ies, um, f, pe, ep, hc, fco, t, xse, oe); break;
          case 3: fused_e_own<TY, 1, true>(p, fa, st, hn0, ies, um, f, pe, ep, hc, fco, t, xse, oe); break;
          case 2: fused_e_own<TY, 1, false>(p, fa, st, hn0, ies, um, f, pe, ep, hc, fco, t, xse, oe); break;
          case 1: fused_e_own<TY, 0, true>(p, fa, st, hn0, ies, um, f, pe, ep, hc, fco, t, xse, oe); break;
          default: fused_e_own<TY, 0, false>(p, fa, st, hn0, ies, um, f, pe, ep, hc, fco, t, xse, oe); break;
        }
      }
#pragma unroll
      for (int c = 0; c < 3; c++) ep[c] = ec[c];
    }
  }
  if (gave_up && tid == 0) {
    // a wait gave up: no further copies were issued; wait (bounded) for those in flight, then leave
    for (int s = swait; s <= issued; s++) mbar_wait(&bars[s % F_NST], (unsigned)((s / F_NST) & 1), nullptr, DRAIN_POLLS);
  }
}

}  // namespace dtmx
