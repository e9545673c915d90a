// dtmx_device.cuh -- device-side data structures and per-plane field updates.
//
// The unit of work is one (z,y) tile of one x-plane: TZ = 32 nodes along z by
// TYT = 16 along y, eight threads a row with four consecutive z nodes each
// (16-byte shared and global accesses).  The y/z taps of the derivatives come
// from shared-memory copies of the neighbouring field's plane tile; the x taps
// from a register queue while a CTA streams along x.  Absorber (CPML or the
// reference split-field PML) and material coefficients are applied in the same
// pass; the Drude/Lorentz ADE nodes (reference countDisp) and the gyrotropic
// current are finished by a pass over the dispersive box after the E half step.
//
// Update equations (reference generator genAlg.py:182-301, defs.h:3-13):
//   H -= dt * curl E,  E += dt/eps * curl H  (c = 1),
//   D f = (27 (f[+1/2] - f[-1/2]) - (f[+3/2] - f[-3/2])) / 24   (order 4)
//   D f = f[+1/2] - f[-1/2]                                     (order 2)
// H nodes take taps at index offsets -2..+1, E nodes at -1..+2.
#pragma once
#include <cstdint>
#include <cuda.h>
#include <cuda_runtime.h>

namespace dtmx {

constexpr int TZ = 32;          // tile extent along z: eight threads of four nodes
constexpr int TYT = 16;          // tile extent along y
constexpr int MAXMAT = 64;
constexpr int MAXPOLE = 2;

// Programmatic dependent launch.  A step is a chain of launches on one stream, on
// small grids of a few microseconds each.  Every kernel of the chain waits for the
// one before (pdl_wait) ahead of anything that one may have written; what comes
// before the wait reads only tables that no step changes.  All but the per-step
// field kernels and the DFT fold let the next one start its set-up (pdl_trigger);
// after those it starts when they end.  Each kernel waits in all its threads (the
// fold is launched without the attribute), so a finished kernel means that all
// before it have finished.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// half-cell offset of component c along axis a (lattice in dtmx.h)
__host__ __device__ __forceinline__ int comp_off(int c, int a) { return c < 3 ? (a != c) : (a == c - 3); }

struct Grid {
  int n[3];
  long long sx, sy;          // element strides of x and y (z stride 1)
  int live_lo[6][3], live_hi[6][3];
  int all_lo[3], all_hi[3];  // index range live for every component
  int btype[3][2], bplane[3][2];
  int bsE[3][2], bsH[3][2];
  int box;                   // box geometry: every node of the array is live, zero outside
};

struct Absorb {
  int kind;                  // 0 none, 1 CPML, 2 split PML
  int L[3][2];               // slab thickness in cells
  float* aux[3][4];          // per axis: 4 slots (2 E comps, 2 H comps) over the slab cells
  const float* c0[3];        // CPML b      | split K1     (indexed by half-coordinate)
  const float* c1[3];        // CPML a      | split K2
  const float* c2[3];        // CPML 1/kappa
};

struct MatTable {
  float inv_eps[MAXMAT][3];
  int npoles[MAXMAT];
  float kEJ[MAXMAT][3][MAXPOLE][2];
  float kE[MAXMAT][3][3];
  float kJ[MAXMAT][3][MAXPOLE][5];
  // magnetised-Drude (gyrotropic) current: decay, rotation cos/sin, E drive, dt/eps_inf (0: not gyrotropic)
  float gA[MAXMAT], gC[MAXMAT], gS[MAXMAT], gB[MAXMAT], gjc[MAXMAT];
};

struct Ade {
  int lo[3], n[3];           // box of cells holding ADE state
  float* Em[3];
  float* Jp[3][MAXPOLE];
  float* Jm[3][MAXPOLE];
  float* Jg[2][3];           // gyrotropic current, double-buffered
};

struct Params {
  Grid g;
  float* f[6];
  float cdt[3];              // dt/dx, dt/dy, dt/dz
  Absorb ab;
  const uint8_t* mat[3];     // per E component material index (nullptr -> material 0)
  const MatTable* mt;
  Ade ade;
  int x0, x1;                // planes [x0, x1) of a wavefront launch
  int xchunk;                // planes per CTA of a streaming launch without a work table
  int* err;                  // device error word (bounded waits that gave up)
  long long wait_limit;      // polls of one bounded wait (2^26; lowered only to test the timeout paths)
  // per (plane, y tile, z tile): the single non-dispersive material of all E
  // nodes of that plane tile, or -1 when mixed/dispersive
  const signed char* umat;
  int ntz, nty;              // tiles along z and y
  // E of the previous step when a pass reads it from another buffer than the
  // one it writes (the single-sweep engine's ADE pass); nullptr: in place
  const float* fe_old[3];
  // design region: per-node 1/eps of the E components over a cell box
  const float* des_ie[3];
  int des_lo[3], des_n[3];
  int des_on;
};

// The piece of work of a CTA of a streaming launch: z tile, y tile, first plane
// and plane past the last, from the block index (equal pieces) or from a table
// (plan_work).  The table is in global memory: as a kernel argument of 4.7 KB it
// was no faster (128^3: 37.5 against 36.7 us).
template <bool TAB> struct Work { const int4* e; };
template <> struct Work<false> {};
template <bool TAB>
__device__ __forceinline__ int4 cta_job(const Params& p, const Work<TAB>& w) {
  if constexpr (TAB) {
    return __ldg(w.e + blockIdx.x);
  } else {
    const int x0 = blockIdx.z * p.xchunk;
    return make_int4(blockIdx.x, blockIdx.y, x0, min(x0 + p.xchunk, p.g.n[0]));
  }
}

__host__ __device__ __forceinline__ long long design_index(const Params& p, int i, int j, int k) {
  if (!p.des_on) return -1;
  const int a = i - p.des_lo[0], b = j - p.des_lo[1], c = k - p.des_lo[2];
  if (a < 0 || a >= p.des_n[0] || b < 0 || b >= p.des_n[1] || c < 0 || c >= p.des_n[2]) return -1;
  return ((long long)a * p.des_n[1] + b) * p.des_n[2] + c;
}

// TMA descriptors of one context: source tiles (40 z x rows y x 1 plane),
// own-value tiles (32 x 16 x 1) of every component and material tiles.
struct TmaMaps {
  CUtensorMap src[6];
  CUtensorMap own[6];
  CUtensorMap mat[3];
};

// storage slot of component c for derivative axis a (-1: c has no derivative along a)
__host__ __device__ __forceinline__ constexpr int slot_of(int c, int a) {
  // Ex: y->0 z->0 ; Ey: x->0 z->1 ; Ez: x->1 y->1 ; Hx: y->2 z->2 ; Hy: x->2 z->3 ; Hz: x->3 y->3
  // (a conditional expression: a table indexed by a run-time c would live in local memory)
  return c == 0 ? (a == 0 ? -1 : 0)
       : c == 1 ? (a == 0 ? 0 : a == 1 ? -1 : 1)
       : c == 2 ? (a == 2 ? -1 : 1)
       : c == 3 ? (a == 0 ? -1 : 2)
       : c == 4 ? (a == 0 ? 2 : a == 1 ? -1 : 3)
                : (a == 2 ? -1 : 3);
}

// Loads: LD = 0 read-only path (field not written during the launch),
// LD = 1 L2-coherent path (written by other CTAs of the same launch).
template <int LD>
__device__ __forceinline__ float ldf(const float* q) { return LD ? __ldcg(q) : __ldg(q); }

// Map index v of component c along axis a to the stored index, applying the
// boundary rule outside the live range; returns -1 when the value is zero.
__device__ __forceinline__ int map_idx(const Grid& g, int c, int a, int v, float& sgn) {
  const int lo = g.live_lo[c][a], hi = g.live_hi[c][a];
  if (v >= lo && v <= hi) return v;
  const int side = v < lo ? 0 : 1;
  if (g.btype[a][side] == 0) return (v >= 0 && v < g.n[a]) ? v : -1;   // non-live cells hold zero
  const int o = comp_off(c, a);
  const int h2 = 2 * g.bplane[a][side] - (2 * v + o);
  const int v2 = (h2 - o) >> 1;
  sgn *= (float)((c < 3) ? g.bsE[a][side] : g.bsH[a][side]);
  if (v2 < lo || v2 > hi) return -1;
  return v2;
}

template <int LD>
__device__ __forceinline__ float fetch(const Params& p, int c, int i, int j, int k) {
  float s = 1.f;
  const int ii = map_idx(p.g, c, 0, i, s);
  const int jj = map_idx(p.g, c, 1, j, s);
  const int kk = map_idx(p.g, c, 2, k, s);
  if ((ii | jj | kk) < 0) return 0.f;
  return s * ldf<LD>(p.f[c] + ii * p.g.sx + jj * p.g.sy + kk);
}

// The node update is written with explicitly rounded operations (__fadd_rn,
// __fmul_rn, __fmaf_rn: no compiler contraction), so every kernel that
// evaluates it -- the per-half-step kernels and the wavefront engine -- gets
// bit-identical results whatever code surrounds it.
template <int ORDER>
__device__ __forceinline__ float dstencil(float v0, float v1, float v2, float v3) {
  if (ORDER == 2) return __fsub_rn(v2, v1);
  return __fmul_rn(__fmaf_rn(27.f, __fsub_rn(v2, v1), __fsub_rn(v0, v3)), 1.f / 24.f);
}
__device__ __forceinline__ float sum3(float a, float b, float c) { return __fadd_rn(__fadd_rn(a, b), c); }

__device__ __forceinline__ bool is_live(const Grid& g, int c, int i, int j, int k) {
  return i >= g.live_lo[c][0] && i <= g.live_hi[c][0] && j >= g.live_lo[c][1] && j <= g.live_hi[c][1] &&
         k >= g.live_lo[c][2] && k <= g.live_hi[c][2];
}

__device__ __forceinline__ bool in_slab(const Params& p, int a, int v) {
  return v < p.ab.L[a][0] || v >= p.g.n[a] - p.ab.L[a][1];
}

__device__ __forceinline__ long long slab_index(const Params& p, int a, int i, int j, int k) {
  const int n = p.g.n[a];
  const int c = a == 0 ? i : a == 1 ? j : k;
  const int lo = p.ab.L[a][0], hi = p.ab.L[a][1];
  int cs;
  if (c < lo) cs = c;
  else if (c >= n - hi) cs = lo + (c - (n - hi));
  else return -1;
  const int th = lo + hi;
  if (a == 0) return ((long long)cs * p.g.n[1] + j) * p.g.n[2] + k;
  if (a == 1) return ((long long)i * th + cs) * p.g.n[2] + k;
  return ((long long)i * p.g.n[1] + j) * th + cs;
}

// Absorber correction of component c at a slab node: the update is
// F_new = F + dif[0] + dif[1] + dif[2] + correction, where for every slab axis a
//   CPML:  correction_a = (1/kappa_a - 1) dif_a + psi_a,  psi_a <- b psi_a + a dif_a
//   split: correction_a = (K1_a - 1) p_a + (K2_a - 1) dif_a,  p_a <- K1_a p_a + K2_a dif_a
// (the split form follows from F = rest + sum p_a with rest += undamped terms).
// Split into a load and an apply step so that callers can issue the slab
// loads early: absorb_load reads the auxiliary value of every slab axis of the
// node (0 elsewhere), absorb_apply computes the correction from those values
// and stores the new ones.
__device__ __forceinline__ void absorb_load(const Params& p, int c, int i, int j, int k, float (&old)[3]) {
  const int idx[3] = {i, j, k};
#pragma unroll
  for (int a = 0; a < 3; a++) {
    old[a] = 0.f;
    const int sl = slot_of(c, a);
    if (sl < 0 || !in_slab(p, a, idx[a])) continue;
    old[a] = p.ab.aux[a][sl][slab_index(p, a, i, j, k)];
  }
}
__device__ __forceinline__ float absorb_apply(const Params& p, int c, int i, int j, int k, const float* dif,
                                              const float (&old)[3]) {
  const int idx[3] = {i, j, k};
  float corr = 0.f;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int sl = slot_of(c, a);
    if (sl < 0 || !in_slab(p, a, idx[a])) continue;
    const long long si = slab_index(p, a, i, j, k);
    const int h = 2 * idx[a] + comp_off(c, a);
    const float k0 = __ldg(p.ab.c0[a] + h), k1 = __ldg(p.ab.c1[a] + h);
    const float nv = __fmaf_rn(k0, old[a], __fmul_rn(k1, dif[a]));
    p.ab.aux[a][sl][si] = nv;
    if (p.ab.kind == 1) corr = __fadd_rn(corr, __fmaf_rn(__fsub_rn(__ldg(p.ab.c2[a] + h), 1.f), dif[a], nv));
    else corr = __fadd_rn(corr, __fsub_rn(__fsub_rn(nv, old[a]), dif[a]));
  }
  return corr;
}

// slab index of a node along axis a (-1 outside that slab); 32-bit: every slab
// array holds fewer than 2^31 values, checked when the absorber is set up
__device__ __forceinline__ int slab_index32(const Params& p, int a, int i, int j, int k) {
  const int n = p.g.n[a], v = a == 0 ? i : a == 1 ? j : k;
  const int lo = p.ab.L[a][0], hi = p.ab.L[a][1];
  int cs;
  if (v < lo) cs = v;
  else if (v >= n - hi) cs = lo + (v - (n - hi));
  else return -1;
  if (a == 0) return (cs * p.g.n[1] + j) * p.g.n[2] + k;
  if (a == 1) return (i * (lo + hi) + cs) * p.g.n[2] + k;
  return (i * p.g.n[1] + j) * (lo + hi) + cs;
}
// slab indices of node (i,j,k); true when it lies in any slab
__device__ __forceinline__ bool node_slabs(const Params& p, int i, int j, int k, int (&si)[3]) {
  si[0] = slab_index32(p, 0, i, j, k);
  si[1] = slab_index32(p, 1, i, j, k);
  si[2] = slab_index32(p, 2, i, j, k);
  return (si[0] & si[1] & si[2]) >= 0;
}
// Per-thread absorber context of one node: which slabs hold it.
__device__ __forceinline__ bool node_in_absorber(const Params& p, bool inx, int j, int k) {
  return p.ab.kind != 0 && (inx || in_slab(p, 1, j) || in_slab(p, 2, k));
}

// ---------------------------------------------------------------- E half step
// ADE branch restates countDisp (dispersion.cpp:85-99).
__device__ __forceinline__ float ade_update(const Params& p, int c, int m, int np, long long ai, float rot, float F) {
  const MatTable& mt = *p.mt;
  const float Em = p.ade.Em[c][ai];
  const float Etmp = F;
  float sum = 0.f;
  float jp[MAXPOLE] = {}, jm[MAXPOLE] = {};
#pragma unroll
  for (int q = 0; q < MAXPOLE; q++)
    if (q < np) { jp[q] = p.ade.Jp[c][q][ai]; jm[q] = p.ade.Jm[c][q][ai]; }
#pragma unroll
  for (int q = 0; q < MAXPOLE; q++)
    if (q < np) sum = __fadd_rn(sum, __fmaf_rn(__ldg(&mt.kEJ[m][c][q][0]), jp[q], __fmul_rn(__ldg(&mt.kEJ[m][c][q][1]), jm[q])));
  const float Ep = __fsub_rn(__fmaf_rn(__ldg(&mt.kE[m][c][0]), Em,
                                       __fmaf_rn(__ldg(&mt.kE[m][c][1]), F, __fmul_rn(__ldg(&mt.kE[m][c][2]), rot))),
                             sum);
#pragma unroll
  for (int q = 0; q < MAXPOLE; q++) {
    if (q >= np) continue;
    float a = __fmul_rn(__ldg(&mt.kJ[m][c][q][4]), Etmp);
    a = __fmaf_rn(__ldg(&mt.kJ[m][c][q][3]), Em, a);
    a = __fmaf_rn(__ldg(&mt.kJ[m][c][q][2]), Ep, a);
    a = __fmaf_rn(__ldg(&mt.kJ[m][c][q][1]), jm[q], a);
    p.ade.Jp[c][q][ai] = __fmaf_rn(__ldg(&mt.kJ[m][c][q][0]), jp[q], a);
    p.ade.Jm[c][q][ai] = jp[q];
  }
  p.ade.Em[c][ai] = Etmp;
  return Ep;
}

// Material coefficients used on the common path, staged in shared memory.
struct MatShared {
  float inv_eps[MAXMAT][3];
  int npoles[MAXMAT];
  float gjc[MAXMAT];
};

// The 1/eps entry of a dispersive material is -0 (dtmx_set_materials): it adds
// nothing to E, and is told from a permittivity too large for 1/eps by its sign.
__device__ __forceinline__ bool is_dispersive(float ie) { return __float_as_uint(ie) == 0x80000000u; }

// ---- four consecutive z nodes a thread (the single sweep, its adjoint and the
// per-step kernels)
struct Q4 { float v[4]; };
__device__ __forceinline__ Q4 ld4(const float* s) {
  const float4 t = *reinterpret_cast<const float4*>(s);
  return Q4{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ void st4(float* d, const Q4& q) { *reinterpret_cast<float4*>(d) = make_float4(q.v[0], q.v[1], q.v[2], q.v[3]); }

// index of coordinate v in the slab of its axis (-1 outside)
__device__ __forceinline__ int slab_cs(const Params& p, int a, int v) {
  const int n = p.g.n[a], lo = p.ab.L[a][0], hi = p.ab.L[a][1];
  return v < lo ? v : (v >= n - hi ? lo + v - (n - hi) : -1);
}

// slab index of node (i, j, k) along axis a from its slab coordinate s on that axis (>= 0)
__device__ __forceinline__ int slab_at(const Params& p, int a, int i, int j, int k, int s) {
  if (a == 0) return (s * p.g.n[1] + j) * p.g.n[2] + k;
  if (a == 1) return (i * (p.ab.L[1][0] + p.ab.L[1][1]) + s) * p.g.n[2] + k;
  return (i * p.g.n[1] + j) * (p.ab.L[2][0] + p.ab.L[2][1]) + s;
}

// What a thread keeps about its row and its four columns during the walk.
struct FNode {
  int y, z;                  // tile-local
  int j, k;
  int nv;                    // nodes of the four inside the grid (0: the row is outside)
  int ys;                    // slab coordinate of the row (-1 outside)
  int zs;                    // slab coordinate of node k (negative or past the slab where zm is 0)
  unsigned zm;               // nodes of the four inside the z slab
  bool vxy, vz;              // 16-byte accesses to the x and y slabs' / the z slab's auxiliaries
};

// Four old auxiliaries / four new ones.  The x and y slab arrays have rows of
// nz floats, so with nz a multiple of 4 every row of four is aligned and whole;
// the z slab's rows are as long as the slab is thick.
template <bool RO>
__device__ __forceinline__ Q4 aux4(const float* q, bool vec, unsigned m) {
  Q4 r{{0.f, 0.f, 0.f, 0.f}};
  if (vec) {
    const float4 t = RO ? __ldg(reinterpret_cast<const float4*>(q)) : *reinterpret_cast<const float4*>(q);
    r = Q4{{t.x, t.y, t.z, t.w}};
  } else {
#pragma unroll
    for (int e = 0; e < 4; e++)
      if ((m >> e) & 1) r.v[e] = RO ? __ldg(q + e) : q[e];
  }
  return r;
}
__device__ __forceinline__ void put4(float* q, bool vec, unsigned m, const Q4& v) {
  if (vec) { st4(q, v); return; }
#pragma unroll
  for (int e = 0; e < 4; e++)
    if ((m >> e) & 1) q[e] = v.v[e];
}

// scale * (u - l) of four nodes; l shifted by one node: the value below the first, then u's own
__device__ __forceinline__ Q4 diff4(float s, const Q4& u, const Q4& l) {
  Q4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) r.v[e] = __fmul_rn(s, __fsub_rn(u.v[e], l.v[e]));
  return r;
}
__device__ __forceinline__ Q4 below4(float first, const Q4& u) { return Q4{{first, u.v[0], u.v[1], u.v[2]}}; }
__device__ __forceinline__ Q4 above4(const Q4& u, float last) { return Q4{{u.v[1], u.v[2], u.v[3], last}}; }
__device__ __forceinline__ Q4 add4(const Q4& a, const Q4& b) {
  Q4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) r.v[e] = __fadd_rn(a.v[e], b.v[e]);
  return r;
}

}  // namespace dtmx

#include "dtmx_stream.cuh"
