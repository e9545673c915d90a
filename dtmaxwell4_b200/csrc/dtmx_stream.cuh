// dtmx_stream.cuh -- TMA-fed streaming kernels (one launch per half step).
//
// A CTA owns one (z,y) tile column and an x chunk, which the H step walks
// upwards and the E step downwards.  For every plane it needs the three
// source-field tiles (with y/z halo), the own values of the three updated
// components and, for the E step on mixed planes, their material indices.  One
// elected thread fetches all of them with cp.async.bulk.tensor (TMA, no
// multicast) into a ring of NST shared-memory stages, ahead of
// the ones the update reads; completion is tracked per stage by an mbarrier
// with a transaction count.  Out-of-array boxes are zero-filled by the TMA
// unit, which is exactly the zero-outside boundary.  Tiles at a mirror boundary
// (reference geometry) then overwrite the rows and columns beyond it from the
// staged nodes inside: a tap reaches two nodes over at most, and their images
// lie in the same box.
//
// Four z nodes a thread, as in the single sweep (dtmx_fused.cuh): the kernels
// with two rows a thread and scalar accesses were bound by instructions.
// Measured: order 4, 192x160x224 with a 10-cell CPML e 100 -> 81 and h 92 -> 75
// us; the reference geometry with split PML, 180x180x128, e 217 -> 67 and h 172 ->
// 59 us (its mirrored tiles were staged element by element); order 2, 384^3 with a
// 12-cell CPML 850 -> 698 us a step, 128^3 66 -> 42 us.
#pragma once
#include "dtmx_device.cuh"

namespace dtmx {

constexpr int STREAM_NT = 8 * TYT;           // eight threads a row

__device__ __forceinline__ unsigned smem_u32(const void* q) { return (unsigned)__cvta_generic_to_shared(q); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred pp;\n mbarrier.try_wait.parity.shared::cta.b64 pp, [%1], %2;\n selp.u32 %0, 1, 0, pp;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after `limit` polls (2^26 unless a test lowers it),
// records the failure in *err and returns false.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, int* err, long long limit = 1LL << 26) {
  for (long long it = 0; !mbar_test(bar, parity); it++) {
    if (it > limit) {
      if (err) atomicExch(err, 1);
      return false;
    }
  }
  return true;
}
// Polls allowed while draining the copies of a CTA that gave up: TMA copies
// that were issued always complete, so this bound only guards a broken
// transaction count.
constexpr long long DRAIN_POLLS = 1LL << 20;
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}

template <int ORDER, bool ISH, int NST_ = 3>
struct Pipe {
  static constexpr int R = ORDER / 2;
  static constexpr int YL = ISH ? R : R - 1, YH = ISH ? R - 1 : R;      // halo rows of the y taps
  static constexpr int W = TZ + 8;                     // source rows: z in [k0-4, k0+36), 16-byte aligned
  static constexpr int ROWS = TYT + YL + YH;
  static constexpr int N_A = (W * ROWS + 31) / 32 * 32, N_B = W * TYT;
  static constexpr int OFF_A = 0;                      // Ex (H step) / Hx (E step): y and z taps
  static constexpr int OFF_B = N_A;                    // Ey / Hy: z and x taps
  static constexpr int OFF_C = OFF_B + N_B;            // Ez / Hz: y and x taps
  static constexpr int OFF_OWN = OFF_C + N_A;          // own values of the three updated components
  static constexpr int OWN = TYT * TZ;
  static constexpr int OFF_MAT = OFF_OWN + 3 * OWN;
  static constexpr int STAGE = OFF_MAT + (ISH ? 0 : 3 * OWN / 4);       // floats, multiple of 32
  static constexpr unsigned BYTES = (2 * W * ROWS + N_B + 3 * OWN) * 4;
  static constexpr unsigned BYTES_MAT = 3 * OWN;
  // The H step walks a chunk upwards in x, the E step downwards (the E update
  // reads only H, so the order of its planes is free).  Plane i needs its own
  // stage, AHEAD further planes along the walk (x taps not reached yet) and
  // BEHIND planes already passed (kept in the register queue): H taps -R..R-1
  // and E taps -(R-1)..R both give AHEAD = R-1 and BEHIND = R along their walk.
  static constexpr int DIR = ISH ? 1 : -1;             // direction of the walk along x
  static constexpr int AHEAD = ORDER == 4 ? 1 : 0;
  static constexpr int BEHIND = ORDER == 4 ? 2 : 1;
  static constexpr int NST = NST_;
  static constexpr int BASE = ISH ? 2 : 1;             // queue slot of x offset 0 (dstencil taps v0..v3)
  static constexpr size_t SMEM_BYTES = (size_t)NST * STAGE * 4 + MAXMAT * 3 * 4 + NST * 8 + 128;
};

template <int ORDER>
__device__ __forceinline__ Q4 stencil4(const Q4& a, const Q4& b, const Q4& c, const Q4& d) {
  Q4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) r.v[e] = dstencil<ORDER>(a.v[e], b.v[e], c.v[e], d.v[e]);
  return r;
}
__device__ __forceinline__ Q4 scale4(float s, const Q4& a) {
  Q4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) r.v[e] = __fmul_rn(s, a.v[e]);
  return r;
}
// y derivative of four nodes: q points at tap row o0 of the thread's columns
template <int ORDER>
__device__ __forceinline__ Q4 ytaps(const float* q, int w) {
  Q4 r0{}, r3{};
  const Q4 r1 = ld4(q + w), r2 = ld4(q + 2 * w);
  if (ORDER == 4) { r0 = ld4(q); r3 = ld4(q + 3 * w); }
  return stencil4<ORDER>(r0, r1, r2, r3);
}
// z derivative of four nodes from the row around them (q at the first of the four)
template <int ORDER, bool ISH>
__device__ __forceinline__ Q4 ztaps(const float* q) {
  float v[7];
#pragma unroll
  for (int e = 0; e < 7; e++) v[e] = 0.f;
  const Q4 m = ld4(q);
  if (ISH) {                                           // taps -2 .. +1
    if (ORDER == 4) { const float2 l = *reinterpret_cast<const float2*>(q - 2); v[0] = l.x; v[1] = l.y; v[6] = q[4]; }
    else v[1] = q[-1];
#pragma unroll
    for (int e = 0; e < 4; e++) v[2 + e] = m.v[e];
  } else {                                             // taps -1 .. +2
    if (ORDER == 4) { v[0] = q[-1]; const float2 h = *reinterpret_cast<const float2*>(q + 4); v[5] = h.x; v[6] = h.y; }
    else v[5] = q[4];
#pragma unroll
    for (int e = 0; e < 4; e++) v[1 + e] = m.v[e];
  }
  Q4 r;
#pragma unroll
  for (int e = 0; e < 4; e++) r.v[e] = dstencil<ORDER>(v[e], v[e + 1], v[e + 2], v[e + 3]);
  return r;
}

// The staged rows and columns of component c beyond a mirror boundary, from
// their images inside the box (map_idx's rule); own columns of the rows, own rows
// of the columns (the taps run along one axis).
template <int YL, int YH>
__device__ __forceinline__ void mirror_rows(const Grid& g, float* box, int w, int c, int j0) {
  const int lo = g.live_lo[c][1], hi = g.live_hi[c][1], o = comp_off(c, 1);
  const int r0 = j0 - YL, r1 = j0 + TYT - 1 + YH;
  for (int side = 0; side < 2; side++) {
    if (g.btype[1][side] == 0) continue;
    const int a = side ? max(r0, hi + 1) : r0, b = side ? min(r1, hi + 2) : min(r1, lo - 1);
    const float s = (float)(c < 3 ? g.bsE[1][side] : g.bsH[1][side]);
    for (int v = a + (int)(threadIdx.x >> 5); v <= b; v += 4) {
      const int m = g.bplane[1][side] - v - o;
      const int z = threadIdx.x & 31;
      const bool in = m >= lo && m <= hi && m >= r0 && m <= r1;
      box[(v - r0) * w + 4 + z] = in ? s * box[(m - r0) * w + 4 + z] : 0.f;
    }
  }
}
__device__ __forceinline__ void mirror_cols(const Grid& g, float* box, int w, int yoff, int c, int k0) {
  const int lo = g.live_lo[c][2], hi = g.live_hi[c][2], o = comp_off(c, 2);
  const int y = threadIdx.x >> 3, q = threadIdx.x & 7;          // eight threads a row: 0-3 below, 4-7 above
  const int side = q >> 2;
  if (g.btype[2][side] == 0) return;
  const int v = side ? hi + 1 + (q & 3) : lo - 1 - (q & 3);
  if ((q & 3) > 1 || v < k0 - 2 || v > k0 + TZ + 1) return;
  const float s = (float)(c < 3 ? g.bsE[2][side] : g.bsH[2][side]);
  const int m = g.bplane[2][side] - v - o;
  const bool in = m >= lo && m <= hi && m >= k0 - 4 && m < k0 + TZ + 4;
  float* row = box + (y + yoff) * w + 4 - k0;
  row[v] = in ? s * row[m] : 0.f;
}

// Absorber auxiliaries of the thread's nodes in plane i: they do not depend on
// the staged tiles, so they are requested before the stage wait.
template <bool ISH>
__device__ __forceinline__ void stream_aux_load(const Params& p, const FNode& f, int i, int xs, Q4 (&o)[3][2]) {
  if (f.nv == 0) return;
  constexpr int S = ISH ? 2 : 0;
  const unsigned nm = (1u << f.nv) - 1u;
  if (xs >= 0) {
    const int s = slab_at(p, 0, i, f.j, f.k, xs);
#pragma unroll
    for (int q = 0; q < 2; q++) o[0][q] = aux4<false>(p.ab.aux[0][S + q] + s, f.vxy, nm);
  }
  if (f.ys >= 0) {
    const int s = slab_at(p, 1, i, f.j, f.k, f.ys);
#pragma unroll
    for (int q = 0; q < 2; q++) o[1][q] = aux4<false>(p.ab.aux[1][S + q] + s, f.vxy, nm);
  }
  if (f.zm) {
    const int s = slab_at(p, 2, i, f.j, f.k, f.zs);
#pragma unroll
    for (int q = 0; q < 2; q++) o[2][q] = aux4<false>(p.ab.aux[2][S + q] + s, f.vz, f.zm);
  }
}

// One axis' absorber term of four nodes of one component (absorb_apply's
// arithmetic): CPML, c = (b, a, 1/kappa - 1); split, c = (K1, K2, -).
// lm: the live nodes of the component.
__device__ __forceinline__ void absorb4(int kind, const Q4& d, const float (&c0)[4], const float (&c1)[4], const float (&c2)[4], unsigned m,
                                        unsigned lm, bool vec, const Q4& old, float* mem, Q4& corr) {
  Q4 nv;
#pragma unroll
  for (int e = 0; e < 4; e++) {
    nv.v[e] = __fmaf_rn(c0[e], old.v[e], __fmul_rn(c1[e], d.v[e]));
    const float t = kind == 1 ? __fmaf_rn(c2[e], d.v[e], nv.v[e]) : __fsub_rn(__fsub_rn(nv.v[e], old.v[e]), d.v[e]);
    corr.v[e] = __fadd_rn(corr.v[e], (m >> e) & 1 ? t : 0.f);
  }
  put4(mem, vec && lm == 15u, m & lm, nv);
}

template <int ORDER, bool ISH, bool TAB, int NST_>
__device__ __forceinline__ void stream_body(const Params& p, const TmaMaps& m, const Work<TAB>& work, float* dsm) {
  using P = Pipe<ORDER, ISH, NST_>;
  constexpr int NST = P::NST, AHEAD = P::AHEAD, BEHIND = P::BEHIND, BASE = P::BASE, DIR = P::DIR;
  constexpr int c0 = ISH ? 0 : 3, cf = ISH ? 3 : 0;          // source and updated components
  constexpr int O = ISH ? 0 : 1;                             // half-coordinate offset of the updated nodes along their derivative axes
  constexpr int YL = P::YL, W = P::W, o0 = ISH ? -2 : -1;    // o0: first of the four taps
  float* ies = dsm + NST * P::STAGE;                         // 1/eps of the material table (E step)
  uint64_t* bars = reinterpret_cast<uint64_t*>(ies + MAXMAT * 3);
  const int tid = threadIdx.x;
  const int4 job = cta_job<TAB>(p, work);
  const int k0 = job.x * TZ, j0 = job.y * TYT;
  const int xa = job.z, xb = job.w;
  const int len = xb - xa;
  const int i0 = DIR > 0 ? xa : xb - 1;      // first plane of the walk; step t works on plane i0 + DIR t
  // the uniform-material entries of the planes this CTA stages (stage number s),
  // read once so that the elected thread issues each stage without a dependent load
  constexpr int UMC = 128;
  __shared__ signed char umc[UMC];
  __shared__ __align__(16) float zc[3][TZ];  // absorber coefficients of the tile's columns
  // set by the thread that waits for the stages when a wait gave up: the CTA
  // then stops issuing and computing, drains its copies in flight and returns
  __shared__ int gave_up;
  const int slast = len - 1 + AHEAD;         // last stage number that has to be staged
  const int kind = p.ab.kind;
  if (tid == 0) {
    for (int q = 0; q < NST; q++) mbar_init(&bars[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    gave_up = 0;
  }
  if (!ISH) {
    for (int q = tid; q < MAXMAT * 3; q += STREAM_NT) ies[q] = __ldg(&p.mt->inv_eps[0][0] + q);
    for (int sq = tid; sq <= slast && sq < UMC; sq += STREAM_NT) {
      const int ip = i0 + DIR * sq;
      umc[sq] = (ip >= 0 && ip < p.g.n[0]) ? __ldg(p.umat + ((long long)ip * p.nty + job.y) * p.ntz + job.x)
                                          : (signed char)0;
    }
  }
  // third coefficient: 1/kappa - 1 (CPML; the split form has none)
  auto coeff = [&](int a, int v, float (&c)[3]) {
    const int h = 2 * v + O;
    const bool in = v >= 0 && v < p.g.n[a];
    c[0] = in ? __ldg(p.ab.c0[a] + h) : 1.f;
    c[1] = in ? __ldg(p.ab.c1[a] + h) : 0.f;
    c[2] = in && kind == 1 ? __fsub_rn(__ldg(p.ab.c2[a] + h), 1.f) : 0.f;
  };
  if (kind != 0 && tid < TZ) {
    float c[3];
    coeff(2, k0 + tid, c);
    zc[0][tid] = c[0]; zc[1][tid] = c[1]; zc[2][tid] = c[2];
  }
  pdl_wait();
  __syncthreads();
  // uniform material of stage number sq (0 for planes outside the array)
  auto um_of = [&](int sq) -> int {
    if (ISH) return 0;
    if (sq < UMC) return umc[sq];
    const int ip = i0 + DIR * sq;
    return (ip >= 0 && ip < p.g.n[0]) ? (int)__ldg(p.umat + ((long long)ip * p.nty + job.y) * p.ntz + job.x) : 0;
  };
  auto issue = [&](int sq) {
    const int ip = i0 + DIR * sq;
    float* st = dsm + (sq % NST) * P::STAGE;
    uint64_t* bar = &bars[sq % NST];
    // the material tile is needed only when this plane is updated with mixed materials
    const bool want_mat = !ISH && ip >= 0 && ip < p.g.n[0] && um_of(sq) < 0;
    mbar_arrive_expect_tx(bar, P::BYTES + (want_mat ? P::BYTES_MAT : 0u));
    tma_load_3d(st + P::OFF_A, &m.src[c0], k0 - 4, j0 - YL, ip, bar);
    tma_load_3d(st + P::OFF_B, &m.src[c0 + 1], k0 - 4, j0, ip, bar);
    tma_load_3d(st + P::OFF_C, &m.src[c0 + 2], k0 - 4, j0 - YL, ip, bar);
#pragma unroll
    for (int c = 0; c < 3; c++) tma_load_3d(st + P::OFF_OWN + c * P::OWN, &m.own[cf + c], k0, j0, ip, bar);
    if (want_mat)
#pragma unroll
      for (int c = 0; c < 3; c++)
        tma_load_3d(reinterpret_cast<uint8_t*>(st + P::OFF_MAT) + c * P::OWN, &m.mat[c], k0, j0, ip, bar);
  };
  int issued = -1;
  if (tid == 0)
    for (int sq = 0; sq < NST && sq <= slast; sq++) { issue(sq); issued = sq; }
  // per-thread constants of the walk
  FNode f;
  f.y = tid >> 3; f.z = 4 * (tid & 7);
  f.j = j0 + f.y; f.k = k0 + f.z;
  f.nv = f.j < p.g.n[1] ? min(4, max(0, p.g.n[2] - f.k)) : 0;
  f.ys = kind != 0 && f.nv > 0 ? slab_cs(p, 1, f.j) : -1;
  f.zs = 0; f.zm = 0;
  if (kind != 0) {
    const int lo = p.ab.L[2][0], hi = p.g.n[2] - p.ab.L[2][1];
    f.zs = f.k < lo ? f.k : f.k + lo - hi;
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (e < f.nv && (f.k + e < lo || f.k + e >= hi)) f.zm |= 1u << e;
  }
  f.vxy = (p.g.n[2] & 3) == 0;
  f.vz = f.zm == 15u && ((p.ab.L[2][0] + p.ab.L[2][1]) & 3) == 0 && (f.zs & 3) == 0;
  float yc[3] = {1.f, 0.f, 0.f};
  if (f.ys >= 0) coeff(1, f.j, yc);
  // live nodes (reference geometry): the z masks of both half-cell offsets, and whether the row is live for them
  unsigned lz[3] = {15u, 15u, 15u};          // per updated component, over y and z
  if (!p.g.box) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const Grid& g = p.g;
      lz[c] = 0;
      if (f.j >= g.live_lo[cf + c][1] && f.j <= g.live_hi[cf + c][1])
#pragma unroll
        for (int e = 0; e < 4; e++)
          if (f.k + e >= g.live_lo[cf + c][2] && f.k + e <= g.live_hi[cf + c][2]) lz[c] |= 1u << e;
    }
  }
  // does the tile's box reach over a mirror boundary?
  const bool mirror = !p.g.box && (j0 - 2 < p.g.all_lo[1] || j0 + TYT + 1 > p.g.all_hi[1] || k0 - 2 < p.g.all_lo[2] || k0 + TZ + 1 > p.g.all_hi[2]);
  const bool own_yz = kind != 0 && (j0 < p.ab.L[1][0] || j0 + TYT > p.g.n[1] - p.ab.L[1][1] || k0 < p.ab.L[2][0] ||
                                    k0 + TZ > p.g.n[2] - p.ab.L[2][1]);
  // x queue: the BEHIND planes before the first one of the walk, from global memory
  Q4 qb[4], qc[4], oa[3][2];
#pragma unroll
  for (int q = 0; q < 4; q++) { qb[q] = Q4{{0.f, 0.f, 0.f, 0.f}}; qc[q] = qb[q]; }
#pragma unroll
  for (int b = 1; b <= BEHIND; b++) {
    const int ip = i0 - DIR * b;
    if (ip >= 0 && ip < p.g.n[0] && f.nv > 0) {
      const long long off = (long long)ip * p.g.sx + (long long)f.j * p.g.sy + f.k;
      qb[BASE - DIR * b] = aux4<true>(p.f[c0 + 1] + off, true, 15u);
      qc[BASE - DIR * b] = aux4<true>(p.f[c0 + 2] + off, true, 15u);
    }
  }
  const float cx = p.cdt[0], cy = p.cdt[1], cz = p.cdt[2];
  for (int t = 0; t < len; t++) {
    const int i = i0 + DIR * t;
    // values that do not depend on the staged tiles are loaded before the stage wait
    const int um = um_of(t);
    const int xs = kind != 0 ? slab_cs(p, 0, i) : -1;
    const bool tab = own_yz || xs >= 0;
    float xc[3] = {1.f, 0.f, 0.f};
    if (tab) {
      stream_aux_load<ISH>(p, f, i, xs, oa);
      if (xs >= 0) coeff(0, i, xc);
    }
    // stages t..t+AHEAD-1 were waited for in earlier steps (all of them at the
    // start); one thread polls the stage barriers and the CTA barrier then releases
    // everybody (and orders the staged data for them) without spinning issue slots
    if (tid == 0)
      for (int a = (t == 0 ? 0 : AHEAD); a <= AHEAD; a++)
        if (!mbar_wait(&bars[(t + a) % NST], (unsigned)(((t + a) / NST) & 1), p.err, p.wait_limit)) gave_up = 1;
    __syncthreads();
    if (gave_up) {
      // stages t .. the last one issued may still be landing: wait for them (bounded) before leaving
      if (tid == 0)
        for (int sq = t; sq <= issued; sq++)
          mbar_wait(&bars[sq % NST], (unsigned)((sq / NST) & 1), nullptr, DRAIN_POLLS);
      return;
    }
    // every thread is past step t - 1: the slot of its stage is free
    if (tid == 0 && t >= 1 && t - 1 + NST <= slast) {
      if (mirror) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      issue(t - 1 + NST);
      issued = t - 1 + NST;
    }
    float* cur = dsm + (t % NST) * P::STAGE;
    if (mirror) {
      mirror_rows<YL, P::YH>(p.g, cur + P::OFF_A, W, c0, j0);
      mirror_rows<YL, P::YH>(p.g, cur + P::OFF_C, W, c0 + 2, j0);
      mirror_cols(p.g, cur + P::OFF_A, W, YL, c0, k0);
      mirror_cols(p.g, cur + P::OFF_B, W, 0, c0 + 1, k0);
      __syncthreads();
    }
#pragma unroll
    for (int a = 0; a <= AHEAD; a++) {
      const float* st = dsm + ((t + a) % NST) * P::STAGE;
      qb[BASE + DIR * a] = ld4(st + P::OFF_B + f.y * W + f.z + 4);
      qc[BASE + DIR * a] = ld4(st + P::OFF_C + (f.y + YL) * W + f.z + 4);
    }
    const float* sA = cur + P::OFF_A + (f.y + YL) * W + f.z + 4;
    const float* sB = cur + P::OFF_B + f.y * W + f.z + 4;
    const float* sC = cur + P::OFF_C + (f.y + YL) * W + f.z + 4;
    // H: Hx -= dt(dy Ez - dz Ey); Hy -= dt(dz Ex - dx Ez); Hz -= dt(dx Ey - dy Ex); E: the opposite signs, times 1/eps
    Q4 d01 = scale4(ISH ? -cy : cy, ytaps<ORDER>(sC + o0 * W, W));
    Q4 d02 = scale4(ISH ? cz : -cz, ztaps<ORDER, ISH>(sB));
    Q4 d10 = scale4(ISH ? cx : -cx, stencil4<ORDER>(qc[0], qc[1], qc[2], qc[3]));
    Q4 d12 = scale4(ISH ? -cz : cz, ztaps<ORDER, ISH>(sA));
    Q4 d20 = scale4(ISH ? -cx : cx, stencil4<ORDER>(qb[0], qb[1], qb[2], qb[3]));
    Q4 d21 = scale4(ISH ? cy : -cy, ytaps<ORDER>(sA + o0 * W, W));
    if (!ISH) {
      if (um >= 0) {
        const float e0 = ies[um * 3], e1 = ies[um * 3 + 1], e2 = ies[um * 3 + 2];
        if (e0 != 1.f || e1 != 1.f || e2 != 1.f) {
          d01 = scale4(e0, d01); d02 = scale4(e0, d02);
          d10 = scale4(e1, d10); d12 = scale4(e1, d12);
          d20 = scale4(e2, d20); d21 = scale4(e2, d21);
        }
      } else {
        // mixed materials or the design region; a dispersive node's table entry is -0, so it
        // keeps its old E here and the ADE pass writes it
        const unsigned* mt = reinterpret_cast<const unsigned*>(cur + P::OFF_MAT);
        unsigned mm[3];
#pragma unroll
        for (int c = 0; c < 3; c++) mm[c] = mt[(c * P::OWN + f.y * TZ + f.z) / 4];
#pragma unroll
        for (int e = 0; e < 4; e++) {
          float ie[3];
#pragma unroll
          for (int c = 0; c < 3; c++) ie[c] = ies[((mm[c] >> (8 * e)) & 255u) * 3 + c];
          if (p.des_on) {
            const long long di = design_index(p, i, f.j, f.k + e);
            if (di >= 0) {
#pragma unroll
              for (int c = 0; c < 3; c++)
                if (!is_dispersive(ie[c])) ie[c] = p.des_ie[c][di];
            }
          }
          d01.v[e] = __fmul_rn(d01.v[e], ie[0]); d02.v[e] = __fmul_rn(d02.v[e], ie[0]);
          d10.v[e] = __fmul_rn(d10.v[e], ie[1]); d12.v[e] = __fmul_rn(d12.v[e], ie[1]);
          d20.v[e] = __fmul_rn(d20.v[e], ie[2]); d21.v[e] = __fmul_rn(d21.v[e], ie[2]);
        }
      }
    }
    Q4 inc[3] = {add4(d01, d02), add4(d10, d12), add4(d20, d21)};
    unsigned lm[3] = {15u, 15u, 15u};
    if (!p.g.box) {
#pragma unroll
      for (int c = 0; c < 3; c++) lm[c] = i >= p.g.live_lo[cf + c][0] && i <= p.g.live_hi[cf + c][0] ? lz[c] : 0u;
    }
    if (tab && f.nv > 0 && (xs >= 0 || f.ys >= 0 || f.zm)) {
      constexpr int S = ISH ? 2 : 0;
      const unsigned nm = (1u << f.nv) - 1u;
      Q4 corr[3];
#pragma unroll
      for (int c = 0; c < 3; c++) corr[c] = Q4{{0.f, 0.f, 0.f, 0.f}};
      auto same = [](float v, float (&r)[4]) { r[0] = r[1] = r[2] = r[3] = v; };
      float b[4], a[4], c[4];
      if (xs >= 0) {
        same(xc[0], b); same(xc[1], a); same(xc[2], c);
        const int s = slab_at(p, 0, i, f.j, f.k, xs);
        absorb4(kind, d10, b, a, c, nm, lm[1], f.vxy, oa[0][0], p.ab.aux[0][S] + s, corr[1]);
        absorb4(kind, d20, b, a, c, nm, lm[2], f.vxy, oa[0][1], p.ab.aux[0][S + 1] + s, corr[2]);
      }
      if (f.ys >= 0) {
        same(yc[0], b); same(yc[1], a); same(yc[2], c);
        const int s = slab_at(p, 1, i, f.j, f.k, f.ys);
        absorb4(kind, d01, b, a, c, nm, lm[0], f.vxy, oa[1][0], p.ab.aux[1][S] + s, corr[0]);
        absorb4(kind, d21, b, a, c, nm, lm[2], f.vxy, oa[1][1], p.ab.aux[1][S + 1] + s, corr[2]);
      }
      if (f.zm) {
        const Q4 tb = ld4(&zc[0][f.z]), ta = ld4(&zc[1][f.z]), tc = ld4(&zc[2][f.z]);
        const int s = slab_at(p, 2, i, f.j, f.k, f.zs);
        absorb4(kind, d02, tb.v, ta.v, tc.v, f.zm, lm[0], f.vz, oa[2][0], p.ab.aux[2][S] + s, corr[0]);
        absorb4(kind, d12, tb.v, ta.v, tc.v, f.zm, lm[1], f.vz, oa[2][1], p.ab.aux[2][S + 1] + s, corr[1]);
      }
#pragma unroll
      for (int q = 0; q < 3; q++) inc[q] = add4(inc[q], corr[q]);
    }
    if (f.nv > 0) {
      const long long off = (long long)i * p.g.sx + (long long)f.j * p.g.sy + f.k;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const Q4 own = ld4(cur + P::OFF_OWN + c * P::OWN + f.y * TZ + f.z);
        Q4 r = add4(own, inc[c]);
        // nodes beyond the grid (row padding) and nodes that are not live keep what they hold
        const unsigned keep = lm[c] & ((1u << f.nv) - 1u);
        if (keep != 15u) {
#pragma unroll
          for (int e = 0; e < 4; e++)
            if (!((keep >> e) & 1)) r.v[e] = own.v[e];
        }
        st4(p.f[cf + c] + off, r);
      }
    }
    // the queue moves one plane along the walk
    if (DIR > 0) {
#pragma unroll
      for (int q = 0; q < 3; q++) { qb[q] = qb[q + 1]; qc[q] = qc[q + 1]; }
    } else {
#pragma unroll
      for (int q = 3; q > 0; q--) { qb[q] = qb[q - 1]; qc[q] = qc[q - 1]; }
    }
  }
}

// CTAs per SM: 4 at order 2, what shared memory allows for 3 stages; 3 at order 4, whose
// registers (146) allow no more, with 3 or 4 stages.  Order 4 holds two of its
// stages resident, so a ring of 3 has one plane in flight: large launches are
// then bound by the copies' latency (640x640x384 without absorber 2318 us a step,
// with 4 stages 1886; 256^3 265 and 223; with a 10-cell CPML 384^3 966 and 859).
// The fourth stage costs a little where a short walk starts from cached fields
// (128^3 39.4 and 41.5 us; stream_stages).
template <int ORDER, bool TAB, int NST>
__global__ void __launch_bounds__(STREAM_NT, ORDER == 2 ? 4 : 3)
    h_kernel(const __grid_constant__ Params p, const __grid_constant__ TmaMaps m, const __grid_constant__ Work<TAB> work) {
  extern __shared__ __align__(128) float dsm[];
  stream_body<ORDER, true, TAB, NST>(p, m, work, dsm);
}

template <int ORDER, bool TAB, int NST>
__global__ void __launch_bounds__(STREAM_NT, ORDER == 2 ? 4 : 3)
    e_kernel(const __grid_constant__ Params p, const __grid_constant__ TmaMaps m, const __grid_constant__ Work<TAB> work) {
  extern __shared__ __align__(128) float dsm[];
  stream_body<ORDER, false, TAB, NST>(p, m, work, dsm);
}

}  // namespace dtmx
