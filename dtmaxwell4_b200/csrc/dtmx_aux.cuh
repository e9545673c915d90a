// dtmx_aux.cuh -- per-step side kernels: TF/SF surface corrections, the 1-D
// incident line of the plane-wave source, soft point sources, probes, running
// DFT and the device step counter.
#pragma once
#include "dtmx_device.cuh"

namespace dtmx {

// One TF/SF correction job: component c over an index box that holds every
// node of c whose taps along one curl axis cross one face of the box.
struct TfsfJob {
  int c;
  int a, g, sg;              // the job's curl term: axis, source component, sign in the curl
  int lo[3], hi[3];
  long long cells;
};
constexpr int MAX_TFSF_JOBS = 12;    // 3 components x 2 curl terms x 2 faces

struct TfsfDev {
  int active_cfg;            // a TF/SF source is configured
  int kind;                  // 0 dipole, 1 plane +x
  int lo[3], hi[3];          // inside-box half-coordinate ranges (inclusive)
  double ctr[3];             // dipole position (box centre, physical, whole-grid coordinates)
  int xo;                    // whole-grid cell index of plane 0 (x slabs; 0 for a whole grid)
  double hd[3];              // half cell sizes dx/2, dy/2, dz/2
  double dt, c, w, kenv, tstop;
  int ntime;
  const double* line_e; const double* line_h; int line_M, line_n;
  int njob[2];               // [0] E half step, [1] H half step
  TfsfJob job[2][MAX_TFSF_JOBS];
};

__device__ __forceinline__ bool tfsf_on(const TfsfDev& t, long long n) {
  if (t.tstop <= 0) return true;
  const long long is = n / t.ntime;
  return (double)(is + 1) * t.ntime * t.dt < t.tstop;
}

__device__ __forceinline__ bool in_box(const TfsfDev& t, int X, int Y, int Z) {
  return X >= t.lo[0] && X <= t.hi[0] && Y >= t.lo[1] && Y <= t.hi[1] && Z >= t.lo[2] && Z <= t.hi[2];
}

// Field of a z-oriented Hertzian dipole with a Hann-windowed sine moment,
// reference DipoleTFSF (signal.hpp:51-97), evaluated in double precision.
__device__ double dipole_field(const TfsfDev& t, int comp, int X, int Y, int Z, double tt) {
  const double nx = (X + 2 * t.xo) * t.hd[0] - t.ctr[0], ny = Y * t.hd[1] - t.ctr[1], nz = Z * t.hd[2] - t.ctr[2];
  const double R = sqrt(nx * nx + ny * ny + nz * nz);
  const double time = tt * t.dt, c = t.c, w = t.w, ke = t.kenv;
  const double ph = w * time - w / c * R;
  double s, co, sk, ck;
  sincos(ph, &s, &co);
  sincos(ph * ke, &sk, &ck);
  double d = s * 0.5 * (1.0 - ck);
  double ds = w * co * 0.5 - 0.5 * w * co * ck + 0.5 * s * w * ke * sk;
  double dss = -w * w * s * 0.5 + 0.5 * w * w * s * ck + w * co * w * ke * sk + 0.5 * s * w * ke * w * ke * ck;
  if (ph * ke < 0.0 || ph * ke > 2.0 * M_PI) { d = 0; ds = 0; dss = 0; }
  const double u0 = nx / R, u1 = ny / R, u2 = nz / R;
  if (comp < 3) {
    // (dss z^ x n) x n  +  3 (ds.n) n - ds  +  3 (d.n) n - d   with moments along z
    const double a0 = -dss * u1, a1 = dss * u0;
    const double cr[3] = {a1 * u2, -a0 * u2, a0 * u1 - a1 * u0};
    const double uu[3] = {u0, u1, u2};
    const double dz = comp == 2 ? 1.0 : 0.0;
    return c * (cr[comp] / (c * c * R) + (3.0 * ds * u2 * uu[comp] - ds * dz) / (c * R * R) +
                (3.0 * d * u2 * uu[comp] - d * dz) / (R * R * R));
  }
  const int q = comp - 3;
  const double b1 = q == 0 ? -dss * u1 : q == 1 ? dss * u0 : 0.0;
  const double b2 = q == 0 ? -ds * u1 : q == 1 ? ds * u0 : 0.0;
  return b1 / (c * c * R) + b2 / (c * R * R);
}

// curl terms of component c: {axis, source component} for (+) and (-) terms
__host__ __device__ __forceinline__ void curl_terms(int c, int& a0, int& g0, int& a1, int& g1) {
  switch (c) {
    case 0: a0 = 1; g0 = 5; a1 = 2; g1 = 4; break;
    case 1: a0 = 2; g0 = 3; a1 = 0; g1 = 5; break;
    case 2: a0 = 0; g0 = 4; a1 = 1; g1 = 3; break;
    case 3: a0 = 1; g0 = 2; a1 = 2; g1 = 1; break;
    case 4: a0 = 2; g0 = 0; a1 = 0; g1 = 2; break;
    default: a0 = 0; g0 = 1; a1 = 1; g1 = 0; break;
  }
}

// TF/SF correction of one half step (genAlg.py:209-234): a tap that crosses
// the box surface gets +inc when the updated node is outside and the tap
// inside, -inc in the opposite case.  The update is linear in the taps, so
// the correction is added after the bulk update as dt/d * D(corrections),
// summed over both curl terms of the node in double precision.
// This is the part of one tap: q of curl term `term` (0 where the tap does not
// cross or the term cannot).
template <int ORDER>
__device__ __forceinline__ double tfsf_tap(const Params& p, const TfsfDev& t, int c, int i, int j, int k, bool isH, double tt, int term, int q) {
  if (ORDER == 2 && (q == 0 || q == 3)) return 0.0;
  int ax[2], gs[2];
  curl_terms(c, ax[0], gs[0], ax[1], gs[1]);
  const int a = term ? ax[1] : ax[0], g = term ? gs[1] : gs[0];
  const int t0 = (isH ? -2 : -1) + q;
  const int S[3] = {2 * i + comp_off(c, 0), 2 * j + comp_off(c, 1), 2 * k + comp_off(c, 2)};
  const int G[3] = {2 * (i + (a == 0 ? t0 : 0)) + comp_off(g, 0), 2 * (j + (a == 1 ? t0 : 0)) + comp_off(g, 1),
                    2 * (k + (a == 2 ? t0 : 0)) + comp_off(g, 2)};
  const bool sin_ = in_box(t, S[0], S[1], S[2]);
  if (in_box(t, G[0], G[1], G[2]) == sin_) return 0.0;
  // (a tap differs from its node along a alone, so it is the face along a that it crosses)
  const double w = ORDER == 2 ? (q == 2 ? 1.0 : -1.0) : q == 0 ? 1.0 / 24.0 : q == 1 ? -27.0 / 24.0 : q == 2 ? 27.0 / 24.0 : -1.0 / 24.0;
  double sg = term == 0 ? 1.0 : -1.0;
  if (isH) sg = -sg;
  const double inc = dipole_field(t, g, G[0], G[1], G[2], tt);
  return sg * (double)p.cdt[a] * w * (sin_ ? -inc : inc);
}

__device__ __forceinline__ bool in_job(const TfsfJob& jb, int i, int j, int k) {
  return i >= jb.lo[0] && i <= jb.hi[0] && j >= jb.lo[1] && j <= jb.hi[1] && k >= jb.lo[2] && k <= jb.hi[2];
}

// TPN threads per node of a job (blockIdx.y), by the number of nodes (kTapNodes2,
// kTapNodes4).  Eight, one for each tap of both curl terms: the incident field of
// a tap is a chain of FP64 sines, and on boxes too small to fill the chip its
// latency is all there is (one thread that walks a node's taps takes 5 to 10 us a
// half step for any small box, eight 3 to 5).  One: a node has one or two crossing
// taps, so of eight threads most wait for the others, and where there are
// enough nodes the work of the warps counts: order 4 on 200^3 with a box of 160
// took 366 us a step for the corrections with eight throughout, 122 now.  The sum
// over the taps is the same tree in both, bit for bit.
// A node that also lies in an earlier job of the same component is left to that
// job, so every node is corrected exactly once with the sum of all its
// crossing taps.
template <int ORDER, int TPN>
__global__ void __launch_bounds__(256) tfsf_kernel(const __grid_constant__ Params p, const __grid_constant__ TfsfDev t, const long long* d_step,
                                                   int isH) {
  static_assert(TPN == 1 || TPN == 8, "a node a thread or a tap a thread");
  pdl_wait();
  pdl_trigger();
  const long long n = *d_step;
  if (!tfsf_on(t, n)) return;
  const int hs = isH ? 1 : 0;
  const int r = blockIdx.y;
  if (r >= t.njob[hs]) return;
  const TfsfJob& jb = t.job[hs][r];
  // a job is a thin shell (cells < 2^31, checked when the jobs are built): 32-bit indexing
  const long long th = (long long)blockIdx.x * 256 + threadIdx.x;
  // (the grid is as wide as the largest job: warps past the end of this one have no node, and in its
  // last warp the threads past it help the last node and store nothing)
  if ((th & ~31LL) / TPN >= jb.cells) return;
  const int cell = (int)min(th / TPN, jb.cells - 1);
  const int ey = jb.hi[1] - jb.lo[1] + 1, ez = jb.hi[2] - jb.lo[2] + 1;
  const int i = jb.lo[0] + cell / (ey * ez);
  const int rest = cell - (i - jb.lo[0]) * (ey * ez);
  const int j = jb.lo[1] + rest / ez;
  const int k = jb.lo[2] + (rest - (j - jb.lo[1]) * ez);
  const int c = jb.c;
  const double tt = isH ? (double)n : (double)n + 0.5;
  double total;
  if (TPN == 8) {
    total = tfsf_tap<ORDER>(p, t, c, i, j, k, isH, tt, (threadIdx.x >> 2) & 1, threadIdx.x & 3);
#pragma unroll
    for (int s = 1; s < 8; s <<= 1) total += __shfl_xor_sync(0xffffffffu, total, s);
  } else {
    total = 0.0;
#pragma unroll 1
    for (int term = 0; term < 2; term++) {
      int ax[2], gs[2];
      curl_terms(c, ax[0], gs[0], ax[1], gs[1]);
      const int a = term ? ax[1] : ax[0], g = term ? gs[1] : gs[0], b1 = (a + 1) % 3, b2 = (a + 2) % 3;
      auto at = [&](int b) { return b == 0 ? i : b == 1 ? j : k; };
      // a tap crosses only where the node lies inside the box' range on the other two axes and near a face along a
      const int B1 = 2 * at(b1) + comp_off(g, b1), B2 = 2 * at(b2) + comp_off(g, b2), S = 2 * at(a) + comp_off(c, a);
      if (B1 < t.lo[b1] || B1 > t.hi[b1] || B2 < t.lo[b2] || B2 > t.hi[b2]) continue;
      if ((S < t.lo[a] - 4 || S > t.lo[a] + 3) && (S < t.hi[a] - 3 || S > t.hi[a] + 4)) continue;
      double low = 0.0, high = 0.0;                              // taps 0 + 1 and 2 + 3
#pragma unroll 1
      for (int q = ORDER == 2 ? 1 : 0; q < (ORDER == 2 ? 3 : 4); q++) {
        const double v = tfsf_tap<ORDER>(p, t, c, i, j, k, isH, tt, term, q);
        if (q < 2) low += v; else high += v;
      }
      total += low + high;
    }
  }
  if (th % TPN != 0 || th / TPN >= jb.cells || total == 0.0 || !is_live(p.g, c, i, j, k)) return;
  for (int q = 0; q < r; q++)
    if (t.job[hs][q].c == c && in_job(t.job[hs][q], i, j, k)) return;
  const long long id = (long long)i * p.g.sx + (long long)j * p.g.sy + k;
  if (!isH) {
    const int mi = p.mat[c] ? (int)p.mat[c][id] : 0;
    const long long di = design_index(p, i, j, k);
    total *= (double)(di >= 0 ? p.des_ie[c][di] : p.mt->inv_eps[mi][c]);
  }
  p.f[c][id] += (float)total;
}

// ---- plane wave: corrections of one half step and the 1-D incident line (Ez
// at odd X, Hy at even X, same stencil and time step) in one launch.  The
// corrections read the line's other field, so neither waits for the other: the
// H half step reads e and advances h, the E half step reads h and advances e.
struct LineDev {
  double* e; double* h;
  int n, src;
  double r, dt, amp, f0, tau, t0;
};

template <int ORDER>
__device__ __forceinline__ void line_update(const LineDev& l, bool isH, long long n, int m0, int stride) {
  const double ts = ((double)n + 0.5) * l.dt - l.t0;
  for (int m = m0; m < l.n; m += stride) {
    if (isH) {
      const double e0 = l.e[m], em1 = m >= 1 ? l.e[m - 1] : 0.0;
      double d = e0 - em1;
      if (ORDER == 4) {
        const double ep1 = m + 1 < l.n ? l.e[m + 1] : 0.0, em2 = m >= 2 ? l.e[m - 2] : 0.0;
        d = (27.0 * (e0 - em1) - (ep1 - em2)) / 24.0;
      }
      l.h[m] += l.r * d;
    } else {
      const double h0 = l.h[m], hp1 = m + 1 < l.n ? l.h[m + 1] : 0.0;
      double d = hp1 - h0;
      if (ORDER == 4) {
        const double hp2 = m + 2 < l.n ? l.h[m + 2] : 0.0, hm1 = m >= 1 ? l.h[m - 1] : 0.0;
        d = (27.0 * (hp1 - h0) - (hp2 - hm1)) / 24.0;
      }
      double v = l.e[m] + l.r * d;
      if (m == l.src) v += l.amp * sin(2.0 * M_PI * l.f0 * ts) * exp(-(ts / l.tau) * (ts / l.tau));
      l.e[m] = v;
    }
  }
}

// A plane wave has only Ez and Hy, so a component has one curl term with an
// incident tap, and on one node it depends on the node's index along the
// term's axis and on x alone.  A warp takes 128 nodes of a row of a job: along
// z, or along y where the job is the face normal to z and a row along z would
// hold one node.  Measured on a 384^3 grid: 18 us a half step with one thread a
// node and the general tap search, 12.5 with this, the line's update included (5
// and 2 us as launches of their own); what is left is a chain of dependent loads.
template <int ORDER>
__global__ void __launch_bounds__(256) tfsf_plane_kernel(const __grid_constant__ Params p, const __grid_constant__ TfsfDev t, const LineDev l,
                                                         const long long* d_step, int isH) {
  pdl_wait();
  pdl_trigger();
  const long long n = *d_step;
  const int hs = isH ? 1 : 0, r = blockIdx.y;
  if (r == t.njob[hs]) {                           // the line's own update
    line_update<ORDER>(l, isH, n, blockIdx.x * 256 + threadIdx.x, gridDim.x * 256);
    return;
  }
  if (!tfsf_on(t, n)) return;
  const TfsfJob& jb = t.job[hs][r];
  const int c = jb.c, a = jb.a, g = jb.g, lane = threadIdx.x & 31;
  const int la = a == 2 ? 1 : 2, ra = a == 2 ? 2 : 1;              // axis of a row, and the other one beside x
  const int nl = jb.hi[la] - jb.lo[la] + 1, nr = jb.hi[ra] - jb.lo[ra] + 1, ni = jb.hi[0] - jb.lo[0] + 1;
  const int parts = (nl + 127) / 128;
  const int unit = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit >= ni * nr * parts) return;
  const int part = unit % parts, row = unit / parts;
  int idx[3];
  idx[0] = jb.lo[0] + row / nr;
  idx[ra] = jb.lo[ra] + row % nr;
  const int first = jb.lo[la] + part * 128 + lane;
  // the correction of the row's nodes, but for 1/eps (a is not the row's axis)
  const int t0 = isH ? -2 : -1, o = comp_off(c, a), og = comp_off(g, a);
  const int S = 2 * idx[a] + o;
  const bool sin_ = S >= t.lo[a] && S <= t.hi[a];
  double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (ORDER == 2 && (q == 0 || q == 3)) continue;
    const int G = 2 * (idx[a] + t0 + q) + og;
    if ((G >= t.lo[a] && G <= t.hi[a]) == sin_) continue;
    const int X = a == 0 ? G : 2 * idx[0] + comp_off(g, 0);
    const int m = (g == 2 ? (X - 1) >> 1 : X >> 1) + t.line_M;
    const double inc = m >= 0 && m < t.line_n ? (g == 2 ? t.line_e[m] : t.line_h[m]) : 0.0;
    v[q] = sin_ ? -inc : inc;
  }
  const double dv = ORDER == 2 ? v[2] - v[1] : (27.0 * (v[2] - v[1]) - (v[3] - v[0])) / 24.0;
  const double total = (isH ? -jb.sg : jb.sg) * (double)p.cdt[a] * dv;
  long long id[4];
  float f[4];
  bool on[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    idx[la] = first + 32 * e;
    on[e] = idx[la] <= jb.hi[la] && is_live(p.g, c, idx[0], idx[1], idx[2]);
    // a node of an earlier job of the component is that job's
    for (int q = 0; q < r && on[e]; q++)
      if (t.job[hs][q].c == c && in_job(t.job[hs][q], idx[0], idx[1], idx[2])) on[e] = false;
    id[e] = (long long)idx[0] * p.g.sx + (long long)idx[1] * p.g.sy + idx[2];
    f[e] = on[e] ? p.f[c][id[e]] : 0.f;
  }
#pragma unroll
  for (int e = 0; e < 4; e++) {
    if (!on[e]) continue;
    double w = total;
    if (!isH) {
      idx[la] = first + 32 * e;
      const int mi = p.mat[c] ? (int)__ldg(p.mat[c] + id[e]) : 0;
      const long long di = design_index(p, idx[0], idx[1], idx[2]);
      w *= (double)(di >= 0 ? p.des_ie[c][di] : __ldg(&p.mt->inv_eps[mi][c]));
    }
    p.f[c][id[e]] = f[e] + (float)w;
  }
}

struct PointSrcDev {
  int comp; long long id; double amp, f0, tau, t0;
};
__device__ __forceinline__ float source_value(const PointSrcDev& s, long long n, double dt) {
  const double u = ((double)n + 0.5) * dt - s.t0;
  return (float)(s.amp * sin(2.0 * M_PI * s.f0 * u) * exp(-(u / s.tau) * (u / s.tau)));
}

// More soft sources than the tail kernel's list holds.  The list is sorted by node
// when it is made, sources on one node in the order they were given; a
// thread adds those of one node: run[q] = {first, count}.  (Without the sorted
// list every thread searched all sources for its node's: 16384 sources took
// 4 ms a step: 64x272x272 cells 4064 us, now 56, without sources 53.)
__global__ void point_source_kernel(const __grid_constant__ Params p, const PointSrcDev* s, const int2* run, int nrun, const long long* d_step,
                                    double dt) {
  pdl_wait();
  pdl_trigger();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nrun) return;
  const int2 r = run[q];
  float* f = p.f[s[r.x].comp] + s[r.x].id;
  const long long n = *d_step;
  float v = *f;
  for (int e = r.x; e < r.x + r.y; e++) v += source_value(s[e], n, dt);
  *f = v;
}

struct ProbeDev { int comp, i, j, k, mode; };

struct DftDev {
  int axis, index, comp_mask, nfreq, n1, n2;
  int lo1, lo2;             // window origin along the two in-plane axes (slow, fast)
  const double* omega;
  double2* acc;             // [ncomp][nfreq][n1*n2]
  float* stage;             // [DFT_STAGE][ncomp][n1*n2] plane samples not yet accumulated
  long long* sstep;         // [DFT_STAGE] step number s of each staged sample
};
constexpr int DFT_STAGE = 16;

// ---- the end of a time step in one launch: soft sources, probes, DFT samples,
// the design region's history and the step counter.  Each of them is small
// (1 to 4 us as a launch of its own, 4.6 us a step together for a dipole run
// with probes, 52 us for a flux box' 18 windows), so they share one: a block
// map assigns the blocks to the DFT planes.
// A source changes a node that a sample may read in the same launch.  So the
// blocks read the fields as they are and add the sources of the node they
// read; the block that finishes last (a ticket) adds them to the fields, after
// every read, and advances the step counter.
constexpr int TAIL_SRC = 32;
struct TailArgs {
  const PointSrcDev* src; int ns; double dt;
  const ProbeDev* pr; int np; float* traces; int cap; int every;
  const DftDev* dft; const int2* map; int nmap; int slot;      // map[block] = {plane, its block of 256 points}
  float* hist; int nd;                                         // design-region E of this step (nullptr: none)
  unsigned* ticket;
  int advance;
};
struct TailSources { float v[TAIL_SRC]; long long id[TAIL_SRC]; int comp[TAIL_SRC]; };

__device__ __forceinline__ float tail_get(const Params& p, const TailSources& s, int ns, int c, int i, int j, int k) {
  if (i < 0 || i >= p.g.n[0] || j < 0 || j >= p.g.n[1] || k < 0 || k >= p.g.n[2]) return 0.f;
  const long long id = (long long)i * p.g.sx + (long long)j * p.g.sy + k;
  float v = p.f[c][id];
  for (int q = 0; q < ns; q++)
    if (s.comp[q] == c && s.id[q] == id) v += s.v[q];
  return v;
}

// Reference Sensor::write averaging (sensor.h:51-83); for Hz the reference's
// second point is never assigned and reads a zero node outside the domain.
__device__ __forceinline__ float tail_probe(const Params& p, const TailSources& s, int ns, const ProbeDev& d) {
  const int c = d.comp, x = d.i, y = d.j, z = d.k;
  if (d.mode == 0) return tail_get(p, s, ns, c, x, y, z);
  const int zM = z == 0 ? z + 1 : z - 1;
  auto get = [&](int i, int j, int k) { return tail_get(p, s, ns, c, i, j, k); };
  switch (c) {
    case 0: return 0.25f * (get(x, y - 1, zM) + get(x, y - 1, z) + get(x, y, zM) + get(x, y, z));
    case 1: return 0.25f * (get(x - 1, y, zM) + get(x - 1, y, z) + get(x, y, zM) + get(x, y, z));
    case 2: return 0.25f * (get(x - 1, y - 1, z) + get(x - 1, y, z) + get(x, y - 1, z) + get(x, y, z));
    case 3: return 0.5f * (get(x - 1, y, z) + get(x, y, z));
    case 4: return 0.5f * (get(x, y - 1, z) + get(x, y, z));
    default: return 0.5f * get(x, y, zM);
  }
}

__global__ void __launch_bounds__(256) tail_kernel(const __grid_constant__ Params p, const __grid_constant__ TailArgs a, long long* d_step) {
  __shared__ TailSources s;
  __shared__ bool last;
  const int tid = threadIdx.x, b = blockIdx.x;
  pdl_wait();
  pdl_trigger();
  const long long n = *d_step;
  if (tid < a.ns) {
    const PointSrcDev& q = a.src[tid];
    s.v[tid] = source_value(q, n, a.dt);
    s.id[tid] = q.id;
    s.comp[tid] = q.comp;
  }
  __syncthreads();
  // a probe a thread (20000 probes in one block took 99 us a step more than 8, spread out they take 3)
  const int pq = b * 256 + tid;
  if (pq < a.np && (n + 1) % a.every == 0) {
    const long long sample = (n + 1) / a.every - 1;
    if (sample < a.cap) a.traces[(long long)pq * a.cap + sample] = tail_probe(p, s, a.ns, a.pr[pq]);
  }
  if (b < a.nmap) {
    const int2 e = a.map[b];
    const DftDev& d = a.dft[e.x];
    const int npts = d.n1 * d.n2, n2 = d.n2, mask = d.comp_mask, ncomp = __popc(mask);
    const int pt = e.y * 256 + tid;
    if (pt == 0) d.sstep[a.slot] = n + 1;
    if (pt < npts) {
      const int u = d.lo1 + pt / n2, v = d.lo2 + pt % n2, axis = d.axis;
      const int i = axis == 0 ? d.index : u, j = axis == 0 ? u : axis == 1 ? d.index : v, k = axis == 2 ? d.index : v;
      float* out = d.stage + (long long)a.slot * ncomp * npts + pt;
      int ci = 0;
#pragma unroll
      for (int c = 0; c < 6; c++)
        if (mask & (1 << c)) out[(long long)(ci++) * npts] = tail_get(p, s, a.ns, c, i, j, k);
    }
  } else if (a.hist && b - a.nmap < (3 * a.nd + 255) / 256) {
    const int q = (b - a.nmap) * 256 + tid;
    if (q < 3 * a.nd) {
      const int c = q / a.nd, di = q - c * a.nd;
      const int i = p.des_lo[0] + di / (p.des_n[1] * p.des_n[2]);
      const int j = p.des_lo[1] + (di / p.des_n[2]) % p.des_n[1];
      const int k = p.des_lo[2] + di % p.des_n[2];
      a.hist[q] = p.f[c][(long long)i * p.g.sx + (long long)j * p.g.sy + k];   // (no source lies in the design region)
    }
  }
  __syncthreads();
  if (tid == 0) {
    last = true;
    if (gridDim.x > 1) {
      __threadfence();
      last = atomicAdd(a.ticket, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!last) return;
  if (tid < a.ns) {
    // the list is sorted by node: the first source of a node adds those that follow it there
    auto same = [&](int q) { return s.comp[q] == s.comp[tid] && s.id[q] == s.id[tid]; };
    if (tid == 0 || !same(tid - 1)) {
      float v = p.f[s.comp[tid]][s.id[tid]];
      for (int q = tid; q < a.ns && same(q); q++) v += s.v[q];
      p.f[s.comp[tid]][s.id[tid]] = v;
    }
  }
  if (tid == 0) {
    if (gridDim.x > 1) *a.ticket = 0u;
    if (a.advance) *d_step = n + 1;
  }
}

// Running DFT with FP64 accumulators: acc += f(t) exp(-i w t) dt, t = s*dt for E,
// (s-1/2)*dt for H, s = steps completed.  Every step stages the planes' values
// (tail_kernel); every DFT_STAGE steps dft_flush_kernel folds the staged
// samples into the accumulators in step order, so the accumulator update
// sequence (and its rounding) is that of a per-step update while the
// accumulators are read and written once per DFT_STAGE steps.
// One launch for all planes: a block takes 256 points of one component and up
// to DFT_FCHUNK frequencies, from a map made once.  (A launch per plane with
// all components and frequencies in one thread took 74 us for each of a flux
// box' 18 windows of 41^2 points and 32 frequencies, seven blocks wide, and 119
// us for a 384^2 plane of 4 components and 16 frequencies, whose accumulators'
// bytes take 47.)
constexpr int DFT_FCHUNK = 8;
struct FlushUnit { int plane, comp, slot, f0, ptb; };
__global__ void __launch_bounds__(256) dft_flush_kernel(const DftDev* tab, const FlushUnit* unit, int nslots, double dt) {
  __shared__ double2 ph[DFT_STAGE][DFT_FCHUNK];
  const FlushUnit u = unit[blockIdx.x];
  const DftDev& d = tab[u.plane];
  const int nf = min(DFT_FCHUNK, d.nfreq - u.f0);
  if (threadIdx.x < DFT_STAGE * DFT_FCHUNK) {
    const int sl = threadIdx.x / DFT_FCHUNK, f = threadIdx.x % DFT_FCHUNK;
    if (sl < nslots && f < nf) {
      const double t = (double)d.sstep[sl] - (u.comp < 3 ? 0.0 : 0.5);
      double sn, cs;
      sincos(d.omega[u.f0 + f] * t * dt, &sn, &cs);
      ph[sl][f] = make_double2(cs * dt, -sn * dt);
    }
  }
  __syncthreads();
  const int npts = d.n1 * d.n2, ncomp = __popc(d.comp_mask);
  const int pt = u.ptb * 256 + threadIdx.x;
  if (pt >= npts) return;
  float val[DFT_STAGE];
  const float* st = d.stage + (long long)u.slot * npts + pt;
#pragma unroll
  for (int sl = 0; sl < DFT_STAGE; sl++) val[sl] = sl < nslots ? st[(long long)sl * ncomp * npts] : 0.f;
  double2* acc = d.acc + ((long long)u.slot * d.nfreq + u.f0) * npts + pt;
  double2 v[DFT_FCHUNK];
#pragma unroll
  for (int f = 0; f < DFT_FCHUNK; f++)
    if (f < nf) v[f] = acc[(long long)f * npts];
#pragma unroll
  for (int sl = 0; sl < DFT_STAGE; sl++)
    if (sl < nslots) {
      const double x = (double)val[sl];
#pragma unroll
      for (int f = 0; f < DFT_FCHUNK; f++)
        if (f < nf) { v[f].x += x * ph[sl][f].x; v[f].y += x * ph[sl][f].y; }
    }
#pragma unroll
  for (int f = 0; f < DFT_FCHUNK; f++)
    if (f < nf) acc[(long long)f * npts] = v[f];
}

// Outward Poynting flux of one face of a flux box at every frequency of its
// DFT patch: out[f] = sgn_area * sum_pts Re(E_b conj(H_c) - E_c conj(H_b)) with
// (a, b, c) = (normal, (a+1)%3, (a+2)%3), so that (b, c, a) is right-handed.
// One block per frequency; every thread sums a fixed stride of points and a
// fixed tree combines the threads, so the value does not depend on timing.
constexpr int FLUX_THREADS = 256;
__device__ __forceinline__ int dft_slot(int mask, int comp) { return __popc(mask & ((1 << comp) - 1)); }
__global__ void __launch_bounds__(FLUX_THREADS) flux_face_kernel(DftDev d, double sgn_area, double* out) {
  __shared__ double red[FLUX_THREADS];
  const int f = blockIdx.x;
  const int a = d.axis, b = (a + 1) % 3, c = (a + 2) % 3;
  const long long npts = (long long)d.n1 * d.n2;
  const double2* Eb = d.acc + ((long long)dft_slot(d.comp_mask, b) * d.nfreq + f) * npts;
  const double2* Ec = d.acc + ((long long)dft_slot(d.comp_mask, c) * d.nfreq + f) * npts;
  const double2* Hb = d.acc + ((long long)dft_slot(d.comp_mask, 3 + b) * d.nfreq + f) * npts;
  const double2* Hc = d.acc + ((long long)dft_slot(d.comp_mask, 3 + c) * d.nfreq + f) * npts;
  double s = 0.0;
  for (long long pt = threadIdx.x; pt < npts; pt += FLUX_THREADS) {
    const double2 eb = Eb[pt], ec = Ec[pt], hb = Hb[pt], hc = Hc[pt];
    s += (eb.x * hc.x + eb.y * hc.y) - (ec.x * hb.x + ec.y * hb.y);
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = FLUX_THREADS / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[f] = sgn_area * red[0];
}

// Near-to-far-field transform of a flux box (surface equivalence): on a face
// with outward normal n = sgn e_a the equivalent currents are J = n x H and
// M = -n x E, i.e. J_c = sgn H_b, J_b = -sgn H_c, M_c = -sgn E_b, M_b = sgn E_c
// ((a, b, c) cyclic), and the radiation vectors are
//   N = sum J(r') exp(i k rhat.r') dA,  L = sum M(r') exp(i k rhat.r') dA,
// k = omega (c = 1).  Both currents must lie on one closed surface: the
// tangential E of the face plane w sits at w + 1/2 along the normal and the
// tangential H at w, so H is averaged over the planes w and w + 1 onto the E
// surface, the box [lo + 1/2, hi + 1/2] on every axis.  In the plane every term
// keeps its component's Yee position, and the sum over a face is a quadrature
// over that box's face: along an in-plane axis, a component at integer
// positions takes the midpoints lo+1 .. hi (weight 1), one at half-integer
// positions the points lo+1/2 .. hi+1/2 with the trapezoid weights (1/2 at the
// ends); the windows hold the indices lo .. hi.  The
// DFT phasors follow x(t) = Re(X exp(i w t)), so an outgoing wave carries
// exp(-i k r) and the far field is
//   r E_theta = -i k/(4 pi) (L_phi + N_theta) e^{-ikr},  r E_phi = i k/(4 pi) (L_theta - N_phi) e^{-ikr},
// with radiation intensity U = k^2/(16 pi^2) (|L_phi + N_theta|^2 + |L_theta - N_phi|^2),
// normalised like the flux box (Re(E x H*) without the 1/2), so that the
// integral of U over the sphere equals the box's power.  One block per
// (direction, frequency); FP64 throughout, fixed-order reduction.
struct NtffFaces {
  DftDev f[6];              // tangential E and H of the face planes, windows [lo, hi] in the plane
  DftDev h[6];              // tangential H of the planes one further along each normal
  double org[3];            // the origin of r' (physical units)
  double ds[3];
  int lo[3], hi[3];         // the box (face plane indices)
};
// quadrature weight of in-plane index v for a component at v + o/2, box [lo + 1/2, hi + 1/2]
__host__ __device__ __forceinline__ double ntff_weight(int v, int o, int lo, int hi) {
  if (o == 0) return (v > lo && v <= hi) ? 1.0 : 0.0;
  if (v == lo || v == hi) return 0.5;
  return (v > lo && v < hi) ? 1.0 : 0.0;
}
__global__ void __launch_bounds__(FLUX_THREADS) ntff_kernel(NtffFaces F, const double* theta, const double* phi,
                                                            int nfreq, double* out) {
  __shared__ double red[12][FLUX_THREADS];
  const int dir = blockIdx.x, f = blockIdx.y;
  const double th = theta[dir], ph = phi[dir];
  double sth, cth, sph, cph;
  sincos(th, &sth, &cth);
  sincos(ph, &sph, &cph);
  const double rh[3] = {sth * cph, sth * sph, cth};
  double acc[12];
#pragma unroll
  for (int q = 0; q < 12; q++) acc[q] = 0.0;
  for (int q = 0; q < 6; q++) {
    const DftDev& d = F.f[q];
    const int a = d.axis, b = (a + 1) % 3, c = (a + 2) % 3;
    const double sgn = (q & 1) ? 1.0 : -1.0;
    const int s1 = a == 0 ? 1 : 0, s2 = a == 2 ? 1 : 2;
    const double k = d.omega[f];
    const double dA = F.ds[s1] * F.ds[s2];
    const long long npts = (long long)d.n1 * d.n2;
    const double2* Eb = d.acc + ((long long)dft_slot(d.comp_mask, b) * d.nfreq + f) * npts;
    const double2* Ec = d.acc + ((long long)dft_slot(d.comp_mask, c) * d.nfreq + f) * npts;
    const double2* Hb = d.acc + ((long long)dft_slot(d.comp_mask, 3 + b) * d.nfreq + f) * npts;
    const double2* Hc = d.acc + ((long long)dft_slot(d.comp_mask, 3 + c) * d.nfreq + f) * npts;
    const DftDev& d2 = F.h[q];
    const double2* Hb2 = d2.acc + ((long long)dft_slot(d2.comp_mask, 3 + b) * d2.nfreq + f) * npts;
    const double2* Hc2 = d2.acc + ((long long)dft_slot(d2.comp_mask, 3 + c) * d2.nfreq + f) * npts;
    const int srcs[4] = {3 + b, 3 + c, b, c};       // terms J_c, J_b, M_c, M_b
    for (long long pt = threadIdx.x; pt < npts; pt += FLUX_THREADS) {
      int idx[3];
      idx[a] = d.index;
      idx[s1] = d.lo1 + (int)(pt / d.n2);
      idx[s2] = d.lo2 + (int)(pt % d.n2);
      const double2 hb = Hb[pt], hb2 = Hb2[pt], hc = Hc[pt], hc2 = Hc2[pt];
      const double2 vals[4] = {make_double2(0.5 * (hb.x + hb2.x), 0.5 * (hb.y + hb2.y)),
                               make_double2(0.5 * (hc.x + hc2.x), 0.5 * (hc.y + hc2.y)), Eb[pt], Ec[pt]};
      const double wts[4] = {sgn, -sgn, -sgn, sgn};
      const int dst[4] = {c, b, c, b};
#pragma unroll
      for (int t = 0; t < 4; t++) {
        double proj = 0.0;
#pragma unroll
        for (int x = 0; x < 3; x++) {
          // along the normal every term sits on the E surface w + 1/2
          const double off = x == a ? 0.5 : 0.5 * comp_off(srcs[t], x);
          proj += rh[x] * ((idx[x] + off) * F.ds[x] - F.org[x]);
        }
        const double qw = ntff_weight(idx[s1], comp_off(srcs[t], s1), F.lo[s1], F.hi[s1]) *
                          ntff_weight(idx[s2], comp_off(srcs[t], s2), F.lo[s2], F.hi[s2]);
        if (qw == 0.0) continue;
        double sn, cs;
        sincos(k * proj, &sn, &cs);
        const double re = wts[t] * qw * dA * (vals[t].x * cs - vals[t].y * sn);
        const double im = wts[t] * qw * dA * (vals[t].x * sn + vals[t].y * cs);
        const int base = (t < 2 ? 0 : 6) + 2 * dst[t];
        acc[base] += re;
        acc[base + 1] += im;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < 12; q++) red[q][threadIdx.x] = acc[q];
  __syncthreads();
  for (int w = FLUX_THREADS / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
#pragma unroll
      for (int q = 0; q < 12; q++) red[q][threadIdx.x] += red[q][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    // N = red[0..5] (x, y, z complex), L = red[6..11]; theta/phi components
    const double tv[3] = {cth * cph, cth * sph, -sth}, pv[3] = {-sph, cph, 0.0};
    double Nt[2] = {0, 0}, Np[2] = {0, 0}, Lt[2] = {0, 0}, Lp[2] = {0, 0};
    for (int x = 0; x < 3; x++)
      for (int r = 0; r < 2; r++) {
        Nt[r] += tv[x] * red[2 * x + r][0];
        Np[r] += pv[x] * red[2 * x + r][0];
        Lt[r] += tv[x] * red[6 + 2 * x + r][0];
        Lp[r] += pv[x] * red[6 + 2 * x + r][0];
      }
    const double k = F.f[0].omega[f];
    const double s = k / (4.0 * M_PI);
    // r E_theta = -i s (Lp + Nt), r E_phi = i s (Lt - Np) (the e^{-ikr} dropped)
    const double at[2] = {Lp[0] + Nt[0], Lp[1] + Nt[1]}, ap[2] = {Lt[0] - Np[0], Lt[1] - Np[1]};
    double* o = out + ((long long)dir * nfreq + f) * 5;
    o[0] = s * s * (at[0] * at[0] + at[1] * at[1] + ap[0] * ap[0] + ap[1] * ap[1]);
    o[1] = s * at[1];
    o[2] = -s * at[0];
    o[3] = -s * ap[1];
    o[4] = s * ap[0];
  }
}

// Magnetised-Drude current over the ADE box (dtmx.h, dtmx_material):
// J^{n+1/2} into buffer 1-cur from J^{n-1/2} (buffer cur) and E^n.

// Thread layout of the passes over the ADE box: 256 threads along the box'
// (y, z) plane, blockIdx.y = x.
__device__ __forceinline__ bool ade_cell(const Params& p, int& bi, int& bj, int& bk, long long& q) {
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= p.ade.n[1] * p.ade.n[2]) return false;
  bj = r / p.ade.n[2];
  bk = r - bj * p.ade.n[2];
  bi = blockIdx.y;
  q = (long long)bi * p.ade.n[1] * p.ade.n[2] + r;
  return true;
}

// The three new current components of the node at box position (bi, bj), box
// index q, from the old ones (buffer cur; 0 outside the box and off the
// gyrotropic nodes) and E^n; m: material indices, E: E^n, on: gyrotropic
__device__ __forceinline__ void gyro_new(const Params& p, int cur, int bi, int bj, long long q, const int (&m)[3], const float (&E)[3],
                                         const bool (&on)[3], float (&J)[3]) {
  const MatTable& mt = *p.mt;
  const int dj = p.ade.n[2];
  const long long di = (long long)p.ade.n[1] * dj;
  const float *Jx = p.ade.Jg[cur][0] + q, *Jy = p.ade.Jg[cur][1] + q;
  const bool im = bi > 0, ip = bi + 1 < p.ade.n[0], jm = bj > 0, jp = bj + 1 < p.ade.n[1];
  // every load before its use
  float own[3], near[2][4];
#pragma unroll
  for (int c = 0; c < 3; c++) own[c] = on[c] ? __ldg(p.ade.Jg[cur][c] + q) : 0.f;
  if (on[0]) {
    near[0][0] = im ? __ldg(Jy - di) : 0.f; near[0][1] = on[1] ? own[1] : __ldg(Jy);
    near[0][2] = im && jp ? __ldg(Jy - di + dj) : 0.f; near[0][3] = jp ? __ldg(Jy + dj) : 0.f;
  }
  if (on[1]) {
    near[1][0] = jm ? __ldg(Jx - dj) : 0.f; near[1][1] = ip && jm ? __ldg(Jx + di - dj) : 0.f;
    near[1][2] = on[0] ? own[0] : __ldg(Jx); near[1][3] = ip ? __ldg(Jx + di) : 0.f;
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    J[c] = 0.f;
    if (!on[c]) continue;
    float t = own[c];
    if (c < 2) {
      const float avg = __fmul_rn(0.25f, __fadd_rn(__fadd_rn(__fadd_rn(near[c][0], near[c][1]), near[c][2]), near[c][3]));
      const float s = __fmul_rn(__ldg(&mt.gS[m[c]]), avg);
      t = __fmaf_rn(__ldg(&mt.gC[m[c]]), own[c], c == 0 ? s : -s);
    }
    J[c] = __fmaf_rn(__ldg(&mt.gA[m[c]]), t, __fmul_rn(__ldg(&mt.gB[m[c]]), E[c]));
  }
}

// J^{n+1/2} into buffer 1-cur (per-step engine: before the E half step changes E)
__global__ void __launch_bounds__(256) gyro_current_kernel(const __grid_constant__ Params p, int cur) {
  pdl_wait();
  pdl_trigger();
  int bi, bj, bk;
  long long q;
  if (!ade_cell(p, bi, bj, bk, q)) return;
  const int i = p.ade.lo[0] + bi, j = p.ade.lo[1] + bj, k = p.ade.lo[2] + bk;
  const long long id = (long long)i * p.g.sx + (long long)j * p.g.sy + k;
  // (E, the old current, materials and table are read-only in this pass)
  int m[3];
  float E[3], J[3];
  bool on[3];
#pragma unroll
  for (int c = 0; c < 3; c++) { m[c] = p.mat[c] ? (int)__ldg(p.mat[c] + id) : 0; E[c] = __ldg(p.f[c] + id); }
#pragma unroll
  for (int c = 0; c < 3; c++) on[c] = __ldg(&p.mt->gjc[m[c]]) != 0.f;
  gyro_new(p, cur, bi, bj, q, m, E, on, J);
#pragma unroll
  for (int c = 0; c < 3; c++)
    if (on[c]) p.ade.Jg[1 - cur][c][q] = J[c];
}

// Dispersive and gyrotropic E nodes, after the field pass (which leaves
// dispersive nodes at their old value): the ADE recursion (countDisp,
// dispersion.cpp:85-99) with rot = dt curl H recomputed from H exactly as the
// field kernels compute it, and E -= dt/eps_inf J^{n+1/2} on gyrotropic nodes.
// One thread per cell of the ADE box; BOX: zero-outside geometry (bounds-checked
// taps).  CUR: the gyrotropic current is advanced here too, from E^n in the
// single sweep's other set (p.fe_old): one pass over it instead of two.
// The three components' loads are issued together (materials, then flags, then
// state and taps: three round trips a cell, where a component at a time made
// nine).  A 236x236x76 gyrotropic layer took 84 + 102 us in two passes and takes
// 78 (98 at three blocks per SM instead of five); the Drude film of the reference
// geometry (8 cells along z, so lanes run along y and z together) 76 -> 32 us.
template <int ORDER, bool BOX, bool CUR>
__global__ void __launch_bounds__(256, CUR ? 5 : 4) ade_node_kernel(const __grid_constant__ Params p, int cur) {
  pdl_wait();
  pdl_trigger();
  const MatTable& mt = *p.mt;
  int bi, bj, bk;
  long long q;
  if (!ade_cell(p, bi, bj, bk, q)) return;
  const int i = p.ade.lo[0] + bi, j = p.ade.lo[1] + bj, k = p.ade.lo[2] + bk;
  const long long id = (long long)i * p.g.sx + (long long)j * p.g.sy + k;
  // (materials, table, H and the old E are read-only in this pass)
  int m[3], np[3];
  float gj[3];
#pragma unroll
  for (int c = 0; c < 3; c++) m[c] = p.mat[c] ? (int)__ldg(p.mat[c] + id) : 0;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const bool live = BOX || is_live(p.g, c, i, j, k);
    np[c] = live ? __ldg(&mt.npoles[m[c]]) : 0;
    gj[c] = live ? __ldg(&mt.gjc[m[c]]) : 0.f;
  }
  if (np[0] > 0 || np[1] > 0 || np[2] > 0) {
    // taps of H: the node's own and, per curl term, those along its axis (E taps at -1..+2)
    float v[3][2][4], E0[3];
    bool inside = true;
    if (!BOX) {
      const int ix[3] = {i, j, k};
#pragma unroll
      for (int a = 0; a < 3; a++) inside = inside && ix[a] - 1 >= p.g.all_lo[a] && ix[a] + 2 <= p.g.all_hi[a];
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (np[c] <= 0) continue;
      E0[c] = p.fe_old[c] ? __ldg(p.fe_old[c] + id) : p.f[c][id];
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const int a = (c + 1 + t) % 3;             // curl axis of term t
        const int g = 3 + (c + 2 - t) % 3;         // source H component of term t
        const long long sa = a == 0 ? p.g.sx : a == 1 ? p.g.sy : 1;
        const int ia = a == 0 ? i : a == 1 ? j : k;
#pragma unroll
        for (int o = 0; o < 4; o++) {
          v[c][t][o] = 0.f;
          if (ORDER == 2 && (o == 0 || o == 3)) continue;
          if (BOX || inside) {
            if (!BOX || (ia + o - 1 >= 0 && ia + o - 1 < p.g.n[a])) v[c][t][o] = __ldg(p.f[g] + id + (long long)(o - 1) * sa);
          } else {
            v[c][t][o] = fetch<1>(p, g, a == 0 ? i + o - 1 : i, a == 1 ? j + o - 1 : j, a == 2 ? k + o - 1 : k);
          }
        }
      }
    }
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (np[c] <= 0) continue;
      float d[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int t = 0; t < 2; t++) {
        const int a = (c + 1 + t) % 3;
        d[a] = __fmul_rn(t == 0 ? p.cdt[a] : -p.cdt[a], dstencil<ORDER>(v[c][t][0], v[c][t][1], v[c][t][2], v[c][t][3]));
      }
      p.f[c][id] = ade_update(p, c, m[c], np[c], q, sum3(d[0], d[1], d[2]), E0[c]);
    }
  }
  bool on[3];
#pragma unroll
  for (int c = 0; c < 3; c++) on[c] = np[c] <= 0 && gj[c] != 0.f;
  if (!(on[0] || on[1] || on[2])) return;
  float J[3], F[3];
  if (CUR) {
    float E[3];
#pragma unroll
    for (int c = 0; c < 3; c++) { F[c] = on[c] ? p.f[c][id] : 0.f; E[c] = on[c] ? __ldg(p.fe_old[c] + id) : 0.f; }
    gyro_new(p, cur, bi, bj, q, m, E, on, J);
#pragma unroll
    for (int c = 0; c < 3; c++)
      if (on[c]) p.ade.Jg[1 - cur][c][q] = J[c];
  } else {
#pragma unroll
    for (int c = 0; c < 3; c++) {
      F[c] = on[c] ? p.f[c][id] : 0.f;
      J[c] = on[c] ? __ldg(p.ade.Jg[1 - cur][c] + q) : 0.f;
    }
  }
#pragma unroll
  for (int c = 0; c < 3; c++)
    if (on[c]) p.f[c][id] = __fsub_rn(F[c], __fmul_rn(gj[c], J[c]));
}

__global__ void mask_nonlive_kernel(Params p, int comp, long long ncell) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < ncell; q += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(q % p.g.n[2]);
    const long long r = q / p.g.n[2];
    const int j = (int)(r % p.g.n[1]);
    const int i = (int)(r / p.g.n[1]);
    if (!is_live(p.g, comp, i, j, k)) p.f[comp][(long long)i * p.g.sx + (long long)j * p.g.sy + k] = 0.f;
  }
}

__global__ void nonfinite_kernel(Params p, int comp, long long ncell, int* flag) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < ncell; q += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(q % p.g.n[2]);
    const long long r = q / p.g.n[2];
    const int j = (int)(r % p.g.n[1]);
    const int i = (int)(r / p.g.n[1]);
    const float v = p.f[comp][(long long)i * p.g.sx + (long long)j * p.g.sy + k];
    if (!isfinite(v)) { atomicExch(flag, 1); return; }
  }
}

}  // namespace dtmx
