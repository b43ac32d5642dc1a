// mpm_batch_kernels.cuh -- kernels of the batched mixed-precision step (see
// mpm_batch.cuh for the layout). FP32 particle math, FP64 grid accumulation.
#pragma once

#include "mpm_batch.cuh"
#include "mpm_kernels.cuh"
#include "mpm_sort.cuh"

namespace mpm {
namespace bm {

__device__ __forceinline__ long long btid() { return (long long)blockIdx.x * blockDim.x + threadIdx.x; }

__device__ __forceinline__ bool scene_live(const BState& b, int s) { return b.sst[s].active != 0; }

// scene of item i (a particle, node or centre node): with one scene resident it
// is known without a load, which heads the chain of dependent ones in each
// kernel (steps: Cook 5.8 k particles 76.4 -> 74.4 us, beam 94 k 98.9 -> 96.9,
// column 4.1 M 1513 -> 1497, slopes unchanged). The stress update and the SGMP
// force kernel read it: there the test costs registers that spill (twelve
// scenes in one batch 306 -> 309 us).
__device__ __forceinline__ int scene_of(const BState& b, const uint16_t* scene, long long i) {
  return b.nscene == 1 ? 0 : (int)scene[i];
}

// local node (jx, jy, jz) of a global node index
// n / d for 0 <= n < 2^32 by the multiplier m of d (Scene::m*; 0: d = 1),
// a 64-bit high multiply instead of an integer division
__device__ __forceinline__ int div_by(long long n, unsigned long long m) {
  return m ? (int)__umul64hi((unsigned long long)n, m) : (int)n;
}

__device__ __forceinline__ void node_xyz(const Scene& sc, long long ln, int& jx, int& jy, int& jz) {
  jz = div_by(ln, sc.mNGxy);
  int rem = (int)(ln - (long long)jz * sc.NGxy);
  jy = div_by(rem, sc.mNGx);
  jx = rem - jy * sc.NGx;
}

// -------------------------------------------------------------- 1-D shapes
// Offsets are node index minus particle cell index (t) or the particle's
// position relative to the node in cells (r); derivatives are per cell.
__device__ __forceinline__ void lin1(int t, float off, float& w, float& d) {
  w = t ? off : 1.f - off;
  d = t ? 1.f : -1.f;
}
__device__ __forceinline__ void gimp1(float r, float& w, float& d) { gimp_1d<float>(r, w, d); }
// the same values as gimp1, every branch evaluated and the result selected:
// a warp's particles sit in different pieces of the shape, and the branches
// of gimp1 would run one after another
__device__ __forceinline__ void gimp1_select(float r, float& w, float& d) {
  const float a = r < 0.f ? -r : r, sg = copysignf(1.f, r);
  const float w1 = (7.f - 16.f * a * a) * 0.125f, d1 = -(4.f * r);
  const float w2 = 1.f - a, d2 = -sg;
  const float t = (5.f - 4.f * a) * 0.25f;
  const float w3 = t * t, d3 = 2.f * r - sg * 2.5f;
  w = a < 0.25f ? w1 : (a < 0.75f ? w2 : (a < 1.25f ? w3 : 0.f));
  d = a < 0.25f ? d1 : (a < 0.75f ? d2 : (a < 1.25f ? d3 : 0.f));
}
__device__ __forceinline__ void bsp1(int t, float off, float& w, float& d) {
  // NShape_Bspline pieces (Grid.f90:927-962) with r = off * 0.2 + 0.4
  float r = off * 0.2f + 0.4f;
  if (t < 0) {
    float a = 3.f - 5.f * r;
    w = 0.5f * a * a;
    d = (5.f * r - 3.f) * 5.f * 0.2f;
  } else if (t == 0) {
    w = -25.f * r * r + 25.f * r - 5.5f;
    d = (-50.f * r + 25.f) * 0.2f;
  } else {
    float a = 5.f * r - 2.f;
    w = 0.5f * a * a;
    d = (5.f * r - 2.f) * 5.f * 0.2f;
  }
}


// per-scene bound slots of the transfers (SceneState::qmax, float bits):
// mass (set when a scene is laid out), momentum of the step's first transfer,
// force, and momentum with the updated velocities (the MUSL transfer's bound
// and the next step's Q_MOM)
enum QSlot { Q_MASS = 0, Q_MOM = 1, Q_FORCE = 2, Q_MOM_MUSL = 3 };

// ------------------------------------------------------------- begin step
// A step starts in two kernels. kb_begin (which scenes take the step, the
// transfers' bounds and counters) touches nothing that the previous step's
// energy / DT reduction reads or writes, so the two may run side by side;
// step_tick (step count, time, the re-sort decision) needs the reduction's DT
// and the mass transfer's count of particles out of order, and runs as the
// last block of the mass finalize.
__global__ void kb_begin(BState b, const int* target) {
  chain_entry();
  int s = (int)btid();
  if (s == 0) b.gbar[0] = 0u;  // the re-sort's barrier
  if (s >= b.nscene) return;
  SceneState& t = b.sst[s];
  t.active = t.istep < target[s] ? 1 : 0;
  b.disorder[s] = 0;
  if (!t.active) return;
  t.active_nodes = 0;
  // the momentum bound taken with the last step's final velocities
  t.qmax[Q_MOM] = t.qmax[Q_MOM_MUSL];
  t.qmax[Q_FORCE] = t.qmax[Q_MOM_MUSL] = 0u;
}

// ---------------------------------------------- FP64 <-> FP32 off the FP64 pipe
// GB300 runs FP64 arithmetic and every conversion to or from a 64-bit type
// on a narrow pipe (1/64 of the FP32 rate); the mixed-precision kernels
// convert between FP64 storage and FP32 arithmetic with integer operations.
// Magnitudes below the FP32 normal range give 0 (sign kept), above it (and
// NaN) infinity; positions, velocities and masses lie far inside it.

// FP32 value of x truncated toward zero (its leading 24 bits)
__device__ __forceinline__ float f32_trunc(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ffu) - 1023 + 127;
  const unsigned mant = ((hi & 0xfffffu) << 3) | (lo >> 29);
  const unsigned mag = e <= 0 ? 0u : (e >= 255 ? 0x7f800000u : ((unsigned)e << 23) | mant);
  return __uint_as_float((hi & 0x80000000u) | mag);
}

// FP32 rounding of x, to nearest even (the value of (float)x)
__device__ __forceinline__ float f32_rn(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ffu) - 1023 + 127;
  const unsigned mant = ((hi & 0xfffffu) << 3) | (lo >> 29);
  // round bit: mantissa bit 28 of the low word; sticky: bits 0..27 (ties to
  // even on the kept last bit); a carry out of the mantissa steps the exponent
  const unsigned inc = ((lo >> 28) & 1u) & (((lo & 0x0fffffffu) != 0u) | (mant & 1u));
  unsigned mag = (((unsigned)e << 23) | mant) + inc;
  mag = e <= 0 ? 0u : (e >= 255 || mag >= 0x7f800000u ? 0x7f800000u : mag);
  return __uint_as_float((hi & 0x80000000u) | mag);
}

// exact FP64 value of an FP32 value (normal or zero)
__device__ __forceinline__ double f64_of(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned e = (u >> 23) & 0xffu;
  const unsigned hi = (u & 0x80000000u) | (e ? ((e + 896u) << 20) | ((u & 0x7fffffu) >> 3) : 0u);
  const unsigned lo = e ? u << 29 : 0u;
  return __hiloint2double((int)hi, (int)lo);
}

// x as hi + lo: hi its leading 24 bits, lo the remaining 29 rounded to FP32
// (one 32-bit integer conversion), so hi + lo = x to 2^-47 relative
__device__ __forceinline__ void f32_split(double x, float& hi, float& lo) {
  hi = f32_trunc(x);
  const unsigned w = (unsigned)__double2hiint(x), l = (unsigned)__double2loint(x);
  const int eb = (int)((w >> 20) & 0x7ffu);
  // lo = (l mod 2^29) * 2^(e - 52), e = eb - 1023: FP32 biased exponent eb - 948
  const float r = __uint2float_rn(l & 0x1fffffffu) * __uint_as_float(eb > 948 ? (unsigned)(eb - 948) << 23 : 0u);
  lo = (w & 0x80000000u) ? -r : r;
}

// cell of a position (InWhichCell, Grid.f90:123-155) and the offset in it, in
// cells (FP32); false off the grid. Every transfer and gather takes a
// particle's cell and shape-function offsets from this one routine (through
// the per-step data the mass transfer writes).
__device__ __forceinline__ bool cell_of(const Scene& sc, const double x[3], int cc[3], float off[3]) {
  bool in = true;
  for (int a = 0; a < 3; ++a) {
    if (x[a] < sc.span0[a] || x[a] > sc.span1[a]) in = false;
    double u = (x[a] - sc.span0[a]) * sc.idcell;
    cc[a] = (int)u;
    off[a] = (float)(u - (double)cc[a]);
  }
  return in && cc[0] < sc.NCx && cc[1] < sc.NCy && cc[2] < sc.NCz;
}

// cell_of for the linear, GIMP and B-spline scenes without FP64
// instructions: x - span0 and its product with 1 / dcell carried as FP32
// hi + lo pairs (to about 2^-46), so the offset is exact to far below its
// FP32 rounding. The cell can differ from cell_of's only for a position
// within about 1e-12 cells of a face (or of the grid's edge), where the
// shape functions of the two cells agree.
__device__ __forceinline__ bool cell_of_df(const Scene& sc, const double x[3], int cc[3], float off[3]) {
  bool in = true;
  const int nc[3] = {sc.NCx, sc.NCy, sc.NCz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float xh, xl;
    f32_split(x[a], xh, xl);
    // d = x - span0: TwoSum of the leading parts, the trailing parts added
    const float s = xh - sc.fspan0[a];
    const float bb = s - xh;
    const float err = (xh - (s - bb)) + (-sc.fspan0[a] - bb);
    const float t = err + (xl - sc.fspan0_lo[a]);
    const float dh = s + t, dl = t - (dh - s);
    // u = d * idcell (the lo * lo term is below the pair's precision)
    const float uh = dh * sc.fidcell;
    const float ul = fmaf(dh, sc.fidcell, -uh) + fmaf(dh, sc.fidcell_lo, dl * sc.fidcell);
    float c = floorf(uh);
    float f = (uh - c) + ul;  // uh - c is exact
    if (f < 0.f) {
      c -= 1.f;
      f += 1.f;
    } else if (f >= 1.f) {
      c += 1.f;
      f -= 1.f;
    }
    in = in && c >= 0.f && c < (float)nc[a];
    cc[a] = in ? (int)c : 0;
    off[a] = f;
  }
  return in;
}

// SGMP dual (cell-centre) cell of a position, CenterInWhichCell
// (Grid.f90:157-190): the flat index of the per-direction truncations, valid
// when it lies in 0..CNC-1. Like the reference, a position within half a cell
// of the upper grid faces yields a per-direction index past the last dual
// cell, and the flat index then continues into the next row / layer.
__device__ __forceinline__ long long dual_cell(const Scene& sc, const double x[3]) {
  long long d = 0;
  int dc[3];
  for (int a = 0; a < 3; ++a) dc[a] = (int)((x[a] - sc.span0[a]) * sc.idcell - 0.5);
  d = ((long long)dc[2] * sc.CNCy + dc[1]) * sc.CNCx + dc[0];
  return (d >= 0 && d < sc.CNC) ? d : -1;
}

// (xh + xl) - (sh + sl) as a pair dh + dl: TwoSum of the leading parts, the
// trailing parts added
__device__ __forceinline__ void df_diff(float xh, float xl, float sh, float sl, float& dh, float& dl) {
  const float s = xh - sh;
  const float bb = s - xh;
  const float err = (xh - (s - bb)) + (-sh - bb);
  const float t = err + (xl - sl);
  dh = s + t;
  dl = t - (dh - s);
}

// The SGMP decisions of a position -- its cell and offsets (cell_of), its
// nearest node (the cell's upper one from half a cell on) and its dual cell
// (dual_cell) -- in FP32 double-float arithmetic: x - span0 and x - span1
// as pairs, the coordinate in cells to about 2^-45. Returns false, leaving
// the decisions to the FP64 routines, for a position outside the grid or
// within 2^-40 (relative) of a grid face, a cell face or a half cell, where
// the roundings of the FP64 arithmetic could decide otherwise; every
// decision it returns is the FP64 one. (The nearest node and the dual cell
// are discontinuous at the half cell, so they must be the FP64 ones.)
__device__ __forceinline__ bool sg_locate_df(const Scene& sc, const double x[3], int cc[3], float off[3], int nd[3],
                                             long long& dual) {
  const int nc[3] = {sc.NCx, sc.NCy, sc.NCz};
  int dc[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float xh, xl, dh, dl, eh, el;
    f32_split(x[a], xh, xl);
    df_diff(xh, xl, sc.fspan0[a], sc.fspan0_lo[a], dh, dl);
    df_diff(xh, xl, sc.fspan1[a], sc.fspan1_lo[a], eh, el);
    const float gtol = 0x1p-40f * fabsf(xh);
    if (!(dh > gtol && eh < -gtol)) return false;  // outside or at a grid face
    const float uh = dh * sc.fidcell;
    const float ul = fmaf(dh, sc.fidcell, -uh) + fmaf(dh, sc.fidcell_lo, dl * sc.fidcell);
    const float cf = floorf(uh), fh = uh - cf;  // (exact)
    // distances to the cell's faces and its half (a rounded sum keeps the
    // sign of the exact one)
    const float r0 = fh + ul, r1 = (fh - 1.f) + ul, rh = (fh - 0.5f) + ul;
    const float tol = 0x1p-40f * fmaxf(1.f, uh);
    if (!(r0 > tol && r1 < -tol && fabsf(rh) > tol)) return false;
    const int c = (int)cf;
    if (c >= nc[a]) return false;
    cc[a] = c;
    off[a] = r0;
    nd[a] = c + (rh > 0.f);
    dc[a] = max(nd[a] - 1, 0);  // trunc(u - 1/2): 0 below half a cell
  }
  const long long d = ((long long)dc[2] * sc.CNCy + dc[1]) * sc.CNCx + dc[0];
  dual = (d >= 0 && d < sc.CNC) ? d : -1;
  return true;
}

// -------------------------------------------------------------- locate
// The step's derived data of a particle at position x (ParticleInitial,
// update_step.f90:408-453, in FP32 form): cell (-1 off the grid) and offset in
// it; for SGMP also the dual cell, the nearest node and the coordinates about
// both. cc, off and dual return what the transfers need.
__device__ __forceinline__ bool locate_one(const BState& b, const Scene& sc, long long i, const double x[3], int cc[3],
                                           float off[3], long long& dual) {
  const long long NP = b.NP;
  int nd[3];
  dual = -1;
  bool in;
  if (sc.shape != 3) {
    in = cell_of_df(sc, x, cc, off);
  } else if (sg_locate_df(sc, x, cc, off, nd, dual)) {
    in = true;
  } else {
    in = cell_of(sc, x, cc, off);
    for (int a = 0; a < 3; ++a) {
      const double u = (x[a] - sc.span0[a]) * sc.idcell;  // (as in cell_of)
      nd[a] = cc[a] + (u - (double)cc[a] >= 0.5);
    }
    dual = dual_cell(sc, x);
  }
  for (int a = 0; a < 3; ++a) b.off[a * NP + i] = off[a];
  b.cell[i] = in ? (cc[2] * sc.NCy + cc[1]) * sc.NCx + cc[0] : -1;
  if (sc.shape == 3) {
    // dual (cell-centre) grid: CenterInWhichCell (as the sort keys) and the
    // nearest node with the particle's coordinates about it, both decided
    // as in FP64 (sg_locate_df or the FP64 routines above: the node must
    // stay the one above the dual cell, deciding on the FP32 offset would
    // move particles within 3e-8 of the half onto the other node);
    // XXN = 2 off - 2 (upper node) or 2 off in FP32
    b.dual[i] = (int)dual;
    bool nin = nd[0] >= 0 && nd[0] < sc.NGx && nd[1] >= 0 && nd[1] < sc.NGy && nd[2] >= 0 && nd[2] < sc.NGz;
    int ln = nin ? (nd[2] * sc.NGy + nd[1]) * sc.NGx + nd[0] : -1;
    b.inode[i] = ln;
    int bd = ln >= 0 ? b.bd[sc.n0 + ln] : 0;
    for (int a = 0; a < 3; ++a) {
      float xxn = off[a] * 2.f - (nd[a] > cc[a] ? 2.f : 0.f);
      if ((bd >> (2 * a)) & 3) xxn = xxn > 0.f ? 1.f : (xxn < 0.f ? -1.f : 0.f);
      b.xxn[a * NP + i] = xxn;
      b.xn[a * NP + i] = off[a] * 2.f - 1.f;
    }
  }
  return in;
}

// sort key of a particle from its cell (linear, B-spline), its nearest node
// (GIMP, the upper one from half a cell on) or its dual cell (SGMP), relative
// to its scene's keys; -1 off the grid. A GIMP particle reaches the nodes
// within 1.25 cells of it (the cpGIMP quarter rule of FindInflNode), i.e. at
// most one node either side of its nearest node in each direction: binned by
// nearest node, a key's particles reach a 3 x 3 x 3 box of nodes instead of
// the 4 x 4 x 4 box of a cell's particles. The scatters' segments are runs of
// equal keys of the same definition.
__device__ __forceinline__ int gimp_key(const Scene& sc, int c[3], const float off[3]) {
  for (int a = 0; a < 3; ++a) c[a] += off[a] >= 0.5f;
  return (c[2] * sc.NGy + c[1]) * sc.NGx + c[0];
}

// ------------------------------------------------------------------ keys
// f(s, i, in) for every particle i of the scenes s that are re-sorted this step
// (BState::resort), in chunks of a block's threads; in: the thread has a
// particle. Every thread of the grid calls it. A block takes a run of chunks: one
// search for its first scene (a search for every chunk: the sort of 4000 scenes of
// 512 particles 340 us for 273).
template <class F>
__device__ __forceinline__ void for_resorted(const BState& b, F f) {
  const int *scene = b.resort + kResortScenes, *first = scene + b.nscene;
  const int n = b.resort[0], chunks = first[n];
  const int per = (chunks + gridDim.x - 1) / gridDim.x;
  const int t0 = min((long long)blockIdx.x * per, (long long)chunks), t1 = min(t0 + per, chunks);
  if (t0 >= t1) return;
  int lo = 0, hi = n - 1;  // the last scene whose first chunk is at or before t0
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (first[mid] <= t0) lo = mid;
    else hi = mid - 1;
  }
  for (int t = t0; t < t1; ++t) {
    while (first[lo + 1] <= t) ++lo;
    const int s = scene[lo];
    const long long l = (long long)(t - first[lo]) * kSortThreads + threadIdx.x;
    f(s, b.scenes[s].p0 + l, l < b.scenes[s].np);
  }
}

// Sort keys and per-key counts of the scenes that are re-sorted this step, from
// the step's derived data; the scene's last key collects the particles outside
// the grid. The sort numbers those scenes' keys and particles without gaps: a
// scene's key k is number k0 + k - kshift[s], its particle i number i - shift[s].
__device__ __forceinline__ void sort_keys(BState& b) {
  const long long NP = b.NP;
  for_resorted(b, [&](int s, long long i, bool in) {
    unsigned key = kNoKey;
    if (in) {
      const Scene& sc = b.scenes[s];
      int k = sc.shape == 3 ? b.dual[i] : b.cell[i];
      if (sc.shape == 1 && k >= 0) {
        int c[3];
        c[2] = div_by(k, sc.mNCxy);
        const int rem = k - c[2] * sc.NCxy;
        c[1] = div_by(rem, sc.mNCx);
        c[0] = rem - c[1] * sc.NCx;
        const float off[3] = {b.off[i], b.off[NP + i], b.off[2 * NP + i]};
        k = gimp_key(sc, c, off);
      }
      key = (unsigned)(sc.k0 - b.kshift[s] + (k >= 0 ? k : sc.nk - 1));
      b.key[i] = key;
    }
    // per-key counts: neighbours mostly share a key -- one atomic per key and
    // warp
    const unsigned grp = __match_any_sync(0xffffffffu, key);
    if (key != kNoKey && (threadIdx.x & 31) == __ffs(grp) - 1) atomicAdd(&b.seg[key], __popc(grp));
  });
}

// ---------------------------------------------------- permutation + derived
// dst[i] = src[perm[i]] for every persistent particle field of the scenes
// being re-sorted, then the step's derived data of the particle at its new
// place; permute_back returns the fields to the set every other kernel
// uses.
__device__ __forceinline__ void permute_one(const BState& src, BState& dst, int s, long long i) {
  // every value is loaded before the first store: the stores could alias the
  // loads as far as the compiler knows, so interleaving them would serialise
  // one memory round trip per field
  const long long NP = src.NP;
  const long long j = src.perm[i - src.shift[s]];
  const Scene& sc = src.scenes[s];
  // (the external forces move only in scenes that have some: elsewhere
  // they are zero and nothing reads them)
  double x[3], v[3], f[3] = {0.0, 0.0, 0.0};
  for (int a = 0; a < 3; ++a) {
    x[a] = src.x[a * NP + j];
    v[a] = src.v[a * NP + j];
    if (sc.has_fxp) f[a] = src.fxp[a * NP + j];
  }
  const double mass = src.mass[j], ie = src.ie[j];
  const float vol = src.vol[j], evol = src.evol[j], sig_y = src.sig_y[j], sm = src.sm[j], seqv = src.seqv[j];
  float sd[6];
  for (int a = 0; a < 6; ++a) sd[a] = src.sd[a * NP + j];
  const float epeff = src.epeff[j], celsius = src.celsius[j], dmg = src.dmg[j], lt = src.lt[j], cp = src.cp[j],
              q = src.q[j];
  const uint8_t failure = src.failure[j];
  const uint16_t body = src.body[j];
  const int orig = src.orig[j];
  if (src.any_uvfp) {
    float fp[18];
    for (int a = 0; a < 18; ++a) fp[a] = src.fp[a * NP + j];
    for (int a = 0; a < 18; ++a) dst.fp[a * NP + i] = fp[a];
  }
  for (int a = 0; a < 3; ++a) {
    dst.x[a * NP + i] = x[a];
    dst.v[a * NP + i] = v[a];
    if (sc.has_fxp) dst.fxp[a * NP + i] = f[a];
  }
  dst.mass[i] = mass;
  dst.ie[i] = ie;
  dst.vol[i] = vol;
  dst.evol[i] = evol;
  dst.sig_y[i] = sig_y;
  dst.sm[i] = sm;
  dst.seqv[i] = seqv;
  for (int a = 0; a < 6; ++a) dst.sd[a * NP + i] = sd[a];
  dst.epeff[i] = epeff;
  dst.celsius[i] = celsius;
  dst.dmg[i] = dmg;
  dst.lt[i] = lt;
  dst.cp[i] = cp;
  dst.q[i] = q;
  dst.failure[i] = failure;
  dst.body[i] = body;
  dst.orig[i] = orig;
  // derived
  int cc[3];
  float off[3];
  long long dual;
  locate_one(dst, sc, i, x, cc, off, dual);
  dst.m32[i] = f32_rn(mass);
  for (int a = 0; a < 3; ++a) dst.v32[a * NP + i] = f32_rn(v[a]);
}

// the re-sorted scenes' fields from the permutation's target set back to the
// working set (a straight copy)
__device__ __forceinline__ void permute_back(const BState& src, BState& dst, int s, long long i) {
  const long long NP = src.NP;
  const Scene& sc = src.scenes[s];
  double x[3], v[3], f[3] = {0.0, 0.0, 0.0};
  for (int a = 0; a < 3; ++a) {
    x[a] = src.x[a * NP + i];
    v[a] = src.v[a * NP + i];
    if (sc.has_fxp) f[a] = src.fxp[a * NP + i];
  }
  const double mass = src.mass[i], ie = src.ie[i];
  const float vol = src.vol[i], evol = src.evol[i], sig_y = src.sig_y[i], sm = src.sm[i], seqv = src.seqv[i];
  float sd[6];
  for (int a = 0; a < 6; ++a) sd[a] = src.sd[a * NP + i];
  const float epeff = src.epeff[i], celsius = src.celsius[i], dmg = src.dmg[i], lt = src.lt[i], cp = src.cp[i],
              q = src.q[i];
  const uint8_t failure = src.failure[i];
  const uint16_t body = src.body[i];
  const int orig = src.orig[i];
  for (int a = 0; a < 3; ++a) {
    dst.x[a * NP + i] = x[a];
    dst.v[a * NP + i] = v[a];
    if (sc.has_fxp) dst.fxp[a * NP + i] = f[a];
  }
  dst.mass[i] = mass;
  dst.ie[i] = ie;
  dst.vol[i] = vol;
  dst.evol[i] = evol;
  dst.sig_y[i] = sig_y;
  dst.sm[i] = sm;
  dst.seqv[i] = seqv;
  for (int a = 0; a < 6; ++a) dst.sd[a * NP + i] = sd[a];
  dst.epeff[i] = epeff;
  dst.celsius[i] = celsius;
  dst.dmg[i] = dmg;
  dst.lt[i] = lt;
  dst.cp[i] = cp;
  dst.q[i] = q;
  dst.failure[i] = failure;
  dst.body[i] = body;
  dst.orig[i] = orig;
  if (src.any_uvfp) {
    float fp[18];
    for (int a = 0; a < 18; ++a) fp[a] = src.fp[a * NP + i];
    for (int a = 0; a < 18; ++a) dst.fp[a * NP + i] = fp[a];
  }
}

// ------------------------------------------- deterministic P2G scatter
// Particle -> node transfers of linear, GIMP and B-spline scenes, and the
// particle -> centre-node transfers of SGMP scenes, are scatters: each cell's
// (dual cell's) particles add their FP32 contributions to the nodes they
// influence. Contributions are quantised to 64-bit fixed point with a
// per-scene, per-quantity power-of-two scale and summed with integer adds, so
// a node's sum is exact and independent of the order of the adds (and of
// which other scenes share the batch). The scale comes from a per-step bound
// B on any single contribution's magnitude (a max over the scene's particles,
// also order-independent): a node sums at most np contributions, np * B <
// 2^E, and contributions are scaled by 2^(61 - E), so no sum can reach 2^62.
// The rounding of a contribution to the fixed-point grid (np * B * 2^-61)
// is far below its FP32 rounding.
// The bounds are taken by the kernels that run before each transfer (layout or
// restore for the first step, force staging, position update).

// Max of non-negative values v[k] over the block into sst[s].qmax[slot[k]],
// per scene s (s < 0: no value). Every thread of the block must call it.
// Warps whose lanes all belong to one scene combine through shared memory,
// so a block usually issues one atomic per slot: a per-warp atomic on the
// same address from every warp of a large scene would serialise in L2.
template <int NS>
__device__ __forceinline__ void block_scene_max(BState& b, int s, const int (&slot)[NS], const float (&v)[NS]) {
  __shared__ int ws[32];
  __shared__ unsigned wv[32][NS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const unsigned grp = __match_any_sync(0xffffffffu, s);
  unsigned mx[NS];
  for (int k = 0; k < NS; ++k) mx[k] = __reduce_max_sync(grp, __float_as_uint(v[k]));
  const bool uniform = grp == 0xffffffffu;
  if (!uniform && s >= 0 && lane == __ffs(grp) - 1)
    for (int k = 0; k < NS; ++k) atomicMax(&b.sst[s].qmax[slot[k]], mx[k]);
  if (lane == 0) {
    ws[warp] = uniform ? s : -1;
    for (int k = 0; k < NS; ++k) wv[warp][k] = mx[k];
  }
  __syncthreads();
  if (warp == 0) {
    const int s2 = lane < nw ? ws[lane] : -1;
    const unsigned g2 = __match_any_sync(0xffffffffu, s2);
    for (int k = 0; k < NS; ++k) {
      const unsigned m2 = __reduce_max_sync(g2, lane < nw ? wv[lane][k] : 0u);
      if (s2 >= 0 && lane == __ffs(g2) - 1) atomicMax(&b.sst[s2].qmax[slot[k]], m2);
    }
  }
}

// Fixed-point shift sh of a scene's channel: contributions are rounded to
// integers after scaling by 2^sh, sh = 61 - E with np * bound < 2^E, so no
// sum of a scene's contributions overflows, and at most 47 - Eb with
// bound < 2^Eb, so that one flushed sum (at most 32 contributions) stays
// below 2^53 for quant (this limit binds below 16384 particles only);
// clamped to the FP32 exponent range, 0 when the bound is 0 and every
// contribution is 0.
__device__ __forceinline__ int q_shift(const Scene& sc, unsigned bound_bits) {
  const float bound = __uint_as_float(bound_bits);
  if (!(bound > 0.f)) return 0;
  int E, Eb;
  frexpf(sc.fnp * bound, &E);  // np < 2^31: the product is exact up to one rounding, covered by E + 1
  frexpf(bound, &Eb);
  return max(-126, min(127, min(61 - E, 47 - Eb)));
}
__device__ __forceinline__ float q_scale(int sh) { return __int_as_float((sh + 127) << 23); }
// f = c * 2^sh rounded to the nearest 64-bit integer (ties to even) for
// |f| <= 2^53, without the FP64 pipe (GB300 converts float to int64 there,
// at a small fraction of the 32-bit conversion rate). f splits exactly into
// h * 2^31 + r: the FP32 sum f + 1.5 * 2^54 lies in the binade whose ulp is
// 2^31, so it is 1.5 * 2^54 + h * 2^31 with h = f / 2^31 rounded to
// nearest, and h is the difference of the two bit patterns; the remainder
// r = f - h * 2^31 has |r| <= 2^30 and is exact (a multiple of f's ulp no
// larger than f), so one 32-bit conversion rounds it. h * 2^31 is an
// integer, so the result equals __float2ll_rn(f).
__device__ __forceinline__ long long quant(float c, float scale) {
  constexpr float M = 0x1.8p54f;
  const float f = c * scale;
  const float t = f + M;
  const int h = __float_as_int(t) - __float_as_int(M);
  const int r = __float2int_rn(f - (t - M));
  return (long long)h * 2147483648LL + r;
}
__device__ __forceinline__ double q_unit(int sh) { return __longlong_as_double((long long)(1023 - sh) << 52); }  // 2^-sh

// influence nodes of a particle along one direction: node = cell + t0 + k
// for k < the returned count (at most 3), weight w[k] and derivative d[k]
// (per cell) -- NShape / the cpGIMP quarter rule of FindInflNode with
// NShape_GIMP / NShape_Bspline. Fixed-size arrays with constant indices (the
// gathers unroll their node loops) stay in registers.
__device__ __forceinline__ int dim_nodes(int shape, float off, int& t0, float w[3], float d[3]) {
  if (shape == 0) {
    t0 = 0;
    lin1(0, off, w[0], d[0]);
    lin1(1, off, w[1], d[1]);
    w[2] = d[2] = 0.f;
    return 2;
  }
  if (shape == 2) {
    t0 = -1;
#pragma unroll
    for (int k = 0; k < 3; ++k) bsp1(k - 1, off, w[k], d[k]);
    return 3;
  }
  t0 = off < 0.25f ? -1 : 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) gimp1((float)(-(t0 + k)) + off, w[k], d[k]);
  return 2 + (off < 0.25f) + (off > 0.75f);
}

// The box of a particle's influence nodes for the gathers: index of its first
// node, strides, and the nodes to visit -- within the particle's count and the
// grid -- as a mask of three bits per axis, so that the unrolled loops over the
// 27 nodes test a bit instead of comparing coordinates (stress update of the
// 1.2 M particle slope 98 -> 85 us, dam break 2 M 153 -> 132; the position
// update, bound by its loads then, 91 -> 90 and 134 -> 129).
struct NodeBox {
  long long first;
  int sy, sz;
  unsigned m;
  __device__ __forceinline__ bool x(int k) const { return m >> k & 1u; }
  __device__ __forceinline__ bool row(int ay, int az) const {
    const unsigned r = 8u << ay | 64u << az;
    return (m & r) == r;
  }
};
__device__ __forceinline__ NodeBox node_box(const Scene& sc, const int c[3], const int t0[3], const int nt[3]) {
  NodeBox q;
  const int n[3] = {sc.NGx, sc.NGy, sc.NGz};
  int j[3];
  q.m = 0u;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    j[a] = c[a] + t0[a];
    // nodes j .. j + nt - 1 cut to 0 .. n - 1
    const int lo = max(-j[a], 0), hi = min(nt[a], n[a] - j[a]);
    q.m |= (((1u << max(hi, 0)) - 1u) & ~((1u << lo) - 1u)) << (3 * a);
  }
  q.sy = sc.NGx;
  q.sz = sc.NGxy;
  q.first = sc.n0 + ((long long)j[2] * sc.NGy + j[1]) * sc.NGx + j[0];
  return q;
}

// The re-sort of the scenes marked by step_tick, in one cooperative launch:
// counting sort by key (mpm_sort.cuh), then every field permuted into the
// second particle set and back; over the marked scenes' particles and keys alone
// (over the whole batch, 500 scenes of 512 particles that fly on their own, of
// which some are re-sorted in every step, took 334 us a step linear, 362 GIMP, 520
// SGMP; now 308, 336, 487). A step in which no scene is re-sorted -- most
// of them -- pays one launch that returns at once: 1.6 us of the step, against
// 10 us for an IF node around the phases as kernels of their own and 16 to 34
// us for those kernels returning one by one (5.8 k to 1.2 M particles). The
// barriers between the phases cost a re-sort about what launches would.
__global__ void __launch_bounds__(kSortThreads, 3) kb_resort(BState a, BState o, int polls, int* stall) {
  chain_entry();
  if (!a.resort[0]) return;
  const long long nk = a.resort[1];  // keys of the scenes to sort
  __shared__ int sm[kSmemSeg];  // (the scan's tile, then the long segments)
  __shared__ int thr[kSortThreads], wsum[32];
  const long long g0 = (long long)blockIdx.x * kSortThreads + threadIdx.x, gs = (long long)gridDim.x * kSortThreads;
  unsigned round = 0;
  for (long long k = g0; k < nk; k += gs) a.seg[k] = 0;
  if (g0 == 0) *a.nbig = 0;
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  sort_keys(a);
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  sort_tile_totals(a.seg, nk, a.tiles, thr, wsum);
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  sort_tile_prefix(nk, a.tiles, thr, wsum);
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  sort_tile_scan(a.seg, a.fill, nk, a.tiles, sm, thr, wsum);
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  for_resorted(a, [&](int, long long i, bool in) { sort_place(in ? a.key[i] : kNoKey, i, a.seg, a.fill, a.perm); });
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  sort_segments(a.seg, nk, a.perm, a.big, a.nbig);
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  sort_long(a.seg, a.perm, a.big, a.nbig, sm, [&](int k, int* p, int n) { order_segment(a.key, (unsigned)k, p, n); });
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  for_resorted(a, [&](int s, long long i, bool in) {
    if (in) permute_one(a, o, s, i);
  });
  if (!grid_barrier(a.gbar, ++round, polls, stall)) return;
  for_resorted(a, [&](int s, long long i, bool in) {
    if (in) permute_back(o, a, s, i);
  });
}

// FP32 mass and velocity of the particles of a scene (-1: of every scene),
// when a layout is new or a scene's state was restored (from then on the
// position update keeps the velocity); bounds: also the mass and momentum
// bounds of the first step, for the scenes marked active (new ones -- the
// others carry the bounds of their last step)
__global__ void kb_init_f32(BState b, int scene, int bounds) {
  const long long i = btid(), NP = b.NP;
  int s = -1;
  float bm = 0.f, bv = 0.f;
  if (i < NP && (scene < 0 || b.scene[i] == scene)) {
    s = b.scene[i];
    bm = f32_rn(b.mass[i]);
    const float v[3] = {f32_rn(b.v[i]), f32_rn(b.v[NP + i]), f32_rn(b.v[2 * NP + i])};
    b.m32[i] = bm;
    for (int a = 0; a < 3; ++a) b.v32[a * NP + i] = v[a];
    bv = bm * fmaxf(fabsf(v[0]), fmaxf(fabsf(v[1]), fabsf(v[2]))) * 1.0001f;
    if (!bounds || !scene_live(b, s)) s = -1;
  }
  block_scene_max<2>(b, s, {Q_MASS, Q_MOM_MUSL}, {bm, bv});
}

// Corner k of the dual cell (dx, dy, dz) as a scene cell (its centre node),
// with the reference's flat arithmetic (CenterCellNode, Grid.f90:380-418:
// first corner plus the corner's flat offset; corners at or past the last
// cell are dropped, and a direction with a single cell -- one dual cell --
// spills into the next row); -1 if dropped.
__device__ __forceinline__ long long sg_corner_cell(const Scene& sc, int dx, int dy, int dz, int k) {
  const long long c1 = ((long long)dz * sc.NCy + dy) * sc.NCx + dx;
  const long long cid = c1 + kCorner[k][0] + (long long)kCorner[k][1] * sc.NCx + (long long)kCorner[k][2] * sc.NCxy;
  return cid < (long long)sc.NCxy * sc.NCz ? cid : -1;
}

// -------------------------------------------- particle-parallel scatter
// Linear, GIMP and B-spline scenes scatter in tasks of 32 consecutive
// particles of one scene (task t of a scene: its sorted particles 32 t ..
// 32 t + 31). The lanes of a task that share a sort key (the key's cell, or
// for GIMP its nearest node) form a segment, and every segment's particles
// reach the same box of node offsets (2^3 linear, 3^3 GIMP / B-spline). The
// shapes are tensor products, N = Wx Wy Wz, so a slot's contribution splits
// into an x factor and a (y, z) factor per channel, e.g. for the force
//   f_x = Dx (-s_xx Wy Wz) + Wx (b_x Wy Wz - s_xy Dy Wz - s_xz Wy Dz).
// Two phases through the warp's shared workspace:
//   1. lane = particle: its x factors (W, and D for the force) per x offset
//      and its (y, z) factors per channel;
//   2. lane = (y, z) row of the box and channel: the walk along the task's
//      particles in storage order (FP32 sums of x factor times (y, z) factor for
//      the row's three nodes). A segment's sums are quantised at its end, and a
//      node's added to its 64-bit accumulator with one integer atomic when the
//      walk leaves the node:
//      a segment whose box lies one node further along x -- the usual next key
//      -- leaves one node of the row, any other box all three.
// Bound by instruction issue and the shared-memory / L1 data pipe (76 and 60 % of
// their slots for the mass transfer, 62 and 60 % for the force, on the 1.2
// M-particle slope; L2 atomics 20 %). A lane per node and all its channels read
// 5 (mass and momentum), 8 (force) and 4 (MUSL) shared words per particle and
// flushed every node at every segment end; a lane per row and channel reads its
// own factors and the x factors that all lanes share (a broadcast): 4, 4 and 2,
// the force's as pairs for paired multiply-adds (two per instruction), and
// flushes under half as often. A node's accumulators are adjacent
// (acc[node][4], one 32-byte sector), which a row's lanes hit together. Force
// 93 -> 80, mass 84 -> 81 us (1.2 M particles, GIMP); 309 -> 256, 282 -> 260,
// MUSL 229 -> 189 us (4.1 M); 120 -> 113, 107 -> 107, 87 -> 81 us (2 M, B-spline).
// The task boundaries are fixed by the scene's own sorted order (32 t from
// the scene's first particle), so a scene's sums are the same alone or in a
// batch. Phase 2's walk and its segment ends are the same for every lane
// (the segment mask comes from a warp vote), so the warp never diverges
// there.
template <int MODE>
struct PartShape {
  static constexpr int PF = MODE == 2 ? 6 : 3;          // (y, z) factors per particle and (ty, tz)
  // floats per (ty, tz) row of 32 particles: the rows' factors of one particle
  // and the particles' of one row both fall on distinct banks
  static constexpr int PITCH = 32 * PF + PF;
  static constexpr int XF = MODE == 2 ? 8 : 4;          // x factors per particle: W, or (D, W), per offset
  static constexpr int XAT = (9 * PITCH + 3) / 4 * 4;   // the x factors' place in the workspace
  static constexpr int STRIDE = 33;                     // row stride of the mass factors and of the SGMP form
  static constexpr int MAT = XAT + 32 * XF;             // the mass factors' place (mode 0)
  static constexpr int WS = MAT + (MODE == 0 ? 9 * STRIDE + 3 : 0);  // workspace floats of a warp (a multiple of 4)
  static constexpr int WARPS = MODE == 2 ? 4 : 8;       // warps (tasks) per block (static shared memory)
};

// acc + a * b on both halves of a pair (one instruction)
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 acc) {
  float2 d;
  asm("{\n\t.reg .b64 a, b, c, d;\n\t"
      "mov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(acc.x), "f"(acc.y));
  return d;
}

// 1-D weight w[t] and derivative d[t] (per unit length) of node offset t
// from the key's base (linear: 0..1 from the cell; B-spline: -1..1 from the
// cell; GIMP: -1..1 from the nearest node)
template <int SH>
__device__ __forceinline__ void part_tab(float off, float idc, float (&w)[3], float (&d)[3]) {
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    if (SH == 0) {
      if (t < 2) lin1(t, off, w[t], d[t]);
      else w[t] = d[t] = 0.f;
    } else if (SH == 2) {
      bsp1(t - 1, off, w[t], d[t]);
    } else {
      gimp1_select(off - (float)(t - 1 + (off >= 0.5f)), w[t], d[t]);  // node = nearest - 1 + t
    }
    d[t] *= idc;
  }
}

// The mass transfer (mode 0) opens the step: it locates the particles and
// stores the step's derived data, and returns how many of the task's
// particles come after one with a larger key (0 otherwise).
__device__ __forceinline__ int count_disorder(int key, int cnt) {
  const int lane = threadIdx.x & 31;
  const unsigned prev = (unsigned)__shfl_up_sync(0xffffffffu, key, 1);
  return __popc(__ballot_sync(0xffffffffu, lane > 0 && lane < cnt && prev > (unsigned)key));
}

template <int MODE, int SH>
__device__ __forceinline__ int part_scatter_task(BState& b, const Scene& sc, long long i0, int cnt, float sA,
                                                 float sB, float* ws) {
  using PS = PartShape<MODE>;
  constexpr int PF = PS::PF, PITCH = PS::PITCH, XF = PS::XF;
  constexpr int nt = SH == 0 ? 2 : 3, tlo = SH == 0 ? 0 : -1, NL = 3 * nt * nt;
  const int lane = threadIdx.x & 31;
  const long long NP = b.NP, i = i0 + lane;
  int c[3] = {0, 0, 0};
  float off[3] = {0.f, 0.f, 0.f};
  int key = -1;
  if (MODE == 0) {
    if (lane < cnt) {
      const double x[3] = {b.x[i], b.x[NP + i], b.x[2 * NP + i]};
      const bool in = cell_of_df(sc, x, c, off);
      const int cl = (c[2] * sc.NCy + c[1]) * sc.NCx + c[0];
#pragma unroll
      for (int a = 0; a < 3; ++a) b.off[a * NP + i] = off[a];
      b.cell[i] = in ? cl : -1;
      if (in) key = SH == 1 ? gimp_key(sc, c, off) : cl;
    }
  } else {
    const int cl = lane < cnt ? b.cell[i] : -1;
    if (cl >= 0) {
      c[2] = div_by(cl, sc.mNCxy);
      const int rem = cl - c[2] * sc.NCxy;
      c[1] = div_by(rem, sc.mNCx);
      c[0] = rem - c[1] * sc.NCx;
#pragma unroll
      for (int a = 0; a < 3; ++a) off[a] = b.off[a * NP + i];
      key = SH == 1 ? gimp_key(sc, c, off) : cl;
    }
  }
  const int dis = MODE == 0 ? count_disorder(key, cnt) : 0;
  // segment ends: the last lane of every run of equal keys
  const int knext = __shfl_down_sync(0xffffffffu, key, 1);
  const unsigned lasts = __ballot_sync(0xffffffffu, key >= 0 && (lane == 31 || knext != key));
  if (lasts == 0u) return dis;  // (uniform) nothing of this task on the grid
  // the segment's first box node (scene-local flat index) and whether the
  // whole box lies inside the grid
  const int nbase = ((c[2] + tlo) * sc.NGy + (c[1] + tlo)) * sc.NGx + (c[0] + tlo);
  const bool inner = c[0] + tlo >= 0 && c[0] + tlo + nt <= sc.NGx && c[1] + tlo >= 0 && c[1] + tlo + nt <= sc.NGy &&
                     c[2] + tlo >= 0 && c[2] + tlo + nt <= sc.NGz;
  // phase 1: the particle's factors (zero for a lane without a key)
  {
    constexpr int NQ = MODE == 2 ? 9 : 4;
    float pv[NQ];
    float w[3][3], d[3][3];
#pragma unroll
    for (int q = 0; q < NQ; ++q) pv[q] = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int t = 0; t < 3; ++t) w[a][t] = d[a][t] = 0.f;
    if (key >= 0) {
      if (MODE == 2) {
#pragma unroll
        for (int q = 0; q < 9; ++q) pv[q] = b.fs[q * NP + i];
      } else {
        pv[0] = b.m32[i];
#pragma unroll
        for (int a = 0; a < 3; ++a) pv[1 + a] = b.v32[a * NP + i];
      }
      const float idc = sc.fidcell;
#pragma unroll
      for (int a = 0; a < 3; ++a) part_tab<SH>(off[a], idc, w[a], d[a]);
    }
    float* xf = ws + PS::XAT + lane * XF;
    if (MODE != 2) {
      *reinterpret_cast<float4*>(xf) = make_float4(w[0][0], w[0][1], w[0][2], 0.f);
    } else {
      *reinterpret_cast<float4*>(xf) = make_float4(d[0][0], w[0][0], d[0][1], w[0][1]);
      if (nt == 3) *reinterpret_cast<float2*>(xf + 4) = make_float2(d[0][2], w[0][2]);
    }
    float* col = ws + lane * PF;
#pragma unroll
    for (int tz = 0; tz < nt; ++tz)
#pragma unroll
      for (int ty = 0; ty < nt; ++ty) {
        float* f = col + (tz * nt + ty) * PITCH;
        const float A = w[1][ty] * w[2][tz];
        if (MODE == 2) {
          const float B = d[1][ty] * w[2][tz], C = w[1][ty] * d[2][tz];
          // per channel: the factor of D and the factor of W
          float2* f2 = reinterpret_cast<float2*>(f);
          f2[0] = make_float2(-pv[0] * A, pv[6] * A - pv[3] * B - pv[5] * C);
          f2[1] = make_float2(-pv[3] * A, pv[7] * A - pv[1] * B - pv[4] * C);
          f2[2] = make_float2(-pv[5] * A, pv[8] * A - pv[4] * B - pv[2] * C);
        } else {
          const float M = pv[0] * A;
          if (MODE == 0) ws[PS::MAT + (tz * nt + ty) * PS::STRIDE + lane] = M;
#pragma unroll
          for (int a = 0; a < 3; ++a) f[a] = M * pv[1 + a];
        }
      }
  }
  __syncwarp();
  // phase 2: lane = (y, z) row of the box and channel, the walk along the
  // particles
  const int yz = lane < NL ? lane / 3 : 0, ch = lane % 3;
  const int sz = yz / nt, sy = yz % nt;
  const int soff = (sz * sc.NGy + sy) * sc.NGx;
  const float* xr = ws + PS::XAT;
  const float* fr = ws + yz * PITCH + (MODE == 2 ? 2 * ch : ch);
  const float* mr = ws + (MODE == 0 ? PS::MAT + yz * PS::STRIDE : 0);
  // segment by segment: the segment ends come from a warp vote, so the walk
  // and its flushes are the same for every lane. A segment's FP32 sums end with
  // it, quantised: q[a] is the lane's channel at node a of its row's window; a
  // segment whose box lies one node further along x slides the window (its
  // first node is flushed, the other two go on), any other box flushes it.
  // (Sums carried on in FP32 over the window's keys were rounded at the size of
  // their total: RMS error of the node forces after 21 steps 4.4e-7 for 3.4e-7
  // on a slope, 5.8e-6 for 3.4e-7 on an SGMP beam, whose internal forces cancel;
  // they took 78 us for the mass and force transfers of the 1.2 M particle slope,
  // this 81 and 80.)
  unsigned long long* an = nullptr;  // the window's first node, and its x
  int wb = -2, wx = 0;
  bool row_in = false;
  long long q[3] = {0, 0, 0}, qm = 0;  // (mode 0: qm = the mass of node ch of the window)
  auto flush = [&](int a) {
    if (q[a] && row_in && wx + a >= 0 && wx + a < sc.NGx)
      atomicAdd(an + 4 * a + (MODE == 0 ? 1 + ch : ch), (unsigned long long)q[a]);
  };
  auto flush_mass = [&](bool mine) {
    if (qm && mine && row_in && wx + ch >= 0 && wx + ch < sc.NGx) atomicAdd(an + 4 * ch, (unsigned long long)qm);
  };
  unsigned rem = lasts;
  int j = 0;
  while (rem) {
    const int e = __ffs(rem) - 1;  // the segment's last lane
    rem &= rem - 1;
    const int nb = __shfl_sync(0xffffffffu, nbase, e), jx = __shfl_sync(0xffffffffu, c[0], e) + tlo;
    if (nb == wb + 1 && jx == wx + 1) {
      flush(0);
      if (MODE == 0) {
        flush_mass(ch == 0);
        qm = __shfl_down_sync(0xffffffffu, qm, 1);
        if (ch == nt - 1) qm = 0;
      }
      q[0] = q[1];
      q[1] = nt == 3 ? q[2] : 0;
      q[2] = 0;
      an += 4;
    } else {
      if (an) {
#pragma unroll
        for (int a = 0; a < nt; ++a) flush(a);
        if (MODE == 0) flush_mass(ch < nt);
      }
      row_in = lane < NL;
      if (!__shfl_sync(0xffffffffu, (int)inner, e)) {  // (uniform) a box at the grid's edge
        const int jy = __shfl_sync(0xffffffffu, c[1], e) + tlo + sy, jz = __shfl_sync(0xffffffffu, c[2], e) + tlo + sz;
        row_in = row_in && jy >= 0 && jy < sc.NGy && jz >= 0 && jz < sc.NGz;
      }
      q[0] = q[1] = q[2] = qm = 0;
      an = b.acc + 4 * (sc.n0 + nb + soff);
    }
    wb = nb;
    wx = jx;
    float acc[3] = {0.f, 0.f, 0.f};
    if (MODE != 2) {
      float mass = 0.f;
#pragma unroll 4
      for (; j <= e; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(xr + j * XF);
        const float f = fr[j * PF];
        acc[0] += x.x * f;
        acc[1] += x.y * f;
        if (nt == 3) acc[2] += x.z * f;
        if (MODE == 0) mass += xr[j * XF + ch] * mr[j];
      }
      if (MODE == 0) qm += quant(mass, sA);
    } else {
      float2 s[3] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 4
      for (; j <= e; ++j) {
        const float4 x = *reinterpret_cast<const float4*>(xr + j * XF);
        const float2 f = *reinterpret_cast<const float2*>(fr + j * PF);
        s[0] = fma2(make_float2(x.x, x.y), f, s[0]);
        s[1] = fma2(make_float2(x.z, x.w), f, s[1]);
        if (nt == 3) s[2] = fma2(*reinterpret_cast<const float2*>(xr + j * XF + 4), f, s[2]);
      }
#pragma unroll
      for (int a = 0; a < 3; ++a) acc[a] = s[a].x + s[a].y;
    }
#pragma unroll
    for (int a = 0; a < nt; ++a) q[a] += quant(acc[a], MODE == 0 ? sB : sA);
  }
#pragma unroll
  for (int a = 0; a < nt; ++a) flush(a);
  if (MODE == 0) flush_mass(ch < nt);
  __syncwarp();
  return dis;
}

// The SGMP form of a particle task: the key is the particle's dual cell,
// whose 8 corners are centre nodes with the SGNShape weights
// 0.125 (1 +- xi)(1 +- eta)(1 +- zeta). Phase 1 (lane = particle) writes the
// 8 corner weights -- times the mass for the momentum transfers -- and the
// transferred values; phase 2 (lane = corner and channel) walks the task's
// particles and flushes each segment's sums, quantised, into the centre
// nodes' 64-bit accumulators. A segment whose dual
// cell lies one further along x shares four corners with the one before: its
// lanes take those sums over and only the four corners left behind are flushed.
// Channels: mode 0 mass and momentum (CenterNode Mg, PXg), 1 momentum with the
// updated velocities, 2 external then internal force (Cfext, Cfint); a lane
// takes the corner lane / 4 (mode 0) or lane / 3 (modes 1, 2: one channel, or
// three force channels g, g + 3, g + 6), corners numbered x + 2 y + 4 z.
template <int MODE>
__device__ __forceinline__ int sg_part_task(BState& b, const Scene& sc, long long i0, int cnt, float sA, float sB,
                                            float* ws) {
  constexpr int ST = PartShape<MODE>::STRIDE;
  constexpr int CH0 = MODE == 2 ? CQ_FE : (MODE == 1 ? CQ_P : CQ_M);  // first accumulator channel
  const int lane = threadIdx.x & 31;
  const long long NP = b.NP, i = i0 + lane;
  int d = -1;
  if (lane < cnt) {
    if (MODE == 0) {
      const double x[3] = {b.x[i], b.x[NP + i], b.x[2 * NP + i]};
      int cc[3];
      float off[3];
      long long dual;
      locate_one(b, sc, i, x, cc, off, dual);
      d = (int)dual;
    } else {
      d = b.dual[i];
    }
  }
  const int dis = MODE == 0 ? count_disorder(d, cnt) : 0;
  const int knext = __shfl_down_sync(0xffffffffu, d, 1);
  const unsigned lasts = __ballot_sync(0xffffffffu, d >= 0 && (lane == 31 || knext != d));
  if (lasts == 0u) return dis;  // (uniform) nothing of this task on the dual grid
  int c1 = -1;  // first corner of the dual cell (sg_corner_cell)
  if (d >= 0) {
    const int dz = div_by(d, sc.mCNCxy), rm = d - dz * sc.CNCxy, dy = div_by(rm, sc.mCNCx), dx = rm - dy * sc.CNCx;
    c1 = (dz * sc.NCy + dy) * sc.NCx + dx;
  }
  // phase 1: rows 0..7 the corner weights (times the mass for modes 0, 1),
  // then the values (velocity, or the 9 force inputs)
  {
    float* col = ws + lane;
    float xx[3] = {0.f, 0.f, 0.f}, m = 0.f;
    if (d >= 0) {
#pragma unroll
      for (int a = 0; a < 3; ++a) xx[a] = b.xxn[a * NP + i];
      if (MODE != 2) m = b.m32[i];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      float w = 0.125f;
#pragma unroll
      for (int a = 0; a < 3; ++a) w *= (k >> a & 1) ? 1.f + xx[a] : 1.f - xx[a];
      col[k * ST] = d < 0 ? 0.f : (MODE == 2 ? w : w * m);
    }
    if (MODE == 2) {
#pragma unroll
      for (int c = 0; c < 9; ++c) col[(8 + c) * ST] = d < 0 ? 0.f : b.fs[(c < 3 ? 6 + c : c - 3) * NP + i];
    } else {
#pragma unroll
      for (int a = 0; a < 3; ++a) col[(8 + a) * ST] = d < 0 ? 0.f : b.v32[a * NP + i];
    }
  }
  __syncwarp();
  // phase 2
  constexpr int NPER = MODE == 0 ? 4 : 3;  // lanes per corner
  const int k = lane / NPER, g = lane - k * NPER;
  const bool active = k < 8, left = (k & 1) == 0;
  const float* wr = ws + (active ? k : 0) * ST;
  const float* vr = ws + (8 + (MODE == 0 ? (g > 0 ? g - 1 : 0) : g)) * ST;
  constexpr int NA = MODE == 2 ? 3 : 1;  // accumulators per lane
  const int koff = (k & 1) + (k >> 1 & 1) * sc.NCx + (k >> 2 & 1) * sc.NCxy;
  const int ncell = sc.NCxy * sc.NCz;
  long long q[NA];  // the lane's sums over the window's segments, quantised segment by segment
#pragma unroll
  for (int a = 0; a < NA; ++a) q[a] = 0;
  int wc = -2;  // first corner of the window
  auto flush = [&](bool mine) {
    const int cid = wc + koff;  // (corners past the last cell are dropped)
    if (!mine || !active || cid >= ncell) return;
    unsigned long long* ca = b.cacc + (CH0 + g) * b.NC + sc.c0 + cid;
#pragma unroll
    for (int a = 0; a < NA; ++a)
      if (q[a]) atomicAdd(ca + 3 * a * b.NC, (unsigned long long)q[a]);
    // every corner of a dual cell with particles takes part in the step,
    // whether or not a sum reached it (the auxiliary weights near a fixed
    // face differ from these)
    if (MODE == 0 && g == 0) b.cact[sc.c0 + cid] = 1;
  };
  unsigned rem = lasts;
  int j = 0;
  while (rem) {  // segment by segment (uniform: the segment ends come from a warp vote)
    const int e = __ffs(rem) - 1;
    rem &= rem - 1;
    const int cj = __shfl_sync(0xffffffffu, c1, e);
    if (cj == wc + 1) {
      flush(left);
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const long long r = __shfl_down_sync(0xffffffffu, q[a], NPER);
        q[a] = left ? r : 0;
      }
    } else {
      if (wc >= 0) flush(true);
#pragma unroll
      for (int a = 0; a < NA; ++a) q[a] = 0;
    }
    wc = cj;
    float acc[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) acc[a] = 0.f;
#pragma unroll 4
    for (; j <= e; ++j) {
      const float w = wr[j];
      if (MODE == 2) {
#pragma unroll
        for (int a = 0; a < 3; ++a) acc[a] += w * vr[3 * a * ST + j];
      } else if (MODE == 0) {
        acc[0] += g == 0 ? w : w * vr[j];
      } else {
        acc[0] += w * vr[j];
      }
    }
#pragma unroll
    for (int a = 0; a < NA; ++a) q[a] += quant(acc[a], MODE == 0 && g != 0 ? sB : sA);
  }
  flush(true);
  __syncwarp();
  return dis;
}

template <int MODE>
__global__ void __launch_bounds__(32 * PartShape<MODE>::WARPS, MODE == 2 ? 6 : 4) kb_part_scatter(BState b) {
  chain_entry();
  using PS = PartShape<MODE>;
  __shared__ __align__(16) float wsp[PS::WARPS][PS::WS];
  const int warp = threadIdx.x >> 5;
  const int nt = b.task0[b.nscene];
  int ds = -1, dis = 0;  // scene of the warp's last task, its particles out of order so far
  for (int t = blockIdx.x * PS::WARPS + warp; t < nt; t += gridDim.x * PS::WARPS) {
    // the scene of the task: the last scene whose first task is at or before t
    int lo = 0, hi = b.nscene - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (b.task0[mid] <= t) lo = mid;
      else hi = mid - 1;
    }
    const int s = lo;
    const Scene& sc = b.scenes[s];
    if (!scene_live(b, s) || (MODE == 1 && !sc.musl)) continue;
    const long long first = (long long)(t - b.task0[s]) * 32;
    const int cnt = (int)min(32LL, sc.np - first);
    const SceneState& st = b.sst[s];
    const float sA = q_scale(q_shift(sc, st.qmax[MODE == 0 ? Q_MASS : (MODE == 1 ? Q_MOM_MUSL : Q_FORCE)]));
    const float sB = MODE == 0 ? q_scale(q_shift(sc, st.qmax[Q_MOM])) : sA;
    float* ws = wsp[warp];
    if (MODE == 0 && s != ds) {
      if (dis && (threadIdx.x & 31) == 0) atomicAdd(&b.disorder[ds], dis);
      ds = s;
      dis = 0;
    }
    switch (sc.shape) {
      case 0: dis += part_scatter_task<MODE, 0>(b, sc, sc.p0 + first, cnt, sA, sB, ws); break;
      case 1: dis += part_scatter_task<MODE, 1>(b, sc, sc.p0 + first, cnt, sA, sB, ws); break;
      case 2: dis += part_scatter_task<MODE, 2>(b, sc, sc.p0 + first, cnt, sA, sB, ws); break;
      default: dis += sg_part_task<MODE>(b, sc, sc.p0 + first, cnt, sA, sB, ws);
    }
  }
  if (MODE == 0 && dis && (threadIdx.x & 31) == 0) atomicAdd(&b.disorder[ds], dis);
}

// Accumulated channels 0..nv-1 of node n in FP64 (the accumulators cleared
// for the next transfer). Returns false for an idle node: nothing
// accumulated and a node mass of +0, so every node field is still zero from
// the last time the node was written and nothing needs writing -- on sparse
// grids most nodes are idle. (A node that no particle reaches is never read
// by a particle, and one whose mass drops to zero is written once.) A
// massless node that received a force or a momentum (IntegrateMomentum
// integrates every node, so its momentum is F * DT) carries a mass of -0 as
// the mark that its fields are not zero, and the next transfer clears them.
__device__ __forceinline__ bool take_acc(BState& b, long long n, int nv, const double* unit, double* out) {
  ulonglong2* qa = reinterpret_cast<ulonglong2*>(b.acc + 4 * n);
  const ulonglong2 lo = qa[0], hi = qa[1];
  const unsigned long long q[4] = {lo.x, lo.y, hi.x, hi.y};
  const unsigned long long any = lo.x | lo.y | hi.x | hi.y;  // (a channel past nv is zero)
  if (any == 0ull && __double_as_longlong(b.mg[n]) == 0ll) return false;
  for (int v = 0; v < nv; ++v) out[v] = (double)(long long)q[v] * unit[v];
  if (any) qa[0] = qa[1] = make_ulonglong2(0ull, 0ull);
  return true;
}

__device__ __forceinline__ void node_finish(BState& b, const Scene& sc, long long n, int bc, int vel) {
  const long long NN = b.NN;
  if (bc) {
    uint8_t f = b.fix[n];
    for (int a = 0; a < 3; ++a)
      if (f & (1 << a)) {
        b.px[a * NN + n] = 0.0;
        b.fx[a * NN + n] = 0.0;
      }
  }
  if (vel) {
    // node velocity for the FP32 particle gathers; nodes at or below the
    // cut-off mass contribute nothing, so they hold zero
    const double m = b.mg[n];
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (m > sc.cutoff) {
      const float m32 = (float)m;
      v.x = (float)b.px[n] / m32;
      v.y = (float)b.px[NN + n] / m32;
      v.z = (float)b.px[2 * NN + n] / m32;
    }
    b.nvxy[n] = make_float2(v.x, v.y);
    b.nz[n].x = v.z;
  }
}

// Step count and time of the scenes taking the step, and which of them are
// re-sorted before the step goes on: a scene on its first step, and one whose
// mass transfer met more than kDisorder out-of-order particles per task of
// 32. Every particle out of order splits a run of equal keys in two (one more
// flush of a node box per transfer), so the order is renewed once that costs
// about as much as a sort does; results depend on the order only through FP32
// partial sums, and the decision only on the scene's own particles and order.
// Also lists the scenes to re-sort and numbers their particles and keys for the
// sort (BState::resort, shift, kshift). One block.
constexpr float kDisorder = 1.f;

__device__ __forceinline__ void step_tick(BState& b, const int* target) {
  __shared__ long long thr[512], wsum[32];
  constexpr int U = 2;  // scenes of a thread whose loads are in flight together
  int *scene = b.resort + kResortScenes, *first = scene + b.nscene;
  int any = 0;
  for (int s0 = threadIdx.x; s0 < b.nscene; s0 += U * blockDim.x) {
    SceneState t[U];
    int last[U], dis[U];
    long long np[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = s0 + u * blockDim.x;
      if (s >= b.nscene) continue;
      t[u].active = b.sst[s].active;
      t[u].istep = b.sst[s].istep;
      t[u].time = b.sst[s].time;
      t[u].dt = b.sst[s].dt;
      last[u] = target[s];
      dis[u] = b.disorder[s];
      np[u] = b.scenes[s].np;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int s = s0 + u * blockDim.x;
      if (s >= b.nscene) continue;
      int rs = 0;
      b.ract[s] = t[u].active;
      if (t[u].active) {
        SceneState& st = b.sst[s];
        const int istep = t[u].istep + 1;
        const double time = t[u].time + t[u].dt;
        st.istep = istep;
        st.time = time;
        st.ftime = (float)time;
        if (istep == last[u]) atomicAdd(&b.ctl->finished, 1);  // the scene's last step
        rs = istep == 1 || (float)dis[u] > kDisorder * (float)((np[u] + 31) / 32);
      }
      b.shift[s] = rs;  // (read below by the thread of the scene's strip)
      any |= rs;
    }
  }
  any = __syncthreads_or(any);
  if (!any) {
    if (threadIdx.x == 0) b.resort[0] = 0;
    return;
  }
  // a strip of scenes per thread: how many of them are marked and their chunks,
  // particles and keys, two sums to a 64-bit value
  const int strip = (b.nscene + blockDim.x - 1) / blockDim.x;
  const int s0 = min((int)threadIdx.x * strip, b.nscene), s1 = min(s0 + strip, b.nscene);
  auto sizes = [&](int s, long long& nc, long long& pk) {
    const Scene& sc = b.scenes[s];
    nc = (1LL << 32) + (sc.np + kSortThreads - 1) / kSortThreads;
    pk = (sc.np << 32) + sc.nk;
  };
  long long nc = 0, pk = 0;
  for (int s = s0; s < s1; ++s)
    if (b.shift[s]) {
      long long c, p;
      sizes(s, c, p);
      nc += c;
      pk += p;
    }
  nc = block_scan<long long, ScanSum>(nc, thr, wsum);
  const long long tnc = thr[blockDim.x - 1];
  __syncthreads();
  pk = block_scan<long long, ScanSum>(pk, thr, wsum);
  const long long tpk = thr[blockDim.x - 1];
  for (int s = s0; s < s1; s += U) {
    long long c[U], p[U], p0[U], k0[U];
    int rs[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      rs[u] = s + u < s1 ? b.shift[s + u] : 0;
      if (!rs[u]) continue;
      sizes(s + u, c[u], p[u]);
      p0[u] = b.scenes[s + u].p0;
      k0[u] = b.scenes[s + u].k0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (!rs[u]) continue;
      const int at = (int)(nc >> 32);
      scene[at] = s + u;
      first[at] = (int)(nc & 0xffffffff);
      b.shift[s + u] = (int)(p0[u] - (pk >> 32));
      b.kshift[s + u] = (int)(k0[u] - (pk & 0xffffffff));
      nc += c[u];
      pk += p[u];
    }
  }
  if (threadIdx.x == 0) {
    const int n = (int)(tnc >> 32);
    b.resort[0] = n;
    b.resort[1] = (int)(tpk & 0xffffffff);
    first[n] = (int)(tnc & 0xffffffff);
  }
}

// the cells next to grid node j that take part in the step (bit dx + 2 dy + 4 dz
// for the cell j - 1 + (dx, dy, dz)), and the flat index of such a cell
__device__ __forceinline__ long long sg_near_cell(const Scene& sc, const int j[3], int k) {
  const int cx = j[0] - 1 + (k & 1), cy = j[1] - 1 + (k >> 1 & 1), cz = j[2] - 1 + (k >> 2);
  return sc.c0 + (cz * sc.NCy + cy) * sc.NCx + cx;
}
__device__ __forceinline__ unsigned sg_active_cells(const BState& b, const Scene& sc, const int j[3]) {
  unsigned m = 0u;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int cx = j[0] - 1 + (k & 1), cy = j[1] - 1 + (k >> 1 & 1), cz = j[2] - 1 + (k >> 2);
    if (cx >= 0 && cx < sc.NCx && cy >= 0 && cy < sc.NCy && cz >= 0 && cz < sc.NCz)
      m |= (unsigned)b.cact[sg_near_cell(sc, j, k)] << k;
  }
  return m;
}

// SG: the nodes of the SGMP scenes (an instantiation of its own: the 8 cells' loads
// in flight take registers that the others would pay for); the nodes n0 .. n1 - 1
// are all of that family; tick: the last block starts the step
template <bool SG>
__global__ void kb_p2g_mass(BState b, long long n0, long long n1, int bc_usf, int vel_usf, const int* target, int tick) {
  chain_entry();
  if (tick && blockIdx.x == gridDim.x - 1) {  // the last block starts the step instead of finishing nodes
    step_tick(b, target);
    return;
  }
  const long long n = n0 + btid();
  bool act = false;
  int s = -1;
  if (n < n1) {
    s = scene_of(b, b.node_scene, n);
    if (scene_live(b, s)) {
      const Scene& sc = b.scenes[s];
      const long long NN = b.NN;
      double M = 0, P0 = 0, P1 = 0, P2 = 0;
      bool live = true;
      if (SG) {
        int j[3];
        node_xyz(sc, n - sc.n0, j[0], j[1], j[2]);
        // centre nodes -> node (GridMomentumInitial of SGMP): 1/8 of the
        // adjacent cells' mass and momentum, cells at or below the cut-off
        // mass left out; the cells' fixed-point sums are added exactly
        const unsigned near = sg_active_cells(b, sc, j);
        live = near || __double_as_longlong(b.mg[n]) != 0ll;  // (else idle, as in take_acc)
        const SceneState& st = b.sst[s];
        const int shm = q_shift(sc, st.qmax[Q_MASS]);
        const double um = q_unit(shm), up = q_unit(q_shift(sc, st.qmax[Q_MOM]));
        // cm = q * um > cutoff  <=>  q > floor(cutoff / um) (um a power of two)
        const double thr = ldexp(sc.cutoff, shm);
        const long long qcut = thr >= 9.0e18 ? LLONG_MAX : (long long)floor(thr);
        long long QM = 0, Q0 = 0, Q1 = 0, Q2 = 0;
        const long long* ca = reinterpret_cast<const long long*>(b.cacc);
#pragma unroll
        for (int k0 = 0; k0 < 8; k0 += 4) {  // (four cells' loads in flight at a time)
          long long q[4][4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const bool on = near >> (k0 + k) & 1u;
            const long long c = sg_near_cell(sc, j, k0 + k);
#pragma unroll
            for (int a = 0; a < 4; ++a) q[k][a] = on ? ca[(CQ_M + a) * b.NC + c] : 0;
          }
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (q[k][0] <= qcut) continue;
            QM += q[k][0];
            Q0 += q[k][1];
            Q1 += q[k][2];
            Q2 += q[k][3];
          }
        }
        M = 0.125 * ((double)QM * um);
        P0 = 0.125 * ((double)Q0 * up);
        P1 = 0.125 * ((double)Q1 * up);
        P2 = 0.125 * ((double)Q2 * up);
      } else {
        const SceneState& st = b.sst[s];
        const double up = q_unit(q_shift(sc, st.qmax[Q_MOM]));
        const double unit[4] = {q_unit(q_shift(sc, st.qmax[Q_MASS])), up, up, up};
        double o[4];
        live = take_acc(b, n, 4, unit, o);
        M = o[0];
        P0 = o[1];
        P1 = o[2];
        P2 = o[3];
      }
      if (live) {
        b.mg[n] = M;
        b.px[n] = P0;
        b.px[NN + n] = P1;
        b.px[2 * NN + n] = P2;
        act = M > 0.0;
        node_finish(b, sc, n, bc_usf && sc.usf, vel_usf && sc.usf);
        if (!(M != 0.0)) {
          // the node goes idle: clear the rest of its fields once (the idle
          // test of the later transfers skips it from now on)
          for (int a = 0; a < 3; ++a) b.fx[a * NN + n] = 0.0;
          b.nvxy[n] = b.nz[n] = b.naxy[n] = make_float2(0.f, 0.f);
          // a momentum without mass (the mass contributions quantised to
          // zero, the momentum ones not) keeps the node marked (take_acc)
          if (b.px[n] != 0.0 || b.px[NN + n] != 0.0 || b.px[2 * NN + n] != 0.0) b.mg[n] = -0.0;
        }
      }
    }
  }
  // per-scene active-node count, combined per block (one atomic per scene
  // and block in the common case)
  __shared__ int ws[32];
  __shared__ unsigned wc[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const unsigned grp = __match_any_sync(0xffffffffu, s);
  const unsigned actg = __ballot_sync(0xffffffffu, act) & grp;
  const bool uniform = grp == 0xffffffffu;
  if (!uniform && s >= 0 && actg && lane == __ffs(grp) - 1)
    atomicAdd(&b.sst[s].active_nodes, (unsigned long long)__popc(actg));
  if (lane == 0) {
    ws[warp] = uniform ? s : -1;
    wc[warp] = uniform ? (unsigned)__popc(actg) : 0u;
  }
  __syncthreads();
  if (warp == 0) {
    const int s2 = lane < nw ? ws[lane] : -1;
    const unsigned g2 = __match_any_sync(0xffffffffu, s2);
    const unsigned c2 = __reduce_add_sync(g2, lane < nw ? wc[lane] : 0u);
    if (s2 >= 0 && c2 && lane == __ffs(g2) - 1) atomicAdd(&b.sst[s2].active_nodes, (unsigned long long)c2);
  }
}

// -------------------------------------------------------------- stress
// ParticleStressUpdate + Constitution for one particle (FP32). The stress pass
// runs twice per step: before the force transfer for USF scenes (usf_pass 1)
// and after the position update for USL / MUSL scenes (usf_pass 0).
// MT != 0: the particles of material type MT (an instantiation for each of
// the common types, fewer registers); MT = 0: every other type
__host__ __device__ constexpr bool stress_specialised(int mat_type) {
  return mat_type == 1 || mat_type == 9 || mat_type == 10 || mat_type == 11;
}

// (the common types capped at 64 registers: four 256-thread blocks per SM)
__device__ __forceinline__ float force_stage(BState& b, const Scene& sc, const SceneState& st, long long i, float vol,
                                             float smq, const float (&sd)[6]);

// stages the particle's force input when its scene's USF pass has its final
// stress here (no Johnson-Cook tail after this kernel) and returns that
// contribution's bound; -1 otherwise. UV: the instantiation for scenes that
// update volumes by Fp (1) or not (0) -- without the Fp state's registers
// when not; uvf: the batch holds both kinds, so each launch takes its own.
template <int MT, int UV>
__device__ __forceinline__ float stress_one(BState& b, long long i, int usf_pass, int filter, int uvf) {
  using P = PMixed;
  using R = float;
  const int s = b.scene[i];
  if (!scene_live(b, s)) return -1.f;
  const Scene& sc = b.scenes[s];
  if (sc.usf != usf_pass || (uvf && sc.uvfp != UV)) return -1.f;
  const DevMaterialF& mt = b.fmats[b.bodies[b.body[i]].mat];
  // every particle goes through the instantiation of its own material type
  // (or the general one), whatever else shares the batch: the compiled FP32
  // arithmetic, and so the result, is the same alone or in a batch (filter
  // 0: the batch needs this instantiation only)
  if (filter && (MT ? mt.mat_type != MT : stress_specialised(mt.mat_type))) return -1.f;
  const long long NP = b.NP;
  const long long o = sc.p0 + b.orig[i];  // position in the reference processing order
  if (sc.has_jc) {
    b.setter[o] = -1;
    b.deferred[i] = 0;
  }
  R de[6] = {0, 0, 0, 0, 0, 0}, vort[3] = {0, 0, 0}, deFp[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  if (sc.shape == 3) {
    int d = b.dual[i];
    if (d < 0) return -1.f;
    int dz = div_by(d, sc.mCNCxy), rem = d - dz * sc.CNCxy, dy = div_by(rem, sc.mCNCx), dx = rem - dy * sc.CNCx;
    float xx[3] = {b.xxn[i], b.xxn[NP + i], b.xxn[2 * NP + i]};
    for (int k = 0; k < 8; ++k) {
      int oc[3] = {kCorner[k][0], kCorner[k][1], kCorner[k][2]};
      const long long cid = sg_corner_cell(sc, dx, dy, dz, k);
      if (cid < 0) continue;
      const long long c = sc.c0 + cid;
      float w = 0.125f;
      for (int a = 0; a < 3; ++a) w *= oc[a] ? 1.f + xx[a] : 1.f - xx[a];
      for (int a = 0; a < 3; ++a) {
        const float4 r = b.cgrad[a * b.NC + c];
        deFp[a][0] += w * r.x;
        deFp[a][1] += w * r.y;
        deFp[a][2] += w * r.z;
      }
    }
  } else {
    const int cl = b.cell[i];
    if (cl < 0) return -1.f;
    int c[3];
    c[2] = div_by(cl, sc.mNCxy);
    int rem = cl - c[2] * sc.NCxy;
    c[1] = div_by(rem, sc.mNCx);
    c[0] = rem - c[1] * sc.NCx;
    float off[3] = {b.off[i], b.off[NP + i], b.off[2 * NP + i]};
    int t0[3], nt[3];
    float wd[3][3], dd[3][3];
    for (int a = 0; a < 3; ++a) nt[a] = dim_nodes(sc.shape, off[a], t0[a], wd[a], dd[a]);
    // velocity gradient L[a][k] = sum_n v_a(n) dN_n / dx_k; the shape is a
    // tensor product, so the node velocities are first summed along x with
    // the x weights and x derivatives, and each (y, z) row then adds its two
    // sums times the y-z factors: 6 multiply-adds per node instead of the 24
    // of forming de, vort and deFp node by node
    float L[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    const NodeBox box = node_box(sc, c, t0, nt);
#pragma unroll
    for (int az = 0; az < 3; ++az)
#pragma unroll
      for (int ay = 0; ay < 3; ++ay) {
        if (!box.row(ay, az)) continue;
        const int o = az * box.sz + ay * box.sy;
        const float2 *rv = b.nvxy + box.first + o, *rz = b.nz + box.first + o;
        float S[3] = {0, 0, 0}, D[3] = {0, 0, 0};
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
          if (!box.x(ax)) continue;
          const float2 vn = rv[ax];  // zero below the cut-off mass
          const float vz = rz[ax].x;
          S[0] += wd[0][ax] * vn.x;
          S[1] += wd[0][ax] * vn.y;
          S[2] += wd[0][ax] * vz;
          D[0] += dd[0][ax] * vn.x;
          D[1] += dd[0][ax] * vn.y;
          D[2] += dd[0][ax] * vz;
        }
        const float fx = wd[1][ay] * wd[2][az], fy = dd[1][ay] * wd[2][az], fz = wd[1][ay] * dd[2][az];
        for (int a = 0; a < 3; ++a) {
          L[a][0] += D[a] * fx;
          L[a][1] += S[a] * fy;
          L[a][2] += S[a] * fz;
        }
      }
    const float idc = sc.fidcell;
    for (int a = 0; a < 3; ++a)
      for (int k = 0; k < 3; ++k) deFp[a][k] = L[a][k] * idc;
  }
  de[0] = deFp[0][0];
  de[1] = deFp[1][1];
  de[2] = deFp[2][2];
  de[3] = deFp[2][1] + deFp[1][2];
  de[4] = deFp[0][2] + deFp[2][0];
  de[5] = deFp[1][0] + deFp[0][1];
  vort[0] = deFp[2][1] - deFp[1][2];
  vort[1] = deFp[0][2] - deFp[2][0];
  vort[2] = deFp[1][0] - deFp[0][1];
  const SceneState& st = b.sst[s];
  const R DT = st.fdt;
  for (int a = 0; a < 6; ++a) de[a] *= DT;
  for (int a = 0; a < 3; ++a) vort[a] = vort[a] * DT / 2.f;
  for (int a = 0; a < 3; ++a)
    for (int k = 0; k < 3; ++k) deFp[a][k] *= DT;
  R Fpn[3][3], Fpn_lo[3][3];
  if (UV) {
    // Fp(n+1) = (I + dF) Fp(n), i.e. H += dF + dF H for H = Fp - I, with H
    // carried as a pair hi + lo of FP32 values: the increment in FP32 from
    // the rounded H, added to the pair without rounding error (TwoSum), so
    // that H keeps the precision of the increments instead of losing an
    // FP32 rounding of its whole size every step (a rotated body has |H|
    // far above its strain)
    R F0[3][3], L0[3][3];
    for (int a = 0; a < 9; ++a) {
      F0[a / 3][a % 3] = b.fp[a * NP + i];
      L0[a / 3][a % 3] = b.fp[(9 + a) * NP + i];
    }
    for (int a = 0; a < 3; ++a)
      for (int k = 0; k < 3; ++k) {
        const R inc = deFp[a][k] + (deFp[a][0] * F0[0][k] + deFp[a][1] * F0[1][k] + deFp[a][2] * F0[2][k]);
        const F2 t = two_sum(F0[a][k], inc);
        const F2 h = two_sum(t.hi, t.lo + L0[a][k]);
        Fpn[a][k] = h.hi;
        Fpn_lo[a][k] = h.lo;
        b.fp[(a * 3 + k) * NP + i] = h.hi;
        b.fp[(9 + a * 3 + k) * NP + i] = h.lo;
      }
  }
  PState<R> ps;
  ps.vol = b.vol[i];
  ps.epeff = b.epeff[i];
  ps.sig_y = b.sig_y[i];
  ps.seqv = b.seqv[i];
  ps.lt = b.lt[i];
  ps.celsius = b.celsius[i];
  ps.ie = (R)b.ie[i];
  ps.mass = b.m32[i];
  ps.dmg = b.dmg[i];
  ps.cp = b.cp[i];
  ps.sm = b.sm[i];
  ps.q = b.q[i];
  for (int a = 0; a < 6; ++a) ps.sd[a] = b.sd[a * NP + i];
  ps.failure = b.failure[i] != 0;
  ps.evol = b.evol[i];
  CResult<R> res;
  constitution<P, MT>(ps, mt, de, vort, deFp, Fpn, UV != 0, DT, st.time, sc.fdcell, sc.fbq1, sc.fbq2, res,
                      UV ? Fpn_lo : nullptr);
  if (res.negative_volume) atomicOr(&b.sst[s].status, (unsigned)ST_NEGATIVE_VOLUME);
  if (!res.eos_ok) atomicOr(&b.sst[s].status, (unsigned)ST_BAD_EOS);
  if (sc.has_jc) {
    if (res.dep_set) {
      b.setter[o] = (int)o;
      b.dep[o] = (double)res.depeff;
    }
    b.deferred[i] = res.defer ? (uint8_t)res.tail : 0;
    if (res.defer && res.tail == 7) {
      b.jc_aux[i] = res.vold;
      b.jc_aux[NP + i] = res.ieinc;
      b.jc_aux[2 * NP + i] = res.dvol;
      b.jc_aux[3 * NP + i] = res.smold;
      b.jc_aux[4 * NP + i] = res.vol_;
    }
  }
  b.vol[i] = ps.vol;
  b.evol[i] = ps.evol;
  b.sm[i] = ps.sm;
  b.seqv[i] = ps.seqv;
  for (int a = 0; a < 6; ++a) b.sd[a * NP + i] = ps.sd[a];
  b.ie[i] = (double)ps.ie;
  b.q[i] = ps.q;
  // (the specialised types leave these as they were: neither read nor written
  // for them. Stress update of the 4.1 M particle column 255 -> 246 us, dam break
  // 2 M 117 -> 113; no type changes cp)
  if (!stress_specialised(MT)) {
    b.sig_y[i] = ps.sig_y;
    b.celsius[i] = ps.celsius;
    b.failure[i] = ps.failure ? 1 : 0;
  }
  if (!stress_specialised(MT) || MT == 10) b.epeff[i] = ps.epeff;
  if (!isfinite(ps.sm) || !isfinite(ps.ie)) atomicOr(&b.sst[s].status, (unsigned)ST_NONFINITE);
  // GridMomentumUpdate follows a USF stress update directly: stage its
  // force input from the registers (the stress state is final unless a
  // Johnson-Cook tail still runs)
  if (!sc.usf || sc.has_jc) return -1.f;
  return force_stage(b, sc, st, i, ps.vol, ps.sm - ps.q, ps.sd);
}

// (Drucker-Prager and the null material run better at 1536 threads per SM -- 40
// registers, some spilled -- than at 1024 with few or none: the 1.2 M particle
// slope 85 us for 91, the 2 M dam break 124 for 136; the other specialised
// models at 1024: elastic block 36 k 11.6 us for 12.4, neo-Hookean beam 94 k
// 17.4 for 21.4. The null material with the deformation gradient spills too
// much at 40: dam break 208 us for 159, 27 k particles 15.2 for 13.3)
template <int MT, int UV>
__global__ void __launch_bounds__(512, MT == 10 || (MT == 9 && !UV) ? 3 : (MT ? 2 : 1))
    kb_stress(BState b, int usf_pass, int filter, int uvf) {
  chain_entry();
  const long long i = btid();
  float bound = -1.f;
  if (i < b.NP) bound = stress_one<MT, UV>(b, i, usf_pass, filter, uvf);
  if (usf_pass) block_scene_max<1>(b, bound >= 0.f ? (int)b.scene[i] : -1, {Q_FORCE}, {fmaxf(bound, 0.f)});
}

// Johnson-Cook tails waiting for the depeff carried from the previous particle
// in the reference order (scene-local input order)
__global__ void kb_depeff_apply(BState b, int usf_pass) {
  chain_entry();
  using P = PMixed;
  using R = float;
  long long i = btid();
  if (i >= b.NP) return;
  const int s = scene_of(b, b.scene, i);
  const Scene& sc = b.scenes[s];
  if (!sc.has_jc || !scene_live(b, s) || sc.usf != usf_pass) return;
  const int tail = b.deferred[i];
  if (tail == 0) return;
  const long long NP = b.NP;
  const long long o = sc.p0 + b.orig[i];
  int last = b.setter_scan[o];
  R D = (R)(last >= sc.p0 && last <= o ? b.dep[last] : b.sst[s].depeff_carry);
  const DevMaterial& mt = b.mats[b.bodies[b.body[i]].mat];
  if (tail == 4) {
    R den_ = (R)b.mass[i] / b.vol[i];
    b.celsius[i] = b.celsius[i] + b.seqv[i] * D / den_ / (R)mt.specheat;
    return;
  }
  Mm<R> m;
  m.epeff_ = b.epeff[i];
  m.sm = b.sm[i];
  m.bqf = b.q[i];
  m.iener = (R)b.ie[i];
  m.seqv = b.seqv[i];
  m.sd[0] = b.sd[i];
  m.sd[1] = b.sd[NP + i];
  m.sd[2] = b.sd[2 * NP + i];
  m.sd[3] = b.sd[4 * NP + i];
  m.sd[4] = b.sd[5 * NP + i];
  m.sd[5] = b.sd[3 * NP + i];
  m.vold = (R)b.jc_aux[i];
  m.ieinc = (R)b.jc_aux[NP + i];
  m.dvol = (R)b.jc_aux[2 * NP + i];
  m.smold = (R)b.jc_aux[3 * NP + i];
  m.vol_ = (R)b.jc_aux[4 * NP + i];
  m.DMG = b.dmg[i];
  m.oldDMG = m.DMG;
  bool failure = b.failure[i] != 0;
  R vol_store = m.vol_;
  jc7_tail<P>(m, mt, failure, D, vol_store);
  R den_ = (R)b.mass[i] / m.vol_;
  b.celsius[i] = b.celsius[i] + m.seqv * D / den_ / (R)mt.specheat;
  b.vol[i] = vol_store;
  b.sm[i] = m.sm;
  b.q[i] = m.bqf;
  b.ie[i] = (double)m.iener;
  b.epeff[i] = m.epeff_;
  b.sd[i] = m.sd[0];
  b.sd[NP + i] = m.sd[1];
  b.sd[2 * NP + i] = m.sd[2];
  b.sd[4 * NP + i] = m.sd[3];
  b.sd[5 * NP + i] = m.sd[4];
  b.sd[3 * NP + i] = m.sd[5];
  b.failure[i] = failure ? 1 : 0;
}

__global__ void kb_depeff_carry(BState b, int usf_pass) {
  chain_entry();
  int s = (int)btid();
  if (s >= b.nscene) return;
  const Scene& sc = b.scenes[s];
  if (!sc.has_jc || !scene_live(b, s) || sc.np == 0 || sc.usf != usf_pass) return;
  int last = b.setter_scan[sc.p0 + sc.np - 1];
  if (last >= sc.p0 && last < sc.p0 + sc.np) b.sst[s].depeff_carry = b.dep[last];
}

// ------------------------------------------------------------ force input
// external force (QuLo ramp, Damp, gravity; update_step.f90:889-903) and
// sigma * vol, staged per particle in FP32 for the force gather, from the
// particle's volume, SM - q and SD; returns the bound of one contribution
__device__ __forceinline__ float force_stage(BState& b, const Scene& sc, const SceneState& st, long long i, float vol,
                                             float smq, const float (&sd)[6]) {
  const long long NP = b.NP;
  // external force in FP32 (the staged force is FP32): load ramp, mass
  // damping, gravity
  float f[3];
  const float m = b.m32[i];
  if (sc.has_fxp) {
    const float ramp = (sc.qload && !(st.time >= sc.qload_time)) ? (float)(st.time / sc.qload_time) : 1.f;
    for (int a = 0; a < 3; ++a) f[a] = (float)b.fxp[a * NP + i] * ramp;
  } else {
    f[0] = f[1] = f[2] = 0.f;
  }
  if (sc.qdamp)
    for (int a = 0; a < 3; ++a) f[a] = f[a] - sc.fdamp * m * b.v32[a * NP + i];
  if (sc.gravity) {
    const DevBody& bd = b.bodies[b.body[i]];
    for (int a = 0; a < 3; ++a) f[a] = f[a] + m * bd.fgravp[a];
  }
  float fs[6];
  for (int a = 0; a < 3; ++a) fs[a] = (smq + sd[a]) * vol;
  for (int a = 3; a < 6; ++a) fs[a] = sd[a] * vol;
  for (int a = 0; a < 6; ++a) b.fs[a * NP + i] = fs[a];
  for (int a = 0; a < 3; ++a) b.fs[(6 + a) * NP + i] = f[a];
  // bound of one contribution: node force (|grad N| <= 1 / h per component,
  // N <= 1), or for SGMP one centre-node channel (N times a staged value)
  const float sig = fabsf(fs[0]) + fabsf(fs[1]) + fabsf(fs[2]) + 2.f * (fabsf(fs[3]) + fabsf(fs[4]) + fabsf(fs[5]));
  const float gscale = sc.shape == 3 ? 1.f : sc.fidcell;
  return (sig * gscale + fabsf(f[0]) + fabsf(f[1]) + fabsf(f[2])) * 1.0001f;
}

// the staging of the particles whose stress kernel did not stage them (scenes
// updating stresses after the position update, and Johnson-Cook scenes, whose
// tails run after the stress kernel)
__device__ __forceinline__ float force_prep_one(BState& b, long long i) {
  const int s = scene_of(b, b.scene, i);
  if (!scene_live(b, s)) return -1.f;
  const Scene& sc = b.scenes[s];
  if (sc.usf && !sc.has_jc) return -1.f;
  const long long NP = b.NP;
  // (every value loaded before the first store, which could alias them)
  const float vol = b.vol[i];
  const float smq = b.sm[i] - b.q[i];
  float sd[6];
  for (int a = 0; a < 6; ++a) sd[a] = b.sd[a * NP + i];
  return force_stage(b, sc, b.sst[s], i, vol, smq, sd);
}

__global__ void kb_force_prep(BState b) {
  chain_entry();
  const long long i = btid();
  float bound = -1.f;
  if (i < b.NP) bound = force_prep_one(b, i);
  block_scene_max<1>(b, bound >= 0.f ? scene_of(b, b.scene, i) : -1, {Q_FORCE}, {fmaxf(bound, 0.f)});
}

// GridMomentumUpdate + IntegrateMomentum for one node
__device__ __forceinline__ void node_integrate(BState& b, const Scene& sc, int s, long long n, const double f[3]) {
  const long long NN = b.NN;
  const SceneState& st = b.sst[s];
  const double dt = st.dt;
  for (int a = 0; a < 3; ++a) {
    b.fx[a * NN + n] = f[a];
    double p = b.px[a * NN + n];
    p = st.istep == 1 ? p + f[a] * dt * 0.5 : p + f[a] * dt;
    b.px[a * NN + n] = p;
  }
  node_finish(b, sc, n, 1, 1);
  const double m = b.mg[n];
  if (m == 0.0) b.mg[n] = -0.0;  // fields not zero at a massless node (take_acc)
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (m > sc.cutoff) {
    const float m32 = (float)m;
    acc.x = (float)b.fx[n] / m32;
    acc.y = (float)b.fx[NN + n] / m32;
    acc.z = (float)b.fx[2 * NN + n] / m32;
  }
  b.naxy[n] = make_float2(acc.x, acc.y);
  b.nz[n].y = acc.z;
}

// (the SGMP form keeps two cells' nine loads in flight at 64 registers)
template <bool SG>
__global__ void __launch_bounds__(512, SG ? 2 : 1) kb_p2g_force(BState b, long long n0, long long n1) {
  chain_entry();
  const long long n = n0 + btid();
  if (n >= n1) return;
  const int s = SG ? (int)b.node_scene[n] : scene_of(b, b.node_scene, n);
  if (!scene_live(b, s)) return;
  const Scene& sc = b.scenes[s];
  double F[3] = {0, 0, 0};
  if (SG) {
    int j[3];
    node_xyz(sc, n - sc.n0, j[0], j[1], j[2]);
    // centre nodes -> node (GridMomentumUpdate of SGMP): 1/8 of the cells'
    // external force minus Cfint . dN, dN = +-1 / (4 Jacobi) per direction
    // by the node's side of the cell; the cells' fixed-point sums are
    // combined exactly, then scaled once
    const unsigned near = sg_active_cells(b, sc, j);
    if (!near && __double_as_longlong(b.mg[n]) == 0ll) return;  // idle node (as in take_acc)
    long long E[3] = {0, 0, 0}, T[3] = {0, 0, 0};
    const long long* ca = reinterpret_cast<const long long*>(b.cacc) + CQ_FE * b.NC;
#pragma unroll
    for (int k0 = 0; k0 < 8; k0 += 2) {  // (two cells' loads in flight at a time)
      long long q[2][9];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const bool on = near >> (k0 + u) & 1u;
        const long long c = sg_near_cell(sc, j, k0 + u);
#pragma unroll
        for (int a = 0; a < 9; ++a) q[u][a] = on ? ca[a * b.NC + c] : 0;
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int k = k0 + u;
        const long long* I = q[u] + 3;
        for (int a = 0; a < 3; ++a) E[a] += q[u][a];
        // signed by the node's side: +dN at the upper corner of the cell
        const bool ux = !(k & 1), uy = !(k & 2), uz = !(k & 4);
        const long long xx = ux ? I[0] : -I[0], xy_x = ux ? I[3] : -I[3], xz_x = ux ? I[5] : -I[5];
        const long long xy_y = uy ? I[3] : -I[3], yy = uy ? I[1] : -I[1], yz_y = uy ? I[4] : -I[4];
        const long long xz_z = uz ? I[5] : -I[5], yz_z = uz ? I[4] : -I[4], zz = uz ? I[2] : -I[2];
        T[0] += xx + xy_y + xz_z;
        T[1] += xy_x + yy + yz_z;
        T[2] += xz_x + yz_y + zz;
      }
    }
    const double u = q_unit(q_shift(sc, b.sst[s].qmax[Q_FORCE]));
    for (int a = 0; a < 3; ++a) F[a] = (0.125 * (double)E[a] - sc.iJacobi4 * (double)T[a]) * u;
  } else {
    const double u = q_unit(q_shift(sc, b.sst[s].qmax[Q_FORCE]));
    const double unit[3] = {u, u, u};
    if (!take_acc(b, n, 3, unit, F)) return;  // idle node
  }
  node_integrate(b, sc, s, n, F);
}

// SGMP: velocity gradient at the centre nodes from the 8 cell nodes (the strain
// rate and spin of the particles are its symmetric and antisymmetric parts)
__global__ void kb_sg_centre_gradient(BState b, int usf_pass) {
  chain_entry();
  long long c = btid();
  if (c >= b.NC) return;
  int s = scene_of(b, b.cscene, c);
  if (!scene_live(b, s)) return;
  const Scene& sc = b.scenes[s];
  if (sc.usf != usf_pass || !b.cact[c]) return;
  const long long NC = b.NC;
  long long lc = c - sc.c0;
  int q[3];
  q[2] = div_by(lc, sc.mNCxy);
  int rem = (int)(lc - (long long)q[2] * sc.NCxy);
  q[1] = div_by(rem, sc.mNCx);
  q[0] = rem - q[1] * sc.NCx;
  float cf[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  const float j4 = sc.fiJacobi4;
  for (int k = 0; k < 8; ++k) {
    long long n = sc.n0 + ((long long)(q[2] + kCorner[k][2]) * sc.NGy + q[1] + kCorner[k][1]) * sc.NGx + q[0] +
                  kCorner[k][0];
    const float2 vxy = b.nvxy[n];  // zero below the cut-off mass
    const float3 v4 = make_float3(vxy.x, vxy.y, b.nz[n].x);
    const float v[3] = {v4.x, v4.y, v4.z};
    const float dx = kSN[0][k] * j4, dy = kSN[1][k] * j4, dz = kSN[2][k] * j4;
    for (int a = 0; a < 3; ++a) {
      cf[a][0] += dx * v[a];
      cf[a][1] += dy * v[a];
      cf[a][2] += dz * v[a];
    }
  }
  for (int a = 0; a < 3; ++a) b.cgrad[a * NC + c] = make_float4(cf[a][0], cf[a][1], cf[a][2], 0.f);
}

// SGMP: centre-node velocity / acceleration (BoundaryAuxiliaryNodeUpdate on
// the fixed / symmetric faces)
__global__ void kb_sg_centre_velocity(BState b) {
  chain_entry();
  long long c = btid();
  if (c >= b.NC) return;
  int s = scene_of(b, b.cscene, c);
  if (!scene_live(b, s)) return;
  if (!b.cact[c]) return;
  const Scene& sc = b.scenes[s];
  long long lc = c - sc.c0;
  int q[3];
  q[2] = div_by(lc, sc.mNCxy);
  int rem = (int)(lc - (long long)q[2] * sc.NCxy);
  q[1] = div_by(rem, sc.mNCx);
  q[0] = rem - q[1] * sc.NCx;
  const int NCd[3] = {sc.NCx, sc.NCy, sc.NCz};
  bool boundary = false;
  for (int a = 0; a < 3; ++a)
    if (NCd[a] > 1 && ((q[a] == 0 && sc.fixs[2 * a] != 0) || (q[a] == NCd[a] - 1 && sc.fixs[2 * a + 1] != 0)))
      boundary = true;
  double cxx[3] = {0, 0, 0};
  if (boundary)
    for (int a = 0; a < 3; ++a)
      if (NCd[a] > 1) cxx[a] = q[a] == NCd[a] - 1 ? -1.0 : (q[a] == 0 ? 1.0 : 0.0);
  float v[3] = {0, 0, 0}, acc[3] = {0, 0, 0};
  for (int k = 0; k < 8; ++k) {
    long long n = sc.n0 + ((long long)(q[2] + kCorner[k][2]) * sc.NGy + q[1] + kCorner[k][1]) * sc.NGx + q[0] +
                  kCorner[k][0];
    float w = 0.125f;
    if (boundary)
      w = ((float)kSN[0][k] * (float)cxx[0] + 1.f) * ((float)kSN[1][k] * (float)cxx[1] + 1.f) *
          ((float)kSN[2][k] * (float)cxx[2] + 1.f) * 0.125f;
    const float2 vxy = b.nvxy[n], axy = b.naxy[n], z = b.nz[n];  // zero below the cut-off mass
    const float3 vn = make_float3(vxy.x, vxy.y, z.x), an = make_float3(axy.x, axy.y, z.y);
    v[0] += w * vn.x;
    v[1] += w * vn.y;
    v[2] += w * vn.z;
    acc[0] += w * an.x;
    acc[1] += w * an.y;
    acc[2] += w * an.z;
  }
  b.cvel[c] = make_float4(v[0], v[1], v[2], 0.f);
  b.cacl[c] = make_float4(acc[0], acc[1], acc[2], 0.f);
  // the force sums are consumed (and so are the momentum sums when the
  // MUSL transfer refills them): cleared for the next scatter
  for (int a = sc.musl ? CQ_P : CQ_FE; a < CQ_N; ++a) b.cacc[a * b.NC + c] = 0ull;
}

// SGMP: clears the mass and momentum sums of the live scenes' centre nodes
// before the step's first transfer (they stay readable between steps) and the
// marks of the cells that took part in the last step. Only marked cells are
// touched here, by the node kernels and by the centre kernels: a beam's grid
// is five sixths empty.
__global__ void kb_sg_clear(BState b) {
  chain_entry();
  const long long c = btid();
  if (c >= b.NC) return;
  if (!scene_live(b, scene_of(b, b.cscene, c)) || !b.cact[c]) return;
  b.cact[c] = 0;
  for (int a = CQ_M; a < CQ_FE; ++a) b.cacc[a * b.NC + c] = 0ull;
}

// ---------------------------------------------------------- G2P position
__device__ __forceinline__ float position_one(BState& b, long long i) {
  const int s = scene_of(b, b.scene, i);
  if (!scene_live(b, s)) return -1.f;
  const Scene& sc = b.scenes[s];
  const SceneState& st = b.sst[s];
  const long long NP = b.NP;
  // the particle's FP64 position and velocity, loaded before the node
  // gathers so that their latency overlaps the gathers'
  double x0[3], v0[3];
  for (int a = 0; a < 3; ++a) {
    x0[a] = b.x[a * NP + i];
    v0[a] = b.v[a * NP + i];
  }
  float v[3] = {0, 0, 0}, acc[3] = {0, 0, 0};
  if (sc.shape == 3) {
    int d = b.dual[i];
    if (d < 0) return -1.f;
    int dz = div_by(d, sc.mCNCxy), rem = d - dz * sc.CNCxy, dy = div_by(rem, sc.mCNCx), dx = rem - dy * sc.CNCx;
    int ln = b.inode[i];
    int bd = ln >= 0 ? b.bd[sc.n0 + ln] : 0;
    float xx[3];
    for (int a = 0; a < 3; ++a) {
      if ((bd >> (2 * a)) & 3) {  // AuxiliaryGridSHP
        float xn = b.xn[a * NP + i];
        xx[a] = xn < 0.f ? 1.f + 2.f * xn : 2.f * xn - 1.f;
      } else {
        xx[a] = b.xxn[a * NP + i];
      }
    }
    if (bd == 0)
      for (int a = 0; a < 3; ++a) xx[a] = b.xxn[a * NP + i];
    for (int k = 0; k < 8; ++k) {
      int oc[3] = {kCorner[k][0], kCorner[k][1], kCorner[k][2]};
      const long long cid = sg_corner_cell(sc, dx, dy, dz, k);
      if (cid < 0) continue;
      const float4 cv = b.cvel[sc.c0 + cid], ca = b.cacl[sc.c0 + cid];
      float w = 0.125f;
      for (int a = 0; a < 3; ++a) w *= oc[a] ? 1.f + xx[a] : 1.f - xx[a];
      v[0] += w * cv.x;
      v[1] += w * cv.y;
      v[2] += w * cv.z;
      acc[0] += w * ca.x;
      acc[1] += w * ca.y;
      acc[2] += w * ca.z;
    }
  } else {
    const int cl = b.cell[i];
    if (cl < 0) return -1.f;
    int c[3];
    c[2] = div_by(cl, sc.mNCxy);
    int rem = cl - c[2] * sc.NCxy;
    c[1] = div_by(rem, sc.mNCx);
    c[0] = rem - c[1] * sc.NCx;
    float off[3] = {b.off[i], b.off[NP + i], b.off[2 * NP + i]};
    int t0[3], nt[3];
    float wd[3][3], dd[3][3];
    for (int a = 0; a < 3; ++a) nt[a] = dim_nodes(sc.shape, off[a], t0[a], wd[a], dd[a]);
    // node rows along x, one multiply per node for its weight (the shape is a
    // tensor product)
    const NodeBox box = node_box(sc, c, t0, nt);
#pragma unroll
    for (int az = 0; az < 3; ++az)
#pragma unroll
      for (int ay = 0; ay < 3; ++ay) {
        if (!box.row(ay, az)) continue;
        const int o = az * box.sz + ay * box.sy;
        const float2 *rv = b.nvxy + box.first + o, *rz = b.nz + box.first + o, *ra = b.naxy + box.first + o;
        const float wyz = wd[1][ay] * wd[2][az];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
          if (!box.x(ax)) continue;
          const float2 vn = rv[ax], z = rz[ax], an = ra[ax];  // zero below the cut-off mass
          const float w = wd[0][ax] * wyz;
          v[0] += w * vn.x;
          v[1] += w * vn.y;
          v[2] += w * z.x;
          acc[0] += w * an.x;
          acc[1] += w * an.y;
          acc[2] += w * z.y;
        }
      }
  }
  // position and velocity integrated in FP64 (the FP32 interpolants
  // converted exactly by integer operations; the FP32 velocity copy
  // likewise)
  const double dt = st.dt;
  float pv[3];
  for (int a = 0; a < 3; ++a) {
    const double xx = x0[a] + f64_of(v[a]) * dt;
    // (XX and, at the end of the step, Xp: nothing in between reads positions)
    b.x[a * NP + i] = xx;
    const double vv = v0[a];
    const double vn = st.istep == 1 ? vv + f64_of(acc[a]) * dt * 0.5 : vv + f64_of(acc[a]) * dt;
    b.v[a * NP + i] = vn;
    pv[a] = f32_rn(vn);
    b.v32[a * NP + i] = pv[a];  // for the momentum transfers of this step (MUSL) and the next
  }
  // bound of those transfers' contributions
  const float m = b.m32[i];
  return m * fmaxf(fabsf(pv[0]), fmaxf(fabsf(pv[1]), fabsf(pv[2]))) * 1.0001f;
}

// (capped at 40 registers: six 256-thread blocks per SM hide the node
// gathers' latency better than fewer blocks with more registers; a pblock of
// 512 still launches)
__global__ void __launch_bounds__(512, 3) kb_position(BState b) {
  chain_entry();
  const long long i = btid();
  float bound = -1.f;
  if (i < b.NP) bound = position_one(b, i);
  block_scene_max<1>(b, bound >= 0.f ? (int)b.scene[i] : -1, {Q_MOM_MUSL}, {fmaxf(bound, 0.f)});
}

// GridMomentumMUSL: momentum re-map with the new particle velocities
template <bool SG>
__global__ void kb_p2g_momentum(BState b, long long n0, long long n1) {
  chain_entry();
  const long long n = n0 + btid();
  if (n >= n1) return;
  const int s = scene_of(b, b.node_scene, n);
  if (!scene_live(b, s)) return;
  const Scene& sc = b.scenes[s];
  if (!sc.musl) return;
  const long long NN = b.NN;
  double P0 = 0, P1 = 0, P2 = 0;
  if (SG) {
    int j[3];
    node_xyz(sc, n - sc.n0, j[0], j[1], j[2]);
    // centre nodes -> node (GridMomentumMUSL of SGMP), exact sums of the
    // cells' fixed-point momenta
    const unsigned near = sg_active_cells(b, sc, j);
    if (!near && __double_as_longlong(b.mg[n]) == 0ll) return;  // idle node (as in take_acc)
    long long Q[3] = {0, 0, 0};
    const long long* ca = reinterpret_cast<const long long*>(b.cacc) + CQ_P * b.NC;
#pragma unroll
    for (int k0 = 0; k0 < 8; k0 += 4) {  // (four cells' loads in flight at a time)
      long long q[4][3];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool on = near >> (k0 + k) & 1u;
        const long long c = sg_near_cell(sc, j, k0 + k);
#pragma unroll
        for (int a = 0; a < 3; ++a) q[k][a] = on ? ca[a * b.NC + c] : 0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        for (int a = 0; a < 3; ++a) Q[a] += q[k][a];
    }
    const double u = q_unit(q_shift(sc, b.sst[s].qmax[Q_MOM_MUSL]));
    P0 = 0.125 * ((double)Q[0] * u);
    P1 = 0.125 * ((double)Q[1] * u);
    P2 = 0.125 * ((double)Q[2] * u);
  } else {
    const double u = q_unit(q_shift(sc, b.sst[s].qmax[Q_MOM_MUSL]));
    const double unit[3] = {u, u, u};
    double o[3];
    if (!take_acc(b, n, 3, unit, o)) return;  // idle node
    P0 = o[0];
    P1 = o[1];
    P2 = o[2];
  }
  b.px[n] = P0;
  b.px[NN + n] = P1;
  b.px[2 * NN + n] = P2;
  if (b.mg[n] == 0.0 && (P0 != 0.0 || P1 != 0.0 || P2 != 0.0))
    b.mg[n] = -0.0;  // momentum at a massless node (take_acc)
  node_finish(b, sc, n, 1, !sc.usf);
}

// ------------------------------------------------------------ reductions
// calcEnergy + UpdateDT per scene: a block per chunk (Scene::chunk particles) of
// one scene (chunks are fixed relative to the scene start, so the sums of a
// scene do not depend on the other scenes of the batch), then a block per
// scene combining its chunks in order.
// the scene totals from its chunks' partial sums (FP64; fixed tree order)
// and, with mode & 2, UpdateDT; every thread of the block calls it
__device__ __forceinline__ void reduce_scene_finish(BState& b, int s, int mode, double (*sh)[256]) {
  const Scene& sc = b.scenes[s];
  double acc[6] = {0, 0, 0, 0, 0, 0};
  for (long long r = sc.r0 + threadIdx.x; r < sc.r0 + sc.nr; r += blockDim.x) {
    // (L2 loads: another SM wrote the partials, and this SM's L1 may hold
    // the last step's)
    for (int k = 0; k < 5; ++k) acc[k] += __ldcg(&b.red_part[k * b.NR + r]);
    acc[5] = fmax(acc[5], __ldcg(&b.red_part[5 * b.NR + r]));
  }
  __shared__ double tot[6];
  reduce_block<6, 256>(sh, acc, tot);
  if (threadIdx.x != 0) return;
  SceneState& st = b.sst[s];
  if (mode & 1) {
    st.ke_prev = st.ke;
    st.ke = tot[0];
    st.ie = tot[1];
    st.mom[0] = tot[2];
    st.mom[1] = tot[3];
    st.mom[2] = tot[4];
  }
  st.max_vp = tot[5];
  if (mode & 2) {
    // the least time over the materials is the fastest one's (both roundings
    // are monotonic)
    double dt = (double)1e6f;
    if (sc.wave >= 0.0) dt = fmin(dt, sc.dcell / (sc.wave + tot[5]));
    st.dt = dt * sc.dtscale;
    st.fdt = (float)st.dt;
  }
}

// calcEnergy / UpdateDT: one block per chunk of particles of a live
// scene sums the chunk in FP64 (the energy balance stays in FP64) and writes
// its partial sums; the scene's last chunk block to finish (a per-scene
// counter, reset by that block) forms the scene totals. On small scenes this
// chain ends after the mass transfer beside it: the block sums by a warp per
// value (reduce_block) took 2 us off the step of 36 k to 160 k particles (70 ->
// 68, 87 -> 85). On large ones it shares memory and FP64 pipe with that
// transfer: two particles per thread in flight and the maximum in integers
// (-0.4 %; four: no gain, eight: +1 %).
__global__ void __launch_bounds__(256) kb_reduce_chunks(BState b, int mode) {
  chain_entry();
  __shared__ double sh[6][256], part[6];
  __shared__ int last;
  const long long r = blockIdx.x;
  const int s = b.rscene[r];
  if (!b.ract[s]) return;  // (uniform: every block of the scene returns)
  const Scene& sc = b.scenes[s];
  const long long NP = b.NP;
  double acc[6] = {0, 0, 0, 0, 0, 0};
  const long long p_begin = sc.p0 + (r - sc.r0) * sc.chunk;
  const long long p_end = min(p_begin + sc.chunk, sc.p0 + sc.np);
  constexpr int U = 2;  // particles of a thread in flight
  unsigned long long top = 0ull;  // largest |velocity component|, as bits (ordered like the values)
  for (long long i0 = p_begin + threadIdx.x; i0 < p_end; i0 += U * blockDim.x) {
    double v[U][3], m[U], e[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long i = i0 + u * blockDim.x;
      const bool in = i < p_end;
      for (int c = 0; c < 3; ++c) v[u][c] = in ? b.v[c * NP + i] : 0.0;
      m[u] = in ? b.mass[i] : 0.0;
      e[u] = in ? b.ie[i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      acc[0] += (v[u][0] * v[u][0] + v[u][1] * v[u][1] + v[u][2] * v[u][2]) * m[u];
      acc[1] += e[u];
      for (int c = 0; c < 3; ++c) {
        acc[2 + c] += m[u] * v[u][c];
        const unsigned long long w = (unsigned long long)__double_as_longlong(v[u][c]) & 0x7fffffffffffffffull;
        top = w > top && w <= 0x7ff0000000000000ull ? w : top;  // (a NaN does not count)
      }
    }
  }
  acc[0] *= 0.5;
  acc[5] = __longlong_as_double((long long)top);
  reduce_block<6, 256>(sh, acc, part);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 6; ++k) b.red_part[k * b.NR + r] = part[k];
    __threadfence();
    last = atomicAdd(&b.sst[s].red_done, 1u) == (unsigned)(sc.nr - 1);
  }
  __syncthreads();
  if (!last) return;
  if (threadIdx.x == 0) b.sst[s].red_done = 0u;
  reduce_scene_finish(b, s, mode, sh);
}

__global__ void kb_dr_damping(BState b) {
  chain_entry();
  long long i = btid();
  if (i >= b.NP) return;
  const int s = scene_of(b, b.scene, i);
  const Scene& sc = b.scenes[s];
  if (!sc.drdamp || !b.ract[s]) return;
  const SceneState& st = b.sst[s];
  if (!(st.ke - st.ke_prev <= 0.0)) return;
  const long long NP = b.NP;
  for (int a = 0; a < 3; ++a) {
    b.v[a * NP + i] = 0;
    b.v32[a * NP + i] = 0.f;
  }
}

__global__ void kb_dr_finish(BState b) {
  chain_entry();
  int s = (int)btid();
  if (s >= b.nscene) return;
  if (!b.scenes[s].drdamp || !b.ract[s]) return;
  SceneState& st = b.sst[s];
  if (st.ke - st.ke_prev <= 0.0) st.ke = 0;
}

// values of a few particles of one scene (by deck index) for the curve output
struct GatherItem {
  long long p;
  int field, comp;
};

// value of particle field `field` (component c) at storage position i
__device__ __forceinline__ double field_value(const BState& b, int field, long long c, long long i) {
  const long long NP = b.NP;
  double v = 0.0;
  switch (field) {
    case MPM_P_XP: v = b.x[c * NP + i]; break;
    case MPM_P_XX: v = b.x[c * NP + i]; break;  // XX equals Xp between steps
    case MPM_P_VXP: v = b.v[c * NP + i]; break;
    case MPM_P_FXP: v = b.scenes[b.scene[i]].has_fxp ? b.fxp[c * NP + i] : 0.0; break;
    case MPM_P_VOL: v = b.vol[i]; break;
    case MPM_P_SIG_Y: v = b.sig_y[i]; break;
    case MPM_P_SM: v = b.sm[i]; break;
    case MPM_P_SEQV: v = b.seqv[i]; break;
    case MPM_P_SD: v = b.sd[c * NP + i]; break;
    case MPM_P_FP: v = (double)b.fp[c * NP + i] + (double)b.fp[(9 + c) * NP + i]; break;
    case MPM_P_EPEFF: v = b.epeff[i]; break;
    case MPM_P_CELSIUS: v = b.celsius[i]; break;
    case MPM_P_DMG: v = b.dmg[i]; break;
    case MPM_P_LT: v = b.lt[i]; break;
    case MPM_P_IE: v = b.ie[i]; break;
    case MPM_P_MASS: v = b.mass[i]; break;
    case MPM_P_CP: v = b.cp[i]; break;
    case MPM_P_Q: v = b.q[i]; break;
    case MPM_P_FAILURE: v = b.failure[i] ? 1.0 : 0.0; break;
    default: v = 0.0; break;
  }
  return v;
}

__global__ void kb_gather(BState b, int scene, const GatherItem* it, int n, double* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const Scene& sc = b.scenes[scene];
  out[k] = field_value(b, it[k].field, it[k].comp, b.inv[sc.p0 + it[k].p]);
}

// one component of a particle field of a scene in deck order (downloads)
__global__ void kb_unpermute(BState b, int scene, int field, int ncomp, double* dst) {
  const Scene& sc = b.scenes[scene];
  const long long t = btid();
  if (t >= sc.np * ncomp) return;
  const int a = (int)(t / sc.np);
  const long long k = t - (long long)a * sc.np;
  dst[t] = field_value(b, field, a, b.inv[sc.p0 + k]);  // component-major, input order
}

// ----------------------------------------------------- stress smoothing
// SmoothStressbyGrid (update_step.f90:1876-2055) for one scene, computed
// from the state after its last step when Spre is read (it feeds only the
// output): -SM * VOL and VOL mapped to the grid, Gpre = their ratio on the
// mapped nodes, Spre interpolated back. Shapes as in the reference: GIMP and
// B-spline at the current position against the step's cell, linear ones at
// the step's offsets, SGMP ones at the step's XXN through the centre nodes
// (nodes above the cut-off mass on the way back). Contributions are FP32,
// quantised per particle and node and summed exactly (64-bit fixed point,
// scales from the scene's largest |SM * VOL| and VOL), so Spre does not
// depend on the other scenes of the batch.

// bounds: bnd[0] = max |SM * VOL|, bnd[1] = max VOL (float bits)
__global__ void kb_smooth_bound(BState b, int scene, unsigned* bnd) {
  const Scene& sc = b.scenes[scene];
  const long long k = btid();
  if (k >= sc.np) return;
  const long long i = sc.p0 + k;
  atomicMax(&bnd[0], __float_as_uint(fabsf(b.sm[i] * b.vol[i]) * 1.0001f));
  atomicMax(&bnd[1], __float_as_uint(fabsf(b.vol[i]) * 1.0001f));
}

// particles -> nodes (SGMP: centre nodes); acc = [2][nodes or cells of the scene]
__global__ void kb_smooth_p2g(BState b, int scene, const unsigned* bnd, unsigned long long* acc) {
  const Scene& sc = b.scenes[scene];
  const long long k = btid();
  if (k >= sc.np) return;
  const long long i = sc.p0 + k, NP = b.NP;
  const float sp = q_scale(q_shift(sc, bnd[0])), sv = q_scale(q_shift(sc, bnd[1]));
  const float pv = -b.sm[i] * b.vol[i], v = b.vol[i];
  if (sc.shape == 3) {
    const int d = b.dual[i];
    if (d < 0) return;
    const int dz = div_by(d, sc.mCNCxy), rem = d - dz * sc.CNCxy, dy = div_by(rem, sc.mCNCx), dx = rem - dy * sc.CNCx;
    const long long nc = sc.nc;
    for (int c = 0; c < 8; ++c) {
      const long long cid = sg_corner_cell(sc, dx, dy, dz, c);
      if (cid < 0) continue;
      float w = 0.125f;
      for (int a = 0; a < 3; ++a) w *= kCorner[c][a] ? 1.f + b.xxn[a * NP + i] : 1.f - b.xxn[a * NP + i];
      const long long qp = quant(w * pv, sp), qv = quant(w * v, sv);
      if (qp) atomicAdd(&acc[cid], (unsigned long long)qp);
      if (qv) atomicAdd(&acc[nc + cid], (unsigned long long)qv);
    }
    return;
  }
  const int cl = b.cell[i];
  if (cl < 0) return;
  int c[3];
  c[2] = div_by(cl, sc.mNCxy);
  c[1] = div_by(cl - c[2] * sc.NCxy, sc.mNCx);
  c[0] = cl - c[2] * sc.NCxy - c[1] * sc.NCx;
  float off[3];
  for (int a = 0; a < 3; ++a)
    off[a] = sc.shape == 0 ? b.off[a * NP + i] : (float)((b.x[a * NP + i] - sc.span0[a]) * sc.idcell - (double)c[a]);
  const int tlo = sc.shape == 0 ? 0 : -1, thi = sc.shape == 1 ? 2 : 1;
  float w1[3][4];
  for (int a = 0; a < 3; ++a)
    for (int t = tlo; t <= thi; ++t) {
      float w, dd;
      if (sc.shape == 0) lin1(t, off[a], w, dd);
      else if (sc.shape == 2) bsp1(t, off[a], w, dd);
      else gimp1((float)(-t) + off[a], w, dd);
      w1[a][t + 1] = w;
    }
  for (int tz = tlo; tz <= thi; ++tz)
    for (int ty = tlo; ty <= thi; ++ty)
      for (int tx = tlo; tx <= thi; ++tx) {
        const float w = w1[0][tx + 1] * w1[1][ty + 1] * w1[2][tz + 1];
        const int jx = c[0] + tx, jy = c[1] + ty, jz = c[2] + tz;
        if (w == 0.f || jx < 0 || jx >= sc.NGx || jy < 0 || jy >= sc.NGy || jz < 0 || jz >= sc.NGz) continue;
        const long long n = ((long long)jz * sc.NGy + jy) * sc.NGx + jx;
        const long long qp = quant(w * pv, sp), qv = quant(w * v, sv);
        if (qp) atomicAdd(&acc[n], (unsigned long long)qp);
        if (qv) atomicAdd(&acc[sc.nn + n], (unsigned long long)qv);
      }
}

// Gpre per node of the scene: the ratio of the sums where volume arrived
// (SGMP: of 1/8 of every adjacent cell's sums; every node counts as mapped,
// 0/0 where none arrived)
__global__ void kb_smooth_node(BState b, int scene, const unsigned* bnd, const unsigned long long* acc, double* gpre) {
  const Scene& sc = b.scenes[scene];
  const long long ln = btid();
  if (ln >= sc.nn) return;
  const double up = q_unit(q_shift(sc, bnd[0])), uv = q_unit(q_shift(sc, bnd[1]));
  if (sc.shape == 3) {
    int j[3];
    node_xyz(sc, ln, j[0], j[1], j[2]);
    long long qp = 0, qv = 0;
    for (int cz = j[2] - 1; cz <= j[2]; ++cz) {
      if (cz < 0 || cz >= sc.NCz) continue;
      for (int cy = j[1] - 1; cy <= j[1]; ++cy) {
        if (cy < 0 || cy >= sc.NCy) continue;
        for (int cx = j[0] - 1; cx <= j[0]; ++cx) {
          if (cx < 0 || cx >= sc.NCx) continue;
          const long long c = ((long long)cz * sc.NCy + cy) * sc.NCx + cx;
          qp += (long long)acc[c];
          qv += (long long)acc[sc.nc + c];
        }
      }
    }
    gpre[ln] = (0.125 * ((double)qp * up)) / (0.125 * ((double)qv * uv));
    return;
  }
  const long long qv = (long long)acc[sc.nn + ln];
  gpre[ln] = qv != 0 ? ((double)(long long)acc[ln] * up) / ((double)qv * uv) : 0.0;
}

// SGMP: nodes above the cut-off mass -> centre nodes
__global__ void kb_smooth_back(BState b, int scene, const double* gpre, double* cgpre) {
  const Scene& sc = b.scenes[scene];
  const long long c = btid();
  if (c >= sc.nc) return;
  const int cz = div_by(c, sc.mNCxy), rem = (int)(c - (long long)cz * sc.NCxy), cy = div_by(rem, sc.mNCx), cx = rem - cy * sc.NCx;
  double g = 0.0;
  for (int k = 0; k < 8; ++k) {
    const long long ln = ((long long)(cz + kCorner[k][2]) * sc.NGy + cy + kCorner[k][1]) * sc.NGx + cx + kCorner[k][0];
    if (b.mg[sc.n0 + ln] > sc.cutoff) g = g + 0.125 * gpre[ln];
  }
  cgpre[c] = g;
}

// (centre) nodes -> particles: Spre in the scene's input order
__global__ void kb_smooth_g2p(BState b, int scene, const double* gpre, const double* cgpre, double* spre) {
  const Scene& sc = b.scenes[scene];
  const long long k = btid();
  if (k >= sc.np) return;
  const long long i = sc.p0 + k, NP = b.NP;
  double s = 0.0;
  if (sc.shape == 3) {
    const int d = b.dual[i];
    if (d >= 0) {
      const int dz = div_by(d, sc.mCNCxy), rem = d - dz * sc.CNCxy, dy = div_by(rem, sc.mCNCx), dx = rem - dy * sc.CNCx;
      for (int c = 0; c < 8; ++c) {
        const long long cid = sg_corner_cell(sc, dx, dy, dz, c);
        if (cid < 0) continue;
        float w = 0.125f;
        for (int a = 0; a < 3; ++a) w *= kCorner[c][a] ? 1.f + b.xxn[a * NP + i] : 1.f - b.xxn[a * NP + i];
        s = s + (double)w * cgpre[cid];
      }
    }
  } else if (b.cell[i] >= 0) {
    const int cl = b.cell[i];
    int c[3];
    c[2] = div_by(cl, sc.mNCxy);
    c[1] = div_by(cl - c[2] * sc.NCxy, sc.mNCx);
    c[0] = cl - c[2] * sc.NCxy - c[1] * sc.NCx;
    float off[3];
    for (int a = 0; a < 3; ++a)
      off[a] = sc.shape == 0 ? b.off[a * NP + i] : (float)((b.x[a * NP + i] - sc.span0[a]) * sc.idcell - (double)c[a]);
    const int tlo = sc.shape == 0 ? 0 : -1, thi = sc.shape == 1 ? 2 : 1;
    float w1[3][4];
    for (int a = 0; a < 3; ++a)
      for (int t = tlo; t <= thi; ++t) {
        float w, dd;
        if (sc.shape == 0) lin1(t, off[a], w, dd);
        else if (sc.shape == 2) bsp1(t, off[a], w, dd);
        else gimp1((float)(-t) + off[a], w, dd);
        w1[a][t + 1] = w;
      }
    for (int tz = tlo; tz <= thi; ++tz)
      for (int ty = tlo; ty <= thi; ++ty)
        for (int tx = tlo; tx <= thi; ++tx) {
          const float w = w1[0][tx + 1] * w1[1][ty + 1] * w1[2][tz + 1];
          const int jx = c[0] + tx, jy = c[1] + ty, jz = c[2] + tz;
          if (w == 0.f || jx < 0 || jx >= sc.NGx || jy < 0 || jy >= sc.NGy || jz < 0 || jz >= sc.NGz) continue;
          s = s + (double)w * gpre[((long long)jz * sc.NGy + jy) * sc.NGx + jx];
        }
  }
  spre[b.orig[i]] = s;
}

// SGMP centre-node mass (comp -1) or momentum component of a scene from
// its fixed-point sums (downloads; the momentum of the last transfer, MUSL
// or not)
__global__ void kb_centre_field(BState b, int scene, int comp, double* dst) {
  const Scene& sc = b.scenes[scene];
  const long long k = btid();
  if (k >= sc.nc) return;
  const SceneState& st = b.sst[scene];
  const int q = comp < 0 ? Q_MASS : (sc.musl ? Q_MOM_MUSL : Q_MOM);
  const int ch = comp < 0 ? CQ_M : CQ_P + comp;
  dst[k] = (double)(long long)b.cacc[ch * b.NC + sc.c0 + k] * q_unit(q_shift(sc, st.qmax[q]));
}

}  // namespace bm
}  // namespace mpm
