// gx_step.cuh -- one step of a track, for the transport engine
// (gx_transport.cu): the track record, the layered calorimeter's navigation, cross
// sections, multiple scattering, the phases of a step, the interaction models'
// dispatch, and the tallies of a block.
#pragma once

#include "gx_internal.cuh"

#include <cstring>
#include <type_traits>

namespace gx {
#ifdef GX_PARITY
namespace parity {
#endif

// ------------------------------------------------------------------ layout
// A track record: 96 bytes (128 in FP64), moved as 16-byte words.  One record
// is three (four) whole sectors wherever it goes, whether one lane of a warp
// writes or all, and takes 6 (8) memory instructions from one address.  As a
// plane per member (23 words from 15 addresses, whose pointers were loaded for
// each record, each written lane a sector per plane) 20000 10 GeV showers took
// 172.0 ms, with these records and relocate() without its division 156.1 ms:
// an e- takes 1.4 steps between a load and a store.
// r0: multiple scattering: range scale of the step limit in the current volume
// (<= 0: unset); rs: MRG32k3a state.
template <class R> struct alignas(16) Rec {
  double pos[3];
  R dir[3], E, nil[3], r0;
  uint32_t rs[6];
  int vol, event, prim, type;
};
static_assert(sizeof(Rec<float>) == 96 && sizeof(Rec<double>) == 128, "record layout");

template <class R> struct Store {
  Rec<R> *rec;
  long long cap;
};

struct Geom {
  int geometry, axis, nlayers, box_mat, charged_local, nvol, nevents;
  int msc;       // multiple scattering of e-/e+
  int field_map; // 1: the context's field map with Runge-Kutta sub-steps, 0: uniform Bz
  double t_abs, pitch, x0, total, half_trans, Bz;
  double box_half[3], box_centre[3];
  CsgView csg; // geometry 2: the context's volume tree
};

constexpr int kNStat = 29;
// S_READ/S_WRITE: track records read and written by the step kernels of a
// type other than its transport kernel (the interaction kernels, the plain
// loop's fused kernel); S_TREAD/S_TWRITE: by its transport kernel (the host
// reports the sums as the type's records read and written); S_TQUEUE: of the
// transport kernel's writes, the records put in an interaction buffer (added
// up by k_finish from the buffers' counters); S_TSTEP: steps completed in the
// transport kernel of a type; S_BOOKED: steps of electrons that the interaction
// kernels book where they stop.
enum { S_STEPS, S_SUBSTEPS, S_TRACKS, S_SEC0, S_SEC1, S_SEC2, S_PAIR, S_ANNIH, S_ERR, S_OVERFLOW,
       S_READ0, S_READ1, S_READ2, S_WRITE0, S_WRITE1, S_WRITE2, S_TREAD0, S_TREAD1, S_TREAD2,
       S_TWRITE0, S_TWRITE1, S_TWRITE2, S_TQUEUE0, S_TQUEUE1, S_TQUEUE2, S_TSTEP0, S_TSTEP1, S_TSTEP2,
       S_BOOKED };

struct Ctl {
  int parity;
  int err_flags;
  long long count[2][3];
  long long stack_count[3];
  long long prim_next, nprim;
  long long take_stack[3], take_prim; // refill plan
  long long stack_dst[3], stack_src[3];
  long long in_flight, pending, peak, iterations;
  unsigned long long stat[kNStat];
  double escaped;
  double retired;     // energy deposited or escaped so far (the rest is still carried by tracks)
  long long extracted; // tracks written out by gx_transport_tracks
  const double *cumE; // inclusive prefix sum of the primary energies
  double wave_energy; // energy carried by live tracks before more primaries are injected, at most
  long long refill_below, stack_cap;
  long long qcount[3][3]; // records in the interaction buffers [particle][process]
  long long take[3];      // tracks of the current stores handed out to the transport kernels
};

// Tracks handed in as a gx_track_soa (gx_transport_tracks) instead of
// primaries: injected with their state as it is.
struct SoaIn {
  const int *type, *status, *event, *primary, *volume;
  const double *x, *y, *z, *dx, *dy, *dz, *ekin, *nil0, *nil1, *nil2, *msc;
  const uint32_t *rng;
  long long cap;
};

struct Prims {
  const int *type, *event;
  const double *E, *pos, *dir;
  double seed[6];
  long long first_substream;
  const uint64_t *jump;
  int from_soa; // 1: inject the tracks of soa
  SoaIn soa;
};

template <class R> struct Args {
  const Data *d;
  Ctl *ctl;
  Store<R> st[2][3];
  Store<R> stack[3];
  Geom g;
  Prims p;
  double *edep;
  int *pstep;
  int nstores;
  long long refill_below;
  // tracks waiting for an interaction, per particle type and process, stored
  // compactly so the interaction kernels read them coalesced (batched engine)
  Store<R> ibuf[3][3];
  long long qcap;
  // steps of one track per transport launch, at most, per particle type; few: when
  // the store has no more tracks than the grid has threads
  int step_budget[3], few_budget[3];
  int fetch_min[3];   // idle lanes of a warp before it takes new records, per particle type
  int book_stops;     // electrons that stop where they are created may be booked there
};

// ---------------------------------------------------------------- geometry
// Component a (the run-time layer axis) of a 3-vector.  Selects instead of an
// indexed access keep the vectors in registers: an array indexed by a run-time
// value lives in local memory.
template <class T> __device__ __forceinline__ T comp(const T *p, int a) { return a == 0 ? p[0] : (a == 1 ? p[1] : p[2]); }
template <class T> __device__ __forceinline__ void set_comp(T *p, int a, T v)
{
  if (a == 0)
    p[0] = v;
  else if (a == 1)
    p[1] = v;
  else
    p[2] = v;
}

// The layered calorimeter along axis a: layer k occupies [x0 + k pitch,
// x0 + (k+1) pitch), absorber first.  vol = 2 layer + slab; -1 outside.
__device__ __forceinline__ int vol_material(const Geom &g, int vol)
{
  if (g.geometry == 2) return g.csg.node[vol].mat;
  return g.geometry == 0 ? g.box_mat : ((vol & 1) ? 2 : 1);
}
__device__ __forceinline__ void slab_bounds(const Geom &g, int vol, double &lo, double &hi)
{
  if (g.geometry == 0) {
    const double c = comp(g.box_centre, g.axis), h = comp(g.box_half, g.axis);
    lo = c - h;
    hi = c + h;
    return;
  }
  double base = g.x0 + (vol >> 1) * g.pitch;
  lo = (vol & 1) ? base + g.t_abs : base;
  hi = (vol & 1) ? base + g.pitch : base + g.t_abs;
}
__device__ __forceinline__ double thalf(const Geom &g, int b) { return g.geometry == 0 ? g.box_half[b] : g.half_trans; }
__device__ __forceinline__ double tcentre(const Geom &g, int b) { return g.geometry == 0 ? g.box_centre[b] : 0.0; }

__device__ __forceinline__ int locate(const Geom &g, const double *p, const double *d)
{
  const double tol = 1e-12;
  int a = g.axis;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    if (b == a) continue;
    double h = thalf(g, b), q = p[b] - tcentre(g, b);
    if (q > h || q < -h) return -1;
    if ((q > h - tol && d[b] > 0) || (q < -h + tol && d[b] < 0)) return -1;
  }
  const double pa = comp(p, a), da = comp(d, a);
  if (g.geometry == 0) {
    double q = pa - comp(g.box_centre, a), h = comp(g.box_half, a);
    if (q > h || q < -h) return -1;
    if ((q > h - tol && da > 0) || (q < -h + tol && da < 0)) return -1;
    return 0;
  }
  double u = pa - g.x0;
  if (u < -tol || u > g.total + tol) return -1;
  if ((u < tol && da < 0) || (u > g.total - tol && da > 0)) return -1;
  int layer = (int)floor(u / g.pitch);
  layer = min(max(layer, 0), g.nlayers - 1);
  double q = u - layer * g.pitch;
  if (q < tol && da < 0 && layer > 0) return 2 * (layer - 1) + 1;
  if (q > g.pitch - tol && da > 0 && layer + 1 < g.nlayers) return 2 * (layer + 1);
  if (fabs(q - g.t_abs) < tol) return 2 * layer + (da > 0 ? 1 : 0);
  return 2 * layer + (q < g.t_abs ? 0 : 1);
}

__device__ __forceinline__ double dist_to_out(const Geom &g, int vol, const double *p, const double *d, int &plane)
{
  int a = g.axis;
  double lo, hi, dist = 1.7976931348623157e308;
  slab_bounds(g, vol, lo, hi);
  plane = 0;
  const double pa = comp(p, a), da = comp(d, a);
  if (da > 0) {
    dist = (hi - pa) / da;
    plane = 1;
  } else if (da < 0) {
    dist = (lo - pa) / da;
    plane = -1;
  }
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    if (b == a) continue;
    double h = thalf(g, b), q = p[b] - tcentre(g, b), t = 1.7976931348623157e308;
    if (d[b] > 0)
      t = (h - q) / d[b];
    else if (d[b] < 0)
      t = (-h - q) / d[b];
    if (t < dist) {
      dist = t;
      plane = 2;
    }
  }
  return dist < 0 ? 0 : dist;
}

// The same distance with one division (the FP32-mixed engine): each plane's
// candidate kept as a fraction num / den with den > 0, candidates compared by
// cross-multiplication in the order the loop above takes them (axis planes
// first, ties to the earlier), and only the nearest divided out.
__device__ __forceinline__ double dist_to_out_1div(const Geom &g, int vol, const double *p, const double *d,
                                                   int &plane)
{
  int a = g.axis;
  double lo, hi;
  slab_bounds(g, vol, lo, hi);
  plane = 0;
  double num = 1.7976931348623157e308, den = 1.0;
  const double pa = comp(p, a), da = comp(d, a);
  if (da > 0) {
    num = hi - pa;
    den = da;
    plane = 1;
  } else if (da < 0) {
    num = pa - lo;
    den = -da;
    plane = -1;
  }
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    if (b == a) continue;
    const double h = thalf(g, b), q = p[b] - tcentre(g, b);
    double n = 0.0, m = 0.0;
    if (d[b] > 0) {
      n = h - q;
      m = d[b];
    } else if (d[b] < 0) {
      n = h + q;
      m = -d[b];
    }
    if (m > 0 && n * den < num * m) {
      num = n;
      den = m;
      plane = 2;
    }
  }
  const double dist = num / den;
  return dist < 0 ? 0 : dist;
}

__device__ __forceinline__ double safety(const Geom &g, int vol, const double *p)
{
  int a = g.axis;
  double lo, hi;
  slab_bounds(g, vol, lo, hi);
  const double pa = comp(p, a);
  double s = fmin(pa - lo, hi - pa);
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    if (b == a) continue;
    s = fmin(s, thalf(g, b) - fabs(p[b] - tcentre(g, b)));
  }
  return s < 0 ? 0 : s;
}

__device__ __forceinline__ int next_volume(const Geom &g, int vol, int plane)
{
  if (plane == 2 || g.geometry == 0) return -1;
  int nv = vol + (plane > 0 ? 1 : -1);
  return (nv < 0 || nv >= 2 * g.nlayers) ? -1 : nv;
}

// Volume after a helix sub-step that started in vol.  An end point within
// kSnap of a face it is moving out through (or past it) is put on that face
// and enters the neighbour; otherwise the point is located.  The reference
// pushes 2e-9 mm past the straight-line boundary and locates the helix end
// point, which lands within rounding of the plane often enough for ulp-level
// differences to decide the crossing; the snap distance is far from both.
constexpr double kSnap = 1e-6;
__device__ __forceinline__ int relocate(const Geom &g, int vol, double *p, const double *d)
{
  int a = g.axis;
  double lo, hi;
  slab_bounds(g, vol, lo, hi);
  bool inside = true;
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    if (b == a) continue;
    double h = thalf(g, b), q = p[b] - tcentre(g, b);
    if ((d[b] > 0 && h - q < kSnap) || (d[b] < 0 && q + h < kSnap)) return -1;
    inside = inside && q <= h && q >= -h;
  }
  const double pa = comp(p, a), da = comp(d, a);
  // clear of both faces and not outside transversely: locating the point, with
  // its division by the pitch, would give this volume again
  if (inside && hi - pa >= kSnap && pa - lo >= kSnap) return vol;
  if (da > 0 && hi - pa < kSnap) {
    set_comp(p, a, hi);
    return next_volume(g, vol, 1);
  }
  if (da < 0 && pa - lo < kSnap) {
    set_comp(p, a, lo);
    return next_volume(g, vol, -1);
  }
  return locate(g, p, d);
}

// Kernel variants, template parameters so that each kernel carries only the
// code it runs: bit 0 follows the field map (Runge-Kutta sub-steps) instead of
// the uniform field's helix, bit 1 navigates the CSG tree (gx_csg.cuh) instead
// of the analytic volumes above, bit 2 applies multiple scattering, bit 3
// (with bit 1, FP32-mixed kernels) navigates a tree of boxes only: the
// navigator's code for the other solids is left out of those kernels.
enum { kKindFieldMap = 1, kKindCsg = 2, kKindMsc = 4, kKindBoxes = 8 };
template <int K> constexpr int kSolidsOf = (K & kKindBoxes) != 0 ? kSolidsBox : kSolidsAll;

template <int K> __device__ __forceinline__ double nav_safety(const Geom &g, int vol, const double *p)
{
  if constexpr ((K & kKindCsg) != 0)
    return csg_safety<kSolidsOf<K>>(g.csg, vol, p);
  else
    return safety(g, vol, p);
}
// Straight-line distance to the next boundary.  plane: the analytic
// navigator's face code, or the CSG child entered (-1: leaving the volume);
// the CSG navigator skips children met only beyond limit.  ONE_DIV (the
// FP32-mixed engine): the analytic navigator's distance with one division.
template <int K, bool ONE_DIV = false>
__device__ __forceinline__ double nav_distance(const Geom &g, int vol, const double *p, const double *d, double limit,
                                               int &plane)
{
  if constexpr ((K & kKindCsg) != 0)
    return csg_step<kSolidsOf<K>>(g.csg, vol, p, d, limit, plane);
  else if constexpr (ONE_DIV)
    return dist_to_out_1div(g, vol, p, d, plane);
  else
    return dist_to_out(g, vol, p, d, plane);
}
template <int K> __device__ __forceinline__ int nav_relocate(const Geom &g, int vol, double *p, const double *d)
{
  if constexpr ((K & kKindCsg) != 0)
    return csg_locate<kSolidsOf<K>>(g.csg, vol, p, d, kSnap);
  else
    return relocate(g, vol, p, d);
}

// ---------------------------------------------------------- cross sections
// A table lookup of the step: the polynomial form (one record per bin); in
// the parity variant the reference's spline form, as the oracle evaluates it.
template <class R> __device__ __forceinline__ R tab_value(const Data &d, const VecDesc &v, R e)
{
#ifdef GX_PARITY
  static_assert(sizeof(R) == 8, "the parity variant is FP64");
  return vec_value_ref(d, v, e);
#else
  return vec_value_fast<R>(d, v, e);
#endif
}

template <class R> __device__ __forceinline__ R lambda_tab(const Data &d, int t, int mat, R e)
{
  const VecDesc &v = d.vec[t][mat];
  if ((double)e <= v.emin) return R(0);
  return tab_value<R>(d, v, e);
}

// Macroscopic cross sections (1/mm): gamma {Compton, conversion, photo-electric},
// e- {ionisation, brems}, e+ {ionisation, brems, annihilation}.
template <class R> __device__ __forceinline__ void cross_sections(const Data &d, int type, int mat, R e, R xs[3])
{
  xs[0] = xs[1] = xs[2] = R(0);
  if (type == 0) {
    xs[0] = (e < R(1)) ? tab_value<R>(d, d.vec[GX_Lambda_compt][mat], e)
                       : tab_value<R>(d, d.vec[GX_LambdaPrim_compt][mat], e) / e;
    xs[1] = lambda_tab<R>(d, GX_Lambda_conv, mat, e);
    if (e >= R(0.2))
      xs[2] = tab_value<R>(d, d.vec[GX_LambdaPrim_phot][mat], e) / e;
    else if constexpr (sizeof(R) == 4)
      xs[2] = pe_xs_sandia_f(d, (int)d.mat_Z[mat], (float)d.mat_density[mat], e);
    else
      xs[2] = (R)pe_xs_sandia(d, (int)d.mat_Z[mat], d.mat_density[mat], (double)e);
  } else if (type == 1) {
    xs[0] = lambda_tab<R>(d, GX_Lambda_eIoni_em, mat, e);
    xs[1] = lambda_tab<R>(d, GX_Lambda_eBrem_em, mat, e);
  } else {
    xs[0] = lambda_tab<R>(d, GX_Lambda_eIoni_ep, mat, e);
    xs[1] = lambda_tab<R>(d, GX_Lambda_eBrem_ep, mat, e);
    xs[2] = annih_xs<R>(d, mat, e);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (!(xs[i] > R(0))) xs[i] = R(0);
}

// ProxyIonization::AlongStepGPIL in physics mode (Geant4 step function, length
// cut); raw: the range table's value at e, which the step's continuous loss
// reuses (the energy does not change before it)
template <class R> __device__ __forceinline__ R range_limit(const Data &d, int type, int mat, R e, R &raw)
{
#ifdef GX_PARITY
  raw = R(-1);
  return ioni_along_gpil_ref(d, 1, type == 2 ? 1 : -1, mat, e);
#endif
  const R dR = R(0.2), finalRange = R(10.0);
  R range = vec_value_fast<R>(d, d.vec[type == 2 ? GX_Range_ep : GX_Range_em][mat], e);
  raw = range;
  if (e < R(kMinE)) range *= e / R(kMinE);
  R cut = (R)d.cut_length[1][mat];
  R finR = (finalRange < cut) ? finalRange : cut;
  if (range <= finR) return range;
  return range * dR + finR * (R(1) - dR) * (R(2) - finR / range);
}

// ProxyIonization::AlongStepDoIt in physics mode; the inverse range (used when
// the loss exceeds 1%, i.e. near the end of the range) is evaluated in FP64.
// range0 >= 0: the range table's value at e, taken at the start of the step.
template <class R>
__device__ __forceinline__ R along_loss(const Data &d, int type, int mat, double step, R &e, R range0 = R(-1))
{
#ifdef GX_PARITY
  double edep = 0.0, ee = e;
  ioni_along_doit_ref(d, 1, type == 2 ? 1 : -1, mat, step, ee, edep);
  e = ee;
  return edep;
#endif
  bool ep = type == 2;
  R energy = e;
  R range = range0 >= R(0) ? range0 : vec_value_fast<R>(d, d.vec[ep ? GX_Range_ep : GX_Range_em][mat], energy);
  if (step >= (double)range || energy <= R(kMinE)) {
    e = R(0);
    return energy;
  }
  R dedx = vec_value_fast<R>(d, d.vec[ep ? GX_DEDX_eIoni_ep : GX_DEDX_eIoni_em][mat], energy);
  if (energy < R(kMinE)) dedx *= M<R>::sqrt(energy / R(kMinE));
  R eloss = (R)step * dedx;
  if (eloss > energy * R(0.01)) {
    const VecDesc &vr = d.vec[ep ? GX_Range_ep : GX_Range_em][mat];
    const VecDesc &vi = d.vec[ep ? GX_InverseRange_ep : GX_InverseRange_em][mat];
    if constexpr (sizeof(R) == 4) {
      // the FP32-mixed engine: bin from the FP32 logarithm, one reciprocal
      const double r64 = vec_value_f64_f32bin(d, vr, (double)energy) - step;
      eloss = (R)((double)energy - vec_invrange_fast(d, vi, r64));
    } else {
      const double r64 = vec_value_fast<double>(d, vr, (double)energy) - step;
      eloss = (R)((double)energy - vec_invrange_ref(d, vi, r64));
    }
  }
  R finalE = energy - eloss;
  if (finalE < R(kMinE)) {
    eloss += finalE;
    finalE = R(0);
  }
  e = finalE;
  return eloss > R(0) ? eloss : R(0);
}

// ---------------------------------------------------------------- one step
template <class R> struct Track {
  int type, vol, event, prim;
  double pos[3];
  R dir[3], E, nil[3];
  R msc_r0;       // multiple scattering: range scale of the step limit in this volume (<= 0: unset)
  uint32_t rs[6]; // MRG32k3a state words; draws go through a Mrg made from them (rng / set_rng)
  __device__ __forceinline__ Mrg rng() const
  {
    Mrg m;
    m.from_words(rs);
    return m;
  }
  __device__ __forceinline__ void set_rng(const Mrg &m) { m.to_words(rs); }
  __device__ __forceinline__ void load_rng(const uint32_t *st, long long n, long long i)
  {
#pragma unroll
    for (int k = 0; k < 6; ++k) rs[k] = st[k * n + i]; // not the read-only path: a kernel may have written them
  }
  __device__ __forceinline__ void store_rng(uint32_t *st, long long n, long long i) const
  {
#pragma unroll
    for (int k = 0; k < 6; ++k) st[k * n + i] = rs[k];
  }
};

struct Local {
  // deposits go to a shared-memory tally when it fits, else to global memory
  double *sm_edep;
  double *g_edep;
  double *sm_esc; // this block's [escaped, retired] energy sums (shared memory)
  int nvol, nevents, sm_bins;
  double retired; // energy this thread took out of the live tracks (deposited or escaped)
  unsigned int st[kNStat];
  int err;
  __device__ __forceinline__ void escape(double e)
  {
    retired += e;
    atomicAdd(sm_esc, e);
  }
  __device__ __forceinline__ void deposit(int event, int vol, double e)
  {
    retired += e;
    if (vol < 0 || vol >= nvol || e == 0.0) return;
    if (event < 0 || event >= nevents) { // a primary with an event index outside the tally
      err |= kErrEvent;
      return;
    }
    int bin = event * nvol + vol;
    if (bin < sm_bins)
      atomicAdd(&sm_edep[bin], e);
    else
      atomicAdd(&g_edep[bin], e);
  }
};

template <class R> struct Secs {
  int n;
  int type[2];
  R E[2], dir[2][3];
  // slot chosen by a branch, not an index, so the record stays in registers
  __device__ __forceinline__ void add(int ty, R e, const R *u)
  {
    if (n == 0) {
      type[0] = ty;
      E[0] = e;
      dir[0][0] = u[0];
      dir[0][1] = u[1];
      dir[0][2] = u[2];
    } else {
      type[1] = ty;
      E[1] = e;
      dir[1][0] = u[0];
      dir[1][1] = u[1];
      dir[1][2] = u[2];
    }
    ++n;
  }
};

// One helix sub-step of length s in a uniform field along z: the reference's
// ConstFieldHelixStepper::DoStep (magneticfield/ConstFieldHelixStepper.hpp:164-239)
// with B = (0, 0, Bz) substituted, where the field-direction terms vanish.
// With rn = p / (kB2C q |Bz|) (signed), phi = -s / rn and sB = sign(Bz):
//   x' = x + rn ((cos phi - 1) dy sB - sin phi dx),   dx' = cos phi dx + sin phi dy sB
//   y' = y + rn (-(cos phi - 1) dx sB - sin phi dy),  dy' = cos phi dy - sin phi dx sB
//   z' = z + s dz,                                     dz' = dz
// (the reference's R v equals rn (dx, dy) since sinVB = |(dx, dy)|), with
// cos phi - 1 = -2 sin^2(phi / 2), free of cancellation at small bending
// angles.  The rotation and the transverse displacement are computed in T, the
// displacement is added to the FP64 position.
__device__ __forceinline__ void sincos_t(float x, float *s, float *c) { sincosf(x, s, c); }
__device__ __forceinline__ void sincos_t(double x, double *s, double *c) { ::sincos(x, s, c); }

template <class T, bool FUSED>
__device__ __forceinline__ void helix_bz(T rn, T sB, double s, const double pos[3], const T dir[3], double np[3],
                                         T nd[3])
{
  const T phi = -(T)s / rn;
  T sh, ch;
  sincos_t(T(0.5) * phi, &sh, &ch);
  const T sinp = T(2) * sh * ch, cm1 = T(-2) * sh * sh, cosp = T(1) + cm1;
  np[2] = pos[2] + s * (double)dir[2];
  // FUSED (the FP32 kernels of the analytic navigator): which product of a sum is
  // fused is written out; left open it differed from one form of their loop to
  // another, and a float's last bit is another track.  The volume tree's kernels
  // fuse others, the same in each form.
  if constexpr (FUSED) {
    const float P = __fmul_rn(sinp, dir[0]), Q = __fmul_rn(sinp, dir[1]);
    np[0] = pos[0] + (double)(rn * __fmaf_rn(__fmul_rn(cm1, dir[1]), sB, -P));
    np[1] = pos[1] + (double)(rn * __fmaf_rn(__fmul_rn(-cm1, dir[0]), sB, -Q));
    nd[0] = __fmaf_rn(cosp, dir[0], __fmul_rn(Q, sB));
    nd[1] = __fmaf_rn(cosp, dir[1], -__fmul_rn(P, sB));
  } else {
    np[0] = pos[0] + (double)(rn * (cm1 * dir[1] * sB - sinp * dir[0]));
    np[1] = pos[1] + (double)(rn * (-cm1 * dir[0] * sB - sinp * dir[1]));
    nd[0] = cosp * dir[0] + sinp * dir[1] * sB;
    nd[1] = cosp * dir[1] - sinp * dir[0] * sB;
  }
  nd[2] = dir[2];
}

template <class R>
__device__ __forceinline__ void run_model(const Data &d, const Geom &g, Track<R> &t, int proc, Secs<R> &sec,
                                          Local &L)
{
  int mat = vol_material(g, t.vol);
  ModelParams mp;
  mp.mode = 1;
  mp.Z = (int)d.mat_Z[mat];
  mp.cut = 0.0;
  mp.density_factor = d.mat_dfactor[mat];
  mp.sb = d.sb + ((mat == 1) ? 2 : 1);
  Inter<R> io;
  io.E = t.E;
  io.dir[0] = t.dir[0];
  io.dir[1] = t.dir[1];
  io.dir[2] = t.dir[2];
  io.edep = R(0);
  io.status = 0;
  io.nsec = 0;
  int err = 0;
  Mrg rng = t.rng();
  if (t.type == 0) {
    if (proc == 0)
      kn_sample(rng, mp, io, &err);
    else if (proc == 1) {
      bh_sample(rng, mp, io, &err);
      if (io.nsec == 2) L.st[S_PAIR]++;
    } else
      sg_sample(rng, d, mp, io, &err);
  } else if (proc == 0) {
    mp.cut = d.cut_energy[1][mat];
    if (t.type == 1)
      mb_sample(rng, mp, io, &err);
    else
      bhabha_sample(rng, mp, io, &err);
  } else if (proc == 1) {
    mp.cut = d.cut_energy[0][mat];
    sb_sample(rng, mp, io, &err);
  } else {
    annih_sample(rng, io, &err);
    L.st[S_ANNIH]++;
  }
  t.set_rng(rng);
  if (err) {
    L.err |= err;
    L.st[S_ERR]++;
  }
  L.deposit(t.event, t.vol, (double)io.edep);
  t.E = io.E;
  t.dir[0] = io.dir[0];
  t.dir[1] = io.dir[1];
  t.dir[2] = io.dir[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    if (s >= io.nsec) break;
    if (g.charged_local && io.sec_type[s] != 0) {
      L.deposit(t.event, t.vol, (double)io.sec_E[s]);
      continue;
    }
    sec.add(io.sec_type[s], io.sec_E[s], io.sec_dir[s]);
  }
  if (io.status == 1) t.E = R(0);
}

// ------------------------------------------------------- multiple scattering
// Multiple scattering of e-/e+ (config msc = 1, or 2 with lateral
// displacement): the Urban model as published
// (L. Urban, CERN-OPEN-2006-077); the reference has only a placeholder
// (proxy/ProxyScattering.hpp:53-71) and ships the transport mean free path
// tables (LambdaMod1.msc: E^2 / lambda1).  The oracle restates the same model
// in the same order of random draws.
//   step limit: t <= max(0.04 r0, 0.6 safety, 1e-5 mm), r0 = max(range,
//     lambda1) at the first step in each volume;
//   paths: geometric z = lambda1 (1 - exp(-t / lambda1)) from the true length t,
//     and back when a boundary stops the step;
//   deflection after the along-step loss: cos(theta) from the model's mixture
//     of a central exponential part (Highland-type width theta0), a power tail
//     and a uniform part, weighted so that <cos theta> = exp(-tau); where the
//     published weights would need a uniform part above 1 it is dropped and
//     the central / tail split keeps that mean; phi uniform;
//   lateral displacement (msc = 2), after a step that ends inside its volume:
//     r = 0.73 r_max, r_max = sqrt(t^2 - z^2) the largest displacement the
//     true and geometric lengths allow (the fixed fraction of early versions
//     of the model), perpendicular to the direction at the start of the step,
//     at the azimuth of the deflection (the displacement follows the turn),
//     cut to 0.99 of the safety at the end point so that it never crosses a
//     boundary, and none within 1e-5 mm of one.
// Not modelled: the e+ correction of theta0.
constexpr double kMscFr = 0.04, kMscFs = 0.6, kMscTmin = 1.0e-5;
constexpr double kMscTauBig = 8.0, kMscTauSmall = 1.0e-16, kMscTauLim = 1.0e-6;

// transport mean free path lambda1 (mm); 0 when the table has nothing
template <class R> __device__ __forceinline__ R msc_lambda1(const Data &d, int type, int mat, R e)
{
  const R v = tab_value<R>(d, d.vec[type == 2 ? GX_LambdaMod1_msc_ep : GX_LambdaMod1_msc_em][mat], e);
  return v > R(0) ? e * e / v : R(0);
}

template <class R> __device__ __forceinline__ R msc_expm1(R x);
template <> __device__ __forceinline__ float msc_expm1(float x) { return expm1f(x); }
template <> __device__ __forceinline__ double msc_expm1(double x) { return dexpm1(x); }
template <class R> __device__ __forceinline__ R msc_log1p(R x);
template <> __device__ __forceinline__ float msc_log1p(float x) { return log1pf(x); }
template <> __device__ __forceinline__ double msc_log1p(double x) { return dlog1p(x); }

template <class R> __device__ __forceinline__ double msc_true_to_geom(double t, R lam)
{
  const R tau = (R)t / lam;
  return tau < R(kMscTauLim) ? t : -(double)lam * (double)msc_expm1<R>(-tau);
}

template <class R> __device__ __forceinline__ double msc_geom_to_true(double z, R lam, double tmax)
{
  const R x = (R)z / lam;
  if (x < R(kMscTauLim)) return z;
  const double t = x < R(1) ? -(double)lam * (double)msc_log1p<R>(-x) : tmax;
  return t < tmax ? t : tmax;
}

// the model's two-function form for large angles: exact first and second moments
template <class R> __device__ __forceinline__ R msc_simple(Mrg &rng, R xm, R x2m)
{
  const R a = (R(2) * xm + R(9) * x2m - R(3)) / (R(2) * xm - R(3) * x2m + R(1));
  const R prob = (a + R(2)) * xm / a;
  const R r0 = rng.template u<R>(), r1 = rng.template u<R>();
  if (r0 < prob) return R(-1) + R(2) * M<R>::exp(M<R>::log(r1) / (a + R(1)));
  return R(-1) + R(2) * r1;
}

// cos(theta) after a true path t; lam0 / lam1 and e0 / e1 at the start and
// the end of the step; c = the material's constants {X0, th1, th2, ca..cd}
template <class R>
__device__ __forceinline__ R msc_cos_theta(Mrg &rng, const double *c, R t, R lam0, R lam1, R e0, R e1)
{
  R tau = t / lam0;
  if (lam1 > R(0) && fabs(lam1 - lam0) > R(0.01) * lam0) tau = t * M<R>::log(lam0 / lam1) / (lam0 - lam1);
  if (tau >= R(kMscTauBig)) return R(-1) + R(2) * rng.template u<R>();
  if (tau < R(kMscTauSmall)) return R(1);
  R xm, x2m;
  if (tau < R(0.01)) {
    xm = R(1) - tau * (R(1) - R(0.5) * tau);
    x2m = R(1) - tau * (R(5) - R(6.25) * tau) / R(3);
  } else {
    xm = M<R>::exp(-tau);
    x2m = (R(1) + R(2) * M<R>::exp(R(-2.5) * tau)) / R(3);
  }
  if (R(1) - e1 / e0 > R(0.5)) return msc_simple<R>(rng, xm, x2m);
  const R m = R(kEMass);
  const R inv0 = (e0 + m) / (e0 * (e0 + R(2) * m)), inv1 = (e1 + m) / (e1 * (e1 + R(2) * m));
  const R X0 = (R)c[0], y = t / X0;
  const R th0 = R(13.6) * M<R>::sqrt(y) * M<R>::sqrt(inv0 * inv1) * ((R)c[1] + (R)c[2] * M<R>::log(y));
  const R th2 = th0 * th0;
  if (th2 < R(kMscTauSmall)) return R(1);
  if (th0 > R(kPi / 6)) return msc_simple<R>(rng, xm, x2m);
  R x = th2 * (R(1) - th2 / R(12));
  if (th2 > R(0.01)) {
    const R s = R(2) * M<R>::sinr(R(0.5) * th0);
    x = s * s;
  }
  const R u = M<R>::exp(M<R>::log(tau) / R(6));
  R xsi = (R)c[3] + u * ((R)c[4] + (R)c[5] * u) + (R)c[6] * M<R>::log((t / tau) / X0);
  if (xsi < R(1.9)) xsi = R(1.9);
  R cc = xsi;
  if (fabs(cc - R(3)) < R(0.001))
    cc = R(3.001);
  else if (fabs(cc - R(2)) < R(0.001))
    cc = R(2.001);
  const R c1 = cc - R(1);
  const R ea = M<R>::exp(-xsi), eaa = R(1) - ea;
  const R xmean1 = R(1) - (R(1) - (R(1) + xsi) * ea) * x / eaa;
  if (xmean1 <= R(0.999) * xm) return msc_simple<R>(rng, xm, x2m);
  const R x0 = R(1) - xsi * x;
  const R b = R(1) + (cc - xsi) * x, b1 = b + R(1), bx = cc * x;
  const R dd = M<R>::exp(c1 * M<R>::log(bx)) / M<R>::exp(c1 * M<R>::log(b1));
  const R xmean2 = (x0 + dd - (bx - b1 * dd) / (cc - R(2))) / (R(1) - dd);
  const R f1x0 = ea / eaa, f2x0 = c1 / (cc * (R(1) - dd));
  R prob = f2x0 / (f1x0 + f2x0);
  R qprob = xm / (prob * xmean1 + (R(1) - prob) * xmean2);
  if (qprob > R(1)) {
    qprob = R(1);
    prob = (xm - xmean2) / (xmean1 - xmean2);
  }
  const R r0 = rng.template u<R>(), r1 = rng.template u<R>();
  if (r0 < qprob) {
    if (r1 < prob) return R(1) + M<R>::log(ea + rng.template u<R>() * eaa) * x;
    R var = (R(1) - dd) * rng.template u<R>();
    if (var < R(0.01) * dd) {
      var /= dd * c1;
      return R(-1) + var * (R(1) - R(0.5) * var * cc) * (R(2) + (cc - xsi) * x);
    }
    return R(1) + x * (cc - xsi - cc * M<R>::exp(-M<R>::log(var + dd) / c1));
  }
  return R(-1) + R(2) * r1;
}

// deflect the direction by the sampled angle (no draw for phi when it is 0)
template <class R>
// Returns false when the direction is kept (no azimuth drawn); sp, cp: the
// azimuth of the deflection.
__device__ __forceinline__ bool msc_deflect(const Data &d, Track<R> &t, int mat, R step, R lam0, R e0, R &sp, R &cp)
{
  const R lam1 = msc_lambda1<R>(d, t.type, mat, t.E);
  Mrg rng = t.rng();
  R ct = msc_cos_theta<R>(rng, d.mat_msc[mat], step, lam0, lam1, e0, t.E);
  if (!(ct < R(1))) {
    t.set_rng(rng);
    return false;
  }
  if (ct < R(-1)) ct = R(-1);
  const R st = M<R>::sqrt((R(1) - ct) * (R(1) + ct));
  M<R>::sincos2pi(rng.template u<R>(), &sp, &cp);
  t.set_rng(rng);
  R u = st * cp, v = st * sp, w = ct;
  rotate_to_lab(u, v, w, t.dir[0], t.dir[1], t.dir[2]);
  t.dir[0] = u;
  t.dir[1] = v;
  t.dir[2] = w;
  return true;
}

// The lateral displacement of a multiple-scattering step that ended inside
// its volume (config msc = 2): 0.73 sqrt(t^2 - z^2) perpendicular to the
// step's starting direction (d0, d1, d2) at the deflection's azimuth, cut to
// 0.99 of the safety at the end point, none within kMscTmin of a boundary.
// Out of line: the common path (msc 0 or 1) carries only the call.
template <class R, int K>
__device__ __noinline__ double3 msc_displacement(const Geom &g, int vol, double x, double y, double z, double t,
                                                 double zg, R cp, R sp, R d0, R d1, R d2)
{
  double3 out = make_double3(0.0, 0.0, 0.0);
  const double rmax2 = (t - zg) * (t + zg);
  if (!(rmax2 > 0.0)) return out;
  const double p[3] = {x, y, z};
  const double saf = nav_safety<K>(g, vol, p);
  if (!(saf > kMscTmin)) return out;
  const double r = fmin(0.73 * sqrt(rmax2), 0.99 * saf);
  R u = cp, v = sp, w = R(0);
  rotate_to_lab(u, v, w, d0, d1, d2);
  out.x = r * (double)u;
  out.y = r * (double)v;
  out.z = r * (double)w;
  return out;
}

#ifndef GX_PARITY
// Whether an electron of energy e that starts at pos in volume vol comes to rest
// in its first step there unless it interacts: its step limit is its range (the
// range is below the step function's final range) and nothing of the volume's
// surface is within it.  Such a step is one straight or helix move that stays in
// the volume and deposits all of e there, whatever the direction (step_gpil,
// field_substep: safety above the remaining length; along_loss: step >= range).
// The margin is far above the move's rounding and the navigator's snap distance.
// range: the step.  S: the solids of the volume tree (0: the analytic volumes).
template <class R, int S>
__device__ __forceinline__ bool stops_at_once(const Data &d, const Geom &g, int vol, const double *pos, int mat, R e,
                                              R &range)
{
  R raw;
  range = range_limit<R>(d, 1, mat, e, raw);
  const R cut = (R)d.cut_length[1][mat], finR = (R(10.0) < cut) ? R(10.0) : cut;
  if (e < R(kMinE)) raw *= e / R(kMinE);
  if (!(raw <= finR)) return false;
  double saf;
  if constexpr (S != 0)
    saf = csg_safety<S>(g.csg, vol, pos);
  else
    saf = safety(g, vol, pos);
  return saf > 1.0001 * (double)range + 2e-6;
}
#endif

enum { kDone = 0, kAlive = 1, kInteract = 2 };

// One OneStep (test_BasicCpuTransport.cpp:408-497 / InnerStep :358-403) in
// physics mode, up to the choice of the post-step interaction, in three
// phases so that a kernel can interleave tracks at different points of their
// steps: step_begin (GPIL and the step limit; a straight-line move completes
// here), field_substep (one helix sub-step, repeated until the step ends) and
// step_end (NIL update, continuous loss, outcome).  The state carried from one
// phase to the next:
template <class R> struct StepCtx {
  // macroscopic cross sections at the start of the step (scalars: an array
  // member of a structure that lives across loop passes ends up in local
  // memory)
  R xs0, xs1, xs2;
  double remaining; // helix: length of the step still to go
  double total;     // length travelled in this step
  int sel;          // process that limits the step (-1: none)
  int vol0;         // volume at the start of the step
  int newvol;       // volume entered (-2: sub-step cap hit)
  int nsub;         // helix sub-steps taken
  bool crossed;     // the step ended on a boundary
  // multiple scattering (lam0 > 0 when it applies to this step): transport
  // mean free path and energy at the start, the step's true length
  R lam0, e0;
  double ttrue;
  R range0; // charged: the range table's value at the step's energy (-1: none)
  __device__ __forceinline__ R xs(int i) const { return i == 0 ? xs0 : (i == 1 ? xs1 : xs2); }
};

// A photon's cross sections in the two calorimeter materials while its energy
// does not change (it stays in a transport kernel until it interacts):
// computed at its first step in each material, reused after.
template <class R> struct GammaXs {
  R pb0, pb1, pb2, ar0, ar1, ar2;
  int have; // bit 0: lead (material 1), bit 1: argon (material 2)
};

// The NILs a track at its GPIL lacks: a primary's, or one that a step stopped by
// a boundary used up to rounding.  Out of line, and copies passed so that the
// track stays in registers: tracks come with their NILs drawn (draw_nils).
template <class R> struct NilDraw {
  R nil[3];
  uint32_t rs[6];
};
template <class R> __device__ __noinline__ void redraw_nils_of(NilDraw<R> *n, int type);
template <class R> __device__ __forceinline__ void redraw_nils(Track<R> &t)
{
  NilDraw<R> n;
#pragma unroll
  for (int i = 0; i < 3; ++i) n.nil[i] = t.nil[i];
#pragma unroll
  for (int k = 0; k < 6; ++k) n.rs[k] = t.rs[k];
  redraw_nils_of(&n, t.type);
#pragma unroll
  for (int i = 0; i < 3; ++i) t.nil[i] = n.nil[i];
#pragma unroll
  for (int k = 0; k < 6; ++k) t.rs[k] = n.rs[k];
}

// GPIL and step limit (PostStepGPIL of the discrete processes, the range and
// multiple-scattering limits): returns the step to move (geometric length),
// and sets the step context.  gx, when given, caches a photon's cross
// sections per material.
template <class R, int K>
__device__ __forceinline__ R step_gpil(const Data &d, const Geom &g, Track<R> &t, StepCtx<R> &c,
                                       GammaXs<R> *gx = nullptr)
{
  const int mat = vol_material(g, t.vol);
  const int np = (t.type == 1) ? 2 : 3;
  const bool charged = t.type != 0;
  R xs[3];
  if (gx && mat == 1 && (gx->have & 1)) {
    xs[0] = gx->pb0;
    xs[1] = gx->pb1;
    xs[2] = gx->pb2;
  } else if (gx && mat == 2 && (gx->have & 2)) {
    xs[0] = gx->ar0;
    xs[1] = gx->ar1;
    xs[2] = gx->ar2;
  } else {
    cross_sections<R>(d, t.type, mat, t.E, xs);
    if (gx && mat == 1) {
      gx->pb0 = xs[0];
      gx->pb1 = xs[1];
      gx->pb2 = xs[2];
      gx->have |= 1;
    } else if (gx && mat == 2) {
      gx->ar0 = xs[0];
      gx->ar1 = xs[1];
      gx->ar2 = xs[2];
      gx->have |= 2;
    }
  }
  c.xs0 = xs[0];
  c.xs1 = xs[1];
  c.xs2 = xs[2];
  // loops over the three process slots are unrolled with the bound as a guard,
  // so xs[] and nil[] are indexed by constants and stay in registers
  bool draw = false;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < np && t.nil[i] <= R(0)) draw = true;
  if (draw) redraw_nils(t);
  R pstep = R(3.0e38);
  int sel = -1;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < np && xs[i] > R(0)) {
      R s = t.nil[i] / xs[i];
      if (s < pstep) {
        pstep = s;
        sel = i;
      }
    }
  c.range0 = R(-1);
  if (charged) {
    R slim = range_limit<R>(d, t.type, mat, t.E, c.range0);
    if (slim < pstep) {
      pstep = slim;
      sel = -1;
    }
  }
  // multiple scattering: its step limit, then the true step becomes the
  // geometric length to move
  c.lam0 = R(0);
  c.e0 = t.E;
  if ((K & kKindMsc) != 0 && charged) {
    const R lam0 = msc_lambda1<R>(d, t.type, mat, t.E);
    if (t.msc_r0 <= R(0)) {
      R range = tab_value<R>(d, d.vec[t.type == 2 ? GX_Range_ep : GX_Range_em][mat], t.E);
      if (t.E < R(kMinE)) range *= t.E / R(kMinE);
      t.msc_r0 = range > lam0 ? range : lam0;
    }
    const double tlim = fmax(fmax(kMscFr * (double)t.msc_r0, kMscFs * nav_safety<K>(g, t.vol, t.pos)), kMscTmin);
    if (tlim < (double)pstep) {
      pstep = (R)tlim;
      sel = -1;
    }
    c.ttrue = (double)pstep;
    if (lam0 > R(0)) {
      c.lam0 = lam0;
      pstep = (R)msc_true_to_geom<R>((double)pstep, lam0);
    }
  }
  c.sel = sel;
  c.vol0 = t.vol;
  c.newvol = t.vol;
  c.crossed = false;
  c.nsub = 0;
  return pstep;
}

// The start of the move by pstep: true when the step continues with helix
// sub-steps (a charged track in a field); otherwise the straight move to pstep
// or the first boundary is made here and false returned.
template <class R, int K>
__device__ __forceinline__ bool step_move_begin(const Geom &g, Track<R> &t, StepCtx<R> &c, R pstep)
{
  if (t.type != 0 && (g.Bz != 0.0 || g.field_map)) {
    c.remaining = (double)pstep;
    c.total = 0.0;
    return true;
  }
  int plane;
  double dir[3] = {(double)t.dir[0], (double)t.dir[1], (double)t.dir[2]};
  double ps = (double)pstep;
  double dd = nav_distance<K, sizeof(R) == 4>(g, t.vol, t.pos, dir, ps, plane);
  if (dd < ps) {
    c.total = dd;
    c.crossed = true;
    if constexpr ((K & kKindCsg) != 0) {
      for (int k = 0; k < 3; ++k) t.pos[k] += dd * dir[k];
      c.newvol = csg_cross<kSolidsOf<K>>(g.csg, t.vol, plane, t.pos, dir);
    } else {
      c.newvol = next_volume(g, t.vol, plane);
      for (int k = 0; k < 3; ++k) t.pos[k] += dd * dir[k];
      if (plane != 2) {
        double lo, hi;
        slab_bounds(g, t.vol, lo, hi);
        set_comp(t.pos, g.axis, plane > 0 ? hi : lo);
      }
    }
  } else {
    c.total = ps;
    for (int k = 0; k < 3; ++k) t.pos[k] += ps * dir[k];
  }
  return false;
}

// GPIL, step limit and the start of the move.  Returns true when the step
// continues with helix sub-steps (a charged track in a field), false when it
// is complete.
template <class R, int K>
__device__ __forceinline__ bool step_begin(const Data &d, const Geom &g, Track<R> &t, StepCtx<R> &c,
                                           GammaXs<R> *gx = nullptr)
{
  const R pstep = step_gpil<R, K>(d, g, t, c, gx);
  return step_move_begin<R, K>(g, t, c, pstep);
}

// One helix sub-step in Bz (FieldPropagationHandler::Propagate /
// PropagateInVolume, magneticfield/src/FieldPropagationHandler.cpp:87-360).
// Positions, the geometry and the step bookkeeping are FP64; the direction,
// the momentum and the sub-step length heuristic are in R (FP32 in the mixed
// build).  Returns true when the step is complete (boundary reached, length
// used up, or the cap of 10000 sub-steps hit: then newvol = -2).
// One classical fourth-order Runge-Kutta step of length s through the field
// map (FP64): position x and unit direction u with du/ds = k u x B(x),
// k = 0.299792458 q / p (MeV, T, mm); four map lookups, direction renormalised.
__device__ __forceinline__ void rk4_map_step(const float4 *__restrict__ fmap, double k, double s, double x[3],
                                             double u[3], const double B0[3])
{
  double xs[3], us[3], B[3], kx[4][3], ku[4][3];
  const double h[3] = {0.5 * s, 0.5 * s, s};
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    kx[0][j] = u[j];
  }
  ku[0][0] = k * (u[1] * B0[2] - u[2] * B0[1]);
  ku[0][1] = k * (u[2] * B0[0] - u[0] * B0[2]);
  ku[0][2] = k * (u[0] * B0[1] - u[1] * B0[0]);
#pragma unroll
  for (int st = 1; st < 4; ++st) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      xs[j] = x[j] + h[st - 1] * kx[st - 1][j];
      us[j] = u[j] + h[st - 1] * ku[st - 1][j];
    }
    field_map_value(fmap, xs, B);
#pragma unroll
    for (int j = 0; j < 3; ++j) kx[st][j] = us[j];
    ku[st][0] = k * (us[1] * B[2] - us[2] * B[1]);
    ku[st][1] = k * (us[2] * B[0] - us[0] * B[2]);
    ku[st][2] = k * (us[0] * B[1] - us[1] * B[0]);
  }
  double m = 0.0;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    x[j] += s / 6.0 * (kx[0][j] + 2.0 * kx[1][j] + 2.0 * kx[2][j] + kx[3][j]);
    u[j] += s / 6.0 * (ku[0][j] + 2.0 * ku[1][j] + 2.0 * ku[2][j] + ku[3][j]);
    m += u[j] * u[j];
  }
  m = 1.0 / ::sqrt(m);
  u[0] *= m;
  u[1] *= m;
  u[2] *= m;
}

// One sub-step through the field map: the sub-step length from the same
// geometry and sagitta limits as the helix (with the field at the start
// point), then a Runge-Kutta step.  Returns the length moved.
template <class R>
__device__ __forceinline__ double field_map_substep(const Data &d, const Geom &g, Track<R> &t, double remaining,
                                                    double saf, double snext)
{
  const double eps = 0.1, charge = (t.type == 1) ? -1.0 : 1.0;
  const double E = (double)t.E, p = ::sqrt(E * (E + 2.0 * kEMass));
  double B0[3], u[3] = {(double)t.dir[0], (double)t.dir[1], (double)t.dir[2]};
  field_map_value(d.fmap, t.pos, B0);
  const double cx = u[1] * B0[2] - u[2] * B0[1], cy = u[2] * B0[0] - u[0] * B0[2], cz = u[0] * B0[1] - u[1] * B0[0];
  const double bperp = ::sqrt(cx * cx + cy * cy + cz * cz); // |u x B|
  double step_field = 1.7976931348623157e308;
  if (bperp > 0.0) step_field = fmax(2.0 * ::sqrt(eps * p / (0.299792458 * bperp)), saf);
  const double step_gp = fmax(fmin(remaining, 1e-4), snext);
  const double s = fmin(fmin(step_gp, step_field), remaining);
  if (bperp > 0.0) {
    rk4_map_step(d.fmap, 0.299792458 * charge / p, s, t.pos, u, B0);
    for (int k = 0; k < 3; ++k) t.dir[k] = (R)u[k];
  } else {
    for (int k = 0; k < 3; ++k) t.pos[k] += s * u[k];
  }
  return s;
}

// K: the kernel variant (kKindFieldMap, kKindCsg, kKindMsc bits).
template <class R, int K>
__device__ __forceinline__ bool field_substep(const Data &d, const Geom &g, Track<R> &t, StepCtx<R> &c, Local &L)
{
  const R eps = R(0.1); // gEpsDeflection = 1e-2 cm
  const R charge = (t.type == 1) ? R(-1) : R(1);
  const R p = M<R>::sqrt(t.E * (t.E + R(2.0 * kEMass)));
  const R absB = (R)fabs(g.Bz), sB = g.Bz >= 0.0 ? R(1) : R(-1);
  const R curv_per_pt = R(0.299792458) * absB; // 1 / radius = curv_per_pt / pt
  int plane;
  double dd[3] = {(double)t.dir[0], (double)t.dir[1], (double)t.dir[2]};
  const double remaining = c.remaining;
  double saf = nav_safety<K>(g, t.vol, t.pos);
  double snext = (saf > remaining)
                     ? remaining
                     : fmax(2e-9, fmin(nav_distance<K, sizeof(R) == 4>(g, t.vol, t.pos, dd, remaining, plane),
                                       remaining) + 2e-9);
  double s;
  if constexpr ((K & kKindFieldMap) != 0) {
    s = field_map_substep<R>(d, g, t, remaining, saf, snext);
  } else {
  double step_gp = fmax(fmin(remaining, 1e-4), snext);
  R pt = p * M<R>::sqrt(fmax(R(1) - t.dir[2] * t.dir[2], R(0)));
  double step_field = 1.7976931348623157e308;
#ifdef GX_PARITY
  // the oracle's form: the sagitta length from the curvature, the general
  // helix step, the direction renormalised by division
  if (pt > 0.0) {
    const double curv = 0.299792458 * fabs(g.Bz) / pt;
    step_field = fmax(2.0 * ::sqrt(eps / curv), saf);
  }
  s = fmin(fmin(step_gp, step_field), remaining);
  if (pt > 0.0) {
    const double B[3] = {0.0, 0.0, g.Bz};
    double np[3], nd[3];
    helix_dostep(kB2C_mm, B, t.pos, t.dir, (double)charge, p, s, np, nd);
    const double m = ::sqrt(nd[0] * nd[0] + nd[1] * nd[1] + nd[2] * nd[2]);
    for (int k = 0; k < 3; ++k) {
      t.pos[k] = np[k];
      t.dir[k] = nd[k] / m;
    }
  } else {
    for (int k = 0; k < 3; ++k) t.pos[k] += s * dd[k];
  }
#else
  if (pt > R(0)) step_field = fmax(2.0 * (double)M<R>::sqrt(eps * pt / curv_per_pt), saf);
  s = fmin(fmin(step_gp, step_field), remaining);
  if (pt > R(0)) {
    const R rn = p / (R(kB2C_mm) * charge * absB);
    double np[3];
    R nd[3];
    constexpr bool kFused = sizeof(R) == 4 && (K & kKindCsg) == 0;
    helix_bz<R, kFused>(rn, sB, s, t.pos, t.dir, np, nd);
    R n2;
    if constexpr (kFused)
      n2 = __fmaf_rn(nd[2], nd[2], __fmaf_rn(nd[1], nd[1], __fmul_rn(nd[0], nd[0])));
    else
      n2 = nd[0] * nd[0] + nd[1] * nd[1] + nd[2] * nd[2];
    const R inv = R(1) / M<R>::sqrt(n2);
    for (int k = 0; k < 3; ++k) {
      t.pos[k] = np[k];
      t.dir[k] = nd[k] * inv;
    }
  } else {
    for (int k = 0; k < 3; ++k) t.pos[k] += s * dd[k];
  }
#endif
  }
  c.total += s;
  c.remaining = remaining - s;
  L.st[S_SUBSTEPS]++;
  dd[0] = (double)t.dir[0];
  dd[1] = (double)t.dir[1];
  dd[2] = (double)t.dir[2];
  int v = nav_relocate<K>(g, t.vol, t.pos, dd);
  if (v != t.vol || c.remaining <= 1e-10) {
    if (v != t.vol) {
      c.crossed = true;
      c.newvol = v;
    }
    return true;
  }
  if (++c.nsub >= 10000) {
    L.err |= kErrFieldCap;
    L.st[S_ERR]++;
    c.crossed = true;
    c.newvol = -2;
    return true;
  }
  return false;
}

// NIL update, continuous loss and the outcome of the step: kDone (track
// finished), kAlive (no interaction this step) or kInteract with *proc set
// (for a stopped e+, proc 2 = annihilation at rest, at E = 0).
template <class R, int K>
__device__ __forceinline__ int step_end(const Data &d, const Geom &g, Track<R> &t, const StepCtx<R> &c, Local &L,
                                        int *proc)
{
  const int np = (t.type == 1) ? 2 : 3;
  // the true length of the step: all of it, or back from where a boundary
  // stopped it
  const bool msc = (K & kKindMsc) != 0 && c.lam0 > R(0); // multiple scattering applied to this step
  const double step = msc ? (c.crossed ? msc_geom_to_true<R>(c.total, c.lam0, c.ttrue) : c.ttrue) : c.total;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < np) t.nil[i] -= (R)step * c.xs(i);
  L.st[S_STEPS]++;
  if (c.newvol == -2) {
    L.deposit(t.event, c.vol0, (double)t.E);
    return kDone;
  }
  if (t.type != 0) {
    R eloss = along_loss<R>(d, t.type, vol_material(g, c.vol0), step, t.E, c.range0);
    L.deposit(t.event, c.vol0, (double)eloss);
    if (t.E <= R(0)) {
      if (t.type == 2) {
        int v = c.crossed ? c.newvol : c.vol0;
        if (v >= 0) {
          t.vol = v;
          t.E = R(0);
          *proc = 2;
          return kInteract;
        }
        L.escape(2.0 * kEMass);
      }
      return kDone;
    }
    if (msc) {
      const R d0 = t.dir[0], d1 = t.dir[1], d2 = t.dir[2]; // the direction the step started in
      R sp, cp;
      const bool turned = msc_deflect<R>(d, t, vol_material(g, c.vol0), (R)step, c.lam0, c.e0, sp, cp);
      if (g.msc == 2 && turned && !c.crossed) {
        const double3 dx =
            msc_displacement<R, K>(g, t.vol, t.pos[0], t.pos[1], t.pos[2], step, c.total, cp, sp, d0, d1, d2);
        t.pos[0] += dx.x;
        t.pos[1] += dx.y;
        t.pos[2] += dx.z;
      }
    }
  }
  if (c.crossed) {
    t.msc_r0 = R(-1); // a new volume: the step limit starts again
    t.vol = c.newvol;
    if (c.newvol < 0) {
      L.escape((double)t.E + ((t.type == 2) ? 2.0 * kEMass : 0.0));
      return kDone;
    }
    return kAlive;
  }
  if (c.sel >= 0) {
#pragma unroll
    for (int i = 0; i < 3; ++i)
      if (i == c.sel) t.nil[i] = R(-1);
    *proc = c.sel;
    return kInteract;
  }
  return kAlive;
}

// The three phases in sequence: one whole step up to the interaction.
template <class R, int K>
__device__ __forceinline__ int transport_part(const Data &d, const Geom &g, Track<R> &t, Local &L,
                                                                 int *proc)
{
  StepCtx<R> c;
  if (step_begin<R, K>(d, g, t, c))
    while (!field_substep<R, K>(d, g, t, c, L)) {
    }
  return step_end<R, K>(d, g, t, c, L, proc);
}

// The whole OneStep, interaction included (the fused form the plain loop
// runs); the oracle's one_step is the same algorithm in the same order of
// random draws.  Returns false when the track is finished.
template <class R, int K>
__device__ bool one_step(const Data &d, const Geom &g, Track<R> &t, Secs<R> &sec, Local &L)
{
  sec.n = 0;
  int proc = -1;
  int r = transport_part<R, K>(d, g, t, L, &proc);
  if (r == kInteract) {
    run_model(d, g, t, proc, sec, L);
    return t.E > R(0);
  }
  return r == kAlive;
}

// ------------------------------------------------------------- load / store
// A record as 32-bit words in registers (constant indices only).
template <class R> struct RecWords {
  static constexpr int kWords = (int)(sizeof(Rec<R>) / 4), kR = (int)(sizeof(R) / 4);
  uint32_t w[kWords];
  __device__ __forceinline__ double get64(int k) const { return __hiloint2double((int)w[k + 1], (int)w[k]); }
  __device__ __forceinline__ void put64(int k, double v)
  {
    w[k] = (uint32_t)__double2loint(v);
    w[k + 1] = (uint32_t)__double2hiint(v);
  }
  __device__ __forceinline__ R real(int k) const // k-th of the R members
  {
    if constexpr (sizeof(R) == 8)
      return get64(6 + 2 * k);
    else
      return __uint_as_float(w[6 + k]);
  }
  __device__ __forceinline__ void real(int k, R v)
  {
    if constexpr (sizeof(R) == 8)
      put64(6 + 2 * k, v);
    else
      w[6 + k] = __float_as_uint(v);
  }
};

template <class R> __device__ __forceinline__ void load_rec(const Rec<R> *p, Track<R> &t)
{
  RecWords<R> u;
  const uint4 *q = reinterpret_cast<const uint4 *>(p);
#pragma unroll
  for (int k = 0; k < u.kWords / 4; ++k) {
    const uint4 v = q[k];
    u.w[4 * k] = v.x;
    u.w[4 * k + 1] = v.y;
    u.w[4 * k + 2] = v.z;
    u.w[4 * k + 3] = v.w;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    t.pos[k] = u.get64(2 * k);
    t.dir[k] = u.real(k);
    t.nil[k] = u.real(4 + k);
  }
  t.E = u.real(3);
  t.msc_r0 = u.real(7);
  constexpr int o = 6 + 8 * RecWords<R>::kR;
#pragma unroll
  for (int k = 0; k < 6; ++k) t.rs[k] = u.w[o + k];
  t.vol = (int)u.w[o + 6];
  t.event = (int)u.w[o + 7];
  t.prim = (int)u.w[o + 8];
  t.type = (int)u.w[o + 9];
}
template <class R> __device__ __forceinline__ void store_rec(Rec<R> *p, const Track<R> &t)
{
  RecWords<R> u;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    u.put64(2 * k, t.pos[k]);
    u.real(k, t.dir[k]);
    u.real(4 + k, t.nil[k]);
  }
  u.real(3, t.E);
  u.real(7, t.msc_r0);
  constexpr int o = 6 + 8 * RecWords<R>::kR;
#pragma unroll
  for (int k = 0; k < 6; ++k) u.w[o + k] = t.rs[k];
  u.w[o + 6] = (uint32_t)t.vol;
  u.w[o + 7] = (uint32_t)t.event;
  u.w[o + 8] = (uint32_t)t.prim;
  u.w[o + 9] = (uint32_t)t.type;
  uint4 *q = reinterpret_cast<uint4 *>(p);
#pragma unroll
  for (int k = 0; k < u.kWords / 4; ++k)
    q[k] = make_uint4(u.w[4 * k], u.w[4 * k + 1], u.w[4 * k + 2], u.w[4 * k + 3]);
}

template <class R> __device__ __forceinline__ void load_track(const Store<R> &s, long long i, int ptype, Track<R> &t)
{
  load_rec(s.rec + i, t);
  if (ptype < 3) t.type = ptype; // known to the compiler
}

template <class R> __device__ __forceinline__ void store_track(const Store<R> &s, long long i, const Track<R> &t)
{
  store_rec(s.rec + i, t);
}

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

__device__ __forceinline__ unsigned lanemask_lt() { return (1u << lane_id()) - 1u; }

// Reserve cnt[q] consecutive slots per lane (0 to 3: a survivor and up to two
// secondaries) in each of the counters ctr[q], q < nq <= 3: next[q] becomes this
// lane's first slot.  The lanes' counts go in as two ballots per counter (their
// bits 0 and 1), so the exclusive prefix is two popcounts; lane q adds to
// counter q, so the three additions are in flight together instead of each
// waiting for the one before.
__device__ __forceinline__ void warp_reserve3(unsigned long long *ctr, int nq, const int cnt[3], long long next[3])
{
  unsigned b0[3], b1[3];
  int mine = 0;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    b0[q] = __ballot_sync(0xffffffffu, cnt[q] & 1);
    b1[q] = __ballot_sync(0xffffffffu, cnt[q] & 2);
    if ((int)lane_id() == q && q < nq) mine = __popc(b0[q]) + 2 * __popc(b1[q]);
  }
  unsigned long long base = 0;
  if (mine) base = atomicAdd(ctr + lane_id(), (unsigned long long)mine);
  const unsigned lt = lanemask_lt();
#pragma unroll
  for (int q = 0; q < 3; ++q)
    next[q] = (long long)__shfl_sync(0xffffffffu, base, q) + __popc(b0[q] & lt) + 2 * __popc(b1[q] & lt);
}

// Write a track to store q, or to q's overflow stack when the store is full.
template <class R> __device__ __forceinline__ void put_track(const Args<R> &a, int q, long long idx, const Track<R> &t, Local &L)
{
  const Store<R> &s = a.st[a.ctl->parity ^ 1][q];
  if (idx < s.cap) {
    store_track(s, idx, t);
    return;
  }
  unsigned long long j = atomicAdd((unsigned long long *)&a.ctl->stack_count[q], 1ULL);
  if ((long long)j < a.stack[q].cap) {
    store_track(a.stack[q], (long long)j, t);
  } else {
    // no room anywhere: the track is retired and its energy scored where it is
    L.err |= kErrOverflow;
    L.st[S_OVERFLOW]++;
    L.deposit(t.event, t.vol, (double)t.E);
  }
}

// ----------------------------------------------------------------- kernels
// Event row 0 of the tally lives in shared memory when it fits.  (The bins in
// several copies, so that fewer lanes of a warp meet on one, were no gain: 8
// copies of 100 bins 135.7 against 134.2 ms for 20000 showers.)
constexpr int kTallyDoubles = 768;

// Shared-memory tally and block statistics of one step kernel.
__device__ __forceinline__ void tally_begin(Local &L, const Geom &g, double *edep, double *sm_edep,
                                            unsigned long long *sm_stat, double *sm_esc, int *sm_err)
{
  L.nvol = g.nvol;
  L.nevents = g.nevents;
  L.g_edep = edep;
  L.sm_edep = sm_edep;
  L.sm_esc = sm_esc;
  L.sm_bins = (g.nvol <= kTallyDoubles) ? g.nvol : 0;
  for (int k = threadIdx.x; k < L.sm_bins; k += blockDim.x) sm_edep[k] = 0.0;
  for (int k = threadIdx.x; k < kNStat; k += blockDim.x) sm_stat[k] = 0;
  if (threadIdx.x == 0) {
    sm_esc[0] = sm_esc[1] = 0.0;
    *sm_err = 0;
  }
  __syncthreads();
  L.retired = 0.0;
  L.err = 0;
#pragma unroll
  for (int k = 0; k < kNStat; ++k) L.st[k] = 0;
}

// The sum of v over the lanes that are here, added to *ctr by one of them: a
// 64-bit (or FP64) addition in shared memory is a compare-and-swap loop, and
// every thread's own at the end of a block kept it there longer than an
// interaction's sampling did.
__device__ __forceinline__ void add_warp(unsigned long long *ctr, unsigned int v)
{
  const unsigned m = __activemask();
  const unsigned sum = __reduce_add_sync(m, v);
  if ((int)lane_id() == __ffs(m) - 1) atomicAdd(ctr, (unsigned long long)sum);
}

// steps_slot >= 0: the stat that also receives this kernel's step count
__device__ __forceinline__ void tally_end(Local &L, Ctl *ctl, double *edep, double *sm_edep,
                                          unsigned long long *sm_stat, double *sm_esc, int *sm_err,
                                          int steps_slot = -1)
{
#pragma unroll
  for (int k = 0; k < kNStat; ++k)
    if (L.st[k]) add_warp(&sm_stat[k], L.st[k]);
  if (steps_slot >= 0 && L.st[S_STEPS]) add_warp(&sm_stat[steps_slot], L.st[S_STEPS]);
  __syncwarp();
  double retired = L.retired;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) retired += __shfl_xor_sync(0xffffffffu, retired, o);
  if (lane_id() == 0 && retired != 0.0) atomicAdd(&sm_esc[1], retired);
  if (L.err) atomicOr(sm_err, L.err);
  __syncthreads();
  for (int k = threadIdx.x; k < L.sm_bins; k += blockDim.x)
    if (sm_edep[k] != 0.0) atomicAdd(&edep[k], sm_edep[k]);
  for (int k = threadIdx.x; k < kNStat; k += blockDim.x)
    if (sm_stat[k]) atomicAdd(&ctl->stat[k], sm_stat[k]);
  if (threadIdx.x == 0) {
    if (sm_esc[0] != 0.0) atomicAdd(&ctl->escaped, sm_esc[0]);
    if (sm_esc[1] != 0.0) atomicAdd(&ctl->retired, sm_esc[1]);
    if (*sm_err) atomicOr(&ctl->err_flags, *sm_err);
  }
}

// Element q of a 3-array by unrolled compare, so the array stays in registers.
template <class T> __device__ __forceinline__ T take3(T (&v)[3], int q, T inc)
{
  T r = 0;
#pragma unroll
  for (int j = 0; j < 3; ++j)
    if (j == q) {
      r = v[j];
      v[j] += inc;
    }
  return r;
}

// The NIL of every discrete process of track t that has none (<= 0), drawn
// from the track's stream in process order -- the draws its next GPIL would
// make first.  Drawn where a track is created or survives an interaction,
// right after the stream's other draws there, they are the same numbers in
// the same order on the same stream, and the transport kernels' GPIL then
// finds them set: the draws run convergently in the kernel that makes the
// tracks instead of for one or two lanes in most passes of a transport warp.
template <class R> __device__ __forceinline__ void draw_nils(Track<R> &t, Mrg &rng)
{
  const int np = (t.type == 1) ? 2 : 3;
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (i < np && t.nil[i] <= R(0)) t.nil[i] = -M<R>::log(rng.template u<R>());
}

template <class R> __device__ __noinline__ void redraw_nils_of(NilDraw<R> *n, int type)
{
  Track<R> t = {};
  t.type = type;
  for (int i = 0; i < 3; ++i) t.nil[i] = n->nil[i];
  for (int k = 0; k < 6; ++k) t.rs[k] = n->rs[k];
  Mrg rng = t.rng();
  draw_nils(t, rng);
  t.set_rng(rng);
  for (int i = 0; i < 3; ++i) n->nil[i] = t.nil[i];
  for (int k = 0; k < 6; ++k) n->rs[k] = t.rs[k];
}

// One store of cap records at `base + off` (off advances past it).
template <class R> inline Store<R> carve(uintptr_t base, size_t &off, long long cap)
{
  Store<R> s;
  s.cap = cap;
  s.rec = (Rec<R> *)(base + off);
  off += (cap * sizeof(Rec<R>) + 255) & ~size_t(255);
  return s;
}

// The variant of the step kernels for a geometry and field (kKind* bits).
template <class R> inline int kernel_kind(const Geom &g)
{
  const bool boxes = sizeof(R) == 4 && g.geometry == 2 && g.csg.solids == kSolidsBox;
  return (g.field_map ? kKindFieldMap : 0) | (g.geometry == 2 ? kKindCsg : 0) | (g.msc ? kKindMsc : 0) |
         (boxes ? kKindBoxes : 0);
}
// Geometry and options of a transport configuration, for the kernels.
inline void make_geom(const Ctx *C, const gx_transport_config *cfg, int nvol, Geom &g)
{
  std::memset(&g, 0, sizeof(g));
  g.geometry = cfg->geometry;
  g.axis = cfg->axis;
  g.nlayers = cfg->nlayers;
  g.box_mat = cfg->box_mat;
  g.charged_local = cfg->charged_local;
  g.nvol = nvol;
  g.nevents = cfg->nevents;
  g.t_abs = cfg->t_abs;
  g.pitch = cfg->t_abs + cfg->t_gap;
  g.x0 = -0.5 * cfg->nlayers * g.pitch;
  g.total = cfg->nlayers * g.pitch;
  g.half_trans = cfg->half_trans;
  g.Bz = cfg->Bz;
  g.msc = cfg->msc;
  g.field_map = cfg->field_map;
  for (int k = 0; k < 3; ++k) {
    g.box_half[k] = cfg->box_half[k];
    g.box_centre[k] = cfg->box_centre[k];
  }
}

#ifdef GX_PARITY
} // namespace parity
#endif
} // namespace gx
