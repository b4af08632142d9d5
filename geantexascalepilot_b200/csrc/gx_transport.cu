// gx_transport.cu -- the transport engine: every alive track takes one or more
// steps per iteration, in FP64 or FP32-mixed arithmetic.
//
// Layout in HBM: per particle type (gamma, e-, e+) two track stores of
// `capacity` records (current / next), one overflow stack and a buffer for each
// process.  A transport kernel reads the current store of its type and steps each
// track, in registers, until it interacts (then it goes to the process's buffer),
// ends, or has had its turn (then to the next store); an interaction kernel per
// process reads its buffer and writes survivors and secondaries to the next
// stores.  All are written at slots reserved per warp (ballots and one atomic for
// each destination), so stores stay compact and particle-pure without a separate
// compaction pass.  Tracks that do not fit go to the stack and are re-injected
// when the stores drain; primaries are injected on the device, with per-primary
// MRG32k3a substreams by skip-ahead, whenever fewer than `refill_below`
// tracks are in flight.  The launches of an iteration (refill, three transport
// kernels, eight interaction kernels on parallel branches, finish) are captured in
// a CUDA graph that repeats on the device while tracks are left.
//
// Times in the comments of this file and of gx_step.cuh, gx_device.cuh and
// gx_internal.cuh are ms per call on a B200 at 1965 MHz, with what is described and
// without it, all else as it was at that time.  "20000 showers": 10^4 electrons and
// 10^4 photons of 10 GeV, 50 layers, 4 T, FP32-mixed; "61 showers": 61 of them;
// "256 events": 25600 electrons of 10 GeV from host arrays, scored in 256 events;
// "two electrons": of 1 GeV, no field, FP64; "photons in lead": 10^4 of 10 MeV in a
// lead cube, no field, FP64.
//
// The "plain" engine runs the same step code as one kernel over one mixed
// store, launched and synchronised from the host every iteration, in FP64: the
// straightforward GPU loop the batched engine is measured against.
//
// The FP64 parity variant: gx_transport_parity.cu compiles this file a second
// time with GX_PARITY defined and without floating-point contraction, into
// namespace gx::parity (FP64 only).  There the step takes the reference's
// spline form for every table lookup, the reference's ionisation GPIL/DoIt,
// the general helix step (ConstFieldHelixStepper::DoStep) with the
// oracle's sub-step length, and the elementary functions of gx_math.h: the
// same operations, in the same order and rounding, as the oracle's step loop,
// so that the two agree track by track (gx_transport_config.fp64_parity).
#include "gx_step.cuh"

#include <algorithm>
#include <mutex>
#include <cmath>
#include <cstring>

namespace gx {
#ifdef GX_PARITY
namespace parity {
#define GX_ENGINE_OF(c) ((c)->parity_engine)
#define GX_RELEASE_ENGINE(c) ::gx::parity::release_engine(c)
#else
#define GX_ENGINE_OF(c) ((c)->engine)
#define GX_RELEASE_ENGINE(c) ::gx::release_engine(c)
#endif

// After a track's interaction: its secondaries (streams seeded from the
// parent, in order, their NILs drawn) and the survivor (its spent NIL drawn
// anew) go to the next stores, destination =
// particle type, or store 0 with one mixed store.  Every lane of the warp
// calls this (the slot reservations are warp-wide); `active` lanes write.
// SRC is the store the tracks were read from (for the write statistics).
template <class R, int SRC>
__device__ __forceinline__ void emit_tracks(const Args<R> &a, Ctl *ctl, int par, bool active, bool alive, Track<R> &t,
                                            const Secs<R> &sec, Local &L)
{
  const bool mixed = a.nstores == 1;
  int cnt[3] = {0, 0, 0};
  if (alive) take3(cnt, mixed ? 0 : t.type, 1);
#pragma unroll
  for (int k = 0; k < 2; ++k)
    if (k < sec.n) take3(cnt, mixed ? 0 : sec.type[k], 1);
  long long next[3];
  warp_reserve3((unsigned long long *)ctl->count[par ^ 1], a.nstores, cnt, next);
  if (!active) return;
  Mrg rng = t.rng();
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (k >= sec.n) break;
    Track<R> c;
    c.type = sec.type[k];
    c.pos[0] = t.pos[0];
    c.pos[1] = t.pos[1];
    c.pos[2] = t.pos[2];
    c.dir[0] = sec.dir[k][0];
    c.dir[1] = sec.dir[k][1];
    c.dir[2] = sec.dir[k][2];
    c.E = sec.E[k];
    c.nil[0] = c.nil[1] = c.nil[2] = R(-1);
    c.msc_r0 = R(-1);
    Mrg cr;
    rng.seed_child(cr);
    draw_nils(c, cr);
    c.set_rng(cr);
    c.vol = t.vol;
    c.event = t.event;
    c.prim = -1;
    const int q = mixed ? 0 : c.type;
    put_track(a, q, take3(next, q, 1LL), c, L);
    unsigned int sc[3] = {L.st[S_SEC0], L.st[S_SEC1], L.st[S_SEC2]};
    take3(sc, c.type, 1u);
    L.st[S_SEC0] = sc[0];
    L.st[S_SEC1] = sc[1];
    L.st[S_SEC2] = sc[2];
    L.st[S_WRITE0 + SRC]++;
  }
  if (alive) draw_nils(t, rng);
  t.set_rng(rng);
  if (alive) {
    const int q = mixed ? 0 : t.type;
    put_track(a, q, take3(next, q, 1LL), t, L);
    L.st[S_WRITE0 + SRC]++;
  }
}

// PT: particle type of the store (0, 1, 2), or 3 for the single mixed store.
// The fused step (transport and interaction in one kernel) of the plain loop.
template <class R, int PT, int K> __device__ __forceinline__ void step_body(const Args<R> &a)
{
  extern __shared__ double sm_edep[];
  __shared__ unsigned long long sm_stat[kNStat];
  __shared__ double sm_esc[2];
  __shared__ int sm_err;
  const Data &d = *a.d;
  Ctl *ctl = a.ctl;
  const int par = ctl->parity;
  constexpr int SRC = (PT < 3) ? PT : 0;
  const Store<R> &cur = a.st[par][SRC];
  const long long n = min(ctl->count[par][SRC], cur.cap);
  Local L;
  tally_begin(L, a.g, a.edep, sm_edep, sm_stat, sm_esc, &sm_err);
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x; base < n; base += stride) {
    long long i = base + threadIdx.x;
    bool active = i < n;
    Track<R> t;
    Secs<R> sec;
    sec.n = 0;
    bool alive = false;
    if (active) {
      load_track(cur, i, PT, t);
      L.st[S_READ0 + SRC]++;
      alive = one_step<R, K>(d, a.g, t, sec, L);
      if (t.prim >= 0 && a.pstep) atomicAdd(&a.pstep[t.prim], 1);
    }
    emit_tracks<R, SRC>(a, ctl, par, active, alive, t, sec, L);
  }
  tally_end(L, ctl, a.edep, sm_edep, sm_stat, sm_esc, &sm_err);
}

// Arguments by value (the allocation-free entry point) or from a device copy.
// Two resident blocks per SM: the fused step needs ~190 registers per thread
// unconstrained, which would leave one 256-thread block (8 warps) per SM.
template <class R, int PT, int K> __global__ void __launch_bounds__(256, 2) k_step(Args<R> a)
{
  step_body<R, PT, K>(a);
}
template <class R, int PT, int K> __global__ void __launch_bounds__(256, 2) k_step_p(const Args<R> *__restrict__ A)
{
  step_body<R, PT, K>(*A);
}

// ------------------------------------------------- batched engine: split step
// Resident 256-thread blocks per SM the step kernels are compiled for: the FP64
// kernels would take 160-180 registers unbounded (12 warps per SM); bounded to
// 128 they keep 16 warps at the cost of a few spills.  The FP32-mixed kernels
// take 110-126 registers unbounded.  Held to 96 (kMaxRegs: the interaction
// kernels and the transport kernels of the uniform field, layered geometry and
// no multiple scattering) five 128-thread blocks fit on an SM instead of four,
// and C3 and C4 run 7-8% faster although the kernels spill 0-30 words; the
// field-map and multiple-scattering variants would spill 50-270 bytes there
// and stay unbounded (255).
template <class R> constexpr int kMinBlocks = sizeof(R) == 8 ? 2 : 0; // 0: no minimum
template <class R, int K> constexpr int kMaxRegs = sizeof(R) == 8 ? 128 : (K == 0 ? 96 : 255);

// Timeline tracing (the library built with GX_TIMELINE, a separate build of
// this file): per iteration and step kernel, the global timer when the first
// block of the kernel starts and when the last one ends, so that a run shows
// how the kernels of an iteration follow or overlap one another.  Kernel ids:
// 0 refill, 1 refill bookkeeping (at a hand-over only), 2-4 transport of gamma, e-, e+, 5 + 3 type +
// process the interaction kernels, 14 end of iteration; 512 iterations kept
// (iteration i in row (i + 1) mod 512; row 0 holds the planning launch).
// Without GX_TIMELINE the marks compile to nothing.
#if defined(GX_TIMELINE) && !defined(GX_PARITY)
constexpr int kTimelineRows = 512, kTimelineKernels = 16;
__device__ unsigned long long g_timeline[kTimelineRows * kTimelineKernels][2];
__device__ __forceinline__ int timeline_slot(const Ctl *ctl, int id)
{
  const long long it = ((volatile const Ctl *)ctl)->iterations + 1;
  return (int)((it & (kTimelineRows - 1)) * kTimelineKernels + id);
}
__device__ __forceinline__ void timeline_mark(int slot, int end)
{
  if (threadIdx.x == 0) {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (end)
      atomicMax(&g_timeline[slot][1], t);
    else
      atomicMin(&g_timeline[slot][0], t);
  }
}
#define GX_TL_BEGIN(ctl, id)                                                                                          \
  const int gx_tl_slot = timeline_slot(ctl, id);                                                                     \
  timeline_mark(gx_tl_slot, 0)
#define GX_TL_END() timeline_mark(gx_tl_slot, 1)
#else
#define GX_TL_BEGIN(ctl, id)
#define GX_TL_END()
#endif

constexpr int kPhotonSteps = 4;

// Transport of the tracks of type PT: each lane keeps its track in registers
// and steps it until the track interacts (it then goes to the interaction
// buffer of its process), dies, leaves the world, or has taken step_budget
// steps in this launch (it then goes to the next store).  A lane without a
// track takes the next one of those that its warp has drawn, in chunks, from a
// work counter shared by the whole grid, so the lanes of a warp stay busy while
// their tracks take different numbers of steps.
// One pass of the loop advances every lane by a few helix sub-steps (charged
// tracks in a field), with the start and the end of a step attached to them, so
// a lane whose step needs many sub-steps does not hold up the others.
// All stores and buffers are written at slots reserved per warp, contiguous.
template <class R, int PT, int K> __device__ __forceinline__ void transport_body(const Args<R> *__restrict__ A)
{
  extern __shared__ double sm_edep[];
  __shared__ unsigned long long sm_stat[kNStat];
  __shared__ double sm_esc[2];
  __shared__ int sm_err;
  const Args<R> &a = *A;
  const Data &d = *a.d;
  Ctl *ctl = a.ctl;
  const int par = ctl->parity;
  const Store<R> &cur = a.st[par][PT];
  GX_TL_BEGIN(ctl, 2 + PT);
  const long long n = min(ctl->count[par][PT], cur.cap);
  // Lanes of a warp that take records: one while the store has no more records than
  // a fifth of the grid's warps (with 5 blocks of 128 threads per SM one for each
  // scheduler, with 4 blocks 0.8), so that none waits for another's branches, else
  // all (two electrons 3.87 against 3.47 ms; spread further, over all the warps, 61
  // showers lost 15%).
  const int lanes = n <= (long long)gridDim.x * blockDim.x / 160 ? 1 : 32;
  if ((long long)blockIdx.x * (blockDim.x / 32) * lanes >= n) { // no work for this block (uniform exit)
    GX_TL_END();
    return;
  }
  Local L;
  tally_begin(L, a.g, a.edep, sm_edep, sm_stat, sm_esc, &sm_err);
  const bool few = n <= (long long)gridDim.x * blockDim.x;
  const int budget = few ? a.few_budget[PT] : a.step_budget[PT];
  // helix sub-steps of a pass (most steps have one, few more than two): 20000
  // showers 121.4 ms with 1, 118.4 with 2, 120.6 with 3, 122.9 with 4; where every
  // lane has one track, its latency counts: 61 showers 8.9 ms with 1, 8.0 with 2,
  // 7.7 with 4, 7.5 with 6, 7.1 with 8
  const int per_pass = few ? 8 : 2;
  const int fetch_min = min(a.fetch_min[PT], lanes);
  Track<R> t;
  StepCtx<R> c;
  GammaXs<R> gxs;
  gxs.have = 0;
  bool have = false, more = true; // `more` is warp-uniform: the work counter is not exhausted
  bool infield = false;           // in the middle of a step (helix sub-steps)
  int nst = 0;
  // records read and written: counted per warp, in registers (the host adds them
  // to the type's totals; those queued for interactions are counted by k_finish
  // from the buffers' counters)
  unsigned read = 0, written = 0;
  // Records handed to this warp and not yet taken by a lane.  They come in
  // chunks of up to 32, one addition to the grid's counter per chunk instead of
  // per pass, and on their way into L2 by the time a lane loads one (a lane asks for
  // the 128-byte line its record starts in; where a record ends in the next line,
  // the next record starts there): 20000 showers 135.2 to 133.3 ms, 256 events 177.4
  // to 174.3.  A chunk is at most a quarter of a warp's share of the store, so that a small store is still spread
  // over all warps (then 0: what is wanted, no more).
  long long pool_base = 0, old_base = 0;
  int pool_n = 0, old_n = 0;
  const int chunk = (int)min(32LL, n / ((long long)gridDim.x * blockDim.x / 8));
  for (;;) {
    // new records once fetch_min lanes are idle (or all are: the last ones)
    const unsigned need = __ballot_sync(0xffffffffu, !have);
    const int want = lanes - 32 + __popc(need);
    if (want > 0 && (more || pool_n) && (want >= fetch_min || need == 0xffffffffu)) {
      if (pool_n < want && more) {
        // the pool runs out: what is left of it is taken first (old_*, gone
        // after this fetch, since more than that is wanted), then the new run
        const int grab = max(want - pool_n, chunk);
        long long base = 0;
        if (lane_id() == 0)
          base = (long long)atomicAdd((unsigned long long *)&ctl->take[PT], (unsigned long long)grab);
        base = __shfl_sync(0xffffffffu, base, 0);
        old_base = pool_base;
        old_n = pool_n;
        const int got = (int)max(0LL, min((long long)grab, n - base));
        pool_base = base;
        pool_n = old_n + got;
        if (base + grab >= n) more = false;
        if ((int)lane_id() < got) asm volatile("prefetch.global.L2 [%0];" ::"l"(cur.rec + base + lane_id()));
      }
      const int rank = __popc(need & lanemask_lt());
      if (!have && rank < min(want, pool_n)) {
        load_track(cur, rank < old_n ? old_base + rank : pool_base + (rank - old_n), PT, t);
        have = true;
        infield = false;
        nst = 0;
        gxs.have = 0; // a new photon energy
      }
      const int used = min(want, pool_n);
      read += used;
      pool_base += used - old_n;
      old_n = 0;
      pool_n -= used;
    }
    if (!__any_sync(0xffffffffu, have)) break;
    int r = kDone, proc = -1;
    bool done = false; // a step ends in this pass
    if constexpr (PT == 0) {
      // A photon's step is short (most cross a slab with the cross sections it
      // has), so a pass takes up to kPhotonSteps of them before the warp looks for
      // new records and results again: 20000 showers 123.9 ms with 1, 123.2 with
      // 2, 122.3 with 4; at 8 the lanes that are done wait too long (128.0).
      if (have) {
#pragma unroll 1
        for (int k = 0; k < kPhotonSteps && !(done && (r != kAlive || nst >= budget)); ++k) {
          step_begin<R, K>(d, a.g, t, c, &gxs);
          r = step_end<R, K>(d, a.g, t, c, L, &proc);
          done = true;
          ++nst;
          if (t.prim >= 0 && a.pstep) atomicAdd(&a.pstep[t.prim], 1);
        }
      }
    } else {
      if (have && !infield) {
        infield = step_begin<R, K>(d, a.g, t, c);
        done = !infield;
      }
      if (have && infield) {
#pragma unroll 1
        for (int k = 0; k < per_pass && infield; ++k) infield = !field_substep<R, K>(d, a.g, t, c, L);
        done = !infield;
      }
      if (done) {
        r = step_end<R, K>(d, a.g, t, c, L, &proc);
        ++nst;
        if (t.prim >= 0 && a.pstep) atomicAdd(&a.pstep[t.prim], 1);
      }
    }
    const bool w_alive = done && r == kAlive && nst >= budget;
    const bool w_int = done && r == kInteract;
    // slots in the next store and the interaction buffers, one per lane that
    // needs one: lane k adds to counter k (store, processes 0 to 2), the
    // additions in flight together
    const unsigned m_al = __ballot_sync(0xffffffffu, w_alive), m0 = __ballot_sync(0xffffffffu, w_int && proc == 0),
                   m1 = __ballot_sync(0xffffffffu, w_int && proc == 1),
                   m2 = PT == 1 ? 0u : __ballot_sync(0xffffffffu, w_int && proc == 2);
    const unsigned wr = m_al | m0 | m1 | m2;
    long long slot = 0, q = 0;
    if (wr) {
      const int k = (int)lane_id();
      const int mine = k > 3 ? 0 : __popc(k == 0 ? m_al : (k == 1 ? m0 : (k == 2 ? m1 : m2)));
      unsigned long long base = 0;
      if (mine)
        base = atomicAdd((unsigned long long *)(k == 0 ? &ctl->count[par ^ 1][PT] : &ctl->qcount[PT][k - 1]),
                         (unsigned long long)mine);
      base = __shfl_sync(0xffffffffu, base, w_int ? proc + 1 : 0);
      const unsigned with = w_int ? (proc == 0 ? m0 : (proc == 1 ? m1 : m2)) : m_al;
      slot = q = (long long)base + __popc(with & lanemask_lt());
    }
    bool queued = false;
    if (w_alive) {
      put_track(a, PT, slot, t, L);
    } else if (w_int) {
      if (q < a.qcap) {
        store_track(a.ibuf[PT][proc], q, t);
        queued = true;
      } else {
        L.err |= kErrOverflow;
        L.st[S_OVERFLOW]++;
        L.deposit(t.event, t.vol, (double)t.E);
      }
    }
    written += __popc(__ballot_sync(0xffffffffu, w_alive || queued));
    if (done && (r != kAlive || nst >= budget)) have = false;
  }
  if (lane_id() == 0) {
    if (read) atomicAdd(&sm_stat[S_TREAD0 + PT], (unsigned long long)read);
    if (written) atomicAdd(&sm_stat[S_TWRITE0 + PT], (unsigned long long)written);
  }
  tally_end(L, ctl, a.edep, sm_edep, sm_stat, sm_esc, &sm_err, S_TSTEP0 + PT);
  GX_TL_END();
}

template <class R, int PT, int K>
__global__ void __launch_bounds__(256, kMinBlocks<R>) __maxnreg__((kMaxRegs<R, K>)) k_transport(const Args<R> *__restrict__ A)
{
  transport_body<R, PT, K>(A);
}
// The FP32 CSG variants: held to the 128 registers of the others they spill
// 100-300 bytes; at 168 (three 128-thread blocks per SM) nearly none.
template <class R, int PT, int K> __global__ void __maxnreg__(168) k_transport_csg(const Args<R> *__restrict__ A)
{
  transport_body<R, PT, K>(A);
}
// Variants for 512- and 1024-thread blocks (the launch-setting sweep): held
// to the 64 registers per thread a 1024-thread block leaves, they spill.
template <class R, int PT, int K> __global__ void __launch_bounds__(1024, 1) k_transport_wide(const Args<R> *__restrict__ A)
{
  transport_body<R, PT, K>(A);
}

#ifndef GX_PARITY
// Electrons that stops_at_once() finds to end in the volume they are created in
// never become records: about half of all e- steps are the only step of a
// photo-electron or a Compton electron, and it leaves nothing but its deposit and
// its counts.  Without multiple scattering, and with enough of them (n, the
// interactions of a launch) that throughput counts: 20000 showers 128.9 to 123.7
// ms, 256 events 169.8 to 163.7, 1001 of 10 GeV through the volume tree 30.4 to
// 29.1, but two electrons 3.06 to 3.16, where the looking is latency on the way to
// the next iteration.  Not in a run whose caller counts its iterations
// (book_stops): what is handed over after them would depend on n.
template <class R> __device__ __forceinline__ bool local_stops(const Args<R> &a, long long n)
{
  return a.book_stops && !a.g.msc && !a.g.charged_local && n >= 1024;
}

template <class R> __device__ __forceinline__ void book_stop(const Geom &g, const Track<R> &t, R e, Local &L)
{
  L.deposit(t.event, t.vol, (double)e);
  L.st[S_SEC1]++;
  L.st[S_STEPS]++;
  if (g.Bz != 0.0 || g.field_map) L.st[S_SUBSTEPS]++;
}

// The photo-electron of photon t, when it stops at once and no process can come
// before (no cross section at its energy): its energy and the shell's are
// deposited, and neither its direction nor its stream is sampled, since nothing
// is left that would use them.
template <class R, int S>
__device__ __forceinline__ bool photo_electron_stops(const Data &d, const Geom &g, Track<R> &t, Local &L)
{
  const int mat = vol_material(g, t.vol);
  const R e = (R)photo_electron_energy(d, (int)d.mat_Z[mat], (double)t.E, 1);
  if (!(e > R(0)) || (double)e > d.vec[GX_Lambda_eIoni_em][mat].emin || (double)e > d.vec[GX_Lambda_eBrem_em][mat].emin)
    return false;
  R range;
  if (!stops_at_once<R, S>(d, g, t.vol, t.pos, mat, e, range)) return false;
  L.deposit(t.event, t.vol, (double)(t.E - e));
  book_stop(g, t, e, L);
  t.E = R(0);
  return true;
}

// emit_tracks for a Compton scattering or photo-electric absorption (at most one
// electron, in the batched engine's three stores): the electron is booked on the
// spot when `local` and it stops at once before any interaction.
template <class R, int S>
__device__ __forceinline__ void emit_electron(const Args<R> &a, Ctl *ctl, int par, bool active, bool alive, Track<R> &t,
                                              const Secs<R> &sec, bool local, Local &L)
{
  const bool child = active && sec.n == 1;
  bool stop = false;
  Track<R> c = t;
  if (active) {
    Mrg rng = t.rng();
    if (child) {
      c.type = 1;
      c.dir[0] = sec.dir[0][0];
      c.dir[1] = sec.dir[0][1];
      c.dir[2] = sec.dir[0][2];
      c.E = sec.E[0];
      c.nil[0] = c.nil[1] = c.nil[2] = R(-1);
      c.msc_r0 = R(-1);
      c.prim = -1;
      Mrg cr;
      rng.seed_child(cr);
      draw_nils(c, cr);
      c.set_rng(cr);
      const int mat = vol_material(a.g, c.vol);
      R range;
      if (local && stops_at_once<R, S>(*a.d, a.g, c.vol, c.pos, mat, c.E, range)) {
        // as step_gpil chooses: a process comes first unless its length is above the range
        R xs[3];
        cross_sections<R>(*a.d, 1, mat, c.E, xs);
        stop = true;
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (xs[i] > R(0) && !(range < c.nil[i] / xs[i])) stop = false;
      }
      if (stop)
        book_stop(a.g, t, c.E, L);
      else
        L.st[S_SEC1]++;
    }
    if (alive) draw_nils(t, rng);
    t.set_rng(rng);
  }
  const int cnt[3] = {alive ? 1 : 0, child && !stop ? 1 : 0, 0};
  long long next[3];
  warp_reserve3((unsigned long long *)ctl->count[par ^ 1], 2, cnt, next);
  if (cnt[1]) put_track(a, 1, next[1], c, L);
  if (cnt[0]) put_track(a, 0, next[0], t, L);
  L.st[S_WRITE0] += cnt[0] + cnt[1];
}
#endif

// Post-step interaction of process PROC for the buffered tracks of type PT:
// one model per kernel, so a warp runs one sampling algorithm; survivor and
// secondaries go to the next stores.
// S: the solids of the volume tree, in the kernels that look at the geometry (0:
// the analytic volumes).
template <class R, int PT, int PROC, int S>
__device__ __forceinline__ void interact_body(const Args<R> *__restrict__ A)
{
  extern __shared__ double sm_edep[];
  __shared__ unsigned long long sm_stat[kNStat];
  __shared__ double sm_esc[2];
  __shared__ int sm_err;
  const Args<R> &a = *A;
  const Data &d = *a.d;
  Ctl *ctl = a.ctl;
  const int par = ctl->parity;
  const Store<R> &buf = a.ibuf[PT][PROC];
  GX_TL_BEGIN(ctl, 5 + 3 * PT + PROC);
  const long long n = min(ctl->qcount[PT][PROC], a.qcap);
  if ((long long)blockIdx.x * blockDim.x >= n) { // no work for this block (uniform exit)
    GX_TL_END();
    return;
  }
  Local L;
  tally_begin(L, a.g, a.edep, sm_edep, sm_stat, sm_esc, &sm_err);
#ifndef GX_PARITY
  const bool local = local_stops(a, n);
#endif
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long base = (long long)blockIdx.x * blockDim.x; base < n; base += stride) {
    long long j = base + threadIdx.x;
    bool active = j < n;
    Track<R> t;
    Secs<R> sec;
    sec.n = 0;
    bool alive = false;
    if (active) {
      load_track(buf, j, PT, t);
      L.st[S_READ0 + PT]++;
      bool sample = true;
#ifndef GX_PARITY
      if (PT == 0 && PROC == 2 && local) sample = !photo_electron_stops<R, S>(d, a.g, t, L);
#endif
      if (sample) {
        run_model(d, a.g, t, PROC, sec, L);
        alive = t.E > R(0);
      }
    }
#ifndef GX_PARITY
    if constexpr (PT == 0 && PROC != 1)
      emit_electron<R, S>(a, ctl, par, active, alive, t, sec, local, L);
    else
#endif
      emit_tracks<R, PT>(a, ctl, par, active, alive, t, sec, L);
  }
  tally_end(L, ctl, a.edep, sm_edep, sm_stat, sm_esc, &sm_err, S_BOOKED);
  GX_TL_END();
}

template <class R, int PT, int PROC, int S>
__global__ void __launch_bounds__(256, kMinBlocks<R>) __maxnreg__((kMaxRegs<R, 0>)) k_interact(const Args<R> *__restrict__ A)
{
  interact_body<R, PT, PROC, S>(A);
}
template <class R, int PT, int PROC>
__global__ void __launch_bounds__(1024, 1) k_interact_wide(const Args<R> *__restrict__ A)
{
  interact_body<R, PT, PROC, 0>(A);
}

// End of an iteration: the refill that opened it is booked, the next stores
// become current, the refill plan for the following iteration is made.
// interacted: the interaction kernels ran in this iteration (their buffers are
// emptied); otherwise the tracks waiting in them count as pending.
__device__ void finish_iteration(Ctl *ctl, long long cap0, long long cap1, long long cap2, int nstores, int interacted)
{
  for (int q = 0; q < 3; ++q) ctl->take_stack[q] = 0;
  ctl->prim_next += ctl->take_prim;
  ctl->take_prim = 0;
  int par = ctl->parity, np = par ^ 1;
  const long long cap[3] = {cap0, cap1, cap2};
  const long long refill_below = ctl->refill_below, stack_cap = ctl->stack_cap;
  long long buffered = 0;
  for (int q = 0; q < 3; ++q) {
    for (int p = 0; p < 3; ++p) {
      if (interacted) {
        // the records the transport kernels queued for this interaction
        ctl->stat[S_TQUEUE0 + q] += (unsigned long long)ctl->qcount[q][p];
        ctl->qcount[q][p] = 0;
      } else {
        buffered += ctl->qcount[q][p];
      }
    }
    ctl->take[q] = 0;
  }
  long long fl = 0;
  for (int q = 0; q < nstores; ++q) {
    // pushes past the end of a full stack were not written (and were counted as errors)
    ctl->stack_count[q] = min(ctl->stack_count[q], stack_cap);
    ctl->count[np][q] = min(ctl->count[np][q], cap[q]);
    ctl->count[par][q] = 0;
    fl += ctl->count[np][q];
  }
  ctl->parity = np;
  ctl->iterations++;
  // refill plan: deferred tracks first (most recent first), then primaries
  long long budget = refill_below - fl;
  long long pend = ctl->nprim - ctl->prim_next + buffered;
  for (int q = 0; q < nstores; ++q) {
    long long room = cap[q] - ctl->count[np][q];
    long long take = 0;
    // all of the stack is pending, also what is taken now: it is in no store yet
    pend += ctl->stack_count[q];
    if (budget > 0) take = min(min(ctl->stack_count[q], room), budget);
    // reserve the slots now: deferred tracks land at the end of the store,
    // primaries are appended after them by the refill kernel
    ctl->take_stack[q] = take;
    ctl->stack_dst[q] = ctl->count[np][q];
    ctl->count[np][q] += take;
    ctl->stack_count[q] -= take;
    ctl->stack_src[q] = ctl->stack_count[q];
    budget -= take;
  }
  // primaries: a shower's population peaks in proportion to its energy, long
  // after it is injected, so primaries are injected only while the energy the
  // live tracks carry (injected minus deposited or escaped) stays within
  // wave_energy; one primary at least once nothing is left in flight
  long long tp = 0;
  if (budget > 0 && ctl->prim_next < ctl->nprim) {
    long long lo = ctl->prim_next, hi = min(ctl->nprim, ctl->prim_next + budget);
    double e0 = lo > 0 ? ctl->cumE[lo - 1] : 0.0;
    const double room = ctl->wave_energy - (e0 - ctl->retired);
    // largest k in [lo, hi] with cumE[k - 1] - e0 <= room
    long long a = lo, b = hi;
    while (a < b) {
      long long m = (a + b + 1) / 2;
      if (ctl->cumE[m - 1] - e0 <= room)
        a = m;
      else
        b = m - 1;
    }
    long long live = 0;
    for (int q = 0; q < nstores; ++q) live += ctl->count[np][q] + ctl->stack_count[q];
    if (a == lo && live == 0) a = lo + 1;
    tp = a - lo;
  }
  ctl->take_prim = tp;
  ctl->in_flight = fl;
  ctl->pending = pend;
  if (fl > ctl->peak) ctl->peak = fl;
}

// One thread's work, on a copy of the control block in shared memory that the
// block reads and writes together: word by word from L2 it took 4.2 us of every
// iteration, and the booking of the refill was a launch of its own.
constexpr int kFinishBlock = 128;
// batch > 0: the last of the `batch` iterations in the body of the conditional
// node `loop`, which repeats while tracks are left, until a multiple of kLoopIters
// is reached (the host then launches it again).  Every pass of the body sets the
// node's condition, whatever the handle's value (0 is not documented as invalid):
// a pass that did not would leave it at its default and repeat for good.
constexpr long long kLoopIters = 4096;
__global__ void __launch_bounds__(kFinishBlock) k_finish(Ctl *ctl, long long cap0, long long cap1, long long cap2,
                                                         int nstores, int interacted, cudaGraphConditionalHandle loop, int batch)
{
  __shared__ Ctl c;
  static_assert(sizeof(Ctl) % 8 == 0, "copied as 64-bit words");
  GX_TL_BEGIN(ctl, 14);
  for (int k = threadIdx.x; k < (int)(sizeof(Ctl) / 8); k += kFinishBlock)
    reinterpret_cast<unsigned long long *>(&c)[k] = reinterpret_cast<const unsigned long long *>(ctl)[k];
  __syncthreads();
  if (threadIdx.x == 0) {
    finish_iteration(&c, cap0, cap1, cap2, nstores, interacted);
    if (batch > 0)
      cudaGraphSetConditional(loop, (c.in_flight || c.pending) &&
                                        c.iterations / kLoopIters == (c.iterations - batch) / kLoopIters);
  }
  __syncthreads();
  for (int k = threadIdx.x; k < (int)(sizeof(Ctl) / 8); k += kFinishBlock)
    reinterpret_cast<unsigned long long *>(ctl)[k] = reinterpret_cast<const unsigned long long *>(&c)[k];
  GX_TL_END();
}

// Inclusive prefix sum of the primary energies, one block: each thread scans a
// contiguous chunk, the chunk totals are scanned in shared memory.
// status (optional): only the entries with status GX_TRACK_ALIVE count.
__global__ void __launch_bounds__(1024) k_prefix_energy(const double *__restrict__ E, long long n,
                                                        double *__restrict__ out, const int *__restrict__ status)
{
  __shared__ double part[1024];
  int t = threadIdx.x, nt = blockDim.x;
  long long chunk = (n + nt - 1) / nt;
  long long b = t * chunk, e = min(n, b + chunk);
  double s = 0.0;
  for (long long i = b; i < e; ++i) s += (!status || status[i] == GX_TRACK_ALIVE) ? E[i] : 0.0;
  part[t] = s;
  __syncthreads();
  if (t == 0)
    for (int k = 1; k < nt; ++k) part[k] += part[k - 1];
  __syncthreads();
  double run = t > 0 ? part[t - 1] : 0.0;
  for (long long i = b; i < e; ++i) {
    run += (!status || status[i] == GX_TRACK_ALIVE) ? E[i] : 0.0;
    out[i] = run;
  }
}

// v := A v modulo m = 2^32 - c (the folding of k_rng_substreams' products)
__device__ __forceinline__ void jump_matvec(const uint64_t *A, uint64_t v[3], uint32_t c, uint32_t m)
{
  uint64_t r[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    uint64_t acc = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const uint64_t x = A[3 * i + k] * v[k];
      acc += (x >> 32) * c + (x & 0xffffffffull);
    }
    r[i] = Mrg::mod_m(acc, c, m);
  }
  v[0] = r[0];
  v[1] = r[1];
  v[2] = r[2];
}

// Execute the refill plan: move deferred tracks back from the stacks, then
// inject primaries (MRG32k3a substream first_substream + primary index).
template <class R> __device__ __forceinline__ void refill_body(const Args<R> &a)
{
  Ctl *ctl = a.ctl;
  int par = ctl->parity;
  long long ts[3] = {ctl->take_stack[0], ctl->take_stack[1], ctl->take_stack[2]};
  long long tp = ctl->take_prim;
  long long total = ts[0] + ts[1] + ts[2] + tp;
  long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    long long j = i;
    int q = 0;
    while (q < 3 && j >= ts[q]) {
      j -= ts[q];
      ++q;
    }
    if (q < 3) {
      Track<R> t;
      load_track(a.stack[q], ctl->stack_src[q] + j, (a.nstores == 1) ? 3 : q, t);
      store_track(a.st[par][q], ctl->stack_dst[q] + j, t);
      continue;
    }
    long long pi = ctl->prim_next + j;
    Track<R> t;
    if (a.p.from_soa) {
      // a track handed in with its state
      const SoaIn &q = a.p.soa;
      if (q.status[pi] != GX_TRACK_ALIVE) continue;
      t.type = q.type[pi];
      t.E = (R)q.ekin[pi];
      t.pos[0] = q.x[pi];
      t.pos[1] = q.y[pi];
      t.pos[2] = q.z[pi];
      t.dir[0] = (R)q.dx[pi];
      t.dir[1] = (R)q.dy[pi];
      t.dir[2] = (R)q.dz[pi];
      t.nil[0] = (R)q.nil0[pi];
      t.nil[1] = (R)q.nil1[pi];
      t.nil[2] = (R)q.nil2[pi];
      t.msc_r0 = q.msc ? (R)q.msc[pi] : R(-1);
      t.load_rng(q.rng, q.cap, pi);
      t.vol = q.volume[pi];
      if (t.vol < -1) {
        double dd[3] = {q.dx[pi], q.dy[pi], q.dz[pi]};
        t.vol = a.g.geometry == 2 ? csg_locate(a.g.csg, 0, t.pos, dd, kCsgTol) : locate(a.g, t.pos, dd);
      }
      t.event = q.event ? q.event[pi] : 0;
      t.prim = q.primary ? q.primary[pi] : -1;
    } else {
      t.type = a.p.type[pi];
      t.E = (R)a.p.E[pi];
      for (int k = 0; k < 3; ++k) {
        t.pos[k] = a.p.pos[3 * pi + k];
        t.dir[k] = (R)a.p.dir[3 * pi + k];
      }
      double dd[3] = {a.p.dir[3 * pi], a.p.dir[3 * pi + 1], a.p.dir[3 * pi + 2]};
      t.vol = a.g.geometry == 2 ? csg_locate(a.g.csg, 0, t.pos, dd, kCsgTol) : locate(a.g, t.pos, dd);
      t.nil[0] = t.nil[1] = t.nil[2] = R(-1);
      t.msc_r0 = R(-1);
      t.event = a.p.event ? a.p.event[pi] : 0;
      t.prim = (int)pi;
      unsigned long long kk = (unsigned long long)(a.p.first_substream + pi);
      uint64_t v1[3] = {(uint64_t)a.p.seed[0], (uint64_t)a.p.seed[1], (uint64_t)a.p.seed[2]};
      uint64_t v2[3] = {(uint64_t)a.p.seed[3], (uint64_t)a.p.seed[4], (uint64_t)a.p.seed[5]};
      for (int b = 0; kk != 0 && b < 64; ++b, kk >>= 1)
        if (kk & 1ULL) {
          jump_matvec(a.p.jump + 9 * b, v1, Mrg::kC1, Mrg::kM1u);
          jump_matvec(a.p.jump + 9 * (64 + b), v2, Mrg::kC2, Mrg::kM2u);
        }
      for (int k = 0; k < 3; ++k) {
        t.rs[k] = (uint32_t)v1[k];
        t.rs[3 + k] = (uint32_t)v2[k];
      }
    }
    atomicAdd(&ctl->stat[S_TRACKS], 1ULL);
    if (t.vol < 0) {
      atomicAdd(&ctl->escaped, (double)t.E);
      atomicAdd(&ctl->retired, (double)t.E);
      continue;
    }
    int qs = (a.nstores == 1) ? 0 : t.type;
    unsigned long long slot = atomicAdd((unsigned long long *)&ctl->count[par][qs], 1ULL);
    if ((long long)slot < a.st[par][qs].cap) {
      store_track(a.st[par][qs], (long long)slot, t);
    } else {
      atomicOr(&ctl->err_flags, (int)kErrOverflow);
      atomicAdd(&ctl->stat[S_OVERFLOW], 1ULL);
    }
  }
}

// launched with the step kernels' block size, up to 1024 threads
template <class R> __global__ void __launch_bounds__(1024) k_refill(Args<R> a) { refill_body(a); }
template <class R> __global__ void __launch_bounds__(1024) k_refill_p(const Args<R> *__restrict__ A)
{
  GX_TL_BEGIN(A->ctl, 0);
  refill_body(*A);
  GX_TL_END();
}

// Bookkeeping after a refill that no iteration follows (the hand-over of live
// tracks): the primary cursor.  One thread.
__global__ void k_refill_done(Ctl *ctl)
{
  GX_TL_BEGIN(ctl, 1);
  GX_TL_END();
  for (int q = 0; q < 3; ++q) ctl->take_stack[q] = 0;
  ctl->prim_next += ctl->take_prim;
  ctl->take_prim = 0;
}

// Tracks of a run: the primaries, and every secondary once.
inline long long total_tracks(const Ctl &c)
{
  return (long long)(c.stat[S_TRACKS] + c.stat[S_SEC0] + c.stat[S_SEC1] + c.stat[S_SEC2]);
}

// ------------------------------------------------------------------ engine
struct Engine {
  int precision = -1, engine = -1;
  long long cap = 0, stack_cap = 0;
  void *pool = nullptr;
  size_t pool_bytes = 0;
  Ctl *ctl = nullptr;
  Ctl *h_ctl = nullptr; // pinned mirror
  cudaGraphExec_t graph = nullptr;
  int graph_iters = 0;
  std::vector<char> graph_args; // launch arguments the graph was captured with
  double *cumE = nullptr;
  long long cumE_cap = 0;
  double *vtally = nullptr; // geometry 2: deposits per (event, touchable), folded into the caller's columns
  long long vtally_cap = 0;
  void *dargs = nullptr; // device copy of the launch arguments (batched engine)
  cudaStream_t s1 = nullptr, s2 = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_j1 = nullptr, ev_j2 = nullptr;
  // per particle type: branches for its second and third interaction kernel
  cudaStream_t side[3][2] = {};
  cudaEvent_t side_fork[3] = {}, side_join[3][2] = {};
};

void release_engine(Ctx *c)
{
  Engine *e = GX_ENGINE_OF(c);
  if (!e) return;
  if (e->graph) cudaGraphExecDestroy(e->graph);
  if (e->pool) cudaFree(e->pool);
  if (e->ctl) cudaFree(e->ctl);
  if (e->cumE) cudaFree(e->cumE);
  if (e->vtally) cudaFree(e->vtally);
  if (e->dargs) cudaFree(e->dargs);
  if (e->h_ctl) cudaFreeHost(e->h_ctl);
  if (e->s1) cudaStreamDestroy(e->s1);
  if (e->s2) cudaStreamDestroy(e->s2);
  if (e->ev_fork) cudaEventDestroy(e->ev_fork);
  if (e->ev_j1) cudaEventDestroy(e->ev_j1);
  if (e->ev_j2) cudaEventDestroy(e->ev_j2);
  for (int q = 0; q < 3; ++q) {
    if (e->side_fork[q]) cudaEventDestroy(e->side_fork[q]);
    for (int k = 0; k < 2; ++k) {
      if (e->side[q][k]) cudaStreamDestroy(e->side[q][k]);
      if (e->side_join[q][k]) cudaEventDestroy(e->side_join[q][k]);
    }
  }
  delete e;
  GX_ENGINE_OF(c) = nullptr;
}


template <class R> struct Launch {
  Args<R> a;
  int block, grid, smem;
};

// Geometry 2: the deposits per (event, touchable) added to the caller's
// tally columns (touchables without a column are dropped).
__global__ void k_fold_touchables(const double *__restrict__ vt, const int *__restrict__ score, int ntouch,
                                  int nscore, long long n, double *__restrict__ edep)
{
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const double e = vt[i];
    const long long ev = i / ntouch;
    const int c = score[i - ev * ntouch];
    if (e != 0.0 && c >= 0) edep[ev * nscore + c] += e;
  }
}

template <class R, int PT, int K> static void (*transport_variant())(const Args<R> *)
{
  if constexpr (sizeof(R) == 4 && (K & kKindCsg) != 0)
    return k_transport_csg<R, PT, K>;
  else
    return k_transport<R, PT, K>;
}
template <class R, int PT> static void (*transport_kernel(int kind))(const Args<R> *)
{
  if constexpr (sizeof(R) == 4) {
    switch (kind) {
    case 10: return transport_variant<R, PT, 10>();
    case 11: return transport_variant<R, PT, 11>();
    case 14: return transport_variant<R, PT, 14>();
    case 15: return transport_variant<R, PT, 15>();
    default: break;
    }
  }
  switch (kind & 7) {
  case 1: return transport_variant<R, PT, 1>();
  case 2: return transport_variant<R, PT, 2>();
  case 3: return transport_variant<R, PT, 3>();
  case 4: return transport_variant<R, PT, 4>();
  case 5: return transport_variant<R, PT, 5>();
  case 6: return transport_variant<R, PT, 6>();
  case 7: return transport_variant<R, PT, 7>();
  default: return transport_variant<R, PT, 0>();
  }
}
template <class R> static void (*step_kernel_p(int kind))(const Args<R> *)
{
  if constexpr (sizeof(R) == 4) {
    switch (kind) {
    case 10: return k_step_p<R, 3, 10>;
    case 11: return k_step_p<R, 3, 11>;
    case 14: return k_step_p<R, 3, 14>;
    case 15: return k_step_p<R, 3, 15>;
    default: break;
    }
  }
  switch (kind & 7) {
  case 1: return k_step_p<R, 3, 1>;
  case 2: return k_step_p<R, 3, 2>;
  case 3: return k_step_p<R, 3, 3>;
  case 4: return k_step_p<R, 3, 4>;
  case 5: return k_step_p<R, 3, 5>;
  case 6: return k_step_p<R, 3, 6>;
  case 7: return k_step_p<R, 3, 7>;
  default: return k_step_p<R, 3, 0>;
  }
}

// The step kernels of one type for a launch: blocks above 256 threads take the
// wide variants (kernel kind 0 only, FP32 and FP64 library kernels).
template <class R, int PT> static void (*transport_for(const Launch<R> &L))(const Args<R> *)
{
#ifndef GX_PARITY
  if (L.block > 256) return k_transport_wide<R, PT, 0>;
#endif
  return transport_kernel<R, PT>(kernel_kind<R>(L.a.g));
}
template <class R, int PT, int PROC> static void (*interact_for(const Launch<R> &L))(const Args<R> *)
{
#ifndef GX_PARITY
  if (L.block > 256) return k_interact_wide<R, PT, PROC>;
  if constexpr (PT == 0 && PROC != 1)
    if (L.a.g.geometry == 2)
      return sizeof(R) == 4 && L.a.g.csg.solids == kSolidsBox ? k_interact<R, PT, PROC, kSolidsBox>
                                                              : k_interact<R, PT, PROC, kSolidsAll>;
#endif
  return k_interact<R, PT, PROC, 0>;
}

// One type's interaction kernels (gamma 3 processes, e- 2, e+ 3): one after
// another, or (e given) the second and third on branches of their own beside
// the first.  They read different buffers and reserve their outputs by atomics;
// with few tracks each is 10 to 20 us of latency whatever its work: 61 showers 13.9 ms
// in a row, 12.5 side by side, two electrons 4.8 and 4.0, a full batch of 20000
// 136.0 and 135.2.
template <class R, int PT>
static void enqueue_interactions(const Launch<R> &L, const Args<R> *A, cudaStream_t s, Engine *e = nullptr)
{
  cudaStream_t to[3] = {s, s, s};
  if (e) {
    cudaEventRecord(e->side_fork[PT], s);
    for (int k = 0; k < (PT == 1 ? 1 : 2); ++k) {
      to[k + 1] = e->side[PT][k];
      cudaStreamWaitEvent(to[k + 1], e->side_fork[PT], 0);
    }
  }
  interact_for<R, PT, 0>(L)<<<L.grid, L.block, L.smem, to[0]>>>(A);
  interact_for<R, PT, 1>(L)<<<L.grid, L.block, L.smem, to[1]>>>(A);
  if constexpr (PT != 1) interact_for<R, PT, 2>(L)<<<L.grid, L.block, L.smem, to[2]>>>(A);
  if (e)
    for (int k = 0; k < (PT == 1 ? 1 : 2); ++k) {
      cudaEventRecord(e->side_join[PT][k], to[k + 1]);
      cudaStreamWaitEvent(s, e->side_join[PT][k], 0);
    }
}

// One iteration.  interact: this iteration runs the interaction kernels (the
// compaction interval: otherwise the interacting tracks wait in their buffers).
template <class R>
static void enqueue_iteration(const Launch<R> &L, Engine *e, cudaStream_t s, bool concurrent, bool interact = true,
                              cudaGraphConditionalHandle loop = 0, int batch = 0)
{
  const Args<R> *A = (const Args<R> *)e->dargs;
  if (L.a.nstores == 1) {
    // plain loop: one fused step kernel over the mixed store
    k_refill_p<R><<<L.grid, L.block, 0, s>>>(A);
    step_kernel_p<R>(kernel_kind<R>(L.a.g))<<<L.grid, L.block, L.smem, s>>>(A);
    k_finish<<<1, kFinishBlock, 0, s>>>(L.a.ctl, L.a.st[0][0].cap, L.a.st[0][1].cap, L.a.st[0][2].cap, L.a.nstores, 1, 0, 0);
    return;
  }
  k_refill_p<R><<<L.grid, L.block, 0, s>>>(A);
  cudaStream_t sg = s, se = s, sp = s;
  if (concurrent) {
    // gamma on s, e- on s1, e+ on s2
    cudaEventRecord(e->ev_fork, s);
    cudaStreamWaitEvent(e->s1, e->ev_fork, 0);
    cudaStreamWaitEvent(e->s2, e->ev_fork, 0);
    se = e->s1;
    sp = e->s2;
  }
  // Each type's transport kernel fills every SM, so the three run nearly one
  // after another, the next one's blocks taking the SMs the previous one's
  // blocks leave.  Positrons go first: their chain (a transport kernel with
  // about one record per lane, then three interaction kernels) is the one
  // that ends an iteration most often when it is dispatched last.
  transport_for<R, 2>(L)<<<L.grid, L.block, L.smem, sp>>>(A);
  if (interact) enqueue_interactions<R, 2>(L, A, sp, concurrent ? e : nullptr);
  transport_for<R, 1>(L)<<<L.grid, L.block, L.smem, se>>>(A);
  if (interact) enqueue_interactions<R, 1>(L, A, se, concurrent ? e : nullptr);
  transport_for<R, 0>(L)<<<L.grid, L.block, L.smem, sg>>>(A);
  if (interact) enqueue_interactions<R, 0>(L, A, sg, concurrent ? e : nullptr);
  if (concurrent) {
    cudaEventRecord(e->ev_j1, e->s1);
    cudaEventRecord(e->ev_j2, e->s2);
    cudaStreamWaitEvent(s, e->ev_j1, 0);
    cudaStreamWaitEvent(s, e->ev_j2, 0);
  }
  k_finish<<<1, kFinishBlock, 0, s>>>(L.a.ctl, L.a.st[0][0].cap, L.a.st[0][1].cap, L.a.st[0][2].cap, L.a.nstores,
                           interact ? 1 : 0, loop, batch);
}

// The graph that runs iterations while tracks are left: a conditional node whose
// body is kLoopBatch iterations (whole compaction intervals).  As 16 iterations
// per launch, with the host looking at the counters in between, a call ran up
// to 15 iterations of empty launches after its last track and waited for the
// host between the launches: photons in lead (8 iterations) 0.52 ms, now 0.44.
// Repeating costs 5 us: a body of one iteration lost what it saved (61 showers
// 9.36 ms against 9.06), bodies of 4 and 8 are equal there.
constexpr int kLoopBatch = 8;
template <class R> static cudaError_t loop_graph(const Launch<R> &L, Engine *e, int every, cudaGraphExec_t *exec)
{
  cudaGraph_t graph = nullptr;
  cudaStream_t cs = nullptr;
  cudaError_t err = cudaGraphCreate(&graph, 0);
  cudaGraphConditionalHandle loop = 0;
  cudaGraphNodeParams p = {};
  p.type = cudaGraphNodeTypeConditional;
  p.conditional.type = cudaGraphCondTypeWhile;
  p.conditional.size = 1;
  cudaGraphNode_t node;
  if (err == cudaSuccess) err = cudaGraphConditionalHandleCreate(&loop, graph, 1, cudaGraphCondAssignDefault);
  p.conditional.handle = loop;
  if (err == cudaSuccess) err = cudaGraphAddNode(&node, graph, nullptr, 0, &p);
  if (err == cudaSuccess) err = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
  if (err == cudaSuccess)
    err = cudaStreamBeginCaptureToGraph(cs, p.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                        cudaStreamCaptureModeThreadLocal);
  if (err == cudaSuccess) {
    const int batch = (kLoopBatch + every - 1) / every * every;
    for (int k = 0; k < batch; ++k)
      enqueue_iteration(L, e, cs, true, (k + 1) % every == 0, loop, k + 1 == batch ? batch : 0);
    cudaGraph_t body = nullptr;
    err = cudaStreamEndCapture(cs, &body);
  }
  if (err == cudaSuccess) err = cudaGraphInstantiate(exec, graph, 0);
  if (cs) cudaStreamDestroy(cs);
  if (graph) cudaGraphDestroy(graph);
  return err;
}

// One particle type's step (transport + its interactions), for the profiling
// pass; `mid` is recorded between the transport kernel and the interactions.
template <class R>
static void enqueue_type(const Launch<R> &L, Engine *e, cudaStream_t s, int q, cudaEvent_t mid, bool interact = true)
{
  const Args<R> *A = (const Args<R> *)e->dargs;
  if (q == 0) {
    transport_for<R, 0>(L)<<<L.grid, L.block, L.smem, s>>>(A);
    cudaEventRecord(mid, s);
    if (interact) enqueue_interactions<R, 0>(L, A, s);
  } else if (q == 1) {
    transport_for<R, 1>(L)<<<L.grid, L.block, L.smem, s>>>(A);
    cudaEventRecord(mid, s);
    if (interact) enqueue_interactions<R, 1>(L, A, s);
  } else {
    transport_for<R, 2>(L)<<<L.grid, L.block, L.smem, s>>>(A);
    cudaEventRecord(mid, s);
    if (interact) enqueue_interactions<R, 2>(L, A, s);
  }
}

// Copy the tracks of a store (or stack), or the not yet injected tracks of a
// handed-in batch, into a caller's gx_track_soa at slots taken from a counter.
template <class R>
__global__ void k_extract(Store<R> src, long long n, int ptype, Ctl *ctl, gx_track_soa out)
{
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    Track<R> t;
    load_track(src, i, ptype, t);
    const long long j = (long long)atomicAdd((unsigned long long *)&ctl->extracted, 1ULL);
    if (j >= out.capacity) continue;
    out.type[j] = t.type;
    out.status[j] = GX_TRACK_ALIVE;
    if (out.event) out.event[j] = t.event;
    if (out.primary) out.primary[j] = t.prim;
    out.volume[j] = t.vol;
    out.next_volume[j] = t.vol;
    out.process[j] = -1;
    out.boundary[j] = 0;
    out.x[j] = t.pos[0];
    out.y[j] = t.pos[1];
    out.z[j] = t.pos[2];
    out.dx[j] = (double)t.dir[0];
    out.dy[j] = (double)t.dir[1];
    out.dz[j] = (double)t.dir[2];
    out.ekin[j] = (double)t.E;
    out.nil0[j] = (double)t.nil[0];
    out.nil1[j] = (double)t.nil[1];
    out.nil2[j] = (double)t.nil[2];
    out.lambda_inv0[j] = out.lambda_inv1[j] = out.lambda_inv2[j] = 0.0;
    out.pstep[j] = out.step[j] = out.snext[j] = out.safety[j] = 0.0;
    if (out.msc_range) out.msc_range[j] = (double)t.msc_r0;
    t.store_rng(out.rng, out.capacity, j);
  }
}

__global__ void k_extract_pending(SoaIn in, long long first, long long n, Ctl *ctl, gx_track_soa out)
{
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const long long i = first + k;
    if (in.status[i] != GX_TRACK_ALIVE) continue;
    const long long j = (long long)atomicAdd((unsigned long long *)&ctl->extracted, 1ULL);
    if (j >= out.capacity) continue;
    out.type[j] = in.type[i];
    out.status[j] = GX_TRACK_ALIVE;
    if (out.event) out.event[j] = in.event ? in.event[i] : 0;
    if (out.primary) out.primary[j] = in.primary ? in.primary[i] : -1;
    out.volume[j] = in.volume[i];
    out.next_volume[j] = in.volume[i];
    out.process[j] = -1;
    out.boundary[j] = 0;
    out.x[j] = in.x[i];
    out.y[j] = in.y[i];
    out.z[j] = in.z[i];
    out.dx[j] = in.dx[i];
    out.dy[j] = in.dy[i];
    out.dz[j] = in.dz[i];
    out.ekin[j] = in.ekin[i];
    out.nil0[j] = in.nil0[i];
    out.nil1[j] = in.nil1[i];
    out.nil2[j] = in.nil2[i];
    out.lambda_inv0[j] = out.lambda_inv1[j] = out.lambda_inv2[j] = 0.0;
    out.pstep[j] = out.step[j] = out.snext[j] = out.safety[j] = 0.0;
    if (out.msc_range) out.msc_range[j] = in.msc ? in.msc[i] : -1.0;
#pragma unroll
    for (int w = 0; w < 6; ++w) out.rng[w * out.capacity + j] = in.rng[w * in.cap + i];
  }
}

// The transport loop.  tin (optional): transport these tracks instead of the
// primaries; max_iter > 0: stop after that many iterations and write every
// track still alive to tout.
template <class R>
static int run(Ctx *C, const gx_transport_config *cfg, int nprim, const int *d_type, const double *d_E,
               const double *d_pos, const double *d_dir, const int *d_event, double *d_edep, int nvol,
               int *d_pstep, gx_transport_stats *stats, cudaStream_t s, const gx_track_soa *tin = nullptr,
               int max_iter = 0, gx_track_soa *tout = nullptr)
{
  const int prec = std::is_same<R, float>::value ? 1 : 0;
  const bool batched = cfg->engine == 1;
  const int nstores = batched ? 3 : 1;
  long long cap = cfg->capacity > 0 ? cfg->capacity : (batched ? (1LL << 24) : (3LL << 24));
  long long stack_cap = std::max(cap, 1LL << 20);
  Engine *&E = GX_ENGINE_OF(C);
  if (E && (E->precision != prec || E->engine != cfg->engine || E->cap != cap)) GX_RELEASE_ENGINE(C);
  cudaError_t err;
  if (!E) {
    E = new Engine();
    E->precision = prec;
    E->engine = cfg->engine;
    E->cap = cap;
    E->stack_cap = stack_cap;
    size_t bytes = 0;
    for (int b = 0; b < 2; ++b)
      for (int q = 0; q < nstores; ++q) carve<R>(0, bytes, cap);
    for (int q = 0; q < nstores; ++q) carve<R>(0, bytes, stack_cap);
    if (batched) // interaction buffers: gamma 3 processes, e- 2, e+ 3
      for (int k = 0; k < 8; ++k) carve<R>(0, bytes, cap);
    err = cudaMalloc(&E->pool, bytes);
    if (err != cudaSuccess) {
      GX_RELEASE_ENGINE(C);
      return cuda_error(err, "transport track stores");
    }
    E->pool_bytes = bytes;
    if ((err = cudaMalloc((void **)&E->ctl, sizeof(Ctl))) != cudaSuccess ||
        (err = cudaMallocHost((void **)&E->h_ctl, sizeof(Ctl))) != cudaSuccess) {
      GX_RELEASE_ENGINE(C);
      return cuda_error(err, "transport control block");
    }
    cudaStreamCreateWithFlags(&E->s1, cudaStreamNonBlocking);
    cudaStreamCreateWithFlags(&E->s2, cudaStreamNonBlocking);
    cudaEventCreateWithFlags(&E->ev_fork, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&E->ev_j1, cudaEventDisableTiming);
    cudaEventCreateWithFlags(&E->ev_j2, cudaEventDisableTiming);
    for (int q = 0; q < 3; ++q) {
      cudaEventCreateWithFlags(&E->side_fork[q], cudaEventDisableTiming);
      for (int k = 0; k < 2; ++k) {
        cudaStreamCreateWithFlags(&E->side[q][k], cudaStreamNonBlocking);
        cudaEventCreateWithFlags(&E->side_join[q][k], cudaEventDisableTiming);
      }
    }
  }
  Launch<R> L;
  std::memset(&L.a, 0, sizeof(L.a));
  size_t off = 0;
  uintptr_t base = (uintptr_t)E->pool;
  for (int b = 0; b < 2; ++b)
    for (int q = 0; q < nstores; ++q) L.a.st[b][q] = carve<R>(base, off, cap);
  for (int q = 0; q < nstores; ++q) L.a.stack[q] = carve<R>(base, off, stack_cap);
  for (int q = nstores; q < 3; ++q) {
    L.a.st[0][q] = L.a.st[0][0];
    L.a.st[1][q] = L.a.st[1][0];
    L.a.stack[q] = L.a.stack[0];
  }
  if (batched) {
    for (int q = 0; q < 3; ++q)
      for (int pr = 0; pr < 3; ++pr)
        if (q != 1 || pr != 2) L.a.ibuf[q][pr] = carve<R>(base, off, cap);
    L.a.qcap = cap;
  }
  {
    // a budget asked for holds whatever the store's size; with
    // steps_per_launch alone e+ get a quarter of it.  A caller that counts
    // iterations (max_iter) gets kCountedSteps, whatever the store's size, and no
    // step beyond them.
    L.a.book_stops = max_iter == 0;
    const int spl = cfg->steps_per_launch;
    for (int q = 0; q < 3; ++q) {
      const int asked = cfg->steps_per_launch_by_type[q] > 0 ? cfg->steps_per_launch_by_type[q]
                        : spl > 0                            ? (q == 2 ? std::max(1, spl / 4) : spl)
                                                             : 0;
      L.a.step_budget[q] = asked ? asked : (max_iter > 0 ? kCountedSteps : kDefaultSteps)[q];
      L.a.few_budget[q] = asked ? asked : (max_iter > 0 ? kCountedSteps : kFewSteps)[q];
    }
    // a warp refills when this many of its lanes are idle: a photon takes a
    // few cheap boundary-crossing steps, so the new-track work (record load,
    // NIL draws, cross sections) would otherwise run for one or two lanes in
    // most passes of the photon kernel
    for (int q = 0; q < 3; ++q)
      L.a.fetch_min[q] = cfg->fetch_min_by_type[q] > 0 ? cfg->fetch_min_by_type[q] : default_fetch_min(*cfg, q);
  }
  if (off > E->pool_bytes) return set_error(GX_ERR_OVERFLOW, "transport pool layout");
  L.a.d = C->dev;
  L.a.ctl = E->ctl;
  Geom &g = L.a.g;
  make_geom(C, cfg, nvol, g);
  uint64_t *jt;
  int rc = get_jump_table(&jt);
  if (rc) return rc;
  L.a.p.type = d_type;
  L.a.p.event = d_event;
  L.a.p.E = d_E;
  L.a.p.pos = d_pos;
  L.a.p.dir = d_dir;
  for (int k = 0; k < 6; ++k) L.a.p.seed[k] = cfg->seed[k];
  L.a.p.first_substream = cfg->first_substream;
  L.a.p.jump = jt;
  if (tin) {
    L.a.p.from_soa = 1;
    L.a.p.soa = SoaIn{tin->type, tin->status, tin->event, tin->primary, tin->volume, tin->x, tin->y, tin->z,
                      tin->dx, tin->dy, tin->dz, tin->ekin, tin->nil0, tin->nil1, tin->nil2, tin->msc_range,
                      tin->rng, (long long)tin->capacity};
  }
  L.a.edep = d_edep;
  L.a.pstep = d_pstep;
  if (cfg->geometry == 2) {
    // the kernels score per (event, touchable); folded into d_edep at the end
    g.csg = CsgView{C->csg_node, C->csg_kids, C->csg_slab, C->csg_cand, C->csg_planes, C->csg_solids};
    g.nvol = C->csg_n;
    const long long nt = (long long)cfg->nevents * C->csg_n;
    if (nt > E->vtally_cap) {
      if (E->vtally) cudaFree(E->vtally);
      E->vtally = nullptr;
      E->vtally_cap = 0;
      if ((err = cudaMalloc((void **)&E->vtally, sizeof(double) * nt)) != cudaSuccess)
        return cuda_error(err, "transport touchable tally");
      E->vtally_cap = nt;
    }
    if ((err = cudaMemsetAsync(E->vtally, 0, sizeof(double) * nt, s)) != cudaSuccess)
      return cuda_error(err, "transport touchable tally");
    L.a.edep = E->vtally;
  }
  L.a.nstores = nstores;
  L.a.refill_below = cfg->refill_below > 0 ? std::min(cfg->refill_below, cap) : cap / 2;
  L.block = cfg->block_size > 0 ? cfg->block_size : default_block(cfg->engine);
  int bpsm = cfg->blocks_per_sm > 0 ? cfg->blocks_per_sm : default_blocks_per_sm(*cfg);
  L.grid = C->num_sms * bpsm;
  L.smem = kTallyDoubles * sizeof(double);

  if (nprim > E->cumE_cap) {
    if (E->cumE) cudaFree(E->cumE);
    E->cumE = nullptr;
    E->cumE_cap = 0;
    if ((err = cudaMalloc((void **)&E->cumE, sizeof(double) * nprim)) != cudaSuccess)
      return cuda_error(err, "transport primary energies");
    E->cumE_cap = nprim;
  }
  if (nprim > 0) k_prefix_energy<<<1, 1024, 0, s>>>(tin ? tin->ekin : d_E, nprim, E->cumE, tin ? tin->status : nullptr);
  Ctl h;
  std::memset(&h, 0, sizeof(h));
  h.nprim = nprim;
  h.iterations = -1; // the planning launch below is not an iteration
  h.cumE = E->cumE;
  h.wave_energy = cfg->wave_energy > 0 ? cfg->wave_energy : default_wave_energy(cap, batched ? kWaveFillBatched : kWaveFillPlain);
  h.refill_below = L.a.refill_below;
  h.stack_cap = stack_cap;
  err = cudaMemcpyAsync(E->ctl, &h, sizeof(Ctl), cudaMemcpyHostToDevice, s);
  if (err != cudaSuccess) return cuda_error(err, "transport control init");
  // first refill plan
  k_finish<<<1, kFinishBlock, 0, s>>>(E->ctl, cap, cap, cap, nstores, 1, 0, 0);
  cudaEvent_t t0, t1;
  cudaEventCreate(&t0);
  cudaEventCreate(&t1);
  cudaEventRecord(t0, s);
  const long long kMaxIter = 2000000LL;
  long long iters = 0;
  // the kernels read their arguments from a device copy (indexing a kernel
  // parameter by a run-time value would copy the whole block to local memory)
  if (!E->dargs && (err = cudaMalloc(&E->dargs, sizeof(Args<double>))) != cudaSuccess)
    return cuda_error(err, "transport arguments");
  if ((err = cudaMemcpyAsync(E->dargs, &L.a, sizeof(Args<R>), cudaMemcpyHostToDevice, s)) != cudaSuccess)
    return cuda_error(err, "transport arguments upload");
  double step_ms[3] = {0, 0, 0}, transport_ms[3] = {0, 0, 0};
  long long step_launches[3] = {0, 0, 0};
  // the compaction interval: the interaction kernels run (and their buffers
  // are emptied into the stores) every `every` iterations; one iteration for
  // the plain loop and for runs that hand their tracks over at the end
  const int every = (batched && !tout && cfg->interaction_interval > 1) ? cfg->interaction_interval : 1;
  if (!batched || cfg->profile || max_iter > 0) {
    // plain loop (and the profiling pass, and runs stopped after a number of
    // iterations): launch, synchronise, look at the counters, every iteration
    cudaEvent_t ea[3], em[3], eb[3];
    for (int q = 0; q < 3; ++q) {
      cudaEventCreate(&ea[q]);
      cudaEventCreate(&em[q]);
      cudaEventCreate(&eb[q]);
    }
    for (;;) {
      if (cfg->profile) {
        k_refill_p<R><<<L.grid, L.block, 0, s>>>((const Args<R> *)E->dargs);
        for (int q = 0; q < nstores; ++q) {
          cudaEventRecord(ea[q], s);
          if (!batched) {
            step_kernel_p<R>(kernel_kind<R>(L.a.g))<<<L.grid, L.block, L.smem, s>>>(
                (const Args<R> *)E->dargs);
            cudaEventRecord(em[q], s);
          } else {
            enqueue_type(L, E, s, q, em[q], (iters + 1) % every == 0);
          }
          cudaEventRecord(eb[q], s);
        }
        k_finish<<<1, kFinishBlock, 0, s>>>(L.a.ctl, L.a.st[0][0].cap, L.a.st[0][1].cap, L.a.st[0][2].cap, L.a.nstores,
                                 (iters + 1) % every == 0 ? 1 : 0, 0, 0);
      } else {
        enqueue_iteration(L, E, s, false, (iters + 1) % every == 0);
      }
      cudaMemcpyAsync(E->h_ctl, E->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s);
      if ((err = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_error(err, "transport iteration");
      if (cfg->profile)
        for (int q = 0; q < nstores; ++q) {
          float t = 0, tt = 0;
          cudaEventElapsedTime(&t, ea[q], eb[q]);
          cudaEventElapsedTime(&tt, ea[q], em[q]);
          step_ms[q] += t;
          transport_ms[q] += tt;
          step_launches[q]++;
        }
      ++iters;
      if (E->h_ctl->in_flight == 0 && E->h_ctl->pending == 0) break;
      if (max_iter > 0 && iters >= max_iter) break;
      if (iters > kMaxIter) return set_error(GX_ERR_ITERCAP, "transport: iteration cap");
    }
    for (int q = 0; q < 3; ++q) {
      cudaEventDestroy(ea[q]);
      cudaEventDestroy(em[q]);
      cudaEventDestroy(eb[q]);
    }
  } else {
    // graph_iters asked for: that many iterations per launch, the host looking at
    // the counters in between; otherwise (G = 0) the graph repeats by itself
    int G = cfg->graph_iters > 0 ? cfg->graph_iters : 0;
    G = ((G + every - 1) / every) * every; // whole compaction intervals
    // (re)capture the iteration graph when its launch shape or its kernels
    // (field kind, geometry kind) change; the arguments themselves are read
    // from the device copy uploaded above
    int shape[6] = {G, L.block, L.grid, L.smem, kernel_kind<R>(L.a.g), every};
    std::vector<char> key(sizeof(shape) + 2 * sizeof(void *));
    const void *ptrs[2] = {E->dargs, E->ctl};
    std::memcpy(key.data(), shape, sizeof(shape));
    std::memcpy(key.data() + sizeof(shape), ptrs, sizeof(ptrs));
    if (!E->graph || E->graph_args != key) {
      if (E->graph) {
        cudaGraphExecDestroy(E->graph);
        E->graph = nullptr;
      }
      if (G == 0) {
        if ((err = loop_graph(L, E, every, &E->graph)) != cudaSuccess) return cuda_error(err, "iteration graph");
      } else {
        cudaStream_t cs;
        cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
        cudaGraph_t graph;
        if ((err = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal)) != cudaSuccess)
          return cuda_error(err, "graph capture");
        for (int k = 0; k < G; ++k) enqueue_iteration(L, E, cs, true, (k + 1) % every == 0);
        if ((err = cudaStreamEndCapture(cs, &graph)) != cudaSuccess) return cuda_error(err, "graph capture end");
        err = cudaGraphInstantiate(&E->graph, graph, 0);
        cudaGraphDestroy(graph);
        cudaStreamDestroy(cs);
        if (err != cudaSuccess) return cuda_error(err, "graph instantiate");
      }
      E->graph_iters = G;
      E->graph_args = key;
    }
    for (;;) {
      if ((err = cudaGraphLaunch(E->graph, s)) != cudaSuccess) return cuda_error(err, "graph launch");
      cudaEventRecord(t1, s);
      cudaMemcpyAsync(E->h_ctl, E->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s);
      if ((err = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_error(err, "transport graph");
      iters = E->h_ctl->iterations;
      if (E->h_ctl->in_flight == 0 && E->h_ctl->pending == 0) break;
      if (iters > kMaxIter) return set_error(GX_ERR_ITERCAP, "transport: iteration cap");
    }
  }
  if (cfg->geometry == 2) {
    const long long nt = (long long)cfg->nevents * C->csg_n;
    k_fold_touchables<<<(int)std::min<long long>((nt + 255) / 256, 4096), 256, 0, s>>>(
        E->vtally, C->csg_score, C->csg_n, C->csg_nscore, nt, d_edep);
  }
  if (tout) {
    // the tracks still alive: carry out the refill plan the last iteration
    // made (deferred tracks back into the stores, the next primaries in), then
    // write out the stores, the stacks and what was never injected
    const Args<R> *A = (const Args<R> *)E->dargs;
    k_refill_p<R><<<L.grid, L.block, 0, s>>>(A);
    k_refill_done<<<1, 1, 0, s>>>(L.a.ctl);
    cudaMemcpyAsync(E->h_ctl, E->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s);
    if ((err = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_error(err, "transport hand-over");
    const Ctl hc = *E->h_ctl;
    const int par = hc.parity;
    const int ptype_of[3] = {batched ? 0 : 3, batched ? 1 : 3, batched ? 2 : 3};
    for (int q = 0; q < nstores; ++q) {
      const long long nc = std::min(hc.count[par][q], cap), ns = std::min(hc.stack_count[q], stack_cap);
      if (nc > 0) k_extract<R><<<(int)std::min<long long>((nc + 255) / 256, 4096), 256, 0, s>>>(
          L.a.st[par][q], nc, ptype_of[q], E->ctl, *tout);
      if (ns > 0) k_extract<R><<<(int)std::min<long long>((ns + 255) / 256, 4096), 256, 0, s>>>(
          L.a.stack[q], ns, ptype_of[q], E->ctl, *tout);
    }
    if (tin && hc.prim_next < hc.nprim) {
      const long long np = hc.nprim - hc.prim_next;
      k_extract_pending<<<(int)std::min<long long>((np + 255) / 256, 4096), 256, 0, s>>>(L.a.p.soa, hc.prim_next,
                                                                                        np, E->ctl, *tout);
    }
  }
  // the graph's last look at the counters is the end, unless something followed it
  if (!batched || cfg->profile || max_iter > 0 || cfg->geometry == 2 || tout) {
    cudaEventRecord(t1, s);
    cudaMemcpyAsync(E->h_ctl, E->ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s);
    if ((err = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_error(err, "transport end");
  }
  float ms = 0;
  cudaEventElapsedTime(&ms, t0, t1);
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  const Ctl &c = *E->h_ctl;
  if (stats) {
    stats->steps = (long long)c.stat[S_STEPS];
    stats->substeps = (long long)c.stat[S_SUBSTEPS];
    stats->tracks = total_tracks(c);
    for (int q = 0; q < 3; ++q) stats->secondaries[q] = (long long)c.stat[S_SEC0 + q];
    stats->n_pair = (long long)c.stat[S_PAIR];
    stats->n_annih = (long long)c.stat[S_ANNIH];
    stats->errors = (long long)(c.stat[S_ERR] + c.stat[S_OVERFLOW]);
    stats->escaped = c.escaped;
    stats->iterations = c.iterations;
    stats->peak_in_flight = c.peak;
    stats->kernel_ms = ms;
    for (int q = 0; q < 3; ++q) {
      stats->step_ms[q] = step_ms[q];
      stats->step_launches[q] = step_launches[q];
      // the transport kernels count their records in the transport entries only
      stats->tracks_read[q] = (long long)(c.stat[S_READ0 + q] + c.stat[S_TREAD0 + q]);
      stats->tracks_written[q] = (long long)(c.stat[S_WRITE0 + q] + c.stat[S_TWRITE0 + q]);
      stats->transport_ms[q] = transport_ms[q];
      stats->transport_read[q] = (long long)c.stat[S_TREAD0 + q];
      stats->transport_written[q] = (long long)c.stat[S_TWRITE0 + q];
      stats->transport_queued[q] = (long long)c.stat[S_TQUEUE0 + q];
      stats->transport_steps[q] = (long long)c.stat[S_TSTEP0 + q];
    }
    stats->booked_steps = (long long)c.stat[S_BOOKED];
    stats->transport_steps[1] += stats->booked_steps;
    stats->bytes_per_track = (long long)sizeof(Rec<R>);
  }
  if (tout) tout->n = (int)std::min<long long>(c.extracted, INT32_MAX);
  if (c.err_flags & kErrEvent)
    return set_error(GX_ERR_ARG, "transport: a primary's event index is outside [0, nevents = %d)", cfg->nevents);
  if (c.err_flags & kErrOverflow) return set_error(GX_ERR_OVERFLOW, "transport: track stores and stacks full");
  if (tout && c.extracted > tout->capacity)
    return set_error(GX_ERR_OVERFLOW, "gx_transport_tracks: %lld tracks alive, the output holds %d", c.extracted,
                     tout->capacity);
  if (c.err_flags) return set_error(GX_ERR_ITERCAP, "transport: an iteration cap was hit (flags %d)", c.err_flags);
  return GX_OK;
}


// ------------------------------------------------- the stages of one step
// gx_gpil, gx_propagate, gx_along_step, gx_post_step: OneStep cut at the
// points where the reference's process interface hands over (GPIL, the move,
// the along-step DoIt, the post-step DoIt), one thread per track of a
// caller's gx_track_soa, FP64; the state carried from one stage to the next
// is the SoA's (lambda_inv*, pstep, process, step, boundary, next_volume).
// Multiple scattering is not offered stage by stage (its along-step state is
// not part of the SoA); K: kKindFieldMap or 0.
struct StageArgs {
  const Data *d;
  Geom g;
  gx_track_soa t, sec;
  double *edep;
  double *escaped;
  int sorted; // the blocks work in the order of stage_track
};

__device__ __forceinline__ void soa_load(const gx_track_soa &s, int i, Track<double> &t)
{
  t.type = s.type[i];
  t.pos[0] = s.x[i];
  t.pos[1] = s.y[i];
  t.pos[2] = s.z[i];
  t.dir[0] = s.dx[i];
  t.dir[1] = s.dy[i];
  t.dir[2] = s.dz[i];
  t.E = s.ekin[i];
  t.nil[0] = s.nil0[i];
  t.nil[1] = s.nil1[i];
  t.nil[2] = s.nil2[i];
  t.msc_r0 = s.msc_range ? s.msc_range[i] : -1.0;
  t.load_rng(s.rng, s.capacity, i);
  t.vol = s.volume[i];
  t.event = s.event ? s.event[i] : 0;
  t.prim = s.primary ? s.primary[i] : -1;
}

// the state a stage may change
__device__ __forceinline__ void soa_store(const gx_track_soa &s, int i, const Track<double> &t)
{
  s.x[i] = t.pos[0];
  s.y[i] = t.pos[1];
  s.z[i] = t.pos[2];
  s.dx[i] = t.dir[0];
  s.dy[i] = t.dir[1];
  s.dz[i] = t.dir[2];
  s.ekin[i] = t.E;
  s.nil0[i] = t.nil[0];
  s.nil1[i] = t.nil[1];
  s.nil2[i] = t.nil[2];
  if (s.msc_range) s.msc_range[i] = t.msc_r0;
  t.store_rng(s.rng, s.capacity, i);
  s.volume[i] = t.vol;
}

// the step context of a track from its SoA fields (after gx_gpil)
__device__ __forceinline__ void soa_ctx(const gx_track_soa &s, int i, const Track<double> &t, StepCtx<double> &c)
{
  c.xs0 = s.lambda_inv0[i];
  c.xs1 = s.lambda_inv1[i];
  c.xs2 = s.lambda_inv2[i];
  c.sel = s.process[i];
  c.vol0 = t.vol;
  c.newvol = t.vol;
  c.crossed = false;
  c.nsub = 0;
  c.remaining = 0.0;
  c.total = 0.0;
  c.lam0 = 0.0;
  c.e0 = t.E;
  c.ttrue = 0.0;
  c.range0 = -1.0;
}

__device__ __forceinline__ void stage_local(Local &L, const StageArgs &a)
{
  L.sm_edep = nullptr;
  L.g_edep = a.edep;
  L.sm_esc = a.escaped;
  L.nvol = a.g.nvol;
  L.nevents = a.g.nevents;
  L.sm_bins = 0;
  L.retired = 0.0;
  L.err = 0;
#pragma unroll
  for (int k = 0; k < kNStat; ++k) L.st[k] = 0;
}

// The tracks of a stage's block in the order of `key` (0 .. 15, -1: nothing to
// do): the thread's track, -1 for none.  A batch in flight mixes particle types
// and processes, whose models a warp of gx_post_step would run one after another;
// sorted within a block of kStageBlock, most warps run one of them (400000 tracks
// 508 us in the batch's order, 196 in this; 100003 99 and 51; 32000 53 and 39;
// 16000 39 and 35; 8000 31 and 35, so from kStageSortFrom on).  The other stages,
// whose types share most of the code, gain nothing by it.  Every thread of the
// block calls it.
constexpr int kStageBlock = 256, kStageSortFrom = 16384;
__device__ __forceinline__ int stage_track(int key)
{
  __shared__ int first[17], order[kStageBlock];
  const int t = threadIdx.x;
  if (t < 17) first[t] = 0;
  order[t] = -1;
  __syncthreads();
  const int rank = key >= 0 ? atomicAdd(&first[key + 1], 1) : 0;
  __syncthreads();
  if (t == 0)
    for (int k = 1; k < 17; ++k) first[k] += first[k - 1];
  __syncthreads();
  if (key >= 0) order[first[key] + rank] = blockIdx.x * blockDim.x + t;
  __syncthreads();
  return order[t];
}
template <int K> __global__ void __launch_bounds__(128) k_stage_gpil(StageArgs a)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.t.n || a.t.status[i] != GX_TRACK_ALIVE) return;
  Track<double> t;
  soa_load(a.t, i, t);
  if (t.vol < -1) t.vol = locate(a.g, t.pos, t.dir);
  if (t.vol < 0) { // outside the world
    a.t.volume[i] = t.vol;
    a.t.status[i] = GX_TRACK_EXITED;
    return;
  }
  StepCtx<double> c;
  const double ps = step_gpil<double, K>(*a.d, a.g, t, c);
  soa_store(a.t, i, t);
  a.t.pstep[i] = ps;
  a.t.process[i] = c.sel;
  a.t.lambda_inv0[i] = c.xs0;
  a.t.lambda_inv1[i] = c.xs1;
  a.t.lambda_inv2[i] = c.xs2;
  a.t.safety[i] = nav_safety<K>(a.g, t.vol, t.pos);
  int plane;
  a.t.snext[i] = fmin(nav_distance<K>(a.g, t.vol, t.pos, t.dir, ps, plane), ps);
}

template <int K> __global__ void __launch_bounds__(128) k_stage_propagate(StageArgs a)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.t.n || a.t.status[i] != GX_TRACK_ALIVE) return;
  Track<double> t;
  soa_load(a.t, i, t);
  StepCtx<double> c;
  soa_ctx(a.t, i, t, c);
  Local L;
  stage_local(L, a);
  if (step_move_begin<double, K>(a.g, t, c, a.t.pstep[i]))
    while (!field_substep<double, K>(*a.d, a.g, t, c, L)) {
    }
  soa_store(a.t, i, t);
  a.t.step[i] = c.total;
  a.t.boundary[i] = c.crossed ? 1 : 0;
  a.t.next_volume[i] = c.crossed ? c.newvol : t.vol;
}

template <int K> __global__ void __launch_bounds__(128) k_stage_along(StageArgs a)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.t.n || a.t.status[i] != GX_TRACK_ALIVE) return;
  Track<double> t;
  soa_load(a.t, i, t);
  StepCtx<double> c;
  soa_ctx(a.t, i, t, c);
  c.crossed = a.t.boundary[i] != 0;
  c.newvol = a.t.next_volume[i];
  c.total = a.t.step[i];
  Local L;
  stage_local(L, a);
  int proc = -1;
  const int r = step_end<double, K>(*a.d, a.g, t, c, L, &proc);
  soa_store(a.t, i, t);
  a.t.process[i] = (r == kInteract) ? proc : -1;
  a.t.status[i] = (r == kInteract) ? GX_TRACK_INTERACT
                  : (r == kAlive)  ? GX_TRACK_ALIVE
                  : (c.crossed && c.newvol == -1) ? GX_TRACK_EXITED
                                                  : GX_TRACK_KILLED;
}

template <int K> __global__ void __launch_bounds__(kStageBlock) k_stage_post(StageArgs a)
{
  const int own = blockIdx.x * blockDim.x + threadIdx.x;
  int key = -1; // interacting: by type and process; 15: only the secondaries' slots to clear
  if (own < a.t.n)
    key = a.t.status[own] == GX_TRACK_INTERACT ? min(max(a.t.type[own] * 3 + a.t.process[own], 0), 14) : 15;
  const int i = a.sorted ? stage_track(key) : (key >= 0 ? own : -1);
  if (i < 0) return;
  int nsec = 0;
  if (a.t.status[i] == GX_TRACK_INTERACT) {
    Track<double> t;
    soa_load(a.t, i, t);
    Secs<double> sec;
    sec.n = 0;
    Local L;
    stage_local(L, a);
    run_model(*a.d, a.g, t, a.t.process[i], sec, L);
    Mrg rng = t.rng();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k >= sec.n) break;
      Track<double> ch;
      ch.type = sec.type[k];
      ch.pos[0] = t.pos[0];
      ch.pos[1] = t.pos[1];
      ch.pos[2] = t.pos[2];
      ch.dir[0] = sec.dir[k][0];
      ch.dir[1] = sec.dir[k][1];
      ch.dir[2] = sec.dir[k][2];
      ch.E = sec.E[k];
      ch.nil[0] = ch.nil[1] = ch.nil[2] = -1.0;
      ch.msc_r0 = -1.0;
      Mrg cr;
      rng.seed_child(cr);
      ch.set_rng(cr);
      ch.vol = t.vol;
      ch.event = t.event;
      ch.prim = -1;
      const int j = 2 * i + k;
      soa_store(a.sec, j, ch);
      a.sec.type[j] = ch.type;
      a.sec.status[j] = GX_TRACK_ALIVE;
      if (a.sec.event) a.sec.event[j] = ch.event;
      if (a.sec.primary) a.sec.primary[j] = -1;
      a.sec.next_volume[j] = ch.vol;
      a.sec.process[j] = -1;
      a.sec.boundary[j] = 0;
      a.sec.lambda_inv0[j] = a.sec.lambda_inv1[j] = a.sec.lambda_inv2[j] = 0.0;
      a.sec.pstep[j] = a.sec.step[j] = a.sec.snext[j] = a.sec.safety[j] = 0.0;
      ++nsec;
    }
    t.set_rng(rng);
    soa_store(a.t, i, t);
    a.t.process[i] = -1;
    a.t.status[i] = t.E > 0.0 ? GX_TRACK_ALIVE : GX_TRACK_KILLED;
  }
  for (int k = nsec; k < 2; ++k) {
    a.sec.status[2 * i + k] = GX_TRACK_KILLED;
    a.sec.type[2 * i + k] = -1;
  }
}

// One stage (0 gpil, 1 propagate, 2 along, 3 post) over a track SoA.
int run_stage(int stage, Ctx *C, const gx_transport_config *cfg, gx_track_soa *t, gx_track_soa *sec, double *d_edep,
              int nvol, cudaStream_t s)
{
  StageArgs a;
  std::memset(&a, 0, sizeof(a));
  a.d = C->dev;
  make_geom(C, cfg, nvol, a.g);
  a.t = *t;
  if (sec) a.sec = *sec;
  a.edep = d_edep;
  a.escaped = C->stage_scratch;
  if (t->n <= 0) return GX_OK;
  a.sorted = stage == 3 && t->n >= kStageSortFrom;
  const int block = a.sorted ? kStageBlock : 128, grid = (t->n + block - 1) / block;
  const bool fm = cfg->field_map != 0;
  switch (stage) {
  case 0: (fm ? k_stage_gpil<kKindFieldMap> : k_stage_gpil<0>)<<<grid, block, 0, s>>>(a); break;
  case 1: (fm ? k_stage_propagate<kKindFieldMap> : k_stage_propagate<0>)<<<grid, block, 0, s>>>(a); break;
  case 2: (fm ? k_stage_along<kKindFieldMap> : k_stage_along<0>)<<<grid, block, 0, s>>>(a); break;
  default: (fm ? k_stage_post<kKindFieldMap> : k_stage_post<0>)<<<grid, block, 0, s>>>(a); break;
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GX_OK : cuda_error(e, "gx stage launch");
}

// gx_transport_tracks in this variant (FP64 here, or FP32-mixed)
int run_tracks(Ctx *C, const gx_transport_config *cfg, const gx_track_soa *in, int max_iter, gx_track_soa *out,
               double *d_edep, int nvol, gx_transport_stats *stats, cudaStream_t s)
{
#ifndef GX_PARITY
  if (cfg->precision == 1)
    return run<float>(C, cfg, in->n, nullptr, nullptr, nullptr, nullptr, nullptr, d_edep, nvol, nullptr, stats, s, in,
                      max_iter, out);
#endif
  return run<double>(C, cfg, in->n, nullptr, nullptr, nullptr, nullptr, nullptr, d_edep, nvol, nullptr, stats, s, in,
                     max_iter, out);
}

#ifdef GX_PARITY
// The FP64 transport of gx_transport_run with gx_transport_config.fp64_parity
int run_transport(Ctx *C, const gx_transport_config *cfg, int nprim, const int *d_type, const double *d_E,
                  const double *d_pos, const double *d_dir, const int *d_event, double *d_edep, int nvol,
                  int *d_pstep, gx_transport_stats *stats, cudaStream_t s)
{
  return run<double>(C, cfg, nprim, d_type, d_E, d_pos, d_dir, d_event, d_edep, nvol, d_pstep, stats, s);
}
} // namespace parity
#endif
} // namespace gx

#ifndef GX_PARITY
using namespace gx;

extern "C" {

void gx_transport_config_default(gx_transport_config *c)
{
  std::memset(c, 0, sizeof(*c));
  c->geometry = 1;
  c->axis = 2;
  c->nlayers = 50;
  c->t_abs = 2.3;
  c->t_gap = 5.7;
  c->half_trans = 200.0;
  c->box_mat = 1;
  c->max_steps = 1000000;
  for (int k = 0; k < 6; ++k) c->seed[k] = 12345.0;
  c->nevents = 1;
  c->precision = 0;
  c->engine = 1;
}

int gx_timeline_reset(gx_ctx *ctx)
{
#ifdef GX_TIMELINE
  if (!ctx) return set_error(GX_ERR_ARG, "gx_timeline_reset: null context");
  cudaError_t e = cudaSetDevice(reinterpret_cast<Ctx *>(ctx)->device);
  if (e != cudaSuccess) return cuda_error(e, "gx_timeline_reset: cudaSetDevice");
  static unsigned long long h[kTimelineRows * kTimelineKernels][2];
  for (int i = 0; i < kTimelineRows * kTimelineKernels; ++i) {
    h[i][0] = ~0ULL; // first start: a minimum
    h[i][1] = 0ULL;  // last end: a maximum
  }
  if ((e = cudaMemcpyToSymbol(g_timeline, h, sizeof(h))) != cudaSuccess) return cuda_error(e, "gx_timeline_reset");
  return GX_OK;
#else
  (void)ctx;
  return set_error(GX_ERR_ARG, "gx_timeline_reset: the library was built without GX_TIMELINE "
                               "(python geantexascalepilot_b200/build.py --timeline builds libgxb200_timeline.so)");
#endif
}

int gx_timeline_read(gx_ctx *ctx, unsigned long long *h_out, long long n)
{
#ifdef GX_TIMELINE
  if (!ctx || !h_out) return set_error(GX_ERR_ARG, "gx_timeline_read: null argument");
  if (n != (long long)kTimelineRows * kTimelineKernels * 2)
    return set_error(GX_ERR_ARG, "gx_timeline_read: n must be %d", kTimelineRows * kTimelineKernels * 2);
  cudaError_t e = cudaSetDevice(reinterpret_cast<Ctx *>(ctx)->device);
  if (e != cudaSuccess) return cuda_error(e, "gx_timeline_read: cudaSetDevice");
  if ((e = cudaDeviceSynchronize()) != cudaSuccess) return cuda_error(e, "gx_timeline_read: synchronize");
  if ((e = cudaMemcpyFromSymbol(h_out, g_timeline, sizeof(g_timeline))) != cudaSuccess)
    return cuda_error(e, "gx_timeline_read");
  return GX_OK;
#else
  (void)ctx;
  (void)h_out;
  (void)n;
  return set_error(GX_ERR_ARG, "gx_timeline_read: the library was built without GX_TIMELINE "
                               "(python geantexascalepilot_b200/build.py --timeline builds libgxb200_timeline.so)");
#endif
}

// The checks of a transport configuration shared by the entry points.
static int check_config(const Ctx *C, const gx_transport_config *cfg, int nvol, const char *who)
{
  if (cfg->geometry == 1 && (cfg->nlayers <= 0 || cfg->t_abs <= 0 || cfg->t_gap <= 0 || cfg->half_trans <= 0 ||
                             nvol < 2 * cfg->nlayers))
    return set_error(GX_ERR_ARG, "%s: bad calorimeter (nvol must be >= 2 nlayers)", who);
  if (cfg->axis < 0 || cfg->axis > 2 || cfg->precision < 0 || cfg->precision > 1 || cfg->engine < 0 ||
      cfg->engine > 1 || cfg->nevents < 1)
    return set_error(GX_ERR_ARG, "%s: bad config", who);
  if (cfg->box_mat < 0 || cfg->box_mat > 2) return set_error(GX_ERR_ARG, "%s: bad box material", who);
  if (cfg->block_size && (cfg->block_size % 32 || cfg->block_size > 1024))
    return set_error(GX_ERR_ARG, "%s: block_size must be a multiple of 32, at most 1024", who);
  if (cfg->block_size > 256 && (cfg->engine != 1 || cfg->fp64_parity || cfg->geometry == 2 || cfg->msc ||
                                cfg->field_map))
    return set_error(GX_ERR_ARG, "%s: blocks above 256 threads are for the batched engine with the uniform field, "
                                 "layered geometry and no multiple scattering", who);
  if (cfg->interaction_interval < 0 || cfg->interaction_interval > 64)
    return set_error(GX_ERR_ARG, "%s: interaction_interval must be 0 .. 64", who);
  for (int q = 0; q < 3; ++q)
    if (cfg->fetch_min_by_type[q] < 0 || cfg->fetch_min_by_type[q] > 32)
      return set_error(GX_ERR_ARG, "%s: fetch_min_by_type must be 0 .. 32", who);
  if (cfg->field_map && !C->host.fmap)
    return set_error(GX_ERR_ARG, "%s: field_map = 1 without a field map (gx_ctx_load_field_map)", who);
  if (cfg->geometry < 0 || cfg->geometry > 2) return set_error(GX_ERR_ARG, "%s: bad geometry", who);
  if (cfg->msc < 0 || cfg->msc > 2) return set_error(GX_ERR_ARG, "%s: msc must be 0, 1 or 2", who);
  if (cfg->geometry == 2 && !C->csg_node)
    return set_error(GX_ERR_ARG, "%s: geometry 2 without a volume tree (gx_ctx_load_geometry)", who);
  if (cfg->geometry == 2 && nvol != C->csg_nscore)
    return set_error(GX_ERR_ARG, "%s: nvol %d, the volume tree has %d scored touchables", who, nvol, C->csg_nscore);
  if (cfg->fp64_parity < 0 || cfg->fp64_parity > 1 || (cfg->fp64_parity && cfg->precision != 0))
    return set_error(GX_ERR_ARG, "%s: fp64_parity must be 0 or 1, and 1 needs precision 0", who);
  return GX_OK;
}

// The arrays every stage and the hand-over read or write.
static bool soa_complete(const gx_track_soa *t)
{
  return t && t->n >= 0 && t->capacity >= t->n && t->type && t->status && t->volume && t->next_volume && t->process &&
         t->boundary && t->x && t->y && t->z && t->dx && t->dy && t->dz && t->ekin && t->nil0 && t->nil1 && t->nil2 &&
         t->lambda_inv0 && t->lambda_inv1 && t->lambda_inv2 && t->pstep && t->step && t->snext && t->safety && t->rng;
}

int gx_transport_run(gx_ctx *ctx, const gx_transport_config *cfg, int nprim, const int *d_type, const double *d_E,
                     const double *d_pos, const double *d_dir, const int *d_event, double *d_edep, int nvol,
                     int *d_primary_steps, gx_transport_stats *stats, gx_stream_t s)
{
  if (!ctx || !cfg) return set_error(GX_ERR_ARG, "gx_transport_run: null argument");
  if (nprim < 0 || (nprim > 0 && (!d_type || !d_E || !d_pos || !d_dir)) || !d_edep || nvol <= 0)
    return set_error(GX_ERR_ARG, "gx_transport_run: bad arguments");
  Ctx *C = reinterpret_cast<Ctx *>(ctx);
  int rc = check_config(C, cfg, nvol, "gx_transport_run");
  if (rc) return rc;
  cudaSetDevice(C->device);
  if (cfg->fp64_parity)
    return parity::run_transport(C, cfg, nprim, d_type, d_E, d_pos, d_dir, d_event, d_edep, nvol, d_primary_steps,
                                 stats, stream_of(s));
  if (cfg->precision == 1)
    return run<float>(C, cfg, nprim, d_type, d_E, d_pos, d_dir, d_event, d_edep, nvol, d_primary_steps, stats,
                      stream_of(s));
  return run<double>(C, cfg, nprim, d_type, d_E, d_pos, d_dir, d_event, d_edep, nvol, d_primary_steps, stats,
                     stream_of(s));
}

static int stage_entry(int stage, gx_ctx *ctx, const gx_transport_config *cfg, gx_track_soa *t, gx_track_soa *sec,
                       double *d_edep, int nvol, gx_stream_t s, const char *who)
{
  if (!ctx || !cfg || !soa_complete(t)) return set_error(GX_ERR_ARG, "%s: null argument or incomplete track SoA", who);
  if (stage >= 2 && (!d_edep || nvol <= 0)) return set_error(GX_ERR_ARG, "%s: no tally", who);
  if (stage == 3 && (!soa_complete(sec) || sec->capacity < 2 * t->n))
    return set_error(GX_ERR_ARG, "%s: the secondaries' SoA needs capacity 2 n", who);
  Ctx *C = reinterpret_cast<Ctx *>(ctx);
  int rc = check_config(C, cfg, nvol > 0 ? nvol : 2 * cfg->nlayers, who);
  if (rc) return rc;
  if (cfg->msc || cfg->geometry == 2)
    return set_error(GX_ERR_ARG, "%s: the stage calls take msc = 0 and geometry 0 or 1 (use gx_transport_tracks)", who);
  cudaSetDevice(C->device);
  if (!C->stage_scratch) {
    cudaError_t e = cudaMalloc((void **)&C->stage_scratch, 8 * sizeof(double));
    if (e != cudaSuccess) return cuda_error(e, "stage scratch");
    C->owned.push_back(C->stage_scratch);
    cudaMemset(C->stage_scratch, 0, 8 * sizeof(double));
  }
  if (stage == 3) sec->n = 2 * t->n;
  if (cfg->fp64_parity) return parity::run_stage(stage, C, cfg, t, sec, d_edep, nvol, stream_of(s));
  return run_stage(stage, C, cfg, t, sec, d_edep, nvol, stream_of(s));
}

int gx_gpil(gx_ctx *ctx, const gx_transport_config *cfg, gx_track_soa *tracks, gx_stream_t s)
{
  return stage_entry(0, ctx, cfg, tracks, nullptr, nullptr, 0, s, "gx_gpil");
}

int gx_propagate(gx_ctx *ctx, const gx_transport_config *cfg, gx_track_soa *tracks, gx_stream_t s)
{
  return stage_entry(1, ctx, cfg, tracks, nullptr, nullptr, 0, s, "gx_propagate");
}

int gx_along_step(gx_ctx *ctx, const gx_transport_config *cfg, gx_track_soa *tracks, double *d_edep, int nvol,
                  gx_stream_t s)
{
  return stage_entry(2, ctx, cfg, tracks, nullptr, d_edep, nvol, s, "gx_along_step");
}

int gx_post_step(gx_ctx *ctx, const gx_transport_config *cfg, gx_track_soa *tracks, gx_track_soa *secondaries,
                 double *d_edep, int nvol, gx_stream_t s)
{
  return stage_entry(3, ctx, cfg, tracks, secondaries, d_edep, nvol, s, "gx_post_step");
}

int gx_transport_tracks(gx_ctx *ctx, const gx_transport_config *cfg, const gx_track_soa *in, int max_iterations,
                        gx_track_soa *out, double *d_edep, int nvol, gx_transport_stats *stats, gx_stream_t s)
{
  if (!ctx || !cfg || !soa_complete(in) || !soa_complete(out) || !d_edep || nvol <= 0 || max_iterations < 0)
    return set_error(GX_ERR_ARG, "gx_transport_tracks: bad arguments");
  if (in->rng == out->rng || in->x == out->x || in->status == out->status)
    return set_error(GX_ERR_ARG, "gx_transport_tracks: in and out share arrays");
  Ctx *C = reinterpret_cast<Ctx *>(ctx);
  int rc = check_config(C, cfg, nvol, "gx_transport_tracks");
  if (rc) return rc;
  cudaSetDevice(C->device);
  out->n = 0;
  if (cfg->fp64_parity) return parity::run_tracks(C, cfg, in, max_iterations, out, d_edep, nvol, stats, stream_of(s));
  return run_tracks(C, cfg, in, max_iterations, out, d_edep, nvol, stats, stream_of(s));
}

int gx_transport_run_host(gx_ctx *ctx, const gx_transport_config *cfg, int nprim, const int *h_type,
                          const double *h_E, const double *h_pos, const double *h_dir, const int *h_event,
                          double *h_edep, int nvol, int *h_primary_steps, gx_transport_stats *stats)
{
  if (!ctx || !cfg || nprim < 0 || !h_edep || nvol <= 0 || (nprim > 0 && (!h_type || !h_E || !h_pos || !h_dir)))
    return set_error(GX_ERR_ARG, "gx_transport_run_host: bad arguments");
  Ctx *C = reinterpret_cast<Ctx *>(ctx);
  cudaSetDevice(C->device);
  const size_t n = (size_t)(nprim > 0 ? nprim : 1), nt = (size_t)cfg->nevents * nvol;
  // one staging buffer and one stream kept by the context, grown when a call
  // needs more: no allocation, no stream creation per call
  auto pad = [](size_t b) { return (b + 255) & ~size_t(255); };
  const size_t b_int = pad(n * sizeof(int)), b_dbl = pad(n * sizeof(double)), b_vec = pad(3 * n * sizeof(double));
  const size_t need = 3 * b_int + 2 * b_vec + b_dbl + pad(nt * sizeof(double));
  cudaError_t e;
  if (!C->host_stream && (e = cudaStreamCreateWithFlags(&C->host_stream, cudaStreamNonBlocking)) != cudaSuccess)
    return cuda_error(e, "gx_transport_run_host: stream");
  if (need > C->host_buf_bytes) {
    if (C->host_buf) cudaFree(C->host_buf);
    C->host_buf = nullptr;
    C->host_buf_bytes = 0;
    if ((e = cudaMalloc(&C->host_buf, need)) != cudaSuccess) return cuda_error(e, "gx_transport_run_host: staging");
    C->host_buf_bytes = need;
  }
  cudaStream_t s = C->host_stream;
  char *b = (char *)C->host_buf;
  int *dt = (int *)b, *dev = (int *)(b + b_int), *dps = (int *)(b + 2 * b_int);
  double *dp = (double *)(b + 3 * b_int), *dd = (double *)(b + 3 * b_int + b_vec);
  double *dE = (double *)(b + 3 * b_int + 2 * b_vec), *ded = (double *)(b + 3 * b_int + 2 * b_vec + b_dbl);
  if (nprim > 0) {
    cudaMemcpyAsync(dt, h_type, nprim * sizeof(int), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dE, h_E, nprim * sizeof(double), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dp, h_pos, 3 * nprim * sizeof(double), cudaMemcpyHostToDevice, s);
    cudaMemcpyAsync(dd, h_dir, 3 * nprim * sizeof(double), cudaMemcpyHostToDevice, s);
    if (h_event) cudaMemcpyAsync(dev, h_event, nprim * sizeof(int), cudaMemcpyHostToDevice, s);
  }
  cudaMemsetAsync(ded, 0, nt * sizeof(double), s);
  if (h_primary_steps) cudaMemsetAsync(dps, 0, n * sizeof(int), s);
  int rc = gx_transport_run(ctx, cfg, nprim, dt, dE, dp, dd, h_event ? dev : nullptr, ded, nvol,
                            h_primary_steps ? dps : nullptr, stats, reinterpret_cast<gx_stream_t>(s));
  if (!rc) {
    cudaMemcpyAsync(h_edep, ded, nt * sizeof(double), cudaMemcpyDeviceToHost, s);
    if (h_primary_steps) cudaMemcpyAsync(h_primary_steps, dps, nprim * sizeof(int), cudaMemcpyDeviceToHost, s);
  }
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess && !rc) rc = cuda_error(e, "gx_transport_run_host copy back");
  return rc;
}

} // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free transport (gx_transport_run_noalloc).
//
// For callers that must not allocate device memory while they run -- a host
// framework whose caching allocator owns the device memory, a process under a
// fixed memory budget, a time-critical loop that cannot absorb the implicit
// device synchronisation of cudaMalloc/cudaFree -- this entry point runs the
// plain FP64 loop on one static device array owned by the library instead of
// allocating track stores, the control block, the primary-energy prefix sums
// and the skip-ahead table.  Limits: at most kNoallocCapacity tracks in
// flight (mixed store), as many deferred on the stack, at most
// kNoallocMaxPrimaries primaries per call.  The array is shared by every call
// on a device and keeps the last call's contents; each call rewrites the parts
// that must start from zero (the control block) before its first launch.
// Calls that overlap on the GPU (two streams, two host threads) race on it.
// The first call on a device sets up that device (cudaGetSymbolAddress and
// the skip-ahead table upload).
// Every call synchronises its stream after each iteration (the host reads the
// control block to decide whether to go on).  The set-up is kept for the life
// of the process: a cudaDeviceReset while the library is loaded is not
// supported (the array would come back zeroed without its skip-ahead table).
namespace gx {

constexpr long long kNoallocCapacity = 16384;
constexpr int kNoallocMaxPrimaries = 4096;
static_assert(kNoallocCapacity == GX_NOALLOC_CAPACITY && kNoallocMaxPrimaries == GX_NOALLOC_MAX_PRIMARIES,
              "the limits of the allocation-free entry point must match gx_abi.h");
constexpr size_t kNoallocStoreBytes = 128 * (size_t)kNoallocCapacity; // FP64 record with type field
constexpr size_t kNoallocCtlBytes = 4096;
constexpr size_t kNoallocCumEBytes = sizeof(double) * kNoallocMaxPrimaries;
constexpr size_t kNoallocJumpBytes = sizeof(uint64_t) * 2 * 64 * 9;
constexpr size_t kNoallocBytes = 3 * kNoallocStoreBytes + kNoallocCtlBytes + kNoallocCumEBytes + kNoallocJumpBytes;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocBytes];

static std::mutex g_noalloc_mu;
static unsigned char *g_noalloc_ptr[64] = {nullptr};

// Once per device, with that device current: the device address of the
// static array, and the skip-ahead table written into it.
static int noalloc_setup(int dev, unsigned char **out)
{
  static_assert(sizeof(Ctl) <= kNoallocCtlBytes, "control block does not fit");
  if (dev < 0 || dev >= 64) return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: device index %d", dev);
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_error(e, "gx_transport_run_noalloc: cudaGetSymbolAddress");
    uint64_t h[2][64][9];
    build_jump_host(h);
    unsigned char *base = (unsigned char *)p;
    e = cudaMemcpy(base + 3 * kNoallocStoreBytes + kNoallocCtlBytes + kNoallocCumEBytes, h, sizeof(h),
                   cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cuda_error(e, "gx_transport_run_noalloc: skip-ahead table");
    g_noalloc_ptr[dev] = base;
  }
  *out = g_noalloc_ptr[dev];
  return GX_OK;
}

} // namespace gx

extern "C" int gx_transport_run_noalloc(gx_ctx *ctx, const gx_transport_config *cfg, int nprim, const int *d_type,
                                        const double *d_E, const double *d_pos, const double *d_dir,
                                        const int *d_event, double *d_edep, int nvol, gx_transport_stats *stats,
                                        gx_stream_t stream)
{
  using namespace gx;
  if (!ctx || !cfg) return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: null argument");
  if (nprim < 0 || (nprim > 0 && (!d_type || !d_E || !d_pos || !d_dir)) || !d_edep || nvol <= 0)
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: bad arguments");
  if (nprim > kNoallocMaxPrimaries)
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: %d primaries exceed the static limit of %d", nprim,
                     kNoallocMaxPrimaries);
  if (cfg->precision != 0)
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: FP64 only (precision must be 0)");
  if (cfg->geometry != 0 && cfg->geometry != 1)
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: geometry 0 or 1 only (the volume tree's per-touchable "
                                 "tally is allocated: use gx_transport_run)");
  if (cfg->geometry == 1 && (cfg->nlayers <= 0 || cfg->t_abs <= 0 || cfg->t_gap <= 0 || cfg->half_trans <= 0 ||
                             nvol < 2 * cfg->nlayers))
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: bad calorimeter (nvol must be >= 2 nlayers)");
  if (cfg->axis < 0 || cfg->axis > 2 || cfg->nevents < 1 || cfg->box_mat < 0 || cfg->box_mat > 2)
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: bad config");
  if (cfg->block_size && (cfg->block_size % 32 || cfg->block_size > 256))
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: block_size must be a multiple of 32, at most 256");
  Ctx *C = reinterpret_cast<Ctx *>(ctx);
  if (cfg->field_map && !C->host.fmap)
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: field_map = 1 without a field map");
  cudaError_t err = cudaSetDevice(C->device);
  if (err != cudaSuccess) return cuda_error(err, "gx_transport_run_noalloc: cudaSetDevice");
  unsigned char *base = nullptr;
  int rc = noalloc_setup(C->device, &base);
  if (rc) return rc;
  cudaStream_t s = stream_of(stream);
  const long long cap = kNoallocCapacity;

  Launch<double> L;
  std::memset(&L.a, 0, sizeof(L.a));
  size_t off = 0;
  uintptr_t b = (uintptr_t)base;
  L.a.st[0][0] = carve<double>(b, off, cap);
  L.a.st[1][0] = carve<double>(b, off, cap);
  L.a.stack[0] = carve<double>(b, off, cap);
  if (off != 3 * kNoallocStoreBytes) return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: layout");
  for (int q = 1; q < 3; ++q) {
    L.a.st[0][q] = L.a.st[0][0];
    L.a.st[1][q] = L.a.st[1][0];
    L.a.stack[q] = L.a.stack[0];
  }
  Ctl *ctl = (Ctl *)(base + 3 * kNoallocStoreBytes);
  double *cumE = (double *)(base + 3 * kNoallocStoreBytes + kNoallocCtlBytes);
  const uint64_t *jump = (const uint64_t *)(base + 3 * kNoallocStoreBytes + kNoallocCtlBytes + kNoallocCumEBytes);
  L.a.d = C->dev;
  L.a.ctl = ctl;
  make_geom(C, cfg, nvol, L.a.g);
  L.a.p.type = d_type;
  L.a.p.event = d_event;
  L.a.p.E = d_E;
  L.a.p.pos = d_pos;
  L.a.p.dir = d_dir;
  for (int k = 0; k < 6; ++k) L.a.p.seed[k] = cfg->seed[k];
  L.a.p.first_substream = cfg->first_substream;
  L.a.p.jump = jump;
  L.a.edep = d_edep;
  L.a.pstep = nullptr;
  L.a.nstores = 1;
  L.a.refill_below = cfg->refill_below > 0 ? std::min(cfg->refill_below, cap) : cap / 2;
  L.block = cfg->block_size > 0 ? cfg->block_size : 256;
  L.grid = C->num_sms * (cfg->blocks_per_sm > 0 ? cfg->blocks_per_sm : 4);
  L.smem = kTallyDoubles * sizeof(double);

  // the control block starts from zero on every call
  Ctl h;
  std::memset(&h, 0, sizeof(h));
  h.nprim = nprim;
  h.iterations = -1;
  h.cumE = cumE;
  h.wave_energy = cfg->wave_energy > 0 ? cfg->wave_energy : default_wave_energy(cap, kWaveFillPlain);
  h.refill_below = L.a.refill_below;
  h.stack_cap = cap;
  if ((err = cudaMemcpyAsync(ctl, &h, sizeof(Ctl), cudaMemcpyHostToDevice, s)) != cudaSuccess ||
      (err = cudaStreamSynchronize(s)) != cudaSuccess)
    return cuda_error(err, "gx_transport_run_noalloc: control block");
  if (nprim > 0) k_prefix_energy<<<1, 1024, 0, s>>>(d_E, nprim, cumE, nullptr);
  k_finish<<<1, kFinishBlock, 0, s>>>(ctl, cap, cap, cap, 1, 1, 0, 0);
  Ctl hc;
  long long iters = 0;
  for (;;) {
    k_refill<double><<<L.grid, L.block, 0, s>>>(L.a);
    (cfg->msc ? (cfg->field_map ? k_step<double, 3, 5> : k_step<double, 3, 4>)
              : (cfg->field_map ? k_step<double, 3, 1> : k_step<double, 3, 0>))<<<L.grid, L.block, L.smem, s>>>(L.a);
    k_finish<<<1, kFinishBlock, 0, s>>>(ctl, cap, cap, cap, 1, 1, 0, 0);
    if ((err = cudaGetLastError()) != cudaSuccess) return cuda_error(err, "gx_transport_run_noalloc: launch");
    if ((err = cudaMemcpyAsync(&hc, ctl, sizeof(Ctl), cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (err = cudaStreamSynchronize(s)) != cudaSuccess)
      return cuda_error(err, "gx_transport_run_noalloc: iteration");
    ++iters;
    if (hc.in_flight == 0 && hc.pending == 0) break;
    if (iters > 2000000LL) return set_error(GX_ERR_ITERCAP, "gx_transport_run_noalloc: iteration cap");
  }
  if (stats) {
    std::memset(stats, 0, sizeof(*stats));
    stats->steps = (long long)hc.stat[S_STEPS];
    stats->substeps = (long long)hc.stat[S_SUBSTEPS];
    stats->tracks = total_tracks(hc);
    for (int q = 0; q < 3; ++q) stats->secondaries[q] = (long long)hc.stat[S_SEC0 + q];
    stats->n_pair = (long long)hc.stat[S_PAIR];
    stats->n_annih = (long long)hc.stat[S_ANNIH];
    stats->errors = (long long)(hc.stat[S_ERR] + hc.stat[S_OVERFLOW]);
    stats->escaped = hc.escaped;
    stats->iterations = hc.iterations;
    stats->peak_in_flight = hc.peak;
    stats->tracks_read[0] = (long long)hc.stat[S_READ0];
    stats->tracks_written[0] = (long long)hc.stat[S_WRITE0];
    stats->bytes_per_track = (long long)sizeof(Rec<double>);
  }
  if (hc.err_flags & kErrEvent)
    return set_error(GX_ERR_ARG, "gx_transport_run_noalloc: a primary's event index is outside [0, nevents = %d)",
                     cfg->nevents);
  if (hc.err_flags & kErrOverflow)
    return set_error(GX_ERR_OVERFLOW, "gx_transport_run_noalloc: more than %lld tracks in flight and deferred",
                     2 * kNoallocCapacity);
  if (hc.err_flags) return set_error(GX_ERR_ITERCAP, "gx_transport_run_noalloc: an iteration cap was hit");
  return GX_OK;
}
#endif // GX_PARITY
