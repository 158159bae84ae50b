// Kernels of the photon-propagation hot path (sm_100a).
//
//  batched_kernel  persistent: each warp pulls runs of photons of any pair from a
//                  device work queue and refills a lane as soon as its photon
//                  ends, so lanes never idle behind a long-lived photon and
//                  thousands of uneven pairs run in one launch.
//  plain_kernel    one pair per launch, one photon per thread at a time
//                  (grid-stride), the straightforward port of the reference's
//                  thread loop (src/photon_prop_cuda.jl:301-380).
//  stacks_kernel   cuda_propagate_photons! with the reference's output layout
//                  (per-block hit stacks, src/photon_prop_cuda.jl:262-386).
//  setup_kernel, fill_kernel   zeroed statistics and histograms, counters,
//                  work queue.
//  normalize_kernel  histograms per photon (PP_OPT_NORMALIZE).
//  eval_kernel     device helpers on test inputs.
//  peak kernels    FP32 / MUFU / INT issue microbenchmarks for the roofline.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "pp_device.cuh"
#include "pp_internal.h"
#include "pp_special.cuh"

namespace ppd {

// ---------------------------------------------------------------------------
// Batched persistent kernel.
//
// The work queue is one row of granules of 32 photons over all pairs
// (granule_offsets; a pair's last granule may be short).  Each warp takes runs
// of granules from it and emits one granule at a time, converged.  What
// follows differs by mode:
//
// Physical mode: photons end after very different numbers of steps (3.4 on
// average in the mixed batch), so the warp stages emissions in a ring of
// kStage photons in shared memory, dead lanes pick staged photons up with
// four 16-byte loads, and all 32 lanes step together.
//
// Compat mode: every photon makes max_steps steps unless it hits, so the 32
// emitted photons step in lockstep to their end: no ring, no refill, and
// the lanes of the few that hit idle.  Where many have hit with many steps
// still to come (at most kThinLive live lanes, at least kThinSteps steps), the
// warp goes over to refilling its idle lanes, kRefill or more at a time, until
// all are idle at once.  One source, 100 steps, 2e8 photons of which 4, 20, 30,
// 45, 80 % hit at once: 82.6, 83.1, 83.4, 84.0, 85.2 ms in lockstep alone; with
// the ring that physical mode has 110.5, 97.3, 87.9, 74.2, 42.5 ms; now
// 80.5, 81.8, 75.2, 62.4, 29.3 ms.  25 steps, 4e8 photons, 20 and 80 %: 43.8 and
// 48.5 ms, 59.0 and 51.2 with the ring, now 43.7 and 25.5.  kThinLive of 18 or 20
// costs 2 to 3 % at 20 % hits, where a granule falls below it by chance;
// kThinSteps of 12 up to 10 % there.  With 10 steps lockstep is twice as
// fast as the ring at any share (24.1 against 46.4 ms at 80 %), and its kernel
// without the other loop (THIN) 2 % faster on 2e7 photons.
//
// Bound by instruction issue (78 % of the issue slots, ALU half-rate pipe
// 48 %); what counts is instructions per photon.  512 mixed pairs (2.52e8
// photons): 6.30e9 -> 4.94e9 warp instructions, 6.99 -> 5.57 ms, by testing
// the reach where a photon stops (in_reach), one emission pass per pair with
// its record by broadcast, and separate loops for the full warp and for the
// last photons; 4096 mixed pairs (5.75e9 photons): 171 -> 138 ms.  Cascade
// pairs: 25.3 warp instructions per photon against 19.6 of the mixed batch
// (3.68 steps against 3.37, a longer emission; its table reads hit L1 and do
// not stall), issue 75 %.  Compat mode (100 distances, 2e9 photons): 139.4 ->
// 90.1 ms, 124 warp instructions per step with the emission's tenth and the
// hits; the last step leaves out the move and turn that nothing follows, steps
// are counted by what hits leave out, a batch of hits adds its sums over the
// warp.  Measured and not kept: the first one or two steps of physical mode
// inside the emission pass (fewer loop iterations, but 180 bytes spilled at 64
// registers: 14 % slower).
constexpr int kStage = 64;  // >= 2 * 32 - 1 staged emissions per warp (power of two)

constexpr unsigned kThinLive = 16, kRefill = 8;
constexpr int kThinSteps = 24;

// The ring holds a photon's 16 words as four arrays of 16-byte words, so that
// neighbouring lanes read and write neighbouring words (one 64-byte record
// per photon put the lanes of a store or load on a quarter of the banks):
//   0: px py pz dx   1: dy dz neg_ln2_len path
//   2: index lo, the first step's counter word, pair, the pair's sphere radius (a refill reads shared memory only)
//   3: the step stream's words, a, q
//
// The part of a warp's run that lies in one pair, with a copy of the pair's
// record, is kept in shared memory too: only the emission pass reads or
// advances it, so the step loop holds no registers for it.  A pass emits
// photons of one pair, so it reads the record by broadcast.
template <int MODE>
struct __align__(16) WarpArea {
  float4 ring[4][MODE == kPhysical ? kStage : 1];
  float4 rec[5];                       // the current pair's pp_pair
  unsigned long long base;             // its next photon index
  unsigned long long run_at, run_end;  // the granules of the run that follow in other pairs
  unsigned left;                       // the pair's photons left in the run
  int pair;
  unsigned long long not_made;  // compat: steps that hits left out
  WarpStats stats;
};
static_assert(sizeof(pp_pair) == 5 * sizeof(float4), "the record is copied as 16-byte words");

// Compat mode hits often: a photon whose line meets the sphere beyond its
// step waits in place, pointing at it, until a step reaches it (3.6 % of the
// photons of make_photon_fits hit, against 4e-5 in physical mode).  There a
// hit lane stages its photon in shared memory and the warp records up to 32
// staged hits together, converged, instead of one or two lanes walking the
// hit path while the others wait.
constexpr unsigned kHitStage = 32;
struct StagedHit {
  float px, py, pz, dx, dy, dz, path;
  uint32_t id_lo, id_hi;
  int32_t pair;
  int32_t left;  // steps that the hit leaves out
};

// Register budget: 64 per thread (1024 threads per SM) for the basic
// emitters; the cascade variant's table lookups in the emission block spill
// at 64, so it gets 80 (768 threads per SM), which runs cone and isotropic
// pairs as fast as the basic variant does.
template <int MODE, int WARPS, int EM, bool THIN = false>
__global__ void __launch_bounds__(WARPS * 32, (EM == kEmCascade ? 768 : 1024) / (WARPS * 32))
    batched_kernel(const RunParams R) {
  __shared__ __align__(16) DevTables T;
  __shared__ WarpArea<MODE> area[WARPS];
  __shared__ StagedHit hstage[MODE == kCompat ? WARPS : 1][kHitStage];
  stage_tables(T, R.tables);
  const unsigned lane = threadIdx.x & 31u;
  WarpArea<MODE>* wa = &area[threadIdx.x >> 5];
  if (lane == 0) {
    wa->stats.pair = -1;
    for (int k = 0; k < 6; ++k) wa->stats.v[k] = 0.0;
    wa->left = 0;
    wa->pair = 0;
    wa->not_made = 0;
    wa->run_at = wa->run_end = 0;
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");  // what the set-up kernel writes is read below

  const unsigned lt_mask = (1u << lane) - 1u;
  WarpStats* ws = &wa->stats;
  StagedHit* hst = hstage[MODE == kCompat ? (threadIdx.x >> 5) : 0];
  unsigned h_count = 0;  // staged hits, warp-uniform
  // records staged hits 0..n-1 (n warp-uniform), one per lane
  auto record_staged = [&](unsigned n) {
    __syncwarp();
    const bool valid = lane < n;
    const StagedHit& g = hst[valid ? lane : 0u];
    Photon p;
    p.px = g.px;
    p.py = g.py;
    p.pz = g.pz;
    p.dx = g.dx;
    p.dy = g.dy;
    p.dz = g.dz;
    p.path = g.path;
    p.neg_ln2_len = 0.f;
    p.id_lo = g.id_lo;
    p.ctr3 = g.id_hi;  // block 0: the index's top bits only
    p.sc0 = p.sc1 = 0u;
    const PairCtx pc{0.f, g.pair};
    const HitValues h = hit_values<MODE, EM>(T, R, R.pairs + g.pair, p);
    add_warp_stats(R, ws, valid, g.pair, h);
    const unsigned less = __reduce_add_sync(kFull, valid ? (unsigned)g.left : 0u);
    if (lane == 0) wa->not_made += less;
    if (valid) store_hit(R, pc, p, h);
    __syncwarp();
  };
  // takes the hits of a step (all lanes call)
  auto take_hits = [&](bool hit, const Photon& p, const PairCtx& c, int left) -> bool {
    if (MODE == kCompat) {
      const unsigned hm = __ballot_sync(kFull, hit);
      if (!hm) return false;
      const unsigned nh = __popc(hm);
      if (h_count + nh > kHitStage) {  // no room: record what is staged first
        record_staged(h_count);
        h_count = 0;
      }
      if (hit) {
        StagedHit& g = hst[h_count + __popc(hm & lt_mask)];
        g.px = p.px;
        g.py = p.py;
        g.pz = p.pz;
        g.dx = p.dx;
        g.dy = p.dy;
        g.dz = p.dz;
        g.path = p.path;
        g.id_lo = p.id_lo;
        g.id_hi = p.ctr3 & 0xFFu;
        g.pair = c.index;
        g.left = left;
      }
      h_count += nh;
      return true;
    }
    if (!__any_sync(kFull, hit)) return false;
    if (hit) {
      const HitValues h = hit_values<MODE, EM>(T, R, R.pairs + c.index, p);
      record_hit_cached(R, ws, c, p, h);
    }
    return true;
  };
  // the next pair of the warp's run, or of its next run, with its record and
  // statistics cache; false when the queue is exhausted.  A run is half the
  // warps' share of what was left when the warp last looked, between one
  // granule and R.max_run of them: long runs while there is much to do (a
  // lookup per 4096 photons), short ones at the end, so that the warps finish
  // together, and a small batch spreads over all of them.
  auto fetch = [&]() {
    __syncwarp();  // every lane has read the run and added its hits' sums before lane 0 writes them
    int p = -1;
    if (lane == 0) {
      unsigned long long at = wa->run_at, end = wa->run_end;
      const unsigned long long total = R.granule_offsets[R.n_pairs];
      if (at >= end) {
        const unsigned long long share = (total - min(end, total)) / (2u * gridDim.x * WARPS);
        const unsigned long long n = max(1ull, min(share, (unsigned long long)R.max_run));
        at = atomicAdd(R.queue, n);
        end = min(at + n, total);
      }
      if (at < end) {
        int hi = (int)R.n_pairs - 1;  // last pair whose first granule <= at
        p = 0;
        while (p < hi) {
          const int mid = (p + hi + 1) >> 1;
          if (R.granule_offsets[mid] <= at) p = mid; else hi = mid - 1;
        }
        const unsigned long long first = R.granule_offsets[p], stop = min(end, R.granule_offsets[p + 1]);
        const unsigned long long start = (at - first) * 32u;
        wa->base = start;
        wa->left = (unsigned)min((stop - at) * 32u, (unsigned long long)R.pairs[p].n_photons - start);
        wa->run_at = stop;
        wa->run_end = end;
        wa->pair = p;
        if (EM == kEmBasic && R.pairs[p].emitter == PP_EMITTER_CASCADE)
          atomicOr(R.counters + 2, 4ull);  // a cascade pair in a launch without PP_OPT_CASCADE
        if (p != ws->pair) {               // the warp's statistics cache follows its run
          flush_warp_stats(R.stats, ws);
          ws->pair = p;
        }
      }
    }
    p = __shfl_sync(kFull, p, 0);
    if (p >= 0 && lane < 5u) wa->rec[lane] = __ldg(reinterpret_cast<const float4*>(R.pairs + p) + lane);
    __syncwarp();
    return p >= 0;
  };
  // emits the pair's next photons, at most `most`, the lane's the one of its
  // rank (lanes past the last emit as well, and drop it); returns whether the
  // lane has one that is in reach
  unsigned steps = 0;  // beyond those that the set-up kernel has counted (physical mode)
  auto emit = [&](Photon& e, PairCtx& c, unsigned rank, unsigned most) {
    const unsigned left = wa->left, n = min(most, left);
    const uint64_t base = wa->base;
    c.index = wa->pair;
    __syncwarp();
    wa->base = base + n;  // by every lane: the same values
    wa->left = left - n;
    set_photon(e, base + rank);
    const PairRec P = staged_pair(wa->rec);
    c.r = P.tgt_r.w;
    const bool near = emit_event<MODE, EM>(T, R, P, e);
    return near && rank < n;
  };

  if constexpr (MODE == kCompat) {
    for (;;) {
      if (wa->left == 0u && !fetch()) break;
      Photon s;
      PairCtx c;
      bool alive = emit(s, c, lane, 32u), hit, more, thin = false;
      for (int left = R.max_steps - 1; left > 0; --left) {
        step_event<MODE>(R, c, s, hit, more);
        hit = hit && alive;
        if (take_hits(hit, s, c, left)) {
          alive = alive && !hit;
          const unsigned live = __popc(__ballot_sync(kFull, alive));
          if (THIN) thin = live <= kThinLive && left >= kThinSteps;
          if (thin || live == 0u) break;
        }
      }
      if (!THIN || !thin) {
        step_event<MODE, true>(R, c, s, hit, more);
        take_hits(hit && alive, s, c, 0);
        continue;
      }
      bool dry = false;  // the queue is exhausted
      for (;;) {         // each lane at its photon's own step, until all are done at once
        const unsigned need = __ballot_sync(kFull, !alive), idle = __popc(need);
        if (need == kFull) break;
        if (!dry && idle >= kRefill) {
          dry = wa->left == 0u && !fetch();
          if (!dry) {
            Photon e;
            PairCtx ec;
            if (emit(e, ec, __popc(need & lt_mask), idle) && !alive) {
              s = e;
              c = ec;
              alive = true;
            }
          }
        }
        step_event<MODE>(R, c, s, hit, more);
        hit = hit && alive;
        take_hits(hit, s, c, R.max_steps + 1 - (int)(s.ctr3 >> 8));
        alive = alive && more;
      }
    }
  } else {
    // warp-uniform state of the ring, and the lane's photon and pair (radius
    // and index: the rest of its record, which only a hit's emission replay
    // needs, is read then)
    unsigned r_head = 0, r_count = 0;
    bool alive = false;
    Photon s;
    s.id_lo = 0;
    s.ctr3 = 1u << 8;
    s.sc0 = s.sc1 = 0u;
    s.px = s.py = s.pz = s.dx = s.dy = s.path = s.neg_ln2_len = 0.f;
    s.dz = 1.f;
    s.a = s.q = 0.f;
    PairCtx c;
    c.r = 0.f;
    c.index = 0;
    // the lane's next photon: the ring's entry of its rank among the lanes in need
    auto take_staged = [&](unsigned need) {
      const unsigned slot = (r_head + __popc(need & lt_mask)) & (kStage - 1);
      const float4 a = wa->ring[0][slot], b = wa->ring[1][slot], d = wa->ring[2][slot], e = wa->ring[3][slot];
      s.px = a.x;
      s.py = a.y;
      s.pz = a.z;
      s.dx = a.w;
      s.dy = b.x;
      s.dz = b.y;
      s.neg_ln2_len = b.z;
      s.path = b.w;
      s.id_lo = __float_as_uint(d.x);
      s.ctr3 = __float_as_uint(d.y);
      c.index = __float_as_int(d.z);
      c.r = d.w;
      s.sc0 = __float_as_uint(e.x);
      s.sc1 = __float_as_uint(e.y);
      s.a = e.z;
      s.q = e.w;
    };
    // While the ring can fill every lane in need, all 32 lanes step together
    // and nothing else is tested.
    for (;;) {
      const unsigned need = __ballot_sync(kFull, !alive), n_need = __popc(need);
      // emission passes, until the ring can (photons that start out of reach
      // are not staged) or the queue is exhausted
      while (r_count < n_need) {
        if (wa->left == 0u && !fetch()) break;
        Photon e;
        PairCtx ec;
        const bool near = emit(e, ec, lane, 32u);
        const unsigned keep = __ballot_sync(kFull, near);
        if (near) {
          const unsigned slot = (r_head + r_count + __popc(keep & lt_mask)) & (kStage - 1);
          wa->ring[0][slot] = make_float4(e.px, e.py, e.pz, e.dx);
          wa->ring[1][slot] = make_float4(e.dy, e.dz, e.neg_ln2_len, e.path);
          wa->ring[2][slot] = make_float4(__uint_as_float(e.id_lo), __uint_as_float(e.ctr3),
                                          __int_as_float(ec.index), ec.r);
          wa->ring[3][slot] = make_float4(__uint_as_float(e.sc0), __uint_as_float(e.sc1), e.a, e.q);
        }
        r_count += __popc(keep);
        __syncwarp();
      }
      if (r_count < n_need) break;
      if (!alive) take_staged(need);
      r_head += n_need;
      r_count -= n_need;
      bool hit, more;
      alive = step_event<MODE>(R, c, s, hit, more);
      steps += more ? 1u : 0u;
      take_hits(hit, s, c, 0);
    }
    // The ring's last photons, then ever fewer lanes.
    for (;;) {
      const unsigned need = __ballot_sync(kFull, !alive);
      if (!alive && __popc(need & lt_mask) < r_count) {
        take_staged(need);
        alive = true;
      }
      if (need == kFull && r_count == 0u) break;  // every lane was idle and none took a photon
      const unsigned took = min((unsigned)__popc(need), r_count);
      r_head += took;
      r_count -= took;
      bool hit = false, more = false;
      if (alive) alive = step_event<MODE>(R, c, s, hit, more);
      steps += more ? 1u : 0u;
      take_hits(hit, s, c, 0);
    }
  }
  if (MODE == kCompat && h_count > 0u) record_staged(h_count);
  __syncwarp();
  if (lane == 0) flush_warp_stats(R.stats, ws);
  // photon-step count for the roofline
  unsigned long long st = steps;
  if (MODE == kCompat) {
    st = 0ull - wa->not_made;
  } else {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) st += __shfl_xor_sync(kFull, st, o);
  }
  if (lane == 0) atomicAdd(R.counters + 1, st);
}

// ---------------------------------------------------------------------------
// Plain kernel: one pair, photons id = gtid + i * stride.
template <int MODE, int EM>
__global__ void __launch_bounds__(512) plain_kernel(const RunParams R, const pp_pair* __restrict__ pair_ptr,
                                                    int pair_index) {
  __shared__ __align__(16) DevTables T;
  stage_tables(T, R.tables);
  __syncthreads();
  const PairCtx c{pair_ptr->radius, pair_index};
  const unsigned long long n = (unsigned long long)pair_ptr->n_photons;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned steps = 0;
  for (unsigned long long id = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; id < n;
       id += stride) {
    Photon s;
    set_photon(s, id);
    s.dx = s.dy = 0.f;
    s.dz = 1.f;
    bool alive = true;
    while (alive) {
      bool hit = false;
      alive = photon_event<MODE, EM>(T, R, pair_ptr, c, s, hit, steps);
      if (hit) {
        const HitValues h = hit_values<MODE, EM>(T, R, pair_ptr, s);
        record_hit(R, c, s, h, 0);
      }
    }
  }
  unsigned long long st = steps;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) st += __shfl_xor_sync(kFull, st, o);
  if ((threadIdx.x & 31u) == 0) atomicAdd(R.counters + 1, st);
}

// ---------------------------------------------------------------------------
// Step events that a propagation of these pairs makes: counters[1] counts the
// step that would only find a photon out of reach, which no kernel makes.
// A diagnostic of the rates' denominators (one thread per photon, nothing
// recorded), so that the batched kernel need not count both.
template <int MODE, int EM>
__global__ void __launch_bounds__(256) made_steps_kernel(const RunParams R, unsigned long long* __restrict__ out) {
  __shared__ __align__(16) DevTables T;
  stage_tables(T, R.tables);
  __syncthreads();
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long made = 0;
  for (int64_t p = blockIdx.y; p < R.n_pairs; p += gridDim.y) {
    const PairCtx c{R.pairs[p].radius, (int)p};
    const long long photons = R.pairs[p].n_photons;
    const unsigned long long n = photons > 0 ? (unsigned long long)photons : 0ull;
    for (unsigned long long id = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; id < n; id += stride) {
      Photon s;
      set_photon(s, id);
      bool hit, more, alive = emit_event<MODE, EM>(T, R, load_pair(R.pairs + p), s);
      for (; alive; ++made) {
        alive = step_event<MODE>(R, c, s, hit, more);
        if (MODE == kCompat) alive = more;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) made += __shfl_xor_sync(kFull, made, o);
  if ((threadIdx.x & 31u) == 0) atomicAdd(out, made);
}

// ---------------------------------------------------------------------------
// cuda_propagate_photons! layout (src/photon_prop_cuda.jl:262-386).  Photon
// ids: thread g simulates ids g + i * (blocks * threads), i < per_thread.
template <int MODE>
__global__ void __launch_bounds__(1024) stacks_kernel(const RunParams R, const pp_pair* __restrict__ pair_ptr,
                                                      float* __restrict__ out_pos, float* __restrict__ out_dir,
                                                      float* __restrict__ out_wl, float* __restrict__ out_dist,
                                                      int32_t* __restrict__ out_sp,
                                                      long long* __restrict__ out_nsim, int stack_len,
                                                      long long per_thread) {
  __shared__ __align__(16) DevTables T;
  __shared__ int cursor;
  stage_tables(T, R.tables);
  const int ix_offset = (int)blockIdx.x * stack_len + 1;  // 1-based, as in the reference
  if (threadIdx.x == 0) cursor = ix_offset;
  __syncthreads();
  const PairCtx c{pair_ptr->radius, 0};
  const int safe_margin = max(0, (int)blockDim.x - 32);
  const unsigned long long G = (unsigned long long)gridDim.x * blockDim.x;
  const unsigned long long g = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long n_sim = 0;
  unsigned steps = 0;
  for (long long i = 0; i < per_thread; ++i) {
    if (*(volatile int*)&cursor > ix_offset + stack_len - safe_margin) break;
    Photon s;
    set_photon(s, g + (unsigned long long)i * G);
    s.dx = s.dy = 0.f;
    s.dz = 1.f;
    bool alive = true;
    while (alive) {
      bool hit = false;
      alive = photon_event<MODE, kEmCascade>(T, R, pair_ptr, c, s, hit, steps);
      if (hit) {
        const HitValues h = hit_values<MODE, kEmCascade>(T, R, pair_ptr, s);
        const int idx = atomicAdd(&cursor, 1);  // 1-based slot
        if (idx < ix_offset + stack_len) {
          const int j = idx - 1;
          out_pos[3 * j + 0] = h.px;
          out_pos[3 * j + 1] = h.py;
          out_pos[3 * j + 2] = h.pz;
          out_dir[3 * j + 0] = h.d0x;
          out_dir[3 * j + 1] = h.d0y;
          out_dir[3 * j + 2] = h.d0z;
          out_wl[j] = h.wl;
          out_dist[j] = h.dist;
          atomicMax(out_sp + blockIdx.x, idx);
        } else {
          atomicOr(R.counters + 2, 1ull);
        }
      }
    }
    ++n_sim;
  }
  atomicAdd(reinterpret_cast<unsigned long long*>(out_nsim), (unsigned long long)n_sim);
  atomicAdd(R.counters + 1, (unsigned long long)steps);
}

// ---------------------------------------------------------------------------
// The outputs of a launch before it: statistics rows (zeros, and the photon
// count in column 6) and zeroed histograms, by threads first, first + stride, ...
__device__ __forceinline__ void fill_outputs(const pp_pair* __restrict__ pairs, int64_t n, double* __restrict__ stats,
                                             double* __restrict__ hist, int64_t hist_len, int64_t first,
                                             int64_t stride) {
  if (stats)
    for (int64_t i = first; i < n * PP_STATS; i += stride)
      stats[i] = i % PP_STATS == 6 ? (double)pairs[i / PP_STATS].n_photons : 0.0;
  if (hist) {  // 16-byte stores from the first 16-byte boundary on
    const int64_t head = min((int64_t)((reinterpret_cast<uintptr_t>(hist) >> 3) & 1u), hist_len);
    double2* body = reinterpret_cast<double2*>(hist + head);
    const int64_t nb = (hist_len - head) / 2;
    for (int64_t i = first; i < nb; i += stride) body[i] = make_double2(0.0, 0.0);
    if (first == 0) {
      if (head) hist[0] = 0.0;
      if (head + 2 * nb < hist_len) hist[hist_len - 1] = 0.0;
    }
  }
}

__global__ void __launch_bounds__(1024) fill_kernel(const pp_pair* __restrict__ pairs, int64_t n,
                                                    double* __restrict__ stats, double* __restrict__ hist,
                                                    int64_t hist_len) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // setup_kernel scans meanwhile
  fill_outputs(pairs, n, stats, hist, hist_len, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
               (int64_t)gridDim.x * blockDim.x);
}

// The work queue of a launch.  Block 0 resets the queue cursor and the
// counters and writes the offsets: offsets[p] = granules (32 photons) of pairs
// 0..p-1, offsets[n] all of them; counters[1] starts as photon_steps per
// photon: physical mode the first one, to which the batched kernel adds the
// others, compat mode max_steps, from which it takes what hits leave out.
// offsets == NULL (the one-pair kernel, which counts all its steps): no queue.
// Further blocks, if any, fill the outputs.
__global__ void __launch_bounds__(1024) setup_kernel(const pp_pair* __restrict__ pairs, int64_t n,
                                                     unsigned long long* __restrict__ offsets,
                                                     unsigned long long* __restrict__ queue,
                                                     unsigned long long* __restrict__ counters,
                                                     double* __restrict__ stats, double* __restrict__ hist,
                                                     int64_t hist_len, unsigned photon_steps) {
  // the batched kernel may start (its blocks wait for this grid to end
  // before they read what it writes)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int t = threadIdx.x;
  if (blockIdx.x > 0) {
    fill_outputs(pairs, n, stats, hist, hist_len, (int64_t)(blockIdx.x - 1) * blockDim.x + t,
                 (int64_t)(gridDim.x - 1) * blockDim.x);
    return;
  }
  __shared__ unsigned long long granules[32], photons[32];
  const unsigned lane = t & 31, warp = t >> 5;
  unsigned long long done = 0, seen = 0;  // granules of the tiles before; this thread's photons
  constexpr int kPer = 4;                 // pairs per thread and tile, loaded together
  if (offsets) {
    for (int64_t tile = 0; tile < n; tile += (int64_t)kPer * blockDim.x) {
      unsigned long long g[kPer], sum = 0;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int64_t i = tile + (int64_t)t * kPer + j;
        const long long np = i < n ? (long long)__ldg(reinterpret_cast<const long long*>(pairs + i) + 6) : 0ll;
        g[j] = np > 0 ? (unsigned long long)np : 0ull;
      }
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        seen += g[j];
        g[j] = (g[j] + 31u) / 32u;
        sum += g[j];
      }
      unsigned long long incl = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(kFull, incl, o);
        if ((int)lane >= o) incl += v;
      }
      if (lane == 31) granules[warp] = incl;
      __syncthreads();
      unsigned long long before = done, all = 0;
#pragma unroll
      for (unsigned w = 0; w < 32; ++w) {  // 32 warps: read by broadcast
        before += w < warp ? granules[w] : 0ull;
        all += granules[w];
      }
      __syncthreads();
      unsigned long long run = before + incl - sum;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const int64_t i = tile + (int64_t)t * kPer + j;
        if (i < n) offsets[i] = run;
        run += g[j];
      }
      done += all;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) seen += __shfl_xor_sync(kFull, seen, o);
  if (lane == 0) photons[warp] = seen;
  __syncthreads();
  if (t == 0) {
    unsigned long long all = 0;
    for (int w = 0; w < 32; ++w) all += photons[w];
    if (offsets) {
      offsets[n] = done;
      queue[0] = 0ull;
    }
    counters[0] = 0ull;
    counters[1] = all * photon_steps;
    counters[2] = 0ull;
    counters[3] = 0ull;
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");  // fill_kernel, where it ran before: its end is part of this grid's
}

// hist[p][:] /= photons.
__global__ void normalize_kernel(const pp_pair* __restrict__ pairs, int64_t n_pairs, double* __restrict__ hist,
                                 int bins) {
  const int64_t total = n_pairs * (int64_t)bins;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double n = (double)pairs[i / bins].n_photons;
    if (n > 0) hist[i] /= n;
  }
}

// ---------------------------------------------------------------------------
__global__ void eval_kernel(int op, const double* __restrict__ in, double* __restrict__ out, int64_t n,
                            const DevTables* __restrict__ tables) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (op == 13 || op == 14) {  // a warp's lanes hold the tables: all take part
    const ppsf::WarpTables W = ppsf::warp_tables();
    const double v = in[min(i, n - 1)], r = op == 13 ? ppsf::exp_tab(v, W) : ppsf::log_tab(v, W);
    if (i < n) out[i] = r;
    return;
  }
  if (i >= n) return;
  const DevTables& T = *tables;
  switch (op) {
    case 0: {
      const double* a = in + 6 * i;
      uint32_t c[4] = {(uint32_t)a[0], (uint32_t)a[1], (uint32_t)a[2], (uint32_t)a[3]};
      philox4x32_10(c, (uint32_t)a[4], (uint32_t)a[5]);
      for (int j = 0; j < 4; ++j) out[4 * i + j] = (double)c[j];
      break;
    }
    case 1: out[i] = (double)u01((uint32_t)in[i]); break;
    case 12: {  // step block: (counter word 0, word 1, key) -> (w0, w1, u0, u1, u2)
      const double* a = in + 3 * i;
      uint32_t w0 = (uint32_t)a[0], w1 = (uint32_t)a[1];
      philox2x32_10(w0, w1, (uint32_t)a[2]);
      const Draw3 d = step_uniforms(w0, w1);
      double* o = out + 5 * i;
      o[0] = (double)w0;
      o[1] = (double)w1;
      o[2] = (double)d.u0;
      o[3] = (double)d.u1;
      o[4] = (double)d.u2;
      break;
    }
    case 2: {
      const float g = (float)in[2 * i];
      const HG h = make_hg(g);
      out[i] = (double)hg_costheta(h, (float)in[2 * i + 1]);
      break;
    }
    case 3: {
      const double* a = in + 6 * i;
      float x, y, z;
      rotate_to_axis((float)a[0], (float)a[1], (float)a[2], (float)a[3], (float)a[4], (float)a[5], x, y, z);
      out[3 * i] = x;
      out[3 * i + 1] = y;
      out[3 * i + 2] = z;
      break;
    }
    case 4: {
      const double* a = in + 7 * i;
      const float st = (float)a[6];
      out[3 * i] = fmaf(st, (float)a[3], (float)a[0]);
      out[3 * i + 1] = fmaf(st, (float)a[4], (float)a[1]);
      out[3 * i + 2] = fmaf(st, (float)a[5], (float)a[2]);
      break;
    }
    case 5: out[i] = (double)draw_wavelength(T, (float)in[i]); break;
    case 6: out[i] = (double)phase_index(T, 1.f / (float)in[i]); break;
    case 7: out[i] = (double)group_index(T, 1.f / (float)in[i]); break;
    case 8: out[i] = (double)scattering_length(T, (float)in[i]); break;
    case 9: out[i] = (double)interp_sorted((float)in[i], T.abs_wl, T.abs_len, T.n_abs); break;
    case 15: ppsf::psi_both(in[i], out[2 * i], out[2 * i + 1]); break;
    case 16: out[i] = ppsf::reciprocal_1_2(in[i]); break;
    case 11: out[i] = (double)cascade_cos_theta(T, 1.f / (float)in[2 * i + 1], (float)in[2 * i]); break;
    case 10:
      out[i] = T.n_pmt > 0 ? (double)interp_sorted((float)in[i], T.pmt_wl, T.pmt_acc, T.n_pmt) : 1.0;
      break;
    default: out[i] = 0.0;
  }
}

// ---------------------------------------------------------------------------
// Issue-rate microbenchmarks: 8 independent dependent chains per thread.
__global__ void peak_fma_kernel(float* out, int iters, float a, float b) {
  float x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = (float)(threadIdx.x + j);
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = fmaf(x[j], a, b);
  }
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += x[j];
  if (s == 1.2345f) out[0] = s;
}

__global__ void peak_mufu_kernel(float* out, int iters) {
  float x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = 0.5f + 0.01f * (float)(threadIdx.x & 7) + 0.001f * j;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = ex2(x[j] * -0.5f);  // ex2 of a value in (0,1): stays in (0,1)
  }
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += x[j];
  if (s == 1.2345f) out[0] = s;
}

__global__ void peak_philox_kernel(unsigned* out, int iters) {
  // independent Philox4x32-10 blocks per thread: the integer work of one photon step
  uint32_t acc = 0;
  for (int i = 0; i < iters; ++i) {
    uint32_t c[4] = {threadIdx.x, blockIdx.x, (uint32_t)i, 0u};
    philox4x32_10(c, 0x12345678u, 0x9abcdef0u);
    acc ^= c[0] ^ c[1] ^ c[2] ^ c[3];
  }
  if (acc == 12345u) out[0] = acc;
}

// Speed of light of the physical step: every lane steps its own photon
// through step_event (one Philox2x32-10 block, the ray-sphere test, the move
// and the Henyey-Greenstein turn) with no emission, refill, hit record or
// loop bookkeeping, at the batched kernel's occupancy (256 threads, 4 CTAs
// per SM, at most 64 registers).  Its step rate bounds what the batched
// kernel can reach on this GPU under instruction-issue limits.  The photons
// start 100 m from a 0.21 m sphere with an unbounded path, so they keep
// moving; the results are kept live through a never-true store.
__global__ void __launch_bounds__(256, 4) peak_step_kernel(const RunParams R, int iters,
                                                           unsigned long long* __restrict__ out) {
  PairCtx c;
  c.r = 0.21f;
  c.index = 0;
  Photon s;
  s.sc0 = 0x9E3779B9u * (blockIdx.x + 1u) ^ threadIdx.x;
  s.sc1 = 0x2545F491u & 0x7FFFFFFu;
  const uint64_t id = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  s.id_lo = (uint32_t)id;
  s.px = 100.f + (float)(threadIdx.x & 31u);
  s.py = 50.f;
  s.pz = -30.f;
  s.dx = 0.6f;
  s.dy = 0.f;
  s.dz = 0.8f;
  s.path = 1e30f;
  s.neg_ln2_len = -kLn2 * 30.f;
  s.ctr3 = ctr_word(id, 1u);
  line_of(s);
  unsigned live = 0, steps = 0;
  for (int i = 0; i < iters; ++i) {
    bool hit, more;
    live += step_event<kPhysical>(R, c, s, hit, more) ? 1u : 0u;
    steps += more ? 1u : 0u;
  }
  if (s.px == 1.2345f && s.dz == 0.5f && live + steps == 7u) out[1] = 1ull;
  if ((threadIdx.x & 31u) == 0) atomicAdd(out, 32ull * (unsigned long long)iters);
}

}  // namespace ppd

// ---------------------------------------------------------------------------
// Launch helpers (host).
namespace pp {

static __host__ ppd::RunParams to_params(const LaunchArgs& a) {
  ppd::RunParams R;
  R.pairs = a.pairs;
  R.n_pairs = a.n_pairs;
  R.granule_offsets = a.granule_offsets;
  R.queue = a.queue;
  R.max_run = std::max(1u, a.chunk / 32u + (a.chunk % 32u != 0u));
  R.pair_base = a.pair_base;
  R.hits = a.hits;
  R.hit_cap = a.hit_cap;
  R.counters = a.counters;
  R.stats = a.stats;
  R.hist = a.hist;
  R.tables = reinterpret_cast<const ppd::DevTables*>(a.tables);
  R.max_steps = a.opts.max_steps;
  R.ctr_limit = ((uint32_t)a.opts.max_steps + 1u) << 8;
  R.t_max = a.opts.t_max;
  R.hist_t0 = a.opts.hist_t0;
  R.inv_bin_width = a.opts.hist_bin_width > 0.f ? 1.f / a.opts.hist_bin_width : 0.f;
  R.hist_bins = a.opts.hist_bins;
  R.flags = a.opts.flags;
  R.hg = ppd::make_hg(a.opts.g);
  return R;
}

size_t dev_tables_size() { return sizeof(ppd::DevTables); }

void fill_dev_tables(void* host_tables, const double coeffs[11], const float* knots, int n_knots,
                     const float* abs_wl, const float* abs_len, int n_abs, const float* pmt_wl,
                     const float* pmt_acc, int n_pmt) {
  ppd::DevTables* t = reinterpret_cast<ppd::DevTables*>(host_tables);
  memset(t, 0, sizeof(*t));
  t->a01 = (float)coeffs[0];
  t->a2 = (float)coeffs[1];
  t->a3 = (float)coeffs[2];
  t->a4 = (float)coeffs[3];
  t->g01 = (float)coeffs[0];
  t->g2 = (float)(2.0 * coeffs[1]);
  t->g3 = (float)(3.0 * coeffs[2]);
  t->g4 = (float)(4.0 * coeffs[3]);
  t->sca0 = (float)coeffs[4];
  t->sca1 = (float)coeffs[5];
  t->sca2 = (float)coeffs[6];
  t->n_knots = n_knots;
  for (int i = 0; i < n_knots; ++i) t->knots[i] = knots[i];
  t->n_cells = n_knots > 1 ? n_knots - 1 : 1;
  if (n_knots == 1) t->knots[1] = t->knots[0];
  t->n_abs = n_abs;
  for (int i = 0; i < n_abs; ++i) {
    t->abs_wl[i] = abs_wl[i];
    t->abs_len[i] = abs_len[i];
  }
  t->n_pmt = n_pmt;
  for (int i = 0; i < n_pmt; ++i) {
    t->pmt_wl[i] = pmt_wl[i];
    t->pmt_acc[i] = pmt_acc[i];
  }
}

void set_cascade_tables(void* host_tables, const float* d_casc, double gmin, double gmax) {
  ppd::DevTables* t = reinterpret_cast<ppd::DevTables*>(host_tables);
  t->casc = d_casc;
  t->casc_nf = kCascNF;
  t->casc_ni = kCascNI;
  t->casc_vmin = (float)kCascVMin;
  t->casc_inv_dv = (float)(kCascNF / (kCascVMax - kCascVMin));
  t->casc_gmin = (float)gmin;
  t->casc_inv_dg = (float)(kCascNI / (gmax - gmin));
}

void get_dev_knots(const void* host_tables, float* out, int* n) {
  const ppd::DevTables* t = reinterpret_cast<const ppd::DevTables*>(host_tables);
  *n = t->n_knots;
  for (int i = 0; i < t->n_knots; ++i) out[i] = t->knots[i];
}

cudaError_t launch_setup(const LaunchArgs& a, int sm_count, cudaStream_t s) {
  const int64_t hist_len = a.hist ? a.n_pairs * (int64_t)a.opts.hist_bins : 0;
  const int64_t words = (a.stats ? a.n_pairs * PP_STATS : 0) + hist_len;
  // 16 words per thread.  What one block fills (a single source, 16 pairs of
  // 1000 bins) is a second block of the set-up kernel, one launch less; beyond,
  // the outputs have a kernel of their own, which the scan's registers do not
  // hold to one block per SM.
  const int64_t blocks = (words + 16383) / 16384;
  const unsigned photon_steps = a.opts.mode == PP_MODE_COMPAT ? (unsigned)a.opts.max_steps : 1u;
  if (blocks <= 1) {
    ppd::setup_kernel<<<1 + (int)blocks, 1024, 0, s>>>(a.pairs, a.n_pairs, a.granule_offsets, a.queue, a.counters,
                                                       a.stats, a.hist, hist_len, photon_steps);
    count_launches(1);
    return cudaGetLastError();
  }
  ppd::fill_kernel<<<(int)std::min<int64_t>(blocks, 2 * (int64_t)sm_count), 1024, 0, s>>>(a.pairs, a.n_pairs, a.stats,
                                                                                          a.hist, hist_len);
  count_launches(1);
  const cudaError_t e = cudaGetLastError();
  if (e) return e;
  return launch_dependent(ppd::setup_kernel, 1, 1024, 0, s, a.pairs, a.n_pairs, a.granule_offsets, a.queue, a.counters,
                          (double*)nullptr, (double*)nullptr, (int64_t)0, photon_steps);
}

namespace {
using BatchedFn = void (*)(ppd::RunParams);
BatchedFn batched_fn(int mode, int block, bool cascade, int max_steps = 0) {
  if (mode == PP_MODE_COMPAT) {
    if (max_steps > ppd::kThinSteps)  // at least kThinSteps steps can be left
      return block == 128 ? ppd::batched_kernel<ppd::kCompat, 4, ppd::kEmBasic, true>
                          : ppd::batched_kernel<ppd::kCompat, 8, ppd::kEmBasic, true>;
    return block == 128 ? ppd::batched_kernel<ppd::kCompat, 4, ppd::kEmBasic>
                        : ppd::batched_kernel<ppd::kCompat, 8, ppd::kEmBasic>;
  }
  if (cascade)
    return block == 128 ? ppd::batched_kernel<ppd::kPhysical, 4, ppd::kEmCascade>
                        : ppd::batched_kernel<ppd::kPhysical, 8, ppd::kEmCascade>;
  return block == 128 ? ppd::batched_kernel<ppd::kPhysical, 4, ppd::kEmBasic>
                      : ppd::batched_kernel<ppd::kPhysical, 8, ppd::kEmBasic>;
}
}  // namespace

// Follows launch_setup on the same stream: the blocks start and stage their
// tables while the set-up kernel runs, then wait for it to end.
cudaError_t launch_batched(const LaunchArgs& a, int grid, int block, cudaStream_t s) {
  const ppd::RunParams R = to_params(a);
  if (block != 128) block = 256;
  const auto fn = batched_fn(a.opts.mode, block, (a.opts.flags & PP_OPT_CASCADE) != 0, a.opts.max_steps);
  return launch_dependent(fn, grid, block, 0, s, R);
}

cudaError_t launch_plain(const LaunchArgs& a, const pp_pair* d_pair, int pair_index, int grid, int block,
                         cudaStream_t s) {
  const ppd::RunParams R = to_params(a);
  if (a.opts.mode == PP_MODE_COMPAT)
    ppd::plain_kernel<ppd::kCompat, ppd::kEmBasic><<<grid, block, 0, s>>>(R, d_pair, pair_index);
  else if (a.opts.flags & PP_OPT_CASCADE)
    ppd::plain_kernel<ppd::kPhysical, ppd::kEmCascade><<<grid, block, 0, s>>>(R, d_pair, pair_index);
  else
    ppd::plain_kernel<ppd::kPhysical, ppd::kEmBasic><<<grid, block, 0, s>>>(R, d_pair, pair_index);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_made_steps(const LaunchArgs& a, unsigned long long* out, int sm_count, cudaStream_t s) {
  const ppd::RunParams R = to_params(a);
  // 32 blocks per SM where the pairs are few, one per pair where they are many
  const int64_t rows = std::min<int64_t>(a.n_pairs, 32768);
  const dim3 grid((unsigned)std::max<int64_t>(1, 32 * (int64_t)sm_count / rows), (unsigned)rows);
  if (a.opts.mode == PP_MODE_COMPAT)
    ppd::made_steps_kernel<ppd::kCompat, ppd::kEmBasic><<<grid, 256, 0, s>>>(R, out);
  else if (a.opts.flags & PP_OPT_CASCADE)
    ppd::made_steps_kernel<ppd::kPhysical, ppd::kEmCascade><<<grid, 256, 0, s>>>(R, out);
  else
    ppd::made_steps_kernel<ppd::kPhysical, ppd::kEmBasic><<<grid, 256, 0, s>>>(R, out);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_stacks(const LaunchArgs& a, const pp_pair* d_pair, float* pos, float* dir, float* wl,
                          float* dist, int32_t* sp, int64_t* nsim, int stack_len, int grid, int block,
                          long long per_thread, cudaStream_t s) {
  const ppd::RunParams R = to_params(a);
  if (a.opts.mode == PP_MODE_COMPAT)
    ppd::stacks_kernel<ppd::kCompat><<<grid, block, 0, s>>>(R, d_pair, pos, dir, wl, dist, sp,
                                                            reinterpret_cast<long long*>(nsim), stack_len,
                                                            per_thread);
  else
    ppd::stacks_kernel<ppd::kPhysical><<<grid, block, 0, s>>>(R, d_pair, pos, dir, wl, dist, sp,
                                                              reinterpret_cast<long long*>(nsim), stack_len,
                                                              per_thread);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_normalize(const pp_pair* pairs, int64_t n, double* hist, int bins, int sm_count, cudaStream_t s) {
  const int64_t total = n * (int64_t)bins;
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, (int64_t)sm_count * 8));
  ppd::normalize_kernel<<<grid, 256, 0, s>>>(pairs, n, hist, bins);
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_eval(int op, const double* in, double* out, int64_t n, const void* tables, cudaStream_t s) {
  const int grid = (int)((n + 127) / 128);
  ppd::eval_kernel<<<grid, 128, 0, s>>>(op, in, out, n, reinterpret_cast<const ppd::DevTables*>(tables));
  count_launches(1);
  return cudaGetLastError();
}

// (both compat variants have the same registers and shared memory)
int batched_max_blocks_per_sm(int mode, int block, bool cascade) {
  int nb = 0;
  if (block != 128) block = 256;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, batched_fn(mode, block, cascade), block, 0);
  return nb;
}

int plain_max_blocks_per_sm(int mode, int block) {
  int nb = 0;
  if (mode == PP_MODE_COMPAT)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ppd::plain_kernel<ppd::kCompat, ppd::kEmBasic>, block, 0);
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, ppd::plain_kernel<ppd::kPhysical, ppd::kEmBasic>, block, 0);
  return nb;
}

cudaError_t run_peaks(int sm_count, double* fp32, double* mufu, double* iops) {
  float* dout = nullptr;
  cudaError_t e = cudaMalloc(&dout, 64);
  if (e != cudaSuccess) return e;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  const int block = 256, grid = sm_count * 8;
  const double threads = (double)grid * block;
  float ms = 0.f;
  // warm-up
  ppd::peak_fma_kernel<<<grid, block>>>(dout, 1000, 0.999f, 0.001f);
  ppd::peak_mufu_kernel<<<grid, block>>>(dout, 100);
  ppd::peak_philox_kernel<<<grid, block>>>(reinterpret_cast<unsigned*>(dout), 100);
  count_launches(3);
  const int it_f = 20000, it_m = 40000, it_i = 4000;
  cudaEventRecord(a);
  ppd::peak_fma_kernel<<<grid, block>>>(dout, it_f, 0.999f, 0.001f);
  cudaEventRecord(b);
  cudaEventSynchronize(b);
  cudaEventElapsedTime(&ms, a, b);
  *fp32 = threads * it_f * 8.0 / (ms * 1e-3);
  cudaEventRecord(a);
  ppd::peak_mufu_kernel<<<grid, block>>>(dout, it_m);
  cudaEventRecord(b);
  cudaEventSynchronize(b);
  cudaEventElapsedTime(&ms, a, b);
  *mufu = threads * it_m * 8.0 / (ms * 1e-3);
  cudaEventRecord(a);
  ppd::peak_philox_kernel<<<grid, block>>>(reinterpret_cast<unsigned*>(dout), it_i);
  cudaEventRecord(b);
  cudaEventSynchronize(b);
  cudaEventElapsedTime(&ms, a, b);
  *iops = threads * it_i / (ms * 1e-3);  // Philox blocks per second
  count_launches(3);
  e = cudaGetLastError();
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  cudaFree(dout);
  return e;
}

cudaError_t run_step_rate(int sm_count, double* steps_per_s) {
  unsigned long long* dout = nullptr;
  cudaError_t e = cudaMalloc(&dout, 16);
  if (e != cudaSuccess) return e;
  cudaMemset(dout, 0, 16);
  LaunchArgs a{};
  a.opts.mode = PP_MODE_PHYSICAL;
  a.opts.max_steps = 1000;
  a.opts.g = 0.95f;
  a.opts.t_max = 1000.f;
  ppd::RunParams R = to_params(a);
  R.ctr_limit = 0xFFFFFFFFu;
  cudaEvent_t t0, t1;
  cudaEventCreate(&t0);
  cudaEventCreate(&t1);
  const int grid = sm_count * 4, block = 256, iters = 20000;
  ppd::peak_step_kernel<<<grid, block>>>(R, 500, dout);  // warm-up
  cudaEventRecord(t0);
  ppd::peak_step_kernel<<<grid, block>>>(R, iters, dout);
  cudaEventRecord(t1);
  cudaEventSynchronize(t1);
  count_launches(2);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, t0, t1);
  *steps_per_s = (double)grid * block * iters / (ms * 1e-3);
  e = cudaGetLastError();
  cudaEventDestroy(t0);
  cudaEventDestroy(t1);
  cudaFree(dout);
  return e;
}

}  // namespace pp
