// sw_kernels.cuh -- the __global__ kernels of the engine.
//
//   k_batched<T, K, LANES>  persistent kernel over a cost-ordered work list;
//                     each warp pulls work items (per group of LANES lanes one
//                     pair for s32 lanes, two for 16-bit halves) from an
//                     atomic queue head.  s16x2 items whose score could have
//                     left int16 are appended to an overflow list that a
//                     second k_batched<LaneS32, K> launch reruns.
//   k_plain<K>        the one-launch-per-batch kernel over the reference's
//                     wire buffer (Seqs || Meta, ipu_batch_affine.cpp:287) with
//                     results in its Scores || ARanges || BRanges layout; one
//                     warp per comparison slot in slot order, s32 lanes.
//   k_exact           one thread per pair with the recurrence written out
//                     cell by cell in int32; used for scoring configurations
//                     that the wavefront kernels do not cover (gI + gE >= 0 or
//                     gE > 0).
//   k_plain16<K>      the same wire-buffer kernel with two slots per warp in
//                     s16x2 halves (a slot that could leave int16 is redone
//                     in s32 by the same warp).
//   k_strips<K>       the strip-team kernel: the warps of a block share the
//                     strips of one item (two pairs in s16x2 halves), each
//                     strip waiting on the boundary rows of the one before
//                     (long pairs whose latency would end the launch).
//   k_bin_*           the cost-binning pre-pass that orders the work list:
//                     k_bin_total (batch cells), k_bin_bound (main-diagonal
//                     bounds of the long pairs, one at a time per warp),
//                     k_bin_count
//                     (class and bucket of every pair), k_bin_scan (list
//                     offsets and class ranges), k_bin_scatter (the list);
//                     k_bin_small does all of it for a few thousand pairs.
#pragma once
#include "sw_device.cuh"
#include "sw_tagged.cuh"

namespace ipuma_dev {

// Pair descriptor of the batched API (matches ipuma_pair in ipuma_b200.h).
struct PairDesc {
  long long a_off;
  long long b_off;
  int a_len;
  int b_len;
};

// Packs (start, end) like codelet_batch_affine.cpp:117-123 (uint16 halves).
__device__ __forceinline__ int pack_range(int start, int end) {
  return (int)(((uint32_t)(uint16_t)start) | (((uint32_t)(uint16_t)end) << 16));
}

// Device-side status words (bounded error reporting, no traps).
struct DevStatus {
  int error;           // first error code seen by any warp (0 = none)
  int overflow_start;  // always 0: {overflow_start, overflow_count} is the
  int overflow_count;  // range of the overflow list for the s32 rerun
  int pad;
};

// Blocks of a class launch that work (those past `blocks` exit at once: all
// of them when the class is empty), and where its strip scratch starts in
// the scratch buffer (int2), so that concurrent launches never share any.
// Written on the device by the binning pre-pass.
struct ClassAllot {
  long long base;
  int blocks;
  int pad;
};

constexpr int ERR_SCRATCH = 1;  // a pass needed more scratch rows than provided
constexpr int ERR_LENGTH = 2;   // a pair exceeded the stated maximum lengths
constexpr int ERR_RANGE = 3;    // a pair's offsets or lengths lie outside the code array
constexpr int ERR_WAIT = 4;     // a strip team's wait for a boundary ran out (kTeamWaitNs)

// What a kernel does with one pair descriptor of a device-resident batch,
// checked before any code is read (the same rules as the host-side check of
// the host-buffer calls): PAIR_OUT for a negative offset or length or a
// sequence reaching past the n_codes residues of the code array (error
// status, zero result), PAIR_EMPTY for an empty sequence (zero result),
// PAIR_LONG beyond the stated maxima (error status, zero result), PAIR_OK.
constexpr int PAIR_OK = 0, PAIR_EMPTY = 1, PAIR_LONG = 2, PAIR_OUT = 3;
__device__ __forceinline__ int pair_state(const PairDesc& d, long long n_codes, int max_a, int max_b) {
  if (d.a_len < 0 || d.b_len < 0 || d.a_off < 0 || d.b_off < 0 || d.a_off > n_codes - d.a_len ||
      d.b_off > n_codes - d.b_len)
    return PAIR_OUT;
  if (d.a_len == 0 || d.b_len == 0) return PAIR_EMPTY;
  if (d.a_len > max_a || d.b_len > max_b) return PAIR_LONG;
  return PAIR_OK;
}

// Records the error of a rejected pair (PAIR_LONG / PAIR_OUT) in the status
// word; the caller writes its zero result.
__device__ __forceinline__ void report_pair(int state, DevStatus* st) {
  if (state == PAIR_LONG) atomicCAS(&st->error, 0, ERR_LENGTH);
  if (state == PAIR_OUT) atomicCAS(&st->error, 0, ERR_RANGE);
}

// Shared-memory layout of the wavefront kernels.
// Per warp: 32 / LANES groups, each with its profile and B-letter ring.
template <class T, int K, int LANES>
struct SmemLayout {
  static constexpr int SW = LANES * K;
  static constexpr int GROUPS = 32 / LANES;
  // M = alphabet size (substitution table), P = letters of the profile.
  __host__ __device__ static int simp_bytes(int M, int P) { return SubTable::bytes(M, P); }
  __host__ __device__ static int prof_bytes(int P) { return T::NP * (P + 1) * LANES * ProfileWords<K>::KP; }
  __host__ __device__ static int ring_bytes() { return 128 * 2 * T::NP; }  // a doubled uint16 ring per pair
  __host__ __device__ static int group_bytes(int P) { return (prof_bytes(P) + ring_bytes() + 15) & ~15; }
  __host__ __device__ static int warp_bytes(int P) { return GROUPS * group_bytes(P); }
  __host__ __device__ static int total(int M, int P, int warps) { return simp_bytes(M, P) + warps * warp_bytes(P); }
};

// One pass of a lane type: tagged 16-bit lanes or sw_pass's lanes.
template <class T>
constexpr bool kTagged = false;
template <int TB, bool LIN, bool SCALED>
constexpr bool kTagged<LaneTag<TB, LIN, SCALED>> = true;
template <>
constexpr bool kTagged<LaneBig> = true;
// Bias (-gE for linear gaps) and scale of a lane type's profile values.
template <class T>
constexpr bool kProfBias = T::LINEAR;
template <class T>
constexpr int kProfShift = 0;
template <int TB, bool LIN, bool SCALED>
constexpr int kProfShift<LaneTag<TB, LIN, SCALED>> = SCALED ? TB : 0;
template <class T, int K, int LANES, bool EARLY = false>
__device__ __forceinline__ bool one_pass(const SwConst& sc, uint8_t* s_prof, const int8_t* s_simp, uint16_t* s_bring,
                                         const PassSeq (&ps)[T::NP], int2* scr, long rowsCap, Best (&out)[T::NP],
                                         PassStop stop = PassStop{}) {
  if constexpr (kTagged<T>)
    return tag_pass<T, K, LANES, EARLY>(sc, s_prof, s_simp, s_bring, ps, scr, rowsCap, out, stop);
  else
    return sw_pass<T, K, LANES>(sc, s_prof, s_simp, s_bring, ps, scr, rowsCap, out);
}

// Forward pass (+ reverse pass unless forwardOnly) for the NP pairs held
// by one lane group.  For 16-bit lanes a pair whose score exceeds the
// lane's limit (or any pair of a warp that gave up) is flagged in `ovf` and
// gets no reverse pass (the s32 rerun redoes it).
// MODE: 0 = by sc.forwardOnly at run time, 1 = forward only, 2 = with the
// reverse pass (a kernel specialised for one mode holds only its code, so
// the forward-only kernels keep their own register allocation).
template <class T, int K, int LANES, int MODE = 0>
__device__ __forceinline__ void align_pairs(const SwConst& sc, uint8_t* s_prof,
                                            const int8_t* s_simp, uint16_t* s_bring, const uint8_t* codes,
                                            const long long (&a0)[T::NP], const long long (&b0)[T::NP],
                                            const int (&alen)[T::NP], const int (&blen)[T::NP],
                                            int2* scr, long rowsCap, Best (&fw)[T::NP],
                                            Best (&rv)[T::NP], bool (&ovf)[T::NP]) {
  constexpr int NP = T::NP;
  PassSeq ps[NP];
#pragma unroll
  for (int h = 0; h < NP; ++h) {
    const bool empty = alen[h] <= 0 || blen[h] <= 0;
    ps[h] = PassSeq{codes, a0[h], b0[h], empty ? 0 : alen[h], empty ? 0 : blen[h], 1, 1};
  }
#pragma unroll
  for (int h = 0; h < NP; ++h) rv[h] = Best{0, 0, 0};
  if (MODE == 1 || (MODE == 0 && sc.forwardOnly)) {
    if constexpr (MODE != 2) {
      const bool done = one_pass<T, K, LANES>(sc, s_prof, s_simp, s_bring, ps, scr, rowsCap, fw);
#pragma unroll
      for (int h = 0; h < NP; ++h) ovf[h] = (NP == 2) && (!done || fw[h].s > Cell<T>::limit(sc));
    }
    return;
  }
  if constexpr (MODE != 1) {
  // With start coordinates both passes run through one copy of the pass: two
  // inlined copies alternating in the instruction cache slowed both down.
  // (A forward-only launch runs only the copy above.)  The reverse pass
  // stops early once every pair reached its forward score (PassStop).
  // Only the kernels specialised for full alignments (MODE 2) take the
  // early stop: it costs registers that the others keep.
  PassStop stop;
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    Best res[NP];
    const bool done = one_pass<T, K, LANES, MODE == 2>(sc, s_prof, s_simp, s_bring, ps, scr, rowsCap, res, stop);
    if (pass == 1) {
#pragma unroll
      for (int h = 0; h < NP; ++h) rv[h] = res[h];
      break;
    }
    bool any = false;
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      fw[h] = res[h];
      ovf[h] = (NP == 2) && (!done || fw[h].s > Cell<T>::limit(sc));
      const bool run = !ovf[h] && fw[h].s > 0;
      any |= run;
      ps[h] = run ? PassSeq{codes, a0[h] + fw[h].j, b0[h] + fw[h].i, fw[h].j + 1, fw[h].i + 1, -1, -1}
                  : PassSeq{codes, a0[h], b0[h], 0, 0, 1, 1};
      stop.target[h] = run ? fw[h].s : 0;
    }
    stop.on = true;
    // Uniform across the warp: every group takes part in the shuffles.
    if (!__any_sync(FULL, any)) break;
  }
  }
}

// One pass of the hybrid class for the two pairs of a 32-lane group: s16x2
// while every strip is provably inside int16, then each pair alone in s32
// lanes from the first strip that is not (its half of the packed boundary
// column as input).  Returns false when the s16x2 part gave up anyway.
template <int K>
__device__ __forceinline__ bool hybrid_pass(const SwConst& sc, uint8_t* s_prof, const int8_t* s_simp,
                                            uint16_t* s_bring, const PassSeq (&ps)[2], int2* scr,
                                            long rowsCap, Best (&out)[2]) {
  PassCtl c16;
  if (!sw_pass<LaneHi, K, 32, true>(sc, s_prof, s_simp, s_bring, ps, scr, rowsCap, out, &c16)) return false;
  if (c16.stoppedAt < 0) return true;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    if (ps[h].alen <= c16.stoppedAt * 32 * K || ps[h].blen <= 0) continue;  // no strip left
    PassCtl c32;
    c32.strip0 = c16.stoppedAt;
    c32.bndHalf = h;
    c32.scrBase = c16.scrBase;
    const PassSeq one[1] = {ps[h]};
    Best o[1] = {out[h]};
    sw_pass<LaneS32, K, 32, true>(sc, s_prof, s_simp, s_bring, one, scr, rowsCap, o, &c32);
    out[h] = o[0];
  }
  return true;
}

// Forward (+ reverse) pass of the hybrid class; as align_pairs (MODE too).
template <int K, int MODE = 0>
__device__ __forceinline__ void align_pairs_hybrid(const SwConst& sc, uint8_t* s_prof, const int8_t* s_simp,
                                                   uint16_t* s_bring, const uint8_t* codes,
                                                   const long long (&a0)[2], const long long (&b0)[2],
                                                   const int (&alen)[2], const int (&blen)[2], int2* scr,
                                                   long rowsCap, Best (&fw)[2], Best (&rv)[2], bool (&ovf)[2]) {
  PassSeq ps[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const bool empty = alen[h] <= 0 || blen[h] <= 0;
    ps[h] = PassSeq{codes, a0[h], b0[h], empty ? 0 : alen[h], empty ? 0 : blen[h], 1, 1};
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) rv[h] = Best{0, 0, 0};
  if (MODE == 1 || (MODE == 0 && sc.forwardOnly)) {
    if constexpr (MODE != 2) {
      const bool done = hybrid_pass<K>(sc, s_prof, s_simp, s_bring, ps, scr, rowsCap, fw);
      ovf[0] = ovf[1] = !done;
    }
    return;
  }
  if constexpr (MODE != 1) {
  // With start coordinates one copy of the hybrid pass serves both
  // directions (as align_pairs).
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    Best res[2];
    const bool done = hybrid_pass<K>(sc, s_prof, s_simp, s_bring, ps, scr, rowsCap, res);
    if (pass == 1) {
      if (done) {
        rv[0] = res[0];
        rv[1] = res[1];
      } else {
        ovf[0] = ovf[1] = true;
      }
      break;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      fw[h] = res[h];
      ovf[h] = !done;
      ps[h] = fw[h].s > 0 ? PassSeq{codes, a0[h] + fw[h].j, b0[h] + fw[h].i, fw[h].j + 1, fw[h].i + 1, -1, -1}
                          : PassSeq{codes, a0[h], b0[h], 0, 0, 1, 1};
    }
    if (!done) break;
  }
  }
}

__device__ __forceinline__ void write_result(const SwConst& sc, const Best& fw, const Best& rv,
                                             int* score, int* arange, int* brange, long idx) {
  const int aend = fw.j, bend = fw.i;
  const int astart = sc.forwardOnly ? 0 : aend - rv.j;
  const int bstart = sc.forwardOnly ? 0 : bend - rv.i;
  score[idx] = fw.s;
  arange[idx] = pack_range(astart, aend);
  brange[idx] = pack_range(bstart, bend);
}

// What the kernels read and write besides their work list.
struct BatchIo {
  const uint8_t* codes;
  const PairDesc* pairs;
  long rowsCap;
  int *score, *arange, *brange, *overflow_list;
  unsigned long long* rerun_cells;
  DevStatus* st;
};

// One work item of a warp: the 32 / LANES * NP list entries from `first`
// on (those below n), lane group g aligning entries [g * NP, g * NP + NP).
//   wsmem : the warp's shared memory (SmemLayout::warp_bytes)
//   wscr  : the warp's strip-boundary scratch
template <class T, int K, int LANES, bool HYB, bool FWD>
__device__ __forceinline__ void batched_item(const SwConst& sc, const BatchIo& io, const int8_t* s_simp, uint8_t* wsmem,
                                             int2* wscr, const int* list, int first, int n) {
  using L = SmemLayout<T, K, LANES>;
  constexpr int NP = T::NP;
  constexpr int NBUF = HYB ? 3 : 2;  // strip-boundary buffers per group
  const int lane32 = threadIdx.x & 31;
  const int group = lane32 / LANES;
  const int glane = lane32 & (LANES - 1);
  uint8_t* s_prof = wsmem + group * L::group_bytes(sc.P);
  uint16_t* s_bring = reinterpret_cast<uint16_t*>(s_prof + L::prof_bytes(sc.P));
  int2* scr = wscr + group * NBUF * io.rowsCap;
  int pid[NP], alen[NP], blen[NP];
  long long a0[NP], b0[NP];
  bool tooLong = false;
#pragma unroll
  for (int h = 0; h < NP; ++h) {
    const int k = first + group * NP + h;
    pid[h] = (k < n) ? list[k] : -1;
    PairDesc d = (pid[h] >= 0) ? io.pairs[pid[h]] : PairDesc{0, 0, 0, 0};
    alen[h] = d.a_len;
    blen[h] = d.b_len;
    a0[h] = d.a_off;
    b0[h] = d.b_off;
    tooLong |= d.b_len > io.rowsCap;
  }
  if (__any_sync(FULL, tooLong)) {
    // The host sizes the scratch for the longest B; report, never trap.
    if (lane32 == 0) atomicCAS(&io.st->error, 0, ERR_SCRATCH);
    return;
  }
  Best fw[NP], rv[NP];
  bool ovf[NP];
  if constexpr (HYB) {
    static_assert(NP == 2 && LANES == 32, "the hybrid class pairs two pairs per 32-lane warp");
    // Mode chosen at run time: specialising the hybrid class made its
    // forward-only kernel spill and slowed the heavy-tailed protein batch.
    align_pairs_hybrid<K, 0>(sc, s_prof, s_simp, s_bring, io.codes, a0, b0, alen, blen, scr, io.rowsCap, fw, rv, ovf);
  } else {
    // 16-bit classes: one kernel per mode (fewer registers, no spills for
    // forward-only; the early reverse stop for full alignments); the s32
    // class keeps the run-time choice for the same reason as the hybrid.
    constexpr int MODE = (T::NP == 1) ? 0 : (FWD ? 1 : 2);
    align_pairs<T, K, LANES, MODE>(sc, s_prof, s_simp, s_bring, io.codes, a0, b0, alen, blen, scr, io.rowsCap, fw, rv,
                                   ovf);
  }
  if (glane == 0) {
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      if (pid[h] < 0) continue;
      if (ovf[h]) {
        const int slot = atomicAdd(&io.st->overflow_count, 1);
        io.overflow_list[slot] = pid[h];
        atomicAdd(io.rerun_cells, (unsigned long long)alen[h] * (unsigned long long)blen[h]);
        continue;
      }
      write_result(sc, fw[h], rv[h], io.score, io.arange, io.brange, pid[h]);
    }
  }
}

// Persistent kernel of one class.  `list` holds pair ids in processing
// order; warps take items from an atomic queue head.
// Register budget: the forward-only kernels get at most 128 registers (4
// blocks of 128 threads per SM when the profile is small); the kernels
// with a reverse pass or a run-time mode (FWD false, or the hybrid class)
// up to 170 (3 blocks per SM, which their shared memory allows anyway), as
// at 128 they spilled.  The affine classes of long pairs, proteins mostly,
// fit two blocks by their shared memory.
template <class T, bool HYB, bool FWD>
constexpr int kBatchedBlocks = (kTagged<T> && !T::LINEAR) ? 2 : (FWD && !HYB) ? 4 : 3;
template <class T, int K, int LANES, bool HYB = false, bool FWD = false>
__global__ void __launch_bounds__(128, kBatchedBlocks<T, HYB, FWD>)
    k_batched(SwConst sc, const int8_t* __restrict__ sim, BatchIo io, const int* __restrict__ list,
              const int* __restrict__ range, int* queue_head, int2* scratch, const ClassAllot* __restrict__ allot,
              unsigned long long* trace) {
  if ((int)blockIdx.x >= allot->blocks) return;  // outside this launch's share
  scratch += allot->base;
  // trace (option "trace"): {~first block start, last warp end} of the launch.
  if (trace && threadIdx.x == 0) atomicMax(&trace[0], ~global_ns());
  using L = SmemLayout<T, K, LANES>;
  constexpr int PER_ITEM = L::GROUPS * T::NP;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warps = blockDim.x >> 5;
  const int wib = threadIdx.x >> 5;
  const int lane32 = threadIdx.x & 31;
  int8_t* s_simp = reinterpret_cast<int8_t*>(smem);
  uint8_t* wsmem = smem + L::simp_bytes(sc.M, sc.P) + wib * L::warp_bytes(sc.P);
  load_table(s_simp, sim, sc, kProfBias<T> ? -sc.gE : 0, kProfShift<T>);
  __syncthreads();

  // range = {first list entry, number of entries}, written by the binning
  // pre-pass (or the overflow counter) on the device.
  const int n = range[1];
  list += range[0];
  const int items = (n + PER_ITEM - 1) / PER_ITEM;
  const long gw = (long)blockIdx.x * warps + wib;
  int2* wscr = scratch + gw * L::GROUPS * (HYB ? 3 : 2) * io.rowsCap;
  while (true) {
    int item = 0;
    if (lane32 == 0) item = atomicAdd(queue_head, 1);
    item = __shfl_sync(FULL, item, 0);
    if (item >= items) break;
    batched_item<T, K, LANES, HYB, FWD>(sc, io, s_simp, wsmem, wscr, list, item * PER_ITEM, n);
  }
  if (trace && lane32 == 0) atomicMax(&trace[1], global_ns());
}

// Strip-team kernel: teams of warps of a block align one item each (two
// pairs in 16-bit halves), taking its 32 * K wide strips round robin
// (tag_pass with TEAM), so a long pair finishes up to `team size` times
// sooner than on one warp.  Each warp keeps the best cell of its own
// strips; the team merges them with the first-strict-maximum order
// (better), the order-independent total order the one-warp pass applies
// strip by strip.  With start coordinates the team then runs the reverse
// pass the same way.  A team that gave up (a 16-bit overflow, or a wait
// past kTeamWaitNs, which also sets ERR_WAIT) sends both pairs to the s32
// rerun.  Block scratch: one boundary column of rowsCap rows per warp.
//
// A block's warps form one team, two or four (team_size): with fewer items
// than blocks only the largest team uses the SM's warps at all; with more,
// a smaller one wastes less on the strips' rounding (9 strips keep 8 warps
// busy 9 of 16 turns, two warps 9 of 10) and on the lag between warps.
constexpr int kTeamMaxWarps = 8;

// Steps a team warp starts behind the warp before it: it reads the boundary
// rows of a block of 32 when it starts the block, and that warp publishes
// them a block later.
constexpr float kTeamLagSteps = 64.f;

// Warps per team: the divisor of the block's warps (down to a quarter, two
// at least) that finishes `items` items like the list's first, its longest,
// soonest -- rounds of items times the steps of one item.  A smaller team
// has to win by a twentieth: with 150 items on 148 blocks teams of four tie
// with teams of eight, but keep every SM half idle for the whole time where
// eight leave all but two SMs to the next launches after half of it.
__device__ __forceinline__ int team_size(int warps, long blocks, int items, int strips, int rows) {
  int best = warps;
  float bestCost = 3.0e38f;
  for (int t = warps; t >= 2 && 4 * t >= warps; t /= 2) {
    const long slots = blocks * (warps / t);
    const float cost = (float)((items + slots - 1) / slots) *
                       ((float)((strips + t - 1) / t) * (float)(rows + 32) +
                        kTeamLagSteps * (float)(min(strips, t) - 1));
    if (cost < 0.95f * bestCost) {
      bestCost = cost;
      best = t;
    }
    if (t & 1) break;
  }
  return best;
}

template <class T, int K>
__global__ void __launch_bounds__(256, T::LINEAR ? 2 : 1)
    k_strips(SwConst sc, const int8_t* __restrict__ sim, BatchIo io, const int* __restrict__ list,
             const int* __restrict__ range, int* queue_head, int2* scratch, const ClassAllot* __restrict__ allot,
             unsigned long long* trace) {
  if ((int)blockIdx.x >= allot->blocks) return;
  scratch += allot->base;
  if (trace && threadIdx.x == 0) atomicMax(&trace[0], ~global_ns());
  using L = SmemLayout<T, K, 32>;
  constexpr int NP = 2;
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr int MAXT = kTeamMaxWarps / 2;  // teams of a block
  __shared__ int s_prog[kTeamMaxWarps];
  __shared__ int s_abort[MAXT], s_item[MAXT];
  __shared__ Best s_res[kTeamMaxWarps][NP];
  __shared__ Best s_bestT[MAXT][2][NP];  // merged best of the forward / reverse pass
  __shared__ bool s_ovfT[MAXT][NP];
  const int warps = blockDim.x >> 5;
  const int wib = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int8_t* s_simp = reinterpret_cast<int8_t*>(smem);
  uint8_t* s_prof = smem + L::simp_bytes(sc.M, sc.P) + wib * L::warp_bytes(sc.P);
  uint16_t* s_bring = reinterpret_cast<uint16_t*>(s_prof + L::prof_bytes(sc.P));
  load_table(s_simp, sim, sc, kProfBias<T> ? -sc.gE : 0, kProfShift<T>);

  __syncthreads();  // s_simp is loaded

  const int n = range[1];
  list += range[0];
  const int items = (n + NP - 1) / NP;
  if (n <= 0) return;
  const PairDesc longest = io.pairs[list[0]];
  const int tsize = team_size(warps, min((long)gridDim.x, (long)allot->blocks), items,
                              (longest.a_len + 32 * K - 1) / (32 * K), longest.b_len);
  const int q = wib / tsize, tw = wib % tsize;  // this warp's team, and its place there
  if (q >= warps / tsize) return;               // warps past the last whole team
  const int tid = tw * 32 + lane;
  // A barrier of the team's warps (barrier 0 is the block's).
  const auto team_sync = [&]() {
    asm volatile("bar.sync %0, %1;" ::"r"(q + 1), "r"(32 * tsize) : "memory");
  };
  Best(&s_best)[2][NP] = s_bestT[q];
  bool(&s_ovf)[NP] = s_ovfT[q];
  int2* scr = scratch + ((long)blockIdx.x * warps + q * tsize) * io.rowsCap;
  const StripTeam team{s_prog + q * tsize, &s_abort[q], &io.st->error, ERR_WAIT, tw, tsize};
  while (true) {
    team_sync();  // the previous item's merge is done
    if (tid == 0) {
      s_item[q] = atomicAdd(queue_head, 1);
      s_abort[q] = 0;
    }
    if (lane == 0) s_prog[wib] = -1;
    team_sync();
    const int item = s_item[q];
    if (item >= items) break;
    int pid[NP];
    PairDesc d[NP];
    bool tooLong = false;
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      const int k = item * NP + h;
      pid[h] = (k < n) ? list[k] : -1;
      d[h] = (pid[h] >= 0) ? io.pairs[pid[h]] : PairDesc{0, 0, 0, 0};
      tooLong |= d[h].b_len > io.rowsCap;
    }
    if (tooLong) {
      // The host sizes the scratch for the longest B; report, never trap.
      if (tid == 0) atomicCAS(&io.st->error, 0, ERR_SCRATCH);
      continue;
    }
    PassSeq ps[NP];
#pragma unroll
    for (int h = 0; h < NP; ++h) {
      const bool empty = d[h].a_len <= 0 || d[h].b_len <= 0;
      ps[h] = PassSeq{io.codes, d[h].a_off, d[h].b_off, empty ? 0 : d[h].a_len, empty ? 0 : d[h].b_len, 1, 1};
    }
    // Pass 0: forward.  Pass 1 (with start coordinates): the same pass over
    // the reversed reads from each pair's end cell (as align_pairs, without
    // the early stop), whose first strict maximum gives the start.  One
    // copy of tag_pass serves both.
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      Best out[NP];
      tag_pass<T, K, 32, false, true>(sc, s_prof, s_simp, s_bring, ps, scr, io.rowsCap, out, PassStop{}, team);
      if (lane == 0) {
#pragma unroll
        for (int h = 0; h < NP; ++h) s_res[wib][h] = out[h];
      }
      team_sync();
      if (tid < NP) {
        const int h = tid;
        Best b = s_res[q * tsize][h];
        for (int w = 1; w < tsize; ++w) {
          const Best c = s_res[q * tsize + w][h];
          if (better(c.s, c.i, c.j, b.s, b.i, b.j)) b = c;
        }
        s_best[pass][h] = b;
        // A team that gave up (in either pass) sends the pair to the rerun.
        if (pass == 0) {
          s_ovf[h] = s_abort[q] != 0 || b.s > Cell<T>::limit(sc);
          s_best[1][h] = Best{0, 0, 0};  // the start of a pair without a reverse pass
        }
        if (pass == 1 && s_abort[q] != 0) s_ovf[h] = true;
      }
      team_sync();
      if (pass == 1 || sc.forwardOnly) break;
      bool any = false;
#pragma unroll
      for (int h = 0; h < NP; ++h) {
        const Best fw = s_best[0][h];
        const bool run = pid[h] >= 0 && !s_ovf[h] && fw.s > 0;
        any |= run;
        ps[h] = run ? PassSeq{io.codes, d[h].a_off + fw.j, d[h].b_off + fw.i, fw.j + 1, fw.i + 1, -1, -1}
                    : PassSeq{io.codes, d[h].a_off, d[h].b_off, 0, 0, 1, 1};
      }
      if (!any) break;  // block-uniform: every thread read the same words
      // A fresh team for the reverse pass (after every warp read s_ovf).
      team_sync();
      if (tid == 0) s_abort[q] = 0;
      if (lane == 0) s_prog[wib] = -1;
      team_sync();
    }
    if (tid < NP) {
      const int h = tid;
      if (pid[h] >= 0) {
        if (s_ovf[h]) {
          const int slot = atomicAdd(&io.st->overflow_count, 1);
          io.overflow_list[slot] = pid[h];
          atomicAdd(io.rerun_cells, (unsigned long long)d[h].a_len * (unsigned long long)d[h].b_len);
        } else {
          write_result(sc, s_best[0][h], s_best[1][h], io.score, io.arange, io.brange, pid[h]);
        }
      }
    }
  }
  if (trace && lane == 0) atomicMax(&trace[1], global_ns());
}

// One-launch-per-batch kernel over the reference wire buffer.
// Comparison slot g = tile * maxBatches + slot reads Meta[4g..4g+3] =
// {a_len, a_off, b_len, b_off}, byte offsets into the tile's Seqs region
// (ipu_batch_affine.cpp:164-167, 881-884), and writes Scores[g],
// ARanges[g], BRanges[g] of the output buffer (ipu_batch_affine.cpp:208-210,
// 288).  Warps take slots g = warp, warp + nwarps, ... in slot order.
template <int K>
__global__ void __launch_bounds__(128) k_plain(SwConst sc, const int8_t* __restrict__ sim,
                                               const int* __restrict__ inputs, long seqWordsPerTile,
                                               long metaOffset, int maxBatches, int totalSlots,
                                               int2* scratch, long rowsCap, int* results,
                                               DevStatus* st) {
  using T = LaneS32;
  using L = SmemLayout<T, K, 32>;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warps = blockDim.x >> 5;
  const int wib = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int8_t* s_simp = reinterpret_cast<int8_t*>(smem);
  uint8_t* wbase = smem + L::simp_bytes(sc.M, sc.P) + wib * L::warp_bytes(sc.P);
  uint8_t* s_prof = wbase;
  uint16_t* s_bring = reinterpret_cast<uint16_t*>(wbase + L::prof_bytes(sc.P));
  load_table(s_simp, sim, sc);
  __syncthreads();
  const long gw = (long)blockIdx.x * warps + wib;
  const long nw = (long)gridDim.x * warps;
  int2* scr = scratch + gw * 2 * rowsCap;
  const int* meta = inputs + metaOffset;
  // Byte codes: residue offsets count bytes from the start of the buffer.
  const uint8_t* bytes = reinterpret_cast<const uint8_t*>(inputs);
  for (long g = gw; g < totalSlots; g += nw) {
    const long long tileBase = (long long)(g / maxBatches) * seqWordsPerTile * 4;
    const int alen = meta[4 * g + 0], aoff = meta[4 * g + 1];
    const int blen = meta[4 * g + 2], boff = meta[4 * g + 3];
    if (blen > rowsCap) {
      if (lane == 0) atomicCAS(&st->error, 0, ERR_SCRATCH);
      continue;
    }
    const long long a0[1] = {tileBase + aoff};
    const long long b0[1] = {tileBase + boff};
    const int al[1] = {alen}, bl[1] = {blen};
    Best fw[1], rv[1];
    bool ovf[1];
    align_pairs<T, K, 32>(sc, s_prof, s_simp, s_bring, bytes, a0, b0, al, bl, scr, rowsCap, fw, rv, ovf);
    if (lane == 0)
      write_result(sc, fw[0], rv[0], results, results + totalSlots, results + 2L * totalSlots, g);
  }
}

// The one-launch-per-batch kernel with s16x2 lanes: the same wire buffer,
// slot order and static stride as k_plain, but one warp aligns two
// consecutive comparison slots (2g, 2g + 1) in the halves of s16x2 lanes,
// whatever their lengths.  A slot whose score could have left int16 is
// redone by the same warp in s32 lanes, so the batch still takes one
// launch.  It isolates what the batched engine gains by sorting, binning
// and packing pairs from what it gains by the lane width.
template <int K>
__global__ void __launch_bounds__(128) k_plain16(SwConst sc, const int8_t* __restrict__ sim,
                                                 const int* __restrict__ inputs, long seqWordsPerTile,
                                                 long metaOffset, int maxBatches, int totalSlots,
                                                 int2* scratch, long rowsCap, int* results,
                                                 DevStatus* st) {
  using L = SmemLayout<Lane16, K, 32>;
  extern __shared__ __align__(16) uint8_t smem[];
  const int warps = blockDim.x >> 5;
  const int wib = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int8_t* s_simp = reinterpret_cast<int8_t*>(smem);
  uint8_t* wbase = smem + L::simp_bytes(sc.M, sc.P) + wib * L::warp_bytes(sc.P);
  uint8_t* s_prof = wbase;  // the s32 redo uses the first half of it
  uint16_t* s_bring = reinterpret_cast<uint16_t*>(wbase + L::prof_bytes(sc.P));
  load_table(s_simp, sim, sc);
  __syncthreads();
  const long gw = (long)blockIdx.x * warps + wib;
  const long nw = (long)gridDim.x * warps;
  int2* scr = scratch + gw * 2 * rowsCap;
  const int* meta = inputs + metaOffset;
  const uint8_t* bytes = reinterpret_cast<const uint8_t*>(inputs);
  for (long g0 = 2 * gw; g0 < totalSlots; g0 += 2 * nw) {
    long long a0[2], b0[2];
    int al[2], bl[2];
    bool tooLong = false;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long g = g0 + h;
      const bool have = g < totalSlots;
      const long long tileBase = have ? (long long)(g / maxBatches) * seqWordsPerTile * 4 : 0;
      al[h] = have ? meta[4 * g + 0] : 0;
      bl[h] = have ? meta[4 * g + 2] : 0;
      a0[h] = tileBase + (have ? meta[4 * g + 1] : 0);
      b0[h] = tileBase + (have ? meta[4 * g + 3] : 0);
      tooLong |= bl[h] > rowsCap;
    }
    if (tooLong) {  // warp-uniform: every lane read the same Meta words
      if (lane == 0) atomicCAS(&st->error, 0, ERR_SCRATCH);
      continue;
    }
    Best fw[2], rv[2];
    bool ovf[2];
    align_pairs<Lane16, K, 32>(sc, s_prof, s_simp, s_bring, bytes, a0, b0, al, bl, scr, rowsCap, fw, rv, ovf);
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      if (g0 + h >= totalSlots) break;
      if (ovf[h]) {  // uniform: the score is the 32-lane group's reduction
        const long long a1[1] = {a0[h]};
        const long long b1[1] = {b0[h]};
        const int al1[1] = {al[h]}, bl1[1] = {bl[h]};
        Best f1[1], r1[1];
        bool o1[1];
        align_pairs<LaneS32, K, 32>(sc, s_prof, s_simp, s_bring, bytes, a1, b1, al1, bl1, scr, rowsCap, f1, r1,
                                    o1);
        fw[h] = f1[0];
        rv[h] = r1[0];
      }
      if (lane == 0)
        write_result(sc, fw[h], rv[h], results, results + totalSlots, results + 2L * totalSlots, g0 + h);
    }
  }
}

// Exact per-thread kernel: one thread per pair, the recurrence written out
// cell by cell in int32 (codelet_batch_affine.cpp:65-115) with C and F rows
// in global scratch (2 * maxA int per thread).  Covers every scoring
// configuration.  A[j] = residue a0 + j * da, B[i] = residue b0 + i * db of
// `codes` (sc.bits per residue).
static __device__ void exact_pass(const uint8_t* codes, int bits, long long a0, int alen, int da, long long b0,
                                  int blen, int db, const int8_t* sim, int M, int gI, int gE, int* C, int* F,
                                  Best& out) {
  int s = 0, bi = 0, bj = 0;
  for (int j = 0; j < alen; ++j) {
    C[j] = 0;
    F[j] = 0;
  }
  for (int i = 0; i < blen; ++i) {
    const int bc = code_at(codes, b0 + (long long)i * db, bits);
    int e = gI, hl = 0, diag = 0;
    for (int j = 0; j < alen; ++j) {
      const int ac = code_at(codes, a0 + (long long)j * da, bits);
      e = max(hl + gI + gE, e + gE);
      const int f = max(C[j] + gI + gE, F[j] + gE);
      F[j] = f;
      int h = max(diag + (int)sim[ac * M + bc], e);
      h = max(max(h, f), 0);
      diag = C[j];
      C[j] = h;
      hl = h;
      if (h > s) {
        s = h;
        bi = i;
        bj = j;
      }
    }
  }
  out = Best{s, bi, bj};
}

// Pairs are checked with pair_state against n_codes and the stated maxima
// (maxA, maxB) before any code is read.
static __global__ void k_exact(SwConst sc, const int8_t* __restrict__ sim, const uint8_t* __restrict__ codes,
                        long long n_codes, const PairDesc* __restrict__ pairs, int n, int* cf_scratch, long maxA,
                        int maxB, int* score, int* arange, int* brange, DevStatus* st) {
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long nt = (long)gridDim.x * blockDim.x;
  int* C = cf_scratch + tid * 2 * maxA;
  int* F = C + maxA;
  for (long p = tid; p < n; p += nt) {
    const PairDesc d = pairs[p];
    const int state = pair_state(d, n_codes, (int)maxA, maxB);
    report_pair(state, st);
    const int alen = state == PAIR_OK ? d.a_len : 0;
    const int blen = state == PAIR_OK ? d.b_len : 0;
    const long long a = state == PAIR_OK ? d.a_off : 0;
    const long long b = state == PAIR_OK ? d.b_off : 0;
    Best fw{0, 0, 0}, rv{0, 0, 0};
    if (alen > 0 && blen > 0 && alen <= maxA) {
      exact_pass(codes, sc.bits, a, alen, 1, b, blen, 1, sim, sc.M, sc.gI, sc.gE, C, F, fw);
      if (!sc.forwardOnly)
        exact_pass(codes, sc.bits, a + fw.j, fw.j + 1, -1, b + fw.i, fw.i + 1, -1, sim, sc.M, sc.gI, sc.gE, C, F,
                   rv);
    }
    write_result(sc, fw, rv, score, arange, brange, p);
  }
}

// -------------------------------------------------------------------------
// Cost-binned work list.  Every pair gets a key = class * NBUCKET + bucket,
// where the class picks the kernel (lane type, lanes per pair, columns per
// lane: |A| decides it) and the bucket orders by descending |B| on a
// log-linear scale; a counting sort over the keys yields the processing
// order: longest first inside each class (the long tail starts early) and
// neighbours of near-equal rows, which share a warp.  Empty pairs get their
// zero result here and are not listed.
// -------------------------------------------------------------------------
constexpr int NROWB = 256;    // row buckets (16 per power of two)
constexpr int NSTRIPB = 16;   // strip-count buckets
constexpr int NBUCKET = NROWB * NSTRIPB;
constexpr int NCLASS_MAX = 29;

// Log-linear bucket of |B| (16 sub-buckets per power of two): pairs that
// share a bucket differ by at most 1/16 in rows, so the groups of a warp
// finish their wavefronts together.
__device__ __forceinline__ int rows_bucket(int b) {
  if (b < 16) return b;
  const int lg = 31 - __clz(b);
  return min(NROWB - 1, (lg - 3) * 16 + ((b >> (lg - 4)) & 15));
}

struct BinParams {
  int nclass;
  int cls_s32;             // class index of the exact-32-bit kernel
  int cls_hi;              // class of pairs whose diagonal bound passes big_limit:
                           // the hybrid class (or cls_s32 when it is off)
  int cls_big;             // class of the other pairs past s16_limit (cls_s32 when
                           // the hybrid class is off), and its strip-team class (-1: none)
  int team_big;
  int big_limit;           // scores above this need more than 16 biased bits
  int s16_max_len;         // min(|A|,|B|) above which the 16-bit lanes could overflow
  int s16_limit;           // scores above this need more than the long class's 16 bits
  // Scores the lanes of the classes by cost hold (a pair past them is rerun in
  // s32 lanes), and the longest min(|A|,|B|) that cannot pass them.  A longer
  // pair goes to cls_over: where by_letters is 0 by its length alone, else if
  // its letters' top scores say so (letters_pass).
  int fit_score, fit_len, by_letters, cls_over;
  int8_t top[32];
  int lanes[NCLASS_MAX];   // lanes per group of each class
  int width[NCLASS_MAX];   // strip width (lanes * K) of each class
  unsigned inv_width[NCLASS_MAX];  // ceil(2^32 / width): strips_of
  float slot_ps[NCLASS_MAX];   // time per cell slot of a strip (autotuned)
  float strip_ps[NCLASS_MAX];  // fixed time per strip (autotuned)
  // One warp item of class c advances one step (row) every step_ps[c], so a
  // pair of `strips` strips takes strips * (|B| + lanes) * step_ps[c]; it
  // counts lat_weight times that beside the batch's modelled time (pair_key).
  float step_ps[NCLASS_MAX];
  float batch_ps_per_cell;     // modelled batch time per cell (strip teams)
  float lat_weight;
  float team_slack;            // kTeamSlackPs, or 0 for a batch that leaves warps idle
  int long_a;                  // |A| above which the widest strips are used
  int widest;                  // class of the widest strips
  int forced_class;        // >= 0: every s16x2 pair goes to this class
  int team_cls;            // strip-team class (-1: none in this batch)
  int team_warps;          // warps per team
  unsigned by_cost;        // classes a pair is given to by its modelled time
  int max_a, max_b;        // stated maxima (violations set ERR_LENGTH)
  long long n_codes;       // residues in the code array (pairs past it set ERR_RANGE)
  int bits;                // bits per residue of the code array (code_at)
  int M;                   // alphabet size of `sim`
  int force_s32;           // 1: every pair goes to the s32 class
  // Per-thread class (k_thread): one thread per two pairs, so a pair's time
  // is long.  A pair may use it only when |B| <= thr_max_rows and its cells
  // stay below thr_cap_scale * (cells of the whole batch): that bounds its
  // latency to a fraction of the batch's time (thr_cap_scale = fraction /
  // pair slots the class keeps resident).
  // Full-occupancy grid and strip scratch (int2) per block of each class,
  // where its launch's scratch starts (a region per stream), and the scratch
  // available.
  long long base[NCLASS_MAX + 1];
  int grid[NCLASS_MAX + 1];
  long long scr_per_block[NCLASS_MAX + 1];
  long long scr_cap;
  int thr_cls;             // class index
  int thr_on;              // 0: the class is never chosen (unless forced)
  int thr_max_rows, thr_fit;   // rows it accepts, and the longest min(|A|,|B|)
  float thr_cap_scale;
  const unsigned long long* total_cells;  // written by k_bin_total
};

// Buckets of the per-thread class: exact strip counts up to 24 (then one
// bucket), rows log-linear with 16 sub-buckets per octave (< 144 for rows
// up to 2048); both descending.
constexpr int THR_NSB = 25;
constexpr int THR_NRB = 144;
static_assert(THR_NSB * THR_NRB <= NBUCKET, "per-thread buckets");

// Best ungapped score along the main diagonal (a lower bound of the local
// alignment score): pairs that surely pass the s16 limit go to the hybrid
// (or s32) class instead of giving up half way in s16x2.  One warp per
// pair: lane l takes the l-th of 32 consecutive segments of the diagonal
// and summarises it as {sum, best prefix, best suffix, best run} (all >= 0
// but the sum); an ordered tree of shuffles joins the summaries, the best
// run of the whole diagonal ending in lane 0 (the maximum-subarray score
// that max(run + s, 0) computes sequentially).
struct DiagRun {
  int sum, pre, suf, best;
};

__device__ __forceinline__ DiagRun join_runs(const DiagRun& l, const DiagRun& r) {
  return DiagRun{l.sum + r.sum, max(l.pre, l.sum + r.pre), max(r.suf, r.sum + l.suf),
                 max(max(l.best, r.best), l.suf + r.pre)};
}

static __device__ int warp_diagonal_bound(const uint8_t* codes, int bits, long long a, long long b, int n,
                                          const int8_t* sim, int M) {
  const int lane = threadIdx.x & 31;
  const int seg = (n + 31) / 32;
  const int k0 = min(n, lane * seg), k1 = min(n, k0 + seg);
  DiagRun r{0, 0, 0, 0};
  int run = 0;
  auto take = [&](int s) {
    r.sum += s;
    r.pre = max(r.pre, r.sum);
    run = max(run + s, 0);
    r.best = max(r.best, run);
  };
  // A code outside the alphabet (no row of the matrix) counts 0 here.
  auto score = [&](int x, int y) { return (x < M && y < M) ? (int)sim[x * M + y] : 0; };
  if (k0 < k1) {
    if (bits == 8) {
      for (int k = k0; k < k1; ++k) take(score(codes[a + k], codes[b + k]));
    } else {
      PackedStream sa(codes, a + k0, bits), sb(codes, b + k0, bits);
      for (int k = k0; k < k1; ++k) {
        const int x = sa.next(), y = sb.next();
        take(score(x, y));
      }
    }
  }
  r.suf = run;  // best sum of a suffix (empty allowed)
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    DiagRun o;
    o.sum = __shfl_down_sync(FULL, r.sum, off);
    o.pre = __shfl_down_sync(FULL, r.pre, off);
    o.suf = __shfl_down_sync(FULL, r.suf, off);
    o.best = __shfl_down_sync(FULL, r.best, off);
    if ((lane & (2 * off - 1)) == 0 && lane + off < 32) r = join_runs(r, o);
  }
  return __shfl_sync(FULL, r.best, 0);
}

// A pair goes to a strip team when its one-warp latency passes the batch's
// modelled time plus this many ps (BinParams::team_slack): below it the
// other pairs' work hides the pair, and a team's fill and idle warps only
// cost throughput -- its block also keeps k_mix off the SM.  The slack is
// what a batch that fills the GPU takes beside its cells; a batch of fewer
// pairs than the widest strips' warps hold has none, since no other work
// fills the rest.  (B200: 1,000 pairs of 1,600-2,000, too few to fill the
// GPU, ran 1.35 ms with every pair in a team, 2.5 without; 4,006 proteins
// 0.97 ms with pairs from 700 residues in teams, 0.67 from 900; 60,000
// heavy-tailed proteins 28 ms with the line at 1.8 times their time.)
constexpr float kTeamSlackPs = 2.5e8f;

// Class of a pair: the kernel with the lowest modelled time
//   strips * ((|B| + lanes) * width * slot_ps + strip_ps)
// where strips * width covers |A|, |B| + lanes counts the fill and drain of
// each strip's wavefront, and slot_ps / strip_ps are the per-class rates
// the autotuner measured.  Key = class, then strip count (descending), then
// rows (descending).
// Strips of class c that cover alen columns: (alen + width - 1) / width by
// multiplication (exact: the numerator times width stays below 2^32).
__device__ __forceinline__ int strips_of(const BinParams& bp, int c, int alen) {
  return (int)__umulhi((unsigned)(alen + bp.width[c] - 1), bp.inv_width[c]);
}

// A strip team's class `tc` for a pair whose one-warp latency is `lat`, or
// cls: taken when even the fastest warp would take a large share of the
// whole batch's modelled time (kTeamSlackPs: below it the other pairs'
// work hides the pair, and a team's fill and idle warps only cost
// throughput) and the team finishes the pair sooner.  Its warps take the
// strips round robin, each starting about kTeamLagSteps behind the warp
// before it.
__device__ __forceinline__ int team_class(const BinParams& bp, int cls, int tc, int alen, int blen, float lat,
                                          float batch_ps) {
  if (tc < 0 || lat <= batch_ps + bp.team_slack) return cls;
  const int strips = strips_of(bp, tc, alen);
  if (strips < 2) return cls;
  const int rounds = (strips + bp.team_warps - 1) / bp.team_warps;
  const float tl = ((float)rounds * (float)(blen + bp.lanes[tc]) +
                    kTeamLagSteps * (float)(min(strips, bp.team_warps) - 1)) *
                   bp.step_ps[tc];
  return tl < lat ? tc : cls;
}

// `flag`: 0, 1 (the diagonal bound passes s16_limit), 2 (big_limit) or 3
// (letters_pass).
__device__ __forceinline__ int pair_key(const BinParams& bp, int alen, int blen, int flag, float thr_cap) {
  int cls;
  if (bp.force_s32) {
    cls = bp.cls_s32;
  } else if (flag == 2) {
    cls = bp.cls_hi;
  } else if (flag == 1) {
    cls = bp.cls_big;
    const float batch_ps = bp.total_cells ? (float)(*bp.total_cells) * bp.batch_ps_per_cell : 0.f;
    const float lat = (float)strips_of(bp, cls, alen) * (float)(blen + bp.lanes[cls]) *
                      bp.step_ps[cls];
    cls = team_class(bp, cls, bp.team_big, alen, blen, lat, batch_ps);
  } else if (bp.forced_class >= 0) {
    cls = bp.forced_class;
  } else {
    const float batch_ps = bp.total_cells ? (float)(*bp.total_cells) * bp.batch_ps_per_cell : 0.f;
    float bestLat = -1.f;  // one-warp latency of the class picked below
    const int shorter = min(alen, blen);
    const bool over = shorter > bp.fit_len && (flag == 3 || !bp.by_letters);
    const int wide = over ? bp.cls_over : bp.widest;
    if (alen > bp.long_a) {
      // Very long pairs are few and each keeps one warp busy for long: their
      // latency, not throughput, sets the end of the launch, and the widest
      // strips finish a pair in the fewest steps.
      cls = wide;
      bestLat = (float)strips_of(bp, cls, alen) * (float)(blen + bp.lanes[cls]) *
                bp.step_ps[cls];
    } else {
      cls = wide;
      float bestCost = -1.f;
      const bool thr_ok = bp.thr_on && blen <= bp.thr_max_rows && shorter <= bp.thr_fit &&
                          (float)alen * (float)blen <= thr_cap;
      // The time of a batch made of this pair alone, as many as hold the
      // batch's cells: its share of the GPU's rate, and once a part of its
      // own latency (the last ones finish alone).
      const float like = bp.total_cells ? (float)(*bp.total_cells) / ((float)alen * (float)blen) : 1.f;
      for (unsigned left = bp.by_cost; left; left &= left - 1) {
        const int c = __ffs(left) - 1;
        if (c == bp.thr_cls ? !thr_ok : over) continue;
        const int strips = strips_of(bp, c, alen);
        const float lat = (float)strips * (float)(blen + bp.lanes[c]) * bp.step_ps[c];
        const float cost =
            (float)strips * ((float)(blen + bp.lanes[c]) * (float)bp.width[c] * bp.slot_ps[c] + bp.strip_ps[c]) *
                like + (c == bp.thr_cls ? 0.f : bp.lat_weight * lat);
        if (bestCost < 0.f || cost < bestCost) {
          bestCost = cost;
          bestLat = lat;
          cls = c;
        }
      }
      if (bestCost < 0.f)  // none of them holds its scores
        bestLat = (float)strips_of(bp, cls, alen) * (float)(blen + bp.lanes[cls]) * bp.step_ps[cls];
    }
    cls = team_class(bp, cls, bp.team_cls, alen, blen, bestLat, batch_ps);
  }
  const int strips = strips_of(bp, cls, alen);
  if (cls == bp.thr_cls) {
    const int sb = THR_NSB - 1 - min(strips - 1, THR_NSB - 1);
    return cls * NBUCKET + sb * THR_NRB + (THR_NRB - 1 - min(rows_bucket(blen), THR_NRB - 1));
  }
  const int sb = NSTRIPB - 1 - min(strips - 1, NSTRIPB - 1);
  return cls * NBUCKET + sb * NROWB + (NROWB - 1 - rows_bucket(blen));
}

// Latency cap of the per-thread class for this batch (cells per pair).
__device__ __forceinline__ float thread_cap(const BinParams& bp) {
  return (bp.thr_on && bp.total_cells) ? (float)(*bp.total_cells) * bp.thr_cap_scale : 0.f;
}

// Sum of |A| * |B| over the pairs the pipeline will align (the batch size
// the per-thread class's latency cap is measured against).
static __global__ void k_bin_total(BinParams bp, const PairDesc* __restrict__ pairs, int n,
                                   unsigned long long* total, int* hist, int nkeys) {
  // The key histogram of the launches after this one starts at zero.
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nkeys; k += gridDim.x * blockDim.x) hist[k] = 0;
  unsigned long long local = 0;
  for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x) {
    const PairDesc d = pairs[p];
    if (pair_state(d, bp.n_codes, bp.max_a, bp.max_b) != PAIR_OK) continue;
    local += (unsigned long long)d.a_len * (unsigned long long)d.b_len;
  }
  for (int off = 16; off > 0; off >>= 1) local += __shfl_xor_sync(FULL, local, off);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(total, local);
}

// A pair whose diagonal bound decides its class: both sequences longer than
// the longest pair that cannot pass the s16 limit.
__device__ __forceinline__ bool bound_candidate(const BinParams& bp, const PairDesc& d) {
  return !bp.force_s32 && min(d.a_len, d.b_len) > bp.s16_max_len &&
         pair_state(d, bp.n_codes, bp.max_a, bp.max_b) == PAIR_OK;
}

// s32_flag of every candidate pair (k_bin_count reads it): warps take 32
// pairs at a time and compute the diagonal bound of each candidate among
// them together (warp_diagonal_bound).  blockDim.x is a multiple of 32.
static __global__ void k_bin_bound(BinParams bp, const uint8_t* __restrict__ codes,
                                   const int8_t* __restrict__ sim, const PairDesc* __restrict__ pairs, int n,
                                   uint8_t* s32_flag) {
  __shared__ int8_t s_sim[32 * 32];
  const bool smemSim = bp.M <= 32;
  if (smemSim)
    for (int k = threadIdx.x; k < bp.M * bp.M; k += blockDim.x) s_sim[k] = sim[k];
  __syncthreads();
  const int8_t* simT = smemSim ? s_sim : sim;
  const int lane = threadIdx.x & 31;
  const long warps = (long)gridDim.x * (blockDim.x / 32);
  for (long base = ((long)blockIdx.x * blockDim.x + threadIdx.x) / 32 * 32; base < n; base += warps * 32) {
    const long p = base + lane;
    const bool cand = p < n && bound_candidate(bp, pairs[p]);
    unsigned m = __ballot_sync(FULL, cand);
    while (m) {
      const long q = base + __ffs(m) - 1;
      m &= m - 1;
      const PairDesc d = pairs[q];
      const int bound =
          warp_diagonal_bound(codes, bp.bits, d.a_off, d.b_off, min(d.a_len, d.b_len), simT, bp.M);
      if (lane == 0) s32_flag[q] = bound > bp.big_limit ? 2 : bound > bp.s16_limit ? 1 : 0;
    }
  }
}

// May this lane's pair, longer than fit_len (`cand`), pass fit_score?  An
// alignment scores no more than the top scores of its shorter sequence's
// letters add up to.  32 of them, at equal distances, give the sum to about a
// sixteenth; from three of those below the limit to a fourth above it 128 do,
// to a thirtieth, against a line a sixteenth below the limit.  The lanes of a
// warp read one candidate's letters, the first samples of up to four at a
// time.  s_top: bp.top in shared memory.
// (B200, 10,000 near-identical proteins of 700-1,300 residues, 80 % of them C,
// H or W: with the mean letter for all 6,328 were rerun in s32, 7.1 ms; now
// 3.7.  Adding up all letters took 9 us of a request of 500; 32 alone, with
// a line an eighth below, sent pairs of 1,200 average residues to the long
// class, 8 % slower with start coordinates.)
__device__ __forceinline__ bool letters_pass(const BinParams& bp, const int8_t* s_top, const uint8_t* codes,
                                             const PairDesc& d, bool cand) {
  const int lane = threadIdx.x & 31;
  const int own_len = min(d.a_len, d.b_len);
  const long long own_off = d.a_len <= d.b_len ? d.a_off : d.b_off;
  const auto top = [&](int x) { return x < 32 ? (int)s_top[x] : 0; };  // past the alphabet: scores nothing
  bool pass = false;
  unsigned m = __ballot_sync(FULL, cand);
  while (m) {
    int src[4], len[4], x[4];
    long long off[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      src[u] = m ? __ffs(m) - 1 : -1;
      m &= m - 1;
      len[u] = __shfl_sync(FULL, own_len, max(src[u], 0));
      off[u] = __shfl_sync(FULL, own_off, max(src[u], 0));
      x[u] = src[u] >= 0 ? code_at(codes, off[u] + lane * len[u] / 32, bp.bits) : 32;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (src[u] < 0) break;
      const long long sampled = (long long)__reduce_add_sync(FULL, top(x[u])) * len[u];  // 32 times the sum
      bool over = sampled > 40ll * bp.fit_score;
      if (!over && sampled > 26ll * bp.fit_score) {
        int y[4], sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) y[q] = code_at(codes, off[u] + (4 * lane + q) * len[u] / 128, bp.bits);
#pragma unroll
        for (int q = 0; q < 4; ++q) sum += top(y[q]);
        over = (long long)__reduce_add_sync(FULL, sum) * len[u] > 120ll * bp.fit_score;
      }
      if (lane == src[u]) pass = over;
    }
  }
  return pass;
}

// Flag of a pair (pair_key); s32_flag as k_bin_bound left it.  All lanes of
// the warp call it.
__device__ __forceinline__ int pair_flag(const BinParams& bp, const int8_t* s_top, const uint8_t* codes, const PairDesc& d,
                                         bool listed, long p, const uint8_t* s32_flag) {
  const int flag = listed && bound_candidate(bp, d) ? s32_flag[p] : 0;
  if (!bp.by_letters) return flag;
  const bool cand = listed && flag == 0 && min(d.a_len, d.b_len) > bp.fit_len;
  return letters_pass(bp, s_top, codes, d, cand) ? 3 : flag;
}

// Sums of the pairs of one class.
struct ClassSums {
  unsigned long long cells;
  int count, pad;
};

// Key of one listed pair; its cells go to the block's class sums
// with one atomic per class among the warp's lanes (shared 64-bit atomics of
// 256 threads on a handful of classes took 17 of the kernel's 22 us for
// 20,000 pairs).  Called by the lanes of `act`.
__device__ __forceinline__ int tally_pair(const BinParams& bp, const PairDesc& d, int flag, ClassSums* s_sum,
                                          unsigned act) {
  const int key = pair_key(bp, d.a_len, d.b_len, flag, thread_cap(bp));
  const unsigned same = __match_any_sync(act, key / NBUCKET);
  const unsigned cells = (unsigned)d.a_len * (unsigned)d.b_len;  // < 2^32: lengths below 65536
  // Sums in 16-bit halves, which 32 lanes cannot carry out of 32 bits.
  const unsigned c0 = __reduce_add_sync(same, cells & 0xffffu), c1 = __reduce_add_sync(same, cells >> 16);
  if ((int)(threadIdx.x & 31) == __ffs(same) - 1) {
    ClassSums& s = s_sum[key / NBUCKET];
    atomicAdd(&s.cells, ((unsigned long long)c1 << 16) + c0);
    atomicAdd(&s.count, __popc(same));
  }
  return key;
}

// Zero result of a pair that is not listed (empty, too long or outside the
// code array).
__device__ __forceinline__ void reject_pair(int state, long p, DevStatus* st, int* score, int* arange, int* brange) {
  report_pair(state, st);
  score[p] = 0;
  arange[p] = 0;
  brange[p] = 0;
}

static __global__ void k_bin_count(BinParams bp, const uint8_t* __restrict__ codes,
                                   const PairDesc* __restrict__ pairs, int n, int* hist, const uint8_t* s32_flag,
                                   int* keys, ClassSums* sums, DevStatus* st, int* score, int* arange, int* brange) {
  __shared__ ClassSums s_sum[NCLASS_MAX];
  __shared__ int8_t s_top[32];
  for (int k = threadIdx.x; k < NCLASS_MAX; k += blockDim.x) s_sum[k] = ClassSums{0, 0, 0};
  if (threadIdx.x < 32) s_top[threadIdx.x] = bp.top[threadIdx.x];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (long base = (long)blockIdx.x * blockDim.x + threadIdx.x - lane; base < n; base += (long)gridDim.x * blockDim.x) {
    const long p = base + lane;
    const PairDesc d = p < n ? pairs[p] : PairDesc{0, 0, 0, 0};
    const int state = pair_state(d, bp.n_codes, bp.max_a, bp.max_b);
    const int flag = pair_flag(bp, s_top, codes, d, p < n && state == PAIR_OK, p, s32_flag);
    if (p >= n) continue;
    if (state != PAIR_OK) {
      reject_pair(state, p, st, score, arange, brange);
      keys[p] = -1;
      continue;
    }
    const unsigned act = __activemask();
    const int key = tally_pair(bp, d, flag, s_sum, act);
    keys[p] = key;
    // One histogram update per distinct key among the warp's lanes.
    const unsigned same = __match_any_sync(act, key);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&hist[key], __popc(same));
  }
  __syncthreads();
  for (int k = threadIdx.x; k < bp.nclass; k += blockDim.x) {
    if (!s_sum[k].count) continue;
    atomicAdd(&sums[k].cells, s_sum[k].cells);
    atomicAdd(&sums[k].count, s_sum[k].count);
  }
}

// One warp: the {start, count} list range of every class, and where its
// launch may run -- on the whole GPU, in the scratch region of its stream.
__device__ __forceinline__ void allot_classes(const BinParams& bp, const ClassSums* sums, int* class_range,
                                              ClassAllot* allot, DevStatus* st) {
  static_assert(NCLASS_MAX <= 32, "a lane per class");
  const int c = threadIdx.x & 31;
  const bool real = c < bp.nclass;
  const int count = real ? sums[c].count : 0;
  int start = count;  // inclusive prefix, then exclusive
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int y = __shfl_up_sync(FULL, start, off);
    if (c >= off) start += y;
  }
  start -= count;
  if (real) {
    int blocks = count > 0 ? bp.grid[c] : 0;
    const long long base = bp.base[c];
    if (base + (long long)blocks * bp.scr_per_block[c] > bp.scr_cap) {
      // Never reached when the host sized the scratch for these regions.
      blocks = (int)max(0ll, (bp.scr_cap - base) / max(bp.scr_per_block[c], 1ll));
      if (blocks == 0) atomicCAS(&st->error, 0, ERR_SCRATCH);
    }
    class_range[2 * c] = start;
    class_range[2 * c + 1] = count;
    allot[c].blocks = blocks;
    allot[c].base = base;
  }
  if (c == 0) {
    // The s32 rerun runs alone after every class: the whole GPU, base 0.
    allot[bp.nclass].blocks = bp.grid[bp.cls_s32];
    allot[bp.nclass].base = 0;
  }
}

// Block c (1024 threads): exclusive scan of class c's part of the histogram
// into `offs`, from the class's list start; block 0 also writes the ranges
// and shares of all classes.  A block per class: one block over all keys,
// tile after tile, took 53 us.
static __global__ void k_bin_scan(BinParams bp, const int* hist, int* offs, const ClassSums* sums, int* class_range,
                                  ClassAllot* allot, DevStatus* st) {
  constexpr int PER = NBUCKET / 1024;
  static_assert(PER == 4, "a 16-byte load per thread");
  __shared__ int s_warp[32];
  const int c = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  if (c == 0 && wid == 0) allot_classes(bp, sums, class_range, allot, st);
  if (sums[c].count == 0) return;
  int start = lane < c ? sums[lane].count : 0;  // pairs of the classes before
  start = __reduce_add_sync(FULL, start);
  const int4 v = reinterpret_cast<const int4*>(hist + c * NBUCKET)[tid];
  const int own = v.x + v.y + v.z + v.w;
  int x = own;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int y = __shfl_up_sync(FULL, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) s_warp[wid] = x;
  __syncthreads();
  const int before = __reduce_add_sync(FULL, lane < wid ? s_warp[lane] : 0);
  int4 o;
  o.x = start + before + x - own;
  o.y = o.x + v.x;
  o.z = o.y + v.y;
  o.w = o.z + v.z;
  reinterpret_cast<int4*>(offs + c * NBUCKET)[tid] = o;
}

// The whole pre-pass of a batch of at most kSmallBin pairs in one block:
// batch cells, keys, class sums and the list, sorted by key in shared memory
// (bitonic).  Four launches and their histogram (NCLASS_MAX * NBUCKET keys)
// took 85 us for 64 pairs, this 9.  s32_flag as in k_bin_count.
constexpr int kSmallBin = 4096;
static __global__ void __launch_bounds__(1024) k_bin_small(BinParams bp, const uint8_t* __restrict__ codes,
                                                           const PairDesc* __restrict__ pairs, int n,
                                                           const uint8_t* s32_flag, unsigned long long* total,
                                                           ClassSums* sums, int* class_range, ClassAllot* allot,
                                                           DevStatus* st, int* list, int* score, int* arange,
                                                           int* brange) {
  __shared__ unsigned long long s_key[kSmallBin];  // key << 32 | pair; rejected pairs and padding last
  __shared__ ClassSums s_sum[NCLASS_MAX];
  const int tid = threadIdx.x;
  __shared__ int8_t s_top[32];
  if (tid < NCLASS_MAX) s_sum[tid] = ClassSums{0, 0, 0};
  if (tid < 32) s_top[tid] = bp.top[tid];
  __syncthreads();
  unsigned long long local = 0;
  for (int p = tid; p < n; p += 1024) {
    const PairDesc d = pairs[p];
    if (pair_state(d, bp.n_codes, bp.max_a, bp.max_b) == PAIR_OK)
      local += (unsigned long long)d.a_len * (unsigned long long)d.b_len;
  }
  for (int off = 16; off > 0; off >>= 1) local += __shfl_xor_sync(FULL, local, off);
  if ((tid & 31) == 0 && local) atomicAdd(total, local);  // bp.total_cells, cleared before the run
  __threadfence();
  __syncthreads();
  int m = 32;  // entries sorted: the power of two that holds n
  while (m < n) m <<= 1;
  for (int p = tid; p < m; p += 1024) {
    unsigned long long e = ~0ull;
    // m is a multiple of 32: whole warps take part.
    const PairDesc d = p < n ? pairs[p] : PairDesc{0, 0, 0, 0};
    const int state = pair_state(d, bp.n_codes, bp.max_a, bp.max_b);
    const int flag = pair_flag(bp, s_top, codes, d, p < n && state == PAIR_OK, p, s32_flag);
    if (p < n) {
      if (state != PAIR_OK) {
        reject_pair(state, p, st, score, arange, brange);
      } else {
        const int key = tally_pair(bp, d, flag, s_sum, __activemask());
        e = ((unsigned long long)key << 32) | (unsigned)p;
      }
    }
    s_key[p] = e;
  }
  __syncthreads();
  for (int k = 2; k <= m; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < m / 2; i += 1024) {
        const int lo = ((i & ~(j - 1)) << 1) | (i & (j - 1)), hi = lo + j;
        const unsigned long long a = s_key[lo], b = s_key[hi];
        if ((a > b) == ((lo & k) == 0)) {
          s_key[lo] = b;
          s_key[hi] = a;
        }
      }
      __syncthreads();
    }
  for (int p = tid; p < n; p += 1024)
    if (s_key[p] != ~0ull) list[p] = (int)(unsigned)s_key[p];
  if (tid < bp.nclass) sums[tid] = s_sum[tid];
  if (tid < 32) allot_classes(bp, s_sum, class_range, allot, st);
}

// keys: of every pair, as k_bin_count left them (-1: not listed).
static __global__ void k_bin_scatter(const int* __restrict__ keys, int n, int* offs, int* list) {
  for (long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x) {
    const int key = keys[p];
    if (key < 0) continue;
    // One atomic per distinct key among the warp's lanes; each lane takes
    // the slot of its rank in the group.
    const unsigned act = __activemask();
    const unsigned same = __match_any_sync(act, key);
    const int lane = (int)(threadIdx.x & 31), leader = __ffs(same) - 1;
    int pos0 = 0;
    if (lane == leader) pos0 = atomicAdd(&offs[key], __popc(same));
    pos0 = __shfl_sync(act, pos0, leader);
    list[pos0 + __popc(same & ((1u << lane) - 1u))] = (int)p;
  }
}

// Synthetic calibration batch for the autotuner: n pairs of |A| = alen,
// |B| = blen; A uniform over `letters`, B = A with 1 in 8 residues
// substituted, then random letters past |A|.  related >= 0: A is drawn from
// the first half of the letters and B from the second, but for `related`
// residues of A's diagonal in equal distances, so that no alignment scores
// more than they do.
static __global__ void k_synth_pairs(uint8_t* codes, PairDesc* pairs, int n, int alen, int blen,
                                     const uint8_t* __restrict__ letters, int nletters, int related, uint32_t seed) {
  const int half = nletters / 2, diag = min(alen, blen);
  const long per = (long)alen + blen;
  for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < (long)n * per;
       k += (long)gridDim.x * blockDim.x) {
    const long p = k / per, i = k % per;
    auto hash = [&](long x) {
      uint32_t h = (uint32_t)x * 0x9E3779B1u ^ seed;
      h ^= h >> 15;
      h *= 0x85EBCA77u;
      h ^= h >> 13;
      h *= 0xC2B2AE3Du;
      return h ^ (h >> 16);
    };
    uint8_t v;
    if (i < alen) {
      v = letters[hash(p * 131071 + i) % (related < 0 ? nletters : half)];
    } else if (related >= 0) {
      const long j = i - alen;
      const bool kept = j < diag && j * related / diag != (j + 1) * related / diag;
      v = letters[kept ? hash(p * 131071 + j) % half : half + hash(p * 524287 + j + 7) % (nletters - half)];
    } else {
      const long j = i - alen;
      const uint32_t r = hash(p * 524287 + j + 7);
      v = (j < alen && (r & 7)) ? letters[hash(p * 131071 + j) % nletters] : letters[(r >> 3) % nletters];
    }
    codes[k] = v;
    if (i == 0) pairs[p] = PairDesc{p * per, p * per + alen, alen, blen};
  }
}

// Validates the Meta section of a device-resident wire buffer: lengths and
// offsets must stay inside their tile.  info = {maxA, maxB, bad slots}.
static __global__ void k_wire_check(const int* __restrict__ inputs, long metaOffset, long tileBytes,
                             int totalSlots, int* info, unsigned long long* cells) {
  for (long g = (long)blockIdx.x * blockDim.x + threadIdx.x; g < totalSlots;
       g += (long)gridDim.x * blockDim.x) {
    const int* m = inputs + metaOffset + 4 * g;
    const int al = m[0], ao = m[1], bl = m[2], bo = m[3];
    if (al == 0 || bl == 0) continue;
    if (al < 0 || bl < 0 || ao < 0 || bo < 0 || (long)ao + al > tileBytes || (long)bo + bl > tileBytes) {
      atomicAdd(&info[2], 1);
      continue;
    }
    atomicMax(&info[0], al);
    atomicMax(&info[1], bl);
    atomicAdd(cells, (unsigned long long)al * (unsigned long long)bl);
  }
}

// Wire buffer -> pair list: slot g of tile g / maxBatches, offsets made
// absolute in bytes from the start of the input buffer.
static __global__ void k_wire_to_pairs(const int* __restrict__ inputs, long seqWordsPerTile, long metaOffset,
                                int maxBatches, int totalSlots, PairDesc* pairs) {
  for (long g = (long)blockIdx.x * blockDim.x + threadIdx.x; g < totalSlots;
       g += (long)gridDim.x * blockDim.x) {
    const int* m = inputs + metaOffset + 4 * g;
    const long base = (g / maxBatches) * seqWordsPerTile * 4;
    pairs[g] = PairDesc{base + m[1], base + m[3], m[0], m[2]};
  }
}

}  // namespace ipuma_dev
