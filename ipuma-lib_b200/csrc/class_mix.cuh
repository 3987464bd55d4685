// class_mix.cuh -- k_mix, one persistent launch over the 16-bit wavefront
// classes of a batch.
//
// A warp takes items of one class after the other, widest strips first and
// longest pair first within a class.  A launch per class left each with a
// tail of its own and, in a batch of a few thousand pairs, cost more in
// launches and events than in cells; here a warp that finds a class finished
// goes on with the next class's, so only the batch has a tail.
// Warps of an SM are in the same or the next class's code most of the time,
// which the instruction cache holds (all classes at once on shares of the
// SMs ran 24 % slower on DNA).
//
// A model is a set of class kernels that share lanes and table scale:
//   kMixLin    linear gaps
//   kMixAff    affine, nucleic acids
//   kMixProt   affine, proteins: their profiles leave room for two blocks an
//              SM, so the kernel is compiled for two (B200, 10,000 pairs of
//              512 x 520: 0.67 ms, at 128 registers 0.74)
//   kMixAny    any score (64-column steps only)
// Each instantiation is a translation unit of its own (mix_*.cu): they hold
// up to 22 inlined passes and compile side by side.  Large 2-bit batches
// with linear gaps (kSepLin8) keep a launch per class: their 8-lane kernels
// use every register of four blocks an SM and lost 5 % in k_mix, more than
// their tails cost (1M DNA pairs 8.2 against 8.6 ms).
#pragma once
#include "sw_kernels.cuh"

namespace ipuma_dev {


// Lanes of the 16-bit classes.  Linear gaps keep four tag bits (2,047
// points), which fit every pair their strips are meant for; affine scorings,
// proteins mostly, keep two (8,191 points) so that only very long or
// near-identical pairs need the long class, whose lanes hold 16 bits.
// Matrices whose scaled values pass a profile byte run unscaled.
using LaneLin = LaneTag<4, true, true>;
using LaneAff = LaneTag<2, false, true>;
using LaneAny = LaneTag<2, false, false>;

constexpr int kMixLin = 0, kMixAff = 1, kMixProt = 2, kMixAny = 3, kSepLin8 = 4;

// Lanes and columns per lane of a class's strips in a model (0 lanes: the
// model has no kernel for it).  Strips of 16 * k columns: 16 lanes, or in
// kSepLin8 8 lanes of twice the columns (B200, 60,000 pairs of 240 x 320:
// 16 lanes 6488, 8 lanes 7061 GCUPS -- a lane's work per step covers twice
// the cells; affine lanes of more than 24 columns spill).
struct MixShape {
  int lanes, k;
};
constexpr MixShape mix_shape(int model, int cls) {
  constexpr int strip_k[16] = {4, 8, 12, 16, 0, 0, 0, 6, 10, 14, 5, 7, 9, 11, 13, 15};
  if (cls == 4) return {32, 12};
  if (cls == 5) return {32, 16};
  if (cls == 27 || cls == 28)
    return model == kMixAny || model == kSepLin8 ? MixShape{0, 0} : MixShape{32, cls == 27 ? 8 : 4};
  if (cls >= 16 && cls <= 20)  // in kSepLin8 those of classes 0, 10, 7, 11 and 1
    return model == kMixAny || model == kSepLin8 ? MixShape{0, 0} : MixShape{8, 2 * (cls - 16) + 8};
  if (cls < 0 || cls > 20 || strip_k[cls < 16 ? cls : 0] == 0) return {0, 0};
  if (model == kSepLin8) return {8, 2 * strip_k[cls]};
  if (model == kMixAny && strip_k[cls] % 4 != 0) return {0, 0};
  return {16, strip_k[cls]};
}

// Classes of a launch (bit c: class c), and the sizes its warps share.
struct MixArgs {
  unsigned mask;
  int warp_bytes;     // shared memory per warp: the largest of the classes
  long scr_per_warp;  // strip scratch (int2) per warp, likewise
};

template <int MODEL>
struct MixLane {
  using T = LaneAff;
};
template <>
struct MixLane<kMixLin> {
  using T = LaneLin;
};
template <>
struct MixLane<kMixAny> {
  using T = LaneAny;
};

using MixKernel = void (*)(SwConst, MixArgs, const int8_t*, BatchIo, const int*, const int*, int*, int2*,
                           unsigned long long*);
// The kernels, by model and mode (defined in mix_*.cu).
template <int MODEL, bool FWD>
MixKernel mix_kernel();

// The items of one class: a loop of its own, so that values of one class's
// passes are never live in another's (one loop over a switch of all classes
// hoisted every class's invariants and spilled thousands of bytes; called
// functions ran at 60 % of the rate).
template <int MODEL, bool FWD, int CLS>
__device__ __forceinline__ void mix_class(const SwConst& sc, const MixArgs& ma, const BatchIo& io, const int8_t* s_simp,
                                          uint8_t* wsmem, int2* wscr, const int* list, const int* ranges, int* heads,
                                          unsigned long long* trace) {
  constexpr MixShape sh = mix_shape(MODEL, CLS);
  if constexpr (sh.lanes > 0) {
    const int n = (ma.mask >> CLS) & 1u ? ranges[2 * CLS + 1] : 0;
    if (n <= 0) return;
    constexpr int PER_ITEM = 32 / sh.lanes * 2;
    const int items = (n + PER_ITEM - 1) / PER_ITEM;
    const int lane32 = threadIdx.x & 31;
    const int* l = list + ranges[2 * CLS];
    bool any = false;
    while (true) {
      int item = 0;
      if (lane32 == 0) item = atomicAdd(heads + CLS, 1);
      item = __shfl_sync(FULL, item, 0);
      if (item >= items) break;
      if (trace && !any && lane32 == 0) atomicMax(&trace[2 * CLS], ~global_ns());
      any = true;
      batched_item<typename MixLane<MODEL>::T, sh.k, sh.lanes, false, FWD>(sc, io, s_simp, wsmem, wscr, l,
                                                                           item * PER_ITEM, n);
    }
    if (trace && any && lane32 == 0) atomicMax(&trace[2 * CLS + 1], global_ns());
  }
}

// ranges: {start, count} of every class's part of the list; heads: a queue
// head per class.  trace: {~first item start, last item end} per class.
template <int MODEL, bool FWD>
__global__ void __launch_bounds__(128, MODEL == kMixProt ? 2 : FWD ? 4 : 3)
    k_mix(SwConst sc, MixArgs ma, const int8_t* __restrict__ sim, BatchIo io, const int* __restrict__ list,
          const int* __restrict__ ranges, int* heads, int2* scratch, unsigned long long* trace) {
  using T = typename MixLane<MODEL>::T;
  extern __shared__ __align__(16) uint8_t smem[];
  const int wib = threadIdx.x >> 5;
  int8_t* s_simp = reinterpret_cast<int8_t*>(smem);
  uint8_t* wsmem = smem + SubTable::bytes(sc.M, sc.P) + wib * ma.warp_bytes;
  int2* wscr = scratch + ((long)blockIdx.x * (blockDim.x >> 5) + wib) * ma.scr_per_warp;
  load_table(s_simp, sim, sc, kProfBias<T> ? -sc.gE : 0, kProfShift<T>);
  __syncthreads();
#define IPUMA_MIX(c) mix_class<MODEL, FWD, c>(sc, ma, io, s_simp, wsmem, wscr, list, ranges, heads, trace);
  IPUMA_MIX(5)
  IPUMA_MIX(4)
  IPUMA_MIX(27)
  IPUMA_MIX(3)
  IPUMA_MIX(15)
  IPUMA_MIX(9)
  IPUMA_MIX(14)
  IPUMA_MIX(2)
  IPUMA_MIX(13)
  IPUMA_MIX(8)
  IPUMA_MIX(12)
  IPUMA_MIX(28)
  IPUMA_MIX(1)
  IPUMA_MIX(20)
  IPUMA_MIX(11)
  IPUMA_MIX(19)
  IPUMA_MIX(7)
  IPUMA_MIX(18)
  IPUMA_MIX(10)
  IPUMA_MIX(17)
  IPUMA_MIX(0)
  IPUMA_MIX(16)
#undef IPUMA_MIX
}

}  // namespace ipuma_dev
