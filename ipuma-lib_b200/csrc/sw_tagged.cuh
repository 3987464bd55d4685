// sw_tagged.cuh -- the wavefront pass of the 16-bit classes (tag_pass).
//
// Same work layout and results as sw_pass (sw_device.cuh); what differs is
// how a cell is issued.  On B200 a scheduler takes two cycles of its ALU
// pipe for every 16-bit maximum, add-max, prmt and lop3, and two cycles of
// its FMA pipe, beside the ALU, for add.s16x2 and imad.  The pass therefore
// keeps only what has to be a maximum on the ALU:
//
//                                     linear gaps (gap_init = 0)     pipe
//   sub = prmt(profile words)         the same                       ALU
//   d   = H(diag) + sub               the same, HG(diag)             FMA
//   F̂   = max(F̂ + gE, H(up))          --                             ALU
//   Y   = max(F̂ + gI + gE, d, 0)      --                             ALU
//   Ê   = max(Ê + gE', Y(left))       --                             ALU
//   H   = max(Ê + gI + gE, Y)         max(d, HG(up), HG(left), 0)    ALU
//                                     HG = H + gE                    FMA
//   T   = H + tag                     inside the row maximum         FMA
//
// (F̂, Ê shifted by -(gI + gE) and gE' as in sw_device.cuh.)  With gap_init
// = 0 an extension never beats a new gap: E and F are HG of the left and
// upper neighbour, held in H's place (the profile holds sub - gE).  Affine
// lanes keep the one-instruction row chain Ê: the three-instruction chain of
// max(d, F, E) saved an ALU instruction but left 8-warp SMs waiting (B200,
// 10,000 protein pairs of 512 x 520: 0.88 against 0.75 ms).
//
// d belongs to the next row and is computed a step ahead: it crosses the
// loop's back edge, so the compiler cannot fold the add into the maximum
// (an add-max would be an ALU instruction), HG[c] is updated in place
// without register moves, and the profile loads have a step to arrive.
//
// Row maxima are tagged.  A cell enters the row's maximum as T, its score
// over TB tag bits that hold 2^TB - 1 - (column mod 2^TB); the maximum of
// 2^TB columns carries the first column that reaches it, and only one word
// per 2^TB columns is kept of the best row, not one per column.  SCALED
// lanes hold every value times 2^TB, so T is one add; the others multiply.
// Scores are limited accordingly (limit()); the limit is checked every 32
// steps, which add at most 32 * maxSub.
//
// Measured on B200 (one class launch, forward pass): 60,000 DNA pairs of
// 240 x 320, linear gaps 1.22 ms before -> 0.66 (16 lanes of 15 columns),
// 0.60 (8 lanes of 30), affine 0.98; 10,000 protein pairs of 512 x 520 0.81
// -> 0.66; 20,000 of 224 x 350 0.57 -> 0.44.  ALU instructions per column
// and warp 8.0 -> 3.9 (linear), 6.6 (affine).  What bounds it now: the ALU
// pipe, 77 % busy over a launch of affine DNA (three blocks an SM) and 70 %
// of proteins (two); linear gaps issue 0.67 to 0.72 instructions a cycle with
// the ALU pipe at 68 to 71 %, which more resident warps did not raise (20 or
// 24 per SM: within 5 %).
#pragma once
#include "sw_device.cuh"

namespace ipuma_dev {

// On every lambda of the pass: its arrays live in registers only if all of
// them are inlined, which the compiler stops doing in a translation unit that
// holds many passes.
#define IPUMA_INLINE __attribute__((always_inline))


__device__ __forceinline__ uint32_t add16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("add.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t maxu16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t minu16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("min.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// Two pairs per lane (pair P low, pair Q high), TB tag bits; LIN: gap_init = 0.
template <int TB, bool LIN, bool SCALED>
struct LaneTag {
  using V = uint32_t;
  static constexpr int NP = 2;
  static constexpr int TAG = TB;
  static constexpr bool LINEAR = LIN;
  static constexpr int SH = SCALED ? TB : 0;  // bits H itself is shifted by
  static constexpr int BIAS = 0;
  static constexpr bool BIG = false;
  static constexpr uint32_t MASK = ((1u << TB) - 1u) * 0x00010001u;  // the tag bits of both halves
  static constexpr uint32_t ONE = 0x00010001u << TB;                 // one score point in both halves
  __device__ __forceinline__ static V splat(int x) {
    return (uint32_t)(x & 0xffff) | ((uint32_t)(x & 0xffff) << 16);
  }
  // Running best: the score with every tag bit set, which a later row has
  // to exceed.
  __device__ __forceinline__ static V best_of(int lo, int hi) {
    return ((uint32_t)(lo << TB) | ((uint32_t)(hi << TB) << 16)) | MASK;
  }
  __device__ __forceinline__ static int score(V best, int h) {
    return (int)((h ? best >> 16 : best & 0xffffu) >> TB);
  }
  // Largest score at a check: the 32 steps to the next one add at most
  // maxSub each, and T must still fit 16 bits.
  __host__ __device__ static int limit(int maxSub) { return (SCALED ? (32767 >> TB) : (1 << (16 - TB)) - 1) - 32 * maxSub; }
};

// Two pairs per lane with all 16 bits for the score, held as an unsigned
// halfword score + BIAS: the sums H + sub, F + gI + gE and E + gI + gE stay
// at or above 0 (sub >= -128, gI + gE > -1000).  No tag bits: the best row
// is kept whole, and the recurrence's floor is the BIAS of Y's 3-way max.
struct LaneBig {
  using V = uint32_t;
  static constexpr int NP = 2;
  static constexpr int TAG = 0;
  static constexpr bool LINEAR = false;
  static constexpr int SH = 0;
  static constexpr int BIAS = 1024;
  static constexpr bool BIG = true;
  static constexpr uint32_t MASK = 0, ONE = 0x00010001u;
  __device__ __forceinline__ static V best_of(int lo, int hi) {
    return (uint32_t)(lo + BIAS) | ((uint32_t)(hi + BIAS) << 16);
  }
  __device__ __forceinline__ static int score(V best, int h) {
    return (int)(h ? best >> 16 : best & 0xffffu) - BIAS;
  }
  __host__ __device__ static int limit(int maxSub) { return 65535 - BIAS - 33 * maxSub; }
};

template <>
struct Cell<LaneBig> {
  __host__ __device__ __forceinline__ static int limit(const SwConst& sc) { return LaneBig::limit(sc.maxSub); }
};

template <int TB, bool LIN, bool SCALED>
struct Cell<LaneTag<TB, LIN, SCALED>> {
  __host__ __device__ __forceinline__ static int limit(const SwConst& sc) { return LaneTag<TB, LIN, SCALED>::limit(sc.maxSub); }
};

template <int C>
__device__ __forceinline__ uint32_t unpack_sub(uint32_t wp, uint32_t wq) {
  return prmt(wp, wq, (uint32_t)(C | ((C | 8) << 4) | ((4 + C) << 8) | (((4 + C) | 8) << 12)));
}

// Profile rows of a pass's B letters.  Packed codes: 32-bit bit positions
// from the word of row 0 (rows < 65536, so they stay below 2^20).
struct RowLetters {
  const uint8_t* p;
  int bit0, step, bits, shift;
  __device__ __forceinline__ RowLetters(const SwConst& sc, const PassSeq& ps) : bits(sc.bits), shift(sc.pshift) {
    if (bits == 8) {
      p = ps.base + ps.b;
      bit0 = 0;
      step = ps.db;
    } else {
      const long long bit = ps.b * bits;
      p = ps.base + (bit >> 5) * 4;
      bit0 = (int)(bit & 31);
      step = ps.db * bits;
      shift = bits == 2 ? shift - 1 : shift;  // 2-bit fields hold code - 1
    }
  }
  __device__ __forceinline__ int at(int r) const {
    const int o = bit0 + r * step;
    if (bits == 8) return (int)p[o] - shift;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(p) + (o >> 5);
    return (int)(__funnelshift_r(__ldg(w), __ldg(w + 1), (uint32_t)o & 31u) & ((1u << bits) - 1u)) - shift;
  }
};

// raise_to_group of tagged bests: the group's best score minus one with
// every tag bit set (a group best of 0 stays 0).
template <class T, int LANES>
__device__ __forceinline__ uint32_t raise_tagged(uint32_t best) {
  uint32_t g = best;
#pragma unroll
  for (int off = LANES / 2; off > 0; off >>= 1) g = maxu16x2(g, __shfl_xor_sync(FULL, g, off, LANES));
  constexpr uint32_t ZERO = (uint32_t)T::BIAS * 0x00010001u + T::MASK;  // score 0
  return maxu16x2(best, maxu16x2(g, ZERO + T::ONE) - T::ONE);
}

// Parameters, scratch and return value as sw_pass; the boundary column
// holds (HG, E) of a strip's last column.
template <class T, int K, int LANES, bool EARLY = false, bool TEAM = false>
__device__ __forceinline__ bool tag_pass(const SwConst& sc, uint8_t* s_prof, const int8_t* s_simp,
                                         uint16_t* s_bring, const PassSeq (&ps)[2], int2* scr, long rowsCap,
                                         Best (&out)[2], PassStop stop = PassStop{}, StripTeam team = StripTeam{}) {
  static_assert(!TEAM || (LANES == 32 && !EARLY), "strip teams run whole-warp passes without an early stop");
  constexpr int TB = T::TAG;
  constexpr bool LINEAR = T::LINEAR;
  constexpr int SW = LANES * K;
  constexpr int KP = ProfileWords<K>::KP;
  constexpr int SWP = LANES * KP;
  constexpr int W = 1 << TB;            // columns per tag group
  constexpr int NG = (K + W - 1) / W;   // tag groups of a lane
  // The next row's profile loads go out before this row's maxima, which a
  // warp alone on its scheduler would otherwise wait for; with more than 16
  // columns they would take the registers of the maxima instead.
  constexpr bool kLoadFirst = K <= 16;
  const int lane = threadIdx.x & (LANES - 1);
  const int P = sc.P;
  const int profStride = (P + 1) * SWP;
  const ProfilePtr<K, LANES> prof{(uint32_t)lane};
  const uint8_t* profQ = s_prof + profStride;

  int rowsG = 0, amax = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    rowsG = max(rowsG, ps[h].blen);
    amax = max(amax, ps[h].alen);
    out[h] = Best{0, 0, 0};
  }
  int rowsW = __reduce_max_sync(FULL, rowsG);
  int rowsMin = __reduce_min_sync(FULL, rowsG);
  const int nstrips = (__reduce_max_sync(FULL, amax) + SW - 1) / SW;
  int capRows[2] = {ps[0].blen, ps[1].blen};  // EARLY: rows each pair still needs
  const unsigned gmask = (LANES == 32) ? FULL : (((1u << LANES) - 1u) << (threadIdx.x & (32 - LANES)));
  const uint32_t vgE = sc.gE2;
  const uint32_t vgIgE = sc.gIgE2;  // also HG, E and F where H = 0 and no gap is open
  const uint32_t vgEp = sc.gEp2;
  const uint32_t tagMul = (uint32_t)sc.one << TB;  // 2^TB that the compiler keeps as an imad
  const int lim = T::limit(sc.maxSub);
  const auto wbuf = [&](int s) IPUMA_INLINE -> int { return TEAM ? s % team.warps : s & 1; };
  bool teamGaveUp = false;
  const RowLetters letter[2] = {RowLetters(sc, ps[0]), RowLetters(sc, ps[1])};

  // TEAM: waits until the previous warp published `need` rows of strip s's
  // boundary.  Warp-uniform; false once the team gave up (as in sw_pass).
  auto team_wait = [&](int s, int need) IPUMA_INLINE -> bool {
    bool ok = true;
    if constexpr (TEAM) {
      const int target = (s << 16) | need;
      const volatile int* pr = team.prog + (team.warp + team.warps - 1) % team.warps;
      const volatile int* ab = team.abort;
      unsigned long long t_start = 0;
      for (int it = 0; *pr < target; ++it) {
        if (*ab != 0) {
          ok = false;
          break;
        }
        if ((it & 255) == 0) {
          const unsigned long long now = global_ns();
          if (it == 0) t_start = now;
          if (now - t_start > kTeamWaitNs || it >= (1 << 26)) {
            atomicCAS(team.err, 0, team.errCode);
            *(volatile int*)team.abort = 1;
            ok = false;
            break;
          }
        }
        __nanosleep(64);
      }
      __threadfence_block();  // the boundary rows are read after the flag
      ok = __all_sync(FULL, ok);
    }
    return ok;
  };

  for (int strip = TEAM ? team.warp : 0; strip < nstrips; strip += TEAM ? team.warps : 1) {
    if constexpr (EARLY) {
      if (stop.on && strip > 0) {
        rowsG = max(min(ps[0].blen, capRows[0]), min(ps[1].blen, capRows[1]));
        rowsW = __reduce_max_sync(FULL, rowsG);
        rowsMin = __reduce_min_sync(FULL, rowsG);
        if (rowsW == 0) break;  // caps only shrink: no later strip can win
      }
    }
    const int col0 = strip * SW;
    const bool hasIn = strip > 0;
    const bool hasOut = strip + 1 < nstrips;
    const int2* scrIn = scr + (hasIn ? wbuf(strip - 1) : 0) * rowsCap;
    int2* scrOut = scr + wbuf(strip) * rowsCap;

    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
      build_profile<K, LANES>(s_prof + h * profStride, s_simp, sc, ps[h], col0, lane);

    // B letters: lane k of `bnext` holds the profile row offsets of one row
    // (pair h in halfword h), parked in the rings a block at a time.  A
    // block of steps starting at t0 reads rows up to t0 + LANES.
    auto fetch_letters = [&](int r) IPUMA_INLINE -> uint32_t {
      uint32_t v = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int x = r < ps[h].blen ? min((uint32_t)letter[h].at(r), (uint32_t)P) : P;
        v |= (uint32_t)(x * SWP) << (16 * h);
      }
      return v;
    };
    auto park_letters = [&](int r, uint32_t v) IPUMA_INLINE {
      const int w = r & 63;
      s_bring[w] = s_bring[w + 64] = (uint16_t)v;
      s_bring[128 + w] = s_bring[192 + w] = (uint16_t)(v >> 16);
    };
    park_letters(lane, fetch_letters(lane));
    uint32_t bnext = fetch_letters(1 + lane);
    __threadfence_block();
    __syncwarp();

    uint32_t H[K], F[K], d[K], snap[NG];
    constexpr uint32_t ZERO = (uint32_t)T::BIAS * 0x00010001u;
    const uint32_t vH0 = LINEAR ? vgE : ZERO;  // H = 0 as held (H + gE for linear gaps)
#pragma unroll
    for (int c = 0; c < K; ++c) {
      H[c] = vH0;
      if constexpr (!LINEAR) F[c] = ZERO;
    }
#pragma unroll
    for (int g = 0; g < NG; ++g) snap[g] = 0;
    uint32_t outH = vH0, outE = ZERO;
    // Running best, started one below the pair's best of the strips before
    // (a cell that ties it can still win on its row), and its row, one
    // halfword per pair (rows < 65536).
    uint32_t best = T::best_of(max(out[0].s - 1, 0), max(out[1].s - 1, 0));
    uint32_t brow = 0;

    // Boundary of the previous strip: lane k of a chunk holds row
    // (chunkBase + k).
    int2 chunk = make_int2(0, 0), chunkNext = make_int2(0, 0);
    if (hasIn) {
      // (A team reads each block's rows when it starts the block: one block
      // less behind the strip before it, for one exposed load.)
      if (!TEAM && lane < rowsG) chunk = scrIn[lane];
      if (!TEAM && LANES + lane < rowsG) chunkNext = scrIn[LANES + lane];
    } else {
      chunk = chunkNext = make_int2((int)vH0, (int)ZERO);  // H = 0 left of the first strip
    }

    // Profile words of the row whose letters lie at `ring`, and its d from
    // the left neighbour's H of the row above, `left`.
    uint32_t wp[KP / 4], wq[KP / 4];
    auto fetch_profile = [&](const uint16_t* ring) IPUMA_INLINE {
      prof.load(wp, s_prof + ring[0]);
      prof.load(wq, profQ + ring[128]);
    };
    auto ahead = [&](uint32_t left) IPUMA_INLINE {
#pragma unroll
      for (int c = 0; c < K; ++c) {
        uint32_t sb;
        switch (c & 3) {
          case 0: sb = unpack_sub<0>(wp[c >> 2], wq[c >> 2]); break;
          case 1: sb = unpack_sub<1>(wp[c >> 2], wq[c >> 2]); break;
          case 2: sb = unpack_sub<2>(wp[c >> 2], wq[c >> 2]); break;
          default: sb = unpack_sub<3>(wp[c >> 2], wq[c >> 2]); break;
        }
        d[c] = add16x2(c == 0 ? left : H[c > 0 ? c - 1 : 0], sb);
      }
    };
    // Row i's maxima; `left` and `e` are the left neighbour's HG and E of
    // this row, rows = i in both halfwords.
    auto row = [&](int i, uint32_t rows, uint32_t left, uint32_t e, auto multi) IPUMA_INLINE {
      uint32_t tv[K];
#pragma unroll
      for (int c = 0; c < K; ++c) {
        uint32_t h;
        if constexpr (LINEAR) {
          h = __vimax3_s16x2_relu(d[c], H[c], left);
          left = H[c] = add16x2(h, vgE);
        } else if constexpr (T::BIG) {
          F[c] = __viaddmax_u16x2(F[c], vgE, H[c]);
          const uint32_t y = __vimax3_u16x2(d[c], add16x2(F[c], vgIgE), ZERO);
          if (c > 0) e = __viaddmax_u16x2(e, vgEp, left);
          h = H[c] = __viaddmax_u16x2(e, vgIgE, y);
          left = y;
        } else {
          F[c] = __viaddmax_s16x2(F[c], vgE, H[c]);
          const uint32_t y = __viaddmax_s16x2_relu(F[c], vgIgE, d[c]);
          if (c > 0) e = __viaddmax_s16x2(e, vgEp, left);
          h = H[c] = __viaddmax_s16x2(e, vgIgE, y);
          left = y;
        }
        const uint32_t tag = (uint32_t)(W - 1 - c % W) * 0x00010001u;
        if constexpr (LINEAR && T::SH > 0)
          tv[c] = c % W ? h : h + tag;  // the other columns' tags are added in the maximum
        else
          tv[c] = T::BIG ? h : T::SH > 0 ? h + tag : h * tagMul + tag;
      }
      outH = H[K - 1];
      if constexpr (T::BIG)
        outE = __viaddmax_u16x2(e, vgEp, left);
      else if constexpr (!LINEAR)
        outE = __viaddmax_s16x2(e, vgEp, left);
      uint32_t gm[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        const int n = (K - g * W) < W ? (K - g * W) : W;
        uint32_t m = tv[g * W];
        if constexpr (LINEAR && T::SH > 0) {
#pragma unroll
          for (int c = 1; c < W; ++c)
            if (c < n) m = __viaddmax_u16x2(tv[g * W + c], (uint32_t)(W - 1 - c) * 0x00010001u, m);
        } else {
#pragma unroll
        for (int c = 1; c < W; c += 2) {
          if (c + 1 < n)
            m = __vimax3_u16x2(m, tv[g * W + c], tv[g * W + c + 1]);
          else if (c < n)
            m = maxu16x2(m, tv[g * W + c]);
        }
        }
        gm[g] = m;
      }
      uint32_t rm = gm[0];
#pragma unroll
      for (int g = 1; g < NG; g += 2) rm = g + 1 < NG ? __vimax3_u16x2(rm, gm[g], gm[g + 1]) : maxu16x2(rm, gm[g]);
      // Strict >: the first row of a score keeps it.  imp = all-ones in the
      // halves that improved.
      const uint32_t up = maxu16x2(best, rm);
      const uint32_t imp = minu16x2(up - best, 0x00010001u) * 0xffffu;
      brow = (brow & ~imp) | (rows & imp);
#pragma unroll
      for (int g = 0; g < NG; ++g) snap[g] = (snap[g] & ~imp) | (gm[g] & imp);
      best = up | T::MASK;
      if constexpr (decltype(multi)::value) {
        if (hasOut && lane == LANES - 1) scrOut[i] = make_int2((int)outH, (int)outE);
      }
    };
    // One wavefront step: lane works on row i = t - lane, then prepares
    // row i + 1 (rows past the end read the padding letter).
    auto step = [&](int i, int k, uint32_t rows, const uint16_t* ring, auto check, auto multi) IPUMA_INLINE {
      uint32_t left = __shfl_up_sync(FULL, outH, 1, LANES);
      uint32_t e = ZERO;
      if constexpr (!LINEAR) e = __shfl_up_sync(FULL, outE, 1, LANES);
      if constexpr (decltype(multi)::value) {
        const uint32_t bh = (uint32_t)__shfl_sync(FULL, chunk.x, k, LANES);
        uint32_t be = 0;
        if constexpr (!LINEAR) be = (uint32_t)__shfl_sync(FULL, chunk.y, k, LANES);
        if (lane == 0) {
          left = bh;
          e = be;
        }
      } else if (lane == 0) {
        left = vH0;
        e = ZERO;
      }
      if constexpr (decltype(check)::value) {
        if (i >= 0 && i < rowsG) row(i, rows, left, e, multi);
        if (i >= -1) {
          fetch_profile(ring);
          ahead(left);
        }
      } else {
        if (kLoadFirst) fetch_profile(ring);
        row(i, rows, left, e, multi);
        if (!kLoadFirst) fetch_profile(ring);
        ahead(left);
      }
    };
    // The row before the first: lane 0 prepares row 0.
    if (lane == 0) {
      fetch_profile(s_bring);
      ahead(vH0);
    }

    const int nsteps = rowsW + LANES - 1;
    bool gaveUp = false;
    int stopAt = nsteps;  // EARLY: end of the block after every pair is done
    for (int t0 = 0; t0 < nsteps; t0 += LANES) {
      if constexpr (EARLY) {
        if (t0 >= stopAt) break;
        if (stop.on && stopAt == nsteps) {
          // Done (warp-uniform): every group reached its target before t0,
          // or all lanes are past its rows.
          bool done = true;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const bool found = (__ballot_sync(FULL, T::score(best, h) >= stop.target[h]) & gmask) != 0;
            done = done && (found || t0 - (LANES - 1) >= min(ps[h].blen, capRows[h]));
          }
          if (__all_sync(FULL, done)) stopAt = t0 + LANES;
        }
      }
      if ((t0 & 31) == 0) {
        if (__any_sync(FULL, T::score(best, 0) > lim || T::score(best, 1) > lim)) {
          gaveUp = true;
          break;
        }
      }
      if constexpr (TEAM) {
        // Another warp gave up: this pass's results are not used.
        if (__any_sync(FULL, *(volatile int*)team.abort != 0)) {
          teamGaveUp = true;
          break;
        }
      }
      if (t0 > 0) best = raise_tagged<T, LANES>(best);
      park_letters(t0 + 1 + lane, bnext);
      bnext = fetch_letters(t0 + LANES + 1 + lane);
      __syncwarp();
      if constexpr (TEAM) {
        if (hasIn) {
          if (!team_wait(strip - 1, min(t0 + LANES, rowsG))) {
            teamGaveUp = true;
            break;
          }
          chunk = (t0 + lane < rowsG) ? scrIn[t0 + lane] : make_int2(0, 0);
        }
      } else if (hasIn && t0 > 0) {
        chunk = chunkNext;
        const int r = t0 + LANES + lane;
        chunkNext = (r < rowsG) ? scrIn[r] : make_int2(0, 0);
      }
      const bool all = t0 >= LANES - 1 && t0 + LANES - 1 < rowsMin;
      int i = t0 - lane;
      uint32_t rows = (uint32_t)i * 0x00010001u;
      const uint16_t* ring = s_bring + ((i + 1) & 63);  // slot of row i + 1, < 64 + LANES
      auto block = [&](auto check, auto multi) IPUMA_INLINE {
#pragma unroll 1
        for (int k = 0; k < LANES; ++k) {
          step(i, k, rows, ring, check, multi);
          ++i;
          rows += 0x00010001u;
          ++ring;
        }
      };
      if (nstrips > 1) {
        if (all) block(std::false_type{}, std::true_type{});
        else block(std::true_type{}, std::true_type{});
      } else {
        if (all) block(std::false_type{}, std::false_type{});
        else block(std::true_type{}, std::false_type{});
      }
      if constexpr (TEAM) {
        // Lane LANES - 1 wrote the boundary rows up to t0 (those below
        // rowsG): release them to the next strip's warp.
        if (hasOut && lane == LANES - 1) {
          __threadfence_block();
          *(volatile int*)(team.prog + team.warp) = (strip << 16) | min(t0 + 1, rowsG);
        }
      }
    }
    if constexpr (TEAM) {
      if (teamGaveUp) break;
    }
    if (!gaveUp) gaveUp = __any_sync(FULL, T::score(best, 0) > lim || T::score(best, 1) > lim);
    if (gaveUp) {
      if constexpr (TEAM) {
        if (lane == 0) *(volatile int*)team.abort = 1;
      }
      return false;
    }
    // Strip result: first column of the lane's best row that holds its best.
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      int s = T::score(best, h);
      int jj = 0;
#pragma unroll
      for (int g = NG - 1; g >= 0; --g) {
        const int v = (int)((snap[g] >> (16 * h)) & 0xffffu) - T::BIAS;
        if ((v >> TB) == s) jj = g * W + W - 1 - (v & (W - 1));
      }
      int ii = (int)((brow >> (16 * h)) & 0xffffu);
      int j = col0 + lane * K + jj;
      if (s <= 0) {
        s = 0;
        ii = 0;
        j = 0;
      }
      group_best_reduce<LANES>(s, ii, j);
      if (better(s, ii, j, out[h].s, out[h].i, out[h].j)) out[h] = Best{s, ii, j};
      if constexpr (EARLY) {
        if (stop.on && out[h].s >= stop.target[h]) capRows[h] = min(capRows[h], out[h].i);
      }
    }
    if (hasOut) {
      __threadfence_block();
      __syncwarp();
    }
  }
  return !teamGaveUp;
}

}  // namespace ipuma_dev
