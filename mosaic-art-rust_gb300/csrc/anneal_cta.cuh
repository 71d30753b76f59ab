// anneal_cta.cuh -- one simulated-annealing chain by one CTA (anneal_cta_kernel,
// for single mosaics and for every chain of a batch).
//
// Reference: optimizer.rs:41-129 MosaicOptimizer::optimize, optimizer.rs:132-198
// optimize_greedy, adjacency.rs:133-214 calculate_swap_delta.
//
// A chain is a sequence of dependent swaps, so its speed is the latency from
// one swap to the next that reads its cells.  Almost everything about a
// proposal is known ahead of the chain: its two cells (a counter-based draw),
// whether it is skipped (swaps never move empty cells, so emptiness is a
// property of the start grid), its temperature (the decay is applied once per
// earlier proposal that is not skipped, whatever was accepted) and with it the
// deltas that are accepted; and which earlier proposals can matter to it: those
// that may swap a cell it reads, i.e. with a position within Manhattan distance
// 1 of its own.  Only the eight neighbour weights need the grid.  So the work is
// split by warp, window of 64 proposals by window:
//   * kProducers warps take a window each in turn: draw and decode, skip flags,
//     the window's temperatures (one chain of multiplications, handed from
//     window to window), the acceptance bounds, and each proposal's level --
//     0 when no earlier proposal of the window is near it, else one more than
//     the highest level among those that are;
//   * kEvalWarps warps evaluate a window level by level, four lanes a proposal
//     (one direction each: a neighbour of either position), decide and swap.
//     Proposals of one level do not
//     touch one another's cells, and a proposal comes after every earlier one
//     near it, so each reads the grid exactly as the sequential chain would;
//   * one warp keeps the books two windows behind: the running cost is summed in
//     proposal order, with the best cost and the counters.
// Acceptance: u < exp(-delta / T) is decided by comparing delta with -T ln u
// when it lies further from it than 1e-4 T (over ten times the error of the
// logarithm, the division and this library's exp together), else by the
// definition itself.
// The warps meet at named barriers only (no spinning): FULL[slot] when a window
// is prepared and the one two before it is done (producer, evaluators, book
// keeper), EMPTY[slot] when the evaluators hold a window's descriptors in
// registers, TEMP[slot] when a window's first temperature is known, EVAL between
// levels and windows.
//
// What bounds it: the latency of a level (shared-memory reads of cells, then
// Lab; square roots and reciprocals; the in-order sum of eight terms; a
// barrier).  A window of 64 takes ~2 000 cycles on a 24 000-cell grid (1.9
// levels on average), issue slots 39% used.  Before, a CTA of four warps drew,
// evaluated, tested all pairs for conflicts and booked 32 (or 16) proposals in
// turn, ~4 000 (2 550) cycles a round.  Measured, GB300, before -> now:
// 64 chains x 100 000 iterations on 179 x 134 cells 6.32 -> 1.49 ms; 32 x 2000
// on 80 x 60 0.203 -> 0.060 ms.  Windows of 32, eight lanes a proposal (16
// warps), and two proposals a group of eight lanes were measured too: 2.1, 1.55
// and 2.0 ms on the first.
#pragma once
#include "mg_internal.h"
#include "roots.cuh"

namespace mg {
namespace anneal_detail {

constexpr uint16_t kNone16 = 0xFFFFu;  // a cell without a tile
constexpr int kWindow = 64;     // proposals per window
constexpr int kEvalWarps = 8;   // four lanes a proposal
constexpr int kEval = kEvalWarps * 32;
constexpr int kProducers = 4;   // warps preparing windows, two proposals a lane; also the descriptor slots
constexpr int kThreads = kEval + 32 * kProducers + 32;
// named barriers (0 is __syncthreads)
constexpr int kBarFull = 1, kBarEmpty = kBarFull + kProducers, kBarTemp = kBarEmpty + kProducers,
              kBarEval = kBarTemp + kProducers;
static_assert(kBarEval < 16, "sixteen barriers a CTA");

struct Proposal {        // a prepared proposal
  int p1, p2;            // cells
  uint32_t flags;        // bits 0-7: neighbour t lies in the grid and is not the other position; 8: adjacent
                         // positions; 9-10: direction of pos2 from pos1; 11: not skipped; 16-21: level
  float lo;              // accepted when delta < lo (delta < 0 always is)
  float hi;              // rejected when delta > hi
  float u, t;            // acceptance uniform, temperature
  int levels;            // levels of the window
};
struct Outcome {  // a window's decisions, for the book keeper
  float delta[kWindow];     // 0 unless accepted
  uint32_t flags[kWindow];  // bit 0: accepted, 1: not skipped
};
constexpr int kTermStride = 36;  // floats between the sets of a warp's terms (four banks apart)
struct ChainShared {
  Proposal ring[kProducers][kWindow];
  Outcome out[3];
  float terms[kEvalWarps][4 * kTermStride];  // old, old, new, new weights: neighbours of pos1, of pos2
  int2 pos[kProducers][kWindow];           // a window's positions, as near_pos takes them
  float temps[kProducers][kWindow + 4];    // the window's first temperature after 0, 1, ... coolings
  float temp[kProducers];                  // first temperature of the window in the slot
  float sums[kWindow];                     // the running cost after each proposal of a window
  int first[4];                            // greedy descent: the lowest level that accepts, in [0] and [1] by turns
};

// Behind it: the writers table (kProducers x 2 x writer_slots words), the
// palette Lab, the grid (one 16-bit material a cell, and an empty cell n).
// More table slots leave fewer chance hits; the largest grids leave room for few.
constexpr int kWriterSlots = 4096, kWriterSlotsShared = 512, kWriterSlotsMin = 64;
__host__ __device__ inline size_t anneal_cta_smem_bytes(int max_cells, int p, bool lab_smem, int writer_slots) {
  return sizeof(ChainShared) + (size_t)kProducers * 2 * 4 * writer_slots + (lab_smem ? (size_t)p * 16 : 0) +
         ((((size_t)max_cells + 1) * 2 + 15) & ~(size_t)15);
}
static_assert(sizeof(ChainShared) % 16 == 0, "16-byte aligned parts");

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// bar_sync; whether v holds in any of the threads.
__device__ __forceinline__ bool bar_any(int id, int threads, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.or.aligned.pred q, %1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(id), "r"(threads), "r"((uint32_t)v)
      : "memory");
  return r != 0u;
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("barrier.cta.arrive.aligned %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
constexpr int kFullThreads = 32 + kEval + 32, kEmptyThreads = kEval + 32, kTempThreads = 64;

// Positions y * S + x with S >= gw + 2: within Manhattan distance 1 exactly
// when they differ by 0, 1 or S.
__device__ __forceinline__ bool near_pos(int a, int b, int S) {
  const int d = abs(a - b);
  return d <= 1 || d == S;
}

// Producer `slot`: prepares windows slot, slot + kProducers, ...; a lane holds
// proposals lane and lane + 32 (h = 0, 1).
__device__ __forceinline__ void produce_windows(const AnnealJob& J, int chain, long long windows, int slot,
                                                ChainShared& S, uint32_t* writers, int writer_slots,
                                                const uint16_t* s_grid) {
  const int lane = threadIdx.x & 31;
  const int gw = J.gw, gh = J.gh, stride = gw + 2;
  const bool greedy_only = J.greedy_only != 0;
  const float decay = J.decay, inf = __int_as_float(0x7f800000);
  const unsigned below = (1u << lane) - 1u;
  int2* pos = S.pos[slot];
  float* temps = S.temps[slot];
  uint2* table = reinterpret_cast<uint2*>(writers) + (size_t)slot * writer_slots;
  const unsigned tmask = (unsigned)writer_slots - 1u;
  for (long long w = slot; w < windows; w += kProducers) {
    int x1[2], y1[2], x2[2], y2[2], c1[2], c2[2];
    float u[2];
    bool skip[2];
    unsigned live[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long my = w * kWindow + 32 * h + lane;
      const uint32_t hi32 = (uint32_t)((unsigned long long)my >> 32);
      const u32x4 a = philox((uint32_t)my, (uint32_t)chain, J.stream, 2u * hi32, J.key0, J.key1);
      const u32x4 b = philox((uint32_t)my, (uint32_t)chain, J.stream, 2u * hi32 + 1u, J.key0, J.key1);
      x1[h] = (int)range_u32(a.x, (uint32_t)gw);
      y1[h] = (int)range_u32(a.y, (uint32_t)gh);
      x2[h] = (int)range_u32(a.z, (uint32_t)gw);
      y2[h] = (int)range_u32(a.w, (uint32_t)gh);
      u[h] = unit_f32(b.x);
      c1[h] = y1[h] * gw + x1[h];
      c2[h] = y2[h] * gw + x2[h];
      // emptiness never changes, so reading beside the evaluators' swaps is safe
      skip[h] = my >= J.iters || c1[h] == c2[h] || s_grid[c1[h]] == kNone16 || s_grid[c2[h]] == kNone16;
      live[h] = __ballot_sync(0xffffffffu, !skip[h]);
      pos[32 * h + lane] = make_int2(y1[h] * stride + x1[h], y2[h] * stride + x2[h]);
    }

    // ---- temperatures: the window's first one comes from the window before.
    // One chain of multiplications; each lane then picks its own.
    if (!greedy_only) {
      if (w > 0) bar_sync(kBarTemp + slot, kTempThreads);
      float tk = w > 0 ? S.temp[slot] : J.t0;
#pragma unroll
      for (int k = 0; k < kWindow; k += 4) {
        float4 v;
        v.x = tk;
        v.y = __fmul_rn(v.x, decay);
        v.z = __fmul_rn(v.y, decay);
        v.w = __fmul_rn(v.z, decay);
        tk = __fmul_rn(v.w, decay);
        *reinterpret_cast<float4*>(temps + k) = v;
      }
      temps[kWindow] = tk;
      __syncwarp();
      if (w + 1 < windows) {
        const int next = (slot + 1) % kProducers;
        if (lane == 0) S.temp[next] = temps[__popc(live[0]) + __popc(live[1])];
        __syncwarp();
        bar_arrive(kBarTemp + next, kTempThreads);
      }
    }

    // ---- levels.  The writers table holds, per (hashed) cell, which proposals
    // of the window may swap it; a proposal looks up the ten cells it reads,
    // keeps the earlier ones and checks each against the positions (chance hits
    // of the hash drop out).
    auto at = [&](int c) -> uint2& { return table[(unsigned)c & tmask]; };
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (!skip[h]) {
        uint32_t* t1 = h ? &at(c1[h]).y : &at(c1[h]).x;
        uint32_t* t2 = h ? &at(c2[h]).y : &at(c2[h]).x;
        atomicOr(t1, 1u << lane);
        atomicOr(t2, 1u << lane);
      }
    __syncwarp();
    unsigned e0 = 0u, e10 = 0u, e11 = 0u;  // earlier proposals near this lane's: h = 0's; h = 1's in either half
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int a = e ? c2[0] : c1[0], b = e ? c2[1] : c1[1];
      e0 |= at(a).x | at(a - 1).x | at(a + 1).x | at(a - gw).x | at(a + gw).x;
      const int bs[5] = {b, b - 1, b + 1, b - gw, b + gw};
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const uint2 v = at(bs[k]);
        e10 |= v.x;
        e11 |= v.y;
      }
    }
    e0 = skip[0] ? 0u : e0 & below;
    e10 = skip[1] ? 0u : e10;
    e11 = skip[1] ? 0u : e11 & below;
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (!skip[h]) at(c1[h]) = at(c2[h]) = make_uint2(0u, 0u);
    {
      const int2 q0 = pos[lane], q1 = pos[32 + lane];
      unsigned m0 = e0, m10 = e10, m11 = e11;
      while (__any_sync(0xffffffffu, (m0 | m10 | m11) != 0u)) {
        // the next unchecked one of the lane: h = 0's first
        const bool f0 = m0 != 0u, f1 = !f0 && m10 != 0u;
        const unsigned m = f0 ? m0 : (f1 ? m10 : m11);
        const int k = (__ffs(m) - 1) & 31;
        const int2 f = pos[k + ((f0 || f1) ? 0 : 32)];
        const int a = f0 ? q0.x : q1.x, b = f0 ? q0.y : q1.y;
        const bool close = near_pos(f.x, a, stride) || near_pos(f.x, b, stride) || near_pos(f.y, a, stride) ||
                           near_pos(f.y, b, stride);
        const unsigned bit = m & (0u - m), drop = close ? 0u : bit;
        m0 &= f0 ? ~bit : ~0u;
        e0 &= f0 ? ~drop : ~0u;
        m10 &= f1 ? ~bit : ~0u;
        e10 &= f1 ? ~drop : ~0u;
        m11 &= (f0 || f1) ? ~0u : ~bit;
        e11 &= (f0 || f1) ? ~0u : ~drop;
      }
    }
    int level[2] = {0, 0}, levels = 1;
    unsigned done0 = __ballot_sync(0xffffffffu, e0 == 0u), done1 = __ballot_sync(0xffffffffu, (e10 | e11) == 0u);
    for (; (done0 & done1) != 0xffffffffu; ++levels) {
      const bool now0 = !((done0 >> lane) & 1u) && (e0 & ~done0) == 0u;
      const bool now1 = !((done1 >> lane) & 1u) && ((e10 & ~done0) | (e11 & ~done1)) == 0u;
      level[0] = now0 ? levels : level[0];
      level[1] = now1 ? levels : level[1];
      done0 |= __ballot_sync(0xffffffffu, now0);
      done1 |= __ballot_sync(0xffffffffu, now1);
    }
    __syncwarp();

    // the slot is free once the evaluators hold the window kProducers back
    if (w >= kProducers) bar_sync(kBarEmpty + slot, kEmptyThreads);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      // the acceptance bounds
      float lo = 0.0f, hi = 0.0f, t = 0.0f;
      if (!greedy_only) {
        t = temps[__popc(live[h] & below) + (h ? __popc(live[0]) : 0)];
        // T in [+0, 1e30], compared as bits (minus zero accepts everything).  Below
        // 1e-30 the bounds are not exact to 1e-4 any more, but need not be: a delta that
        // is not zero is 2^-90 at least (the weights' last bits), far beyond them.
        const bool ok = u[h] > 0.0f && __float_as_uint(t) <= __float_as_uint(1e30f);
        const float theta = -t * __logf(u[h]), margin = 1e-4f * t;
        lo = ok ? fmaxf(theta - margin, 0.0f) : -inf;
        hi = ok ? theta + margin : inf;
      }
      const int dx = x2[h] - x1[h], dy = y2[h] - y1[h];
      const bool adjacent = (dx == 0 && (dy == 1 || dy == -1)) || (dy == 0 && (dx == 1 || dx == -1));
      const uint32_t dir12 = dy == -1 ? 0u : (dy == 1 ? 1u : (dx == -1 ? 2u : 3u));
      uint32_t flags = (y1[h] > 0 ? 1u : 0u) | (y1[h] < gh - 1 ? 2u : 0u) | (x1[h] > 0 ? 4u : 0u) |
                       (x1[h] < gw - 1 ? 8u : 0u) | (y2[h] > 0 ? 16u : 0u) | (y2[h] < gh - 1 ? 32u : 0u) |
                       (x2[h] > 0 ? 64u : 0u) | (x2[h] < gw - 1 ? 128u : 0u);
      flags = adjacent ? (flags & ~((1u << dir12) | (16u << (dir12 ^ 1u)))) | 0x100u | (dir12 << 9) : flags;
      flags |= (skip[h] ? 0u : 0x800u) | ((uint32_t)level[h] << 16);
      int4* d = reinterpret_cast<int4*>(&S.ring[slot][32 * h + lane]);
      d[0] = make_int4(c1[h], c2[h], (int)flags, __float_as_int(lo));
      d[1] = make_int4(__float_as_int(hi), __float_as_int(u[h]), __float_as_int(t), levels);
    }
    __syncwarp();
    bar_arrive(kBarFull + slot, kFullThreads);
  }
}

// The evaluators: the group of four lanes g of warp v takes proposal 8 v + g of
// a window, lane `dir` the neighbour of each position in one direction (up,
// down, left, right).
template <bool kLabSmem, bool kGreedy>
__device__ __forceinline__ void evaluate_windows(const float4* __restrict__ pal, int p, const AnnealJob& J,
                                                 long long windows, ChainShared& S, const float4* s_lab,
                                                 uint16_t* s_grid) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gw = J.gw, n = gw * J.gh;
  const int grp = lane >> 2, dir = lane & 3;
  const int q = warp * 8 + grp;
  const int step = dir == 0 ? -gw : (dir == 1 ? gw : (dir == 2 ? -1 : 1));
  float* put = &S.terms[warp][lane];
  // even lanes sum the old weights, odd lanes the new ones
  const float* get = &S.terms[warp][(dir & 1) * 2 * kTermStride + grp * 4];
  const uint32_t last = (uint32_t)max(p - 1, 0);
  auto lab = [&](uint16_t g) -> float4 {  // a colour of the palette for an empty cell, too
    const uint32_t i = min((uint32_t)g, last);
    return kLabSmem ? s_lab[i] : __ldg(pal + i);
  };
  // A window's descriptor, read while the window before it waits for its cells.
  struct Desc {
    int p1, p2, n1, n2, level, levels;
    uint32_t flags;
    float lo, hi, u, t;
  };
  int slot = 0;
  auto take = [&](long long w) -> Desc {
    bar_sync(kBarFull + slot, kFullThreads);
    const int4 d = *reinterpret_cast<const int4*>(&S.ring[slot][q]);
    const int4 e = *(reinterpret_cast<const int4*>(&S.ring[slot][q]) + 1);
    Desc D;
    D.p1 = d.x;
    D.p2 = d.y;
    D.flags = (uint32_t)d.z;
    D.lo = __int_as_float(d.w);
    D.hi = __int_as_float(e.x);
    D.u = __int_as_float(e.y);
    D.t = __int_as_float(e.z);
    D.levels = e.w;
    D.level = (D.flags & 0x800u) ? (int)((D.flags >> 16) & 63u) : -1;
    const bool mutual = (D.flags & 0x100u) != 0u && dir == (int)((D.flags >> 9) & 3u);
    // cell n of the grid is an empty one for the neighbours outside it
    D.n1 = (((D.flags >> dir) & 1u) || mutual) ? D.p1 + step : n;
    D.n2 = ((D.flags >> (4 + dir)) & 1u) ? D.p2 + step : n;
    if (w + kProducers < windows) bar_arrive(kBarEmpty + slot, kEmptyThreads);
    slot = slot + 1 == kProducers ? 0 : slot + 1;
    return D;
  };
  // Proposal D, whose cells hold g1 and g2, this lane's neighbours a1 and a2:
  // its outcome where `act`, its swap where `swap`.  Whether it is accepted.
  auto decide = [&](const Desc& D, uint16_t g1, uint16_t g2, uint16_t a1, uint16_t a2, Outcome& O, bool act,
                    bool swap) -> bool {
    const float4 l1 = lab(g1), l2 = lab(g2), c1 = lab(a1), c2 = lab(a2);
    const float2 u1 = weight_of_sq2(sq_dist(l1.x, l1.y, l1.z, c1.x, c1.y, c1.z),
                                    sq_dist(l2.x, l2.y, l2.z, c1.x, c1.y, c1.z));
    const float2 u2 = weight_of_sq2(sq_dist(l1.x, l1.y, l1.z, c2.x, c2.y, c2.z),
                                    sq_dist(l2.x, l2.y, l2.z, c2.x, c2.y, c2.z));
    const bool use1 = ((D.flags >> dir) & 1u) && a1 != kNone16, use2 = a2 != kNone16;
    put[0] = use1 ? u1.x : 0.0f;
    put[kTermStride] = use2 ? u2.y : 0.0f;
    put[2 * kTermStride] = use1 ? u1.y : 0.0f;
    put[3 * kTermStride] = use2 ? u2.x : 0.0f;
    __syncwarp();
    // the reference's order of summation
    const float4 s0 = *reinterpret_cast<const float4*>(get), s1 = *reinterpret_cast<const float4*>(get + kTermStride);
    float cost = __fadd_rn(__fadd_rn(s0.x, s0.y), s0.z);  // weights are >= 0: 0 + s0.x is s0.x
    cost = __fadd_rn(__fadd_rn(cost, s0.w), s1.x);
    cost = __fadd_rn(__fadd_rn(cost, s1.y), s1.z);
    cost = __fadd_rn(cost, s1.w);
    if (__any_sync(0xffffffffu, (D.flags & 0x100u) != 0u)) {  // the mutual weight, last on both sides
      const float m = __shfl_sync(0xffffffffu, u1.x, (grp << 2) + (int)((D.flags >> 9) & 3u));
      if (D.flags & 0x100u) cost = __fadd_rn(cost, m);
    }
    const float other = __shfl_xor_sync(0xffffffffu, cost, 1);
    bool accept = false;
    if (dir == 0 && act) {
      const float delta = g1 == g2 ? 0.0f : __fsub_rn(other, cost);
      accept = delta < D.lo;
      if (!accept && !(delta > D.hi))
        accept = delta < 0.0f || (!kGreedy && D.u < exp_spec(__fdiv_rn(-delta, D.t)));
      if (accept && swap) {
        s_grid[D.p1] = g2;
        s_grid[D.p2] = g1;
      }
      O.delta[q] = accept ? delta : 0.0f;
      O.flags[q] = accept ? 3u : 2u;
    }
    __syncwarp();  // the terms are read before the next level writes them
    return accept;
  };
  Desc next{};
  if (windows > 0) next = take(0);
  int o = 0;  // the window's outcome slot
  int turn = 0;
  for (long long w = 0; w < windows; ++w) {
    const Desc D = next;
    Outcome& O = S.out[o];
    o = o == 2 ? 0 : o + 1;
    {
      const uint16_t g1 = s_grid[D.p1], g2 = s_grid[D.p2], a1 = s_grid[D.n1], a2 = s_grid[D.n2];
      if (w + 1 < windows) next = take(w + 1);
      const bool act = kGreedy ? D.level >= 0 : D.level == 0;
      bool accept = false;
      if (__any_sync(0xffffffffu, act)) accept = decide(D, g1, g2, a1, a2, O, act, !kGreedy);
      if (D.level < 0 && dir == 0) {
        O.delta[q] = 0.0f;
        O.flags[q] = 0u;
      }
      // Greedy descent ends in windows that accept nothing, and then what every
      // level finds on the grid as it is stands: one pass.  Else that holds up to
      // the lowest level that accepts; its swaps are made and the levels above it
      // are looked at again, all at once.  (With a temperature, where windows
      // accept at most levels, one level after the other is faster: 1.53 against 1.70 ms
      // for 100 000 on 179 x 134.)  5000 iterations on 8 x 6 cells, 8 chains, a whole
      // call: 562 -> 240 us (471 in rounds of 16 proposals).
      if (kGreedy) {
        for (;;) {
          const int lowest = __reduce_min_sync(0xffffffffu, accept ? D.level : kWindow);
          if (lane == 0 && lowest < kWindow) atomicMin(&S.first[turn], lowest);
          if (!bar_any(kBarEval, kEval, accept)) break;
          const int done = S.first[turn];
          if (accept && D.level == done) {
            const uint16_t t = s_grid[D.p1];  // (no other swap of the level touches these)
            s_grid[D.p1] = s_grid[D.p2];
            s_grid[D.p2] = t;
          }
          turn ^= 1;
          if (tid == 0) S.first[turn] = kWindow;
          bar_sync(kBarEval, kEval);  // the level's swaps are in place
          if (done + 1 >= D.levels) break;
          accept = false;
          if (__any_sync(0xffffffffu, D.level > done))
            accept = decide(D, s_grid[D.p1], s_grid[D.p2], s_grid[D.n1], s_grid[D.n2], O, D.level > done, false);
        }
        continue;
      }
    }
    for (int l = 1; l < D.levels; ++l) {
      bar_sync(kBarEval, kEval);
      if (__any_sync(0xffffffffu, D.level == l))
        decide(D, s_grid[D.p1], s_grid[D.p2], s_grid[D.n1], s_grid[D.n2], O, D.level == l, true);
    }
    __syncwarp();
    bar_sync(kBarEval, kEval);  // the window's swaps are in place
  }
}

// One chain by one CTA of kThreads threads.  smem: anneal_cta_smem_bytes bytes, 16-byte
// aligned; writer_slots a power of two.
template <bool kLabSmem>
__device__ __forceinline__ void anneal_chain_cta(const float4* __restrict__ pal, int p, const AnnealJob& J, int chain,
                                                 int writer_slots, uint8_t* smem) {
  // the warp index through a shuffle: the compiler then knows each warp's path as converged
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int gw = J.gw, gh = J.gh, n = gw * gh;
  ChainShared& S = *reinterpret_cast<ChainShared*>(smem);
  uint32_t* writers = reinterpret_cast<uint32_t*>(smem + sizeof(ChainShared));
  float4* s_lab = reinterpret_cast<float4*>(writers + kProducers * 2 * writer_slots);
  uint16_t* s_grid = reinterpret_cast<uint16_t*>(s_lab + (kLabSmem ? p : 0));
  if (kLabSmem)
    for (int i = tid; i < p; i += kThreads) s_lab[i] = pal[i];
  for (int i = tid; i <= n; i += kThreads) {
    const int g = i < n ? __ldcg(J.grid_in + i) : -1;
    s_grid[i] = g < 0 ? kNone16 : (uint16_t)g;
  }
  for (int i = tid; i < kProducers * 2 * writer_slots; i += kThreads) writers[i] = 0u;
  if (tid < 2) S.first[tid] = kWindow;
  __syncthreads();
  const long long windows = (J.iters + kWindow - 1) / kWindow;

  if (warp < kEvalWarps) {
    if (J.greedy_only) evaluate_windows<kLabSmem, true>(pal, p, J, windows, S, s_lab, s_grid);
    else evaluate_windows<kLabSmem, false>(pal, p, J, windows, S, s_lab, s_grid);
    __syncthreads();
  } else if (warp < kEvalWarps + kProducers) {
    produce_windows(J, chain, windows, warp - kEvalWarps, S, writers, writer_slots, s_grid);
    __syncthreads();
  } else {
    // ---- the book keeper.  Initial cost: calculate_total_cost of the start
    // grid (sequential FP32 sum), read from global memory as the evaluators may
    // be swapping already.
    float current;
    if (J.initial_cost) {
      current = __ldcg(J.initial_cost);
    } else {
      // 32 cells at a time, their cells read two steps ahead of the sum and their
      // Lab one (216 x 160 cells, 36 iterations, a whole call: 1104 -> 800 us).
      auto lab = [&](int i) -> float4 { return kLabSmem ? s_lab[i] : __ldg(pal + i); };
      struct Cells {
        int cur, right, down;
      };
      auto cells = [&](int c0) -> Cells {
        const int c = c0 + lane, x = c % gw, y = c / gw;
        Cells v{-1, -1, -1};
        if (c < n) {
          v.cur = __ldcg(J.grid_in + c);
          if (x < gw - 1) v.right = __ldcg(J.grid_in + c + 1);
          if (y < gh - 1) v.down = __ldcg(J.grid_in + c + gw);
        }
        return v;
      };
      struct Labs {
        float4 cur, right, down;
        bool r, d;
      };
      auto labs = [&](const Cells& v) -> Labs {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        Labs l{zero, zero, zero, v.cur >= 0 && v.right >= 0, v.cur >= 0 && v.down >= 0};
        if (v.cur >= 0) l.cur = lab(v.cur);
        if (l.r) l.right = lab(v.right);
        if (l.d) l.down = lab(v.down);
        return l;
      };
      current = 0.0f;
      Labs now = labs(cells(0));
      Cells next = cells(32);
      for (int c0 = 0; c0 < n; c0 += 32) {
        const float tr = now.r ? wgt(now.cur, now.right) : 0.0f, td = now.d ? wgt(now.cur, now.down) : 0.0f;
        now = labs(next);
        next = cells(c0 + 64);
        const int cnt = min(32, n - c0);
        for (int s = 0; s < cnt; ++s) {
          current = __fadd_rn(current, __shfl_sync(0xffffffffu, tr, s));
          current = __fadd_rn(current, __shfl_sync(0xffffffffu, td, s));
        }
      }
    }
    const float initial = current;
    float best = current;
    long long accepted = 0, cooled = 0, improved = 0;
    // A proposal that was not accepted adds 0 and is no new best, so every
    // proposal is booked alike: one chain of additions, its partial sums to
    // shared memory; when one of them is a new best, each lane compares two of
    // them with the least before.
    auto book = [&](const Outcome& O) {
      float d[kWindow];
#pragma unroll
      for (int h = 0; h < kWindow; h += 4) *reinterpret_cast<float4*>(d + h) = *reinterpret_cast<const float4*>(O.delta + h);
#pragma unroll
      for (int h = 0; h < kWindow; ++h) {
        current = __fadd_rn(current, d[h]);
        d[h] = current;
      }
#pragma unroll
      for (int h = 0; h < kWindow; h += 4) *reinterpret_cast<float4*>(S.sums + h) = *reinterpret_cast<const float4*>(d + h);
      __syncwarp();
      float c[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t f = O.flags[32 * h + lane];
        accepted += __popc(__ballot_sync(0xffffffffu, (f & 1u) != 0u));
        cooled += __popc(__ballot_sync(0xffffffffu, (f & 2u) != 0u));
        c[h] = S.sums[32 * h + lane];
      }
      if (__any_sync(0xffffffffu, c[0] < best || c[1] < best)) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float least = c[h];  // of this lane's and the earlier ones
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float v = __shfl_up_sync(0xffffffffu, least, o);
            least = lane >= o ? fminf(least, v) : least;
          }
          float before = __shfl_up_sync(0xffffffffu, least, 1);
          before = lane == 0 ? best : fminf(best, before);
          improved += __popc(__ballot_sync(0xffffffffu, c[h] < before));
          best = fminf(best, __shfl_sync(0xffffffffu, least, 31));
        }
      }
      __syncwarp();
    };
    int slot = 0;
    for (long long w = 0; w < windows; ++w) {
      bar_sync(kBarFull + slot, kFullThreads);  // window w is prepared, the evaluators are in window w - 1
      if (w > 1) book(S.out[(w - 2) % 3]);
      slot = slot + 1 == kProducers ? 0 : slot + 1;
    }
    __syncthreads();
    if (windows > 1) book(S.out[(windows - 2) % 3]);
    if (windows > 0) book(S.out[(windows - 1) % 3]);
    if (lane == 0) {
      ChainResult r;
      r.initial_cost = initial;
      r.final_cost = current;
      r.best_cost = J.greedy_only ? current : best;
      r.pad = 0.0f;
      r.accepted = accepted;
      r.improved = J.greedy_only ? accepted : improved;
      r.cooled = cooled;
      r.pad2 = 0;
      J.results[chain] = r;
    }
  }
  int32_t* out = J.chain_grids + (size_t)chain * n;
  for (int i = tid; i < n; i += kThreads) {
    const uint16_t g = s_grid[i];
    out[i] = g == kNone16 ? -1 : (int32_t)g;
  }
}

}  // namespace anneal_detail
}  // namespace mg
