// k_greedy.cu -- (d) the standalone greedy placement kernels.
//
// Reference: main.rs:529-545 (row-major walk), main.rs:335-418
// find_and_use_best_tile_with_position, main.rs:420-475 fallback_tile_selection,
// main.rs:309-333 can_place_at_position, lib.rs:57-89 UsageTracker,
// adjacency.rs:63-88 calculate_penalty.  The decision rule and its exact
// shortcuts are described in greedy_walk.cuh.
//
// Two kernels:
//  - greedy_kernel: one warp walks one mosaic (greedy_walk.cuh).  Used for
//    palettes above 65535 materials, grids narrower than 8 cells and walks
//    whose three-CTA form does not fit in shared memory.
//  - greedy_pair_kernel: a cluster of three CTAs per mosaic.  The walk is a
//    chain of dependent decisions, so its speed is the latency of one decision.
//    One warp of CTA 0 (the walker) makes them; everything that does not depend
//    on the last few is prepared ahead of it, in two steps:
//    * 62 scout warps in CTAs 1 and 2, on other SMs, turn each cell's candidate
//      row into a record, kScoutLead cells ahead: the first 32 candidates (list
//      order) that differ from the cell above and were under the usage cap in a
//      snapshot of the counters (a copy that a follower warp keeps in each of
//      those CTAs), with distance, Lab and weight against the cell above; also
//      the first 32 candidates regardless of the counters, for use after a reset;
//    * kRefiners warps of CTA 0 turn each record into a list of eight entries,
//      kRefineLag cells ahead, from the counters themselves (see ListShared).
//    Counters only grow between resets, so a candidate that failed the cap in a
//    snapshot still fails it when the walker arrives: the walker's choice is the
//    list entry of lowest rank that passes the fresh counter and is not the left
//    neighbour's material -- one warp minimum -- whenever the list settles it,
//    bit for bit the reference's.  In every other case (nothing of the list
//    passes, something beyond it might win, a reset since the snapshot) the
//    walker decides from the record (window_cell) or evaluates the cell in full,
//    exactly as greedy_walk does.  A reset bumps an epoch that invalidates older
//    records and lists: the cells up to the first new list are decided in runs
//    from their records alone (record_cells), and so is a whole walk of cap 1
//    over few materials, whose lists hold nothing by the time they are used.  Where the 16-bit grid does not fit, the walker's shared
//    memory holds a ring of the last placed cells instead, so a mosaic of any
//    cell count walks in this form.  calculate_total_cost: by a warp of CTA 0
//    that follows the walk (with the ring: by CTA 1 after it), one sequential
//    FP32 sum in the reference's order.
//
//    What bounds it: the walker's loop, ~100 cycles a cell (the minimum 22, the
//    rotation, test and exclusion before it ~20, two branches ~40), and lists
//    that are not there in time: ~500 cycles from trigger to list, ~1 000 when
//    penalties decide.  Measured, GB300, before (records alone, no lists; 64
//    scouts that read the counters through distributed shared memory) -> now:
//    80 x 60 cells, 506 materials 0.551 -> 0.326 ms; 179 x 134, 5000 materials
//    3.49 -> 1.75; 61 x 43, 112 materials, cap 2 0.518 -> 0.255; 64 mosaics of
//    300 to 17 900 cells, 10 000 materials 4.6 -> 1.62; whole calls of 140 x 100
//    cells, resets every few cells: 5 materials, cap 1 4.77 -> 4.30, 30 materials,
//    cap 1 1.93 -> 1.77, 100 materials, cap 2 3.75 -> 1.28 (without the runs from
//    records 6.4, 3.9 and 1.9).  Measured and not kept:
//    blocks of 2 or 4 cells without branches (80 cycles a cell alone, but a list
//    that is late costs a whole block), lists made 10, 14 or 20 cells ahead (late;
//    or, with caps of 2, filled before they are used), 11 or 20 refiners (too
//    few; or in each other's way), refiners on the walker's scheduler, 124
//    scouts, counters gathered two rounds at once.
#include <cstddef>
#include <type_traits>

#include "greedy_walk.cuh"

namespace mg {
namespace {
using namespace greedy_detail;

template <bool kLabSmem, bool kUsageSmem>
__global__ void __launch_bounds__(32) greedy_kernel(const float4* __restrict__ pal, int p,
                                                    const GreedyJob* __restrict__ jobs, uint32_t* usage_global,
                                                    uint32_t* err) {
  extern __shared__ __align__(128) uint8_t smem[];
  const GreedyJob J = jobs[blockIdx.x];
  greedy_walk<kLabSmem, kUsageSmem>(pal, p, J, smem, usage_global ? usage_global + (size_t)blockIdx.x * p : nullptr,
                                    err);
}

// ---- the scouted walk -------------------------------------------------------------------
// A cluster of 1 + kScoutCtas CTAs per mosaic.  CTA 0 walks (warp 0; the
// state of the walk lives in its shared memory) with the refiners on its other
// schedulers; the other CTAs, on other SMs, hold the scouts and a follower each
// that copies the walk for them, so the walker's SM is read by one warp of each
// and written the records, through distributed shared memory.  (Four scout CTAs
// gained nothing over two.)
constexpr int kScoutCtas = 2;
constexpr int kThreads = 1024;      // per CTA
constexpr int kScoutWarpsMax = 32;  // warps of a scout CTA
constexpr uint32_t kInvalidEpoch = 0xFFFFFFFFu;
constexpr uint32_t kWalkPolls = 1u << 24;      // the walker's bounded wait for a record
constexpr uint32_t kInjectedWalkPolls = 1u << 12;  // ... when a timeout is injected (well under a millisecond)
constexpr uint32_t kScoutPolls = 1u << 24;  // polls of about 0.3 us each
// Records are built at most kScoutLead cells ahead of the walker: far enough
// that they are there in time, and no further, as every placement made since a
// snapshot may have filled one of its entries.
constexpr int kScoutLead = 80;
// With caps of 1 and 2 they are: a palette of few materials is used up, and the
// counters reset, within a few rows.  Records are then built less far ahead
// (140 x 100 cells, cap 1, weight 0.25, against 80 cells ahead: 50 materials
// 3.81 -> 2.07 ms, 100 materials 4.56 -> 2.03, 200 materials 2.67 -> 1.74; cap 2,
// 50 materials 2.11 -> 1.46, 100 materials 1.93 -> 1.40; caps of 4 and more lose
// a tenth; at a quarter of a palette above 320 the distance is 80 again).
__host__ __device__ inline int scout_ahead(int gw, int p, uint32_t max_usage) {
  int a = kScoutLead;
  if (max_usage == 1u) a = p / 4 > 32 ? p / 4 : 32;
  if (max_usage == 2u) a = 5 * (p / 8) > 48 ? 5 * (p / 8) : 48;
  if (a > kScoutLead) a = kScoutLead;
  return a < gw ? a : gw;
}
// Lists of a cap-1 palette below this many materials would go unused: the cells
// placed since a list was made have what it held (200 materials, cap 1: 2.68 ms
// with them, 1.62 without; 1000 materials: 1.29 and 1.60).  Such a walk makes none
// and goes by the records alone.
constexpr int kCapOneLists = 512;
__device__ __forceinline__ bool walks_by_lists(int p, uint32_t max_usage) {
  return max_usage > 1u || p >= kCapOneLists;
}
constexpr uint32_t kRefinePolls = 1u << 26;  // the refiners' bounded waits (seconds)
constexpr int kCostChunk = 2048;  // cells per pass of the final cost sum
constexpr uint32_t kFollowPolls = 1u << 26;  // the cost warp's bounded wait for a placement (seconds)
enum Ctrl { kProgress = 0, kEpoch = 1, kAbort = 2 };

// A cell's prepared decision: two candidate lists of up to 32 entries in list
// (= ascending distance) order, entry i for walker lane i, both without the
// cell above:
//  f: the candidates under the usage cap in the scout's snapshot (valid while
//     the epoch is unchanged);
//  r: all candidates (valid in any epoch, used after a reset).
// Entry i is the key (i << 17 | blocked << 16 | palette index), ~0 where the
// list is shorter, so the lowest key among eligible entries is the first
// eligible one.  `blocked` is clear when no later entry of the list (nor
// anything beyond it) lies inside the 2*weight window of entry i -- then, if
// entry i is the first eligible one, the penalty cannot change the decision.
// Palette indices are 16-bit (palettes of at most 65535).
// The record also carries, for each f entry, its distance, its weight against
// the cell above (0 in the first row) and its Lab, and `f_next`, the distance
// of the first entry after the list (+inf when the list holds every entry
// under the cap): the walker then settles a cell whose penalty window holds
// several entries from shared memory (window_cell).
struct __align__(16) CellRecord {
  uint32_t kf[32];
  uint32_t kr[32];
  uint32_t epoch;
  float f_next;
  uint32_t pad[2];
  float wd[32];
  float wu[32];
  float4 wl[32];
};
// A scout's working copy of one record (in its own CTA).
struct ScoutStage {
  uint32_t kf[32], kr[32];
  float df[32], dr[32];
};

// Records live in a ring of R slots.  A scout writes cell c's record once the
// walker has placed cell c - ahead, and that is when the slot's last one, of cell
// c - R, must have no reader any more.  The walker is past it and reads two ahead
// of its cell at most.  A refiner may be later than the walker, which goes kTurn
// cells past one whose list it has not seen, at most: R >= ahead + kTurn.  Where a
// ring of that size does not fit, ahead is shorter (rows of 28 cells, a ring of 32
// for 64: 0.45 -> 0.60 ms a call of 2800 cells, 30 materials, cap 2).
constexpr int kLists = 16;         // ring of the prepared lists (below)
constexpr int kTurn = kLists - 2;  // (fast_cells reads the list two cells on)
__host__ __device__ inline int ring_size(int gw, bool roomy) {
  const int lead = gw < kScoutLead ? gw : kScoutLead;
  int r = 32;
  while (r < lead + (roomy ? kTurn : 4)) r <<= 1;
  return r;
}

// The placed cells live in the walker CTA's shared memory in one of two forms:
//  - the grid, 16-bit, kUnplaced until placed (copied to global memory after
//    the walk);
//  - when the grid does not fit: a ring of words (cell index & 0xFFFF) << 16 |
//    material, one 32-bit store publishing a placement and naming its cell.
//    The walker reads the cell above its own; a scout reads its lead cell and
//    the cell above its cell.  The walker never passes a cell whose record is
//    missing, so no cell read is more than gw + kScoutLead + 64 behind the
//    newest placement, and a ring of more slots than that keeps every cell
//    until it is read.  The global grid receives each placement as it is made.
constexpr uint16_t kUnplaced = 0xFFFFu;
constexpr uint32_t kNoCell = 0xFFFFFFFFu;  // a ring slot no placement has written yet
__host__ __device__ inline int cell_ring_size(int gw) {
  int r = 64;
  while (r < gw + kScoutLead + 72) r <<= 1;
  return r;
}
__device__ __forceinline__ uint32_t cell_word(int c, int t) { return ((uint32_t)c << 16) | ((uint32_t)t & 0xFFFFu); }

// The prepared lists.  Beside the walker (warp 0), refiner warps of its CTA --
// none on the walker's scheduler -- turn each cell's record into what the
// decision needs last, kRefineLag cells ahead of the walker: the first kList
// entries under the usage cap *now* (a record's snapshot is up to kScoutLead
// placements old).  A list is written in list (= distance) order first, each
// entry with whether the next one lies outside its 2*weight window: then, if it
// is the first that may be taken, the penalty cannot change the decision.  When
// every entry is clear like that, the list is done.  Else a second form follows,
// ~500 cycles later: each entry's rank by score (then position), given each
// entry of the previous cell's list as the left neighbour -- the one part of a
// score not known before.  (When one of the first kEarly entries is not clear,
// the second form is the only one.)
// An entry of a list is one 64-bit word:
//   low:  eight 4-bit ranks, rotated so that a left rotation by 4 j + 2 brings
//         the one for previous entry j to the top (first form: the position):
//         15 when the entry is absent, 14 when its score exceeds the distance
//         of the first entry after the list (something beyond it might win);
//   high: epoch (its low bits, list_tag) << 28 | position << 25 | clear << 24 | parity of the
//         cell's turn of the ring << 23 | 1 << 16 | material (p when absent).
// With j known from the previous decision the walker's choice is one warp
// minimum over (rank, position, counter, material) of the entries still under
// the cap and not the left neighbour's material: entries after a list have
// distances, and so scores, of at least the first one's distance, so an entry
// of score up to that is the reference's choice (ties go to the lower position).
constexpr int kList = 8;
constexpr int kRefiners = 17;   // warps 2, 3, 5, 6, 7, 9, ... of the walker's CTA
constexpr int kRefineLag = 12;
constexpr int kEarly = 3;       // entries that must be clear for the first form (2 to 8 differ by 3%)
constexpr uint32_t kRankOpen = 14, kClear = 1u << 24;
constexpr uint32_t kNotThere = 0xFFFFu;  // the packed word of an entry whose list is not there
constexpr int kResetLog = 128;  // more resets than cells between the walker and its followers
// The tag bits of a list tell cell c's from the one a turn of the ring before (cell
// c - kLists), not from older ones: a reader of cell c's slot knows that the list of
// c - kLists has been there (the walker's `behind`).  Between a list's making and
// its use lie fewer than 32 cells, so fewer than 32 resets.
constexpr uint32_t kTagMask = 0xF0820000u, kTagCell = 0x00800000u;
__device__ __forceinline__ uint32_t list_tag(int c, uint32_t epoch) {
  return (epoch << 28) | ((epoch & 16u) << 13) | (((uint32_t)c & kLists) ? kTagCell : 0u);
}
static_assert((kLists & (kLists - 1)) == 0 && kLists <= 32 && kRefineLag + 4 <= kLists, "the list ring");
struct __align__(16) ListShared {
  unsigned long long ent[kLists][kList];  // first form
  unsigned long long fin[kLists][kList];  // second form
  unsigned long long spare[2];      // written where an entry has no place
  uint32_t done[kLists];         // cell + 1 once all of its lists are written
  float4 sel[kLists][kList + 1];    // Lab, material bits (the last one: what the list does not take)
  uint32_t seq[kLists];             // cell + 1 once sel is complete
  float2 dw[kRefiners][kList + 1];  // distance, weight against the cell above
  unsigned long long reset_at[kResetLog];  // epoch e << 32 | the cell that began it, at e % kResetLog
};
static_assert(sizeof(ListShared) % 16 == 0, "16-byte aligned parts");

// Shared memory of the walker CTA: control words, lists, record ring, sequence
// words, the placed cells (grid or ring), usage counters (and one more, full, for
// absent entries), optionally the palette Lab.
__host__ __device__ inline size_t cells_bytes(int gw, int n, bool ring) {
  return ring ? (size_t)cell_ring_size(gw) * 4 : align16((size_t)n * 2);
}
__host__ __device__ inline size_t walker_smem_bytes(int gw, int n, int p, bool lab_smem, bool ring, bool roomy) {
  const int R = ring_size(gw, roomy);
  size_t b = 16 + sizeof(ListShared) + (size_t)R * sizeof(CellRecord) + (size_t)R * 4;
  b += cells_bytes(gw, n, ring);
  b += align16(((size_t)p + 1) * 4);
  if (lab_smem) b += (size_t)p * 16;
  return b;
}
// Shared memory of a scout CTA: staging per warp, the cost terms, and its copy
// of the walk (follow_walk): control words, counters, the last placed cells.
struct ScoutLayout {
  ScoutStage* stage;
  float* terms;
  uint32_t* ctl;  // Follow
  uint32_t* usage;
  uint16_t* cells;  // ring of cell_ring_size(gw)
};
enum Follow { kFollowed = 0, kFollowEpoch = 1, kFollowAbort = 2 };
__device__ inline ScoutLayout scout_layout(uint8_t* smem, int p) {
  ScoutLayout S;
  S.stage = reinterpret_cast<ScoutStage*>(smem);
  S.terms = reinterpret_cast<float*>(S.stage + kScoutWarpsMax);
  S.ctl = reinterpret_cast<uint32_t*>(S.terms + 2 * kCostChunk);
  S.usage = S.ctl + 4;
  S.cells = reinterpret_cast<uint16_t*>(reinterpret_cast<uint8_t*>(S.usage) + align16((size_t)p * 4));
  return S;
}
__host__ __device__ inline size_t scout_cta_smem_bytes(int gw, int p) {
  return (size_t)kScoutWarpsMax * sizeof(ScoutStage) + (size_t)kCostChunk * 8 + 16 + align16((size_t)p * 4) +
         (size_t)cell_ring_size(gw) * 2;
}
__host__ __device__ inline size_t pair_smem_bytes(int gw, int n, int p, bool lab_smem, bool ring, bool roomy = false) {
  const size_t a = walker_smem_bytes(gw, n, p, lab_smem, ring, roomy), b = scout_cta_smem_bytes(gw, p);
  return a > b ? a : b;
}

// The exact decision for one cell (greedy_walk's per-cell rule, candidate rows
// read from global memory).  Updates the counters; a fallback resets them and
// bumps the epoch.  Returns the chosen palette index.
// The whole candidate row (k <= 100: four entries per lane) and the neighbours'
// Lab are read at once, then the Lab of the candidates inside the penalty
// window: two dependent memory round trips whatever the depth of the first
// eligible entry (reading on until one is eligible: 5.1 ms against 4.1 for
// 140 x 100 cells, 100 materials, cap 1).
template <class LabFn>
__device__ int full_cell(LabFn lab, const uint32_t* __restrict__ ci, const float* __restrict__ cd, int k, int p,
                         int up, int left, uint32_t* usage, uint32_t max_usage, float weight, uint32_t* ctrl,
                         uint32_t& epoch, int& resets, int lane, unsigned long long* reset_at, int c) {
  constexpr int kRounds = 4;  // ceil(100 / 32)
  const bool use_pen = weight > 0.0f;
  const float two_w = __fmul_rn(2.0f, weight);
  const float kInf = __int_as_float(0x7f800000);
  uint32_t tr[kRounds];
  float dr[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const int j = r * 32 + lane;
    tr[r] = j < k ? __ldg(ci + j) : kNoCand;
    dr[r] = j < k ? __ldg(cd + j) : kInf;
  }
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 lab_up = use_pen && up >= 0 ? lab(up) : zero;
  const float4 lab_left = use_pen && left >= 0 ? lab(left) : zero;
  auto okf = [&](uint32_t t) { return t < (uint32_t)p && (int)t != up && (int)t != left && usage[t] < max_usage; };
  int r0 = -1;
  unsigned m = 0;
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const unsigned mr = __ballot_sync(0xffffffffu, okf(tr[r]));
    if (r0 < 0 && mr) {
      r0 = r;
      m = mr;
    }
  }
  int t;
  if (r0 >= 0) {
    const int e0l = __ffs(m) - 1;
    int win = r0 * 32 + e0l;
    uint32_t t_win = 0;
#pragma unroll
    for (int r = 0; r < kRounds; ++r)
      if (r == r0) t_win = __shfl_sync(0xffffffffu, tr[r], e0l);
    if (use_pen) {
      float d0 = 0.0f;
#pragma unroll
      for (int r = 0; r < kRounds; ++r)
        if (r == r0) d0 = __shfl_sync(0xffffffffu, dr[r], e0l);
      const float b0 = __fadd_rn(d0, two_w);
      // another eligible entry after e0 inside [d0, d0 + 2w): penalties decide
      bool any_in = false;
#pragma unroll
      for (int r = 0; r < kRounds; ++r) any_in |= r * 32 + lane > win && dr[r] < b0 && okf(tr[r]);
      if (__any_sync(0xffffffffu, any_in)) {
        float4 lt[kRounds];
        bool in[kRounds];
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
          in[r] = r * 32 + lane >= win && dr[r] < b0 && okf(tr[r]);
          lt[r] = in[r] ? lab((int)tr[r]) : zero;
        }
        uint32_t best_s = 0xFFFFFFFFu;
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
          uint32_t sb = 0xFFFFFFFFu;
          if (in[r]) {
            float pen = 0.0f;
            if (up >= 0) pen = __fadd_rn(pen, wgt(lt[r], lab_up));
            if (left >= 0) pen = __fadd_rn(pen, wgt(lt[r], lab_left));
            sb = __float_as_uint(__fadd_rn(dr[r], __fmul_rn(pen, weight)));
          }
          const uint32_t mn = __reduce_min_sync(0xffffffffu, sb);
          if (mn < best_s) {  // strict: the earliest entry keeps a tie
            best_s = mn;
            const int l = __ffs(__ballot_sync(0xffffffffu, sb == mn)) - 1;
            win = r * 32 + l;
            t_win = __shfl_sync(0xffffffffu, tr[r], l);
          }
        }
      }
    }
    t = (int)t_win;
    __syncwarp();
    if (lane == 0) usage[t] += 1u;
  } else {
    // main.rs:420-475: global reset, first candidate passing can_place, else nearest.
    ++resets;
    __syncwarp();
    for (int i = lane; i < p; i += 32) usage[i] = 0;
    t = -1;
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int tj = (int)tr[r];
      const unsigned mask = __ballot_sync(0xffffffffu, tr[r] != kNoCand && tj >= 0 && tj < p && tj != up && tj != left);
      if (t < 0 && mask) t = __shfl_sync(0xffffffffu, tj, __ffs(mask) - 1);
    }
    if (t < 0) t = (int)__shfl_sync(0xffffffffu, tr[0], 0);
    __syncwarp();  // with the release: the zeroed counters are seen no later than the epoch
    ++epoch;
    if (lane == 0) {
      usage[t] = 1u;
      // one word for the followers, which need no order with anything else; the
      // epoch for the refiners of this CTA, after the zeroed counters
      *reinterpret_cast<volatile unsigned long long*>(&reset_at[epoch % kResetLog]) =
          (unsigned long long)epoch << 32 | (uint32_t)c;
      st_release_cta(&ctrl[kEpoch], epoch);
    }
  }
  return t;
}

// The walker CTA's shared-memory layout (both CTAs compute it; the scouts map
// it into the walker CTA's window).
struct WalkerLayout {
  uint32_t* ctrl;
  ListShared* lists;
  CellRecord* rec;
  uint32_t* seq;
  uint32_t* ring;    // the placed cells as a ring (kRing) ...
  uint16_t* grid16;  // ... or as the 16-bit grid; the same address
  uint32_t* usage;
  float4* lab;
};
__device__ inline WalkerLayout walker_layout(uint8_t* smem, int gw, int n, int p, int R, bool ring) {
  WalkerLayout L;
  L.ctrl = reinterpret_cast<uint32_t*>(smem);
  L.lists = reinterpret_cast<ListShared*>(smem + 16);
  L.rec = reinterpret_cast<CellRecord*>(L.lists + 1);
  L.seq = reinterpret_cast<uint32_t*>(L.rec + R);
  L.ring = L.seq + R;
  L.grid16 = reinterpret_cast<uint16_t*>(L.ring);
  L.usage = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(L.ring) + cells_bytes(gw, n, ring));
  L.lab = reinterpret_cast<float4*>(reinterpret_cast<uint8_t*>(L.usage) + align16(((size_t)p + 1) * 4));
  return L;
}

// The follower warp of a scout CTA keeps a copy of the walk in that CTA's shared
// memory: the cells placed so far, the counters, the epoch.  The scouts then
// read nothing from the walker's SM -- gathering up to a hundred counters there
// for every cell kept its shared memory busier than the walk did, and a scout
// 5 us a cell (64 scouts: 175 cycles a cell).  The copy lags; counters that lag
// only list entries that are full by now, and an epoch that lags only makes the
// record one of the earlier epoch.
template <bool kRing>
__device__ void follow_walk(const GreedyJob& J, int p, uint8_t* smem, int R, uint32_t* err) {
  const int lane = threadIdx.x & 31;
  const int gw = J.gw, n = gw * J.gh;
  const WalkerLayout L = walker_layout(smem, gw, n, p, R, kRing);
  const ScoutLayout S = scout_layout(smem, p);
  const uint32_t r_abort = cluster_map(&L.ctrl[kAbort], 0);
  const uint32_t r_cells = cluster_map(L.ring, 0), r_log = cluster_map(L.lists->reset_at, 0);
  const int cmask = cell_ring_size(gw) - 1;
  uint32_t mine = 0, polls = 0;
  for (int pos = 0; pos < n;) {
    const int cc = pos + lane;
    uint32_t v = 0;
    bool placed = false;
    if (cc < n) {
      v = kRing ? ld_cluster_u32(r_cells + 4u * (uint32_t)(cc & cmask)) : ld_cluster_u16(r_cells + 2u * (uint32_t)cc);
      placed = kRing ? (v >> 16) == ((uint32_t)cc & 0xFFFFu) : v != kUnplaced;
      v &= 0xFFFFu;
    }
    const unsigned missing = __ballot_sync(0xffffffffu, !placed);
    const int run = missing ? __ffs(missing) - 1 : 32;
    if (run == 0) {
      const bool out = ++polls > kScoutPolls;
      if (__any_sync(0xffffffffu, out || ld_cluster_u32(r_abort) != 0u)) {
        if (lane == 0) {
          if (out) {
            atomicOr(err, kErrTimeout);
            st_cluster_u32(r_abort, 1u);
          }
          *reinterpret_cast<volatile uint32_t*>(&S.ctl[kFollowAbort]) = 1u;
        }
        return;
      }
      __nanosleep(100);
      continue;
    }
    polls = 0;
    int from = 0;  // the run's cells before it are counted
    for (;;) {
      const unsigned long long log =
          __shfl_sync(0xffffffffu, ld_cluster_u64(r_log + 8u * ((mine + 1u) % kResetLog)), 0);
      if ((uint32_t)(log >> 32) != mine + 1u) break;
      const int at = (int)(uint32_t)log;
      if (at >= pos + run) break;  // not there yet
      if (lane == 0) st_release_cta(&S.ctl[kFollowEpoch], kInvalidEpoch);
      __threadfence_block();
      __syncwarp();
      for (int i = lane; i < p; i += 32) S.usage[i] = 0;
      __syncwarp();
      // (a reset seen late: the cells counted since it)
      for (int i = at + lane; i < pos; i += 32) atomicAdd(&S.usage[S.cells[i & cmask]], 1u);
      from = max(from, at - pos);
      __threadfence_block();
      __syncwarp();
      ++mine;
      if (lane == 0) st_release_cta(&S.ctl[kFollowEpoch], mine);
      __syncwarp();
    }
    if (lane >= from && lane < run) atomicAdd(&S.usage[v], 1u);
    if (lane < run) S.cells[cc & cmask] = (uint16_t)v;
    __syncwarp();
    pos += run;
    if (lane == 0) st_release_cta(&S.ctl[kFollowed], (uint32_t)pos);
    __syncwarp();
  }
}

// A scout warp: prepares the records of cells s, s + kScouts, s + 2 kScouts, ...
// Returns false when the walk was aborted.
// (The layout is recomputed here rather than passed by reference: a struct
// whose address escapes would turn the walker's shared-memory pointers into
// generic ones.)
// inject.timeout: build the records but never publish them (the walker's wait for
// the first record then runs out); inject.scout_ns: publish each that much later.
template <bool kRing, int kScouts>
__device__ bool scout_cells(int s, const GreedyJob& J, const float4* __restrict__ pal, int p, uint8_t* smem,
                            ScoutStage& S, int R, uint32_t* err, const WalkInject& inject) {
  const int lane = threadIdx.x & 31;
  const int gw = J.gw, k = J.k, n = gw * J.gh;
  const WalkerLayout L = walker_layout(smem, gw, n, p, R, kRing);
  const ScoutLayout F = scout_layout(smem, p);
  const uint32_t max_usage = J.max_usage;
  const bool use_pen = J.weight > 0.0f;
  const float two_w = __fmul_rn(2.0f, J.weight);
  const int ahead = min(scout_ahead(gw, p, max_usage), R - kTurn);
  const int nr = (k + 31) >> 5;
  const float inf = __int_as_float(0x7f800000);
  const unsigned lt = (1u << lane) - 1u;
  const int cmask = cell_ring_size(gw) - 1;
  // the walker CTA's records, in the cluster window
  const uint32_t r_rec = cluster_map(L.rec, 0), r_seq = cluster_map(L.seq, 0);
  for (int c = s; c < n; c += kScouts) {
    const int y = c / gw;
    const uint32_t* ci = J.cand_idx + (size_t)c * k;
    const float* cd = J.cand_dist + (size_t)c * k;
    uint32_t t[4];
    float d[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int j = r * 32 + lane;
      t[r] = kNoCand;
      d[r] = inf;
      if (r < nr && j < k) {
        t[r] = __ldg(ci + j);
        d[r] = __ldg(cd + j);
      }
    }
    // Wait until the follower has cell c - ahead: the cell above is
    // then known, and the counters this record is filtered by are at most `ahead`
    // placements (and the follower's lag) old (in a region of one colour a row's
    // placements cap dozens of the nearest materials; a record built a whole
    // row ahead would list none left).  The walker read that cell's record
    // before placing it (the placement depends on it), so the walker is done
    // with the ring slot this record reuses, and so are the refiners (ring_size).
    const int lead = c - ahead;
    for (uint32_t polls = 0;
         lead >= 0 && !__all_sync(0xffffffffu, (int)ld_acquire_cta(&F.ctl[kFollowed]) > lead);) {
      const bool out = ++polls > kScoutPolls;
      if (__any_sync(0xffffffffu, out || ld_volatile_u32(&F.ctl[kFollowAbort]) != 0u)) {
        if (out && lane == 0) {
          atomicOr(err, kErrTimeout);
          st_cluster_u32(cluster_map(&L.ctrl[kAbort], 0), 1u);
        }
        return false;
      }
      __nanosleep(100);
    }
    const int up = y == 0 ? -1 : (int)*reinterpret_cast<const volatile uint16_t*>(&F.cells[(c - gw) & cmask]);
    const uint32_t ep0 = ld_acquire_cta(&F.ctl[kFollowEpoch]);
    int bf = 0, br = 0;
    float af = inf, ar = inf;  // distance of the 33rd entry
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      if (r < nr && (bf <= 32 || br <= 32)) {
        const bool in = t[r] < (uint32_t)p && (int)t[r] != up;
        const bool okf = in && ld_volatile_u32(&F.usage[t[r]]) < max_usage;
        const unsigned mf = __ballot_sync(0xffffffffu, okf), mr = __ballot_sync(0xffffffffu, in);
        const int pf = bf + __popc(mf & lt), pr = br + __popc(mr & lt);
        if (okf && pf < 32) {
          S.kf[pf] = ((uint32_t)pf << 17) | t[r];
          S.df[pf] = d[r];
        }
        if (in && pr < 32) {
          S.kr[pr] = ((uint32_t)pr << 17) | t[r];
          S.dr[pr] = d[r];
        }
        const unsigned f32 = __ballot_sync(0xffffffffu, okf && pf == 32);
        const unsigned r32 = __ballot_sync(0xffffffffu, in && pr == 32);
        if (f32) af = __shfl_sync(0xffffffffu, d[r], __ffs(f32) - 1);
        if (r32) ar = __shfl_sync(0xffffffffu, d[r], __ffs(r32) - 1);
        bf += __popc(mf);
        br += __popc(mr);
      }
    }
    __threadfence_block();
    const uint32_t ep1 = ld_acquire_cta(&F.ctl[kFollowEpoch]);
    __syncwarp();
    const int cf = min(bf, 32), cr = min(br, 32);
    // static window test of entry `lane` against the next entry of its list
    const float dfi = lane < cf ? S.df[lane] : inf, dfn = lane + 1 < cf ? S.df[lane + 1] : af;
    const float dri = lane < cr ? S.dr[lane] : inf, drn = lane + 1 < cr ? S.dr[lane + 1] : ar;
    const bool blocked_f = use_pen && dfn < __fadd_rn(dfi, two_w);
    const bool blocked_r = use_pen && drn < __fadd_rn(dri, two_w);
    const uint32_t slot = (uint32_t)(c & (R - 1));
    const uint32_t rr = r_rec + slot * (uint32_t)sizeof(CellRecord);
    // final keys into the local copy, then 16-byte stores to the walker's SM
    // (fewer requests on its shared memory)
    const uint32_t kf_final = lane < cf ? S.kf[lane] | (blocked_f ? 0x10000u : 0u) : 0xFFFFFFFFu;
    const uint32_t kr_final = lane < cr ? S.kr[lane] | (blocked_r ? 0x10000u : 0u) : 0xFFFFFFFFu;
    __syncwarp();
    S.kf[lane] = kf_final;
    S.kr[lane] = kr_final;
    __syncwarp();
    if (lane < 16) {
      const uint4 v = reinterpret_cast<const uint4*>(lane < 8 ? S.kf : S.kr)[lane & 7];
      st_cluster_v4(rr + 16u * (uint32_t)lane, v);
    }
    if (lane == 0) st_cluster_u32(rr + 256u, ep0 == ep1 ? ep0 : kInvalidEpoch);
    {
      // distance, weight against the cell above and Lab of each f entry (wgt
      // as full_cell computes it), and the distance after the list
      float d = inf, wu = 0.0f;
      float4 la = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lane < cf) {
        d = S.df[lane];
        la = __ldg(pal + (kf_final & 0xFFFFu));
        if (use_pen && up >= 0) wu = wgt(la, __ldg(pal + up));
      }
      const uint32_t wrec = rr + (uint32_t)offsetof(CellRecord, wd);
      st_cluster_u32(wrec + 4u * (uint32_t)lane, __float_as_uint(d));
      st_cluster_u32(rr + (uint32_t)offsetof(CellRecord, wu) + 4u * (uint32_t)lane, __float_as_uint(wu));
      st_cluster_v4(rr + (uint32_t)offsetof(CellRecord, wl) + 16u * (uint32_t)lane,
                    make_uint4(__float_as_uint(la.x), __float_as_uint(la.y), __float_as_uint(la.z), 0u));
      if (lane == 0) st_cluster_u32(rr + (uint32_t)offsetof(CellRecord, f_next), __float_as_uint(cf < 32 ? inf : af));
    }
    if (inject.scout_ns) __nanosleep(inject.scout_ns);
    fence_cluster();
    __syncwarp();
    if (lane == 0 && !inject.timeout) st_release_cluster(r_seq + 4u * slot, (uint32_t)(c + 1));
  }
  return true;
}

// Refiner r: prepares the lists of cells r, r + kRefiners, ...  Every wait is
// bounded; one that runs out aborts the walk.
template <bool kLabSmem, bool kRing>
__device__ void refine_cells(int r, const GreedyJob& J, const float4* __restrict__ pal, int p, uint8_t* smem, int R,
                             uint32_t* err, uint32_t delay_ns) {
  const int lane = threadIdx.x & 31;
  const int gw = J.gw, k = J.k, n = gw * J.gh;
  const WalkerLayout L = walker_layout(smem, gw, n, p, R, kRing);
  ListShared& Q = *L.lists;
  const float4* s_lab = L.lab;
  auto lab = [&](int i) -> float4 { return kLabSmem ? s_lab[i] : __ldg(pal + i); };
  const int cmask = cell_ring_size(gw) - 1;
  const uint32_t max_usage = J.max_usage;
  const float weight = J.weight, two_w = __fmul_rn(2.0f, weight), inf = __int_as_float(0x7f800000);
  const bool use_pen = weight > 0.0f;
  const unsigned lt = (1u << lane) - 1u;
  const int i = lane & 7, j0 = lane >> 3;
  // polls until ok() in every lane; false (in every lane): aborted
  auto wait = [&](auto ok) -> bool {
    for (uint32_t polls = 0; !__all_sync(0xffffffffu, ok());) {
      if ((++polls & 15u) == 0u) {
        const bool out = polls > kRefinePolls;
        if (__any_sync(0xffffffffu, out || ld_volatile_u32(&L.ctrl[kAbort]) != 0u)) {
          if (out && lane == 0) {
            atomicOr(err, kErrTimeout);
            *reinterpret_cast<volatile uint32_t*>(&L.ctrl[kAbort]) = 1u;
          }
          return false;
        }
      }
    }
    return true;
  };
  auto at = [&](int c) -> uint32_t {  // a placed cell's material
    return kRing ? ld_volatile_u32(&L.ring[c & cmask]) & 0xFFFFu
                 : (uint32_t)*reinterpret_cast<const volatile uint16_t*>(&L.grid16[c]);
  };
  const uint32_t usage0 = smem_u32(L.usage);
  // Whether the record of cell c (this warp's) is published; a probe looks at
  // the warp's next 8 (lane l at cell c + l * kRefiners).
  int ready_until = 0;
  auto published = [&](int c) -> bool {
    if (c < ready_until) return true;
    const int cc = c + (lane & 7) * kRefiners;
    const bool mine = cc >= n || ld_acquire_cluster(smem_u32(&L.seq[cc & (R - 1)])) == (uint32_t)(cc + 1);
    const unsigned no = __ballot_sync(0xffffffffu, !mine) & 0xFFu;
    ready_until = c + (no ? __ffs(no) - 1 : 8) * kRefiners;
    return c < ready_until;
  };
  // A cell's candidates, one a lane: the record's list, or, when it is of an
  // earlier epoch, the first 32 candidates of the row.  m = p: none.
  uint32_t m = (uint32_t)p, rec_epoch = 0;
  float d = inf, after = inf, wu = 0.0f;
  float4 la = make_float4(0.f, 0.f, 0.f, 0.f);
  auto load_row = [&](int c) {
    const uint32_t* ci = J.cand_idx + (size_t)c * k;
    const float* cd = J.cand_dist + (size_t)c * k;
    m = lane < k ? __ldg(ci + lane) : kNoCand;
    d = lane < k ? __ldg(cd + lane) : inf;
    after = k > 32 ? __ldg(cd + 32) : inf;
    const int up = c >= gw ? (int)at(c - gw) : -1;
    if ((int)m == up || m >= (uint32_t)p) m = (uint32_t)p;
    wu = 0.0f;
    la = make_float4(0.f, 0.f, 0.f, 0.f);
    if (m < (uint32_t)p) {
      la = lab((int)m);
      if (use_pen && up >= 0) wu = wgt(la, lab(up));
    }
  };
  bool use_f = false;
  auto load_record = [&](int c) {
    const CellRecord& Rc = L.rec[c & (R - 1)];
    rec_epoch = Rc.epoch;
    const uint32_t key = Rc.kf[lane];
    m = key == 0xFFFFFFFFu ? (uint32_t)p : key & 0xFFFFu;
    d = Rc.wd[lane];
    wu = Rc.wu[lane];
    la = Rc.wl[lane];
    after = Rc.f_next;
  };
  int x = r % gw;
  bool have = false;  // the cell's record is read
  for (int c = r; c < n; c += kRefiners) {
    const int slot = c & (kLists - 1);
    if (!have) {
      if (!wait([&] { return published(c); })) return;
      load_record(c);
    }
    // the slot is free: its last cell's lists are done, and the next cell's,
    // which reads this one's (the walker may have passed both on first forms)
    const int past = c - kLists;
    if (past >= 0 && !wait([&] {
          return (int)ld_acquire_cta(&Q.done[slot]) > past &&
                 (int)ld_acquire_cta(&Q.done[(past + 1) & (kLists - 1)]) > past + 1;
        }))
      return;
    if (delay_ns) __nanosleep(delay_ns);
    use_f = __all_sync(0xffffffffu, rec_epoch == ld_volatile_u32(&L.ctrl[kEpoch]));
    if (!use_f) load_row(c);
    const int lead = c - kRefineLag;
    if (lead >= 0 && !wait([&] {
          return kRing ? (ld_volatile_u32(&L.ring[lead & cmask]) >> 16) == ((uint32_t)lead & 0xFFFFu)
                       : at(lead) != kUnplaced;
        }))
      return;
    // the epoch, then the counters: they only grow within an epoch, so an entry
    // at the cap now stays there
    const uint32_t epoch = ld_acquire_cta(&L.ctrl[kEpoch]);
    auto counter = [&] {
      uint32_t u;
      asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(u) : "r"(usage0 + 4u * m) : "memory");
      return u;
    };
    uint32_t used = counter();
    if (use_f && __any_sync(0xffffffffu, rec_epoch != epoch)) {  // a reset while it waited
      load_row(c);
      used = counter();
    }
    const bool under = used < max_usage;
    const unsigned um = __ballot_sync(0xffffffffu, under);
    const int cnt = __popc(um), rk = __popc(um & lt);
    // every entry of the list against the window of the one before it
    const unsigned later = um & ~((2u << lane) - 1u);
    float dn = __shfl_sync(0xffffffffu, d, later ? __ffs(later) - 1 : lane);
    if (!later) dn = after;
    const bool in = under && rk < kList;
    const bool clear = !use_pen || dn >= __fadd_rn(d, two_w);
    const bool flat = __all_sync(0xffffffffu, !in || clear);
    const uint32_t tag = 0x00010000u | list_tag(c, epoch);
    // (every lane stores, the same instructions: no branch to come together from)
    auto entry = [&](unsigned long long* to, uint32_t ranks, uint32_t mat, int pos, bool clear) {
      *reinterpret_cast<volatile unsigned long long*>(to) =
          (unsigned long long)(tag | ((uint32_t)pos << 25) | (clear ? kClear : 0u) | mat) << 32 |
          __funnelshift_r(ranks, ranks, 2);
    };
    if (cnt < kList) {
      const bool none = lane < kList && lane >= cnt;
      entry(none ? &Q.ent[slot][lane] : &Q.spare[0], 0xFFFFFFFFu, (uint32_t)p, lane & 7, true);
      entry(none ? &Q.fin[slot][lane] : &Q.spare[0], 0xFFFFFFFFu, (uint32_t)p, lane & 7, true);
    }
    // the first form at once when the entries that mostly win are clear
    const bool early = __all_sync(0xffffffffu, !under || rk >= kEarly || clear);
    if (early) entry(in ? &Q.ent[slot][rk] : &Q.spare[0], 0x11111111u * (uint32_t)min(rk, 15), m & 0xFFFFu, rk & 7, clear);
    // the list, for this cell's table and the next one's
    const int put = in ? rk : kList;
    Q.sel[slot][put] = make_float4(la.x, la.y, la.z, __uint_as_float(m));
    Q.dw[r][put] = make_float2(d, wu);
    __syncwarp();
    st_release_cta(&Q.seq[slot], (uint32_t)(c + 1));
    if (!flat) {
      const float beyond =  // the distance of the first entry after the list
          cnt > kList
              ? __uint_as_float(__reduce_min_sync(0xffffffffu, under && rk == kList ? __float_as_uint(d) : 0xFFFFFFFFu))
              : after;
      // lane (i, j0) ranks entry i for previous entries j0 and j0 + 4
      const bool absent = i >= cnt;
      const float4 ei = Q.sel[slot][absent ? 0 : i];
      const float2 di = Q.dw[r][absent ? 0 : i];
      const float up_pen = __fadd_rn(0.0f, di.y);
      float wa = 0.0f, wb = 0.0f;
      if (x > 0) {
        const int prev = (c - 1) & (kLists - 1);
        if (!wait([&] { return ld_acquire_cta(&Q.seq[prev]) == (uint32_t)c; })) return;
        const float4 ea = Q.sel[prev][j0], eb = Q.sel[prev][j0 + 4];  // stale beyond its length: never looked up
        const float2 w = weight_of_sq2(sq_dist(ei.x, ei.y, ei.z, ea.x, ea.y, ea.z), sq_dist(ei.x, ei.y, ei.z, eb.x, eb.y, eb.z));
        wa = w.x;
        wb = w.y;
      }
      const float sa = absent ? inf : __fadd_rn(di.x, __fmul_rn(__fadd_rn(up_pen, wa), weight));
      const float sb = absent ? inf : __fadd_rn(di.x, __fmul_rn(__fadd_rn(up_pen, wb), weight));
      uint32_t ra = 0u, rb = 0u;
#pragma unroll
      for (int o = 1; o < kList; ++o) {
        const int q = (i + o) & 7;
        const float va = __shfl_sync(0xffffffffu, sa, (lane & 24) | q), vb = __shfl_sync(0xffffffffu, sb, (lane & 24) | q);
        ra += va < sa || (va == sa && q < i) ? 1u : 0u;
        rb += vb < sb || (vb == sb && q < i) ? 1u : 0u;
      }
      if (!(sa <= beyond)) ra = kRankOpen;
      if (!(sb <= beyond)) rb = kRankOpen;
      uint32_t ranks = (ra << (28 - 4 * j0)) | (rb << (12 - 4 * j0));
      ranks |= __shfl_xor_sync(0xffffffffu, ranks, 8);
      ranks |= __shfl_xor_sync(0xffffffffu, ranks, 16);
      // (the four lanes of an entry hold the same word)
      entry(absent ? &Q.spare[0] : early ? &Q.fin[slot][i] : &Q.ent[slot][i], ranks, __float_as_uint(ei.w) & 0xFFFFu, i, true);
    }
    __syncwarp();
    st_release_cta(&Q.done[slot], (uint32_t)(c + 1));
    // the next cell's record
    const int next = c + kRefiners;
    have = next < n && published(next);
    if (have) load_record(next);
    x += kRefiners;
    while (x >= gw) x -= gw;
  }
}

template <bool kLabSmem, bool kRing>
__global__ void __cluster_dims__(1 + kScoutCtas, 1, 1) __launch_bounds__(kThreads, 1)
    greedy_pair_kernel(const float4* __restrict__ pal, int p, const GreedyJob* __restrict__ jobs, uint32_t* err,
                       uint32_t walk_polls, bool roomy, WalkInject inject) {
  extern __shared__ __align__(128) uint8_t smem[];
  const GreedyJob J = jobs[blockIdx.x / (1 + kScoutCtas)];
  const uint32_t rank = cluster_ctarank();
  // the warp index through a shuffle: the compiler then knows each warp's path
  // as converged (without, every warp collective of the walker's loop comes with
  // a convergence step: 138 against 86 cycles a cell in a copy of the loop)
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int gw = J.gw, gh = J.gh, k = J.k, n = gw * gh;
  const int R = ring_size(gw, roomy);
  const WalkerLayout L = walker_layout(smem, gw, n, p, R, kRing);
  if (rank == 0) {
    for (int i = threadIdx.x; i <= p; i += blockDim.x) {
      L.usage[i] = i < p ? 0u : 0x7FFFFFFFu;  // absent entries have no room under any cap
      if (kLabSmem && i < p) L.lab[i] = pal[i];
    }
    for (int i = threadIdx.x; i < kLists * kList; i += blockDim.x)  // lists of no cell, their entries absent
      (&L.lists->ent[0][0])[i] = (unsigned long long)(kTagCell | (uint32_t)p) << 32;
    if (threadIdx.x < kResetLog) L.lists->reset_at[threadIdx.x] = 0;
    if (threadIdx.x < kLists) L.lists->seq[threadIdx.x] = L.lists->done[threadIdx.x] = 0;
    for (int i = threadIdx.x; i < R; i += blockDim.x) L.seq[i] = 0;
    if (kRing)
      for (int i = threadIdx.x; i < cell_ring_size(gw); i += blockDim.x) L.ring[i] = kNoCell;
    else
      for (int i = threadIdx.x; i < n; i += blockDim.x) L.grid16[i] = kUnplaced;
    if (threadIdx.x < 4) L.ctrl[threadIdx.x] = 0;
  }
  if (rank > 0) {
    const ScoutLayout F = scout_layout(smem, p);
    for (int i = threadIdx.x; i < p; i += blockDim.x) F.usage[i] = 0;
    if (threadIdx.x < 4) F.ctl[threadIdx.x] = 0;
  }
  cluster_sync_all();  // the walker CTA's state exists before any follower reads it

  if (rank >= 1) {
    // ---- the scouts, then (CTA 1) the final cost of the walk
    const ScoutLayout F = scout_layout(smem, p);
    float* terms = F.terms;
    constexpr int kPer = kScoutWarpsMax - 1;  // scouts in this CTA; its last warp follows the walk
    bool ok = true;
    if (warp < kPer)
      ok = scout_cells<kRing, kScoutCtas * kPer>(
          (int)(rank - 1) * kPer + warp, J, pal, p, smem, F.stage[warp], R, err, inject);
    else
      follow_walk<kRing>(J, p, smem, R, err);
    if (rank > 1) {
      cluster_sync_all();
      return;
    }
    if (!kRing) {  // the walker CTA's cost warp follows the walk instead
      cluster_sync_all();
      return;
    }
    // calculate_total_cost (adjacency.rs:91-130) of the placed grid once the
    // walk is complete: terms in parallel, one sequential FP32 sum in the
    // reference's order (right then down, row-major).
    __shared__ uint32_t s_ok;
    if (threadIdx.x == 0) s_ok = 1u;
    __syncthreads();
    if (!ok) s_ok = 0u;
    __syncthreads();
    if (threadIdx.x == 0 && s_ok) {
      const uint32_t r_progress = cluster_map(&L.ctrl[kProgress], 0), r_abort = cluster_map(&L.ctrl[kAbort], 0);
      uint32_t polls = 0;
      while (ld_acquire_cluster(r_progress) < (uint32_t)n) {
        if (ld_cluster_u32(r_abort) || ++polls > kScoutPolls) {
          s_ok = 0u;
          break;
        }
        __nanosleep(256);
      }
    }
    __syncthreads();
    if (s_ok) {
      float total = 0.0f;
      for (int c0 = 0; c0 < n; c0 += kCostChunk) {
        const int m = min(kCostChunk, n - c0);
        for (int i = threadIdx.x; i < m; i += blockDim.x) {
          const int c = c0 + i, x = c % gw, y = c / gw;
          const int cur = J.grid[c];
          float tr = 0.0f, td = 0.0f;
          if (cur >= 0) {
            const float4 lc = __ldg(pal + cur);
            if (x < gw - 1) {
              const int r = J.grid[c + 1];
              if (r >= 0) tr = wgt(lc, __ldg(pal + r));
            }
            if (y < gh - 1) {
              const int d = J.grid[c + gw];
              if (d >= 0) td = wgt(lc, __ldg(pal + d));
            }
          }
          terms[2 * i] = tr;
          terms[2 * i + 1] = td;
        }
        __syncthreads();
        if (threadIdx.x == 0)
          for (int i = 0; i < 2 * m; ++i) total = __fadd_rn(total, terms[i]);  // (the loads run ahead)
        __syncthreads();
      }
      if (threadIdx.x == 0 && J.total_cost) *J.total_cost = total;
    }
    cluster_sync_all();
    return;
  }
  if (!kRing && warp == 1) {
    // ---- CTA 0, warp 1: calculate_total_cost (adjacency.rs:91-130) following
    // the walk, and the placed grid into global memory.  Cell c's terms (right,
    // then down) are final once cells c, c + 1 and c + gw are placed (each is
    // written once, so a value seen is the final one); one FP32 sum in the
    // reference's order, 32 cells behind a row of the walker at most, so the
    // total is ready when the walk ends.  On another SMSP than the walker.
    auto lab_of = [&](int i) -> float4 { return kLabSmem ? L.lab[i] : __ldg(pal + i); };
    const volatile uint16_t* g16 = L.grid16;
    float total = 0.0f;
    bool ok = true;
    for (int c0 = 0; c0 < n && ok; c0 += 32) {
      const int c = c0 + lane, x = c % gw, y = c / gw;
      int cur = 0, rt = 0, dn = 0;
      bool lane_ok = true;
      if (c < n) {
        uint32_t polls = 0;
        for (;;) {
          cur = g16[c];
          rt = x < gw - 1 ? g16[c + 1] : 0;
          dn = y < gh - 1 ? g16[c + gw] : 0;
          if (cur != kUnplaced && rt != kUnplaced && dn != kUnplaced) break;
          if (ld_volatile_u32(&L.ctrl[kAbort]) || ++polls > kFollowPolls) {
            lane_ok = false;
            break;
          }
          __nanosleep(128);
        }
      }
      ok = __all_sync(0xffffffffu, lane_ok);
      if (!ok) break;
      float tr = 0.0f, td = 0.0f;
      if (c < n) {
        const float4 lc = lab_of(cur);
        if (x < gw - 1) tr = wgt(lc, lab_of(rt));
        if (y < gh - 1) td = wgt(lc, lab_of(dn));
        J.grid[c] = cur;
      }
      const int m = min(32, n - c0);
      for (int i = 0; i < m; ++i) {
        const float a = __shfl_sync(0xffffffffu, tr, i), b = __shfl_sync(0xffffffffu, td, i);
        total = __fadd_rn(__fadd_rn(total, a), b);
      }
    }
    if (ok) {
      if (lane == 0 && J.total_cost) *J.total_cost = total;
    } else {
      // the walk gave up: every cell empty (this warp is the grid's only writer)
      for (int i = lane; i < n; i += 32) J.grid[i] = -1;
      if (lane == 0) atomicOr(err, kErrTimeout);
    }
    cluster_sync_all();
    return;
  }
  if (warp != 0) {
    // ---- CTA 0, the refiners (not on the walker's scheduler)
    const int r = warp - warp / 4 - 2;
    if (walks_by_lists(p, J.max_usage) && (warp & 3) != 0 && r >= 0 && r < kRefiners)
      refine_cells<kLabSmem, kRing>(r, J, pal, p, smem, R, err, inject.refiner_ns);
    cluster_sync_all();
    return;
  }

  // ---- CTA 0, warp 0: the walker
  uint32_t* ctrl = L.ctrl;
  CellRecord* rec = L.rec;
  uint32_t* ring = L.ring;
  uint16_t* grid16 = L.grid16;
  ListShared& Q = *L.lists;
  const int cmask = cell_ring_size(gw) - 1;
  // a placement: the 16-bit grid, or the ring word and the global grid
  auto place = [&](int cc, int tt) {
    if (kRing) {
      ring[cc & cmask] = cell_word(cc, tt);
      J.grid[cc] = tt;
    } else {
      grid16[cc] = (uint16_t)tt;
    }
  };
  uint32_t* usage = L.usage;
  const float4* s_lab = L.lab;
  const uint32_t max_usage = J.max_usage;
  const float weight = J.weight;
  auto lab = [=](int i) -> float4 { return kLabSmem ? s_lab[i] : __ldg(pal + i); };
  uint32_t epoch = 0;
  int resets = 0, last = -1, x = 0;
  bool aborted = false;
  // A cell whose list does not settle it is decided from its record: the
  // lowest key among the entries under the cap, not the left neighbour, is the
  // reference's choice when its window is clear.
  struct Cur {
    uint32_t key, ti, ui;
    bool f;  // the key is the record's f entry (its epoch is the walk's)
    bool there;  // the record was published when it was read
  };
  auto record_entry = [&](int c) {
    Cur r;
    // (the refiner that sets this word saw the record published)
    r.there = ld_acquire_cta(&Q.seq[c & (kLists - 1)]) == (uint32_t)(c + 1);
    const CellRecord& Rc = rec[c & (R - 1)];
    r.f = Rc.epoch == epoch;
    r.key = r.f ? Rc.kf[lane] : Rc.kr[lane];
    r.ti = r.key & 0xFFFFu;
    r.ui = (r.key != 0xFFFFFFFFu && r.ti < (uint32_t)p) ? usage[r.ti] : 0xFFFFFFFFu;
    return r;
  };
  // A cell (not a row start) whose first eligible f entry has later entries
  // inside its penalty window, settled from the record: the window's entries
  // are the list's entries under the cap now, other than the left neighbour's
  // material, with distance below d(first) + 2*weight (f_next >= that bound
  // closes the window inside the list); each scores d + (w_up + w_left) *
  // weight in full_cell's arithmetic and the lowest score, then the lowest
  // position, wins -- full_cell's decision.  Commits it and returns the
  // material; -1 when the window may reach past the list (then full_cell
  // decides).  e0: the position of the first eligible entry.
  auto window_cell = [&](int cc, const Cur& cu, int left, bool has_up, int e0) -> int {
    const CellRecord& Rc = rec[cc & (R - 1)];
    const bool elig = cu.key != 0xFFFFFFFFu && cu.ui < max_usage && (int)cu.ti != left;
    const float dl = Rc.wd[lane];
    const float b0 = __fadd_rn(Rc.wd[e0], __fmul_rn(2.0f, weight));
    if (!(Rc.f_next >= b0)) return -1;
    const bool in = elig && lane >= e0 && dl < b0;
    float pen = has_up ? Rc.wu[lane] : 0.0f;  // 0 + w_up, exactly
    pen = __fadd_rn(pen, wgt(Rc.wl[lane], lab(left)));
    const uint32_t sb = in ? __float_as_uint(__fadd_rn(dl, __fmul_rn(pen, weight))) : 0xFFFFFFFFu;
    const uint32_t mn = __reduce_min_sync(0xffffffffu, sb);
    const bool wins = mn == 0xFFFFFFFFu ? lane == e0 : (in && sb == mn);
    const uint32_t wn = __reduce_min_sync(0xffffffffu, wins ? ((uint32_t)lane << 16) | cu.ti : 0xFFFFFFFFu);
    const int win = (int)(wn >> 16), tw = (int)(wn & 0xFFFFu);
    if (lane == win) {
      usage[cu.ti] = cu.ui + 1u;
      place(cc, tw);
    }
    return tw;
  };
  // The walk is a chain of dependent decisions, so its speed is the latency of
  // one decision in one warp.  Per cell that is a rotation and an OR (the ranks'
  // column for the previous choice), one warp minimum, and the commit, made by
  // every lane with the same stores so that no lane waits on another.  All else
  // runs ahead: a list is read two cells early, unconditionally (one not there
  // yet, or of another epoch, shows by its tag), its counters one cell early --
  // the one commit in between is the left neighbour's, which the cell may not
  // take -- and formed into the packed word beside the minimum of the cell
  // before: rank << 28 | position << 25 | clear << 24 | counter + 1 << 16 | material;
  // bits 23-27 are then the rotation that brings up the next column.  Counters pack to 7 bits: with caps
  // beyond that (kWide) one of 127 or more is read again at its commit.
  struct Entry {
    uint32_t ranks, hi;
  };
  auto load_entry = [&](int c) {
    const unsigned long long v = *reinterpret_cast<const volatile unsigned long long*>(&Q.ent[c & (kLists - 1)][lane & 7]);
    return Entry{(uint32_t)v, (uint32_t)(v >> 32)};
  };
  const uint32_t cap = lane < kList ? max_usage : 0u;  // lanes past the list never take part
  // Decides cells from c on, not past `end` (the row's), the first one from
  // lists and counters read afresh; b: the word of the choice before c.
  // Returns the first cell left open.
  auto fast_cells = [&](auto wide, int c, int end, uint32_t& b, Entry e0) -> int {
    constexpr bool kWide = decltype(wide)::value;
    uint32_t w, ranks;
    auto form = [&](const Entry& e, uint32_t u, int cell) {
      const uint32_t v = e.hi ^ list_tag(cell, epoch);
      const bool there = (v & kTagMask) == 0u;
      w = u < cap ? v + ((kWide ? min(u, 126u) : u) << 16) : 0xFFFFFFFFu;
      w = there ? w : kNotThere;
      ranks = there ? e.ranks : 0u;
    };
    // clear, and a rank below 8
    auto settles = [](uint32_t best) { return ((best ^ kClear) & (0x80000000u | kClear)) == 0u; };
    // the entry's word given the choice before: its rank's column, out if it is that material
    auto choice = [&](uint32_t b) -> uint32_t {
      const uint32_t word = w | (__funnelshift_l(ranks, ranks, b >> 23) & 0xF0000000u);
      return ((w ^ b) & 0xFFFFu) == 0u ? 0xFFFFFFFFu : word;
    };
    for (uint32_t polls = 0;;) {
      uint32_t stop = 0u;  // the word that stopped the run
      const uint32_t u0 = usage[e0.hi & 0xFFFFu];
      Entry e1 = load_entry(c + 1);
      form(e0, u0, c);
      uint32_t u1 = usage[e1.hi & 0xFFFFu];
      bool ok = true;
      while (c < end) {
        const uint32_t word = choice(b);
        const Entry e2 = load_entry(c + 2);
        const uint32_t best = __reduce_min_sync(0xffffffffu, word);
        form(e1, u1, c + 1);
        stop = best;
        ok = settles(best);
        if (!ok) break;
        uint32_t u = __byte_perm(best, 0u, 0x4442);
        if (kWide && u == 127u) u = usage[best & 0xFFFFu] + 1u;
        usage[best & 0xFFFFu] = u;
        place(c, (int)(best & 0xFFFFu));
        u1 = usage[e2.hi & 0xFFFFu];
        b = best;
        e1 = e2;
        ++c;
      }
      // done; or cell c is open; or its list is not there, or its first entry
      // not clear and the second form decides: a short wait for that
      if (ok || stop >= kRankOpen << 28) return c;
      if (stop == kNotThere) {
        do {
          if (++polls > 256u) return c;
          e0 = load_entry(c);
        } while (!__all_sync(0xffffffffu, ((e0.hi ^ list_tag(c, epoch)) & kTagMask) == 0u));
      } else {
        while (!__all_sync(0xffffffffu, ld_acquire_cta(&Q.done[c & (kLists - 1)]) == (uint32_t)(c + 1)))
          if (++polls > 256u) return c;
        const unsigned long long v = Q.fin[c & (kLists - 1)][lane & 7];
        e0 = Entry{(uint32_t)v, (uint32_t)(v >> 32)};
      }
    }
  };
  // A run of cells from c on, not past `end` (the row's), from their records
  // alone, in the manner of fast_cells: for cells whose lists are of the epoch
  // before, or hold nothing.  Stops at a cell that its record does not settle
  // by a clear entry.  The word: position << 27 | not clear (or a counter that
  // does not fit) << 26 | counter << 16 | material.  Measured: 140 x 100 cells,
  // 30 materials, cap 1: 3.89 -> 1.77 ms a call.  (Its result and what follows
  // from it go through a shuffle: the compiler else takes the walker's loops for
  // divergent, 1.0 -> 1.4 ms for 5000 materials, which never come here.)
  int rec_ready = 0;  // the records of the cells from the walker's to before it are published
  // The word beside a record names the cell it is of.
  auto record_there = [&](int c) -> bool {
    return __all_sync(0xffffffffu, ld_acquire_cluster(smem_u32(&L.seq[c & (R - 1)])) == (uint32_t)(c + 1));
  };
  // After `polls` polls: whether the walk ends here.
  auto gives_up = [&](uint32_t polls) -> bool {
    aborted = polls > walk_polls || __any_sync(0xffffffffu, ld_volatile_u32(&ctrl[kAbort]) != 0u);
    return aborted;
  };
  auto record_cells = [&](int c, int end, int left) -> int {
    if (c >= rec_ready) {
      const int cc = c + lane;
      const unsigned no = __ballot_sync(
          0xffffffffu, cc >= n || ld_acquire_cluster(smem_u32(&L.seq[cc & (R - 1)])) != (uint32_t)(cc + 1));
      rec_ready = __shfl_sync(0xffffffffu, c + (no ? __ffs(no) - 1 : 32), 0);
    }
    end = min(end, rec_ready);
    struct Head {
      uint32_t epoch, kf, kr;
    };
    auto head = [&](int c) {
      const CellRecord& Rc = rec[c & (R - 1)];
      return Head{Rc.epoch, Rc.kf[lane], Rc.kr[lane]};
    };
    auto pick = [&](const Head& h) { return h.epoch == epoch ? h.kf : h.kr; };
    auto counter = [&](uint32_t key) { return usage[min(key & 0xFFFFu, (uint32_t)p)]; };  // (p: full)
    uint32_t key = pick(head(c)), u = counter(key);
    Head h1 = head(c + 1);
    while (c < end) {
      const uint32_t key1 = pick(h1), u1 = counter(key1);
      const Head h2 = head(c + 2);
      const bool takes = u < max_usage && (int)(key & 0xFFFFu) != left;
      const uint32_t w = (key >> 17) << 27 | (key & 0x10000u) << 10 | min(u, 1023u) << 16 | (key & 0xFFFFu) |
                         (u < 1023u ? 0u : 1u << 26);
      const uint32_t best = __reduce_min_sync(0xffffffffu, takes ? w : 0xFFFFFFFFu);
      if (best & (1u << 26)) break;
      left = (int)(best & 0xFFFFu);
      usage[left] = ((best >> 16) & 1023u) + 1u;
      place(c, left);
      key = key1;
      u = u1;
      h1 = h2;
      ++c;
    }
    return __shfl_sync(0xffffffffu, c, 0);  // (uniform for the compiler)
  };
  const bool lists = walks_by_lists(p, max_usage);
  int old_lists = 0;         // lists of cells before it may be of an earlier epoch
  constexpr int kNoneBehind = 0x7FFF0000;
  int behind = kNoneBehind;  // the first cell passed by a run whose list the walker has not seen
  bool known = true;         // b names the previous choice's position in its list
  uint32_t b = kClear;
  int c = 0;
  while (c < n) {
    // the list of cell c, or, in a walk without lists, its record (bounded waits:
    // who makes them waits for nothing the walker has yet to do)
    Entry e = load_entry(c);
    if (lists) {
      // A cell passed by its list has been in its slot; a run from records leaves cells
      // behind whose lists may be late.  Until those are done, the walk stays
      // within a turn of the ring of the first of them.
      if (c + 4 > behind + kTurn) {
        const int j = c - kLists + (lane & (kLists - 1));
        for (uint32_t polls = 0;
             !__all_sync(0xffffffffu, j < behind || (int)ld_acquire_cta(&Q.done[j & (kLists - 1)]) > j);)
          if (gives_up(++polls)) break;
        if (aborted) break;
        behind = __shfl_sync(0xffffffffu, kNoneBehind, 0);
        e = load_entry(c);  // (read before, it may be of two turns ago)
      }
      for (uint32_t polls = 0; !__all_sync(0xffffffffu, ((e.hi ^ list_tag(c, 0)) & kTagCell) == 0u);) {
        if (gives_up(++polls)) break;
        e = load_entry(c);
      }
    } else if (c >= rec_ready) {
      for (uint32_t polls = 0; !record_there(c);)
        if (gives_up(++polls)) break;
    }
    if (aborted) break;
    if (!lists || c < old_lists) {
      const int c0 = c;
      c = record_cells(c, min(c + gw - x, lists ? min(old_lists, behind + kTurn) : n), x == 0 ? -1 : last);
      __syncwarp();
      if (c > c0) {
        behind = __shfl_sync(0xffffffffu, min(behind, c0 + 1), 0);
        x += c - c0;
        if (x == gw) x = 0;
        last = __shfl_sync(0xffffffffu, kRing ? (int)(ring[(c - 1) & cmask] & 0xFFFFu) : (int)grid16[c - 1], 0);
        // its place in the list of cell c - 1, if that is there: its maker sets seq
        // when the slot has held the list of the turn before
        const bool made = __all_sync(0xffffffffu, ld_acquire_cta(&Q.seq[(c - 1) & (kLists - 1)]) == (uint32_t)c);
        const Entry before = load_entry(c - 1);
        const unsigned at = __ballot_sync(0xffffffffu, lane < kList && (before.hi & 0xFFFFu) == (uint32_t)last);
        known = made && at != 0u && __all_sync(0xffffffffu, ((before.hi ^ list_tag(c - 1, 0)) & kTagCell) == 0u);
        b = kClear | (known ? (uint32_t)(__ffs(at) - 1) << 25 : 0u) | (uint32_t)last;
        continue;
      }
    }
    const bool fresh = __all_sync(0xffffffffu, ((e.hi ^ list_tag(c, epoch)) & kTagMask) == 0u);
    if (lists && fresh && (x == 0 || known)) {
      const int c0 = c;
      if (x == 0) b |= 0xFFFFu;  // no left neighbour
      const int end = min(c + gw - x, behind + kTurn);
      if (max_usage < 127u) c = fast_cells(std::false_type{}, c, end, b, e);
      else c = fast_cells(std::true_type{}, c, end, b, e);
      __syncwarp();
      if (c > c0) {
        last = (int)(b & 0xFFFFu);
        known = true;
        x += c - c0;
        if (x == gw) x = 0;
        continue;
      }
    }
    // ---- cell c from its record, or in full
    const bool row_start = x == 0;
    Cur cu = record_entry(c);
    for (uint32_t polls = 0; !__all_sync(0xffffffffu, cu.there || !lists);) {
      if (gives_up(++polls)) break;
      cu = record_entry(c);
    }
    if (aborted) break;
    const uint32_t key = __reduce_min_sync(
        0xffffffffu, cu.ui < max_usage && (row_start || (int)cu.ti != last) ? cu.key : 0xFFFFFFFFu);
    int t = (int)(key & 0xFFFFu);
    bool done = key != 0xFFFFFFFFu && !(key & 0x10000u);
    if (done) {
      if (lane == (int)(key >> 17)) {
        usage[cu.ti] = cu.ui + 1u;
        place(c, t);
      }
    } else if (!row_start && key != 0xFFFFFFFFu && cu.f) {
      const int tw = window_cell(c, cu, last, c >= gw, (int)(key >> 17));
      done = tw >= 0;
      if (done) t = tw;
    }
    if (!done) {
      const int up = c < gw ? -1 : kRing ? (int)(ring[(c - gw) & cmask] & 0xFFFFu) : (int)grid16[c - gw];
      const uint32_t* ci = J.cand_idx + (size_t)c * k;
      const float* cd = J.cand_dist + (size_t)c * k;
      const int was = resets;
      t = full_cell(lab, ci, cd, k, p, up, row_start ? -1 : last, usage, max_usage, weight, ctrl, epoch, resets, lane,
                    Q.reset_at, c);
      old_lists = __shfl_sync(0xffffffffu, resets != was ? c + kRefineLag : old_lists, 0);
      if (lane == 0) place(c, t);
    }
    __syncwarp();
    last = t;
    const unsigned at = __ballot_sync(0xffffffffu, lane < kList && (e.hi & 0xFFFFu) == (uint32_t)t);
    known = at != 0u;
    b = kClear | (known ? (uint32_t)(__ffs(at) - 1) << 25 : 0u) | (uint32_t)t;
    ++c;
    x = x + 1 == gw ? 0 : x + 1;
  }
  if (aborted) {
    if (lane == 0) {
      atomicOr(err, kErrTimeout);
      *reinterpret_cast<volatile uint32_t*>(&ctrl[kAbort]) = 1u;
    }
    // every cell empty, so the stages after the walk read no stale index (in
    // the 16-bit grid form the cost warp writes the global grid)
    if (kRing)
      for (int i = lane; i < n; i += 32) J.grid[i] = -1;
    if (lane == 0 && J.n_resets) *J.n_resets = 0;
  } else {
    // the placed grid in global memory (every lane's stores visible) before the
    // completion the scout CTA waits for; in the 16-bit grid form the cost warp
    // writes it
    if (kRing) __threadfence();
    if (lane == 0 && J.n_resets) *J.n_resets = resets;
    __syncwarp();
    if (lane == 0) st_release_cluster(smem_u32(&ctrl[kProgress]), (uint32_t)n);
  }
  cluster_sync_all();  // the scouts are done with this CTA's shared memory
}

}  // namespace

size_t greedy_shared_bytes(int k, int gw, int p, bool lab_smem, bool usage_smem) {
  return greedy_smem_bytes(k, gw, p, lab_smem, usage_smem);
}

bool greedy_scouted_fits(int gw, int n, int p) {
  constexpr size_t kMaxSmem = 227 * 1024 - 128;  // beside the kernel's static words
  // the largest ring any row width uses, the palette Lab outside shared memory
  return gw >= 8 && p <= 65535 &&
         (pair_smem_bytes(gw, n, p, false, false) <= kMaxSmem || pair_smem_bytes(gw, n, p, false, true) <= kMaxSmem);
}

int launch_greedy(const float4* pal, int p, const GreedyJob* jobs_dev, int n_jobs, int k, int max_gw,
                  int max_cells, uint32_t* usage_scratch, uint32_t* err, cudaStream_t stream, bool one_warp,
                  WalkInject inject) {
  if (n_jobs <= 0) return MG_OK;
  if (k < 1 || k > 100) return fail(MG_ERR_ARG, "candidate count must be in 1..100");
  constexpr size_t kMaxSmem = 227 * 1024 - 128;  // beside the kernel's static words
  static int configured_device = -1;
  int dev = 0;
  MG_CUDA(cudaGetDevice(&dev));
  if (configured_device != dev) {
    const int m = (int)kMaxSmem;
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    MG_CUDA(cudaFuncSetAttribute(greedy_kernel<true, true>, a, m));
    MG_CUDA(cudaFuncSetAttribute(greedy_kernel<false, true>, a, m));
    MG_CUDA(cudaFuncSetAttribute(greedy_kernel<false, false>, a, m));
    MG_CUDA(cudaFuncSetAttribute(greedy_pair_kernel<true, false>, a, m));
    MG_CUDA(cudaFuncSetAttribute(greedy_pair_kernel<false, false>, a, m));
    MG_CUDA(cudaFuncSetAttribute(greedy_pair_kernel<true, true>, a, m));
    MG_CUDA(cudaFuncSetAttribute(greedy_pair_kernel<false, true>, a, m));
    configured_device = dev;
  }
  // The scouted walk: counters in shared memory, 16-bit palette indices, rows
  // of at least 8 cells.
  if (!one_warp && max_gw >= 8 && p <= 65535) {
    // the grid before the ring (a shorter walker loop), the palette Lab in shared memory before global
    const bool fit[4] = {pair_smem_bytes(max_gw, max_cells, p, true, false) <= kMaxSmem,
                         pair_smem_bytes(max_gw, max_cells, p, false, false) <= kMaxSmem,
                         pair_smem_bytes(max_gw, max_cells, p, true, true) <= kMaxSmem,
                         pair_smem_bytes(max_gw, max_cells, p, false, true) <= kMaxSmem};
    const int form = fit[0] ? 0 : fit[1] ? 1 : fit[2] ? 2 : fit[3] ? 3 : -1;
    if (form >= 0) {
      const bool lab_smem = form == 0 || form == 2, ring = form >= 2;
      const bool roomy = pair_smem_bytes(max_gw, max_cells, p, lab_smem, ring, true) <= kMaxSmem;
      const size_t bytes = pair_smem_bytes(max_gw, max_cells, p, lab_smem, ring, roomy);
      const uint32_t polls = inject.timeout ? kInjectedWalkPolls : kWalkPolls;
      auto go = [&](auto kernel) {
        kernel<<<(unsigned)((1 + kScoutCtas) * n_jobs), kThreads, bytes, stream>>>(pal, p, jobs_dev, err, polls, roomy, inject);
      };
      if (form == 0) go(greedy_pair_kernel<true, false>);
      else if (form == 1) go(greedy_pair_kernel<false, false>);
      else if (form == 2) go(greedy_pair_kernel<true, true>);
      else go(greedy_pair_kernel<false, true>);
      g_launches += 1;
      MG_CUDA(cudaGetLastError());
      return MG_OK;
    }
  }
  bool lab_smem = true, usage_smem = true;
  size_t bytes = greedy_smem_bytes(k, max_gw, p, lab_smem, usage_smem);
  if (bytes > kMaxSmem) {
    lab_smem = false;
    bytes = greedy_smem_bytes(k, max_gw, p, lab_smem, usage_smem);
  }
  if (bytes > kMaxSmem) {
    usage_smem = false;
    bytes = greedy_smem_bytes(k, max_gw, p, lab_smem, usage_smem);
  }
  if (bytes > kMaxSmem) return fail(MG_ERR_ARG, "grid row too wide for the greedy walk");
  if (!usage_smem && !usage_scratch) return fail(MG_ERR_ARG, "usage scratch required for this palette size");
  if (lab_smem)
    greedy_kernel<true, true><<<n_jobs, 32, bytes, stream>>>(pal, p, jobs_dev, usage_scratch, err);
  else if (usage_smem)
    greedy_kernel<false, true><<<n_jobs, 32, bytes, stream>>>(pal, p, jobs_dev, usage_scratch, err);
  else
    greedy_kernel<false, false><<<n_jobs, 32, bytes, stream>>>(pal, p, jobs_dev, usage_scratch, err);
  g_launches += 1;
  MG_CUDA(cudaGetLastError());
  return MG_OK;
}

}  // namespace mg
