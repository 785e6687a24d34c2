// Exact sweep: the body of FluidSim::tick (src/fluid.rs:584-651) over the region's CTA, eight lanes per
// cell (one thread in long rounds), with results bit-identical to the reference's sequential loop.
//
// The order of the sequential loop matters only between cells that touch a common cell, so the
// sweep runs in rounds over the dependency graph of the drained cells:
//   * Dependencies. A cell reads and writes {self, below, +-x, +-z} and, if it may attempt a pull,
//     reads the cell above. Two cells conflict iff they are on one layer within manhattan distance
//     2, on adjacent layers within distance 1, or (the lower one may pull) two layers apart in one
//     column: 12 later positions per cell. Each cell counts its earlier conflicting cells in a byte
//     of shared memory; a finished cell decrements its successors' counts and appends those that
//     reach zero to the next round's list. Cells of one round never conflict. Solid cells only erase
//     their own partial entry, which nothing in the sweep reads: they are done in the prepass.
//   * Pressure pulls (fluid.rs:511-561) read cells far away and write one cell on a higher layer.
//     A pull at layer y sees, above y, the state at the tick's start changed by earlier pulls only
//     (every cell above y comes later in sorted order), and on y the writes of earlier cells. So
//     cells above y wait until no cell up to y can still pull, and on y itself a search reads the
//     value a cell held before the writes of later cells that already ran (LvOld); a search that
//     finds an unfinished earlier writer of a cell it reads is run again later.
//   * Who can pull. Nothing a cell does before its turn can lift a neighbour to 1 - 1e-4 or more
//     (a side flow stops at MIN_FLOW, falls fill the layer below, pulls only take), except a pull
//     that fills its own cell. So the cells that attempt are those below 1 - 1e-4 at the tick's start
//     plus the full ones an earlier pull takes from, and those that can find a start cell (`pp`)
//     have a full neighbour at the tick's start, were taken from, or follow a cell a pull filled.
//     Pulls run in the sorted order of `pp`; the 4096-attempt budget (fluid.rs:594) is a prefix count
//     that is exact at each of them.
// Nothing is undone or run twice, and no thread waits for another except at the CTA's barriers.
//
// What bounds it: the number of rounds times the latency of one (list entry -> 32-byte record -> 7
// cells -> plan -> stores -> successor counts -> barrier), on one SM per region, and between the rounds warp 0's
// chain of pulls: a lone warp takes ~8 cycles for each dependent instruction (a cell 1,700, a search round
// 1,600, a search's start 1,200 cycles). Dam break, first 16 ticks: 817 M SM cycles when every cell waited
// for its conflicts in rows of the sorted order and conflicting pulls were undone, 204 M here.
#pragma once
#include "engine_dev.cuh"

namespace vfe {

constexpr unsigned GRID_CLAIM = 0x80000000u;   // grid word while a CTA gives out slots: | writer's key << 8 | uniform value
constexpr int MAX_WARPS = 16;                  // warps of a CTA running the sweep
constexpr unsigned SOLO_CELLS = 4;             // a list this short is run by one warp (eight lanes per cell)
constexpr unsigned SOLO_ENTRIES = 6;           // queue entries one warp examines per search round
constexpr unsigned SOLO_WAIT = SOLO_ENTRIES;   // a search with more entries waiting goes to all warps
constexpr unsigned VIS_SLOTS = 4096;           // visited set, emptied when VIS_FULL cells have been added
constexpr int VIS_SHIFT = 20;                  // hash bits kept: 32 - log2(VIS_SLOTS)
constexpr unsigned VIS_FULL = 1536;            // one search adds <= 6 + 512 + one round's 5 per entry (480)
constexpr unsigned VIS_RANKS = 4096;           // ranks of one search: 6 + 5 * 512 at most
constexpr unsigned NGROUPS = (MAX_CELLS_PER_TICK + 31) / 32;
constexpr unsigned LIST_CAP = 2048;   // a round's list kept in shared memory; the rest goes to global
constexpr unsigned NOSUCC = 0xFFFFu;
static_assert(SOLO_CELLS <= LIST_CAP, "a short list is in shared memory");
static_assert(MAX_CELLS_PER_TICK < NOSUCC, "sorted positions fit 16 bits");
constexpr unsigned DONE = 0x80u;           // dependency byte of a finished cell: DONE | the footprint slots it wrote
constexpr int GATE_MAX = 31;               // range of the gate knob's radii (accepted, unused)

// What a round reads of a drained cell, made in the prepass: one 32-byte sector, a word per lane of the
// eight that run the cell.
struct __align__(16) LvCell {
  unsigned short succ[12];  // later conflicting positions (succ_offset's order), NOSUCC = none
  unsigned cid;             // domain id
  unsigned ye;              // layer | bits 27-31: may a pull start from the cell's up, +x, -x, +z, -z neighbour
                            // (x and z >= 0, fluid.rs:519)
};
static_assert(sizeof(LvCell) == 32, "LvCell");
constexpr unsigned YE_Y = 0x07FFFFFFu;  // layers: a domain has fewer than 2^31 cells and 65 x 65 columns or more

// The footprint volumes a cell of the gate layer found, for searches of earlier cells.
struct __align__(16) LvOld {
  float vol[8];
};

// The pressure search under way.
enum SearchStatus { SS_NONE = 0, SS_SUCCESS = 1, SS_BLOCKED = 2, SS_MORE = 3 };
struct Search {
  uint2 q[PRESSURE_SEARCH];  // queued cells: domain id | ABOVE where it lies above the pulling layer, volume
  // Visited set: a key stays where a search put it; what tells searches apart is the rank, whose
  // base falls from search to search, so that an older search's rank never wins (a set emptied after
  // every search cost ~700 cycles of each pull).
  unsigned vkey[VIS_SLOTS];     // cells tested by this or earlier searches (EMPTY_ID = free)
  unsigned vrank[VIS_SLOTS];    // rank base + earliest (entry, direction) that tested the cell
  unsigned rank0, nvis;         // the search's rank base, keys added since the set was last empty
  unsigned m_win[MAX_WARPS], m_side[MAX_WARPS], m_new[MAX_WARPS];
  unsigned blk;                 // 1 + an unfinished earlier cell the search depends on (0: none)
  unsigned pos, status, i, qlen, side;  // the cell, and the search's progress
  float vol, got, here;         // its volume, what the pull takes, the source's volume
  unsigned cid, skey;           // the pulling cell, the source's queue key
};
constexpr unsigned ABOVE = 0x80000000u;

// What warp 0 asks of the CTA between rounds.
enum SoloRequest { SR_LIST = 0, SR_GATE = 1, SR_SEARCH = 2, SR_END = 3 };
// The first pp cell and what is known about it.
struct HeadState {
  unsigned head, word;  // its position (n: none), its group
  unsigned blk;         // 1 + the cell its search waits for (0: none)
  unsigned test;        // lv_prune: 0 to be tested, 1 + the cell the test waits for, or TEST_FAILED
  int gate;             // its layer: cells above it wait
};
constexpr unsigned TEST_FAILED = 0xFFFFFFFFu;

struct LvSmem {
  unsigned dep[(MAX_CELLS_PER_TICK + 3) / 4];  // a byte per cell: unfinished earlier conflicting cells, or DONE | slots
  unsigned att[NGROUPS + 1];   // bit per cell: not solid and below 1 - 1e-4 at the tick's start
  unsigned pp[NGROUPS + 1];    // bit per unfinished cell that may find a start cell within the budget
  unsigned short gpre[NGROUPS + 1];  // att bits before each group of 32
  unsigned short list[2][LIST_CAP];
  unsigned cnt[3];             // list lengths, rotating: this round's, the next, the one being cleared
  unsigned cur, cc;            // the list and the counter of the next round
  unsigned park_n[2], pb;      // ready cells above the gate, and which parked list holds them
  unsigned kp;                 // positions from here on cannot pull (budget spent before them)
  unsigned nx;                 // full cells pulls took from (Region::pxlist)
  HeadState h;
  unsigned req, rounds, resume, timeout;
  unsigned n_succ, n_searches, n_again;
  unsigned long long n_entries;
  unsigned hard;               // the last long search found nothing: the next may well be hopeless
  unsigned flood_n[5];
  uint2 flood[2][16][32];      // search_hopeless: rows of its two floods
  Search s;
};

__device__ __forceinline__ unsigned vld(const unsigned* p) { return *(volatile const unsigned*)p; }
// A global word that only this CTA's threads write (grid words): a relaxed load at CTA scope. It is
// coherent with the CTA's stores and atomics but may be served by the SM's L1.
__device__ __forceinline__ unsigned gld(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.cta.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}

__device__ __forceinline__ CD load_cell_par(const Region& R, const int* ring, int x, int y, int z) {
  CD c;
  c.part = 0.0f;
  c.slot = NOSLOT;
  c.gi = 0;
  c.mat = 0;
  c.out = outside(R, ring, x, y, z);
  if (c.out) return c;
  c.gi = grid_index(R, x >> 3, y >> 3, z >> 3);
  const unsigned g = gld(R.grid + c.gi);
  if (g < 256u) {
    c.mat = (unsigned char)g;
    return c;
  }
  c.slot = g - 256u;
  const size_t o = (size_t)c.slot * 512u + local_index(x, y, z);
  c.mat = R.amat[o];
  c.part = R.avol[o];
  return c;
}

// Atlas slots for the bricks a CTA's threads are about to write first (sparse_volume.rs:250-266): bit q of
// `mask` names brick gi[q]. Slots are given out in the order of the writes (thread, then q), which is
// the program's order where the callers pass cells in it: whatever follows the slots' order (the rows
// of the proposal's features) is the same in every run. A brick goes to its first writer, found by an
// atomic minimum in the grid word itself. All threads; callers skip it when nothing is needed.
// (By value: a Region behind a reference would keep the caller's copy out of registers.)
struct AtlasRef {
  unsigned* grid;
  unsigned char* amat;
  float* avol;
  Ctl* ctl;
  unsigned atlas_cap;
};
template <int K>
__device__ __noinline__ void give_slots(AtlasRef R, unsigned mask, const unsigned (&gi)[K]) {
  __shared__ unsigned s_cnt[32], s_base;
  const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, nw = blockDim.x >> 5;
  static_assert(1024 * K <= 1 << 23, "keys fit the grid word");
  __syncthreads();  // nobody reads the grid any more
#pragma unroll
  for (int q = 0; q < K; ++q) {
    if (!((mask >> q) & 1u)) continue;
    unsigned* gp = R.grid + gi[q];
    unsigned g = __ldcg(gp);
    while (g < 256u || g >= GRID_CLAIM) {
      const unsigned mine = GRID_CLAIM | (tid * K + q) << 8 | (g & 255u);
      if (g >= GRID_CLAIM && g <= mine) break;
      const unsigned old = atomicCAS(gp, g, mine);
      if (old == g) break;
      g = old;
    }
  }
  __syncthreads();
  unsigned win = 0, fill[K];
#pragma unroll
  for (int q = 0; q < K; ++q) {
    fill[q] = 0;
    if (!((mask >> q) & 1u)) continue;
    const unsigned g = __ldcg(R.grid + gi[q]);
    if (g < GRID_CLAIM || (g & ~GRID_CLAIM) >> 8 != tid * K + q) continue;
    win |= 1u << q;
    fill[q] = g & 255u;
  }
  const unsigned k = (unsigned)__popc(win);
  unsigned pre = k;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned v = __shfl_up_sync(FULLMASK, pre, o);
    if (lane >= (unsigned)o) pre += v;
  }
  if (lane == 31u) s_cnt[warp] = pre;
  __syncthreads();
  const unsigned c = lane < nw ? s_cnt[lane] : 0u;
  const unsigned before = __reduce_add_sync(FULLMASK, lane < warp ? c : 0u), total = __reduce_add_sync(FULLMASK, c);
  if (tid == 0) s_base = atomicAdd(&R.ctl->atlas_used, total);
  __syncthreads();
  unsigned next = s_base + before + pre - k;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const bool w = (win >> q) & 1u;
    const unsigned s = w ? next++ : NOSLOT;
    const bool ok = w && s < R.atlas_cap;
    if (w && !ok) {
      if (atomicCAS(&R.ctl->status, 0, ST_OOM) == 0) R.ctl->err_info = 1;
      atomicExch(R.grid + gi[q], fill[q]);
    }
    for (unsigned m = __ballot_sync(FULLMASK, ok); m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const unsigned sl = __shfl_sync(FULLMASK, s, l);
      const unsigned fv = __shfl_sync(FULLMASK, fill[q], l) * 0x01010101u;
      reinterpret_cast<uint4*>(R.amat + (size_t)sl * 512u)[lane] = make_uint4(fv, fv, fv, fv);
      uint4* vv = reinterpret_cast<uint4*>(R.avol + (size_t)sl * 512u);
#pragma unroll
      for (int p = 0; p < 4; ++p) vv[lane + 32 * p] = make_uint4(0, 0, 0, 0);
    }
    if (ok) atomicExch(R.grid + gi[q], 256u + s);
  }
  __syncthreads();
}
// The same for one brick a thread, and the slot it got. All threads.
__device__ __forceinline__ void materialize_cta(const Region& R, bool need, unsigned gi, unsigned& slot) {
  if (!__syncthreads_or(need)) return;
  const unsigned a[1] = {gi};
  give_slots<1>(AtlasRef{R.grid, R.amat, R.avol, R.ctl, R.atlas_cap}, need ? 1u : 0u, a);
  if (need) {
    const unsigned g = __ldcg(R.grid + gi);
    slot = g >= 256u ? g - 256u : NOSLOT;
  }
}

// FluidSim::set_volume (fluid.rs:327-355) split into the decision and the stores.
struct SVPlan {
  float npart;
  unsigned char nmat;
  bool wpart, wmat, ch;
  int dp;
};
__device__ __forceinline__ SVPlan sv_plan(float part, unsigned char mat, bool has, float vol) {
  SVPlan p;
  const bool is_water = mat == WATER;
  const bool low = vol <= 1e-6f;
  const bool high = !low && vol >= full_level();
  const bool mid = !low && !high;
  const bool had = has && part > 0.0f;
  p.npart = mid ? vol : 0.0f;
  p.nmat = low ? (unsigned char)0
         : high ? (unsigned char)WATER
         : (is_water && vol < HIDE_BELOW) ? (unsigned char)0
         : (!is_water && vol >= SHOW_AT) ? (unsigned char)WATER
         : mat;
  p.wpart = has && (mid || had);
  p.wmat = has && p.nmat != mat;
  p.ch = mid ? p.wmat : p.nmat != mat;
  p.dp = ((mid && has && !had) ? 1 : 0) - ((!mid && had) ? 1 : 0);
  return p;
}
__device__ __forceinline__ void sv_apply(const Region& R, const CD& c, unsigned id, unsigned local, const SVPlan& p) {
  const size_t o = (size_t)c.slot * 512u + local;
  if (p.wpart) R.avol[o] = p.npart;
  if (p.wmat) R.amat[o] = p.nmat;
  dense_put(R, id, p.nmat, p.npart);
}

// Footprint slot offsets: 0 self, 1 below, 2 up, 3 +x, 4 -x, 5 +z, 6 -z.
__device__ __forceinline__ void fp_off(int l, int& ox, int& oy, int& oz) {
  ox = (l == 3) - (l == 4);
  oy = (l == 2) - (l == 1);
  oz = (l == 5) - (l == 6);
}
// The q-th (0..11) later position a cell conflicts with; s = +1, or -1 on odd ticks (whose order
// mirrors x and z). 0..5 lie on the cell's layer, 6..10 on the one above, 11 two above.
__device__ __forceinline__ void succ_offset(int q, int s, int& dx, int& dy, int& dz) {
  dx = q == 0 ? s : q == 1 ? 2 * s : q == 2 ? -1 : q == 4 ? 1 : q == 7 ? 1 : q == 8 ? -1 : 0;
  dy = q < 6 ? 0 : q < 11 ? 1 : 2;
  dz = (q >= 2 && q <= 4) ? s : q == 5 ? 2 * s : q == 9 ? 1 : q == 10 ? -1 : 0;
}

// ------------------------------------------------------------------------------- the lists
// A cell enters a list once and the parked list once, so neither outgrows the tick's cells; the bounds
// are checked all the same where an entry goes to global memory.
__device__ __forceinline__ unsigned list_get(const Region& R, const LvSmem& L, unsigned b, unsigned t) {
  return t < LIST_CAP ? L.list[b][t] : R.lv_over[(size_t)b * MAX_CELLS_PER_TICK + t];
}
__device__ __forceinline__ void list_put(const Region& R, LvSmem& L, unsigned b, unsigned t, unsigned i) {
  if (t < LIST_CAP) L.list[b][t] = (unsigned short)i;
  else if (t < MAX_CELLS_PER_TICK) R.lv_over[(size_t)b * MAX_CELLS_PER_TICK + t] = (unsigned short)i;
  else set_status(R, ST_RANGE, 51);
}
__device__ __forceinline__ void park_put(const Region& R, unsigned b, unsigned t, unsigned i) {
  if (t < MAX_CELLS_PER_TICK) R.lv_park[(size_t)b * MAX_CELLS_PER_TICK + t] = (unsigned short)i;
  else set_status(R, ST_RANGE, 52);
}
// Four cells' bytes share a word, and in a round of the CTA one warp finishes a cell while others count down its
// neighbours: there every access is to the whole word, and every change an atomic one (cell_done_now, cell_finish;
// bit_now for pp). Where nobody else is at work, warp 0 between rounds and code between barriers, bytes are read and
// written as such (words everywhere: +3% of the sweep's cycles, on warp 0's chain).
__device__ __forceinline__ unsigned dep_byte(const LvSmem& L, unsigned i) { return reinterpret_cast<const volatile unsigned char*>(L.dep)[i]; }
__device__ __forceinline__ bool cell_done(const LvSmem& L, unsigned i) { return dep_byte(L, i) >= DONE; }
__device__ __forceinline__ bool cell_done_now(const LvSmem& L, unsigned i) { return (vld(&L.dep[i >> 2]) >> ((i & 3u) * 8u)) & DONE; }
template <bool SOLO>
__device__ __forceinline__ void cell_finish(LvSmem& L, unsigned i, unsigned slots) {  // (the byte of a cell that runs is 0)
  if (SOLO) reinterpret_cast<volatile unsigned char*>(L.dep)[i] = (unsigned char)(DONE | slots);
  else atomicOr(&L.dep[i >> 2], (DONE | slots) << ((i & 3u) * 8u));
}
__device__ __forceinline__ bool bit_of(const unsigned* w, unsigned i) { return (w[i >> 5] >> (i & 31u)) & 1u; }
__device__ __forceinline__ bool bit_now(const unsigned* w, unsigned i) { return (vld(w + (i >> 5)) >> (i & 31u)) & 1u; }
// att bits before position i
__device__ __forceinline__ unsigned attempts_before(const LvSmem& L, unsigned i) {
  return (unsigned)L.gpre[i >> 5] + (unsigned)__popc(L.att[i >> 5] & ((1u << (i & 31u)) - 1u));
}

// -------------------------------------------------------------------------------- the cells
// Lane constants of the eight lanes that run a cell: lane l < 7 holds footprint slot l.
struct LaneSlot {
  int off;               // the slot's offset in domain ids
  unsigned end;          // cells from this position on leave the lane's slot unread: 0 for lane 7, and kp for the
                         // cell above, which only a cell that may pull looks at (another of the round may write it)
  unsigned open1, open2; // the lane's two successors: one layer up (bit per successor), two layers up
};
__device__ __forceinline__ int fp_id(const Region& R, int l) {
  int ox, oy, oz;
  fp_off(l, ox, oy, oz);
  return ox + (oz * R.PY + oy) * R.PX;
}
__device__ __forceinline__ LaneSlot lane_slot(const Region& R, unsigned kp) {
  const int l = (int)(threadIdx.x & 7u);
  LaneSlot s;
  s.off = l < 7 ? fp_id(R, l) : 0;
  s.end = l == 7 ? 0u : l == 2 ? kp : MAX_CELLS_PER_TICK;
  s.open1 = l == 3 || l == 4 ? 3u : l == 5 ? 1u : 0u;  // successors 6..10
  s.open2 = l == 5 ? 2u : 0u;                          // successor 11
  return s;
}

// What a lane holds of its cell: fetched in two steps, so that a long list's next cells travel while the
// warp runs the ones before (cells of a round do not touch each other's footprints).
struct LaneCell {
  bool has;
  unsigned i, w;  // sorted position, the lane's word of the record
  uint2 ce;       // cid, ye
  unsigned u;     // the lane's slot
};
__device__ __forceinline__ LaneCell cell_record(const Region& R, bool has, unsigned i) {
  LaneCell c{has, i, 0xFFFFFFFFu, make_uint2(0u, 0u), DC_SOLID};
  if (has) {
    c.w = reinterpret_cast<const unsigned*>(R.lv + i)[threadIdx.x & 7u];
    c.ce = reinterpret_cast<const uint2*>(R.lv + i)[3];
  }
  return c;
}
__device__ __forceinline__ void cell_slot(const Region& R, const LaneSlot& S, LaneCell& c) {
  if (c.has && c.i < S.end) c.u = R.dense[(int)c.ce.x + S.off];
}

// A lone warp touches its cells' successors' records, some of which it runs next: they come from L2 (~850
// cycles) while it works (the prefetch instruction to L1 does nothing here). What was read is looked at
// in the next call, when it has long arrived.
struct Touch {
  unsigned a = 0, b = 0, seen = 0;  // domain ids: below 2^31
};

// Four cells at sorted positions i (fluid.rs:584-651), eight lanes each, warp-collective (groups
// without a cell: `has` false). `pulled`: the cell's pull has run and took `got` (event bits `ev`);
// otherwise a cell with a start cell is left for its pull (lv_solo). Ready successors join list nb or, above
// the gate, parked list pb; their counts are the caller's registers (SOLO: no other warp runs) or
// L.cnt[nc] and L.park_n[pb]. Returns the cell's volume afterwards.
//
// Eight lanes rather than one thread per cell: a round is a latency chain (a few dozen to a few
// hundred cells on 16 warps), and a lane that holds one slot issues one load, one set_volume and two
// successor counts where a thread issues seven, six and twelve. A lone warp takes ~8 cycles for every
// dependent instruction, so what counts is their number and that the counts and the volumes travel
// together: the code is one straight line, and successors are counted down before the volumes are
// looked at (nobody reads the next list before the round has ended). The sweep writes the dense words only;
// sweep_flush brings the atlas in step.
template <bool SOLO>
__device__ __forceinline__ float lv_cells(const Region& R, LvSmem& L, const LaneSlot& S, const LaneCell& c, bool pulled, float got, unsigned ev, int gate,
                                          unsigned kp, unsigned nb, unsigned nc, unsigned& cnt, unsigned pb, unsigned& park, Touch& T, int& pd) {
  const float FULL = full_level();
  const unsigned lane = lane_id(), l = lane & 7u, base = lane & 24u;
  const unsigned i = c.i, w = c.w, u = c.u;
  const uint2 ce = c.ce;
  bool has = c.has;
  const bool pp = has && i < kp && (SOLO ? bit_of(L.pp, i) : bit_now(L.pp, i));
  const int y = (int)(ce.y & YE_Y), at = (int)ce.x + S.off;
  // ---- a cell that attempts a pull and has a start cell waits for the pull
  if (__any_sync(FULLMASK, pp && !pulled)) {
    const float v = dc_volume(u);
    const unsigned starts = (__ballot_sync(FULLMASK, l >= 2u && l < 7u && ((ce.y >> (25u + l)) & 1u) && !dc_solid(u) && v >= FULL) >> base) & 0xFFu;
    const float self = __shfl_sync(FULLMASK, v, 0, 8);
    if (!pulled && pp && self < FULL && starts) has = false;
  }
  // ---- successors whose last earlier cell this was
  const unsigned a = w & 0xFFFFu, b = w >> 16, sa = (a & 3u) * 8u, sb = (b & 3u) * 8u;
  const bool cnts = has && l < 6u;
  unsigned oa = 0, ob = 0;
  if (cnts && a != NOSUCC) oa = atomicSub(&L.dep[a >> 2], 1u << sa);
  if (cnts && b != NOSUCC) ob = atomicSub(&L.dep[b >> 2], 1u << sb);
  {
    T.seen |= T.a | T.b;
    if (cnts && a != NOSUCC) T.a = R.lv[a].cid;
    if (cnts && b != NOSUCC) T.b = R.lv[b].cid;
  }
  // ---- 1. fall into the free capacity below, 2. share with lower sides when supported, 3. evaporate
  // crumbs (fluid.rs:606-650). Every side's flow depends on the volume after the fall and its own
  // volume only; the running volume subtracts the flows in side order (a side without one: 0).
  const bool solid = dc_solid(u);
  const float v = solid ? 0.0f : dc_volume(u);
  const float v0 = __shfl_sync(FULLMASK, v, 0, 8), bv = __shfl_sync(FULLMASK, v, 1, 8);
  const bool below_solid = (__ballot_sync(FULLMASK, solid) >> (base + 1u)) & 1u;
  float vol = pulled && got > 0.0f ? __fadd_rn(v0, got) : v0;
  const bool live = has && vol > 0.0f;  // fluid.rs:602-604
  const float ff = fminf(vol, __fsub_rn(1.0f, bv));
  const bool w_below = live && !below_solid && ff > 1e-6f;
  const float below_new = __fadd_rn(bv, ff);
  vol = w_below ? __fsub_rn(vol, ff) : vol;
  const float below_after = w_below ? (below_new >= FULL ? 1.0f : below_new) : bv;
  const bool spread = live && vol > MIN_SPREAD && (below_solid || below_after >= FULL);
  const float f = __fmul_rn(__fsub_rn(vol, v), 0.2f);
  const bool ok = spread && l >= 3u && !solid && !(v >= vol) && !(f < MIN_FLOW) && !(__fsub_rn(vol, f) < MIN_SPREAD * 0.5f);
  const float fs = ok ? f : 0.0f;
  const float f3 = __shfl_sync(FULLMASK, fs, 3, 8), f4 = __shfl_sync(FULLMASK, fs, 4, 8);
  const float f5 = __shfl_sync(FULLMASK, fs, 5, 8), f6 = __shfl_sync(FULLMASK, fs, 6, 8);
  vol = __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(vol, f3), f4), f5), f6);
  vol = vol < EVAPORATE ? 0.0f : vol;
  const float dv = fabsf(__fsub_rn(vol, v0));
  // ---- set_volume of the lane's cell (fluid.rs:327-355): snapped to 0 or full the entry goes; water
  // shows from 0.5 and hides below 0.3 (a snapped volume lies on the same side of both)
  const bool wr = l == 0u ? (live && dv > 1e-7f) : l == 1u ? w_below : ok;
  const float wv = l == 0u ? vol : l == 1u ? below_new : __fadd_rn(v, f);
  const bool is_water = (int)u > 0, mid = wv > 1e-6f && wv < FULL, had = v > 0.0f && v < 1.0f;
  const bool wet = wv >= (is_water ? HIDE_BELOW : SHOW_AT);
  const unsigned nu = mid ? (__float_as_uint(wv) | (wet ? 0u : DC_AIR)) : (wet ? DC_FULL : 0u);
  const bool put = wr && nu != u;
  if (put) R.dense[at] = nu;
  pd += put ? (mid ? 1 : 0) - (had ? 1 : 0) : 0;
  if (has && y == gate) R.lv_old[i].vol[l] = v;
  const unsigned pm = __ballot_sync(FULLMASK, put) >> base;
  const unsigned cm = __ballot_sync(FULLMASK, put && wet != is_water) >> base;
  // activation slots: 2 below, 3..6 the sides, 7 the cell itself
  const unsigned am = __ballot_sync(FULLMASK, l == 2u ? w_below : l == 7u ? live && dv > SLEEP : ok && f > SLEEP) >> base;
  // ---- the ready ones to the next list, or parked above the gate
  const bool r0 = ((oa >> sa) & 0xFFu) == 1u, r1 = ((ob >> sb) & 0xFFu) == 1u;
  const unsigned shut = (y + 1 > gate ? S.open1 : 0u) | (y + 2 > gate ? S.open2 : 0u);
  const bool p0 = r0 && !(shut & 1u), p1 = r1 && !(shut & 2u);
  const unsigned g0 = __ballot_sync(FULLMASK, p0), g1 = __ballot_sync(FULLMASK, p1);
  const unsigned h0 = __ballot_sync(FULLMASK, r0 && !p0), h1 = __ballot_sync(FULLMASK, r1 && !p1);
  if (g0 | g1) {
    const unsigned k = (unsigned)(__popc(g0) + __popc(g1));
    unsigned t = cnt;
    if (SOLO) {
      cnt += k;
    } else {
      if (lane == 0u) t = atomicAdd(&L.cnt[nc], k);
      t = __shfl_sync(FULLMASK, t, 0);
    }
    const unsigned t0 = t + (unsigned)__popc(g0 & lanemask_lt()), t1 = t + (unsigned)(__popc(g0) + __popc(g1 & lanemask_lt()));
    if (t + k <= LIST_CAP) {
      if (p0) L.list[nb][t0] = (unsigned short)a;
      if (p1) L.list[nb][t1] = (unsigned short)b;
    } else {
      if (p0) list_put(R, L, nb, t0, a);
      if (p1) list_put(R, L, nb, t1, b);
    }
  }
  if (h0 | h1) {
    const unsigned k = (unsigned)(__popc(h0) + __popc(h1));
    unsigned t = park;
    if (SOLO) {
      park += k;
    } else {
      if (lane == 0u) t = atomicAdd(&L.park_n[pb], k);
      t = __shfl_sync(FULLMASK, t, 0);
    }
    if (r0 && !p0) park_put(R, pb, t + (unsigned)__popc(h0 & lanemask_lt()), a);
    if (r1 && !p1) park_put(R, pb, t + (unsigned)(__popc(h0) + __popc(h1 & lanemask_lt())), b);
  }
  if (SOLO) __syncwarp();  // the counts are down before a byte beside them is written
  if (has && l == 0u) {
    R.lv_ev[i] = ev | (am & 0xFCu) | ((am & 0x80u) << 9) | ((cm & 0x7Fu) << 8);  // bit 16: seeds itself
    cell_finish<SOLO>(L, i, pm & 0x7Fu);
    if (pp) atomicAnd(&L.pp[i >> 5], ~(1u << (i & 31u)));
  }
  __syncwarp();
  return vol;
}

// The same for a long list, one thread per cell, warp-collective: a warp's instructions then serve 32
// cells instead of four, and it is the number of instructions that bounds a round of hundreds of cells
// (the chain of one thread, twelve counts and seven cells, is longer: rounds of fewer than THREAD_CELLS take
// eight lanes).
constexpr unsigned THREAD_CELLS = 192;  // lake: 5.1 M cycles of rounds from 192 on, 6.0 from 256 on, 5.9 without; ring rain 7.9 against 14.4
__device__ __forceinline__ void lv_cell_thread(const Region& R, LvSmem& L, bool has, unsigned i, int gate, unsigned kp, unsigned nb, unsigned nc, unsigned pb,
                                               int& pd) {
  const float FULL = full_level();
  const unsigned lane = lane_id();
  uint4 ra = make_uint4(~0u, ~0u, ~0u, ~0u), rb = make_uint4(~0u, ~0u, 0u, 0u);
  if (has) {
    ra = reinterpret_cast<const uint4*>(R.lv + i)[0];
    rb = reinterpret_cast<const uint4*>(R.lv + i)[1];
  }
  const unsigned w[6] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y}, ye = rb.w;
  const int cid = (int)rb.z, y = (int)(ye & YE_Y);
  const bool pp = has && i < kp && bit_now(L.pp, i);
  unsigned u[7];
#pragma unroll
  for (int l = 0; l < 7; ++l) {
    u[l] = DC_SOLID;
    if (l == 2 ? pp : has) u[l] = R.dense[cid + fp_id(R, l)];
  }
  if (pp && dc_volume(u[0]) < FULL) {  // a cell that attempts a pull and has a start cell waits for the pull
    bool start = false;
#pragma unroll
    for (int l = 2; l < 7; ++l) start |= ((ye >> (25 + l)) & 1u) && !dc_solid(u[l]) && dc_volume(u[l]) >= FULL;
    if (start) has = false;
  }
  // ---- successors whose last earlier cell this was (succ_offset's order: 6..10 one layer up, 11 two)
  unsigned ready = 0;
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    const unsigned a = (q & 1) ? w[q >> 1] >> 16 : w[q >> 1] & 0xFFFFu, sh = (a & 3u) * 8u;
    unsigned o = 0;
    if (has && a != NOSUCC) o = atomicSub(&L.dep[a >> 2], 1u << sh);
    ready |= ((o >> sh) & 0xFFu) == 1u ? 1u << q : 0u;
  }
  // ---- the rules, as in lv_cells
  const float v0 = dc_volume(u[0]);
  const bool below_solid = dc_solid(u[1]);
  const float bv = below_solid ? 0.0f : dc_volume(u[1]);
  float vol = v0;
  const bool live = has && vol > 0.0f;
  const float ff = fminf(vol, __fsub_rn(1.0f, bv));
  const bool w_below = live && !below_solid && ff > 1e-6f;
  const float below_new = __fadd_rn(bv, ff);
  vol = w_below ? __fsub_rn(vol, ff) : vol;
  const float below_after = w_below ? (below_new >= FULL ? 1.0f : below_new) : bv;
  const bool spread = live && vol > MIN_SPREAD && (below_solid || below_after >= FULL);
  float wv[7], v[7], run = vol;
  bool wr[7];
  unsigned am = w_below ? 4u : 0u;
#pragma unroll
  for (int l = 3; l < 7; ++l) {
    const bool solid = dc_solid(u[l]);
    v[l] = solid ? 0.0f : dc_volume(u[l]);
    const float f = __fmul_rn(__fsub_rn(vol, v[l]), 0.2f);
    wr[l] = spread && !solid && !(v[l] >= vol) && !(f < MIN_FLOW) && !(__fsub_rn(vol, f) < MIN_SPREAD * 0.5f);
    wv[l] = __fadd_rn(v[l], f);
    run = __fsub_rn(run, wr[l] ? f : 0.0f);
    am |= wr[l] && f > SLEEP ? 1u << l : 0u;
  }
  run = run < EVAPORATE ? 0.0f : run;
  const float dv = fabsf(__fsub_rn(run, v0));
  am |= live && dv > SLEEP ? 0x80u : 0u;
  v[0] = v0;
  v[1] = bv;
  wr[0] = live && dv > 1e-7f;
  wv[0] = run;
  wr[1] = w_below;
  wv[1] = below_new;
  unsigned pm = 0, cm = 0;
#pragma unroll
  for (int l = 0; l < 7; ++l) {
    if (l == 2) continue;
    const bool is_water = (int)u[l] > 0, mid = wv[l] > 1e-6f && wv[l] < FULL, had = v[l] > 0.0f && v[l] < 1.0f;
    const bool wet = wv[l] >= (is_water ? HIDE_BELOW : SHOW_AT);
    const unsigned nu = mid ? (__float_as_uint(wv[l]) | (wet ? 0u : DC_AIR)) : (wet ? DC_FULL : 0u);
    if (wr[l] && nu != u[l]) {
      R.dense[cid + fp_id(R, l)] = nu;
      pd += (mid ? 1 : 0) - (had ? 1 : 0);
      pm |= 1u << l;
      cm |= wet != is_water ? 1u << l : 0u;
    }
  }
  if (has && y == gate) {  // (a search asks for slots 0 and 3..6)
    float4* o = reinterpret_cast<float4*>(R.lv_old + i);
    o[0] = make_float4(v[0], v[1], 0.0f, v[3]);
    o[1] = make_float4(v[4], v[5], v[6], 0.0f);
  }
  if (has) {
    R.lv_ev[i] = (am & 0xFCu) | ((am & 0x80u) << 9) | cm << 8;
    cell_finish<false>(L, i, pm);
    if (pp) atomicAnd(&L.pp[i >> 5], ~(1u << (i & 31u)));
  }
  // ---- the ready ones to the next list, or parked above the gate: places by a scan over the warp
  const unsigned shut = (y + 1 > gate ? 0x7C0u : 0u) | (y + 2 > gate ? 0x800u : 0u), go = ready & ~shut, stay = ready & shut;
  const unsigned both = (unsigned)__popc(go) | (unsigned)__popc(stay) << 16;
  unsigned pre = both;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned x = __shfl_up_sync(FULLMASK, pre, o);
    if (lane >= (unsigned)o) pre += x;
  }
  unsigned t = 0, p = 0;
  if (lane == 31u) {
    if (pre & 0xFFFFu) t = atomicAdd(&L.cnt[nc], pre & 0xFFFFu);
    if (pre >> 16) p = atomicAdd(&L.park_n[pb], pre >> 16);
  }
  t = __shfl_sync(FULLMASK, t, 31) + ((pre - both) & 0xFFFFu);
  p = __shfl_sync(FULLMASK, p, 31) + ((pre - both) >> 16);
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    const unsigned a = (q & 1) ? w[q >> 1] >> 16 : w[q >> 1] & 0xFFFFu;
    if ((go >> q) & 1u) list_put(R, L, nb, t++, a);
    if (q >= 6 && ((stay >> q) & 1u)) park_put(R, pb, p++, a);
  }
  __syncwarp();
}

// After the sweep: every cell it wrote (the slots in the dependency bytes, the pulls' sources) to the
// atlas, all at once, in batches of one drained cell per thread in sorted order. Bricks written for
// the first time get their slots in the program's order (a pull's source before its cell). All threads.
__device__ __forceinline__ void sweep_flush(const Region& R, const LvSmem& L, unsigned n) {
  for (unsigned base = 0; base < n; base += blockDim.x) {
    const unsigned i = base + threadIdx.x;
    unsigned w = 0, need = 0;  // entry 0: the source, 1 + l: slot l (never 2, the cell above)
    unsigned gi[8], g[8], u[8], at[8];  // brick, its grid word, the dense word, the cell in its brick
    if (i < n) {
      w = (dep_byte(L, i) & 0x7Fu) << 1 | (R.lv_ev[i] & 1u);
      if (w) {
        const unsigned cid = R.lv[i].cid, sid = (w & 1u) ? R.lv_src[i] : cid;
        int x, y, z;
        dom_xyz(R, cid, x, y, z);
        const unsigned gc = grid_index(R, x >> 3, y >> 3, z >> 3), gw = gld(R.grid + gc);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          if (q == 3 || !((w >> q) & 1u)) continue;
          int ax, ay, az;
          unsigned id = sid;
          if (q == 0) {
            dom_xyz(R, sid, ax, ay, az);
          } else {
            fp_off(q - 1, ax, ay, az);
            id = (unsigned)((int)cid + fp_id(R, q - 1));
            ax += x;
            ay += y;
            az += z;
          }
          u[q] = R.dense[id];
          gi[q] = gc;
          g[q] = gw;
          if (((ax ^ x) | (ay ^ y) | (az ^ z)) & ~7) {  // another brick
            gi[q] = grid_index(R, ax >> 3, ay >> 3, az >> 3);
            g[q] = gld(R.grid + gi[q]);
          }
          at[q] = local_index(ax, ay, az);
          need |= g[q] < 256u ? 1u << q : 0u;
        }
      }
    }
    if (__syncthreads_or(need != 0u)) {
      unsigned a[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = gi[q];
      give_slots<8>(AtlasRef{R.grid, R.amat, R.avol, R.ctl, R.atlas_cap}, need, a);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if ((need >> q) & 1u) g[q] = __ldcg(R.grid + gi[q]);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (q == 3 || !((w >> q) & 1u) || g[q] < 256u) continue;  // (no slot left: the status says so)
      const size_t o = (size_t)(g[q] - 256u) * 512u + at[q];
      const float v = dc_volume(u[q]);
      R.avol[o] = v < 1.0f ? v : 0.0f;
      R.amat[o] = (int)u[q] > 0 ? WATER : (unsigned char)0;
    }
  }
}

// --------------------------------------------------------------------------- pressure search
__device__ __forceinline__ unsigned vis_slot(Search& C, unsigned key) {
  unsigned h = (key * 2654435761u) >> VIS_SHIFT;
  while (true) {
    const unsigned old = atomicCAS(&C.vkey[h], EMPTY_ID, key);
    if (old == EMPTY_ID || old == key) return h;
    h = (h + 1u) & (VIS_SLOTS - 1u);
  }
}

// The set empty and the rank base at its top; by the threads of one warp or of the CTA.
__device__ __forceinline__ void vis_reset(Search& C, unsigned t0, unsigned nt) {
  for (unsigned t = t0; t < VIS_SLOTS; t += nt) {
    C.vkey[t] = EMPTY_ID;
    C.vrank[t] = 0xFFFFFFFFu;
  }
  if (t0 == 0u) {
    C.rank0 = 0xFFFFFFFFu - VIS_RANKS;
    C.nvis = 0u;
  }
}

// The volume a cell of the pulling layer holds at the turn of the cell at position k, given the volume
// `v` it holds now and the positions j of its writers (itself, and the cells it is a side of): later
// ones that already ran and wrote it are looked through (the earliest such write's old value); an
// unfinished earlier writer is reported in blk.
__device__ __forceinline__ float old_volume(const Region& R, const LvSmem& L, unsigned k, const unsigned (&j)[5], float v, unsigned& blk) {
  unsigned best = NOSLOT, slot = 0u;
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const unsigned fl = q == 0 ? 0u : q + 2u;
    const unsigned b = j[q] != NOSLOT ? dep_byte(L, j[q]) : DONE;
    if (j[q] < k && b < DONE) blk = max(blk, j[q] + 1u);
    if (j[q] > k && b >= DONE && ((b >> fl) & 1u) && j[q] < best) {
      best = j[q];
      slot = fl;
    }
  }
  return best != NOSLOT ? R.lv_old[best].vol[slot] : v;
}

// The direction d of a search round's lane: up, +x, -x, +z, -z (none for lanes 30 and 31).
struct SearchLane {
  int off;        // its step in domain ids
  bool up, neg;   // d = 0; negative coordinates have to be looked for (fluid.rs:542): a ring world's only
};
__device__ __forceinline__ SearchLane search_lane(const Region& R, unsigned d) {
  const int row = R.PX * R.PY;
  return SearchLane{d == 0u ? R.PX : d == 1u ? 1 : d == 2u ? -1 : d == 3u ? row : -row, d == 0u, R.ring_w && (R.px0 < 0 || R.pz0 < 0)};
}
// What a search round's thread finds: its queue entry's neighbour. blk: 1 + an unfinished earlier cell
// that what it read depends on (0: none).
struct SearchRead {
  unsigned key;  // the neighbour's queue key
  float here, v;
  bool win, cand, side;
  unsigned blk;
};
__device__ __forceinline__ SearchRead search_read(const Region& R, const LvSmem& L, const SearchLane& D, bool act, unsigned e, bool sides) {
  const Search& C = L.s;
  const uint2 q = C.q[act ? e : 0u];  // (a lane without an entry looks at the first one's neighbour for nothing)
  SearchRead r;
  const int id = (int)(q.x & ~ABOVE) + D.off;  // the neighbours of a cell of the world lie inside the padded domain
  const bool above0 = q.x >= ABOVE, above = above0 || D.up;
  r.key = (unsigned)id | (above ? ABOVE : 0u);
  r.here = __uint_as_float(q.y);
  r.blk = 0u;
  // Once the 24 side checks at the start level are spent, what its cells hold no longer matters.
  bool rd = act && (sides || above);
  const unsigned u = R.dense[id];
  r.v = dc_volume(u);
  if (D.neg) {
    int x, y, z;
    dom_xyz(R, (unsigned)id, x, y, z);
    rd = rd && (D.up || (x >= 0 && z >= 0));
  }
  const bool level = rd && !above && !dc_solid(u);
  if (__any_sync(FULLMASK, level)) {
    if (level) {
      const unsigned* st = R.stamp + id;
      const int row = R.PX * R.PY;
      const unsigned j[5] = {st[0], st[-1], st[1], st[-row], st[row]};
      r.v = old_volume(R, L, C.pos, j, r.v, r.blk);
    }
  }
  // the surface test of the entry on its up neighbour (fluid.rs:534-535), else an expansion
  r.cand = rd && !dc_solid(u) && r.v > 0.0f;
  r.win = act && D.up && !r.cand && above0 && r.here > 0.0f;
  r.side = r.cand && !above;
  return r;
}

__device__ __forceinline__ void search_won(Search& C, const SearchRead& r, unsigned e) {
  C.skey = C.q[e].x;
  C.here = r.here;
  C.got = fminf(__fsub_rn(1.0f, C.vol), r.here);
  C.status = SS_SUCCESS;
  C.i = e + 1u;
}

// FluidSim::pressure_pull (fluid.rs:511-561) of the cell at position k: its start, by one warp. Writes
// nothing but L.s. A search examines at most 24 sides on its own layer, so nearly all it reads there is
// written by the cells within three rows and columns: `wait` gets 1 + the last unfinished earlier one
// of them (0: none), one probe per lane instead of a search that finds out. Returns whether there is
// anything to examine.
__device__ __forceinline__ bool search_begin(const Region& R, LvSmem& L, const LaneSlot& S, unsigned k, int sgn, unsigned& wait) {
  Search& C = L.s;
  const float FULL = full_level();
  const unsigned lane = lane_id();
  const unsigned cid = R.lv[k].cid, ye = R.lv[k].ye;
  // lanes 0..20: the three rows before, x - 3 .. x + 3; 21..23: the three cells before in the row
  const int row = (int)lane / 7, ndx = lane < 21u ? (int)lane - 7 * row - 3 : -sgn * ((int)lane - 20);
  const int ndz = lane < 21u ? -sgn * (row + 1) : 0;
  unsigned near = NOSLOT, u = DC_SOLID;
  if (lane < 24u) near = R.stamp[(int)cid + ndx + ndz * R.PX * R.PY];
  if (lane < 7u) u = R.dense[(int)cid + S.off];
  const float v = dc_solid(u) ? 0.0f : dc_volume(u);
  wait = __reduce_max_sync(FULLMASK, near != NOSLOT && !cell_done(L, near) ? near + 1u : 0u);
  if (wait) return false;
  const float vol = __shfl_sync(FULLMASK, v, 0);
  unsigned starts = (__ballot_sync(FULLMASK, lane >= 2u && lane < 7u && ((ye >> (25u + lane)) & 1u) && v >= FULL) >> 2) & 31u;
  unsigned before = attempts_before(L, k);
  if (before + L.nx >= MAX_PULLS_PER_TICK) {  // near the budget: the cells before this one that pulls took below full
    unsigned c = 0;
    for (unsigned t = lane; t < L.nx; t += 32u) c += R.pxlist[t] < k ? 1u : 0u;
    before += __reduce_add_sync(FULLMASK, c);
  }
  if (!(vol < FULL) || before >= MAX_PULLS_PER_TICK) starts = 0u;
  if (starts && (C.nvis > VIS_FULL || C.rank0 < VIS_RANKS)) {
    vis_reset(C, lane, 32u);
    __syncwarp();
  }
  const unsigned rank0 = C.rank0 - VIS_RANKS;
  __syncwarp();
  if (lane == 0) {
    C.pos = k;
    C.status = SS_NONE;
    C.blk = 0u;
    C.i = 0u;
    C.side = 0u;
    C.qlen = (unsigned)__popc(starts);
    C.vol = vol;
    C.got = 0.0f;
    C.cid = cid;
    if (starts) {
      C.rank0 = rank0;
      C.nvis += 6u;
    }
  }
  if (starts) {
    // the start cells in direction order; visited ranks 0 (the cell itself), 1..5
    const unsigned d = lane - 2u;
    const bool st = lane >= 2u && lane < 7u && ((starts >> d) & 1u);
    if (st || lane == 0u) {
      const unsigned key = (unsigned)((int)cid + S.off) | (lane == 2u ? ABOVE : 0u);  // (slot 0: the cell)
      C.vrank[vis_slot(C, key)] = rank0 + (st ? d + 1u : 0u);
      if (st) {
        const unsigned p = (unsigned)__popc(starts & ((1u << d) - 1u));
        C.q[p] = make_uint2(key, __float_as_uint(v));
      }
    }
  }
  __syncwarp();
  return starts != 0u;
}

// Search rounds by one warp, SOLO_ENTRIES queue entries each, one neighbour per lane, the reference's
// queue order kept exactly: the first surface entry in queue order wins; the 24 side checks at the
// start level are counted in (entry, direction) order; a cell several lanes find belongs to the
// earliest. Ends with C.status, or SS_MORE when many entries wait (all warps take over).
__device__ __forceinline__ void search_solo(const Region& R, LvSmem& L) {
  Search& C = L.s;
  const unsigned lane = lane_id(), j = lane / 5u, d = lane - 5u * j;
  const SearchLane D = search_lane(R, d);
  unsigned i = C.i, qlen = C.qlen, side = C.side, status = SS_NONE, nvis = 0u;
  const unsigned rank0 = C.rank0 + 6u;
  while (i < qlen) {
    if (qlen - i > SOLO_WAIT || qlen + 5u * SOLO_ENTRIES > PRESSURE_SEARCH) {
      status = SS_MORE;
      break;
    }
    const unsigned kk = min(SOLO_ENTRIES, qlen - i);
    const SearchRead r = search_read(R, L, D, j < kk, i + j, side < 24u);
    if (__any_sync(FULLMASK, r.blk != 0u)) {  // an earlier cell has yet to write what the search read: run it again later
      const unsigned blk = __reduce_max_sync(FULLMASK, r.blk);
      if (lane == 0) C.blk = blk;
      status = SS_BLOCKED;
      break;
    }
    const unsigned wm = __ballot_sync(FULLMASK, r.win);
    if (wm) {
      const unsigned wl = (unsigned)__ffs(wm) - 1u;
      if (lane == wl) {
        search_won(C, r, i + j);
        C.nvis += nvis;
      }
      __syncwarp();
      return;
    }
    const unsigned sm = __ballot_sync(FULLMASK, r.side);
    const bool cand = r.cand && !(r.side && side + (unsigned)__popc(sm & lanemask_lt()) + 1u > 24u);
    side += (unsigned)__popc(sm);
    const unsigned rank = rank0 + (i + j) * 5u + d;
    unsigned h = 0;
    if (cand) {
      h = vis_slot(C, r.key);
      atomicMin(&C.vrank[h], rank);
    }
    __syncwarp();
    const bool isnew = cand && vld(&C.vrank[h]) == rank;
    const unsigned nm = __ballot_sync(FULLMASK, isnew);
    const unsigned pos = qlen + (unsigned)__popc(nm & lanemask_lt());
    if (isnew && pos < PRESSURE_SEARCH) C.q[pos] = make_uint2(r.key, __float_as_uint(r.v));
    qlen += (unsigned)__popc(nm);
    nvis += (unsigned)__popc(nm);
    i += kk;
    __syncwarp();
  }
  if (lane == 0) {
    C.status = status;
    C.i = i;
    C.qlen = qlen;
    C.side = side;
    C.nvis += nvis;
  }
  __syncwarp();
}

// Is the search hopeless, that is, certain to examine its 512 entries and find no surface? In deep water
// nearly every search is, and in queue order it takes ~9 rounds to find out (~19,000 cycles of the CTA); counting
// takes no order. Two floods from the start cells over bit masks of the surroundings, one step at a time:
//   sup  every cell that can be queued within s steps (on the pulling layer: every cell not solid);
//   sub  cells above the layer that are sure to be queued within s steps.
// The queue is in order of steps, so with 512 cells in sub and no surface cell in sup, the first 512
// entries, all that a search examines (fluid.rs:530), hold no surface. Warp = layer dy above the pulling
// one, lane = row dz + 16, bit = dx + 16. What lies beyond the rows loaded (|dz| + dy <= 14) counts as dry:
// reached within 13 steps it makes the cell below it a surface, which is the safe side. True: hopeless.
// All threads of a CTA of 16 warps; ends with a barrier. ~7,000 cycles.
// It is asked after a search that examined 512 entries for nothing, until it says no: regions of 50% size, 32 of
// them, 206 -> 174 ms (asked for 4,557 of the busiest
// region's 5,651 searches, 4,071 times yes), with edits 248 -> 223 (4,352 of 8,780, 3,949); a quarter dam asks 3 times.
constexpr int FLOOD_STEPS = 13;  // 9 steps hold 670 cells of open water; a corner of it takes a few more
__device__ __noinline__ bool search_hopeless(const Region& Rs, LvSmem& L) {
  const Region R = Rs;
  const Search& C = L.s;
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const int dy = (int)warp, row = R.PX * R.PY, cid = (int)C.cid;
  unsigned* rows = reinterpret_cast<unsigned*>(L.flood);  // water masks [dy][dz + 16]
  int x, y, z;
  dom_xyz(R, C.cid, x, y, z);
  const bool in_x = (unsigned)(x - R.px0 + (int)lane - 16) < (unsigned)R.PX;
  rows[tid] = 0u;
  if (tid < 5u) L.flood_n[tid] = 0u;
  // rows of layers 1..14, 27 - 2 (dy - 1) of them each: layers p + 1 and 14 - p share 28; then 27 rows of the
  // pulling layer. All of a warp's loads are under way before the first is looked at.
  constexpr int MINE = (196 + 27 + 15) / 16;
  unsigned u[MINE];
  int slot[MINE];
#pragma unroll
  for (int k = 0; k < MINE; ++k) {
    const unsigned m = warp + 16u * k;
    const int p = (int)(m / 28u), r = (int)(m % 28u), n0 = 27 - 2 * p;
    const int ly = m >= 196u ? 0 : r < n0 ? p + 1 : 14 - p;
    const int dz = m >= 196u ? (int)m - 196 - 13 : r < n0 ? r - (13 - p) : r - n0 - p;
    const bool in = in_x && m < 196u + 27u && (unsigned)(y + ly) < (unsigned)R.PY && (unsigned)(z - R.pz0 + dz) < (unsigned)R.PZ;
    slot[k] = m < 196u + 27u ? ly * 32 + dz + 16 : -1;
    u[k] = DC_SOLID;
    if (in) u[k] = R.dense[cid + (int)lane - 16 + (dz * R.PY + ly) * R.PX];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < MINE; ++k) {
    const unsigned b = __ballot_sync(FULLMASK, !dc_solid(u[k]) && (slot[k] < 32 || dc_volume(u[k]) > 0.0f));
    if (lane == 0u && slot[k] >= 0) rows[slot[k]] = b;
  }
  __syncthreads();
  const unsigned wet = rows[tid], over = warp < 15u ? rows[tid + 32u] : 0u;
  const unsigned surface = warp ? wet & ~over : 0u;
  unsigned sup = 0u, sub = 0u, late = 0u;  // late: sure to be queued by the first step
  for (unsigned e = 0; e < C.qlen; ++e) {  // at most five start cells
    const int d = (int)(C.q[e].x & ~ABOVE) - cid;
    const int sx = d == 1 ? 1 : d == -1 ? -1 : 0, sz = d == row ? 1 : d == -row ? -1 : 0, sy = (sx | sz) ? 0 : 1;
    if ((int)lane - 16 != sz) continue;
    const unsigned bit = 1u << (16 + sx);
    if (dy == sy) sup |= bit;
    if (dy == 1) (sy ? sub : late) |= bit;
  }
  __syncthreads();
  bool found = false;
  for (int s = 1; s <= FLOOD_STEPS; ++s) {
    L.flood[s & 1][dy][lane] = make_uint2(sup, sub);
    __syncthreads();
    const uint2 under = dy ? L.flood[s & 1][dy - 1][lane] : make_uint2(0u, 0u);
    const unsigned pu = __shfl_up_sync(FULLMASK, sup, 1), pd = __shfl_down_sync(FULLMASK, sup, 1);
    const unsigned bu = __shfl_up_sync(FULLMASK, sub, 1), bd = __shfl_down_sync(FULLMASK, sub, 1);
    sup = (sup | sup << 1 | sup >> 1 | pu | pd | under.x) & wet;
    sub = (sub | sub << 1 | sub >> 1 | bu | bd | under.y | late) & wet;
    if (s >= 9) {
      const unsigned n = __reduce_add_sync(FULLMASK, (unsigned)__popc(sub));
      if (lane == 0u) atomicAdd(&L.flood_n[s - 9], n);
      if (__syncthreads_or((sup & surface) != 0u)) break;
      if (L.flood_n[s - 9] >= PRESSURE_SEARCH) {
        found = true;
        break;
      }
    }
  }
  __syncthreads();
  return found;
}

// The same rounds by all warps of the CTA, six entries each in queue order, until the search ends.
// Entries past the 512th are never examined (fluid.rs:530), so appends stop there. All threads; ends
// with a barrier.
__device__ __noinline__ void search_cta(const Region& Rs, LvSmem& L) {
  const Region R = Rs;
  Search& C = L.s;
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, nw = blockDim.x >> 5;
  const unsigned jl = lane / 5u, d = lane - 5u * jl, j = warp * SOLO_ENTRIES + jl;  // lanes 30, 31 idle
  const SearchLane D = search_lane(R, d);
  if (L.hard) {
    const bool hopeless = search_hopeless(Rs, L);
    if (tid == 0) {
      if (hopeless) {
        C.status = SS_NONE;
        C.i = PRESSURE_SEARCH;
      } else {
        L.hard = 0u;
      }
    }
    __syncthreads();
    if (hopeless) return;
  }
  unsigned i = C.i, qlen = C.qlen, side = C.side;
  const unsigned rank0 = C.rank0 + 6u;
  while (i < qlen && i < PRESSURE_SEARCH) {
    const unsigned kk = min(SOLO_ENTRIES * nw, min(qlen, PRESSURE_SEARCH) - i);
    const SearchRead r = search_read(R, L, D, jl < SOLO_ENTRIES && j < kk, i + j, side < 24u);
    if (r.blk) atomicMax(&C.blk, r.blk);
    const unsigned wm = __ballot_sync(FULLMASK, r.win), smk = __ballot_sync(FULLMASK, r.side);
    // no more than 24 side checks at the start level (fluid.rs:546-549): their order over the warps
    // matters only in the round that passes the limit
    if (lane == 0) {
      C.m_win[warp] = wm;
      C.m_side[warp] = smk;
    }
    __syncthreads();
    if (C.blk) {
      if (tid == 0) C.status = SS_BLOCKED;
      break;
    }
    const unsigned wmine = lane < nw ? C.m_win[lane] : 0u, smine = lane < nw ? C.m_side[lane] : 0u;
    const unsigned wany = __ballot_sync(FULLMASK, wmine != 0u), sany = __ballot_sync(FULLMASK, smine != 0u);
    if (wany) {
      if (warp == (unsigned)__ffs(wany) - 1u && lane == (unsigned)__ffs(wm) - 1u) search_won(C, r, i + j);
      break;
    }
    bool cand = r.cand;
    if (sany) {
      const unsigned c = (unsigned)__popc(smine);
      const unsigned before = __reduce_add_sync(FULLMASK, lane < warp ? c : 0u);
      if (r.side && side + before + (unsigned)__popc(smk & lanemask_lt()) + 1u > 24u) cand = false;
      side += __reduce_add_sync(FULLMASK, c);
    }
    if (qlen < PRESSURE_SEARCH) {
      const unsigned rank = rank0 + (i + j) * 5u + d;
      unsigned h = 0;
      if (cand) {
        h = vis_slot(C, r.key);
        atomicMin(&C.vrank[h], rank);
      }
      __syncthreads();
      const bool isnew = cand && vld(&C.vrank[h]) == rank;
      const unsigned nm = __ballot_sync(FULLMASK, isnew);
      if (lane == 0) C.m_new[warp] = (unsigned)__popc(nm);
      __syncthreads();
      const unsigned c = lane < nw ? C.m_new[lane] : 0u;
      const unsigned before = __reduce_add_sync(FULLMASK, lane < warp ? c : 0u), all = __reduce_add_sync(FULLMASK, c);
      const unsigned pos = qlen + before + (unsigned)__popc(nm & lanemask_lt());
      if (isnew && pos < PRESSURE_SEARCH) C.q[pos] = make_uint2(r.key, __float_as_uint(r.v));
      qlen += all;
    }
    i += kk;
    __syncthreads();
  }
  __syncthreads();
  if (tid == 0) {
    if (C.status == SS_MORE) {
      C.status = SS_NONE;
      C.i = i;
      // (negative coordinates, which a search passes over, and narrower CTAs: always in queue order)
      L.hard = i >= PRESSURE_SEARCH && !D.neg && nw == 16u ? 1u : 0u;
    }
    C.nvis += qlen;  // (keys of the last round that found no place in the queue: fewer than VIS_SLOTS - VIS_FULL - 518)
  }
  __syncthreads();
}

// The end of a pull, one warp: the source's write (fluid.rs:536-540), then the cell itself.
__device__ __forceinline__ void pull_end(const Region& R, LvSmem& L, const LaneSlot& S, int gate, unsigned kp, unsigned cur, unsigned& cnt, unsigned pb,
                                         unsigned& park, Touch& T, int& pd) {
  Search& C = L.s;
  const unsigned lane = lane_id(), k = C.pos;
  unsigned ev = 0u;
  if (C.status == SS_SUCCESS) {
    if (lane == 0) {
      const unsigned sid = C.skey & ~ABOVE;
      const unsigned u = R.dense[sid], j = R.stamp[sid];
      const float nv = __fsub_rn(C.here, C.got), v = dc_volume(u);
      const bool is_water = (int)u > 0, mid = nv > 1e-6f && nv < full_level(), wet = nv >= (is_water ? HIDE_BELOW : SHOW_AT);
      R.dense[sid] = mid ? (__float_as_uint(nv) | (wet ? 0u : DC_AIR)) : (wet ? DC_FULL : 0u);
      pd += (mid ? 1 : 0) - (v < 1.0f ? 1 : 0);  // (a source holds water)
      R.lv_src[k] = sid;
      // activation slots 0 (the source) and 1 (around the cell); bit 17 seeds the source
      ev = 3u | (wet != is_water ? 0x8000u : 0u) | (2u << 16);
      // a drained source that was full attempts a pull of its own when its turn comes
      if (j != NOSLOT && nv < full_level() && !bit_of(L.att, j) && !((R.pextra[j >> 5] >> (j & 31u)) & 1u)) {
        R.pextra[j >> 5] |= 1u << (j & 31u);
        R.pxlist[L.nx] = j;
        L.nx += 1u;
        if (j < kp) L.pp[j >> 5] |= 1u << (j & 31u);
      }
      L.n_succ += 1u;
    }
    ev = __shfl_sync(FULLMASK, ev, 0);
  }
  if (lane == 0) {
    L.n_entries += C.i;
    L.n_searches += 1u;
  }
  __syncwarp();
  LaneCell c = cell_record(R, lane < 8u, k);
  cell_slot(R, S, c);
  const float vol = lv_cells<true>(R, L, S, c, true, C.got, ev, gate, kp, cur, 0u, cnt, pb, park, T, pd);
  if (lane == 0u && ev && vol >= full_level()) {
    // a pull that leaves its own cell full gives its later neighbours on the layer a start cell
    const LvCell& rc = R.lv[k];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const unsigned nb = rc.succ[q == 0 ? 0 : 3];
      if (nb != NOSUCC && nb < kp && bit_of(L.att, nb)) L.pp[nb >> 5] |= 1u << (nb & 31u);
    }
  }
  __syncwarp();
}

// Finds the first pp cell in sorted order and its layer (the gate), one warp.
__device__ __forceinline__ void lv_head(const Region& R, LvSmem& L, unsigned n, HeadState& H) {
  const unsigned lane = lane_id(), ngrp = (n + 31u) / 32u;
  unsigned w = H.word, P = 0, any = 0;
  while (w < ngrp) {
    P = w + lane < ngrp ? vld(&L.pp[w + lane]) : 0u;
    any = __ballot_sync(FULLMASK, P != 0u);
    if (any) break;
    w += 32u;
  }
  H.blk = H.test = 0u;
  if (!any) {
    H.word = ngrp;
    H.head = n;
    H.gate = 0x7FFFFFFF;
    return;
  }
  const int fl = __ffs(any) - 1;
  H.word = w + (unsigned)fl;
  H.head = H.word * 32u + (unsigned)__ffs(__shfl_sync(FULLMASK, P, fl)) - 1u;
  H.gate = (int)(R.lv[H.head].ye & YE_Y);  // (its search or its test reads the record next)
}

// The first pp cell has yet to have its turn: can it still find a start cell then? A full neighbour
// stays full unless it runs before the cell does and falls: a side earlier in sorted order, over a
// cell that no unfinished cell writes and that has room (a full cell makes no attempt, and a fall of
// 2e-4 leaves it below 1 - 1e-4). A cell whose full neighbours all do that will not pull and leaves
// pp: later pulls need not wait for it. Returns 0 = it will not pull, 1 + a cell to wait for before
// the test can tell, or TEST_FAILED.
__device__ __forceinline__ unsigned lv_prune(const Region& R, LvSmem& L, unsigned k) {
  const unsigned lane = lane_id();
  const unsigned cid = R.lv[k].cid, ye = R.lv[k].ye;
  const float FULL = full_level();
  // lanes 8m .. 8m + 7 (m = 0..3) look at side m; lane 0 at the cell above too
  const unsigned m = lane >> 3, q = lane & 7u;
  const int row = R.PX * R.PY, at = (int)cid + (m == 0u ? 1 : m == 1u ? -1 : m == 2u ? row : -row);
  const int w5 = at - R.PX + (q == 1u ? 1 : q == 2u ? -1 : q == 3u ? row : q == 4u ? -row : 0);  // who may write the cell below it
  const unsigned us = R.dense[at], ub = q == 1u ? R.dense[at - R.PX] : DC_SOLID, ps = q == 0u ? R.stamp[at] : NOSLOT;
  const unsigned uu = lane == 0u ? R.dense[(int)cid + R.PX] : DC_SOLID;
  // (a side that is solid has no start cell, and what lies around it may be outside the domain)
  const bool full = ((ye >> (28u + m)) & 1u) && !dc_solid(us) && dc_volume(us) >= FULL;
  bool fail = lane == 0u && ((ye >> 27) & 1u) && !dc_solid(uu) && dc_volume(uu) >= FULL;
  unsigned wait = 0u;
  if (full) {
    if (q == 0u) fail |= ps == NOSLOT || ps > k || cell_done(L, ps);  // the side itself: earlier and unfinished
    if (q == 1u) fail |= dc_solid(ub) || !(__fsub_rn(1.0f, dc_volume(ub)) >= 2e-4f);  // room below it
    if (q < 5u) {
      const unsigned p = R.stamp[w5];
      if (p != NOSLOT && !cell_done(L, p)) wait = p + 1u;
    }
  }
  // room below is final only once nobody writes it: wait first
  const unsigned hard = __ballot_sync(FULLMASK, fail && q != 1u), soft = __ballot_sync(FULLMASK, fail);
  const unsigned w = __reduce_max_sync(FULLMASK, wait);
  return hard ? TEST_FAILED : w ? w : soft ? TEST_FAILED : 0u;
}

// Between the CTA's rounds, warp 0: the pulls whose turn has come, in order, and the rounds that are
// too short for the CTA. Ends with a request to the CTA: run the list, open the gate (L.gate changed
// from `gate`), carry on the search, or the sweep's end. Returns the change in partial entries.
__device__ __noinline__ int lv_solo(const Region& Rs, LvSmem& L, unsigned n, int gate, int sgn, unsigned long long cap) {
  const Region R = Rs;
  int pd = 0;
  __syncwarp();
  const unsigned lane = lane_id(), kp = L.kp;
  const LaneSlot S = lane_slot(R, kp);
  HeadState H = L.h;
  const unsigned pb = L.pb, cc = L.cc;
  unsigned req, cur = L.cur, cnt = L.cnt[cc], park = L.park_n[pb], rounds = L.rounds;  // (nobody else adds to the lists now)
  bool finish = L.resume != 0u;
  unsigned steps = 0;
  Touch T;
  while (true) {
    if (++steps > 8u * MAX_CELLS_PER_TICK) {  // more than the tick's pulls and rounds: cannot happen
      if (lane == 0) L.timeout = 1u;
      req = SR_END;
      break;
    }
    if (!finish && H.head < n) {
      if (!((vld(&L.pp[H.head >> 5]) >> (H.head & 31u)) & 1u)) {
        lv_head(R, L, n, H);
        if (H.gate != gate) {
          req = SR_GATE;
          break;
        }
      }
      const unsigned dep = dep_byte(L, H.head);
      if (dep == 0u) {  // its turn has come
        if (H.blk == 0u || cell_done(L, H.blk - 1u)) {
          if (search_begin(R, L, S, H.head, sgn, H.blk)) {
            if (vld(&L.hard)) {  // all warps look at it at once
              if (lane == 0) L.s.status = SS_MORE;
              __syncwarp();
            } else {
              search_solo(R, L);
            }
            if (L.s.status == SS_MORE) {
              req = SR_SEARCH;
              break;
            }
          }
          finish = H.blk == 0u;
        }
      } else if (H.test == 0u || (H.test != TEST_FAILED && cell_done(L, H.test - 1u))) {
        H.test = lv_prune(R, L, H.head);
        if (H.test == 0u) {
          if (lane == 0) L.pp[H.head >> 5] &= ~(1u << (H.head & 31u));
          __syncwarp();
          continue;
        }
      }
    }
    if (finish) {
      finish = false;
      if (L.s.status == SS_BLOCKED) {
        H.blk = L.s.blk;
        if (lane == 0) L.n_again += 1u;
      } else {
        pull_end(R, L, S, gate, kp, cur, cnt, pb, park, T, pd);
      }
      continue;
    }
    if (cnt == 0u || rounds >= cap) {  // with a pull pending a listed cell is always left: a stuck sweep ends as a timeout
      if (lane == 0) L.timeout = cnt != 0u || H.head < n ? 1u : 0u;
      req = SR_END;
      break;
    }
    if (cnt > SOLO_CELLS) {
      req = SR_LIST;
      break;
    }
    const unsigned t = lane >> 3;
    const unsigned i = t < cnt ? L.list[cur][t] : 0u;
    const bool run = t < cnt && !cell_done(L, i);
    cnt = 0u;
    LaneCell c = cell_record(R, run, i);
    cell_slot(R, S, c);
    lv_cells<true>(R, L, S, c, false, 0.0f, 0u, gate, kp, cur ^ 1u, 0u, cnt, pb, park, T, pd);
    cur ^= 1u;
    ++rounds;
  }
  if ((T.seen | T.a | T.b) >> 31) set_status(R, ST_RANGE, 53);
  __syncwarp();
  if (lane == 0) {
    L.req = req;
    L.resume = req == SR_SEARCH ? 1u : 0u;
    L.h = H;
    L.cur = cur;
    L.cnt[0] = L.cnt[1] = L.cnt[2] = 0u;
    L.cnt[cc] = cnt;
    L.park_n[pb] = park;
    L.rounds = rounds;
  }
  return pd;
}

// Rounds of THREAD_CELLS cells and more, by the whole CTA, one thread per cell: one while pulls are still possible
// (warp 0 looks after every round), else as long as the lists are that long. All threads; ends with a barrier.
// Returns the thread's change in partial entries. (The long rounds, those of four cells a warp and warp 0's work
// are functions of their own for the registers: one holding two of them slowed the shorter one by 6-15%.)
__device__ __noinline__ int lv_long(const Region& Rs, LvSmem& L, unsigned n, int gate, unsigned long long cap) {
  const Region R = Rs;
  const unsigned tid = threadIdx.x;
  const bool alive = L.h.head < n;
  const unsigned pb = L.pb, kp = L.kp;
  unsigned cur = L.cur, cc = L.cc, rounds = L.rounds, fcount = min(L.cnt[cc], MAX_CELLS_PER_TICK);
  int pd = 0;
  do {
    const unsigned nc = cc == 2u ? 0u : cc + 1u, zc = nc == 2u ? 0u : nc + 1u;
    if (tid == 0) L.cnt[zc] = 0u;
    for (unsigned at = tid & ~31u; at < fcount; at += blockDim.x) {
      const unsigned t = at + lane_id(), i = t < fcount ? list_get(R, L, cur, t) : 0u;
      lv_cell_thread(R, L, t < fcount && !cell_done_now(L, i), i, gate, kp, cur ^ 1u, nc, pb, pd);
    }
    __syncthreads();
    cur ^= 1u;
    cc = nc;
    ++rounds;
    fcount = min(L.cnt[cc], MAX_CELLS_PER_TICK);
  } while (!alive && fcount >= THREAD_CELLS && rounds < cap);
  __syncthreads();  // everybody has read the count
  if (tid == 0) {
    L.cur = cur;
    L.cc = cc;
    L.rounds = rounds;
  }
  return pd;
}

// Rounds by the whole CTA, four cells a warp at a time: one while pulls are still possible (warp 0 looks
// after every round), else until the list is short or long. All threads; ends with a barrier. A long list's
// records are fetched two steps ahead and its volumes one (a function of its own for the registers
// that takes): ring rain 18.6 -> 13.8 M cycles of its rounds, lake 7.6 -> 6.3 M. Returns the thread's change in
// partial entries.
__device__ __noinline__ int lv_wide(const Region& Rs, LvSmem& L, unsigned n, int gate, unsigned long long cap) {
  const Region R = Rs;
  const unsigned tid = threadIdx.x, lane = tid & 31u, step = (blockDim.x >> 5) * 4u, t0 = (tid >> 5) * 4u;
  const bool alive = L.h.head < n;
  const unsigned pb = L.pb, kp = L.kp;
  const LaneSlot S = lane_slot(R, kp);
  unsigned cur = L.cur, cc = L.cc, rounds = L.rounds, fcount = min(L.cnt[cc], MAX_CELLS_PER_TICK), unused = 0;
  Touch T;
  int pd = 0;
  do {
    const unsigned nb = cur ^ 1u, nc = cc == 2u ? 0u : cc + 1u, zc = nc == 2u ? 0u : nc + 1u;
    if (tid == 0) L.cnt[zc] = 0u;
    auto record = [&](unsigned at) {
      const unsigned t = at + (lane >> 3), i = t < fcount ? list_get(R, L, cur, t) : 0u;
      return cell_record(R, t < fcount && !cell_done_now(L, i), i);
    };
    if (fcount <= step) {
      if (t0 < fcount) {
        LaneCell c = record(t0);
        cell_slot(R, S, c);
        lv_cells<false>(R, L, S, c, false, 0.0f, 0u, gate, kp, nb, nc, unused, pb, unused, T, pd);
      }
    } else if (t0 < fcount) {
      LaneCell c = record(t0), d = record(t0 + step);
      cell_slot(R, S, c);
      for (unsigned at = t0; at < fcount; at += step) {
        const LaneCell e = record(at + 2u * step);
        cell_slot(R, S, d);
        lv_cells<false>(R, L, S, c, false, 0.0f, 0u, gate, kp, nb, nc, unused, pb, unused, T, pd);
        c = d;
        d = e;
      }
    }
    __syncthreads();
    cur = nb;
    cc = nc;
    ++rounds;
    fcount = min(L.cnt[cc], MAX_CELLS_PER_TICK);
  } while (!alive && fcount > SOLO_CELLS && fcount < THREAD_CELLS && rounds < cap);
  if ((T.seen | T.a | T.b) >> 31) set_status(R, ST_RANGE, 53);
  __syncthreads();  // everybody has read the count
  if (tid == 0) {
    L.cur = cur;
    L.cc = cc;
    L.rounds = rounds;
  }
  return pd;
}

}  // namespace vfe
