// Exact parallel sweep: the body of FluidSim::tick (src/fluid.rs:584-651) over the region's CTA, one
// thread per cell, with results bit-identical to the reference's sequential loop.
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
// What bounds it: the number of rounds times the latency of one (list entry -> 64-byte record -> 7
// cells -> plan -> stores -> successor counts -> barrier), on one SM per region.
#pragma once
#include "engine_dev.cuh"

namespace vfe {

constexpr unsigned GRID_LOCKED = 0xFFFFFFFFu;  // grid word while a warp materialises the brick
constexpr int MAX_WARPS = 16;                  // warps of a CTA running the sweep
constexpr int TEAM_WARPS = 4;                  // warps that run one pressure search together
constexpr int TEAM_THREADS = 32 * TEAM_WARPS;
constexpr int MAX_TEAMS = MAX_WARPS / TEAM_WARPS;
constexpr unsigned TEAM_ENTRIES = TEAM_THREADS / 5;  // queue entries a search examines per round
constexpr unsigned VIS_SLOTS = 1024;  // visited set of one search: <= 6 + 512 + 5 * TEAM_ENTRIES cells
static_assert(6 + PRESSURE_SEARCH + 5 * TEAM_ENTRIES < VIS_SLOTS, "visited set");
constexpr unsigned NGROUPS = (MAX_CELLS_PER_TICK + 31) / 32;
constexpr unsigned LIST_CAP = 4096;   // a round's list kept in shared memory; the rest goes to global
constexpr unsigned NOSUCC = 0xFFFFu;
static_assert(MAX_CELLS_PER_TICK < NOSUCC, "sorted positions fit 16 bits");
constexpr unsigned UNIFORM = 0x80000000u;  // LvCell::slot of a brick that was a uniform grid value
constexpr unsigned DONE = 0xFFu;           // dependency byte of a finished cell
constexpr int GATE_MAX = 31;               // range of the gate knob's radii (accepted, unused)

// What a round reads of a drained cell, made in the prepass (one 64-byte line segment per cell).
struct __align__(16) LvCell {
  unsigned slot[7];         // atlas slots of the footprint (self, below, up, +x, -x, +z, -z), or UNIFORM
  unsigned cid;             // domain id
  unsigned short succ[12];  // later conflicting positions (succ_offset's order), NOSUCC = none
  unsigned flags;           // bits 0-6 solid footprint cells; 8-12 cells a pull may start from (up,
                            // +x, -x, +z, -z: not solid, x and z >= 0); 16-24 brick voxel index
  int y;
};
static_assert(sizeof(LvCell) == 64, "LvCell");

// The footprint volumes a cell of the gate layer found, for searches of earlier cells.
struct __align__(16) LvOld {
  float vol[7];
  unsigned wmask;  // footprint slots it wrote
};

// One pressure search (a team of TEAM_WARPS warps).
enum SearchStatus { SS_NONE = 0, SS_SUCCESS = 1, SS_BLOCKED = 2 };
struct Search {
  unsigned q[PRESSURE_SEARCH];  // queued cells, relative to the pulling cell (rel_pack)
  float qv[PRESSURE_SEARCH];    // their volume
  unsigned vkey[VIS_SLOTS];     // visited cells (EMPTY_ID = free)
  unsigned vrank[VIS_SLOTS];    // earliest (entry, direction) that tested the cell
  float fv[8];                  // the pulling cell's footprint volumes
  unsigned m_win[TEAM_WARPS], m_side[TEAM_WARPS], m_new[TEAM_WARPS];
  unsigned blk;                 // 1 + an unfinished earlier cell the search depends on (0: none)
  unsigned before;              // cells before this one that pulls took below full
  unsigned pos, status, entries, qlen, hit, full;
  float got, here;
  int cx, cy, cz;               // the pulling cell
  int sx, sy, sz;               // the source
};

struct LvSmem {
  unsigned dep[(MAX_CELLS_PER_TICK + 3) / 4];  // a byte per cell: unfinished earlier conflicting cells, DONE
  unsigned att[NGROUPS + 1];   // bit per cell: not solid and below 1 - 1e-4 at the tick's start
  unsigned pp[NGROUPS + 1];    // bit per unfinished cell that may find a start cell within the budget
  unsigned pend[NGROUPS + 1];  // bit per cell that reached its turn and has a start cell
  unsigned short gpre[NGROUPS + 1];  // att bits before each group of 32
  unsigned short list[2][LIST_CAP];
  unsigned cnt[3];             // list lengths, rotating: this round's, the next, the one being cleared
  unsigned park_n[2];          // ready cells above the gate
  unsigned kp;                 // positions from here on cannot pull (budget spent before them)
  unsigned nx;                 // full cells pulls took from (Region::pxlist)
  unsigned head, hword, hblk;  // first pp cell, its group, 1 + the cell its search waits for
  int gate;                    // layer of the first pp cell: cells above it wait
  unsigned lend;               // first position after that layer
  unsigned nsearch, ncommit;   // pulls whose turn has come, those that commit
  unsigned cand[MAX_TEAMS];
  unsigned res_ev[MAX_TEAMS];
  unsigned n_succ, n_searches, n_again;
  unsigned long long n_entries;
  Search s[MAX_TEAMS];
};

__device__ __forceinline__ unsigned vld(const unsigned* p) { return *(volatile const unsigned*)p; }
// A global word that only this CTA's threads write (grid words): a relaxed load at CTA scope. It is
// coherent with the CTA's stores and atomics but may be served by the SM's L1.
__device__ __forceinline__ unsigned gld(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.cta.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}

// Back-off of a polling loop after n polls: a few polls at full rate, then sleeps of up to 1 us.
__device__ __forceinline__ void backoff(unsigned long long n) {
  if (n > 4) __nanosleep(min(32u << (unsigned)min((n - 4) >> 2, 5ull), 1024u));
}

// The grid word of a brick, past a lock another warp holds while it materialises it (a lock's holder
// waits for nobody, so the wait is short; it is bounded all the same).
__device__ __forceinline__ unsigned grid_word(const Region& R, unsigned gi, unsigned long long cap) {
  unsigned g = gld(R.grid + gi);
  unsigned long long spins = 0;
  while (g == GRID_LOCKED) {
    if (++spins > cap) {
      set_status(R, ST_TIMEOUT, 30);
      return 0u;
    }
    backoff(spins);
    g = gld(R.grid + gi);
  }
  __threadfence_block();
  return g;
}

__device__ __forceinline__ CD load_cell_par(const Region& R, const int* ring, int x, int y, int z, unsigned long long cap) {
  CD c;
  c.part = 0.0f;
  c.slot = NOSLOT;
  c.gi = 0;
  c.mat = 0;
  c.out = outside(R, ring, x, y, z);
  if (c.out) return c;
  c.gi = grid_index(R, x >> 3, y >> 3, z >> 3);
  const unsigned g = grid_word(R, c.gi, cap);
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

// Atlas slots for the bricks lanes with `need` are about to write (sparse_volume.rs:250-266), warp-
// collective. The first warp to take a brick's grid word (CAS to GRID_LOCKED) allocates and fills the
// slot and publishes it; the others read the published slot. A warp publishes every brick it has
// locked before it waits for one, so two warps never wait for each other.
__device__ void materialize_par(const Region& R, bool need, unsigned gi, unsigned& slot, unsigned long long cap) {
  const unsigned lane = lane_id();
  const unsigned key = need ? gi : (0xFFFFFFFFu - lane);
  const unsigned peers = __match_any_sync(FULLMASK, key);
  bool open = need && !(peers & lanemask_lt());
  unsigned s = NOSLOT;
  unsigned long long spins = 0;
  while (__any_sync(FULLMASK, open)) {
    unsigned g = 0;
    bool fill = false;
    if (open) {
      g = gld(R.grid + gi);
      if (g < 256u) {
        if (atomicCAS(R.grid + gi, g, GRID_LOCKED) == g) {
          s = atomicAdd(&R.ctl->atlas_used, 1u);
          if (s >= R.atlas_cap) {
            set_status(R, ST_OOM, 1);
            atomicExch(R.grid + gi, g);
            s = NOSLOT;
            open = false;
          } else {
            fill = true;
          }
        }
      } else if (g != GRID_LOCKED) {
        s = g - 256u;
        open = false;
      } else if (++spins > cap) {
        set_status(R, ST_TIMEOUT, 31);
        open = false;
      } else {
        backoff(spins);
      }
    }
    for (unsigned m = __ballot_sync(FULLMASK, fill); m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const unsigned sl = __shfl_sync(FULLMASK, s, l);
      unsigned fv = __shfl_sync(FULLMASK, g, l) & 255u;
      fv |= fv << 8;
      fv |= fv << 16;
      reinterpret_cast<uint4*>(R.amat + (size_t)sl * 512u)[lane] = make_uint4(fv, fv, fv, fv);
      uint4* vv = reinterpret_cast<uint4*>(R.avol + (size_t)sl * 512u);
#pragma unroll
      for (int k = 0; k < 4; ++k) vv[lane + 32 * k] = make_uint4(0, 0, 0, 0);
    }
    __syncwarp();
    __threadfence_block();
    if (fill) {
      atomicExch(R.grid + gi, 256u + s);
      open = false;
    }
  }
  const int src = need ? (__ffs(peers) - 1) : (int)lane;
  const unsigned s2 = __shfl_sync(FULLMASK, s, src);
  if (need) slot = s2;
  __syncwarp();
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
__device__ __forceinline__ void sv_apply(const Region& R, size_t o, const SVPlan& p) {
  if (p.wpart) R.avol[o] = p.npart;
  if (p.wmat) R.amat[o] = p.nmat;
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

__device__ __forceinline__ unsigned rank_at(const Region& R, int x, int y, int z) {
  if (!in_dom(R, x, y, z)) return NOSLOT;
  return R.stamp[dom_id(R, x, y, z)];
}

// Cells relative to a pulling cell: a search examines 512 entries, so it stays within 513 steps.
__device__ __forceinline__ unsigned rel_pack(int dx, int dy, int dz) {
  return (unsigned)(dx + 1024) | (unsigned)(dz + 1024) << 11 | (unsigned)dy << 22;
}
__device__ __forceinline__ void rel_unpack(unsigned k, int& dx, int& dy, int& dz) {
  dx = (int)(k & 2047u) - 1024;
  dz = (int)((k >> 11) & 2047u) - 1024;
  dy = (int)(k >> 22);
}

// The flow part of a cell's update (fluid.rs:606-650) from its footprint volumes, its solid cells
// (bits) and its volume `vol` (> 0): 1. fall into the free capacity below, 2. share with lower sides
// when supported, 3. evaporate crumbs. Every side's flow depends only on the volume after the fall
// and that side's volume; only the running volume subtracts them in side order.
struct FlowPlan {
  float vol;          // the cell's volume afterwards (before the write-back test)
  float below_new;    // the cell below's new volume when w_below
  float side_new[4];  // +x, -x, +z, -z new volumes when their bit of wside is set
  bool w_below;
  unsigned wside;     // bit i: side i is written
  unsigned amask;     // activation slots 2 (below) and 3..6 (sides)
};
__device__ __forceinline__ FlowPlan flow_plan(const float (&v)[7], unsigned solid, float vol) {
  const float FULL = full_level();
  FlowPlan P;
  const bool below_solid = (solid >> 1) & 1u;
  const float bv = below_solid ? 0.0f : v[1];
  const float ff = fminf(vol, __fsub_rn(1.0f, bv));
  P.w_below = !below_solid && ff > 1e-6f;
  P.below_new = __fadd_rn(bv, ff);
  vol = P.w_below ? __fsub_rn(vol, ff) : vol;
  const float below_after = P.w_below ? (P.below_new >= FULL ? 1.0f : P.below_new) : bv;
  const bool spread = vol > MIN_SPREAD && (below_solid || below_after >= FULL);
  const float here = vol;
  P.wside = 0u;
  P.amask = P.w_below ? (1u << 2) : 0u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool open = !((solid >> (3 + i)) & 1u);
    const float nv = open ? v[3 + i] : 0.0f;
    const float f = __fmul_rn(__fsub_rn(here, nv), 0.2f);
    const bool ok = spread && open && !(nv >= here) && !(f < MIN_FLOW) && !(__fsub_rn(here, f) < MIN_SPREAD * 0.5f);
    P.side_new[i] = __fadd_rn(nv, f);
    P.wside |= ok ? (1u << i) : 0u;
    vol = ok ? __fsub_rn(vol, f) : vol;
    P.amask |= (ok && f > SLEEP) ? (1u << (3 + i)) : 0u;
  }
  P.vol = vol < EVAPORATE ? 0.0f : vol;
  return P;
}

// ------------------------------------------------------------------------------- the lists
__device__ __forceinline__ unsigned list_get(const Region& R, const LvSmem& L, unsigned b, unsigned t) {
  return t < LIST_CAP ? L.list[b][t] : R.lv_over[(size_t)b * MAX_CELLS_PER_TICK + t];
}
__device__ __forceinline__ void list_put(const Region& R, LvSmem& L, unsigned b, unsigned t, unsigned i) {
  if (t < LIST_CAP) L.list[b][t] = (unsigned short)i;
  else R.lv_over[(size_t)b * MAX_CELLS_PER_TICK + t] = (unsigned short)i;
}
__device__ __forceinline__ bool cell_done(const LvSmem& L, unsigned i) { return ((vld(&L.dep[i >> 2]) >> ((i & 3u) * 8u)) & 0xFFu) == DONE; }
__device__ __forceinline__ bool bit_of(const unsigned* w, unsigned i) { return (w[i >> 5] >> (i & 31u)) & 1u; }
// att bits before position i
__device__ __forceinline__ unsigned attempts_before(const LvSmem& L, unsigned i) {
  return (unsigned)L.gpre[i >> 5] + (unsigned)__popc(L.att[i >> 5] & ((1u << (i & 31u)) - 1u));
}

// -------------------------------------------------------------------------------- the cells
// Lane constants of the eight lanes that run a cell: lane l < 7 holds footprint slot l.
struct LaneSlot {
  int ox, oy, oz;        // the slot's offset
  unsigned lm, la;       // brick voxel index of the slot: the axis' bits, and what is added to them
  unsigned open1, open2; // the lane's two successors: one layer up (bit per successor), two layers up
};
__device__ __forceinline__ LaneSlot lane_slot() {
  const int l = (int)(threadIdx.x & 7u);
  LaneSlot s;
  fp_off(l, s.ox, s.oy, s.oz);
  s.lm = l == 7 || l == 0 ? 0u : l <= 2 ? 0x38u : l <= 4 ? 7u : 0x1C0u;
  s.la = (unsigned)(s.ox + 8 * s.oy + 64 * s.oz);
  s.open1 = l == 3 || l == 4 ? 3u : l == 5 ? 1u : 0u;  // successors 6..10
  s.open2 = l == 5 ? 2u : 0u;                          // successor 11
  return s;
}

// Four cells at sorted positions i (fluid.rs:584-651), eight lanes each, warp-collective (groups
// without a cell: `has` false). `pulled`: the cell's pull has run and took `got` (event bits `ev`);
// otherwise a cell with a start cell is left pending for its pull. nb / nc: the next round's list and
// its counter; pb: the parked list.
//
// Eight lanes rather than one thread per cell: a round is a latency chain (a few dozen to a few
// hundred cells on 16 warps), and a lane that holds one slot issues one address, one pair of loads,
// one set_volume and two successor counts where a thread issues seven, seven, six and twelve. The
// exchange costs seven shuffles and five ballots.
__device__ __forceinline__ void lv_cells(const Region& R, LvSmem& L, const LaneSlot& S, bool has, unsigned i, bool pulled, float got, unsigned ev,
                                         int gate, unsigned kp, unsigned nb, unsigned nc, unsigned pb, int& pd, unsigned long long cap) {
  const float FULL = full_level();
  const unsigned lane = lane_id(), l = lane & 7u, base = lane & 24u;
  unsigned w1 = UNIFORM, w2 = 0xFFFFFFFFu;
  if (has) {
    const unsigned* p = reinterpret_cast<const unsigned*>(R.lv + i) + l;
    w1 = p[0];
    w2 = p[8];
  }
  const unsigned flags = __shfl_sync(FULLMASK, w2, 6, 8);
  const unsigned cid = __shfl_sync(FULLMASK, w1, 7, 8);
  const int y = (int)__shfl_sync(FULLMASK, w2, 7, 8);
  const bool cell = has && l < 7u && !((flags >> l) & 1u);  // the lane holds a cell that is not solid
  const unsigned loc = flags >> 16, at = (loc & ~S.lm) | ((loc + S.la) & S.lm);
  unsigned slot = cell ? w1 : UNIFORM, gi = 0;
  if (cell && (slot & UNIFORM)) {  // uniform at the tick's start: the value, or the slot the brick has now
    int x, yy, z;
    dom_xyz(R, cid, x, yy, z);
    gi = grid_index(R, (x + S.ox) >> 3, (yy + S.oy) >> 3, (z + S.oz) >> 3);
    const unsigned g = grid_word(R, gi, cap);
    slot = g < 256u ? (UNIFORM | g) : g - 256u;
  }
  float part = 0.0f;
  unsigned mat = slot & 255u;
  if (!(slot & UNIFORM)) {
    const size_t o = (size_t)slot * 512u + at;
    part = R.avol[o];
    mat = R.amat[o];
  }
  const float v = part > 0.0f ? part : (cell && mat == WATER ? 1.0f : 0.0f);
  // ---- a cell that attempts a pull and has a start cell waits for the pull
  const unsigned starts = (__ballot_sync(FULLMASK, cell && l >= 2u && ((flags >> (6u + l)) & 1u) && v >= FULL) >> base) & 0xFFu;
  const float v0 = __shfl_sync(FULLMASK, v, 0, 8), bv = __shfl_sync(FULLMASK, v, 1, 8);
  if (has && !pulled && i < kp && v0 < FULL && starts) {
    if (l == 0u) {
      atomicOr(&L.pend[i >> 5], 1u << (i & 31u));
      if (!bit_of(L.pp, i)) set_status(R, ST_RANGE, 50);  // every cell that finds a start cell is in pp
    }
    has = false;
  }
  // ---- 1. fall into the free capacity below, 2. share with lower sides when supported, 3. evaporate
  // crumbs (fluid.rs:606-650). Every side's flow depends on the volume after the fall and its own
  // volume only; the running volume subtracts the flows in side order (a side without one: 0).
  float vol = pulled && got > 0.0f ? __fadd_rn(v0, got) : v0;
  const bool live = has && vol > 0.0f;  // fluid.rs:602-604
  const bool below_solid = (flags >> 1) & 1u;
  const float ff = fminf(vol, __fsub_rn(1.0f, bv));
  const bool w_below = live && !below_solid && ff > 1e-6f;
  const float below_new = __fadd_rn(bv, ff);
  vol = w_below ? __fsub_rn(vol, ff) : vol;
  const float below_after = w_below ? (below_new >= FULL ? 1.0f : below_new) : bv;
  const bool spread = live && vol > MIN_SPREAD && (below_solid || below_after >= FULL);
  const float f = __fmul_rn(__fsub_rn(vol, v), 0.2f);
  const bool ok = spread && l >= 3u && cell && !(v >= vol) && !(f < MIN_FLOW) && !(__fsub_rn(vol, f) < MIN_SPREAD * 0.5f);
  const float fs = ok ? f : 0.0f;
  const float f3 = __shfl_sync(FULLMASK, fs, 3, 8), f4 = __shfl_sync(FULLMASK, fs, 4, 8);
  const float f5 = __shfl_sync(FULLMASK, fs, 5, 8), f6 = __shfl_sync(FULLMASK, fs, 6, 8);
  vol = __fsub_rn(__fsub_rn(__fsub_rn(__fsub_rn(vol, f3), f4), f5), f6);
  vol = vol < EVAPORATE ? 0.0f : vol;
  const float dv = fabsf(__fsub_rn(vol, v0));
  const bool wr = l == 0u ? (live && dv > 1e-7f) : l == 1u ? w_below : ok;
  const float wv = l == 0u ? vol : l == 1u ? below_new : __fadd_rn(v, f);
  // ---- set_volume of the lane's cell (fluid.rs:327-355)
  const bool need = wr && (slot & UNIFORM) && (wv <= 1e-6f ? mat == WATER : wv >= FULL ? mat != WATER : true);
  if (__any_sync(FULLMASK, need)) {
    unsigned s = NOSLOT;
    materialize_par(R, need, gi, s, cap);
    if (need && s != NOSLOT) slot = s;
  }
  const bool hs = !(slot & UNIFORM);
  SVPlan p{};
  if (wr) {
    p = sv_plan(part, (unsigned char)mat, hs, wv);
    if (hs) sv_apply(R, (size_t)slot * 512u + at, p);
    pd += p.dp;
  }
  const unsigned wm = (__ballot_sync(FULLMASK, wr) >> base) & 0x7Fu;
  const unsigned cm = (__ballot_sync(FULLMASK, wr && p.ch) >> base) & 0x7Fu;
  const unsigned am = (__ballot_sync(FULLMASK, l == 1u ? w_below : ok && f > SLEEP) >> base) & 0x7Au;  // slots 1, 3..6
  bool r0 = false, r1 = false;  // the lane's successors whose last earlier cell this was
  if (has) {
    if (y == gate) reinterpret_cast<unsigned*>(R.lv_old + i)[l] = l == 7u ? wm : __float_as_uint(v);
    if (l == 0u) {
      // activation slots: 2 below, 3..6 the sides, 7 the cell itself
      const bool self = live && dv > SLEEP;
      R.lv_ev[i] = ev | (am & 0x78u) | ((am & 2u) << 1) | (self ? 0x10080u : 0u) | (cm << 8);
      atomicOr(&L.dep[i >> 2], DONE << ((i & 3u) * 8u));
      if (i < kp && bit_of(L.pp, i)) atomicAnd(&L.pp[i >> 5], ~(1u << (i & 31u)));
    }
    if (l < 6u) {
      const unsigned a = w2 & 0xFFFFu, b = w2 >> 16;
      unsigned oa = 0, ob = 0;
      if (a != NOSUCC) oa = atomicSub(&L.dep[a >> 2], 1u << ((a & 3u) * 8u));
      if (b != NOSUCC) ob = atomicSub(&L.dep[b >> 2], 1u << ((b & 3u) * 8u));
      r0 = a != NOSUCC && ((oa >> ((a & 3u) * 8u)) & 0xFFu) == 1u;
      r1 = b != NOSUCC && ((ob >> ((b & 3u) * 8u)) & 0xFFu) == 1u;
    }
  }
  // ---- the ready ones: to the next round, or parked above the gate
  const unsigned shut = (y + 1 > gate ? S.open1 : 0u) | (y + 2 > gate ? S.open2 : 0u);
  const unsigned g0 = __ballot_sync(FULLMASK, r0 && !(shut & 1u)), g1 = __ballot_sync(FULLMASK, r1 && !(shut & 2u));
  if (g0 | g1) {
    unsigned t = 0;
    if (lane == 0u) t = atomicAdd(&L.cnt[nc], (unsigned)(__popc(g0) + __popc(g1)));
    t = __shfl_sync(FULLMASK, t, 0);
    if (r0 && !(shut & 1u)) list_put(R, L, nb, t + (unsigned)__popc(g0 & lanemask_lt()), w2 & 0xFFFFu);
    if (r1 && !(shut & 2u)) list_put(R, L, nb, t + (unsigned)(__popc(g0) + __popc(g1 & lanemask_lt())), w2 >> 16);
  }
  if ((r0 && (shut & 1u)) || (r1 && (shut & 2u))) {
    unsigned t = atomicAdd(&L.park_n[pb], (r0 && (shut & 1u) ? 1u : 0u) + (r1 && (shut & 2u) ? 1u : 0u));
    if (r0 && (shut & 1u)) R.lv_park[(size_t)pb * MAX_CELLS_PER_TICK + t++] = (unsigned short)(w2 & 0xFFFFu);
    if (r1 && (shut & 2u)) R.lv_park[(size_t)pb * MAX_CELLS_PER_TICK + t] = (unsigned short)(w2 >> 16);
  }
  __syncwarp();
}

// --------------------------------------------------------------------------- pressure search
__device__ __forceinline__ void team_sync(int team) { asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "r"(TEAM_THREADS) : "memory"); }

__device__ __forceinline__ unsigned vis_slot(Search& C, unsigned key) {
  unsigned h = (key * 2654435761u) >> 22;  // 10 bits
  while (true) {
    const unsigned old = atomicCAS(&C.vkey[h], EMPTY_ID, key);
    if (old == EMPTY_ID || old == key) return h;
    h = (h + 1u) & (VIS_SLOTS - 1u);
  }
}

// The volume a cell (a, y, c) of the pulling layer holds at the turn of the cell at position k, given
// the volume `v` it holds now: later cells that already ran and wrote it are looked through (the
// earliest such write's old value); an unfinished earlier writer is reported in C.blk.
__device__ float old_volume(const Region& R, const LvSmem& L, Search& C, unsigned k, int a, int y, int c, float v) {
  unsigned j[5];
#pragma unroll
  for (int q = 0; q < 5; ++q)  // the writers of the cell: itself, and the sides it is a side of
    j[q] = rank_at(R, a - (q == 1) + (q == 2), y, c - (q == 3) + (q == 4));
  unsigned best = NOSLOT;
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    if (j[q] == NOSLOT || j[q] == k) continue;
    const bool done = cell_done(L, j[q]);
    if (j[q] < k) {
      if (!done) atomicMax(&C.blk, j[q] + 1u);
    } else if (done && j[q] < best) {
      const LvOld& o = R.lv_old[j[q]];
      const int fl = q == 0 ? 0 : q + 2;
      if ((o.wmask >> fl) & 1u) {
        best = j[q];
        v = o.vol[fl];
      }
    }
  }
  return v;
}

// FluidSim::pressure_pull (fluid.rs:511-561) of the cell at position k, by one team; writes nothing but
// C. TEAM_ENTRIES queue entries per round, one neighbour per thread, the reference's queue order kept
// exactly: the first surface entry in queue order wins; the 24 side checks at the start level are
// counted in (entry, direction) order; a cell found by several threads of a round belongs to the
// earliest (vrank). Entries past the 512th are never examined, so appends stop there.
__device__ void lv_search(const Region& R, LvSmem& L, const int* ring, int team, unsigned k, unsigned long long cap) {
  Search& C = L.s[team];
  const float FULL = full_level();
  const unsigned tt = threadIdx.x % TEAM_THREADS, tw = tt >> 5, lane = tt & 31u;
  const LvCell& rc = R.lv[k];
  const unsigned flags = rc.flags;
  int x, y, z;
  dom_xyz(R, rc.cid, x, y, z);
  for (unsigned t = tt; t < VIS_SLOTS; t += TEAM_THREADS) {
    C.vkey[t] = EMPTY_ID;
    C.vrank[t] = 0xFFFFFFFFu;
  }
  if (tt < 7u) {
    int ox, oy, oz;
    fp_off((int)tt, ox, oy, oz);
    const CD c = load_cell_par(R, ring, x + ox, y + oy, z + oz, cap);
    C.fv[tt] = cd_solid(c) ? 0.0f : cd_volume(c);
  }
  if (tt == 0) {
    C.blk = 0u;
    C.before = 0u;
    C.pos = k;
    C.status = SS_NONE;
    C.entries = 0u;
    C.qlen = 0u;
    C.hit = 0u;
    C.full = 0u;
    C.got = 0.0f;
    C.cx = x;
    C.cy = y;
    C.cz = z;
  }
  team_sync(team);
  {
    unsigned c = 0;
    for (unsigned t = tt; t < L.nx; t += TEAM_THREADS) c += R.pxlist[t] < k ? 1u : 0u;
    if (c) atomicAdd(&C.before, c);
  }
  team_sync(team);
  const float vol = C.fv[0];
  unsigned starts = 0u;
#pragma unroll
  for (int d = 0; d < 5; ++d) starts |= (((flags >> (8 + d)) & 1u) && C.fv[2 + d] >= FULL) ? (1u << d) : 0u;
  if (!(vol < FULL) || attempts_before(L, k) + C.before >= MAX_PULLS_PER_TICK || !starts) return;
  if (tt == 0) {
    C.vrank[vis_slot(C, rel_pack(0, 0, 0))] = 0u;
    unsigned p = 0;
    for (int d = 0; d < 5; ++d) {
      if (!((starts >> d) & 1u)) continue;
      int dx, dy, dz;
      dir5(d, dx, dy, dz);
      const unsigned key = rel_pack(dx, dy, dz);
      C.q[p] = key;
      C.qv[p] = C.fv[2 + d];
      C.vrank[vis_slot(C, key)] = ++p;
    }
  }
  team_sync(team);
  const unsigned j = tt / 5u, d = tt - 5u * j;
  unsigned qlen = (unsigned)__popc(starts), i = 0, side = 0;
  while (i < qlen && i < PRESSURE_SEARCH) {
    const unsigned kk = min(TEAM_ENTRIES, min(qlen, PRESSURE_SEARCH) - i);
    const bool act = j < kk;
    int a = 0, b = 0, c = 0, dx = 0, dy = 0, dz = 0;
    float here = 0.0f, v = 0.0f;
    bool rd = false, so = true;
    unsigned key = 0;
    if (act) {
      key = C.q[i + j];
      here = C.qv[i + j];
      rel_unpack(key, a, b, c);
      dir5((int)d, dx, dy, dz);
      dx += a;
      dy += b;
      dz += c;
      const int na = x + dx, nb = y + dy, nc = z + dz;
      rd = d == 0u ? nb < R.ny : (na >= 0 && nc >= 0);
      if (rd) {
        const CD cd = load_cell_par(R, ring, na, nb, nc, cap);
        so = cd_solid(cd);
        v = so ? 0.0f : cd_volume(cd);
        if (!so && dy == 0) v = old_volume(R, L, C, k, na, nb, nc, v);
      }
    }
    // surface test of each entry on its up neighbour (fluid.rs:534-535)
    const bool top = so || v <= 0.0f;
    const bool win = act && d == 0u && top && b > 0 && here > 0.0f;
    bool cand = rd && !top;
    const bool scnt = cand && d >= 1u && dy == 0;
    const unsigned wmk = __ballot_sync(FULLMASK, win), smk = __ballot_sync(FULLMASK, scnt);
    if (lane == 0) {
      C.m_win[tw] = wmk;
      C.m_side[tw] = smk;
    }
    team_sync(team);
    if (C.blk) {  // an earlier cell has yet to write what the search read: run it again later
      if (tt == 0) C.status = SS_BLOCKED;
      return;
    }
    int wt = -1;
    unsigned sbefore = side, sall = side;
#pragma unroll
    for (int w = 0; w < TEAM_WARPS; ++w) {
      const unsigned m = C.m_win[w];
      if (m && wt < 0) wt = 32 * w + __ffs(m) - 1;
      const unsigned sc = (unsigned)__popc(C.m_side[w]);
      if ((unsigned)w < tw) sbefore += sc;
      sall += sc;
    }
    if (wt >= 0) {
      if ((int)tt == wt) {
        C.sx = x + a;
        C.sy = y + b;
        C.sz = z + c;
        C.here = here;
        C.got = fminf(__fsub_rn(1.0f, vol), here);
        C.status = SS_SUCCESS;
        C.entries = i + j + 1u;
        C.qlen = min(qlen, PRESSURE_SEARCH);
      }
      team_sync(team);
      break;
    }
    if (qlen < PRESSURE_SEARCH) {
      // expansions (fluid.rs:541-556)
      if (scnt && sbefore + (unsigned)__popc(smk & lanemask_lt()) + 1u > 24u) cand = false;
      side = sall;
      const unsigned rank = 6u + (i + j) * 5u + d;
      unsigned h = 0;
      if (cand) {
        key = rel_pack(dx, dy, dz);
        h = vis_slot(C, key);
        atomicMin(&C.vrank[h], rank);
      }
      team_sync(team);
      const bool isnew = cand && vld(&C.vrank[h]) == rank;
      const unsigned nmk = __ballot_sync(FULLMASK, isnew);
      if (lane == 0) C.m_new[tw] = nmk;
      team_sync(team);
      unsigned pos = qlen + (unsigned)__popc(nmk & lanemask_lt()), all = 0;
#pragma unroll
      for (int w = 0; w < TEAM_WARPS; ++w) {
        const unsigned nw = (unsigned)__popc(C.m_new[w]);
        if ((unsigned)w < tw) pos += nw;
        all += nw;
      }
      if (isnew && pos < PRESSURE_SEARCH) {
        C.q[pos] = key;
        C.qv[pos] = v;
      }
      qlen += all;
    }
    i += kk;
    team_sync(team);
  }
  if (tt == 0) {
    if (C.status != SS_SUCCESS) {
      C.entries = i;
      C.qlen = min(qlen, PRESSURE_SEARCH);
    } else {
      // does the pull leave its own cell full? (its flow is planned on the footprint just read)
      float fv[7];
#pragma unroll
      for (int l = 0; l < 7; ++l) fv[l] = C.fv[l];
      const FlowPlan P = flow_plan(fv, flags & 0x7Fu, __fadd_rn(vol, C.got));
      C.full = P.vol >= FULL ? 1u : 0u;
    }
  }
}

// Did the search of team w read the source of team o's pull (as a queue entry or beside one)?
__device__ void lv_hits(LvSmem& L, int w, int o) {
  Search& C = L.s[w];
  const Search& S = L.s[o];
  const int rx = S.sx - C.cx, ry = S.sy - C.cy, rz = S.sz - C.cz;
  bool hit = false;
  for (unsigned t = threadIdx.x % TEAM_THREADS; t < C.qlen; t += TEAM_THREADS) {
    int a, b, c;
    rel_unpack(C.q[t], a, b, c);
    const int ex = abs(rx - a), ey = ry - b, ez = abs(rz - c);
    hit |= (ey == 0 || ey == 1) && ex + ez + ey <= 1;
  }
  if (hit) atomicOr(&C.hit, 1u << o);
}

// The write of a committed pull's source (fluid.rs:536-540), one warp.
__device__ void lv_source(const Region& R, LvSmem& L, const int* ring, int team, int& pd, unsigned long long cap) {
  const Search& C = L.s[team];
  const unsigned lane = lane_id();
  const float nv = __fsub_rn(C.here, C.got);
  CD c = CD{0.0f, NOSLOT, 0u, 0, true};
  if (lane == 0) c = load_cell_par(R, ring, C.sx, C.sy, C.sz, cap);
  const bool need = lane == 0 && c.slot == NOSLOT && set_volume_needs_slot(c, nv);
  if (__any_sync(FULLMASK, need)) materialize_par(R, need, c.gi, c.slot, cap);
  if (lane == 0) {
    const unsigned sid = dom_id(R, C.sx, C.sy, C.sz);
    const SVPlan p = sv_plan(c.part, c.mat, c.slot != NOSLOT, nv);
    if (c.slot != NOSLOT) sv_apply(R, (size_t)c.slot * 512u + local_index(C.sx, C.sy, C.sz), p);
    pd += p.dp;
    R.lv_src[C.pos] = sid;
    // activation slots 0 (the source) and 1 (around the cell); bit 17 seeds the source
    L.res_ev[team] = 3u | (p.ch ? 0x8000u : 0u) | (2u << 16);
    // a drained source that was full attempts a pull of its own when its turn comes
    const unsigned j = R.stamp[sid];
    if (j != NOSLOT && nv < full_level() && !bit_of(L.att, j) && !(atomicOr(R.pextra + (j >> 5), 1u << (j & 31u)) & (1u << (j & 31u)))) {
      R.pxlist[atomicAdd(&L.nx, 1u)] = j;
      if (j < L.kp) atomicOr(&L.pp[j >> 5], 1u << (j & 31u));
    }
  }
  __syncwarp();
}

// After a round, one warp: the first pp cell in sorted order and its layer (the gate), and the pulls
// whose turn has come: the first pp cells that are all pending, up to one per team (none while the
// first one waits for an earlier cell).
__device__ void lv_head(const Region& R, LvSmem& L, unsigned n, int teams) {
  const unsigned lane = lane_id(), ngrp = (n + 31u) / 32u;
  if (L.head < n && bit_of(L.pp, L.head) && (!bit_of(L.pend, L.head) || (L.hblk && !cell_done(L, L.hblk - 1u)))) {
    if (lane == 0) L.nsearch = 0u;  // the first pp cell has yet to have its turn
    return;
  }
  unsigned w = L.hword;
  unsigned P = 0, any = 0;
  while (w < ngrp) {
    P = w + lane < ngrp ? L.pp[w + lane] : 0u;
    any = __ballot_sync(FULLMASK, P != 0u);
    if (any) break;
    w += 32u;
  }
  if (!any) {
    if (lane == 0) {
      L.hword = ngrp;
      L.head = n;
      L.gate = 0x7FFFFFFF;
      L.nsearch = 0u;
    }
    return;
  }
  const int fl = __ffs(any) - 1;
  const unsigned head = (w + (unsigned)fl) * 32u + (unsigned)__ffs(__shfl_sync(FULLMASK, P, fl)) - 1u;
  const unsigned old = L.head, hblk = head == old ? L.hblk : 0u;
  int gate = L.gate;
  unsigned lend = L.lend;
  if (head >= lend) {  // a new gate layer: its first position after the layer, by a 32-way search
    gate = R.lv[head].y;
    const unsigned lim = (unsigned)(gate + 1) * (unsigned)R.PZ * (unsigned)R.PX;
    unsigned lo = head, hi = n;  // cells[lo] is on the layer; the answer lies in (lo, hi]
    while (hi - lo > 1u) {
      const unsigned st = (hi - lo + 31u) / 32u, p = lo + (lane + 1u) * st;
      const unsigned b = __ballot_sync(FULLMASK, p < hi && R.cells[p] < lim);
      const unsigned k = (unsigned)__popc(b);  // keys ascend: the first k probes are on the layer
      const unsigned nlo = lo + k * st, nhi = min(hi, lo + (k + 1u) * st);
      lo = nlo;
      hi = nhi;
    }
    lend = hi;
  }
  __syncwarp();
  const bool ready = bit_of(L.pend, head) && (hblk == 0u || cell_done(L, hblk - 1u));
  unsigned m = 0;
  if (ready) {
    const unsigned D = w + lane < ngrp ? L.pend[w + lane] : 0u;
    const unsigned no = P & ~D;  // pp cells whose turn has not come: candidates end before the first
    const unsigned nb = __ballot_sync(FULLMASK, no != 0u);
    const int nl = nb ? __ffs(nb) - 1 : 32;
    unsigned c = (int)lane < nl ? P : ((int)lane == nl ? P & ((no & (0u - no)) - 1u) : 0u);
    while (m < (unsigned)teams) {
      const unsigned cb = __ballot_sync(FULLMASK, c != 0u);
      if (!cb) break;
      if ((int)lane == __ffs(cb) - 1) {
        L.cand[m] = (w + lane) * 32u + (unsigned)__ffs(c) - 1u;
        c &= c - 1u;
      }
      ++m;
    }
  }
  if (lane == 0) {
    L.hword = w + (unsigned)fl;
    L.head = head;
    L.hblk = hblk;
    L.gate = gate;
    L.lend = lend;
    L.nsearch = m;
  }
}

// The searches of the pulls lv_head picked, side by side; the longest prefix whose searches would have
// found the same one after another commits. All threads; ends with a barrier.
__device__ void lv_pulls(const Region& R, LvSmem& L, const int* ring, int m, int& pd, unsigned long long cap) {
  const unsigned tid = threadIdx.x;
  const int team = (int)(tid / TEAM_THREADS);
  if (team < m) lv_search(R, L, ring, team, L.cand[team], cap);
  __syncthreads();
  if (m > 1) {
    if (team < m && L.s[team].status != SS_BLOCKED)
      for (int o = 0; o < team; ++o)
        if (L.s[o].status == SS_SUCCESS) lv_hits(L, team, o);
    __syncthreads();
  }
  if (tid == 0) {
    int c = 0;
    unsigned won = 0u;
    while (c < m) {
      const Search& S = L.s[c];
      if (S.status == SS_BLOCKED) {
        if (c == 0) L.hblk = S.blk;
        L.n_again += 1u;
        break;
      }
      if (S.hit & won) break;
      L.res_ev[c] = 0u;
      L.pend[S.pos >> 5] &= ~(1u << (S.pos & 31u));
      bool stop = false;
      if (S.status == SS_SUCCESS) {
        won |= 1u << c;
        L.n_succ += 1u;
        if (S.full) {  // its later neighbours on the layer may start from it
          const LvCell& rc = R.lv[S.pos];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const unsigned nb = rc.succ[q == 0 ? 0 : 3];
            if (nb == NOSUCC || nb >= L.kp || !bit_of(L.att, nb) || bit_of(L.pp, nb)) continue;
            L.pp[nb >> 5] |= 1u << (nb & 31u);
            stop |= c + 1 < m && nb < L.cand[c + 1];
          }
        }
      }
      L.n_entries += S.entries;
      L.n_searches += 1u;
      ++c;
      if (stop) break;
    }
    L.ncommit = (unsigned)c;
  }
  __syncthreads();
  if (team < (int)L.ncommit && L.s[team].status == SS_SUCCESS && tid % TEAM_THREADS < 32u) lv_source(R, L, ring, team, pd, cap);
  __syncthreads();
}

}  // namespace vfe
