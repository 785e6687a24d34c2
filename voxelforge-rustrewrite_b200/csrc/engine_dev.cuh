// Warp-cooperative device rules of the reference's fluid (src/fluid.rs:292-657) shared by the tick and
// the host edits: cell loads, set_volume, activation, brick allocation and the one-warp parts of the
// levelling.
#pragma once
#include "engine.cuh"

namespace vfe {

constexpr unsigned FULLMASK = 0xFFFFFFFFu;

__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// f32 constant 1.0 - 1e-4 folded in f32 (fluid.rs:323, :337, :513, :594).
__device__ __forceinline__ float full_level() { return __fsub_rn(1.0f, 1e-4f); }

// ---------------------------------------------------------------------------- world reads
__device__ __forceinline__ bool chunk_loaded(const Region& R, const int* ring, int cx, int cz) {  // sparse_volume.rs:164-170
  int m = R.ring_w - 1;
  int i = ((cz & m) * R.ring_w + (cx & m)) * 3;
  return ring[i + 2] != 0 && ring[i] == cx && ring[i + 1] == cz;
}

__device__ __forceinline__ bool outside(const Region& R, const int* ring, int x, int y, int z) {  // fluid.rs:212-217
  if (y < 0 || y >= R.ny) return true;
  if (R.ring_w) return !chunk_loaded(R, ring, x >> 7, z >> 7);
  return x < 0 || z < 0 || x >= R.nx || z >= R.nz;
}

__device__ __forceinline__ unsigned local_index(int x, int y, int z) { return ((unsigned)(z & 7) << 6) | ((unsigned)(y & 7) << 3) | (unsigned)(x & 7); }

__device__ __forceinline__ CD load_cell(const Region& R, const int* ring, int x, int y, int z) {
  CD c;
  c.part = 0.0f;
  c.slot = NOSLOT;
  c.gi = 0;
  c.mat = 0;
  c.out = outside(R, ring, x, y, z);
  if (c.out) return c;
  c.gi = grid_index(R, x >> 3, y >> 3, z >> 3);
  unsigned g = R.grid[c.gi];
  if (g < 256u) {
    c.mat = (unsigned char)g;
    return c;
  }
  c.slot = g - 256u;
  size_t o = (size_t)c.slot * 512u + local_index(x, y, z);
  c.mat = R.amat[o];
  c.part = R.avol[o];
  return c;
}

// Warp-uniform scheduler state of one region: a tick's, or a host edit's.
struct WS {
  unsigned long long qhead, qtail;
  unsigned long long activations, pull_attempts, pull_success, bfs_visits, level_cells_total;
  long long pdelta;        // partial_count delta (lane-local, reduced at the end)
  unsigned nseeds;
  unsigned llc;            // last_level_cells
  unsigned ndrain;         // layers drained to a film (fluid.rs:456-481) since the handle's start
  bool level_round;
  bool changed;
  // Inside a tick the scheduler side effects are logged in program order and committed in
  // parallel at the tick's end (deferred); host edits apply them at once.
  bool deferred;
  unsigned nact, nseed, nchg;  // event-log cursors (deferred mode)
};

constexpr unsigned EMPTY_ID = 0xFFFFFFFFu;

struct Smem {
  const int* ring;
};

__device__ __forceinline__ void set_status(const Region& R, int st, unsigned info) {
  if (atomicCAS(&R.ctl->status, 0, st) == 0) R.ctl->err_info = info;
}

// ---------------------------------------------------------------------- materialisation
// Bricks that are uniform grid values get an atlas slot before their first write (the
// reference's SparseVolume::materialize, sparse_volume.rs:250-266; partial pages, fluid.rs:108-128).
// Lanes with `need` name a grid index; one leader per distinct index allocates, the warp fills.
__device__ void materialize_lanes(const Region& R, bool need, unsigned gi, unsigned& slot) {
  const unsigned lane = lane_id();
  unsigned key = need ? gi : (0xFFFFFFFFu - lane);
  unsigned peers = __match_any_sync(FULLMASK, key);
  bool leader = need && !(peers & lanemask_lt());
  unsigned lead_mask = __ballot_sync(FULLMASK, leader);
  if (!lead_mask) return;
  unsigned s = NOSLOT;
  unsigned g = 0;
  if (leader) {
    g = R.grid[gi];
    if (g >= 256u) {
      s = g - 256u;
    } else {
      s = atomicAdd(&R.ctl->atlas_used, 1u);
      if (s >= R.atlas_cap) {
        set_status(R, ST_OOM, 1);
        s = NOSLOT;
      }
    }
  }
  // cooperative fill of each new slot
  for (unsigned m = lead_mask; m; m &= m - 1) {
    int l = __ffs(m) - 1;
    unsigned sl = __shfl_sync(FULLMASK, s, l);
    unsigned gv = __shfl_sync(FULLMASK, g, l);
    if (sl != NOSLOT && gv < 256u) {
      unsigned fill = gv & 255u;
      fill |= fill << 8;
      fill |= fill << 16;
      uint4 f4 = make_uint4(fill, fill, fill, fill);
      reinterpret_cast<uint4*>(R.amat + (size_t)sl * 512u)[lane] = f4;
      uint4 z4 = make_uint4(0, 0, 0, 0);
      uint4* vv = reinterpret_cast<uint4*>(R.avol + (size_t)sl * 512u);
#pragma unroll
      for (int k = 0; k < 4; ++k) vv[lane + 32 * k] = z4;
    }
  }
  __syncwarp();
  // publish the slot after its fill (release)
  __threadfence_block();
  if (leader && s != NOSLOT && g < 256u) *(volatile unsigned*)(R.grid + gi) = 256u + s;
  int src = need ? (__ffs(peers) - 1) : (int)lane;
  unsigned s2 = __shfl_sync(FULLMASK, s, src);
  if (need) slot = s2;
  __syncwarp();
}

// --------------------------------------------------------------------------- writes
__device__ __forceinline__ void record_change(const Region& R, unsigned id) {
  unsigned old = atomicOr(&R.chgbits[id >> 5], 1u << (id & 31));
  if (!(old & (1u << (id & 31)))) {
    unsigned long long i = atomicAdd(&R.ctl->nchg, 1ull);
    if (i < R.chg_cap) R.chg[i] = id;
    else set_status(R, ST_OOM, 2);
  }
}

// The dense word of a cell after its atlas entry was written.
__device__ __forceinline__ void dense_put(const Region& R, unsigned id, unsigned mat, float part) { R.dense[id] = dense_code(false, mat, __float_as_uint(part)); }
__device__ __forceinline__ float dc_volume(unsigned u) { return __uint_as_float(u & 0x7FFFFFFFu); }
// FluidSim::volume as the levelling tests it (> 0, >= 1 - 1e-4): a solid cell's partial entry counts as
// water there (fluid.rs:251-260 looks at the entry first).
__device__ __forceinline__ float dc_level(unsigned u) { return u == DC_SOLID ? 0.0f : u == DC_SOLID_PART ? 1.0f : dc_volume(u); }
__device__ __forceinline__ unsigned dense_at(const Region& R, int x, int y, int z) { return in_dom(R, x, y, z) ? R.dense[dom_id(R, x, y, z)] : DC_SOLID; }

__device__ __forceinline__ void erase_part(const Region& R, CD& c, unsigned l, unsigned id, long long& pdelta) {
  if (c.slot != NOSLOT && c.part > 0.0f) {
    R.avol[(size_t)c.slot * 512u + l] = 0.0f;
    dense_put(R, id, c.mat, 0.0f);
    c.part = 0.0f;
    pdelta -= 1;
  }
}

// Does set_volume(c, vol) write into the brick (so a uniform brick needs a slot first)?
__device__ __forceinline__ bool set_volume_needs_slot(const CD& c, float vol) {
  if (c.slot != NOSLOT) return false;
  bool is_water = c.mat == WATER;
  if (vol <= 1e-6f) return is_water;
  if (vol >= full_level()) return !is_water;
  return true;
}

// FluidSim::set_volume (fluid.rs:327-355) on one lane's cell; c.slot must be valid when
// set_volume_needs_slot said so. Returns "the voxel changed". Written as selects: the snapping
// (<= 1e-6 -> 0, >= 1-1e-4 -> full), the partial entry and the show/hide hysteresis each decide a
// value, and the stores are predicated.
__device__ __forceinline__ bool set_volume_lane(const Region& R, CD& c, int x, int y, int z, unsigned id, float vol, long long& pdelta,
                                                bool deferred = false) {
  const unsigned l = local_index(x, y, z);
  const bool is_water = c.mat == WATER;
  const bool has = c.slot != NOSLOT;  // false only when materialisation failed (status set)
  const bool low = vol <= 1e-6f;
  const bool high = !low && vol >= full_level();
  const bool mid = !low && !high;
  const bool had = has && c.part > 0.0f;
  const float npart = mid ? vol : 0.0f;
  const unsigned char nmat = low ? (unsigned char)0
                           : high ? (unsigned char)WATER
                           : (is_water && vol < HIDE_BELOW) ? (unsigned char)0
                           : (!is_water && vol >= SHOW_AT) ? (unsigned char)WATER
                           : c.mat;
  const bool wpart = has && (mid || had);
  const bool wmat = has && nmat != c.mat;
  const bool ch = mid ? wmat : nmat != c.mat;
  pdelta += (mid && has && !had) ? 1 : 0;
  pdelta -= (!mid && had) ? 1 : 0;
  if (wpart) R.avol[(size_t)c.slot * 512u + l] = npart;
  if (wmat) R.amat[(size_t)c.slot * 512u + l] = nmat;
  if (has) c.part = npart;
  if (wmat) c.mat = nmat;
  if (has) dense_put(R, id, c.mat, npart);
  if (wmat && !deferred) record_change(R, id);
  return ch;
}

// Append per-lane events (lane order) to a log; returns the new cursor.
__device__ __forceinline__ unsigned log_append(const Region& R, unsigned* log, unsigned cap, unsigned cur, bool v, unsigned id, unsigned site) {
  unsigned b = __ballot_sync(FULLMASK, v);
  if (v) {
    unsigned pos = cur + (unsigned)__popc(b & lanemask_lt());
    if (pos < cap) log[pos] = id;
    else set_status(R, ST_OOM, site);
  }
  return cur + (unsigned)__popc(b);
}

// Warp: lanes with `w` write `vol` into their cell through set_volume. Returns whether any
// voxel changed.
__device__ bool warp_set_volume(const Region& R, WS& W, bool w, CD& c, int x, int y, int z, float vol) {
  bool need = w && set_volume_needs_slot(c, vol);
  if (__any_sync(FULLMASK, need)) materialize_lanes(R, need, c.gi, c.slot);
  bool ch = false;
  const unsigned id = (w && in_dom(R, x, y, z)) ? dom_id(R, x, y, z) : 0u;
  if (w) ch = set_volume_lane(R, c, x, y, z, id, vol, W.pdelta, W.deferred);
  if (W.deferred) W.nchg = log_append(R, R.ev_chg, R.ev_chg_cap, W.nchg, ch, id, 9);
  __syncwarp();
  return __any_sync(FULLMASK, ch);
}

// ---------------------------------------------------------------------------- activation
// Push cells (one per lane, lane order = program order) that are not active yet.
__device__ __forceinline__ void activate_round(const Region& R, WS& W, bool valid, int x, int y, int z) {
  const unsigned lane = lane_id();
  unsigned id = 0;
  if (valid) {
    if (y < 0) valid = false;  // fluid.rs:293-295
    else if (!in_dom(R, x, y, z)) {
      set_status(R, ST_RANGE, 3);
      valid = false;
    } else {
      id = dom_id(R, x, y, z);
    }
  }
  unsigned peers = __match_any_sync(FULLMASK, valid ? id : (0xFFFFFFFFu - lane));
  bool first = valid && !(peers & lanemask_lt());
  if (W.deferred) {  // inside a tick: log in program order, the tick's end commits
    W.nact = log_append(R, R.ev_act, R.ev_act_cap, W.nact, first, id, 10);
    __syncwarp();
    return;
  }
  bool isnew = false;
  if (first) isnew = !((R.active[id >> 5] >> (id & 31)) & 1u);
  unsigned nb = __ballot_sync(FULLMASK, isnew);
  if (isnew) {
    unsigned long long pos = W.qtail + (unsigned long long)__popc(nb & lanemask_lt());
    R.queue[pos & R.qmask] = id;
    atomicOr(&R.active[id >> 5], 1u << (id & 31));
  }
  W.qtail += (unsigned long long)__popc(nb);
  W.activations += (unsigned long long)__popc(nb);
  __syncwarp();
}

// Activation-log word: the cell id, bit 31 set for a wake_around centre (7 cells).
constexpr unsigned ACT_AROUND = 0x80000000u;

// ------------------------------------------------------------------------ level fill
// LayerMarks::test_and_set (fluid.rs:194-200): one bit per cell in 64x64 tiles per layer; the
// tiles touched during a levelling round are listed so the round's end clears only those.
__device__ __forceinline__ bool mark_tas(const Region& R, int x, int y, int z) {
  if (!in_dom(R, x, y, z)) {  // cannot happen for neighbours of addressable cells; never write out of range
    set_status(R, ST_RANGE, 8);
    return true;
  }
  unsigned xr = (unsigned)(x - R.px0), zr = (unsigned)(z - R.pz0);
  unsigned tile = ((zr >> 6) * (unsigned)R.PY + (unsigned)y) * (unsigned)R.TX + (xr >> 6);
  unsigned bit = ((zr & 63u) << 6) | (xr & 63u);
  unsigned old = atomicOr(&R.marks[(size_t)tile * 128u + (bit >> 5)], 1u << (bit & 31));
  if (R.mark_tflag[tile] == 0u && atomicExch(&R.mark_tflag[tile], 1u) == 0u) {
    unsigned k = atomicAdd(&R.ctl->mark_ntiles, 1u);
    R.mark_list[k] = tile;
  }
  return (old >> (bit & 31)) & 1u;
}

// LayerMarks::test_and_set of a cell known to be unmarked, in two halves so that the caller's other
// loads overlap them: mark_begin sets the bit (no result wanted) and reads the tile's listed flag,
// mark_end lists the tile if nobody has.
__device__ __forceinline__ unsigned mark_begin(const Region& R, int x, int y, int z, unsigned& tile) {
  const unsigned xr = (unsigned)(x - R.px0), zr = (unsigned)(z - R.pz0);
  tile = ((zr >> 6) * (unsigned)R.PY + (unsigned)y) * (unsigned)R.TX + (xr >> 6);
  const unsigned bit = ((zr & 63u) << 6) | (xr & 63u);
  atomicOr(&R.marks[(size_t)tile * 128u + (bit >> 5)], 1u << (bit & 31));
  return __ldcg(R.mark_tflag + tile);  // set by atomics (in L2): read past L1
}
__device__ __forceinline__ void mark_end(const Region& R, unsigned tile, unsigned listed) {
  if (listed == 0u && atomicExch(&R.mark_tflag[tile], 1u) == 0u) {
    const unsigned k = atomicAdd(&R.ctl->mark_ntiles, 1u);
    R.mark_list[k] = tile;
  }
}

__device__ __forceinline__ void side4(int d, int& dx, int& dz) {  // SIDES (fluid.rs:228)
  dx = (d == 0) - (d == 1);
  dz = (d == 2) - (d == 3);
}

// FluidSim::level_layer's membership test (fluid.rs:413-415) of (x, y, z): !solid && vol > 0 &&
// supported && vol(above) <= 0. Returns the cell's volume through *v.
__device__ __forceinline__ bool level_member(const Region& R, int x, int y, int z, float* v) {
  const unsigned c = dense_at(R, x, y, z);
  *v = dc_level(c);
  if (dc_solid(c) || !(*v > 0.0f)) return false;
  const unsigned b = dense_at(R, x, y - 1, z), a = dense_at(R, x, y + 1, z);  // inside the domain: the cell is in the world
  return (dc_solid(b) || dc_volume(b) >= full_level()) && !(dc_level(a) > 0.0f);
}

// The flood fill of FluidSim::level_layer (fluid.rs:425-446) continued by one warp from queue
// entry i of len (R.lvl_id / R.lvl_vol): entries are examined in order, each testing its four
// sides once (LayerMarks) and appending the members. Stops early, with i < len, when `hand` or
// more entries wait (the CTA takes the layer over from there). Returns the length.
__device__ unsigned level_bfs_warp(const Region& R, Smem& S, unsigned& i, unsigned len, unsigned hand) {
  const unsigned lane = lane_id();
  const float FULL = full_level();
  while (i < len) {
    if (len >= MAX_LEVEL_CELLS) {  // the rest is only summed (fluid.rs:436-438)
      i = len;
      break;
    }
    if (len - i >= hand) break;
    unsigned cid = R.lvl_id[i];
    ++i;
    int x, y, z;
    dom_xyz(R, cid, x, y, z);
    // lanes 0..11: side d = lane/3, j = lane%3 (0 the neighbour, 1 below it, 2 above it)
    int d = (int)lane / 3, j = (int)lane % 3;
    int dx = 0, dz = 0;
    if (lane < 12) side4(d, dx, dz);
    int nx = x + dx, nz = z + dz;
    bool skip = lane >= 12 || (R.ring_w == 0 && (nx < 0 || nz < 0));
    unsigned tas = 0;
    if (!skip && j == 0) tas = mark_tas(R, nx, y, nz);
    const unsigned c = skip ? DC_SOLID : dense_at(R, nx, y + (j == 1 ? -1 : (j == 2 ? 1 : 0)), nz);
    // gather the three cells of each side at its j==0 lane
    const bool sol = dc_solid(c);
    const float v = dc_level(c);
    float v1 = __shfl_down_sync(FULLMASK, v, 1), v2 = __shfl_down_sync(FULLMASK, v, 2);
    bool s1 = __shfl_down_sync(FULLMASK, (unsigned)sol, 1) != 0u;
    bool push = !skip && j == 0 && !tas && !sol && v > 0.0f && (s1 || v1 >= FULL) && v2 <= 0.0f;
    unsigned pm = __ballot_sync(FULLMASK, push);
    if (push) {
      unsigned pos = len + (unsigned)__popc(pm & lanemask_lt());
      R.lvl_id[pos] = dom_id(R, nx, y, nz);
      R.lvl_vol[pos] = v;
    }
    len += (unsigned)__popc(pm);
    __syncwarp();
  }
  return len;
}

// The sum and range of the gathered volumes in queue order (fluid.rs:431-434), one lane adding in
// f64 in order; the result is broadcast to the warp.
__device__ void level_sum_warp(const Region& R, unsigned len, double& sum, float& lo, float& hi) {
  double s = 0.0;
  float l = 2.0f, h = -1.0f;
  if (lane_id() == 0) {
    for (unsigned i = 0; i < len; ++i) {
      const float v = R.lvl_vol[i];
      s = __dadd_rn(s, (double)v);
      l = fminf(l, v);
      h = fmaxf(h, v);
    }
  }
  sum = __shfl_sync(FULLMASK, s, 0);
  lo = __shfl_sync(FULLMASK, l, 0);
  hi = __shfl_sync(FULLMASK, h, 0);
}

// What FluidSim::level_layer does with a gathered layer (fluid.rs:446-485), one warp: count the
// cells, then level to the average or drain the film. Returns "a voxel changed".
__device__ bool level_finish(const Region& R, WS& W, Smem& S, unsigned len, double sum, float lo, float hi);

// FluidSim::level_layer (fluid.rs:412-486), one warp. Cells are gathered in the exact BFS order of
// the reference and summed in that order in f64. A layer whose flood fill grows to `hand` waiting
// entries is handed over: returns true with the queue state in qi / qlen, nothing levelled yet.
__device__ bool level_layer(const Region& R, WS& W, Smem& S, int sx, int sy, int sz, unsigned hand, unsigned& qi,
                            unsigned& qlen) {
  const unsigned lane = lane_id();
  unsigned was = 0;
  if (lane == 0) was = mark_tas(R, sx, sy, sz);
  was = __shfl_sync(FULLMASK, was, 0);
  if (was) return false;
  float v0 = 0.0f;
  const bool member = level_member(R, sx, sy, sz, &v0);
  if (!member) return false;
  if (lane == 0) {
    R.lvl_id[0] = dom_id(R, sx, sy, sz);
    R.lvl_vol[0] = v0;
  }
  __syncwarp();
  unsigned i = 0;
  const unsigned len = level_bfs_warp(R, S, i, 1u, hand);
  if (i < len) {
    qi = i;
    qlen = len;
    return true;
  }
  double sum;
  float lo, hi;
  level_sum_warp(R, len, sum, lo, hi);
  W.changed |= level_finish(R, W, S, len, sum, lo, hi);
  return false;
}

__device__ bool level_finish(const Region& R, WS& W, Smem& S, unsigned len, double sum, float lo, float hi) {
  const unsigned lane = lane_id();
  W.llc += len;
  W.level_cells_total += len;
  bool changed = false;
  if (len >= 2 && __fsub_rn(hi, lo) >= SLEEP) {
    const float avg = __double2float_rn(__ddiv_rn(sum, (double)len));
    if (avg >= MIN_SPREAD) {  // fluid.rs:449-455
      for (unsigned b0 = 0; b0 < len; b0 += 32) {
        unsigned k = b0 + lane;
        bool wv = false;
        int x = 0, y = 0, z = 0;
        CD c = CD{0.0f, NOSLOT, 0u, 0, true};
        if (k < len) {
          dom_xyz(R, R.lvl_id[k], x, y, z);
          c = load_cell(R, S.ring, x, y, z);
          wv = fabsf(__fsub_rn(cd_volume(c), avg)) > 1e-6f;
        }
        changed |= warp_set_volume(R, W, wv, c, x, y, z, avg);
      }
    } else {  // drain into the water under the film (fluid.rs:456-481)
      W.ndrain += 1;
      double left = sum;
      bool stop = false;
      for (unsigned b0 = 0; b0 < len && !stop; b0 += 32) {
        unsigned k = b0 + lane;
        int x = 0, y = 0, z = 0;
        CD c = CD{0.0f, NOSLOT, 0u, 0, true};
        bool ok = false;
        if (k < len) {
          dom_xyz(R, R.lvl_id[k], x, y, z);
          if (y != 0) {
            c = load_cell(R, S.ring, x, y - 1, z);
            ok = !cd_solid(c);
          }
        }
        float bel = cd_volume(c);
        // sequential in cell order: take = min(left, 1 - below)
        bool wv = false;
        float nvv = 0.0f;
        unsigned n_here = min(32u, len - b0);
        for (unsigned t = 0; t < n_here; ++t) {
          bool okt = __shfl_sync(FULLMASK, ok, t);
          float bt = __shfl_sync(FULLMASK, bel, t);
          if (!okt) continue;
          float take = __double2float_rn(fmin(left, (double)__fsub_rn(1.0f, bt)));
          if (take <= 0.0f) continue;
          if (lane == t) {
            wv = true;
            nvv = __fadd_rn(bt, take);
          }
          left = __dsub_rn(left, (double)take);
          if (left <= 1e-6) {
            stop = true;
            break;
          }
        }
        changed |= warp_set_volume(R, W, wv, c, x, y - 1, z, nvv);
        // activations in cell order (fluid.rs:472)
        unsigned am = __ballot_sync(FULLMASK, wv);
        for (unsigned m = am; m; m &= m - 1) {
          int l = __ffs(m) - 1;
          int ax = __shfl_sync(FULLMASK, x, l), ay = __shfl_sync(FULLMASK, y, l), az = __shfl_sync(FULLMASK, z, l);
          activate_round(R, W, lane == 0, ax, ay - 1, az);
        }
      }
      const float rest = __double2float_rn(__ddiv_rn(left, (double)len));
      const float rv = rest < EVAPORATE ? 0.0f : rest;
      for (unsigned b0 = 0; b0 < len; b0 += 32) {
        unsigned k = b0 + lane;
        int x = 0, y = 0, z = 0;
        CD c = CD{0.0f, NOSLOT, 0u, 0, true};
        bool wv = k < len;
        if (wv) {
          dom_xyz(R, R.lvl_id[k], x, y, z);
          c = load_cell(R, S.ring, x, y, z);
        }
        changed |= warp_set_volume(R, W, wv, c, x, y, z, rv);
      }
    }
  }
  return changed;
}

}  // namespace vfe
