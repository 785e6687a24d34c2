// Kernels of the CA-water engine: the tick (drain -> sort -> sweep -> levelling) for one or many
// regions, host-edit kernels (wake, displace, brush, emitters, set_partial) and inspection
// kernels (digests, dense export, change download).
#pragma once
#include <cuda_fp16.h>

#include "engine_dev.cuh"
#include "sweep_lvl.cuh"

namespace vfe {

// blockDim-derived thread / warp counts of the running CTA
#define NT_ ((unsigned)blockDim.x)
#define NW_ ((unsigned)(blockDim.x >> 5))

// Launch shape: MAX_WARPS warps per region. CTA-wide helpers use the launched block size; shared arrays
// are sized for the full one.
constexpr int PAR_THREADS = MAX_WARPS * 32;

// ---------------------------------------------------------------- CTA radix sort (LSD, 8 bit)
// Stable within each warp's contiguous chunk; chunks in order -> stable overall. Sorts n unique
// keys in place (tmp is scratch). hist: NW_*256 u32 of shared memory.
__device__ void cta_radix_sort(unsigned* keys, unsigned* tmp, unsigned n, unsigned* hist, unsigned* sred) {
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (n <= 1) return;
  // key range -> number of passes
  unsigned mn = 0xFFFFFFFFu, mx = 0;
  for (unsigned i = tid; i < n; i += NT_) {
    unsigned k = keys[i];
    mn = min(mn, k);
    mx = max(mx, k);
  }
  for (int o = 16; o; o >>= 1) {
    mn = min(mn, __shfl_xor_sync(FULLMASK, mn, o));
    mx = max(mx, __shfl_xor_sync(FULLMASK, mx, o));
  }
  if (lane == 0) {
    sred[warp] = mn;
    sred[NW_ + warp] = mx;
  }
  __syncthreads();
  if (tid == 0) {
    unsigned a = 0xFFFFFFFFu, b = 0;
    for (int w = 0; w < NW_; ++w) {
      a = min(a, sred[w]);
      b = max(b, sred[NW_ + w]);
    }
    sred[2 * NW_] = a;
    sred[2 * NW_ + 1] = b;
  }
  __syncthreads();
  const unsigned kmin = sred[2 * NW_], range = sred[2 * NW_ + 1] - kmin;
  __syncthreads();
  const int bits = range ? 32 - __clz(range) : 0;
  const int passes = (bits + 7) / 8;
  const unsigned chunk = (n + NW_ - 1) / NW_;
  const unsigned b0 = min(n, warp * chunk), b1 = min(n, b0 + chunk);
  unsigned* src = keys;
  unsigned* dst = tmp;
  for (int p = 0; p < passes; ++p) {
    const int sh = 8 * p;
    for (unsigned i = tid; i < NW_ * 256; i += NT_) hist[i] = 0;
    __syncthreads();
    for (unsigned i = b0 + lane; i < b1; i += 128) {  // four loads under way at a time
      unsigned k[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) k[q] = i + 32u * q < b1 ? src[i + 32u * q] : 0u;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (i + 32u * q < b1) atomicAdd(&hist[warp * 256 + (((k[q] - kmin) >> sh) & 255u)], 1u);
    }
    __syncthreads();
    // offsets: digit-major, warp-minor
    if (tid < 256) {
      unsigned s = 0;
      for (int w = 0; w < NW_; ++w) s += hist[w * 256 + tid];
      sred[tid] = s;
    }
    __syncthreads();
    if (tid < 32) {
      // exclusive scan of 256 digit totals by one warp (8 per lane)
      unsigned v[8], t = 0;
      for (int k = 0; k < 8; ++k) {
        v[k] = sred[lane * 8 + k];
        t += v[k];
      }
      unsigned incl = t;
      for (int o = 1; o < 32; o <<= 1) {
        unsigned u = __shfl_up_sync(FULLMASK, incl, o);
        if (lane >= (unsigned)o) incl += u;
      }
      unsigned run = incl - t;
      for (int k = 0; k < 8; ++k) {
        sred[256 + lane * 8 + k] = run;
        run += v[k];
      }
    }
    __syncthreads();
    if (tid < 256) {
      unsigned run = sred[256 + tid];
      for (int w = 0; w < NW_; ++w) {
        unsigned c = hist[w * 256 + tid];
        hist[w * 256 + tid] = run;
        run += c;
      }
    }
    __syncthreads();
    unsigned ahead[3];  // the next three keys are on their way
#pragma unroll
    for (int q = 0; q < 3; ++q) ahead[q] = b0 + 32u * q + lane < b1 ? src[b0 + 32u * q + lane] : 0u;
    for (unsigned base = b0; base < b1; base += 32) {
      unsigned i = base + lane;
      bool valid = i < b1;
      const unsigned k = ahead[0];
      ahead[0] = ahead[1];
      ahead[1] = ahead[2];
      ahead[2] = i + 96u < b1 ? src[i + 96u] : 0u;
      unsigned d = valid ? (((k - kmin) >> sh) & 255u) : (256u + lane);
      unsigned peers = __match_any_sync(FULLMASK, d);
      unsigned rank = __popc(peers & lanemask_lt());
      unsigned pos = 0;
      if (valid) pos = hist[warp * 256 + d] + rank;
      __syncwarp();
      if (valid) {
        dst[pos] = k;
        if (rank == 0) hist[warp * 256 + d] += __popc(peers);
      }
      __syncwarp();
    }
    __syncthreads();
    unsigned* t = src;
    src = dst;
    dst = t;
  }
  if (src != keys) {
    for (unsigned i = tid; i < n; i += NT_) keys[i] = src[i];
    __syncthreads();
  }
}

// ----------------------------------------------------------------------------- the tick
// Launch-time knobs of the tick (results do not depend on them).
struct Tune {
  int gate;       // bits 16-20: warps of the region's CTA (0: MAX_WARPS); the other bits are unused
  unsigned long long spin_cap;  // rounds of the sweep before the tick gives up (ST_TIMEOUT)
};

struct TickSmem {
  unsigned sred[2 * 256 + 64];
  int ring[3 * 16 * 16];
  unsigned scan[MAX_WARPS + 1];
  union {
    LvSmem p;   // the sweep
    struct {    // before and after the sweep: the sort's histograms, then the levelling's tables
      unsigned hist[MAX_WARPS * 256];
      unsigned fills[MAX_WARPS * 1024];  // LevelFill per warp
    } x;
  } u;
};

__device__ void load_ws(const Region& R, WS& W) {
  const Ctl& c = *R.ctl;
  W.qhead = c.qhead;
  W.qtail = c.qtail;
  W.activations = 0;
  W.pull_attempts = 0;
  W.pull_success = 0;
  W.bfs_visits = 0;
  W.level_cells_total = 0;
  W.pdelta = 0;
  W.nseeds = c.nseeds;
  W.llc = c.last_level_cells;
  W.ndrain = 0;
  W.level_round = c.level_round != 0;
  W.changed = false;
  W.deferred = false;
  W.nact = W.nseed = W.nchg = 0;
}

// ----------------------------------------------------------------- CTA-wide ordered commits
// Exclusive prefix of per-thread flags over the CTA (in thread order). Returns this thread's
// offset; *total gets the CTA total. All threads must call.
__device__ unsigned cta_scan(TickSmem& sm, bool f, unsigned* total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  unsigned b = __ballot_sync(FULLMASK, f);
  if (lane == 0) sm.scan[warp] = __popc(b);
  __syncthreads();
  unsigned before = 0, all = 0;
  for (int w = 0; w < NW_; ++w) {
    unsigned c = sm.scan[w];
    if ((unsigned)w < warp) before += c;
    all += c;
  }
  __syncthreads();
  *total = all;
  return before + __popc(b & lanemask_lt());
}

// First occurrence of each cell id in an event log (stamp = lowest event index).
__device__ void stamp_first(const Region& R, const unsigned* ev, unsigned n) {
  for (unsigned i = threadIdx.x; i < n; i += NT_) atomicMin(&R.stamp[ev[i]], i);
  __syncthreads();
}
__device__ void stamp_clear(const Region& R, const unsigned* ev, unsigned n) {
  __syncthreads();
  for (unsigned i = threadIdx.x; i < n; i += NT_) R.stamp[ev[i]] = 0xFFFFFFFFu;
  __syncthreads();
}

// The sweep's FluidSim::activate calls in program order (fluid.rs:292-300): a cell joins the
// FIFO at its first activation if it was not active already.
// Exclusive prefix of per-thread counts over the CTA (thread order); *total = the CTA sum.
__device__ unsigned cta_scan_count(TickSmem& sm, unsigned c, unsigned* total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  unsigned incl = c;
  for (int o = 1; o < 32; o <<= 1) {
    unsigned u = __shfl_up_sync(FULLMASK, incl, o);
    if (lane >= (unsigned)o) incl += u;
  }
  if (lane == 31) sm.scan[warp] = incl;
  __syncthreads();
  const unsigned s = lane < NW_ ? sm.scan[lane] : 0u;
  const unsigned before = __reduce_add_sync(FULLMASK, lane < warp ? s : 0u);
  *total = __reduce_add_sync(FULLMASK, s);
  __syncthreads();
  return before + incl - c;
}

// Cell o of an activation-log word: a single cell, or wake_around's order self, +x, -x, +y, -y,
// +z, -z (fluid.rs:302-310). Returns false for cells activate() ignores (y < 0).
__device__ __forceinline__ bool act_cell(const Region& R, unsigned word, int o, unsigned& id) {
  const unsigned c = word & ~ACT_AROUND;
  if (!(word & ACT_AROUND)) {
    id = c;
    return o == 0;
  }
  const unsigned px = (unsigned)R.PX, pxy = px * (unsigned)R.PY;
  switch (o) {
    case 0: id = c; return true;
    case 1: id = c + 1u; return true;
    case 2: id = c - 1u; return true;
    case 3: id = c + px; return true;
    case 4: {  // y - 1 < 0
      id = c - px;
      const unsigned t = udiv(c, px, R.mx);
      return t != udiv(t, (unsigned)R.PY, R.my) * (unsigned)R.PY;
    }
    case 5: id = c + pxy; return true;
    default: id = c - pxy; return true;
  }
}

// The tick's FluidSim::activate calls in program order (fluid.rs:292-300): a cell joins the
// FIFO at its first activation if it was not active already. Log word i covers activation
// indices 8i..8i+6, which keeps program order for the first-occurrence stamps.
__device__ void commit_acts(const Region& R, TickSmem& sm, unsigned n, unsigned long long& qtail, unsigned long long qhead) {
  for (unsigned i = threadIdx.x; i < n; i += NT_) {
    unsigned w = R.ev_act[i], id;
    for (int o = 0; o < 7; ++o)
      if (act_cell(R, w, o, id)) atomicMin(&R.stamp[id], i * 8u + (unsigned)o);
  }
  __syncthreads();
  __shared__ unsigned long long s_tail;
  if (threadIdx.x == 0) s_tail = qtail;
  __syncthreads();
  for (unsigned base = 0; base < n; base += NT_) {
    const unsigned i = base + threadIdx.x;
    unsigned newmask = 0, w = 0;
    if (i < n) {
      w = R.ev_act[i];
      // the word's cells, then all their stamps and active words in flight together
      unsigned ids[7], st[7], ac[7];
      bool ok[7];
#pragma unroll
      for (int o = 0; o < 7; ++o) ok[o] = act_cell(R, w, o, ids[o]);
#pragma unroll
      for (int o = 0; o < 7; ++o) {
        st[o] = ok[o] ? R.stamp[ids[o]] : 0xFFFFFFFFu;
        ac[o] = ok[o] ? R.active[ids[o] >> 5] : 0u;
      }
#pragma unroll
      for (int o = 0; o < 7; ++o)
        if (ok[o] && st[o] == i * 8u + (unsigned)o && !((ac[o] >> (ids[o] & 31u)) & 1u)) newmask |= 1u << o;
    }
    unsigned total;
    unsigned off = cta_scan_count(sm, __popc(newmask), &total);
    for (int o = 0; o < 7; ++o) {
      if (!(newmask & (1u << o))) continue;
      unsigned id;
      act_cell(R, w, o, id);
      R.queue[(s_tail + off) & R.qmask] = id;
      atomicOr(&R.active[id >> 5], 1u << (id & 31));
      ++off;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_tail += total;
    __syncthreads();
  }
  qtail = s_tail;
  if (threadIdx.x == 0 && s_tail - qhead > R.qmask + 1ull) set_status(R, ST_OOM, 12);
  __syncthreads();
  for (unsigned i = threadIdx.x; i < n; i += NT_) {
    unsigned w = R.ev_act[i], id;
    for (int o = 0; o < 7; ++o)
      if (act_cell(R, w, o, id)) R.stamp[id] = 0xFFFFFFFFu;
  }
  __syncthreads();
}

// FluidSim::seed_level calls in order (fluid.rs:312-316): first insertion of a cell not yet a
// seed, while the set holds fewer than MAX_LEVEL_SEEDS.
__device__ void commit_seeds(const Region& R, TickSmem& sm, unsigned n, unsigned& nseeds) {
  stamp_first(R, R.ev_seed, n);
  __shared__ unsigned s_ns;
  if (threadIdx.x == 0) s_ns = nseeds;
  __syncthreads();
  for (unsigned base = 0; base < n; base += NT_) {
    unsigned i = base + threadIdx.x;
    bool isnew = false;
    unsigned id = 0;
    if (i < n) {
      id = R.ev_seed[i];
      isnew = R.stamp[id] == i && !((R.seedbits[id >> 5] >> (id & 31)) & 1u);
    }
    unsigned total;
    unsigned off = cta_scan(sm, isnew, &total);
    unsigned pos = s_ns + off;
    if (isnew && pos < MAX_LEVEL_SEEDS) {
      R.seeds[pos] = id;
      atomicOr(&R.seedbits[id >> 5], 1u << (id & 31));
    }
    __syncthreads();
    if (threadIdx.x == 0) s_ns = min(MAX_LEVEL_SEEDS, s_ns + total);
    __syncthreads();
  }
  nseeds = s_ns;
  stamp_clear(R, R.ev_seed, n);
}

// Voxel changes for the host (order irrelevant; the host sorts and dedups its dirty list).
__device__ void commit_chgs(const Region& R, unsigned n) {
  for (unsigned i = threadIdx.x; i < n; i += NT_) record_change(R, R.ev_chg[i]);
  __syncthreads();
}

// ------------------------------------------------------------------- the sweep
// Sum of a per-thread value over the CTA (all threads call).
__device__ unsigned long long cta_sum(TickSmem& sm, unsigned long long v) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(FULLMASK, v, o);
  __shared__ unsigned long long s_part[MAX_WARPS];
  if ((threadIdx.x & 31u) == 0) s_part[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned long long t = 0;
  for (unsigned w = 0; w < NW_; ++w) t += s_part[w];
  __syncthreads();
  return t;
}

// The sweep of one tick by the CTA (sweep_lvl.cuh describes the schedule). On return the tick's
// activation, seed and change logs hold the sweep's events in program order and sW its counters.
__device__ __noinline__ void sweep_levels(const Region& Rs, TickSmem& sm, WS& sW, const int* ring, unsigned n, bool flip, Tune tune) {
  LvSmem& L = sm.u.p;
  // The region's constants in registers: a round is a chain of dependent instructions, and behind
  // every store the compiler would read them from shared memory again (~30 cycles each).
  const Region R = Rs;
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const float FULL = full_level();
  const unsigned long long cap = tune.spin_cap;
  const unsigned ngrp = (n + 31u) / 32u;
  long long tp0 = clock64();
  auto plap = [&](int k) {
    if (tid == 0) {
      const long long now = clock64();
      R.ctl->pprof[k] += (unsigned long long)(now - tp0);
      tp0 = now;
    }
  };
  int pd = 0;
  // ---- positions, footprints, and the cells that attempt a pull or may find a start cell
  for (unsigned g = ngrp + tid; g <= NGROUPS; g += NT_) L.att[g] = L.pp[g] = 0u;
  for (unsigned g = tid; g < ngrp; g += NT_) R.pextra[g] = 0u;
  vis_reset(L.s, tid, NT_);
  if (tid == 0) {
    L.cnt[0] = L.cnt[1] = L.cnt[2] = 0u;
    L.cur = L.cc = L.pb = 0u;
    L.park_n[0] = L.park_n[1] = 0u;
    L.nx = 0u;
    L.kp = n;
    L.rounds = L.resume = L.timeout = 0u;
    L.n_succ = L.n_searches = L.n_again = 0u;
    L.n_entries = 0ull;
    L.hard = 0u;
  }
  for (unsigned g = warp; g < ngrp; g += NW_) {
    const unsigned i = g * 32u + lane;
    bool att = false, pp = false;
    if (i < n) {
      const unsigned cid = key_to_id(R, R.cells[i], flip);
      const unsigned u = R.dense[cid];
      R.lv_ev[i] = 0u;
      if (dc_solid(u)) {
        reinterpret_cast<unsigned char*>(L.dep)[i] = DONE;
        if (u == DC_SOLID_PART) {  // fluid.rs:586-589; nothing reads a solid cell's partial volume
          int x, y, z;
          dom_xyz(R, cid, x, y, z);
          const CD c = load_cell(R, ring, x, y, z);
          R.avol[(size_t)c.slot * 512u + local_index(x, y, z)] = 0.0f;
          R.dense[cid] = DC_SOLID;
          pd -= 1;
        }
      } else {
        unsigned nu[5];  // up, +x, -x, +z, -z
#pragma unroll
        for (int d = 0; d < 5; ++d) nu[d] = R.dense[(int)cid + fp_id(R, 2 + d)];
        reinterpret_cast<unsigned char*>(L.dep)[i] = 0;
        R.stamp[cid] = i;
        int x, y, z;
        dom_xyz(R, cid, x, y, z);
        unsigned ye = (unsigned)y;
        att = dc_volume(u) < FULL;
#pragma unroll
        for (int d = 0; d < 5; ++d) {
          const bool st = x + (d == 1) - (d == 2) >= 0 && z + (d == 3) - (d == 4) >= 0;
          ye |= st ? 1u << (27 + d) : 0u;
          pp |= att && st && !dc_solid(nu[d]) && dc_volume(nu[d]) >= FULL;
        }
        reinterpret_cast<uint2*>(R.lv + i)[3] = make_uint2(cid, ye);
      }
    }
    const unsigned ab = __ballot_sync(FULLMASK, att), pb = __ballot_sync(FULLMASK, pp);
    if (lane == 0) {
      L.att[g] = ab;
      L.pp[g] = pb;
    }
  }
  __syncthreads();
  // ---- attempts before each group, and the position from which the budget is spent at the latest
  unsigned total_att;
  {
    const unsigned per = (ngrp + NT_ - 1u) / NT_, g0 = min(ngrp, tid * per), g1 = min(ngrp, g0 + per);
    unsigned c = 0;
    for (unsigned g = g0; g < g1; ++g) c += (unsigned)__popc(L.att[g]);
    unsigned run = cta_scan_count(sm, c, &total_att);
    for (unsigned g = g0; g < g1; ++g) {
      const unsigned a = L.att[g], k = (unsigned)__popc(a);
      L.gpre[g] = (unsigned short)run;
      if (run < MAX_PULLS_PER_TICK && run + k >= MAX_PULLS_PER_TICK) {
        unsigned b = a;
        for (unsigned r = run + 1u; r < MAX_PULLS_PER_TICK; ++r) b &= b - 1u;
        L.kp = g * 32u + (unsigned)__ffs(b);  // after the last attempt of the budget
      }
      run += k;
    }
  }
  __syncthreads();
  const unsigned kp = L.kp;
  for (unsigned g = kp / 32u + tid; g < ngrp; g += NT_) L.pp[g] &= g == kp / 32u ? (1u << (kp & 31u)) - 1u : 0u;
  // ---- the later conflicting cells of every cell, and how many earlier ones each waits for
  const int sgn = flip ? -1 : 1;
  for (unsigned i = tid; i < n; i += NT_) {
    if (cell_done_now(L, i)) continue;
    const unsigned cid = R.lv[i].cid;
    unsigned s[12];
#pragma unroll
    for (int q = 0; q < 12; ++q) {
      int dx, dy, dz;
      succ_offset(q, sgn, dx, dy, dz);
      // (a cell of the world: what lies within two cells of it is inside the padded domain)
      const unsigned r = (q < 11 || i < kp) ? R.stamp[(int)cid + dx + (dz * R.PY + dy) * R.PX] : NOSLOT;
      s[q] = r == NOSLOT ? NOSUCC : r;
    }
#pragma unroll
    for (int q = 0; q < 12; ++q)
      if (s[q] != NOSUCC) atomicAdd(&L.dep[s[q] >> 2], 1u << ((s[q] & 3u) * 8u));
    uint4* o = reinterpret_cast<uint4*>(R.lv + i);
    o[0] = make_uint4(s[0] | s[1] << 16, s[2] | s[3] << 16, s[4] | s[5] << 16, s[6] | s[7] << 16);
    reinterpret_cast<uint2*>(o)[2] = make_uint2(s[8] | s[9] << 16, s[10] | s[11] << 16);
  }
  __syncthreads();
  if (warp == 0) {
    HeadState H{n, 0u, 0u, 0u, -1};
    lv_head(R, L, n, H);
    if (lane == 0) L.h = H;
  }
  __syncthreads();
  int gate = L.h.gate;
  // ---- the first round: cells that wait for nobody
  for (unsigned i = tid; i < n; i += NT_) {
    if (dep_byte(L, i) != 0u) continue;
    if ((int)(R.lv[i].ye & YE_Y) <= gate) list_put(R, L, 0u, atomicAdd(&L.cnt[0], 1u), i);
    else park_put(R, 0u, atomicAdd(&L.park_n[0], 1u), i);
  }
  __syncthreads();
  plap(0);
  // ---- rounds
  long long t_wide = 0, t_search = 0;
  while (true) {
    // warp 0 alone decides what comes next: nobody else reads the lists' state while it runs
    if (warp == 0) pd += lv_solo(Rs, L, n, gate, sgn, cap);
    __syncthreads();
    const unsigned req = L.req;
    if (req == SR_END) break;
    if (req == SR_SEARCH) {
      const long long c0 = clock64();
      search_cta(Rs, L);
      t_search += clock64() - c0;
    } else if (req == SR_GATE) {
      gate = L.h.gate;
      const unsigned pb = L.pb, np = min(L.park_n[pb], MAX_CELLS_PER_TICK), lb = L.cur, lc = L.cc;
      for (unsigned t = tid; t < np; t += NT_) {
        const unsigned i = R.lv_park[(size_t)pb * MAX_CELLS_PER_TICK + t];
        if ((int)(R.lv[i].ye & YE_Y) <= gate) list_put(R, L, lb, atomicAdd(&L.cnt[lc], 1u), i);
        else park_put(R, pb ^ 1u, atomicAdd(&L.park_n[pb ^ 1u], 1u), i);
      }
      __syncthreads();
      if (tid == 0) {
        L.park_n[pb] = 0u;
        L.pb = pb ^ 1u;
      }
      __syncthreads();
    } else {
      const long long c0 = clock64();
      pd += L.cnt[L.cc] >= THREAD_CELLS ? lv_long(Rs, L, n, gate, cap) : lv_wide(Rs, L, n, gate, cap);
      t_wide += clock64() - c0;
    }
  }
  if (L.timeout) {
    if (tid == 0) set_status(R, ST_TIMEOUT, 38);
    __syncthreads();
    return;
  }
  plap(1);
  if (tid == 0) {
    unsigned long long* q = R.ctl->pprof;
    q[7] += (unsigned long long)t_search;
    q[8] += (unsigned long long)t_wide;
    q[9] += n;
    q[14] += L.n_searches;
    q[15] += L.rounds;
    R.ctl->par_segments += L.rounds;
    R.ctl->par_rollbacks += L.n_again;
    R.ctl->par_replayed += L.n_searches;
  }
  sweep_flush(R, L, n);
  // ---- the cells' events in sorted order -> the tick's event logs (program order), and the position map
  // back to idle. A batch's events are on their way while the one before is logged.
  const unsigned pxy = (unsigned)R.PX * (unsigned)R.PY;
  const bool lr = sW.level_round;
  unsigned any_chg = 0, s_na = 0, s_ns = 0, s_nc = 0;  // (the same in every thread)
  unsigned ev_next = tid < n ? R.lv_ev[tid] : 0u, key_next = tid < n ? R.cells[tid] : 0u;
  for (unsigned base = 0; base < n; base += NT_) {
    const unsigned i = base + tid, ev = ev_next, key = key_next;
    if (i + NT_ < n) {
      ev_next = R.lv_ev[i + NT_];
      key_next = R.cells[i + NT_];
    }
    unsigned am = 0, fl = 0, cm = 0, src = 0, cid = 0;
    if (i < n) {
      am = ev & 0xFFu;
      cm = (ev >> 8) & 0xFFu;
      fl = ev >> 16;
      cid = key_to_id(R, key, flip);
      R.stamp[cid] = 0xFFFFFFFFu;
      if (am & 1u) src = R.lv_src[i];
      any_chg |= cm;
    }
    const unsigned ns = lr ? 0u : (unsigned)__popc(fl & 3u);
    unsigned ta, ts = 0u, os = 0u;  // activations and changes in one scan: at most 8 a cell
    static_assert(8 * PAR_THREADS < 1 << 16, "two counts in a word");
    const unsigned oa = cta_scan_count(sm, (unsigned)__popc(am) | (unsigned)__popc(cm) << 16, &ta);
    if (!lr) os = cta_scan_count(sm, ns, &ts);
    if (i < n) {
      // activations: slot 0 the source (one cell), slots 1..7 wake_around centres
      unsigned pa = s_na + (oa & 0xFFFFu);
      for (int g = 0; g < 8; ++g) {
        if (!((am >> g) & 1u)) continue;
        unsigned w;
        switch (g) {
          case 0: w = src; break;
          case 2: w = (cid - (unsigned)R.PX) | ACT_AROUND; break;
          case 3: w = (cid + 1u) | ACT_AROUND; break;
          case 4: w = (cid - 1u) | ACT_AROUND; break;
          case 5: w = (cid + pxy) | ACT_AROUND; break;
          case 6: w = (cid - pxy) | ACT_AROUND; break;
          default: w = cid | ACT_AROUND; break;  // 1 and 7: the cell itself
        }
        if (pa < R.ev_act_cap) R.ev_act[pa] = w;
        else set_status(R, ST_OOM, 40);
        ++pa;
      }
      unsigned psd = s_ns + os;
      if (ns) {  // the pull's source, then the cell itself
        if (fl & 2u) {
          if (psd < R.ev_seed_cap) R.ev_seed[psd] = src;
          else set_status(R, ST_OOM, 41);
          ++psd;
        }
        if (fl & 1u) {
          if (psd < R.ev_seed_cap) R.ev_seed[psd] = cid;
          else set_status(R, ST_OOM, 41);
        }
      }
      unsigned pc = s_nc + (oa >> 16);
      for (int l = 0; l < 8; ++l) {
        if (!((cm >> l) & 1u)) continue;
        unsigned id;
        switch (l) {
          case 0: id = cid; break;
          case 1: id = cid - (unsigned)R.PX; break;
          case 3: id = cid + 1u; break;
          case 4: id = cid - 1u; break;
          case 5: id = cid + pxy; break;
          case 6: id = cid - pxy; break;
          default: id = src; break;
        }
        if (pc < R.ev_chg_cap) R.ev_chg[pc] = id;
        else set_status(R, ST_OOM, 42);
        ++pc;
      }
    }
    s_na += ta & 0xFFFFu;
    s_ns += ts;
    s_nc += ta >> 16;
  }
  const unsigned long long c_pd = cta_sum(sm, (unsigned long long)(long long)pd);
  any_chg = __syncthreads_or((int)any_chg);
  if (tid == 0) {
    sW.nact = s_na;
    sW.nseed = s_ns;
    sW.nchg = s_nc;
    sW.pull_attempts = min(MAX_PULLS_PER_TICK, total_att + L.nx);
    sW.pull_success = L.n_succ;
    sW.bfs_visits = L.n_entries;
    sW.pdelta = (long long)c_pd;
    sW.changed = any_chg != 0;
  }
  __syncthreads();
  plap(3);
}

// ------------------------------------------------------------------ levelling, all warps
// LayerMarks probe without setting (mark_tas's tile and bit); cells outside the domain read as
// marked, as mark_tas treats them. Marks are set by atomics (in L2): read past L1.
__device__ __forceinline__ bool mark_test(const Region& R, int x, int y, int z) {
  if (!in_dom(R, x, y, z)) return true;
  const unsigned xr = (unsigned)(x - R.px0), zr = (unsigned)(z - R.pz0);
  const unsigned tile = ((zr >> 6) * (unsigned)R.PY + (unsigned)y) * (unsigned)R.TX + (xr >> 6);
  const unsigned bit = ((zr & 63u) << 6) | (xr & 63u);
  return (__ldcg(R.marks + (size_t)tile * 128u + (bit >> 5)) >> (bit & 31u)) & 1u;
}

// The flood fill of FluidSim::level_layer (fluid.rs:425-446) continued from queue entry qs of qe,
// batch by batch over the CTA. The batch is every waiting entry; entry p's side d is tried in the
// reference's order p-major, d-minor: its rank 4(p - qs) + d claims the cell (the lowest rank is
// the reference's first test, which sets the mark; the others find it set), and the members are
// appended in rank order, so the queue is the reference's queue. A batch that could carry the
// queue to MAX_LEVEL_CELLS (where the reference stops expanding part-way) finishes on one warp.
// Returns the final length.
__device__ __noinline__ unsigned level_bfs_cta(const Region& R, TickSmem& sm, Smem& S, unsigned qs, unsigned qe) {
  __shared__ unsigned s_run, s_len;
  const unsigned tid = threadIdx.x;
  while (qs < qe) {
    const unsigned F = qe - qs;
    if ((unsigned long long)qe + 4ull * F >= MAX_LEVEL_CELLS) {
      if (tid < 32u) {
        unsigned i = qs;
        const unsigned len = level_bfs_warp(R, S, i, qe, 0xFFFFFFFFu);
        if (tid == 0) s_len = len;
      }
      __syncthreads();
      return s_len;
    }
    // claims
    for (unsigned t = tid; t < 4u * F; t += NT_) {
      int x, y, z, dx, dz;
      dom_xyz(R, R.lvl_id[qs + t / 4u], x, y, z);
      side4((int)(t & 3u), dx, dz);
      const int nx = x + dx, nz = z + dz;
      if (R.ring_w == 0 && (nx < 0 || nz < 0)) continue;
      if (!in_dom(R, nx, y, nz)) {  // cannot happen for neighbours of addressable cells
        set_status(R, ST_RANGE, 8);
        continue;
      }
      if (mark_test(R, nx, y, nz)) continue;
      atomicMin(R.rb + dom_id(R, nx, y, nz), t);
    }
    if (tid == 0) s_run = 0;
    __syncthreads();
    // the winners set the mark, test and append, in rank order
    for (unsigned base = 0; base < 4u * F; base += NT_) {
      const unsigned t = base + tid;
      unsigned f = 0, nid = 0;
      float v = 0.0f;
      if (t < 4u * F) {
        int x, y, z, dx, dz;
        dom_xyz(R, R.lvl_id[qs + t / 4u], x, y, z);
        side4((int)(t & 3u), dx, dz);
        const int nx = x + dx, nz = z + dz;
        if (!(R.ring_w == 0 && (nx < 0 || nz < 0)) && in_dom(R, nx, y, nz)) {
          nid = dom_id(R, nx, y, nz);
          if (__ldcg(R.rb + nid) == t) {  // set by atomics (in L2): read past L1
            R.rb[nid] = 0xFFFFFFFFu;
            unsigned tile;
            const unsigned listed = mark_begin(R, nx, y, nz, tile);  // unmarked: it won the claim
            f = level_member(R, nx, y, nz, &v) ? 1u : 0u;
            mark_end(R, tile, listed);
          }
        }
      }
      unsigned tot;
      const unsigned off = cta_scan_count(sm, f, &tot);
      if (f) {
        R.lvl_id[qe + s_run + off] = nid;
        R.lvl_vol[qe + s_run + off] = v;
      }
      __syncthreads();
      if (tid == 0) s_run += tot;
      __syncthreads();
    }
    qs = qe;
    qe += s_run;
    __syncthreads();
  }
  return qe;
}

// A layer whose one-warp flood fill has this many entries waiting continues over the CTA.
constexpr unsigned LEVEL_HAND = 16;

// Minimum and maximum of a float over the CTA.
__device__ void cta_minmax(float& lo, float& hi) {
  __shared__ float s_lo[MAX_WARPS], s_hi[MAX_WARPS];
  for (int o = 16; o; o >>= 1) {
    lo = fminf(lo, __shfl_xor_sync(FULLMASK, lo, o));
    hi = fmaxf(hi, __shfl_xor_sync(FULLMASK, hi, o));
  }
  if ((threadIdx.x & 31u) == 0) {
    s_lo[threadIdx.x >> 5] = lo;
    s_hi[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  for (unsigned w = 0; w < NW_; ++w) {
    lo = fminf(lo, s_lo[w]);
    hi = fmaxf(hi, s_hi[w]);
  }
  __syncthreads();
}

// Cells of levelled layers, one per thread in order: each takes its layer's average (fluid.rs:457-470).
// Returns the thread's change in partial entries. All threads.
__device__ __forceinline__ int level_write(const Region& R, TickSmem& sm, WS& sW, const int* ring, bool has, unsigned id, float avg) {
  int x = 0, y = 0, z = 0;
  bool wv = false;
  CD c = CD{0.0f, NOSLOT, 0u, 0, true};
  if (has) {
    dom_xyz(R, id, x, y, z);
    c = load_cell_par(R, ring, x, y, z);
    wv = fabsf(__fsub_rn(cd_volume(c), avg)) > 1e-6f;
  }
  materialize_cta(R, wv && set_volume_needs_slot(c, avg), c.gi, c.slot);
  bool ch = false;
  int pd = 0;
  if (wv) {
    const SVPlan p = sv_plan(c.part, c.mat, c.slot != NOSLOT, avg);
    if (c.slot != NOSLOT) sv_apply(R, c, id, local_index(x, y, z), p);
    ch = p.ch;
    pd = p.dp;
  }
  unsigned tot;
  const unsigned off = cta_scan(sm, ch, &tot);
  if (ch) {
    const unsigned pos = sW.nchg + off;
    if (pos < R.ev_chg_cap) R.ev_chg[pos] = id;
    else set_status(R, ST_OOM, 9);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    sW.nchg += tot;
    if (tot) sW.changed = true;
  }
  __syncthreads();
  return pd;
}

// What FluidSim::level_layer does with a gathered layer of len cells (fluid.rs:430-485), over the
// CTA. The f64 sum in queue order is formed exactly whenever every partial sum is representable:
// all volumes are multiples of 2^L (L from the smallest, lo) and every partial sum is below
// len * hi < 2^H, so H - L <= 53 makes each f64 addition exact and the integer sum of v / 2^L is
// the reference's sum, in any order. Otherwise one thread adds in queue order. Levelling to the
// average writes each cell once, in parallel, the change log in cell order; the drain branch
// (`left` runs through the cells in order) and layers left as they are go to warp 0's
// level_finish.
__device__ __noinline__ void level_finish_cta(const Region& R, TickSmem& sm, WS& sW, Smem& S, unsigned len) {
  __shared__ double s_sum;
  const unsigned tid = threadIdx.x;
  float lo = 2.0f, hi = -1.0f;
  for (unsigned k = tid; k < len; k += NT_) {
    const float v = R.lvl_vol[k];
    lo = fminf(lo, v);
    hi = fmaxf(hi, v);
  }
  cta_minmax(lo, hi);
  int el, eh;
  frexpf(lo, &el);
  frexp((double)len * (double)hi, &eh);
  const int L = el - 24;  // lo = m 2^el, m in [0.5, 1): its last mantissa bit is 2^(el - 24)
  double sum;
  if (lo >= 1.17549435e-38f && eh - L <= 53) {
    unsigned long long q = 0;
    for (unsigned k = tid; k < len; k += NT_) q += (unsigned long long)ldexp((double)R.lvl_vol[k], -L);
    sum = ldexp((double)cta_sum(sm, q), L);
  } else {
    if (tid == 0) {
      double a = 0.0;
      for (unsigned k = 0; k < len; ++k) a = __dadd_rn(a, (double)R.lvl_vol[k]);
      s_sum = a;
    }
    __syncthreads();
    sum = s_sum;
    __syncthreads();
  }
  const bool spread = len >= 2 && __fsub_rn(hi, lo) >= SLEEP;
  const float avg = spread ? __double2float_rn(__ddiv_rn(sum, (double)len)) : 0.0f;
  if (!spread || avg < MIN_SPREAD) {
    if (tid < 32u) {
      WS W = sW;
      W.pdelta = 0;
      const bool ch = level_finish(R, W, S, len, sum, lo, hi);
      long long pd = W.pdelta;
      for (int o = 16; o; o >>= 1) pd += __shfl_xor_sync(FULLMASK, pd, o);
      if (tid == 0) {
        W.pdelta = sW.pdelta + pd;
        W.changed |= ch;
        sW = W;
      }
      __syncwarp();
    }
    __syncthreads();
    return;
  }
  long long pd = 0;
  for (unsigned base = 0; base < len; base += NT_) {
    const unsigned k = base + tid;
    pd += level_write(R, sm, sW, S.ring, k < len, k < len ? R.lvl_id[k] : 0u, avg);
  }
  const long long dp = (long long)cta_sum(sm, (unsigned long long)pd);
  if (tid == 0) {
    sW.pdelta += dp;
    sW.llc += len;
    sW.level_cells_total += len;
  }
  __syncthreads();
}

// A small layer's flood fill by one warp, without touching the marks: the cells in the reference's
// order, and every cell it tested (a set: the marks it would leave). Several run side by side; the
// layers of one batch are the same or disjoint (their members do not change while it lasts), so the
// smallest cell id tells them apart. Bound by the longest layer of a group, ~1,200 cycles for each
// one or two of its entries (ring rain: 14.4 M cycles of levelling with one a step, 11.4 with two).
constexpr unsigned FILL_CELLS = 64, FILL_SLOTS = 512;
static_assert(4 * FILL_CELLS + 1 < FILL_SLOTS, "tested cells of a small layer");
enum FillKind { FK_KEEP = 0, FK_LEVEL = 1, FK_DRAIN = 2, FK_BIG = 3, FK_DUP = 4 };
struct LevelFill {
  unsigned id[FILL_CELLS];
  float vol[FILL_CELLS];
  unsigned key[FILL_SLOTS];  // tested cells (EMPTY_ID = free)
  unsigned len, kind, min_id;
  float avg;
};

__device__ void level_fill_small(const Region& R, LevelFill& F, unsigned sid) {
  const unsigned lane = lane_id();
  const float FULL = full_level();
  for (unsigned t = lane; t < FILL_SLOTS; t += 32u) F.key[t] = EMPTY_ID;
  __syncwarp();
  auto test = [&](unsigned id) {  // true: tested before
    unsigned h = (id * 2654435761u) >> 23;
    while (true) {
      const unsigned old = atomicCAS(&F.key[h], EMPTY_ID, id);
      if (old == EMPTY_ID) return false;
      if (old == id) return true;
      h = (h + 1u) & (FILL_SLOTS - 1u);
    }
  };
  int sx, sy, sz;
  dom_xyz(R, sid, sx, sy, sz);
  float v0;
  level_member(R, sx, sy, sz, &v0);
  if (lane == 0) {
    test(sid);
    F.id[0] = sid;
    F.vol[0] = v0;
  }
  __syncwarp();
  unsigned len = 1, kind = FK_KEEP, mn = sid;
  // two queue entries a step where two wait: lanes 0..11 the first, 12..23 the second; of an entry's lanes, side
  // d = lane / 3, its cell (j = 0), the one below (1) and above (2)
  const unsigned half = lane >= 12u ? 1u : 0u, r = lane - 12u * half;
  const int d = (int)r / 3, j = (int)r % 3;
  int dx = 0, dz = 0;
  if (lane < 24u) side4(d, dx, dz);
  for (unsigned i = 0, step; i < len; i += step) {
    step = min(len - i, 2u);
    int x, y, z;
    dom_xyz(R, F.id[i + (half < step ? half : 0u)], x, y, z);
    const int nx = x + dx, nz = z + dz;
    const bool skip = lane >= 24u || half >= step || (R.ring_w == 0 && (nx < 0 || nz < 0));
    const bool look = !skip && j == 0 && in_dom(R, nx, y, nz);
    const unsigned nid = look ? dom_id(R, nx, y, nz) : EMPTY_ID;
    bool seen = true;
    if (look) seen = mark_test(R, nx, y, nz);
    // a cell both entries test is the first one's
    const unsigned peers = __match_any_sync(FULLMASK, nid);
    if (look && !seen) seen = (peers & lanemask_lt()) != 0u || test(nid);
    const unsigned c = skip ? DC_SOLID : dense_at(R, nx, y + (j == 1 ? -1 : (j == 2 ? 1 : 0)), nz);
    const bool sol = dc_solid(c);
    const float v = dc_level(c);
    const float v1 = __shfl_down_sync(FULLMASK, v, 1), v2 = __shfl_down_sync(FULLMASK, v, 2);
    const bool s1 = __shfl_down_sync(FULLMASK, (unsigned)sol, 1) != 0u;
    const bool push = !skip && j == 0 && !seen && !sol && v > 0.0f && (s1 || v1 >= FULL) && v2 <= 0.0f;
    const unsigned pm = __ballot_sync(FULLMASK, push);
    if (len + (unsigned)__popc(pm) > FILL_CELLS || len - i > LEVEL_HAND) {  // large: goes to the CTA
      kind = FK_BIG;
      break;
    }
    if (push) {
      const unsigned p = len + (unsigned)__popc(pm & lanemask_lt());
      F.id[p] = nid;
      F.vol[p] = v;
    }
    mn = min(mn, __reduce_min_sync(FULLMASK, push ? nid : EMPTY_ID));
    len += (unsigned)__popc(pm);
    __syncwarp();
  }
  if (lane == 0) {
    F.len = len;
    F.min_id = mn;
    if (kind != FK_BIG) {  // fluid.rs:430-456: the sum in queue order
      double a = 0.0;
      float lo = 2.0f, hi = -1.0f;
      for (unsigned k = 0; k < len; ++k) {
        a = __dadd_rn(a, (double)F.vol[k]);
        lo = fminf(lo, F.vol[k]);
        hi = fmaxf(hi, F.vol[k]);
      }
      if (len >= 2u && __fsub_rn(hi, lo) >= SLEEP) {
        F.avg = __double2float_rn(__ddiv_rn(a, (double)len));
        kind = F.avg >= MIN_SPREAD ? FK_LEVEL : FK_DRAIN;
      }
    }
    F.kind = kind;
  }
  __syncwarp();
}

// The marks a small layer's fill leaves behind, one warp.
__device__ __forceinline__ void level_mark_small(const Region& R, const LevelFill& F) {
  const unsigned lane = lane_id();
  for (unsigned t = lane; t < FILL_SLOTS; t += 32u) {
    if (F.key[t] == EMPTY_ID) continue;
    int x, y, z;
    dom_xyz(R, F.key[t], x, y, z);
    mark_tas(R, x, y, z);
  }
}

// FluidSim::level_surfaces (fluid.rs:489-507) from sW.llc on, over the CTA, in batches of up to one
// seed per thread (LIFO order = thread order). Every thread walks its seed up to the top water cell
// (fluid.rs:496-499) and tests the start: a start that is marked, repeats an earlier start of the
// batch, or is not a layer member needs no flood fill. Levelling a layer to its average changes no
// cell's solidity, its "vol > 0" or "supported", so these tests stay true while the batch's
// earlier layers are levelled; a drained layer (which can change them) ends the batch. The
// remaining starts, the candidates, are levelled in order, each marked at its turn as the reference
// does; the budget (fluid.rs:492) ends the batch after the candidate that spends it. Where the budget
// cannot run out in between, one candidate per warp is filled at once (level_fill_small) and those
// before the first large or drained layer commit together; a large layer starts on warp 0 and is
// handed to the CTA as it grows. (Rain on the ring world: ~3,000 puddles of ~8 cells a levelling tick,
// 57 M SM cycles one after another.) The popped seeds leave the seed set and their starts are
// marked (a start that is not a member is marked, and skipped by every later flood fill, either
// way). sW.level_round is updated at the end.
__device__ __noinline__ void level_round_cta(const Region& R, TickSmem& sm, WS& sW, Smem& S) {
  __shared__ unsigned s_ns, s_stop, s_brk, s_pend, s_qi, s_ql, s_cur, s_m, s_group[MAX_WARPS];
  LevelFill* const fills = reinterpret_cast<LevelFill*>(sm.u.x.fills);  // the sweep's shared memory is free now
  static_assert(sizeof(LevelFill) * MAX_WARPS <= sizeof(sm.u.x.fills) && sizeof(sm.u.x) <= sizeof(LvSmem), "level fills");
  const unsigned tid = threadIdx.x;
  unsigned* b_start = sm.u.x.hist;          // the batch's starts (domain ids), by seed
  unsigned* b_cand = sm.u.x.hist + NT_;     // candidate seeds in order
  while (true) {
    if (tid == 0) s_ns = (sW.llc < LEVEL_BUDGET) ? sW.nseeds : 0u;
    __syncthreads();
    const unsigned ns = s_ns;
    if (ns == 0u) break;
    const unsigned B = min(ns, NT_);
    // ---- starts and their tests, one seed per thread
    unsigned sid = 0;
    int x = 0, y = 0, z = 0;
    if (tid < B) {
      dom_xyz(R, R.seeds[ns - 1u - tid], x, y, z);
      while (true) {  // four cells of the column per step
        bool up[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int yy = y + 1 + q;
          up[q] = false;
          if (yy < R.ny) {
            const unsigned c = dense_at(R, x, yy, z);
            up[q] = !dc_solid(c) && dc_volume(c) > 0.0f;
          }
        }
        const int steps = !up[0] ? 0 : !up[1] ? 1 : !up[2] ? 2 : !up[3] ? 3 : 4;
        y += steps;
        if (steps < 4) break;
      }
      sid = dom_id(R, x, y, z);
      b_start[tid] = sid;
      atomicMin(R.rb + sid, tid);
    }
    __syncthreads();
    const bool first = tid < B && __ldcg(R.rb + sid) == tid;  // set by atomics (in L2): read past L1
    __syncthreads();
    unsigned cand = 0, single = 0;
    if (first) {
      R.rb[sid] = 0xFFFFFFFFu;
      float v;
      cand = (!mark_test(R, x, y, z) && level_member(R, x, y, z, &v)) ? 1u : 0u;
      // a start none of whose sides is an unmarked member is a layer of one cell: no flood fill
      // (marks only grow and membership holds through the batch, so this stays true)
      if (cand) {
        single = 1u;
        for (int d = 0; d < 4 && single; ++d) {
          int dx, dz;
          side4(d, dx, dz);
          const int nx = x + dx, nz = z + dz;
          if (R.ring_w == 0 && (nx < 0 || nz < 0)) continue;
          if (!mark_test(R, nx, y, nz) && level_member(R, nx, y, nz, &v)) single = 0u;
        }
      }
    }
    unsigned nc;
    const unsigned off = cta_scan_count(sm, cand, &nc);
    if (cand) b_cand[off] = tid | (single << 31);
    if (tid == 0) {
      s_stop = B;
      s_brk = 0;
      s_cur = 0;  // the next candidate to level
    }
    __syncthreads();
    // ---- the candidates in order. One-cell layers only count (fluid.rs:446, len < 2); a start
    // that an earlier layer's flood fill marked is skipped, as its test_and_set would return
    // (entry bits: 31 one cell, 30 marked since the batch began, 0-29 the seed)
    while (true) {
      if (tid == 0 && !s_brk) {
        unsigned c = s_cur;
        while (c < nc && (b_cand[c] >> 30)) {
          if (b_cand[c] >> 31) {
            sW.llc += 1u;
            sW.level_cells_total += 1u;
            if (sW.llc >= LEVEL_BUDGET) {
              s_stop = (b_cand[c] & 0x3FFFFFFFu) + 1u;
              s_brk = 1u;
            }
          }
          ++c;
          if (s_brk) break;
        }
        s_cur = c;
      }
      __syncthreads();
      if (s_brk || s_cur >= nc) break;
      const unsigned cur = s_cur;
      const unsigned j = b_cand[cur];
      if (tid == 0) {
        unsigned m = 0;
        if (sW.llc + nc + FILL_CELLS * NW_ < LEVEL_BUDGET)
          for (unsigned c = cur; c < nc && m < NW_; ++c)
            if (!(b_cand[c] >> 30)) s_group[m++] = b_cand[c];
        s_m = m;
      }
      __syncthreads();
      const unsigned m = s_m;
      if (m) {
        const unsigned w = tid >> 5;
        if (w < m) level_fill_small(R, fills[w], b_start[s_group[w]]);
        __syncthreads();
        if (tid == 0) {
          unsigned k = 0, cells = 0;
          for (; k < m; ++k) {
            if (fills[k].kind == FK_BIG || fills[k].kind == FK_DRAIN) break;
            bool dup = false;  // an earlier fill of the group covers it: its start is marked by then
            for (unsigned o = 0; o < k; ++o) dup |= fills[o].kind != FK_DUP && fills[o].min_id == fills[k].min_id;
            if (dup) fills[k].kind = FK_DUP;
            else cells += fills[k].len;
          }
          s_m = k;
          sW.llc += cells;
          sW.level_cells_total += cells;
        }
        __syncthreads();
        const unsigned done = s_m;
        if (w < done && fills[w].kind != FK_DUP) level_mark_small(R, fills[w]);
        // the cells of the layers that are levelled, in order, one per thread
        int pd = 0;
        for (unsigned base = 0;; base += NT_) {
          unsigned k = base + tid, f = 0, total = 0;
          for (unsigned o = 0; o < done; ++o) {
            const unsigned l = fills[o].kind == FK_LEVEL ? fills[o].len : 0u;
            total += l;
            if (k >= total) f = o + 1u;
            else if (f == o) k -= total - l;
          }
          if (base >= total) break;
          const bool has = base + tid < total;
          pd += level_write(R, sm, sW, S.ring, has, has ? fills[f].id[k] : 0u, has ? fills[f].avg : 0.0f);
        }
        if (pd) atomicAdd(reinterpret_cast<unsigned long long*>(&sW.pdelta), (unsigned long long)(long long)pd);
        __syncthreads();
        if (done) {  // the group's starts, and the later ones its fills marked
          for (unsigned c = cur + tid; c < nc; c += NT_) {
            const unsigned e = b_cand[c];
            if (e >> 30) continue;
            int cx, cy, cz;
            dom_xyz(R, b_start[e], cx, cy, cz);
            if (mark_test(R, cx, cy, cz)) b_cand[c] = e | (1u << 30);
          }
          __syncthreads();
          continue;
        }
      }
      if (tid < 32u) {
        WS W = sW;
        W.pdelta = 0;
        int cx, cy, cz;
        dom_xyz(R, b_start[j], cx, cy, cz);
        unsigned qi = 0, ql = 0;
        const bool pend = level_layer(R, W, S, cx, cy, cz, LEVEL_HAND, qi, ql);
        long long pd = W.pdelta;
        for (int o = 16; o; o >>= 1) pd += __shfl_xor_sync(FULLMASK, pd, o);
        if (tid == 0) {
          W.pdelta = sW.pdelta + pd;
          sW = W;
          s_pend = pend ? 1u : 0u;
          s_qi = qi;
          s_ql = ql;
        }
        __syncwarp();
      }
      __syncthreads();
      if (s_pend) {
        const unsigned len = level_bfs_cta(R, sm, S, s_qi, s_ql);
        level_finish_cta(R, sm, sW, S, len);
      }
      // the later candidates this layer's flood fill marked
      for (unsigned c = cur + 1u + tid; c < nc; c += NT_) {
        const unsigned e = b_cand[c];
        if (e >> 30) continue;
        int cx, cy, cz;
        dom_xyz(R, b_start[e], cx, cy, cz);
        if (mark_test(R, cx, cy, cz)) b_cand[c] = e | (1u << 30);
      }
      if (tid == 0) {
        if (sW.llc >= LEVEL_BUDGET || sW.ndrain != 0u) {
          s_stop = j + 1u;
          s_brk = 1u;
        }
        s_cur += 1u;
      }
      __syncthreads();  // (s_brk is looked at after the next barrier only: thread 0 may set it before that)
    }
    // ---- the popped seeds: out of the seed set, starts marked (and the sides a one-cell layer's
    // flood fill tested)
    const unsigned stop = s_stop;
    if (tid < stop) {
      const unsigned k = R.seeds[ns - 1u - tid];
      atomicAnd(&R.seedbits[k >> 5], ~(1u << (k & 31u)));
      int sx, sy, sz;
      dom_xyz(R, b_start[tid], sx, sy, sz);
      mark_tas(R, sx, sy, sz);
      if (single) {
        for (int d = 0; d < 4; ++d) {
          int dx, dz;
          side4(d, dx, dz);
          const int nx = sx + dx, nz = sz + dz;
          if (R.ring_w == 0 && (nx < 0 || nz < 0)) continue;
          if (in_dom(R, nx, sy, nz)) mark_tas(R, nx, sy, nz);
        }
      }
    }
    __syncthreads();
    if (tid == 0) {
      sW.nseeds = ns - stop;
      sW.ndrain = 0u;
    }
    __syncthreads();
  }
  if (tid == 0) sW.level_round = sW.nseeds != 0u;
  __syncthreads();
}

// FluidSim::tick (fluid.rs:564-657) for region R, n_ticks times. All threads of the CTA enter.
// Per tick, all by the CTA: drain the FIFO head and sort it, the sweep, the seed log's commit,
// levelling, then the activation and change logs' commits. The logs keep program order, so the committed FIFO and seed list are exactly
// the reference's.
__device__ void run_ticks(const Region& R, TickSmem& sm, int n_ticks, Tune tune) {
  const unsigned tid = threadIdx.x, warp = tid >> 5;
  const int* ring = R.ring;
  if (R.ring_w && R.ring_w <= 16) {
    for (int i = tid; i < 3 * R.ring_w * R.ring_w; i += NT_) sm.ring[i] = R.ring[i];
    ring = sm.ring;
  }
  __shared__ unsigned s_n, s_flip, s_clear, s_abort, s_nseeds, s_lv;
  __shared__ unsigned long long s_qtail;
  __shared__ WS sW;
  if (tid == 0) {
    load_ws(R, sW);
    sW.deferred = true;
    s_abort = R.ctl->status != 0;
    s_clear = 0;
  }
  __syncthreads();
  long long tp = clock64();
  auto lap = [&](int k) {
    if (tid == 0) {
      long long now = clock64();
      R.ctl->prof[k] += (unsigned long long)(now - tp);
      tp = now;
    }
  };
  for (int t = 0; t < n_ticks; ++t) {
    if (s_abort) break;
    lap(15);
    // ---- drain the FIFO head (fluid.rs:565-572)
    if (tid == 0) {
      unsigned tick = R.ctl->tick_no + 1u;
      R.ctl->tick_no = tick;
      unsigned long long len = sW.qtail - sW.qhead;
      s_n = (unsigned)min(len, (unsigned long long)MAX_CELLS_PER_TICK);
      s_flip = tick & 1u;
    }
    __syncthreads();
    const unsigned n = s_n;
    const bool flip = s_flip != 0;
    const unsigned long long qh = sW.qhead;
    const unsigned tick_now = R.ctl->tick_no;
    for (unsigned i = tid; i < n; i += NT_) {
      unsigned id = R.queue[(qh + i) & R.qmask];
      atomicAnd(&R.active[id >> 5], ~(1u << (id & 31)));
      R.cells[i] = sort_key(R, id, flip);
      // wake history of materialised bricks (training labels of the wake proposal)
      int x, y, z;
      dom_xyz(R, id, x, y, z);
      if (!outside(R, ring, x, y, z)) {
        unsigned g = R.grid[grid_index(R, x >> 3, y >> 3, z >> 3)];
        if (g >= 256u) R.last_woken[g - 256u] = tick_now;
      }
    }
    __syncthreads();
    if (tid == 0) {
      sW.qhead = qh + n;
      sW.changed = false;
      sW.activations = sW.pull_attempts = sW.pull_success = sW.bfs_visits = sW.level_cells_total = 0;
      sW.pdelta = 0;
      sW.nact = sW.nseed = sW.nchg = 0;
    }
    __syncthreads();
    // ---- ring worlds: a drained cell of an evicted chunk is solid (outside), and the sweep erases its
    // partial entry (fluid.rs:586-589); entries kept for evicted chunks are erased here, which nothing
    // in the tick can tell apart (an outside cell's volume reads 0)
    if (R.detbits && vld(&R.ctl->ndetached) != 0u) {
      unsigned long long er = 0;
      for (unsigned i = tid; i < n; i += NT_) {
        const unsigned id = R.queue[(qh + i) & R.qmask];
        int x, y, z;
        dom_xyz(R, id, x, y, z);
        if (!outside(R, ring, x, y, z)) continue;
        const unsigned bit = 1u << (id & 31u);
        if (atomicAnd(R.detbits + (id >> 5), ~bit) & bit) ++er;
      }
      er = cta_sum(sm, er);
      if (tid == 0) {
        R.ctl->partial_count -= (long long)er;
        R.ctl->ndetached -= (unsigned)er;
      }
      __syncthreads();
    }
    lap(0);
    // ---- sort (fluid.rs:575-580)
    cta_radix_sort(R.cells, R.cells_tmp, n, sm.u.x.hist, sm.sred);
    __syncthreads();
    lap(1);
    // ---- the sweep (fluid.rs:584-651)
    sweep_levels(R, sm, sW, ring, n, flip, tune);
    lap(2);
    if (vld((const unsigned*)&R.ctl->status) != 0u) {
      if (tid == 0) s_abort = 1;
      __syncthreads();
      break;
    }
    // ---- level seeds logged by the sweep (fluid.rs:312-316)
    if (tid == 0) s_nseeds = sW.nseeds;
    __syncthreads();
    unsigned nseeds = s_nseeds;
    commit_seeds(R, sm, min(sW.nseed, R.ev_seed_cap), nseeds);
    if (tid == 0) sW.nseeds = nseeds;
    __syncthreads();
    lap(7);
    // ---- levelling (fluid.rs:652-655)
    if (tid == 0) s_lv = (sW.level_round || (R.ctl->tick_no % LEVEL_TICKS) == 0u) ? 1u : 0u;
    __syncthreads();
    if (s_lv) {
      Smem S{ring};
      if (tid == 0) sW.llc = 0;
      __syncthreads();
      level_round_cta(R, sm, sW, S);
      if (tid == 0) s_clear = sW.level_round ? 0u : 1u;
    }
    __syncthreads();
    lap(8);
    // ---- FIFO appends and voxel changes logged during the tick
    if (tid == 0) s_qtail = sW.qtail;
    __syncthreads();
    unsigned long long qt = s_qtail;
    commit_acts(R, sm, min(sW.nact, R.ev_act_cap), qt, sW.qhead);
    lap(9);
    commit_chgs(R, min(sW.nchg, R.ev_chg_cap));
    lap(10);
    if (tid == 0) {
      Ctl& c = *R.ctl;
      c.activations += qt - s_qtail;
      sW.qtail = qt;
      c.last_cells = n;
      c.cells_total += n;
      c.pull_attempts += sW.pull_attempts;
      c.pull_success += sW.pull_success;
      c.bfs_visits += sW.bfs_visits;
      c.level_cells_total += sW.level_cells_total;
      c.partial_count += sW.pdelta;
      c.last_level_cells = sW.llc;
      c.nseeds = sW.nseeds;
      c.level_round = sW.level_round ? 1u : 0u;
      if (sW.changed) c.changed = 1u;
      c.qhead = sW.qhead;
      c.qtail = sW.qtail;
      s_abort = c.status != 0;
    }
    __syncthreads();
    // ---- end of a levelling round: clear the marks it touched (fluid.rs:503-505)
    if (s_clear) {
      const unsigned nt = R.ctl->mark_ntiles;
      for (unsigned k = warp; k < nt; k += NW_) {
        unsigned tile = R.mark_list[k];
        for (unsigned w = lane_id(); w < 128; w += 32) R.marks[(size_t)tile * 128u + w] = 0u;
        if (lane_id() == 0) R.mark_tflag[tile] = 0u;
      }
      __syncthreads();
      if (tid == 0) {
        R.ctl->mark_ntiles = 0;
        s_clear = 0;
      }
      __syncthreads();
    }
    lap(11);
  }
}

// One CTA of up to PAR_THREADS per region.
__global__ void __launch_bounds__(PAR_THREADS, 1) k_tick_par(Region* regs, int nreg, int n_ticks, Tune tune) {
  extern __shared__ __align__(16) unsigned char smraw[];
  TickSmem& sm = *reinterpret_cast<TickSmem*>(smraw);
  // The region's constants (sizes, array bases): a copy in shared memory keeps them off the L1, which
  // the sweep's records and dense words stream through.
  __shared__ Region s_reg;
  for (int r = blockIdx.x; r < nreg; r += gridDim.x) {
    if (threadIdx.x == 0) s_reg = regs[r];
    __syncthreads();
    run_ticks(s_reg, sm, n_ticks, tune);
    __syncthreads();
  }
}

// -------------------------------------------------------------------------- host edits
// Activate a box in z, y, x order (FluidSim::wake, fluid.rs:358-366). One CTA; ordered by a
// CTA-wide exclusive scan per chunk of cells.
__global__ void __launch_bounds__(1024) k_wake_box(Region R, int x0, int y0, int z0, int x1, int y1, int z1) {
  __shared__ unsigned warp_cnt[32];
  __shared__ unsigned long long s_tail;
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  if (tid == 0) s_tail = R.ctl->qtail;
  __syncthreads();
  const long long sx = (long long)x1 - x0 + 1, sy = (long long)y1 - y0 + 1, sz = (long long)z1 - z0 + 1;
  if (sx <= 0 || sy <= 0 || sz <= 0) return;
  const long long total = sx * sy * sz;
  for (long long base = 0; base < total; base += 1024) {
    long long t = base + tid;
    bool isnew = false;
    unsigned id = 0;
    if (t < total) {
      long long xx = t % sx, rest = t / sx;
      int x = x0 + (int)xx, y = y0 + (int)(rest % sy), z = z0 + (int)(rest / sy);
      if (y >= 0) {
        if (!in_dom(R, x, y, z)) {
          if (atomicCAS(&R.ctl->status, 0, ST_RANGE) == 0) R.ctl->err_info = 5;
        } else {
          id = dom_id(R, x, y, z);
          isnew = !((R.active[id >> 5] >> (id & 31)) & 1u);
        }
      }
    }
    unsigned b = __ballot_sync(FULLMASK, isnew);
    if (lane == 0) warp_cnt[warp] = __popc(b);
    __syncthreads();
    unsigned before = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
      unsigned c = warp_cnt[w];
      if ((unsigned)w < warp) before += c;
      all += c;
    }
    if (isnew) {
      unsigned long long pos = s_tail + before + __popc(b & lanemask_lt());
      R.queue[pos & R.qmask] = id;
      atomicOr(&R.active[id >> 5], 1u << (id & 31));
    }
    __syncthreads();
    if (tid == 0) {
      s_tail += all;
      R.ctl->activations += all;
    }
    __syncthreads();
  }
  if (tid == 0) {
    R.ctl->qtail = s_tail;
    if (s_tail - R.ctl->qhead > R.qmask + 1ull) atomicCAS(&R.ctl->status, 0, ST_OOM);
  }
}

// A single warp running sequential host edits with the tick's device rules.
struct EditSmem {
  int ring[3 * 16 * 16];
};

__device__ const int* edit_ring(const Region& R, int* smring) {
  if (R.ring_w && R.ring_w <= 16) {
    for (int i = lane_id(); i < 3 * R.ring_w * R.ring_w; i += 32) smring[i] = R.ring[i];
    __syncwarp();
    return smring;
  }
  return R.ring;
}

__device__ void commit_ws(const Region& R, WS& W) {
  long long pd = W.pdelta;
  for (int o = 16; o; o >>= 1) pd += __shfl_xor_sync(FULLMASK, pd, o);
  if (lane_id() == 0) {
    Ctl& c = *R.ctl;
    c.partial_count += pd;
    c.qtail = W.qtail;
    c.activations += W.activations;
    c.nseeds = W.nseeds;
    if (W.changed) c.changed = 1u;
  }
  __syncwarp();
}

__device__ void wake_box_warp(const Region& R, WS& W, int x0, int y0, int z0, int x1, int y1, int z1) {
  // small boxes (displace's 3^3): z, y, x order, 32 cells per round
  int sx = x1 - x0 + 1, sy = y1 - y0 + 1, sz = z1 - z0 + 1;
  int total = sx * sy * sz;
  for (int base = 0; base < total; base += 32) {
    int t = base + (int)lane_id();
    bool v = t < total;
    int x = 0, y = 0, z = 0;
    if (v) {
      x = x0 + t % sx;
      y = y0 + (t / sx) % sy;
      z = z0 + t / (sx * sy);
    }
    activate_round(R, W, v, x, y, z);
  }
}

// The column a displacement looks at first: lane q holds the cell q above (x, y, z).
__device__ __forceinline__ CD load_column(const Region& R, const int* ring, int x, int y, int z) {
  const int yy = y + (int)lane_id();
  return yy < R.ny ? load_cell(R, ring, x, yy, z) : CD{0.0f, NOSLOT, 0u, 0, true};
}

// Hand out `amount` over the lanes' cells in lane order (fluid.rs:381-393, :396-406): each open one
// takes min(amount, 1 - its volume) while more than 1e-6 is left, is written and activated. Cells
// already full take nothing, so only the others are visited.
__device__ float give_lanes(const Region& R, WS& W, bool open, CD c, int x, int y, int z, float amount) {
  const float cur = cd_volume(c);
  float nv = 0.0f;
  bool w = false;
  for (unsigned m = __ballot_sync(FULLMASK, open && __fsub_rn(1.0f, cur) > 0.0f); m && amount > 1e-6f; m &= m - 1u) {
    const int q = __ffs(m) - 1;
    const float cq = __shfl_sync(FULLMASK, cur, q);
    const float take = fminf(amount, __fsub_rn(1.0f, cq));
    if (take > 0.0f) {
      if ((int)lane_id() == q) {
        w = true;
        nv = __fadd_rn(cq, take);
      }
      amount = __fsub_rn(amount, take);
    }
  }
  if (__any_sync(FULLMASK, w)) {
    W.changed |= warp_set_volume(R, W, w, c, x, y, z, nv);
    activate_round(R, W, w, x, y, z);
  }
  return amount;
}

// FluidSim::displace (fluid.rs:370-408), one warp; col: load_column of the cell. The column is read 32
// cells at a time and the sides together, where a walk cell by cell paid two dependent loads for each
// cell on the way to the surface.
__device__ void displace_warp(const Region& R, WS& W, const int* ring, int x, int y, int z, CD col) {
  const unsigned lane = lane_id();
  float amount = __shfl_sync(FULLMASK, cd_volume(col), 0);
  if (lane == 0 && !col.out) erase_part(R, col, local_index(x, y, z), dom_id(R, x, y, z), W.pdelta);
  __syncwarp();
  wake_box_warp(R, W, x - 1, y - 1, z - 1, x + 1, y + 1, z + 1);
  if (amount <= 0.0f) return;
  for (int y0 = y;; y0 += 32) {
    const unsigned stop = __ballot_sync(FULLMASK, cd_solid(col) && !(y0 == y && lane == 0u));  // solid, or past the top
    const unsigned below = stop ? (stop & (0u - stop)) - 1u : 0xFFFFFFFFu;
    const bool open = ((below >> lane) & 1u) && !(y0 == y && lane == 0u);
    amount = give_lanes(R, W, open, col, x, y0 + (int)lane, z, amount);
    if (stop || amount <= 1e-6f) break;
    col = load_column(R, ring, x, y0 + 32, z);
  }
  if (amount <= 1e-6f) return;
  int dx = 0, dz = 0;
  if (lane < 4u) side4((int)lane, dx, dz);
  CD c = CD{0.0f, NOSLOT, 0u, 0, true};
  if (lane < 4u) c = load_cell(R, ring, x + dx, y, z + dz);
  give_lanes(R, W, lane < 4u && !cd_solid(c), c, x + dx, y, z + dz, amount);
}

// One cell of apply_brush (src/edit/brush.rs:93-111) with displace as on_water; returns 1 if the voxel
// was written.
__device__ unsigned brush_warp(const Region& R, WS& W, const int* ring, int x, int y, int z, unsigned char m) {
  const unsigned lane = lane_id();
  const CD col = load_column(R, ring, x, y, z);
  const unsigned own = __shfl_sync(FULLMASK, (unsigned)col.mat | ((unsigned)col.out << 8), 0);
  if (own >> 8) return 0u;  // in_brush_world (brush.rs:82-87)
  const bool empty = own == 0u || own == WATER;
  if ((m == 0) == empty) return 0u;
  if (own == WATER) displace_warp(R, W, ring, x, y, z, col);
  // SparseVolume::set_voxel (sparse_volume.rs:268-293); the displacement may have given the brick a slot
  unsigned slot = col.slot;
  const bool differs = lane == 0u && own != m;
  materialize_lanes(R, differs && slot == NOSLOT, col.gi, slot);
  if (differs && slot != NOSLOT) {
    const size_t o = (size_t)slot * 512u + local_index(x, y, z);
    R.amat[o] = m;
    dense_put(R, dom_id(R, x, y, z), m, R.avol[o]);
    record_change(R, dom_id(R, x, y, z));
  }
  __syncwarp();
  return 1u;
}

// Host voxel writes (x, y, z, m quads) in list order, SparseVolume::set_voxel each (sparse_volume.rs:
// 268-293), one CTA. The order matters only between writes of one voxel, where the last one stands and
// the voxel has changed iff some write differs from what it held, so the list runs in parallel: the
// writes claim their voxel (rb, the last wins), those that differ record the change and give the
// brick a slot, and the winners store. A warp going through the list one write after another spent
// ~1.5 us on each (16,000 writes 24 ms; here 0.1 ms).
constexpr int EDIT_THREADS = 1024;
__global__ void __launch_bounds__(EDIT_THREADS) k_voxel_edits(Region R, const int4* edits, unsigned n) {
  const unsigned nt = blockDim.x;
  for (unsigned base = 0; base < n; base += nt) {
    const unsigned i = base + threadIdx.x;
    if (i >= n) continue;
    const int4 e = edits[i];
    if (!outside(R, R.ring, e.x, e.y, e.z)) atomicMin(R.rb + dom_id(R, e.x, e.y, e.z), n - 1u - i);
  }
  for (unsigned base = 0; base < n; base += nt) {  // nothing is stored yet: every write sees what its voxel held
    const unsigned i = base + threadIdx.x;
    int4 e = make_int4(0, 0, 0, 0);
    CD c = CD{0.0f, NOSLOT, 0u, 0, true};
    if (i < n) {
      e = edits[i];
      c = load_cell_par(R, R.ring, e.x, e.y, e.z);
    }
    const bool differs = !c.out && c.mat != (unsigned char)e.w;
    unsigned slot = c.slot;
    materialize_cta(R, differs && slot == NOSLOT, c.gi, slot);
    if (differs && slot != NOSLOT) record_change(R, dom_id(R, e.x, e.y, e.z));
  }
  __syncthreads();
  for (unsigned base = 0; base < n; base += nt) {
    const unsigned i = base + threadIdx.x;
    if (i >= n) continue;
    const int4 e = edits[i];
    if (outside(R, R.ring, e.x, e.y, e.z)) continue;
    const unsigned id = dom_id(R, e.x, e.y, e.z);
    if (__ldcg(R.rb + id) != n - 1u - i) continue;  // set by atomics (in L2): read past L1
    const CD c = load_cell_par(R, R.ring, e.x, e.y, e.z);
    if (c.slot != NOSLOT) {
      R.amat[(size_t)c.slot * 512u + local_index(e.x, e.y, e.z)] = (unsigned char)e.w;
      dense_put(R, id, (unsigned)e.w & 255u, c.part);
    }
    R.rb[id] = 0xFFFFFFFFu;
  }
}

// Exclusive prefix of a per-thread flag over a CTA of up to 1024 threads; *total = the count. `cnt`: 32
// words of shared memory. All threads; two barriers.
__device__ __forceinline__ unsigned edit_scan(unsigned* cnt, bool f, unsigned* total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned b = __ballot_sync(FULLMASK, f);
  if (lane == 0u) cnt[warp] = (unsigned)__popc(b);
  __syncthreads();
  const unsigned c = lane < nw ? cnt[lane] : 0u;
  const unsigned before = __reduce_add_sync(FULLMASK, lane < warp ? c : 0u);
  *total = __reduce_add_sync(FULLMASK, c);
  __syncthreads();
  return before + (unsigned)__popc(b & lanemask_lt());
}

// Rain emitters in list order (for each cell: vol' = min(1, vol + amount) through set_volume, then
// activate it), one CTA. Cells of the list that differ do not touch each other, so a chunk of 1024
// runs at once; the first entry of a cell (claims in rb) takes the later ones of the chunk with it, one
// after another in registers, and the activations join the FIFO in list order by a scan. One warp in order
// spent ~0.8 us per emitter of a cell listed before and 1.2 per new one (1,024 of one cell: 845 us; in rounds of the
// chunk, one entry of each cell a round, 1.4 ms).
__global__ void __launch_bounds__(EDIT_THREADS) k_emit(Region R, const int* xyz, unsigned long long n, float amount) {
  __shared__ unsigned cnt[32], s_more[EDIT_THREADS];
  __shared__ int s_pd, s_ch;
  const unsigned tid = threadIdx.x;
  if (tid == 0) s_pd = s_ch = 0;
  unsigned long long tail = R.ctl->qtail;
  const unsigned long long head = R.ctl->qhead, tail0 = tail;
  __syncthreads();
  for (unsigned long long base = 0; base < n; base += blockDim.x) {
    const unsigned long long i = base + tid;
    int x = 0, y = 0, z = 0;
    bool open = false;
    unsigned id = 0;
    CD c = CD{0.0f, NOSLOT, 0u, 0, true};
    if (i < n) {
      x = xyz[3 * i];
      y = xyz[3 * i + 1];
      z = xyz[3 * i + 2];
      c = load_cell_par(R, R.ring, x, y, z);
      open = !cd_solid(c);
      if (open) id = dom_id(R, x, y, z);
    }
    s_more[tid] = 0u;
    if (open) atomicMin(R.rb + id, tid);
    __syncthreads();
    const unsigned first = open ? __ldcg(R.rb + id) : tid;  // set by atomics (in L2): read past L1
    const bool act = open && first == tid;
    if (first != tid) atomicAdd(&s_more[first], 1u);
    __syncthreads();
    // (an entry that needs no slot changes nothing, and so do the later ones of its cell)
    materialize_cta(R, act && set_volume_needs_slot(c, fminf(1.0f, __fadd_rn(cd_volume(c), amount))), c.gi, c.slot);
    int pd = 0;
    if (act) {
      bool wpart = false, wmat = false, ch = false;
      for (unsigned k = s_more[tid] + 1u; k; --k) {
        const SVPlan p = sv_plan(c.part, c.mat, c.slot != NOSLOT, fminf(1.0f, __fadd_rn(cd_volume(c), amount)));
        wpart |= p.wpart;
        wmat |= p.wmat;
        ch |= p.ch;
        pd += p.dp;
        if (!p.wmat && !(p.wpart && __float_as_uint(p.npart) != __float_as_uint(c.part))) break;  // the later ones do the same
        if (p.wpart) c.part = p.npart;
        if (p.wmat) c.mat = p.nmat;
      }
      if (c.slot != NOSLOT) {
        const size_t o = (size_t)c.slot * 512u + local_index(x, y, z);
        if (wpart) R.avol[o] = c.part;
        if (wmat) R.amat[o] = c.mat;
        dense_put(R, id, c.mat, c.part);
      }
      if (wmat) record_change(R, id);
      if (ch) s_ch = 1;
      R.rb[id] = 0xFFFFFFFFu;
    }
    if (pd) atomicAdd(&s_pd, pd);
    const bool isnew = act && !((__ldcg(&R.active[id >> 5]) >> (id & 31u)) & 1u);
    unsigned total;
    const unsigned off = edit_scan(cnt, isnew, &total);
    if (isnew) {
      R.queue[(tail + off) & R.qmask] = id;
      atomicOr(&R.active[id >> 5], 1u << (id & 31u));
    }
    tail += total;
  }
  __syncthreads();
  if (tid == 0) {
    Ctl& c = *R.ctl;
    c.partial_count += s_pd;
    c.qtail = tail;
    c.activations += tail - tail0;
    if (s_ch) c.changed = 1u;
    if (tail - head > R.qmask + 1ull) set_status(R, ST_OOM, 7);
  }
}

// apply_brush with an empty material (src/edit/brush.rs:93-111), one CTA: every listed solid voxel
// becomes air, once. Nothing is displaced or woken, so the list has no order to keep; the voxels are
// claimed (rb) so that one listed twice counts once.
__global__ void __launch_bounds__(EDIT_THREADS) k_carve(Region R, const int* xyz, unsigned long long n, unsigned long long* out_count) {
  __shared__ unsigned s_n;
  const unsigned tid = threadIdx.x;
  if (tid == 0) s_n = 0u;
  __syncthreads();
  for (unsigned long long base = 0; base < n; base += blockDim.x) {
    const unsigned long long i = base + tid;
    int x = 0, y = 0, z = 0;
    unsigned id = 0;
    bool hit = false;
    CD c = CD{0.0f, NOSLOT, 0u, 0, true};
    if (i < n) {
      x = xyz[3 * i];
      y = xyz[3 * i + 1];
      z = xyz[3 * i + 2];
      c = load_cell_par(R, R.ring, x, y, z);
      hit = !c.out && c.mat != 0 && c.mat != WATER;
    }
    if (hit) {
      id = dom_id(R, x, y, z);
      atomicMin(R.rb + id, tid);
    }
    __syncthreads();
    const bool win = hit && __ldcg(R.rb + id) == tid;  // set by atomics (in L2): read past L1
    __syncthreads();
    const bool need = win && c.slot == NOSLOT;
    materialize_cta(R, need, c.gi, c.slot);
    if (win) {
      if (c.slot != NOSLOT) {
        R.amat[(size_t)c.slot * 512u + local_index(x, y, z)] = 0;
        dense_put(R, id, 0u, c.part);
        record_change(R, id);
      }
      R.rb[id] = 0xFFFFFFFFu;
      atomicAdd(&s_n, 1u);
    }
    __syncthreads();
  }
  if (tid == 0 && out_count) *out_count = s_n;
}

// apply_brush with a solid material (src/edit/brush.rs:93-111) over a long list, one CTA. A listed water
// cell's water goes up its own column (FluidSim::displace, fluid.rs:370-408), so the columns of a stroke
// are independent as long as the cells of a column with water are listed upwards and it finds room above: a
// warp then takes a column, in registers. In chunks of the list: the voxels and columns are claimed (rb, stamp); every
// column is tried without writing, up to its first cell that does not fit (water that goes to the sides, a
// cell of such a column after one above it, a voxel listed twice, a column of more than 96 rows, water that
// goes to more than three cells). What the list holds before the first of those commits to the dense words and logs what
// each listed cell did, and the log is followed in list order: slots, the atlas, and the
// activations (27 around a displaced cell, then those that took its water), 16 cells at a time, each cell
// activated by its first mention. That first cell then takes its turn as brush_warp does (up to 64 cells when
// the next chunks stop early too), and the rest is the next chunk. One warp in list order spent 3.2 us
// on each displaced cell and 1.2 on a dry one: 257 dry cells 375 us in any order (here 80; 410 in an order that goes
// down while such columns had to be listed upwards too).
constexpr int BRUSH_THREADS = 512;
constexpr unsigned BRUSH_CHUNK = 4096, BRUSH_MIN = 12;
constexpr int BRUSH_ROWS = 4, BRUSH_TARGETS = 3;
constexpr int BRUSH_BELOW = 32;  // rows of a column that may lie below its first cell
static_assert(BRUSH_CHUNK * sizeof(uint4) <= MAX_CELLS_PER_TICK * sizeof(LvCell), "the log lies where a tick keeps its records");
// A log entry: .x = cells that took water | 4 placed | 8 it was water | 16 << t: cell t's voxel changed |
// 128 it keeps an entry; .y, .z, .w those cells, or the entry's volume.

// The listed cells before entry `limit` of the column of entry `lead`, from the lowest up, by one warp. Returns the
// first entry that does not fit, or `limit` (nothing is written unless `commit`).
__device__ __forceinline__ unsigned brush_column(const Region& R, const int* xyz, unsigned lead, unsigned limit, bool commit, uint4* log, int& pd,
                                                 unsigned& placed) {
  const unsigned lane = lane_id();
  const int x = xyz[3 * lead], z = xyz[3 * lead + 2];
  const int y = min(xyz[3 * lead + 1], (int)(__ldcg(R.stamp + dom_id(R, x, 1, z)) >> 1));  // (idle: 2^31 - 1)
  const unsigned id0 = dom_id(R, x, y, z);
  unsigned u[BRUSH_ROWS], at[BRUSH_ROWS], dirty = 0;
#pragma unroll
  for (int k = 0; k < BRUSH_ROWS; ++k) {
    const int up = 32 * k + (int)lane;
    const bool in = y + up < R.ny;
    u[k] = in ? R.dense[id0 + (unsigned)(up * R.PX)] : DC_SOLID;
    at[k] = in ? __ldcg(R.rb + id0 + (unsigned)(up * R.PX)) : NOSLOT;
  }
  // A column with water to displace is listed upwards up to `limit`: it ends before the first entry with an earlier
  // one above it. A later end then only takes the column's last cells away, so the commit finds what the try found.
  // (Cells without water touch nothing but themselves: their order is free.)
  bool wet = false;
#pragma unroll
  for (int k = 0; k < BRUSH_ROWS; ++k) wet |= at[k] < limit && dc_water(u[k]);
  if (!commit && __any_sync(FULLMASK, wet)) {
    unsigned above = NOSLOT, bad = NOSLOT;  // the earliest entry of the rows above
#pragma unroll
    for (int k = BRUSH_ROWS - 1; k >= 0; --k) {
      if (!__any_sync(FULLMASK, at[k] != NOSLOT)) continue;
      unsigned first = at[k];  // the earliest entry of the lane's cell and those above it
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_down_sync(FULLMASK, first, o);
        first = min(first, lane + (unsigned)o < 32u ? v : above);
      }
      const unsigned over = __shfl_down_sync(FULLMASK, first, 1);
      if (at[k] != NOSLOT && at[k] > (lane < 31u ? over : above)) bad = at[k] < bad ? at[k] : bad;
      above = __shfl_sync(FULLMASK, first, 0);
    }
    limit = min(limit, __reduce_min_sync(FULLMASK, bad));
  }
  bool ok = true;
#pragma unroll
  for (int k = 0; k < BRUSH_ROWS; ++k) {
    for (unsigned listed = __ballot_sync(FULLMASK, at[k] != NOSLOT); listed && ok; listed &= listed - 1u) {
      const unsigned b = (unsigned)__ffs(listed) - 1u;
      const unsigned i = __shfl_sync(FULLMASK, at[k], b), own = __shfl_sync(FULLMASK, u[k], b);
      if (i >= limit || dc_solid(own)) continue;  // (left for the next chunk, cells above it may come before it in the list)
      unsigned nt = 0, t[BRUSH_TARGETS] = {0, 0, 0}, flags = 4u;
      if ((int)own > 0) {
        flags |= 8u;
        float amount = dc_volume(own);
        if (lane == 0u && amount < 1.0f) pd -= 1;  // its entry goes
        bool shut = false;
#pragma unroll
        for (int kk = 0; kk < BRUSH_ROWS; ++kk) {
          if (kk < k || shut || amount <= 1e-6f) continue;
          const unsigned over = kk > k ? 0xFFFFFFFFu : ~((2u << b) - 1u);
          const unsigned solid = __ballot_sync(FULLMASK, dc_solid(u[kk])) & over;
          const unsigned below = solid ? (solid & (0u - solid)) - 1u : 0xFFFFFFFFu;
          const float cur = dc_volume(u[kk]);
          unsigned room = __ballot_sync(FULLMASK, !dc_solid(u[kk]) && __fsub_rn(1.0f, cur) > 0.0f) & over & below;
          for (; room && amount > 1e-6f; room &= room - 1u) {
            const unsigned q = (unsigned)__ffs(room) - 1u;
            const float cq = __shfl_sync(FULLMASK, cur, q);
            const unsigned uq = __shfl_sync(FULLMASK, u[kk], q);
            const float take = fminf(amount, __fsub_rn(1.0f, cq));
            if (!(take > 0.0f)) continue;
            const float nv = __fadd_rn(cq, take);
            amount = __fsub_rn(amount, take);
            const bool is_water = (int)uq > 0, mid = nv > 1e-6f && nv < full_level(), had = cq > 0.0f && cq < 1.0f;
            const bool wet = nv >= (is_water ? HIDE_BELOW : SHOW_AT);
            if (lane == q) {
              u[kk] = mid ? (__float_as_uint(nv) | (wet ? 0u : DC_AIR)) : (wet ? DC_FULL : 0u);
              dirty |= 1u << kk;
            }
            if (lane == 0u) pd += (mid ? 1 : 0) - (had ? 1 : 0);
            if (wet != is_water) flags |= 16u << nt;
            const unsigned tid_ = id0 + (unsigned)((32 * kk + (int)q) * R.PX);
            if (nt == 0u) t[0] = tid_;
            if (nt == 1u) t[1] = tid_;
            if (nt == 2u) t[2] = tid_;
            ++nt;
            if (nt > BRUSH_TARGETS) {
              ok = false;
              amount = 0.0f;
            }
          }
          shut = solid != 0u;
        }
        if (!commit && ok && amount > 1e-6f) {
          // to the sides, if one of them has room: during a stroke a cell only fills or turns solid, so one without
          // room stays so; where none has any, the water is gone (fluid.rs:396-408). Asked while nothing is written
          // (a commit goes no further than its try did): the side columns may be other warps'.
          const int row = R.PX * R.PY;
          const int off = lane == 0u ? 1 : lane == 1u ? -1 : lane == 2u ? row : -row;
          const unsigned us = lane < 4u ? R.dense[(int)(id0 + (32u * k + b) * (unsigned)R.PX) + off] : DC_SOLID;
          ok = shut && !__any_sync(FULLMASK, !dc_solid(us) && __fsub_rn(1.0f, dc_volume(us)) > 0.0f);
        }
      } else if (own != 0u) {  // a film of hidden water: its entry stays in the solid cell
        flags |= 128u;
        t[0] = __float_as_uint(dc_volume(own));
      }
      if (lane == b) {
        u[k] = (flags & 128u) ? DC_SOLID_PART : DC_SOLID;
        dirty |= 1u << k;
      }
      placed += 1u;
      if (!ok) limit = i;
      if (commit && lane == 0u) log[i] = make_uint4(flags | nt, t[0], t[1], t[2]);
    }
  }
  if (commit) {
#pragma unroll
    for (int k = 0; k < BRUSH_ROWS; ++k)
      if ((dirty >> k) & 1u) R.dense[id0 + (unsigned)((32 * k + (int)lane) * R.PX)] = u[k];
  }
  return limit;
}

__global__ void __launch_bounds__(BRUSH_THREADS) k_brush(Region R, const int* list, unsigned long long n, int m, unsigned long long* out_count) {
  __shared__ EditSmem es;
  __shared__ unsigned cnt[32], s_placed, s_ch, s_limit;
  __shared__ int s_pd;
  const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const int* ring = edit_ring(R, es.ring);
  uint4* log = reinterpret_cast<uint4*>(R.lv);
  if (tid == 0) {
    s_placed = s_ch = 0u;
    s_pd = 0;
  }
  unsigned long long serial = 0;
  unsigned turns = 1, size = BRUSH_CHUNK;  // cells that take their turn by themselves when a chunk stops early; the next chunk
  for (unsigned long long base = 0; base < n;) {
    const int* xyz = list + 3 * base;
    const unsigned all = (unsigned)min((unsigned long long)size, n - base);
    if (tid == 0) s_limit = all;
    __syncthreads();
    // ---- claims: a voxel's first entry, a column's first entry (at its layer 0), its lowest cell below that one (layer 1)
    for (unsigned i = tid; i < all; i += BRUSH_THREADS) {
      const int x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
      log[i] = make_uint4(0u, 0u, 0u, 0u);
      if (outside(R, ring, x, y, z)) continue;
      atomicMin(R.rb + dom_id(R, x, y, z), i);
      atomicMin(R.stamp + dom_id(R, x, 0, z), i);
    }
    __syncthreads();
    for (unsigned i = tid; i < all; i += BRUSH_THREADS) {
      const int x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
      if (outside(R, ring, x, y, z)) continue;
      const unsigned id = dom_id(R, x, y, z), lead = __ldcg(R.stamp + dom_id(R, x, 0, z));
      const int yl = xyz[3 * lead + 1];
      bool end = __ldcg(R.rb + id) != i || y - yl >= 32 * BRUSH_ROWS - BRUSH_BELOW || yl - y > BRUSH_BELOW;
      if (y < yl && !end) {  // (water in one of the two: the try would find it too, after trying more)
        end = dc_water(R.dense[id]) || dc_water(R.dense[dom_id(R, x, yl, z)]);
        if (!end) atomicMin(R.stamp + dom_id(R, x, 1, z), 2u * (unsigned)y + 1u);
      }
      if (end) atomicMin(&s_limit, i);
    }
    __syncthreads();
    // ---- the columns: tried, then committed
    int pd = 0;
    unsigned placed = 0, len = 0;
    for (int commit = 0; commit < 2; ++commit) {
      len = s_limit;
      pd = 0;
      placed = 0;
      __syncthreads();
      for (unsigned b0 = warp; b0 < len; b0 += BRUSH_THREADS) {  // neighbours in the list to different warps: often a row of columns
        const unsigned i = b0 + lane * (BRUSH_THREADS / 32);
        bool lead = false;
        if (i < len) {
          const int x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
          lead = !outside(R, ring, x, y, z) && __ldcg(R.stamp + dom_id(R, x, 0, z)) == i;
        }
        for (unsigned mask = __ballot_sync(FULLMASK, lead); mask; mask &= mask - 1u) {
          const unsigned fit = brush_column(R, xyz, b0 + ((unsigned)__ffs(mask) - 1u) * (BRUSH_THREADS / 32), len, commit != 0, log, pd, placed);
          if (lane == 0u && fit < len) atomicMin(&s_limit, fit);
        }
      }
      __syncthreads();
    }
    for (unsigned i = tid; i < all; i += BRUSH_THREADS) {
      const int x = xyz[3 * i], y = xyz[3 * i + 1], z = xyz[3 * i + 2];
      if (outside(R, ring, x, y, z)) continue;
      R.rb[dom_id(R, x, y, z)] = 0xFFFFFFFFu;
      R.stamp[dom_id(R, x, 0, z)] = 0xFFFFFFFFu;
      R.stamp[dom_id(R, x, 1, z)] = 0xFFFFFFFFu;
    }
    __syncthreads();
    if (pd) atomicAdd(&s_pd, pd);
    if (lane == 0u && placed) atomicAdd(&s_placed, placed);
    // ---- the atlas, in list order: the cells that took a cell's water, then the cell
    for (unsigned b0 = 0; b0 < len; b0 += BRUSH_THREADS) {
      const unsigned i = b0 + tid;
      uint4 e = make_uint4(0u, 0u, 0u, 0u);
      if (i < len) e = log[i];
      const unsigned nt = e.x & 3u;
      unsigned w = (e.x & 4u) ? (1u << nt) - 1u | 8u : 0u, need = 0, id[4] = {e.y, e.z, e.w, 0u}, gi[4], g[4], at[4];
      if (w) id[3] = dom_id(R, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2]);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        gi[q] = g[q] = at[q] = 0u;
        if (!((w >> q) & 1u)) continue;
        int x, y, z;
        dom_xyz(R, id[q], x, y, z);
        gi[q] = grid_index(R, x >> 3, y >> 3, z >> 3);
        at[q] = local_index(x, y, z);
        g[q] = __ldcg(R.grid + gi[q]);
        need |= g[q] < 256u ? 1u << q : 0u;
      }
      if (__syncthreads_or(need != 0u)) {
        give_slots<4>(AtlasRef{R.grid, R.amat, R.avol, R.ctl, R.atlas_cap}, need, gi);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if ((need >> q) & 1u) g[q] = __ldcg(R.grid + gi[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (!((w >> q) & 1u)) continue;
        if (q == 3 || ((e.x >> (4 + q)) & 1u)) {
          record_change(R, id[q]);
          if (q < 3) s_ch = 1u;
        }
        if (g[q] < 256u) continue;  // (no slot left: the status says so)
        const size_t o = (size_t)(g[q] - 256u) * 512u + at[q];
        if (q == 3) {
          R.avol[o] = (e.x & 128u) ? __uint_as_float(e.y) : 0.0f;
          R.amat[o] = (unsigned char)m;
          continue;
        }
        const unsigned u = R.dense[id[q]];
        if (dc_solid(u)) continue;  // placed later in the list
        const float v = dc_volume(u);
        R.avol[o] = v < 1.0f ? v : 0.0f;
        R.amat[o] = (int)u > 0 ? WATER : (unsigned char)0;
      }
    }
    __syncthreads();
    // ---- the activations, in list order, a displaced cell per warp
    unsigned long long tail = R.ctl->qtail;
    const unsigned long long tail0 = tail;
    for (unsigned b0 = 0; b0 < len; b0 += BRUSH_THREADS / 32) {
      const unsigned i = b0 + warp;
      bool act = false;
      unsigned id = 0;
      if (i < len) {
        const uint4 e = log[i];
        if (e.x & 8u) {
          if (lane < 27u) {
            const int x = xyz[3 * i] - 1 + (int)lane % 3, y = xyz[3 * i + 1] - 1 + (int)lane / 3 % 3, z = xyz[3 * i + 2] - 1 + (int)lane / 9;
            act = y >= 0;
            if (act && !in_dom(R, x, y, z)) {
              set_status(R, ST_RANGE, 3);
              act = false;
            }
            if (act) id = dom_id(R, x, y, z);
          } else if (lane - 27u < (e.x & 3u)) {
            act = true;
            id = lane == 27u ? e.y : lane == 28u ? e.z : e.w;
          }
        }
      }
      if (!__syncthreads_or(act)) continue;
      if (act) atomicMin(R.rb + id, tid);
      __syncthreads();
      const bool first = act && __ldcg(R.rb + id) == tid;
      const bool isnew = first && !((__ldcg(&R.active[id >> 5]) >> (id & 31u)) & 1u);
      unsigned total;
      const unsigned off = edit_scan(cnt, isnew, &total);
      if (isnew) {
        R.queue[(tail + off) & R.qmask] = id;
        atomicOr(&R.active[id >> 5], 1u << (id & 31u));
      }
      if (first) R.rb[id] = 0xFFFFFFFFu;
      tail += total;
    }
    __syncthreads();
    if (tid == 0) {
      R.ctl->qtail = tail;
      R.ctl->activations += tail - tail0;
      if (tail - R.ctl->qhead > R.qmask + 1ull) set_status(R, ST_OOM, 7);
    }
    __syncthreads();
    base += len;
    if (len == all) {
      size = min(4u * size, BRUSH_CHUNK);
      continue;
    }
    // ---- the cell that did not fit
    const unsigned k = (unsigned)min((unsigned long long)turns, n - base);
    if (warp == 0) {
      WS W;
      load_ws(R, W);
      for (unsigned i = len; i < len + k; ++i) serial += brush_warp(R, W, ring, xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], (unsigned char)m);
      if (W.qtail - W.qhead > R.qmask + 1ull) set_status(R, ST_OOM, 7);
      commit_ws(R, W);
    }
    __syncthreads();
    base += k;
    turns = len >= 64u ? 1u : min(2u * turns, 64u);
    size = min(max(128u, 2u * len), BRUSH_CHUNK);  // (what lies behind the next such cell is tried for nothing)
  }
  if (tid == 0) {
    R.ctl->partial_count += s_pd;
    if (s_ch) R.ctl->changed = 1u;
    if (out_count) *out_count = serial + s_placed;
  }
}

enum EditKind { ED_DISPLACE = 1, ED_BRUSH = 2, ED_EMIT = 3, ED_SET_PARTIAL = 4 };

// kind/args: ED_DISPLACE: xyz[0..3]; ED_BRUSH: n cells, m; ED_SET_PARTIAL: xyz[0..3], amount.
__global__ void __launch_bounds__(32) k_edit(Region R, int kind, const int* xyz, unsigned long long n, int m, float amount,
                                             unsigned long long* out_count) {
  __shared__ EditSmem es;
  const unsigned lane = lane_id();
  const int* ring = edit_ring(R, es.ring);
  WS W;
  load_ws(R, W);
  unsigned long long cnt = 0;
  if (kind == ED_DISPLACE) {
    displace_warp(R, W, ring, xyz[0], xyz[1], xyz[2], load_column(R, ring, xyz[0], xyz[1], xyz[2]));
  } else if (kind == ED_BRUSH) {
    // apply_brush (src/edit/brush.rs:93-111), cell after cell: a displacement moves water into cells
    // that may be listed later. The list is read 32 cells at a time.
    for (unsigned long long base = 0; base < n; base += 32ull) {
      const unsigned long long i = base + lane;
      const int lx = i < n ? xyz[3 * i] : 0, ly = i < n ? xyz[3 * i + 1] : 0, lz = i < n ? xyz[3 * i + 2] : 0;
      const int here = (int)min(n - base, 32ull);
      for (int k = 0; k < here; ++k)
        cnt += brush_warp(R, W, ring, __shfl_sync(FULLMASK, lx, k), __shfl_sync(FULLMASK, ly, k), __shfl_sync(FULLMASK, lz, k), (unsigned char)m);
    }
  } else if (kind == ED_SET_PARTIAL) {
    // FluidSim::set_partial (fluid.rs:278-282): PartialField::set only, voxel untouched
    int x = xyz[0], y = xyz[1], z = xyz[2];
    if (amount > 0.0f && amount < 1.0f) {
      CD c = load_cell(R, ring, x, y, z);
      if (c.out) {
        if (lane == 0 && atomicCAS(&R.ctl->status, 0, ST_RANGE) == 0) R.ctl->err_info = 6;
      } else {
        bool need = lane == 0 && c.slot == NOSLOT;
        materialize_lanes(R, need, c.gi, c.slot);
        if (lane == 0 && c.slot != NOSLOT) {
          if (!(c.part > 0.0f)) W.pdelta += 1;
          R.avol[(size_t)c.slot * 512u + local_index(x, y, z)] = amount;
          dense_put(R, dom_id(R, x, y, z), c.mat, amount);
        }
      }
    }
  }
  if (W.qtail - W.qhead > R.qmask + 1ull) set_status(R, ST_OOM, 7);
  commit_ws(R, W);
  if (lane == 0 && out_count) *out_count = cnt;
}

// The first cell of the brick at grid index gi; false where a ring world's slot holds no chunk.
__device__ __forceinline__ bool brick_origin(const Region& R, unsigned gi, int& x, int& y, int& z) {
  int bx = (int)(gi % (unsigned)R.bx), bz = (int)(gi / ((unsigned)R.bx * (unsigned)R.by));
  y = (int)((gi / (unsigned)R.bx) % (unsigned)R.by) * 8;
  if (R.ring_w) {
    const int* s = R.ring + 3 * ((bz >> 4) * R.ring_w + (bx >> 4));
    if (!s[2]) return false;
    bx = s[0] * 16 + (bx & 15);
    bz = s[1] * 16 + (bz & 15);
  }
  x = bx * 8;
  z = bz * 8;
  return true;
}

// The dense words of a box of columns from the grid and the atlas, a row of cells per CTA: the whole domain
// after an upload, one chunk's 128 x 128 columns when it comes or goes. Bound by the words' stores
// (a 576 x 160 x 576 domain: 212 MB; a chunk of 256 layers: 19 MB, where the whole domain of 9 x 9 chunks is 1.7 GB:
// an eviction and a paste there 6.3 ms with it, 4.2 with the chunk).
__global__ void __launch_bounds__(256) k_dense(Region R, int x0, int z0, int sx, int sz) {
  for (unsigned row = blockIdx.x; row < (unsigned)sz * (unsigned)R.PY; row += gridDim.x) {
    const int dz = (int)udiv(row, (unsigned)R.PY, R.my), y = (int)(row - (unsigned)dz * (unsigned)R.PY), z = z0 + dz;
    for (int x = x0 + (int)threadIdx.x; x < x0 + sx; x += (int)blockDim.x) {
      const CD c = load_cell(R, R.ring, x, y, z);
      R.dense[dom_id(R, x, y, z)] = dense_code(c.out, c.mat, __float_as_uint(c.part));
    }
  }
}

// The dense words after a reset: the partial volumes are gone, the materials stand, so that only the cells of
// bricks with a slot can differ (slot_gi: k_slot_map's), a warp each. Latency: a brick is one round of loads and 64
// sectors of stores.
__global__ void __launch_bounds__(256) k_dense_slots(Region R, const int* slot_gi, unsigned nslots) {
  const unsigned lane = lane_id();
  for (unsigned s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslots; s += (gridDim.x * blockDim.x) >> 5) {
    const int gi = slot_gi[s];
    int x0, y0, z0;
    if (gi < 0 || !brick_origin(R, (unsigned)gi, x0, y0, z0)) continue;
    const bool held = !R.ring_w || chunk_loaded(R, R.ring, x0 >> 7, z0 >> 7);
    unsigned char mat[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) mat[k] = R.amat[(size_t)s * 512u + 32u * k + lane];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const unsigned v = 32u * k + lane;
      const int x = x0 + (int)(v & 7u), y = y0 + (int)((v >> 3) & 7u), z = z0 + (int)(v >> 6);
      const bool out = !held || y >= R.ny || (!R.ring_w && (x >= R.nx || z >= R.nz));
      if (in_dom(R, x, y, z)) R.dense[dom_id(R, x, y, z)] = dense_code(out, mat[k], 0u);
    }
  }
}

// ------------------------------------------------------------------------- inspection
__device__ __forceinline__ unsigned long long cell_hash(int x, int y, int z, unsigned m, unsigned vb) {
  return fmix64(ref_key(x, y, z) * 0x9E3779B97F4A7C15ULL + (((unsigned long long)m << 32) | vb));
}

// Sum over cells with (material, partial bits) != (0, 0) of cell_hash; one thread per voxel.
__global__ void k_state_digest(Region R, unsigned long long* out) {
  const unsigned long long nb = (unsigned long long)R.bx * R.by * R.bz;
  unsigned long long acc = 0;
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < nb * 512ull;
       t += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long gi = t >> 9;
    unsigned l = (unsigned)(t & 511u);
    int bx = (int)(gi % R.bx), by = (int)((gi / R.bx) % R.by), bz = (int)(gi / ((unsigned long long)R.bx * R.by));
    int ax = bx, az = bz;
    if (R.ring_w) {
      const int* s = R.ring + 3 * ((bz / 16) * R.ring_w + (bx / 16));
      if (!s[2]) continue;
      ax = s[0] * 16 + bx % 16;
      az = s[1] * 16 + bz % 16;
    }
    int x = ax * 8 + (int)(l & 7u), y = by * 8 + (int)((l >> 3) & 7u), z = az * 8 + (int)(l >> 6);
    if (y >= R.ny) continue;
    unsigned g = R.grid[gi];
    unsigned m;
    float p = 0.0f;
    if (g < 256u) {
      m = g;
    } else {
      // atlas local index == voxel index here (x|y<<3|z<<6 with l's bit layout)
      m = R.amat[(size_t)(g - 256u) * 512u + l];
      p = R.avol[(size_t)(g - 256u) * 512u + l];
    }
    unsigned vb = __float_as_uint(p);
    if (m == 0 && vb == 0) continue;
    acc += cell_hash(x, y, z, m, vb);
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULLMASK, acc, o);
  if ((threadIdx.x & 31u) == 0) atomicAdd(out, acc);
}

// Partial entries kept for evicted ring chunks (x, y, z, volume bits, cell id per entry) whose cell
// still has its detbits bit: hashed like cells outside the loaded chunks (material 0).
__global__ void k_detached_digest(Region R, const int4* ent, const unsigned* ids, unsigned n, unsigned long long* out) {
  unsigned long long acc = 0;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned id = ids[i];
    if (!((R.detbits[id >> 5] >> (id & 31u)) & 1u)) continue;
    const int4 e = ent[i];
    acc += cell_hash(e.x, e.y, e.z, 0u, (unsigned)e.w);
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULLMASK, acc, o);
  if ((threadIdx.x & 31u) == 0) atomicAdd(out, acc);
}

// Ring paste/evict helpers: gather the partial volumes of atlas slots; write whole bricks (materials
// and volumes) into slots; set, clear or read bits of cells.
__global__ void k_gather_vol(const float* avol, const unsigned* slots, unsigned n, float* out) {
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n * 512u; t += gridDim.x * blockDim.x)
    out[t] = avol[(size_t)slots[t >> 9] * 512u + (t & 511u)];
}
__global__ void k_scatter_bricks(unsigned char* amat, float* avol, const unsigned* slots, unsigned n, const unsigned char* mats,
                                 const float* vols) {
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n * 512u; t += gridDim.x * blockDim.x) {
    const size_t o = (size_t)slots[t >> 9] * 512u + (t & 511u);
    amat[o] = mats[t];
    avol[o] = vols[t];
  }
}
// op 0: clear, 1: set, 2: read into out
__global__ void k_cell_bits(unsigned* bits, const unsigned* ids, unsigned n, int op, unsigned* out) {
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const unsigned id = ids[i], bit = 1u << (id & 31u);
    if (op == 0) atomicAnd(bits + (id >> 5), ~bit);
    else if (op == 1) atomicOr(bits + (id >> 5), bit);
    else out[i] = (bits[id >> 5] & bit) ? 1u : 0u;
  }
}

// Order-dependent digest of a list of domain ids: sum fmix64(ref_key * golden + position).
__global__ void k_list_digest(Region R, const unsigned* ids, unsigned long long n, unsigned long long head, unsigned long long mask,
                              unsigned long long* out) {
  unsigned long long acc = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned id = ids[(head + i) & mask];
    int x, y, z;
    dom_xyz(R, id, x, y, z);
    acc += fmix64(ref_key(x, y, z) * 0x9E3779B97F4A7C15ULL + i);
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(FULLMASK, acc, o);
  if ((threadIdx.x & 31u) == 0) atomicAdd(out, acc);
}

__global__ void k_export_box(Region R, int x0, int y0, int z0, int sx, int sy, int sz, unsigned char* mat, float* part) {
  const unsigned long long total = (unsigned long long)sx * sy * sz;
  for (unsigned long long t = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; t < total; t += (unsigned long long)gridDim.x * blockDim.x) {
    int x = x0 + (int)(t % sx), y = y0 + (int)((t / sx) % sy), z = z0 + (int)(t / ((unsigned long long)sx * sy));
    CD c = load_cell(R, R.ring, x, y, z);
    // get_voxel reads 0 outside (sparse_volume.rs:238-241); partials of outside cells are none
    if (mat) mat[t] = c.out ? 0 : c.mat;
    if (part) part[t] = c.out ? 0.0f : c.part;
  }
}

// Gather pending voxel changes (final material) for the host and clear their bits.
struct Voxel {
  int x, y, z;
  unsigned char m, pad[3];
};
__global__ void k_gather_changes(Region R, unsigned long long n, Voxel* out) {
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n; i += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned id = R.chg[i];
    int x, y, z;
    dom_xyz(R, id, x, y, z);
    CD c = load_cell(R, R.ring, x, y, z);
    Voxel v;
    v.x = x;
    v.y = y;
    v.z = z;
    v.m = c.mat;
    v.pad[0] = v.pad[1] = v.pad[2] = 0;
    out[i] = v;
    atomicAnd(&R.chgbits[id >> 5], ~(1u << (id & 31)));
  }
}

// Partial entries in (z, y, x) order, which is the order of domain ids: a count per row of cells from the bricks that
// have a slot (no other cell has an entry), sums over chunks of rows, and every chunk writes its rows behind the
// ones before it. What is read follows the bricks and the rows with entries, not the domain: passes over all its dense
// words took 700 us a call on the world of 9 x 9 chunks, entries gathered by slot and sorted on the host 180 us with
// hardly an entry and 610 with 9,656 (dam break).
constexpr unsigned PART_TILE = 128, PART_CHUNKS = 4096;  // rows of a chunk: a multiple of the tile, so few chunks that each adds up those before it
__device__ __forceinline__ bool dc_has_part(unsigned u) { return dc_solid(u) ? u == DC_SOLID_PART : dc_volume(u) > 0.0f && dc_volume(u) < 1.0f; }
__device__ __forceinline__ unsigned block_sum(unsigned v) {
  __shared__ unsigned s[32];
  v = __reduce_add_sync(FULLMASK, v);
  __syncthreads();
  if ((threadIdx.x & 31u) == 0u) s[threadIdx.x >> 5] = v;
  __syncthreads();
  return __reduce_add_sync(FULLMASK, (threadIdx.x & 31u) < (blockDim.x >> 5) ? s[threadIdx.x & 31u] : 0u);
}
// Entries per row (z - pz0) * PY + y; a warp per slot, eight lanes per row of its brick.
__global__ void __launch_bounds__(256) k_part_rows(Region R, const int* slot_gi, unsigned nslots, unsigned* rows) {
  const unsigned lane = lane_id();
  for (unsigned s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslots; s += (gridDim.x * blockDim.x) >> 5) {
    const int gi = slot_gi[s];
    int x0, y0, z0;
    if (gi < 0 || !brick_origin(R, (unsigned)gi, x0, y0, z0)) continue;
    unsigned u[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const unsigned v = 32u * k + lane;
      const int x = x0 + (int)(v & 7u), y = y0 + (int)((v >> 3) & 7u), z = z0 + (int)(v >> 6);
      u[k] = in_dom(R, x, y, z) ? R.dense[dom_id(R, x, y, z)] : 0u;
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const unsigned c = (unsigned)__popc((__ballot_sync(FULLMASK, dc_has_part(u[k])) >> (lane & 24u)) & 0xFFu);
      const unsigned v = 32u * k + lane;
      if (c && (lane & 7u) == 0u) atomicAdd(rows + (size_t)(z0 + (int)(v >> 6) - R.pz0) * (unsigned)R.PY + (unsigned)(y0 + (int)((v >> 3) & 7u)), c);
    }
  }
}
__global__ void __launch_bounds__(PART_TILE) k_part_sums(const unsigned* rows, unsigned nrows, unsigned per, unsigned* sums) {
  unsigned c = 0;
  const unsigned r0 = blockIdx.x * per, r1 = min(nrows, r0 + per);
  for (unsigned r = r0 + threadIdx.x; r < r1; r += PART_TILE) c += rows[r];
  c = block_sum(c);
  if (threadIdx.x == 0) sums[blockIdx.x] = c;
}
__global__ void __launch_bounds__(PART_TILE) k_part_write(Region R, const unsigned* rows, unsigned nrows, unsigned per, const unsigned* sums, int* xyz, float* vol,
                                                          unsigned long long cap) {
  __shared__ unsigned s_cnt[PART_TILE / 32], s_nz[PART_TILE / 32], s_row[PART_TILE], s_at[PART_TILE];
  const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  if (sums[blockIdx.x] == 0u) return;
  unsigned before = 0;
  for (unsigned b = tid; b < blockIdx.x; b += PART_TILE) before += sums[b];
  before = block_sum(before);
  const unsigned r0 = blockIdx.x * per, r1 = min(nrows, r0 + per);
  for (unsigned base = r0; base < r1; base += PART_TILE) {
    // ---- the tile's rows with entries, and where each one's begin
    const unsigned c = base + tid < r1 ? rows[base + tid] : 0u;
    unsigned pre = c;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(FULLMASK, pre, o);
      if (lane >= (unsigned)o) pre += v;
    }
    const unsigned b = __ballot_sync(FULLMASK, c != 0u);
    __syncthreads();
    if (lane == 31u) {
      s_cnt[warp] = pre;
      s_nz[warp] = (unsigned)__popc(b);
    }
    __syncthreads();
    unsigned at = before + pre - c, k0 = (unsigned)__popc(b & lanemask_lt()), full = 0;
#pragma unroll
    for (unsigned w = 0; w < PART_TILE / 32; ++w) {
      at += w < warp ? s_cnt[w] : 0u;
      k0 += w < warp ? s_nz[w] : 0u;
      before += s_cnt[w];
      full += s_nz[w];
    }
    if (c) {
      s_row[k0] = base + tid;
      s_at[k0] = at;
    }
    __syncthreads();
    // ---- a row per warp
    for (unsigned k = warp; k < full; k += PART_TILE / 32) {
      const unsigned row = s_row[k];
      const unsigned id0 = row * (unsigned)R.PX;
      unsigned long long p = s_at[k];
      for (unsigned x0 = 0; x0 < (unsigned)R.PX; x0 += 128u) {  // four loads under way at a time
        unsigned u[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) u[e] = x0 + 32u * e + lane < (unsigned)R.PX ? R.dense[id0 + x0 + 32u * e + lane] : 0u;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const bool has = dc_has_part(u[e]);
          const unsigned m = __ballot_sync(FULLMASK, has);
          const unsigned long long i = p + (unsigned)__popc(m & lanemask_lt());
          if (has && i < cap) {
            int x, y, z;
            dom_xyz(R, id0 + x0 + 32u * e + lane, x, y, z);
            xyz[3 * i] = x;
            xyz[3 * i + 1] = y;
            xyz[3 * i + 2] = z;
            vol[i] = dc_solid(u[e]) ? load_cell(R, R.ring, x, y, z).part : dc_volume(u[e]);
          }
          p += (unsigned)__popc(m);
        }
      }
    }
  }
}

__global__ void k_slot_map(Region R, int* slot_brick, unsigned nslots) {
  const unsigned long long nb = (unsigned long long)R.bx * R.by * R.bz;
  for (unsigned long long gi = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; gi < nb; gi += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned g = R.grid[gi];
    if (g >= 256u && g - 256u < nslots) slot_brick[g - 256u] = (int)gi;
  }
}

}  // namespace vfe

namespace vfe {

// ------------------------------------------------------------------ wake-proposal features
// Per materialised brick (atlas slot): aggregates of its 512 cells.
struct SlotAggr {
  float wsum, wmax;
  unsigned npart, nwater, nsolid, nactive, ntop;
  int gi;  // grid index, -1 for a slot no brick uses
};

__global__ void k_slot_aggr(Region R, const int* slot_gi, unsigned nslots, SlotAggr* out) {
  __shared__ float s_sum[4], s_max[4];
  __shared__ unsigned s_cnt[4][5];
  const unsigned tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;  // 128 threads
  for (unsigned s = blockIdx.x; s < nslots; s += gridDim.x) {
    const int gi = slot_gi[s];
    float sum = 0.f, mx = 0.f;
    unsigned c[5] = {0, 0, 0, 0, 0};
    if (gi >= 0) {
      int bx = gi % R.bx, by = (gi / R.bx) % R.by, bz = gi / (R.bx * R.by);
      if (R.ring_w) {
        const int* rs = R.ring + 3 * ((bz / 16) * R.ring_w + (bx / 16));
        bx = rs[0] * 16 + bx % 16;
        bz = rs[1] * 16 + bz % 16;
      }
      for (unsigned l = tid; l < 512u; l += 128u) {
        const size_t o = (size_t)s * 512u + l;
        const unsigned m = R.amat[o];
        const float p = R.avol[o];
        const float v = p > 0.f ? p : (m == WATER ? 1.f : 0.f);
        sum += v;
        mx = fmaxf(mx, v);
        c[0] += p > 0.f;
        c[1] += m == WATER;
        c[2] += (m != 0u && m != WATER);
        const int x = bx * 8 + (int)(l & 7u), y = by * 8 + (int)((l >> 3) & 7u), z = bz * 8 + (int)(l >> 6);
        if (in_dom(R, x, y, z)) {
          unsigned id = dom_id(R, x, y, z);
          c[3] += (R.active[id >> 5] >> (id & 31)) & 1u;
        }
        if (v > 0.f && ((l >> 3) & 7u) < 7u) {  // water with air above (within the brick)
          const unsigned m2 = R.amat[o + 8];
          const float p2 = R.avol[o + 8];
          c[4] += (m2 == 0u && !(p2 > 0.f));
        }
      }
    }
    for (int off = 16; off; off >>= 1) {
      sum += __shfl_xor_sync(FULLMASK, sum, off);
      mx = fmaxf(mx, __shfl_xor_sync(FULLMASK, mx, off));
      for (int k = 0; k < 5; ++k) c[k] += __shfl_xor_sync(FULLMASK, c[k], off);
    }
    if (lane == 0) {
      s_sum[warp] = sum;
      s_max[warp] = mx;
      for (int k = 0; k < 5; ++k) s_cnt[warp][k] = c[k];
    }
    __syncthreads();
    if (tid == 0) {
      SlotAggr a;
      a.wsum = s_sum[0] + s_sum[1] + s_sum[2] + s_sum[3];
      a.wmax = fmaxf(fmaxf(s_max[0], s_max[1]), fmaxf(s_max[2], s_max[3]));
      unsigned t[5];
      for (int k = 0; k < 5; ++k) t[k] = s_cnt[0][k] + s_cnt[1][k] + s_cnt[2][k] + s_cnt[3][k];
      a.npart = t[0];
      a.nwater = t[1];
      a.nsolid = t[2];
      a.nactive = t[3];
      a.ntop = t[4];
      a.gi = gi;
      out[s] = a;
    }
    __syncthreads();
  }
}

// Aggregate of the face neighbour (dx,dy,dz) of grid cell gi: its slot's, or the uniform value's.
__device__ __forceinline__ void neighbour_aggr(const Region& R, const SlotAggr* aggr, int gi, int dx, int dy, int dz, float& wsum,
                                               float& act, int& nslot) {
  int bx = gi % R.bx + dx, by = (gi / R.bx) % R.by + dy, bz = gi / (R.bx * R.by) + dz;
  wsum = 0.f;
  act = 0.f;
  nslot = -1;
  if (by < 0 || by >= R.by) return;
  if (!R.ring_w && (bx < 0 || bz < 0 || bx >= R.bx || bz >= R.bz)) return;
  unsigned g = R.grid[grid_index(R, bx, by, bz)];
  if (g >= 256u) {
    nslot = (int)(g - 256u);
    wsum = aggr[nslot].wsum;
    act = (float)aggr[nslot].nactive;
  } else if (g == WATER) {
    wsum = 512.f;
  }
}

// Features (32 fp16 per slot): water sum, max level, partial/water/solid/active counts, exposed
// surface, the six face neighbours' water sums and active counts, water-sum changes over the last
// four calls (own and the faces': the flux proxy), wake recency, height, bias.
__global__ void k_slot_features(Region R, const SlotAggr* aggr, unsigned nslots, const float* hist, unsigned hpos, unsigned tick,
                                __half* X) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < nslots; s += gridDim.x * blockDim.x) {
    float f[32];
    for (int k = 0; k < 32; ++k) f[k] = 0.f;
    const SlotAggr a = aggr[s];
    if (a.gi >= 0) {
      const float old = hist[(size_t)s * 4 + ((hpos + 1) & 3u)];
      f[0] = a.wsum / 512.f;
      f[1] = a.wmax;
      f[2] = a.npart / 512.f;
      f[3] = a.nwater / 512.f;
      f[4] = a.nsolid / 512.f;
      f[5] = a.nactive / 512.f;
      f[6] = a.ntop / 64.f;
      const int D[6][3] = {{1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1}};
      for (int k = 0; k < 6; ++k) {
        float w, ac;
        int ns;
        neighbour_aggr(R, aggr, a.gi, D[k][0], D[k][1], D[k][2], w, ac, ns);
        f[7 + k] = w / 512.f;
        f[13 + k] = ac / 512.f;
        f[20 + k] = ns >= 0 ? (w - hist[(size_t)ns * 4 + ((hpos + 1) & 3u)]) / 64.f : 0.f;
      }
      f[19] = (a.wsum - old) / 64.f;
      const unsigned lw = R.last_woken[s];
      const unsigned age = lw ? tick - lw : 0xFFFFFFFFu;
      f[26] = age <= 1u ? 1.f : 0.f;
      f[27] = age <= 4u ? 1.f : 0.f;
      f[28] = lw ? 1.f / (1.f + (float)age) : 0.f;
      f[29] = (float)(((a.gi / R.bx) % R.by) * 8) / (float)R.ny;
      f[30] = 1.f;
      f[31] = a.nactive ? 1.f : 0.f;
    }
    __half2* out = reinterpret_cast<__half2*>(X + (size_t)s * 32);
    for (int k = 0; k < 16; ++k) out[k] = __floats2half2_rn(f[2 * k], f[2 * k + 1]);
  }
}

__global__ void k_slot_hist(const SlotAggr* aggr, unsigned nslots, float* hist, unsigned hpos) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < nslots; s += gridDim.x * blockDim.x)
    hist[(size_t)s * 4 + (hpos & 3u)] = aggr[s].gi >= 0 ? aggr[s].wsum : 0.f;
}

// Label: a cell of the slot's brick was drained in ticks (since, now].
__global__ void k_slot_labels(Region R, unsigned nslots, unsigned since, unsigned now, float* y) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < nslots; s += gridDim.x * blockDim.x) {
    const unsigned lw = R.last_woken[s];
    y[s] = (lw > since && lw <= now) ? 1.f : 0.f;
  }
}

// Pre-stage the bricks the proposal expects to wake: what the sweep and its searches read of their cells, the dense
// words (64 rows of one sector), into L2. `staged` counts the slots, a thread each; a thread per grid word finds
// their bricks. It gains little, for most of a region's words are in L2: 40 ticks of the ring world 117.2 ms, 117.7
// when it fetched the atlas, which the sweep no longer reads.
__global__ void k_stage(Region R, unsigned nslots, const float* prob, float thr, unsigned* staged) {
  const unsigned t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
  for (unsigned s = t0; s < nslots; s += nt)
    if (prob[s] >= thr) atomicAdd(staged, 1u);
  const unsigned nb = (unsigned)R.bx * (unsigned)R.by * (unsigned)R.bz;
  for (unsigned long long gi = t0; gi < nb; gi += nt) {
    const unsigned g = R.grid[gi];
    if (g < 256u || g - 256u >= nslots || !(prob[g - 256u] >= thr)) continue;
    int x, y, z;
    if (!brick_origin(R, (unsigned)gi, x, y, z) || !in_dom(R, x, y, z) || !in_dom(R, x + 7, y + 7, z + 7)) continue;
    const unsigned* row = R.dense + dom_id(R, x, y, z);
    for (int lz = 0; lz < 8; ++lz)
      for (int ly = 0; ly < 8; ++ly) asm volatile("prefetch.global.L2 [%0];" ::"l"(row + (unsigned)((lz * R.PY + ly) * R.PX)));
  }
}

}  // namespace vfe
