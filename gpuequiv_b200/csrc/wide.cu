// wide.cu - the energy-game fixpoint for every EnergyConf outside the
// thermometer codecs of codec.cuh: energies of several words (e.g. {30, 3},
// two words), fields too wide for a thermometer code (ONE_DIMENSION =
// {1, u32::MAX}), updates of several words.
//
// Reference: the same path as engine.cu -- EnergyGame::run ->
// GPURunner::execute_gpu (src/energygame.rs:379-383, :1461-1523) with the
// arithmetic the shader preprocessor generates for any conf
// (src/energygame/shadergen.rs:55-157): IMPL_LESS_EQ / IMPL_EQ field-wise on
// the packed words, UPDATE1 (+1 in u32 arithmetic, then min with max),
// UPDATE_MIN (merges in index order), MAX_SUPREMUM.
//
// Layout: energies stay in the crate's packed form (energy_size words, a
// field never straddles a word since energy_bits is a power of two).  Every
// position's list is a slice of one energy arena (descriptor = first energy
// << 24 | count).  The rounds are the reference's Jacobi rounds: a round
// reads only committed lists and writes new lists to fresh arena space; the
// commit publishes them and marks the predecessors of changed positions for
// the next frontier (a bitmap turned into a list).
//
// One warp per frontier position.  A position's new list is built as an
// antichain: of energies of one, two or four words in shared memory, 32
// candidates (inverse-updated successor energies, suprema) at a time
// (insert32); of others, and beyond 256 members, in the warp's slice of a
// global scratch, where each candidate is tested against the members by the 32
// lanes at once and either dropped or inserted while the members it dominates
// are removed.  Field-wise <= and max run word by word
// with SWAR arithmetic (fields of 1-16 bits in guarded 2k-bit slots; 32-bit
// fields directly).  A position whose antichain outgrows its scratch is
// recorded and computed again in the same round with a larger scratch; a
// round whose results outgrow the arena is run again after the arena has
// been compacted and grown.  Either way only committed lists are read, so a
// repeated computation gives the same lists.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <chrono>
#include <cstring>

#include "geq_internal.h"
#include "wide_arith.cuh"

namespace geq {
namespace wide {

constexpr uint32_t ES_MAX = 64;   // words per energy
constexpr uint32_t US_MAX = 128;  // words per update
constexpr uint32_t WARPS = 4;
constexpr uint32_t BLOCK_T = 32 * WARPS;
constexpr unsigned long long NOCHANGE = ~0ull;
constexpr uint32_t CNT_BITS = 24;
constexpr unsigned long long CNT_MASK = (1ull << CNT_BITS) - 1ull;

struct Ctr {
  unsigned long long arena_top;  // energies in use
  unsigned long long rounds;     // completed by k_wide_rounds
  unsigned long long positions, edges, bytes;
  uint32_t next_slot;   // slots handed out to warps
  uint32_t n_ovf;       // slots whose antichain outgrew the warp scratch
  uint32_t arena_full;  // a new list found no arena space
  uint32_t next_size;   // size of the next frontier
  uint32_t flip;        // k_wide_rounds: 1 when `next` holds the frontier
  uint32_t pad;
};

struct P {
  const uint32_t *row, *col, *wt, *rrow, *rcol;
  const uint8_t *att;
  unsigned long long *desc;
  uint32_t *arena;
  unsigned long long arena_cap;  // energies
  const uint32_t *front;
  const uint32_t *slots;  // null: item i is slot i
  uint32_t n_items;
  unsigned long long *slot_new;
  uint32_t *ovf;
  uint32_t *scratch;
  unsigned long long scratch_words;  // per warp
  Ctr *ctr;
  uint32_t *mark, *next;
  uint32_t n_nodes, mwords;
  uint32_t n_warps;  // warps with a scratch slice (the others of the last block idle)
  uint32_t el, mx, eb, em, ub, um, es, us;
  Swar sw;
  WideConf wc;
};

// Inverse update of one energy in place (UPDATE1 then UPDATE_MIN); u = the
// edge's update words, null for the zero update of an attacker's own list.
__device__ __forceinline__ void inv_update(const P &p, uint32_t *x, const uint32_t *u) { wide_inv_update(p.wc, x, u); }
__device__ __forceinline__ bool leq_w(uint32_t a, uint32_t b, const Swar &s) { return swar_leq(a, b, s); }
__device__ __forceinline__ uint32_t max_w(uint32_t a, uint32_t b, const Swar &s) { return swar_max(a, b, s); }

// The warp's antichain: members in `ac` (es words each), an "own energy" flag
// per member in `fl` (attacker tie rule).
struct Ac {
  uint32_t *ac;
  uint8_t *fl;
  uint32_t n, cap;
};

// Insert candidate x (shared memory, es words): dropped when a member is <=
// x (an equal member takes x's own flag when x is own, as the later copy
// wins); else the members above x leave and x joins.  false: no room.
__device__ bool ac_insert(const P &p, Ac &a, const uint32_t *x, bool own, uint32_t lane) {
  const uint32_t es = p.es;
  bool dom = false, rm = false;
  int eqi = -1;
  for (uint32_t j = lane; j < a.n; j += 32) {
    const uint32_t *m = a.ac + (size_t)j * es;
    bool le = true, ge = true, eq = true;
    for (uint32_t w = 0; w < es && (le || ge); w++) {
      const uint32_t mv = m[w], xv = x[w];
      le = le && leq_w(mv, xv, p.sw);
      ge = ge && leq_w(xv, mv, p.sw);
      eq = eq && mv == xv;
    }
    if (le) {
      dom = true;
      if (eq) eqi = (int)j;
    } else if (ge) {
      rm = true;
    }
  }
  if (__any_sync(0xffffffffu, dom)) {
    if (own && eqi >= 0) a.fl[eqi] = 1;
    return true;
  }
  uint32_t n = a.n;
  if (__any_sync(0xffffffffu, rm)) {
    // remove the members above x, keeping the order (reads of a chunk's word
    // before its writes; destinations never pass their sources)
    uint32_t out = 0;
    for (uint32_t base = 0; base < a.n; base += 32) {
      const uint32_t j = base + lane;
      bool keep = false;
      if (j < a.n) {
        const uint32_t *m = a.ac + (size_t)j * es;
        bool ge = true;
        for (uint32_t w = 0; w < es && ge; w++) ge = leq_w(x[w], m[w], p.sw);
        keep = !ge;
      }
      const uint32_t bal = __ballot_sync(0xffffffffu, keep);
      const uint32_t dst = out + __popc(bal & ((1u << lane) - 1u));
      for (uint32_t w = 0; w < es; w++) {
        const uint32_t val = keep ? a.ac[(size_t)j * es + w] : 0u;
        __syncwarp();
        if (keep) a.ac[(size_t)dst * es + w] = val;
        __syncwarp();
      }
      const uint8_t f = keep ? a.fl[j] : 0;
      __syncwarp();
      if (keep) a.fl[dst] = f;
      __syncwarp();
      out += __popc(bal);
    }
    n = out;
  }
  if (n >= a.cap) return false;
  for (uint32_t w = lane; w < es; w += 32) a.ac[(size_t)n * es + w] = x[w];
  if (lane == 0) a.fl[n] = own ? 1 : 0;
  __syncwarp();
  a.n = n + 1;
  return true;
}

// Append x without a dominance test (a single-successor defender's list is
// its successor's updated list as is).
__device__ bool ac_append(const P &p, Ac &a, const uint32_t *x, uint32_t lane) {
  if (a.n >= a.cap) return false;
  for (uint32_t w = lane; w < p.es; w += 32) a.ac[(size_t)a.n * p.es + w] = x[w];
  if (lane == 0) a.fl[a.n] = 0;
  __syncwarp();
  a.n++;
  return true;
}

__device__ __forceinline__ uint32_t dcnt(unsigned long long d) { return (uint32_t)(d & CNT_MASK); }
__device__ __forceinline__ unsigned long long doff(unsigned long long d) { return d >> CNT_BITS; }

// shared memory of one warp: the update words, 32 staged energies, one candidate
__device__ __forceinline__ uint32_t *warp_smem(const P &p, uint32_t *base, uint32_t wib) {
  return base + (size_t)wib * (p.us + 33u * p.es);
}

// Stage energies [b0, b0+32) of list d, each inverse-updated by u (null: own
// list, clamped); returns how many were staged.
__device__ uint32_t stage(const P &p, uint32_t *stg, unsigned long long d, uint32_t b0, const uint32_t *u,
                          uint32_t lane) {
  const uint32_t cnt = dcnt(d), k = min(32u, cnt - b0);
  if (lane < k) {
    uint32_t *x = stg + (size_t)lane * p.es;
    const uint32_t *src = p.arena + (doff(d) + b0 + lane) * p.es;
    for (uint32_t w = 0; w < p.es; w++) x[w] = src[w];
    inv_update(p, x, u);
  }
  __syncwarp();
  return k;
}

__device__ void load_update(const P &p, uint32_t *ush, unsigned long long k, uint32_t lane) {
  __syncwarp();
  for (uint32_t w = lane; w < p.us; w += 32) ush[w] = p.wt[k * p.us + w];
  __syncwarp();
}

// One position; returns false when its antichain outgrew the scratch.
__device__ bool solve_one(const P &p, uint32_t slot, uint32_t *sm, uint32_t lane, unsigned long long &edges,
                          unsigned long long &bytes) {
  const uint32_t v = p.front[slot];
  const uint32_t e0 = p.row[v], e1 = p.row[v + 1], deg = e1 - e0;
  const bool attacker = p.att[v] != 0;
  uint32_t *ush = sm, *stg = sm + p.us, *xb = stg + 32u * p.es;
  uint32_t *ws = p.scratch + (size_t)(((blockIdx.x * BLOCK_T) + threadIdx.x) >> 5) * p.scratch_words;
  // scratch: two antichains of cap energies and their flags
  const unsigned long long cap_e = p.scratch_words / (2ull * p.es + 1ull);
  const uint32_t cap = (uint32_t)(cap_e < 0xFFFFFFull ? cap_e : 0xFFFFFFull);
  Ac A{ws, (uint8_t *)(ws + 2ull * cap * p.es), 0, cap};
  Ac B{ws + (size_t)cap * p.es, A.fl + cap, 0, cap};
  const unsigned long long esb = 4ull * p.es;
  if (attacker) {
    for (uint32_t k = e0; k < e1; k++) {
      const unsigned long long d = p.desc[p.col[k]];
      bytes += 16 + esb * dcnt(d);
      load_update(p, ush, k, lane);
      for (uint32_t b0 = 0; b0 < dcnt(d); b0 += 32) {
        const uint32_t n = stage(p, stg, d, b0, ush, lane);
        for (uint32_t t = 0; t < n; t++)
          if (!ac_insert(p, A, stg + (size_t)t * p.es, false, lane)) return false;
        __syncwarp();
      }
    }
    edges += deg;
    const unsigned long long dv = p.desc[v];
    bytes += 12 + esb * dcnt(dv);
    for (uint32_t b0 = 0; b0 < dcnt(dv); b0 += 32) {
      const uint32_t n = stage(p, stg, dv, b0, nullptr, lane);
      for (uint32_t t = 0; t < n; t++)
        if (!ac_insert(p, A, stg + (size_t)t * p.es, true, lane)) return false;
      __syncwarp();
    }
    // changed iff a kept energy came from a successor (attack_minimize.wgsl:95-101)
    bool from_succ = false;
    for (uint32_t j = lane; j < A.n; j += 32) from_succ |= A.fl[j] == 0;
    if (!__any_sync(0xffffffffu, from_succ)) {
      if (lane == 0) p.slot_new[slot] = NOCHANGE;
      return true;
    }
  } else {
    // defenders wait until every successor has a list (energygame.rs:789-792)
    bool empty = false;
    for (uint32_t k = e0 + lane; k < e1; k += 32) empty |= dcnt(p.desc[p.col[k]]) == 0;
    if (deg == 0 || __any_sync(0xffffffffu, empty)) {
      if (lane == 0) p.slot_new[slot] = NOCHANGE;
      return true;
    }
    edges += deg;
    bytes += 12;
    {
      const unsigned long long d = p.desc[p.col[e0]];
      bytes += 16 + esb * dcnt(d);
      load_update(p, ush, e0, lane);
      for (uint32_t b0 = 0; b0 < dcnt(d); b0 += 32) {
        const uint32_t n = stage(p, stg, d, b0, ush, lane);
        for (uint32_t t = 0; t < n; t++) {
          const uint32_t *x = stg + (size_t)t * p.es;
          if (!(deg == 1 ? ac_append(p, A, x, lane) : ac_insert(p, A, x, false, lane))) return false;
        }
        __syncwarp();
      }
    }
    // fold: minimal elements of the pairwise suprema, successor by successor
    for (uint32_t k = e0 + 1; k < e1; k++) {
      const unsigned long long d = p.desc[p.col[k]];
      bytes += 16 + esb * dcnt(d);
      load_update(p, ush, k, lane);
      B.n = 0;
      for (uint32_t b0 = 0; b0 < dcnt(d); b0 += 32) {
        const uint32_t n = stage(p, stg, d, b0, ush, lane);
        for (uint32_t t = 0; t < n; t++) {
          const uint32_t *y = stg + (size_t)t * p.es;
          for (uint32_t i = 0; i < A.n; i++) {
            const uint32_t *a = A.ac + (size_t)i * p.es;
            for (uint32_t w = lane; w < p.es; w += 32) xb[w] = max_w(a[w], y[w], p.sw);
            __syncwarp();
            if (!ac_insert(p, B, xb, false, lane)) return false;
            __syncwarp();
          }
        }
        __syncwarp();
      }
      Ac t = A;
      A = B;
      B = t;
    }
    // changed iff the list differs from the old one (EnergyArray ==,
    // energy.rs:334-350: same length and every new energy in the old list)
    const unsigned long long dv = p.desc[v];
    bool same = dcnt(dv) == A.n;
    if (same) {
      bool miss = false;
      for (uint32_t j = lane; j < A.n; j += 32) {
        const uint32_t *x = A.ac + (size_t)j * p.es;
        bool found = false;
        for (uint32_t q = 0; q < dcnt(dv) && !found; q++) {
          const uint32_t *o = p.arena + (doff(dv) + q) * p.es;
          bool eq = true;
          for (uint32_t w = 0; w < p.es && eq; w++) eq = o[w] == x[w];
          found = eq;
        }
        miss |= !found;
      }
      same = !__any_sync(0xffffffffu, miss);
    }
    if (same) {
      if (lane == 0) p.slot_new[slot] = NOCHANGE;
      return true;
    }
  }
  // the new list into fresh arena space
  unsigned long long off = 0;
  if (lane == 0) off = atomicAdd(&p.ctr->arena_top, (unsigned long long)A.n);
  off = __shfl_sync(0xffffffffu, off, 0);
  if (off + A.n > p.arena_cap) {
    if (lane == 0) {
      atomicExch(&p.ctr->arena_full, 1u);
      p.slot_new[slot] = NOCHANGE;
    }
    return true;
  }
  for (size_t w = lane; w < (size_t)A.n * p.es; w += 32) p.arena[off * p.es + w] = A.ac[w];
  bytes += esb * A.n;
  if (lane == 0) p.slot_new[slot] = (off << CNT_BITS) | A.n;
  return true;
}

__global__ void __launch_bounds__(BLOCK_T) k_wide_round(const P p) {
  extern __shared__ uint32_t smem[];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  if (blockIdx.x * WARPS + wib >= p.n_warps) return;
  uint32_t *sm = warp_smem(p, smem, wib);
  unsigned long long edges = 0, bytes = 0, pos = 0;
  for (;;) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(&p.ctr->next_slot, 1u);
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= p.n_items) break;
    const uint32_t slot = p.slots ? p.slots[i] : i;
    if (!solve_one(p, slot, sm, lane, edges, bytes)) {
      if (lane == 0) p.ovf[atomicAdd(&p.ctr->n_ovf, 1u)] = slot;
    } else {
      pos++;
    }
    __syncwarp();
  }
  if (lane == 0) {
    atomicAdd(&p.ctr->positions, pos);
    atomicAdd(&p.ctr->edges, edges);
    atomicAdd(&p.ctr->bytes, bytes);
  }
}

// ---- energies of one, two or four words: antichains in shared memory ----------
// A candidate at a time against an antichain in global memory is a chain of a
// few hundred cycles per candidate, with one lane busy while a list of one
// energy is updated.  Here 32 candidates, taken across the successors' lists,
// are updated by one lane each and inserted together: every lane compares its
// candidate with all members (broadcast reads of shared memory), the ones left
// meet one another by shuffles.  What remains, and its order, is what inserting
// them in turn leaves: the members without a candidate below them, then the
// candidates without a member at or below, a strictly smaller candidate or an
// equal earlier one.  An antichain beyond SCAP members is left to k_wide_round
// (Ctr::n_ovf).
constexpr uint32_t SCAP = 256;
template <int ES>
struct SWarp {
  uint32_t A[SCAP * ES], B[SCAP * ES];  // members
  uint32_t Y[32 * ES];                  // a chunk of updated energies
  uint32_t Q[64 * ES];                  // suprema that wait to be inserted
  uint32_t inc[32];
  uint8_t fl[SCAP];                     // own energy (attacker tie rule)
};

template <int ES>
__device__ __forceinline__ bool leq_es(const uint32_t (&a)[ES], const uint32_t (&b)[ES], const Swar &sw) {
  bool r = true;
#pragma unroll
  for (int w = 0; w < ES; w++) r = r && leq_w(a[w], b[w], sw);
  return r;
}
template <int ES>
__device__ __forceinline__ bool eq_es(const uint32_t (&a)[ES], const uint32_t (&b)[ES]) {
  bool r = true;
#pragma unroll
  for (int w = 0; w < ES; w++) r = r && a[w] == b[w];
  return r;
}

// Insert the lanes' candidates (valid ones, in lane order) into the n members
// at M.  false: no room.
template <int ES>
__device__ __forceinline__ bool insert32(const P &p, uint32_t *M, uint8_t *fl, uint32_t &n, const uint32_t (&x)[ES],
                                         bool valid, bool own, uint32_t lane) {
  constexpr uint32_t FULL = 0xffffffffu;
  // Most candidates lie above a member: that is looked for first, four members
  // at a time until every lane has one; only the candidates left are compared
  // the other way, each with 32 members at once.
  bool dom = !valid;
  for (uint32_t m0 = 0; m0 < n && !__all_sync(FULL, dom); m0 += 4u) {
#pragma unroll
    for (uint32_t k = 0; k < 4u; k++) {
      const uint32_t m = min(m0 + k, n - 1u);
      uint32_t mv[ES];
#pragma unroll
      for (int w = 0; w < ES; w++) mv[w] = M[m * ES + w];
      if (leq_es<ES>(mv, x, p.sw)) {
        dom = true;
        if (own && valid && eq_es<ES>(mv, x)) fl[m] = 1;
      }
    }
  }
  bool live = !dom;
  uint32_t lm = __ballot_sync(FULL, live);
  for (uint32_t r = lm; r; r &= r - 1u) {
    const uint32_t j = (uint32_t)__ffs((int)r) - 1u;
    uint32_t xj[ES];
#pragma unroll
    for (int w = 0; w < ES; w++) xj[w] = __shfl_sync(FULL, x[w], j);
    if (j != lane && leq_es<ES>(xj, x, p.sw) && (j < lane || !eq_es<ES>(xj, x))) live = false;
  }
  lm = __ballot_sync(FULL, live);
  __syncwarp();  // flags set above are read by other lanes; ballots order no memory
  if (!lm) return true;
  uint32_t rm = 0;  // bit k: member 32k + lane leaves
  for (uint32_t r = lm; r; r &= r - 1u) {
    const uint32_t j = (uint32_t)__ffs((int)r) - 1u;
    uint32_t xj[ES];
#pragma unroll
    for (int w = 0; w < ES; w++) xj[w] = __shfl_sync(FULL, x[w], j);
    for (uint32_t m = lane; m < n; m += 32u) {
      uint32_t mv[ES];
#pragma unroll
      for (int w = 0; w < ES; w++) mv[w] = M[m * ES + w];
      if (leq_es<ES>(xj, mv, p.sw)) rm |= 1u << (m >> 5);
    }
  }
  const bool any_rm = __any_sync(FULL, rm != 0u);
  __syncwarp();
  if (any_rm) {
    uint32_t out = 0;
    for (uint32_t b0 = 0; b0 < n; b0 += 32u) {
      const uint32_t m = b0 + lane;
      const bool keep = m < n && !((rm >> (b0 >> 5)) & 1u);
      uint32_t mv[ES];
      uint8_t f = 0;
      if (keep) {
#pragma unroll
        for (int w = 0; w < ES; w++) mv[w] = M[m * ES + w];
        f = fl[m];
      }
      const uint32_t bal = __ballot_sync(FULL, keep);
      __syncwarp();
      if (keep) {
        const uint32_t d = out + (uint32_t)__popc(bal & ((1u << lane) - 1u));
#pragma unroll
        for (int w = 0; w < ES; w++) M[d * ES + w] = mv[w];
        fl[d] = f;
      }
      __syncwarp();
      out += (uint32_t)__popc(bal);
    }
    n = out;
  }
  const uint32_t bal = __ballot_sync(FULL, live);
  const uint32_t k = (uint32_t)__popc(bal);
  if (n + k > SCAP) return false;
  if (live) {
    const uint32_t d = n + (uint32_t)__popc(bal & ((1u << lane) - 1u));
#pragma unroll
    for (int w = 0; w < ES; w++) M[d * ES + w] = x[w];
    fl[d] = own ? 1 : 0;
  }
  n += k;
  __syncwarp();
  return true;
}

// solve_one with the antichains in shared memory.
template <int ES>
__device__ bool solve_es(const P &p, uint32_t slot, SWarp<ES> &s, uint32_t lane, unsigned long long &edges,
                         unsigned long long &bytes) {
  constexpr uint32_t FULL = 0xffffffffu;
  const uint32_t v = p.front[slot];
  const uint32_t e0 = p.row[v], e1 = p.row[v + 1], deg = e1 - e0;
  const bool attacker = p.att[v] != 0;
  const unsigned long long dv = p.desc[v];
  constexpr unsigned long long esb = 4ull * ES;
  uint32_t *A = s.A, *B = s.B;
  uint32_t n = 0;
  if (!attacker) {
    // defenders wait until every successor has a list (energygame.rs:789-792)
    bool empty = false;
    for (uint32_t k = e0 + lane; k < e1; k += 32) empty |= dcnt(p.desc[p.col[k]]) == 0;
    if (deg == 0 || __any_sync(FULL, empty)) {
      if (lane == 0) p.slot_new[slot] = NOCHANGE;
      return true;
    }
  }
  unsigned long long by = 12ull + 16ull * deg;
  auto fetch = [&](unsigned long long d, uint32_t q, const uint32_t *u, uint32_t (&x)[ES]) {
    const uint32_t *src = p.arena + (doff(d) + q) * ES;
#pragma unroll
    for (int w = 0; w < ES; w++) x[w] = src[w];
    wide_inv_update(p.wc, x, u);
  };
  if (attacker) {
    for (uint32_t k0 = e0; k0 < e1; k0 += 32u) {
      const uint32_t k = k0 + lane;
      const unsigned long long d = k < e1 ? p.desc[p.col[k]] : 0ull;
      const uint32_t c = k < e1 ? dcnt(d) : 0u;
      uint32_t inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, inc, o);
        if (lane >= (uint32_t)o) inc += y;
      }
      const uint32_t total = __shfl_sync(FULL, inc, 31);
      by += esb * total;
      __syncwarp();
      s.inc[lane] = inc;
      __syncwarp();
      for (uint32_t t0 = 0; t0 < total; t0 += 32u) {
        const uint32_t t = t0 + lane;
        const bool valid = t < total;
        uint32_t lo = 0;  // the successor whose range holds candidate t
        if (valid) {
          uint32_t hi = 31;
          while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (s.inc[mid] > t) hi = mid;
            else lo = mid + 1;
          }
        }
        const unsigned long long dk = __shfl_sync(FULL, d, lo);
        uint32_t x[ES] = {};
        if (valid) fetch(dk, t - (lo ? s.inc[lo - 1] : 0u), p.wt + (unsigned long long)(k0 + lo) * p.us, x);
        if (!insert32<ES>(p, A, s.fl, n, x, valid, false, lane)) return false;
      }
    }
    by += esb * dcnt(dv);
    for (uint32_t q0 = 0; q0 < dcnt(dv); q0 += 32u) {
      const bool valid = q0 + lane < dcnt(dv);
      uint32_t x[ES] = {};
      if (valid) fetch(dv, q0 + lane, nullptr, x);
      if (!insert32<ES>(p, A, s.fl, n, x, valid, true, lane)) return false;
    }
    edges += deg;
    // changed iff a kept energy came from a successor (attack_minimize.wgsl:95-101)
    bool from_succ = false;
    for (uint32_t j = lane; j < n; j += 32) from_succ |= s.fl[j] == 0;
    if (!__any_sync(FULL, from_succ)) {
      if (lane == 0) p.slot_new[slot] = NOCHANGE;
      bytes += by;
      return true;
    }
  } else {
    for (uint32_t k = e0; k < e1; k++) {
      const unsigned long long d = p.desc[p.col[k]];
      const uint32_t *u = p.wt + (unsigned long long)k * p.us;
      by += esb * dcnt(d);
      uint32_t nb = 0, nq = 0;
      auto drain = [&](uint32_t c) {  // the first c waiting suprema go in
        __syncwarp();
        uint32_t z[ES] = {}, r[ES] = {};
#pragma unroll
        for (int w = 0; w < ES; w++) {
          if (lane < c) z[w] = s.Q[lane * ES + w];
          if (lane + c < nq) r[w] = s.Q[(lane + c) * ES + w];
        }
        __syncwarp();
        if (lane + c < nq) {
#pragma unroll
          for (int w = 0; w < ES; w++) s.Q[lane * ES + w] = r[w];
        }
        nq -= c;
        return insert32<ES>(p, B, s.fl, nb, z, lane < c, false, lane);
      };
      for (uint32_t q0 = 0; q0 < dcnt(d); q0 += 32u) {
        const uint32_t ny = min(32u, dcnt(d) - q0);
        uint32_t x[ES] = {};
        if (lane < ny) fetch(d, q0 + lane, u, x);
        if (k == e0) {
          // a single successor's updated list as is, else the first list minimised
          if (deg == 1u) {
            if (n + ny > SCAP) return false;
            if (lane < ny) {
#pragma unroll
              for (int w = 0; w < ES; w++) A[(n + lane) * ES + w] = x[w];
            }
            n += ny;
            __syncwarp();
          } else if (!insert32<ES>(p, A, s.fl, n, x, lane < ny, false, lane)) {
            return false;
          }
          continue;
        }
        // minimal elements of the pairwise suprema, in the order (energy, member)
        if (lane < ny) {
#pragma unroll
          for (int w = 0; w < ES; w++) s.Y[lane * ES + w] = x[w];
        }
        __syncwarp();
        if (ny * n == 1u) {  // nothing to leave out
          if (nq && !drain(nq)) return false;
          uint32_t z[ES];
#pragma unroll
          for (int w = 0; w < ES; w++) z[w] = max_w(A[w], s.Y[w], p.sw);
          if (!insert32<ES>(p, B, s.fl, nb, z, lane == 0, false, lane)) return false;
          continue;
        }
        // Where a member lies at or below y, y itself is a supremum and every
        // other one with y lies above it; likewise where an energy of this
        // chunk lies at or below a member.  Only what is left is inserted:
        // conf {30, 3}, 12,000 positions 8.1 -> 6.3 ms, {16, 7}, 20,000 positions
        // 4.2 -> 3.5 ms on one B200.
        bool hy = lane >= ny;
        uint32_t ha = 0;  // bit j: member 32j + lane
        for (uint32_t m = 0; m < n && !__all_sync(FULL, hy); m++) {
          uint32_t mv[ES];
#pragma unroll
          for (int w = 0; w < ES; w++) mv[w] = A[m * ES + w];
          hy = hy || leq_es<ES>(mv, x, p.sw);
        }
        const uint32_t hits = __ballot_sync(FULL, hy);
        for (uint32_t m = lane; m < n; m += 32u) {
          uint32_t mv[ES], yv[ES];
#pragma unroll
          for (int w = 0; w < ES; w++) mv[w] = A[m * ES + w];
          bool h = false;
          for (uint32_t q = 0; q < ny && !h; q++) {
#pragma unroll
            for (int w = 0; w < ES; w++) yv[w] = s.Y[q * ES + w];
            h = leq_es<ES>(yv, mv, p.sw);
          }
          if (h) ha |= 1u << (m >> 5);
        }
        __syncwarp();
        uint32_t yq = lane / n, am = lane - yq * n;
        for (uint32_t i0 = 0; i0 < ny * n; i0 += 32u) {
          const bool valid = i0 + lane < ny * n;
          const uint32_t hm = __shfl_sync(FULL, ha, am & 31u);
          bool keep = valid;
          uint32_t z[ES] = {};
          if (valid) {
            bool ey = true, ea = true;  // the supremum is y, is the member
#pragma unroll
            for (int w = 0; w < ES; w++) {
              const uint32_t av = A[am * ES + w], yv = s.Y[yq * ES + w];
              z[w] = max_w(av, yv, p.sw);
              ey = ey && z[w] == yv;
              ea = ea && z[w] == av;
            }
            keep = (ey || !((hits >> yq) & 1u)) && (ea || !((hm >> (am >> 5)) & 1u));
          }
          const uint32_t bal = __ballot_sync(FULL, keep);
          if (keep) {
            const uint32_t d = nq + (uint32_t)__popc(bal & ((1u << lane) - 1u));
#pragma unroll
            for (int w = 0; w < ES; w++) s.Q[d * ES + w] = z[w];
          }
          nq += (uint32_t)__popc(bal);
          if (nq >= 32u && !drain(32u)) return false;
          for (am += 32u; am >= n; am -= n) yq++;
        }
        __syncwarp();
      }
      if (k != e0) {
        if (nq && !drain(nq)) return false;
        uint32_t *t = A;
        A = B;
        B = t;
        n = nb;
      }
    }
    edges += deg;
    // changed iff the list differs from the old one (EnergyArray ==,
    // energy.rs:334-350: same length and every new energy in the old list)
    bool same = dcnt(dv) == n;
    if (same) {
      bool miss = false;
      for (uint32_t j = lane; j < n; j += 32) {
        bool found = false;
        for (uint32_t q = 0; q < n && !found; q++) {
          const uint32_t *o = p.arena + (doff(dv) + q) * ES;
          bool eq = true;
#pragma unroll
          for (int w = 0; w < ES; w++) eq = eq && o[w] == A[j * ES + w];
          found = eq;
        }
        miss |= !found;
      }
      same = !__any_sync(FULL, miss);
    }
    if (same) {
      if (lane == 0) p.slot_new[slot] = NOCHANGE;
      bytes += by;
      return true;
    }
  }
  unsigned long long off = 0;
  if (lane == 0) off = atomicAdd(&p.ctr->arena_top, (unsigned long long)n);
  off = __shfl_sync(FULL, off, 0);
  bytes += by;
  if (off + n > p.arena_cap) {
    if (lane == 0) {
      atomicExch(&p.ctr->arena_full, 1u);
      p.slot_new[slot] = NOCHANGE;
    }
    return true;
  }
  for (uint32_t w = lane; w < n * ES; w += 32) p.arena[off * ES + w] = A[w];
  bytes += esb * n;
  if (lane == 0) p.slot_new[slot] = (off << CNT_BITS) | n;
  __syncwarp();
  return true;
}

// A round by all warps of the device (the first attempt at every slot).
template <int ES>
__global__ void __launch_bounds__(BLOCK_T) k_wide_round_es(const P p) {
  __shared__ SWarp<ES> sw[WARPS];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  unsigned long long edges = 0, bytes = 0, pos = 0;
  for (;;) {
    uint32_t i = 0;
    if (lane == 0) i = atomicAdd(&p.ctr->next_slot, 1u);
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= p.n_items) break;
    if (!solve_es<ES>(p, i, sw[wib], lane, edges, bytes)) {
      if (lane == 0) p.ovf[atomicAdd(&p.ctr->n_ovf, 1u)] = i;
    } else {
      pos++;
    }
    __syncwarp();
  }
  if (lane == 0 && pos) {
    atomicAdd(&p.ctr->positions, pos);
    atomicAdd(&p.ctr->edges, edges);
    atomicAdd(&p.ctr->bytes, bytes);
  }
}

// Rounds inside one launch, four barriers a round in place of three launches,
// four fills, two read-backs and the waits for them: of a cluster of blocks
// (GRID = false) for small games, whose rounds are shorter than a barrier of
// the whole device, else of a block per SM (a cooperative launch).  Leaves
// before the commit of a round that met a full arena or antichains beyond SCAP
// members, for the host to finish that round.
constexpr uint32_t CWARPS = 16, CTHREADS = 32 * CWARPS;
template <int ES, bool GRID>
__global__ void __launch_bounds__(CTHREADS, 1) k_wide_rounds(P p, uint32_t fs, uint32_t max_rounds) {
  extern __shared__ __align__(16) unsigned char dsm[];
  const uint32_t rank = blockIdx.x, blocks = gridDim.x;  // one cluster, or the grid
  auto sync = [] {
    if constexpr (GRID) cooperative_groups::this_grid().sync();
    else cooperative_groups::this_cluster().sync();
  };
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  SWarp<ES> &s = ((SWarp<ES> *)dsm)[warp];
  const uint32_t gw = warp * blocks + rank, warps = blocks * CWARPS;
  const uint32_t tid = gw * 32u + lane, threads = warps * 32u;
  Ctr *c = p.ctr;
  unsigned long long edges = 0, bytes = 0, pos = 0;
  uint32_t *front = const_cast<uint32_t *>(p.front), *next = p.next;
  uint32_t rounds = 0, flip = 0;
  bool stop = false;
  while (fs && rounds < max_rounds) {
    p.front = front;
    // the fuller warps of a round are not known beforehand: slots by a counter
    for (;;) {
      uint32_t i = 0;
      if (lane == 0) i = atomicAdd(&c->next_slot, 1u);
      i = __shfl_sync(0xffffffffu, i, 0);
      if (i >= fs) break;
      if (!solve_es<ES>(p, i, s, lane, edges, bytes)) {
        if (lane == 0) p.ovf[atomicAdd(&c->n_ovf, 1u)] = i;
      } else {
        pos++;
      }
      __syncwarp();
    }
    sync();
    stop = *(volatile uint32_t *)&c->n_ovf != 0u || *(volatile uint32_t *)&c->arena_full != 0u;
    if (stop) break;
    for (uint32_t k = tid; k < fs; k += threads) {
      const unsigned long long d = p.slot_new[k];
      if (d == NOCHANGE) continue;
      const uint32_t v = front[k];
      p.desc[v] = d;
      for (uint32_t e = p.rrow[v]; e < p.rrow[v + 1]; e++) {
        const uint32_t u = p.rcol[e];
        atomicOr(&p.mark[u >> 5], 1u << (u & 31u));
      }
    }
    if (rank == 0 && threadIdx.x == 0) {
      c->next_slot = 0u;
      c->next_size = 0u;
    }
    sync();
    for (uint32_t w = tid; w < p.mwords; w += threads) {
      uint32_t b = p.mark[w];
      if (!b) continue;
      p.mark[w] = 0u;
      uint32_t at = atomicAdd(&c->next_size, (uint32_t)__popc(b));
      for (; b; b &= b - 1u) next[at++] = w * 32u + (uint32_t)__ffs((int)b) - 1u;
    }
    sync();
    fs = *(volatile uint32_t *)&c->next_size;
    uint32_t *t = front;
    front = next;
    next = t;
    flip ^= 1u;
    rounds++;
    sync();  // everyone has read the size
  }
  if (lane == 0 && pos) {
    atomicAdd(&c->positions, pos);
    atomicAdd(&c->edges, edges);
    atomicAdd(&c->bytes, bytes);
  }
  if (rank == 0 && threadIdx.x == 0) {
    c->rounds = c->rounds + rounds;
    c->next_size = fs;
    c->flip = flip;
  }
  sync();
}

// publish the round's lists and mark the predecessors of changed positions
__global__ void k_wide_commit(const P p, uint32_t n_slots) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n_slots) return;
  const unsigned long long d = p.slot_new[s];
  if (d == NOCHANGE) return;
  const uint32_t v = p.front[s];
  p.desc[v] = d;
  for (uint32_t k = p.rrow[v]; k < p.rrow[v + 1]; k++) {
    const uint32_t u = p.rcol[k];
    atomicOr(&p.mark[u >> 5], 1u << (u & 31u));
  }
}

// the next frontier from the bitmap (clears it)
__global__ void k_wide_fill(const P p) {
  const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= p.mwords) return;
  uint32_t b = p.mark[w];
  if (!b) return;
  p.mark[w] = 0;
  uint32_t at = atomicAdd(&p.ctr->next_size, (uint32_t)__popc(b));
  while (b) {
    const uint32_t i = (uint32_t)__ffs((int)b) - 1u;
    b &= b - 1u;
    p.next[at++] = w * 32u + i;
  }
}

// initial visit lists: predecessors of the to_reach positions (energygame.rs:1461-1465)
__global__ void k_wide_mark_reach(const P p, const uint32_t *reach, uint32_t n_reach) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_reach) return;
  const uint32_t v = reach[i];
  for (uint32_t k = p.rrow[v]; k < p.rrow[v + 1]; k++) {
    const uint32_t u = p.rcol[k];
    atomicOr(&p.mark[u >> 5], 1u << (u & 31u));
  }
}

// arena compaction: every position's list copied to its new place
__global__ void k_wide_move(const unsigned long long *desc, const unsigned long long *noff, uint32_t n,
                            const uint32_t *src, uint32_t *dst, uint32_t es) {
  const uint32_t v = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  if (v >= n) return;
  const unsigned long long d = desc[v];
  const size_t words = (size_t)dcnt(d) * es;
  for (size_t w = lane; w < words; w += 32) dst[noff[v] * es + w] = src[doff(d) * es + w];
}

__global__ void k_wide_redesc(unsigned long long *desc, const unsigned long long *noff, uint32_t n) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < n) desc[v] = (noff[v] << CNT_BITS) | dcnt(desc[v]);
}

// ---- host side ----------------------------------------------------------------
#define WCU(x)                                                                          \
  do {                                                                                  \
    const cudaError_t e_ = (x);                                                         \
    if (e_ != cudaSuccess) return fail(e_ == cudaErrorMemoryAllocation ? GEQ_ERR_OUT_OF_MEMORY : GEQ_ERR_CUDA, \
                                       "%s: %s", #x, cudaGetErrorString(e_));           \
  } while (0)

// Device buffers of one solve (all work is on the engine's stream).  Blocks up
// to POOL_MAX come from the engine's pool: the device's stream-ordered pool gives
// its memory back at every wait unless told otherwise, which for a solve's 18
// buffers cost 10 to 60 ms.  Larger ones -- arenas of big games, the warps'
// scratch of up to 4 GB -- come from that pool and go back to the device when
// the solve ends.  (A line of 32 MB instead: games that use the smallest
// scratch, 155 MB, 11.5 -> 14.1 ms.)
struct Bufs {
  static constexpr size_t POOL_MAX = 256u << 20;
  struct Block {
    void *p;
    size_t bytes;
    bool pooled;
  };
  Engine &eng;
  std::vector<Block> blocks;
  cudaStream_t stream() const { return (cudaStream_t)eng.stream_handle(); }
  template <class T>
  geq_status get(T *&p, size_t n) {
    Block b{nullptr, std::max<size_t>(n, 1) * sizeof(T), false};
    b.pooled = b.bytes <= POOL_MAX;
    if (!b.pooled && cudaMallocAsync(&b.p, b.bytes, stream()) != cudaSuccess) {
      cudaGetLastError();
      b.p = nullptr;
      b.pooled = true;  // the engine's pool gives up its idle blocks first
    }
    if (b.pooled) b.p = eng.pool_get(b.bytes);
    if (!b.p) return fail(GEQ_ERR_OUT_OF_MEMORY, "device allocation of %zu bytes for the wide solver failed", b.bytes);
    blocks.push_back(b);
    p = (T *)b.p;
    return GEQ_OK;
  }
  void give(const Block &b) {
    if (b.pooled) eng.pool_put(b.p, b.bytes);
    else cudaFreeAsync(b.p, stream());
  }
  void put(void *q) {
    for (size_t i = 0; i < blocks.size(); i++)
      if (blocks[i].p == q) {
        give(blocks[i]);
        blocks.erase(blocks.begin() + i);
        return;
      }
  }
  ~Bufs() {
    cudaStreamSynchronize(stream());  // error paths leave work behind
    for (auto &b : blocks) give(b);
  }
};

// The cluster kernels on the current device: blocks per cluster, 0: none.
template <int ES>
static uint32_t cluster_setup_es() {
  const size_t smem = sizeof(SWarp<ES>) * CWARPS;
  if (cudaFuncSetAttribute(k_wide_rounds<ES, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaFuncSetAttribute(k_wide_rounds<ES, false>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (uint32_t b = 16; b >= 8; b /= 2) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(b);
    cfg.blockDim = dim3(CTHREADS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = b;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_wide_rounds<ES, false>, &cfg) == cudaSuccess && n > 0) return b;
    cudaGetLastError();
  }
  return 0;
}
static uint32_t cluster_blocks(Engine &eng, uint32_t es) {
  if (es != 1 && es != 2 && es != 4) return 0;
  if (eng.wide_cluster < 0)
    eng.wide_cluster = (int)std::min({cluster_setup_es<1>(), cluster_setup_es<2>(), cluster_setup_es<4>()});
  return (uint32_t)eng.wide_cluster;
}
template <int ES>
static cudaError_t launch_cluster_es(const P &p, uint32_t blocks, uint32_t fs, uint32_t max_rounds, cudaStream_t S) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(CTHREADS);
  cfg.dynamicSmemBytes = sizeof(SWarp<ES>) * CWARPS;
  cfg.stream = S;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = blocks;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_wide_rounds<ES, false>, p, fs, max_rounds);
}
// The same over the whole device: blocks of a cooperative launch, 0: none.
template <int ES>
static uint32_t grid_setup_es(int device) {
  const size_t smem = sizeof(SWarp<ES>) * CWARPS;
  int sms = 0, coop = 0, per = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess || !coop ||
      cudaFuncSetAttribute(k_wide_rounds<ES, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
          cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_wide_rounds<ES, true>, CTHREADS, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return per > 0 ? (uint32_t)sms : 0u;
}
static uint32_t grid_blocks(Engine &eng, int device, uint32_t es) {
  if (es != 1 && es != 2 && es != 4) return 0;
  if (eng.wide_grid < 0)
    eng.wide_grid = (int)std::min({grid_setup_es<1>(device), grid_setup_es<2>(device), grid_setup_es<4>(device)});
  return (uint32_t)eng.wide_grid;
}
template <int ES>
static cudaError_t launch_rounds_es(P p, bool grid, uint32_t blocks, uint32_t fs, uint32_t max_rounds,
                                    cudaStream_t S) {
  if (!grid) return launch_cluster_es<ES>(p, blocks, fs, max_rounds, S);
  void *args[3] = {&p, &fs, &max_rounds};
  return cudaLaunchCooperativeKernel((void *)k_wide_rounds<ES, true>, dim3(blocks), dim3(CTHREADS), args,
                                     sizeof(SWarp<ES>) * CWARPS, S);
}
// Games of up to so many positions run their rounds in launches of one cluster,
// of up to so many in cooperative launches.  Median per call on one B200, all
// rounds in cluster launches / in cooperative ones:
//   conf {30, 3}, 300 / 2,000 / 4,000 / 12,000 positions
//     0.42 / 4.15 / 2.15 / 6.30 ms against 0.50 / 4.30 / 2.25 / 6.09;
//   {16, 7}, 2,000 / 20,000 positions 1.37 / 3.41 against 1.47 / 2.88 ms;
//   {1, u32::MAX}, 2,000 / 20,000 positions 0.60 / 1.75 against 0.70 / 1.58 ms.
// Rounds as kernels with read-backs against cooperative launches: {16, 7},
// 100,000 positions 10.2-10.9 against 8.4 ms, {1, u32::MAX}, 150,000 positions
// 8.5 against 7.1 ms.  Warps per block: 8, 16 and 24 warps of a cluster took
// 8.6, 8.1 and 8.6 ms for the 12,000 positions (when every supremum was
// inserted).
constexpr uint32_t WIDE_CLUSTER_POSITIONS = 8192, WIDE_GRID_POSITIONS = 262144;
constexpr uint32_t WIDE_CLUSTER_ROUNDS = 256;  // per launch

static geq_status check_game(const GameInput &gi, const Conf &c) {
  const geq_game_graph &g = gi.g;
  const uint32_t n = g.n_vertices, us = c.update_size(), ub = c.update_bits(), um = c.update_mask();
  const uint64_t m = g.row_offsets[n];
  for (uint32_t v = 0; v < n; v++)
    if (g.row_offsets[v + 1] < g.row_offsets[v]) return fail(GEQ_ERR_INVALID_INPUT, "row_offsets not monotone at %u", v);
  for (uint64_t k = 0; k < m; k++)
    if (g.column_indices[k] >= n) return fail(GEQ_ERR_INVALID_INPUT, "Node index too high: successor %u of %u positions",
                                              g.column_indices[k], n);
  // update codes: 0 Zero, 1 Decrement, k+2 Min into element k < elements;
  // bits past the last field are padding and must be clear
  const uint64_t fields_bits = (uint64_t)ub * c.elements;
  for (uint64_t k = 0; k < m; k++) {
    const uint32_t *u = g.weights + k * us;
    uint32_t any = 0;
    for (uint32_t w = 0; w < us; w++) any |= u[w];
    if (!any) continue;
    for (uint32_t i = 0; i < c.elements; i++) {
      const uint32_t bit = i * ub, code = (u[bit >> 5] >> (bit & 31u)) & um;
      if (code >= 2 && code - 2 >= c.elements)
        return fail(GEQ_ERR_INVALID_INPUT, "edge %llu: update code %u names no element", (unsigned long long)k, code);
    }
    if (fields_bits % 32) {
      const uint32_t pad = ~0u << (fields_bits % 32);
      if (u[us - 1] & pad) return fail(GEQ_ERR_INVALID_INPUT, "edge %llu: update padding bits set", (unsigned long long)k);
    }
  }
  return GEQ_OK;
}

// One game on the engine's stream.
static geq_status solve_one_game(Engine &eng, int device, const GameInput &gi, const Conf &c, geq_solution &sol,
                                 uint32_t g_index) {
  cudaStream_t S = (cudaStream_t)eng.stream_handle();
  const int n_sms = eng.n_sms;
  const geq_game_graph &g = gi.g;
  const uint32_t n = g.n_vertices, es = c.energy_size(), us = c.update_size();
  const uint64_t m = g.row_offsets[n];
  geq_status st = check_game(gi, c);
  if (st) return st;
  // reverse CSR (energygame.rs:235-250), predecessors in increasing order
  std::vector<uint32_t> rrow(n + 1, 0), rcol(m);
  for (uint64_t k = 0; k < m; k++) rrow[g.column_indices[k] + 1]++;
  for (uint32_t v = 0; v < n; v++) rrow[v + 1] += rrow[v];
  {
    std::vector<uint32_t> fill(rrow.begin(), rrow.end() - 1);
    for (uint32_t v = 0; v < n; v++)
      for (uint32_t k = g.row_offsets[v]; k < g.row_offsets[v + 1]; k++) rcol[fill[g.column_indices[k]]++] = v;
  }
  // initial lists: given, or {0} at the to_reach positions (with_reach, energygame.rs:355-365)
  std::vector<unsigned long long> desc(n, 0);
  std::vector<uint32_t> init_words;
  if (gi.init) {
    for (uint32_t v = 0; v < n; v++) {
      const uint64_t a = gi.init->offsets[v], b = gi.init->offsets[v + 1];
      desc[v] = ((unsigned long long)a << CNT_BITS) | (b - a);
    }
    init_words.assign(gi.init->data, gi.init->data + gi.init->offsets[n] * es);
  } else {
    for (uint32_t i = 0; i < gi.n_reach; i++) {
      const uint32_t v = gi.to_reach[i];
      if (desc[v]) continue;
      desc[v] = ((unsigned long long)(init_words.size() / es) << CNT_BITS) | 1ull;
      init_words.insert(init_words.end(), es, 0u);
    }
  }
  const unsigned long long init_e = init_words.size() / es;

  Bufs B{eng, {}};
  P p{};
  uint32_t *d_row, *d_col, *d_wt, *d_rrow, *d_rcol, *d_front, *d_next, *d_ovf, *d_mark, *d_reach, *d_arena,
      *d_scratch;
  uint8_t *d_att;
  unsigned long long *d_desc, *d_slot;
  Ctr *d_ctr;
  const uint32_t mwords = (n + 31) / 32;
  if ((st = B.get(d_row, n + 1)) || (st = B.get(d_col, m)) || (st = B.get(d_wt, m * us)) ||
      (st = B.get(d_rrow, n + 1)) || (st = B.get(d_rcol, m)) || (st = B.get(d_att, n)) ||
      (st = B.get(d_desc, n)) || (st = B.get(d_front, n)) || (st = B.get(d_next, n)) ||
      (st = B.get(d_ovf, n)) || (st = B.get(d_mark, mwords)) || (st = B.get(d_slot, n)) ||
      (st = B.get(d_ctr, 1)) || (st = B.get(d_reach, gi.n_reach)))
    return st;
  unsigned long long arena_cap = std::max<unsigned long long>(4 * init_e + 16ull * (n + m), 1ull << 16);
  if ((st = B.get(d_arena, arena_cap * es))) return st;
  const uint32_t max_warps = (uint32_t)n_sms * 16;
  unsigned long long scratch_words = 1ull << 14;  // per warp
  uint32_t scratch_warps = max_warps;
  // the scratch of energies of one, two or four words is taken when an
  // antichain outgrows shared memory
  d_scratch = nullptr;
  if (es != 1 && es != 2 && es != 4 && (st = B.get(d_scratch, scratch_words * scratch_warps))) return st;

  WCU(cudaMemcpyAsync(d_row, g.row_offsets, (n + 1) * 4ull, cudaMemcpyHostToDevice, S));
  if (m) {
    WCU(cudaMemcpyAsync(d_col, g.column_indices, m * 4, cudaMemcpyHostToDevice, S));
    WCU(cudaMemcpyAsync(d_wt, g.weights, m * us * 4, cudaMemcpyHostToDevice, S));
    WCU(cudaMemcpyAsync(d_rcol, rcol.data(), m * 4, cudaMemcpyHostToDevice, S));
  }
  WCU(cudaMemcpyAsync(d_rrow, rrow.data(), (n + 1) * 4ull, cudaMemcpyHostToDevice, S));
  std::vector<uint8_t> att(n);
  for (uint32_t v = 0; v < n; v++) att[v] = g.attacker_pos[v] ? 1 : 0;
  if (n) {
    WCU(cudaMemcpyAsync(d_att, att.data(), n, cudaMemcpyHostToDevice, S));
    WCU(cudaMemcpyAsync(d_desc, desc.data(), n * 8ull, cudaMemcpyHostToDevice, S));
  }
  if (!init_words.empty())
    WCU(cudaMemcpyAsync(d_arena, init_words.data(), init_words.size() * 4, cudaMemcpyHostToDevice, S));
  if (gi.n_reach) WCU(cudaMemcpyAsync(d_reach, gi.to_reach, gi.n_reach * 4ull, cudaMemcpyHostToDevice, S));
  WCU(cudaMemsetAsync(d_mark, 0, mwords * 4ull, S));
  {
    // new lists go after the initial ones
    Ctr h0{};
    h0.arena_top = init_e;
    WCU(cudaMemcpyAsync(d_ctr, &h0, sizeof(Ctr), cudaMemcpyHostToDevice, S));
    WCU(cudaStreamSynchronize(S));  // h0 is on the stack
  }

  p.row = d_row; p.col = d_col; p.wt = d_wt; p.rrow = d_rrow; p.rcol = d_rcol; p.att = d_att;
  p.desc = d_desc; p.arena = d_arena; p.arena_cap = arena_cap;
  p.front = d_front; p.slots = nullptr; p.slot_new = d_slot; p.ovf = d_ovf;
  p.scratch = d_scratch; p.scratch_words = scratch_words; p.ctr = d_ctr;
  p.mark = d_mark; p.next = d_next; p.n_nodes = n; p.mwords = mwords;
  p.el = c.elements; p.mx = c.max; p.eb = c.energy_bits(); p.em = c.energy_mask();
  p.ub = c.update_bits(); p.um = c.update_mask(); p.es = es; p.us = us;
  p.sw = make_swar(p.eb);
  p.wc = WideConf{p.el, p.mx, p.eb, p.em, p.ub, p.um};
  const size_t smem = (size_t)WARPS * (us + 33u * es) * 4;
  WCU(cudaFuncSetAttribute(k_wide_round, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));

  cudaEvent_t ev0, ev1;
  WCU(cudaEventCreate(&ev0));
  WCU(cudaEventCreate(&ev1));
  struct EvGuard {
    cudaEvent_t a, b;
    ~EvGuard() { cudaEventDestroy(a); cudaEventDestroy(b); }
  } evg{ev0, ev1};
  WCU(cudaEventRecord(ev0, S));
  unsigned long long launches = 0;
  if (gi.n_reach) {
    k_wide_mark_reach<<<(gi.n_reach + 255) / 256, 256, 0, S>>>(p, d_reach, gi.n_reach);
    launches++;
  }
  Ctr h{};
  auto fill_next = [&](uint32_t &size) -> geq_status {
    WCU(cudaMemsetAsync(&d_ctr->next_size, 0, 4, S));
    k_wide_fill<<<(mwords + 255) / 256, 256, 0, S>>>(p);
    launches++;
    WCU(cudaMemcpyAsync(&h, d_ctr, sizeof(Ctr), cudaMemcpyDeviceToHost, S));
    WCU(cudaStreamSynchronize(S));
    size = h.next_size;
    return GEQ_OK;
  };
  uint32_t fsize = 0;
  if (n && (st = fill_next(fsize))) return st;
  std::swap(d_front, d_next);
  p.front = d_front;
  p.next = d_next;
  uint64_t rounds = 0;
  uint64_t compactions = 0;
  uint32_t *d_items = nullptr;  // the slots of a round that are computed again
  const bool grid = n > WIDE_CLUSTER_POSITIONS && n <= WIDE_GRID_POSITIONS && grid_blocks(eng, device, es) != 0u;
  const uint32_t cluster = grid                       ? grid_blocks(eng, device, es)
                           : n <= WIDE_GRID_POSITIONS ? cluster_blocks(eng, es)
                                                      : 0u;
  const auto t_start = std::chrono::steady_clock::now();
  while (fsize) {
    bool first_try = true;  // of this round's slots
    if (cluster) {
      // rounds in one launch; a round it left unfinished goes on below
      WCU(cudaMemsetAsync(&d_ctr->next_slot, 0, 12, S));  // next_slot, n_ovf, arena_full
      p.slots = nullptr;
      WCU(es == 1   ? launch_rounds_es<1>(p, grid, cluster, fsize, WIDE_CLUSTER_ROUNDS, S)
          : es == 2 ? launch_rounds_es<2>(p, grid, cluster, fsize, WIDE_CLUSTER_ROUNDS, S)
                    : launch_rounds_es<4>(p, grid, cluster, fsize, WIDE_CLUSTER_ROUNDS, S));
      launches++;
      WCU(cudaMemcpyAsync(&h, d_ctr, sizeof(Ctr), cudaMemcpyDeviceToHost, S));
      WCU(cudaStreamSynchronize(S));
      fsize = h.next_size;
      if (h.flip) std::swap(d_front, d_next);
      p.front = d_front;
      p.next = d_next;
      if (std::chrono::steady_clock::now() - t_start > std::chrono::seconds(600))
        return fail(GEQ_ERR_TIMEOUT, "no fixpoint after 600 s (%llu rounds)", (unsigned long long)(rounds + h.rounds));
      if (!h.n_ovf && !h.arena_full) continue;
      first_try = false;
    }
    rounds++;
    if (std::chrono::steady_clock::now() - t_start > std::chrono::seconds(600))
      return fail(GEQ_ERR_TIMEOUT, "no fixpoint after 600 s (%llu rounds)", (unsigned long long)rounds);
    // the round, repeated for positions whose antichain outgrew the scratch
    p.slots = nullptr;
    p.n_items = fsize;
    const bool shared_ac = es == 1 || es == 2 || es == 4;
    bool fresh = shared_ac;  // all slots, antichains in shared memory; else in the warps' scratch
    for (;;) {
      if (first_try || !cluster) {
        WCU(cudaMemsetAsync(&d_ctr->next_slot, 0, 12, S));  // next_slot, n_ovf, arena_full
        const uint32_t warps = std::min<uint32_t>(scratch_warps, std::max<uint32_t>(p.n_items, 1));
        p.n_warps = warps;
        if (fresh) {
          const unsigned blocks = std::min<unsigned>((p.n_items + WARPS - 1) / WARPS, (unsigned)n_sms * 4u);
          if (es == 1) k_wide_round_es<1><<<blocks, BLOCK_T, 0, S>>>(p);
          else if (es == 2) k_wide_round_es<2><<<blocks, BLOCK_T, 0, S>>>(p);
          else k_wide_round_es<4><<<blocks, BLOCK_T, 0, S>>>(p);
        } else {
          k_wide_round<<<(warps + WARPS - 1) / WARPS, BLOCK_T, smem, S>>>(p);
        }
        launches++;
        WCU(cudaGetLastError());
        WCU(cudaMemcpyAsync(&h, d_ctr, sizeof(Ctr), cudaMemcpyDeviceToHost, S));
        WCU(cudaStreamSynchronize(S));
      }
      first_try = true;
      if (h.arena_full) {
        // compact the committed lists into a larger arena and run the round again
        compactions++;
        std::vector<unsigned long long> hd(n), noff(n);
        WCU(cudaMemcpyAsync(hd.data(), d_desc, n * 8ull, cudaMemcpyDeviceToHost, S));
        WCU(cudaStreamSynchronize(S));
        unsigned long long live = 0;
        for (uint32_t v = 0; v < n; v++) {
          noff[v] = live;
          live += hd[v] & CNT_MASK;
        }
        const unsigned long long cap2 = std::max(2 * arena_cap, 4 * live + (1ull << 16));
        uint32_t *na;
        unsigned long long *d_noff;
        if ((st = B.get(na, cap2 * es)) || (st = B.get(d_noff, n))) return st;
        WCU(cudaMemcpyAsync(d_noff, noff.data(), n * 8ull, cudaMemcpyHostToDevice, S));
        k_wide_move<<<(n + 7) / 8, 256, 0, S>>>(d_desc, d_noff, n, d_arena, na, es);
        k_wide_redesc<<<(n + 255) / 256, 256, 0, S>>>(d_desc, d_noff, n);
        launches += 2;
        B.put(d_arena);
        B.put(d_noff);
        d_arena = na;
        arena_cap = cap2;
        p.arena = d_arena;
        p.arena_cap = arena_cap;
        WCU(cudaMemcpyAsync(&d_ctr->arena_top, &live, 8, cudaMemcpyHostToDevice, S));
        p.slots = nullptr;
        p.n_items = fsize;
        fresh = shared_ac;
        continue;
      }
      if (!h.n_ovf) break;
      // positions whose antichain did not fit: in the warps' scratch, then
      // again with 8x the scratch each, on as many warps as the memory allows
      if (!fresh) scratch_words *= 8;
      fresh = false;
      if (scratch_words > (1ull << 31)) return fail(GEQ_ERR_OUT_OF_MEMORY, "antichain beyond 8 GB of warp scratch");
      if (d_scratch) B.put(d_scratch);
      scratch_warps = (uint32_t)std::max<unsigned long long>(
          1, std::min<unsigned long long>(max_warps, (4ull << 30) / (scratch_words * 4)));
      if ((st = B.get(d_scratch, scratch_words * scratch_warps))) return st;
      // the overflowed slots become the items (copied: the kernel appends to ovf)
      if (d_items) B.put(d_items);  // (its last reader is ahead on the stream)
      if ((st = B.get(d_items, h.n_ovf))) return st;
      WCU(cudaMemcpyAsync(d_items, d_ovf, h.n_ovf * 4ull, cudaMemcpyDeviceToDevice, S));
      p.scratch = d_scratch;
      p.scratch_words = scratch_words;
      p.slots = d_items;
      p.n_items = h.n_ovf;
    }
    k_wide_commit<<<(fsize + 255) / 256, 256, 0, S>>>(p, fsize);
    launches++;
    if ((st = fill_next(fsize))) return st;
    std::swap(d_front, d_next);
    p.front = d_front;
    p.next = d_next;
  }
  WCU(cudaEventRecord(ev1, S));
  // download: offsets and words of every list
  std::vector<unsigned long long> hd(n);
  if (n) WCU(cudaMemcpyAsync(hd.data(), d_desc, n * 8ull, cudaMemcpyDeviceToHost, S));
  WCU(cudaMemcpyAsync(&h, d_ctr, sizeof(Ctr), cudaMemcpyDeviceToHost, S));
  WCU(cudaStreamSynchronize(S));
  std::vector<unsigned long long> noff(n);
  unsigned long long total = 0;
  for (uint32_t v = 0; v < n; v++) {
    noff[v] = total;
    total += hd[v] & CNT_MASK;
  }
  uint32_t *d_out = nullptr;
  unsigned long long *d_noff = nullptr;
  if ((st = B.get(d_out, total * es)) || (st = B.get(d_noff, n))) return st;
  if (n) {
    WCU(cudaMemcpyAsync(d_noff, noff.data(), n * 8ull, cudaMemcpyHostToDevice, S));
    k_wide_move<<<(n + 7) / 8, 256, 0, S>>>(d_desc, d_noff, n, d_arena, d_out, es);
    launches++;
  }
  const uint64_t ob = sol.offsets.size(), db = sol.data.size() / es;
  sol.n_vertices.push_back(n);
  sol.offsets_base.push_back(ob);
  sol.data_base.push_back(db);
  sol.offsets.resize(ob + n + 1);
  for (uint32_t v = 0; v < n; v++) sol.offsets[ob + v] = noff[v];
  sol.offsets[ob + n] = total;
  sol.data.resize((db + total) * es);
  if (total) WCU(cudaMemcpyAsync(sol.data.data() + db * es, d_out, total * es * 4, cudaMemcpyDeviceToHost, S));
  WCU(cudaStreamSynchronize(S));
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ev0, ev1);
  sol.stats.rounds += rounds + h.rounds;
  sol.stats.positions_computed += h.positions;
  sol.stats.edges_relaxed += h.edges;
  sol.stats.algorithmic_bytes += h.bytes;
  sol.stats.arena_compactions += compactions;
  sol.stats.kernel_launches += launches;
  sol.stats.device_ms += ms;
  (void)g_index;
  return GEQ_OK;
}

}  // namespace wide

bool wide_supported(const Conf &c, std::string *why) {
  if (c.energy_size() > wide::ES_MAX || c.update_size() > wide::US_MAX) {
    if (why)
      *why = "EnergyConf {" + std::to_string(c.elements) + ", " + std::to_string(c.max) + "} needs " +
             std::to_string(c.energy_size()) + " energy / " + std::to_string(c.update_size()) +
             " update words (the solver takes up to " + std::to_string(wide::ES_MAX) + " / " +
             std::to_string(wide::US_MAX) + ")";
    return false;
  }
  return c.elements >= 1;
}

geq_status solve_wide(Engine &e, int device, std::vector<GameInput> &in, geq_solution &sol) {
  if (in.empty()) return fail(GEQ_ERR_INVALID_INPUT, "no games");
  const Conf c(in[0].g.conf);
  std::string why;
  if (!wide_supported(c, &why)) return fail(GEQ_ERR_UNSUPPORTED, "%s", why.c_str());
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != device) cudaSetDevice(device);
  struct Restore {
    int prev, dev;
    ~Restore() { if (prev != dev && prev >= 0) cudaSetDevice(prev); }
  } restore{prev, device};
  sol.energy_size = c.energy_size();
  for (uint32_t g = 0; g < in.size(); g++) {
    GameInput &gi = in[g];
    if (gi.std_reach) {
      gi.reach_storage = standard_reach_of(gi.g);
      gi.to_reach = gi.reach_storage.data();
      gi.n_reach = (uint32_t)gi.reach_storage.size();
      gi.std_reach = false;
    }
    const geq_status st = wide::solve_one_game(e, device, gi, c, sol, g);
    if (st) return st;
  }
  return GEQ_OK;
}

}  // namespace geq
