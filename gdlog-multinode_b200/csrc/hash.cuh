// hash.cuh — update relations of wide domains deduplicated by a hash set.
//
// Beyond the bitmaps (ids from 2^16 on, or arity 3) the list form sorts every
// iteration's candidates and merges them into all of FULL: for a sparse graph
// a fixpoint is a dozen kernels an iteration whose cost follows |FULL|, not
// the new tuples (the 64 x 64 grid's path lengths: 126 iterations of 13
// launches, 4.3 M tuples merged each time, 21 ms).  When no operator reads
// FULL as a list during the loop (every inner is a static relation, DELTA and
// a tmp NEWT are only outers), order is needed once, at the end.  Then:
//   * FULL is an unsorted list plus a set of its keys: open addressing, 8-byte
//     slots, at most three quarters full when an iteration commits, ~0 empty;
//   * a join probes, expands and inserts in one pass (k_join_hash): a
//     candidate that takes an empty slot is new and is appended to FULL and to
//     the next DELTA, any other is dropped, most of them by a plain load;
//   * a tmp relation's NEWT is appended to without deduplication, as the
//     reference does;
//   * after the loop FULL is sorted once by the radix sort.
// A candidate costs one random 8-byte access (an L2 hit while the set is
// below 100 MB), whatever |FULL| is.  The iterations run in one resident
// launch (k_hash_loop, as loop.cuh): a barrier an operator.
//
// Dependent columns (src/lie.cu:131-138): a tuple is new only if no FULL
// tuple has its other columns, and tuples of one iteration that differ in
// dependent columns only are all new.  Keys hash by their prefix, so the
// tuples of one prefix share a probe chain.  Each slot's ordinal in FULL
// (`hord`) says whether its tuple was there when the iteration began: a
// candidate that meets its prefix in such a slot is known.  One that meets it
// in a slot of this iteration, with another dependent part, is put aside (in
// the relation's NEWT, otherwise unused here), and k_hash_aside decides it
// after the joins.  (On a random graph most paths are derived again, longer.
// Put aside like the others, an atomic of one counter each, the shortest paths
// over 2^12 ids and 8,000 R-MAT edges took 9.7 ms, now 2.1; 5.1 on sorted
// lists.)
//
// A key takes its slot before the list's counter counts it, so an iteration
// may pass the three quarters before the overflow is seen: up to 224 keys a
// warp wait uncounted, and a warp looks at the overflow flag every four steps
// of 32 candidates.  A set may even fill up.  Probe chains are therefore
// bounded (kHashMaxProbe): past the bound the iteration ends uncommitted and
// runs again, from a larger set where the rows counted ask for one, else (the
// chain is the tuples of one prefix, which no larger set shortens) on sorted
// lists.
#pragma once

#include "common.cuh"
#include "dense.cuh"
#include "index.cuh"
#include "join.cuh"
#include "loop.cuh"

namespace gdl {

constexpr u64 kHashEmpty = ~0ull;
// A set holds up to three quarters of its slots.  The first has room for
// kHashGrowth times the largest relation that the LIE starts from, up to 2^23
// slots, 64 MB: half of L2, and 6.3 M tuples.  (With 2^23 whatever the input,
// a three-edge graph took 384 MB for its sets and lists, twenty relations of
// one tuple 4.6 GB.  The 64 x 64 grid's shortest paths are 533 for an edge,
// the most of the benchmarks' programs.)
__host__ __device__ constexpr u64 hash_rows(u64 slots) { return slots / 4 * 3; }
constexpr u64 kHashFirstRows = hash_rows(1ull << 23);
constexpr u64 kHashGrowth = 1024;

struct HashJoinArgs {
  JoinArgs j;
  RelDev *out;
  int hashed;     // out is an update relation kept as a set, else a tmp list
  u64 prefix;     // key bits that decide membership (~0 without dependent columns)
  int need_full, need_delta, need_newt;  // need slots of out
};

// Slots a probe looks at.  The longest chain of random keys in a set three
// quarters full is about ln(slots) / 0.038 slots (Knuth vol. 3, 6.4): 420 of
// 2^23, 570 of 2^31.
constexpr u32 kHashMaxProbe = 2048;

// The iteration cannot be committed with this set.
__device__ __forceinline__ void hash_chain_long(Ctl *ctl) {
  ctl->hash_long = 1;
  atomicExch(&ctl->overflow, 1u);
}

// One candidate: 0 known, 1 new (its slot in *slot), 2 this iteration derived
// its prefix with another dependent part, 3 its probe chain is too long.
// hord: with dependent columns, each slot's ordinal; FULL had full_n tuples
// when the iteration began (slots taken since have ordinals from there on, or
// none yet).
__device__ __forceinline__ int hash_insert(u64 *set, u64 mask, u64 prefix, const u32 *hord,
                                           u64 full_n, u64 k, u64 *slot) {
  if (k == kHashEmpty) {
    // the one key that looks like an empty slot has a slot of its own
    *slot = mask + 1;
    return atomicCAS((unsigned long long *)&set[mask + 1], kHashEmpty, 0ull) == kHashEmpty;
  }
  u64 h = mix64(k & prefix) & mask;
  for (u32 step = 0; step < kHashMaxProbe; step++) {
    u64 s = *((volatile u64 *)&set[h]);
    if (s == kHashEmpty) {
      s = atomicCAS((unsigned long long *)&set[h], kHashEmpty, k);
      if (s == kHashEmpty) {
        *slot = h;
        return 1;
      }
    }
    if (s == k) return 0;
    if (((s ^ k) & prefix) == 0) return *((volatile const u32 *)&hord[h]) < full_n ? 0 : 2;
    h = (h + 1) & mask;
  }
  return 3;
}

// A warp's new keys wait in shared memory until kOutCap - 32 are there, so
// that the list's counter, one address for the whole grid, takes an atomic
// per couple of hundred keys instead of one per step.
constexpr u32 kOutCap = 256;
struct WarpOut {
  u64 key[kOutCap];
  u32 slot[kOutCap];  // (with dependent columns)
};

// Lists of `out`: its new tuples (FULL and the next DELTA), or its NEWT.
__device__ __forceinline__ void hash_flush(const HashJoinArgs &a, bool fresh, WarpOut &w, u32 n) {
  if (n == 0) return;
  const int lane = threadIdx.x & 31;
  RelDev *r = a.out;
  __syncwarp();
  u64 base = 0;
  if (lane == 0)
    base = atomicAdd((unsigned long long *)(fresh ? &r->delta_next.n : &r->newt.n),
                     (unsigned long long)n);
  base = __shfl_sync(0xffffffffu, base, 0);
  if (!fresh) {
    u64 *dst = r->newt.ptr;
    const u64 cap = r->newt.cap;
    for (u32 i = lane; i < n; i += 32)
      if (base + i < cap) dst[base + i] = w.key[i];
    if (base + n > cap && lane == 0) {
      atomicMax((unsigned long long *)&a.j.ctl->need[a.need_newt], base + n);
      atomicExch(&a.j.ctl->overflow, 1u);
    }
    __syncwarp();
    return;
  }
  u64 *delta = r->delta_next.ptr, *full = r->full.ptr;
  u32 *hord = r->hord;
  const u64 ord0 = r->full.n + base;
  const u64 cap = r->delta_next.cap, fcap = min(r->full.cap, hash_rows(r->hmask + 1));
  for (u32 i = lane; i < n; i += 32)
    if (base + i < cap && ord0 + i < fcap) {
      delta[base + i] = w.key[i];
      full[ord0 + i] = w.key[i];
      if (hord) hord[w.slot[i]] = (u32)(ord0 + i);
    }
  if ((base + n > cap || ord0 + n > fcap) && lane == 0) {
    // the iteration runs again from FULL's committed rows
    atomicMax((unsigned long long *)&a.j.ctl->need[a.need_full], ord0 + n);
    atomicMax((unsigned long long *)&a.j.ctl->need[a.need_delta], base + n);
    atomicExch(&a.j.ctl->overflow, 1u);
  }
  __syncwarp();
}
// The lanes with `take` add their key; n: keys waiting (warp-uniform).
__device__ __forceinline__ void hash_put(const HashJoinArgs &a, bool fresh, WarpOut &w, u32 &n,
                                         bool take, u64 k, u64 slot) {
  const unsigned m = __ballot_sync(0xffffffffu, take);
  if (!m) return;
  if (take) {
    const u32 at = n + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
    w.key[at] = k;
    if (a.prefix != ~0ull) w.slot[at] = (u32)slot;
  }
  n += __popc(m);
  if (n > kOutCap - 32) {
    hash_flush(a, fresh, w, n);
    n = 0;
  }
}

// One candidate a lane; set aside (rare, so unbuffered): a candidate whose
// prefix is present with another dependent part.
__device__ __forceinline__ void hash_emit(const HashJoinArgs &a, WarpOut &w, u32 &n, u64 k,
                                          bool valid) {
  if (!a.hashed) {
    hash_put(a, false, w, n, valid, k, 0);
    return;
  }
  u64 slot = 0;
  const int st = valid ? hash_insert(a.out->hset, a.out->hmask, a.prefix, a.out->hord,
                                     a.out->full.n, k, &slot)
                       : 0;
  hash_put(a, true, w, n, st == 1, k, slot);
  if (st == 3) hash_chain_long(a.j.ctl);
  if (st == 2) {
    RelDev *r = a.out;
    const u64 pos = atomicAdd((unsigned long long *)&r->newt.n, 1ull);
    if (pos < r->newt.cap) {
      r->newt.ptr[pos] = k;
    } else {
      atomicMax((unsigned long long *)&a.j.ctl->need[a.need_newt], pos + 1);
      atomicExch(&a.j.ctl->overflow, 1u);
    }
  }
}

// A join's candidates into a hash set or a tmp list: probe and expand as
// k_join_bm (dense.cuh), 32 candidates of a warp's 32 outer rows a step; runs
// longer than kHeavyRun are cut into pieces for k_join_hash_heavy.
struct HashSmem {
  FuseSmem<256> fuse;
  WarpOut out[8];
};
__device__ __forceinline__ void hash_join(const HashJoinArgs &a, HashSmem &hs) {
  FuseSmem<256> &sm = hs.fuse;
  WarpOut *s_out = hs.out;
  const JoinArgs &j = a.j;
  const u64 n_outer = eff_count(j.outer, j.outer_vis);
  const u64 n_inner = eff_count(j.inner, j.inner_vis);
  if (n_outer == 0 || n_inner == 0) {
    join_empty_side(j, n_outer);
    return;
  }
  if (j.once) {
    if (*j.once) {
      if (blockIdx.x == 0 && threadIdx.x == 0 && *j.produced) *j.phantom = 1;
      return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *j.once_pending = 1;
  }
  const Index ix = *j.inner_idx;
  const u64 *inner = j.inner->ptr;
  const u64 *outer = j.outer->ptr;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const u64 chunks = (n_outer + 31) / 32;
  const u64 nw = (u64)gridDim.x * 8;
  u64 cand = 0;
  bool emitted = false;
  u32 waiting = 0;
  for (u64 c = (u64)blockIdx.x * 8 + wid; c < chunks; c += nw) {
    // (not before a warp's first chunk, whose loads would wait for this one:
    // 0.3 us of an iteration that has one chunk a warp)
    u32 over = 0;
    if (c >= nw) {
      over = *((volatile u32 *)&j.ctl->overflow);
      if (__any_sync(0xffffffffu, over != 0)) break;
    }
    const u64 i = c * 32 + lane;
    u64 row = 0;
    u32 s = 0, l = 0;
    if (i < n_outer) {
      row = outer[i];
      l = index_probe(ix, key_c0(row), &s);
    }
    if (l > kHeavyRun) {
      const u32 np = (l + kHeavyPiece - 1) / kHeavyPiece;
      const u64 pos = reserve_pieces(j, np);
      if (pos != ~0ull) {
        for (u32 k = 0; k < np; k++) {
          j.crow_key[pos + k] = row;
          j.crow_start[pos + k] = s + k * kHeavyPiece;
          j.crow_len[pos + k] = min(kHeavyPiece, l - k * kHeavyPiece);
        }
        l = 0;
      }  // else: no room, the warp expands the run itself
    }
    u64 inc = l;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u64 y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += y;
    }
    const u64 total = __shfl_sync(0xffffffffu, inc, 31);
    sm.row[wid][lane] = row;
    sm.start[wid][lane] = s;
    sm.excl[wid][lane] = inc - l;
    __syncwarp();
    for (u64 base = 0; base < total; base += 32) {
      // (a chunk may hold thousands of candidates: a look every four steps,
      // its load under way with the step's others)
      const bool look = (base & 96) == 96;
      if (look) over = *((volatile u32 *)&j.ctl->overflow);
      const u64 p = base + lane;
      u64 t = 0;
      bool ok = false;
      if (p < total) {
        int r = 0;
#pragma unroll
        for (int h = 16; h > 0; h >>= 1)
          if (sm.excl[wid][r + h] <= p) r += h;
        t = join_out(j, inner[sm.start[wid][r] + (p - sm.excl[wid][r])], sm.row[wid][r]);
        ok = pred_ok(j.pred, t);
      }
      emitted |= ok;
      hash_emit(a, s_out[wid], waiting, t, ok);
      if (look && __any_sync(0xffffffffu, over != 0)) break;
    }
    __syncwarp();
    cand += total;
  }
  hash_flush(a, a.hashed, s_out[wid], waiting);
  if (__any_sync(0xffffffffu, emitted) && lane == 0) {
    if (a.hashed) a.out->c_newt_n = 1;  // NEWT is not empty (src/lie.cu:114-121)
    if (j.produced) *j.produced = 1;
  }
  if (lane == 0) prof_add(j.ctl, kPJoinMat, cand * 16);
  if (blockIdx.x == 0 && threadIdx.x == 0) prof_add(j.ctl, kPJoinMat, n_outer * 24);
}
__global__ void __launch_bounds__(256) k_join_hash(HashJoinArgs a) {
  __shared__ HashSmem sm;
  if (ctl_stop(a.j.ctl)) return;
  hash_join(a, sm);
}

// The first np pieces of long runs, a block per piece.
__device__ __forceinline__ void hash_heavy(const HashJoinArgs &a, u64 np, WarpOut *s_out) {
  const JoinArgs &j = a.j;
  const u64 *inner = j.inner->ptr;
  u64 cand = 0;
  bool emitted = false;
  u32 waiting = 0;
  for (u64 k = blockIdx.x; k < np; k += gridDim.x) {
    if (__any_sync(0xffffffffu, *((volatile u32 *)&j.ctl->overflow) != 0)) break;
    const u64 row = j.crow_key[k];
    const u32 s = j.crow_start[k], l = j.crow_len[k];
    for (u32 j0 = threadIdx.x & ~31u; j0 < l; j0 += blockDim.x) {  // (warp-uniform)
      const bool look = ((j0 / blockDim.x) & 3) == 3;
      const u32 over = look ? *((volatile u32 *)&j.ctl->overflow) : 0u;
      const u32 q = j0 + (threadIdx.x & 31);
      u64 t = 0;
      bool ok = false;
      if (q < l) {
        t = join_out(j, inner[s + q], row);
        ok = pred_ok(j.pred, t);
      }
      emitted |= ok;
      hash_emit(a, s_out[threadIdx.x >> 5], waiting, t, ok);
      if (look && __any_sync(0xffffffffu, over != 0)) break;
    }
    cand += l;
  }
  hash_flush(a, a.hashed, s_out[threadIdx.x >> 5], waiting);
  if (__any_sync(0xffffffffu, emitted) && (threadIdx.x & 31) == 0) {
    if (a.hashed) a.out->c_newt_n = 1;
    if (j.produced) *j.produced = 1;
  }
  if (threadIdx.x == 0) prof_add(j.ctl, kPJoinMat, cand * 16);
}
// (The last block empties the piece list.  An overflow may be raised while
// blocks of this launch are still starting: every block comes to the end.)
__global__ void __launch_bounds__(256) k_join_hash_heavy(HashJoinArgs a) {
  __shared__ int s_stop;
  __shared__ WarpOut s_out[8];
  if (threadIdx.x == 0) s_stop = ctl_stop(a.j.ctl);
  __syncthreads();
  hash_heavy(a, s_stop ? 0 : min(a.j.op->nc, a.j.crow_cap), s_out);
  if (launch_rec_finish(a.j.rec) && threadIdx.x == 0) a.j.op->nc = 0;
}

// The candidates put aside: new unless a tuple of their prefix was in FULL
// when the iteration began; each kept once.  (A slot taken by this launch or
// the joins has an ordinal from FULL's count on, or none yet.)
__device__ __forceinline__ void hash_aside(const HashJoinArgs &a, WarpOut *s_out) {
  RelDev *r = a.out;
  u32 waiting = 0;
  const u64 n = min(r->newt.n, r->newt.cap);
  const u64 full_n = r->full.n, mask = r->hmask;
  const int lane = threadIdx.x & 31;
  for (u64 i0 = ((u64)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; i0 < n;
       i0 += (u64)gridDim.x * blockDim.x) {
    if (__any_sync(0xffffffffu, *((volatile u32 *)&a.j.ctl->overflow) != 0)) break;
    bool is_new = false;
    u64 k = 0, slot = 0;
    if (i0 + lane < n) {
      k = r->newt.ptr[i0 + lane];
      u64 h = mix64(k & a.prefix) & mask;
      u32 step = 0;
      for (; step < kHashMaxProbe; step++) {
        u64 s = *((volatile u64 *)&r->hset[h]);
        if (s == kHashEmpty) {
          s = atomicCAS((unsigned long long *)&r->hset[h], kHashEmpty, k);
          if (s == kHashEmpty) {
            is_new = true;
            slot = h;
            break;
          }
        }
        if (s == k) break;
        if (((s ^ k) & a.prefix) == 0 && *((volatile u32 *)&r->hord[h]) < full_n) break;
        h = (h + 1) & mask;
      }
      if (step == kHashMaxProbe) hash_chain_long(a.j.ctl);
    }
    hash_put(a, true, s_out[threadIdx.x >> 5], waiting, is_new, k, slot);
  }
  hash_flush(a, true, s_out[threadIdx.x >> 5], waiting);
}
__global__ void __launch_bounds__(256) k_hash_aside(HashJoinArgs a) {
  __shared__ WarpOut s_out[8];
  if (ctl_stop(a.j.ctl)) return;
  hash_aside(a, s_out);
}

constexpr int kHashLoopOps = 16;
constexpr int kHashLoopCtasPerSm = 4;

struct HashLoopArgs {
  const HashJoinArgs *ops;  // n_ops joins, then (to n_all) the relations whose
  int n_ops, n_all;         // candidates may be put aside
  RelDev *rels;
  LieDev *lie;
  Ctl *ctl;
};

// Every iteration of a LIE.  A join's barrier tells whether it left pieces of
// long runs, the last join's whether candidates were put aside; when neither,
// that barrier commits.  An overflow ends the loop uncommitted, at the first
// barrier after it.
__global__ void __launch_bounds__(256, kHashLoopCtasPerSm) k_hash_loop(HashLoopArgs a) {
  __shared__ HashSmem sm;
  __shared__ HashJoinArgs s_op[kHashLoopOps];
  __shared__ int s_go;
  for (u32 i = threadIdx.x; i < a.n_ops * sizeof(HashJoinArgs) / 4; i += 256)
    reinterpret_cast<u32 *>(s_op)[i] = reinterpret_cast<const u32 *>(a.ops)[i];
  __syncthreads();
  Ctl *ctl = a.ctl;
  u32 gen = ctl->bar_word >> 2;
  // (not the overflow flag: a block may start after another has raised it, and
  // each of them arrives at the first barrier or none does)
  u32 flags = (ctl->done | ctl->pause | ctl->timeout) ? 1u : 0u;
  const LaneLists lists = lane_lists(a.lie, threadIdx.x & 31);
  // the asides' counts, a relation a lane
  const u64 *aside_n = nullptr;
  if ((int)(threadIdx.x & 31) < a.n_all - a.n_ops)
    aside_n = &a.ops[a.n_ops + (threadIdx.x & 31)].out->newt.n;
  auto finish = [&](int lane) -> u32 {
    return loop_commit<true>(a.rels, a.lie, ctl, lists, lane) ? 1u : 0u;
  };
  // What the last block decides after a join: 1 an overflow ends the loop, 2
  // pieces (nc) or, after the last join, asides are left, else it may commit.
  // One round trip: every word is loaded before one is looked at.
  auto decide = [&](int lane, const u64 *nc, bool last) -> u32 {
    const u64 left = nc ? *((volatile const u64 *)nc) : 0;
    const u64 put = aside_n ? *((volatile const u64 *)aside_n) : 0;
    if (*((volatile u32 *)&ctl->overflow)) return 1u;
    if (left) return 2u;
    if (!last) return 0u;
    return __any_sync(0xffffffffu, put != 0) ? 2u : finish(lane);
  };
  while (!(flags & 1u)) {
    bool committed = false;
    for (int i = 0; i < a.n_ops && !(flags & 1u); i++) {
      const HashJoinArgs &op = s_op[i];
      const bool last = i == a.n_ops - 1;
      hash_join(op, sm);
      // bit 1: more to do before the next join (or the commit)
      flags = loop_barrier_flags(ctl, gen, &s_go, [&](int lane) -> u32 {
        return decide(lane, &op.j.op->nc, last);
      });
      if (flags & 1u) break;
      if (!(flags & 2u)) {
        committed = last;
        continue;
      }
      const u64 np = min(*((volatile u64 *)&op.j.op->nc), op.j.crow_cap);
      if (np) {
        hash_heavy(op, np, sm.out);
        flags = loop_barrier_flags(ctl, gen, &s_go, [&](int lane) -> u32 {
          if (lane == 0) op.j.op->nc = 0;
          return decide(lane, nullptr, last);
        });
        if (flags & 1u) break;
        if (!(flags & 2u)) {
          committed = last;
          continue;
        }
      }
    }
    if ((flags & 1u) || committed) continue;
    for (int i = a.n_ops; i < a.n_all && !(flags & 1u); i++) {
      hash_aside(a.ops[i], sm.out);
      const bool end = i == a.n_all - 1;
      flags = loop_barrier_flags(ctl, gen, &s_go, [&](int lane) -> u32 {
        if (*((volatile u32 *)&ctl->overflow)) return 1u;
        return end ? finish(lane) : 0u;
      });
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (*((volatile u32 *)&ctl->overflow))  // (pieces of an iteration that runs again)
      for (int i = 0; i < a.n_ops; i++) a.ops[i].j.op->nc = 0;
    if (ctl->cond_set)
      cudaGraphSetConditional((cudaGraphConditionalHandle)ctl->cond_handle, 0u);
  }
}

// The set of FULL's committed rows (the set is all empty when this starts;
// rows of one prefix are entries of their own).  Rows past the chains' bound
// are left out: the iteration that opens next (k_begin) ends the loop, which
// goes on on sorted lists.
__global__ void __launch_bounds__(256) k_hash_fill(RelDev *r, u64 prefix, Ctl *ctl) {
  if (ctl_stop(ctl)) return;
  const u64 n = r->full.n, mask = r->hmask;
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x) {
    const u64 k = r->full.ptr[i];
    u64 h;
    if (k == kHashEmpty) {
      h = mask + 1;
      r->hset[h] = 0;
    } else {
      h = mix64(k & prefix) & mask;
      u32 step = 0;
      for (; step < kHashMaxProbe; step++) {
        if (atomicCAS((unsigned long long *)&r->hset[h], kHashEmpty, k) == kHashEmpty) break;
        if ((step & 255u) == 255u && *((volatile u32 *)&r->hlong)) return;
        h = (h + 1) & mask;
      }
      if (step == kHashMaxProbe) {
        r->hlong = 1;
        continue;
      }
    }
    if (r->hord) r->hord[h] = (u32)i;
  }
}

}  // namespace gdl
