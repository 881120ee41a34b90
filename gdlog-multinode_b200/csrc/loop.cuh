// loop.cuh — a LIE's iterations in one resident kernel.
//
// Over small domains an iteration is a few kernels of two to four
// microseconds each, and the graph's while-node spends ten times that
// between them: a 64 x 64 grid's closure (126 iterations of a join, an
// update pass and a commit over 2 MB bitmaps) took 25 us an iteration.  Here
// the whole loop is one cooperative launch: its blocks stay resident, run
// the iteration's steps in operator order and meet at a grid barrier after
// each.  The last block to arrive does the step's bookkeeping before it
// opens the barrier, so the commit (control.cuh) costs no launch either.
//
// Used up to 2^kLoopMaxBits ids (bitmaps of at most 8 MB, which stay in L2)
// when every operator is a row-gather join, a product below 2^12 ids
// or a swapping ACopy, and every update relation has the fused update step.
// From 2^14 ids an iteration's own work is larger than the launches, and the
// TMA passes (tma.cuh) do it faster than the passes here.
//
// Every wait is bounded: a block that gives up raises Ctl::timeout and leaves,
// and the others leave when they see it.  At a barrier a block waits for the
// others' whole steps, not for one tile, so the bound there is kBarrierPolls
// or Ctl::spin_limit, whichever is more.
#pragma once

#include "common.cuh"
#include "control.cuh"
#include "dense.cuh"
#include "product.cuh"
#include "pull.cuh"

namespace gdl {

constexpr int kLoopBlock = 256;
constexpr int kLoopMaxBits = 13;

constexpr u32 kBarrierPolls = 1u << 25;  // some twenty seconds

constexpr int kLoopMaxSteps = 64;  // at most 32 of one level
constexpr int kLoopMaxUpd = 32;

enum LoopKind { kLoopRows = 0, kLoopProduct, kLoopTranspose, kLoopFold };

// One step.  Steps of one level touch nothing another of them writes
// (products may OR into one bitmap) and run without a barrier between them.
struct LoopStep {
  int kind, level;
  int level_end;   // one past the last step of its level
  // joins: descriptors for the emptiness rules (src/join.cu:38-45)
  const DArr *outer, *inner;
  u32 *outer_vis;        // null: a NEWT outer
  const u32 *inner_vis;
  u32 *outer_bm;         // NEWT outer: its bitmap and words
  u64 outer_words;
  int op;                // place in the LIE
  int delta_rel;         // product: relation whose DELTA is the outer, else -1
  u64 before;            // product: the steps (by number) of operators before
                         // this one with the same DELTA as their outer
  // product: OT, F -> dst; rows: O -> dst; transpose and fold: src -> dst
  const u32 *src, *F;
  u32 *dst;
  // transpose: if set, the bits counted into *count_acc and published
  DArr *count_to;
  u64 *count_acc;
  // rows
  const u32 *inv_keys, *inv_ys;
  u32 n_edges, unit;
  int dst_zero, clear_diag;
  const u32 *once;
  u32 *once_pending, *produced, *phantom;
};

// The update step of one relation, or (rd null) a tmp NEWT to clear.
struct LoopUpd {
  RelDev *rd;
  u32 *F, *G;      // FULL; NEWT's rows
  u32 *gt;         // NEWT as its transposed twin instead (G unused), or null
  u32 *dn, *dt;    // DELTA's rows / DELTA transposed, or null
  u8 *clean;       // per tile: DELTA's tiles are known to be zero
};

struct LoopArgs {
  const LoopStep *steps;
  const LoopUpd *upd;
  int n_steps, n_upd;
  int dk;
  u32 side, splits;
  RelDev *rels;
  LieDev *lie;
  Ctl *ctl;
};

// Grid barrier, all threads of all blocks.  The last block's first warp runs
// fin(lane), which returns flags every block gets: bit 0 stops the loop, bit 1
// is the caller's.  One round trip to count arrivals and one to see the word
// the last block releases, which carries the barrier's number and the flags.
// A wait that gives up returns the stop bit.
template <class Fin>
__device__ __forceinline__ u32 loop_barrier_flags(Ctl *ctl, u32 &gen, int *s_go, Fin fin) {
  __syncthreads();
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    u32 last = 0;
    if (lane == 0) {
      u32 before;
      asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;"
                   : "=r"(before)
                   : "l"(&ctl->bar_count)
                   : "memory");
      last = before == gridDim.x - 1;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    __syncwarp();
    u32 word = 0;
    if (last) {
      const u32 flags = fin(lane);
      __syncwarp();
      if (lane == 0) {
        ctl->bar_count = 0;
        word = ((gen + 1) << 2) | flags;
        asm volatile("st.release.gpu.u32 [%0], %1;" ::"l"(&ctl->bar_word),
                     "r"(word)
                     : "memory");
      }
    } else if (lane == 0) {
      const u32 limit = max(ctl->spin_limit, kBarrierPolls);
      for (u32 polls = 0;; polls++) {
        asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(word) : "l"(&ctl->bar_word) : "memory");
        if ((word >> 2) != gen) break;
        if ((polls & 63u) == 63u && *((volatile u32 *)&ctl->timeout)) {
          word = 1;
          break;
        }
        if (polls > limit) {
          atomicOr(&ctl->timeout, 1u);
          word = 1;
          break;
        }
      }
    }
    if (lane == 0) *s_go = (int)(word & 3u);
  }
  __syncthreads();
  gen = (gen + 1) & 0x3FFFFFFFu;
  return (u32)*s_go;
}
// ... with fin returning whether the loop stops; false when it does.
template <class Fin>
__device__ __forceinline__ bool loop_barrier(Ctl *ctl, u32 &gen, int *s_go, Fin fin) {
  return !(loop_barrier_flags(ctl, gen, s_go, [&](int lane) { return fin(lane) ? 1u : 0u; }) & 1u);
}

// k_commit's bookkeeping (control.cuh) for relations kept as bitmaps with
// the fused update step, then the next iteration's opening.  One warp; every
// load of a lane is issued before any of them is used.  With bitmaps DELTA's
// lists are not written during the loop and only counts change; the hash
// form (hash.cuh) swaps its two DELTA lists.
template <bool HASH>
__device__ __forceinline__ bool loop_commit(RelDev *rels, LieDev *lie, Ctl *ctl,
                                            const LaneLists &x, int lane) {
  const u64 it = ctl->iteration, trace_base = ctl->trace_base, trace_rows = ctl->trace_rows;
  const u64 max_it = ctl->max_iteration, stop_at = ctl->stop_at;
  u64 *trace = lie->trace;
  bool grew = false;
#pragma unroll
  for (int j = 0; j < kListPerLane; j++) {
    const int i = lane + 32 * j;
    if (i < x.nu) {
      RelDev &r = rels[x.upd[j]];
      const u64 nd = HASH ? r.delta_next.n : r.scan.total_a;
      const u64 nn = HASH ? r.c_newt_n : r.scan.pop_g, nf = r.full.n;
      u64 *dp = nullptr, *np = nullptr;
      u64 dc = 0, nc = 0;
      if (HASH) dp = r.delta.ptr, dc = r.delta.cap, np = r.delta_next.ptr, nc = r.delta_next.cap;
      const u32 ph = r.newt_phantom, wv = r.w_full_vis;
      const u64 row = it - trace_base;
      u64 *tr = (trace && row < trace_rows) ? trace + (row * x.nu + i) * 3 : nullptr;
      const bool none = nn == 0 && !ph;  // src/lie.cu:114-121: no new tuple
      const u64 dn = none ? 0 : nd;
      const u32 fv = dn ? 1u : wv;
      if (dn) r.full.n = nf + dn;
      grew = grew || dn != 0;
      r.delta.n = dn;
      r.full_vis = r.w_full_vis = fv;
      r.delta_vis = r.w_delta_vis = 1;
      if (tr) {
        tr[0] = none ? kNoTrace : dn;
        tr[1] = dn;
        tr[2] = nf + dn;
      }
      if (HASH) {
        if (!none) r.delta.ptr = np, r.delta.cap = nc, r.delta_next.ptr = dp, r.delta_next.cap = dc;
        r.delta_next.n = 0;
        r.c_newt_n = 0;
      } else {
        r.scan.total_a = 0;
        r.scan.pop_g = 0;
      }
      r.newt.n = 0;
      r.newt_phantom = 0;
    }
    if (i < x.ns) {
      RelDev &r = rels[x.sta[j]];
      const u32 f = r.w_full_vis, d = r.w_delta_vis;
      r.full_vis = f;
      r.delta_vis = d;
    }
    if (i < x.nt) {
      RelDev &r = rels[x.tmp[j]];
      const u32 f = r.full_vis, d = r.delta_vis;
      r.newt.n = 0;  // src/lie.cu:85-87
      r.w_full_vis = f;
      r.w_delta_vis = d;
    }
    if (i < x.no) {
      const u32 p = lie->jonce_pending[i];
      if (p) {
        lie->jonce[i] |= p;
        lie->jonce_pending[i] = 0;
      }
    }
  }
  const bool fixpoint = !__any_sync(0xffffffffu, grew);
  const u64 next = it + 1;
  const bool done = fixpoint || next > max_it;
  const bool pause = !done && next >= stop_at;
  if (lane == 0) {
    ctl->iteration = next;
    ctl->generation = ctl->generation + 1;
    if (done) ctl->done = 1;
    if (pause) ctl->pause = 1;
  }
  return done || pause;
}

// dst |= transpose(src) and src cleared, by tiles.
__device__ __forceinline__ void loop_fold(u32 *src, u32 *dst, int rs, u32 side, u32 block,
                                          u32 (*s_t)[9]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (u32 t = block; t < side * side; t += gridDim.x) {
    const u32 tr = t / side, tc = t % side;
    const u64 at = (((u64)tr * 256 + threadIdx.x) << rs) + tc * 8;
    const u64 dw = (((u64)tc * 256 + threadIdx.x) << rs) + tr * 8;
    u32 v[8];
    load8(src + at, v);
    const bool any = (v[0] | v[1] | v[2] | v[3] | v[4] | v[5] | v[6] | v[7]) != 0u;
    uint4 *pd = reinterpret_cast<uint4 *>(dst + dw);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    if (any) {
      uint4 *ps = reinterpret_cast<uint4 *>(src + at);
      ps[0] = zero;
      ps[1] = zero;
    }
    // (also orders the last tile's reads of s_t)
    if (__syncthreads_or(any)) {
#pragma unroll
      for (int i = 0; i < 8; i++) s_t[i * 32 + lane][wid] = transpose32(v[i], lane);
      __syncthreads();
      const u32 *q = s_t[threadIdx.x];
      u32 d[8];
      load8(dst + dw, d);
#pragma unroll
      for (int i = 0; i < 8; i++) d[i] |= q[i];
      pd[0] = make_uint4(d[0], d[1], d[2], d[3]);
      pd[1] = make_uint4(d[4], d[5], d[6], d[7]);
    }
  }
}

// dst := transpose(src), its bits added to *count_acc if set.
__device__ __forceinline__ void loop_transpose(const u32 *src, u32 *dst, u64 *count_acc, int rs,
                                               u32 side, u32 block, u32 (*s_t)[9]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  u32 bits = 0;
  for (u32 t = block; t < side * side; t += gridDim.x) {
    const u32 tr = t / side, tc = t % side;
    u32 v[8];
    load8(src + ((((u64)tr * 256 + threadIdx.x) << rs) + tc * 8), v);
    bool any = false;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      any |= v[i] != 0u;
      bits += __popc(v[i]);
    }
    uint4 *pd = reinterpret_cast<uint4 *>(dst + ((((u64)tc * 256 + threadIdx.x) << rs) + tr * 8));
    if (__syncthreads_or(any)) {
#pragma unroll
      for (int i = 0; i < 8; i++) s_t[i * 32 + lane][wid] = transpose32(v[i], lane);
      __syncthreads();
      const u32 *q = s_t[threadIdx.x];
      pd[0] = make_uint4(q[0], q[1], q[2], q[3]);
      pd[1] = make_uint4(q[4], q[5], q[6], q[7]);
    } else {
      pd[0] = make_uint4(0, 0, 0, 0);
      pd[1] = make_uint4(0, 0, 0, 0);
    }
  }
  if (count_acc) {
    bits = __reduce_add_sync(0xffffffffu, bits);
    if (lane == 0 && bits)
      atomicAdd(reinterpret_cast<unsigned long long *>(count_acc), (unsigned long long)bits);
  }
  __syncthreads();  // (s_t may be the next step's)
}

// src/join.cu:42-45: an empty inner zeroes the outer's count ...
__device__ __forceinline__ void loop_empty_inner(const LoopStep &st) {
  if (st.outer_vis)
    *st.outer_vis = 0;
  else
    const_cast<DArr *>(st.outer)->n = 0;
}
// ... and the bitmap of a NEWT outer.
__device__ __forceinline__ void loop_clear(const LoopStep &st) {
  uint4 *p = reinterpret_cast<uint4 *>(st.outer_bm);
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < st.outer_words / 4;
       i += (u64)gridDim.x * blockDim.x)
    p[i] = make_uint4(0, 0, 0, 0);
}

// One tile of k_bm_update_t's pass (pull.cuh): DELTA = NEWT & ~FULL written
// as u asks, FULL |= NEWT, NEWT cleared.  A tile without NEWT bits only
// clears what its DELTA tiles still hold.
__device__ __forceinline__ void loop_update_tile(const LoopUpd &u, int rs, u32 tr, u32 tc,
                                                 u32 side, u32 (*s_t)[9], u32 &n_delta,
                                                 u32 &n_newt) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const u64 src = (((u64)tr * 256 + tid) << rs) + tc * 8;
  const u64 mir = (((u64)tc * 256 + tid) << rs) + tr * 8;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  u32 *np = u.gt ? u.gt + mir : u.G + src;
  u32 v[8];
  load8(np, v);
  const bool clean = u.rd && u.clean[tr * side + tc];
  const bool any_v = (v[0] | v[1] | v[2] | v[3] | v[4] | v[5] | v[6] | v[7]) != 0u;
  if (any_v) {
    reinterpret_cast<uint4 *>(np)[0] = zero;
    reinterpret_cast<uint4 *>(np)[1] = zero;
  }
  if (!u.rd) return;  // a tmp NEWT (uniform over the launch)
  // (also orders the last tile's reads of s_t, and the reads of `clean`)
  if (!__syncthreads_or(any_v)) {
    if (!clean) {
      if (u.dn) {
        reinterpret_cast<uint4 *>(u.dn + src)[0] = zero;
        reinterpret_cast<uint4 *>(u.dn + src)[1] = zero;
      }
      if (u.dt) {
        reinterpret_cast<uint4 *>(u.dt + mir)[0] = zero;
        reinterpret_cast<uint4 *>(u.dt + mir)[1] = zero;
      }
      if (tid == 0) u.clean[tr * side + tc] = 1;
    }
    return;
  }
  u32 f[8];
  load8(u.F + src, f);
  if (u.gt) {
#pragma unroll
    for (int i = 0; i < 8; i++) s_t[i * 32 + lane][wid] = transpose32(v[i], lane);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = s_t[tid][i];
  }
  bool any_d = false;
  u32 d[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    d[i] = v[i] & ~f[i];
    any_d |= d[i] != 0u;
    n_delta += __popc(d[i]);
    n_newt += __popc(v[i]);
    f[i] |= v[i];
  }
  if (any_d) {
    reinterpret_cast<uint4 *>(u.F + src)[0] = make_uint4(f[0], f[1], f[2], f[3]);
    reinterpret_cast<uint4 *>(u.F + src)[1] = make_uint4(f[4], f[5], f[6], f[7]);
  }
  const bool tile_d = __syncthreads_or(any_d);  // (and the reads of s_t above)
  if (!tile_d && clean) return;
  if (u.dn) {
    reinterpret_cast<uint4 *>(u.dn + src)[0] = make_uint4(d[0], d[1], d[2], d[3]);
    reinterpret_cast<uint4 *>(u.dn + src)[1] = make_uint4(d[4], d[5], d[6], d[7]);
  }
  if (u.dt) {
    if (tile_d) {
#pragma unroll
      for (int i = 0; i < 8; i++) s_t[i * 32 + lane][wid] = transpose32(d[i], lane);
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 8; i++) d[i] = s_t[tid][i];
    }
    reinterpret_cast<uint4 *>(u.dt + mir)[0] = make_uint4(d[0], d[1], d[2], d[3]);
    reinterpret_cast<uint4 *>(u.dt + mir)[1] = make_uint4(d[4], d[5], d[6], d[7]);
  }
  if (tid == 0) u.clean[tr * side + tc] = !tile_d;
}

// V: as k_join_rows_bm; 0 below 2^12 ids, where joins are products.
template <int V>
__global__ void __launch_bounds__(kLoopBlock, 2) k_lie_loop(LoopArgs a) {
  __shared__ u32 s_t[256][9];
  __shared__ LoopStep s_step[kLoopMaxSteps];
  __shared__ LoopUpd s_upd[kLoopMaxUpd];
  __shared__ int s_go;
  Ctl *ctl = a.ctl;
  u32 gen = ctl->bar_word >> 2;  // (it cannot change before this block arrives)
  bool go = !ctl_stop(ctl);
  const int rs = a.dk - 5;
  const LaneLists lists = lane_lists(a.lie, threadIdx.x & 31);
  for (u32 i = threadIdx.x; i < a.n_steps * sizeof(LoopStep) / 4; i += kLoopBlock)
    reinterpret_cast<u32 *>(s_step)[i] = reinterpret_cast<const u32 *>(a.steps)[i];
  for (u32 i = threadIdx.x; i < a.n_upd * sizeof(LoopUpd) / 4; i += kLoopBlock)
    reinterpret_cast<u32 *>(s_upd)[i] = reinterpret_cast<const u32 *>(a.upd)[i];
  __syncthreads();
  // (a block's number differs from step to step, so that steps with little
  // work do not all fall to the first blocks)
  auto block_for = [&](u32 i) { return (blockIdx.x + i * 61u) % gridDim.x; };
  while (go) {
    // Products whose inner is empty, by step.  Inners are FULLs that only the
    // commit changes, so the iteration's first level looks at all of them.  An
    // empty inner zeroes its outer's DELTA for the operators after its own
    // (src/join.cu:42-45): levels reorder steps, so each step knows which
    // operators those are (LoopStep::before).
    u64 no_inner = 0;
    for (int i = 0; i < a.n_steps && go;) {
      // the steps of one level; lane k looks at the outer of the k-th (the
      // loads take one round trip together)
      const int i0 = i, i1 = s_step[i0].level_end;
      u32 no_outer = 0;
      if (V == 0) {
        const int lane = threadIdx.x & 31;
        bool ni[2] = {false, false}, no = false;
        if (i0 == 0) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const LoopStep &st = s_step[lane + 32 * h];
            if (lane + 32 * h < a.n_steps && st.kind == kLoopProduct)
              ni[h] = eff_count(st.inner, st.inner_vis) == 0;
          }
        }
        if (i0 + lane < i1) {
          const LoopStep &st = s_step[i0 + lane];
          if (st.kind == kLoopProduct) no = eff_count(st.outer, st.outer_vis) == 0;
        }
        if (i0 == 0)
          no_inner = __ballot_sync(0xffffffffu, ni[0]) |
                     ((u64)__ballot_sync(0xffffffffu, ni[1]) << 32);
        no_outer = __ballot_sync(0xffffffffu, no);
      }
      for (; i < i1; i++) {
        const LoopStep &st = s_step[i];
        if (st.kind == kLoopRows) {
          if (V > 0) {
            RowsArgs ra;
            ra.j.outer = st.outer;
            ra.j.outer_vis = st.outer_vis;
            ra.j.inner = st.inner;
            ra.j.inner_vis = st.inner_vis;
            ra.j.ctl = nullptr;
            ra.j.once = st.once;
            ra.j.once_pending = st.once_pending;
            ra.j.produced = st.produced;
            ra.j.phantom = st.phantom;
            ra.O = st.src;
            ra.outer_clear = st.outer_bm;
            ra.outer_words = st.outer_words;
            ra.inv_keys = st.inv_keys;
            ra.inv_ys = st.inv_ys;
            ra.inv_off = nullptr;
            ra.n_edges = st.n_edges;
            ra.unit = st.unit;
            ra.dst = st.dst;
            ra.dirty = nullptr;
            ra.dst_zero = st.dst_zero;
            ra.clear_diag = st.clear_diag;
            ra.dk = a.dk;
            if (st.n_edges)
              join_rows<V == 0 ? 1 : V>(ra);
            else if (blockIdx.x == 0 && threadIdx.x == 0)
              loop_empty_inner(st);
            if (!st.n_edges && st.outer_bm) loop_clear(st);
          }
        } else if (st.kind == kLoopProduct) {
          if (V == 0) {
            if ((no_inner >> i) & 1ull) {
              if (!st.outer_vis) loop_clear(st);  // (its count: by the barrier)
            } else if (!((no_outer >> (i - i0)) & 1u) && !(no_inner & st.before)) {
              ProdArgs pa;
              pa.j.ctl = nullptr;
              pa.OT = st.src;
              pa.F = st.F;
              pa.G = st.dst;
              pa.dirty = nullptr;
              pa.dk = a.dk;
              pa.side = a.side;
              pa.splits = a.splits;
              product_small(pa, block_for(i));
            }
          }
        } else if (st.kind == kLoopTranspose) {
          loop_transpose(st.src, st.dst, st.count_to ? st.count_acc : nullptr, rs, a.side,
                         block_for(i), s_t);
        } else {
          loop_fold(const_cast<u32 *>(st.src), st.dst, rs, a.side, block_for(i), s_t);
        }
      }
      go = loop_barrier(ctl, gen, &s_go, [&](int lane) {
        for (int k = i0 + lane; k < i1; k += 32) {
          const LoopStep &st = s_step[k];
          if (st.kind == kLoopTranspose && st.count_to) {
            st.count_to->n = *st.count_acc;
            *st.count_acc = 0;
          }
          if (((no_inner >> k) & 1ull) && !st.outer_vis) loop_empty_inner(st);
        }
        return false;
      });
    }
    if (!go) break;
    // the update step of every relation
    const u32 tiles = a.side * a.side;
    for (int r = 0; r < a.n_upd; r++) {
      const LoopUpd u = s_upd[r];
      u32 nd = 0, nn = 0;
      for (u32 t = block_for(r); t < tiles; t += gridDim.x)
        loop_update_tile(u, rs, t / a.side, t % a.side, a.side, s_t, nd, nn);
      if (!u.rd) continue;
      nd = __reduce_add_sync(0xffffffffu, nd);
      nn = __reduce_add_sync(0xffffffffu, nn);
      if ((threadIdx.x & 31) == 0) {
        if (nd) atomicAdd((unsigned long long *)&u.rd->scan.total_a, (unsigned long long)nd);
        if (nn) atomicAdd((unsigned long long *)&u.rd->scan.pop_g, (unsigned long long)nn);
      }
    }
    go = loop_barrier(ctl, gen, &s_go, [&](int lane) {
      return loop_commit<false>(a.rels, a.lie, ctl, lists, lane);
    });
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && ctl->cond_set)
    cudaGraphSetConditional((cudaGraphConditionalHandle)ctl->cond_handle, 0u);
}

}  // namespace gdl
