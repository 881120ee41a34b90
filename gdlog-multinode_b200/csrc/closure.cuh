// closure.cuh — linear recursion over a static relation, one pass an iteration.
//
// A LIE whose one operator is  P(x, z) :- E(y, x), P(y, z)  (output (inner
// column 1, outer column 1), inner a static FULL, outer P's DELTA; test/tc.cu:
// 61-78) makes row x of the next DELTA from the DELTA rows of x's sources:
//     DELTA'[x] = (OR over (y, x) in E of DELTA[y]) & ~FULL[x];  FULL[x] |= DELTA'[x]
// so a join, a NEWT bitmap, an update pass and a commit are one pass over
// rows, each row owned by one group of lanes, without atomics.  Two DELTA
// bitmaps alternate.  Each row of DELTA has an extent, the words between its
// first and last bit: only those are read and written, and nothing is ever
// cleared (a word outside the extent is never read).  On layered graphs a
// row's DELTA is one layer wide: the 384-DAG batch reads 200 bytes an active
// row and iteration, where the scans read 1.8 GB of bitmap and the join
// expanded every candidate tuple (122 ms a batch).
//
// The loop is resident (loop.cuh): one grid barrier an iteration.  A warp
// looks at up to 32 rows at once (a lane a row: its sources' extents), then
// takes the rows with something to do: four at a time by eight lanes each
// (their loads overlap), a single one with a long extent by all lanes.  A row
// with many sources is one warp's serial work, so in-degrees are bounded by
// kClosureMaxDegree; beyond it the edge-balanced join (pull.cuh,
// k_join_rows_bm) runs instead.
//
// Both layouts: the square domain (row x at x << rs) and the batched form's
// block diagonal (rows numbered through all instances).
#pragma once

#include "common.cuh"
#include "dense.cuh"
#include "index.cuh"
#include "loop.cuh"

namespace gdl {

constexpr u32 kClosureMaxDegree = 64;
constexpr u32 kClosureLongExtent = 32;  // words from which a lone row takes a warp
constexpr u32 kNoWord = 0xFFFFFFFFu;
constexpr int kClosureCtasPerSm = 3;

struct ClosureArgs {
  const u32 *start, *end;  // per row: its sources are adj[start .. end)
  const u32 *adj;
  const u32 *row_word;     // per row: its first word; null: row << rs
  const u32 *row_inst;     // per row: its instance; null: not batched
  u64 *inst_last;          // per instance: last iteration (+1) with new tuples
  u32 *F;
  u32 *D[2];
  uint2 *ext[2];           // per row: words [x, y) of D hold its bits
  u32 rows, chunk;         // chunk: rows a warp looks at together (4 .. 32)
  int rs;
  RelDev *rd;
  LoopArgs loop;           // for the commit
};

__device__ __forceinline__ u32 closure_word(const ClosureArgs &a, u32 row) {
  return a.row_word ? a.row_word[row] : row << a.rs;
}

// One row by the lanes of a group of G (lane gl of it); on: the group has a
// row.  Returns the row's new tuples counted by this lane; *found: this lane
// met a tuple, new or not.  All 32 lanes call it.
template <int G>
__device__ __forceinline__ u32 closure_row(const ClosureArgs &a, bool on, u32 row, u32 s, u32 e,
                                           u32 lo, u32 hi, const u32 *Dc, u32 *Dn,
                                           const uint2 *ec, uint2 *en, u64 it, bool *found) {
  const u32 gl = threadIdx.x & (G - 1);
  constexpr int kPre = 4;  // sources held in registers
  const u32 *src[kPre];
  uint2 x[kPre];
#pragma unroll
  for (int j = 0; j < kPre; j++) {
    src[j] = Dc;
    x[j] = make_uint2(kNoWord, 0);
    if (on && s + j < e) {
      const u32 k = a.adj[s + j];
      x[j] = ec[k];
      src[j] = Dc + closure_word(a, k);
    }
  }
  const u32 rw = on ? closure_word(a, row) : 0u;
  u32 nlo = kNoWord, nhi = 0, cnt = 0;
  if (on) {
#pragma unroll 4
    for (u32 w = lo + gl; w < hi; w += G) {
      const u32 f = a.F[rw + w];
      u32 v = 0;
#pragma unroll
      for (int j = 0; j < kPre; j++)
        if (w >= x[j].x && w < x[j].y) v |= src[j][w];
      for (u32 j = s + kPre; j < e; j++) {
        const u32 k = a.adj[j];
        const uint2 y = ec[k];
        if (w >= y.x && w < y.y) v |= Dc[closure_word(a, k) + w];
      }
      const u32 d = v & ~f;
      Dn[rw + w] = d;
      if (v) *found = true;
      if (d) {
        a.F[rw + w] = f | d;
        cnt += __popc(d);
        nlo = min(nlo, w);
        nhi = max(nhi, w + 1);
      }
    }
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    nlo = min(nlo, __shfl_xor_sync(0xffffffffu, nlo, o));
    nhi = max(nhi, __shfl_xor_sync(0xffffffffu, nhi, o));
  }
  if (on && gl == 0) {
    en[row] = make_uint2(nlo, nhi);
    if (a.row_inst && nhi) {
      u64 *last = a.inst_last + a.row_inst[row];
      if (*last != it + 1) *last = it + 1;
    }
  }
  return cnt;
}

__global__ void __launch_bounds__(kLoopBlock, kClosureCtasPerSm) k_closure_loop(ClosureArgs a) {
  __shared__ int s_go;
  Ctl *ctl = a.loop.ctl;
  u32 gen = ctl->bar_word >> 2;
  bool go = !ctl_stop(ctl);
  const int lane = threadIdx.x & 31;
  const LaneLists lists = lane_lists(a.loop.lie, lane);
  const u32 nw = gridDim.x * (kLoopBlock / 32);
  const u32 wid = blockIdx.x * (kLoopBlock / 32) + (threadIdx.x >> 5);
  while (go) {
    const u64 it = ctl->iteration;
    const int cur = (int)(it & 1);
    const uint2 *ec = a.ext[cur];
    uint2 *en = a.ext[cur ^ 1];
    const u32 *Dc = a.D[cur];
    u32 *Dn = a.D[cur ^ 1];
    u64 n_new = 0;
    bool found = false;
    for (u32 c = wid; (u64)c * a.chunk < a.rows; c += nw) {
      const u32 base = c * a.chunk, r = base + lane;
      u32 s = 0, e = 0, lo = kNoWord, hi = 0;
      if (lane < (int)a.chunk && r < a.rows) {
        s = a.start[r];
        e = a.end[r];
        for (u32 j = s; j < e; j++) {
          const uint2 x = ec[a.adj[j]];
          lo = min(lo, x.x);
          hi = max(hi, x.y);
        }
        if (hi == 0) en[r] = make_uint2(kNoWord, 0);
      }
      u32 todo = __ballot_sync(0xffffffffu, hi != 0);
      if (__popc(todo) == 1 && __any_sync(0xffffffffu, hi != 0 && hi - lo > kClosureLongExtent)) {
        const int q = __ffs(todo) - 1;
        todo = 0;
        n_new += closure_row<32>(a, true, base + q, __shfl_sync(0xffffffffu, s, q),
                                 __shfl_sync(0xffffffffu, e, q), __shfl_sync(0xffffffffu, lo, q),
                                 __shfl_sync(0xffffffffu, hi, q), Dc, Dn, ec, en, it, &found);
      }
      while (todo) {
        // group g takes the g-th row left
        int q = 0;
        bool on = false;
        u32 rest = todo;
#pragma unroll
        for (int g = 0; g < 4; g++) {
          if (rest && g == lane >> 3) {
            q = __ffs(rest) - 1;
            on = true;
          }
          rest &= rest - 1;  // (0 stays 0)
        }
        todo = rest;
        n_new += closure_row<8>(a, on, base + q, __shfl_sync(0xffffffffu, s, q),
                                __shfl_sync(0xffffffffu, e, q), __shfl_sync(0xffffffffu, lo, q),
                                __shfl_sync(0xffffffffu, hi, q), Dc, Dn, ec, en, it, &found);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n_new += __shfl_xor_sync(0xffffffffu, n_new, o);
    if (lane == 0 && n_new)
      atomicAdd((unsigned long long *)&a.rd->scan.total_a, (unsigned long long)n_new);
    if (__any_sync(0xffffffffu, found) && lane == 0) a.rd->scan.pop_g = 1;  // NEWT is not empty
    go = loop_barrier(ctl, gen, &s_go,
                      [&](int ln) {
                        return loop_commit<false>(a.loop.rels, a.loop.lie, ctl, lists, ln);
                      });
  }
  if (blockIdx.x == 0 && threadIdx.x == 0 && ctl->cond_set)
    cudaGraphSetConditional((cudaGraphConditionalHandle)ctl->cond_handle, 0u);
}

// Setup ---------------------------------------------------------------------

// The batched form's rows: instance i owns rows row_first[i] .. + n of them.
struct ClosureRows {
  const SegInfo *seg;
  const u32 *row_first;
  u32 n_inst;
  int shift;  // ids are instance << shift | local
};
// The row of an id; kNoWord when it lies in no instance.
__device__ __forceinline__ u32 closure_row_of(const ClosureRows &m, u32 id) {
  if (!m.row_first) return id;
  const u32 i = id >> m.shift, x = id & ((1u << m.shift) - 1u);
  return i < m.n_inst && x < m.seg[i].n ? m.row_first[i] + x : kNoWord;
}

// Whether both columns lie in one instance.
__device__ __forceinline__ bool closure_inside(const ClosureRows &m, u64 k) {
  return !m.row_first || (((key_c0(k) ^ key_c1(k)) >> m.shift) == 0 &&
                          closure_row_of(m, key_c0(k)) != kNoWord &&
                          closure_row_of(m, key_c1(k)) != kNoWord);
}

__global__ void __launch_bounds__(256) k_closure_rows(ClosureRows m, u32 *row_word, u32 *row_inst) {
  for (u32 i = blockIdx.x; i < m.n_inst; i += gridDim.x) {
    const SegInfo s = m.seg[i];
    for (u32 x = threadIdx.x; x < s.n; x += blockDim.x) {
      row_word[m.row_first[i] + x] = (u32)s.base_word + (x << s.row_shift);
      row_inst[m.row_first[i] + x] = i;
    }
  }
}

// Column-swapped keys of a list (to be sorted by column 1).
__global__ void __launch_bounds__(256) k_closure_swap(const DArr *list, u64 *out) {
  const u64 n = list->n;
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x) {
    const u64 k = list->ptr[i];
    out[i] = (k << 32) | (k >> 32);
  }
}

// Sources per row, and the most of one row (both zero before).  An edge out of
// the instances or between two of them is written to *bad: the general path
// runs, whose bit-sets report it.
__global__ void __launch_bounds__(256) k_closure_count(const u64 *edges, u64 n, ClosureRows m,
                                                       u32 *count, u32 *most, u32 *bad) {
  u32 mx = 0;
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x) {
    if (closure_inside(m, edges[i]))
      mx = max(mx, atomicAdd(&count[closure_row_of(m, key_c1(edges[i]))], 1u) + 1);
    else
      *bad = 1;
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(most, mx);
}

// From keys (row id, source id) sorted: adj, and each row's range (rows
// without sources keep start = end = 0).
__global__ void __launch_bounds__(256) k_closure_adj(const u64 *keys, u64 n, ClosureRows m,
                                                     u32 *start, u32 *end, u32 *adj) {
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x) {
    const u64 k = keys[i];
    const u32 row = closure_row_of(m, key_c0(k));
    adj[i] = closure_row_of(m, key_c1(k));
    if (i == 0 || key_c0(keys[i - 1]) != key_c0(k)) {
      start[row] = (u32)i;
      end[row] = (u32)run_end(keys, n, i);
    }
  }
}

__global__ void __launch_bounds__(256) k_closure_degree(const u32 *start, const u32 *end, u32 rows,
                                                        u32 *max_degree) {
  u32 m = 0;
  for (u32 r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x)
    m = max(m, end[r] - start[r]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(max_degree, m);
}

// The first DELTA's tuples out of the instances or between two: as bad edges.
__global__ void __launch_bounds__(256) k_closure_check(const u64 *keys, u64 n, ClosureRows m,
                                                       u32 *bad) {
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x)
    if (!closure_inside(m, keys[i])) *bad = 1;
}

// The first DELTA: extents of its rows, those words zeroed, then the bits
// set (k_bm_from_list).
__global__ void __launch_bounds__(256) k_closure_ext(const DArr *list, ClosureRows m, uint2 *ext) {
  const u64 n = list->n;
  for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (u64)gridDim.x * blockDim.x) {
    const u64 k = list->ptr[i];
    if (!closure_inside(m, k)) continue;  // (no extent past its row)
    const u32 r = closure_row_of(m, key_c0(k));
    const u32 c = m.row_first ? key_c1(k) & ((1u << m.shift) - 1u) : key_c1(k);
    atomicMin(&ext[r].x, c >> 5);
    atomicMax(&ext[r].y, (c >> 5) + 1);
  }
}
__global__ void __launch_bounds__(256) k_closure_ext_init(uint2 *e0, uint2 *e1, u32 rows) {
  for (u32 r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
    e0[r] = make_uint2(kNoWord, 0);
    e1[r] = make_uint2(kNoWord, 0);
  }
}
__global__ void __launch_bounds__(256) k_closure_zero(ClosureArgs a) {
  const int lane = threadIdx.x & 31;
  for (u32 r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < a.rows;
       r += (gridDim.x * blockDim.x) >> 5) {
    const uint2 x = a.ext[0][r];
    const u32 rw = closure_word(a, r);
    for (u32 w = x.x + lane; w < x.y; w += 32) a.D[0][rw + w] = 0;
  }
}

}  // namespace gdl
