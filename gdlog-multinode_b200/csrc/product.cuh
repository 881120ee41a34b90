// product.cuh — joins into bitmaps as boolean matrix products.
//
// A pull-form join (pull.cuh: output (outer column 1, inner column 1), or
// its transpose, joined on column 0) over an inner FULL kept as a bitmap is
// the boolean product  Out[x] |= OR over k of OT[x][k] & F[k]:  the outer
// transposed (row x, bit k) times the inner's rows.  Points-to analysis
// (test/cspa.cu:279-352) spends its time in nine such products of relations
// that fill a fifth to nine tenths of their domain; listing the inner,
// indexing it and expanding candidate tuples cost 11 ms a join at 20,000
// ids.  Here no list and no index exist.
//
// k_join_product: a block owns MR output rows by a slice of 1024 columns (a
// word a lane, MR / 32 rows a warp, accumulated in registers) and walks the
// keys 32 at a time.  Per 32 keys (one word of each row of OT), by the bits
// its rows hold:
//   * many: the four-Russians method (Arlazarov, Dinic, Kronrod, Faradzev
//     1970).  For each of the word's four bytes the 256 ORs of its eight
//     inner rows are tabled in shared memory (1024 entries of 128 bytes,
//     built from registers, a store an entry), and a row takes four table
//     reads instead of one read per key.
//   * few: the row's keys one by one from the inner rows staged in shared
//     memory, rows without a key skipped by a ballot.
//   * none, or no inner row with bits in the slice: skipped.
// The bound is shared-memory bandwidth, one 128-byte read a row and byte of
// keys, so MR = 1024 rows share a table (its 1024 stores are a fifth of the
// 4096 + 512 reads).  The integer pipe comes second: the outer's words are
// staged as their bytes' table offsets (two a word, byte * 128), so an
// address is one instruction, and rows are taken four at a time without a
// branch.  The next 256 keys' operands load (cp.async for the inner's rows,
// registers for the outer's words) while these are used.
//
// k_join_product_rows: a row of few keys would leave that kernel scanning
// empty words for every slice.  A block takes 8 rows of OT, lists their keys
// in shared memory and its warps OR equal shares of the listed inner rows,
// whole rows at a time, at L2's rate (6 TB/s: 0.4 ns a key at 20,000 ids,
// where a row costs the tables 350 ns however many keys it has).
// Both run: k_prod_rows counts each row's keys and lists the long ones, and by
// those counts both kernels decide which rows k_join_product takes (points-to
// relations are reflexive, so half the rows hold a few keys and the others
// thousands; 20,000 variables: 260 -> 195 ms).
//
// A tmp NEWT outer (points-to's two-step rule) is derived anew in every
// iteration, mostly the tuples of the iteration before: joined with all of
// FULL then, and their results are in the output's FULL now.  So with few
// fresh tuples only those are joined with FULL, and the whole NEWT with the
// inner's DELTA (as the product the other way round: its few rows against
// NEWT's), semi-naive within the rule.  The transpose that makes OT keeps the
// last one's to compare with; the device decides by the counts.  Late
// iterations at 20,000 variables: 6.5 -> 0.5 to 1.2 ms a product.
//
// product_small: below 2^kProdTableBits ids there are too few rows to fill
// the GPU with tables.  A warp takes one output row and a share of its keys
// and ORs the inner's rows straight from L1 / L2, four keys' loads in flight
// (at 512 ids two keys a load instruction, at 256 four).
#pragma once

#include "common.cuh"
#include "dense.cuh"
#include "join.cuh"

namespace gdl {

constexpr int kProdBlock = 1024;
constexpr int kProdWarps = kProdBlock / 32;
constexpr int kProdStep = 256;       // keys per staged step: 8 words of a row
constexpr int kProdTableBits = 12;   // tables from 2^12 ids on
// Output rows per warp: 32 warps of 32 rows, not 16 of 64 (the same 1024
// accumulators a lane column), halve the unrolled code a warp runs through
// (instruction fetch was a tenth of its stalls) and double the warps that
// hide the reads' latency.
constexpr int kProdWarpRows = 32;
constexpr u32 kProdRows = kProdWarps * kProdWarpRows;  // per block
constexpr u32 kProdUnits = 6;        // units of work a block, at least
constexpr int kProdPart = 4;         // words of a step staged together
// Which rows the tables take, decided on the device from what k_prod_rows
// counts: the rows with a 64th of the ids or more (long), those with an eighth
// or more (full; a sixteenth once the inner's bitmap is beyond L2), or none.
// The costs compared are in keys listed (k_join_product_rows reads a row of
// the inner a key).  Points-to, ms with every long row in the tables / now
// (variables, facts a variable; in brackets before there were products):
//    2,100, 0.8:  10.4 /  6.2  (7.6)        8,100, 2.75:  20.5 / 20.2  (100)
//    3,000, 0.55: 11.2 /  7.2  (8.7)       12,000, 0.8:   27.8 / 21.1  (46)
//    4,000, 2.75:  8.1 /  7.6  (34)        16,300, 0.8:   46.2 / 36.2  (62)
//    6,000, 0.8:  13.2 /  9.5  (15.3)      20,000, 2.75:   172 / 166   (1109)
constexpr u32 kProdLong = 64;
__device__ __forceinline__ u32 prod_full_part(int dk) { return dk <= 14 ? 8u : 16u; }
__device__ __forceinline__ bool prod_reaches(u32 keys, u32 part, u32 side) {
  return keys * part >= side * 256;
}
// ProdArgs::list: the counts of the full rows and of the long ones, their keys
// (in 32s), then the rows themselves.
enum ProdKind : u32 { kProdFullRows = 0, kProdLongRows = 1, kProdNone = 2 };
constexpr u32 kProdListHead = 4, kProdListRows = 1u << 16;
__host__ __device__ constexpr u32 prod_list_at(u32 kind) {
  return kProdListHead + kind * kProdListRows;
}
constexpr u32 kProdListWords = kProdListHead + 2 * kProdListRows;
// The units of work of n rows in the tables: row blocks by column slices by
// key ranges.  The key range is split until there are kProdUnits units a
// block: at 20,000 ids 400 row-by-column blocks share 148 SMs unevenly (3
// rounds for 2.7), and few long rows are few blocks.
struct ProdSplit {
  u32 n_rb, n_sl, ksteps, n_kc;
};
__device__ __forceinline__ ProdSplit prod_split(u32 n, u32 side, u32 sms) {
  ProdSplit x;
  x.n_rb = (n + kProdRows - 1) / kProdRows;
  x.n_sl = (side + 3) / 4;
  x.ksteps = max(2u, side * x.n_rb * x.n_sl / (kProdUnits * sms));
  x.n_kc = (side + x.ksteps - 1) / x.ksteps;
  return x;
}
// What n rows cost in the tables, in 32 listed keys.  A block of 1024 rows
// takes 4.3 us a word of keys and slice, a fifth of it to build the tables, and
// a listed key side x 5.3 ps (20,000 ids: 0.42 ns; 840 keys a row are the
// same).  Fewer units than SMs cost as many times more.  (Whole numbers, so
// that both kernels decide alike; 32 bits hold them: units are fewer than SMs
// below 2^14 ids only.)
__device__ __forceinline__ u32 prod_table_cost(u32 n, u32 side, u32 sms) {
  const ProdSplit x = prod_split(n, side, sms);
  const u32 units = x.n_rb * x.n_sl * x.n_kc;
  const u32 keys = side * (68 * x.n_rb + 17 * n / 64);
  return units - 1 < sms - 1 ? keys * sms / units : keys;
}
__device__ __forceinline__ u32 prod_kind(const u32 *list, u32 side, u32 sms) {
  // (reset by the second kernel's last block, when all have read them)
  const uint4 c = *reinterpret_cast<const uint4 *>(list);
  const u32 all = prod_table_cost(c.y, side, sms);
  const u32 full = prod_table_cost(c.x, side, sms) + (c.w - c.z);
  return c.w <= min(all, full) ? kProdNone : full < all ? kProdFullRows : kProdLongRows;
}
// Dynamic shared memory: the tables, two stages of 256 inner row slices, and
// kProdPart of a step's 8 outer words, as two words each.
constexpr u32 kProdSmem = 4 * 256 * 128 + 2 * kProdStep * 128 + 2 * kProdPart * kProdRows * 4;

struct ProdArgs {
  JoinArgs j;      // descriptors for the emptiness rules, launch record, ctl
  const u32 *OT;   // the outer, transposed
  const u32 *F;    // the inner's rows
  u32 *G;          // output rows: the output's NEWT or its transposed twin
  u8 *dirty;       // dirty map of G, or null
  LaunchRec *rows_rec;  // launch record of k_join_product_rows
  u32 *list;       // long rows of OT (prod_kind, prod_list_at)
  u32 sms;         // blocks of k_join_product
  int dk;          // rows of 2^(dk-5) words
  u32 side;        // 256-id groups that hold ids
  // Repeated outer: the fresh part of OT and its size; part 1 takes it in
  // place of OT when it is small, part 2 (OT the inner's DELTA, F NEWT's rows)
  // runs in that case only.  0: neither.
  int part;
  const u32 *OT_fresh;
  const u64 *n_fresh;
  const DArr *newt, *delta;  // the outer, and the inner's DELTA
  u32 splits;      // product_small: warps a row's keys are shared among
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src, u32 bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (u32)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}

// The two parts against the whole: by their tuples, with room for what they
// cost beyond that (at 20,000 variables: 8.2 ms for 6.6 where a tenth of NEWT
// was fresh or DELTA, 1.2 for 6.6 at a fiftieth).
__device__ __forceinline__ bool prod_few_fresh(const ProdArgs &a) {
  return a.part && (*a.n_fresh + a.delta->n) * 16 <= a.newt->n;
}
// The outer a launch reads, null when there is nothing for it to do.
__device__ __forceinline__ const u32 *prod_outer(const ProdArgs &a) {
  if (a.part == 0) return a.OT;
  const bool few = prod_few_fresh(a);
  if (a.part == 1) return few ? a.OT_fresh : a.OT;
  return few && a.j.outer->n && a.j.inner->n ? a.OT : nullptr;
}

// src/join.cu:38-45 for a product: an empty inner empties the OUTER (every
// block calls this; a NEWT outer's bitmap is cleared too).  Returns whether
// there is nothing to join.  The inner is looked at first: no block reads
// the outer's count while block 0 may be zeroing it.
__device__ __forceinline__ bool product_empty(const JoinArgs &j, u64 *n_outer) {
  if (eff_count(j.inner, j.inner_vis) == 0) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      if (j.outer_vis)
        *j.outer_vis = 0;
      else
        ((DArr *)j.outer)->n = 0;
    }
    if (!j.outer_vis && j.outer_bm) {
      uint4 *p = reinterpret_cast<uint4 *>(j.outer_bm);
      for (u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x; i < j.outer_bm_words / 4;
           i += (u64)gridDim.x * blockDim.x)
        p[i] = make_uint4(0, 0, 0, 0);
    }
    return true;
  }
  *n_outer = eff_count(j.outer, j.outer_vis);
  return *n_outer == 0;
}

// The full and the long rows of OT, listed for k_join_product
// (k_join_product_rows sets the counts back to zero), nearly in order: 32 rows
// a block, two atomics a list.
__global__ void __launch_bounds__(256) k_prod_rows(ProdArgs a) {
  __shared__ u32 s_keys[32];
  if (ctl_stop(a.j.ctl)) return;
  const u64 n_outer = eff_count(a.j.outer, a.j.outer_vis);
  if (n_outer == 0 || eff_count(a.j.inner, a.j.inner_vis) == 0) return;
  const u32 *OT = prod_outer(a);
  if (!OT) return;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const u32 n4 = a.side * 2;
  for (u32 g = blockIdx.x; g < a.side * 8; g += gridDim.x) {
    __syncthreads();
    // this warp's four rows
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint4 *p =
          reinterpret_cast<const uint4 *>(OT + ((u64)(g * 32 + wid * 4 + q) << (a.dk - 5)));
      u32 keys = 0;
      for (u32 i = lane; i < n4; i += 32) {
        const uint4 v = p[i];
        keys += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
      }
      keys = __reduce_add_sync(0xffffffffu, keys);
      if (lane == 0) s_keys[wid * 4 + q] = keys;
    }
    __syncthreads();
    if (wid < 2) {  // a warp a list, a row a lane
      const u32 keys = s_keys[lane];
      const bool on = prod_reaches(keys, wid ? kProdLong : prod_full_part(a.dk), a.side);
      const u32 b = __ballot_sync(0xffffffffu, on);
      const u32 sum = __reduce_add_sync(0xffffffffu, on ? keys / 32 : 0u);
      u32 base = 0;
      if (lane == 0 && b) {
        base = atomicAdd(&a.list[wid], (u32)__popc(b));
        atomicAdd(&a.list[2 + wid], sum);
      }
      base = __shfl_sync(0xffffffffu, base, 0);
      if (on)
        a.list[prod_list_at(wid) + base + __popc(b & ((1u << lane) - 1u))] = g * 32 + lane;
    }
  }
}

__global__ void __launch_bounds__(kProdBlock, 1) k_join_product(ProdArgs a) {
  constexpr int RW = kProdWarpRows;
  constexpr u32 MR = kProdRows;
  static_assert(MR == kProdBlock, "a thread loads one outer row");
  constexpr u32 kNoRow = 0xFFFFFFFFu;
  constexpr int kPart = kProdPart;
  extern __shared__ __align__(128) u32 prod_mem[];
  u32 *tab = prod_mem;
  u32 *sB = tab + 4 * 256 * 32;
  u32 *sA = sB + 2 * kProdStep * 32;
  __shared__ u32 s_cnt[2][8];            // bits of the outer per word of keys
  __shared__ u32 s_rows[8];              // inner rows with bits, per word of keys
  __shared__ long long s_unit;
  if (ctl_stop(a.j.ctl)) return;
  u64 n_outer;
  if (a.part != 2 && product_empty(a.j, &n_outer)) return;
  const u32 *OT = prod_outer(a);
  if (!OT) return;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int rs = a.dk - 5;
  const u32 row_words = 1u << rs;
  const u32 ids = a.side * 256;  // at most 2^dk
  const u32 kind = prod_kind(a.list, a.side, a.sms);
  const u32 n_rows = kind == kProdNone ? 0u : *((volatile u32 *)&a.list[kind]);
  const u32 *rows = a.list + prod_list_at(kind == kProdNone ? 0 : kind);
  const ProdSplit split = prod_split(n_rows, a.side, a.sms);
  const u32 n_sl = split.n_sl, n_kc = split.n_kc, ksteps = split.ksteps;
  const u32 units = split.n_rb * n_sl * n_kc;
  const u32 lane4 = lane * 4;
  u64 flushed = 0;
  while (true) {
    if (tid < 16) s_cnt[tid >> 3][tid & 7] = 0;
    const long long g = grab_tile(a.j.rec, &s_unit);
    if (g >= (long long)units) break;
    const u32 u = (u32)g;
    const u32 kc = u % n_kc, sl = (u / n_kc) % n_sl, rb = u / n_kc / n_sl;
    const u32 k0 = kc * ksteps, k1 = min(k0 + ksteps, a.side);
    u32 acc[RW];
#pragma unroll
    for (int r = 0; r < RW; r++) acc[r] = 0;
    // this thread's outer row (also lane l's: output row l of the warp)
    const u32 my_row = rb * MR + tid < n_rows ? rows[rb * MR + tid] : kNoRow;
    u32 av[8];
    auto load_a = [&](u32 s) {
      if (my_row != kNoRow) {
        load8(OT + ((u64)my_row << rs) + s * 8, av);
      } else {
#pragma unroll
        for (int w = 0; w < 8; w++) av[w] = 0;
      }
    };
    // 256 inner rows of 128 bytes (zeros past the row's end)
    auto load_b = [&](u32 s, u32 st) {
#pragma unroll
      for (int i = 0; i < kProdStep * 8 / kProdBlock; i++) {
        const u32 c = tid + i * kProdBlock, r = c >> 3, w = sl * 32 + (c & 7) * 4;
        const bool in = w < row_words;
        cp_async16(sB + (st * kProdStep + r) * 32 + (c & 7) * 4,
                   a.F + ((u64)(s * kProdStep + r) << rs) + (in ? w : 0), in ? 16 : 0);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load_a(k0);
    load_b(k0, 0);
    for (u32 s = k0; s < k1; s++) {
      const u32 st = (s - k0) & 1;
#pragma unroll
      for (int w = 0; w < 8; w++) {
        const u32 c = __reduce_add_sync(0xffffffffu, (u32)__popc(av[w]));
        if (lane == 0 && c) atomicAdd(&s_cnt[st][w], c);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      const u32 *B = sB + st * kProdStep * 32;
#pragma unroll
      for (int part = 0; part < 8; part += kPart) {
        // the outer's words of this part, as table offsets: bytes 0, 1 (times
        // 128) in one word, bytes 2, 3 in the next
#pragma unroll
        for (int w = 0; w < kPart; w++) {
          const u32 x = av[part + w];
          reinterpret_cast<uint2 *>(sA)[w * MR + tid] =
              make_uint2(((x & 0xFFu) << 7) | ((x & 0xFF00u) << 15),
                         ((x >> 9) & 0x7F80u) | ((x >> 1) & 0x7F800000u));
        }
        __syncthreads();  // the step's operands and counts
        if (part + kPart == 8 && s + 1 < k1) {
          load_a(s + 1);
          load_b(s + 1, st ^ 1);
        }
        u32 any = 0;
#pragma unroll
        for (int w = 0; w < 8; w++) any |= s_cnt[st][w];
        if (any) {  // (block-uniform)
          if (part == 0) {
            u32 m = 0;
#pragma unroll
            for (int j = 0; j < kProdStep / kProdWarps; j++)
              if (__any_sync(0xffffffffu,
                             B[(wid * (kProdStep / kProdWarps) + j) * 32 + lane] != 0u))
                m |= 1u << j;
            // (eight rows a warp: byte wid % 4 of word wid / 4)
            if (lane == 0) reinterpret_cast<u8 *>(s_rows)[wid] = (u8)m;
            __syncthreads();
          }
          for (int wp = 0; wp < kPart; wp++) {
            const int w = part + wp;
            const u32 cnt = s_cnt[st][w];
            const u32 bm = s_rows[w];
            if (cnt == 0 || bm == 0) continue;  // (block-uniform)
            const u32 *Bw = B + w * 32 * 32 + lane;
            if (cnt > MR) {
              {
                // warp wid: byte wid / 8, the 32 entries with top bits wid % 8
                const u32 *r = Bw + (wid >> 3) * 8 * 32;
                u32 lo[8], hi[4];
                lo[0] = 0;
                lo[1] = r[0];
                lo[2] = r[32];
                lo[3] = lo[1] | lo[2];
                const u32 r2 = r[64];
#pragma unroll
                for (int i = 0; i < 4; i++) lo[4 + i] = lo[i] | r2;
                hi[0] = ((wid & 1) ? r[5 * 32] : 0u) | ((wid & 2) ? r[6 * 32] : 0u) |
                        ((wid & 4) ? r[7 * 32] : 0u);
                hi[1] = hi[0] | r[96];
                const u32 r4 = r[128];
                hi[2] = hi[0] | r4;
                hi[3] = hi[1] | r4;
                u32 *t = tab + ((wid >> 3) * 256 + (wid & 7) * 32) * 32 + lane;
#pragma unroll
                for (int i = 0; i < 32; i++) t[i * 32] = lo[i & 7] | hi[i >> 3];
              }
              __syncthreads();
              const char *tb = reinterpret_cast<const char *>(tab);
              const uint4 *Aw = reinterpret_cast<const uint4 *>(sA) + (wp * MR + wid * RW) / 2;
#pragma unroll
              for (int q = 0; q < RW / 4; q++) {
                const uint4 x0 = Aw[2 * q], x1 = Aw[2 * q + 1];
                if (x0.x | x0.y | x0.z | x0.w | x1.x | x1.y | x1.z | x1.w) {
                  const u32 xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
#pragma unroll
                  for (int i = 0; i < 4; i++) {
                    const u32 lo = xs[2 * i], hi = xs[2 * i + 1];
                    const u32 t0 = *(const u32 *)(tb + ((lo & 0x7F80u) | lane4));
                    const u32 t1 = *(const u32 *)(tb + 32768 + ((lo >> 16) + lane4));
                    const u32 t2 = *(const u32 *)(tb + 65536 + ((hi & 0x7F80u) | lane4));
                    const u32 t3 = *(const u32 *)(tb + 98304 + ((hi >> 16) + lane4));
                    acc[q * 4 + i] |= t0 | t1 | t2 | t3;
                  }
                }
              }
              __syncthreads();  // the table is rebuilt for the next word
            } else {
              const uint2 *Aw = reinterpret_cast<const uint2 *>(sA) + wp * MR + wid * RW;
#pragma unroll
              for (int h = 0; h < RW / 32; h++) {
                const uint2 mine = Aw[h * 32 + lane];
                const u32 some = __ballot_sync(0xffffffffu, (mine.x | mine.y) != 0u);
                if (!some) continue;
#pragma unroll
                for (int r = 0; r < 32; r++) {
                  if (!((some >> r) & 1u)) continue;
                  const uint2 p = Aw[h * 32 + r];
                  u32 x = ((p.x >> 7) & 0xFFu) | ((p.x >> 15) & 0xFF00u) |
                          ((p.y & 0x7F80u) << 9) | ((p.y & 0x7F800000u) << 1);
                  // (two reads in flight; the last key twice when they are odd)
                  for (x &= bm; x; ) {
                    const u32 b0 = __ffs(x) - 1;
                    x &= x - 1;
                    const u32 b1 = x ? __ffs(x) - 1 : b0;
                    x &= x - 1;
                    acc[h * 32 + r] |= Bw[b0 * 32] | Bw[b1 * 32];
                  }
                }
              }
            }
          }
        }
        __syncthreads();  // every read of this part's words (and, last, of the inner's rows)
        if (part + kPart == 8 && tid < 8) s_cnt[st][tid] = 0;  // (next used two steps on)
      }
    }
    // nonzero words out; units that share rows differ in their keys only
    const u32 col = sl * 32 + lane;
#pragma unroll
    for (int r = 0; r < RW; r++) {
      const u32 v = acc[r];
      const u32 row = __shfl_sync(0xffffffffu, my_row, r);
      if (v && col < row_words) {
        const u64 gw = ((u64)row << rs) + col;
        asm volatile("red.global.or.b32 [%0], %1;" ::"l"(a.G + gw), "r"(v) : "memory");
        if (a.dirty) a.dirty[gw / kBmChunkWords] = 1;
        flushed++;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) flushed += __shfl_xor_sync(0xffffffffu, flushed, o);
  // algorithmic bytes of both kernels together: OT and the inner once, 4 per
  // word reduced into the output
  if (lane == 0) prof_add(a.j.ctl, kPJoinMat, 4 * flushed);
  if (launch_rec_finish(a.j.rec) && tid == 0)
    prof_add(a.j.ctl, kPJoinMat, (u64)ids * a.side * 32);
}

// A product that leaves the repeated tuples out still counts as having found
// theirs (NEWT is not empty, src/lie.cu:114-121): *phantom is set when some
// key of OT has an inner row with bits.  Warps stop at the first such key, as
// a rule at once.
__global__ void __launch_bounds__(256) k_prod_repeats(ProdArgs a, u32 *phantom) {
  if (ctl_stop(a.j.ctl) || !prod_few_fresh(a)) return;
  if (a.newt->n == 0 || eff_count(a.j.inner, a.j.inner_vis) == 0) return;
  const int lane = threadIdx.x & 31;
  const u32 words = a.side * 8, rows = a.side * 256;
  for (u32 r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows;
       r += (gridDim.x * blockDim.x) >> 5) {
    for (u32 w0 = 0; w0 < words; w0 += 32) {
      if (*((volatile u32 *)phantom)) return;
      const u32 mine = w0 + lane < words ? a.OT[((u64)r << (a.dk - 5)) + w0 + lane] : 0u;
      for (u32 some = __ballot_sync(0xffffffffu, mine != 0u); some; some &= some - 1) {
        const int j = __ffs(some) - 1;
        for (u32 x = __shfl_sync(0xffffffffu, mine, j); x; x &= x - 1) {
          const u32 *row = a.F + ((u64)((w0 + j) * 32 + __ffs(x) - 1) << (a.dk - 5));
          u32 any = 0;
          for (u32 i = lane; i < words; i += 32) any |= row[i];
          if (__any_sync(0xffffffffu, any != 0u)) {
            if (lane == 0) *phantom = 1;
            return;
          }
        }
      }
    }
  }
}

// One warp: output row `row`, the keys of its words [w0, w1) (at most 32
// words).  RS: rows of 2^RS words, 8 to 64.  With rows shorter than a warp,
// 32 >> RS keys are read at once, one per group of 2^RS lanes.
template <int RS>
__device__ __forceinline__ void product_small_row(const ProdArgs &a, u32 row, u32 w0, u32 w1,
                                                  u32 *keys_used) {
  constexpr u32 RWD = 1u << RS;
  constexpr int LOADS = RS >= 5 ? 4 : 4 >> (5 - RS);  // load instructions per 4 keys
  const int lane = threadIdx.x & 31;
  const u32 mine = w0 + lane < w1 ? a.OT[(row << RS) + w0 + lane] : 0u;
  u32 some = __ballot_sync(0xffffffffu, mine != 0u);
  if (!some) return;
  u32 acc0 = 0, acc1 = 0, used = 0;
  const u32 grp = RS >= 5 ? 0 : (u32)lane >> RS, at = RS >= 5 ? (u32)lane : lane & (RWD - 1);
  for (; some; some &= some - 1) {
    const int j = __ffs(some) - 1;
    u32 x = __shfl_sync(0xffffffffu, mine, j);
    used += __popc(x);
    const u32 *base = a.F + ((w0 + j) << (5 + RS)) + at;
    while (x) {
      // four keys (the last one repeated when fewer are left)
      u32 k[4];
      k[0] = __ffs(x) - 1;
      x &= x - 1;
#pragma unroll
      for (int i = 1; i < 4; i++) {
        k[i] = x ? __ffs(x) - 1 : k[i - 1];
        x &= x - 1;
      }
#pragma unroll
      for (int i = 0; i < LOADS; i++) {
        u32 key = k[i];
        if (RS == 4) key = grp ? k[2 * i + 1] : k[2 * i];
        if (RS == 3) key = grp == 0 ? k[0] : grp == 1 ? k[1] : grp == 2 ? k[2] : k[3];
        acc0 |= base[key << RS];
        if (RS == 6) acc1 |= base[(key << RS) + 32];
      }
    }
  }
  if (RS < 5) {
#pragma unroll
    for (int o = 16; o >= (int)RWD; o >>= 1) acc0 |= __shfl_xor_sync(0xffffffffu, acc0, o);
  }
  const u32 out = (row << RS) + at;
  if (acc0 && grp == 0) {
    asm volatile("red.global.or.b32 [%0], %1;" ::"l"(a.G + out), "r"(acc0) : "memory");
    if (a.dirty) a.dirty[out / kBmChunkWords] = 1;
  }
  if (RS == 6 && acc1) {
    asm volatile("red.global.or.b32 [%0], %1;" ::"l"(a.G + out + 32), "r"(acc1) : "memory");
    if (a.dirty) a.dirty[out / kBmChunkWords] = 1;  // (rows of one chunk)
  }
  *keys_used += used;
}

// The product over 2^8 .. 2^11 ids by the calling grid's warps (block: the
// caller's number for this one), both sides non-empty.
__device__ __forceinline__ void product_small(const ProdArgs &a, u32 block) {
  const u32 rows = a.side * 256, words = a.side * 8;
  const u32 per = (words + a.splits - 1) / a.splits;
  u32 used = 0;
  const u32 nw = gridDim.x * (blockDim.x >> 5);
  for (u32 u = (block * blockDim.x + threadIdx.x) >> 5; u < rows * a.splits; u += nw) {
    const u32 row = u / a.splits, w0 = (u % a.splits) * per, w1 = min(w0 + per, words);
    switch (a.dk) {
      case 8: product_small_row<3>(a, row, w0, w1, &used); break;
      case 9: product_small_row<4>(a, row, w0, w1, &used); break;
      case 10: product_small_row<5>(a, row, w0, w1, &used); break;
      default: product_small_row<6>(a, row, w0, w1, &used); break;
    }
  }
  // algorithmic bytes: each word of OT, an inner row per key
  if (!a.j.ctl) return;  // (the resident loop keeps no account)
  if ((threadIdx.x & 31) == 0 && used) prof_add(a.j.ctl, kPJoinMat, (u64)used << (a.dk - 3));
  if (blockIdx.x == 0 && threadIdx.x == 0) prof_add(a.j.ctl, kPJoinMat, (u64)rows * words * 4);
}

__global__ void __launch_bounds__(256) k_join_product_small(ProdArgs a) {
  if (ctl_stop(a.j.ctl)) return;
  u64 n_outer;
  if (product_empty(a.j, &n_outer)) return;
  product_small(a, blockIdx.x);
}

// Warps a row's keys are shared among: 8 words of keys (256) each from 2^10
// ids on, 4 below, so that a full row is at most 64 rounds of four reads.
__host__ __device__ constexpr u32 prod_small_splits(u32 side) {
  return side >= 4 ? side : 2 * side;
}

constexpr int kProdRowsBlock = 256;
constexpr u32 kProdListCap = 4096;  // listed keys per round
constexpr u32 kProdListTake = kProdListCap / kProdRowsBlock;

// V: 16-byte words of a row per lane, 2^(dk-12).  Lane l holds words
// j * 32 + l; words past the last id's group are neither read nor written.
template <int V>
__global__ void __launch_bounds__(kProdRowsBlock, V <= 8 ? 2 : 1) k_join_product_rows(ProdArgs a) {
  __shared__ u32 s_list[kProdListCap];  // row of the tile << 16 | key
  __shared__ u64 s_scan[kProdRowsBlock / 32];
  __shared__ long long s_tile;
  if (ctl_stop(a.j.ctl)) return;
  const u64 n_outer = eff_count(a.j.outer, a.j.outer_vis);
  // (the launch before this one applied the empty-side rule)
  if (n_outer == 0 || eff_count(a.j.inner, a.j.inner_vis) == 0) return;
  const u32 *OT = prod_outer(a);
  if (!OT) return;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int kRows = kProdRowsBlock / 32;
  const int rs = a.dk - 5;
  const u32 n4 = a.side * 2;  // 16-byte words of a row that hold ids
  const u32 tiles = a.side * 256 / kRows;
  // (without the rows that the launch before this one took)
  const u32 kind = prod_kind(a.list, a.side, a.sms);
  const u32 part = kind == kProdNone       ? 0u
                   : kind == kProdFullRows ? prod_full_part(a.dk)
                                           : kProdLong;
  u64 words_out = 0;
  while (true) {
    const long long t = grab_tile(a.rows_rec, &s_tile);
    if (t >= (long long)tiles) break;
    // (rows of a tile lie far apart: long rows, often neighbours, go to
    // different blocks)
    auto row_no = [&](u32 r) { return (u32)t + r * tiles; };
    u32 w[V * 4];
    u32 left = 0;
    {
      const uint4 *p = reinterpret_cast<const uint4 *>(OT + ((u64)row_no(wid) << rs));
#pragma unroll
      for (int j = 0; j < V; j++) {
        const uint4 x = j * 32 + lane < n4 ? p[j * 32 + lane] : make_uint4(0, 0, 0, 0);
        w[4 * j] = x.x, w[4 * j + 1] = x.y, w[4 * j + 2] = x.z, w[4 * j + 3] = x.w;
        left += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
      }
      if (prod_reaches(__reduce_add_sync(0xffffffffu, left), part, a.side)) left = 0;
    }
    while (true) {
      // all keys that are left, or when they do not fit the list a share of
      // every thread's
      u64 total;
      u64 ex = block_excl_scan<kProdRowsBlock>(left, s_scan, &total);
      if (total == 0) break;  // (block-uniform)
      u32 take = left;
      if (total > kProdListCap) {
        take = min(left, kProdListTake);
        ex = block_excl_scan<kProdRowsBlock>(take, s_scan, &total);
      }
      left -= take;
      u32 pos = (u32)ex;
      const u32 end = pos + take;
#pragma unroll
      for (int j = 0; j < V * 4; j++) {
        const u32 key0 = (((j >> 2) * 32 + lane) * 4 + (j & 3)) * 32;
        while (w[j] && pos < end) {
          s_list[pos++] = ((u32)wid << 16) | (key0 + __ffs(w[j]) - 1);
          w[j] &= w[j] - 1;
        }
      }
      __syncthreads();
      const u32 n = (u32)total;
      // an equal share of the list a warp, two rows in flight
      u32 i = (u32)((u64)n * wid / kRows);
      const u32 iend = (u32)((u64)n * (wid + 1) / kRows);
      uint4 acc[V];
      const uint4 none = make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int j = 0; j < V; j++) acc[j] = none;
      auto row_of = [&](u32 e, uint4 *b) {
        const uint4 *p = reinterpret_cast<const uint4 *>(a.F + ((u64)(e & 0xFFFFu) << rs));
#pragma unroll
        for (int j = 0; j < V; j++) b[j] = j * 32 + lane < n4 ? p[j * 32 + lane] : none;
      };
      auto flush = [&](u32 r) {
        u32 *d = a.G + ((u64)row_no(r) << rs);
#pragma unroll
        for (int j = 0; j < V; j++) {
          const uint4 v = acc[j];
          acc[j] = none;
          if ((v.x | v.y | v.z | v.w) == 0u) continue;
          u32 *o = d + (j * 32 + lane) * 4;
          if (v.x) asm volatile("red.global.or.b32 [%0], %1;" ::"l"(o + 0), "r"(v.x) : "memory");
          if (v.y) asm volatile("red.global.or.b32 [%0], %1;" ::"l"(o + 1), "r"(v.y) : "memory");
          if (v.z) asm volatile("red.global.or.b32 [%0], %1;" ::"l"(o + 2), "r"(v.z) : "memory");
          if (v.w) asm volatile("red.global.or.b32 [%0], %1;" ::"l"(o + 3), "r"(v.w) : "memory");
          if (a.dirty) a.dirty[(o - a.G) / kBmChunkWords] = 1;
          words_out += 4;
        }
      };
      auto or_in = [&](const uint4 *b) {
#pragma unroll
        for (int j = 0; j < V; j++)
          acc[j].x |= b[j].x, acc[j].y |= b[j].y, acc[j].z |= b[j].z, acc[j].w |= b[j].w;
      };
      if (i < iend) {
        u32 cur = s_list[i] >> 16;
        for (; i < iend; i += 2) {
          const u32 e0 = s_list[i], e1 = s_list[min(i + 1, iend - 1)];
          uint4 b0[V], b1[V];
          row_of(e0, b0);
          row_of(e1, b1);
          if ((e0 >> 16) != cur) {
            flush(cur);
            cur = e0 >> 16;
          }
          or_in(b0);
          if ((e1 >> 16) != cur) {
            flush(cur);
            cur = e1 >> 16;
          }
          or_in(b1);  // (the last entry twice when the share is odd)
        }
        flush(cur);
      }
      __syncthreads();  // the list is rewritten
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) words_out += __shfl_xor_sync(0xffffffffu, words_out, o);
  if (lane == 0) prof_add(a.j.ctl, kPJoinMat, 4 * words_out);
  if (launch_rec_finish(a.rows_rec) && tid == 0) {
    for (u32 i = 0; i < kProdListHead; i++) a.list[i] = 0;
    prof_add(a.j.ctl, kPJoinMat, (u64)a.side * 256 * a.side * 32);
  }
}

}  // namespace gdl
