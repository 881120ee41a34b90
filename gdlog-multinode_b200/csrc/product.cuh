// product.cuh — joins into bitmaps as boolean matrix products.
//
// A pull-form join (pull.cuh: output (outer column 1, inner column 1), or
// its transpose, joined on column 0) over an inner FULL kept as a bitmap is
// the boolean product  Out[x] |= OR over k of OT[x][k] & F[k]:  the outer
// transposed (row x, bit k) times the inner's rows.  Points-to analysis
// (test/cspa.cu:279-352) spends its time in nine such products of relations
// that fill a fifth to nine tenths of their domain; listing the inner,
// indexing it and expanding candidate tuples cost 11 ms a join at 20,000
// ids.  Here no list and no index exist: a block owns MR output rows by a
// slice of 1024 columns (a word a lane, MR / 16 rows a warp, accumulated in
// registers) and walks the keys 32 at a time.
//
// Per 32 keys (one word of each row of OT), by the bits its rows hold:
//   * many: the four-Russians method (Arlazarov, Dinic, Kronrod, Faradzev
//     1970).  For each of the word's four bytes the 256 ORs of its eight
//     inner rows are tabled in shared memory (1024 entries of 128 bytes,
//     built from registers, a store an entry), and a row takes four table
//     reads instead of one read per key.
//   * few: the row's keys one by one from the inner rows staged in shared
//     memory.
//   * none, or no inner row with bits in the slice: skipped.
// The bound is shared-memory bandwidth: one 128-byte read a row and byte of
// keys, so MR = 1024 rows share a table (its 1024 stores are a fifth of the
// 4096 + 256 reads).  The next 256 keys' operands load (cp.async for the
// inner's rows, registers for the outer's words) while these are used.
//
// Small domains (below 2^kProdTableBits ids) have too few rows to fill the
// GPU with tables: blocks of 64 rows, keys one by one, several blocks an SM.
#pragma once

#include "common.cuh"
#include "dense.cuh"
#include "join.cuh"

namespace gdl {

constexpr int kProdBlock = 512;
constexpr int kProdWarps = kProdBlock / 32;
constexpr int kProdStep = 256;       // keys per staged step: 8 words of a row
constexpr int kProdTableBits = 12;   // tables from 2^12 ids on
constexpr int kProdBigRows = 64;     // rows per warp with tables
constexpr int kProdSmallRows = 4;    // ... and without

__host__ __device__ constexpr u32 prod_rows(bool tables) {
  return kProdWarps * (tables ? kProdBigRows : kProdSmallRows);
}
// dynamic shared memory: the tables, two stages of 256 inner row slices, and
// the outer's words [8][rows]
__host__ __device__ constexpr u32 prod_smem(bool tables) {
  return (tables ? 4 * 256 * 128 : 0) + 2 * kProdStep * 128 + 8 * prod_rows(tables) * 4;
}

struct ProdArgs {
  JoinArgs j;      // descriptors for the emptiness rules, launch record, ctl
  const u32 *OT;   // the outer, transposed
  const u32 *F;    // the inner's rows
  u32 *G;          // output rows: the output's NEWT or its transposed twin
  u8 *dirty;       // dirty map of G, or null
  int dk;          // rows of 2^(dk-5) words
  u32 side;        // 256-id groups that hold ids
  u32 ksteps;      // groups per unit of work (the key range is split)
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src, u32 bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (u32)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes)
               : "memory");
}

template <int RW, bool TAB>
__global__ void __launch_bounds__(kProdBlock, TAB ? 1 : 2) k_join_product(ProdArgs a) {
  constexpr u32 MR = kProdWarps * RW;
  constexpr int RPT = MR >= kProdBlock ? MR / kProdBlock : 1;  // outer rows loaded per thread
  extern __shared__ __align__(128) u32 prod_mem[];
  u32 *tab = prod_mem;
  u32 *sB = tab + (TAB ? 4 * 256 * 32 : 0);
  u32 *sA = sB + 2 * kProdStep * 32;
  __shared__ u32 s_cnt[2][8];            // bits of the outer per word of keys
  __shared__ u32 s_half[kProdWarps];     // inner rows with bits, 16 a warp
  __shared__ long long s_unit;
  if (ctl_stop(a.j.ctl)) return;
  const u64 n_outer = eff_count(a.j.outer, a.j.outer_vis);
  const u64 n_inner = eff_count(a.j.inner, a.j.inner_vis);
  if (n_outer == 0 || n_inner == 0) {
    join_empty_side(a.j, n_outer);
    return;
  }
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int rs = a.dk - 5;
  const u32 row_words = 1u << rs;
  const u32 ids = a.side * 256;  // at most 2^dk
  const u32 n_rb = (ids + MR - 1) / MR, n_sl = (ids + 1023) / 1024;
  const u32 n_kc = (a.side + a.ksteps - 1) / a.ksteps;
  const u32 units = n_rb * n_sl * n_kc;
  const u32 lane4 = lane * 4;
  u64 used = 0, flushed = 0;
  while (true) {
    if (tid < 16) s_cnt[tid >> 3][tid & 7] = 0;
    const long long g = grab_tile(a.j.rec, &s_unit);
    if (g >= (long long)units) break;
    const u32 u = (u32)g;
    const u32 kc = u % n_kc, sl = (u / n_kc) % n_sl, rb = u / n_kc / n_sl;
    const u32 k0 = kc * a.ksteps, k1 = min(k0 + a.ksteps, a.side);
    u32 acc[RW];
#pragma unroll
    for (int r = 0; r < RW; r++) acc[r] = 0;
    u32 av[RPT][8];
    auto load_a = [&](u32 s) {
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const u32 lr = tid + i * kProdBlock, row = rb * MR + lr;
        if (lr < MR && row < ids) {
          load8(a.OT + ((u64)row << rs) + s * 8, av[i]);
        } else {
#pragma unroll
          for (int w = 0; w < 8; w++) av[i][w] = 0;
        }
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
        u32 c = 0;
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          if (tid + i * kProdBlock < MR) sA[w * MR + tid + i * kProdBlock] = av[i][w];
          c += __popc(av[i][w]);
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0 && c) atomicAdd(&s_cnt[st][w], c);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // the step's operands and counts
      if (s + 1 < k1) {
        load_a(s + 1);
        load_b(s + 1, st ^ 1);
      }
      if (tid < 8) s_cnt[st ^ 1][tid] = 0;
      const u32 *B = sB + st * kProdStep * 32;
      u32 any = 0;
#pragma unroll
      for (int w = 0; w < 8; w++) any |= s_cnt[st][w];
      if (any) {  // (block-uniform)
        u32 m = 0;
#pragma unroll
        for (int j = 0; j < 16; j++)
          if (__any_sync(0xffffffffu, B[(wid * 16 + j) * 32 + lane] != 0u)) m |= 1u << j;
        if (lane == 0) s_half[wid] = m;
        __syncthreads();
        for (int w = 0; w < 8; w++) {
          const u32 cnt = s_cnt[st][w];
          const u32 bm = s_half[2 * w] | (s_half[2 * w + 1] << 16);
          if (cnt == 0 || bm == 0) continue;  // (block-uniform)
          if (tid == 0) used += cnt;
          const u32 *Bw = B + w * 32 * 32 + lane;
          const uint4 *Aw = reinterpret_cast<const uint4 *>(sA + w * MR + wid * RW);
          if (TAB && cnt > 2 * MR) {
            {
              // warp wid: byte wid / 4, the 64 entries with top bits wid % 4
              const u32 *r = Bw + (wid >> 2) * 8 * 32;
              u32 lo[8], hi[8];
              lo[0] = 0;
              lo[1] = r[0];
              lo[2] = r[32];
              lo[3] = lo[1] | lo[2];
              const u32 r2 = r[64];
#pragma unroll
              for (int i = 0; i < 4; i++) lo[4 + i] = lo[i] | r2;
              hi[0] = ((wid & 1) ? r[6 * 32] : 0u) | ((wid & 2) ? r[7 * 32] : 0u);
              hi[1] = hi[0] | r[96];
              const u32 r4 = r[128], r5 = r[160];
              hi[2] = hi[0] | r4;
              hi[3] = hi[1] | r4;
#pragma unroll
              for (int i = 0; i < 4; i++) hi[4 + i] = hi[i] | r5;
              u32 *t = tab + ((wid >> 2) * 256 + (wid & 3) * 64) * 32 + lane;
#pragma unroll
              for (int i = 0; i < 64; i++) t[i * 32] = lo[i & 7] | hi[i >> 3];
            }
            __syncthreads();
            const char *tb = reinterpret_cast<const char *>(tab);
#pragma unroll
            for (int q = 0; q < RW / 4; q++) {
              const uint4 x4 = Aw[q];
              const u32 xs[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
              for (int i = 0; i < 4; i++) {
                const u32 x = xs[i];
                if (x) {
                  const u32 t0 = *(const u32 *)(tb + (((x << 7) & 0x7f80u) | lane4));
                  const u32 t1 = *(const u32 *)(tb + 32768 + (((x >> 1) & 0x7f80u) | lane4));
                  const u32 t2 = *(const u32 *)(tb + 65536 + (((x >> 9) & 0x7f80u) | lane4));
                  const u32 t3 = *(const u32 *)(tb + 98304 + (((x >> 17) & 0x7f80u) | lane4));
                  acc[q * 4 + i] |= t0 | t1 | t2 | t3;
                }
              }
            }
            __syncthreads();  // the table is rebuilt for the next word
          } else {
#pragma unroll
            for (int q = 0; q < RW / 4; q++) {
              const uint4 x4 = Aw[q];
              const u32 xs[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
              for (int i = 0; i < 4; i++)
                for (u32 x = xs[i] & bm; x; x &= x - 1) acc[q * 4 + i] |= Bw[(__ffs(x) - 1) * 32];
            }
          }
        }
      }
      __syncthreads();  // every read of the step's operands, before the next step's stores
    }
    // nonzero words out; units that share rows differ in their keys only
    const u32 col = sl * 32 + lane;
#pragma unroll
    for (int r = 0; r < RW; r++) {
      const u32 v = acc[r];
      if (v && col < row_words) {
        const u64 gw = ((u64)(rb * MR + wid * RW + r) << rs) + col;
        asm volatile("red.global.or.b32 [%0], %1;" ::"l"(a.G + gw), "r"(v) : "memory");
        if (a.dirty) a.dirty[gw / kBmChunkWords] = 1;
        flushed++;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) flushed += __shfl_xor_sync(0xffffffffu, flushed, o);
  // algorithmic bytes: 4 per word of OT, a slice of an inner row per key
  // used, 4 per word reduced into the output
  if (lane == 0) prof_add(a.j.ctl, kPJoinMat, 4 * flushed);
  if (tid == 0) prof_add(a.j.ctl, kPJoinMat, used * min(128u, 4u << rs));
  if (launch_rec_finish(a.j.rec) && tid == 0)
    prof_add(a.j.ctl, kPJoinMat, (u64)ids * a.side * 32);
}

}  // namespace gdl
