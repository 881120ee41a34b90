// export.cuh — a sorted version's keys to the caller's rows (host code).
//
// The keys come over in pieces through a pinned buffer that the engine keeps,
// and threads unpack each piece as it lands: the caller's pages are mostly
// untouched before (one thread spent 25 of 35 ms on faulting them in for 4.3 M
// rows of three columns).
//
// Pinned memory costs some 0.65 ms a megabyte when it is first taken, more than
// the pieces save in one export below kExportFirst keys: those take the keys in
// one copy until as many have been exported.  (Taken by every first export,
// 1.3 M rows took 6.2 ms the first time, 2.4 after that; 3.8 in one copy.  4.3
// M rows of three columns: 27, 3.4 and 25 ms; 14.6 M rows: 38, 8.7 and 90.)
//
// What the copies need from the device is behind Api, so that the order of the
// steps and every failure of one can be run without a device:
//   Key *buffer(keys, &cap)  pinned room for cap keys (at most `keys`), or null
//   bool marks(n)            marks 0 .. n - 1 can be set
//   bool copy(dst, src, n)   n keys queued from the device
//   bool mark(i)             mark i queued behind them
//   bool wait(i)             mark i passed (called from several threads)
//   bool finish()            everything queued has ended
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <exception>
#include <thread>
#include <vector>

namespace gdl {

constexpr uint64_t kExportPiece = 1ull << 18;   // keys
constexpr uint64_t kExportPinned = 1ull << 23;  // keys the pinned buffer holds at most
constexpr uint64_t kExportFirst = 1ull << 22;   // keys of an export that takes it at once

// Whether an export of n keys goes in pieces, `before` keys having been
// exported and the buffer having room for cap.
inline bool export_in_pieces(uint64_t n, uint64_t before, uint64_t cap) {
  return n > kExportPiece &&
         (cap >= std::min(n, kExportPinned) || n >= kExportFirst || before >= n);
}

enum ExportEnd { kExported = 0, kExportNoRoom, kExportFailed };

// kExportNoRoom: no buffer or no marks, nothing was written.
template <class Api, class Key>
ExportEnd export_pieces(Api &api, const Key *keys, uint64_t n, int arity, int k2,
                        uint64_t *rows, uint64_t piece = kExportPiece,
                        uint64_t pinned = kExportPinned) {
  Key room = 0;
  Key *pin = api.buffer(std::min(n, pinned), &room);
  const uint64_t cap = room;
  if (!pin || cap == 0) return kExportNoRoom;
  if (!api.marks((std::min(n, cap) + piece - 1) / piece)) return kExportNoRoom;
  const unsigned hc = std::thread::hardware_concurrency();
  const uint64_t threads = std::min<uint64_t>(std::min(hc ? hc : 1u, 8u), n / piece + 1);
  for (uint64_t base = 0; base < n; base += cap) {
    const uint64_t m = std::min(n - base, cap);
    const uint64_t pieces = (m + piece - 1) / piece;
    bool queued = true;
    for (uint64_t q = 0; q < pieces && queued; q++) {
      const uint64_t o = q * piece, c = std::min(piece, m - o);
      queued = api.copy(pin + o, keys + base + o, c) && api.mark(q);
    }
    if (!queued) {
      api.finish();  // (the copies queued before)
      return kExportFailed;
    }
    std::atomic<uint64_t> next{0};
    std::atomic<bool> bad{false};
    auto work = [&] {
      for (uint64_t q; !bad && (q = next.fetch_add(1)) < pieces;) {
        if (!api.wait(q)) {
          bad = true;
          return;
        }
        const uint64_t o = q * piece, c = std::min(piece, m - o);
        const Key *k = pin + o;
        uint64_t *d = rows + (base + o) * arity;
        if (arity == 2) {
          for (uint64_t i = 0; i < c; i++) {
            d[2 * i] = k[i] >> 32;
            d[2 * i + 1] = (uint32_t)k[i];
          }
        } else {
          const uint64_t low = (1ull << k2) - 1;
          for (uint64_t i = 0; i < c; i++) {
            d[3 * i] = k[i] >> 32;
            d[3 * i + 1] = (uint32_t)k[i] >> k2;
            d[3 * i + 2] = k[i] & low;
          }
        }
      }
    };
    std::vector<std::thread> pool;
    try {
      pool.reserve(threads);
      while (pool.size() + 1 < threads) pool.emplace_back(work);
    } catch (const std::exception &) {
      // (fewer threads then)
    }
    work();
    for (std::thread &t : pool) t.join();
    if (!api.finish() || bad) return kExportFailed;
  }
  return kExported;
}

}  // namespace gdl
