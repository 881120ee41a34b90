// export_pieces (csrc/export.cuh) over a fake device whose copies land late,
// and whose calls fail one at a time.  Prints "ok" or the failing check.
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <vector>

#include "../../gdlog-multinode_b200/csrc/export.cuh"

using u64 = uint64_t;

struct Fake {
  enum Call { kNone, kBuffer, kMarks, kCopy, kMark, kWait, kFinish };
  Call fail = kNone;
  u64 fail_at = 0;  // the call of that kind that fails
  u64 most = 1000;  // keys the buffer can hold
  u64 calls[7] = {};
  std::vector<u64> pin;
  struct Copy {
    u64 *dst;
    const u64 *src;
    u64 n;
  };
  std::vector<Copy> queue;     // not landed yet
  std::vector<u64> behind;     // per mark: copies queued before it
  std::mutex mu;
  bool step(Call c) { return !(calls[c]++ == fail_at && c == fail); }
  void land(u64 n) {
    for (u64 i = 0; i < n; i++) {
      for (u64 j = 0; j < queue[i].n; j++) queue[i].dst[j] = queue[i].src[j];
      queue[i].n = 0;
    }
  }
  u64 *buffer(u64 keys, u64 *cap) {
    if (!step(kBuffer)) return nullptr;
    *cap = keys < most ? keys : most;
    pin.assign(*cap, ~0ull);
    return pin.data();
  }
  bool marks(u64 n) {
    behind.assign(n, 0);
    return step(kMarks);
  }
  bool copy(u64 *dst, const u64 *src, u64 n) {
    if (!step(kCopy)) return false;
    if (dst < pin.data() || dst + n > pin.data() + pin.size()) {
      printf("copy past the buffer\n");
      exit(1);
    }
    queue.push_back({dst, src, n});
    return true;
  }
  bool mark(u64 i) {
    if (!step(kMark)) return false;
    behind.at(i) = queue.size();
    return true;
  }
  bool wait(u64 i) {
    std::lock_guard<std::mutex> lock(mu);
    if (!step(kWait)) return false;
    land(behind.at(i));
    return true;
  }
  bool finish() {
    std::lock_guard<std::mutex> lock(mu);
    land(queue.size());
    queue.clear();
    return step(kFinish);
  }
};

static int check(int arity, u64 n, Fake::Call fail, u64 at, gdl::ExportEnd want) {
  const int k2 = 10;
  std::vector<u64> keys(n), rows(n * arity + 1, 77);
  for (u64 i = 0; i < n; i++) keys[i] = (i * 3 << 32) | (i % 1024 << k2) | (i % 1000);
  Fake api;
  api.fail = fail;
  api.fail_at = at;
  const gdl::ExportEnd end = gdl::export_pieces(api, keys.data(), n, arity, k2, rows.data(), 64, 1000);
  const char *what = end != want ? "wrong end"
                     : !api.queue.empty() && end != gdl::kExportNoRoom ? "copies left in flight"
                     : rows[n * arity] != 77 ? "row past the end"
                                             : nullptr;
  for (u64 i = 0; i < n && !what; i++) {
    const u64 *r = &rows[i * arity], k = keys[i];
    if (end == gdl::kExportNoRoom) {
      if (r[0] != 77 || r[1] != 77) what = "written without a buffer";
    } else if (end == gdl::kExported) {
      const bool ok = arity == 2 ? r[0] == k >> 32 && r[1] == (uint32_t)k
                                 : r[0] == k >> 32 && r[1] == (uint32_t)k >> k2 && r[2] == k % 1024;
      if (!ok) what = "wrong row";
    }
  }
  if (what) printf("%s: arity %d, n %llu, call %d at %llu\n", what, arity, (unsigned long long)n,
                   (int)fail, (unsigned long long)at);
  return what != nullptr;
}

int main() {
  int bad = 0;
  for (int arity : {2, 3})
    for (u64 n : {1, 63, 64, 65, 999, 1000, 1001, 4000, 4111}) {
      bad += check(arity, n, Fake::kNone, 0, gdl::kExported);
      bad += check(arity, n, Fake::kBuffer, 0, gdl::kExportNoRoom);
      bad += check(arity, n, Fake::kMarks, 0, gdl::kExportNoRoom);
      for (Fake::Call c : {Fake::kCopy, Fake::kMark, Fake::kWait}) {
        const u64 pieces = (n / 1000) * 16 + (n % 1000 + 63) / 64;
        for (u64 at : {u64(0), pieces / 2, pieces - 1})
          bad += check(arity, n, c, at, gdl::kExportFailed);
      }
      bad += check(arity, n, Fake::kFinish, (n - 1) / 1000, gdl::kExportFailed);
    }
  const u64 some = gdl::kExportPiece + 1, first = gdl::kExportFirst, pinned = gdl::kExportPinned;
  const struct {
    u64 n, before, cap;
    bool pieces;
  } rule[] = {{some - 1, 9 * some, pinned, false}, {some, 0, 0, false},    {some, some - 1, 0, false},
              {some, some, 0, true},               {some, 0, some, true},  {some, 0, some - 1, false},
              {first - 1, 0, some, false},         {first, 0, 0, true},    {4 * pinned, 0, 0, true},
              {4 * pinned, 0, pinned, true}};
  for (auto &x : rule)
    if (gdl::export_in_pieces(x.n, x.before, x.cap) != x.pieces) {
      printf("rule: n %llu\n", (unsigned long long)x.n);
      bad++;
    }
  if (!bad) printf("ok\n");
  return bad != 0;
}
