"""What the contexts of a device share (csrc/gd_shared.h) over a stand-in for
the runtime whose CUDA contexts come and go: contexts released in any order,
more of them than a pinned block has room for, several devices, a device reset
under live contexts, workspaces lent and given back, and failures on the way."""
import pytest

from tests import native

FAKE = r"""
#include <map>
#include <set>
#include <vector>
#include "gd_shared.h"
struct State {
  int device = 0, pins = 0, fail_in = 0;
  std::map<int, uint64_t> serial{{0, 7}, {1, 8}};
  std::map<void *, uint64_t> pinned;   // live blocks, by the serial they belong to
  std::map<void *, uint64_t> mem;      // device allocations
  std::map<int, bool> ended;           // events: whether the work before them has ended
  int allocs = 0, queries = 0, next_event = 1;
  bool wrong = false;                  // something dead was given back
  void reset(int d, uint64_t s) {      // everything of the old CUDA context goes
    for (auto it = pinned.begin(); it != pinned.end();)
      if (it->second == serial[d]) { std::free(it->first); it = pinned.erase(it); } else ++it;
    for (auto it = mem.begin(); it != mem.end();)
      if (it->second == serial[d]) { std::free(it->first); it = mem.erase(it); } else ++it;
    serial[d] = s;
  }
};
struct Fake {
  using Error = int;
  using Stream = int;
  using Event = int;
  State *s;
  static bool ok(int e) { return e == 0; }
  uint64_t serial() { return s->serial[s->device]; }
  bool fails() { return s->fail_in > 0 && --s->fail_in == 0; }
  int pin(void **p, size_t n) {
    if (fails()) return 2;
    *p = std::malloc(n);
    s->pinned[*p] = serial();
    s->pins++;
    return 0;
  }
  int alloc(void **p, size_t, int) {
    if (fails()) return 2;
    *p = std::malloc(1);
    s->mem[*p] = serial();
    s->allocs++;
    return 0;
  }
  void free(void *p, int) {
    auto it = s->mem.find(p);
    if (it == s->mem.end()) { s->wrong = true; return; }
    std::free(p);
    s->mem.erase(it);
  }
  int event(int *e) { *e = s->next_event++; s->ended[*e] = true; return 0; }
  int record(int e, int) { s->ended[e] = false; return 0; }
  bool done(int e) { s->queries++; return s->ended[e]; }
  void drop(int e) { if (!s->ended.erase(e)) s->wrong = true; }
  void unpin(void *p) {
    auto it = s->pinned.find(p);
    if (it == s->pinned.end()) { s->wrong = true; return; }
    std::free(p);
    s->pinned.erase(it);
  }
};
using Shared = gd::DeviceShared<Fake>;
using Lease = Shared::Lease;
// whether the lease's block lies in pinned memory that is still there
bool live(State &s, const Lease &l, size_t n) {
  for (auto &x : s.pinned) {
    auto *b = (unsigned char *)x.first, *p = (unsigned char *)l.block;
    if (p >= b && p + n <= b + 4 * n) return true;
  }
  return false;
}
"""

CASES = {
    # six contexts, released out of order and taken again: blocks are distinct,
    # everything goes with the last of them
    "mixed_order": r"""
  State s;
  Shared S(512, 64 << 20, Fake{&s});
  Lease l[6];
  for (auto &x : l) CHECK(S.acquire(0, &x) == 0);
  CHECK(s.pins == 3);  // a block of four, two of their own
  std::set<void *> seen;
  for (auto &x : l) { seen.insert(x.block); CHECK(live(s, x, 512)); }
  CHECK(seen.size() == 6);
  void *b1 = l[1].block;
  S.release(&l[4], nullptr, 0);
  S.release(&l[1], nullptr, 0);
  S.release(&l[0], nullptr, 0);
  Lease again;
  CHECK(S.acquire(0, &again) == 0 && s.pins == 3 && again.block != l[2].block &&
        again.block != l[3].block && live(s, again, 512));
  CHECK(S.acquire(0, &l[1]) == 0 && s.pins == 3);
  CHECK(again.block == b1 || l[1].block == b1);
  for (Lease *x : {&l[3], &again, &l[5], &l[1]}) S.release(x, nullptr, 0);
  S.release(&l[2], nullptr, 0);
  CHECK(s.pinned.empty() && s.mem.empty() && s.ended.empty() && !s.wrong);
  S.release(&l[2], nullptr, 0);  // a lease is given back once
""",
    # the block of device 1's context is not device 0's to take away
    "devices": r"""
  State s;
  Shared S(512, 64 << 20, Fake{&s});
  Lease a, b;
  CHECK(S.acquire(0, &a) == 0);
  s.device = 1;
  CHECK(S.acquire(1, &b) == 0);
  s.device = 0;
  S.release(&a, nullptr, 0);
  s.reset(0, 9);
  CHECK(live(s, b, 512));
  s.device = 1;
  S.release(&b, nullptr, 0);
  CHECK(s.pinned.empty() && s.mem.empty() && s.ended.empty() && !s.wrong);
""",
    # a reset under live contexts: the next context gets a block that
    # exists, and releasing the old ones later gives nothing dead back
    "reset": r"""
  State s;
  Shared S(512, 64 << 20, Fake{&s});
  Lease old[6], now[2];
  for (auto &x : old) CHECK(S.acquire(0, &x) == 0);
  s.reset(0, 9);
  CHECK(S.acquire(0, &now[0]) == 0 && live(s, now[0], 512));
  S.release(&old[5], nullptr, 0);
  S.release(&old[0], nullptr, 0);
  CHECK(S.acquire(0, &now[1]) == 0 && live(s, now[1], 512));
  CHECK(now[0].block != now[1].block && now[0].group == now[1].group);
  for (int k : {1, 2, 3, 4}) S.release(&old[k], nullptr, 0);
  CHECK(live(s, now[0], 512) && !s.wrong);
  S.release(&now[0], nullptr, 0);
  S.release(&now[1], nullptr, 0);
  CHECK(s.pinned.empty() && s.mem.empty() && s.ended.empty() && !s.wrong);
""",
    # no serial number: nothing is shared
    "unknown": r"""
  State s;
  s.serial[0] = 0;
  Shared S(512, 64 << 20, Fake{&s});
  Lease a, b;
  CHECK(S.acquire(0, &a) == 0 && S.acquire(0, &b) == 0 && a.group != b.group && s.pins == 2);
  S.release(&a, nullptr, 0);
  CHECK(live(s, b, 512));
  S.release(&b, nullptr, 0);
  CHECK(s.pinned.empty() && s.mem.empty() && s.ended.empty() && !s.wrong);
""",
    # the block or a fifth context's own cannot be had
    "failures": r"""
  State s;
  Shared S(512, 64 << 20, Fake{&s});
  Lease l[5];
  s.fail_in = 1;
  CHECK(S.acquire(0, &l[0]) != 0 && s.pinned.empty());
  for (int k = 0; k < 4; ++k) CHECK(S.acquire(0, &l[k]) == 0);
  s.fail_in = 1;
  CHECK(S.acquire(0, &l[4]) != 0 && s.pinned.size() == 1);
  for (int k = 0; k < 4; ++k) S.release(&l[k], nullptr, 0);
  CHECK(s.pinned.empty() && s.mem.empty() && s.ended.empty() && !s.wrong);
""",
    # slabs: kept from call to call; another context's only once its work has ended
    "slabs": r"""
  State s;
  Shared S(512, 64 << 20, Fake{&s});
  const size_t MB = 1 << 20;
  Lease l[3];
  for (auto &x : l) CHECK(S.acquire(0, &x) == 0);
  auto *g = l[0].group;
  int A, B, C;  // contexts
  auto *a = S.lend(g, &A, 1, 3 * MB - 5);
  CHECK(a && a->bytes == 3 * MB && s.allocs == 1);
  auto *a2 = S.lend(g, &A, 1, MB);  // another thread of the same context
  CHECK(a2 && a2 != a && s.allocs == 2);
  S.give_back(g, a, &A, 1, MB);
  S.give_back(g, a2, &A, 1, MB);
  const int q = s.queries;
  CHECK(S.lend(g, &A, 1, 2 * MB) == a && s.allocs == 2);  // its own stream orders them
  CHECK(s.queries == q);
  S.give_back(g, a, &A, 1, 2 * MB);
  auto *b = S.lend(g, &B, 2, 2 * MB);  // A's work has not ended
  CHECK(b && b != a && b != a2 && s.allocs == 3);
  S.give_back(g, b, &B, 2, 2 * MB);
  for (auto &e : s.ended) e.second = true;
  auto *c = S.lend(g, &C, 3, MB);  // the smallest that fits
  CHECK(c == a2 && s.allocs == 3);
  S.give_back(g, c, &C, 3, MB);
  CHECK(S.lend(g, &B, 2, MB) == b && s.allocs == 3);  // its own first
  S.give_back(g, b, &B, 2, 5 * MB);  // it would have needed more: larger for the next
  CHECK(s.allocs == 4 && b->bytes == 5 * MB && s.mem.size() == 3);
  S.release(&l[1], &B, 2);
  CHECK(!S.lend(g, &A, 1, 65 * MB));  // more than is kept
  s.fail_in = 1;
  CHECK(!S.lend(g, &A, 1, 20 * MB));  // cannot be had
  CHECK(s.mem.size() == 2);           // (in the place of an ended one)
  S.release(&l[0], &A, 1);
  S.release(&l[2], &C, 3);
  CHECK(s.pinned.empty() && s.mem.empty() && s.ended.empty() && !s.wrong);
""",
    # never more than `keep` bytes, never one that is lent
    "slabs_bounded": r"""
  State s;
  Shared S(512, 64 << 20, Fake{&s});
  const size_t MB = 1 << 20;
  Lease l;
  CHECK(S.acquire(0, &l) == 0);
  std::vector<std::pair<Shared::Slab *, int>> lent;
  uint64_t x = 88172645463325252ull;
  int ctx[4];
  for (int i = 0; i < 20000; ++i) {
    x ^= x << 13, x ^= x >> 7, x ^= x << 17;
    const int k = (x >> 8) % 4;
    if ((x & 1) || lent.empty()) {
      const size_t need = 1 + (x >> 20) % (30 * MB);
      auto *b = S.lend(l.group, &ctx[k], k, need);
      if (b) {
        CHECK(b->bytes >= need && b->p);
        for (auto &y : lent) CHECK(y.first != b);
        // lent to another context only when its work has ended
        CHECK(b->user == nullptr || b->user == &ctx[k] || s.ended[b->done]);
        lent.push_back({b, k});
      }
    } else {
      const size_t j = (x >> 12) % lent.size();
      S.give_back(l.group, lent[j].first, &ctx[lent[j].second], lent[j].second,
                  (x >> 20) % (40 * MB));
      lent.erase(lent.begin() + j);
    }
    if (x % 5 == 0)
      for (auto &e : s.ended) e.second = e.second || (x >> 30) % 2;
    size_t total = 0;
    for (auto &b : l.group->slabs) total += b.bytes;
    CHECK(total <= 64 * MB && s.mem.size() <= 8);
    s.fail_in = x % 50 == 0 ? 1 : 0;
  }
  for (auto &y : lent) S.give_back(l.group, y.first, &ctx[y.second], y.second, 0);
  for (auto &c : ctx) (void)c;
  S.release(&l, nullptr, 0);
  CHECK(s.pinned.empty() && s.mem.empty() && s.ended.empty() && !s.wrong);
""",
    # a reset while slabs are kept: the next context's are of the new CUDA context
    "slabs_reset": r"""
  State s;
  Shared S(512, 64 << 20, Fake{&s});
  Lease old, now;
  int A, B;
  CHECK(S.acquire(0, &old) == 0);
  auto *a = S.lend(old.group, &A, 1, 100);
  S.give_back(old.group, a, &A, 1, 100);
  s.reset(0, 9);
  CHECK(S.acquire(0, &now) == 0 && now.group != old.group);
  auto *b = S.lend(now.group, &B, 2, 100);
  CHECK(b && s.mem.count(b->p));
  S.give_back(now.group, b, &B, 2, 100);
  S.release(&old, &A, 1);
  CHECK(s.mem.size() == 1 && !s.wrong);
  S.release(&now, &B, 2);
  CHECK(s.pinned.empty() && s.mem.empty() && !s.wrong);
""",
}


@pytest.mark.parametrize("case", CASES)
def test_shared(tmp_path, case):
    native.run(tmp_path, CASES[case], FAKE)
