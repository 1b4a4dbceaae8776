"""What the contexts of a device share (csrc/gd_shared.h) over a stand-in for
the runtime whose CUDA contexts come and go: contexts released in any order,
more of them than a pinned block has room for, several devices, a device reset
under live contexts, and failures on the way."""
import pytest

from tests import native

FAKE = r"""
#include <map>
#include <set>
#include "gd_shared.h"
struct State {
  int device = 0, pins = 0, fail_in = 0;
  std::map<int, uint64_t> serial{{0, 7}, {1, 8}};
  std::map<void *, uint64_t> pinned;   // live blocks, by the serial they belong to
  bool wrong = false;                  // something dead was given back
  void reset(int d, uint64_t s) {      // everything of the old CUDA context goes
    for (auto it = pinned.begin(); it != pinned.end();)
      if (it->second == serial[d]) { std::free(it->first); it = pinned.erase(it); } else ++it;
    serial[d] = s;
  }
};
struct Fake {
  using Error = int;
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
  Shared S(512, Fake{&s});
  Lease l[6];
  for (auto &x : l) CHECK(S.acquire(0, &x) == 0);
  CHECK(s.pins == 3);  // a block of four, two of their own
  std::set<void *> seen;
  for (auto &x : l) { seen.insert(x.block); CHECK(live(s, x, 512)); }
  CHECK(seen.size() == 6);
  void *b1 = l[1].block;
  S.release(&l[4]);
  S.release(&l[1]);
  S.release(&l[0]);
  Lease again;
  CHECK(S.acquire(0, &again) == 0 && s.pins == 3 && again.block != l[2].block &&
        again.block != l[3].block && live(s, again, 512));
  CHECK(S.acquire(0, &l[1]) == 0 && s.pins == 3);
  CHECK(again.block == b1 || l[1].block == b1);
  for (Lease *x : {&l[3], &again, &l[5], &l[1]}) S.release(x);
  S.release(&l[2]);
  CHECK(s.pinned.empty() && !s.wrong);
  S.release(&l[2]);  // a lease is given back once
""",
    # the block of device 1's context is not device 0's to take away
    "devices": r"""
  State s;
  Shared S(512, Fake{&s});
  Lease a, b;
  CHECK(S.acquire(0, &a) == 0);
  s.device = 1;
  CHECK(S.acquire(1, &b) == 0);
  s.device = 0;
  S.release(&a);
  s.reset(0, 9);
  CHECK(live(s, b, 512));
  s.device = 1;
  S.release(&b);
  CHECK(s.pinned.empty() && !s.wrong);
""",
    # a reset under live contexts: the next context gets a block that
    # exists, and releasing the old ones later gives nothing dead back
    "reset": r"""
  State s;
  Shared S(512, Fake{&s});
  Lease old[6], now[2];
  for (auto &x : old) CHECK(S.acquire(0, &x) == 0);
  s.reset(0, 9);
  CHECK(S.acquire(0, &now[0]) == 0 && live(s, now[0], 512));
  S.release(&old[5]);
  S.release(&old[0]);
  CHECK(S.acquire(0, &now[1]) == 0 && live(s, now[1], 512));
  CHECK(now[0].block != now[1].block && now[0].group == now[1].group);
  for (int k : {1, 2, 3, 4}) S.release(&old[k]);
  CHECK(live(s, now[0], 512) && !s.wrong);
  S.release(&now[0]);
  S.release(&now[1]);
  CHECK(s.pinned.empty() && !s.wrong);
""",
    # no serial number: nothing is shared
    "unknown": r"""
  State s;
  s.serial[0] = 0;
  Shared S(512, Fake{&s});
  Lease a, b;
  CHECK(S.acquire(0, &a) == 0 && S.acquire(0, &b) == 0 && a.group != b.group && s.pins == 2);
  S.release(&a);
  CHECK(live(s, b, 512));
  S.release(&b);
  CHECK(s.pinned.empty() && !s.wrong);
""",
    # the block or a fifth context's own cannot be had
    "failures": r"""
  State s;
  Shared S(512, Fake{&s});
  Lease l[5];
  s.fail_in = 1;
  CHECK(S.acquire(0, &l[0]) != 0 && s.pinned.empty());
  for (int k = 0; k < 4; ++k) CHECK(S.acquire(0, &l[k]) == 0);
  s.fail_in = 1;
  CHECK(S.acquire(0, &l[4]) != 0 && s.pinned.size() == 1);
  for (int k = 0; k < 4; ++k) S.release(&l[k]);
  CHECK(s.pinned.empty() && !s.wrong);
""",
}


@pytest.mark.parametrize("case", CASES)
def test_shared(tmp_path, case):
    native.run(tmp_path, CASES[case], FAKE)
