// gd_shared.h -- what the contexts of a device share: blocks of pinned memory,
// and the device memory kept for their calls' workspaces.
//
// Pinning memory takes 1 .. 3 ms up to 1 MB and mapping a workspace of tens of MB
// up to 10 ms, so a device's contexts have them together, from the first of them
// to the last.  Both belong to the device's CUDA context and end with it
// (cudaDeviceReset), whether or not the handles that use them were destroyed
// first.  So they are kept by device and by the serial number of its CUDA
// context: a context created after a reset leaves the old group to the handles
// that still name it and starts a new one, and nothing of a group whose CUDA
// context is gone is handed out, written or given back to the runtime.  Where
// the serial number is not to be had (0), every context has a group of its own.
//
// Workspaces (slabs) are lent to one call at a time.  The work of a call goes to
// its context's stream and may still run when the call returns a slab; the next
// call has it only if it is of the same context, whose stream orders the two, or
// if that work has ended.  No call waits for another: one that finds no slab
// makes a new one while all of them take at most `keep` bytes, or else allocates
// for itself.
//
// Rt is the runtime (tests put one of their own in its place): the types Error,
// Stream and Event, ok(Error), serial(), pin(void **, size_t), unpin(void *),
// alloc(void **, size_t, Stream), free(void *, Stream), event(Event *),
// record(Event, Stream), done(Event) and drop(Event), all of them about the
// current device.
#pragma once
#include <cstddef>
#include <cstdint>
#include <map>
#include <memory>
#include <mutex>

namespace gd {

template <class Rt>
class DeviceShared {
 public:
  using Error = typename Rt::Error;
  using Stream = typename Rt::Stream;
  static constexpr int kSlots = 4;  // contexts per pinned block; later ones pin their own
  static constexpr int kSlabs = 8;  // workspaces kept at most
  static constexpr size_t kStep = 1 << 20;

  struct Slab {
    unsigned char *p = nullptr;  // nullptr: no such slab
    size_t bytes = 0;
    const void *user = nullptr;  // the context whose call had it last
    bool lent = false;
    typename Rt::Event done{};  // the end of that call's work
  };
  struct Group {
    int device = 0;
    uint64_t serial = 0;
    int users = 0;
    unsigned char *pinned = nullptr;
    unsigned used = 0;  // a bit per slot of `pinned`
    Slab slabs[kSlabs];
  };
  // One context's part.
  struct Lease {
    Group *group = nullptr;
    void *block = nullptr;  // block_bytes of pinned memory
    int slot = -1;          // in group->pinned, or -1: pinned for this lease
  };

  // keep: most bytes of a device's slabs together
  DeviceShared(size_t block_bytes, size_t keep, Rt rt = Rt())
      : rt_(rt), block_bytes_(block_bytes), keep_(keep) {}

  // `device` is current.
  Error acquire(int device, Lease *out) {
    std::lock_guard<std::mutex> lk(mu_);
    const uint64_t serial = rt_.serial();
    Group *&current = current_[device];
    // a group of another serial: its CUDA context is gone, its users free it
    if (current && (serial == 0 || current->serial != serial)) current = nullptr;
    Error e{};
    std::unique_ptr<Group> fresh;
    if (!current) {
      fresh.reset(new Group);
      fresh->device = device;
      fresh->serial = serial;
      e = rt_.pin((void **)&fresh->pinned, block_bytes_ * kSlots);
      if (!rt_.ok(e)) return e;
    }
    Group *g = fresh ? fresh.get() : current;
    Lease l;
    l.group = g;
    for (int k = 0; k < kSlots && l.slot < 0; ++k)
      if (!(g->used >> k & 1u)) l.slot = k;
    if (l.slot >= 0) {
      l.block = g->pinned + (size_t)l.slot * block_bytes_;
      g->used |= 1u << l.slot;
    } else {
      e = rt_.pin(&l.block, block_bytes_);
      if (!rt_.ok(e)) return e;
    }
    g->users += 1;
    fresh.release();
    if (serial != 0) current = g;
    *out = l;
    return e;
  }

  // The lease's device is current; `user`'s work on s, its stream, has ended.
  void release(Lease *l, const void *user, Stream s) {
    Group *g = l->group;
    if (!g) return;
    std::lock_guard<std::mutex> lk(mu_);
    const bool alive = rt_.serial() == g->serial;
    if (l->slot >= 0)
      g->used &= ~(1u << l->slot);
    else if (alive)
      rt_.unpin(l->block);
    *l = Lease{};
    for (Slab &b : g->slabs)
      if (b.user == user) b.user = nullptr;
    if (--g->users > 0) return;
    if (alive) {
      rt_.unpin(g->pinned);
      for (Slab &b : g->slabs)
        if (b.p) discard(b, s);
    }
    Group *&current = current_[g->device];
    if (current == g) current = nullptr;
    delete g;
  }

  // A slab of at least `bytes` for a call of `user` on s, or nullptr.
  Slab *lend(Group *g, const void *user, Stream s, size_t bytes) {
    bytes = (bytes + kStep - 1) / kStep * kStep;
    if (bytes > keep_) return nullptr;
    std::lock_guard<std::mutex> lk(mu_);
    Slab *fit = nullptr;
    // the user's own first: no event is queried then (another thread of the
    // process may have a stream under capture, which a query can end)
    for (Slab &b : g->slabs)
      if (b.p && !b.lent && b.user == user && b.bytes >= bytes && (!fit || b.bytes < fit->bytes))
        fit = &b;
    if (fit) {
      fit->lent = true;
      return fit;
    }
    Slab *small = nullptr, *none = nullptr;
    size_t total = 0;
    for (Slab &b : g->slabs) {
      total += b.bytes;
      if (!b.p) none = &b;
      if (!b.p || !free_for(b, user)) continue;
      if (b.bytes < bytes) {
        if (!small || b.bytes < small->bytes) small = &b;
      } else if (!fit || b.bytes < fit->bytes) {
        fit = &b;
      }
    }
    if (!fit) {
      // in the place of a smaller one that nobody needs now, or beside the others
      if (small) {
        total -= small->bytes;
        discard(*small, s);
        none = small;
      }
      if (!none || total + bytes > keep_ || !make(*none, bytes, s)) return nullptr;
      fit = none;
    }
    fit->lent = true;
    return fit;
  }

  // The call's work is all on s.  want: what it would have needed, for the next.
  void give_back(Group *g, Slab *b, const void *user, Stream s, size_t want) {
    std::lock_guard<std::mutex> lk(mu_);
    size_t total = 0;
    for (const Slab &x : g->slabs) total += x.bytes;
    want = (want + kStep - 1) / kStep * kStep;
    b->lent = false;
    b->user = user;
    if (want > b->bytes && total - b->bytes + want <= keep_) {
      discard(*b, s);
      if (!make(*b, want, s)) return;
      b->user = user;
    }
    if (!rt_.ok(rt_.record(b->done, s))) discard(*b, s);
  }

 private:
  bool free_for(const Slab &b, const void *user) {
    return !b.lent && (b.user == user || rt_.done(b.done));
  }
  bool make(Slab &b, size_t bytes, Stream s) {
    b = Slab{};
    if (!rt_.ok(rt_.event(&b.done))) return false;
    if (!rt_.ok(rt_.alloc((void **)&b.p, bytes, s))) {
      rt_.drop(b.done);
      b = Slab{};
      return false;
    }
    b.bytes = bytes;
    return true;
  }
  // (in the order of s: its own work, or work that has ended)
  void discard(Slab &b, Stream s) {
    rt_.free(b.p, s);
    rt_.drop(b.done);
    b = Slab{};
  }

  Rt rt_;
  const size_t block_bytes_, keep_;
  std::mutex mu_;
  std::map<int, Group *> current_;  // by device
};

}  // namespace gd
