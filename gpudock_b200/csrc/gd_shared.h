// gd_shared.h -- what the contexts of a device share: blocks of pinned memory.
//
// Pinning memory takes 1 .. 3 ms up to 1 MB, so a device's contexts share blocks
// of it, from the first of them to the last.  A block belongs to the device's
// CUDA context and ends with it (cudaDeviceReset), whether or not the handles
// that use it were destroyed first.  So blocks are kept by device and by the
// serial number of its CUDA context: a context created after a reset leaves the
// old block to the handles that still name it and starts a new one, and nothing
// of a block whose CUDA context is gone is handed out, written or given back to
// the runtime.  Where the serial number is not to be had (0), every context has
// a block of its own.
//
// Rt is the runtime (tests put one of their own in its place): the type Error,
// ok(Error), serial(), pin(void **, size_t) and unpin(void *), all of them about
// the current device.
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
  static constexpr int kSlots = 4;  // contexts per pinned block; later ones pin their own

  struct Group {
    int device = 0;
    uint64_t serial = 0;
    int users = 0;
    unsigned char *pinned = nullptr;
    unsigned used = 0;  // a bit per slot of `pinned`
  };
  // One context's part.
  struct Lease {
    Group *group = nullptr;
    void *block = nullptr;  // block_bytes of pinned memory
    int slot = -1;          // in group->pinned, or -1: pinned for this lease
  };

  explicit DeviceShared(size_t block_bytes, Rt rt = Rt()) : rt_(rt), block_bytes_(block_bytes) {}

  Rt &runtime() { return rt_; }

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

  // The lease's device is current.
  void release(Lease *l) {
    Group *g = l->group;
    if (!g) return;
    std::lock_guard<std::mutex> lk(mu_);
    const bool alive = rt_.serial() == g->serial;
    if (l->slot >= 0)
      g->used &= ~(1u << l->slot);
    else if (alive)
      rt_.unpin(l->block);
    *l = Lease{};
    if (--g->users > 0) return;
    if (alive) rt_.unpin(g->pinned);
    Group *&current = current_[g->device];
    if (current == g) current = nullptr;
    delete g;
  }

 private:
  Rt rt_;
  const size_t block_bytes_;
  std::mutex mu_;
  std::map<int, Group *> current_;  // by device
};

}  // namespace gd
