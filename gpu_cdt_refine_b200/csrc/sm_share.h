// Multiprocessors for cooperative launches that run side by side.
//
// A cooperative launch starts when all its blocks fit, so launches that each
// take the whole GPU run one after another.  A refinement or a triangulation is
// a chain of dependent loads that a part of the multiprocessors serves nearly as
// fast: contexts used by several threads are better off with a part each.  Every
// such call registers here with its size (triangles) for as long as it runs.  One
// that is alone takes what it asks for; beside others it takes the part of its
// size in the sum of sizes or, if that is more, what nobody holds or is about to
// take.  A launch that finds less free than it was given waits for another's end.
// The number of blocks never changes a result.
//
// Time of one call with four threads calling, each launch on the whole GPU and
// with this rule (B200; as launches of one phase each, before: in brackets):
// refinement of 10,000 points 3.4 and 2.7 ms (6.8), of 100,000 points 22.5 and
// 7.1 ms (12.6), of 300,000 points 25.7 and 10.8 ms (16.5); triangulation of
// 200,000 points 4.8 and 2.7 ms (3.6), of 1,000,000 points 12.0 and 9.8 ms (9.4).
#pragma once
#include <algorithm>
#include <mutex>

namespace gqm_share {

struct Device {
  std::mutex m;
  double size = 0.0;     // of all calls under way
  double waiting = 0.0;  // of those that hold no blocks, as far as they will soon take some
  int calls = 0, blocks = 0;
};
constexpr int kDevices = 64;
inline Device g_devices[kDevices];

// One call's registration.
class Ticket {
 public:
  Ticket() = default;
  Ticket(const Ticket &) = delete;
  Ticket &operator=(const Ticket &) = delete;
  ~Ticket() { close(); }
  // busy: the part of its time for which the call holds blocks
  void open(int device, double size, double busy) {
    close();
    if (device < 0 || device >= kDevices) return;
    d_ = &g_devices[device];
    size_ = std::max(1.0, size);
    soon_ = busy * size_;
    std::lock_guard<std::mutex> lock(d_->m);
    d_->calls++;
    d_->size += size_;
    d_->waiting += soon_;
  }
  void close() {
    if (!d_) return;
    give();
    std::lock_guard<std::mutex> lock(d_->m);
    d_->size -= size_;
    d_->waiting -= soon_;
    if (--d_->calls == 0) d_->size = d_->waiting = 0.0;  // no rounding is left behind
    d_ = nullptr;
  }
  // Blocks for this call's next launch: at most `want` of the `most` that can be
  // resident together.
  int take(int want, int most) {
    if (!d_) return want;
    give();
    std::lock_guard<std::mutex> lock(d_->m);
    d_->waiting -= soon_;
    int n = want;
    if (d_->calls > 1) {
      const double part = most * size_ / d_->size;
      const double free = most - d_->blocks - most * d_->waiting / d_->size;
      n = std::max(1, std::min(want, (int)std::max(part, free)));
    }
    held_ = n;
    d_->blocks += n;
    return n;
  }
  // The launch has ended.
  void give() {
    if (!held_) return;
    std::lock_guard<std::mutex> lock(d_->m);
    d_->blocks -= held_;
    d_->waiting += soon_;
    held_ = 0;
  }

 private:
  Device *d_ = nullptr;
  double size_ = 0.0, soon_ = 0.0;
  int held_ = 0;
};

}  // namespace gqm_share
