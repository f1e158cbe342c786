// Host state that the entry points share.
#pragma once
#include <atomic>

namespace cps {

// A persistent launch in flight on a device, from before it is queued until
// its results are back.  The flow solve asks whether it is the only one: its
// cluster form takes whole SMs and leaves no room for other contexts' launches
// beside it, the grid form (the same results) does.
class InFlight {
 public:
  explicit InFlight(int device)
      : count_(counts()[(unsigned)device % kDevices]), alone_(count_.fetch_add(1, std::memory_order_relaxed) == 0) {}
  ~InFlight() { count_.fetch_sub(1, std::memory_order_relaxed); }
  InFlight(const InFlight&) = delete;
  InFlight& operator=(const InFlight&) = delete;
  bool alone() const { return alone_; }  // when this launch was made

 private:
  static constexpr unsigned kDevices = 64;
  static std::atomic<int>* counts() {
    static std::atomic<int> c[kDevices];
    return c;
  }
  std::atomic<int>& count_;
  const bool alone_;
};

}  // namespace cps
