// What the engine thread tells a flush: how many launches it has looked back on, the last of them that found work or did not
// get to look, and the last that found frames no neighbour had acknowledged.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstdint>

namespace st {

class QuietWatch {
 public:
  // ---- engine thread
  void begin() { looked_.store(launched_.load()); }  // launches of an earlier run that were not looked back on
  void launched() { launched_.fetch_add(1); }
  // `cut_short`: a group left before it had looked at its tiles (an update wanted the SMs, a wait ran out).  That says nothing
  // about them, so the launch does not count as one that found nothing.
  void looked(bool found_work, bool cut_short, uint64_t now_ns, bool unacknowledged = false) {
    const uint64_t n = looked_.load() + 1;
    if (unacknowledged) open_launch_.store(n);
    if (found_work || cut_short) {
      busy_ns_.store(now_ns);
      busy_launch_.store(n);
    }
    looked_.store(n);
  }

  // ---- flush
  uint64_t launches() const { return launched_.load(); }
  // The last `count` launches found nothing and were all begun after launch number `before`.  (The launches are read before
  // the busy one, which is written before them: a busy launch is never counted.)
  bool quiet_launches(uint64_t before, uint64_t count) const {
    const uint64_t n = looked_.load(), busy = busy_launch_.load();
    return n >= std::max(before, busy) + count;
  }
  // The last `count` launches found every frame acknowledged.
  bool acknowledged(uint64_t count) const {
    const uint64_t n = looked_.load(), open = open_launch_.load();
    return n >= open + count;
  }
  // Three passes (of `windows` launches each), all begun after launch number `before`, count nothing to do, and the last one no
  // frame without an acknowledgement (unless nobody is waited for: `alone`).  What a launch counts may be read along with the
  // counts of up to `ahead` launches before it, as many as may be in flight behind a launch whose counts are read: so that the
  // last pass has surely looked at all tiles and found nothing, nothing may have been counted in those either.
  bool settled(uint64_t before, uint64_t windows, uint64_t ahead, bool alone) const {
    return quiet_launches(before, std::max(3 * windows, windows + ahead)) && (alone || acknowledged(windows + ahead));
  }
  // How long no launch has found work, counted from `start_ns` at the earliest.  The engine thread may have found some since
  // the caller took the time.
  uint64_t quiet_for(uint64_t start_ns, uint64_t now_ns) const {
    const uint64_t since = std::max(start_ns, busy_ns_.load());
    return now_ns > since ? now_ns - since : 0;
  }

 private:
  std::atomic<uint64_t> launched_{0}, looked_{0}, busy_launch_{0}, busy_ns_{0}, open_launch_{0};
};

}  // namespace st
