// Which limit of dynamic shared memory each kernel has been given, so that it is set when it has to rise and
// not at every launch.  Host code only.
#pragma once
#include <cstddef>
#include <map>
#include <mutex>
#include <utility>

namespace cssm {

// The limit is one attribute of a kernel that all threads share, and a launch reads it some time after
// raise() has returned.  So it never falls (a smaller request of another thread must not undercut a launch
// that is still to come), and check, call and record are one step under the lock: when raise() returns
// success the limit holds `bytes` and keeps doing so.
//
// The attribute lives as long as the context it was set in: `context` is an id that is never given twice, so
// that after a cudaDeviceReset nothing is believed that was set before (0: unknown, nothing is remembered).
class SmemLimits {
 public:
  // get(&limit) reads the limit in force, set(bytes) changes it; both return 0 on success
  template <class Get, class Set>
  int raise(const void* kern, unsigned long long context, std::size_t bytes, Get&& get, Set&& set) {
    std::lock_guard<std::mutex> lock(mu_);
    const auto it = known_.find({kern, context});
    if (context != 0 && it != known_.end() && it->second >= bytes) return 0;
    std::size_t now = 0;
    int e = get(&now);
    if (e == 0 && now < bytes) {
      e = set(bytes);
      now = bytes;
    }
    if (e == 0 && context != 0) {
      if (known_.size() >= MAX_KNOWN) known_.clear();      // of dead contexts, mostly; the rest is read again
      known_[{kern, context}] = now;
    }
    return e;
  }

 private:
  static constexpr std::size_t MAX_KNOWN = 4096;
  std::mutex mu_;
  std::map<std::pair<const void*, unsigned long long>, std::size_t> known_;
};

}  // namespace cssm
