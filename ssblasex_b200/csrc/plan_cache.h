// Which plans of grouped calls are kept, found again and dropped. Free of CUDA, so that it is unit-tested on
// the CPU.
#pragma once

#include <stddef.h>

#include <memory>
#include <utility>
#include <vector>

namespace ssb {

// Plan: `size_t scratch` (bytes), `unsigned long tick` (last use, set here) and `bool captured`: a CUDA graph
// holds launches of it. At most MAX_PLANS others are kept, and beyond the newest of them only as long as
// their scratch stays within MAX_SCRATCH; a captured plan stays until clear(), since the graph holds its
// addresses, and is left to graphs, since no ordinary call can tell when they run.
template <class Plan, size_t MAX_PLANS, size_t MAX_SCRATCH>
class PlanCache {
 public:
  // A plan that `match` accepts, for an ordinary call or one under capture (which may take either kind, a
  // captured one first).
  template <class Match>
  Plan* find(bool captured, const Match& match) {
    Plan* other = nullptr;
    for (auto& p : plans_) {
      if (p->captured && !captured) continue;
      if (other && !p->captured) continue;
      if (!match(*p)) continue;
      if (p->captured == captured) return p.get();
      other = p.get();
    }
    return other;
  }
  // Drops the least recently used plans until one of `scratch` bytes fits beside the others.
  void make_room(size_t scratch) {
    for (;;) {
      size_t oldest = plans_.size(), count = 0, bytes = scratch;
      for (size_t i = 0; i < plans_.size(); ++i) {
        if (plans_[i]->captured) continue;
        ++count;
        bytes += plans_[i]->scratch;
        if (oldest == plans_.size() || plans_[i]->tick < plans_[oldest]->tick) oldest = i;
      }
      if (count == 0 || (count < MAX_PLANS && bytes <= MAX_SCRATCH)) return;
      plans_.erase(plans_.begin() + (long)oldest);
    }
  }
  Plan* add(std::unique_ptr<Plan> p) {
    plans_.push_back(std::move(p));
    return plans_.back().get();
  }
  void use(Plan& p) { p.tick = ++tick_; }
  void clear() { plans_.clear(); }
  size_t size() const { return plans_.size(); }

 private:
  std::vector<std::unique_ptr<Plan>> plans_;
  unsigned long tick_ = 0;
};

}  // namespace ssb
