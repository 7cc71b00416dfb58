// One host thread instead of a team for small inputs (library-internal).
#pragma once
#include <omp.h>

#include <cstdint>

namespace bcg {

// Below this many vertices and this many arcs the host loops run on the calling thread: a
// loop over them takes less than waking a team, most of all where other work
// shares the cores. Decomposition of random graphs of 8 edges a vertex on 8
// threads / 1: 1,000 vertices 0.60 / 0.40 ms, 2,000 1.14 / 0.94, 4,000 1.98 /
// 2.02, 8,000 2.86 / 3.97.
constexpr int64_t kTeamWork = 1 << 15;

// Keeps the parallel regions that the calling thread meets in its lifetime to
// one thread, when the work is small (the setting is the calling thread's own).
class SmallTeam {
 public:
  SmallTeam(int64_t vertices, int64_t arcs)
      : was_(vertices < kTeamWork && arcs < kTeamWork ? omp_get_max_threads() : 0) {
    if (was_) omp_set_num_threads(1);
  }
  ~SmallTeam() {
    if (was_) omp_set_num_threads(was_);
  }
  SmallTeam(const SmallTeam &) = delete;
  SmallTeam &operator=(const SmallTeam &) = delete;

 private:
  int was_;
};

}  // namespace bcg
