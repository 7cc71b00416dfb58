// One host thread instead of a team for small inputs (library-internal).
#pragma once
#include <omp.h>

#include <cstdint>

namespace bcg {

// Below this many vertices and this many arcs the host loops run on the calling thread: a
// loop over them takes less than waking a team, most of all where other work
// shares the cores. Graphs from edges on 16 threads / 1: rings with as many or 7
// times as many chords, 4,000 arcs 0.043 / 0.028 ms, 16,000 0.149 / 0.120, 32,000
// 0.184 / 0.167 and 0.226 / 0.252, 64,000 0.386 / 0.399.
constexpr int64_t kTeamWork = 1 << 15;
// The decomposition and a plan's routing do more for a vertex, their team pays
// earlier: the same graphs of 1,000 vertices 0.29 / 0.24 and 0.59 / 0.54 ms, of
// 2,000 0.52 / 0.51 and 1.07 / 1.11, of 4,000 0.94 / 1.07 and 1.94 / 1.95, of 8,000
// 1.60 / 2.19; PLAIN plans of 40 and 70 BA graphs (4,300 and 7,700 vertices) 0.29 /
// 0.35 and 0.42 / 0.58. The line lies where the gain begins to outweigh the waits
// for a team whose cores are busy with something else, milliseconds a call.
constexpr int64_t kTeamVertices = 1 << 12;

// Keeps the parallel regions that the calling thread meets in its lifetime to
// one thread, when the work is small (the setting is the calling thread's own).
class SmallTeam {
 public:
  SmallTeam(int64_t vertices, int64_t arcs, int64_t below = kTeamWork)
      : was_(vertices < below && arcs < kTeamWork ? omp_get_max_threads() : 0) {
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
