// side_streams.h -- which of a few streams each of a batch's single launches
// takes (host logic, no CUDA).  Launches on one graph share its workspace, so
// they follow one another on one stream; different graphs take the streams in
// turn.  A graph is its handle: a batch may list one handle at several indices.
#pragma once

#include <cstddef>
#include <utility>
#include <vector>

namespace grus {

// How many of the single launches run at a time, with one CTA an SM each, and
// whether the workers' kernel runs beside them.  Its CTAs and theirs take a slot
// each, of which an SM has `per_sm`; the launches wait at grid barriers, so all
// their CTAs have to find one whatever the workers hold.  The workers keep to the
// slots that are left; where that is fewer than half as many workers as there
// are tasks, or leaves one launch at a time, the kernel waits for the launches.
struct SidePlan {
  int streams;
  int workers;  // of the workers' kernel
  bool beside;
};

inline SidePlan plan_sides(int most, int per_sm, int sms, int cluster, int workers, int tasks) {
  const int w = tasks < workers ? tasks : workers;
  const int all = most < per_sm ? most : per_sm;
  if (tasks == 0) return {all, workers, false};
  for (int k = all; k >= 2; --k) {
    const int room = (per_sm - k) * sms / cluster;
    if (w <= room) return {k, w, true};
    if (k == 2 && room > 0 && tasks <= 2 * room) return {k, room < w ? room : w, true};
  }
  return {all, workers, false};
}

class SideStreams {
 public:
  explicit SideStreams(int streams) : n_(streams) {}
  void limit(int streams) { n_ = streams; }  // before the first of()
  int of(const void *graph) {
    for (const auto &g : at_)
      if (g.first == graph) return g.second;
    at_.emplace_back(graph, (int)(at_.size() % (size_t)n_));
    return at_.back().second;
  }
  size_t graphs() const { return at_.size(); }

 private:
  int n_;
  std::vector<std::pair<const void *, int>> at_;
};

}  // namespace grus
