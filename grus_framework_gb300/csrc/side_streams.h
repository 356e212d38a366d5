// side_streams.h -- which of a few streams each of a batch's single launches
// takes (host logic, no CUDA).  Launches on one graph share its workspace, so
// they follow one another on one stream; different graphs take the streams in
// turn.  A graph is its handle: a batch may list one handle at several indices.
#pragma once

#include <cstddef>
#include <utility>
#include <vector>

namespace grus {

class SideStreams {
 public:
  explicit SideStreams(int streams) : n_(streams) {}
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
