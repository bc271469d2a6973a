// Which shared distance searches run before an admission pass.  Host code without CUDA, a
// function of the queue and the free slots alone.
#pragma once
#include <algorithm>
#include <map>
#include <vector>

namespace gst {

// A query that waits to be admitted.
struct Waiting {
  int kind;       // of the shared search it may take part in: 0 unbounded, D, or -1 none
  bool searched;  // a search has covered it; if not (and kind >= 0) it waits for one
};

// The kinds to search now, in the order their first waiting queries stand in the queue: those
// whose searched queries are fewer than the free slots.  An admission pass that steps over
// waiting queries (a batch) can take every searched one.  In arrival order (a server) it ends
// at the first waiting one, so only those ahead of it count: a query that comes back after a
// capacity overflow stands before queries that its first search covered too, and they can
// not be admitted until it has been searched again.  Counting those as well, a server whose
// head waited with as many behind it as it has slots neither searched nor admitted.
inline std::vector<int> kinds_due(const std::vector<Waiting>& queue, int free_slots, bool in_order) {
  std::map<int, int> ready;
  std::vector<int> seen, due;
  if (!in_order)
    for (const Waiting& w : queue) ready[w.kind] += w.searched;
  for (const Waiting& w : queue) {
    if (w.searched) {
      if (in_order) ready[w.kind]++;
    } else if (w.kind >= 0 && std::find(seen.begin(), seen.end(), w.kind) == seen.end()) {
      seen.push_back(w.kind);
      if (ready[w.kind] < free_slots) due.push_back(w.kind);
    }
  }
  return due;
}

}  // namespace gst
