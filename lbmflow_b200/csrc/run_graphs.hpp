// The captured graphs of a loop, one per length, all for one key.
//
// A key holds everything that the captured launches were given; a graph of
// another key would replay the old arguments. Graphs are made when a call
// first needs their length, so one key's set grows over several calls.
#pragma once
#include <cstring>
#include <type_traits>

namespace lbmb {

// Key: plain bytes (compared with memcmp, padding zeroed by its maker).
// Graph: a handle, null when empty; Free: functor that frees one.
template <class Key, class Graph, class Free, int N>
class GraphSet {
 public:
  GraphSet() = default;
  GraphSet(const GraphSet&) = delete;
  GraphSet& operator=(const GraphSet&) = delete;
  ~GraphSet() { drop(); }

  Graph operator[](int i) const { return g_[i]; }

  void drop() {
    for (Graph& g : g_)
      if (g) {
        Free()(g);
        g = Graph();
      }
  }

  // Makes the graphs that `need` names exist for `key`: those of another key
  // go first, capture(i) makes a missing one. A capture that throws takes
  // every graph with it, so none is left whose key is not `key_`.
  template <class Capture>
  void prepare(const Key& key, const bool (&need)[N], const Capture& capture) {
    static_assert(std::is_trivially_copyable<Key>::value, "keys are compared byte by byte");
    if (std::memcmp(&key, &key_, sizeof(Key)) != 0) {
      drop();
      std::memcpy(&key_, &key, sizeof(Key));
    }
    try {
      for (int i = 0; i < N; ++i)
        if (need[i] && !g_[i]) g_[i] = capture(i);
    } catch (...) {
      drop();
      throw;
    }
  }

 private:
  Key key_{};
  Graph g_[N] = {};
};

}  // namespace lbmb
