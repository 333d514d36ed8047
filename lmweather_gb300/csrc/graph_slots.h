// The captured step graphs that an engine keeps. A run's chunks (keyed by step size and length: the guard-sized chunk and
// the remainders) share CHUNKS slots, of which the least recently used gives way. step() has one slot of its own, so that a
// program that alternates step() with runs of many lengths does not lose its graph to them.
#pragma once
#include <algorithm>
#include <vector>

namespace lmw {

template <class Exec> class GraphSlots {
 public:
  static constexpr size_t CHUNKS = 4;
  // step() with one dt is launched kernel by kernel this often before its graph is captured: the capture costs what the graph
  // saves in eight to ten steps (T21: 39 us against 87 - 83 us a step; T42: 40 against 101 - 96)
  static constexpr int REPEATS = 8;

  // the graph of `steps` steps of dt, or null
  Exec chunk(double dt, int steps) {
    for (size_t i = 0; i < chunks.size(); i++)
      if (chunks[i].dt == dt && chunks[i].steps == steps) {
        std::rotate(chunks.begin() + static_cast<long>(i), chunks.begin() + static_cast<long>(i) + 1, chunks.end());
        return chunks.back().exec;
      }
    return Exec{};
  }
  template <class Destroy> void keep_chunk(double dt, int steps, Exec g, Destroy destroy) {
    if (chunks.size() >= CHUNKS) {
      destroy(chunks.front().exec);
      chunks.erase(chunks.begin());
    }
    chunks.push_back({dt, steps, g});
  }

  // one more step() of dt: true when it takes a graph, step_graph() or, where that is null, one captured now
  bool step(double dt) {
    if (dt != step_dt) {
      step_dt = dt;
      seen = 0;
    }
    return ++seen > REPEATS;
  }
  Exec step_graph() const { return step_dt == kept_dt ? kept : Exec{}; }
  template <class Destroy> void keep_step(Exec g, Destroy destroy) {
    if (kept) destroy(kept);
    kept = g;
    kept_dt = step_dt;
  }

  template <class Destroy> void clear(Destroy destroy) {
    for (const Chunk &c : chunks) destroy(c.exec);
    chunks.clear();
    if (kept) destroy(kept);
    kept = Exec{};
  }

 private:
  struct Chunk {
    double dt;
    int steps;
    Exec exec;
  };
  std::vector<Chunk> chunks;
  double step_dt = 0, kept_dt = 0;
  int seen = 0;  // step() calls in a row with step_dt
  Exec kept{};
};

}  // namespace lmw
