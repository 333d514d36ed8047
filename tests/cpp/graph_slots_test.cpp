// csrc/graph_slots.h with numbers for graphs: prints how many graphs each pattern of calls captures, and how many are alive
// too long or twice destroyed at its end.
#include <cmath>
#include <cstdio>
#include <set>
#include "graph_slots.h"

struct Engine {
  lmw::GraphSlots<int> slots;
  std::set<int> alive;
  int next = 1, captures = 0, wrong = 0;
  int capture() {
    captures++;
    alive.insert(next);
    return next++;
  }
  void destroy(int g) { wrong += alive.erase(g) ? 0 : 1; }
  void step(double dt) {
    if (!slots.step(dt)) return;
    if (!slots.step_graph()) slots.keep_step(capture(), [&](int g) { destroy(g); });
    wrong += alive.count(slots.step_graph()) ? 0 : 1;
  }
  void chunk(double dt, int steps) {
    int g = slots.chunk(dt, steps);
    if (!g) {
      g = capture();
      slots.keep_chunk(dt, steps, g, [&](int x) { destroy(x); });
    }
    wrong += alive.count(g) ? 0 : 1;
  }
  void done(const char *name) {
    const int most = static_cast<int>(lmw::GraphSlots<int>::CHUNKS) + 1;
    wrong += static_cast<int>(alive.size()) > most ? 1 : 0;
    slots.clear([&](int g) { destroy(g); });
    wrong += static_cast<int>(alive.size());
    std::printf("%s %d %d\n", name, captures, wrong);
  }
};

int main() {
  {
    Engine e;  // step(dt) between runs, each with two chunk lengths of its own step size
    for (int k = 0; k < 100; k++) {
      e.step(600.0);
      e.chunk(500.0 + k, 64);
      e.chunk(500.0 + k, 17);
    }
    e.done("alternating");
  }
  {
    Engine e;  // a guard-sized chunk in every run, remainders of many lengths
    for (int k = 0; k < 100; k++) {
      e.chunk(600.0, 64);
      e.chunk(600.0, 4 + k % 60);
    }
    e.done("remainders");
  }
  {
    Engine e;  // a few steps with each of many step sizes; not a number never takes a graph
    for (int k = 0; k < 100; k++)
      for (int i = 0; i < 2; i++) e.step(600.0 + k);
    for (int i = 0; i < 100; i++) e.step(std::nan(""));
    e.done("short");
  }
  {
    Engine e;  // two step sizes, many steps each, with the engine's graphs dropped in between
    for (int k = 0; k < 4; k++) {
      for (int i = 0; i < 50; i++) e.step(k & 1 ? 300.0 : 600.0);
      e.slots.clear([&](int g) { e.destroy(g); });
      for (int i = 0; i < 50; i++) e.step(k & 1 ? 300.0 : 600.0);
    }
    e.done("long");
  }
  return 0;
}
