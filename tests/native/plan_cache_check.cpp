// PlanCache: a plan whose upload fails half-way is not kept, and the next call builds it again;
// a plan that the planner refuses is asked for once; a complete one is built once.
#include <cstdio>
#include <new>

#include "internal.h"

struct Bufs {
  int n = 0;
  bool complete = false;
};

int main() {
  mpf::PlanCache<std::pair<int, int>, Bufs> cache;
  int built = 0;
  bool fail = true;
  auto build = [&](Bufs& b) {
    ++built;
    b.n = 7;
    if (fail) throw std::bad_alloc();  // the first of its uploads
    b.complete = true;
    return true;
  };
  for (int k = 0; k < 2; ++k) {
    bool threw = false;
    try {
      cache.get({4, 8}, build);
    } catch (const std::bad_alloc&) {
      threw = true;
    }
    if (!threw || built != k + 1) return 1;
  }
  fail = false;
  const Bufs* p = cache.get({4, 8}, build);
  if (!p || !p->complete || p->n != 7 || built != 3) return 2;
  if (cache.get({4, 8}, build) != p || built != 3) return 3;
  int asked = 0;
  for (int k = 0; k < 2; ++k)
    if (cache.get({8, 8}, [&](Bufs&) { return ++asked < 0; }) != nullptr) return 4;
  if (asked != 1) return 5;
  cache.clear();
  if (!cache.get({4, 8}, build) || built != 4) return 6;
  std::printf("ok\n");
  return 0;
}
