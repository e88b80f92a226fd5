// Sweep plans of several grids in one handle, some without a variable in B'' (every bus but the
// slack is PV): each island of the handle has its range of steps, empty where it has no
// supernode, and the islands' steps together are the plan.
#include <cstdio>
#include <numeric>

#include "internal.h"

using namespace mpf;

int main() {
  long plans = 0;
  // buses of each grid; negative: all PV
  const std::vector<std::vector<int>> sets = {{30, -6}, {-6, 30}, {30, -6, 12, -2}, {-6, -9}, {-2, -2, -2}};
  for (auto& set : sets) {
    std::vector<mpf_bus> bus;
    std::vector<mpf_branch> br;
    for (int nb : set) {
      const int n = nb < 0 ? -nb : nb, off = (int)bus.size();
      for (int i = 0; i < n; ++i)
        bus.push_back(mpf_bus{i == 0 ? MPF_BUS_SLACK : nb < 0 ? MPF_BUS_PV : MPF_BUS_PQ, 0, 1.0, 0.0, -0.01, 0.0, 0.0, 0.0});
      for (int i = 1; i < n; ++i) br.push_back(mpf_branch{off + (i - 1) / 2, off + i, 1, 0, 0.02, 0.1, 0.0, 0.0, 0.0});
      if (n > 3) br.push_back(mpf_branch{off + n - 1, off + 1, 1, 0, 0.02, 0.1, 0.0, 0.0, 0.0});
    }
    GridSymbolic g;
    const std::string msg = build_symbolic(bus.data(), (int)bus.size(), br.data(), (int)br.size(), g);
    if (!msg.empty() || g.n_islands != (int)set.size()) {
      std::printf("%s\n", msg.c_str());
      return 1;
    }
    auto check = [&](const LUSymbolic& s, const std::vector<int>& var, const std::vector<int>* var2) {
      std::vector<int> vi(s.n, 0), si, count(g.n_islands, 0);
      for (int i = 0; i < g.nb; ++i) {
        if (var[i] >= 0) vi[var[i]] = g.bus_island[i];
        if (var2 && (*var2)[i] >= 0) vi[(*var2)[i]] = g.bus_island[i];
      }
      for (int k = 0; k < s.nsn; ++k) {
        si.push_back(vi[s.sn_rows[s.sn_rptr[k]]]);
        ++count[si.back()];
      }
      for (bool compact : {false, true}) {
        SweepPlan P;
        if (!build_sweep_plan(s, si, compact, 4, 8, 8 * 1024, 16 * 1024, P, g.n_islands)) return false;
        if ((int)P.step_ptr.size() != g.n_islands + 1 || (int)P.down_ptr.size() != g.n_islands) return false;
        if (P.step_ptr[0] != 0 || P.step_ptr.back() != (int)P.step.size()) return false;
        for (int k = 0; k < g.n_islands; ++k) {
          const int a = P.step_ptr[k], b = P.step_ptr[k + 1], d = P.down_ptr[k];
          int up = 0, down = 0;  // supernodes of each direction
          for (int q = a; q < b; ++q) {
            if ((q < d) != (P.step[q].up == 1)) return false;
            (q < d ? up : down) += P.step[q].nsolo + P.step[q].nbig;
          }
          if (a > b || d < a || d > b || up != count[k] || down != count[k]) return false;
        }
        ++plans;
      }
      return true;
    };
    bool ok = check(g.jac, g.var_va, &g.var_vm);
    for (int v = 0; v < 2; ++v) ok = ok && check(g.bp[v].lu, g.bp[v].var, nullptr) && check(g.bpp[v].lu, g.bpp[v].var, nullptr);
    if (!ok) {
      std::printf("bad plan: %d islands, first of %d buses\n", g.n_islands, set[0]);
      return 1;
    }
  }
  std::printf("plans %ld\n", plans);
  return 0;
}
