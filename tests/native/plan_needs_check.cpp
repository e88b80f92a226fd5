// What is known of the plans before they are built: sweep_peak_cb is every compact sweep plan's
// peak; a factorisation plan is built exactly where factor_needs says that its largest task fits
// a ring slot and its contribution blocks with one front the rest, and costs no less than the
// needs' cycles.  Small transmission grids have factorisation plans at every lane count (a uniform random graph need not).
#include <cstdio>

#include "internal.h"

using namespace mpf;

int main() {
  long built = 0, refused = 0, sweeps = 0;
  const int shapes[][5] = {{30, 41, 5, 0, 0}, {118, 179, 53, 0, 0}, {300, 411, 69, 0, 0}, {300, 435, 60, 1, 0},
                           {1354, 1991, 259, 0, 0}, {1354, 1991, 259, 1, 1}, {2869, 4582, 509, 0, 1}};
  for (auto& sh : shapes) {
    std::vector<mpf_bus> bus(sh[0]);
    std::vector<mpf_branch> br(sh[1]);
    mpf_synth_params p;
    mpf_synth_default(&p);
    p.n_bus = sh[0];
    p.n_branch = sh[1];
    p.n_pv = sh[2];
    p.topology = sh[3];
    p.seed = 3;
    GridSymbolic g;
    if (mpf_synth_grid(&p, bus.data(), br.data()) != 0 ||
        !build_symbolic(bus.data(), sh[0], br.data(), sh[1], g).empty())
      return 1;
    for (const LUSymbolic* s : {&g.jac, &g.bp[0].lu, &g.bpp[1].lu})
      for (int G : {8, 1})
        for (size_t slot : {(size_t)6 * 1024, (size_t)48 * 1024}) {
          SweepPlan P;
          if (!build_sweep_plan(*s, {}, true, G, 4, slot, 16 * 1024, P)) continue;
          ++sweeps;
          if (P.peak_cb != sweep_peak_cb(*s, {})) return 2;
        }
    const FactorNeeds needs = factor_needs(g.jac, g.ah_ptr);
    for (int ws : {4, 8})
      for (int G = 32 / ws; G >= 1; G /= 2) {
        bool any = false;
        for (size_t slot = 24 * 1024; slot >= 3 * 1024; slot = slot * 2 / 3 / 16 * 16) {
          const size_t smem = 200 * 1024 - 3 * slot;
          FactorPlan P;
          const bool ok = build_factor_plan(g.jac, g.ah_ptr, g.ah_loc, G, ws, slot, smem, P);
          if (ok != needs.fits(G, ws, slot, smem)) {
            std::printf("%d buses, G %d, value %d, slot %zu: built %d\n", sh[0], G, ws, slot, (int)ok);
            return 3;
          }
          if (ok && (P.cycles < needs.cycles || P.peak_cb != needs.peak_cb || P.most < needs.front)) return 4;
          any = any || ok;
          ++(ok ? built : refused);
        }
        if (!any && sh[0] <= 300 && sh[3] == 0) {
          std::printf("no plan: %d buses, G %d, value %d\n", sh[0], G, ws);
          return 5;
        }
        if (sh[4] && G * ws == 32 && any) return 6;  // (these must be refused)
      }
  }
  std::printf("built %ld refused %ld sweeps %ld\n", built, refused, sweeps);
  return 0;
}
