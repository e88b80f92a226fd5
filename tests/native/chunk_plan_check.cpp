// Checks build_sweep_plan on the Newton, B' and B'' systems of synthetic grids (one island
// and two): a step's panels are adjacent and fit its slot with its index block, its teams fit
// the block, its warps, its named barriers and the scratch; and both pairs of substitutions
// walked over the plan, each step reading only its own index block and what earlier steps
// wrote, equal a plain supernode-by-supernode substitution on random panels.  Prints the number of plans and the
// largest relative difference.
#include <cmath>
#include <cstdio>
#include <vector>

#include "internal.h"

using namespace mpf;

static long plans = 0;
static double worst = 0.0;

enum { FWD, BWD, FWD_T, BWD_T };

// plain substitution: supernodes in level order, carried entries in cbr
static std::vector<double> plain(const LUSymbolic& s, const std::vector<double>& pan, std::vector<double> x, int kind) {
  const bool up = kind == FWD || kind == FWD_T;
  std::vector<double> c(s.cbr_off.back() + 1, 0.0);
  for (int q = 0; q < (int)s.lev_sn.size(); ++q) {
    const int n = s.lev_sn[up ? q : (int)s.lev_sn.size() - 1 - q];
    const int w = s.sn_w[n], f = s.sn_f[n];
    const int* rows = &s.sn_rows[s.sn_rptr[n]];
    const double* P = &pan[s.pan_off[n]];
    auto Lv = [&](int i, int p) { return i < w ? P[i * f + p] : P[w * f + (i - w) * w + p]; };
    std::vector<double> b(f, 0.0);
    for (int i = 0; i < f; ++i) b[i] = (i < w || !up) ? x[rows[i]] : 0.0;
    if (up) {
      for (int e = s.child_ptr[n]; e < s.child_ptr[n + 1]; ++e) {
        const int ch = s.child_list[e];
        for (int a = 0; a < s.sn_f[ch] - s.sn_w[ch]; ++a) b[s.relmap[s.rel_ptr[ch] + a]] += c[s.cbr_off[ch] + a];
      }
      for (int p = 0; p < w; ++p) {
        if (kind == FWD_T) b[p] /= P[p * f + p];
        for (int i = p + 1; i < f; ++i) b[i] -= (kind == FWD ? Lv(i, p) : P[p * f + i]) * b[p];
      }
      if (s.sn_parent[n] >= 0)
        for (int a = 0; a < f - w; ++a) c[s.cbr_off[n] + a] = b[w + a];
    } else {
      for (int p = w - 1; p >= 0; --p) {
        for (int i = p + 1; i < f; ++i) b[p] -= (kind == BWD ? P[p * f + i] : Lv(i, p)) * b[i];
        if (kind == BWD) b[p] /= P[p * f + p];
      }
    }
    for (int p = 0; p < w; ++p) x[rows[p]] = b[p];
  }
  return x;
}

static bool check(const LUSymbolic& s, const std::vector<int>& isl, bool compact, int G, int wsize, size_t slot, Rng& rng) {
  const size_t scratch = 16 * 1024;
  SweepPlan P;
  if (!build_sweep_plan(s, isl, compact, G, wsize, slot, scratch, P)) {
    // refused only where a front does not fit the scratch
    for (int n = 0; n < s.nsn; ++n)
      if ((size_t)(s.sn_f[n] + 3) / 4 * 4 * G * wsize > scratch) return true;
    std::printf("refused without a reason\n");
    return false;
  }
  ++plans;
  std::vector<double> pan(s.nnz), x0(s.n);
  for (double& v : pan) v = rng.uniform() - 0.5;
  for (int n = 0; n < s.nsn; ++n)
    for (int p = 0; p < s.sn_w[n]; ++p) pan[s.pan_off[n] + (size_t)p * s.sn_f[n] + p] = 8.0 + rng.uniform();
  for (double& v : x0) v = rng.uniform() - 0.5;
  int nisl = 1;
  for (int v : isl) nisl = v + 1 > nisl ? v + 1 : nisl;
  if ((int)P.step_ptr.size() != nisl + 1 || (int)P.down_ptr.size() != nisl) return false;
  for (int k = 0; k < nisl; ++k)  // up to down_ptr leaves to root, then root to leaves
    for (int q = P.step_ptr[k]; q < P.step_ptr[k + 1]; ++q)
      if ((P.step[q].up != 0) != (q < P.down_ptr[k])) return false;
  size_t most = 0, widest = 0;
  for (bool tr : {false, true}) {
    std::vector<double> x = x0;
    std::vector<int> seen(s.n, 0);
    for (int k = 0; k < nisl; ++k) {
      std::vector<double> c(compact ? P.peak_cb + 1 : s.cbr_off.back() + 1, std::nan(""));
      for (int q = P.step_ptr[k]; q < P.step_ptr[k + 1]; ++q) {
        // the kernel reads the record's first four ints from the step array, the rest and
        // everything else from the step's index block
        const SweepStep& R = P.step[q];
        if (R.i0 % 4 || R.ni % 4 || R.i0 + R.ni > (int)P.idx.size() || R.e0 + R.ne > s.nnz) return false;
        const size_t bytes = ((size_t)R.ne * G * wsize + 15) / 16 * 16 + (size_t)R.ni * 4;
        if (bytes > slot) return false;
        if (bytes > widest) widest = bytes;
        const int* ib = &P.idx[R.i0];
        const bool up = ib[4] != 0;
        const int split = 1 << ib[5], nsolo = ib[6], nbig = ib[7], team = 1 << ib[8], nteams = ib[9], xstride = ib[10], direct = ib[11];
        if (direct && (R.ne != 0 || nsolo != 0 || nbig != 1 || ib[0] != R.e0 || ib[2] != R.i0)) return false;
        if (split < 1 || split * G > 32 || (split & (split - 1))) return false;
        if (nbig > 0) {
          if (team % 32 || nteams < 1 || team * nteams > kChunkThreads || (team > 32 && nteams > 15)) return false;
          if ((size_t)nteams * xstride * G * wsize > scratch) return false;
          if ((size_t)nteams * xstride > most) most = (size_t)nteams * xstride;
        } else if (nteams != 0) {
          return false;
        }
        const std::vector<double> cr = c, xr = x;  // what earlier steps left
        std::vector<char> cw(c.size(), 0);
        for (int t = 0; t < nsolo + nbig; ++t) {
          const int* h = ib + kStepInts + 4 * t;
          const int w = h[1] & 0xffff, f = h[1] >> 16, cbo = h[3];
          if ((t < nsolo) != (solo_task(w, f) && !direct) || (t >= nsolo && f > xstride)) return false;
          if (!direct && h[0] + w * (2 * f - w) > R.ne) return false;
          const int* xi = ib + h[2] + (up ? 2 : 0);
          const int layers = up ? xi[-2] : 0;
          const int* pr = xi + ((w + 1) & ~1);
          if (up && (pr - &P.idx[0]) % 2) return false;
          if ((up ? pr + 2 * f * layers : xi + f) > (direct ? &P.idx[0] + P.idx.size() : ib + R.ni)) return false;
          const double* M = &pan[R.e0 + h[0]];
          auto Lv = [&](int i, int p) { return i < w ? M[i * f + p] : M[w * f + (i - w) * w + p]; };
          std::vector<double> b(f, 0.0);
          for (int i = 0; i < (up ? w : f); ++i) b[i] = xr[xi[i]];
          if (up) {
            for (int e = 0; e < layers; ++e)
              for (int i = 0; i < f; ++i)
                for (int z = 0; z < 2; ++z)
                  if (pr[2 * (e * f + i) + z] >= 0) b[i] += cr[pr[2 * (e * f + i) + z]];
            for (int p = 0; p < w; ++p) {
              if (tr) b[p] /= M[p * f + p];
              for (int i = p + 1; i < f; ++i) b[i] -= (tr ? M[p * f + i] : Lv(i, p)) * b[p];
            }
            for (int a = 0; a < f - w && cbo >= 0; ++a) {
              if (cbo + a >= (int)c.size() || cw[cbo + a]) return false;
              cw[cbo + a] = 1;
              c[cbo + a] = b[w + a];
            }
          } else {
            for (int p = w - 1; p >= 0; --p) {
              for (int i = p + 1; i < f; ++i) b[p] -= (tr ? Lv(i, p) : M[p * f + i]) * b[i];
              if (!tr) b[p] /= M[p * f + p];
            }
          }
          for (int p = 0; p < w; ++p) {
            x[xi[p]] = b[p];
            ++seen[xi[p]];
          }
        }
      }
    }
    for (int v : seen)
      if (v != 2) return false;
    const std::vector<double> ref = plain(s, pan, plain(s, pan, x0, tr ? FWD_T : FWD), tr ? BWD_T : BWD);
    for (int i = 0; i < s.n; ++i) {
      const double e = std::fabs(x[i] - ref[i]) / (1.0 + std::fabs(ref[i]));
      if (!(e < 1e-12)) return false;
      if (e > worst) worst = e;
    }
  }
  return most == P.scratch && widest == P.slot;
}

// The factorisation's plan: its steps hold every arrowhead value once, in order; a step fits
// its slot, its teams and warps the block and the shared memory; contribution blocks are
// written once per slot and step and read only in later steps.  The factorisation walked over
// the plan equals the dense front-by-front one bit for bit.
static bool check_factor(const LUSymbolic& s, const std::vector<int>& ah_ptr, const std::vector<int>& ah_loc, int G,
                         int wsize, size_t slot, size_t smem, Rng& rng) {
  auto area = [](int f) { return (size_t)f * ((f + 1) | 1); };
  FactorPlan P;
  if (!build_factor_plan(s, ah_ptr, ah_loc, G, wsize, slot, smem, P)) return true;
  ++plans;
  const int nA = ah_ptr[s.nsn];
  std::vector<double> A(nA), x0(s.n);
  for (double& v : A) v = rng.uniform() - 0.5;
  for (int n = 0; n < s.nsn; ++n)
    for (int e = ah_ptr[n]; e < ah_ptr[n + 1]; ++e) {
      const int RS = (s.sn_f[n] + 1) | 1;
      if (ah_loc[e] / RS == ah_loc[e] % RS) A[e] = 20.0 + rng.uniform();
    }
  for (double& v : x0) v = rng.uniform() - 0.5;
  // a front's partial LU, right-looking (columns f: the right-hand side)
  auto lu = [](std::vector<double>& F, int f, int w) {
    const int RS = (f + 1) | 1;
    for (int p = 0; p < w; ++p) {
      const double inv = 1.0 / F[p * RS + p];
      for (int i = p + 1; i < f; ++i) {
        const double l = F[i * RS + p] * inv;
        F[i * RS + p] = l;
        for (int q = p + 1; q <= f; ++q) F[i * RS + q] -= l * F[p * RS + q];
      }
    }
  };
  std::vector<double> pan(s.nnz, 0.0), ref(s.nnz, 0.0), x = x0, xr = x0;
  {
    std::vector<std::vector<double>> cb(s.nsn);
    for (int q = 0; q < s.nsn; ++q) {
      const int n = s.lev_sn[q], w = s.sn_w[n], f = s.sn_f[n], m = f - w, RS = (f + 1) | 1;
      std::vector<double> F((size_t)f * RS, 0.0);
      for (int e = ah_ptr[n]; e < ah_ptr[n + 1]; ++e) F[ah_loc[e]] = A[e];
      for (int p = 0; p < w; ++p) F[p * RS + f] = xr[s.sn_rows[s.sn_rptr[n] + p]];
      for (int c = s.child_ptr[n]; c < s.child_ptr[n + 1]; ++c) {
        const int ch = s.child_list[c], mc = s.sn_f[ch] - s.sn_w[ch];
        const int* rel = &s.relmap[s.rel_ptr[ch]];
        for (int a = 0; a < mc; ++a) {
          for (int b = 0; b < mc; ++b) F[rel[a] * RS + rel[b]] += cb[ch][a * mc + b];
          F[rel[a] * RS + f] += cb[ch][mc * mc + a];
        }
      }
      lu(F, f, w);
      for (int i = 0; i < f; ++i)
        for (int j = 0; j < (i < w ? f : w); ++j) ref[s.pan_off[n] + (i < w ? i * f + j : w * f + (i - w) * w + j)] = F[i * RS + j];
      for (int p = 0; p < w; ++p) xr[s.sn_rows[s.sn_rptr[n] + p]] = F[p * RS + f];
      cb[n].resize(m * m + m);
      for (int a = 0; a < m; ++a) {
        for (int b = 0; b < m; ++b) cb[n][a * m + b] = F[(w + a) * RS + w + b];
        cb[n][m * m + a] = F[(w + a) * RS + f];
      }
    }
  }
  std::vector<double> cb(P.peak_cb + 1, std::nan(""));
  int at = 0;
  size_t most = 0;
  for (const FactorStep& st : P.step) {
    if (st.e0 != at || st.i0 % 4 || st.ni % 4 || st.i0 + st.ni > (int)P.idx.size()) return false;
    at += st.ne;
    const size_t bytes = ((size_t)st.ne * G * wsize + 15) / 16 * 16 + (size_t)st.ni * 4;
    if (bytes > slot || bytes > P.slot) return false;
    const int* ib = &P.idx[st.i0];
    const int nbig = ib[4], nsmall = ib[5], lteam = ib[6], nteams = ib[7], bstride = ib[8], sstride = ib[9];
    const int busy = nteams << lteam;
    if (busy > kChunkThreads || (nbig > 0) != (nteams > 0) || (lteam > 5 && nteams > 15)) return false;
    if ((size_t)bstride * G * wsize % 16 || (size_t)sstride * G * wsize % 16) return false;
    const size_t big = (size_t)nteams * bstride;
    const size_t small = nsmall > 0 ? (kChunkThreads - (busy < kChunkThreads ? busy : 0)) / 32 * (size_t)sstride : 0;
    const size_t held = busy < kChunkThreads ? big + small : big > small ? big : small;
    if (held > most) most = held;
    const std::vector<double> cr = cb, xs = x;
    std::vector<char> cw(cb.size(), 0);
    for (int t = 0; t < nbig + nsmall; ++t) {
      const int* h = ib + kStepInts + 8 * t;
      const int na = h[1], w = h[2] & 0xffff, f = h[2] >> 16, m = f - w, RS = (f + 1) | 1;
      if (area(f) > (size_t)(t < nbig ? bstride : sstride) || h[0] < 0 || h[0] + na > st.ne) return false;
      const int *loc = ib + h[3], *rows = loc + na, *kid = rows + w;
      std::vector<double> F((size_t)f * RS, 0.0);
      for (int e = 0; e < na; ++e) F[loc[e]] = A[st.e0 + h[0] + e];
      for (int p = 0; p < w; ++p) F[p * RS + f] = xs[rows[p]];
      for (int c = 0; c < h[5]; ++c) {
        const int ne = kid[1];
        const int* to = kid + 2;
        if (to + ne > ib + st.ni) return false;
        std::vector<char> once(F.size(), 0);
        for (int e = 0; e < ne; ++e) {
          if (to[e] < 0 || to[e] >= f * RS || once[to[e]]++) return false;  // distinct within a child
          F[to[e]] += cr[kid[0] + e];
        }
        kid = to + ne;
      }
      lu(F, f, w);
      for (int i = 0; i < f; ++i)
        for (int j = 0; j < (i < w ? f : w); ++j) pan[h[6] + (i < w ? i * f + j : w * f + (i - w) * w + j)] = F[i * RS + j];
      for (int p = 0; p < w; ++p) x[rows[p]] = F[p * RS + f];
      for (int a = 0; a < m && h[4] >= 0; ++a)
        for (int b = 0; b <= m; ++b) {
          const int to = h[4] + (b < m ? a * m + b : m * m + a);
          if (to >= P.peak_cb || cw[to]) return false;
          cw[to] = 1;
          cb[to] = F[(w + a) * RS + (b < m ? w + b : f)];
        }
    }
  }
  if (at != nA || most != P.most || (P.most + P.peak_cb) * G * wsize > smem) return false;
  return pan == ref && x == xr;
}

int main() {
  const int shapes[][4] = {{2, 1, 0, 0}, {30, 41, 5, 0}, {118, 179, 53, 0}, {300, 411, 69, 0},
                           {1354, 1991, 259, 0}, {1354, 1991, 259, 1}, {2869, 4582, 509, 0}, {700, 699, 0, 2}};
  Rng rng(7);
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
    if (sh[0] == 2) {
      bus[0] = mpf_bus{MPF_BUS_SLACK, 0, 1.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      bus[1] = mpf_bus{MPF_BUS_PQ, 0, 1.0, 0.0, -0.1, -0.05, 0.0, 0.0};
      br[0] = mpf_branch{0, 1, 1, 0, 0.02, 0.1, 0.0, 0.0, 0.0};
    } else if (sh[3] == 2) {
      // a hub with hundreds of neighbours: one front row adds hundreds of carried entries
      for (int i = 0; i < sh[0]; ++i) bus[i] = mpf_bus{i == 1 ? MPF_BUS_SLACK : MPF_BUS_PQ, 0, 1.0, 0.0, -1e-4, 0.0, 0.0, 0.0};
      for (int i = 1; i < sh[0]; ++i) br[i - 1] = mpf_branch{i < 600 ? 0 : i - 500, i, 1, 0, 0.02, 0.1, 0.0, 0.0, 0.0};
    } else if (mpf_synth_grid(&p, bus.data(), br.data()) != 0) {
      return 1;
    }
    // the grid alone, and twice as two islands of one system
    for (int copies = 1; copies <= (sh[0] > 2000 ? 1 : 2); ++copies) {
      std::vector<mpf_bus> b2;
      std::vector<mpf_branch> r2;
      for (int k = 0; k < copies; ++k) {
        b2.insert(b2.end(), bus.begin(), bus.end());
        for (mpf_branch x : br) {
          x.from += k * sh[0];
          x.to += k * sh[0];
          r2.push_back(x);
        }
      }
      GridSymbolic g;
      const std::string msg = build_symbolic(b2.data(), (int)b2.size(), r2.data(), (int)r2.size(), g);
      if (!msg.empty()) {
        std::printf("%s\n", msg.c_str());
        return 1;
      }
      auto islands = [&](const LUSymbolic& s, const std::vector<int>& var, const std::vector<int>* var2) {
        std::vector<int> vi(s.n, 0), si;
        if (g.n_islands <= 1) return si;
        for (int i = 0; i < g.nb; ++i) {
          if (var[i] >= 0) vi[var[i]] = g.bus_island[i];
          if (var2 && (*var2)[i] >= 0) vi[(*var2)[i]] = g.bus_island[i];
        }
        for (int k = 0; k < s.nsn; ++k) si.push_back(vi[s.sn_rows[s.sn_rptr[k]]]);
        return si;
      };
      const LUSymbolic* sys[3] = {&g.jac, &g.bp[0].lu, &g.bpp[0].lu};
      const std::vector<int> isl[3] = {islands(g.jac, g.var_va, &g.var_vm), islands(g.bp[0].lu, g.bp[0].var, nullptr),
                                       islands(g.bpp[0].lu, g.bpp[0].var, nullptr)};
      for (int G : {8, 2, 1})
        for (size_t slot : {(size_t)3 * 1024, (size_t)16 * 1024})
          for (int ws : {4, 8})
            if (!check_factor(g.jac, g.ah_ptr, g.ah_loc, G, ws, slot, 170 * 1024, rng)) {
              std::printf("bad factor plan: %d buses, copies %d, G %d, value %d, slot %zu\n", sh[0], copies, G, ws, slot);
              return 1;
            }
      for (int k = 0; k < 3; ++k)
        for (bool compact : {false, true})
          for (int G : {8, 1})
            for (size_t slot : {(size_t)6 * 1024, (size_t)20 * 1024, (size_t)48 * 1024})
              if (!check(*sys[k], isl[k], compact, G, 4, slot, rng) || !check(*sys[k], isl[k], compact, G / 2 + G % 2, 8, slot, rng)) {
                std::printf("bad plan: %d buses, copies %d, system %d, compact %d, G %d, slot %zu\n", sh[0], copies, k,
                            (int)compact, G, slot);
                return 1;
              }
    }
  }
  std::printf("plans %ld worst %.2e\n", plans, worst);
  return 0;
}
