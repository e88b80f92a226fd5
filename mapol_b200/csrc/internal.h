// Host-side internals shared by the library's translation units.
#ifndef MPF_INTERNAL_H_
#define MPF_INTERNAL_H_

#include <cstdint>
#include <map>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "mpf.h"

#ifdef __CUDACC__
#define MPF_HD __host__ __device__
#else
#define MPF_HD
#endif

namespace mpf {

// A block of len entries stored in lane pairs ([16 pairs][len][2 lanes], contribution blocks
// between two large fronts): the values that hold lanes lane .. lane + G - 1 (lane a multiple of
// G) are the pair_values(len, G) from pair_first(len, lane) on.  One lane's values lie among
// its pair's.
MPF_HD inline long long pair_first(long long len, int lane) { return (lane >> 1) * len * 2; }
MPF_HD inline long long pair_values(long long len, int G) { return len * (G > 2 ? G : 2); }

uint64_t splitmix64(uint64_t& x);

// xoshiro256** seeded with splitmix64: identical streams on every machine.
struct Rng {
  uint64_t s[4];
  explicit Rng(uint64_t seed);
  uint64_t next();
  double uniform();            // [0, 1)
  uint64_t below(uint64_t n);  // [0, n)
  double normal();             // N(0, 1), Box-Muller
};

int find_bridges(const mpf_branch* br, int nbr, int nb, std::vector<uint8_t>& is_bridge);

// Branch pi-model admittances (complex as re/im pairs), makeYbus.h:40-107 (CPU)
// and :306-366 (GPU): Ys = stat/(R+jX), Bc = stat*jB, t = tap*e^{j*pi*shift/180}
// (tap 0 -> 1), Ytt = Ys + Bc/2, Yff = Ytt/|t|^2, Yft = -Ys/conj(t), Ytf = -Ys/t.
struct BranchY {
  double ff[2], ft[2], tf[2], tt[2];
};
BranchY branch_admittance(double r, double x, double b, double tap, double shift_deg, int stat);

// Multifrontal symbolic LU of a structurally symmetric n x n matrix factorised
// without pivoting (diagonal pivots) in a fixed elimination order.
//
// Supernode s owns w_s pivot variables and its front rows R_s =
// sn_rows[sn_rptr[s] .. sn_rptr[s+1]) (f_s of them, ascending; the first w_s are
// the pivots, every other row is a later variable).  Pivots of an amalgamated
// supernode need not be consecutive.  The front is the dense f x f matrix
// A(R_s, R_s) restricted to the arrowhead of the pivots plus the contribution
// blocks (CB) of the children; a partial LU of its first w pivots produces
//   U-panel  F(0:w, 0:f)          w*f entries, row-major (holds L of the diagonal
//                                 block below its diagonal, unit diagonal implied)
//   L-panel  F(w:f, 0:w)          (f-w)*w entries, row-major
//   CB       F(w:f, w:f)          (f-w)^2 entries, added into the parent's front
//   CB-RHS   b(w:f) - L y         (f-w) entries (forward solve carried upward)
// Panels of all supernodes are concatenated (pan_off) and hold exactly nnz(L+U)
// entries.
struct LUSymbolic {
  int n = 0;
  int64_t nnz = 0;                   // entries of L+U (= sum of panel sizes)
  std::vector<int> etree_parent;     // per variable, -1 for roots
  int nsn = 0;
  std::vector<int> sn_w;             // pivots
  std::vector<int> sn_f;             // front size
  std::vector<int> sn_rptr, sn_rows; // front rows
  std::vector<int> sn_parent;        // -1 for roots
  std::vector<int> sn_level;         // 0 for leaves, parent = 1 + max(children)
  int nlevels = 0;
  std::vector<int> lev_ptr, lev_sn;  // supernodes grouped by level, by front size within a level
  std::vector<int> child_ptr, child_list;
  std::vector<int64_t> pan_off;      // nsn+1, entries (order_panels); [nsn] = total
  // offsets of each supernode's contribution block ((f-w)^2 entries) and carried
  // right-hand side (f-w); siblings adjacent; [nsn] = the totals
  std::vector<int64_t> cb_off;       // nsn+1
  std::vector<int64_t> cbr_off;      // nsn+1
  std::vector<int> rel_ptr, relmap;  // per supernode: CB index -> index in the parent's front
  std::vector<int> sn_of;            // per variable
  int max_front = 0;
  int64_t flops = 0;                 // 2 * multiply-adds of one factorisation
  int64_t sum_cb = 0;                // sum of (f-w)^2
  int64_t nnz_l = 0;                 // strictly lower entries

  int local(int s, int var) const;               // index of var in R_s or -1
  int64_t entry_pos(int row, int col) const;     // panel position of LU entry or -1
};

// Relaxed supernode amalgamation: a child joins its parent's front when the merged
// front has at most max_pivots pivots and max_front rows and gains at most
// max(max_zeros, max_zero_frac * size) explicit zeros.  max_pivots <= 1 disables it.
// Measured on the 9241-bus workload (1000 N-1 cases, mixed precision, solves/s):
// none 20.5k, zero-free merges only 21.3k, (4, 0.1) 21.9k, (16, 0.3) 20.4k,
// (32, 0.4) 18.3k, (64, 0.5) 16.7k: the kernels' per-task cost is now low enough
// that explicit zeros cost more than the tasks they save.  Again with the launch DAG
// and the two-pivot kernels: these defaults 29.7k; zeros (8, 0.15) 28.9k, (2, 0.05)
// 29.0k; 48 pivots / 100 rows 29.7k; 16 pivots 29.6k.
struct Relax {
  int max_pivots = 32;
  int max_front = 83;
  long long max_zeros = 4;
  double max_zero_frac = 0.1;
};

// Builds the symbolic LU of the pattern given as symmetric adjacency (no diagonal)
// in the already-permuted variable numbering.
void lu_symbolic(int n, const std::vector<std::vector<int>>& adj, LUSymbolic& s, const Relax& relax = Relax());

// Panel storage: by island (sn_island, empty: one), level, solo or not, pivots and front size,
// the order in which a block walks the supernodes (build_sweep_plan), so that a level's panels
// are adjacent and similar fronts side by side.
void order_panels(LUSymbolic& s, const std::vector<int>& sn_island);

// Groups matrix entries (rows[e], cols[e]) by the supernode that owns min(row, col)
// (its arrowhead).  a_index[e] = position of entry e in the grouped ("A-array")
// order; supernode s owns A-array range [ah_ptr[s], ah_ptr[s+1]); ah_loc[k] is the
// flat position row * RS + col of A-array entry k inside the front, with the row
// stride RS = (f + 1) | 1 (the front carries a right-hand-side column f; the odd
// stride spreads consecutive rows over shared-memory banks).
void arrowhead_layout(const LUSymbolic& s, const std::vector<int>& rows,
                      const std::vector<int>& cols, std::vector<int>& a_index,
                      std::vector<int>& ah_ptr, std::vector<int>& ah_loc);

// Minimum-degree ordering of an undirected graph (adjacency lists without self
// loops).  Returns perm with perm[k] = vertex eliminated k-th.  Ties: lowest index.
std::vector<int> minimum_degree(int n, const std::vector<std::vector<int>>& adj);

// Minimum-deficiency (minimum fill-in) ordering: eliminates next the vertex whose
// elimination adds the fewest edges among its neighbours, each missing edge (a, b)
// counted weight[a] x weight[b] (weight null: 1).  Ties: smaller weighted degree,
// then lowest index.  Returns perm as minimum_degree, or an empty vector once the work
// of counting fill (which grows with it) passes max_work (0: no limit).
std::vector<int> minimum_fill(int n, const std::vector<std::vector<int>>& adj, const std::vector<int>* weight,
                              long long max_work = 0);

// Plan of one block's substitutions over the elimination tree (kernels_chunk.cuh): leaves to
// root, then root to leaves, as one sequence of steps.  A step is a run of supernodes of one
// level whose panels are adjacent in storage (pan_off is in this order), small enough for a
// slot of the block's ring buffer.  Supernodes of at most kSoloPivots pivots and kSoloFront
// rows are solo tasks (1 to 8 threads per lane, no barriers), the others are worked on beside
// them by nteams teams of `team` threads.
constexpr int kChunkThreads = 512;
constexpr int kSoloPivots = 4, kSoloFront = 16;
constexpr int kRingSlots = 3;
struct SweepStep {
  int e0, ne;          // panel entries [e0, e0 + ne)
  int i0, ni;          // index block: idx[i0 .. i0 + ni), both multiples of 4
  int up, lsplit;      // 1: leaves to root; log2 of the threads per lane of a solo task
  int nsolo, nbig;     // tasks of the index block: solo ones first
  int lteam, nteams;   // log2 of a team's threads
  int xstride;         // values per lane a team needs for its front
  int direct;          // 1: one team task too large for a slot: its panel and list are read
                       // where they are (ne = 0; the list follows the block in idx)
};
constexpr int kStepInts = sizeof(SweepStep) / 4;
inline bool solo_task(int w, int f) { return w <= kSoloPivots && f <= kSoloFront; }
// Index block of a step: the SweepStep itself, a header of four ints per task, then the
// tasks' index lists.  Header: panel entry relative to e0; w | f << 16; start of the task's
// list in the block; where the rows below the pivots are carried (-1: no parent).  List, root
// to leaves: the x indices of the front [f].  Leaves to root: the number of layers and a 0,
// the x indices of the pivots [w] (an even number of ints), and per layer f pairs: the
// carried entries that front row i adds, two per layer, children in order (-1: none).
struct SweepPlan {
  std::vector<SweepStep> step;
  std::vector<int> step_ptr;   // [islands + 1]: steps of each island (none where it has no supernode)
  std::vector<int> down_ptr;   // [islands]: of them, the first root-to-leaves step
  std::vector<int> idx;
  int peak_cb = 0;             // carried entries alive at once (most over the islands)
  size_t scratch = 0;          // values per lane of shared memory the teams need
  size_t slot = 0;             // bytes of the largest step
};
// Plan of one block's factorisation (one island), streamed like the substitutions: a step is
// a run of supernodes of one level whose arrowhead values are adjacent.  Its larger fronts go
// to nteams teams of 1 << lteam threads, the others to the remaining warps, one front per
// warp; bstride / sstride: shared-memory values per lane of a team's / a warp's front.
struct FactorStep {
  int e0, ne;          // arrowhead values [e0, e0 + ne)
  int i0, ni;          // index block: idx[i0 .. i0 + ni), both multiples of 4
  int nbig, nsmall;    // tasks of the index block: large fronts first
  int lteam, nteams;
  int bstride, sstride;
  int pad[2];
};
static_assert(sizeof(FactorStep) == sizeof(SweepStep), "both records start an index block");
// Index block: the FactorStep, eight ints per task (first value relative to e0, values; w |
// f << 16; start of the task's list in the block, where its contribution block goes (-1: no
// parent), children, panel entry, 0), then the lists: places of the arrowhead values in the
// front, the pivots' x indices, and per child its contribution block's place, its length m m +
// m and the place in the front of each of its values: m x m, then the m carried right-hand
// sides.
// Row stride of a front in shared memory (front_stride() of the kernels)
inline int plan_front_stride(int f) { return (f + 1) | 1; }
struct FactorPlan {
  std::vector<FactorStep> step;
  std::vector<int> idx;
  int peak_cb = 0;             // values per lane of the contribution blocks alive at once
  size_t most = 0;             // values per lane of the fronts worked on side by side
  size_t slot = 0;             // bytes of the largest step
  double cycles = 0.0;         // estimated clock cycles of a factorisation
};
// What every factorisation plan needs, whatever its lanes: a plan that does not fit() is refused
// without being built.  cycles: less than any plan's.
struct FactorNeeds {
  int peak_cb = 0;             // as FactorPlan
  size_t front = 0;            // values per lane of the largest front
  double cycles = 0.0;
  std::vector<std::pair<int64_t, int64_t>> tasks;  // a step of one supernode: arrowhead values, ints
  bool fits(int G, int wsize, size_t slot, size_t smem) const;
};
FactorNeeds factor_needs(const LUSymbolic& s, const std::vector<int>& ah_ptr);

// G lanes of wsize-byte values; slot: most bytes of a step; smem: bytes for contribution blocks
// and fronts.  False when they do not fit.
bool build_factor_plan(const LUSymbolic& s, const std::vector<int>& ah_ptr, const std::vector<int>& ah_loc, int G,
                       int wsize, size_t slot, size_t smem, FactorPlan& out);

// SweepPlan::peak_cb of the plans with compact carried entries (any lanes and slot)
int sweep_peak_cb(const LUSymbolic& s, const std::vector<int>& sn_island);

// sn_island: each supernode's island (empty: one island); n_islands: how many there are, also
// those without a supernode (0: as many as sn_island names).
// compact_cb: carried entries get slots that are reused once the parent has read them (else
// their storage in cbr).  G lanes of wsize-byte values; slot: most bytes of a step; scratch:
// bytes for the teams' fronts.  False when a front does not fit the scratch.
bool build_sweep_plan(const LUSymbolic& s, const std::vector<int>& sn_island, bool compact_cb, int G, int wsize,
                      size_t slot, size_t scratch, SweepPlan& out, int n_islands = 0);

// Plans kept by what they depend on.  A plan enters the cache when it is complete: a build
// that throws (an allocation or a copy that failed) leaves no trace and is tried again by the
// next call; one that returns false (the planner refuses) is remembered as null.
template <class Key, class Plan>
class PlanCache {
 public:
  template <class Build>  // bool build(Plan&)
  const Plan* get(const Key& key, Build&& build) {
    auto it = plans_.find(key);
    if (it == plans_.end()) {
      auto p = std::make_unique<Plan>();
      if (!build(*p)) p.reset();
      it = plans_.emplace(key, std::move(p)).first;
    }
    return it->second.get();
  }
  void clear() { plans_.clear(); }
  template <class F>  // f(const Plan&) for every plan kept
  void each(F&& f) const {
    for (const auto& p : plans_)
      if (p.second) f(*p.second);
  }

 private:
  std::map<Key, std::unique_ptr<Plan>> plans_;
};

// Everything that does not depend on the case batch.
struct GridSymbolic {
  int nb = 0, nbr = 0, npv = 0, npq = 0, slack = -1, n_slack = 0;
  int n_islands = 0;                 // connected islands with a slack (grids of a multi-grid handle)
  std::vector<int> bus_island;       // per bus: island, -1 for buses of slack-less islands without equations
  std::vector<int> br_island;        // per branch: island of its buses
  std::vector<int> pv, pq;           // bus-index order (Topology.h:100-126)
  std::vector<int> bus_type;
  // Ybus superset pattern (every branch, in or out of service), CSR, columns sorted
  std::vector<int> y_rowptr, y_col;
  std::vector<double> y_val;         // base values, 2 per entry (re, im)
  std::vector<int> y_diag;           // position of (i, i)
  std::vector<int> br_pos;           // 4 per branch: ff, ft, tf, tt positions in Ybus
  std::vector<double> br_y;          // 8 per branch: ff, ft, tf, tt (re, im), with status
  std::vector<int> br_from, br_to, br_status;
  std::vector<double> sbus;          // 2 per bus
  std::vector<double> v0;            // 2 per bus: start point (runpf.h:211-226)

  // Newton system: variables = Va of every PV/PQ bus, Vm of every PQ bus
  std::vector<int> bus_order;        // elimination order of PV/PQ buses
  int ordering = 0;                  // the method that produced it (MPF_ORDER_*)
  std::vector<int> var_va, var_vm;   // per bus: LU variable index or -1
  LUSymbolic jac;
  int nnz_jac = 0;
  std::vector<int> jpos;             // 4 per Ybus entry: J-array index of the
                                     // (Va,Va), (Va,Vm), (Vm,Va), (Vm,Vm) block entries or -1
  std::vector<int> ah_ptr, ah_loc;   // arrowhead of supernode s: J-array range
                                     // [ah_ptr[s], ah_ptr[s+1]) and flat front positions
  std::vector<int> mis_rows;         // PV/PQ buses (rows of the mismatch)

  // Fast-decoupled systems (B': Va of PV/PQ buses; B'': Vm of PQ buses), for
  // XB (alg 1) and BX (alg 2) variants (makeB.h:311-501)
  struct FDSystem {
    LUSymbolic lu;
    std::vector<int> var;            // per bus: variable index or -1
    std::vector<double> base;        // arrowhead values of the base case (A-array order)
    std::vector<int> ah_ptr, ah_loc; // arrowhead of each supernode (as for the Newton system)
    std::vector<int> br_pos;         // 4 per branch: A-array index (ff, ft, tf, tt) or -1
    std::vector<double> br_val;      // 4 per branch: B contributions (ff, ft, tf, tt)
    std::vector<int> diag_pos;       // per bus: A-array index of its diagonal or -1
  };
  FDSystem bp[2], bpp[2];            // [0] = XB, [1] = BX
  std::vector<int> bpp_order;
};

// Validates the grid and fills g.  Returns empty string on success, else a message.
// vm_free (nullable): PV buses that also get a Vm variable and a Q equation (buses
// whose reactive limits may switch them to PQ).
// ordering: MPF_ORDER_* of the Newton system's bus elimination order (AUTO picks the
// candidate with the least estimated factorisation time).
std::string build_symbolic(const mpf_bus* buses, int nb, const mpf_branch* br, int nbr,
                           GridSymbolic& g, const std::vector<char>* vm_free = nullptr, int ordering = 0);

}  // namespace mpf

#endif  // MPF_INTERNAL_H_
