// dem_internal.cuh -- shared definitions of the CUDA DEM library.
//
// Device layout (n = MAX_PIP):
//   pos4[b][i] = (x, y, z, radius)      double4, double-buffered (b = 0/1)
//   vel4[b][i] = (u, v, w, pmass)       double4, double-buffered
//   omg4[b][i] = (wx, wy, wz, omoi)     double4, one array (omg4[0] and
//                                       omg4[1] are the same): the spin is
//                                       updated in place, and a particle with
//                                       no torque under Euler is not touched
//   state[i]   int8 PARTICLE_STATE, phase[i] uint8 (0-based)
//   fc, tow    (n,3) column blocks, as FC/TOW of discretelement_mod.f:630
//   pairs      CSR half list: row_end[i] = pairs in rows 0..i,
//              nbrs[P] 0-based, pft[b] = PFT_NEIGHBOR as three planes of
//              pair_cap (one per component),
//              and the transpose in_start[n+1] / in_pair[] = (owner, cc)
//              sorted by owner so each particle can gather the forces of
//              the pairs it does not own in the serial reference's order.
// Packing a particle's position with its radius (and velocity with mass,
// spin with inverse inertia) makes each neighbour gather one 32-byte sector
// per quantity.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <deque>
#include <string>
#include <vector>

#include "../../include/dem_b200.h"
#include "quotient.cuh"

namespace demb {

// Neighbours per particle kept by the count pass of the pair build.
constexpr int NSLOT = 16;
constexpr double SMALL_NUMBER = 1.0e-15;       // param1_mod.f:26
constexpr double UNDEFINED_D  = 9.87654321e31; // param1_mod.f:20
constexpr int MAXP = DEM_MAX_PHASES;

// Error word bits (device -> host)
enum : unsigned {
  EF_ZERO_DIST   = 1u << 0,
  EF_WALL_SLOTS  = 1u << 1,
  EF_PAIR_CAP    = 1u << 2,
  EF_ROGUE_FATAL = 1u << 3,
  EF_CELL_CAP    = 1u << 4,
  EF_NONFINITE   = 1u << 5,
  EF_INFLOW_CAP  = 1u << 6,   // fewer NONEXISTENT slots than particles to seed
};

// Per-pair flag bits (pflag) between force passes.
enum : uint8_t {
  PF_CONTACT = 1,   // in contact at the last force pass (its record is valid)
  PF_HIST    = 2,   // its tangential history PFT is nonzero
};

// The candidate list of a single-system handle's pair build (neighbor.cu):
// pairs within the search radius plus a skin, kept while the displacement
// bound since its build stays within half the skin.
struct CandState {
  double disp;  // displacement bound since the list was built
  int have;     // the list is complete (built, within its capacity)
  int ok;       // this build filters the list (set at the start of each build)
  int build;    // this build makes a new list
  int total;    // entries of the last list build
  int uses;     // builds that filtered the current list
  int cool;     // builds left before the next list is made (after one expired unused)
};

// Contacts of a split-precision pair pass whose onset-of-slip test lies
// near its threshold (force_split.cu): 2 * pair index + 1 when the pair
// had a history.  The count starts at zero and the split gather, which follows
// every pass, clears it; past SLIP_FIX_CAP a contact keeps its FP32
// decision.
constexpr int SLIP_FIX_CAP = 4096;
struct SlipFix {
  unsigned count;
  unsigned pad;
  long long pair[SLIP_FIX_CAP];
};

// Contacts of a force pass.
struct ContactCount {
  unsigned long long pairs, walls;
};

struct DevErr {
  unsigned flags;
  int first_rogue;   // smallest rogue particle index of the last build (n if none)
  int zero_a, zero_b;  // particles of a zero-distance pair
  // two sets: a force pass on state buffer c counts into count[c], and its
  // integrating gather clears the other for the next pass
  ContactCount count[2];
  unsigned long long rogue_removed;
  unsigned long long outflow_removed;
  int cand_lists;     // candidate lists built (complete) so far
  int cand_filtered;  // pair builds that filtered a candidate list so far
};

// Parameters as kernels see them (passed by value).
struct DevParams {
  int n;
  int coll, intg, nph, no_k, cmax, remove_rogue, first_pass, prec;
  int per[3];
  int istart1, iend1, istart2, iend2;
  int jstart1, jend1, jstart2, jend2;
  int kstart1, kend1, kstart2, kend2;
  int c1, c2, c3, ncell2;
  double dt, grav[3];
  double kn, kt, kn_w, kt_w, mew, mew_w, mew_r, mew_rw;
  double factor_rlm, max_radius;
  double dg_start[3], dg_inv[3];
  double lo[3], hi[3], L[3], inv_L[3];  // inv_L = 1 / L
  double etan[MAXP * MAXP], etat[MAXP * MAXP], hkn[MAXP * MAXP], hkt[MAXP * MAXP];
  double etanw[MAXP], etatw[MAXP], hkwn[MAXP], hkwt[MAXP];
  // FP32 copies for the split-precision pair force: HERT_KN, HERT_KT,
  // DES_ETAN*sqrt(HERT_KN), DES_ETAT*sqrt(HERT_KT) (Hertz), DES_ETAN,
  // DES_ETAT, KN, KT (linear spring-dashpot), MEW
  float hkn32[MAXP * MAXP], hkt32[MAXP * MAXP], etan_sq32[MAXP * MAXP], etat_sq32[MAXP * MAXP];
  float etan32[MAXP * MAXP], etat32[MAXP * MAXP];
  float kn32, kt32, mew32;
  // search grid of the pair build: fn[a] interior cells of width 1/f_inv[a]
  // over the DES-grid interior, plus one ghost layer on each side
  int fn[3], fc1, fc2, nfcell;
  double f_inv[3];
  // place of the system in a batch handle (0 for an ordinary handle):
  // particles [p_begin, p_end), DES cells from cell_off, search cells from
  // fcell_off in the handle-wide cell arrays; n stays the handle-wide count
  int p_begin, p_end, cell_off, fcell_off;
};

// Batch view of a kernel: the parameter block of every system and the
// system of every particle.  Kernels instantiated with B = false use the
// by-value block of the handle's single system and never touch the view.
struct BatchView {
  const DevParams* tab;       // [system]
  const uint16_t* sys_of;     // [particle]
  const uint8_t* due;         // [system] 1 = rebuild its pair list now, 2 = first build (no history)
  int* first_rogue;           // [system] smallest rogue particle of the last build
};

template <bool B>
__device__ __forceinline__ const DevParams& sysp(const DevParams& p, const BatchView& bv, int particle) {
  if constexpr (B) return bv.tab[bv.sys_of[particle]];
  else return p;
}

// What the two particles of a contact pair need to add the pair's terms to
// FC/TOW in the reference's order: FC_TMP, CROSS(NORMAL, FT) with the two
// lever arms (the torques are DIST_CL*TOW_force and DIST_CI*TOW_force), and
// KN_DES and OVERLAP_N for the rolling-friction torque.
struct PairRec {
  double fc[3], tf[3], dcl2, dci2, kn, ov;
};
// The record in memory, 80 bytes a pair in two arrays: (fc, tf, dcl2, dci2)
// as two aligned 32-byte words, read and written with one instruction each,
// and (kn, ov), which only a system with rolling friction writes and reads.
struct RecStore {
  double4* main;   // [2 * pair], [2 * pair + 1]
  double2* roll;   // [pair]
};

struct FacetBinEntry {  // one entry of facets_at_dg(cell)
  double mn, mx;        // facet extent along dir
  int id;               // 0-based facet
  int dir;              // 0-based axis of smallest extent
};

// ---------------------------------------------------------------------------
// Host-side handle
struct DevBuf {
  void* p = nullptr;
  size_t bytes = 0;
};

// Host bookkeeping of one system of a batch handle.
struct SysSlot {
  bool live = false;          // the slot holds a system
  bool clean = true;          // no rows of an earlier occupant left under this id
  bool started = false;       // its pair list exists and it steps
  bool have_state = false;
  dem_params prm;
  DevParams dp;               // p_begin/p_end/cell_off/fcell_off filled in
  int cap = 0;                // particles reserved (p_end - p_begin)
  int nn = 1;                 // NN of its next DES_TIME_STEP
  bool first_pass = true;
  long long steps_done = 0;
  double s_time = 0.0;
  int fac_off = 0, nf = 0;     // its wall facets in the handle-wide facet arrays
  int bin_off = 0, nbin = 0;   // its facet-bin entries
};

// First-fit allocator over an index range (particles or cells of a batch).
struct RangeAlloc {
  std::vector<std::pair<int, int>> free_;  // (begin, length), sorted by begin
  void reset(int total) { free_.assign(1, {0, total}); }
  int take(int len, int align);             // begin, or -1 when nothing fits
  void give(int begin, int len);
};

}  // namespace demb

struct dem_handle {
  dem_params prm;
  demb::DevParams dp;
  int n = 0;

  // batch of independent systems (dem_batch_create); empty otherwise
  std::vector<demb::SysSlot> sys;
  demb::RangeAlloc part_alloc, cell_alloc, fcell_alloc, fac_alloc, bin_alloc;
  int max_facets = 0, max_bins = 0;
  demb::DevParams* d_sys = nullptr;   // device copy of sys[*].dp
  uint16_t* sys_of = nullptr;         // [particle] system
  uint8_t* d_due = nullptr;           // 3 masks of max_systems: eager events, and the idle
                                      // and rebuild steps of a captured period
  const uint8_t* due_cur = nullptr;   // the mask the next kernels read
  int* d_first_rogue = nullptr;       // [system]
  int ncell_total = 0, nfcell_total = 0;
  int n_act = 0, nfc_act = 0;         // extent of the live systems' particle and search-cell ranges
  int n_built = 0;                    // the particle extent of the current pair list's build
  bool batch() const { return !sys.empty(); }
  // The particles and search cells the step kernels cover: for a batch the
  // extent of its live systems (the ranges past it belong to no system: no
  // particle exists there and no cell is read), else all of them.
  int nl() const { return batch() ? n_act : n; }
  int nfl() const { return batch() ? nfc_act : dp.nfcell; }
  demb::BatchView bview() const { return demb::BatchView{d_sys, sys_of, due_cur, d_first_rogue}; }
  int dev = 0;
  cudaStream_t stream = 0;
  std::string err;
  long long launches = 0;
  bool have_state = false, have_pairs = false;
  int cur = 0;  // current state buffer
  int pcur = 0; // current pft buffer
  bool first_pass = true;
  long long steps_done = 0;
  double s_time = 0.0;

  // particle state
  double4* pos4[2] = {nullptr, nullptr};
  double4* vel4[2] = {nullptr, nullptr};
  double4* omg4[2] = {nullptr, nullptr};
  int8_t* state = nullptr;
  uint8_t* phase = nullptr;
  double* fc = nullptr;   // (n,3)
  double* tow = nullptr;
  double* acc_old = nullptr;
  double* rot_acc_old = nullptr;

  // DES grid
  int* dg_pijk = nullptr;     // 1-based cell, 0 = none
  int* cell_cnt = nullptr;    // ncell2
  int* cell_fill = nullptr;   // ncell2
  int* fcell_key = nullptr;   // n: search-grid cell of each particle (0-based; -1: not binned)
  int* fcell_slot = nullptr;  // n: its place in the cell
  int* fcell_cnt = nullptr;   // nfcell+1, zero between the passes that count into it
  int* fcell_start = nullptr; // nfcell+1
  double4* spos = nullptr;    // n: positions in search-cell order (pair build)
  float4* sposf = nullptr;    // n: the same rounded to FP32 (conservative distance pre-check)
  int4* sinfo = nullptr;      // n: (particle, packed DES cell (i,j,k), state, search cell) in that order
  uint32_t* nslot = nullptr;  // n * NSLOT: rows kept by the count pass of the pair build, by particle
  int* long_rows = nullptr;   // n + 1: sorted-copy places of the rows longer than NSLOT, count at [n]
  // candidate list (single-system handles): particle i's candidates are entries
  // [cand_start[i], cand_start[i + 1]) of cand_nb (particle indices); cand_cnt
  // and cand_fill are build scratch, qof[i] the particle's place in the sorted
  // copy (-1 when not in it)
  int* cand_cnt = nullptr;
  int* cand_start = nullptr;
  int* cand_fill = nullptr;
  int* qof = nullptr;
  int* cand_nb = nullptr;
  long long cand_cap = 0;
  demb::CandState* cand = nullptr;

  demb::SlipFix* slipfix = nullptr;  // split pair pass: contacts near the onset of slip

  // pairs
  long long pair_cap = 0;
  long long arr_bytes = 0;    // device bytes of the arrays sized by the counts (handle_arrays and the batch tables)
  long long n_pairs = 0;      // host copy of the pair count (valid when !np_stale)
  bool np_stale = false;      // the last build ran without reading the count back
  int* d_np = nullptr;        // device pair count (persistent pair kernels read it); [1]: the count of the
                              // list being built, which becomes [0] when its rows are filled
  int n_sm = 148;             // multiprocessors of the device
  // launch shapes of the hot kernels (dem_autotune picks them)
  struct Tune {
    int pair_threads = 256, pair_bpsm = 8;  // pair kernel: threads per block, resident blocks per SM
    int gather_threads = 256;               // gather kernel: threads per block
    int neigh_threads = 128;                // pair-build scan: threads per block
  } tune;
  bool tuned = false;         // the shapes were measured or set; otherwise pair_shape chooses
  // Launch shape of the pair kernel.  The FP64 one keeps 512 threads on a
  // multiprocessor (128 registers).  With eight windows of pairs or more for each resident
  // warp: blocks of two warps, as many as fit the device once, since a second
  // wave of these persistent blocks only waits for the first and small blocks
  // end more evenly (the bed of 1,000,000 spheres, 34,000 windows: 354 us per
  // step against 365 with 1184 blocks of eight warps).  With fewer: blocks of
  // eight warps, whose neighbouring windows share an L1 (coupled bed of 500,000,
  // five windows a warp: 281 us per step against 288 in blocks of two; gas of
  // 200,003, less than one: 60 us against 66).  The split kernel, with twice
  // the warps, gains nothing from small blocks (a batch of columns loses 1 %).
  // The loops over the list take any grid.
  struct Shape {
    int threads, blocks;
  };
  Shape pair_shape(bool split) const {
    constexpr int resident = 512;
    if (!split && !tuned && n_pairs / 128 >= 8ll * n_sm * resident / 32) return {64, n_sm * (resident / 64)};
    return {tune.pair_threads, n_sm * tune.pair_bpsm};
  }
  // Threads of a block of the gathers: a block leaves when its slowest warp
  // does, so small ones refill sooner (1 % of a step of a bed of 150,001 and of
  // one of 1,000,000 against blocks of 256).  The split gather stages its warps'
  // records in shared memory for 128 threads at most.
  static constexpr int SPLIT_GATHER_MAX = 128;
  int gather_block(bool split) const {
    const int t = tuned ? tune.gather_threads : 128;
    return split && t > SPLIT_GATHER_MAX ? SPLIT_GATHER_MAX : t;
  }
  bool capturing = false;     // inside a CUDA graph capture: no host syncs
  cudaStream_t own_stream = nullptr;
  // the wall kernels of a force pass run on side_stream beside the pair
  // kernel (they write disjoint arrays); ev_fork / ev_join order them
  cudaStream_t side_stream = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  bool joined = false;        // the next launch follows a wait for the other stream, a copy or a memset
  bool chain = false;         // eager launches that follow one another with nothing in between
  cudaGraphExec_t graphs[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  long long graph_launches = 0;
  long long graph_kernels[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // kernels per graph replay
  bool no_graphs = false;
  int* row_cnt = nullptr;     // n
  int* row_end[2] = {nullptr, nullptr};   // n (current / previous build)
  int* nbrs[2] = {nullptr, nullptr};      // cap
  // 3*cap, a plane of cap values per component (neighbouring pairs' values
  // lie side by side); pft[pcur] is current, the other takes the carry-over
  // of a rebuild
  double* pft[2] = {nullptr, nullptr};
  int* in_cnt = nullptr;      // n, zero between the builds that count into it
  int* in_start = nullptr;    // n+1
  int* in_mid = nullptr;      // n: the first slot of each incoming list whose owner has a higher index (the
                              // list's end when none)
  int2* in_pair = nullptr;    // cap
  int* in_pos = nullptr;      // cap: slot of each pair in its neighbour's incoming list (inverse of in_pair; during
                              // a build its place in the list as found)
  uint8_t* in_flag = nullptr; // cap: PF_CONTACT of the pair at each incoming slot
  int* pair_owner = nullptr;  // cap
  // cap: PF_* bits of each pair, one array per history buffer: pflagb[pcur]
  // goes with pft[pcur] (the other is stencil-rank scratch during a build
  // and the output of a split-precision force pass)
  uint8_t* pflagb[2] = {nullptr, nullptr};
  uint8_t* pflag() const { return pflagb[pcur]; }
  uint8_t* touched = nullptr; // n: 1 = in some pair contact at the current force pass
  uint8_t* wall_hit = nullptr; // n: 1 = in some wall contact (its terms are in wf)
  float* pgap = nullptr;      // cap: gap |d| - (r_i + r_j) of each pair at the last build, rounded down
  double* skin = nullptr;     // [0]: bound on any particle's displacement since the last build
  // per-step displacement bounds, as float bits, in two sets of 32 slots:
  // set `cur` holds what has not been added to skin yet (the last integrating
  // gather's), and the next moves are noted in the other
  unsigned* vslot = nullptr;
  unsigned* vslot_pending() const { return vslot + 32 * cur; }
  unsigned* vslot_note() const { return vslot + 32 * (1 - cur); }
  int count_set = 0;          // set of derr->count that the last force pass counted into
  bool count_dirty = false;   // a pass that did not integrate has left its counts in place
  void* prec = nullptr;       // 80*cap bytes: contact terms of the last force pass
  demb::RecStore recs() const {
    return {static_cast<double4*>(prec), reinterpret_cast<double2*>(static_cast<char*>(prec) + 64 * pair_cap)};
  }
  int rb = 0;                 // which row_end/nbrs buffer is current

  // walls
  int nf = 0;
  double* vertex = nullptr;   // [f][v][c]
  double* norm_face = nullptr;// [f][c]
  int8_t* ignore_edge = nullptr; // [f][4]
  int* fbin_start = nullptr;  // ncell2+1
  demb::FacetBinEntry* fbin = nullptr;
  int n_fbin = 0;
  int* wall_fid = nullptr;    // [i][cmax]
  double* wall_pft = nullptr; // [i][cmax][3]
  uint8_t* wall_live = nullptr; // [i] 1 when some wall slot may be in use
  uint8_t* wall_cand = nullptr; // [i] 1 when the particle's DES cell holds facets
  float* wgap = nullptr;        // [i] clearance from the facets of its DES cell at the last build
  // outflow boundaries (single handles): host copy, device copy, the
  // FIRST_PASS of UPDATE_EXIT_DES_VEL
  std::vector<dem_outflow_bc> obc;
  dem_outflow_bc* d_obc = nullptr;
  bool exit_first_pass = true;
  // mass-inflow boundaries (single handles): host copies with their layout
  // arrays, the device copy (membership and entering test), the queue and
  // generator of the uniform numbers, the particles seeded since the last
  // DESGRID_PIC (not yet in its cell lists) and the seed records
  struct Inflow {
    dem_inflow_bc bc;
    std::vector<double> p, q;
    std::vector<int32_t> layout;
    std::vector<int32_t> w, hh;  // DEM_MI%W, %H for restart records (zeros when not given)
  };
  std::vector<Inflow> ibc;
  dem_inflow_bc* d_ibc = nullptr;
  std::deque<double> irand;
  uint64_t irng = 0;
  uint8_t* pic_fresh = nullptr;
  void* d_seed = nullptr;
  int seed_cap = 0;
  long long inflow_added = 0;
  double* wf = nullptr;       // [i][6] wall force and torque of the last force pass (valid with wall_hit)

  // scan scratch
  int* scan_tmp = nullptr;
  size_t scan_tmp_elems = 0;

  // error word
  demb::DevErr* derr = nullptr;
  demb::DevErr* herr = nullptr;   // pinned mirror

  // reductions for stats
  double* red = nullptr;      // scratch doubles
  int red_elems = 0;

  // coupling (see coupling.cu)
  struct Gas* gas = nullptr;

  int fail_alloc = 0;  // > 0: the allocation that fails (dem_test_fail_alloc)

  // host<->device staging (kept between calls)
  void* stage = nullptr;
  size_t stage_bytes = 0;

  // kernel-time accounting (dem_set_profiling)
  int prof = 0;                // 0 off, 1 kernel classes, 2 also the parts of the force step
  struct ProfEv { int cls; cudaEvent_t a, b; };
  std::vector<ProfEv> prof_pending;
  std::vector<cudaEvent_t> ev_pool;
  double prof_ms[DEM_PROF_N] = {0};
  long long prof_n[DEM_PROF_N] = {0};
};

namespace demb {

// set by every API entry point on failure
int set_err(dem_handle* h, int code, const std::string& msg);
int check_cuda(dem_handle* h, cudaError_t e, const char* what);
// capi.cu: cudaMalloc; a failure leaves a null pointer and no pending error
cudaError_t alloc_bytes(dem_handle* h, void** p, size_t bytes);
template <class T>
cudaError_t dev_alloc(dem_handle* h, T** p, size_t bytes) {
  return alloc_bytes(h, reinterpret_cast<void**>(p), bytes);
}

// scan.cu: exclusive scan of n ints into out (out may alias in); total
// written to *d_total (device pointer) when non-null; `clear` zeroes the
// input behind it (not with out == in); with `go` (device pointer) nothing is
// done unless *go is set.
int exclusive_scan(dem_handle* h, int* in, int* out, int n, int* d_total, bool clear = false,
                   const int* go = nullptr);
// The scratch of a scan of n ints, so that the scan itself cannot fail for
// memory.  Counters that a clearing scan leaves at zero (fcell_cnt, in_cnt,
// pic_cnt) are only counted into behind it: a call that returned between the
// count and its scan would leave them for the next one to add to.
int reserve_scan(dem_handle* h, int n);

// desgrid.cu / neighbor.cu / force.cu / walls.cu host drivers
int run_desgrid_pic(dem_handle* h, bool sort_cells);
int run_neighbour(dem_handle* h, bool carry_history);
int run_force(dem_handle* h, bool fused);
int run_force_open(dem_handle* h);              // forces into FC/TOW, ended by a kernel of the caller's (end_step, the other state buffer)
int run_cfnewvalues(dem_handle* h);
int run_bin_facets(dem_handle* h, const double* vertex_fortran, const double* norm_fortran, int nf);
int run_split_force_error(dem_handle* h, double* rel_err);
void launch_pairs_split(dem_handle* h);         // force_split.cu
void launch_gather_split(dem_handle* h, int mode);
int ensure_pair_capacity(dem_handle* h, long long need);
int build_transpose(dem_handle* h, int nb, bool counted);    // neighbor.cu
void launch_neigh_count(dem_handle* h, const int* skip = nullptr);        // neighbor.cu: count pass of the pair build
void reset_neigh_count(dem_handle* h);         // neighbor.cu: what it counts into, to zero
void set_hist_flags(dem_handle* h);            // neighbor.cu: PF_HIST from the current history
// neighbor.cu: the history of pairs [first, first + count) between its planes
// and PFT_NEIGHBOR's (3,P) order on the host
int download_history(dem_handle* h, long long first, long long count, double* pf);
int upload_history(dem_handle* h, long long count, const double* pf);
void launch_skin(dem_handle* h);               // force.cu: adds the noted displacements to the bound
void clear_counts(dem_handle* h);              // force.cu: both sets of contact counts to zero
void skin_unknown(dem_handle* h);              // force.cu: positions changed from outside: no pair skipped
void launch_wall_gaps(dem_handle* h);          // force.cu: wall clearances at a build (with the pair gaps)
int run_cfnewvalues_outflow(dem_handle* h, bool* force_nsearch);  // outflow.cu: exit velocities, CFNEWVALUES, MASS_OUTFLOW_DEM
int run_mass_inflow(dem_handle* h);  // inflow.cu: MASS_INFLOW_DEM (entering test, seeding)
void launch_wall_cand(dem_handle* h);          // desgrid.cu: facet-cell flag of every particle
void launch_pairs_only(dem_handle* h, bool walls);  // force.cu: pair kernel of the handle's precision; walls: with
                                               // the wall work, where they are one launch (walls_with_pairs)
bool walls_with_pairs(const dem_handle* h, bool split);  // force.cu
void launch_gather_only(dem_handle* h);        // force.cu: gather kernel, forces into FC/TOW
// capi.cu: parameter block of a system with handle-wide particle count n
void fill_devparams(const dem_params& q, int n, DevParams& p);
bool des_grid_ok(const dem_params& q);
int alloc_handle(dem_handle* h, int nc, int nfc, long long pairs);
// Device bytes of the pair-list arrays for cap pairs (ensure_pair_capacity).
long long pair_array_bytes(long long cap);

// The arrays of a handle for n particles, nc DES cells and nfc search cells
// (COLLISION_ARRAY_MAX from h->dp), each given to A(&pointer, bytes): the
// allocation list of alloc_handle, and what dem_batch_footprint counts.
template <class F>
void handle_arrays(dem_handle* h, size_t n, size_t nc, size_t nfc, F&& A) {
  const size_t cmax = (size_t)h->dp.cmax;
  for (int b = 0; b < 2; ++b) {
    A((void**)&h->pos4[b], sizeof(double4) * n);
    A((void**)&h->vel4[b], sizeof(double4) * n);
    A((void**)&h->row_end[b], sizeof(int) * n);
  }
  // the spin is one array under both buffer names: the kernels that write it
  // in a step (the integrating gathers, k_coupled_step, k_integrate and its
  // outflow form, the deletions) each write the thread's own particle, behind
  // every kernel that reads other particles' spins
  A((void**)&h->omg4[0], sizeof(double4) * n);
  h->omg4[1] = h->omg4[0];
  A((void**)&h->state, n);
  A((void**)&h->phase, n);
  A((void**)&h->fc, sizeof(double) * 3 * n);
  A((void**)&h->tow, sizeof(double) * 3 * n);
  A((void**)&h->acc_old, sizeof(double) * 3 * n);
  A((void**)&h->rot_acc_old, sizeof(double) * 3 * n);
  A((void**)&h->dg_pijk, sizeof(int) * n);
  A((void**)&h->cell_cnt, sizeof(int) * (nc + 1));
  A((void**)&h->cell_fill, sizeof(int) * (nc + 1));
  A((void**)&h->fcell_key, sizeof(int) * n);
  A((void**)&h->fcell_cnt, sizeof(int) * (nfc + 1));
  A((void**)&h->fcell_start, sizeof(int) * (nfc + 1));
  A((void**)&h->fcell_slot, sizeof(int) * n);
  A((void**)&h->spos, sizeof(double4) * n);
  A((void**)&h->sposf, sizeof(float4) * n);
  A((void**)&h->sinfo, sizeof(int4) * n);
  A((void**)&h->nslot, sizeof(uint32_t) * NSLOT * n);
  A((void**)&h->long_rows, sizeof(int) * (n + 1));
  A((void**)&h->row_cnt, sizeof(int) * n);
  A((void**)&h->in_cnt, sizeof(int) * n);
  A((void**)&h->in_start, sizeof(int) * (n + 1));
  A((void**)&h->in_mid, sizeof(int) * n);
  A((void**)&h->fbin_start, sizeof(int) * (nc + 1));
  A((void**)&h->wall_fid, sizeof(int) * cmax * n);
  A((void**)&h->wall_pft, sizeof(double) * 3 * cmax * n);
  A((void**)&h->wall_live, n);
  A((void**)&h->wf, sizeof(double) * 6 * n);
  A((void**)&h->touched, n);
  A((void**)&h->wall_hit, n);
  A((void**)&h->wall_cand, n);
  A((void**)&h->wgap, sizeof(float) * n);
  A((void**)&h->skin, sizeof(double));
  A((void**)&h->vslot, sizeof(unsigned) * 64);
  A((void**)&h->derr, sizeof(DevErr));
  A((void**)&h->d_np, 2 * sizeof(int));
  A((void**)&h->slipfix, sizeof(SlipFix));
  if (!h->batch()) {
    A((void**)&h->cand_cnt, sizeof(int) * n);
    A((void**)&h->cand_start, sizeof(int) * (n + 1));
    A((void**)&h->cand_fill, sizeof(int) * n);
    A((void**)&h->qof, sizeof(int) * n);
    A((void**)&h->cand, sizeof(CandState));
  }
}
int upload_range(dem_handle* h, int off, int cnt, int nph, const double* pos, const double* vel,
                 const double* omega, const double* radius, const double* pmass, const double* omoi,
                 const int8_t* state, const int32_t* phase, bool note_moves = false);
int download_range(dem_handle* h, int off, int cnt, double* pos, double* vel, double* omega, int8_t* state);
int stats_range(dem_handle* h, int off, int cnt, dem_stats* s);
// walls.cu: facets of batch system `sys` binned to its DES cells
int run_bin_facets_sys(dem_handle* h, int sys, const double* vertex_fortran, const double* norm_fortran, int nf);
int fetch_errors(dem_handle* h);
void* stage_buffer(dem_handle* h, size_t bytes);
void free_gas(dem_handle* h);                   // coupling.cu
long long host_pairs(dem_handle* h);            // pair count on the host (syncs when stale)
void invalidate_graphs(dem_handle* h);

// Grid of the persistent kernels over the pair list: a fixed number of
// resident blocks.
inline unsigned pair_grid(const dem_handle* h, int threads) {
  return (unsigned)(h->n_sm * (2048 / threads));
}

// Brackets the kernels issued in its scope with CUDA events when the
// handle's profiling is on.
struct ProfScope {
  dem_handle* h;
  int idx = -1;
  ProfScope(dem_handle* hh, int cls);
  ~ProfScope();
};

// ---------------------------------------------------------------------------
// 32-byte loads and stores (one instruction per lane where double4 takes
// two; the address must be 32-byte aligned).  A lane that gathers a particle's
// state or a contact record touches one sector per word, and the kernels
// that do so are bound by the number of such accesses the L1 takes in.  The
// loads are for arrays that the kernel does not write.
__device__ __forceinline__ double4 ld32(const double4* p) {
  double4 v;
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// 16 bytes from global to shared memory, asynchronously; copy_wait() returns
// when the thread's copies are there.
__device__ __forceinline__ void copy16(void* shared, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(shared)),
               "l"(global)
               : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void st32(double4* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// Contact bits (PF_CONTACT, bit 0 of each flag byte) of flags[base,
// base + cnt), cnt <= 32, as a mask: the bytes are read as aligned 32-bit
// words (the flag arrays carry 16 bytes of padding past their capacity).
__device__ __forceinline__ unsigned contact_mask(const uint8_t* __restrict__ flags, int base, int cnt) {
  static_assert(PF_CONTACT == 1, "contact bit is bit 0");
  unsigned mask = 0u;
  const int w0 = base & ~3;
  for (int w = w0; w < base + cnt; w += 4) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(flags + w) & 0x01010101u;
    const unsigned b4 = (v | (v >> 7) | (v >> 14) | (v >> 21)) & 0xFu;  // byte k -> bit k
    const int sh = w - base;
    mask |= sh >= 0 ? (b4 << sh) : (b4 >> -sh);
  }
  return cnt >= 32 ? mask : (mask & ((1u << cnt) - 1u));
}

// The pairs of a warp's window [c0, c0 + WIN_PAIRS) that a pair kernel has to
// look at, as a queue in shared memory: pair offset in the window, PF_HIST
// and PF_CONTACT of the last pass above it, and the two particles.  A pair
// whose gap at the build exceeds `reach` (twice the displacement bound since, rounded up) with a
// zero history is apart without a look at its particles: its flags are
// cleared and it is left out.  A lane screens four consecutive pairs from one
// load of flags and one of gaps; the queue then gives every lane a pair, so
// the contact arithmetic and its gathers run on full warps (about 0.4 of a
// dense bed's pairs are in contact).  The particles of all 128 pairs are loaded
// with the flags, in whole lines: looked up for the queued pairs alone they
// were one more round of loads in the chain (bed of 1,000,000 spheres 334 us
// per step, 321 us so; split 249 and 244 us; a batch of 16 columns 111 and 108
// us).  Returns the queue's length, the same in every lane.
// Also tried: the queue carried over from window to window, so that only full
// warps take from it (1 % faster in FP64, 5 % slower in split), and a block's
// windows side by side over several turns (4 to 10 % slower): what counts is
// that all blocks work at one place of the list, whose particles the L2 holds.
constexpr int WIN_PAIRS = 128;
constexpr int WQ_CONTACT = 1 << 7, WQ_HIST = 1 << 8;
struct WinQueue {
  int2 who[WIN_PAIRS];
  uint16_t e[WIN_PAIRS];
};
__device__ __forceinline__ int screen_window(long long c0w, long long np, uint8_t* __restrict__ pflag,
                                             uint8_t* __restrict__ in_flag, const int* __restrict__ in_pos,
                                             const float* __restrict__ pgap, const int* __restrict__ owner,
                                             const int* __restrict__ nbrs, float reach, WinQueue* queue) {
  static_assert(PF_CONTACT << 7 == WQ_CONTACT && PF_HIST << 7 == WQ_HIST, "flags move up by seven bits");
  const int lane = threadIdx.x & 31;
  const long long c0 = c0w + 4 * lane;
  uint32_t fw = 0;  // the four flags, one per byte
  float g[4] = {0.f, 0.f, 0.f, 0.f};
  int live = 4, ow[4] = {0, 0, 0, 0}, nb[4] = {0, 0, 0, 0};
  if (c0 + 3 < np) {
    fw = *reinterpret_cast<const uint32_t*>(pflag + c0);
    const float4 gq = *reinterpret_cast<const float4*>(pgap + c0);
    g[0] = gq.x; g[1] = gq.y; g[2] = gq.z; g[3] = gq.w;
    const int4 oq = *reinterpret_cast<const int4*>(owner + c0), nq = *reinterpret_cast<const int4*>(nbrs + c0);
    ow[0] = oq.x; ow[1] = oq.y; ow[2] = oq.z; ow[3] = oq.w;
    nb[0] = nq.x; nb[1] = nq.y; nb[2] = nq.z; nb[3] = nq.w;
  } else {
    live = c0 < np ? (int)(np - c0) : 0;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j < live) { fw |= (uint32_t)pflag[c0 + j] << (8 * j); g[j] = pgap[c0 + j]; ow[j] = owner[c0 + j]; nb[j] = nbrs[c0 + j]; }
  }
  unsigned need = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (j >= live) break;
    const uint8_t f = (uint8_t)(fw >> (8 * j));
    if ((f & PF_HIST) || !(g[j] > reach)) {
      need |= 1u << j;
    } else if (f) {
      pflag[c0 + j] = 0;
      if (f & PF_CONTACT) in_flag[in_pos[c0 + j]] = 0;
    }
  }
  const int mine = __popc(need);
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  int at = incl - mine;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if ((need >> j) & 1u) {
      queue->who[at] = make_int2(ow[j], nb[j]);
      queue->e[at++] = (uint16_t)((4 * lane + j) | (((fw >> (8 * j)) & (PF_CONTACT | PF_HIST)) << 7));
    }
  __syncwarp();
  return __shfl_sync(0xffffffffu, incl, 31);
}

// ---------------------------------------------------------------------------
// Device helpers.  All FP64 arithmetic in the parity kernels is compiled
// without FMA contraction so each expression rounds like the Fortran.
__device__ __forceinline__ double dot3(const double a[3], const double b[3]) {
  return a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
}
__device__ __forceinline__ void cross3(const double x[3], const double y[3], double o[3]) {
  o[0] = x[1] * y[2] - x[2] * y[1];
  o[1] = x[2] * y[0] - x[0] * y[2];
  o[2] = x[0] * y[1] - x[1] * y[0];
}

__device__ __forceinline__ int dg_funijk(const DevParams& p, int i, int j, int k) {
  return j + i * p.c1 + k * p.c2 + p.c3;
}
__device__ __forceinline__ int dg_jof(const DevParams& p, int ijk) {
  return ((ijk - 1) % p.c2) % p.c1 + p.jstart2;
}
__device__ __forceinline__ int dg_iof(const DevParams& p, int ijk) {
  return ((ijk - dg_jof(p, ijk) + p.jstart2 - 1) % p.c2) / p.c1 + p.istart2;
}
__device__ __forceinline__ int dg_kof(const DevParams& p, int ijk) {
  return (ijk - p.c3 - dg_iof(p, ijk) * p.c1 - dg_jof(p, ijk)) / p.c2;
}
// A DES cell as (i, j, k) in one int: 10 bits for i and k, 12 for j (the
// handle set-up checks the grid fits).
constexpr int DG_MAX_IK = 1023, DG_MAX_J = 4095;
__device__ __forceinline__ int pack_ijk(int i, int j, int k) { return i | (j << 10) | (k << 22); }
__device__ __forceinline__ void unpack_ijk(int c, int& i, int& j, int& k) {
  i = c & 1023;
  j = (c >> 10) & 4095;
  k = (c >> 22) & 1023;
}

// Cells of the DES grid, and of the search grid of the pair build, at most
// (with their ghost layers): every cell index and count fits an int.
constexpr long long MAX_GRID_CELLS = 1LL << 28;
// Cells of the search grid of one system when it is finer than its DES grid.
constexpr long long SEARCH_CELLS_CAP = 1LL << 22;

constexpr int MAX_PARTICLES = (1 << 27) - 1;  // particle index in 27 bits of a kept key

__device__ __forceinline__ int dg_ofpos(const DevParams& p, int ax, double x, int start1) {
  return (int)floor((x - p.dg_start[ax]) * p.dg_inv[ax]) + start1;
}

// DESGRID_PIC for one existing particle at x (desgrid_mod.f:877-995): on a
// periodic axis a coordinate whose cell left the domain's cells moves by one
// period (the serial self-exchange of DES_PAR_EXCHANGE,
// mpi_funs_des_mod.f:38-160); then the clamped DES cell.  Returns whether x
// moved.
__device__ __forceinline__ bool dg_place(const DevParams& p, bool per, double4& x, int& cell) {
  bool moved = false;
  if (per) {
    if (p.per[0]) {
      int ci = dg_ofpos(p, 0, x.x, p.istart1);
      if (ci > p.iend1) { x.x = x.x - p.L[0]; moved = true; }
      else if (ci < p.istart1) { x.x = x.x + p.L[0]; moved = true; }
    }
    if (p.per[1]) {
      int cj = dg_ofpos(p, 1, x.y, p.jstart1);
      if (cj > p.jend1) { x.y = x.y - p.L[1]; moved = true; }
      else if (cj < p.jstart1) { x.y = x.y + p.L[1]; moved = true; }
    }
    if (p.per[2] && !p.no_k) {
      int ck = dg_ofpos(p, 2, x.z, p.kstart1);
      if (ck > p.kend1) { x.z = x.z - p.L[2]; moved = true; }
      else if (ck < p.kstart1) { x.z = x.z + p.L[2]; moved = true; }
    }
  }
  int li = min(p.iend2, max(p.istart2, dg_ofpos(p, 0, x.x, p.istart1)));
  int lj = min(p.jend2, max(p.jstart2, dg_ofpos(p, 1, x.y, p.jstart1)));
  int lk = p.no_k ? 1 : min(p.kend2, max(p.kstart2, dg_ofpos(p, 2, x.z, p.kstart1)));
  cell = dg_funijk(p, li, lj, lk);
  return moved;
}

// Minimum-image shift for periodic axes (the copy of j that the reference's
// ghost exchange places next to i).
__device__ __forceinline__ double periodic_shift(const DevParams& p, int ax, double d) {
  if (!p.per[ax]) return 0.0;
  double L = p.L[ax];
  if (d > 0.5 * L) return -L;
  if (d < -0.5 * L) return L;
  return 0.0;
}

// The bound on any particle's displacement since the build: what has been
// added up plus the pending step's largest (called by whole warps).
__device__ __forceinline__ double displacement_bound(const double* __restrict__ skin,
                                                     const unsigned* __restrict__ pending) {
  return skin[0] + (double)__uint_as_float(__reduce_max_sync(0xffffffffu, pending[threadIdx.x & 31]));
}

// What the integrating gather's first warp does for the step besides: the
// pending displacement joins the bound (and the candidate list's) and its
// slots are cleared for the step after the next, and the next pass's contact
// counts start at zero.  No other kernel of the step reads these then.
struct StepEnd {
  double* skin;
  unsigned* pending;
  CandState* cand;
  ContactCount* next;
};
__device__ __forceinline__ void add_displacement(double* __restrict__ skin, CandState* __restrict__ cand,
                                                 unsigned* __restrict__ slots) {
  const unsigned m = __reduce_max_sync(0xffffffffu, slots[threadIdx.x & 31]);
  slots[threadIdx.x & 31] = 0;
  if ((threadIdx.x & 31) == 0) {
    skin[0] = skin[0] + (double)__uint_as_float(m);
    if (cand) cand->disp = cand->disp + (double)__uint_as_float(m);
  }
}
__device__ __forceinline__ void end_step(const StepEnd& e) {
  if (blockIdx.x != 0 || threadIdx.x >= 32) return;
  add_displacement(e.skin, e.cand, e.pending);
  if (threadIdx.x == 0) *e.next = ContactCount{0ull, 0ull};
}

// Adds a particle's displacement bound of this step (max(|v|, |v_new|)*dt,
// as float bits rounded up) to the per-step maximum.  Called by every active
// lane of a warp; one atomic per warp, spread over 32 slots.
__device__ __forceinline__ void note_displacement(unsigned* __restrict__ vslot, double disp) {
  const unsigned bits = __float_as_uint(__double2float_ru(disp));
  const unsigned mask = __activemask();
  const unsigned m = __reduce_max_sync(mask, bits);
  const int lane = threadIdx.x & 31;
  if (lane == __ffs(mask) - 1 && m)
    atomicMax(&vslot[((blockIdx.x * blockDim.x + threadIdx.x) >> 5) & 31], m);
}

// The larger of two speeds (the square root is monotonic, so one does).
__device__ __forceinline__ double max_speed(const double a[3], const double b[3]) {
  return sqrt(fmax(dot3(a, a), dot3(b, b)));
}

// Result of the force sum of one particle: either stored into FC/TOW
// (MODE 0) or integrated as CFUPDATEOLD + CFNEWVALUES (cfupdateold.f:33-41,
// cfnewvalues.f:700-812) into the other state buffer (MODE 1 = Euler,
// MODE 2 = Adams-Bashforth).  Velocity updates apply to NORMAL particles,
// position updates to states below NORMAL_GHOST.
// Outputs of DESGRID_PIC when the integration does it for the new positions
// (a null dg_pijk: not done there).
struct CellOut {
  int* dg_pijk = nullptr;
  uint8_t* wall_cand = nullptr;
  const int* fbin_start = nullptr;
  float* wgap = nullptr;  // facet clearance of the last build: -1 (unknown) on a change of cell
};

template <int MODE>
__device__ __forceinline__ double4 finish_particle(const DevParams& p, int me, int8_t st, const double x[3],
                                                const double v[3], const double w[3], double r, double m,
                                                double omoi, const double f[3], const double t[3],
                                                double4* __restrict__ pos_n, double4* __restrict__ vel_n,
                                                double4* __restrict__ omg_n, double* __restrict__ fc,
                                                double* __restrict__ tow, double* __restrict__ acc_old,
                                                double* __restrict__ rot_acc_old, unsigned* __restrict__ vslot,
                                                CellOut cells = CellOut{}, bool keep_w = false) {
  const size_t n = (size_t)p.n;
  if (MODE == 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c) { fc[c * n + me] = f[c]; tow[c * n + me] = t[c]; }
    return make_double4(x[0], x[1], x[2], r);
  }
  const double dt = p.dt;
  double xn[3], vn[3], wn[3], fm[3], ab[6];
  if (MODE == 2) {
    // all six before the first store (for the compiler they might alias)
#pragma unroll
    for (int c = 0; c < 3; ++c) { ab[c] = acc_old[c * n + me]; ab[3 + c] = rot_acc_old[c * n + me]; }
  }
  div3(f, m, fm);
  if (MODE == 1) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      vn[c] = v[c];
      if (st == DEM_STATE_NORMAL) vn[c] = v[c] + dt * (fm[c] + p.grav[c]);
      xn[c] = x[c];
      if (st < DEM_STATE_NORMAL_GHOST) xn[c] = x[c] + vn[c] * dt;
      wn[c] = w[c];
      if (st == DEM_STATE_NORMAL) wn[c] = w[c] + t[c] * omoi * dt;
    }
  } else {
    const bool fp_ok = !(st == DEM_STATE_NONEXISTENT || st == DEM_STATE_ENTERING || st == 102 ||
                         st == DEM_STATE_NORMAL_GHOST || st == 110);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double ao = ab[c], ro = ab[3 + c];
      if (p.first_pass && fp_ok) { ao = fm[c] + p.grav[c]; ro = t[c]; }
      double a = f[c];
      if (st == DEM_STATE_NORMAL) a = fm[c] + p.grav[c];
      vn[c] = v[c];
      if (st == DEM_STATE_NORMAL) vn[c] = v[c] + 0.5 * (3.0 * a - ao) * dt;
      acc_old[c * n + me] = a;
      xn[c] = x[c];
      if (st < DEM_STATE_NORMAL_GHOST) xn[c] = x[c] + 0.5 * (v[c] + vn[c]) * dt;
      wn[c] = w[c];
      if (st == DEM_STATE_NORMAL) {
        wn[c] = w[c] + 0.5 * (3.0 * t[c] * omoi - ro) * dt;
        ro = t[c] * omoi;
      }
      rot_acc_old[c * n + me] = ro;
    }
  }
  double4 xo = make_double4(xn[0], xn[1], xn[2], r);
  if (cells.dg_pijk) {
    // the step's DESGRID_PIC for a periodic system, on the new position
    if (st == DEM_STATE_NONEXISTENT) {
      cells.dg_pijk[me] = 0;
      cells.wall_cand[me] = 0;
    } else {
      int c;
      dg_place(p, true, xo, c);
      if (cells.dg_pijk[me] != c) cells.wgap[me] = -1.0f;
      cells.dg_pijk[me] = c;
      const int fc = p.cell_off + c - 1;
      cells.wall_cand[me] = cells.fbin_start[fc + 1] > cells.fbin_start[fc] ? 1 : 0;
    }
  }
  pos_n[me] = xo;
  vel_n[me] = make_double4(vn[0], vn[1], vn[2], m);
  // keep_w: the spin stays as it is (the gather did not read it)
  if (!keep_w) omg_n[me] = make_double4(wn[0], wn[1], wn[2], omoi);
  // |x_new - x| <= max(|v|, |v_new|) * dt for both integrators
  note_displacement(vslot, st < DEM_STATE_NORMAL_GHOST ? max_speed(v, vn) * dt : 0.0);
  return xo;  // the new position
}

}  // namespace demb

#define DEM_LAUNCH(h) ((h)->launches++)

namespace demb {
// A kernel that may start while the one before it on the stream drains
// (programmatic dependent launch): it calls pdl_wait() before it touches
// memory, which returns when that kernel is complete, and pdl_next() lets the
// one after it start likewise.  Between two kernels of a captured step this
// leaves out most of the launch latency.  pdl_wait() returns a zero that the
// compiler does not know: every address that the kernel reads through a
// read-only pointer has it in its index, since such a load could otherwise be
// moved ahead of the wait.
// With the wall work in the pair launch, and the displacement bound and the
// counters moved into the gather, a step of the 4,000-sphere box went from
// 24.4 to 17.8 us; the hoppers' from 68 to 59 us.
__device__ __forceinline__ int pdl_wait() {
  int zero;
  asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, 0;" : "=r"(zero)::"memory");
  return zero;
}
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class... P, class... A>
inline void launch_pdl(dem_handle* h, void (*kernel)(P...), unsigned grid, unsigned threads, A&&... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(threads);
  c.stream = h->stream;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  // Only where what comes before is known to be a kernel: in a captured period
  // (copies and the waits for the other stream marked by `joined`) and where a
  // caller says that nothing else comes between (chain).
  c.numAttrs = (h->capturing || h->chain) && h->stream && !h->joined ? 1 : 0;
  h->joined = false;
  cudaLaunchKernelEx(&c, kernel, P(args)...);
  DEM_LAUNCH(h);
}
}  // namespace demb

namespace demb {
// A single handle with a periodic axis places its particles in their DES
// cells in the integrating gather (the step's DESGRID_PIC then runs only on
// neighbour-search steps, where it repeats the same placement).
inline bool cells_in_gather(const dem_handle* h) {
  const DevParams& p = h->dp;
  // not with flow boundaries: their cell tests read the cells of the last
  // DESGRID_PIC, which the placement would move ahead
  return !h->batch() && h->obc.empty() && h->ibc.empty() && (p.per[0] || p.per[1] || (p.per[2] && !p.no_k));
}
inline StepEnd step_end(const dem_handle* h) {
  return StepEnd{h->skin, h->vslot_pending(), h->cand, &h->derr->count[1 - h->cur]};
}
template <int MODE, bool B>
inline CellOut gather_cells(const dem_handle* h) {
  CellOut c;
  if (MODE != 0 && !B && cells_in_gather(h)) {
    c.dg_pijk = h->dg_pijk;
    c.wall_cand = h->wall_cand;
    c.fbin_start = h->fbin_start;
    c.wgap = h->wgap;
  }
  return c;
}
}  // namespace demb
