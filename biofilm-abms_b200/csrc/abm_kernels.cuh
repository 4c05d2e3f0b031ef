// Kernel-side shared types and launch wrappers of the B200 mechanics step.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "abm_device.cuh"

namespace abm {

const int MAX_STAGES = 7;

// Controller modes of one iteration (simulation.hpp:1690-1769)
// MODE_COMMIT: the learned controller's proposal passed the error test; the final
// attempt copies its candidate state instead of re-running the step.
enum CtrlMode { MODE_TRIAL = 0, MODE_RETRY = 1, MODE_FINAL = 2, MODE_COMMIT = 3 };

// How a kernel of an iteration is launched.  FLOW_STEP: as one iteration of its own.  The loop
// graph advances many: rounds of FLOW_FAST iterations, in which the kernels follow one another
// without a conditional node and leave at once when there is nothing to do (no iteration
// left, or Ctrl::hold), and after each round, only where Ctrl::hold asks for it, what the fast
// iterations wait for: the FLOW_SLOW rest of an iteration whose first attempt failed, or a
// division.
enum LoopFlow { FLOW_STEP = 0, FLOW_FAST = 1, FLOW_SLOW = 2 };
// Ctrl::hold: the next iteration has to start with the division launch (a cell has reached
// the division length, or the colony its limit); or the running one waits for its retries.
enum LoopHold { HOLD_NONE = 0, HOLD_START = 1, HOLD_RETRY = 2 };

// Ctrl::halted: the population has reached its limit; or a wait among a launch's blocks has run
// out, after which the barrier record, the bin counts and the neighbor set are not to be used:
// every kernel that would leaves at once, and the status stays ST_BARRIER.
enum HaltBits { HALT_CELLS = 1, HALT_LOST = 2 };

// Step-size network: 32 features -> 64 -> 64 -> 1 (log dt ratio)
const int MLP_IN = 32, MLP_H = 64;
const int MLP_OFF_W1 = 0, MLP_OFF_B1 = MLP_OFF_W1 + MLP_H * MLP_IN, MLP_OFF_W2 = MLP_OFF_B1 + MLP_H;
const int MLP_OFF_B2 = MLP_OFF_W2 + MLP_H * MLP_H, MLP_OFF_W3 = MLP_OFF_B2 + MLP_H, MLP_OFF_B3 = MLP_OFF_W3 + MLP_H;
const int MLP_NPARAM = MLP_OFF_B3 + 1;
// log row: 32 features, ln(dt_max / dt_first), ln(dt_first / dt_prev), log10 E, passed,
// the proposal's error-model baseline, 3 spare columns
const int MLP_LOG_COLS = 40;
const int HIST = 8;
const int STAT_V2_SHIFT = 20, STAT_G_SHIFT = 32;

// Status bits raised on the device and turned into ABM_ERR_* by the host.
enum StatusBits {
    ST_NAN = 1,            // NaN/Inf in the error norm or velocities
    ST_NBR_OVERFLOW = 2,   // more neighbors than cap_neighbors_per_cell
    ST_BIN_OVERFLOW = 4,   // grid needs more bins than allocated
    ST_CELL_OVERFLOW = 8,  // division would exceed cap_cells
    ST_BARRIER = 16,       // a grid barrier's bounded wait ran out
};

// Blocks of a launch whose blocks wait for one another: one cluster, or a cooperative grid
struct LaunchShape {
    int blocks = 1;
    int cluster = 0;
};
// `threads` threads of work in blocks of `block`, on a `share`-th of the chip (the contexts of a
// batch run side by side).  A cooperative grid starts when all its blocks have room, so one that
// fills the chip waits for every other context's work and holds up theirs: a batch of 24 growing
// colonies of 20,000 cells took 2.8 ms an iteration with whole-chip grids (2.6 as the chain of
// plain kernels before them) and takes 0.97 with a 24th of the chip each; 8 of them at rest 108
// and 56 us.
LaunchShape make_shape(const void* kernel, int block, long long threads, bool cluster, int num_sms, int share);
// the runtime's answer: a launch that it refuses did not happen
cudaError_t launch_shape(const void* kernel, const LaunchShape& shape, int block, void** args, cudaStream_t st);

// Record of a barrier over the blocks of a cooperative launch (abm_grid.cuh)
struct GridBar {
    unsigned int count, gen;
};

// Device-resident clock, controller and population state.  Fetched and put back whole by the
// last block of every attempt: 72 words, whole sectors; one more took up to 0.27 us an iteration
// (200 iterations of 64 cells 5.31 against 5.26 ms), so fields for rare events sit in the gaps of
// the alignment.
struct Ctrl {
    double t, dt;               // simulated time, current step size
    double dt_try;              // step size of the next attempt
    double factor;              // controller factor (simulation.hpp:1710-1757)
    double last_max_error;
    double last_trial_error;
    unsigned long long err_bits;    // max scaled error of the running attempt (ordered bits)
    unsigned int blocks_done;       // last-block counter of the running attempt
    int iter;
    int mode;                   // CtrlMode
    int tries;                  // j in simulation.hpp:1716
    int attempt;                // attempt index within the iteration (noise stream)
    int status;                 // StatusBits
    int n;                      // cells
    int n_dir;                  // directed neighbor entries (2 x pairs)
    int no_table;               // the last build found no neighbor set (an overflow): it is empty
    int path_valid;             // as screen_valid, but that a loaded checkpoint keeps it (see path)
    long long attempts, retries, iterations, rebuilds, divisions;
    unsigned long long eval_err_bits;   // scaled max error of the last API attempt
    int n_pairs;                // pair records made so far by a running build
    int n_sorted;               // cells placed so far by its counting sort
    int n_divided;              // mothers of the last division launch
    int last_div_tries;
    int n_parents;              // length of the lineage vector
    long long div_events;       // iterations in which cells divided
    // step-size features (filled when StepParams::stats_on)
    // sums in fixed point so that their value does not depend on the order of the atomics
    unsigned long long st_vmax_bits;    // max |v_r| of the last accepted step (ordered bits)
    unsigned long long st_ovl_bits[2];  // max overlap of the pair-force passes of even / odd iterations
    unsigned long long st_v2_fx;        // sum |v_r|^2 * 2^STAT_V2_SHIFT
    unsigned long long st_g_fx;         // sum of growth rates * 2^STAT_G_SHIFT
    unsigned long long st_near_div;     // cells with l > 0.9 Ldiv
    int since_div;                      // accepted steps so far (feature 31, abm_propose.cuh)
    int waiting;                        // HALT_CELLS, while a call evaluates a colony at its limit
    double hist_dt[HIST], hist_err[HIST];   // accepted dt and its scaled error, newest at hist_pos - 1
    int hist_acc[HIST];                 // 1 if that iteration's first attempt passed the error test
    int hist_pos;
    int first_passed;                   // the running iteration's first attempt passed
    double dt_prev;                     // accepted dt before the running iteration
    long long rejected;                 // iterations whose first attempt failed the error test
    long long log_rows;                 // feature rows written (ring position = log_rows % capacity)
    // cell-count stop on the device (terminate(), simulation.hpp:1600-1615): decided at the
    // start of each iteration by the division count; a halted context skips its iterations
    int halt_n;                         // 0 = no limit
    int halted;                         // HaltBits
    long long cell_steps;               // sum of the population over accepted steps
    // screened pair pass: the active list (pairs that passed the bound test with the
    // skin at the last refresh) and the motion since then
    int n_surv;                         // active pairs
    int n_surv_next;                    // pairs appended by a refresh in progress
    int screen_valid;                   // 0 after a rebuild, an upload or a division
    unsigned int surv_blocks;           // last-block counter of the pair pass
    int n_order;                        // cells covered by the attempt order (0: index order)
    // frames: an accepted step whose time crosses a multiple of dt_write marks a frame,
    // which the snapshot kernel at the end of the iteration copies into a ring slot
    double dt_write;                    // 0: no frames
    int frame_due, frames_taken;
    unsigned int frame_blocks;          // last-block counter of the snapshot kernel
    // friction: candidate pairs of the last pair pass, pairs whose decisions change with the
    // stage, and the trial loop's state (a trial pass is pending; a check changed a decision)
    int fr_ncand, fr_ncand_next;
    int fr_nflip, fr_nflip_next;
    int fr_pending, fr_changed;
    unsigned int fr_blocks;
    // basal-only compaction: cells kept by the last test, cells dropped so far
    int n_keep;
    long long basal_dropped;
    double drift;                       // max over cells of the segment's motion since the last refresh
    unsigned long long drift_bits;      // block maxima of the running attempt (ordered bits)
    // mixed precision: the sum over the accepted steps of the largest motion in each.  A pass
    // whose list would be stale by this sum takes ROUND_STALE (dist_geom_mixed), whether or not
    // the list is stale by `drift`: the rule keeps mixed-precision trajectories bit for bit.
    // A loaded checkpoint brings the sum and path_valid back, so that the first pass after it
    // rounds as the uninterrupted run's does, although its list has to be made anew.
    double path;
    unsigned long long path_bits;
    // the loop graph (LoopFlow): iterations still to take, and why the plain ones wait
    int todo;
    int hold;                           // LoopHold
    int div_any;                        // a cell grew past Ldiv in the running attempt's step
    int rounds;                         // rounds of the loop graph left (a bound)
};

// Nothing to do for a kernel of the loop graph?
__device__ __forceinline__ bool loop_idle(const Ctrl* c, int flow)
{
    return flow != FLOW_STEP && (c->todo <= 0 || c->hold != (flow == FLOW_FAST ? HOLD_NONE : HOLD_RETRY));
}

struct Grid {
    double x0, y0, z0, edge, inv_edge;
    int nx, ny, nz, nbins;
    double max_half_l;
    double reach;               // no two neighbors' centres are farther apart
    float max_reach;            // largest segment_reach
    float margin;               // of the FP32 distance tests on sorted positions
};

struct StepParams {
    MechParams mp;
    int s;                      // stages
    double A[MAX_STAGES][MAX_STAGES], b[MAX_STAGES], bs[MAX_STAGES];
    double inv_q1;              // 1 / (error_order + 1)
    double tol, min_error, min_stepsize, max_stepsize;
    int max_tries, iter_update_stepsize;
    double noise_max[6];
    int noise_on;
    uint64_t seed;
    // 2-D model: composite drag eta0 + eta1 rho_c / R (2D/include/mechanics.hpp:264-279)
    double rho_c;
    double max_noise_2d;
    // step-size control
    int propose;                // 1: every iteration's first attempt runs at a proposed dt and is
                                // accepted as is when its error passes (learned and PI controllers)
    int network;                // 1: the step-size network makes the proposal (learned controller)
    int pi;                     // 1: the PI rule makes the proposal after each accepted step
    int mixed;                  // 1: mixed precision (3-D): cells in surface contact take the FP32
                                // contact branch of the velocity solve
    int fric;                   // 1: cell-cell kinetic friction (3-D, FP64)
    int div_on;                 // 1: cells may divide
    double Ldiv;
    int stats_on;               // accumulate the network's features (learned or logging)
    double near_div_length;     // 0.9 Ldiv
    double4* stat_part;         // per-block (max |v_r|, sum |v_r|^2, sum growth, near-division count)
    float* log_buf;             // MLP_LOG_COLS floats per row, log_cap rows (ring)
    int log_cap;
    const int* order;           // attempt order of the first ctrl->n_order cells (3-D), or null
    int order_cap;              // its entries
};

struct ForceParams {
    double R, Rcell, E0;
    double pf0, pf1, pf2;       // repulsion prefactors (simulation.hpp:1270-1274)
    double max_overlap;         // 2 (R - Rcell)
    int adhesion;
    int jkr_n;
    double jkr_step;            // spacing of the overlap mesh
    // variable-gamma table (IsotropicJKRDataVariableGamma, mechanics.hpp:159-199): radii on
    // the overlap mesh x the gamma mesh, overlap-major; jkr_ng = 0 without it
    int jkr_ng;
    double jkr_gstep;           // spacing of the gamma mesh
    const double* jkr_gam;      // gamma mesh (jkr_ng)
    const double* jkr_rad2;     // radii (jkr_n x jkr_ng)
    int stats;                  // record the max overlap (step-size features)
    double skin;                // screened pair pass: margin of the active list (um)
    // 2-D model (ABM-2d): Hertz prefactors of 2D/include/simulation.hpp:232-235 and
    // the JKR-Lagrange adhesion of 2D/include/adhesion.hpp:403-448
    double pf2d[3];
    double adh_strength, adh_mindist;
    const unsigned char* adhere;    // per CSR entry: to_adhere at the last rebuild
    // cell-cell kinetic friction (cellCellFrictionForces, mechanics.hpp:1031-1175), FP64, 3-D
    int fric;
    int surface;                    // a surface is present (the planar-contact rule applies)
    double coulomb_cc;              // Coulomb cap coefficient (not positive: no cap)
    const Vel* vel;                 // stored velocities of the cells (dr, dn)
    const double* feta;             // friction coefficient of each cell
    double4* fbuf;                  // per active share: its change when the planar decision flips
    int* fmask;                     // per active share: FR_* bits
    int* fr_list;                   // active pairs with a planar-contact candidate, this pass
};

// Friction: a contact with |dz / d| < 1e-3 whose two contact points lie below 1.01 R is taken
// in the xy-plane (mechanics.hpp:1090-1110).  The positions enter only through that test, so
// an attempt's pair forces are fixed but for those candidate pairs, whose planar decision can
// change from stage to stage.  Per CSR entry: FR_CAND, FR_D0 = the decision at y0, and bits
// 0-7 = the stages whose decision differs from FR_D0.
const int FR_CAND = 1 << 16, FR_D0 = 1 << 17, FR_FLIPS = 0xFF;

struct BuildParams {
    double threshold;           // neighbor_threshold
    double prefilter;           // neighbor_threshold + Ldiv + 2 R (mechanics.hpp:551)
    int cap_per_cell;
};

// The active pairs: those within 2R + skin at the last refresh.  Each cell's active shares
// lie at the start of its row's slots in `jbuf`, in the row's column order.
struct ActiveList {
    int4* act;                  // (i, j, slot of i's share, slot of j's share); j's sign bit: to_adhere (2-D)
    int* n_act;                 // active shares of each cell
    unsigned char* keep;        // per CSR entry: active (made and read by a refresh)
    Geom* gref;                 // the cells at the last refresh
    const int* row_ptr;
    GridBar* bar;
    int cluster;                // the pass's blocks are one cluster
    double4* pbuf;              // velocity Verlet: the JKR part of each share (else null)
};
const int ACT_ADHERE = (int)0x80000000;

// Where an attempt finds the pair force when it completes the sum itself:
// fused = 2: jbuf holds both shares of every active pair, as double4;
// fused = 3: the same as float4 (mixed precision);
// fused = 0: fcc already holds the total.
struct PairGather {
    int fused;
    const int* row_ptr;
    const int* n_act;
    const double4* jbuf;
    Gen6* fcc_w;
    const Geom* gref;
    // friction: the planar-contact corrections of each stage, and the stage states of the
    // cells with candidate contacts (z and n_z per stage, written by the trial passes)
    const double4* fbuf;
    const int* fmask;
    double2* ystage;
    int ystage_ld;
};

// ---- launch wrappers (abm_kernels.cu) ----
void launch_cells_from_colmajor(const double* cm, int n, int ncols, int ld, int has_gamma,
                                Geom* geom, Vel* vel, Phys* phys, cudaStream_t st);
void launch_cells_to_colmajor(const Geom* geom, const Vel* vel, const Phys* phys, int n, int ncols,
                              int ld, int has_gamma, double* cm, cudaStream_t st);
// 2-D layout (ABM-2d/ABM-2d-cpp/include/indices.hpp) <-> records with z = 0
void launch_cells_from_colmajor_2d(const double* cm, int n, int ncols, int ld, Geom* geom, Vel* vel, Phys* phys,
                                   cudaStream_t st);
void launch_cells_to_colmajor_2d(const Geom* geom, const Vel* vel, const Phys* phys, int n, int ncols, int ld,
                                 double* cm, cudaStream_t st);
// 2-D dE/dq (n x 4) from the pair sums (F, S): torques projected with the current n
void launch_pair_dEdq_2d(const Geom* geom, const Gen6* fcc, const Ctrl* ctrl, double* cm, int cap_cells,
                         cudaStream_t st);
void launch_gen6_to_colmajor(const Gen6* g, int n, double* cm, cudaStream_t st);

// exclusive scan of len (device int) entries; out has len + 1 entries, out[len] = total
void launch_scan(const int* in, const int* len, int* out, int* block_sums, int cap, cudaStream_t st);
size_t scan_block_sums_size(int cap);

// pass over the active pairs (both shares into jbuf), refreshing the active list when it is
// stale; with_sum also writes each cell's total into fcc.  cells: about how many there are
// (the launch's shape; more only take longer); share: as for make_shape.
cudaError_t launch_pair_screened(const Geom* geom, Ctrl* ctrl, ForceParams fp, const double* jkr_delta,
                                 const double* jkr_radius, Gen6* fcc, double4* jbuf, int mixed, int max_entries,
                                 int cap_cells, int num_sms, cudaStream_t st, int with_sum, int dims, int tile,
                                 int blocks_per_sm, const int4* pairs, int* surv, ActiveList al, int cells, int share,
                                 const StepParams* sp = nullptr, const float* mlp_w = nullptr, int flow = FLOW_STEP);
// kind: MODE_TRIAL / MODE_RETRY / MODE_FINAL for the loop, 3 = evaluation for the API
// (writes candidates and errors without touching the controller)
// cond / use_cond: WHILE-node handle that the trial and retry attempts set to 1
// when the controller asks for another retry (only inside a CUDA graph)
struct AttemptArgs {
    Geom* geom;
    Vel* vel;
    Phys* phys;
    const Gen6* fcc;
    Ctrl* ctrl;
    const StepParams* sp;
    Geom* geom_c;
    Vel* vel_c;
    Gen6* k0buf;
    int cap_cells;
    int cells, num_sms;         // cells there are, as far as the host knows (the kernel's shape)
    PairGather pg;
    // the API's evaluation
    Gen6* err_out;
    double eval_dt;
    int eval_attempt;
    // graph conditions
    unsigned long long cond;
    int use_cond;
    unsigned long long cond_run;
    int flow;                   // LoopFlow
};
void launch_attempt(int kind, const AttemptArgs& a, int dims, cudaStream_t st);
// one translation unit per stage count (abm_attempt.cuh)
void launch_attempt_2(int kind, const AttemptArgs& a, int dims, cudaStream_t st);
void launch_attempt_4(int kind, const AttemptArgs& a, int dims, cudaStream_t st);
void launch_attempt_6(int kind, const AttemptArgs& a, int dims, cudaStream_t st);
void launch_attempt_7(int kind, const AttemptArgs& a, int dims, cudaStream_t st);
// one frame of the ring: the state after the accepted step that marked it
struct FrameInfo {
    double t;
    int iter, n, n_parents, pad;
};
// copies the cells into ring slot frames_taken % slots when a frame is due
void launch_frame_snapshot(const Geom* geom, const Vel* vel, const Phys* phys, Ctrl* ctrl, Geom* snap_geom,
                           Vel* snap_vel, Phys* snap_phys, FrameInfo* info, int slots, int cap_cells,
                           cudaStream_t st, const double* feta = nullptr, double* snap_feta = nullptr);
void launch_velocities(const Geom* geom, const Vel* vel, const Phys* phys, const Gen6* fcc,
                       const Ctrl* ctrl, const StepParams& sp, Gen6* v_out, int cap_cells,
                       cudaStream_t st, int dims = 3);
void launch_grow(Geom* geom, Phys* phys, const Ctrl* ctrl, double R, double dt, int cap_cells,
                 cudaStream_t st);

void launch_count_lower(const Ctrl* ctrl, const int* row_ptr, const int* col, int* cnt,
                        int cap_cells, cudaStream_t st);
void launch_table_rows(const Ctrl* ctrl, const int* row_ptr, const int* col, const int* pos,
                       const Geom* geom, double* out, int ld, int cap_cells, cudaStream_t st, int dims = 3);

// step-size network (abm_mlp.cu); weights are the flat FP32 master copy
void launch_mlp_forward(const float* master, const float* X, int n, float* Y, cudaStream_t st);
void launch_mlp_grad(const float* master, const float* X, const float* T, int n, float* G, float* loss,
                     cudaStream_t st);
void launch_mlp_train(float* master, float* m1, float* m2, float* G, const float* X, const float* T, int n,
                      int epochs, float lr, unsigned seed, float* loss_out, cudaStream_t st);
const int AT_T = 128;           // threads of an attempt block, one cell each
int attempt_blocks(int cap_cells);

// division (growth.hpp:66-426), abm_divide.cuh
struct DivideParams {
    double R, Rcell, Ldiv;
    double growth_mean, growth_std, daughter_length_std, angle_xy_bound, angle_z_bound;
    uint64_t seed;
    int cap_cells;
    // phenotype switching: the daughters' growth rates come from the mother's group
    // (growth.hpp:634-644), and with inherited switching one daughter of a pair may move
    // to the other group at division (switch.hpp:97-142, simulation.hpp:1650-1656)
    int group_growth;
    double gmean[2], gstd[2];
    int inherit, n_start_switch;
    double rates[4];
    double* feta;               // friction coefficient of each cell (daughters inherit it), or null
};
// Neighbor set and division (abm_build.cu): one cooperative launch
struct BuildArgs {
    Geom* geom;
    Vel* vel;
    Phys* phys;
    Ctrl* ctrl;
    GridBar* bar;
    int cluster;                            // the blocks are one cluster (else a cooperative grid)
    // cell list
    int* bbox;                              // 8 per block
    int2* part;                             // per-block partial sums of the scans
    int *bin_count, *bin_start, *key, *slot, *sorted_cell, *sorted_key;
    float4 *sorted_pos, *sorted_dir;        // (r, reach) from the box's corner; (n, h)
    int cap_bins, cap_cells;
    // neighbor set
    BuildParams bp;
    MechParams mp;
    int *scratch, *count, *row_ptr, *col, *lower_end;
    int4* pairs;
    int* order;                             // attempt order (3-D), or null
    unsigned char* adhere;                  // to_adhere of every CSR entry (2-D adhesion), or null
    // division
    DivideParams dp;
    int *flags, *mothers, *check, *sat, *ok;
    Geom *d1, *d2;
    double *dlen, *dgrowth;
    int* parents;
};
enum BuildWhat { BUILD_NEIGHBORS, BUILD_GROWTH, BUILD_DIVIDE, BUILD_RECORDS };
const int BUILD_CLUSTER_CELLS = 8192;       // launches shaped for more are cooperative grids
const int PAIR_CLUSTER_CELLS = BUILD_CLUSTER_CELLS / 2;
LaunchShape build_shape(int cells, int num_sms, int share = 1);
cudaError_t launch_build(const BuildArgs& args, int what, const LaunchShape& shape, cudaStream_t st, int flow = FLOW_STEP);

// the loop graph: `todo` iterations ahead (of each of n contexts); then, once per round,
// whether a slow iteration runs and whether another round follows
// (divides: the first iteration starts with a look for mothers and the cell limit)
void launch_loop_begin(Ctrl* ctrl, int divides, int todo, cudaStream_t st);
void launch_loop_begin_all(Ctrl* const* ctrls, const int* divides, int n, int todo, cudaStream_t st);
// a slow iteration starts: its first retry is pending (a handle's default value holds for
// the first pass through its graph only)
void launch_retry_begin(Ctrl* ctrl, unsigned long long cond, cudaStream_t st);
void launch_loop_round(Ctrl* ctrl, unsigned long long cond_slow, unsigned long long cond_loop, cudaStream_t st);
// Phenotype switching between two groups and what it drives, after each accepted step
// (abm_switch.cu): Markov switching (switch.hpp:45-95), the attribute and gamma ramps
// (simulation.hpp:1872-1957), local viscosity (simulation.hpp:1958-2020) and basal-only
// compaction (simulation.hpp:1831-1856).  Random draws: Philox, purpose SWITCH, counters
// (iteration, cell or division pair, slot).
struct SwitchParams {
    uint64_t seed;
    int mode;                   // 0 none, 1 Markov, 2 inherited at division
    int n_start;                // switching starts once the colony has this many cells
    double rates[4];            // 2 x 2, row = current group: rates (Markov) or probabilities
    double gmean[2], gstd[2];   // growth-rate distribution of each group
    double timescale;           // ramp time; 0: the attributes jump to their targets
    int n_attr;
    int attr_field[4];          // switched attributes as Phys fields: 2 eta0, 3 eta1, 4 sigma0
    double target[2][4];        // their targets in group 1 and group 2
    int gamma_ramp;             // adhesion on: gamma ramps up (group 1) or down (group 2)
    double max_gamma;
    int modulate;               // eta0 from the share of group-1 cells among the contacts
    double visc[4];             // (min, max) eta0 of group 1, then of group 2
    int max_coord;
    double R;
    int basal;                  // basal-only compaction (surface present)
    double basal_min_overlap;
};
void launch_switch_cells(Geom* geom, Phys* phys, const Ctrl* ctrl, const SwitchParams& sw, int cap_cells,
                         cudaStream_t st);
void launch_modulate_viscosity(const Geom* geom, Phys* phys, const Ctrl* ctrl, const int* row_ptr, const int* col,
                               const SwitchParams& sw, int cap_cells, cudaStream_t st);
void launch_basal_flags(const Geom* geom, const Ctrl* ctrl, const SwitchParams& sw, int* keep, int cap_cells,
                        cudaStream_t st);
void launch_basal_decide(Ctrl* ctrl, const int* keep, const int* rank, unsigned long long cond, int use_cond,
                         cudaStream_t st);
void launch_basal_compact(Geom* geom, Vel* vel, Phys* phys, Geom* geom_tmp, Vel* vel_tmp, Phys* phys_tmp,
                          Ctrl* ctrl, const int* keep, const int* rank, int cap_cells, cudaStream_t st,
                          double* feta = nullptr, double* feta_tmp = nullptr);
void launch_periodic_rebuild_cond(const Ctrl* ctrl, int every, unsigned long long cond, cudaStream_t st);

// velocity Verlet (abm_verlet.cu): the cells' part of one step of integration mode 0 at
// ctrl->dt; phase 0 after the pair pass at the current state (half kick, drift to geom_c /
// vel_c), phase 1 after the pass at the drifted state (kick, growth, bookkeeping)
struct VerletArgs {
    Geom* geom;
    Vel* vel;
    Geom* geom_c;
    Vel* vel_c;
    Phys* phys;
    double4* whalf;          // half-step angular velocity of each cell
    const int* row_ptr;
    const int* n_act;
    const double4* jbuf;
    const double4* pbuf;
    const Geom* gref;        // the cells at the last refresh of the active pairs
    double rho;              // cell density M0 / (pi ((4/3) R^3 + R^2 L0))
};
void launch_verlet_cells(int phase, const VerletArgs& a, Ctrl* ctrl, const StepParams& sp, int cap_cells,
                         cudaStream_t st);

// friction: before an attempt, trial passes that run the stages of the cells with
// candidate contacts and checks that recompute the candidates' planar decisions from
// the stage states, until the decisions agree with the states (at most stages - 1 rounds)
void launch_friction_rounds(int kind, const AttemptArgs& a, const int4* act, const int* fr_list, int* fmask, double R,
                            cudaStream_t st);
void launch_friction_rounds_2(int kind, const AttemptArgs& a, const int4* act, const int* fr_list, int* fmask,
                              double R, cudaStream_t st);
void launch_friction_rounds_4(int kind, const AttemptArgs& a, const int4* act, const int* fr_list, int* fmask,
                              double R, cudaStream_t st);
void launch_friction_rounds_6(int kind, const AttemptArgs& a, const int4* act, const int* fr_list, int* fmask,
                              double R, cudaStream_t st);
void launch_friction_rounds_7(int kind, const AttemptArgs& a, const int4* act, const int* fr_list, int* fmask,
                              double R, cudaStream_t st);

}   // namespace abm
