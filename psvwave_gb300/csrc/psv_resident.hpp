// FP32 time stepping of grids held on chip for every time step of a launch
// (psv_resident_core.cuh).
//
// A simulation runs on a team of CTAs, each owning a tile. Every thread keeps
// its points' wave fields and medium in registers for all steps, and the tile's
// fields lie in shared memory for the neighbours' stencils. After each half-step
// the tile's edges go to the neighbouring CTAs, by one of two links. A team of up
// to 16 CTAs is one thread-block cluster (tiles of up to 152 columns) and writes
// straight into its neighbours' shared memory, counted on their mbarriers. Any
// other (tiles of up to 64 columns, one or two CTAs on an SM) goes through
// mailboxes in global memory (L2), whose 128-bit words carry three values and the
// step's number, so that the receiver needs no flag, fence or barrier. Global
// memory otherwise carries only the initial and final state, receivers,
// snapshots, correlations and injection.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "psv_tma.hpp"

namespace psv {
namespace resident {

// A grid to split: its size, and the cells (ix nz + iz) of its receivers, of
// each shot's injection points, and of its injection terms (a cell per term).
struct Grid {
  int nx = 0, nz = 0;
  std::vector<int> receivers;
  std::vector<std::vector<int>> sources, terms;
};

// How one simulation is split: tiles_x x tiles_z CTAs, blocks of `threads`
// with `groups` thread groups of at most `rows` rows each, shared rows of
// `stride` floats; n_rec, n_inj, n_term: the most receivers, injection points
// and terms of a tile. cluster: the team is one thread-block cluster; otherwise its edges go
// through mailboxes. No CTAs: the grid does not fit.
struct Plan {
  int tiles_x = 0, tiles_z = 0, groups = 0, rows = 0, threads = 0, stride = 0;
  int n_rec = 0, n_inj = 0, n_term = 0;
  bool cluster = false;
  size_t smem = 0;
  int ctas() const { return tiles_x * tiles_z; }
};

// The split of a grid for one simulation at a time: the largest cluster that
// holds it, else mailboxes over the whole device. These calls set launch
// attributes as a side effect (call outside stream capture). Measured, one
// simulation, us a step: 250 x 150 points in one cluster of 16 CTAs 1.7, by
// mailboxes 2.6 to 3.6 (32 to 152 CTAs); 1103 x 497 points 3.9 by mailboxes.
// Clusters of 16 | 8 | 4 | 2 | 1 CTAs, forward: 24 x 20 points 1.03 | 1.04 | 1.06 |
// 0.97 | 0.99, 40 x 40 0.96 | 1.06 | 0.98 | 1.09 | 1.31, 68 x 56 0.99 | 1.04 | 1.24 |
// 1.58 | 2.06, 100 x 80 1.03 | 1.21 | 1.61 | 2.5 | -.
Plan plan(const Grid &g);
// A cluster of exactly nc CTAs.
Plan plan_cluster(const Grid &g, int nc);
// Mailboxes over at most max_ctas CTAs (0: as many as are resident at once),
// per_sm (1 or 2) of them sharing an SM.
Plan plan_mailbox(const Grid &g, int max_ctas, int per_sm);

// States saved during a run: the state before step j of the launch goes to
// base + (j / every) * stride when j % every == 0 (five planes of
// nx * pitch floats).
struct Dump {
  float *base = nullptr;
  size_t stride = 0;
  int every = 1;
};

// Mailbox bytes of a plan (0 for a cluster).
size_t mailbox_bytes(const Plan &p);

// n_steps steps of simulation d from set `parity` (forward: it0, it0 + 1,
// ...; adjoint: it0, it0 - 1, ...), final state in set parity ^ (n_steps & 1);
// forward snapshots when store. zero: start from zero fields instead of the
// set's. mail: mailbox_bytes(p) of scratch (cleared here on s). One launch. *err is raised when a bounded wait for a neighbour runs
// out.
cudaError_t steps(const tma::SimDesc &d, const Plan &p, bool adjoint, int it0, int n_steps,
                  int parity, bool zero, bool store, const Dump &dump, void *mail, int *err,
                  cudaStream_t s);

// ---- exact gradients (psv_resident_exact.cu) ----

// The split of an exact gradient of one simulation: forward steps that keep
// their rates, and the exact adjoint's steps, on the same tiles. n_src: the
// most source points of a tile; smem, rate_smem: the adjoint's and the keeping
// forward steps'. lanes: how many run at
// once, each on its share of the device.
struct ExactPlan {
  Plan p;
  int n_src = 0, n_term = 0;
  size_t smem = 0, rate_smem = 0;
  size_t rate_stride = 0;  // float2 per step
};
ExactPlan plan_exact(const Grid &g, int lanes);

// Steps it0, it0 + 1, ... of d from set 0 (zero: from zero fields), as
// steps() takes them, keeping the rates of step it0 + k at
// rates + k * rate_stride; final state in set n_steps & 1.
cudaError_t steps_keeping_rates(const tma::SimDesc &d, const ExactPlan &p, int it0, int n_steps,
                                bool zero, float2 *rates, void *mail, int *err, cudaStream_t s);

// The exact adjoint (notation in psv_exact.cuh) of steps first + n_steps - 1
// down to first: d.set[0] holds l of the last of them (zero: it is zero)
// and takes l of the first; d.plan's terms add the series a_ux, a_uz to the
// adjoint velocities. The gradients of lm, mu (with lambda = lm - 2 mu) and b
// are summed in FP32 for `flush` steps at a time, which are logged (log: three
// planes of nx * pitch for each multiple of `flush` among the steps) and then
// added to float-float pairs `sums` of nx * nz, later steps first; what a
// launch leaves unlogged it hands to the next in part (three planes).
struct ExactSteps {
  int first = 0, n_steps = 0;
  bool zero = false;
  const float2 *rates = nullptr;
  InjPlan src{};  // the shot's source terms
  float *part = nullptr, *log = nullptr;
  float2 *sums[3] = {nullptr, nullptr, nullptr};
  int flush = 1;
};
// Entries of the log for n_steps steps at most.
inline int log_entries(int n_steps, int flush) { return (n_steps - 1) / flush + 1; }
cudaError_t exact_steps(const tma::SimDesc &d, const ExactPlan &p, const ExactSteps &x,
                        void *mail, int *err, cudaStream_t s);

// ---- batches: forward steps of many simulations from zero fields ----

// One member of a batched launch: its CTAs first .. first + tiles_x tiles_z - 1
// run simulation `sim` of the table.
struct Member {
  int sim, first, tiles_x, tiles_z, groups, n_rec, n_inj, n_term;
};
// One launch: CTAs first_cta .. first_cta + ctas - 1 of the CTA table (the
// launch's member of each), members from first_member on. team > 0: clusters
// of `team` CTAs, one member each, as many as there are (they queue for the
// device); team = 0: a cooperative launch whose teams exchange edges through
// mailboxes. All members have plans of `rows` and `stride`; threads and smem
// are their largest.
struct Launch {
  int first_member = 0, first_cta = 0, ctas = 0, team = 0;
  int rows = 0, stride = 0, threads = 0;
  size_t smem = 0;
};
size_t launch_mailbox_bytes(const Launch &l);
cudaError_t steps_batch(const tma::SimDesc *sims, const Member *members, const int *cta_member,
                        const Launch &l, int n_steps, bool store, void *mail, int *err,
                        cudaStream_t s);
// CTAs resident at once in a cooperative launch of per_sm CTAs per SM.
int resident_slots(int per_sm);
// The mailbox split with the fewest CTAs, and the same with tiles_x tiles
// along x (false, p unchanged: does not fit).
Plan plan_smallest(const Grid &g, int per_sm);
bool set_tiles_x(Plan &p, const Grid &g, int tiles_x, int per_sm);

}  // namespace resident
}  // namespace psv
