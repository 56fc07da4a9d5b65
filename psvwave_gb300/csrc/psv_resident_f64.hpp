// FP64 time stepping with the grid resident on chip (psv_resident_f64.cu):
// the arithmetic of the two-kernel step, bit for bit, in one launch for all
// time steps.
#pragma once

#include <cuda_runtime.h>

#include "psv_resident.hpp"
#include "psv_solver.hpp"

namespace psv {
namespace resident64 {

// tiles_x x tiles_z CTAs of `threads` threads, `help` warps of them helpers;
// the others hold at most `rows` (1, 2 or 4) points each. n_rec, n_term: the
// most receivers and injection terms of a tile; box: mailbox words of a CTA. No
// CTAs: does not fit.
struct Plan {
  int tiles_x = 0, tiles_z = 0, rows = 0, help = 0, threads = 0;
  int n_rec = 0, n_term = 0, box = 0;
  size_t smem = 0;
  int ctas() const { return tiles_x * tiles_z; }
};
// g.sources: the cells of each launch's injection terms, one entry a term.
Plan plan(const resident::Grid &g, double dx, double dz);
size_t mailbox_bytes(const Plan &p);

// n_steps steps of shot `shot` (forward: it0, it0 + 1, ...; adjoint: it0,
// it0 - 1, ...) on the fields of `a`, in place, as forward_f64 / adjoint_f64
// run them (forward: receivers' raw velocities are recorded; snapshots with
// store). zero: from zero fields. mail: mailbox_bytes of scratch. One
// cooperative launch; *err is raised when a bounded wait runs out.
cudaError_t steps(const SolverArgs &a, const InjPlan &inj, const Plan &p, int shot, bool adjoint,
                  int it0, int n_steps, bool zero, bool store, void *mail, int *err,
                  cudaStream_t s);

}  // namespace resident64
}  // namespace psv
