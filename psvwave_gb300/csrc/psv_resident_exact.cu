// Exact gradients with the grid resident on chip (psv_resident_core.cuh).
//
// The exact adjoint step (psv_exact.cuh) has the shape of a forward step: the
// velocity transpose's stencils read w = b dt T l_v as the stress half-step's
// read v, and the stress transpose's read p = dt C T l_t as the velocity
// half-step's read tau. So one member_steps serves both: the adjoint state
// and the medium stay in registers, w and p lie in the shared planes and
// cross between CTAs as v and tau do.
//
// Its gradient terms need the forward step's strain rates and accelerations at
// the thread's own points only. The recomputing forward pass keeps those five
// numbers instead of the state (the same bytes), in the thread's own order:
// the adjoint needs no stencil, no halo and no second look at them. A helper
// fetches a step's numbers with bulk copies, three fields for the stress half
// while the velocity half runs and two the other way round. The sums of the
// gradients stay in shared memory.
//
// What bounds it: the per-step kernels it replaces moved 51 planes of the grid
// per step and shot through L2 and DRAM (13 a forward step, 25 an adjoint
// step) in three launches; this moves 10, in two launches per segment. Then, as
// for all resident steps, computation and the exchange of edges. us per step
// and shot, those kernels -> these: 250 x 150 25.0 -> 7.4 (one shot), 8.6 -> 1.2
// (eight at a time); 500 x 300 29.6 -> 8.3, 10.2 -> 5.6; 900 x 450 36.6 -> 11.8,
// 15.5 -> 11.0; 1100 x 500 35.9 -> 16.6, 19.0 -> 15.7. Grids that do not fit with
// the adjoint's shared memory keep them.
#include "psv_resident_core.cuh"

namespace psv {
namespace resident {
namespace {

template <int MODE, int K, int S, bool CLUSTER>
__global__ void __launch_bounds__(kMaxThreads, 1)
    resident_exact(const __grid_constant__ tma::SimDesc d, const Team team, int it0, int n_steps,
                   int zero, const RateIo io, int *err) {
  Team t = team;
  t.k = (int)blockIdx.x;
  member_steps<MODE, K, S, CLUSTER>(d, t, it0, n_steps, 0, zero != 0, 0, Dump(), io, err);
}

template <int MODE, class T>
cudaError_t run(T, const tma::SimDesc &d, const ExactPlan &q, int it0, int n_steps, bool zero,
                const RateIo &io, void *mail, int *err, cudaStream_t s) {
  auto kern = resident_exact<MODE, T::K, T::S, T::CL>;
  static std::atomic<unsigned long long> configured{0};
  cudaError_t e = configure(kern, T::CL, configured);
  if (e != cudaSuccess) return e;
  const Plan &p = q.p;
  if (!p.cluster) {
    e = cudaMemsetAsync(mail, 0, mailbox_bytes(p), s);
    if (e != cudaSuccess) return e;
  }
  const Team team{0, p.tiles_x, p.tiles_z, p.groups, p.n_rec, p.n_inj, q.n_src,
                  MODE == kExact ? q.n_term : p.n_term, static_cast<Word *>(mail)};
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t lc = config(&attr, T::CL, p.ctas(), p.ctas(), p.threads,
                                 MODE == kExact ? q.smem : q.rate_smem, s);
  return cudaLaunchKernelEx(&lc, kern, d, team, it0, n_steps, zero ? 1 : 0, io, err);
}

// Adds the log's entries to the pairs, the last entry first, with each addition's
// rounding error kept in lo (Knuth's TwoSum).
__global__ void __launch_bounds__(128) add_log(int nx, int nz, int pitch, int entries,
                                               const float *log, float2 *a, float2 *b, float2 *c) {
  const int iz = blockIdx.x * blockDim.x + threadIdx.x, ix = blockIdx.y, p = blockIdx.z;
  if (iz >= nz) return;
  float2 *const to = (p == 0 ? a : p == 1 ? b : c) + (size_t)ix * nz + iz;
  const size_t plane = (size_t)nx * pitch;
  const float *from = log + p * plane + (size_t)ix * pitch + iz;
  float2 v = *to;
  for (int k = entries - 1; k >= 0; --k) {
    const float x = from[(size_t)k * 3 * plane];
    const float s = v.x + x, t = s - v.x;
    v = make_float2(s, v.y + ((v.x - (s - t)) + (x - t)));
  }
  *to = v;
}

}  // namespace

cudaError_t steps_keeping_rates(const tma::SimDesc &d, const ExactPlan &p, int it0, int n_steps,
                                bool zero, float2 *rates, void *mail, int *err, cudaStream_t s) {
  if (n_steps <= 0) return cudaSuccess;
  RateIo io;
  io.rates = rates;
  io.stride = p.rate_stride;
  io.first = it0;
  return with_plan(p.p.rows, p.p.stride, p.p.cluster, [&](auto t) {
    return run<kRates>(t, d, p, it0, n_steps, zero, io, mail, err, s);
  });
}

cudaError_t exact_steps(const tma::SimDesc &d, const ExactPlan &p, const ExactSteps &x,
                        void *mail, int *err, cudaStream_t s) {
  if (x.n_steps <= 0) return cudaSuccess;
  RateIo io;
  io.rates = const_cast<float2 *>(x.rates);
  io.stride = p.rate_stride;
  io.first = x.first;
  io.src = x.src;
  io.part = x.part;
  io.log = x.log;
  io.flush = x.flush;
  io.first_log = (x.first + x.flush - 1) / x.flush;
  cudaError_t e = with_plan(p.p.rows, p.p.stride, p.p.cluster, [&](auto t) {
    return run<kExact>(t, d, p, x.first + x.n_steps - 1, x.n_steps, x.zero, io, mail, err, s);
  });
  const int entries = (x.first + x.n_steps - 1) / x.flush - io.first_log + 1;
  if (e != cudaSuccess || entries <= 0) return e;
  const dim3 grid((d.nz + 127) / 128, d.nx, 3);
  add_log<<<grid, 128, 0, s>>>(d.nx, d.nz, d.pitch, entries, x.log, x.sums[0], x.sums[1], x.sums[2]);
  return cudaGetLastError();
}

}  // namespace resident
}  // namespace psv
