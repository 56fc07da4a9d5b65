// FP32 forward and adjoint steps resident on chip (psv_resident_core.cuh): one
// simulation, or a batch's members.
#include "psv_resident_core.cuh"

namespace psv {
namespace resident {
namespace {

template <int MODE, int K, int S, bool CLUSTER>
__global__ void __launch_bounds__(kMaxThreads, 1)
    resident_steps(const __grid_constant__ tma::SimDesc d, int tiles_x, int tiles_z, int groups,
                   int n_rec, int n_inj, int n_term, int it0, int n_steps, int parity, int zero, int store,
                   const Dump dump, Word *mail, int *err) {
  const Team t{(int)blockIdx.x, tiles_x, tiles_z, groups, n_rec, n_inj, 0, n_term, mail};
  member_steps<MODE, K, S, CLUSTER>(d, t, it0, n_steps, parity, zero != 0, store, dump, RateIo(),
                                    err);
}

// Mailbox link: the members' teams side by side in one cooperative launch.
// Cluster link: cluster m runs members[m].
template <int K, int S, bool CLUSTER>
__global__ void __launch_bounds__(kMaxThreads, 1)
    resident_steps_batch(const tma::SimDesc *__restrict__ sims, const Member *__restrict__ members,
                         const int *__restrict__ cta_member, int n_steps, int store, Word *mail,
                         int *err) {
  const Member m = members[cta_member[blockIdx.x]];
  const Team t{(int)blockIdx.x - m.first, m.tiles_x, m.tiles_z, m.groups, m.n_rec, m.n_inj,
               0, m.n_term, mail + (size_t)m.first * kBox};
  member_steps<kForward, K, S, CLUSTER, true>(sims[m.sim], t, 0, n_steps, 0, true, store, Dump(),
                                              RateIo(), err);
}

size_t smem_bytes(int Rm, int S, int nr, int n_points, int n_terms) {
  return (size_t)5 * (Rm + 4) * S * sizeof(float) + (size_t)n_points * 12 +
         (size_t)n_terms * 28 + (size_t)nr * 8 +
         (size_t)Rm * (S - 4) * sizeof(unsigned short) + 16;
}

template <int MODE, class T>
cudaError_t run(T, const tma::SimDesc &d, const Plan &p, int it0, int n_steps, int parity, int zero,
                int store, const Dump &dump, void *mail, int *err, cudaStream_t s) {
  auto kern = resident_steps<MODE, T::K, T::S, T::CL>;
  static std::atomic<unsigned long long> configured{0};
  cudaError_t e = configure(kern, T::CL, configured);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t lc = config(&attr, T::CL, p.ctas(), p.ctas(), p.threads, p.smem, s);
  return cudaLaunchKernelEx(&lc, kern, d, p.tiles_x, p.tiles_z, p.groups, p.n_rec, p.n_inj, p.n_term, it0,
                            n_steps, parity, zero, store, dump, static_cast<Word *>(mail), err);
}

// How many clusters of a plan the device runs at once.
int active_clusters(const Plan &p) {
  int n = 0;
  with_plan(p.rows, p.stride, true, [&](auto t) {
    using T = decltype(t);
    auto kern = resident_steps_batch<T::K, T::S, true>;
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = configure(kern, true, configured);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t lc = config(&attr, true, p.ctas(), p.ctas(), p.threads, p.smem, nullptr);
    return cudaOccupancyMaxActiveClusters(&n, kern, &lc);
  });
  cudaGetLastError();
  return n;
}

// The tile a point falls in when n items are split over parts.
int part_of(int i, int parts, int n) {
  int k = (int)(((long long)i * parts) / n);
  while (k + 1 < parts && split(k + 1, parts, n) <= i) ++k;
  while (k > 0 && split(k, parts, n) > i) --k;
  return k;
}

// The most points of a list (cells ix nz + iz) that one tile holds.
int most_per_tile(const Plan &p, int nx, int nz, const std::vector<int> &cells) {
  std::vector<int> count((size_t)p.ctas(), 0);
  int most = 0;
  for (int cell : cells) {
    const int ti = part_of(cell / nz, p.tiles_x, nx);
    const int tj = part_of(cell % nz / 2, p.tiles_z, pairs(nz));
    most = std::max(most, ++count[(size_t)ti * p.tiles_z + tj]);
  }
  return most;
}

// Fills groups, rows, threads and shared memory for a tiling; false when it
// does not fit. per_sm: CTAs that share an SM.
bool fit(Plan &p, const Device &q, const Grid &g, int per_sm) {
  const int max_threads = kMaxThreads / per_sm;
  const int P = pairs(g.nz);
  if (p.tiles_x < 1 || p.tiles_z < 1 || P / p.tiles_z < 2 || g.nx / p.tiles_x < 2) return false;
  const int r_min = g.nx / p.tiles_x, r_max = (g.nx + p.tiles_x - 1) / p.tiles_x;
  const int C = (P + p.tiles_z - 1) / p.tiles_z;
  if (C <= (kNarrow - 4) / 2)
    p.stride = kNarrow;
  else if (p.cluster && C <= (kWide - 4) / 2)
    p.stride = kWide;
  else
    return false;
  // Helper warps: one for a cluster; enough for the tile's words otherwise,
  // one per SM partition on full blocks (their polls then cost each
  // partition's compute warps alike: at 1103 x 497 points 12 + 4 warps take
  // 4.7 us a step, 12 + 2 warps 5.0).
  int help = 1;
  if (!p.cluster) {
    if (words(r_max, C) > kBoxWords) return false;
    help = std::max(2, (words(r_max, C) + 32 * kCommWords - 1) / (32 * kCommWords));
  }
  // Groups of at least two rows each, as many as the threads allow.
  auto groups_for = [&](int helpers) {
    return std::min((max_threads - 32 * helpers) / (p.cluster ? C : 32), r_min / 2);
  };
  p.groups = groups_for(help);
  if (!p.cluster && per_sm == 1 && p.groups > 12 && (r_max + 11) / 12 <= kMaxK) {
    help = std::max(help, 4);
    p.groups = groups_for(help);
  }
  if (p.groups < 1) return false;
  p.rows = std::max(kMinK, (r_max + p.groups - 1) / p.groups);
  if (p.rows > kMaxK) return false;
  p.threads = (p.cluster ? (p.groups * C + 31) / 32 * 32 : 32 * p.groups) + 32 * help;
  p.n_rec = most_per_tile(p, g.nx, g.nz, g.receivers);
  p.n_inj = most_per_tile(p, g.nx, g.nz, g.receivers);  // the adjoint injects at receivers
  for (const auto &cells : g.sources) p.n_inj = std::max(p.n_inj, most_per_tile(p, g.nx, g.nz, cells));
  p.n_term = 2 * p.n_rec;  // of the adjoint
  for (const auto &cells : g.terms) p.n_term = std::max(p.n_term, most_per_tile(p, g.nx, g.nz, cells));
  p.smem = smem_bytes(r_max, p.stride, p.n_rec, p.n_inj, p.n_term);
  // (1 KB of every resident CTA's share is the system's.)
  return (p.smem + 1024 + 64) * per_sm <= (size_t)q.optin + 1024;
}

}  // namespace

Plan plan(const Grid &g) {
  Device q;
  if (g.nx < 4 || g.nz < 4 || !device(q)) return Plan();
  // One cluster, of as many CTAs as it can hold.
  for (int nc = kMaxCluster; nc >= 1; --nc) {
    Plan t = plan_cluster(g, nc);
    if (t.ctas() > 0) return t;
  }
  return plan_mailbox(g, 0, 1);
}

Plan plan_cluster(const Grid &g, int nc) {
  Device q;
  Plan t;
  if (g.nx < 4 || g.nz < 4 || nc < 1 || nc > kMaxCluster || !device(q)) return t;
  t.cluster = true;
  t.tiles_z = (pairs(g.nz) + (kWide - 4) / 2 - 1) / ((kWide - 4) / 2);
  t.tiles_x = nc / t.tiles_z;
  if (nc % t.tiles_z || t.tiles_x < 1 || g.nx / t.tiles_x < 4 || !fit(t, q, g, 1) ||
      active_clusters(t) < 1)
    return Plan();
  return t;
}

Plan plan_mailbox(const Grid &g, int max_ctas, int per_sm) {
  Device q;
  Plan p;
  if (g.nx < 4 || g.nz < 4 || !device(q)) return p;
  if (max_ctas <= 0 || max_ctas > per_sm * q.sms) max_ctas = per_sm * q.sms;
  p.tiles_z = (pairs(g.nz) + (kNarrow - 4) / 2 - 1) / ((kNarrow - 4) / 2);
  p.tiles_x = std::min(max_ctas / p.tiles_z, g.nx / 4);
  return fit(p, q, g, per_sm) ? p : Plan();
}

ExactPlan plan_exact(const Grid &g, int lanes) {
  Device q;
  ExactPlan e;
  if (!device(q) || lanes < 1) return e;
  // Fills what the adjoint adds to a plan; false when it does not fit.
  auto complete = [&](const Plan &p) {
    if (p.ctas() <= 0) return false;
    const int P = pairs(g.nz), C = (P + p.tiles_z - 1) / p.tiles_z;
    const int R = (g.nx + p.tiles_x - 1) / p.tiles_x;
    const size_t cw = p.cluster ? (p.groups * C + 31) / 32 * 32 : 32 * p.groups;
    const size_t rates = 5 * (size_t)p.rows * cw * sizeof(float2);
    e.p = p;
    e.n_src = 0;
    for (const auto &cells : g.sources)
      e.n_src = std::max(e.n_src, most_per_tile(p, g.nx, g.nz, cells));
    // Both the receivers' and the shot's terms.
    e.n_term = 0;
    for (const auto &cells : g.terms) e.n_term = std::max(e.n_term, most_per_tile(p, g.nx, g.nz, cells));
    e.n_term += 2 * p.n_rec;
    if (e.n_term > 0xFFFF) return false;
    e.rate_stride = p.ctas() * rates / sizeof(float2);
    e.rate_smem = p.smem + rates;
    e.smem = e.rate_smem + (size_t)4 * R * (p.stride - 4) * sizeof(float) + (size_t)e.n_src * 12 +
             (size_t)(e.n_term - p.n_term) * 28;
    if (p.n_inj > 256 || e.n_src > 256) return false;  // byte tables
    return e.smem + 64 <= (size_t)q.optin;
  };
  for (int nc = kMaxCluster; nc >= 1; --nc) {
    const Plan p = plan_cluster(g, nc);
    if (p.ctas() <= 0) continue;
    if (complete(p)) return e;
    break;  // fewer CTAs hold less
  }
  if (complete(plan_mailbox(g, q.sms / lanes, 1))) return e;
  return ExactPlan();
}

size_t mailbox_bytes(const Plan &p) {
  return p.cluster ? 0 : (size_t)p.ctas() * kBox * sizeof(Word);
}

cudaError_t steps(const tma::SimDesc &d, const Plan &p, bool adjoint, int it0, int n_steps,
                  int parity, bool zero, bool store, const Dump &dump, void *mail, int *err,
                  cudaStream_t s) {
  if (n_steps <= 0) return cudaSuccess;
  if (p.ctas() <= 0) return cudaErrorInvalidValue;
  if (!p.cluster) {
    cudaError_t e = cudaMemsetAsync(mail, 0, mailbox_bytes(p), s);
    if (e != cudaSuccess) return e;
  }
  const int z = zero ? 1 : 0, st = store ? 1 : 0;
  return with_plan(p.rows, p.stride, p.cluster, [&](auto t) {
    return adjoint ? run<kAdjoint>(t, d, p, it0, n_steps, parity, z, st, dump, mail, err, s)
                   : run<kForward>(t, d, p, it0, n_steps, parity, z, st, dump, mail, err, s);
  });
}

cudaError_t steps_batch(const tma::SimDesc *sims, const Member *members, const int *cta_member,
                        const Launch &l, int n_steps, bool store, void *mail, int *err,
                        cudaStream_t s) {
  if (n_steps <= 0 || l.ctas <= 0) return cudaSuccess;
  if (!l.team) {
    cudaError_t e = cudaMemsetAsync(mail, 0, launch_mailbox_bytes(l), s);
    if (e != cudaSuccess) return e;
  }
  const int st = store ? 1 : 0;
  return with_plan(l.rows, l.stride, l.team > 0, [&](auto t) {
    using T = decltype(t);
    auto kern = resident_steps_batch<T::K, T::S, T::CL>;
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = configure(kern, T::CL, configured);
    if (e != cudaSuccess) return e;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t lc = config(&attr, T::CL, l.team, l.ctas, l.threads, l.smem, s);
    return cudaLaunchKernelEx(&lc, kern, sims, members + l.first_member, cta_member + l.first_cta,
                              n_steps, st, static_cast<Word *>(mail), err);
  });
}

size_t launch_mailbox_bytes(const Launch &l) {
  return l.team ? 0 : (size_t)l.ctas * kBox * sizeof(Word);
}

int resident_slots(int per_sm) {
  Device q;
  return device(q) ? per_sm * q.sms : 0;
}

bool set_tiles_x(Plan &p, const Grid &g, int tiles_x, int per_sm) {
  Device q;
  if (!device(q)) return false;
  Plan t = p;
  t.tiles_x = tiles_x;
  if (!fit(t, q, g, per_sm)) return false;
  p = t;
  return true;
}

Plan plan_smallest(const Grid &g, int per_sm) {
  Device q;
  Plan p;
  if (g.nx < 4 || g.nz < 4 || !device(q)) return p;
  p.tiles_z = (pairs(g.nz) + (kNarrow - 4) / 2 - 1) / ((kNarrow - 4) / 2);
  for (p.tiles_x = 1; p.tiles_x * p.tiles_z <= per_sm * q.sms && p.tiles_x <= g.nx / 4; ++p.tiles_x)
    if (fit(p, q, g, per_sm)) return p;
  return Plan();
}

}  // namespace resident
}  // namespace psv
