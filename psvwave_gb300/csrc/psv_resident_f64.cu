// FP64 time stepping with the grid resident on chip; see
// psv_resident_f64.hpp. Built with -fmad=false.
//
// What bounds it: GB300 issues two FP64 operations per SM and clock, so a step
// costs the FP64 operations of an SM's points, 94 a point, and the work is
// split evenly over all SMs (6.3 us a step at 250 x 150). The two-kernel step
// took two launches a step and the divisions of every point (about 200
// operations): 17.8 us; this one 8.0 us.
//
// Split: tiles as in psv_resident_f32.cu (mailbox link), one, two or four
// points a thread. A thread's points keep their five fields and medium in
// registers; the tile's fields lie in shared memory with two halo rows and
// columns on each side, from which all stencils read. The points that
// neighbours wait for, a ring two wide, go to the first warps, which send
// them to the neighbours' mailboxes as soon as they are computed: 128-bit
// words of a value and the step's tag written and read as single relaxed
// accesses (a word whose tag matches carries its value). Helper warps put
// arriving words into the halo; only the ring's warps wait for them, the
// others compute meanwhile (with all warps meeting at one barrier 9.4 to 10.6
// us a step). Two parities of each box suffice, as there. One more warp
// records the receivers and forms the injection terms.
//
// Every expression keeps the operation order of psv_kernels.cuh. A quotient
// by dx or dz is formed from the divisor's reciprocal y = RN(1 / d) and its
// error z = RN(1 / d - y): q = RN(a y + RN(a z)) is within one unit in the
// last place of a / d, and RN(q + y RN(a - d q)) is then the correctly rounded
// quotient (P. Markstein, IBM J. Res. Dev. 34, 1990; N. Brisebarre, J.-M.
// Muller and S. K. Raina, IEEE Trans. Comput. 53, 2004) as long as nothing
// under- or overflows; other operands take the division itself.
//
// Every wait is bounded: a thread whose wait runs out raises *err and stops
// waiting for the rest of the launch, which then ends by itself.
#include "psv_resident_f64.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <vector>

#include "psv_kernels.cuh"

namespace psv {
namespace resident64 {
namespace {

// Most rows of a thread and the threads that leave it registers for them.
constexpr int kRows[3] = {1, 2, 4};
constexpr int max_threads(int rows) { return rows == 4 ? 384 : 512; }
constexpr int kMaxTile = 64;           // most rows or columns of a tile
constexpr int kCommWords = 12;         // words of one helper thread at most
constexpr uint32_t kPolls = 1u << 20;  // about a second

__host__ __device__ __forceinline__ int split(int k, int parts, int n) {
  return (int)(((long long)k * n) / parts);
}

// Words of a box; a CTA has four: [kind 2][parity 2].
__host__ __device__ __forceinline__ int box_words(int R, int C) { return 6 * (R + C); }

struct alignas(16) Word {
  double v;
  unsigned long long tag;
};
__device__ __forceinline__ void post(Word *p, double v, uint32_t tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = tag;
  asm volatile(
      "{\n .reg .b128 w;\n mov.b128 w, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], w;\n}" ::"l"(p),
      "l"(b), "l"(t));
}
__device__ __forceinline__ Word peek(const Word *p) {
  unsigned long long b, t;
  asm volatile("{\n .reg .b128 w;\n ld.relaxed.gpu.global.b128 w, [%2];\n mov.b128 {%0, %1}, w;\n}"
               : "=l"(b), "=l"(t)
               : "l"(p)
               : "memory");
  Word w;
  w.v = __longlong_as_double((long long)b);
  w.tag = t;
  return w;
}

// A divisor with its reciprocal and the reciprocal's error.
struct Divisor {
  double d, y, z;
};
template <bool Z>
__device__ __forceinline__ double normal_quotient(double a, const Divisor &q) {
  const double q0 = Z ? __fma_rn(a, q.y, __dmul_rn(a, q.z)) : __dmul_rn(a, q.y);
  return __fma_rn(__fma_rn(-q.d, q0, a), q.y, q0);
}
// The rest: infinities, NaN and huge operands by the division, tiny ones
// scaled by 2^600. Scaling the quotient q back rounds it
// once more where it is subnormal, to t with an exact error e = q - t 2^600;
// only where e is half a unit of t can the exact quotient, q + r / d, lie on
// the other side of the tie that was broken.
template <bool Z>
__device__ __noinline__ double other_quotient(double a, double d, double y, double z) {
  if (!(fabs(a) < 1.0)) return a / d;
  const Divisor s = {d, y, z};
  const double b = __dmul_rn(a, 0x1p600), q = normal_quotient<Z>(b, s);
  double t = __dmul_rn(q, 0x1p-600);
  const double e = __fma_rn(t, -0x1p600, q);
  if (fabs(e) == 0x1p-475) {
    const double r = __fma_rn(-d, q, b);
    if (r != 0.0 && (r > 0.0) == (e > 0.0)) t = __dadd_rn(t, copysign(0x1p-1074, e));
  }
  return t;
}
template <bool Z>
__device__ __forceinline__ double quotient(double a, const Divisor &q) {
  const uint32_t e = (uint32_t)(__double2hiint(a) >> 20) & 0x7FFu;
  if (e - 123u < 1800u) return normal_quotient<Z>(a, q);  // 2^-900 <= |a| < 2^900
  if ((__double_as_longlong(a) << 1) == 0) return a;      // +-0
  return other_quotient<Z>(a, q.d, q.y, q.z);
}

struct Args {
  int nx, nz, pitch, np, nt, nr, si;
  int tiles_x, tiles_z, help, n_rec, n_term;
  double dt, sidt;
  Divisor dx, dz;
  double *f[5];
  const double *lm, *la, *mu, *b, *taper;
  double *accu[5];  // this shot's snapshots (null: none)
  double *krho, *klam, *kmu;
  int fx0, fx1, fz0, fz1;
  const int *rec_cell;
  double *rec_vx, *rec_vz;
  InjPlan plan;
  const double *stf, *a_ux, *a_uz;
  int it0, n_steps, zero;
  Word *mail;
  int *err;
};

template <bool ADJ, int K, bool Z>
__global__ void __launch_bounds__(max_threads(K), 1) resident_steps_f64(const Args a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nx = a.nx, nz = a.nz, ps = a.pitch, cta = blockIdx.x;
  const int ti = cta / a.tiles_z, tj = cta - ti * a.tiles_z;
  const int x0 = split(ti, a.tiles_x, nx), R = split(ti + 1, a.tiles_x, nx) - x0;
  const int z0 = split(tj, a.tiles_z, nz), C = split(tj + 1, a.tiles_z, nz) - z0;
  const int Rm = (nx + a.tiles_x - 1) / a.tiles_x, Cm = (nz + a.tiles_z - 1) / a.tiles_z;
  const int box_n = box_words(Rm, Cm), cta_box = 4 * box_n;
  const int S = Cm + 4, FS = (Rm + 4) * S;  // strides of a row and of a field
  double *const F = reinterpret_cast<double *>(smem_raw);
  double *const VX = F, *const VZ = F + FS, *const TXX = F + 2 * FS, *const TZZ = F + 3 * FS,
               *const TXZ = F + 4 * FS;
  // Values of the tile's injection terms this step, the terms, and for every
  // point of the tile its first term's place (low 16 bits) and their number.
  double *const term_v = F + 5 * FS;
  int *const term_id = reinterpret_cast<int *>(term_v + a.n_term);
  int *const rec_off = term_id + a.n_term, *const rec_id = rec_off + a.n_rec;
  uint32_t *const point = reinterpret_cast<uint32_t *>(rec_id + a.n_rec);
  // The tile's points (row << 8 | column), those that neighbours wait for
  // first.
  uint16_t *const order = reinterpret_cast<uint16_t *>(point + Rm * Cm);
  __shared__ int s_count[2];
  // Warps: compute warps, one for receivers and injection terms, receivers of
  // the halo.
  const int tid = threadIdx.x, NT = blockDim.x, CW = NT - 32 * (a.help + 1);
  const bool helper = tid >= CW;
  const bool up = ti > 0, down = ti + 1 < a.tiles_x, left = tj > 0, right = tj + 1 < a.tiles_z;

  for (int i = tid; i < 5 * FS; i += NT) F[i] = 0.0;
  for (int i = tid; i < Rm * Cm; i += NT) point[i] = 0;
  const int sides = 2 * C + 4 * (R - 4), ring = sides + 2 * C;
  for (int i = tid; i < R * C; i += NT) {
    const int r = i / C, c = i - r * C;
    int at;
    if (r < 2)
      at = i;
    else if (r >= R - 2)
      at = sides + (r - (R - 2)) * C + c;
    else if (c < 2 || c >= C - 2)
      at = 2 * C + (r - 2) * 4 + (c < 2 ? c : c - C + 4);
    else
      at = ring + (r - 2) * (C - 4) + c - 2;
    order[at] = (uint16_t)(r << 8 | c);
  }
  if (tid < 2) s_count[tid] = 0;
  __syncthreads();
  auto in_tile = [&](int ix, int iz) {
    return ix >= x0 && ix < x0 + R && iz >= z0 && iz < z0 + C;
  };
  const InjPlan &pl = a.plan;
  for (int i = tid; i < pl.n; i += NT) {
    const int cell = pl.terms[i].cell, ix = cell / nz, iz = cell - ix * nz;
    if (!in_tile(ix, iz) || (i > 0 && pl.terms[i - 1].cell == cell)) continue;
    int n = 1;
    while (i + n < pl.n && pl.terms[i + n].cell == cell) ++n;
    const int at = atomicAdd(&s_count[0], n);
    for (int k = 0; k < n; ++k) term_id[at + k] = i + k;
    point[(ix - x0) * Cm + iz - z0] = (uint32_t)at | (uint32_t)n << 16;
  }
  if (!ADJ)
    for (int r = tid; r < a.nr; r += NT) {
      const int cell = a.rec_cell[r], ix = cell / ps, iz = cell - ix * ps;
      if (in_tile(ix, iz)) {
        const int q = atomicAdd(&s_count[1], 1);
        rec_off[q] = (2 + ix - x0) * S + 2 + iz - z0;
        rec_id[q] = r;
      }
    }

  // Own points.
  double vx[K], vz[K], xx[K], zz[K], xz[K], lm[K], la[K], md[K], bd[K], tp[K];
  uint32_t inside = 0;
  int rc[K], my[K];  // row << 8 | column, place in a field
  const int n_pts = helper ? 0 : R * C;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    vx[k] = vz[k] = xx[k] = zz[k] = xz[k] = lm[k] = la[k] = md[k] = bd[k] = tp[k] = 0.0;
    rc[k] = my[k] = 0;
    if (tid + k * CW >= n_pts) continue;
    rc[k] = order[tid + k * CW];
    const int x = x0 + (rc[k] >> 8), z = z0 + (rc[k] & 255);
    my[k] = (2 + x - x0) * S + 2 + z - z0;
    const size_t o = (size_t)x * ps + z;
    if (!a.zero) {
      vx[k] = a.f[0][o];
      vz[k] = a.f[1][o];
      xx[k] = a.f[2][o];
      zz[k] = a.f[3][o];
      xz[k] = a.f[4][o];
    }
    VX[my[k]] = vx[k];
    VZ[my[k]] = vz[k];
    lm[k] = a.lm[o];
    la[k] = a.la[o];
    md[k] = a.dt * a.mu[o];
    bd[k] = a.b[o] * a.dt;
    tp[k] = a.taper[min(min(min(x + 1, nx - x), min(z + 1, nz - z)), a.np)];
    if (x >= 2 && x < nx - 2 && z >= 2 && z < nz - 2) inside |= 1u << k;
  }
  // The velocities around the tile, for the first half-step.
  if (!a.zero) {
    auto edge = [&](int r, int q) {  // tile row r, column q
      const int x = x0 + r, iz = z0 + q;
      if (x < 0 || x >= nx || iz < 0 || iz >= nz) return;
      VX[(2 + r) * S + 2 + q] = a.f[0][(size_t)x * ps + iz];
      VZ[(2 + r) * S + 2 + q] = a.f[1][(size_t)x * ps + iz];
    };
    for (int i = tid; i < 4 * C; i += NT) edge(i / C < 2 ? i / C - 2 : R + i / C - 2, i % C);
    for (int i = tid; i < 4 * R; i += NT) edge(i / 4, i % 4 < 2 ? i % 4 - 2 : C + i % 4 - 2);
  }
  const Word *const box = a.mail + (size_t)cta * cta_box;
  auto box_at = [&](int kind, uint32_t tag) { return (kind * 2 + (int)(tag & 1)) * box_n; };
  // Words of a box: 3 C from above (P row -1, M rows -2, -1; P the field of
  // the forward x difference, M of the backward one), 3 C from below (P rows
  // R, R + 1, M row R), 3 R from the left (forward z difference: column -1,
  // backward: -2, -1), 3 R from the right (forward: C, C + 1, backward: C).
  __syncthreads();

  // Two barriers a half-step. `tile`: compute warps and the receivers' and
  // terms' warp, once the tile's own values are in. `halo`: the warps that
  // hold points of the ring (they alone read the halo) and the halo's warps,
  // once its words are in. So the inner points' warps go on while words
  // travel. No halo word can be overwritten early: a neighbour sends its next
  // one of a side after it has the words of all points that read that side.
  const int ringers = min(CW, (ring + 31) & ~31);
  const int halo_threads = ringers + 32 * a.help;
  auto tile_sync = [&] { asm volatile("barrier.sync 1, %0;" ::"r"(CW + 32) : "memory"); };
  auto halo_sync = [&] { asm volatile("barrier.sync 2, %0;" ::"r"(halo_threads) : "memory"); };

  if (helper && tid < CW + 32) {
    const int n_term = s_count[0], n_rec = s_count[1];
    for (int j = 0; j < a.n_steps; ++j) {
      const int it = ADJ ? a.it0 - j : a.it0 + j;
      if (!ADJ)
        for (int i = tid - CW; i < n_rec; i += 32) {
          a.rec_vx[(size_t)rec_id[i] * a.nt + it] = VX[rec_off[i]];
          a.rec_vz[(size_t)rec_id[i] * a.nt + it] = VZ[rec_off[i]];
        }
      for (int i = tid - CW; i < n_term; i += 32) {
        const InjTerm t = pl.terms[term_id[i]];
        const int ix = t.cell / nz, iz = t.cell - ix * nz;
        const double b = a.b[(size_t)ix * ps + iz];
        double v;
        if (t.kind == 0) {
          v = (((t.coef * a.stf[(size_t)t.index * a.nt + it]) * a.dt) * b) / t.div;
        } else {
          const double *src = t.field == 0 ? a.a_ux : a.a_uz;
          v = ((a.dt * b) * src[(size_t)t.index * a.nt + it]) / t.div;
        }
        term_v[i] = v;
      }
      tile_sync();
      tile_sync();
    }
    return;
  }
  if (helper) {
    const int ct = tid - CW - 32, CT = NT - CW - 32;
    int at[kCommWords], to[kCommWords];  // slot, cell (field, row, column) after a velocity half-step
#pragma unroll
    for (int q = 0; q < kCommWords; ++q) {
      const int i = ct + q * CT;
      at[q] = -1;
      to[q] = 0;
      if (i < 6 * C) {
        const int s = i / (3 * C), w = (i - s * 3 * C) / C, l = i - (3 * s + w) * C;
        if (!(s ? down : up)) continue;
        const bool p = s ? w < 2 : w == 0;
        const int row = s ? (w == 1 ? R + 3 : R + 2) : (w == 1 ? 0 : 1);
        at[q] = i;
        to[q] = (p ? 0 : FS) + row * S + 2 + l;
      } else if (i < 6 * C + 6 * R) {
        const int t = i - 6 * C, s = t / (3 * R), w = (t - s * 3 * R) / R, r = t - (3 * s + w) * R;
        if (!(s ? right : left)) continue;
        const bool fwd = s ? w < 2 : w == 0;
        const int col = s ? (w == 1 ? C + 3 : C + 2) : (w == 1 ? 0 : 1);
        at[q] = i;
        to[q] = (fwd ? 0 : FS) + (2 + r) * S + col;
      }
    }
    bool alive = true;
    auto receive = [&](int kind, uint32_t tag) {
      const Word *const from = box + box_at(kind, tag);
      uint32_t open = 0;
#pragma unroll
      for (int q = 0; q < kCommWords; ++q)
        if (at[q] >= 0) open |= 1u << q;
      for (uint32_t i = 0; open && alive; ++i) {
#pragma unroll
        for (int q = 0; q < kCommWords; ++q) {
          if (!(open >> q & 1u)) continue;
          const Word w = peek(from + at[q]);
          if ((uint32_t)w.tag != tag) continue;
          // The stress half-step sends txz, txx along x and tzz, txz along z
          // where the velocity half-step sends vx, vz.
          int o = to[q];
          if (!kind) o += at[q] < 6 * C ? (o < FS ? 4 * FS : FS) : 3 * FS;
          F[o] = w.v;
          open &= ~(1u << q);
        }
        if (i == kPolls) {
          alive = false;
          atomicOr(a.err, 4);
        }
      }
    };
    for (int j = 0; j < a.n_steps; ++j) {
      const uint32_t tag = (uint32_t)(j + 1);
      receive(0, tag);
      halo_sync();
      if (j + 1 < a.n_steps) receive(1, tag);
      halo_sync();
    }
    return;
  }

  // Sends this thread's edge points of a half-step: p, m the x stencils'
  // forward- and backward-difference fields, f, b the z stencils'.
  Word *const to_up = a.mail + (size_t)(cta - a.tiles_z) * cta_box + 3 * C;
  Word *const to_dn = a.mail + (size_t)(cta + a.tiles_z) * cta_box;
  const int Cl = left ? z0 - split(tj - 1, a.tiles_z, nz) : 0;
  const int Cr = right ? split(tj + 2, a.tiles_z, nz) - z0 - C : 0;
  Word *const to_l = a.mail + (size_t)(cta - 1) * cta_box + 6 * Cl + 3 * R;
  Word *const to_r = a.mail + (size_t)(cta + 1) * cta_box + 6 * Cr;
  auto publish = [&](int k, double p, double m, double f, double b, int at, uint32_t tag) {
    const int r = rc[k] >> 8, c = rc[k] & 255;
    if (up && r < 2) {
      post(to_up + at + r * C + c, p, tag);
      if (r == 0) post(to_up + at + 2 * C + c, m, tag);
    }
    if (down && r >= R - 2) {
      if (r == R - 1) post(to_dn + at + c, p, tag);
      post(to_dn + at + (r == R - 1 ? 2 : 1) * C + c, m, tag);
    }
    if (left && c < 2) {
      post(to_l + at + c * R + r, f, tag);
      if (c == 0) post(to_l + at + 2 * R + r, b, tag);
    }
    if (right && c >= C - 2) {
      if (c == C - 1) post(to_r + at + r, f, tag);
      post(to_r + at + (c == C - 1 ? 2 : 1) * R + r, b, tag);
    }
  };
  const double c1 = 9.0 / 8.0, c2 = 1.0 / 24.0;
  const bool snaps = a.accu[0] != nullptr;
  int to_snap = ADJ ? a.it0 % a.si : (a.si - a.it0 % a.si) % a.si;
  for (int j = 0; j < a.n_steps; ++j) {
    const int it = ADJ ? a.it0 - j : a.it0 + j;
    const uint32_t tag = (uint32_t)(j + 1);
    if (snaps && to_snap == 0) {
      const size_t soff = (size_t)(it / a.si) * nx * nz;
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (tid + k * CW >= n_pts) continue;
        const int x = x0 + (rc[k] >> 8), z = z0 + (rc[k] & 255);
        const size_t u = (size_t)x * nz + z;
        if (!ADJ) {
          a.accu[0][soff + u] = vx[k];
          a.accu[1][soff + u] = vz[k];
          a.accu[2][soff + u] = xx[k];
          a.accu[3][soff + u] = zz[k];
          a.accu[4][soff + u] = xz[k];
        } else if (x >= a.fx0 && x < a.fx1 && z >= a.fz0 && z < a.fz1) {
          kern::Corr<double>::apply(a.sidt, lm[k], la[k], a.mu[(size_t)x * ps + z],
                                    a.accu[0][soff + u], a.accu[1][soff + u], a.accu[2][soff + u],
                                    a.accu[3][soff + u], a.accu[4][soff + u], vx[k], vz[k], xx[k],
                                    zz[k], xz[k], a.krho + u, a.klam + u, a.kmu + u);
        }
      }
    }
    to_snap = to_snap == 0 ? a.si - 1 : to_snap - 1;
    // ---- stresses ----
    int at = box_at(0, tag);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (tid + k * CW >= n_pts) continue;
      const int i = my[k];
      if (inside >> k & 1u) {
        const double dvx = c1 * (VX[i + S] - vx[k]) + c2 * (VX[i - S] - VX[i + 2 * S]);
        const double dvz = c1 * (vz[k] - VZ[i - 1]) + c2 * (VZ[i - 2] - VZ[i + 1]);
        const double sxx = quotient<Z>(lm[k] * dvx, a.dx) + quotient<Z>(la[k] * dvz, a.dz);
        const double szz = quotient<Z>(la[k] * dvx, a.dx) + quotient<Z>(lm[k] * dvz, a.dz);
        const double sxz =
            quotient<Z>(c1 * (VX[i + 1] - vx[k]) + c2 * (VX[i - 1] - VX[i + 2]), a.dz) +
            quotient<Z>(c1 * (vz[k] - VZ[i - S]) + c2 * (VZ[i - 2 * S] - VZ[i + S]), a.dx);
        if (!ADJ) {
          xx[k] = tp[k] * (xx[k] + a.dt * sxx);
          zz[k] = tp[k] * (zz[k] + a.dt * szz);
          xz[k] = tp[k] * (xz[k] + md[k] * sxz);
        } else {
          xx[k] = tp[k] * (xx[k] - a.dt * sxx);
          zz[k] = tp[k] * (zz[k] - a.dt * szz);
          xz[k] = tp[k] * (xz[k] - md[k] * sxz);
        }
      }
      TXX[i] = xx[k];
      TZZ[i] = zz[k];
      TXZ[i] = xz[k];
      publish(k, xz[k], xx[k], zz[k], xz[k], at, tag);
    }
    tile_sync();
    if (tid < ringers) halo_sync();
    // ---- velocities ----
    at = box_at(1, tag);
    const bool more = j + 1 < a.n_steps;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (tid + k * CW >= n_pts) continue;
      const int i = my[k];
      if (inside >> k & 1u) {
        const double ax =
            quotient<Z>(c1 * (xx[k] - TXX[i - S]) + c2 * (TXX[i - 2 * S] - TXX[i + S]), a.dx) +
            quotient<Z>(c1 * (xz[k] - TXZ[i - 1]) + c2 * (TXZ[i - 2] - TXZ[i + 1]), a.dz);
        const double az =
            quotient<Z>(c1 * (TXZ[i + S] - xz[k]) + c2 * (TXZ[i - S] - TXZ[i + 2 * S]), a.dx) +
            quotient<Z>(c1 * (TZZ[i + 1] - zz[k]) + c2 * (TZZ[i - 1] - TZZ[i + 2]), a.dz);
        if (!ADJ) {
          vx[k] = tp[k] * (vx[k] + bd[k] * ax);
          vz[k] = tp[k] * (vz[k] + bd[k] * az);
        } else {
          vx[k] = tp[k] * (vx[k] - bd[k] * ax);
          vz[k] = tp[k] * (vz[k] - bd[k] * az);
        }
      }
      const uint32_t pt = point[(rc[k] >> 8) * Cm + (rc[k] & 255)];
      for (uint32_t q = 0; q < pt >> 16; ++q) {
        const int t = (int)(pt & 0xFFFFu) + (int)q;
        if (pl.terms[term_id[t]].field == 0)
          vx[k] = vx[k] + term_v[t];
        else
          vz[k] = vz[k] + term_v[t];
      }
      VX[i] = vx[k];
      VZ[i] = vz[k];
      if (more) publish(k, vx[k], vz[k], vx[k], vz[k], at, tag);
    }
    tile_sync();
    if (tid < ringers) halo_sync();
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (tid + k * CW >= n_pts) continue;
    const size_t o = (size_t)(x0 + (rc[k] >> 8)) * ps + z0 + (rc[k] & 255);
    a.f[0][o] = vx[k];
    a.f[1][o] = vz[k];
    a.f[2][o] = xx[k];
    a.f[3][o] = zz[k];
    a.f[4][o] = xz[k];
  }
}

Divisor divisor(double d) {
  Divisor q;
  q.d = d;
  q.y = 1.0 / d;
  const double e = std::fma(-d, q.y, 1.0);
  // Up to 2^-54 (about two divisors of three) RN(a y) is within one unit in
  // the last place by itself.
  q.z = std::fabs(e) <= 0x1p-54 ? 0.0 : e / d;
  return q;
}

size_t smem_bytes(const Plan &p, int R, int C) {
  return (size_t)5 * (R + 4) * (C + 4) * 8 + (size_t)p.n_term * 12 + (size_t)p.n_rec * 8 +
         (size_t)R * C * 6 + 16;
}

}  // namespace

Plan plan(const resident::Grid &g, double dx, double dz) {
  Plan best;
  int dev = 0, sms = 0, optin = 0, coop = 0;
  // quotient()'s range check assumes spacings of ordinary size.
  auto ordinary = [](double d) { return d > 0x1p-60 && d < 0x1p60; };
  if (g.nx < 8 || g.nz < 8 || !ordinary(dx) || !ordinary(dz) || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
          cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop)
    return best;
  // Each quarter of an SM has its own FP64 pipe, which takes a warp's 32 lanes
  // whether they have points or not: fewest warps per quarter times points a
  // thread of the fullest CTA, then the fewest halo words, then the fewest
  // points a thread.
  long best_cost = 0;
  for (int tz = 1; tz <= std::min(sms, g.nz / 4); ++tz) {
    const int C = (g.nz + tz - 1) / tz;
    if (C > kMaxTile) continue;
    for (int tx = 1; tx * tz <= sms && tx <= g.nx / 4; ++tx) {
      const int R = (g.nx + tx - 1) / tx;
      if (R > kMaxTile) continue;
      const int help = 6 * (R + C) > 256 ? 3 : 2;
      if (6 * (R + C) > 32 * help * kCommWords) continue;
      for (int rows : kRows) {
        const int warps = (R * C + 32 * rows - 1) / (32 * rows);
        if (32 * (warps + 1 + help) > max_threads(rows)) continue;
        const long cost = (long)((warps + 3) / 4) * rows * 10000 + R + C;
        if (best.ctas() && cost >= best_cost) continue;
        best_cost = cost;
        best.tiles_x = tx;
        best.tiles_z = tz;
        best.rows = rows;
        best.help = help;
        best.threads = 32 * (warps + 1 + help);
      }
    }
  }
  if (!best.ctas()) return best;
  // The most receivers and terms of a tile.
  auto most = [&](const std::vector<int> &cells) {
    std::vector<int> n((size_t)best.ctas(), 0);
    int m = 0;
    for (int cell : cells) {
      auto part = [](int i, int parts, int total) {
        int k = (int)(((long long)i * parts) / total);
        while (k + 1 < parts && split(k + 1, parts, total) <= i) ++k;
        while (k > 0 && split(k, parts, total) > i) --k;
        return k;
      };
      const int t = part(cell / g.nz, best.tiles_x, g.nx) * best.tiles_z +
                    part(cell % g.nz, best.tiles_z, g.nz);
      m = std::max(m, ++n[t]);
    }
    return m;
  };
  best.n_rec = most(g.receivers);
  best.box = 4 * box_words((g.nx + best.tiles_x - 1) / best.tiles_x,
                           (g.nz + best.tiles_z - 1) / best.tiles_z);
  for (const auto &cells : g.sources) best.n_term = std::max(best.n_term, most(cells));
  best.smem = smem_bytes(best, (g.nx + best.tiles_x - 1) / best.tiles_x,
                         (g.nz + best.tiles_z - 1) / best.tiles_z);
  if (best.smem + 64 > (size_t)optin || best.n_term > 0xFFFF) return Plan();
  return best;
}

size_t mailbox_bytes(const Plan &p) { return (size_t)p.ctas() * p.box * sizeof(Word); }

namespace {
template <bool ADJ, int K, bool Z>
cudaError_t launch(const Args &a, const Plan &p, cudaStream_t s) {
  static std::atomic<unsigned long long> configured{0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(configured & bit)) {
    int optin = 0;
    e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(resident_steps_f64<ADJ, K, Z>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               optin - 64);
    if (e != cudaSuccess) return e;
    configured |= bit;
  }
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(p.ctas());
  lc.blockDim = dim3(p.threads);
  lc.dynamicSmemBytes = p.smem;
  lc.stream = s;
  lc.attrs = &attr;
  lc.numAttrs = 1;
  return cudaLaunchKernelEx(&lc, resident_steps_f64<ADJ, K, Z>, a);
}
template <int K>
cudaError_t run(const Args &a, const Plan &p, bool adjoint, cudaStream_t s) {
  const bool z = a.dx.z != 0 || a.dz.z != 0;
  if (adjoint) return z ? launch<true, K, true>(a, p, s) : launch<true, K, false>(a, p, s);
  return z ? launch<false, K, true>(a, p, s) : launch<false, K, false>(a, p, s);
}
}  // namespace

cudaError_t steps(const SolverArgs &q, const InjPlan &inj, const Plan &p, int shot, bool adjoint,
                  int it0, int n_steps, bool zero, bool store, void *mail, int *err,
                  cudaStream_t s) {
  if (n_steps <= 0) return cudaSuccess;
  if (!p.ctas()) return cudaErrorInvalidValue;
  Args a{};
  a.nx = q.nx;
  a.nz = q.nz;
  a.pitch = q.pitch;
  a.np = q.np;
  a.nt = q.nt;
  a.nr = q.nr;
  a.si = q.si;
  a.tiles_x = p.tiles_x;
  a.tiles_z = p.tiles_z;
  a.help = p.help;
  a.n_rec = p.n_rec;
  a.n_term = p.n_term;
  a.dt = q.dt;
  a.sidt = q.si * q.dt;
  a.dx = divisor(q.dx);
  a.dz = divisor(q.dz);
  void *f[5] = {q.vx, q.vz, q.txx, q.tzz, q.txz};
  const size_t snap = (size_t)shot * q.snapshots * q.nx * q.nz;
  for (int k = 0; k < 5; ++k) {
    a.f[k] = static_cast<double *>(f[k]);
    a.accu[k] = adjoint || store ? static_cast<double *>(q.accu[k]) + snap : nullptr;
  }
  a.lm = static_cast<const double *>(q.lm);
  a.la = static_cast<const double *>(q.la);
  a.mu = static_cast<const double *>(q.mu);
  a.b = static_cast<const double *>(q.b);
  a.taper = static_cast<const double *>(q.taper_tab);
  a.krho = q.k_rho;
  a.klam = q.k_lam;
  a.kmu = q.k_mu;
  a.fx0 = q.fx0;
  a.fx1 = q.fx1;
  a.fz0 = q.fz0;
  a.fz1 = q.fz1;
  a.rec_cell = q.rec_cell;
  a.rec_vx = static_cast<double *>(q.rec_raw);
  a.rec_vz = a.rec_vx ? a.rec_vx + (size_t)q.nr * q.nt : nullptr;
  a.plan = inj;
  a.stf = q.stf;
  a.a_ux = q.a_stf_ux + (size_t)shot * q.nr * q.nt;
  a.a_uz = q.a_stf_uz + (size_t)shot * q.nr * q.nt;
  a.it0 = it0;
  a.n_steps = n_steps;
  a.zero = zero ? 1 : 0;
  a.mail = static_cast<Word *>(mail);
  a.err = err;
  cudaError_t e = cudaMemsetAsync(mail, 0, mailbox_bytes(p), s);
  if (e != cudaSuccess) return e;
  if (p.rows == 1) return run<1>(a, p, adjoint, s);
  if (p.rows == 2) return run<2>(a, p, adjoint, s);
  return run<4>(a, p, adjoint, s);
}

}  // namespace resident64
}  // namespace psv
