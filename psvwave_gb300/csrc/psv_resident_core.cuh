// FP32 time stepping with the grid resident on chip; see psv_resident.hpp.
// Included by psv_resident_f32.cu and psv_resident_exact.cu.
//
// Work split: a team's CTAs form tiles_x x tiles_z tiles. A tile of R rows
// and C column pairs is split over `groups` groups of C threads: thread
// (g, c) owns columns 2c, 2c + 1 of the group's kn consecutive rows (2 <= kn
// <= K). Its points' five wave fields, lm, mu, b and taper factors stay in
// registers for every step. Shared memory holds the tile's fields
// F[R + 4][5][S] (vx vz txx tzz txz; S a compile-time stride) with two halo
// rows and two halo columns on each side: a thread reads z neighbours, and x
// neighbours outside its run, from there as float2.
//
// One time step is a stress and a velocity half-step. In a half-step each
// thread advances its points, writes them to shared memory and sends the
// tile's edge values (two rows, two columns) to the neighbouring CTAs. A
// half-step's x stencils read one field with the forward difference (one row
// before, two after) and one with the backward difference (two before, one
// after): three words per column pair and side; its z stencils read a pair
// of columns of two fields on each side. The CTA's last warps (helpers)
// record the receivers and evaluate the injection terms meanwhile.
//
// Two links carry the edges:
//  * Cluster (teams of up to 16 CTAs, one thread-block cluster): st.async
//    writes a word straight into the neighbour's halo and counts its bytes on
//    the neighbour's mbarrier, which completes a half-step once every thread
//    of the CTA has arrived and every incoming byte has landed. (A halo cell
//    is overwritten only after the neighbour has received all words of the
//    previous half-step from that side, and each is sent by a thread that
//    has finished reading that side's halo.)
//  * Mailbox (any team, cooperative launch; a group is a warp): 128-bit words
//    in global memory carry three values and the step's tag, written and read
//    as single relaxed accesses, so a word whose tag matches carries its
//    values, with no flag, fence or barrier between CTAs; the helpers wait for
//    the tile's words and put them into the halo before the CTA's barrier. A
//    warp sends its rows' edge columns with one store, its lanes reading them
//    back from shared memory: one store a row and side, from one lane, cost
//    0.4 us a half-step at 58 x 62 points. Two parities of every
//    box suffice: a CTA writes step j + 2 only after it has received step
//    j + 1, which its neighbour sent after a barrier that follows its reads of
//    step j.
//
// Points outside the updated region [2, n - 2) carry lm = mu = b = 0 and a
// taper factor of 1: their update adds zero, or NaN where a diverging run has
// infinities around them. That goes no further than the infinities do (such a
// point is next to updated ones along one axis only, and reads and is read along
// it), and leaves as the zero it replaced. (Points excepted from the update
// one by one, by selects or predicated multiplications, cost 1 to 4 % of every
// run.) Arithmetic is written with explicit fused multiply-adds so that every
// instantiation rounds alike.
//
// Every wait is bounded: a thread whose wait runs out raises *err and stops
// waiting for the rest of the launch, which then ends by itself.
#pragma once

#include "psv_resident.hpp"

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <vector>

#include "psv_tma_ptx.cuh"
#include "psv_tma_terms.cuh"

namespace psv {
namespace resident {
namespace cg = cooperative_groups;
namespace {

constexpr int kMaxThreads = 512;
constexpr int kMinK = 3, kMaxK = 5;
constexpr uint32_t kPolls = 1u << 20;  // about a second
constexpr int kCommWords = 4;          // words received by one helper thread
constexpr int kMaxCluster = 16;

// First item of part k when n items are split evenly over parts.
__host__ __device__ __forceinline__ int split(int k, int parts, int n) {
  return (int)(((long long)k * n) / parts);
}
__host__ __device__ __forceinline__ int pairs(int nz) { return (nz + 1) / 2; }
// Shared row strides: column pairs of a tile at most (S - 4) / 2. Mailbox tiles
// have a warp a group, 32 pairs. A cluster keeps its tiles one column wide as
// long as it can (152 columns: 76 pairs, six groups of them in a block), for the
// rows of a group then stay in one CTA: 250 x 150 points 1.72 us a step in 16 x 1
// tiles, 1.90 in 8 x 2; 100 x 80 1.03 and 1.12.
constexpr int kNarrow = 68, kWide = 156;

// Mailbox word: three values and the tag, one 16-byte access. The x stencils
// of a column need three values from a side (both fields' rows), the z
// stencils of a row three as well (two columns of one field, one of the
// other). Incoming words of a tile of R rows and C pairs: from above, from
// below (2 C columns each), from the left and from the right (R rows each).
struct alignas(16) Word {
  float a, b, c;
  uint32_t tag;
};
__host__ __device__ __forceinline__ int words(int R, int C) { return 4 * C + 2 * R; }
constexpr int kBoxWords = 320;
constexpr int kBox = 4 * kBoxWords;  // words of one CTA: [kind 2][parity 2][words]

// (post and push carry no memory clobber: nothing else in the thread depends on
// what they write, and a clobber in the row loop would keep the next row's
// shared loads from being issued ahead.)
__device__ __forceinline__ void post(Word *p, float a, float b, float c, uint32_t tag) {
  const unsigned long long lo = (unsigned long long)__float_as_uint(b) << 32 | __float_as_uint(a);
  const unsigned long long hi = (unsigned long long)tag << 32 | __float_as_uint(c);
  asm volatile(
      "{\n .reg .b128 w;\n mov.b128 w, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], w;\n}" ::"l"(p),
      "l"(lo), "l"(hi));
}
__device__ __forceinline__ Word peek(const Word *p) {
  unsigned long long lo, hi;
  asm volatile("{\n .reg .b128 w;\n ld.relaxed.gpu.global.b128 w, [%2];\n mov.b128 {%0, %1}, w;\n}"
               : "=l"(lo), "=l"(hi)
               : "l"(p)
               : "memory");
  Word w;
  w.a = __uint_as_float((uint32_t)lo);
  w.b = __uint_as_float((uint32_t)(lo >> 32));
  w.c = __uint_as_float((uint32_t)hi);
  w.tag = (uint32_t)(hi >> 32);
  return w;
}

__device__ __forceinline__ uint32_t remote(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Writes a pair of columns into a neighbour's halo; its bytes complete on
// the neighbour's mbarrier.
__device__ __forceinline__ void push(uint32_t addr, float2 v, uint32_t bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::
          "r"(addr),
      "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(bar));
}

__device__ __forceinline__ float2 lds2(const float *p) {
  return *reinterpret_cast<const float2 *>(p);
}
__device__ __forceinline__ void sts2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }

// a1 (p - m) + a2 (l - r): one staggered difference with folded coefficients.
__device__ __forceinline__ float diff(float a1, float p, float m, float a2, float l, float r) {
  return __fmaf_rn(a2, __fsub_rn(l, r), __fmul_rn(a1, __fsub_rn(p, m)));
}
// acc + the same.
__device__ __forceinline__ float diff_add(float acc, float a1, float p, float m, float a2, float l,
                                          float r) {
  return __fmaf_rn(a2, __fsub_rn(l, r), __fmaf_rn(a1, __fsub_rn(p, m), acc));
}

struct Team {
  int k, tiles_x, tiles_z, groups;
  // Most receivers, injection points, source points (kExact) and terms of a tile.
  int n_rec, n_inj, n_src, n_term;
  Word *mail;  // mailbox link: boxes of the team's CTA 0
};

// Rates kept by kRates and read by kExact: per step (from step `first` on) and
// CTA, five quantities of every thread's rows -- e_x, e_z, g_xz, then the
// accelerations a_x, a_z, all times dt. kExact also: the shot's source terms,
// the sums between launches (lm, mu, b: planes of nx * pitch), and the log into
// which they go every `flush` steps: those of step n to entry n / flush -
// first_log, three such planes.
struct RateIo {
  float2 *rates = nullptr;
  size_t stride = 0;
  int first = 0;
  InjPlan src{};
  float *part = nullptr;
  float *log = nullptr;
  int flush = 1, first_log = 0;
};

// What member_steps runs: forward steps, the reference's adjoint steps, forward
// steps that also keep their strain rates and accelerations, and the exact
// adjoint's steps, which read them.
enum Mode { kForward, kAdjoint, kRates, kExact };

// Bulk copy of global memory into shared memory, counted on a barrier (addresses
// and size multiples of 16 bytes).
__device__ __forceinline__ void bulk_load(void *to, const void *from, uint32_t bytes,
                                          uint64_t *bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tma::smem_u32(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(tma::smem_u32(to)),
      "l"(from), "r"(bytes), "r"(tma::smem_u32(bar))
      : "memory");
}
// And back (the writes to shared memory it reads must be ordered before it with
// a proxy fence); wait_stored: the group's shared memory may be reused.
__device__ __forceinline__ void bulk_store(void *to, const void *from, uint32_t bytes) {
  asm volatile(
      "cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n"
      "cp.async.bulk.commit_group;" ::"l"(to),
      "r"(tma::smem_u32(from)), "r"(bytes)
      : "memory");
}
__device__ __forceinline__ void wait_stored() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  return make_float2(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y));
}

// (BATCH: the final state is nobody's output.)
template <int MODE, int K, int S, bool CLUSTER, bool BATCH = false>
__device__ __forceinline__ void member_steps(const tma::SimDesc &d, const Team &tm, int it0,
                                             int n_steps, int parity, bool zero, int store,
                                             const Dump &dump, const RateIo &io, int *err) {
  constexpr bool ADJ = MODE == kAdjoint, EX = MODE == kExact, RATES = MODE == kRates;
  constexpr bool BACK = ADJ || EX;  // time runs backwards
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int RS = 5 * S;  // one row of the five fields
  constexpr int oVX = 0, oVZ = S, oXX = 2 * S, oZZ = 3 * S, oXZ = 4 * S;
  const int nx = d.nx, nz = d.nz, ps = d.pitch;
  const int ti = tm.k / tm.tiles_z, tj = tm.k - ti * tm.tiles_z;
  const int x0 = split(ti, tm.tiles_x, nx), R = split(ti + 1, tm.tiles_x, nx) - x0;
  const int c0 = split(tj, tm.tiles_z, pairs(nz)), C = split(tj + 1, tm.tiles_z, pairs(nz)) - c0;
  const int z0 = 2 * c0;
  const int Rm = (nx + tm.tiles_x - 1) / tm.tiles_x;
  float *const F = reinterpret_cast<float *>(smem_raw);
  const InjPlan &pl = d.plan;
  // kRates, kExact: the step's rates (three for the stresses, two for the
  // velocities) of every thread's rows; kExact: the points' gradient sums of lm,
  // mu and b, and b T (in registers, with the rest, it made K = 5 spill).
  const int CW = CLUSTER ? (tm.groups * ((pairs(nz) + tm.tiles_z - 1) / tm.tiles_z) + 31) & ~31
                         : 32 * tm.groups;
  float2 *const rate_a = reinterpret_cast<float2 *>(F + (Rm + 4) * RS);
  float2 *const rate_b = rate_a + (EX || RATES ? 3 * K * CW : 0);
  float *const G = reinterpret_cast<float *>(rate_b + (EX || RATES ? 2 * K * CW : 0));
  // Injection terms of the tile (weight, next sample, series, field); its
  // injection points: the value each adds this step (vx, vz), its first term and
  // their number (<< 16), and the points' slots by (row, column); receivers.
  double *const term_w = reinterpret_cast<double *>(G + (EX ? 4 * Rm * (S - 4) : 0));
  double *const term_next = term_w + tm.n_term;
  const double **const term_src = reinterpret_cast<const double **>(term_next + tm.n_term);
  float2 *const INJ = reinterpret_cast<float2 *>(term_src + tm.n_term);
  const int n_points = tm.n_inj + (EX ? tm.n_src : 0);  // kExact: then source points
  uint32_t *const inj_terms = reinterpret_cast<uint32_t *>(INJ + n_points);
  int *const term_field = reinterpret_cast<int *>(inj_terms + n_points);
  int *const rec_off = term_field + tm.n_term, *const rec_id = rec_off + tm.n_rec;
  unsigned short *const slot_of = reinterpret_cast<unsigned short *>(rec_off + 2 * tm.n_rec);
  // kExact: bytes, of injection points and of source points.
  unsigned char *const slots_of = reinterpret_cast<unsigned char *>(slot_of);
  __shared__ int s_count[5];
  __shared__ __align__(8) uint64_t s_bar[2];  // of stress and velocity half-steps
  __shared__ __align__(8) uint64_t s_rate[2];  // kExact: of the rates' copies
  const int tid = threadIdx.x, NT = blockDim.x;

  // Compute threads come first, helper warps after them.
  const bool helper = tid >= CW;
  const int g = CLUSTER ? tid / C : tid >> 5, c = CLUSTER ? tid - g * C : tid & 31;
  const bool mine = !helper && g < tm.groups && c < C;
  const bool in_group = !helper && g < tm.groups;
  const int r0 = in_group ? split(g, tm.groups, R) : 0;
  const int kn = in_group ? split(g + 1, tm.groups, R) - r0 : 2;
  auto has = [&](int k) { return k < 2 || k < kn; };
  const bool up = ti > 0, down = ti + 1 < tm.tiles_x;
  const bool left = tj > 0, right = tj + 1 < tm.tiles_z;
  const bool send_up = up && mine && g == 0, send_dn = down && mine && g == tm.groups - 1;
  const bool send_z = mine && ((left && c == 0) || (right && c == C - 1));
  const int z = z0 + 2 * c;
  float *const my = F + (2 + r0) * RS + 2 + 2 * c;  // own first row

  // Shared fields (halo rows and columns at the grid's edges stay zero).
  for (int i = tid; i < (Rm + 4) * RS; i += NT) F[i] = 0.f;
  if (tid < 5) s_count[tid] = 0;
  if (EX && tid == 0)
    for (int k = 0; k < 2; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tma::smem_u32(&s_rate[k])),
                   "r"(1)
                   : "memory");
  if ((CLUSTER || EX) && tid == 0) {
    for (int k = 0; CLUSTER && k < 2; ++k)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tma::smem_u32(&s_bar[k])),
                   "r"(NT)
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto in_tile = [&](int ix, int iz) {
    return ix >= x0 && ix < x0 + R && iz >= z0 && iz < z0 + 2 * C;
  };
  // The tile's injection points and receivers. (kExact: the receivers' terms are
  // the series themselves, and a source's derivative by b drops b.)
  auto point = [&](const InjPlan &p, int i, int q) {
    const int cell = p.terms[i].cell, ix = cell / nz, iz = cell - ix * nz;
    int n = 1;
    while (i + n < p.n && p.terms[i + n].cell == cell) ++n;
    const int first = atomicAdd(&s_count[3], n);
    inj_terms[q] = (uint32_t)first | (uint32_t)n << 16;
    INJ[q] = make_float2(0.f, 0.f);
    int per_field[2] = {0, 0};
    for (int k = 0; k < n; ++k) {
      const InjTerm t = p.terms[i + k];
      const double b = EX ? 1.0 : (double)d.b[(size_t)ix * ps + iz];
      const double *src = (t.kind == 0 ? d.stf : t.field == 0 ? d.a_ux : d.a_uz) +
                          (size_t)t.index * d.nt;
      term_w[first + k] =
          EX && t.kind != 0 ? 1.0 : (t.kind == 0 ? t.coef : 1.0) * d.dt_d * b / t.div;
      term_src[first + k] = src;
      term_next[first + k] = src[it0];
      term_field[first + k] = t.field;
      ++per_field[t.field != 0];
    }
    if (per_field[0] > 1 || per_field[1] > 1) s_count[4] = 1;  // several terms in one item
  };
  auto first_in_tile = [&](const InjPlan &p, int i, int &at) {
    const int cell = p.terms[i].cell, ix = cell / nz, iz = cell - ix * nz;
    at = (ix - x0) * (S - 4) + iz - z0;
    return in_tile(ix, iz) && (i == 0 || p.terms[i - 1].cell != cell);
  };
  for (int i = tid, at; i < pl.n; i += NT)
    if (first_in_tile(pl, i, at)) {
      const int q = atomicAdd(&s_count[0], 1);
      point(pl, i, q);
      if (EX)
        slots_of[2 * at] = (unsigned char)q;
      else
        slot_of[at] = (unsigned short)q;
    }
  if (EX)
    for (int i = tid, at; i < io.src.n; i += NT)
      if (first_in_tile(io.src, i, at)) {
        const int q = atomicAdd(&s_count[2], 1);
        point(io.src, i, tm.n_inj + q);
        slots_of[2 * at + 1] = (unsigned char)q;
      }
  if (!BACK)
    for (int r = tid; r < d.nr; r += NT) {
      const int cell = d.rec_cell[r], ix = cell / ps, iz = cell - ix * ps;
      if (in_tile(ix, iz)) {
        const int q = atomicAdd(&s_count[1], 1);
        rec_off[q] = (ix - x0 + 2) * RS + 2 + iz - z0;
        rec_id[q] = r;
      }
    }

  // Own points: state, medium, taper.
  float2 vx[K], vz[K], xx[K], zz[K], xz[K], lm[K], mu[K], bb[K], tp[K];
  // Bits 2 k + e of a thread's points: with injection terms, with source
  // terms (kExact), in the updated region.
  uint32_t inj_mask = 0, src_mask = 0, inside = 0;
  const fast::Fields in = d.set[parity];
  auto load = [&](const float *src, int x, int zc) {
    if (x < 0 || x >= nx || zc < 0 || zc >= nz) return make_float2(0.f, 0.f);
    float2 v = *reinterpret_cast<const float2 *>(src + (size_t)x * ps + zc);
    if (zc + 1 >= nz) v.y = 0.f;
    return v;
  };
  const float2 zero2 = make_float2(0.f, 0.f);
  auto taper_at = [&](int x, int iz) {
    const int n = min(min(x + 1, nx - x), min(iz + 1, nz - iz));
    return n < d.np ? d.taper_tab[n] : 1.f;
  };
  auto in_region = [&](int x, int iz) {
    return x >= 2 && x < nx - 2 && iz >= 2 && iz < nz - 2;
  };
  // kExact: b T at a pair of points, 0 outside the updated region.
  auto scale = [&](int x, int zc) {
    float2 b = load(d.b, x, zc);
    b.x = in_region(x, zc) ? b.x * taper_at(x, zc) : 0.f;
    b.y = in_region(x, zc + 1) ? b.y * taper_at(x, zc + 1) : 0.f;
    return b;
  };
#pragma unroll
  for (int k = 0; k < K; ++k) {
    vx[k] = vz[k] = xx[k] = zz[k] = xz[k] = lm[k] = mu[k] = bb[k] = zero2;
    tp[k] = make_float2(1.f, 1.f);
    if (k >= kn || !mine) continue;
    const int x = x0 + r0 + k;
    if (!zero) {
      vx[k] = load(in.vx, x, z);
      vz[k] = load(in.vz, x, z);
      xx[k] = load(in.txx, x, z);
      zz[k] = load(in.tzz, x, z);
      xz[k] = load(in.txz, x, z);
    }
    const float2 l = load(d.lm, x, z), m = load(d.mu, x, z), b = load(d.b, x, z);
    if (in_region(x, z)) {
      inside |= 1u << (2 * k);
      lm[k].x = l.x;
      mu[k].x = m.x;
      bb[k].x = b.x;
      tp[k].x = taper_at(x, z);
    }
    if (in_region(x, z + 1)) {
      inside |= 2u << (2 * k);
      lm[k].y = l.y;
      mu[k].y = m.y;
      bb[k].y = b.y;
      tp[k].y = taper_at(x, z + 1);
    }
    if (EX) {
      sts2(G + ((r0 + k) * 4 + 3) * (S - 4) + 2 * c, scale(x, z));
      const size_t gp = (size_t)nx * ps, o = (size_t)x * ps + z;
      for (int p = 0; p < 3; ++p)
        sts2(G + ((r0 + k) * 4 + p) * (S - 4) + 2 * c,
             zero ? zero2 : *reinterpret_cast<const float2 *>(io.part + p * gp + o));
      if (io.src.n && x >= io.src.x0 && x < io.src.x0 + io.src.w)
        for (int e = 0; e < 2; ++e)
          if (z + e >= io.src.z0 && z + e < io.src.z0 + io.src.h && z + e < nz &&
              io.src.map[(x - io.src.x0) * io.src.h + (z + e - io.src.z0)] >= 0)
            src_mask |= 1u << (2 * k + e);
    }
    if (pl.n && x >= pl.x0 && x < pl.x0 + pl.w)
      for (int e = 0; e < 2; ++e)
        if (z + e >= pl.z0 && z + e < pl.z0 + pl.h && z + e < nz &&
            pl.map[(x - pl.x0) * pl.h + (z + e - pl.z0)] >= 0)
          inj_mask |= 1u << (2 * k + e);
  }
  // The first stress half-step's velocities with their halos.
  if (!zero)
    for (int i = tid; i < (R + 4) * (C + 2); i += NT) {
      const int r = i / (C + 2), q = i - r * (C + 2);
      const int o = r * RS + 2 * q;
      const int x = x0 - 2 + r, zc = z0 - 2 + 2 * q;
      float2 a = load(in.vx, x, zc), b = load(in.vz, x, zc);
      if (EX) {
        const float2 w = scale(x, zc);
        a = mul2(w, a);
        b = mul2(w, b);
      }
      sts2(F + oVX + o, a);
      sts2(F + oVZ + o, b);
    }

  // Where this thread's edge values go. Mailbox link: slots of the
  // neighbours' boxes. Cluster link: cells of the neighbours' halos (in
  // bytes, field vx) and their mbarriers.
  const Word *const box = tm.mail + (size_t)tm.k * kBox;
  Word *out_up = nullptr, *out_dn = nullptr, *out_z = nullptr;
  const float *z_from = F;  // the edge columns this lane sends
  uint32_t far_up = 0, far_dn = 0, far_z = 0, bar_up = 0, bar_dn = 0, bar_z = 0, in_bytes = 0;
  if (CLUSTER) {
    const uint32_t base = tma::smem_u32(F), bar = tma::smem_u32(&s_bar[0]);
    const int k_up = tm.k - tm.tiles_z, k_dn = tm.k + tm.tiles_z;
    const int k_z = c == 0 && left ? tm.k - 1 : tm.k + 1;
    if (send_up) {
      const int Ru = x0 - split(ti - 1, tm.tiles_x, nx);
      far_up = remote(base + 4u * ((Ru + 2) * RS + 2 + 2 * c), k_up);
      bar_up = remote(bar, k_up);
    }
    if (send_dn) {
      far_dn = remote(base + 4u * (2 + 2 * c), k_dn);
      bar_dn = remote(bar, k_dn);
    }
    if (send_z) {
      const int Cl = c0 - split(tj - 1, tm.tiles_z, pairs(nz));
      far_z = remote(base + 4u * ((2 + r0) * RS + (k_z < tm.k ? 2 + 2 * Cl : 0)), k_z);
      bar_z = remote(bar, k_z);
    }
    in_bytes = 8u * ((up ? 3 * C : 0) + (down ? 3 * C : 0) + (left ? 2 * R : 0) + (right ? 2 * R : 0));
  } else {
    out_up = tm.mail + (size_t)(tm.k - tm.tiles_z) * kBox + 2 * C + 2 * c;
    out_dn = tm.mail + (size_t)(tm.k + tm.tiles_z) * kBox + 2 * c;
    // Lanes 0 .. 7 send the group's rows to the left, 16 .. 23 to the right
    // (a neighbour's box follows its own column count).
    const int l = tid & 31, k = l & 7;
    if (in_group && k < kn && !(l & 8)) {
      if (l < 16 && left) {
        const int Cl = c0 - split(tj - 1, tm.tiles_z, pairs(nz));
        out_z = tm.mail + (size_t)(tm.k - 1) * kBox + 4 * Cl + R + r0 + k;
      } else if (l >= 16 && right) {
        const int Cr = split(tj + 2, tm.tiles_z, pairs(nz)) - c0 - C;
        out_z = tm.mail + (size_t)(tm.k + 1) * kBox + 4 * Cr + r0 + k;
      }
      z_from = F + (2 + r0 + k) * RS + (l < 16 ? 2 : 2 * C);
    }
  }
  auto box_at = [&](int kind, uint32_t tag) { return (kind * 2 + (int)(tag & 1)) * kBoxWords; };
  // End of a half-step (kind 0 stress, 1 velocity): every thread has written
  // its points, and the halo words of the half-step have arrived. (Two
  // mbarriers: a neighbour may send the next half-step's words while threads
  // of this CTA still finish this one.)
  bool alive = true;
  uint32_t phase = 0;
  auto meet = [&](int kind, bool incoming) {
    if (!CLUSTER) {
      asm volatile("bar.sync 0;" ::: "memory");
      return;
    }
    const uint32_t bar = tma::smem_u32(&s_bar[kind]);
    if (tid == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                   "r"(incoming ? in_bytes : 0u)
                   : "memory");
    else
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
    if (alive && !tma::mbar_wait(&s_bar[kind], phase, kPolls)) {
      alive = false;
      atomicOr(err, 4);
    }
    phase ^= (uint32_t)kind;
  };

  const float c1x = ADJ ? -d.coef[0] : d.coef[0], c2x = ADJ ? -d.coef[1] : d.coef[1];
  const float c1z = ADJ ? -d.coef[2] : d.coef[2], c2z = ADJ ? -d.coef[3] : d.coef[3];
  if (CLUSTER)
    cg::this_cluster().sync();
  else
    __syncthreads();

  // ---- helper warps ----
  if (helper) {
    const int ct = tid - CW, CT = NT - CW;
    const int n_inj = s_count[0], n_rec = s_count[1];
    const int n_items = 2 * (n_inj + (EX ? s_count[2] : 0));
    // Mailbox link: this thread's incoming words, where they lie in a box and
    // where their values go in shared memory after a stress (0) and a velocity
    // (1) half-step.
    int in_at[kCommWords], to_a[kCommWords], to_b[kCommWords], to_c[kCommWords];
    if (!CLUSTER) {
      // Cells are given for the velocity half-step (vx, vz); the stress
      // half-step's fields take their places below.
#pragma unroll
      for (int q = 0; q < kCommWords; ++q) {
        const int i = ct + q * CT;
        in_at[q] = -1;
        to_a[q] = to_b[q] = to_c[q] = 0;
        if (i < 4 * C) {
          const int s = i / (2 * C), o = 2 + i - s * 2 * C;
          if (!(s ? down : up)) continue;
          in_at[q] = i;
          // Above: P row -1, M rows -2, -1; below: P rows R, R + 1, M row R.
          to_a[q] = (s ? R + 2 : 1) * RS + oVX + o;
          to_b[q] = s ? (R + 3) * RS + oVX + o : oVZ + o;
          to_c[q] = (s ? R + 2 : 1) * RS + oVZ + o;
        } else if (i < words(R, C)) {
          const int t = i - 4 * C, s = t / R, o = (2 + t - s * R) * RS + (s ? 2 + 2 * C : 0);
          if (!(s ? right : left)) continue;
          in_at[q] = i;
          // Left: forward-difference field's second column, both of the other;
          // right: both of the forward-difference field, first of the other.
          to_a[q] = o + oVX + (s ? 0 : 1);
          to_b[q] = o + (s ? oVX + 1 : oVZ);
          to_c[q] = o + oVZ + (s ? 0 : 1);
        }
      }
    }
    // The stress half-step sends txz, txx along x and tzz, txz along z where
    // the velocity half-step sends vx, vz.
    auto cell = [&](int q, int to, int kind) {
      if (kind) return to;
      const bool vz_ = to % RS >= oVZ;
      if (in_at[q] < 4 * C) return to + (vz_ ? oXX - oVZ : oXZ - oVX);
      return to + (vz_ ? oXZ - oVZ : oZZ - oVX);
    };
    int st_a[kCommWords], st_b[kCommWords], st_c[kCommWords];
#pragma unroll
    for (int q = 0; q < kCommWords; ++q) {
      st_a[q] = cell(q, to_a[q], 0);
      st_b[q] = cell(q, to_b[q], 0);
      st_c[q] = cell(q, to_c[q], 0);
    }
    // Waits for this thread's words of a half-step and puts them into the halo.
    auto receive = [&](int kind, uint32_t tag) {
      if (CLUSTER) return;
      const Word *const from = box + box_at(kind, tag);
      uint32_t open = 0;  // words still to come
#pragma unroll
      for (int q = 0; q < kCommWords; ++q)
        if (in_at[q] >= 0) open |= 1u << q;
      for (uint32_t i = 0; open && alive; ++i) {
        Word w[kCommWords];
#pragma unroll
        for (int q = 0; q < kCommWords; ++q)
          if (open >> q & 1u) w[q] = peek(from + in_at[q]);
#pragma unroll
        for (int q = 0; q < kCommWords; ++q)
          if ((open >> q & 1u) && w[q].tag == tag) {
            F[kind ? to_a[q] : st_a[q]] = w[q].a;
            F[kind ? to_b[q] : st_b[q]] = w[q].b;
            F[kind ? to_c[q] : st_c[q]] = w[q].c;
            open &= ~(1u << q);
          }
        if (i == kPolls) {
          alive = false;
          atomicOr(err, 4);
        }
      }
    };
    // What the injection points add in this step: item 2 q + f is field f of point
    // q (injection points first, then source points, in their own part of the
    // list). A thread keeps its first item's term in registers, its next sample
    // requested a step ahead; where an item has several terms or a thread
    // several items, the rest come from the table, whose next samples are
    // fetched in the velocity half-step (all of them from the table: 1.36
    // instead of 1.24 us a step on a grid of 68 x 56 points).
    const int n_terms = s_count[3];
    const bool table = s_count[4] != 0 || n_items > CT;
    auto place = [&](int i) {
      return EX && (i >> 1) >= n_inj ? tm.n_inj + (i >> 1) - n_inj : i >> 1;
    };
    // v and the terms of item i after the first `skip`, added one by one in the
    // plan's order, so that an item's sum does not depend on the thread it falls
    // to. (-0 adds to a first term without a trace.)
    auto item_value = [&](int i, float v, int skip) {
      const uint32_t t = inj_terms[place(i)];
      for (uint32_t k = t & 0xFFFFu; k < (t & 0xFFFFu) + (t >> 16); ++k)
        if (term_field[k] == (i & 1) && skip-- <= 0) v += (float)(term_w[k] * term_next[k]);
      return v;
    };
    float *const values = reinterpret_cast<float *>(INJ);
    const double *own_src = nullptr;
    double own_w = 0.0, own_next = 0.0;
    if (ct < n_items) {
      const uint32_t t = inj_terms[place(ct)];
      for (uint32_t k = (t & 0xFFFFu) + (t >> 16); k-- > (t & 0xFFFFu);)
        if (term_field[k] == (ct & 1)) {
          own_src = term_src[k];
          own_w = term_w[k];
          own_next = term_next[k];
        }
    }
    float *const own_value = values + 2 * place(ct) + (ct & 1);
    auto add_terms = [&] {
      if (own_src) {
        float v = (float)(own_w * own_next);
        if (table) v = item_value(ct, v, 1);
        *own_value = v;
      }
      for (int i = ct + CT; i < n_items; i += CT)
        values[2 * place(i) + (i & 1)] = item_value(i, -0.f, 0);
    };
    auto fetch_terms = [&](int it) {
      if (!table) return;
#pragma unroll 4
      for (int k = ct; k < n_terms; k += CT) term_next[k] = term_src[k][it];
    };
    // kExact: the CTA's rates of a step, three per row for the stress half-step
    // and two for the velocity one, each fetched as its buffer becomes free.
    const uint32_t rate_bytes = 8u * K * CW;
    auto fetch = [&](int j, int half) {
      if (!EX || ct != 0 || j >= n_steps) return;
      const float2 *from = io.rates + (size_t)(it0 - j - io.first) * io.stride +
                           (size_t)tm.k * 5 * K * CW + (half ? 3 * K * CW : 0);
      bulk_load(half ? rate_b : rate_a, from, (half ? 2 : 3) * rate_bytes, &s_rate[half]);
    };
    fetch(0, 0);
    fetch(0, 1);
    // kRates: a step's rates go out after its half-steps' barriers, while the
    // next half-step runs (stored by every thread as they were formed, they
    // stood before the edge words: 6.9 us a step at 1100 x 500 against 4.6
    // without rates).
    auto put = [&](int j, int half) {
      if (!RATES || ct != 0) return;
      float2 *to = io.rates + (size_t)(it0 + j - io.first) * io.stride + (size_t)tm.k * 5 * K * CW +
                   (half ? 3 * K * CW : 0);
      bulk_store(to, half ? rate_b : rate_a, (half ? 2 : 3) * rate_bytes);
    };
    auto put_done = [&] {
      if (RATES && ct == 0) wait_stored();
    };
    for (int j = 0; j < n_steps; ++j) {
      const int it = BACK ? it0 - j : it0 + j;
      const uint32_t tag = (uint32_t)(j + 1);
      const bool more = j + 1 < n_steps;
      // Receivers: pre-step velocities.
      if (!BACK)
        for (int i = ct; i < n_rec; i += CT) {
          const size_t o = (size_t)rec_id[i] * d.nt + it;
          d.rec_vx[o] = F[oVX + rec_off[i]];
          d.rec_vz[o] = F[oVZ + rec_off[i]];
        }
      add_terms();
      if (own_src && more) own_next = own_src[BACK ? it - 1 : it + 1];
      receive(0, tag);
      put_done();
      meet(0, true);
      fetch(j + 1, 0);
      put(j, 0);
      if (more) fetch_terms(BACK ? it - 1 : it + 1);
      if (more) receive(1, tag);
      put_done();
      meet(1, more);
      fetch(j + 1, 1);
      put(j, 1);
    }
    put_done();
    if (CLUSTER) cg::this_cluster().sync();
    return;
  }

  // Before a thread's fields leave the launch: NaN of points outside the updated
  // region (b = 0 tells them, which no finite density has) back to zero. Threads
  // without such points pass by.
  auto put_back = [&] {
    if (x0 + r0 >= 2 && x0 + r0 + kn <= nx - 2 && z >= 2 && z + 2 <= nz - 2) return;
    auto clear = [](float2 &v, float2 b) {
      if (isnan(v.x) && b.x == 0.f) v.x = 0.f;
      if (isnan(v.y) && b.y == 0.f) v.y = 0.f;
    };
#pragma unroll
    for (int k = 0; k < K; ++k) {
      clear(vx[k], bb[k]);
      clear(vz[k], bb[k]);
      clear(xx[k], bb[k]);
      clear(zz[k], bb[k]);
      clear(xz[k], bb[k]);
    }
  };
  // kExact: the same for gradient sums of row k.
  auto sums_back = [&](float2 v, int k) {
    const int x = x0 + r0 + k;
    if (isnan(v.x) && !in_region(x, z)) v.x = 0.f;
    if (isnan(v.y) && !in_region(x, z + 1)) v.y = 0.f;
    return v;
  };
  auto save = [&](float *base) {
    const size_t gp = (size_t)nx * ps;
    put_back();
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (k >= kn) continue;
      float *q = base + (size_t)(x0 + r0 + k) * ps + z;
      if (z + 1 < nz) {
        sts2(q, vx[k]);
        sts2(q + gp, vz[k]);
        sts2(q + 2 * gp, xx[k]);
        sts2(q + 3 * gp, zz[k]);
        sts2(q + 4 * gp, xz[k]);
      } else {
        q[0] = vx[k].x;
        q[gp] = vz[k].x;
        q[2 * gp] = xx[k].x;
        q[3 * gp] = zz[k].x;
        q[4 * gp] = xz[k].x;
      }
    }
  };

  // Cluster link: sends the tile's edge columns of row k (the first thread of
  // a group to the left, the last to the right): fields at o0, o1 of a row.
  auto push_z = [&](int k, float2 f0, int o0, float2 f1, int o1, int kind) {
    if (!CLUSTER || !send_z) return;
    const uint32_t bar = bar_z + 8u * kind;
    push(far_z + 4u * (k * RS + o0), f0, bar);
    push(far_z + 4u * (k * RS + o1), f1, bar);
  };
  // Mailbox link: the same for the group's rows at once, read back from shared
  // memory: the z stencils' forward-difference field at of, the other at ob.
  auto post_z = [&](int of, int ob, int at, uint32_t tag) {
    if (CLUSTER || !(left || right)) return;
    __syncwarp();
    if (!out_z) return;
    const float2 f = lds2(z_from + of), b = lds2(z_from + ob);
    if ((tid & 31) < 16)
      post(out_z + at, f.x, f.y, b.x, tag);
    else
      post(out_z + at, f.y, b.x, b.y, tag);
  };
  // Sends the edge rows of a half-step's forward- (p, at op of a row) and
  // backward-difference (m, at om) fields to the neighbours above and below.
  auto publish_x = [&](auto &&p, int op, auto &&m, int om, int kind, int at, uint32_t tag) {
    const uint32_t b8 = 8u * kind;
    if (send_up) {
      if (CLUSTER) {
        push(far_up + 4u * op, p(0), bar_up + b8);
        push(far_up + 4u * (RS + op), p(1), bar_up + b8);
        push(far_up + 4u * om, m(0), bar_up + b8);
      } else {
        post(out_up + at, p(0).x, p(1).x, m(0).x, tag);
        post(out_up + at + 1, p(0).y, p(1).y, m(0).y, tag);
      }
    }
    if (send_dn) {
      float2 pl1 = p(1), ml2 = m(0), ml1 = m(1);  // the last rows
#pragma unroll
      for (int k = 2; k < K; ++k)
        if (has(k)) {
          pl1 = p(k);
          ml2 = m(k - 1);
          ml1 = m(k);
        }
      if (CLUSTER) {
        push(far_dn + 4u * (RS + op), pl1, bar_dn + b8);
        push(far_dn + 4u * om, ml2, bar_dn + b8);
        push(far_dn + 4u * (RS + om), ml1, bar_dn + b8);
      } else {
        post(out_dn + at, pl1.x, ml2.x, ml1.x, tag);
        post(out_dn + at + 1, pl1.y, ml2.y, ml1.y, tag);
      }
    }
  };
  // Row i of a field: own, or one of the rows after the run.
  auto row = [&](auto &&own, int i, float2 a0, float2 a1) {
    if (i < K && has(i)) return own(i);
    return i == kn ? a0 : a1;
  };

  // The fields that a half-step's stencils read, row k of the run. kExact: the
  // scaled adjoint velocities w = b T l_v, and p = C T l_t (px, pz, q in the
  // places of txx, tzz, txz).
  auto f_vx = [&](int k) { return EX ? lds2(my + k * RS + oVX) : vx[k]; };
  auto f_vz = [&](int k) { return EX ? lds2(my + k * RS + oVZ) : vz[k]; };
  auto la_of = [&](int k) {
    return make_float2(__fmaf_rn(-2.f, mu[k].x, lm[k].x), __fmaf_rn(-2.f, mu[k].y, lm[k].y));
  };
  auto f_xx = [&](int k) {
    if (!EX) return xx[k];
    const float2 la = la_of(k), a = mul2(la, zz[k]);
    return make_float2(__fmaf_rn(lm[k].x, xx[k].x, a.x), __fmaf_rn(lm[k].y, xx[k].y, a.y));
  };
  auto f_zz = [&](int k) {
    if (!EX) return zz[k];
    const float2 la = la_of(k), a = mul2(la, xx[k]);
    return make_float2(__fmaf_rn(lm[k].x, zz[k].x, a.x), __fmaf_rn(lm[k].y, zz[k].y, a.y));
  };
  auto f_xz = [&](int k) { return EX ? mul2(mu[k], xz[k]) : xz[k]; };
  // kRates: keeps rate q of row k, 0 outside the updated region.
  auto keep = [&](int q, int k, float a, float b) {
    if (!(inside >> (2 * k) & 1u)) a = 0.f;
    if (!(inside >> (2 * k) & 2u)) b = 0.f;
    rate_a[(q * K + k) * CW + tid] = make_float2(a, b);
  };
  auto kept = [&] {
    if (RATES) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  };
  // kExact: waits for the rates of half-step `half`.
  bool rates_in = true;
  auto rates_ready = [&](int half, int j) {
    if (rates_in && !tma::mbar_wait(&s_rate[half], (uint32_t)(j & 1), kPolls)) {
      rates_in = false;
      atomicOr(err, 4);
    }
  };

  // Steps until the next snapshot step, and until the next saved state.
  const bool snaps = (MODE == kForward || ADJ) && d.accu[0] != nullptr && (ADJ || store);
  int to_snap = ADJ ? it0 % d.si : (d.si - it0 % d.si) % d.si;
  int to_dump = 0;
  for (int j = 0; j < n_steps; ++j) {
    const int it = BACK ? it0 - j : it0 + j;
    const bool snap = snaps && to_snap == 0;
    to_snap = to_snap == 0 ? d.si - 1 : to_snap - 1;
    if (MODE == kForward && dump.base) {
      if (to_dump == 0 && mine) save(dump.base + (size_t)(j / dump.every) * dump.stride);
      to_dump = to_dump == 0 ? dump.every - 1 : to_dump - 1;
    }
    if (snap && mine) {
      const size_t soff = (size_t)(it / d.si) * nx * nz;
      if (!ADJ) put_back();
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (k >= kn) continue;
        const int x = x0 + r0 + k;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int iz = z + e;
          if (iz >= nz) continue;
          const int gi = x * nz + iz;
          const float a = e ? vx[k].y : vx[k].x, b = e ? vz[k].y : vz[k].x,
                      sx = e ? xx[k].y : xx[k].x, sz = e ? zz[k].y : zz[k].x,
                      sh = e ? xz[k].y : xz[k].x;
          if (!ADJ) {
            d.accu[0][soff + gi] = a;
            d.accu[1][soff + gi] = b;
            d.accu[2][soff + gi] = sx;
            d.accu[3][soff + gi] = sz;
            d.accu[4][soff + gi] = sh;
          } else if (x >= d.fx0 && x < d.fx1 && iz >= d.fz0 && iz < d.fz1) {
            const float *as[5] = {d.accu[0] + soff, d.accu[1] + soff, d.accu[2] + soff,
                                  d.accu[3] + soff, d.accu[4] + soff};
            const size_t gp = (size_t)x * ps + iz;
            tma::correlate(d, as, gi, d.lm[gp], d.mu[gp], a, b, sx, sz, sh);
          }
        }
      }
    }
    const uint32_t tag = (uint32_t)(j + 1);
    // ---- stresses ----
    int at = box_at(0, tag);
    if (mine) {
      if (EX) rates_ready(0, j);
      // Rows around the run.
      const float *const end = my + kn * RS;
      const float2 p_b1 = lds2(my + oVX - RS), p_a0 = lds2(end + oVX), p_a1 = lds2(end + oVX + RS);
      const float2 m_b2 = lds2(my + oVZ - 2 * RS), m_b1 = lds2(my + oVZ - RS),
                   m_a0 = lds2(end + oVZ);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (has(k)) {
          const float2 xm1 = k >= 1 ? f_vx(k - 1) : p_b1, x0v = f_vx(k),
                       xp1 = row(f_vx, k + 1, p_a0, p_a1), xp2 = row(f_vx, k + 2, p_a0, p_a1);
          const float2 zm2 = k >= 2 ? f_vz(k - 2) : (k == 1 ? m_b1 : m_b2),
                       zm1 = k >= 1 ? f_vz(k - 1) : m_b1, z0v = f_vz(k),
                       zp1 = row(f_vz, k + 1, m_a0, m_a0);
          const float *pv = my + k * RS;
          const float2 vxl = lds2(pv + oVX - 2), vxr = lds2(pv + oVX + 2);
          const float2 vzl = lds2(pv + oVZ - 2), vzr = lds2(pv + oVZ + 2);
          const float ex0 = diff(c1x, xp1.x, x0v.x, c2x, xm1.x, xp2.x);
          const float ex1 = diff(c1x, xp1.y, x0v.y, c2x, xm1.y, xp2.y);
          const float ez0 = diff(c1z, z0v.x, vzl.y, c2z, vzl.x, z0v.y);
          const float ez1 = diff(c1z, z0v.y, z0v.x, c2z, vzl.y, vzr.x);
          const float g0 = diff_add(diff(c1z, x0v.y, x0v.x, c2z, vxl.y, vxr.x), c1x, z0v.x, zm1.x,
                                    c2x, zm2.x, zp1.x);
          const float g1 = diff_add(diff(c1z, vxr.x, x0v.y, c2z, x0v.x, vxr.y), c1x, z0v.y, zm1.y,
                                    c2x, zm2.y, zp1.y);
          if (RATES) {
            keep(0, k, ex0, ex1);
            keep(1, k, ez0, ez1);
            keep(2, k, g0, g1);
          }
          if (EX) {
            // l_t~ = l_t + A^T w, then y = T l_t~.
            xx[k] = make_float2(__fmul_rn(tp[k].x, __fsub_rn(xx[k].x, ex0)),
                                __fmul_rn(tp[k].y, __fsub_rn(xx[k].y, ex1)));
            zz[k] = make_float2(__fmul_rn(tp[k].x, __fsub_rn(zz[k].x, ez0)),
                                __fmul_rn(tp[k].y, __fsub_rn(zz[k].y, ez1)));
            xz[k] = make_float2(__fmul_rn(tp[k].x, __fsub_rn(xz[k].x, g0)),
                                __fmul_rn(tp[k].y, __fsub_rn(xz[k].y, g1)));
            // Sums of lm, (y_xx + y_zz)(e_x + e_z), and of mu, y_xz g - 2 (y_xx
            // e_z + y_zz e_x): the forward step forms lambda = lm - 2 mu.
            const float2 rx = rate_a[k * CW + tid], rz = rate_a[(K + k) * CW + tid],
                         rg = rate_a[(2 * K + k) * CW + tid];
            float *const sum = G + (r0 + k) * 4 * (S - 4) + 2 * c;
            float2 sl = lds2(sum), sm = lds2(sum + (S - 4));
            sl.x = __fmaf_rn(__fadd_rn(xx[k].x, zz[k].x), __fadd_rn(rx.x, rz.x), sl.x);
            sl.y = __fmaf_rn(__fadd_rn(xx[k].y, zz[k].y), __fadd_rn(rx.y, rz.y), sl.y);
            sm.x += __fmaf_rn(xz[k].x, rg.x,
                              -2.f * __fmaf_rn(xx[k].x, rz.x, __fmul_rn(zz[k].x, rx.x)));
            sm.y += __fmaf_rn(xz[k].y, rg.y,
                              -2.f * __fmaf_rn(xx[k].y, rz.y, __fmul_rn(zz[k].y, rx.y)));
            sts2(sum, sl);
            sts2(sum + (S - 4), sm);
          } else {
            const float la0 = __fmaf_rn(-2.f, mu[k].x, lm[k].x);
            const float la1 = __fmaf_rn(-2.f, mu[k].y, lm[k].y);
            xx[k].x = __fmul_rn(tp[k].x, __fadd_rn(xx[k].x, __fmaf_rn(lm[k].x, ex0, __fmul_rn(la0, ez0))));
            xx[k].y = __fmul_rn(tp[k].y, __fadd_rn(xx[k].y, __fmaf_rn(lm[k].y, ex1, __fmul_rn(la1, ez1))));
            zz[k].x = __fmul_rn(tp[k].x, __fadd_rn(zz[k].x, __fmaf_rn(la0, ex0, __fmul_rn(lm[k].x, ez0))));
            zz[k].y = __fmul_rn(tp[k].y, __fadd_rn(zz[k].y, __fmaf_rn(la1, ex1, __fmul_rn(lm[k].y, ez1))));
            xz[k].x = __fmul_rn(tp[k].x, __fmaf_rn(mu[k].x, g0, xz[k].x));
            xz[k].y = __fmul_rn(tp[k].y, __fmaf_rn(mu[k].y, g1, xz[k].y));
          }
          float *to = my + k * RS;
          const float2 sxx = f_xx(k), szz = f_zz(k), sxz = f_xz(k);
          sts2(to + oXX, sxx);
          sts2(to + oZZ, szz);
          sts2(to + oXZ, sxz);
          push_z(k, szz, oZZ, sxz, oXZ, 0);
        }
      }
      publish_x(f_xz, oXZ, f_xx, oXX, 0, at, tag);
    }
    post_z(oZZ, oXZ, at, tag);
    kept();
    meet(0, true);
    // ---- velocities ----
    at = box_at(1, tag);
    const bool more = j + 1 < n_steps;  // the last step's velocities stay here
    if (mine) {
      if (EX) rates_ready(1, j);
      const float *const end = my + kn * RS;
      const float2 p_b1 = lds2(my + oXZ - RS), p_a0 = lds2(end + oXZ), p_a1 = lds2(end + oXZ + RS);
      const float2 m_b2 = lds2(my + oXX - 2 * RS), m_b1 = lds2(my + oXX - RS),
                   m_a0 = lds2(end + oXX);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (has(k)) {
          const float2 am2 = k >= 2 ? f_xx(k - 2) : (k == 1 ? m_b1 : m_b2),
                       am1 = k >= 1 ? f_xx(k - 1) : m_b1, a0 = f_xx(k),
                       ap1 = row(f_xx, k + 1, m_a0, m_a0);
          const float2 bm1 = k >= 1 ? f_xz(k - 1) : p_b1, b0 = f_xz(k),
                       bp1 = row(f_xz, k + 1, p_a0, p_a1), bp2 = row(f_xz, k + 2, p_a0, p_a1);
          const float *pt = my + k * RS;
          const float2 zl = lds2(pt + oZZ - 2), zr = lds2(pt + oZZ + 2);
          const float2 sl = lds2(pt + oXZ - 2), sr = lds2(pt + oXZ + 2);
          const float2 z0v = f_zz(k);
          const float ax0 = diff_add(diff(c1x, a0.x, am1.x, c2x, am2.x, ap1.x), c1z, b0.x, sl.y,
                                     c2z, sl.x, b0.y);
          const float ax1 = diff_add(diff(c1x, a0.y, am1.y, c2x, am2.y, ap1.y), c1z, b0.y, b0.x,
                                     c2z, sl.y, sr.x);
          const float az0 = diff_add(diff(c1x, bp1.x, b0.x, c2x, bm1.x, bp2.x), c1z, z0v.y, z0v.x,
                                     c2z, zl.y, zr.x);
          const float az1 = diff_add(diff(c1x, bp1.y, b0.y, c2x, bm1.y, bp2.y), c1z, zr.x, z0v.y,
                                     c2z, z0v.x, zr.y);
          if (RATES) {
            keep(3, k, ax0, ax1);
            keep(4, k, az0, az1);
          }
          if (EX) {
            // Sum of b: T l_v . A tau, and the source terms times l_v; then
            // v-bar = T l_v + E^T p.
            const float2 ra = rate_b[k * CW + tid], rb = rate_b[(K + k) * CW + tid];
            const float2 tx = mul2(tp[k], vx[k]), tz = mul2(tp[k], vz[k]);
            float *const sum = G + ((r0 + k) * 4 + 2) * (S - 4) + 2 * c;
            float2 sb = lds2(sum);
            sb.x = __fadd_rn(sb.x, __fmaf_rn(tx.x, ra.x, __fmul_rn(tz.x, rb.x)));
            sb.y = __fadd_rn(sb.y, __fmaf_rn(tx.y, ra.y, __fmul_rn(tz.y, rb.y)));
            if (src_mask >> (2 * k) & 3u) {
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                if (!(src_mask >> (2 * k + e) & 1u)) continue;
                const float2 add = INJ[tm.n_inj + slots_of[2 * ((r0 + k) * (S - 4) + 2 * c + e) + 1]];
                if (e)
                  sb.y = __fadd_rn(sb.y, __fmaf_rn(add.x, vx[k].y, __fmul_rn(add.y, vz[k].y)));
                else
                  sb.x = __fadd_rn(sb.x, __fmaf_rn(add.x, vx[k].x, __fmul_rn(add.y, vz[k].x)));
              }
            }
            sts2(sum, sb);
            vx[k] = make_float2(__fsub_rn(tx.x, ax0), __fsub_rn(tx.y, ax1));
            vz[k] = make_float2(__fsub_rn(tz.x, az0), __fsub_rn(tz.y, az1));
          } else {
            vx[k].x = __fmul_rn(tp[k].x, __fmaf_rn(bb[k].x, ax0, vx[k].x));
            vx[k].y = __fmul_rn(tp[k].y, __fmaf_rn(bb[k].y, ax1, vx[k].y));
            vz[k].x = __fmul_rn(tp[k].x, __fmaf_rn(bb[k].x, az0, vz[k].x));
            vz[k].y = __fmul_rn(tp[k].y, __fmaf_rn(bb[k].y, az1, vz[k].y));
          }
          if (inj_mask >> (2 * k) & 3u) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              if (!(inj_mask >> (2 * k + e) & 1u)) continue;
              const int p = (r0 + k) * (S - 4) + 2 * c + e;
              const float2 add = INJ[EX ? slots_of[2 * p] : slot_of[p]];
              if (e) {
                vx[k].y += add.x;
                vz[k].y += add.y;
              } else {
                vx[k].x += add.x;
                vz[k].x += add.y;
              }
            }
          }
          float *to = my + k * RS;
          float2 wx = vx[k], wz = vz[k];
          if (EX) {
            const float2 w = lds2(G + ((r0 + k) * 4 + 3) * (S - 4) + 2 * c);
            wx = mul2(w, wx);
            wz = mul2(w, wz);
          }
          sts2(to + oVX, wx);
          sts2(to + oVZ, wz);
          if (more) push_z(k, wx, oVX, wz, oVZ, 1);
        }
      }
      if (more) publish_x(f_vx, oVX, f_vz, oVZ, 1, at, tag);
      // kExact: every so often the sums go out and start again.
      if (EX && it % io.flush == 0) {
        float *to = io.log + (size_t)(it / io.flush - io.first_log) * 3 * nx * ps +
                    (size_t)(x0 + r0) * ps + z;
        float *sum = G + r0 * 4 * (S - 4) + 2 * c;
#pragma unroll 1
        for (int k = 0; k < kn; ++k, to += ps, sum += 4 * (S - 4))
          for (int p = 0; p < 3; ++p) {
            sts2(to + (size_t)p * nx * ps, sums_back(lds2(sum + p * (S - 4)), k));
            sts2(sum + p * (S - 4), zero2);
          }
      }
    }
    if (more) post_z(oVX, oVZ, at, tag);
    kept();
    meet(1, more);
  }

  if (mine) {
    const fast::Fields out = d.set[parity ^ (n_steps & 1)];
    if (!EX && !BATCH) put_back();
    float *const dst[5] = {out.vx, out.vz, out.txx, out.tzz, out.txz};
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (k >= kn) continue;
      const size_t o = (size_t)(x0 + r0 + k) * ps + z;
      const float2 v[5] = {vx[k], vz[k], xx[k], zz[k], xz[k]};
#pragma unroll
      for (int f = 0; f < 5; ++f) {
        dst[f][o] = v[f].x;
        if (z + 1 < nz) dst[f][o + 1] = v[f].y;
      }
      if (EX)
        for (int p = 0; p < 3; ++p)
          *reinterpret_cast<float2 *>(io.part + (size_t)p * nx * ps + o) =
              sums_back(lds2(G + ((r0 + k) * 4 + p) * (S - 4) + 2 * c), k);
    }
  }
  if (CLUSTER) cg::this_cluster().sync();
}

struct Device {
  int sms = 0, optin = 0;
};
bool device(Device &q) {
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess &&
         cudaDeviceGetAttribute(&q.sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
         cudaDeviceGetAttribute(&q.optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) ==
             cudaSuccess;
}

// Per-device launch attributes of a kernel, set once: the device's largest
// shared memory, and clusters above the portable size.
template <class Kern>
cudaError_t configure(Kern kern, bool cluster, std::atomic<unsigned long long> &configured) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (configured & bit) return cudaSuccess;
  int optin = 0;
  e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, kern);
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           optin - (int)fa.sharedSizeBytes);
  if (e == cudaSuccess && cluster)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) configured |= bit;
  return e;
}

// A cluster launch, or a cooperative one: either way a team's CTAs are
// resident at once, as CTAs that wait on one another require.
cudaLaunchConfig_t config(cudaLaunchAttribute *attr, bool cluster, int team, int ctas, int threads,
                          size_t smem, cudaStream_t s) {
  if (cluster) {
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = team;
    attr->val.clusterDim.y = 1;
    attr->val.clusterDim.z = 1;
  } else {
    attr->id = cudaLaunchAttributeCooperative;
    attr->val.cooperative = 1;
  }
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(ctas);
  lc.blockDim = dim3(threads);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  lc.attrs = attr;
  lc.numAttrs = 1;
  return lc;
}

// Calls f with the K, S and link of a plan as compile-time values.
template <int K_, int S_, bool CL_>
struct Tag {
  static constexpr int K = K_, S = S_;
  static constexpr bool CL = CL_;
};
template <class F>
cudaError_t with_plan(int rows, int stride, bool cluster, F &&f) {
  if (cluster && stride == kWide) {
    if (rows == 3) return f(Tag<3, kWide, true>{});
    if (rows == 4) return f(Tag<4, kWide, true>{});
    if (rows == 5) return f(Tag<5, kWide, true>{});
  } else if (cluster && stride == kNarrow) {
    if (rows == 3) return f(Tag<3, kNarrow, true>{});
    if (rows == 4) return f(Tag<4, kNarrow, true>{});
    if (rows == 5) return f(Tag<5, kNarrow, true>{});
  } else if (stride == kNarrow) {
    if (rows == 3) return f(Tag<3, kNarrow, false>{});
    if (rows == 4) return f(Tag<4, kNarrow, false>{});
    if (rows == 5) return f(Tag<5, kNarrow, false>{});
  }
  return cudaErrorInvalidValue;
}

}  // namespace
}  // namespace resident
}  // namespace psv
