// Surrogate network kernels (forward, backward, Adam) and the coarse-to-grid
// parameter map of the Monte Carlo workload; see psv_cnn.hpp.
//
// The convolutions run on the tensor cores as tcgen05 implicit GEMMs with
// BF16 hi + lo operand splits and FP32 accumulators in TMEM: one kernel takes
// an image through every layer (net_images: forward, and for training the
// loss and the input gradients), one sums the weight and bias gradients
// (net_weights, fixed-order partial sums), so every result is deterministic.
#include "psv_cnn.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/psvwave.h"

namespace psv {
namespace cnn {

namespace {

size_t layer_size(int l) { return (size_t)kCout[l] * kCin[l] * 9 + kCout[l]; }


__device__ __forceinline__ void tap(int k, int dil, int &dh, int &dc) {
  dh = (k / 3 - 1) * dil;
  dc = (k % 3 - 1) * dil;
}

// ---- tensor-core convolutions (tcgen05) -------------------------------------
//
// Every convolution is an implicit GEMM in kind::f16 MMAs (BF16 x BF16 ->
// FP32 in TMEM). FP32 operands are split into BF16 parts, hi = bf16(x) and
// lo = bf16(x - hi), which keeps 16 significant bits (about 2^-17 relative;
// products of BF16 values are exact in FP32). Tensors between the
// convolutions are stored as such pairs, one 32-bit word (hi in the upper
// half), split once by their producer, [image][channel][kPW] with kPW = 208
// words a channel (200 positions and zeros, which taps outside the image
// read).
//
// A lies in TMEM: a thread owns a row (lane) and writes its columns straight
// from registers (tcgen05.st, two BF16 a 32-bit column). Through shared memory
// A's stores and the MMAs' reads of it took more of the shared-memory
// bandwidth than the gather itself. B's operands are K-major in shared memory
// without swizzle: 8 x 16-byte core
// matrices, element (r, k) at (r / 8) * kTcSBO + (k / 8) * 128 +
// (r % 8) * 16 + (k % 8) * 2; the descriptor's leading byte offset (between
// K-adjacent core matrices) is 128, its stride byte offset (between 8-row
// groups) kTcSBO.
constexpr int kPW = 208;
constexpr int kTcM = 128, kTcKc = 64, kTcCi = 7;
constexpr int kTcLBO = 128, kTcSBO = (kTcKc / 8) * 128;

__device__ __forceinline__ uint32_t tc_saddr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__host__ __device__ __forceinline__ int tc_off(int r, int k) {
  return (r >> 3) * kTcSBO + (k >> 3) * kTcLBO + (r & 7) * 16 + (k & 7) * 2;
}
// Shared-memory matrix descriptor: start address >> 4 (bits 0-13), leading
// byte offset >> 4 (16-29), stride byte offset >> 4 (32-45), descriptor
// version 1 (bit 46), no swizzle (61-63 = 0).
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(kTcLBO >> 4) << 16) |
         ((uint64_t)(kTcSBO >> 4) << 32) | ((uint64_t)1 << 46);
}
// Instruction descriptor: D FP32 (bits 4-5 = 1), A and B BF16 (7-9 = 1,
// 10-12 = 1), both K-major, N >> 3 (17-22), M >> 4 (24-28).
__device__ __forceinline__ uint32_t tc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(kTcM >> 4) << 24);
}
__device__ __forceinline__ void tc_mma(uint32_t tmem, uint32_t a, uint64_t b, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(tmem),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// One lane of the calling (whole) warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t pred;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(pred));
  return pred != 0;
}
// A thread's columns of A: N registers into TMEM columns ta .. ta + N - 1 of
// its lane.
template <int N>
__device__ __forceinline__ void tc_store(uint32_t ta, const uint32_t *v);
template <>
__device__ __forceinline__ void tc_store<8>(uint32_t ta, const uint32_t *v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(ta), "r"(v[0]),
      "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
      : "memory");
}
template <>
__device__ __forceinline__ void tc_store<4>(uint32_t ta, const uint32_t *v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(ta), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3])
               : "memory");
}
__device__ __forceinline__ void tc_stored() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}
__device__ __forceinline__ void tc_load16(uint32_t ta, uint32_t v[16]) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(ta));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_alloc(uint32_t *holder, int cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   tc_saddr(holder)),
               "r"(cols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t tmem, int cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols)
               : "memory");
}
__device__ __forceinline__ void bar_init(uint64_t *bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_saddr(bar)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_saddr(bar)) : "memory");
}
// Bounded wait on phase `parity` (about a second). *fail is the CTA's flag:
// once a wait has run out no thread waits again, so that the kernel ends.
__device__ __forceinline__ void bar_wait(uint64_t *bar, uint32_t parity, volatile int *fail) {
  const uint32_t addr = tc_saddr(bar);
  for (uint32_t i = 0; i < (1u << 20); ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(done)
        : "r"(addr), "r"(parity), "r"(1000u)
        : "memory");
    if (done || *fail) return;
  }
  *fail = 1;
}
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_saddr(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(tc_saddr(dst)),
      "l"(src), "r"(bytes), "r"(tc_saddr(bar))
      : "memory");
}
__device__ __forceinline__ uint32_t split_word(float x) {
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  const __nv_bfloat16 l = __float2bfloat16_rn(x - __bfloat162float(h));
  return (uint32_t)__bfloat16_as_ushort(h) << 16 | __bfloat16_as_ushort(l);
}
// Packed weights: the B operand of every chunk of seven gathered channels (63
// columns and a zero column), in its shared-memory layout, forward layers 0-3
// then input gradients of layers 3, 2, 1 (rows are the layer's input channels,
// columns its (output channel, tap)).
constexpr int kSteps = 7;
__host__ __device__ constexpr int step_layer(int s) { return s < kLayers ? s : 7 - s; }
__host__ __device__ constexpr int layer_cin(int l) { return l == 0 ? 5 : l == 1 ? 32 : 64; }
__host__ __device__ constexpr int layer_cout(int l) { return l == 0 ? 32 : l == 3 ? 4 : 64; }
// Channels gathered, and columns of D.
__host__ __device__ constexpr int step_k(int s) {
  return s < kLayers ? layer_cin(step_layer(s)) : layer_cout(step_layer(s));
}
__host__ __device__ constexpr int step_n(int s) {
  return s < kLayers ? (s == 3 ? 16 : layer_cout(s)) : layer_cin(step_layer(s));
}
static_assert(layer_cin(0) == kCin[0] && layer_cin(1) == kCin[1] && layer_cin(2) == kCin[2] &&
                  layer_cin(3) == kCin[3] && layer_cout(0) == kCout[0] &&
                  layer_cout(1) == kCout[1] && layer_cout(2) == kCout[2] &&
                  layer_cout(3) == kCout[3],
              "the layers' channels");
__host__ __device__ constexpr int step_chunks(int s) { return (step_k(s) + kTcCi - 1) / kTcCi; }
__host__ __device__ constexpr int step_bytes(int s) { return step_chunks(s) * step_n(s) * kTcKc * 2; }
__host__ __device__ constexpr int step_offset(int s) {
  int o = 0;
  for (int i = 0; i < s; ++i) o += step_bytes(i);
  return o;
}
constexpr int kPackedBytes = step_offset(kSteps);

__global__ void pack_weights(const __nv_bfloat16 *__restrict__ wbf, unsigned char *__restrict__ out,
                             const int4 offs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // element of the packed operands
  if (i >= kPackedBytes / 2) return;
  int s = 0, base = 0;
  while (2 * i >= base + step_bytes(s)) base += step_bytes(s++);
  const int e = i - base / 2, per = step_n(s) * kTcKc;
  const int ch = e / per, r = (e - ch * per) / kTcKc, kk = e - ch * per - r * kTcKc;
  const int l = step_layer(s), cin = layer_cin(l), cout = layer_cout(l), k = ch * 9 * kTcCi + kk;
  const __nv_bfloat16 *w = wbf + (l == 0 ? offs.x : l == 1 ? offs.y : l == 2 ? offs.z : offs.w);
  __nv_bfloat16 v = __float2bfloat16_rn(0.f);
  if (kk < 9 * kTcCi && k < 9 * step_k(s)) {
    if (s < kLayers) {
      if (r < cout) v = w[(size_t)r * cin * 9 + k];
    } else if (r < cin) {
      v = w[((size_t)(k / 9) * cin + r) * 9 + k % 9];
    }
  }
  *reinterpret_cast<__nv_bfloat16 *>(out + base + ch * per * 2 + tc_off(r, kk)) = v;
}

// One image per CTA, all layers: the forward convolutions and the head, and
// for training the loss and the input gradients back to layer 1, with the
// image's tensor in shared memory between layers.
//
// Thread t < 200 owns position t: it gathers the 63 columns of a chunk for
// its row of A (the tap offsets are per-thread addresses, the channel a
// compile-time offset, so a column is one shared load), and later reads its
// TMEM lane, adds the bias and the ReLU (or applies the ReLU mask) and
// writes its column of the next tensor. Warp 7 streams the packed weights (a
// ring of eight chunks, bulk copies) and issues the MMAs: two tiles of 128
// rows, per 16 columns hi * W then lo * W. A has three stages, so that a
// chunk's MMAs run under the next chunks' gathers. (Tiles straddling images,
// gathered from global memory with the weights fetched element by element,
// took 71 us a layer at 512 images.)
constexpr int kImgThreads = 256, kImgRows = 7;  // 7 row warps
struct ImageArgs {
  int batch;
  const float *x;
  const unsigned char *packed;
  const float *bias[kLayers];
  float *misfit, *grad;                        // prediction, normalised units
  // Prediction at states in physical units: x is [B][3][kP], coords the two
  // coordinate channels, misfit m0 + ms m, gradient gs g.
  const float *coords, *gs;
  double m0, ms;
  double *misfit_d;
  const float *m_true, *g_true;                // training
  float w_m, w_g;
  double *loss;
  uint32_t *xq, *act[3], *dq[4];               // split tensors for the weight gradients
  int *err;
};
// ST stages of A (TMEM: D of the two row tiles, 64 columns each, then per
// stage and tile the 32 columns of hi and of lo) and a ring of weights. With
// at most one image per SM, three stages and one CTA per SM; with more
// images, one stage and two CTAs per SM, which overlap each other's gather,
// MMAs and epilogues (256 images, training: 139 us with one CTA per SM). The
// CTAs of an SM never ask for more than its 512 columns, so no allocation
// waits; the shared memory asked for sees to it.
template <int ST>
struct Img {
  static constexpr int RING = ST > 1 ? 8 : 4, AHEAD = RING - 2;
  static constexpr int COLS = ST > 1 ? 512 : 256;
  static constexpr int USED = RING * 64 * kTcKc * 2 + 64 * kPW * 4 + 1024;
  static constexpr int SMEM = ST > 1 ? 120 * 1024 : USED;
  static_assert(USED <= SMEM && 128 + 128 * ST <= COLS, "one image");
};
constexpr int kImgW = 64 * kTcKc * 2, kImgACol = 128;

struct ImageShared {
  uint64_t full[3], done[3], w[8];
  int2 chunk[64];  // offset and bytes of each chunk's weights
  uint32_t tmem;
  volatile int fail;
  float red[256];
  float y[4 * kP];
};

// TMEM columns of A: stage s, row tile m, hi; lo follows 32 columns on.
__device__ __forceinline__ uint32_t a_col(uint32_t tmem, int s, int m) {
  return tmem + kImgACol + 128u * s + 64u * m;
}

template <int REM>
__device__ __forceinline__ void gather_chunk(const uint32_t *const src[9], uint32_t ta) {
  constexpr int COLS = 9 * REM, GROUPS = (COLS + 15) / 16;
  uint32_t w[16 * GROUPS];
#pragma unroll
  for (int k = 0; k < 16 * GROUPS; ++k) w[k] = k < COLS ? src[k % 9][kPW * (k / 9)] : 0u;
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    uint32_t h[8], l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      h[e] = __byte_perm(w[16 * g + 2 * e], w[16 * g + 2 * e + 1], 0x7632);
      l[e] = __byte_perm(w[16 * g + 2 * e], w[16 * g + 2 * e + 1], 0x5410);
    }
    tc_store<8>(ta + 8 * g, h);
    tc_store<8>(ta + 32 + 8 * g, l);
  }
}

// The row warps' part of step S: gather every chunk, then wait for the
// products. n: chunks so far.
template <int S, int ST>
__device__ __forceinline__ void gather_step(ImageShared &sh, const uint32_t *act, uint32_t tmem,
                                            int t, int &n) {
  constexpr bool BWD = S >= kLayers;
  constexpr int DIL = kDil[step_layer(S)], K = step_k(S);
  constexpr int CHUNKS = step_chunks(S), REM = K - (CHUNKS - 1) * kTcCi;
  const int h = t / kW, c = t - h * kW;
  const uint32_t *src[9];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    int dh, dc;
    tap(q, DIL, dh, dc);
    const int hh = BWD ? h - dh : h + dh, cc = BWD ? c - dc : c + dc;
    const bool ok = t < kP && hh >= 0 && hh < kH && cc >= 0 && cc < kW;
    src[q] = act + (ok ? hh * kW + cc : kP);
  }
  const uint32_t lanes = (uint32_t)(32 * ((t >> 5) & 3)) << 16;
  for (int ch = 0; ch < CHUNKS; ++ch, ++n) {
    const int s = n % ST;
    if (n >= ST)
      bar_wait(&sh.done[s], (uint32_t)(n / ST - 1) & 1u, &sh.fail);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    const uint32_t ta = a_col(tmem, s, t >> 7) + lanes;
    if (REM != kTcCi && ch == CHUNKS - 1)
      gather_chunk<REM>(src, ta);
    else
      gather_chunk<kTcCi>(src, ta);
#pragma unroll
    for (int q = 0; q < 9; ++q) src[q] += kPW * kTcCi;
    tc_stored();
    __syncwarp();
    if ((t & 31) == 0) bar_arrive(&sh.full[s]);
  }
  // The step's last commit covers all its products.
  bar_wait(&sh.done[(n - 1) % ST], (uint32_t)((n - 1) / ST) & 1u, &sh.fail);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Warp 7: the weights of chunk q of the kernel's chunk list (one lane).
template <int ST>
__device__ __forceinline__ void load_weights(ImageShared &sh, const unsigned char *packed,
                                             unsigned char *ring, int q, int total) {
  if (q >= total) return;
  const int2 c = sh.chunk[q];
  bulk_load(ring + (q % Img<ST>::RING) * kImgW, packed + c.x, (uint32_t)c.y, &sh.w[q % Img<ST>::RING]);
}

// The MMAs of step S (the whole warp 7; one lane issues).
template <int S, int ST>
__device__ __forceinline__ void mma_step(ImageShared &sh, const unsigned char *packed,
                                         unsigned char *ring, uint32_t tmem, int total, int &n) {
  constexpr int CHUNKS = step_chunks(S), REM = step_k(S) - (CHUNKS - 1) * kTcCi;
  const uint32_t idesc = tc_idesc(step_n(S));
  for (int ch = 0; ch < CHUNKS; ++ch, ++n) {
    const int s = n % ST, slot = n % Img<ST>::RING;
    // The slot of the chunk loaded now held chunk n - 2: its products must be
    // done. (With one stage they are: chunk n - 1 was gathered after them. A
    // wait here could miss that phase, the barrier having gone two on.)
    if (ST > 1 && n >= 2)
      bar_wait(&sh.done[(n - 2) % ST], (uint32_t)((n - 2) / ST) & 1u, &sh.fail);
    __syncwarp();
    if (elect_one()) load_weights<ST>(sh, packed, ring, n + Img<ST>::AHEAD, total);
    __syncwarp();
    bar_wait(&sh.w[slot], (uint32_t)(n / Img<ST>::RING) & 1u, &sh.fail);
    bar_wait(&sh.full[s], (uint32_t)(n / ST) & 1u, &sh.fail);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    const uint32_t a = a_col(tmem, s, 0);
    const uint64_t bd = tc_desc(tc_saddr(ring + slot * kImgW));
    const int steps = ch == CHUNKS - 1 ? (9 * REM + 15) / 16 : 4;
    if (elect_one()) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (k >= steps) break;
        const uint64_t b = bd + (uint64_t)(k * 2 * kTcLBO >> 4);
        // hi of both tiles, then lo: successive products do not share D.
        const uint32_t acc = (ch > 0 || k > 0) ? 1u : 0u, ak = a + 8u * k;
        tc_mma(tmem, ak, b, idesc, acc);
        tc_mma(tmem + 64u, ak + 64u, b, idesc, acc);
        tc_mma(tmem, ak + 32u, b, idesc, 1u);
        tc_mma(tmem + 64u, ak + 96u, b, idesc, 1u);
      }
      tc_commit(tc_saddr(&sh.done[s]));
    }
    __syncwarp();
  }
}

// Barrier of the row warps.
__device__ __forceinline__ void rows_sync() {
  asm volatile("barrier.sync 1, %0;" ::"n"(32 * kImgRows) : "memory");
}

// Epilogue of a hidden step: thread t's outputs into the image's tensor in
// shared memory (and, for training, global memory). Forward: bias and ReLU;
// backward: the ReLU mask of the layer's input activation.
template <int S, bool TRAIN>
__device__ __forceinline__ void finish_step(const ImageArgs &g, uint32_t *act, uint32_t tmem, int t,
                                            int image) {
  constexpr bool BWD = S >= kLayers;
  constexpr int L = step_layer(S), N = BWD ? kCin[L] : kCout[L];
  const uint32_t ta = tmem + ((uint32_t)(32 * ((t >> 5) & 3)) << 16) + 64u * (t >> 7);
  uint32_t *out = !TRAIN ? nullptr : BWD ? g.dq[L - 1] : g.act[L < 3 ? L : 0];
  const uint32_t *mask = BWD ? g.act[L - 1 < 3 ? (L > 0 ? L - 1 : 0) : 0] : nullptr;
  const size_t at = (size_t)image * N * kPW + t;
#pragma unroll
  for (int c0 = 0; c0 < N; c0 += 16) {
    uint32_t v[16], m[16];
    if (BWD && t < kP)
#pragma unroll
      for (int j = 0; j < 16; ++j) m[j] = mask[at + (size_t)(c0 + j) * kPW];
    tc_load16(ta + c0, v);
    if (t >= kP) continue;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int co = c0 + j;
      float r = __uint_as_float(v[j]);
      if (BWD)
        r = (int)m[j] > 0 ? r : 0.f;
      else
        r = fmaxf(r + __ldg(g.bias[L] + co), 0.f);
      const uint32_t w = split_word(r);
      act[co * kPW + t] = w;
      if (TRAIN) out[at + (size_t)co * kPW] = w;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  rows_sync();
}

// Fixed-order sum over 256 values, the row warps' 224 and zeros.
__device__ float rows_sum(float v, float *red, int t) {
  red[t] = v;
  if (t < 32) red[32 * kImgRows + t] = 0.f;
  rows_sync();
  for (int s = 128; s > 0; s >>= 1) {
    if (t < s) red[t] += red[t + s];
    rows_sync();
  }
  const float r = red[0];
  rows_sync();
  return r;
}

template <bool TRAIN, int ST>
__global__ void __launch_bounds__(kImgThreads, ST > 1 ? 1 : 2) net_images(const ImageArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ ImageShared sh;
  unsigned char *const base = smem + (1024 - (tc_saddr(smem) & 1023)) % 1024;
  unsigned char *const ring = base;
  uint32_t *const act = reinterpret_cast<uint32_t *>(ring + Img<ST>::RING * kImgW);
  const int t = threadIdx.x, image = blockIdx.x;
  constexpr int STEPS = TRAIN ? kSteps : kLayers;
  int total = 0;
#pragma unroll
  for (int s = 0; s < STEPS; ++s) total += step_chunks(s);
  if (t == 0) {
    sh.fail = 0;
    for (int i = 0; i < ST; ++i) {
      bar_init(&sh.full[i], kImgRows);
      bar_init(&sh.done[i], 1);
    }
    for (int i = 0; i < Img<ST>::RING; ++i) bar_init(&sh.w[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (t >= 32 * kImgRows) tc_alloc(&sh.tmem, Img<ST>::COLS);
  if (t < total) {
    int s = 0, c = t, o = 0;
    while (c >= step_chunks(s)) {
      c -= step_chunks(s);
      o += step_bytes(s++);
    }
    const int bytes = step_n(s) * kTcKc * 2;
    sh.chunk[t] = make_int2(o + c * bytes, bytes);
  }
  // The image's features, split; zeros past each channel.
  for (int i = t; i < 64 * kPW; i += kImgThreads) {
    const int c = i / kPW, p = i - c * kPW;
    uint32_t w = 0;
    if (c < layer_cin(0) && p < kP) {
      const float *from = !TRAIN && g.coords
                              ? (c < 3 ? g.x + ((size_t)image * 3 + c) * kP : g.coords + (c - 3) * kP)
                              : g.x + ((size_t)image * layer_cin(0) + c) * kP;
      w = split_word(__ldg(from + p));
      if (TRAIN) g.xq[((size_t)image * layer_cin(0) + c) * kPW + p] = w;
    }
    act[i] = w;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = sh.tmem;
  int n = 0;
  if (t >= 32 * kImgRows) {
    if (elect_one())
      for (int q = 0; q < Img<ST>::AHEAD; ++q) load_weights<ST>(sh, g.packed, ring, q, total);
    __syncwarp();
    mma_step<0, ST>(sh, g.packed, ring, tmem, total, n);
    mma_step<1, ST>(sh, g.packed, ring, tmem, total, n);
    mma_step<2, ST>(sh, g.packed, ring, tmem, total, n);
    mma_step<3, ST>(sh, g.packed, ring, tmem, total, n);
    if (TRAIN) {
      mma_step<4, ST>(sh, g.packed, ring, tmem, total, n);
      mma_step<5, ST>(sh, g.packed, ring, tmem, total, n);
      mma_step<6, ST>(sh, g.packed, ring, tmem, total, n);
    }
  } else {
    gather_step<0, ST>(sh, act, tmem, t, n);
    finish_step<0, TRAIN>(g, act, tmem, t, image);
    gather_step<1, ST>(sh, act, tmem, t, n);
    finish_step<1, TRAIN>(g, act, tmem, t, image);
    gather_step<2, ST>(sh, act, tmem, t, n);
    finish_step<2, TRAIN>(g, act, tmem, t, image);
    gather_step<3, ST>(sh, act, tmem, t, n);
    // Head: gradient map = channels 0 .. 2, misfit = sum of channel 3.
    uint32_t v[16];
    tc_load16(tmem + ((uint32_t)(32 * ((t >> 5) & 3)) << 16) + 64u * (t >> 7), v);
    float y[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c] = __uint_as_float(v[c]) + __ldg(g.bias[3] + c);
    const float m = rows_sum(t < kP ? y[3] : 0.f, sh.red, t);
    if (!TRAIN) {
      if (t < kP)
        for (int c = 0; c < 3; ++c)
          g.grad[((size_t)image * 3 + c) * kP + t] =
              g.coords ? __fmul_rn(__ldg(g.gs + c * kP + t), y[c]) : y[c];
      if (t == 0) {
        if (g.coords)
          g.misfit_d[image] = __dadd_rn(g.m0, __dmul_rn(g.ms, (double)m));
        else
          g.misfit[image] = m;
      }
    } else {
      // Loss = w_m mean_b (m - m*)^2 + w_g mean_{b,c,p} (g - g*)^2 and its
      // gradient with respect to the head's inputs. (The squares are summed
      // in the order of 256 threads striding over [3][200].)
      const float dm = m - g.m_true[image], ng = (float)g.batch * 3 * kP;
      if (t < kP) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float diff = y[c] - g.g_true[((size_t)image * 3 + c) * kP + t];
          sh.y[c * kP + t] = diff * diff;
          y[c] = 2.f * g.w_g * diff / ng;
        }
        y[3] = 2.f * g.w_m * dm / (float)g.batch;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t w = split_word(y[c]);
          act[c * kPW + t] = w;
          g.dq[3][((size_t)image * 4 + c) * kPW + t] = w;
        }
      }
      rows_sync();
      // Threads 224 .. 255 of that order are summed by the first warp.
      auto strided = [&](int k) {
        float s = 0.f;
        for (int i = k; i < 3 * kP; i += 256) s += sh.y[i];
        return s;
      };
      sh.red[t] = strided(t);
      if (t < 32) sh.red[32 * kImgRows + t] = strided(32 * kImgRows + t);
      rows_sync();
      for (int s = 128; s > 0; s >>= 1) {
        if (t < s) sh.red[t] += sh.red[t + s];
        rows_sync();
      }
      if (t == 0)
        g.loss[image] = (double)g.w_m * dm * dm / g.batch + (double)g.w_g * sh.red[0] / ng;
      rows_sync();
      gather_step<4, ST>(sh, act, tmem, t, n);
      finish_step<4, TRAIN>(g, act, tmem, t, image);
      gather_step<5, ST>(sh, act, tmem, t, n);
      finish_step<5, TRAIN>(g, act, tmem, t, image);
      gather_step<6, ST>(sh, act, tmem, t, n);
      finish_step<6, TRAIN>(g, act, tmem, t, image);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (t == 0 && sh.fail) {
    atomicOr(g.err, 1);
    // Bounded: give products in flight more time before the TMEM is freed.
    sh.fail = 0;
    bar_wait(&sh.done[0], 0u, &sh.fail);
  }
  __syncthreads();
  if (t >= 32 * kImgRows) tc_dealloc(tmem, Img<ST>::COLS);
}

// ---- tensor-core weight gradients --------------------------------------------
//
// dW[co][k] = sum_pos dy[pos][co] X[pos][k] and db[co] = sum_pos dy[pos][co]
// as a GEMM whose reduction runs over the positions of the batch's images:
// D[k][co] (M = 128 rows of k = ci * 9 + tap per CTA, the bias as row
// k = cin * 9 with X = 1). Both operands are split pairs; hi.hi + hi.lo +
// lo.hi per 16 positions carry the products to about 2^-16 relative.
// blockIdx.x is a tile of rows of one layer, blockIdx.y one of kChunks ranges
// of images, whose partial sums sum_partials adds in order (deterministic).
// Per image the tile's channels (with a border of zeros, so that a tap is an
// offset) and dy go to shared memory; the next image's words are loaded into
// registers meanwhile. Thread t builds row t % 128 of A: a position is a
// compile-time offset, one shared load; positions run in chunks of 64 (the
// last 16) through two stages, so that a chunk's MMAs run under the next
// chunk's gather. Gathering every element from global memory with two-byte
// shared stores took 780 us a layer at 512 images.
constexpr int kWgThreads = 256;
// (Row and channel pitches that spread a warp's 32 rows, three or four
// channels of nine taps 1, 2 or 4 apart, over the banks.)
constexpr int kPadW = kW + 9, kPadH = kH + 8, kPadP = kPadW * kPadH + 1, kDyP = 209;
constexpr int kWgStage = 2 * 64 * kTcKc * 2;  // B hi, lo
// TMEM: D (64 columns), then per stage 32 columns of A's hi and of its lo.
constexpr int kWgCols = 256, kWgACol = 64;
constexpr int kWgSmem = 2 * kWgStage + 16 * kPadP * 4 + 64 * kDyP * 4 + 1024;
static_assert(kWgSmem > 114 * 1024, "one CTA per SM: its TMEM columns are then free");
constexpr int kWgTiles[kLayers] = {1, 3, 5, 5};  // ceil((cin * 9 + 1) / 128)

struct WeightArgs {
  int batch;
  const uint32_t *x[kLayers], *dy[kLayers];
  float *partial;  // [kChunks][num_params]
  size_t len;      // num_params
  size_t off[kLayers];
  int *err;
};
struct WeightShared {
  uint64_t done[2];
  uint32_t tmem;
  volatile int fail;
};

// Groups G0 .. G0 + NG - 1 (eight positions each, 64 Q + 8 g + e) of chunk Q
// of a row, as hi and lo pairs.
template <int Q, int G0, int NG, bool PAD>
__device__ __forceinline__ void weight_row(const uint32_t *src, uint32_t h[4 * NG],
                                           uint32_t l[4 * NG]) {
  uint32_t w[8 * NG];
#pragma unroll
  for (int i = 0; i < 8 * NG; ++i) {
    const int p = 64 * Q + 8 * G0 + i;
    w[i] = p < kP ? src[PAD ? (p / kW) * kPadW + p % kW : p] : 0u;
  }
#pragma unroll
  for (int i = 0; i < 4 * NG; ++i) {
    h[i] = __byte_perm(w[2 * i], w[2 * i + 1], 0x7632);
    l[i] = __byte_perm(w[2 * i], w[2 * i + 1], 0x5410);
  }
}
// The same into B's row at hi, lo.
template <int Q, int G0, int NG>
__device__ __forceinline__ void weight_row_b(const uint32_t *src, unsigned char *hi,
                                             unsigned char *lo) {
  uint32_t h[4 * NG], l[4 * NG];
  weight_row<Q, G0, NG, false>(src, h, l);
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    *reinterpret_cast<uint4 *>(hi + (G0 + g) * kTcLBO) =
        make_uint4(h[4 * g], h[4 * g + 1], h[4 * g + 2], h[4 * g + 3]);
    *reinterpret_cast<uint4 *>(lo + (G0 + g) * kTcLBO) =
        make_uint4(l[4 * g], l[4 * g + 1], l[4 * g + 2], l[4 * g + 3]);
  }
}

template <int L>
__device__ void weight_tile(const WeightArgs &g, WeightShared &sh, unsigned char *base, int mtile) {
  constexpr int CIN = kCin[L], COUT = kCout[L], DIL = kDil[L], K = CIN * 9;
  constexpr int NPAD = COUT < 16 ? 16 : COUT, NCH = CIN < 16 ? CIN : 16;
  const int t = threadIdx.x;
  const int b0 = (int)((long long)g.batch * blockIdx.y / gridDim.y);
  const int b1 = (int)((long long)g.batch * (blockIdx.y + 1) / gridDim.y);
  const int m0 = mtile * kTcM, ci0 = m0 / 9 < CIN - NCH ? m0 / 9 : CIN - NCH;
  float *const out = g.partial + (size_t)blockIdx.y * g.len + g.off[L];
  uint32_t *const xs = reinterpret_cast<uint32_t *>(base + 2 * kWgStage);
  uint32_t *const ds = xs + 16 * kPadP;
  for (int i = t; i < 16 * kPadP; i += kWgThreads) xs[i] = 0;
  for (int i = t; i < 64 * kDyP; i += kWgThreads) ds[i] = 0;
  // Row t % 128 of A, the half of its groups given by t / 128; row t % 64 of
  // B, a quarter of its groups.
  const int k = m0 + (t & 127), part = t >> 7;
  const int ci = k / 9, tp = k - 9 * ci;
  int dh, dc;
  tap(tp, DIL, dh, dc);
  const uint32_t *const src =
      xs + (k < K ? (ci - ci0) * kPadP + (4 + dh) * kPadW + 4 + dc : 0);
  const int co = t & 63, quarter = t >> 6;
  const uint32_t *const dsrc = ds + co * kDyP;
  const uint32_t lanes = (uint32_t)(32 * ((t >> 5) & 3)) << 16;
  const int brow = (co >> 3) * kTcSBO + (co & 7) * 16;
  const uint32_t idesc = tc_idesc(NPAD), tmem = sh.tmem;
  // Thread t < 200 carries position t of every channel.
  uint32_t px[NCH], pd[COUT];
  auto fetch = [&](int b) {
    if (t >= kP) return;
    const uint32_t *x = g.x[L] + ((size_t)b * CIN + ci0) * kPW + t;
    const uint32_t *d = g.dy[L] + (size_t)b * COUT * kPW + t;
#pragma unroll
    for (int c = 0; c < NCH; ++c) px[c] = __ldg(x + c * kPW);
#pragma unroll
    for (int c = 0; c < COUT; ++c) pd[c] = __ldg(d + c * kPW);
  };
  uint32_t *const xo = xs + (t / kW + 4) * kPadW + t % kW + 4;
  if (b0 < b1) fetch(b0);
  int n = 0;
  auto chunk = [&](auto build, int steps, bool first) {
    const int s = n & 1;
    if (n >= 2) bar_wait(&sh.done[s], (uint32_t)((n >> 1) - 1) & 1u, &sh.fail);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncwarp();
    unsigned char *const bh = base + s * kWgStage, *const bl = bh + 64 * kTcKc * 2;
    const uint32_t a = tmem + kWgACol + 64u * s;
    build(a + lanes, bh + brow, bl + brow);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_stored();
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (t < 32 && elect_one()) {
      const uint64_t dh_ = tc_desc(tc_saddr(bh)), dl_ = tc_desc(tc_saddr(bl));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= steps) break;
        const uint64_t ko = (uint64_t)(q * 2 * kTcLBO >> 4);
        const uint32_t ah = a + 8u * q, al = ah + 32u;
        tc_mma(tmem, ah, dh_ + ko, idesc, (first && q == 0) ? 0u : 1u);
        tc_mma(tmem, ah, dl_ + ko, idesc, 1u);
        tc_mma(tmem, al, dh_ + ko, idesc, 1u);
      }
      tc_commit(tc_saddr(&sh.done[s]));
    }
    ++n;
  };
  __syncthreads();
  for (int b = b0; b < b1; ++b) {
    if (t < kP) {
#pragma unroll
      for (int c = 0; c < NCH; ++c) xo[c * kPadP] = px[c];
#pragma unroll
      for (int c = 0; c < COUT; ++c) ds[c * kDyP + t] = pd[c];
    }
    __syncthreads();
    if (b + 1 < b1) fetch(b + 1);
    const bool first = b == b0;
    // NA groups of the row for each half, NB of B's row for each quarter. Rows
    // past the weights hold ones (the bias row, at valid positions) or zeros.
#define PSV_CHUNK(Q, NA, NB)                                                              \
  chunk(                                                                                  \
      [&](uint32_t ta, unsigned char *bh, unsigned char *bl) {                            \
        uint32_t h[4 * NA], l[4 * NA];                                                    \
        if (part == 0)                                                                    \
          weight_row<Q, 0, NA, true>(src, h, l);                                          \
        else                                                                              \
          weight_row<Q, NA, NA, true>(src, h, l);                                         \
        if (k >= K) {                                                                     \
          _Pragma("unroll") for (int i = 0; i < 4 * NA; ++i) {                            \
            const int p = 64 * Q + 8 * NA * part + 2 * i;                                 \
            h[i] = k == K && p < kP ? 0x3F803F80u : 0u;                                   \
            l[i] = 0u;                                                                    \
          }                                                                               \
        }                                                                                 \
        __syncwarp();                                                                     \
        if (NA == 4) {                                                                    \
          tc_store<8>(ta + 16 * part, h);                                                 \
          tc_store<8>(ta + 16 * part + 8, h + 8 * (NA / 4));                              \
          tc_store<8>(ta + 32 + 16 * part, l);                                            \
          tc_store<8>(ta + 32 + 16 * part + 8, l + 8 * (NA / 4));                         \
        } else {                                                                          \
          tc_store<4>(ta + 4 * part, h);                                                  \
          tc_store<4>(ta + 32 + 4 * part, l);                                             \
        }                                                                                 \
        if (co < NPAD) {                                                                  \
          if (quarter == 0) weight_row_b<Q, 0, NB>(dsrc, bh, bl);                         \
          if (quarter == 1) weight_row_b<Q, NB, NB>(dsrc, bh, bl);                        \
          if (quarter == 2 && Q < 3) weight_row_b<Q, 2 * NB, NB>(dsrc, bh, bl);           \
          if (quarter == 3 && Q < 3) weight_row_b<Q, 3 * NB, NB>(dsrc, bh, bl);           \
        }                                                                                 \
        __syncwarp();                                                                     \
      },                                                                                  \
      Q < 3 ? 4 : 1, first && Q == 0)
    PSV_CHUNK(0, 4, 2);
    PSV_CHUNK(1, 4, 2);
    PSV_CHUNK(2, 4, 2);
    PSV_CHUNK(3, 1, 1);
#undef PSV_CHUNK
    // (The chunks' barriers have ordered every read of xs and ds before the
    // next image's words.)
  }
  if (n) bar_wait(&sh.done[(n - 1) & 1], (uint32_t)((n - 1) >> 1) & 1u, &sh.fail);
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  // Row 32 w + lane of the accumulator is k; warps 4 - 7 have none.
  if (t < kTcM) {
#pragma unroll
    for (int c0 = 0; c0 < NPAD; c0 += 16) {
      uint32_t v[16];
      tc_load16(tmem + ((uint32_t)(32 * (t >> 5)) << 16) + c0, v);
      if (k <= K)
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c0 + j < COUT)
            out[k < K ? (size_t)(c0 + j) * K + k : (size_t)COUT * K + c0 + j] =
                n ? __uint_as_float(v[j]) : 0.f;
    }
  }
}

__global__ void __launch_bounds__(kWgThreads, 1) net_weights(const WeightArgs g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ WeightShared sh;
  unsigned char *const base = smem + (1024 - (tc_saddr(smem) & 1023)) % 1024;
  const int t = threadIdx.x;
  if (t < 32) tc_alloc(&sh.tmem, kWgCols);
  if (t == 0) {
    sh.fail = 0;
    for (int i = 0; i < 2; ++i) bar_init(&sh.done[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const int x = blockIdx.x;
  if (x < 5)
    weight_tile<2>(g, sh, base, x);
  else if (x < 10)
    weight_tile<3>(g, sh, base, x - 5);
  else if (x < 13)
    weight_tile<1>(g, sh, base, x - 10);
  else
    weight_tile<0>(g, sh, base, x - 13);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (t == 0 && sh.fail) {
    atomicOr(g.err, 1);
    sh.fail = 0;
    bar_wait(&sh.done[0], 0u, &sh.fail);
  }
  __syncthreads();
  if (t < 32) tc_dealloc(sh.tmem, kWgCols);
}
constexpr int kWgTileCount = 14;
static_assert(kWgTiles[0] + kWgTiles[1] + kWgTiles[2] + kWgTiles[3] == kWgTileCount, "row tiles");

__global__ void sum_partials(size_t len, const float *__restrict__ partial,
                             float *__restrict__ out) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= len) return;
  float s = 0.f;
#pragma unroll 8
  for (int c = 0; c < kChunks; ++c) s += partial[(size_t)c * len + i];
  out[i] = s;
}

__global__ void adam_step(size_t n, float *__restrict__ p, const float *__restrict__ g,
                          float *__restrict__ m, float *__restrict__ v,
                          __nv_bfloat16 *__restrict__ wbf, float lr, float b1, float b2, float eps,
                          float bc1, float bc2) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  p[i] = pi;
  wbf[i] = __float2bfloat16_rn(pi);
}

__global__ void to_bf16(size_t n, const float *__restrict__ p, __nv_bfloat16 *__restrict__ wbf) {
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) wbf[i] = __float2bfloat16_rn(p[i]);
}

unsigned blocks(size_t n, int t = 256) { return static_cast<unsigned>((n + t - 1) / t); }

void check(cudaError_t e, const char *what) { cuda_check(e, what); }

}  // namespace

size_t weight_offset(int layer) {
  size_t off = 0;
  for (int l = 0; l < layer; ++l) off += layer_size(l);
  return off;
}

size_t bias_offset(int layer) { return weight_offset(layer) + (size_t)kCout[layer] * kCin[layer] * 9; }

size_t num_params() { return weight_offset(kLayers); }

Net::Net(int device, int max_batch) : device_(device), max_batch_(max_batch) {
  if (max_batch <= 0) throw Error(PSV_ERR_INVALID_ARGUMENT, "max_batch must be positive");
  DeviceGuard guard(device_);
  check(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "cudaStreamCreate");
  const size_t n = num_params();
  params_.allocate(n * sizeof(float), false);
  wbf_.allocate(n * sizeof(__nv_bfloat16), false);
  grads_.allocate(n * sizeof(float), false);
  adam_m_.allocate(n * sizeof(float), false);
  adam_v_.allocate(n * sizeof(float), false);
  packed_.allocate(kPackedBytes, false);
  partials_.allocate(kChunks * n * sizeof(float), false);
  const size_t image = (size_t)max_batch * kPW * sizeof(uint32_t);
  xq_.allocate(image * kCin[0], false);
  for (int l = 0; l < 3; ++l) act_[l].allocate(image * kCout[l], false);
  for (int l = 0; l < kLayers; ++l) dq_[l].allocate(image * kCout[l], false);
  // Per-image losses, then the error flag: one copy back a call.
  result_.allocate((size_t)(max_batch + 1) * sizeof(double), false);
  result_h_.resize(max_batch + 1);
  for (auto f : {net_images<true, 3>, net_images<false, 3>})
    check(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, Img<3>::SMEM),
          "smem");
  for (auto f : {net_images<true, 1>, net_images<false, 1>})
    check(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, Img<1>::SMEM),
          "smem");
  check(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, device_), "SMs");
  check(cudaFuncSetAttribute(net_weights, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem),
        "smem");
  // (The buffers were cleared on the legacy stream, for which stream_ does not
  // wait.)
  check(cudaStreamSynchronize(cudaStreamLegacy), "network");
}

int *Net::err() { return reinterpret_cast<int *>(result_.as<double>() + max_batch_); }

// Waits for the stream and returns the sum of the per-image losses. Raises
// when a bounded wait of a kernel ran out (the flag is cleared for the next
// call).
double Net::collect(int batch) {
  // (The losses lie before the flag; with none to read, only the flag comes.)
  const int first = max_batch_ - batch;
  check(cudaMemcpyAsync(result_h_.data() + first, result_.as<double>() + first,
                        (size_t)(batch + 1) * sizeof(double), cudaMemcpyDeviceToHost, stream_),
        "result");
  check(cudaStreamSynchronize(stream_), "network");
  int flag = 0;
  std::memcpy(&flag, &result_h_[max_batch_], sizeof(int));
  if (flag) {
    check(cudaMemsetAsync(err(), 0, sizeof(int), stream_), "err");
    throw Error(PSV_ERR_CUDA, "a tensor-core convolution timed out waiting for its products");
  }
  double loss = 0;
  for (int i = 0; i < batch; ++i) loss += result_h_[first + i];
  return loss;
}

Net::~Net() {
  if (stream_) {
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device_);
    cudaStreamSynchronize(stream_);
    cudaStreamDestroy(stream_);
    cudaSetDevice(prev);
  }
}

void Net::check_batch(int batch) const {
  if (batch <= 0 || batch > max_batch_)
    throw Error(PSV_ERR_INVALID_ARGUMENT, "batch must be in [1, max_batch]");
}

void Net::refresh_bf16() {
  const size_t n = num_params();
  to_bf16<<<blocks(n), 256, 0, stream_>>>(n, params_.as<float>(), wbf_.as<__nv_bfloat16>());
  check(cudaGetLastError(), "to_bf16");
  repack();
}

void Net::repack() {
  const int4 offs = make_int4((int)weight_offset(0), (int)weight_offset(1), (int)weight_offset(2),
                              (int)weight_offset(3));
  pack_weights<<<blocks(kPackedBytes / 2), 256, 0, stream_>>>(
      wbf_.as<__nv_bfloat16>(), packed_.as<unsigned char>(), offs);
  check(cudaGetLastError(), "pack weights");
}

void Net::set_params(const float *host) {
  DeviceGuard guard(device_);
  const size_t n = num_params();
  check(cudaMemcpyAsync(params_.get(), host, n * sizeof(float), cudaMemcpyHostToDevice, stream_),
        "set params");
  check(cudaMemsetAsync(adam_m_.get(), 0, n * sizeof(float), stream_), "adam");
  check(cudaMemsetAsync(adam_v_.get(), 0, n * sizeof(float), stream_), "adam");
  step_ = 0;
  refresh_bf16();
  check(cudaStreamSynchronize(stream_), "set params");
}

void Net::get_params(float *host) {
  DeviceGuard guard(device_);
  check(cudaMemcpyAsync(host, params_.get(), num_params() * sizeof(float), cudaMemcpyDeviceToHost,
                        stream_),
        "get params");
  check(cudaStreamSynchronize(stream_), "get params");
}

// The arguments both kinds of call share.
static ImageArgs image_args(int batch, const float *x, const unsigned char *packed,
                            const float *params, int *err) {
  ImageArgs g{};
  g.batch = batch;
  g.x = x;
  g.packed = packed;
  for (int l = 0; l < kLayers; ++l) g.bias[l] = params + bias_offset(l);
  g.err = err;
  return g;
}

template <bool TRAIN>
static void launch_images(const ImageArgs &g, bool two_per_sm, cudaStream_t s) {
  if (two_per_sm)
    net_images<TRAIN, 1><<<g.batch, kImgThreads, Img<1>::SMEM, s>>>(g);
  else
    net_images<TRAIN, 3><<<g.batch, kImgThreads, Img<3>::SMEM, s>>>(g);
}

// Forward, loss and parameter gradient (into grads_), without waiting.
void Net::gradient(int batch, const float *x, const float *m_true, const float *g_true,
                   float w_misfit, float w_grad) {
  ImageArgs g = image_args(batch, x, packed_.as<unsigned char>(), params_.as<float>(), err());
  g.m_true = m_true;
  g.g_true = g_true;
  g.w_m = w_misfit;
  g.w_g = w_grad;
  g.loss = result_.as<double>() + (max_batch_ - batch);
  g.xq = xq_.as<uint32_t>();
  for (int l = 0; l < 3; ++l) g.act[l] = act_[l].as<uint32_t>();
  for (int l = 0; l < kLayers; ++l) g.dq[l] = dq_[l].as<uint32_t>();
  launch_images<true>(g, batch > sms_, stream_);
  check(cudaGetLastError(), "network forward and input gradients");
  WeightArgs w{};
  w.batch = batch;
  for (int l = 0; l < kLayers; ++l) {
    w.x[l] = l == 0 ? xq_.as<uint32_t>() : act_[l - 1].as<uint32_t>();
    w.dy[l] = dq_[l].as<uint32_t>();
    w.off[l] = weight_offset(l);
  }
  w.partial = partials_.as<float>();
  w.len = num_params();
  w.err = err();
  net_weights<<<dim3(kWgTileCount, kChunks), kWgThreads, kWgSmem, stream_>>>(w);
  check(cudaGetLastError(), "weight gradients");
  sum_partials<<<blocks(w.len), 256, 0, stream_>>>(w.len, partials_.as<float>(),
                                                   grads_.as<float>());
  check(cudaGetLastError(), "sum of partials");
}

void Net::predict(int batch, const float *x, float *misfit, float *grad) {
  check_batch(batch);
  DeviceGuard guard(device_);
  ImageArgs g = image_args(batch, x, packed_.as<unsigned char>(), params_.as<float>(), err());
  g.misfit = misfit;
  g.grad = grad;
  launch_images<false>(g, batch > sms_, stream_);
  check(cudaGetLastError(), "network forward");
  collect(0);
}

void Net::predict_states(int batch, const float *z, const float *coords, double m0, double ms,
                         const float *gs, double *misfit, float *grad) {
  check_batch(batch);
  DeviceGuard guard(device_);
  ImageArgs g = image_args(batch, z, packed_.as<unsigned char>(), params_.as<float>(), err());
  g.coords = coords;
  g.m0 = m0;
  g.ms = ms;
  g.gs = gs;
  g.misfit_d = misfit;
  g.grad = grad;
  launch_images<false>(g, batch > sms_, stream_);
  check(cudaGetLastError(), "network forward");
  collect(0);
}

double Net::loss_grad(int batch, const float *x, const float *m_true, const float *g_true,
                      float w_misfit, float w_grad, float *dparams_host) {
  check_batch(batch);
  DeviceGuard guard(device_);
  gradient(batch, x, m_true, g_true, w_misfit, w_grad);
  if (dparams_host)
    check(cudaMemcpyAsync(dparams_host, grads_.get(), num_params() * sizeof(float),
                          cudaMemcpyDeviceToHost, stream_),
          "grads");
  return collect(batch);
}

double Net::train_step(int batch, const float *x, const float *m_true, const float *g_true,
                       float w_misfit, float w_grad, const Adam &opt) {
  check_batch(batch);
  DeviceGuard guard(device_);
  gradient(batch, x, m_true, g_true, w_misfit, w_grad);
  // (As before the update: a time-out leaves the parameters alone.)
  const double loss = collect(batch);
  ++step_;
  const float bc1 = 1.f - std::pow(opt.beta1, (float)step_);
  const float bc2 = 1.f - std::pow(opt.beta2, (float)step_);
  const size_t n = num_params();
  adam_step<<<blocks(n), 256, 0, stream_>>>(n, params_.as<float>(), grads_.as<float>(),
                                            adam_m_.as<float>(), adam_v_.as<float>(),
                                            wbf_.as<__nv_bfloat16>(), opt.lr, opt.beta1, opt.beta2,
                                            opt.eps, bc1, bc2);
  check(cudaGetLastError(), "adam");
  repack();
  return loss;
}

}  // namespace cnn

// ---- coarse-to-grid map ---------------------------------------------------

namespace {

__global__ void coarse_to_fields(int batch, int nx, int nz, int ncx, int ncz,
                                 const int *__restrict__ x0, const int *__restrict__ x1,
                                 const double *__restrict__ wx, const int *__restrict__ z0,
                                 const int *__restrict__ z1, const double *__restrict__ wz,
                                 const double *__restrict__ mean, const double *__restrict__ sigma,
                                 const float *__restrict__ z, double *__restrict__ fields) {
  const size_t n = (size_t)batch * 3 * nx * nz;
  const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int iz = (int)(i % nz);
  const int ix = (int)((i / nz) % nx);
  const int c = (int)((i / ((size_t)nx * nz)) % 3);
  const int b = (int)(i / ((size_t)3 * nx * nz));
  const size_t cb = (size_t)c * ncx * ncz;
  const float *zb = z + (size_t)b * 3 * ncx * ncz + cb;
  auto theta = [&](int a, int d) {
    const size_t k = (size_t)a * ncz + d;
    return mean[cb + k] + sigma[cb + k] * (double)zb[k];
  };
  const double fx = wx[ix], fz = wz[iz];
  const int a0 = x0[ix], a1 = x1[ix], d0 = z0[iz], d1 = z1[iz];
  fields[i] = (1.0 - fx) * ((1.0 - fz) * theta(a0, d0) + fz * theta(a0, d1)) +
              fx * ((1.0 - fz) * theta(a1, d0) + fz * theta(a1, d1));
}

__global__ void fields_to_coarse(int nx, int nz, int ncx, int ncz, const int *__restrict__ x0,
                                 const int *__restrict__ x1, const double *__restrict__ wx,
                                 const int *__restrict__ z0, const int *__restrict__ z1,
                                 const double *__restrict__ wz, const int *__restrict__ xs,
                                 const int *__restrict__ xe, const int *__restrict__ zs,
                                 const int *__restrict__ ze, const double *__restrict__ sigma,
                                 double scale, const double *__restrict__ g,
                                 float *__restrict__ gz) {
  const int bc = blockIdx.x;  // b * 3 + c
  const int c = bc % 3;
  const double *gb = g + (size_t)bc * nx * nz;
  for (int k = threadIdx.x; k < ncx * ncz; k += blockDim.x) {
    const int a = k / ncz, d = k - a * ncz;
    double acc = 0;
    for (int ix = xs[a]; ix < xe[a]; ++ix) {
      const double ax = (x0[ix] == a ? 1.0 - wx[ix] : 0.0) + (x1[ix] == a ? wx[ix] : 0.0);
      if (ax == 0.0) continue;
      double row = 0;
      for (int iz = zs[d]; iz < ze[d]; ++iz) {
        const double az = (z0[iz] == d ? 1.0 - wz[iz] : 0.0) + (z1[iz] == d ? wz[iz] : 0.0);
        row += az * gb[(size_t)ix * nz + iz];
      }
      acc += ax * row;
    }
    gz[(size_t)bc * ncx * ncz + k] =
        (float)(scale * sigma[(size_t)c * ncx * ncz + k] * acc);
  }
}

// 1-D interpolation weights and supports along one axis of n fine points
// (np boundary frames each side) over nc coarse nodes.
void axis_weights(int n, int np, int nc, std::vector<int> &i0, std::vector<int> &i1,
                  std::vector<double> &w, std::vector<int> &s, std::vector<int> &e) {
  const int inner = n - 2 * np;
  const double f = static_cast<double>(inner) / nc;
  i0.resize(n);
  i1.resize(n);
  w.resize(n);
  s.assign(nc, n);
  e.assign(nc, 0);
  for (int x = 0; x < n; ++x) {
    const int xi = std::min(std::max(x - np, 0), inner - 1);
    double u = (xi + 0.5) / f - 0.5;
    u = std::min(std::max(u, 0.0), static_cast<double>(nc - 1));
    int a = static_cast<int>(std::floor(u));
    a = std::min(a, nc - 1);
    i0[x] = a;
    i1[x] = std::min(a + 1, nc - 1);
    w[x] = u - a;
    for (int k : {i0[x], i1[x]}) {
      s[k] = std::min(s[k], x);
      e[k] = std::max(e[k], x + 1);
    }
  }
}

template <class V>
void upload(DeviceBuffer &d, const V &v) {
  d.allocate(std::max<size_t>(v.size(), 1) * sizeof(v[0]));
  if (!v.empty())
    cuda_check(cudaMemcpy(d.get(), v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice),
               "upload coarse map");
}

}  // namespace

CoarseMap::CoarseMap(int device, int nx_, int nz_, int np_, int ncx_, int ncz_, const double *mean,
                     const double *sigma)
    : nx(nx_), nz(nz_), np(np_), ncx(ncx_), ncz(ncz_), device_(device) {
  if (nx <= 2 * np || nz <= 2 * np || ncx <= 0 || ncz <= 0 || ncx > nx - 2 * np ||
      ncz > nz - 2 * np)
    throw Error(PSV_ERR_INVALID_ARGUMENT, "coarse grid does not fit the inner grid");
  DeviceGuard guard(device_);
  std::vector<int> x0, x1, xs, xe, z0, z1, zs, ze;
  std::vector<double> wx, wz;
  axis_weights(nx, np, ncx, x0, x1, wx, xs, xe);
  axis_weights(nz, np, ncz, z0, z1, wz, zs, ze);
  upload(x0_, x0);
  upload(x1_, x1);
  upload(wx_, wx);
  upload(z0_, z0);
  upload(z1_, z1);
  upload(wz_, wz);
  upload(xs_, xs);
  upload(xe_, xe);
  upload(zs_, zs);
  upload(ze_, ze);
  const size_t n = (size_t)3 * ncx * ncz;
  upload(mean_, std::vector<double>(mean, mean + n));
  upload(sigma_, std::vector<double>(sigma, sigma + n));
  // (On the legacy stream, for which stream_ does not wait.)
  cuda_check(cudaStreamSynchronize(cudaStreamLegacy), "upload coarse map");
  cuda_check(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "cudaStreamCreate");
}

CoarseMap::~CoarseMap() {
  if (stream_) {
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(device_);
    cudaStreamSynchronize(stream_);
    cudaStreamDestroy(stream_);
    cudaSetDevice(prev);
  }
}

void CoarseMap::to_fields(int batch, const float *z, double *fields, cudaStream_t s) const {
  DeviceGuard guard(device_);
  const size_t n = (size_t)batch * 3 * nx * nz;
  if (!n) return;
  cudaStream_t use = s ? s : stream_;
  coarse_to_fields<<<static_cast<unsigned>((n + 255) / 256), 256, 0, use>>>(
      batch, nx, nz, ncx, ncz, x0_.as<int>(), x1_.as<int>(), wx_.as<double>(), z0_.as<int>(),
      z1_.as<int>(), wz_.as<double>(), mean_.as<double>(), sigma_.as<double>(), z, fields);
  cuda_check(cudaGetLastError(), "coarse to fields");
  if (!s) cuda_check(cudaStreamSynchronize(stream_), "coarse to fields");
}

void CoarseMap::gradient(int batch, const double *gfields, float *gz, double scale,
                         cudaStream_t s) const {
  DeviceGuard guard(device_);
  if (batch <= 0) return;
  cudaStream_t use = s ? s : stream_;
  fields_to_coarse<<<batch * 3, 256, 0, use>>>(nx, nz, ncx, ncz, x0_.as<int>(), x1_.as<int>(),
                                               wx_.as<double>(), z0_.as<int>(), z1_.as<int>(),
                                               wz_.as<double>(), xs_.as<int>(), xe_.as<int>(),
                                               zs_.as<int>(), ze_.as<int>(), sigma_.as<double>(),
                                               scale, gfields, gz);
  cuda_check(cudaGetLastError(), "fields to coarse");
  if (!s) cuda_check(cudaStreamSynchronize(stream_), "fields to coarse");
}

}  // namespace psv
