// nrldpc_train_tape.cu — float32 training kernels of the unrolled layered float
// min-sum that keep a tape instead of checkpoints: the forward stores the
// extrinsic input rel_j of every edge of every iteration, and the backward
// recomputes nothing.  Values and gradients are those of nrldpc_train.cu (which
// holds the float64 kernels and the checkpoint form), whose file comment states
// the arithmetic (deep_learning/deeplearning_ldpc_model.py:315-410).
//
// All of a row's forward follows from its rel_j: minima, signs, magnitudes, the
// clipped sums.  So the backward walks the tape in reverse, row by row, with dLQ
// in shared memory and the carry (the gradient of each edge's message for the
// iteration before) in a per-CTA buffer that stays in L2:
//   g_v = g_LQ[c_j] * [|v| within clip],   g_lrt = g_carry_j + g_v,  g_mag = (prod s) s_j g_lrt
//   S = sum of g_mag over j != idx,        g2 = g_mag of idx
//   g_alpha += S r1 + g2 r2,               g_a[idx] = S k1, g_a[idx2] = g2 k2, g_beta -= both
// with r = max(min - beta, 0) and k = alpha [min - beta >= 0] of the two minima.
// The tape is [T][batch][nnz][Zc] floats: 197 words per lifted column of BG2
// (a checkpoint of LQ and compressed messages takes 52 + 168), 316 of BG1 (68 + 184).
//
// The message of a check row (two magnitudes, flips and minimum position in one
// word) waits for the next iteration in the row's own tape slot of that
// iteration (every row has at least three edges); the row takes it from there
// just before it writes its rel over it.
//
// One code block per CTA where its Zc threads fill their warps, so a row's
// barrier holds two to twelve warps and a dozen blocks per SM hide each other's
// latency.  Both kernels are then bound by instruction issue.
//   batch 4096, 10 iterations, us    forward        backward
//   BG2 Zc64                      1422 -> 1012    6133 -> 1652
//   BG1 Zc112                     3500 -> 2990   16300 -> 6010
//   (before: a checkpoint per iteration, recomputed by the backward, six-block CTAs)
// ALU pipe 69 % (forward) and 59 % (backward) busy, 3.1 and 3.3 TB/s of HBM.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

#include "nrldpc_internal.h"

namespace nrldpc {
namespace {

// Rows between the tape's L2 prefetch and its use.
constexpr int kTapeAhead = 4;

// Ask L2 for the 16-byte-aligned interior of [lo, lo + bytes) with one
// cp.async.bulk.prefetch.L2 (a hint: nothing waits for it).
__device__ __forceinline__ void bulk_prefetch_l2(const void* lo, size_t bytes) {
  const uintptr_t a = (reinterpret_cast<uintptr_t>(lo) + 15u) & ~(uintptr_t)15u;
  const uintptr_t b = (reinterpret_cast<uintptr_t>(lo) + bytes) & ~(uintptr_t)15u;
  if (b > a) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)(b - a)));
}

// Byte address of edge e's word for lifted row zx4 / 4 (edge: {column * Zc * 4, (V mod Zc) * 4}).
__device__ __forceinline__ uint32_t tape_addr(const TrainTapeParams& p, int e, uint32_t zx4) {
  const uint2 ed = p.edge4[e];
  const uint32_t t = zx4 + ed.y;
  return min(t, t - 4u * (uint32_t)p.Zc) + ed.x;
}

// Word of edge j of lifted row zx in a row's slice of D Zc floats.  With Zc a
// multiple of 4: groups of four edges as one float4 per row, then what is left as a
// float2 and a float, so a row moves D floats in a quarter to a half of the
// instructions; otherwise one plane of Zc floats per edge.  Either way a thread's
// words are its own.
template <int kAccess>
__device__ __forceinline__ int tape_place(int D, int j, int zx, int Zc) {
  const int quads = D / 4 * 4;
  if (kAccess == kTapePlanes) return j * Zc + zx;
  if (j < quads) return (j & ~3) * Zc + 4 * zx + (j & 3);
  if ((D & 2) && j < quads + 2) return quads * Zc + 2 * zx + (j - quads);
  return (D - 1) * Zc + zx;
}
template <int D, int kAccess>
__device__ __forceinline__ void load_row(const float* slice, int zx, int Zc, float (&v)[D]) {
  if constexpr (kAccess == kTapeGroups) {
#pragma unroll
    for (int c = 0; c < D / 4; ++c) {
      const float4 q = __ldcs(reinterpret_cast<const float4*>(slice + 4 * c * Zc) + zx);
      v[4 * c] = q.x;
      v[4 * c + 1] = q.y;
      v[4 * c + 2] = q.z;
      v[4 * c + 3] = q.w;
    }
    constexpr int b = D / 4 * 4;
    const float* rest = slice + b * Zc;
    if constexpr ((D & 2) != 0) {
      const float2 q = __ldcs(reinterpret_cast<const float2*>(rest) + zx);
      v[b] = q.x;
      v[b + 1] = q.y;
    }
    if constexpr ((D & 1) != 0) v[D - 1] = __ldcs(rest + ((D & 2) ? 2 * Zc : 0) + zx);
  } else {
#pragma unroll
    for (int j = 0; j < D; ++j) v[j] = __ldcs(slice + tape_place<kAccess>(D, j, zx, Zc));
  }
}
// kStream: written once and read much later (the tape); otherwise kept near (the carry).
template <int D, int kAccess, bool kStream>
__device__ __forceinline__ void store_row(float* slice, int zx, int Zc, const float (&v)[D]) {
  const auto put = [](auto* a, auto x) {
    if constexpr (kStream) __stcs(a, x);
    else *a = x;
  };
  if constexpr (kAccess == kTapeGroups) {
#pragma unroll
    for (int c = 0; c < D / 4; ++c)
      put(reinterpret_cast<float4*>(slice + 4 * c * Zc) + zx, make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]));
    constexpr int b = D / 4 * 4;
    float* rest = slice + b * Zc;
    if constexpr ((D & 2) != 0) put(reinterpret_cast<float2*>(rest) + zx, make_float2(v[b], v[b + 1]));
    if constexpr ((D & 1) != 0) put(rest + ((D & 2) ? 2 * Zc : 0) + zx, v[D - 1]);
  } else {
#pragma unroll
    for (int j = 0; j < D; ++j) put(slice + tape_place<kAccess>(D, j, zx, Zc), v[j]);
  }
}

// A row's message in its tape slot of the next iteration, in words of the
// thread's own: magnitudes of the edges that carry the first and the second
// minimum, and a word with edge j's sign flip in bit D - 1 - j and the second
// minimum's edge from bit 20.
struct TapeMsg {
  float n1, n2;
  uint32_t f;
};
template <int D, int kAccess>
__device__ __forceinline__ TapeMsg load_msg(const float* slice, int zx, int Zc) {
  if constexpr (kAccess == kTapeGroups && D >= 4) {
    const float4 q = reinterpret_cast<const float4*>(slice)[zx];
    return TapeMsg{q.x, q.y, __float_as_uint(q.z)};
  } else if constexpr (kAccess == kTapeGroups) {
    const float2 q = reinterpret_cast<const float2*>(slice)[zx];
    return TapeMsg{q.x, q.y, __float_as_uint(slice[2 * Zc + zx])};
  } else {
    const auto at = [&](int j) { return slice[tape_place<kAccess>(D, j, zx, Zc)]; };
    return TapeMsg{at(0), at(1), __float_as_uint(at(2))};
  }
}
template <int D, int kAccess>
__device__ __forceinline__ void store_msg(float* slice, int zx, int Zc, const TapeMsg& m) {
  if constexpr (kAccess == kTapeGroups && D >= 4) {
    reinterpret_cast<float4*>(slice)[zx] = make_float4(m.n1, m.n2, __uint_as_float(m.f), 0.0f);
  } else if constexpr (kAccess == kTapeGroups) {
    reinterpret_cast<float2*>(slice)[zx] = make_float2(m.n1, m.n2);
    slice[2 * Zc + zx] = __uint_as_float(m.f);
  } else {
    slice[tape_place<kAccess>(D, 0, zx, Zc)] = m.n1;
    slice[tape_place<kAccess>(D, 1, zx, Zc)] = m.n2;
    slice[tape_place<kAccess>(D, 2, zx, Zc)] = __uint_as_float(m.f);
  }
}

// Sign of x as the model takes it, in bit 31: set where x < 0.  (Adding +0.0
// turns -0.0 into +0.0, and the sum of a NaN has its sign bit clear.)
__device__ __forceinline__ uint32_t sign_of(float x) { return __float_as_uint(__fadd_rn(x, 0.0f)); }

// Forward of one lifted check row: rel goes to the row's slice of this iteration's
// tape, from where the old message is taken first (zero in the first iteration),
// and the new message to the slice of the next iteration (none after the last).
// Without kKeep (evaluation) there is no tape, only the message's slice.
template <int D, int kAccess, bool kKeep>
__device__ __forceinline__ void tape_row_fwd(const TrainTapeParams& p, char* __restrict__ lq, int zx, int e0, float alpha,
                                             float beta, bool first, float* slice, float* next) {
  const float clip = p.clip;
  TapeMsg m{0.0f, 0.0f, 0u};
  if (!first) m = load_msg<D, kAccess>(slice, zx, p.Zc);
  const int ix = (int)(m.f >> 20);
  float rel[D];
  uint32_t addr[D];
  uint32_t sg = 0u;
  float m1 = INFINITY, m2 = INFINITY;
  int idx = 0;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    addr[j] = tape_addr(p, e0 + j, 4u * (uint32_t)zx);
    const uint32_t old = __float_as_uint(ix == j ? m.n2 : m.n1) ^ ((m.f << (32 - D + j)) & 0x80000000u);
    const float r = __fsub_rn(*reinterpret_cast<const float*>(lq + addr[j]), __uint_as_float(old));
    rel[j] = r;
    sg ^= sign_of(r);
    const float a = fabsf(r);
    const bool lt = a < m1;   // a NaN is never below, and fminf passes it over
    m2 = lt ? m1 : fminf(m2, a);
    m1 = fminf(m1, a);
    idx = lt ? j : idx;
  }
  if constexpr (kKeep) store_row<D, kAccess, true>(slice, zx, p.Zc, rel);
  const float s1 = __fmul_rn(alpha, fmaxf(__fsub_rn(m1, beta), 0.0f));
  const float s2 = __fmul_rn(alpha, fmaxf(__fsub_rn(m2, beta), 0.0f));
  uint32_t flips = 0u;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    const uint32_t f = sign_of(rel[j]) ^ sg;
    flips = __funnelshift_l(f, flips, 1);
    const uint32_t msg = __float_as_uint((j == idx) ? s2 : s1) ^ (f & 0x80000000u);
    const float v = __fadd_rn(rel[j], __uint_as_float(msg));
    *reinterpret_cast<float*>(lq + addr[j]) = fminf(fmaxf(v, -clip), clip);
  }
  if (next) store_msg<D, kAccess>(next, zx, p.Zc, TapeMsg{s1, s2, flips | (uint32_t)idx << 20});
}

// What a row's backward needs besides its loop over edges.
struct BwdRow {
  float s1, s2, r1, r2, k1, k2;
};
__device__ __forceinline__ BwdRow bwd_row(float m1, float m2, float alpha, float beta) {
  BwdRow b;
  const float o1 = __fsub_rn(m1, beta), o2 = __fsub_rn(m2, beta);
  b.r1 = fmaxf(o1, 0.0f);
  b.r2 = fmaxf(o2, 0.0f);
  b.k1 = o1 >= 0.0f ? alpha : 0.0f;   // d mag / d u
  b.k2 = o2 >= 0.0f ? alpha : 0.0f;
  b.s1 = __fmul_rn(alpha, b.r1);
  b.s2 = __fmul_rn(alpha, b.r2);
  return b;
}

// Backward of one lifted check row with infinities or NaN among its inputs: the
// loops of tape_row_bwd with every test of the model spelled out, over values
// read again from memory.
template <int kAccess>
__device__ __noinline__ void tape_row_bwd_odd(const TrainTapeParams& p, char* glq, int zx, int e0, int D, float alpha,
                                              float beta, const float* slice, float* carry, bool last, bool first, float* ga,
                                              float* gb) {
  const auto at = [&](int j) { return tape_place<kAccess>(D, j, zx, p.Zc); };
  bool neg = false;
  float m1 = INFINITY, m2 = INFINITY;
  int idx = -1, idx2 = -1;
  for (int j = 0; j < D; ++j) {
    const float rel = slice[at(j)], a = fabsf(rel);
    neg ^= rel < 0.0f;
    const bool lt1 = a < m1, lt2 = a < m2;
    idx2 = lt1 ? idx : (lt2 ? j : idx2);
    idx = lt1 ? j : idx;
    m2 = lt1 ? m1 : (lt2 ? a : m2);
    m1 = lt1 ? a : m1;
  }
  idx = idx < 0 ? 0 : idx;
  const BwdRow b = bwd_row(m1, m2, alpha, beta);
  const auto incoming = [&](int j, float rel, bool flip) {
    const float mag = j == idx ? b.s2 : b.s1;
    const float v = __fadd_rn(rel, flip ? -mag : mag);
    return v >= -p.clip && v <= p.clip ? *reinterpret_cast<const float*>(glq + tape_addr(p, e0 + j, 4u * (uint32_t)zx)) : 0.0f;
  };
  float sum1 = 0.0f, gm2 = 0.0f;
  for (int j = 0; j < D; ++j) {
    const float rel = slice[at(j)];
    const bool flip = (rel < 0.0f) != neg;
    const float g_lrt = (last ? 0.0f : carry[at(j)]) + incoming(j, rel, flip);
    const float g_mag = flip ? -g_lrt : g_lrt;
    if (j == idx) gm2 = g_mag;
    else sum1 += g_mag;
  }
  *ga += sum1 * b.r1 + gm2 * b.r2;
  const float g1 = sum1 * b.k1, g2 = gm2 * b.k2;
  *gb -= g1 + g2;
  for (int j = 0; j < D; ++j) {
    const float rel = slice[at(j)];
    const float gv = incoming(j, rel, (rel < 0.0f) != neg);
    const float g_a = j == idx ? g1 : (j == idx2 ? g2 : 0.0f);
    const float g_rel = p.detach ? 0.0f : gv + (rel > 0.0f ? g_a : (rel < 0.0f ? -g_a : 0.0f));
    *reinterpret_cast<float*>(glq + tape_addr(p, e0 + j, 4u * (uint32_t)zx)) = g_rel;
    if (!first) carry[at(j)] = -g_rel;
  }
}

// Backward of one lifted check row (see the file comment).  kClip: LLRs are
// clipped, so a sum outside the range passes no gradient.
template <int D, int kAccess, bool kClip>
__device__ __forceinline__ void tape_row_bwd(const TrainTapeParams& p, char* __restrict__ glq, int zx, int e0, float alpha,
                                             float beta, const float* slice, float* carry, bool last, bool first, float* ga,
                                             float* gb) {
  const int Zc = p.Zc;
  float rel[D];
  load_row<D, kAccess>(slice, zx, Zc, rel);
  float cv[D];
  if (last) {
#pragma unroll
    for (int j = 0; j < D; ++j) cv[j] = 0.0f;
  } else {
    load_row<D, kAccess>(carry, zx, Zc, cv);
  }
  uint32_t sg = 0u;
  float m1 = INFINITY, m2 = INFINITY, total = 0.0f;
  // idx: first minimum; idx2: first minimum of the others (torch.min's choices)
  int idx = 0, idx2 = 0;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    sg ^= sign_of(rel[j]);
    const float a = fabsf(rel[j]);
    total += a;
    const bool lt1 = a < m1, lt2 = a < m2;
    idx2 = lt1 ? idx : (lt2 ? j : idx2);
    idx = lt1 ? j : idx;
    m2 = lt1 ? m1 : fminf(m2, a);
    m1 = fminf(m1, a);
  }
  const BwdRow b = bwd_row(m1, m2, alpha, beta);
  if (!(total + fabsf(b.s1) + fabsf(b.s2) < INFINITY)) {   // an infinity or a NaN in the row
    tape_row_bwd_odd<kAccess>(p, glq, zx, e0, D, alpha, beta, slice, carry, last, first, ga, gb);
    return;
  }
  // From here every |rel| is finite: a clip test can only fail by the range, and
  // rel is zero at idx (idx2) exactly when m1 (m2) is.
  float sum1 = 0.0f, gm2 = 0.0f;   // g_mag of the edges that carry the first minimum (summed), and of edge idx
#pragma unroll
  for (int j = 0; j < D; ++j) {
    const uint32_t f = (sign_of(rel[j]) ^ sg) & 0x80000000u;   // the message is negated
    float gv = *reinterpret_cast<const float*>(glq + tape_addr(p, e0 + j, 4u * (uint32_t)zx));
    if constexpr (kClip) {
      const float v = __fadd_rn(rel[j], __uint_as_float(__float_as_uint(j == idx ? b.s2 : b.s1) ^ f));
      gv = fabsf(v) <= p.clip ? gv : 0.0f;
    }
    const float g_mag = __uint_as_float(__float_as_uint(cv[j] + gv) ^ f);
    cv[j] = gv;
    if (j == idx) gm2 = g_mag;
    else sum1 += g_mag;
  }
  *ga += sum1 * b.r1 + gm2 * b.r2;
  float g1 = sum1 * b.k1, g2 = gm2 * b.k2;   // gradients of the two minima
  *gb -= g1 + g2;
  g1 = m1 > 0.0f ? g1 : 0.0f;                // d|rel| / d rel is 0 at 0
  g2 = m2 > 0.0f ? g2 : 0.0f;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    const float g_a = j == idx ? g1 : (j == idx2 ? g2 : 0.0f);
    const float g_rel = p.detach ? 0.0f : cv[j] + __uint_as_float(__float_as_uint(g_a) ^ (__float_as_uint(rel[j]) & 0x80000000u));
    *reinterpret_cast<float*>(glq + tape_addr(p, e0 + j, 4u * (uint32_t)zx)) = g_rel;
    cv[j] = -g_rel;
  }
  if (!first) store_row<D, kAccess, false>(carry, zx, Zc, cv);
}

#define NRLDPC_TAPE_DISPATCH(deg, CALL) \
  switch (deg) {                        \
    case 3: { CALL(3); break; }         \
    case 4: { CALL(4); break; }         \
    case 5: { CALL(5); break; }         \
    case 6: { CALL(6); break; }         \
    case 7: { CALL(7); break; }         \
    case 8: { CALL(8); break; }         \
    case 9: { CALL(9); break; }         \
    case 10: { CALL(10); break; }       \
    default: { CALL((kMaxD > 10 ? 19 : 10)); break; } \
  }

// kMaxD: the largest row degree of the base graph (19 for BG1, 10 for BG2); a
// BG2 instantiation carries no degree-19 code and needs fewer registers.  The
// launch bound sets the registers: 72 for BG2, 14 CTAs of 64 threads on an SM
// (backward at Zc=64 1774 us; 1930 with 80 registers and 12 CTAs, 2009 with 64;
// before rows were staged), and 80 for BG1, whose degree-19 rows would spill
// (Zc=112 6261 us; 6494 with 72).
constexpr int launch_threads(int max_deg) { return max_deg <= 10 ? 448 : kThreadsTarget; }

// A row of iteration t, staged in shared memory: one 16-byte load instead of
// parameter and global loads and their address arithmetic in every row.
struct __align__(16) RowDesc {
  uint16_t e0, deg;
  uint32_t off;   // floats before the row's slice
  float alpha, beta;
};
template <bool kKeep>
__device__ __forceinline__ void stage_rows(const TrainTapeParams& p, RowDesc* s_rows, int t) {
  for (int r = threadIdx.x; r < p.R; r += blockDim.x)
    s_rows[r] = RowDesc{p.row_off[r], (uint16_t)(p.row_off[r + 1] - p.row_off[r]),
                        (uint32_t)(kKeep ? p.row_off[r] : kTapeMessageWords * r) * (uint32_t)p.Zc, p.alpha[t * p.R + r],
                        p.beta[t * p.R + r]};
}

// kKeep: the tape is kept for a backward.  Otherwise (evaluation) the rows' messages
// lie in slices of kTapeMessageWords Zc floats, the same ones in every iteration.
template <int kMaxD, int kAccess, bool kKeep>
__global__ void __launch_bounds__(launch_threads(kMaxD), 2) tape_forward_kernel(const __grid_constant__ TrainTapeParams p) {
  extern __shared__ __align__(16) float s_lq[];
  __shared__ RowDesc s_rows[kMaxRows];
  const float clip = p.clip;
  const int tid = threadIdx.x;
  const int g = tid / p.Zc, zx = tid - g * p.Zc;
  const bool active = g < p.G;
  float* lq = s_lq + (active ? g : 0) * p.n;
  for (int item = blockIdx.x; item * p.G < p.batch; item += gridDim.x) {
    const int cw = item * p.G + g;
    const bool valid = active && cw < p.batch;
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) lq[i] = fminf(fmaxf(p.llr[(size_t)cw * p.n + i], -clip), clip);
    for (int t = 0; t < p.T; ++t) {
      stage_rows<kKeep>(p, s_rows, t);   // the last row's barrier lies between its reads and this
      __syncthreads();
      float* tape = p.tape + ((kKeep ? (size_t)t * p.batch : 0) + (valid ? cw : 0)) * p.tape_words;
      float* tnext = kKeep ? tape + (size_t)p.batch * p.tape_words : tape;
      for (int row = 0; row < p.R; ++row) {
        if (valid) {
          const RowDesc d = s_rows[row];
          const int e0 = d.e0, deg = d.deg;
          float* slice = tape + d.off;
          float* next = t + 1 < p.T ? tnext + d.off : nullptr;
#define NRLDPC_FWD(D) tape_row_fwd<D, kAccess, kKeep>(p, reinterpret_cast<char*>(lq), zx, e0, d.alpha, d.beta, t == 0, slice, next)
          NRLDPC_TAPE_DISPATCH(deg, NRLDPC_FWD)
#undef NRLDPC_FWD
        }
        __syncthreads();
      }
      if (p.iter_llr) {
        if (valid)
          for (int i = zx; i < p.n; i += p.Zc) p.iter_llr[((size_t)t * p.batch + cw) * p.n + i] = lq[i];
        __syncthreads();   // read before the next iteration's rows write
      }
    }
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) p.final_llr[(size_t)cw * p.n + i] = lq[i];
    __syncthreads();
  }
}

// Sum of a (lane 0) and b (lane 16) over the warp: the first step trades halves,
// so both sums take five shuffles.
__device__ __forceinline__ float warp_sum_pair(float a, float b) {
  const bool hi = (threadIdx.x & 16) != 0;
  float v = (hi ? b : a) + __shfl_xor_sync(0xFFFFFFFFu, hi ? a : b, 16);
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}

template <int kMaxD, int kAccess, bool kClip>
__global__ void __launch_bounds__(launch_threads(kMaxD), 2) tape_backward_kernel(const __grid_constant__ TrainTapeParams p) {
  // dLQ of each code block; the iteration's alpha / beta gradients per row and
  // warp, [R][2][warps]; the CTA's sums of them, [T][R][2], added to the outputs
  // at the end (with very many iterations they do not fit, and every iteration
  // adds its own).
  extern __shared__ __align__(16) float s_glq[];
  __shared__ RowDesc s_rows[kMaxRows];
  const int tid = threadIdx.x;
  const int warps = blockDim.x >> 5;
  float* s_part = s_glq + (size_t)p.G * p.n;
  float* s_acc = s_part + 2 * p.R * warps;
  const int g = tid / p.Zc, zx = tid - g * p.Zc;
  const bool active = g < p.G;
  float* glq = s_glq + (active ? g : 0) * p.n;
  float* carry = p.carry + (size_t)blockIdx.x * p.carry_per_cta + (size_t)(active ? g : 0) * p.tape_words;
  if (p.acc)
    for (int k = tid; k < 2 * p.T * p.R; k += blockDim.x) s_acc[k] = 0.0f;
  for (int item = blockIdx.x; item * p.G < p.batch; item += gridDim.x) {
    const int cw = item * p.G + g;
    const bool valid = active && cw < p.batch;
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) glq[i] = p.g_final ? p.g_final[(size_t)cw * p.n + i] : 0.0f;
    for (int t = p.T - 1; t >= 0; --t) {
      // own indices i = zx + k Zc, like the loads above; rows need all of them
      if (valid && p.g_iter)
        for (int i = zx; i < p.n; i += p.Zc) glq[i] += p.g_iter[((size_t)t * p.batch + cw) * p.n + i];
      stage_rows<true>(p, s_rows, t);
      __syncthreads();   // also: the sums over s_part below have been read
      const float* tape = p.tape + ((size_t)t * p.batch + (valid ? cw : 0)) * p.tape_words;
      for (int row = p.R - 1; row >= 0; --row) {
        float ga = 0.0f, gb = 0.0f;
        if (valid) {
          const RowDesc d = s_rows[row];
          const int e0 = d.e0, deg = d.deg;
          // the tape comes from HBM: a row's slice a few rows ahead of its use
          if (zx == 0 && row >= kTapeAhead) {
            const RowDesc a = s_rows[row - kTapeAhead];
            bulk_prefetch_l2(tape + a.off, (size_t)a.deg * (size_t)p.Zc * 4u);
          }
          const float* slice = tape + d.off;
          float* cs = carry + d.off;
#define NRLDPC_BWD(D) \
  tape_row_bwd<D, kAccess, kClip>(p, reinterpret_cast<char*>(glq), zx, e0, d.alpha, d.beta, slice, cs, t == p.T - 1, t == 0, &ga, &gb)
          NRLDPC_TAPE_DISPATCH(deg, NRLDPC_BWD)
#undef NRLDPC_BWD
        }
        const float v = warp_sum_pair(ga, gb);
        if ((tid & 15) == 0) s_part[(2 * row + ((tid >> 4) & 1)) * warps + (tid >> 5)] = v;
        __syncthreads();
      }
      // the iteration's gradients, summed over the CTA's warps
      for (int k = tid; k < 2 * p.R; k += blockDim.x) {
        float s = 0.0f;
        for (int w = 0; w < warps; ++w) s += s_part[k * warps + w];
        if (p.acc) s_acc[2 * t * p.R + k] += s;
        else if (s != 0.0f) atomicAdd(((k & 1) ? p.g_beta : p.g_alpha) + t * p.R + (k >> 1), s);
      }
    }
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) {
        const float x = p.llr[(size_t)cw * p.n + i];
        p.g_llr[(size_t)cw * p.n + i] = (x >= -p.clip && x <= p.clip) ? glq[i] : 0.0f;
      }
    // the next item's first writes are to this thread's own words
  }
  if (p.acc)   // every thread wrote, and now adds, the same entries
    for (int k = tid; k < 2 * p.R; k += blockDim.x)
      for (int t = 0; t < p.T; ++t) {
        const float s = s_acc[2 * t * p.R + k];
        if (s != 0.0f) atomicAdd(((k & 1) ? p.g_beta : p.g_alpha) + t * p.R + (k >> 1), s);
      }
}

template <typename K>
int launch_tape(K kernel, const TrainTapeParams& p, int grid, int block, int smem, void* stream) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return (int)e;
  kernel<<<grid, block, smem, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  count_launch();
  return (int)cudaGetLastError();
}

template <typename K>
int occupancy_tape_one(K kernel, int block, int smem) {
  int n = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, block, smem);
  return n;
}

}  // namespace

namespace {

// Calls op(kernel) with the instance of a launch.
template <typename Op>
int with_tape_kernel(TapePass pass, bool bg2, int access, bool clipped, Op op) {
  const auto tape = [&](auto max_degree, auto mode) {
    constexpr int d = decltype(max_degree)::value, m = decltype(mode)::value;
    if (pass == kTapeEvaluate) return op(tape_forward_kernel<d, m, false>);
    if (pass == kTapeForward) return op(tape_forward_kernel<d, m, true>);
    return clipped ? op(tape_backward_kernel<d, m, true>) : op(tape_backward_kernel<d, m, false>);
  };
  const auto graph = [&](auto max_degree) {
    switch (access) {
      case kTapePlanes: return tape(max_degree, std::integral_constant<int, kTapePlanes>{});
      case kTapeGroupWords: return tape(max_degree, std::integral_constant<int, kTapeGroupWords>{});
      default: return tape(max_degree, std::integral_constant<int, kTapeGroups>{});
    }
  };
  return bg2 ? graph(std::integral_constant<int, 10>{}) : graph(std::integral_constant<int, 19>{});
}

}  // namespace

int launch_train_tape(const TrainTapeParams& p, TapePass pass, int grid, int block, int smem, void* stream) {
  return with_tape_kernel(pass, p.R == NRLDPC_BG2_ROWS, p.access, isfinite(p.clip),
                          [&](auto k) { return launch_tape(k, p, grid, block, smem, stream); });
}

int occupancy_train_tape(const TrainTapeParams& p, TapePass pass, int block, int smem) {
  return with_tape_kernel(pass, p.R == NRLDPC_BG2_ROWS, p.access, isfinite(p.clip),
                          [&](auto k) { return occupancy_tape_one(k, block, smem); });
}

}  // namespace nrldpc
