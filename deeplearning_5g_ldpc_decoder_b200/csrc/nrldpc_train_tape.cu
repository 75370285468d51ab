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
//   BG2 Zc64, batch 4096, 10 iterations: forward 1422 -> 1207 us, backward 6133 -> 2837 us
//   (before: a checkpoint per iteration, recomputed by the backward, six-block CTAs)
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

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

__device__ __forceinline__ uint32_t tape_addr(const TrainTapeParams& p, int e, uint32_t zx) {
  const uint32_t ed = p.edge[e];
  uint32_t t = zx + (ed >> 16);
  t = min(t, t - (uint32_t)p.Zc);
  return (ed & 0xFFFFu) + t;
}

// Forward of one lifted check row: the old message comes from the row's slot of
// this iteration (none in the first), rel goes there, and the new message to the
// slot of the next iteration (none after the last).
template <int D>
__device__ __forceinline__ void tape_row_fwd(const TrainTapeParams& p, float* __restrict__ lq, uint32_t zx, int e0,
                                              float alpha, float beta, bool first, float* slot, float* next) {
  const int Zc = p.Zc;
  const float clip = p.clip;
  float n1 = 0, n2 = 0;
  uint32_t fl = 0u;   // flips in bits 0..18, position of the minimum from bit 20
  if (!first) {
    n1 = slot[0];
    n2 = slot[Zc];
    fl = __float_as_uint(slot[2 * Zc]);
  }
  const int ix = (int)(fl >> 20);
  float rel[D];
  uint32_t addr[D];
  bool neg = false;
  float m1 = INFINITY, m2 = INFINITY;
  int idx = 0;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    addr[j] = tape_addr(p, e0 + j, zx);
    float old = ix == j ? n2 : n1;
    old = ((fl >> j) & 1u) ? -old : old;
    const float r = __fsub_rn(lq[addr[j]], old);
    rel[j] = r;
    neg ^= (r < 0.0f);
    const float a = fabsf(r);
    const bool lt1 = a < m1;
    m2 = lt1 ? m1 : (a < m2 ? a : m2);
    m1 = lt1 ? a : m1;
    idx = lt1 ? j : idx;
  }
#pragma unroll
  for (int j = 0; j < D; ++j) __stcs(slot + (size_t)j * Zc, rel[j]);
  const float s1 = __fmul_rn(alpha, fmaxf(__fsub_rn(m1, beta), 0.0f));
  const float s2 = __fmul_rn(alpha, fmaxf(__fsub_rn(m2, beta), 0.0f));
  uint32_t flips = (uint32_t)idx << 20;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    const bool flip = (rel[j] < 0.0f) != neg;
    const float mag = (j == idx) ? s2 : s1;
    flips |= (flip ? 1u : 0u) << j;
    float v = __fadd_rn(rel[j], flip ? -mag : mag);
    v = fminf(fmaxf(v, -clip), clip);
    lq[addr[j]] = v;
  }
  if (next) {
    next[0] = s1;
    next[Zc] = s2;
    next[2 * Zc] = __uint_as_float(flips);
  }
}

// Backward of one lifted check row (see the file comment).
template <int D>
__device__ __forceinline__ void tape_row_bwd(const TrainTapeParams& p, float* __restrict__ glq, uint32_t zx, int e0,
                                              float alpha, float beta, const float* slot, float* carry, bool last, bool first,
                                              float* ga, float* gb) {
  const int Zc = p.Zc;
  const float clip = p.clip;
  // Rows of more than 10 edges keep only rel in registers: edge addresses are
  // recomputed and the incoming gradient is read again in the last pass (no
  // other edge of the row writes that word).
  constexpr bool kLean = D > 10;
  constexpr int kKeep = kLean ? 1 : D;
  float rel[D];
  float cv[kKeep], g_in[kKeep];
  uint32_t addr[kKeep];
#pragma unroll
  for (int j = 0; j < D; ++j) rel[j] = __ldcs(slot + (size_t)j * Zc);
  if constexpr (!kLean) {
#pragma unroll
    for (int j = 0; j < D; ++j) cv[j] = last ? 0.0f : carry[(size_t)j * Zc];
  }
  bool neg = false;
  float m1 = INFINITY, m2 = INFINITY;
  // idx: first minimum; idx2: first minimum of the others (torch.min's choices),
  // none (-1) where no other is below infinity
  int idx = -1, idx2 = -1;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    neg ^= (rel[j] < 0.0f);
    const float a = fabsf(rel[j]);
    const bool lt1 = a < m1, lt2 = a < m2;
    idx2 = lt1 ? idx : (lt2 ? j : idx2);
    idx = lt1 ? j : idx;
    m2 = lt1 ? m1 : (lt2 ? a : m2);
    m1 = lt1 ? a : m1;
  }
  idx = idx < 0 ? 0 : idx;
  const float o1 = __fsub_rn(m1, beta), o2 = __fsub_rn(m2, beta);
  const float r1 = fmaxf(o1, 0.0f), r2 = fmaxf(o2, 0.0f);
  const float k1 = o1 >= 0.0f ? alpha : 0.0f;   // d mag / d u
  const float k2 = o2 >= 0.0f ? alpha : 0.0f;
  const float s1 = __fmul_rn(alpha, r1), s2 = __fmul_rn(alpha, r2);
  // g_mag of the edges that carry the first minimum (summed), and of edge idx
  float sum1 = 0, gm2 = 0;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    const uint32_t a = tape_addr(p, e0 + j, zx);
    const bool flip = (rel[j] < 0.0f) != neg;
    const float mag = (j == idx) ? s2 : s1;
    const float v = __fadd_rn(rel[j], flip ? -mag : mag);
    const float gv = (v >= -clip && v <= clip) ? glq[a] : 0.0f;
    if constexpr (!kLean) {
      addr[j] = a;
      g_in[j] = gv;
    }
    const float g_lrt = (kLean ? (last ? 0.0f : carry[(size_t)j * Zc]) : cv[kLean ? 0 : j]) + gv;
    const float g_mag = flip ? -g_lrt : g_lrt;
    if (j == idx) gm2 = g_mag;
    else sum1 += g_mag;
  }
  *ga += sum1 * r1 + gm2 * r2;
  const float g1 = sum1 * k1, g2 = gm2 * k2;   // gradients of the two minima
  *gb -= g1 + g2;
#pragma unroll
  for (int j = 0; j < D; ++j) {
    uint32_t a;
    float gv;
    if constexpr (kLean) {
      a = tape_addr(p, e0 + j, zx);
      const bool flip = (rel[j] < 0.0f) != neg;
      const float mag = (j == idx) ? s2 : s1;
      const float v = __fadd_rn(rel[j], flip ? -mag : mag);
      gv = (v >= -clip && v <= clip) ? glq[a] : 0.0f;
    } else {
      a = addr[j];
      gv = g_in[j];
    }
    float g_rel = 0;
    if (!p.detach) {
      const float g_a = j == idx ? g1 : (j == idx2 ? g2 : 0.0f);
      g_rel = gv + (rel[j] > 0.0f ? g_a : (rel[j] < 0.0f ? -g_a : 0.0f));
    }
    glq[a] = g_rel;
    if (!first) carry[(size_t)j * Zc] = -g_rel;
  }
}

#define NRLDPC_TAPE_DISPATCH(FN, deg, ...)   \
  switch (deg) {                                 \
    case 3: FN<3>(__VA_ARGS__); break;        \
    case 4: FN<4>(__VA_ARGS__); break;        \
    case 5: FN<5>(__VA_ARGS__); break;        \
    case 6: FN<6>(__VA_ARGS__); break;        \
    case 7: FN<7>(__VA_ARGS__); break;        \
    case 8: FN<8>(__VA_ARGS__); break;        \
    case 9: FN<9>(__VA_ARGS__); break;        \
    case 10: FN<10>(__VA_ARGS__); break;      \
    default: FN<(kMaxD > 10 ? 19 : 10)>(__VA_ARGS__); break;      \
  }

// kMaxD: the largest row degree of the base graph (19 for BG1, 10 for BG2); a
// BG2 instantiation carries no degree-19 code and needs fewer registers.
template <int kMaxD>
__global__ void __launch_bounds__(kThreadsTarget, 2)
    tape_forward_kernel(const __grid_constant__ TrainTapeParams p) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  float* s_lq = reinterpret_cast<float*>(s_raw);
  const float* llr = p.llr;
  const float* alpha_t = p.alpha;
  const float* beta_t = p.beta;
  float* final_llr = p.final_llr;
  float* iter_llr = p.iter_llr;
  const float clip = p.clip;
  const int tid = threadIdx.x;
  const int g = tid / p.Zc, zx = tid - g * p.Zc;
  const bool active = g < p.G;
  float* lq = s_lq + (active ? g : 0) * p.n;
  for (int item = blockIdx.x; item * p.G < p.batch; item += gridDim.x) {
    const int cw = item * p.G + g;
    const bool valid = active && cw < p.batch;
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) lq[i] = fminf(fmaxf(llr[(size_t)cw * p.n + i], -clip), clip);
    __syncthreads();
    for (int t = 0; t < p.T; ++t) {
      float* tape = p.tape + ((size_t)t * p.batch + (valid ? cw : 0)) * p.tape_words + zx;
      float* tnext = tape + (size_t)p.batch * p.tape_words;
      for (int row = 0; row < p.R; ++row) {
        if (valid) {
          const int e0 = p.row_off[row], deg = p.row_off[row + 1] - e0;
          const float alpha = alpha_t[t * p.R + row], beta = beta_t[t * p.R + row];
          float* slot = tape + (size_t)e0 * p.Zc;
          float* next = t + 1 < p.T ? tnext + (size_t)e0 * p.Zc : nullptr;
          NRLDPC_TAPE_DISPATCH(tape_row_fwd, deg, p, lq, (uint32_t)zx, e0, alpha, beta, t == 0, slot, next)
        }
        __syncthreads();
      }
      if (valid && iter_llr) {
        for (int i = zx; i < p.n; i += p.Zc) iter_llr[((size_t)t * p.batch + cw) * p.n + i] = lq[i];
      }
      if (iter_llr) __syncthreads();   // read before the next iteration's rows write
    }
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) final_llr[(size_t)cw * p.n + i] = lq[i];
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

template <int kMaxD>
__global__ void __launch_bounds__(kThreadsTarget, 2)
    tape_backward_kernel(const __grid_constant__ TrainTapeParams p) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ float s_red[2][2][kThreadsTarget / 32];   // [row parity][alpha, beta][warp]
  float* s_glq = reinterpret_cast<float*>(s_raw);       // dLQ of each code block
  // Sums of the CTA's alpha / beta gradients, [T][R][2], added to the outputs at
  // the end; with very many iterations they do not fit and every row adds its own.
  float* s_acc = s_glq + (size_t)p.G * p.n;
  const float* llr = p.llr;
  const float* alpha_t = p.alpha;
  const float* beta_t = p.beta;
  const float* g_final = p.g_final;
  const float* g_iter = p.g_iter;
  float* g_llr = p.g_llr;
  float* g_alpha = p.g_alpha;
  float* g_beta = p.g_beta;
  const float clip = p.clip;
  const int tid = threadIdx.x;
  const int warps = blockDim.x >> 5;
  const int g = tid / p.Zc, zx = tid - g * p.Zc;
  const bool active = g < p.G;
  float* glq = s_glq + (active ? g : 0) * p.n;
  float* carry = p.carry + (size_t)blockIdx.x * p.carry_per_cta +
                (size_t)(active ? g : 0) * (size_t)p.nnz * p.Zc + zx;
  if (p.acc)
    for (int k = tid; k < 2 * p.T * p.R; k += blockDim.x) s_acc[k] = 0;
  for (int item = blockIdx.x; item * p.G < p.batch; item += gridDim.x) {
    const int cw = item * p.G + g;
    const bool valid = active && cw < p.batch;
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) glq[i] = g_final ? g_final[(size_t)cw * p.n + i] : 0.0f;
    for (int t = p.T - 1; t >= 0; --t) {
      // own indices i = zx + k Zc, like the loads above; rows need all of them
      if (valid && g_iter)
        for (int i = zx; i < p.n; i += p.Zc) glq[i] += g_iter[((size_t)t * p.batch + cw) * p.n + i];
      __syncthreads();
      const float* tape = p.tape + ((size_t)t * p.batch + (valid ? cw : 0)) * p.tape_words + zx;
      for (int row = p.R - 1; row >= 0; --row) {
        float ga = 0, gb = 0;
        if (valid) {
          const int e0 = p.row_off[row], deg = p.row_off[row + 1] - e0;
          // the tape comes from HBM: a row's slice a few rows ahead of its use
          if (zx == 0 && row >= kTapeAhead) {
            const int ep = p.row_off[row - kTapeAhead];
            bulk_prefetch_l2(tape + (size_t)ep * p.Zc, (size_t)(p.row_off[row - kTapeAhead + 1] - ep) * (size_t)p.Zc * 4u);
          }
          const float alpha = alpha_t[t * p.R + row], beta = beta_t[t * p.R + row];
          const float* slot = tape + (size_t)e0 * p.Zc;
          NRLDPC_TAPE_DISPATCH(tape_row_bwd, deg, p, glq, (uint32_t)zx, e0, alpha, beta, slot,
                                carry + (size_t)e0 * p.Zc, t == p.T - 1, t == 0, &ga, &gb)
        }
        // Sum of the row's alpha / beta gradient over the CTA.  Double-buffered
        // by row parity: the next row's writes never meet this row's reads,
        // which end before the barrier after that row.
        const float v = warp_sum_pair(ga, gb);
        if ((tid & 15) == 0) s_red[row & 1][(tid >> 4) & 1][tid >> 5] = v;
        __syncthreads();
        if (tid < 2) {
          float s = 0;
          for (int w = 0; w < warps; ++w) s += s_red[row & 1][tid][w];
          const int k = t * p.R + row;
          if (p.acc) s_acc[2 * k + tid] += s;
          else if (s != 0.0f) atomicAdd((tid ? g_beta : g_alpha) + k, s);
        }
      }
    }
    if (valid)
      for (int i = zx; i < p.n; i += p.Zc) {
        const float x = llr[(size_t)cw * p.n + i];
        g_llr[(size_t)cw * p.n + i] = (x >= -clip && x <= clip) ? glq[i] : 0.0f;
      }
    // the next item's first writes are to this thread's own words
  }
  if (p.acc) {
    __syncthreads();
    for (int k = tid; k < 2 * p.T * p.R; k += blockDim.x)
      if (s_acc[k] != 0.0f) atomicAdd(((k & 1) ? g_beta : g_alpha) + (k >> 1), s_acc[k]);
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

int launch_train_tape(const TrainTapeParams& p, bool backward, int grid, int block, int smem, void* stream) {
  const bool bg2 = p.R == NRLDPC_BG2_ROWS;
  if (backward)
    return bg2 ? launch_tape(tape_backward_kernel<10>, p, grid, block, smem, stream)
               : launch_tape(tape_backward_kernel<19>, p, grid, block, smem, stream);
  return bg2 ? launch_tape(tape_forward_kernel<10>, p, grid, block, smem, stream)
             : launch_tape(tape_forward_kernel<19>, p, grid, block, smem, stream);
}

int occupancy_train_tape(bool backward, bool bg2, int block, int smem) {
  if (backward)
    return bg2 ? occupancy_tape_one(tape_backward_kernel<10>, block, smem)
               : occupancy_tape_one(tape_backward_kernel<19>, block, smem);
  return bg2 ? occupancy_tape_one(tape_forward_kernel<10>, block, smem)
             : occupancy_tape_one(tape_forward_kernel<19>, block, smem);
}

}  // namespace nrldpc
