// nrldpc_channel.cu — device LLR front-end: NR QAM mapping, complex AWGN,
// max-log demapping and int16 quantisation, for batches of code blocks.
//
// Restates the reference's test channel (c_lib/tx_rx_process.c:20-324):
//  * TS 38.211 5.1 constellations with the reference's float expressions
//    (bit_sign(b) = 1 - 2b, nested amplitude, times A = 1/sqrt(2|10|42|170)),
//  * piecewise-linear max-log LLRs per bit pair (:101-268), evaluated as
//    ((c1*A) * (s*r + c2*A)) / noise_var with the reference's segment
//    boundaries and strict "<" comparisons, round-to-nearest float ops,
//  * quantisation round(128*llr) (away from zero), clipped to +-10000 (:27-40).
// The noise comes from a counter-based generator (splitmix64 of seed, block,
// symbol; Box-Muller) instead of libc rand(); the noisy symbols can be returned
// so the demapper can be checked against a host restatement.
#include <cuda_runtime.h>
#include <stdint.h>

#include "nrldpc_internal.h"

namespace nrldpc {
namespace {

// One segment of a piecewise max-log LLR: for r < thr*A (last: always),
// llr = (c1*A) * (s*r + c2*A) / noise_var.
struct Seg {
  float thr, c1, s, c2;
};
constexpr float kInf = 3.0e38f;

// Segment tables per bit pair (re/im share them), restating
// c_lib/tx_rx_process.c:101-231.
__constant__ Seg kQam16[2][3] = {
    {{-2, 8, 1, 1}, {2, 4, 1, 0}, {kInf, 8, 1, -1}},
    {{0, 4, 1, 2}, {kInf, 4, -1, 2}, {kInf, 0, 0, 0}},
};
__constant__ int kQam16N[2] = {3, 2};
__constant__ Seg kQam64[3][7] = {
    {{-6, 16, 1, 3}, {-4, 12, 1, 2}, {-2, 8, 1, 1}, {2, 4, 1, 0}, {4, 8, 1, -1}, {6, 12, 1, -2}, {kInf, 16, 1, -3}},
    {{-6, 8, 1, 5}, {-2, 4, 1, 4}, {0, 8, 1, 3}, {2, 8, -1, 3}, {6, 4, -1, 4}, {kInf, 8, -1, 5}, {kInf, 0, 0, 0}},
    {{-4, 4, 1, 6}, {0, 4, -1, -2}, {4, 4, 1, -2}, {kInf, 4, -1, 6}, {kInf, 0, 0, 0}, {kInf, 0, 0, 0},
     {kInf, 0, 0, 0}},
};
__constant__ int kQam64N[3] = {7, 6, 4};
__constant__ Seg kQam256[4][15] = {
    {{-14, 32, 1, 7}, {-12, 28, 1, 6}, {-10, 24, 1, 5}, {-8, 20, 1, 4}, {-6, 16, 1, 3}, {-4, 12, 1, 2},
     {-2, 8, 1, 1}, {2, 4, 1, 0}, {4, 8, 1, -1}, {6, 12, 1, -2}, {8, 16, 1, -3}, {10, 20, 1, -4},
     {12, 24, 1, -5}, {14, 28, 1, -6}, {kInf, 32, 1, -7}},
    {{-14, 16, 1, 11}, {-12, 12, 1, 10}, {-10, 8, 1, 9}, {-6, 4, 1, 8}, {-4, 8, 1, 7}, {-2, 12, 1, 6},
     {0, 16, 1, 5}, {2, 16, -1, 5}, {4, 12, -1, 6}, {6, 8, -1, 7}, {10, 4, -1, 8}, {12, 8, -1, 9},
     {14, 12, -1, 10}, {kInf, 16, -1, 11}, {kInf, 0, 0, 0}},
    {{-14, 8, 1, 13}, {-10, 4, 1, 12}, {-8, 8, 1, 11}, {-6, 8, -1, -5}, {-2, 4, -1, -4}, {0, 8, -1, -3},
     {2, 8, 1, -3}, {6, 4, 1, -4}, {8, 8, 1, -5}, {10, 8, -1, 11}, {14, 4, -1, 12}, {kInf, 8, -1, 13},
     {kInf, 0, 0, 0}, {kInf, 0, 0, 0}, {kInf, 0, 0, 0}},
    {{-12, 4, 1, 14}, {-8, 4, -1, -10}, {-4, 4, 1, 6}, {0, 4, -1, -2}, {4, 4, 1, -2}, {8, 4, -1, 6},
     {12, 4, 1, -10}, {kInf, 4, -1, 14}, {kInf, 0, 0, 0}, {kInf, 0, 0, 0}, {kInf, 0, 0, 0}, {kInf, 0, 0, 0},
     {kInf, 0, 0, 0}, {kInf, 0, 0, 0}, {kInf, 0, 0, 0}},
};
__constant__ int kQam256N[4] = {15, 14, 12, 8};

// x / nv, correctly rounded, from r = RN(1 / nv) by two remainder steps
// (Markstein's theorem: with a correctly rounded reciprocal and a quotient
// within an ulp, q + r (x - q nv) in fused operations rounds correctly).  The
// host asks for it only where neither the reciprocal nor a remainder can leave
// the normal range.
__device__ __forceinline__ float div_nv(float x, float nv, float r) {
  float q = __fmul_rn(x, r);
  q = __fmaf_rn(__fmaf_rn(-q, nv, x), r, q);
  return __fmaf_rn(__fmaf_rn(-q, nv, x), r, q);
}

__device__ __forceinline__ int16_t quantize(float llr) {
  const float scaled = __fmul_rn(llr, 128.0f);
  int32_t q = (int32_t)(scaled >= 0.0f ? __fadd_rn(scaled, 0.5f) : __fsub_rn(scaled, 0.5f));
  q = q > 10000 ? 10000 : (q < -10000 ? -10000 : q);
  return (int16_t)q;
}

__device__ __forceinline__ uint64_t splitmix(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// PAM cell of r for 2^m levels spaced 2A: the number of boundaries
// (2 c - 2^m) A, c = 1 .. 2^m - 1, that r is not below.  The cell is the floor of
// r / 2A + 2^(m-1), held a quarter away from the ends of the range (a NaN gives
// cell 0); that estimate is within 1e-5 of the exact quotient, so only
// one within 1e-4 of an integer needs the boundaries themselves.
template <int m>
__device__ __forceinline__ int pam_cell(float r, float A, float inv_2a) {
  constexpr int n = 1 << m;
  const float x = fminf(fmaxf(__fmaf_rn(r, inv_2a, (float)(n / 2)), 0.25f), (float)n - 0.25f);
  const float t = __fadd_rz(x, 8388608.0f);   // 2^23 + floor(x): the floor in the low mantissa bits
  int c = (int)(__float_as_uint(t) & (uint32_t)(n - 1));
  const float d = x - (t - 8388608.0f);
  if (fabsf(d - 0.5f) > 0.4999f) {
    if (c > 0 && r < __fmul_rn((float)(2 * c - n), A)) {
      --c;
    } else if (c < n - 1 && !(r < __fmul_rn((float)(2 * c + 2 - n), A))) {
      ++c;
    }
  }
  return c;
}

// Two quantised LLRs in one word, from scaled = 128 LLR (finite): the integer part
// of |scaled| + 0.5, at most 10000, taken from the mantissa after a truncating
// add of 2^23, and the signs applied to both halves at once.
__device__ __forceinline__ uint32_t quantize_pair(float s0, float s1) {
  const float n0 = __fadd_rz(fminf(__fadd_rn(fabsf(s0), 0.5f), 10000.5f), 8388608.0f);
  const float n1 = __fadd_rz(fminf(__fadd_rn(fabsf(s1), 0.5f), 10000.5f), 8388608.0f);
  const uint32_t n = __byte_perm(__float_as_uint(n0), __float_as_uint(n1), 0x5410);
  uint32_t neg;   // all ones in the half of a negative value
  asm("prmt.b32 %0, %1, %2, 0xFFBB;" : "=r"(neg) : "r"(__float_as_uint(s0)), "r"(__float_as_uint(s1)));
  return __vadd2(n ^ neg, neg & 0x00010001u);
}

// 128 x / nv.  Scaling by a power of two commutes with the rounding of the
// division, so the fast form divides 128 x.
template <bool kFast>
__device__ __forceinline__ uint32_t llr_pair(float x0, float x1, float nv, float rnv) {
  if constexpr (kFast) {
    return quantize_pair(div_nv(x0, nv, rnv), div_nv(x1, nv, rnv));
  } else {
    return (uint32_t)(uint16_t)quantize(__fdiv_rn(x0, nv)) | (uint32_t)(uint16_t)quantize(__fdiv_rn(x1, nv)) << 16;
  }
}

// Constellation point of the Qm bits in the low bits of w, first bit on top, by
// the reference's float expressions.
template <int Qm>
__device__ __forceinline__ float2 map_symbol(uint32_t w, float A) {
  const auto sign = [&](int j) { return (w >> (Qm - 1 - j)) & 1u ? -1.0f : 1.0f; };   // 1 - 2 b_j
  float re, im;
  if constexpr (Qm == 1) {
    re = im = __fmul_rn(sign(0), A);
  } else if constexpr (Qm == 2) {
    re = __fmul_rn(sign(0), A);
    im = __fmul_rn(sign(1), A);
  } else if constexpr (Qm == 4) {
    re = __fmul_rn(__fmul_rn(sign(0), __fsub_rn(2.0f, sign(2))), A);
    im = __fmul_rn(__fmul_rn(sign(1), __fsub_rn(2.0f, sign(3))), A);
  } else if constexpr (Qm == 6) {
    re = __fmul_rn(__fmul_rn(sign(0), __fsub_rn(4.0f, __fmul_rn(sign(2), __fsub_rn(2.0f, sign(4))))), A);
    im = __fmul_rn(__fmul_rn(sign(1), __fsub_rn(4.0f, __fmul_rn(sign(3), __fsub_rn(2.0f, sign(5))))), A);
  } else {
    re = __fmul_rn(__fmul_rn(sign(0), __fsub_rn(8.0f, __fmul_rn(sign(2), __fsub_rn(4.0f,
                   __fmul_rn(sign(4), __fsub_rn(2.0f, sign(6))))))), A);
    im = __fmul_rn(__fmul_rn(sign(1), __fsub_rn(8.0f, __fmul_rn(sign(3), __fsub_rn(4.0f,
                   __fmul_rn(sign(5), __fsub_rn(2.0f, sign(7))))))), A);
  }
  return make_float2(re, im);
}

constexpr int kChannelThreads = 256;
constexpr int kGroup = 4;   // symbols per thread and step

// One thread takes four consecutive symbols: their 4 Qm bits start on a nibble,
// and their 4 Qm LLRs are one run of 8 Qm bytes, stored in the widest pieces that
// every row's start allows (`align`: bytes; by halves, 2048 x 25338 LLRs, 64QAM, took
// 312 us, and 286 us with one symbol per thread; 94 us in words, 86 us where rows are
// 16-byte aligned).  The symbol's point and every pair's max-log line
// come from shared tables, the line by the PAM cell of the coordinate (one cell
// per coordinate serves all Qm / 2 pairs); the line's 8-byte entries, at most 16
// per pair, conflict for no lane pattern.  The division by the noise power, the
// same for every LLR, is a multiplication and two remainder steps, and nothing is
// converted on the slow conversion pipe.  Bound by instruction issue: the counter
// generator's four 64-bit products, logf, sqrtf and sincospif per symbol take half
// of it, then 13 instructions per LLR.
// 2048 x 25344 LLRs, 64QAM: 286 us with one symbol per thread, a search of the
// segments in constant memory and 2-byte stores; 107 us with the tables for the
// lines alone; 84 us in this form.
template <int Qm, bool kFast>
__global__ void __launch_bounds__(kChannelThreads) channel_kernel(const uint8_t* __restrict__ rm, int64_t rm_stride, int32_t num_cw, int32_t E,
                               float nv, float sigma, float A, uint64_t seed,
                               int16_t* __restrict__ llr, int64_t llr_stride, float* __restrict__ symbols, int align) {
  constexpr int m = Qm > 2 ? Qm / 2 : 1, kCells = 1 << m;
  constexpr float kScale = kFast ? 128.0f : 1.0f;   // the fast form divides 128 x (llr_pair)
  // per pair and cell: s c1 A (scaled) and c2 A of the line (c1 A) (s r + c2 A); c1 A > 0
  __shared__ float2 s_line[m][kCells];
  __shared__ float2 s_point[1 << Qm];   // constellation
  if constexpr (Qm > 2) {
    for (int k = threadIdx.x; k < m * kCells; k += blockDim.x) {
      const int p = k / kCells, c = k - p * kCells;
      const Seg* seg = Qm == 4 ? kQam16[p & 1] : Qm == 6 ? kQam64[p % 3] : kQam256[p & 3];
      const int n = Qm == 4 ? kQam16N[p & 1] : Qm == 6 ? kQam64N[p % 3] : kQam256N[p & 3];
      int j = 0;
      while (j < n - 1 && seg[j].thr <= (float)(2 * c - kCells)) ++j;   // segments the cell lies above
      s_line[p][c] = make_float2(copysignf(__fmul_rn(__fmul_rn(seg[j].c1, A), kScale), seg[j].s), __fmul_rn(seg[j].c2, A));
    }
  }
  for (int k = threadIdx.x; k < (1 << Qm); k += blockDim.x) s_point[k] = map_symbol<Qm>((uint32_t)k, A);
  __syncthreads();
  const float rnv = kFast ? __frcp_rn(nv) : 0.0f;
  const float inv_2a = 0.5f / A;
  const uint32_t nsym = (uint32_t)(E / Qm);
  const uint32_t groups = (nsym + kGroup - 1) / kGroup;
  const uint64_t total = (uint64_t)groups * (uint64_t)num_cw;
  for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < total; g += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t cw = total <= 0xFFFFFFFFull ? (uint32_t)g / groups : (uint32_t)(g / groups);
    const uint32_t gi = (uint32_t)(g - (uint64_t)cw * groups);
    const uint32_t s0 = gi * kGroup;
    const uint32_t left = min((uint32_t)kGroup, nsym - s0);
    // the group's 4 Qm bits, first bit on top (bits past E are not used)
    uint32_t word = 0u;
    {
      const uint8_t* in = rm + (int64_t)cw * rm_stride;
      const uint32_t byte0 = (uint32_t)(((uint64_t)s0 * Qm) >> 3);
      const uint32_t nbytes = (uint32_t)(((uint64_t)E + 7) >> 3);
#pragma unroll
      for (int j = 0; j < (4 * Qm + 7) / 8; ++j)
        if (byte0 + j < nbytes) word |= (uint32_t)__ldg(in + byte0 + j) << (24 - 8 * j);
      if (Qm == 1 && (gi & 1u)) word <<= 4;
    }
    uint32_t q[2 * Qm];   // 4 Qm int16 LLRs
#pragma unroll
    for (int i = 0; i < kGroup; ++i) {
      const float2 point = s_point[(word >> (32 - (i + 1) * Qm)) & ((1u << Qm) - 1u)];
      // Box-Muller from a counter-based generator.
      const uint64_t z = splitmix(seed ^ splitmix(((uint64_t)cw << 32) ^ (uint64_t)(s0 + i)));
      const float u1 = ((float)(z >> 40) + 1.0f) * (1.0f / 16777218.0f);
      const float u2 = ((float)((z >> 16) & 0xFFFFFFu) + 1.0f) * (1.0f / 16777218.0f);
      const float rad = sqrtf(-2.0f * logf(u1));
      float sn, cs;
      sincospif(2.0f * u2, &sn, &cs);
      const float re = __fadd_rn(point.x, __fmul_rn(sigma, __fmul_rn(rad, cs)));
      const float im = __fadd_rn(point.y, __fmul_rn(sigma, __fmul_rn(rad, sn)));
      if (symbols && (uint32_t)i < left) {
        float* o = symbols + 2 * ((int64_t)cw * nsym + s0 + i);
        o[0] = re;
        o[1] = im;
      }
      if constexpr (Qm == 1) {
        const float x = __fmul_rn(__fmul_rn(__fmul_rn(4.0f, __fadd_rn(re, im)), A), kScale);
        const uint32_t v = llr_pair<kFast>(x, x, nv, rnv);
        q[i >> 1] = i & 1 ? (q[i >> 1] & 0xFFFFu) | (v & 0xFFFF0000u) : v;
      } else if constexpr (Qm == 2) {
        q[i] = llr_pair<kFast>(__fmul_rn(__fmul_rn(__fmul_rn(4.0f, re), A), kScale),
                               __fmul_rn(__fmul_rn(__fmul_rn(4.0f, im), A), kScale), nv, rnv);
      } else {
        const int cr = pam_cell<m>(re, A, inv_2a), ci = pam_cell<m>(im, A, inv_2a);
        // (c1 A) (s r + c2 A): the sign of the table's first entry is s
        const auto line = [](float2 l, float r) {
          const float sr = __uint_as_float(__float_as_uint(r) ^ (__float_as_uint(l.x) & 0x80000000u));
          return __fmul_rn(fabsf(l.x), __fadd_rn(sr, l.y));
        };
#pragma unroll
        for (int p = 0; p < m; ++p)
          q[i * m + p] = llr_pair<kFast>(line(s_line[p][cr], re), line(s_line[p][ci], im), nv, rnv);
      }
    }
    int16_t* out = llr + (int64_t)cw * llr_stride + (int64_t)s0 * Qm;
    if (align >= 16 && Qm > 1 && left == kGroup) {
#pragma unroll
      for (int k = 0; k < Qm / 2; ++k)
        reinterpret_cast<uint4*>(out)[k] = make_uint4(q[4 * k], q[4 * k + 1], q[4 * k + 2], q[4 * k + 3]);
    } else if (align >= 8 && left == kGroup) {
#pragma unroll
      for (int k = 0; k < Qm; ++k) reinterpret_cast<uint2*>(out)[k] = make_uint2(q[2 * k], q[2 * k + 1]);
    } else if (left == kGroup && (reinterpret_cast<uintptr_t>(out) & 2u) == 0u) {
#pragma unroll
      for (int k = 0; k < 2 * Qm; ++k) reinterpret_cast<uint32_t*>(out)[k] = q[k];
    } else if (left == kGroup) {   // halfway between words
      out[0] = (int16_t)q[0];
#pragma unroll
      for (int k = 0; k < 2 * Qm - 1; ++k) reinterpret_cast<uint32_t*>(out + 1)[k] = __byte_perm(q[k], q[k + 1], 0x5432);
      out[4 * Qm - 1] = (int16_t)(q[2 * Qm - 1] >> 16);
    } else {
#pragma unroll
      for (int k = 0; k < kGroup * Qm; ++k)
        if ((uint32_t)k < left * Qm) out[k] = (int16_t)(q[k >> 1] >> (16 * (k & 1)));
    }
  }
}

template <int Qm>
void launch_channel_qm(bool fast, int grid, cudaStream_t s, const uint8_t* rm, int64_t rm_stride, int32_t num_cw,
                       int32_t E, float nv, float sigma, float A, uint64_t seed, int16_t* llr, int64_t llr_stride,
                       float* symbols, int align) {
  if (fast)
    channel_kernel<Qm, true><<<grid, kChannelThreads, 0, s>>>(rm, rm_stride, num_cw, E, nv, sigma, A, seed, llr,
                                                              llr_stride, symbols, align);
  else
    channel_kernel<Qm, false><<<grid, kChannelThreads, 0, s>>>(rm, rm_stride, num_cw, E, nv, sigma, A, seed, llr,
                                                               llr_stride, symbols, align);
}

}  // namespace

int launch_channel(const uint8_t* rm, int64_t rm_stride, int32_t num_cw, int32_t E, int32_t Qm, float nv,
                   float sigma, float A, uint64_t seed, int16_t* llr, int64_t llr_stride, float* symbols,
                   void* stream) {
  const int64_t groups = ((int64_t)(E / Qm) + kGroup - 1) / kGroup;
  const int64_t total = groups * num_cw;
  if (total == 0) return 0;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t want = (total + kChannelThreads - 1) / kChannelThreads;
  const int grid = (int)(want < 16LL * sms ? want : 16LL * sms);
  // Remainder-step division: with nv in this range the reciprocal is normal,
  // quotients of the coordinates' magnitudes (below 2^32) stay finite, and the
  // remainder of any quotient that does not quantise to 0 is normal.
  const bool fast = nv > 0x1p-60f && nv < 0x1p60f;
  // largest power of two up to 16 that divides every row's address
  const uintptr_t low = reinterpret_cast<uintptr_t>(llr) | (num_cw > 1 ? (uintptr_t)(llr_stride * 2) : 0u) | 16u;
  const int align = (int)(low & (0u - low));
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  switch (Qm) {
    case 1: launch_channel_qm<1>(fast, grid, s, rm, rm_stride, num_cw, E, nv, sigma, A, seed, llr, llr_stride, symbols, align); break;
    case 2: launch_channel_qm<2>(fast, grid, s, rm, rm_stride, num_cw, E, nv, sigma, A, seed, llr, llr_stride, symbols, align); break;
    case 4: launch_channel_qm<4>(fast, grid, s, rm, rm_stride, num_cw, E, nv, sigma, A, seed, llr, llr_stride, symbols, align); break;
    case 6: launch_channel_qm<6>(fast, grid, s, rm, rm_stride, num_cw, E, nv, sigma, A, seed, llr, llr_stride, symbols, align); break;
    default: launch_channel_qm<8>(fast, grid, s, rm, rm_stride, num_cw, E, nv, sigma, A, seed, llr, llr_stride, symbols, align); break;
  }
  count_launch();
  return (int)cudaGetLastError();
}

}  // namespace nrldpc
