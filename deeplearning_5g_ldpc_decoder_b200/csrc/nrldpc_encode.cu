// nrldpc_encode.cu — batched 5G NR LDPC encoder + rate matching for sm_100a.
//
// Restates the reference's transmit chain (c_lib/c_ldpc_5g_encoder.c:66-88):
//  * CRC attach (calculate_crc over A/8 payload bytes, MSB first),
//  * QC-LDPC encoding (c_lib/ldpc_encoder.c:52-242): syndromes of the first
//    four base-graph rows over the systematic part, the double-diagonal core
//    parity solve (pc0 from the summed syndromes through the I2 / I4
//    circulant, pc1/pc3 through I1 / I3, pc2 from row 2 / row 1), then every
//    extension row's parity as a plain XOR over systematic + core columns,
//  * bit selection from k0 over the circular buffer without filler bits and
//    the Qm row/column interleave, packed MSB first
//    (c_lib/ldpc_rate_match.c:27-106).
//
// One CTA per code block, 32 bits per word throughout (bit i of a bit string
// in bit i mod 32 of word i / 32):
//  * A base column of the systematic and core parts is kept twice in a row
//    (2 Zc bits), so a circulant is one funnel shift per 32 rows: word w of
//    column c shifted by s starts at bit s + 32 w of the doubled column.
//  * Parity words are ORed into the compacted circular buffer (no punctured
//    columns, no filler) at their bit position; rate matching then reads the
//    Qm interleaved streams as 32-bit windows of that buffer.
//  * 32 symbols are interleaved at once: an 8 x 8 bit transpose per 8 symbols
//    gives one byte per symbol, and Qm < 8 packs the bytes' top Qm bits.
// The kernel is bound by instruction issue (about 8000 warp instructions for a
// BG1 Zc=384 block, 64 % of the issue slots; leaving out the CRC saves 15 % of the
// time, the interleave 16 %, the extension rows 11 %) and, for one block, by the
// latency of its eight phases.  4096 blocks of BG1 Zc=384, E=25344, Qm=8: 783 us with
// one byte per bit and a gather per output bit, 47 us in this form.
#include <cuda_runtime.h>
#include <stdint.h>

#include "nrldpc_internal.h"

namespace nrldpc {

namespace {

constexpr int kEncThreads = 128;
constexpr int kEncCols = 26;                                   // systematic + core columns of BG1
constexpr int kEncDoubled = (2 * kMaxZc + 31) / 32 + 1;        // words of a doubled column
constexpr int kEncZcWords = kMaxZc / 32;

// 32 bits of the bit string a from bit pos.
__device__ __forceinline__ uint32_t bits32(const uint32_t* a, uint32_t pos) {
  const uint32_t w = pos >> 5;
  return __funnelshift_r(a[w], a[w + 1], pos & 31u);
}
// 32 bits of the Zc-bit cyclic string at bit `base` of a, from start < Zc.  Only
// the first 2 Zc - start of them are meaningful when Zc < 32.
__device__ __forceinline__ uint32_t cyclic32(const uint32_t* a, uint32_t base, uint32_t Zc, uint32_t start) {
  uint32_t v = bits32(a, base + start);
  const uint32_t n = Zc - start;
  if (n < 32u) v = (v & ((1u << n) - 1u)) | (bits32(a, base) << n);
  return v;
}
// 32 bits of the cyclic buffer of Nv bits from position c < Nv.
__device__ __forceinline__ uint32_t window32(const uint32_t* a, uint32_t Nv, uint32_t c) {
  uint32_t n = Nv - c;
  uint32_t v = bits32(a, c);
  while (n < 32u) {   // wraps: append the buffer from its start (more than once if it is short)
    v = (v & ((1u << n) - 1u)) | (bits32(a, 0u) << n);
    n += Nv;
  }
  return v;
}

// 32-bit little-endian word k of a row of `len` bytes (bytes past the end are zero).
__device__ __forceinline__ uint32_t row_word(const uint8_t* row, int k, int len, bool vec) {
  if (vec && 4 * k + 4 <= len) return __ldg(reinterpret_cast<const uint32_t*>(row) + k);
  uint32_t v = 0u;
  for (int b = 0; b < 4; ++b)
    if (4 * k + b < len) v |= (uint32_t)__ldg(row + 4 * k + b) << (8 * b);
  return v;
}

// One 8 x 8 bit transpose: byte j (from the top) of x:y becomes the bits
// 7 - j of the eight input bytes, first byte's bit on top (Hacker's Delight,
// transpose8).
__device__ __forceinline__ void transpose8(uint32_t& x, uint32_t& y) {
  uint32_t t = (x ^ (x >> 7)) & 0x00AA00AAu;
  x ^= t ^ (t << 7);
  t = (y ^ (y >> 7)) & 0x00AA00AAu;
  y ^= t ^ (t << 7);
  t = (x ^ (x >> 14)) & 0x0000CCCCu;
  x ^= t ^ (t << 14);
  t = (y ^ (y >> 14)) & 0x0000CCCCu;
  y ^= t ^ (t << 14);
  t = (x & 0xF0F0F0F0u) | ((y >> 4) & 0x0F0F0F0Fu);
  y = ((x << 4) & 0xF0F0F0F0u) | (y & 0x0F0F0F0Fu);
  x = t;
}

// Top Qm bits of the four bytes of t, concatenated from the top of the word.
template <int Qm>
__device__ __forceinline__ uint32_t pack_symbols(uint32_t t) {
  if constexpr (Qm == 8) return t;
  constexpr uint32_t m = (0xFFu << (8 - Qm)) & 0xFFu;
  const uint32_t u = (t & (m * 0x01000100u)) | ((t & (m * 0x00010001u)) << (8 - Qm));   // 2 Qm bits per half
  constexpr uint32_t h = (0xFFFFu << (16 - 2 * Qm)) & 0xFFFFu;
  return (u & (h << 16)) | ((u & h) << (16 - 2 * Qm));
}

// Rate-matched bytes of one block from its compacted circular buffer: 32 symbols
// (Qm words) per thread and step.
// stream[b]: buffer position of bit 0 of stream b.
template <int Qm>
__device__ __forceinline__ void rate_match(const EncodeParams& p, const uint32_t* comp, const uint32_t* stream, uint8_t* out,
                                           bool vec) {
  const int nbytes = (p.E + 7) >> 3;
  for (int s0 = 32 * threadIdx.x; s0 < p.symbols; s0 += 32 * blockDim.x) {
    const int left = p.symbols - s0;
    uint32_t v[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      v[b] = 0u;
      if (b < Qm) {
        uint32_t c = stream[b] + (uint32_t)s0;
        if (c >= (uint32_t)p.Nv) {
          c -= (uint32_t)p.Nv;
          if (c >= (uint32_t)p.Nv) c %= (uint32_t)p.Nv;   // E beyond the buffer: repetition
        }
        v[b] = window32(comp, (uint32_t)p.Nv, c);
        if (left < 32) v[b] &= (1u << left) - 1u;
        v[b] = __brev(v[b]);   // symbol s0 on top
      }
    }
    uint32_t o[8];
    if constexpr (Qm == 1) {
      o[0] = v[0];
    } else {
      uint32_t piece[8];   // four symbols each
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const uint32_t sel = half ? 0x5140u : 0x7362u;   // low / high two bytes of each pair
        const uint32_t a = __byte_perm(v[1], v[0], sel), b = __byte_perm(v[3], v[2], sel);
        const uint32_t c = __byte_perm(v[5], v[4], sel), d = __byte_perm(v[7], v[6], sel);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t x = __byte_perm(b, a, q ? 0x5410u : 0x7632u);
          uint32_t y = __byte_perm(d, c, q ? 0x5410u : 0x7632u);
          transpose8(x, y);
          piece[4 * half + 2 * q] = pack_symbols<Qm>(x);
          piece[4 * half + 2 * q + 1] = pack_symbols<Qm>(y);
        }
      }
      // pieces of 4 Qm bits -> Qm words
      if constexpr (Qm == 8) {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = piece[j];
      } else if constexpr (Qm == 6) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t* q = piece + 4 * j;
          o[3 * j] = q[0] | (q[1] >> 24);
          o[3 * j + 1] = (q[1] << 8) | (q[2] >> 16);
          o[3 * j + 2] = (q[2] << 16) | (q[3] >> 8);
        }
      } else if constexpr (Qm == 4) {
#pragma unroll
        for (int j = 0; j < 4; ++j) o[j] = piece[2 * j] | (piece[2 * j + 1] >> 16);
      } else {
#pragma unroll
        for (int j = 0; j < 2; ++j)
          o[j] = piece[4 * j] | (piece[4 * j + 1] >> 8) | (piece[4 * j + 2] >> 16) | (piece[4 * j + 3] >> 24);
      }
    }
    const int byte0 = (s0 >> 3) * Qm;
#pragma unroll
    for (int j = 0; j < Qm; ++j) {
      const int y = byte0 + 4 * j;
      if (vec && y + 4 <= nbytes) {
        *reinterpret_cast<uint32_t*>(out + y) = __byte_perm(o[j], 0u, 0x0123u);
      } else {
        for (int b = 0; b < 4; ++b)
          if (y + b < nbytes) out[y + b] = (uint8_t)(o[j] >> (24 - 8 * b));
      }
    }
  }
}

__global__ void __launch_bounds__(kEncThreads, 12) encode_kernel(const __grid_constant__ EncodeParams p) {
  __shared__ uint32_t s_lin[(kMaxB + 31) / 32 + 3];            // K systematic bits: payload, CRC, filler zeros
  __shared__ uint32_t s_col[kEncCols * kEncDoubled + 2];       // doubled columns, W2 words each (and two read past the last)
  __shared__ uint32_t s_comp[(66 * kMaxZc + 31) / 32 + 4];     // compacted circular buffer
  __shared__ uint32_t s_par[4][kEncZcWords + 2];               // core parities, Zc bits each
  __shared__ uint32_t s_L[4][kEncZcWords + 2];                 // syndromes, then [0]: their sum
  __shared__ uint32_t s_sum[kEncZcWords + 2];
  __shared__ uint32_t s_edge[kMaxNnz];                         // word offset in s_col | bit shift << 16
  __shared__ uint16_t s_off[kMaxRows + 1];
  __shared__ uint32_t s_stream[8];
  __shared__ uint32_t s_crc;
  const int tid = threadIdx.x, nt = blockDim.x;
  const uint32_t Zc = (uint32_t)p.Zc;
  const int W = (p.Zc + 31) >> 5;
  const int W2 = p.W2;
  const uint32_t last = (Zc & 31u) ? (1u << (Zc & 31u)) - 1u : 0xFFFFFFFFu;   // valid bits of a column's last word
  const int info_bits = p.B - 2 * p.Zc;                        // systematic bits of the circular buffer
  const int info_words = (info_bits + 31) >> 5;
  const int comp_words = ((info_bits + p.R * p.Zc + 31) >> 5) + 3;
  const int lin_words = ((p.K + 31) >> 5) + 2;
  const uint32_t mul_w2 = 65536u / (uint32_t)W2 + 1u, mul_w = 65536u / (uint32_t)W + 1u;
  const uint32_t mul_w1 = 65536u / (uint32_t)((W + 1) >> 1) + 1u;   // exact for the small indices below
  for (int e = tid; e < p.num_edges; e += nt) s_edge[e] = p.edge[e];
  for (int r = tid; r <= p.R; r += nt) s_off[r] = p.row_off[r];
  // stream b of the interleave starts at de-interleaved bit b (E / Qm)
  if (tid < p.Qm) s_stream[tid] = (uint32_t)(p.c0 + tid * p.symbols) % (uint32_t)p.Nv;
  const bool whole = (p.Zc & 31) == 0;   // columns are whole words: no shifts where they are only copied

  for (int cw = blockIdx.x; cw < p.num_cw; cw += gridDim.x) {
    const uint8_t* info = p.info + (int64_t)cw * p.info_stride;
    if (tid == 0) s_crc = 0u;
    for (int k = tid; k < lin_words; k += nt)
      s_lin[k] = __byte_perm(__brev(row_word(info, k, p.A >> 3, p.info_vec != 0)), 0u, 0x0123u);
    for (int k = info_words + tid; k < comp_words; k += nt) s_comp[k] = 0u;
    for (int k = tid; k < 4 * (kEncZcWords + 2); k += nt) {
      s_L[0][k] = 0u;
      s_par[0][k] = 0u;
    }
    for (int k = tid; k < kEncZcWords + 2; k += nt) s_sum[k] = 0u;
    __syncthreads();
    // CRC remainder sum_i bit_i x^(A-1-i+W) mod g(x), four bits and one 16-byte
    // table load per step (A is a multiple of 8).
    {
      uint32_t r = 0u;
      for (int i0 = 4 * tid; i0 < p.A; i0 += 4 * nt) {
        const uint32_t w = s_lin[i0 >> 5] >> (i0 & 31);
        const uint4 t = __ldg(reinterpret_cast<const uint4*>(p.crc_tab + (p.A - 4 - i0)));
        r ^= ((0u - (w & 1u)) & t.w) ^ ((0u - ((w >> 1) & 1u)) & t.z) ^ ((0u - ((w >> 2) & 1u)) & t.y) ^
             ((0u - ((w >> 3) & 1u)) & t.x);
      }
      r = __reduce_xor_sync(0xFFFFFFFFu, r);
      if ((tid & 31) == 0 && r) atomicXor(&s_crc, r);
    }
    __syncthreads();
    if (tid == 0) {
      const int L = p.B - p.A;
      const uint32_t rc = __brev(s_crc) >> (32 - L);           // first CRC bit in bit 0
      const int sh = p.A & 31;
      s_lin[p.A >> 5] |= rc << sh;
      if (sh + L > 32) s_lin[(p.A >> 5) + 1] |= rc >> (32 - sh);
    }
    __syncthreads();
    // Doubled systematic columns, and the systematic part of the circular buffer.
    for (int k = tid; k < p.Kb * W2; k += nt) {
      const uint32_t c = ((uint32_t)k * mul_w2) >> 16;
      if (whole) {
        int w = k - (int)c * W2;
        w -= w >= W ? W : 0;
        w -= w >= W ? W : 0;   // the word after the second copy
        s_col[k] = s_lin[(int)c * W + w];
        continue;
      }
      uint32_t start = 32u * ((uint32_t)k - c * (uint32_t)W2);
      while (start >= Zc) start -= Zc;
      s_col[k] = cyclic32(s_lin, c * Zc, Zc, start);
    }
    for (int k = tid; k < info_words; k += nt) {
      uint32_t v = bits32(s_lin, 2u * Zc + 32u * (uint32_t)k);
      const int n = info_bits - 32 * k;
      if (n < 32) v &= (1u << n) - 1u;
      s_comp[k] = v;
    }
    __syncthreads();
    // Syndromes of rows 0..3 over the systematic columns, each row's edges split
    // over `parts` threads.
    {
      const int parts = max(1, min(4, nt / (4 * W)));
      for (int k = tid; k < 4 * W * parts; k += nt) {
        const int q = k / (4 * W), rw = k - q * 4 * W;
        const int r = (int)(((uint32_t)rw * mul_w) >> 16), w = rw - r * W;
        uint32_t s = 0u;
        for (int e = s_off[r] + q; e < s_off[r + 1]; e += parts) {
          const uint32_t ed = s_edge[e];
          const uint32_t* a = s_col + (ed & 0xFFFFu) + w;
          s ^= __funnelshift_r(a[0], a[1], ed >> 16);
        }
        if (w == W - 1) s &= last;
        atomicXor(&s_L[r][w], s);
      }
    }
    __syncthreads();
    if (tid < 32) {   // core parities: at most 12 words, one warp
      const bool on = tid < W;
      const uint32_t m = tid == W - 1 ? last : 0xFFFFFFFFu;
      uint32_t l0 = 0u, l1 = 0u, l2 = 0u, l3 = 0u;
      if (on) {
        l0 = s_L[0][tid];
        l1 = s_L[1][tid];
        l2 = s_L[2][tid];
        l3 = s_L[3][tid];
        s_sum[tid] = l0 ^ l1 ^ l2 ^ l3;
      }
      __syncwarp();
      uint32_t start = 32u * (uint32_t)tid + Zc - (uint32_t)p.shift1;   // pc0: I2^-1 / I4^-1 applied to the sum
      if (start >= Zc) start -= Zc;
      if (on) s_par[0][tid] = cyclic32(s_sum, 0u, Zc, start) & m;
      __syncwarp();
      start = 32u * (uint32_t)tid + (uint32_t)p.shift0;
      if (start >= Zc) start -= Zc;
      if (on) {
        const uint32_t t = cyclic32(s_par[0], 0u, Zc, start) & m;
        const uint32_t pc1 = l0 ^ t, pc3 = l3 ^ t;
        s_par[1][tid] = pc1;
        s_par[3][tid] = pc3;
        s_par[2][tid] = p.bgn == 1 ? l2 ^ pc3 : l1 ^ pc1;
      }
    }
    __syncthreads();
    for (int k = tid; k < 4 * W2; k += nt) {
      const uint32_t c = ((uint32_t)k * mul_w2) >> 16;
      uint32_t start = 32u * ((uint32_t)k - c * (uint32_t)W2);
      while (start >= Zc) start -= Zc;
      s_col[p.Kb * W2 + k] = cyclic32(s_par[c], 0u, Zc, start);
    }
    __syncthreads();
    // Every row's parity words: rows 0..3 are solved, an extension row is the XOR
    // over its systematic + core columns.  Two words per thread share an edge's
    // record and the word between them.
    const int W1 = (W + 1) >> 1;
    for (int k = tid; k < p.R * W1; k += nt) {
      const int r = (int)(((uint32_t)k * mul_w1) >> 16), w = 2 * (k - r * W1);
      uint32_t s0 = 0u, s1 = 0u;
      if (r < 4) {
        s0 = s_par[r][w];
        s1 = s_par[r][w + 1];
      } else {
        const int e1 = s_off[r + 1];
#pragma unroll 2
        for (int e = s_off[r]; e < e1; ++e) {
          const uint32_t ed = s_edge[e];
          const uint32_t* a = s_col + (ed & 0xFFFFu) + w;
          const uint32_t mid = a[1];
          s0 ^= __funnelshift_r(a[0], mid, ed >> 16);
          s1 ^= __funnelshift_r(mid, a[2], ed >> 16);   // (unused past the last word)
        }
        if (w == W - 1) s0 &= last;
        if (w + 1 == W - 1) s1 &= last;
      }
      if (w + 1 >= W) s1 = 0u;
      const uint32_t pos = (uint32_t)(info_bits + r * p.Zc + 32 * w), sh = pos & 31u;
      uint32_t* d = s_comp + (pos >> 5);
      atomicOr(d, s0 << sh);
      const uint32_t carry = __funnelshift_l(s0, s1, sh);   // s1 << sh | s0 >> (32 - sh)
      if (carry) atomicOr(d + 1, carry);
      const uint32_t top = sh ? s1 >> (32u - sh) : 0u;
      if (top) atomicOr(d + 2, top);
    }
    __syncthreads();
    uint8_t* out = p.rm + (int64_t)cw * p.rm_stride;
    switch (p.Qm) {
      case 1: rate_match<1>(p, s_comp, s_stream, out, p.rm_vec != 0); break;
      case 2: rate_match<2>(p, s_comp, s_stream, out, p.rm_vec != 0); break;
      case 4: rate_match<4>(p, s_comp, s_stream, out, p.rm_vec != 0); break;
      case 6: rate_match<6>(p, s_comp, s_stream, out, p.rm_vec != 0); break;
      default: rate_match<8>(p, s_comp, s_stream, out, p.rm_vec != 0); break;
    }
    __syncthreads();   // the shared arrays are reused by the next block
  }
}

}  // namespace

int launch_encode(const EncodeParams& p, int num_sms, void* stream) {
  // 16 CTAs of 128 threads fill an SM's 2048 threads
  const int grid = p.num_cw < 16 * num_sms ? p.num_cw : 16 * num_sms;
  encode_kernel<<<grid, kEncThreads, 0, reinterpret_cast<cudaStream_t>(stream)>>>(p);
  count_launch();
  return (int)cudaGetLastError();
}

}  // namespace nrldpc
