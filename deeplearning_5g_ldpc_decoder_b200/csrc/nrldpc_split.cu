// nrldpc_split.cu — fixed-point layered min-sum decoder (algos 1, 2, 3) for
// batches too small to fill the GPU: one code block per CTA, each lifted check
// row split over four or eight lanes.
//
// Bit-exact with c_lib/fixedpoint_ldpc_decoder.c:103-222 like the pair kernel
// (nrldpc_fixed.cu), from which it differs in where the parallelism comes from:
//  * int16x2 words pair rows of ONE block.  With H = Zc / 2, word w of a base
//    column holds its beliefs w (half 0) and w + H (half 1), and a thread's two
//    rows are zx and zx + H.  Both rows of an edge lie in the one word
//    (zx + V) mod H, in this order or the other: a byte permute on load and
//    store.  (An odd Zc, 3 to 15, keeps one belief per word: H = Zc, no permute.)
//  * Four or eight lanes (kLanes) share a row pair's edges: lane l takes edges l,
//    l + kLanes, ...  Minima and sign parity meet in two or three shuffle steps.  The edge that carries
//    the second minimum is found by |rel| == min1 afterwards; at a tie both
//    minima are equal, so marking several edges changes no message.
//  * Two consecutive layers without a common base column touch disjoint beliefs
//    and commute, so two groups of threads take one each in the same step: 32
//    steps instead of 46 layers (BG1), 29 instead of 42 (BG2); no order of the
//    rows that keeps shared columns in sequence has fewer than 32 and 28.
//  * All state is in shared memory: beliefs, and one word per edge for the
//    negated old messages of the two rows (not the pair kernel's compressed
//    form, whose packing and unpacking is a third of its instructions).  Up to
//    the lifting size where it fits, a table holds each thread's edge addresses
//    and permute selectors too; above it they are computed.  A row's addresses
//    and old messages are loaded while the row before it still computes, so
//    only the beliefs' load follows the layer barrier.
//
// A step is one dependent chain of about 140 instructions (four lanes) in each of
// a few warps, 600 to 700 cycles (a thread that walks a whole row takes over 1000
// cycles a layer), so what bounds the kernel is that chain, not a throughput.
// 64 blocks, 8 iterations: BG1 Zc=24 198 us in the pair kernel, 85 us here; BG2 Zc=64
// 133 and 78 us.  Per iteration, when it was written: 11.2 us for BG1 Zc=24, 8.9 for
// BG2 Zc=64, 15.8 for BG1 Zc=112; with one group per step 18.2, 10.7 and 17.8 us; with
// the pair kernel's compressed messages (16 or 32 flag bits per lane) and one group
// 21, 14 and 23 us.  With eight lanes a thread has one edge of a row of up to eight;
// the shuffle step and the warps more cost more than that gives where an SM holds
// many threads (the rule in nrldpc_api.cu).
#include <cuda_runtime.h>
#include <stdint.h>

#include "nrldpc_decode_common.cuh"
#include "nrldpc_fixed_row.cuh"
#include "nrldpc_internal.h"

namespace nrldpc {
namespace {

using namespace fixedrow;

constexpr int kAhead = 3;          // slots per lane loaded a row ahead (degree <= 12 with four lanes, all with eight)
constexpr int kGroupsPerStep = 2;
// Two groups of kLanes H threads: Zc <= 208 or 104 (what fits shared memory may end
// below that).  Larger ones lose to the pair kernel: one block, 8 iterations, four lanes
// / pair kernel BG1 Zc 192 233 / 243 us, 208 260 / 256 us, 224 262 / 245 us, BG2 Zc 208
// 147 / 184 us, 224 200 / 174 us, 256 208 / 176 us.  The launch bound also sets the
// registers: 64 for 1024 threads, 72 for 832 (BG1 Zc 160 219 -> 204 us, BG2 Zc 64 with
// an offset 94 -> 84 us).
constexpr int kSplitThreads = 832;

// Permute selectors: the word as it is, and with its halves swapped.
constexpr uint32_t kStraight = 0x3210u, kSwapBit = 0x2222u;

struct Geometry {
  int H;               // words per base column
  uint32_t h4, swap;   // 4 H; kSwapBit, or 0 where words hold one belief
  uint32_t limit;      // bytes of beliefs, the neutral word included
  uint32_t zc_magic;   // ceil(2^32 / Zc): i / Zc as a high multiply for i < 2^16
};

// 16-bit slot of belief i in the shared beliefs.
__device__ __forceinline__ int slot_of(const Geometry& g, int Zc, int i) {
  const int c = (int)__umulhi((uint32_t)i, g.zc_magic);
  int off = i - c * Zc;
  const int hi = off >= g.H ? 1 : 0;
  off -= hi ? g.H : 0;
  return 2 * (c * g.H + off) + hi;
}

// Where an edge's word lies for a thread, in one word: byte address in the high
// half, permute selector in the low half (prmt reads the low 16 bits only).
// Edge record: {4 H column, 4 (V mod H), selector of V's half, -}.
__device__ __forceinline__ uint32_t locate(const Geometry& g, const uint4& e, uint32_t zx4) {
  const uint32_t a = zx4 + e.y;
  const uint32_t b = a - g.h4;                       // negative: no wrap
  const uint32_t sel = e.z ^ (~(uint32_t)((int32_t)b >> 31) & g.swap);
  return ((min(a, b) + e.x) << 16) | sel;
}

// A row's slots for this thread: where their words lie, and the negated old
// messages.  A lane without an edge in the last slot points at a neutral word
// (32767 in both halves, never stored to) and keeps a zero message.
struct Slots {
  uint32_t at[kAhead], nr[kAhead];
};

// One layer for one thread: K = ceil(degree / kLanes) slots.  Threads that own no rows
// (`active` false) only take part in the shuffles; `tail`: the last slot has an edge.
template <int K, int kLanes, int kClip, typename AtSlot>
__device__ __forceinline__ void split_row(const DecodeParams& p, const Geometry& g, char* __restrict__ lq, const Slots& in,
                                          AtSlot at_slot, uint32_t* __restrict__ msg, int stride, bool active, bool tail, int32_t alpha,
                                          int32_t beta) {
  uint32_t at[K], rel[K], mag[K];
  uint32_t sg = 0u, m1 = 0x7FFF7FFFu, m2 = 0x7FFF7FFFu;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    at[k] = k < kAhead ? in.at[k < kAhead ? k : 0] : at_slot(k);
    const uint32_t addr = at[k] >> 16;
    const uint32_t q = NRLDPC_INBOUNDS(addr, g.limit, kBoundsLq)
                           ? __byte_perm(*reinterpret_cast<const uint32_t*>(lq + addr), 0u, at[k])
                           : 0u;
    const uint32_t x = __vadd2(q, k < kAhead ? in.nr[k < kAhead ? k : 0] : msg[k * stride]);
    const uint32_t a = abs_u16x2(x);
    rel[k] = x;
    mag[k] = a;
    sg ^= x;
    m2 = __vmaxu2(m1, __vminu2(m2, a));
    m1 = __vminu2(m1, a);
  }
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) {
    const uint32_t o1 = __shfl_xor_sync(0xFFFFFFFFu, m1, o);
    const uint32_t o2 = __shfl_xor_sync(0xFFFFFFFFu, m2, o);
    sg ^= __shfl_xor_sync(0xFFFFFFFFu, sg, o);
    m2 = __vminu2(__vmaxu2(m1, o1), __vminu2(m2, o2));
    m1 = __vminu2(m1, o1);
  }
  const uint32_t maxp = ((uint32_t)(uint16_t)p.max_llr) * 0x10001u;
  const uint32_t minp = ((uint32_t)(uint16_t)p.min_llr) * 0x10001u;
  uint32_t s1, s2;
  if constexpr (kClip == kClipOpenMax) {
    s1 = scale_open(m1, alpha);
    s2 = scale_open(m2, alpha);
  } else {
    s1 = scale_pair(__vmins2(m1, maxp), alpha, beta, alpha, beta);
    s2 = scale_pair(__vmins2(m2, maxp), alpha, beta, alpha, beta);
  }
  uint32_t ovf = 0u;
  const uint32_t m_active = active ? 0xFFFFFFFFu : 0u, m_tail = tail ? 0xFFFFFFFFu : 0u;
  uint32_t lr[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint32_t mf = sign_mask(sg ^ rel[k]);
    // per half: 1 unless |rel| is the minimum, then all ones or zero
    const uint32_t ne = __vminu2(mag[k] ^ m1, 0x00010001u) * 0xFFFFu;
    const uint32_t v = bsel(ne, s1, s2);
    lr[k] = __vadd2(v ^ mf, mf & 0x00010001u);      // mf ? -v : v
    uint32_t nq, over = 0u;
    if constexpr (kClip == kClipOpenMax) {
      // v >= 0 here (no offset, no negative alpha), so the sum is taken with the
      // message's sign put on the other operand: w = rel ^ mf, (w + v) ^ mf is
      // rel + message, and it overflows only where w is not negative and w + v
      // is.  8 iterations, 64 blocks: BG1 Zc24 106 -> 103.6 us, BG2 Zc64 85 ->
      // 83.2 us.
      const uint32_t w = rel[k] ^ mf, u = __vadd2(w, v);
      over = u & ~w;
      nq = __vmaxs2(u ^ mf, minp);
    } else if constexpr (kClip == kClipClamp) {
      const uint32_t sum = __vadd2(rel[k], lr[k]);
      over = (sum ^ rel[k]) & ~(rel[k] ^ lr[k]);
      nq = __vmins2(__vmaxs2(sum, minp), maxp);
    } else {
      const int32_t lo = (int32_t)(int16_t)(rel[k] & 0xFFFFu) + (int32_t)(int16_t)(lr[k] & 0xFFFFu);
      const int32_t hi = (((int32_t)rel[k]) >> 16) + (((int32_t)lr[k]) >> 16);
      nq = clip_half_degen(lo, p.max_llr, p.min_llr) | (clip_half_degen(hi, p.max_llr, p.min_llr) << 16);
    }
    // A slot without an edge stores nothing, and must not flag its sum either: the
    // neutral word plus any message overflows, in every second row with an idle lane.
    // 8 iterations, 64 blocks, flagged / not: BG1 Zc112 150 / 131 us, BG2 Zc64 87 / 80 us.
    ovf |= over & (k < K - 1 ? m_active : m_tail);
    if ((k < K - 1 ? active : tail) && NRLDPC_INBOUNDS(at[k] >> 16, g.limit, kBoundsLq)) {
      *reinterpret_cast<uint32_t*>(lq + (at[k] >> 16)) = __byte_perm(nq, 0u, at[k]);
      msg[k * stride] = __vadd2(~lr[k], 0x00010001u);
    }
  }
  if (kClip != kClipDegen && (ovf & 0x80008000u) != 0u) {   // rare: a sum left the int16 range
#pragma unroll
    for (int k = 0; k < K; ++k)
      if ((k < K - 1 ? active : tail) && NRLDPC_INBOUNDS(at[k] >> 16, g.limit, kBoundsLq))
        *reinterpret_cast<uint32_t*>(lq + (at[k] >> 16)) =
            __byte_perm(__vmins2(__vmaxs2(__vaddss2(rel[k], lr[k]), minp), maxp), 0u, at[k]);
  }
}

// Rate recovery of code block cw into the beliefs, with its soft buffer (the
// same values as recover_position at every position).
__device__ __forceinline__ void split_recover(const DecodeParams& p, const Geometry& g, int16_t* lq16, int cw) {
  const int16_t* in = p.llr + (int64_t)cw * p.llr_stride;
  int16_t* hq = p.harq ? p.harq + (int64_t)cw * p.harq_stride : nullptr;
  const int nt = blockDim.x;
  for (int i = threadIdx.x; i < p.lq_len; i += nt) {
    const int32_t init = (p.harq_on && hq) ? hq[i] : 0;
    const int32_t a = p.rr_scatter ? (i >= p.B && i < p.K ? p.fill : init) : recover_position(p, in, i, init);
    if (hq && !p.rr_scatter) hq[i] = (int16_t)a;
    lq16[slot_of(g, p.Zc, i)] = (int16_t)a;
  }
  __syncthreads();
  if (!p.rr_scatter) return;
  const uint32_t E = (uint32_t)p.E;
  uint32_t e = 8u * threadIdx.x;
  if (p.rr_vec) {
    for (; e + 8u <= E; e += 8u * nt) {
      const int4 v = __ldg(reinterpret_cast<const int4*>(in + e));
      const uint32_t w4[4] = {(uint32_t)v.x, (uint32_t)v.y, (uint32_t)v.z, (uint32_t)v.w};
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int pos = scatter_position(p, e + (uint32_t)q);
        if (!NRLDPC_INBOUNDS(pos, p.lq_len, kBoundsLq)) continue;
        int16_t* d = lq16 + slot_of(g, p.Zc, pos);
        *d = (int16_t)(*d + (int16_t)(w4[q >> 1] >> (16 * (q & 1))));
      }
    }
  }
  for (; e < E; e += 8u * nt)
    for (uint32_t q = e; q < e + 8u && q < E; ++q) {
      const int pos = scatter_position(p, q);
      if (!NRLDPC_INBOUNDS(pos, p.lq_len, kBoundsLq)) continue;
      int16_t* d = lq16 + slot_of(g, p.Zc, pos);
      *d = (int16_t)(*d + __ldg(in + q));
    }
  __syncthreads();
  if (hq)
    for (int i = threadIdx.x; i < p.lq_len; i += nt) hq[i] = lq16[slot_of(g, p.Zc, i)];
}

// A row of a step, staged in shared memory: x = degree (0: none) | first edge << 16,
// y = word of the thread-0 slot in the slot arrays, z = alpha | beta << 16, w = row.
// kTable: the slots' words come from a table in shared memory (beside the
// messages: one 8-byte load per slot) instead of being computed from the edge
// records.
template <int kClip, bool kTable, int kLanes>
__global__ void __launch_bounds__(kSplitThreads, 1) split_kernel(const __grid_constant__ DecodeParams p) {
  // beliefs [cols][H], four words (the neutral one first), slots [slots][threads of a group]
  extern __shared__ __align__(16) uint32_t s_lq[];
  __shared__ uint4 s_edges[kMaxNnz];
  __shared__ uint4 s_steps[kMaxRows * kGroupsPerStep];
  __shared__ uint32_t s_crc;
  constexpr int kMostSlots = (kMaxDegree + kLanes - 1) / kLanes;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int cw = blockIdx.x;
  const int T = nt / kGroupsPerStep;                 // threads of a group, whole warps
  const int grp = tid >= T ? 1 : 0, t = tid - grp * T;
  Geometry g;
  g.H = (p.Zc & 1) ? p.Zc : p.Zc >> 1;
  g.h4 = 4u * (uint32_t)g.H;
  g.swap = (p.Zc & 1) ? 0u : kSwapBit;
  const int words = (p.lq_len / p.Zc * g.H + 3) & ~3;   // the slots start 16-byte aligned
  g.limit = 4u * (uint32_t)(words + 1);
  g.zc_magic = bp_magic(p.Zc);
  const int nnz = p.row_off[p.R];
  for (int e = tid; e < nnz; e += nt) {
    const uint32_t ed = p.edge[e];   // column * Zc | (V mod Zc) << 16
    const uint32_t s = ed >> 16;
    const bool upper = (p.Zc & 1) == 0 && s >= (uint32_t)g.H;
    s_edges[e] = make_uint4((ed & 0xFFFFu) * ((p.Zc & 1) ? 4u : 2u), 4u * (s - (upper ? (uint32_t)g.H : 0u)),
                            kStraight ^ (upper ? kSwapBit : 0u), 0u);
  }
  // lr_off[r] = first slot of the row | step << 16 | group << 24
  const int steps = (int)(p.lr_off[p.R] >> 16), slots = (int)(p.lr_off[p.R] & 0xFFFFu);
  for (int k = tid; k < steps * kGroupsPerStep; k += nt) s_steps[k] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    s_crc = 0u;
    s_lq[words] = 0x7FFF7FFFu;
  }
  constexpr int kSlotWords = kTable ? 2 : 1;
  uint32_t* s_slot = s_lq + words + 4;
  for (int k = tid; k < slots * T * kSlotWords; k += nt) s_slot[k] = 0u;   // first iteration: zero messages
  __syncthreads();
  for (int r = tid; r < p.R; r += nt) {
    const uint32_t o = p.lr_off[r];
    s_steps[((o >> 16) & 0xFFu) * kGroupsPerStep + (o >> 24)] =
        make_uint4((uint32_t)(p.row_off[r + 1] - p.row_off[r]) | (uint32_t)p.row_off[r] << 16,
                   (o & 0xFFFFu) * (uint32_t)(T * kSlotWords), p.w_inline[r], (uint32_t)r);
  }
  split_recover(p, g, reinterpret_cast<int16_t*>(s_lq), cw);
  __syncthreads();

  const int lane = tid & (kLanes - 1);
  const bool active = (t / kLanes) < g.H;
  const uint32_t zx4 = active ? 4u * (uint32_t)(t / kLanes) : 0u;
  const uint32_t neutral = ((uint32_t)(4 * words) << 16) | kStraight;
  char* lq = reinterpret_cast<char*>(s_lq);
  // slot k of the row d
  const auto compute_slot = [&](const uint4& d, int k) {
    const int j = lane + kLanes * k;
    return active && j < (int)(d.x & 0xFFFFu) ? locate(g, s_edges[(d.x >> 16) + j], zx4) : neutral;
  };
  if constexpr (kTable) {
    for (int s = 0; s < steps; ++s) {
      const uint4 d = s_steps[s * kGroupsPerStep + grp];
      for (int k = 0; kLanes * k < (int)(d.x & 0xFFFFu); ++k) s_slot[d.y + 2 * (k * T + t)] = compute_slot(d, k);
    }
  }
  uint32_t* const mine = s_slot + kSlotWords * t;
  const int stride = kSlotWords * T;
  Slots nxt;
  const auto load_slots = [&](const uint4& d) {
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (kLanes * k < (int)(d.x & 0xFFFFu)) {
        if constexpr (kTable) {
          const uint2 v = *reinterpret_cast<const uint2*>(mine + d.y + k * stride);
          nxt.at[k] = v.x;
          nxt.nr[k] = v.y;
        } else {
          nxt.at[k] = compute_slot(d, k);
          nxt.nr[k] = mine[d.y + k * stride];
        }
      }
  };
  uint4 dn = s_steps[grp];
  load_slots(dn);
  int it = 0;
  bool pass = false;
  for (; it < p.max_it; ++it) {
    for (int step = 0; step < steps; ++step) {
      const Slots cur = nxt;
      const uint4 d = dn;
      const int deg = (int)(d.x & 0xFFFFu);
      // the group's next row (that of step 0 of the next iteration after the
      // last step): nothing this step writes is among its slots
      dn = s_steps[(step + 1 < steps ? step + 1 : 0) * kGroupsPerStep + grp];
      load_slots(dn);
      if (deg > 0) {   // uniform over the group's warps
        const uint32_t ab = p.weights_T > 0 ? __ldg(p.weights + (min(it, p.weights_T - 1) * p.R + (int)d.w)) : d.z;
        const int32_t alpha = (int32_t)(int16_t)(ab & 0xFFFFu), beta = ((int32_t)ab) >> 16;
        uint32_t* msg = mine + d.y + (kTable ? 1 : 0);
        const auto at_slot = [&](int k) { return kTable ? msg[k * stride - 1] : compute_slot(d, k); };
        const int left = deg - lane;   // slot k has an edge while kLanes k < left
        if (deg <= kLanes) {
          split_row<1, kLanes, kClip>(p, g, lq, cur, at_slot, msg, stride, active, active && left > 0, alpha, beta);
        } else if (deg <= 2 * kLanes) {
          split_row<2, kLanes, kClip>(p, g, lq, cur, at_slot, msg, stride, active, active && left > kLanes, alpha, beta);
        } else if (deg <= 3 * kLanes) {
          split_row<3, kLanes, kClip>(p, g, lq, cur, at_slot, msg, stride, active, active && left > 2 * kLanes, alpha, beta);
        } else {
          split_row<kMostSlots, kLanes, kClip>(p, g, lq, cur, at_slot, msg, stride, active, active && left > (kMostSlots - 1) * kLanes,
                                       alpha, beta);
        }
      }
      __syncthreads();
    }
    // Hard decisions and CRC: XOR of T[B-1-i] over the set bits i < B.
    {
      uint32_t r = 0u;
      const int words = ((p.B + p.Zc - 1) / p.Zc) * g.H;
      const uint32_t h_magic = bp_magic(g.H);
      for (int k = tid; k < words; k += nt) {
        const int c = g.H == 1 ? k : div_bp(k, h_magic);
        const int i0 = k + c * (p.Zc - g.H), i1 = i0 + g.H;
        const uint32_t w = s_lq[k];
        if (i0 < p.B) r ^= crc_term(p, i0) & sign_of_byte1(w);
        if (g.swap && i1 < p.B) r ^= crc_term(p, i1) & sign_of_byte3(w);
      }
      r = __reduce_xor_sync(0xFFFFFFFFu, r);
      if ((tid & 31) == 0 && r) atomicXor(&s_crc, r);
    }
    __syncthreads();
    pass = s_crc == 0u;
    __syncthreads();
    if (tid == 0) s_crc = 0u;   // ordered before the next iteration's use by its rows' barriers
    if (pass) {
      ++it;
      break;
    }
  }
  // Outputs.
  const int16_t* lq16 = reinterpret_cast<const int16_t*>(s_lq);
  if (it > 0 && p.bits) {
    const int nbytes = (p.B + 7) >> 3;
    uint8_t* out = p.bits + (int64_t)cw * p.bits_stride;
    for (int y = tid; y < nbytes; y += nt) {
      uint32_t v = 0u;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const int i = 8 * y + b;
        v = (v << 1) | (i < p.B && lq16[slot_of(g, p.Zc, i)] < 0 ? 1u : 0u);
      }
      out[y] = (uint8_t)v;
    }
  }
  if (p.app) {
    int16_t* out = reinterpret_cast<int16_t*>(p.app) + (int64_t)cw * p.app_stride;
    for (int i = tid; i < p.lq_len; i += nt) out[i] = lq16[slot_of(g, p.Zc, i)];
  }
  if (tid == 0) {
    if (p.status) p.status[cw] = pass ? 0 : 1;
    if (p.iters) p.iters[cw] = it;
  }
}

// Opt-in shared memory per CTA less the static arrays.
constexpr int kSplitSmemMax = 227 * 1024 - 16 * (kMaxNnz + kGroupsPerStep * kMaxRows) - 128;

template <int kClip, bool kTable, int kLanes>
int split_op(const DecodeParams* p, int block, int smem, cudaStream_t s, int* occ) {
  static std::atomic<uint32_t> attr_done{0};
  const int err = raise_smem_limit_once(split_kernel<kClip, kTable, kLanes>, &attr_done, kSplitSmemMax);
  if (err != 0) return err;
  if (occ) return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, split_kernel<kClip, kTable, kLanes>, block, smem);
  split_kernel<kClip, kTable, kLanes><<<p->num_cw, block, smem, s>>>(*p);
  count_launch();
  return (int)cudaGetLastError();
}

template <bool kTable, int kLanes>
int split_clip(const DecodeParams* p, int block, int smem, int clip_mode, cudaStream_t s, int* occ) {
  switch (clip_mode) {
    case kClipDegen: return split_op<kClipDegen, kTable, kLanes>(p, block, smem, s, occ);
    case kClipOpen:   // this kernel keeps no parity words
    case kClipOpenMax: return split_op<kClipOpenMax, kTable, kLanes>(p, block, smem, s, occ);
    default: return split_op<kClipClamp, kTable, kLanes>(p, block, smem, s, occ);
  }
}

// Eight lanes always have their table: they are for lifting sizes where it fits.
int split_dispatch(const DecodeParams* p, const SplitShape& sh, int clip_mode, cudaStream_t s, int* occ) {
  if (sh.lanes == 8) return split_clip<true, 8>(p, sh.block, sh.smem, clip_mode, s, occ);
  return sh.table ? split_clip<true, 4>(p, sh.block, sh.smem, clip_mode, s, occ)
                  : split_clip<false, 4>(p, sh.block, sh.smem, clip_mode, s, occ);
}

int split_smem(const SplitShape& s) { return 4 * (s.words + 4 + (s.table ? 2 : 1) * s.slots * s.block / kGroupsPerStep); }

}  // namespace

int bounds_read_split(uint32_t* out, bool reset) { return bounds_read_tu(out, reset); }

namespace {

// lr_off of a base graph for split_kernel: each row's first slot, step and group
// (a row joins the step of the row before it when that one is alone there and
// they share no column), and in lr_off[rows] the numbers of slots and steps.
void make_split_layout(const BaseGraph& g, int lanes, uint32_t* lr_off) {
  uint32_t slot = 0;
  int step = -1, group = kGroupsPerStep;
  for (int r = 0; r < g.rows; ++r) {
    bool joins = group + 1 < kGroupsPerStep;
    for (int a = g.row_off[r > 0 ? r - 1 : 0]; joins && a < g.row_off[r]; ++a)
      for (int b = g.row_off[r]; b < g.row_off[r + 1]; ++b)
        if (g.col[a] == g.col[b]) joins = false;
    group = joins ? group + 1 : 0;
    step += joins ? 0 : 1;
    lr_off[r] = slot | (uint32_t)step << 16 | (uint32_t)group << 24;
    slot += (uint32_t)((g.degree[r] + lanes - 1) / lanes);
  }
  lr_off[g.rows] = slot | (uint32_t)(step + 1) << 16;
}

struct SplitLayouts {
  uint32_t off[2][2][kMaxRows + 1];   // [base graph][lanes 4, 8]
  SplitLayouts() {
    for (int b = 0; b < 2; ++b)
      for (int l = 0; l < 2; ++l) make_split_layout(base_graph(b + 1), l ? 8 : 4, off[b][l]);
  }
};

}  // namespace

// A layout depends on the base graph and the lanes alone, and comparing neighbouring
// rows edge by edge takes longer than the rest of a small batch's planning (a call's
// host time 18.1 -> 16.3 us where all three lane choices are tried), so the four of
// them are made once.
const uint32_t* split_layout(int bgn, int lanes) {
  static const SplitLayouts t;
  return t.off[bgn - 1][lanes == 8 ? 1 : 0];
}

bool split_shape(int Zc, int cols, int lanes, int slots, SplitShape* out) {
  SplitShape s;
  const int H = (Zc & 1) ? Zc : Zc / 2;
  s.lanes = lanes;
  s.words = (cols * H + 3) & ~3;
  s.slots = slots;
  s.block = kGroupsPerStep * ((lanes * H + 31) & ~31);
  s.table = true;
  s.smem = split_smem(s);
  if (s.smem > kSplitSmemMax && lanes == 4) {
    s.table = false;
    s.smem = split_smem(s);
  }
  *out = s;
  return s.block <= kSplitThreads && s.smem <= kSplitSmemMax;
}

int launch_split(const DecodeParams& p, const SplitShape& s, int clip_mode, void* stream) {
  return split_dispatch(&p, s, clip_mode, reinterpret_cast<cudaStream_t>(stream), nullptr);
}
int occupancy_split(const SplitShape& s, int clip_mode) {
  int n = 0;
  split_dispatch(nullptr, s, clip_mode, nullptr, &n);
  return n;
}

}  // namespace nrldpc
