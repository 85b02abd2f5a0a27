// Flash-decode for odml.scaled_dot_product_attention, one query row per sequence, where there are bytes to wait for
// (sdpa_split_faster; sdpa_decode.cu has the kernels for short caches): ragged lengths, up to eight
// query heads per KV head, fp16 / int8 / float32 caches, optional additive mask and logit cap.
//
// Math (tflite/experimental/genai/sdpa.cc:361-662): for each query head, out = softmax_s(scale * q.k_s + mask_s) . v_s
// over the first len[b] cached tokens of the head's KV head.
//
// Bound by the cache's bytes, so the work is cut by bytes: the cached tokens of all (sequence, KV head) pairs form
// one row of 16-token units and every SM gets an equal piece of it, whatever the lengths are. (A grid of fixed
// chunks per sequence left some SMs two chunks and others one or none: 16 ragged sequences of up to 8192 tokens,
// 8 heads x 256, fp16, caches in L2: 23.7 us; equal pieces: 16.8 at the time.) A piece that covers parts of several pairs
// leaves one partial record (un-normalised output, maximum, sum) per pair; a second kernel merges a pair's records.
#include <cuda.h>
#include <math_constants.h>

#include <cstdlib>

#include "common.cuh"
#include "kernels.h"
#include "quant.cuh"

namespace b200 {

namespace {

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kUnit = 16;  // tokens per unit: the rows of one MMA tile and of one copy box

enum : int { kKvF16 = 0, kKvI8 = 1, kKvF32 = 2 };

template <int KV, int H, bool QF32>
struct Split {
  static constexpr int kElem = KV == kKvI8 ? 1 : (KV == kKvF16 ? 2 : 4);
  static constexpr int kRowBytes = H * kElem;
  static constexpr int kBoxBytes = kRowBytes < 128 ? kRowBytes : 128;  // inner extent of a copy box: one swizzle row
  static constexpr int kBoxes = kRowBytes / kBoxBytes;
  // Tokens per stage: 64 KB of keys and values, 128 tokens at most. A stage's chain of waits, products, exponentials
  // and barriers takes 0.5 us however few tokens it has, so rows of half the bytes want twice the tokens (and QK warps).
  static constexpr int kTokens = 2 * 128 * kRowBytes <= 64 * 1024 ? 128 : (2 * 64 * kRowBytes <= 64 * 1024 ? 64 : 32);
  static constexpr int kUnits = kTokens / kUnit;
  static constexpr int kQkWarps = kUnits;
  static constexpr int kPvWarps = H / 64;
  static constexpr int kThreads = 32 * (1 + kQkWarps + kPvWarps);
  static constexpr int kUnitBytes = kUnit * kRowBytes;
  static constexpr int kOperandBytes = kTokens * kRowBytes;
  static constexpr int kQBytes = 8 * H * (QF32 ? 4 : 2);    // the query heads of a pair
  static constexpr int kSlotBytes = 2 * kOperandBytes + kQBytes;
  // About 128 KB in flight per SM: with a third 64 KB stage the same launch is 1.1 us slower (17.9 against 16.8 us, 16
  // ragged sequences of up to 8192 tokens, caches resident in L2).
  static constexpr int kStagesRaw = 146 * 1024 / kSlotBytes;
  static constexpr int kStages = kStagesRaw > 8 ? 8 : kStagesRaw;
  static constexpr int kChunkElems = 16 / kElem;            // elements of a 16-byte piece
  static constexpr int kChunks = H / (4 * kChunkElems);     // pieces of a key row per thread
  static constexpr int kRec = H + 4;                        // floats of a record per head: outputs, maximum, sum, padding
  static_assert(kStages >= 2 && kBoxes >= 1 && (kChunks >= 1), "layout");
};

struct SplitShared {
  uint64_t full_k[8], full_v[8], empty_k[8], empty_v[8];
  uint64_t p_full[2], p_empty[2];
  uint4 p[2][8][32];       // softmax weights of a stage, as the B fragments of the second product: heads, remainders
  float alpha[2][8];       // factor on the earlier stages' output, per head
  uint4 smag[2][2];        // int8 rows: the eight warps' largest value scales over a stage, as bits
  float unit_of[2];        // int8 rows: what the stage's weights are multiples of
  float smax[2][8][8];     // the warps' maxima over a stage
  float ssum[8][8];
  int pair_b, pair_kvh, unit, units_cta;
  int abort_flag;
};

template <int KV, int H, bool QF32>
constexpr size_t split_smem_bytes() {
  using S = Split<KV, H, QF32>;
  return 1024 + (size_t)S::kStages * S::kSlotBytes + sizeof(SplitShared);
}

__device__ __forceinline__ int row_length(const SdpaParams& p, int b) {
  return p.lengths ? max(0, min(p.lengths[b], p.s_max)) : p.s_max;
}
__device__ __forceinline__ int units_of(int len) { return (len + kUnit - 1) / kUnit; }

// How `total` units are cut: `ctas` pieces, the first `rest` of them one unit longer than the others. No piece is
// shorter than min_units, so that short caches are not scattered over more records than they are worth.
struct Pieces {
  int ctas, size, rest;
  __device__ __forceinline__ Pieces(int total, int grid, int min_units) {
    ctas = max(1, min(grid, (total + min_units - 1) / min_units));
    size = total / ctas;
    rest = total - size * ctas;
  }
  __device__ __forceinline__ int begin(int c) const { return c * size + min(c, rest); }
  __device__ __forceinline__ int owner(int u) const {
    const int longer = rest * (size + 1);
    return u < longer ? u / (size + 1) : rest + (u - longer) / size;
  }
};

// Units of all rows, and of the rows below `b`. Whole warp. (32 bits hold them: see sdpa_split_supported.)
__device__ __forceinline__ void count_units(const SdpaParams& p, int b, int lane, int* total, int* below) {
  int all = 0, low = 0;
  for (int i = lane; i < p.b; i += 32) {
    const int u = units_of(row_length(p, i)) * p.nkv;
    all += u;
    if (i < b) low += u;
  }
  *total = (int)__reduce_add_sync(0xffffffffu, (unsigned)all);
  *below = (int)__reduce_add_sync(0xffffffffu, (unsigned)low);
}

__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// What the fp16 roundings of a and b leave, as fp16.
__device__ __forceinline__ uint32_t half2_remainder(float a, float b, uint32_t rounded) {
  const float2 r = __half22float2(*reinterpret_cast<const __half2*>(&rounded));
  return half2_bits(a - r.x, b - r.y);
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
// Exponent field of a magnitude (sign cleared), such that the field and 254 minus it both name normal numbers.
__device__ __forceinline__ int magnitude_exponent(uint32_t bits) {
  return min(max((int)(bits >> 23), 1), 253);
}
// Four int8 -> two half2, exactly: bias to unsigned, splice into 1024 + u, subtract 1152.
__device__ __forceinline__ void widen_s8x4(uint32_t w, uint32_t& lo_bits, uint32_t& hi_bits) {
  const __half2 bias = __floats2half2_rn(1152.0f, 1152.0f);
  w ^= 0x80808080u;
  uint32_t lo = __byte_perm(w, 0x64646464u, 0x4140), hi = __byte_perm(w, 0x64646464u, 0x4342);
  const __half2 l = __hsub2(*reinterpret_cast<__half2*>(&lo), bias), h = __hsub2(*reinterpret_cast<__half2*>(&hi), bias);
  lo_bits = *reinterpret_cast<const uint32_t*>(&l);
  hi_bits = *reinterpret_cast<const uint32_t*>(&h);
}

// A 16-byte piece of a key row as kChunkElems / 2 half2 words.
template <int KV>
__device__ __forceinline__ void widen16(const uint4 v, uint32_t* out) {
  if constexpr (KV == kKvF16) {
    out[0] = v.x, out[1] = v.y, out[2] = v.z, out[3] = v.w;
  } else if constexpr (KV == kKvI8) {
    widen_s8x4(v.x, out[0], out[1]);
    widen_s8x4(v.y, out[2], out[3]);
    widen_s8x4(v.z, out[4], out[5]);
    widen_s8x4(v.w, out[6], out[7]);
  } else {
    out[0] = half2_bits(__uint_as_float(v.x), __uint_as_float(v.y));
    out[1] = half2_bits(__uint_as_float(v.z), __uint_as_float(v.w));
  }
}

__device__ __forceinline__ void bulk_g2s_at(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int x0, int x1, int x2, int x3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(map), "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, int x0, int x1, int x2, int x3, int x4, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(
          dst),
      "l"(map), "r"(x0), "r"(x1), "r"(x2), "r"(x3), "r"(x4), "r"(smem_u32(bar))
      : "memory");
}

// Tensor maps of the two caches: a unit (16 tokens x one head) per copy, and a whole stage of units per copy. A copy
// costs the copy engine about 60 ns however small it is, so a stage of 64 KB must not be made of 2 KB boxes (measured:
// 1.75 us per stage, three times what HBM takes). Both leave [unit][swizzle row of the head][16 tokens][128 bytes].
struct SplitMaps {
  CUtensorMap unit[2], stage[2];
};

// One CTA per SM: a producer warp, kQkWarps warps for the first product and the softmax, kPvWarps for the second.
//  * The producer fetches 16-token boxes of K and V (tensor maps with 128-byte swizzling, so that every fragment
//    load below is free of bank conflicts, whatever the number of KV heads between two rows) into a ring of
//    stages; keys and values have barriers of their own, a key slot is free again before its value slot.
//  * A QK warp takes 16 tokens of the stage: S^T[token, head] = K . Q^T with the up-to-eight query heads as the
//    8-wide side of the MMA. The stage's maximum goes through shared memory (one barrier of the QK warps), the
//    weights leave as the B fragments of the second product (one 8 x 8 transpose each).
//    One fp16 rounding of a weight costs 2^-12 on average: float16 and float32 rows carry the remainders as a second
//    fragment (error against 64 bits, 60 draws of 64 to 8192 tokens, fp16: 2.6e-4 -> 2.1e-4, of which 1.7e-4 are the
//    output's own rounding; +0.4 us at 16 x 8192). int8 rows' weights hold the value scales, which may be far below
//    fp16's range: they are in units of a power of two next to the largest scale so far (scales of 3e-4: 4.5e-4 ->
//    2.9e-4; +0.5 us).
//  * A PV warp takes 64 of the head's dimensions for all tokens of the stage: O^T[d, head] += V^T . P^T, the rows
//    paired up by byte permutes. So no output has to be merged between warps, and while the PV warps work on a
//    stage the QK warps are at the next.
// Measured on B200 with the merge, replayed, against a grid of fixed chunks per sequence (16 sequences, lengths uniform
// up to 8192, 8 heads x 256 on one KV head; caches resident in L2 / read from HBM): fp16 rows 28.8 / 31.1 -> 15.4 / 19.1 us
// (61 MB: 3.2 TB/s from HBM; about 6 us are the two kernels' hand-offs, the first copies' latency and the merge), int8 rows
// 25.3 / 30.8 -> 16.6 / 17.9 (bound by instruction issue: widening the bytes and pairing them up); 4 x 2000 masked float32
// tokens of two KV heads 13.7 / 16.2 -> 7.7 / 9.1.
template <int KV, int H, bool QF32>
__global__ void __launch_bounds__(Split<KV, H, QF32>::kThreads, 1)
    sdpa_split_kernel(const __grid_constant__ SplitMaps maps, const SdpaParams p, const int min_units) {
  using S = Split<KV, H, QF32>;
  extern __shared__ uint8_t split_smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(split_smem_raw) + 1023) & ~uintptr_t(1023));
  SplitShared& sh = *reinterpret_cast<SplitShared*>(ring + (size_t)S::kStages * S::kSlotBytes);
  const uint32_t ring_a = smem_u32(ring);
  const uint32_t q_smem = ring_a + (uint32_t)S::kStages * 2 * S::kOperandBytes;  // per slot: the queries of a segment that starts there
  volatile int* abort_flag = &sh.abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int group = p.n / p.nkv;  // query heads per KV head

  if (tid == 0) {
    for (int i = 0; i < S::kStages; ++i) {
      mbar_init(&sh.full_k[i], 1);
      mbar_init(&sh.full_v[i], 1);
      mbar_init(&sh.empty_k[i], S::kQkWarps);
      mbar_init(&sh.empty_v[i], S::kPvWarps);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sh.p_full[i], S::kQkWarps);
      mbar_init(&sh.p_empty[i], S::kPvWarps);
    }
    sh.abort_flag = p.expired;
    mbar_fence_init();
    for (int op = 0; op < 2; ++op) {
      asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.stage[op]) : "memory");
      asm volatile("prefetch.tensormap [%0];" ::"l"(&maps.unit[op]) : "memory");
    }
  }
  pdl_wait();
  // (only now: what a dependent kernel does ahead of its own wait may then read this kernel's inputs, such as the
  // lengths, because whatever wrote them is complete)
  pdl_launch_dependents();
  if (warp == 0) {
    // this CTA's piece, and the pair in which it starts
    int units = lane < p.b ? units_of(row_length(p, lane)) : 0;
    int total, below;
    if (p.b <= 32) {
      total = (int)__reduce_add_sync(0xffffffffu, (unsigned)(units * p.nkv));
    } else {
      count_units(p, 0, lane, &total, &below);
    }
    const Pieces cut(total, gridDim.x, min_units);
    const int c = blockIdx.x;
    const int u0 = c < cut.ctas ? cut.begin(c) : 0, u1 = c < cut.ctas ? cut.begin(c + 1) : 0;
    int base = 0;
    for (int b0 = 0; b0 < p.b && u0 < u1; b0 += 32) {
      if (b0 > 0) units = b0 + lane < p.b ? units_of(row_length(p, b0 + lane)) : 0;
      int upto = units * p.nkv;  // inclusive prefix sum over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += y;
      }
      const int mine = base + upto - units * p.nkv;
      const bool here = units > 0 && mine <= u0 && u0 < mine + units * p.nkv;
      if (here) {
        sh.pair_b = b0 + lane;
        sh.pair_kvh = (u0 - mine) / units;
        sh.unit = (u0 - mine) % units;
      }
      if (__any_sync(0xffffffffu, here)) break;
      base += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (lane == 0) sh.units_cta = u1 - u0;
  }
  __syncthreads();
  int left = sh.units_cta;
  int b = sh.pair_b, kvh = sh.pair_kvh, unit = sh.unit;
  if (left == 0) return;
  int len = row_length(p, b);
  // the next pair with cached tokens (a pair is there as long as `left` is positive)
  auto next_pair = [&]() {
    unit = 0;
    if (++kvh < p.nkv) return;
    kvh = 0;
    do {
      ++b;
      len = row_length(p, b);
    } while (len == 0);
  };
  uint32_t it = 0;  // stages so far

  if (warp == 0) {
    // ---------------- producer ----------------
    if (lane == 0) {
      uint32_t armed[2] = {0, 0};  // copies of keys and values
      bool stop = false;
      while (left > 0 && !stop) {
        const int seg = min(left, units_of(len) - unit);
        const int row0 = (p.rows_per_kv > 1 ? b / p.rows_per_kv : b) * p.s_max;
        for (int j = 0; j < seg && !stop; j += S::kUnits, ++it) {
          const int s = it % S::kStages;
          const uint32_t ph = (it / S::kStages) & 1u;
          const int n = min(S::kUnits, seg - j);
          const int tok = row0 + (unit + j) * kUnit;
#pragma unroll 1
          for (int op = 0; op < 2; ++op) {
            uint64_t* full = op ? &sh.full_v[s] : &sh.full_k[s];
            mbar_wait_bounded(op ? &sh.empty_v[s] : &sh.empty_k[s], ph ^ 1u, abort_flag, p.status, kStatusWaitTimeoutEmpty);
            // After an abort that wait says nothing: the slot's last copy may be in flight, and a barrier must not be
            // armed twice in a phase.
            stop = *abort_flag != 0;
            if (stop) break;
            const bool with_q = op == 0 && j == 0;  // the segment's queries come with its first keys
            const uint32_t q_bytes = (uint32_t)(group * H * (QF32 ? 4 : 2));
            mbar_arrive_expect_tx(full, (uint32_t)(n * kUnit * S::kRowBytes) + (with_q ? q_bytes : 0u));
            ++armed[op];
            if (with_q)
              bulk_g2s_at(q_smem + (uint32_t)s * S::kQBytes,
                          static_cast<const uint8_t*>(p.q) + ((size_t)b * p.n + kvh * group) * H * (QF32 ? 4 : 2), q_bytes, full);
            const uint32_t dst = ring_a + (uint32_t)(s * 2 + op) * S::kOperandBytes;
            // (the last rows of a stage box are not checked against the cache's end: whole units only)
            if (n == S::kUnits && (unit + j + n) * kUnit <= p.s_max) {
              tma_load_5d(dst, &maps.stage[op], 0, tok, 0, 0, kvh, full);
            } else {
              for (int i = 0; i < n; ++i) tma_load_4d(dst + (uint32_t)i * S::kUnitBytes, &maps.unit[op], 0, tok + i * kUnit, 0, kvh, full);
            }
          }
        }
        left -= seg;
        if (left > 0) next_pair();
      }
      // never leave with copies in flight (only possible after an abort)
#pragma unroll 1
      for (int op = 0; op < 2; ++op)
        for (uint32_t back = 0; back < (uint32_t)S::kStages && back < armed[op]; ++back) {
          const uint32_t j = armed[op] - 1 - back;
          mbar_drain_bounded(op ? &sh.full_v[j % S::kStages] : &sh.full_k[j % S::kStages], (j / S::kStages) & 1u);
        }
    }
  } else if (warp <= S::kQkWarps) {
    // ---------------- first product and softmax ----------------
    const int w = warp - 1;
    const float scale_log2 = p.scale * kLog2e;
    while (left > 0) {
      const int seg = min(left, units_of(len) - unit);
      uint32_t qf[S::kChunks][S::kChunkElems / 2];
      auto load_queries = [&](int s) {
        // thread (g, t) keeps head g, the pieces of a row that it will load of the keys
        const uint32_t row = q_smem + (uint32_t)s * S::kQBytes + (uint32_t)(g * H * (QF32 ? 4 : 2));
#pragma unroll
        for (int q = 0; q < S::kChunks; ++q) {
          const int d0 = S::kBoxBytes == 128 ? ((q >> 1) * 8 + 2 * t + (q & 1)) * S::kChunkElems : t * S::kChunkElems;
#pragma unroll
          for (int e = 0; e < S::kChunkElems / 2; e += 2) {
            if (g >= group) {
              qf[q][e] = qf[q][e + 1] = 0u;
            } else if constexpr (QF32) {
              const uint4 f = lds128(row + (uint32_t)(d0 + 2 * e) * 4);
              qf[q][e] = half2_bits(__uint_as_float(f.x), __uint_as_float(f.y));
              qf[q][e + 1] = half2_bits(__uint_as_float(f.z), __uint_as_float(f.w));
            } else {
              const uint2 f = lds64(row + (uint32_t)(d0 + 2 * e) * 2);
              qf[q][e] = f.x;
              qf[q][e + 1] = f.y;
            }
          }
        }
      };
      const size_t tok_row0 = (size_t)(p.rows_per_kv > 1 ? b / p.rows_per_kv : b) * p.s_max;
      const float* ksc = KV == kKvI8 ? p.k_scale + tok_row0 * p.nkv + kvh : nullptr;
      const float* vsc = KV == kKvI8 ? p.v_scale + tok_row0 * p.nkv + kvh : nullptr;
      const float* maskp = p.mask ? p.mask + (size_t)b * p.s_max : nullptr;
      const int t_end = min(len, (unit + seg) * kUnit);
      // per-token factors of a stage (scales of int8 rows, mask), requested one stage ahead of their use
      struct Factors {
        float ka, kb, sa, sb, ma, mb;
      };
      auto factors = [&](int j) {
        const int ta = (unit + j + w) * kUnit + g, tb = ta + 8;
        const bool va = ta < t_end, vb = tb < t_end;
        Factors f{1.0f, 1.0f, 1.0f, 1.0f, 0.0f, 0.0f};
        if constexpr (KV == kKvI8) {
          f.ka = va ? __ldg(ksc + (size_t)ta * p.nkv) : 0.0f;
          f.kb = vb ? __ldg(ksc + (size_t)tb * p.nkv) : 0.0f;
          f.sa = va ? __ldg(vsc + (size_t)ta * p.nkv) : 0.0f;
          f.sb = vb ? __ldg(vsc + (size_t)tb * p.nkv) : 0.0f;
        }
        if (maskp) {
          f.ma = va ? __ldg(maskp + ta) : 0.0f;
          f.mb = vb ? __ldg(maskp + tb) : 0.0f;
        }
        return f;
      };
      float m_run[2] = {-CUDART_INF_F, -CUDART_INF_F}, l_run[2] = {0.0f, 0.0f};
      uint32_t mag_run = 0;  // int8: the largest value scale so far, as bits
      Factors next = factors(0);
      for (int j = 0; j < seg; j += S::kUnits, ++it) {
        const int s = it % S::kStages;
        const uint32_t ph = (it / S::kStages) & 1u;
        const int pb = it & 1;
        const int ta = (unit + j + w) * kUnit + g, tb = ta + 8;
        const bool va = ta < t_end, vb = tb < t_end;
        const Factors f = next;
        if constexpr (KV == kKvI8) {
          next = factors(j + S::kUnits);
        } else if (maskp) {
          next = factors(j + S::kUnits);
        }
        float sc[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
        mbar_wait_bounded(&sh.full_k[s], ph, abort_flag, p.status, kStatusWaitTimeoutFull);
        if (j == 0) load_queries(s);
        if (j + w < seg) {
          const uint32_t base = ring_a + (uint32_t)(s * 2) * S::kOperandBytes + (uint32_t)w * S::kUnitBytes + (uint32_t)g * S::kBoxBytes;
          float part[4][4];  // independent accumulation chains
#pragma unroll
          for (int c = 0; c < 4; ++c) part[c][0] = part[c][1] = part[c][2] = part[c][3] = 0.0f;
#pragma unroll
          for (int q = 0; q < S::kChunks; ++q) {
            // swizzled place of the piece: rows g and g + 8 of the unit have the same row index modulo 8
            const uint32_t at = S::kBoxBytes == 128
                                    ? (uint32_t)((q >> 1) * kUnit * 128) + (uint32_t)(((2 * t + (q & 1)) ^ g) << 4)
                                    : (uint32_t)((t ^ ((g >> 1) & 3)) << 4);
            uint32_t xa[S::kChunkElems / 2], xb[S::kChunkElems / 2];
            widen16<KV>(lds128(base + at), xa);
            widen16<KV>(lds128(base + at + 8 * S::kBoxBytes), xb);
#pragma unroll
            for (int e = 0; e < S::kChunkElems / 2; e += 2)
              mma_f16(part[(q * (S::kChunkElems / 4) + e / 2) & 3], xa[e], xb[e], xa[e + 1], xb[e + 1], qf[q][e], qf[q][e + 1]);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[e] = (part[0][e] + part[1][e]) + (part[2][e] + part[3][e]);
          const float ka = scale_log2 * f.ka, kb = scale_log2 * f.kb;
          sc[0] *= ka;
          sc[1] *= ka;
          sc[2] *= kb;
          sc[3] *= kb;
          if (p.logit_cap > 0.0f) {
            const float c = p.logit_cap * kLog2e, ic = 1.0f / c;
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[e] = c * tanhf(sc[e] * ic);
          }
          const float ma = f.ma * kLog2e, mb = f.mb * kLog2e;
          sc[0] = va ? sc[0] + ma : -CUDART_INF_F;
          sc[1] = va ? sc[1] + ma : -CUDART_INF_F;
          sc[2] = vb ? sc[2] + mb : -CUDART_INF_F;
          sc[3] = vb ? sc[3] + mb : -CUDART_INF_F;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.empty_k[s]);
        // maximum over the stage: the warp's tokens, then the warps
        float mx[2] = {fmaxf(sc[0], sc[2]), fmaxf(sc[1], sc[3])};
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
          mx[0] = fmaxf(mx[0], __shfl_xor_sync(0xffffffffu, mx[0], o));
          mx[1] = fmaxf(mx[1], __shfl_xor_sync(0xffffffffu, mx[1], o));
        }
        if (g == 0) *reinterpret_cast<float2*>(&sh.smax[pb][w][2 * t]) = make_float2(mx[0], mx[1]);
        if constexpr (KV == kKvI8) {
          const uint32_t mag = __reduce_max_sync(0xffffffffu, max(__float_as_uint(fabsf(f.sa)), __float_as_uint(fabsf(f.sb))));
          if (lane == 0) reinterpret_cast<uint32_t*>(sh.smag[pb])[w] = mag;
        }
        named_barrier(1, 32 * S::kQkWarps);
        float alpha[2], m_use[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float m_new = m_run[e];
#pragma unroll
          for (int i = 0; i < S::kQkWarps; ++i) m_new = fmaxf(m_new, sh.smax[pb][i][2 * t + e]);
          m_use[e] = m_new == -CUDART_INF_F ? 0.0f : m_new;  // everything masked so far
          alpha[e] = exp2f(m_run[e] - m_use[e]);             // exp2(-inf) = 0 at first
          m_run[e] = m_new;
        }
        float pa0 = exp2f(sc[0] - m_use[0]), pa1 = exp2f(sc[1] - m_use[1]);
        float pb0 = exp2f(sc[2] - m_use[0]), pb1 = exp2f(sc[3] - m_use[1]);
        l_run[0] = l_run[0] * alpha[0] + (pa0 + pb0);
        l_run[1] = l_run[1] * alpha[1] + (pa1 + pb1);
        float unit_now = 1.0f;
        if constexpr (KV == kKvI8) {
          static_assert(S::kQkWarps == 8, "two words of four warps");
          const uint4 m0 = sh.smag[pb][0], m1 = sh.smag[pb][1];
          const int was = magnitude_exponent(mag_run);
          mag_run = max(max(max(mag_run, m0.x), max(m0.y, m0.z)), max(max(m0.w, m1.x), max(m1.y, max(m1.z, m1.w))));
          const int now = magnitude_exponent(mag_run);
          if (now != was) {  // the earlier stages' outputs are in the smaller unit
            const float f = exp2f((float)(was - now));
            alpha[0] *= f;
            alpha[1] *= f;
          }
          unit_now = __int_as_float(now << 23);
          const float per_unit = __int_as_float((254 - now) << 23);
          const float sa = f.sa * per_unit, sb = f.sb * per_unit;
          pa0 *= sa;
          pa1 *= sa;
          pb0 *= sb;
          pb1 *= sb;
        }
        // rows = tokens g (g + 8), columns = heads 2t, 2t + 1 -> head g; tokens 2t, 2t + 1 (2t + 8, 2t + 9)
        const uint32_t wa = half2_bits(pa0, pa1), wb = half2_bits(pb0, pb1);
        uint4 frag = make_uint4(transpose8x8(wa), transpose8x8(wb), 0u, 0u);
        if constexpr (KV != kKvI8) {
          frag.z = transpose8x8(half2_remainder(pa0, pa1, wa));
          frag.w = transpose8x8(half2_remainder(pb0, pb1, wb));
        }
        mbar_wait_bounded(&sh.p_empty[pb], ((it >> 1) & 1u) ^ 1u, abort_flag, p.status, kStatusWaitTimeoutEmpty);
        if constexpr (KV == kKvI8) {
          *reinterpret_cast<uint2*>(&sh.p[pb][w][lane]) = make_uint2(frag.x, frag.y);
          if (w == 0 && lane == 0) sh.unit_of[pb] = unit_now;
        } else {
          sh.p[pb][w][lane] = frag;
        }
        if (w == 0 && g == 0) *reinterpret_cast<float2*>(&sh.alpha[pb][2 * t]) = make_float2(alpha[0], alpha[1]);
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh.p_full[pb]);
      }
      // the record's maximum and sum
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) l_run[e] += __shfl_xor_sync(0xffffffffu, l_run[e], o);
      if (g == 0) *reinterpret_cast<float2*>(&sh.ssum[w][2 * t]) = make_float2(l_run[0], l_run[1]);
      named_barrier(1, 32 * S::kQkWarps);
      if (w == 0 && g == 0) {
        float* rec = p.ws + ((size_t)blockIdx.x + (size_t)b * p.nkv + kvh) * 8 * S::kRec;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float l = 0.0f;
#pragma unroll
          for (int i = 0; i < S::kQkWarps; ++i) l += sh.ssum[i][2 * t + e];
          *reinterpret_cast<float2*>(rec + (2 * t + e) * S::kRec + H) = make_float2(m_run[e], l);
        }
      }
      left -= seg;
      if (left > 0) next_pair();
    }
  } else {
    // ---------------- second product: 64 head dimensions per warp ----------------
    const int w = warp - 1 - S::kQkWarps;
    // where in a unit this thread's piece of a token's row lies (its 8 head dimensions)
    auto piece_at = [&](int row) -> uint32_t {
      if constexpr (KV == kKvF16) return (uint32_t)((w * kUnit + row) * 128) + (uint32_t)((g ^ (row & 7)) << 4);
      if constexpr (KV == kKvF32) return (uint32_t)((2 * w * kUnit + row) * 128) + (uint32_t)((g ^ (row & 7)) << 4);
      if constexpr (S::kBoxBytes == 64) return (uint32_t)(row * 64) + (uint32_t)(((g >> 1) ^ ((row >> 1) & 3)) << 4) + (uint32_t)(g & 1) * 8;
      return (uint32_t)(((w >> 1) * kUnit + row) * 128) + (uint32_t)((((w & 1) * 4 + (g >> 1)) ^ (row & 7)) << 4) + (uint32_t)(g & 1) * 8;
    };
    const uint32_t row_at[4] = {piece_at(2 * t), piece_at(2 * t + 1), piece_at(2 * t + 8), piece_at(2 * t + 9)};
    while (left > 0) {
      const int seg = min(left, units_of(len) - unit);
      const int t_end = min(len, (unit + seg) * kUnit);
      float o[4][4], rem[4][4], unit_now = 1.0f;  // rem: what the weights' remainders give (chains of their own)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.0f;
        rem[i][0] = rem[i][1] = rem[i][2] = rem[i][3] = 0.0f;
      }
      for (int j = 0; j < seg; j += S::kUnits, ++it) {
        const int s = it % S::kStages;
        const uint32_t ph = (it / S::kStages) & 1u;
        const int pb = it & 1;
        const int n = min(S::kUnits, seg - j);
        const int last = t_end - 1 - (unit + j) * kUnit;  // last valid row of the stage
        mbar_wait_bounded(&sh.full_v[s], ph, abort_flag, p.status, kStatusWaitTimeoutFull);
        mbar_wait_bounded(&sh.p_full[pb], (it >> 1) & 1u, abort_flag, p.status, kStatusWaitTimeoutFull);
        const float2 al = *reinterpret_cast<const float2*>(&sh.alpha[pb][2 * t]);
        if constexpr (KV == kKvI8) unit_now = sh.unit_of[pb];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          o[i][0] *= al.x;
          o[i][1] *= al.y;
          o[i][2] *= al.x;
          o[i][3] *= al.y;
          if constexpr (KV != kKvI8) {
            rem[i][0] *= al.x;
            rem[i][1] *= al.y;
            rem[i][2] *= al.x;
            rem[i][3] *= al.y;
          }
        }
        const uint32_t vbase = ring_a + (uint32_t)(s * 2 + 1) * S::kOperandBytes;
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
          uint4 pf;
          if constexpr (KV == kKvI8) {
            const uint2 v = *reinterpret_cast<const uint2*>(&sh.p[pb][k][lane]);
            pf = make_uint4(v.x, v.y, 0u, 0u);
          } else {
            pf = sh.p[pb][k][lane];
          }
          const uint32_t ubase = vbase + (uint32_t)k * S::kUnitBytes;
          const int last_row = last - k * kUnit;
          uint32_t vr[4][4];  // 8 head dimensions of tokens 2t, 2t + 1, 2t + 8, 2t + 9
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            uint32_t at = ubase + row_at[r];
            // (rows beyond the last token have weight 0; they read a valid row, so that 0 x NaN cannot arise)
            if (last_row < kUnit - 1) at = ubase + piece_at(min(2 * t + (r & 1) + 8 * (r >> 1), last_row));
            if constexpr (KV == kKvF16) {
              const uint4 v = lds128(at);
              vr[r][0] = v.x, vr[r][1] = v.y, vr[r][2] = v.z, vr[r][3] = v.w;
            } else if constexpr (KV == kKvI8) {
              const uint2 v = lds64(at);
              widen_s8x4(v.x, vr[r][0], vr[r][1]);
              widen_s8x4(v.y, vr[r][2], vr[r][3]);
            } else {
#pragma unroll
              for (int x = 0; x < 2; ++x) {
                const uint4 v = lds128(at + (uint32_t)(x * kUnit * 128));
                vr[r][2 * x] = half2_bits(__uint_as_float(v.x), __uint_as_float(v.y));
                vr[r][2 * x + 1] = half2_bits(__uint_as_float(v.z), __uint_as_float(v.w));
              }
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {  // MMA row g <-> the thread's dimension 2 i, row g + 8 <-> 2 i + 1
            const uint32_t a0 = __byte_perm(vr[0][i], vr[1][i], 0x5410), a1 = __byte_perm(vr[0][i], vr[1][i], 0x7632);
            const uint32_t a2 = __byte_perm(vr[2][i], vr[3][i], 0x5410), a3 = __byte_perm(vr[2][i], vr[3][i], 0x7632);
            mma_f16(o[i], a0, a1, a2, a3, pf.x, pf.y);
            if constexpr (KV != kKvI8) mma_f16(rem[i], a0, a1, a2, a3, pf.z, pf.w);
          }
        }
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&sh.empty_v[s]);
          mbar_arrive(&sh.p_empty[pb]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = KV == kKvI8 ? o[i][e] * unit_now : o[i][e] + rem[i][e];
      float* rec = p.ws + ((size_t)blockIdx.x + (size_t)b * p.nkv + kvh) * 8 * S::kRec;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (2 * t + e >= group) continue;
        float* dst = rec + (2 * t + e) * S::kRec;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int d = KV == kKvF32 ? 64 * w + 32 * x + 4 * g : 64 * w + 8 * g + 4 * x;
          *reinterpret_cast<float4*>(dst + d) = make_float4(o[2 * x][e], o[2 * x][2 + e], o[2 * x + 1][e], o[2 * x + 1][2 + e]);
        }
      }
      left -= seg;
      if (left > 0) next_pair();
    }
  }
  if (!__syncthreads_or(*abort_flag)) return;
  // the records are made of whatever the ring held
  left = sh.units_cta, b = sh.pair_b, kvh = sh.pair_kvh, unit = sh.unit;
  len = row_length(p, b);
  while (left > 0) {
    const int seg = min(left, units_of(len) - unit);
    if (tid < 8) p.ws[((size_t)blockIdx.x + (size_t)b * p.nkv + kvh) * 8 * S::kRec + tid * S::kRec + H + 1] = kLostRecord;
    left -= seg;
    if (left > 0) next_pair();
  }
}

// Records of one (row, KV head) pair: the first one, and how many.
struct PairRecords {
  const float* first;
  int count;
};
template <int H>
__device__ __forceinline__ PairRecords pair_records(const SdpaParams& p, int b, int kvh, int units, int below, const Pieces& cut) {
  PairRecords r{nullptr, 0};
  if (units == 0) return r;
  const int u0 = below + kvh * units;
  const int c0 = cut.owner(u0), c1 = cut.owner(u0 + units - 1);
  r.first = p.ws + ((size_t)c0 + (size_t)b * p.nkv + kvh) * 8 * (H + 4);
  r.count = c1 - c0 + 1;
  return r;
}

// Weights exp2(m_record - m) of a head's records, from their (maximum, sum) pairs at `ml`; returns the softmax
// denominator, or kLostRecord where a record is one. Whole warp; the first 64 pairs in one round trip.
__device__ __forceinline__ float record_weights(const float* ml, size_t stride, int count, int lane, float* weights) {
  const float2 none = make_float2(-CUDART_INF_F, 0.0f);
  const float2 a = lane < count ? __ldcg(reinterpret_cast<const float2*>(ml + lane * stride)) : none;
  const float2 b = lane + 32 < count ? __ldcg(reinterpret_cast<const float2*>(ml + (lane + 32) * stride)) : none;
  float mm = fmaxf(a.x, b.x);
  for (int c = lane + 64; c < count; c += 32) mm = fmaxf(mm, __ldcg(ml + c * stride));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, o));
  const float muse = mm == -CUDART_INF_F ? 0.0f : mm;
  const float fa = exp2f(a.x - muse), fb = exp2f(b.x - muse);
  float l = fa * a.y + fb * b.y;
  bool lost = a.y == kLostRecord || b.y == kLostRecord;
  if (lane < count) weights[lane] = fa;
  if (lane + 32 < count) weights[lane + 32] = fb;
  for (int c = lane + 64; c < count; c += 32) {
    const float2 v = __ldcg(reinterpret_cast<const float2*>(ml + c * stride));
    const float f = exp2f(v.x - muse);
    weights[c] = f;
    l += f * v.y;
    lost = lost || v.y == kLostRecord;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  return __any_sync(0xffffffffu, lost) ? kLostRecord : l;
}

// Sum of a head's records, weighted, for the four outputs d4 .. d4 + 3: records grp, grp + groups, ...
// (`first`: the first kBatch of them, requested earlier).
template <int kBatch>
__device__ __forceinline__ float4 merge_quad(const float* base, size_t stride, int count, int grp, int groups, const float* weights,
                                             const float4 (&first)[kBatch]) {
  float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  auto add = [&](float w, const float4& v) {
    acc.x += w * v.x;
    acc.y += w * v.y;
    acc.z += w * v.z;
    acc.w += w * v.w;
  };
#pragma unroll
  for (int j = 0; j < kBatch; ++j) {
    const int c = grp + j * groups;
    if (c < count) add(weights[c], first[j]);
  }
  for (int c0 = grp + kBatch * groups; c0 < count; c0 += 4 * groups) {
    float4 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c0 + j * groups < count) v[j] = __ldcg(reinterpret_cast<const float4*>(base + (size_t)(c0 + j * groups) * stride));
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (c0 + j * groups < count) add(weights[c0 + j * groups], v[j]);
  }
  return acc;
}
template <int kBatch>
__device__ __forceinline__ void request_quads(float4 (&v)[kBatch], const float* base, size_t stride, int count, int grp, int groups) {
#pragma unroll
  for (int j = 0; j < kBatch; ++j) {
    const int c = grp + j * groups;
    v[j] = c < count ? __ldcg(reinterpret_cast<const float4*>(base + (size_t)c * stride)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
}

// Merges the records of one (row, query head): grid (n, b), 256 threads. What it costs are L2 round trips (0.7 us
// each), so there are as few as possible: where the records are is worked out ahead of the dependency wait, then every
// thread requests four outputs of up to 16 records at once (256 / (H / 4) threads share a record's row: 64 records of
// 256 outputs in one trip) while the first warp gathers the maxima and sums. (One thread per output, eight records in
// flight: a sequence cut into 74 records took 5 us.)
constexpr int kMergeThreads = 256;
template <int H, bool QF32>
__global__ void __launch_bounds__(kMergeThreads) sdpa_split_merge_kernel(const SdpaParams p, const int split_ctas, const int min_units) {
  constexpr int kRec = H + 4, kQuads = H / 4, kGroups = kMergeThreads / kQuads, kMergeBatch = 16;
  constexpr size_t kStride = 8 * (size_t)kRec;
  extern __shared__ float merge_w[];  // one weight exp2(m_record - m) per record
  __shared__ float4 s_part[kMergeThreads];
  __shared__ float s_l;
  pdl_launch_dependents();
  const int b = blockIdx.y, head = blockIdx.x, lane = threadIdx.x & 31;
  const int quad = threadIdx.x % kQuads, grp = threadIdx.x / kQuads;
  const int group = p.n / p.nkv;
  int total, below;
  count_units(p, b, lane, &total, &below);
  const PairRecords rec =
      pair_records<H>(p, b, head / group, units_of(row_length(p, b)), below, Pieces(total, split_ctas, min_units));
  const float* base = rec.first + (head % group) * kRec;
  pdl_wait();
  float4 first[kMergeBatch];
  request_quads(first, base + 4 * quad, kStride, rec.count, grp, kGroups);
  if (threadIdx.x < 32) {
    const float l = record_weights(base + H, kStride, rec.count, lane, merge_w);
    if (lane == 0) s_l = l;
  }
  __syncthreads();
  s_part[threadIdx.x] = merge_quad(base + 4 * quad, kStride, rec.count, grp, kGroups, merge_w, first);
  __syncthreads();
  if (grp > 0) return;
  float4 acc = s_part[quad];
#pragma unroll 2
  for (int i = 1; i < kGroups; ++i) {
    const float4 v = s_part[i * kQuads + quad];
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  }
  const float l = s_l;
  acc = make_float4(head_output(acc.x, l), head_output(acc.y, l), head_output(acc.z, l), head_output(acc.w, l));
  const size_t oi = ((size_t)b * p.n + head) * H + 4 * quad;
  if constexpr (QF32) {
    float* o = static_cast<float*>(p.out) + oi;
    o[0] = acc.x, o[1] = acc.y, o[2] = acc.z, o[3] = acc.w;
  } else {
    __half* o = static_cast<__half*>(p.out) + oi;
    o[0] = __float2half_rn(acc.x), o[1] = __float2half_rn(acc.y), o[2] = __float2half_rn(acc.z), o[3] = __float2half_rn(acc.w);
  }
}

// The merge fused with the per-row asymmetric int8 quantization that the next hybrid FULLY_CONNECTED applies to the
// attention output: one CTA per row over all n * H outputs. Writes the tiled int8 row (+ scale, zero point) and, when
// p.out is set, the floats. 256 threads of up to 112 registers: they fit on an SM beside a CTA of the split kernel, so
// that the early launch is one.
constexpr int kMergeQuantThreads = 256;
template <int H>
__global__ void __launch_bounds__(kMergeQuantThreads, 2) sdpa_split_merge_quant_kernel(const SdpaParams p, const int split_ctas, const int min_units) {
  constexpr int kRec = H + 4, kMergeBatch = 6;
  constexpr size_t kStride = 8 * (size_t)kRec;
  extern __shared__ float xs[];  // n * H merged outputs, then n * split_ctas weights
  __shared__ float red[32];
  __shared__ float s_l[64];  // softmax denominator per head
  pdl_launch_dependents();
  const int b = blockIdx.x, lane = threadIdx.x & 31;
  const int group = p.n / p.nkv;
  int total, below;
  count_units(p, b, lane, &total, &below);
  const Pieces cut(total, split_ctas, min_units);
  const int units = units_of(row_length(p, b));
  const int width = p.n * H, quads = width / 4;
  float* wts = xs + width;
  pdl_wait();
  // the first quad's records are requested before anything else, so that their round trip overlaps the statistics'
  auto quad_base = [&](int quad, int* count) {
    const int head = quad * 4 / H;
    const PairRecords rec = pair_records<H>(p, b, head / group, units, below, cut);
    *count = rec.count;
    return rec.first + (head % group) * kRec + quad * 4 % H;
  };
  float4 first[2][kMergeBatch];
  int count[2] = {0, 0};
  const float* base[2] = {nullptr, nullptr};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int quad = threadIdx.x + e * blockDim.x;
    if (quad < quads) base[e] = quad_base(quad, &count[e]);
    request_quads(first[e], base[e], kStride, count[e], 0, 1);
  }
  bool lost = false;
  for (int hd = threadIdx.x >> 5; hd < p.n; hd += blockDim.x >> 5) {
    const PairRecords r = pair_records<H>(p, b, hd / group, units, below, cut);
    const float l = record_weights(r.first + (hd % group) * kRec + H, kStride, r.count, lane, wts + hd * split_ctas);
    if (lane == 0) s_l[hd & 63] = l;
    lost = lost || l == kLostRecord;
  }
  lost = __syncthreads_or(lost) != 0;
  float mn = 3.402823466e+38f, mx = -3.402823466e+38f;
  auto finish = [&](int quad, const float* from, int n, const float4 (&requested)[kMergeBatch]) {
    const int head = quad * 4 / H;
    float4 acc = merge_quad(from, kStride, n, 0, 1, wts + head * split_ctas, requested);
    const float l = s_l[head & 63];  // an empty sequence gives a zero row
    acc = make_float4(head_output(acc.x, l), head_output(acc.y, l), head_output(acc.z, l), head_output(acc.w, l));
    *reinterpret_cast<float4*>(xs + 4 * quad) = acc;
    if (p.out) {
      float* o = static_cast<float*>(p.out) + (size_t)b * width + 4 * quad;
      o[0] = acc.x, o[1] = acc.y, o[2] = acc.z, o[3] = acc.w;
    }
    mn = fminf(mn, fminf(fminf(acc.x, acc.y), fminf(acc.z, acc.w)));
    mx = fmaxf(mx, fmaxf(fmaxf(acc.x, acc.y), fmaxf(acc.z, acc.w)));
  };
#pragma unroll
  for (int e = 0; e < 2; ++e)
    if ((int)(threadIdx.x + e * blockDim.x) < quads) finish(threadIdx.x + e * blockDim.x, base[e], count[e], first[e]);
#pragma unroll 1
  for (int quad = threadIdx.x + 2 * blockDim.x; quad < quads; quad += blockDim.x) {
    base[0] = quad_base(quad, &count[0]);
    request_quads(first[0], base[0], kStride, count[0], 0, 1);
    finish(quad, base[0], count[0], first[0]);
  }
  const int k_pad = (width + 127) / 128 * 128;
  quantize_smem_row(xs, width, k_pad, b, p.m_alloc, mn, mx, p.q_tiled_out, p.out_scales, p.out_zps, red);
  if (lost && threadIdx.x == 0) p.out_scales[b] = __int_as_float(0x7fffffff);  // (integers hold no NaN; their scale does)
}

// Shortest piece worth a CTA of its own: one unit where no sequence can leave more than 64 records, the merge's single
// round trip; longer pieces for longer caches. (Four units whatever the cache made one CTA walk through several short
// sequences in turn: 16 ragged sequences of up to 64 tokens, 8 heads x 256, fp16 8.8 us, one unit 6.9.)
int split_min_units(int s_max) {
  if (const char* e = tuning_env("B200_SDPA_MIN_UNITS")) {  // measurement knob
    if (atoi(e) > 0) return atoi(e);
  }
  return s_max <= 64 * kUnit ? 1 : s_max <= 128 * kUnit ? 2 : 4;
}
// CTAs of a launch: one per SM, fewer when even full caches give no piece for some.
int split_ctas(int b, int nkv, int s_max) {
  const long long most = (long long)b * nkv * ((s_max + kUnit - 1) / kUnit);
  const long long n = (most + split_min_units(s_max) - 1) / split_min_units(s_max);
  const int sms = device_sm_count();
  return n < sms ? (int)n : sms;
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult st;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &st) != cudaSuccess ||
        st != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      f = nullptr;
    }
    return reinterpret_cast<EncodeTiled>(f);
  }();
  return fn;
}

// A cache [rows, nkv, H] as bytes, seen as (byte of a swizzle row, token, swizzle row of the head, [unit,] head). The
// unit dimension overlaps the token's: unit u of a box starts 16 u tokens behind it.
template <int KV, int H>
bool cache_maps(SplitMaps* maps, int op, const void* base, int nkv, long long rows) {
  using S = Split<KV, H, false>;
  const EncodeTiled encode = encode_tiled();
  if (!encode) return false;
  const cuuint64_t row = (cuuint64_t)S::kRowBytes, pitch = row * nkv;
  const cuuint64_t dims4[4] = {(cuuint64_t)S::kBoxBytes, (cuuint64_t)rows, (cuuint64_t)S::kBoxes, (cuuint64_t)nkv};
  const cuuint64_t strides4[3] = {pitch, (cuuint64_t)S::kBoxBytes, row};
  const cuuint32_t box4[4] = {(cuuint32_t)S::kBoxBytes, (cuuint32_t)kUnit, (cuuint32_t)S::kBoxes, 1};
  const cuuint64_t dims5[5] = {dims4[0], dims4[1], dims4[2], (cuuint64_t)S::kUnits, dims4[3]};
  const cuuint64_t strides5[4] = {pitch, (cuuint64_t)S::kBoxBytes, pitch * kUnit, row};
  const cuuint32_t box5[5] = {box4[0], box4[1], box4[2], (cuuint32_t)S::kUnits, 1};
  const cuuint32_t steps[5] = {1, 1, 1, 1, 1};
  const CUtensorMapSwizzle swizzle = S::kBoxBytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
  void* addr = const_cast<void*>(base);
  return encode(&maps->unit[op], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, addr, dims4, strides4, box4, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS &&
         encode(&maps->stage[op], CU_TENSOR_MAP_DATA_TYPE_UINT8, 5, addr, dims5, strides5, box5, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename K>
cudaError_t allow_smem(K kernel, size_t bytes, bool (&done)[64]) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (done[dev]) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done[dev] = true;
  return e;
}

template <int KV, int H, bool QF32>
cudaError_t launch_split(const SdpaParams& p, cudaStream_t s) {
  using S = Split<KV, H, QF32>;
  const long long rows = (long long)(p.rows_per_kv > 1 ? p.b / p.rows_per_kv : p.b) * p.s_max;
  SplitMaps maps;
  if (!cache_maps<KV, H>(&maps, 0, p.k, p.nkv, rows) || !cache_maps<KV, H>(&maps, 1, p.v, p.nkv, rows)) return cudaErrorNotSupported;
  const int min_units = split_min_units(p.s_max), ctas = split_ctas(p.b, p.nkv, p.s_max);
  static bool done[64] = {false};
  constexpr size_t smem = split_smem_bytes<KV, H, QF32>();
  cudaError_t e = allow_smem(sdpa_split_kernel<KV, H, QF32>, smem, done);
  if (e != cudaSuccess) return e;
  e = launch_chained(sdpa_split_kernel<KV, H, QF32>, dim3(ctas), dim3(S::kThreads), smem, s, maps, p, min_units);
  if (e != cudaSuccess) return e;
  if (p.q_tiled_out) {
    if (p.n > 64) return cudaErrorInvalidValue;
    const size_t msmem = sizeof(float) * ((size_t)p.n * H + (size_t)p.n * ctas);
    static bool mdone[64] = {false};
    e = allow_smem(sdpa_split_merge_quant_kernel<H>, sizeof(float) * 64 * (H + 160), mdone);
    if (e != cudaSuccess) return e;
    return launch_chained(sdpa_split_merge_quant_kernel<H>, dim3(p.b), dim3(kMergeQuantThreads), msmem, s, p, ctas, min_units);
  }
  return launch_chained(sdpa_split_merge_kernel<H, QF32>, dim3(p.n, p.b), dim3(kMergeThreads), sizeof(float) * (size_t)ctas, s, p, ctas,
                        min_units);
}

template <int KV, bool QF32>
cudaError_t launch_split_h(const SdpaParams& p, cudaStream_t s) {
  if (p.h == 256) return launch_split<KV, 256, QF32>(p, s);
  if (p.h == 128) return launch_split<KV, 128, QF32>(p, s);
  return launch_split<KV, 64, QF32>(p, s);
}

}  // namespace

bool sdpa_split_supported(const SdpaParams& p) {
  const int group = p.nkv > 0 ? p.n / p.nkv : 0;
  return group >= 1 && group <= 8 && p.n % p.nkv == 0 && (p.h == 64 || p.h == 128 || p.h == 256) && !p.shared_kv &&
         ((reinterpret_cast<uintptr_t>(p.k) | reinterpret_cast<uintptr_t>(p.v) | reinterpret_cast<uintptr_t>(p.q) |
           reinterpret_cast<uintptr_t>(p.ws)) & 15) == 0 &&
         (long long)p.b * p.nkv * ((p.s_max + kUnit - 1) / kUnit) <= INT32_MAX && p.ws != nullptr &&
         p.ws_bytes >= sdpa_split_workspace_bytes(p.b, p.nkv, p.h, p.s_max);
}

// Where the split kernel is the faster one: its chain of barriers and hand-offs costs more than a chunk's loop until there
// are bytes to wait for, and many pairs of few tokens make a CTA walk through several of them in turn. Over 873 launches
// of 1 to 16 ragged sequences of up to 8192 tokens, six head layouts, replayed, against the kernels over chunks: 0.89 of
// their time on average by this rule, 1.0 if everything is split. 16 sequences of up to 512 tokens, 8 heads x 64 on 8 KV
// heads, int8: 9.0 us over chunks, 13.7 split; of up to 4096 tokens, 8 heads x 256, fp16: 15.6 and 11.3; 300 query tokens
// over 300, 8 heads x 128, fp16: 22.8 and 33.4. The fused quantization is faster split at every size. (The kernels over
// chunks keep a weight as one fp16 operand: 2.45e-4 against 64 bits for fp16 rows, 2.1e-4 here.)
bool sdpa_split_faster(const SdpaParams& p) {
  if (const char* e = tuning_env("B200_SDPA_SPLIT")) return e[0] != '0';  // measurement knob
  if (p.q_tiled_out) return true;
  const long long pairs = (long long)p.b * p.nkv, rows = pairs * p.s_max;
  const bool long_enough = pairs <= 64 || p.s_max > (p.h == 256 ? 256 : 512);
  if (p.kv_dtype == kKvF32) return p.h == 64 ? rows > 16384 && pairs <= 256 : long_enough;  // (chunks without staging)
  if (p.kv_dtype == kKvF16) return p.h == 256 ? long_enough : p.h == 128 ? rows > 8192 && p.s_max > 512 : p.s_max > 2048;
  return p.s_max > 2048 && rows > 8192 && (p.h > 64 || pairs < 64);
}

size_t sdpa_split_workspace_bytes(int b, int nkv, int h, int s_max) {
  // a record (8 heads, padded) per CTA and pair at most: pieces and pairs are both in order, so that CTA + pair names one
  return ((size_t)split_ctas(b, nkv, s_max) + (size_t)b * nkv) * 8 * (h + 4) * sizeof(float);
}

cudaError_t launch_sdpa_split(const SdpaParams& p, cudaStream_t s) {
  const bool qf32 = p.q_dtype == 1;
  if (p.kv_dtype == kKvF16) return qf32 ? launch_split_h<kKvF16, true>(p, s) : launch_split_h<kKvF16, false>(p, s);
  if (p.kv_dtype == kKvI8) return qf32 ? launch_split_h<kKvI8, true>(p, s) : launch_split_h<kKvI8, false>(p, s);
  return qf32 ? launch_split_h<kKvF32, true>(p, s) : launch_split_h<kKvF32, false>(p, s);
}

}  // namespace b200
