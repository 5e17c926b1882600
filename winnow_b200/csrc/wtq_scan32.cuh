// The page scan at head_dim 64 in fp32 on the CUDA cores: one 32-token window of the
// online softmax for up to eight query heads, used by wtq_decode_fused.cu.
//
// Queries, centroids, probabilities and value weights are fp32, as in
// decode_generic_kernel: 16-bit operands, as the scan of head_dim 128 has them, cost three
// digits here (relative error of an fp32 call 3.4e-4 against 5e-7 and, because
// probability x value norm turned subnormal, 1e-2 for values of norm 1e-4).
//
// Scores: lane (tq, part) takes tokens tq, tq + 8, tq + 16, tq + 24 and the sixteen
// coordinates 16 part .. of all eight heads, so a centroid feeds eight multiply-adds and a
// query word four; two exchanges leave every lane with one token's eight scores.  Values:
// lane (gq, dq) takes tokens gq, gq + 4, .. and coordinates 8 dq .. of all heads.  Both
// run two multiply-adds an instruction (fma.rn.f32x2, each rounded as fmaf).  Bound by
// shared-memory operands and issue slots, evenly: 566 cycles a window.  Calls with 14 query
// and 2 kv heads, 4 bits, on decode_generic_kernel and here: 8 sequences of 700 to 5000
// tokens 66.7 -> 16.5 us, one of 131072 336 -> 157, 128 of 8192 1189 -> 166 (16-bit operands
// 10.3, 57.7 and 66.3); error against 64 bits 5.9e-7 -> 3.5e-7.
#pragma once

#include "wtq_scan.cuh"

namespace wtq {
namespace scan32 {

constexpr int kD = 64, kHeads = 8;
constexpr uint32_t kWeightRow = 48;                    // bytes of a token's eight value weights (+ pad: no conflicts)
constexpr uint32_t kWeights = kIterTokens * kWeightRow;

constexpr uint32_t table_bytes(int bw_k, int bw_v) { return 256u << (bw_k > bw_v ? bw_k : bw_v); }
// Word of the fp32 tables for (index, side) number `pair`, the same for every lane; the
// layout is that of wtq_lut.cuh with index = a code at every width.
__device__ __forceinline__ uint32_t table_word(int pair, int bw_k, int bw_v, const float *ck, const float *cv) {
  const int index = pair >> 1, side = pair & 1;
  return index < (1 << (side ? bw_v : bw_k)) ? __float_as_uint(__ldg((side ? cv : ck) + index)) : 0u;
}
// Rotated queries lie as [coordinate][head], a pad of four words per sixteen coordinates.
constexpr uint32_t kQueryWords = kD * kHeads + 4 * (kD / 16);
__device__ __forceinline__ uint32_t query_word(int d, int h) { return (uint32_t)(d * kHeads + 4 * (d >> 4) + h); }

__device__ __forceinline__ void lds_pairs(uint32_t a, uint64_t &x, uint64_t &y) {
  asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];\n" : "=l"(x), "=l"(y) : "r"(a));
}
__device__ __forceinline__ void sts_f4(uint32_t a, float x, float y, float z, float w) {
  asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

struct State {
  uint64_t acc[kHeads / 2][8];                         // [head pair][coordinate 8 dq + i], this lane's tokens
  float M[kHeads], l[kHeads];                          // reference (the same in every lane); this lane's sum
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int h = 0; h < kHeads; ++h) {
      M[h] = -INFINITY;
      l[h] = 0.f;
    }
#pragma unroll
    for (int p = 0; p < kHeads / 2; ++p)
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[p][i] = 0;
  }
};

// Coordinates I .. 15 of the lane's sixteen: s[token][head pair] += q x centroid.
template <int BW, int I>
__device__ __forceinline__ void score_steps(const uint32_t (&w)[4][BW / 2], uint32_t sel, uint32_t q_at,
                                            uint64_t (&s)[4][kHeads / 2]) {
  if constexpr (I < 16) {
    uint64_t q[4], c[4];
    lds_pairs(q_at + 32u * I, q[0], q[1]);
    lds_pairs(q_at + 32u * I + 16u, q[2], q[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = twice(__uint_as_float(lut_code<BW, I>(w[k], sel)));
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int p = 0; p < 4; ++p) fma2(s[k][p], c[k], q[p]);
    score_steps<BW, I + 1>(w, sel, q_at, s);
  }
}
// Coordinates I .. 7 of the lane's eight: acc += weight x centroid.
template <int BW, int I, int NW>
__device__ __forceinline__ void value_steps(const uint32_t (&w)[NW], uint32_t sel, const uint64_t (&p)[4],
                                            uint64_t (&acc)[kHeads / 2][8]) {
  if constexpr (I < 8) {
    const uint64_t c = twice(__uint_as_float(lut_code<BW, I>(w, sel)));
#pragma unroll
    for (int k = 0; k < 4; ++k) fma2(acc[k][I], p[k], c);
    value_steps<BW, I + 1>(w, sel, p, acc);
  }
}

// One window of two tiles at shared address `slot0`, first token `wtok`, tokens from `tok1`
// on and those of tiles that are not in `loaded` left out.  `q_at`: the rotated queries,
// `weights`: kWeights bytes of this warp.
template <class T>
__device__ __forceinline__ void window(State &st, uint32_t slot0, int wtok, int tok1, uint32_t loaded, int lane,
                                       uint32_t sel_k, uint32_t sel_v, uint32_t q_at, uint32_t weights) {
  constexpr uint32_t kFull = 0xffffffffu;
  const int tq = lane >> 2, part = lane & 3;
  // ---- scores -------------------------------------------------------------------
  float s[kHeads];
  {
    uint32_t w[4][T::BWK / 2];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      load_words<2 * T::BWK>(slot0 + (k >> 1) * T::kSlot + (tq + 8 * (k & 1)) * T::NBK + part * (2 * T::BWK), w[k]);
    uint64_t acc[4][kHeads / 2];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int p = 0; p < 4; ++p) acc[k][p] = 0;
    score_steps<T::BWK, 0>(w, sel_k, q_at + 4u * query_word(16 * part, 0), acc);
    // the four parts of a token meet: lane (tq, part) ends with token tq + 8 (2 (part & 1) + (part >> 1))
    const bool odd = part & 1, high = part & 2;
    float half[2][kHeads];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float2 a = halves(acc[k][p]), b = halves(acc[k + 2][p]);
        half[k][2 * p] = (odd ? b.x : a.x) + __shfl_xor_sync(kFull, odd ? a.x : b.x, 1);
        half[k][2 * p + 1] = (odd ? b.y : a.y) + __shfl_xor_sync(kFull, odd ? a.y : b.y, 1);
      }
#pragma unroll
    for (int h = 0; h < kHeads; ++h)
      s[h] = (high ? half[1][h] : half[0][h]) + __shfl_xor_sync(kFull, high ? half[0][h] : half[1][h], 2);
  }
  const int tile = part & 1, row = tq + 8 * (part >> 1), token = 16 * tile + row;
  const uint32_t norms = slot0 + tile * T::kSlot + 2 * row;
  const bool ok = ((loaded >> tile) & 1u) && wtok + token < tok1;
  const float nk = lds_half(norms + T::kOffNK), nv = lds_half(norms + T::kOffNV);
  bool above = false;
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
    s[h] = ok ? s[h] * nk : -INFINITY;
    above |= s[h] > st.M[h];
  }
  // ---- a score above its head's reference: new references, state rescaled ---------
  if (__any_sync(kFull, above)) {
    float alpha[kHeads];
#pragma unroll
    for (int h = 0; h < kHeads; ++h) {
      const float mx = warp_max(s[h]);
      const float now = mx > st.M[h] ? mx + kSlack : st.M[h];
      alpha[h] = now != st.M[h] ? ex2(st.M[h] - now) : 1.f;       // (2^(-inf - x) = 0: nothing seen yet)
      st.M[h] = now;
      st.l[h] *= alpha[h];
    }
#pragma unroll
    for (int p = 0; p < kHeads / 2; ++p) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 a = halves(st.acc[p][i]);
        st.acc[p][i] = pair(a.x * alpha[2 * p], a.y * alpha[2 * p + 1]);
      }
    }
  }
  // ---- probabilities; weights of the values -> shared memory ----------------------
  float v[kHeads];
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
    const float pr = ex2(s[h] - (st.M[h] == -INFINITY ? 0.f : st.M[h]));
    st.l[h] += pr;
    v[h] = ok ? pr * nv : 0.f;                                    // (the norm of a token that is not there is anything)
  }
  sts_f4(weights + token * kWeightRow, v[0], v[1], v[2], v[3]);
  sts_f4(weights + token * kWeightRow + 16, v[4], v[5], v[6], v[7]);
  __syncwarp();
  // ---- values ---------------------------------------------------------------------
  const int gq = lane >> 3, dq = lane & 7;
  constexpr int NB = T::BWV, NW = (NB + 3) / 4;                   // bytes and words of eight codes
#pragma unroll 4
  for (int it = 0; it < kIterTokens / 4; ++it) {
    const uint32_t at = slot0 + (it >> 2) * T::kSlot + T::kOffV + (4 * (it & 3) + gq) * T::kVRow;
    uint32_t w[NW];
    if constexpr (NB % 4 == 0) {
      load_words<NB>(at + dq * NB, w);
    } else {                                                      // six bytes: half-word aligned
      static_assert(NB == 6, "six bytes");
      const uint32_t word = at + ((dq * NB) & ~3), x = lds32(word), y = lds32(word + 4), sh = (dq & 1) * 16;
      w[0] = __funnelshift_r(x, y, sh);
      w[1] = y >> sh;
    }
    uint64_t p[4];
    lds_pairs(weights + (4 * it + gq) * kWeightRow, p[0], p[1]);
    lds_pairs(weights + (4 * it + gq) * kWeightRow + 16, p[2], p[3]);
    value_steps<T::BWV, 0>(w, sel_v, p, st.acc);
  }
}

// The warp's state [head][coordinate], then m[8], l[8], to shared address `at`.
__device__ __forceinline__ void store_state(State &st, uint32_t at, int lane) {
  constexpr uint32_t kFull = 0xffffffffu;
  // lanes that share coordinates add up: heads 4 (gq & 1) + 2 (gq >> 1) + {0, 1} stay
  const bool odd = lane & 8, high = lane & 16;
  float x[2][8];                                                  // [head of the pair][coordinate]
  uint64_t kept[2][8];
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint64_t give = odd ? st.acc[k][i] : st.acc[k + 2][i], keep = odd ? st.acc[k + 2][i] : st.acc[k][i];
      const float2 g = halves(give), m = halves(keep);
      kept[k][i] = pair(m.x + __shfl_xor_sync(kFull, g.x, 8), m.y + __shfl_xor_sync(kFull, g.y, 8));
    }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 g = halves(high ? kept[0][i] : kept[1][i]), m = halves(high ? kept[1][i] : kept[0][i]);
    x[0][i] = m.x + __shfl_xor_sync(kFull, g.x, 16);
    x[1][i] = m.y + __shfl_xor_sync(kFull, g.y, 16);
  }
  const int head = (odd ? 4 : 0) + (high ? 2 : 0);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t dst = at + 4u * ((head + k) * kD + 8 * (lane & 7));
    sts_f4(dst, x[k][0], x[k][1], x[k][2], x[k][3]);
    sts_f4(dst + 16, x[k][4], x[k][5], x[k][6], x[k][7]);
  }
#pragma unroll
  for (int h = 0; h < kHeads; ++h) {
    const float l = warp_sum(st.l[h]);
    if (lane == 0) {
      sts32(at + 4u * (kHeads * kD + h), __float_as_uint(st.M[h]));
      sts32(at + 4u * (kHeads * kD + kHeads + h), __float_as_uint(l));
    }
  }
}

}  // namespace scan32
}  // namespace wtq
