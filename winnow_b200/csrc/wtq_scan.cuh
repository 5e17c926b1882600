// The page scan of the one-launch decode kernel (wtq_decode_fused.cu): how a 16-token
// tile lies in shared memory, and at head_dim 128 the fragments of the score and value
// MMAs built from packed codes and one 32-token window of the online softmax, by the
// steps of the split-K scan (wtq_decode_mma.cu, which keeps its own: see there).
#pragma once

#include <type_traits>

#include "wtq_decode.cuh"
#include "wtq_lut.cuh"

namespace wtq {
namespace mma {

constexpr int kTileTokens = 16;
constexpr int kTilesPerIter = 2;                       // 32 tokens per window
constexpr int kIterTokens = kTileTokens * kTilesPerIter;
constexpr uint32_t kSmemLimit = 227 * 1024;
constexpr float kPreciseAbove = 8.0f;   // |score| (log2 units) that triggers fp32 rescoring
constexpr float kSlack = 4.0f;          // the softmax reference is set this far above a new maximum

constexpr int cmax(int a, int b) { return a > b ? a : b; }
constexpr int cmin(int a, int b) { return a < b ? a : b; }

// One tile slot: K rows | V rows (VROW apart) | fp16 norms of K | of V.
template <int D_, int BWK_, int BWV_, int VROW_> struct Slot {
  static constexpr int D = D_, BWK = BWK_, BWV = BWV_;
  static constexpr int NBK = D * BWK / 8, NBV = D * BWV / 8;    // bytes per packed row
  static constexpr int kVRow = VROW_;
  static constexpr int kOffV = kTileTokens * NBK;
  static constexpr int kOffNK = kOffV + kTileTokens * kVRow;
  static constexpr int kOffNV = kOffNK + 32;
  static constexpr int kSlot = kOffNV + 32;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void griddep_wait() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}
__device__ __forceinline__ void griddep_launch() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

}  // namespace mma

using namespace mma;

// Value side of one tile: the lane holds coordinates (D/8)g .. of tokens 2t,
// 2t+1 (A, B) and 2t+8, 2t+9 (C, D); `rows` = address of row 2t of the value
// rows.  MMA j takes coordinates (D/8)g+2j (row g) and (D/8)g+2j+1 (row g+8)
// of the output tile.
template <int D, int BW, int VROW>
__device__ __forceinline__ void value_mmas(uint32_t rows, int g, uint32_t sel, uint32_t pb0,
                                           uint32_t pb1, float (&acc)[D / 16][4]) {
  constexpr int NB8 = D / 8 * BW / 8;               // bytes of the lane's D / 8 codes
  if constexpr (BW == 4) {
    constexpr int NW = NB8 / 4;
    const uint32_t at = rows + g * NB8;
    uint32_t wa[NW], wb[NW], wc[NW], wd[NW];
    load_words<NB8>(at, wa);
    load_words<NB8>(at + VROW, wb);
    load_words<NB8>(at + 8 * VROW, wc);
    load_words<NB8>(at + 9 * VROW, wd);
    // byte j of lo_* : low nibbles of tokens (A | B << 4) at coordinate (D/8)g+2j
    // byte j of hi_* : high nibbles, coordinate (D/8)g+2j+1
    uint32_t lo_ab[NW], hi_ab[NW], lo_cd[NW], hi_cd[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      lo_ab[i] = (wa[i] & 0x0F0F0F0Fu) | ((wb[i] << 4) & 0xF0F0F0F0u);
      hi_ab[i] = ((wa[i] >> 4) & 0x0F0F0F0Fu) | (wb[i] & 0xF0F0F0F0u);
      lo_cd[i] = (wc[i] & 0x0F0F0F0Fu) | ((wd[i] << 4) & 0xF0F0F0F0u);
      hi_cd[i] = ((wc[i] >> 4) & 0x0F0F0F0Fu) | (wd[i] & 0xF0F0F0F0u);
    }
    // The sixteen table addresses of a word are formed first, then the sixteen
    // lookups are issued, then the four MMAs: a lookup never waits for the
    // byte-permute that builds its own address.
#pragma unroll
    for (int h = 0; h < NW; ++h) {
      uint32_t ad[4][4], f[4][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t src = q == 0 ? lo_ab[h] : q == 1 ? hi_ab[h] : q == 2 ? lo_cd[h] : hi_cd[h];
        ad[0][q] = lut_addr<0>(src, sel); ad[1][q] = lut_addr<1>(src, sel);
        ad[2][q] = lut_addr<2>(src, sel); ad[3][q] = lut_addr<3>(src, sel);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) f[j][q] = lds32(ad[j][q]);
#pragma unroll
      for (int j = 0; j < 4; ++j) mma16816(acc[4 * h + j], f[j][0], f[j][1], f[j][2], f[j][3], pb0, pb1);
    }
  } else {
    constexpr int NW = NB8 / 4;
    uint32_t wa[NW], wb[NW], wc[NW], wd[NW];
    const uint32_t at = rows + g * NB8;
    load_words<NB8>(at, wa);
    load_words<NB8>(at + VROW, wb);
    load_words<NB8>(at + 8 * VROW, wc);
    load_words<NB8>(at + 9 * VROW, wd);
    auto one = [&](auto jc) {
      constexpr int j = decltype(jc)::value;
      mma16816(acc[j],
               join(lut_code<BW, 2 * j>(wa, sel), lut_code<BW, 2 * j>(wb, sel)),
               join(lut_code<BW, 2 * j + 1>(wa, sel), lut_code<BW, 2 * j + 1>(wb, sel)),
               join(lut_code<BW, 2 * j>(wc, sel), lut_code<BW, 2 * j>(wd, sel)),
               join(lut_code<BW, 2 * j + 1>(wc, sel), lut_code<BW, 2 * j + 1>(wd, sel)), pb0, pb1);
    };
    one(std::integral_constant<int, 0>{}); one(std::integral_constant<int, 1>{});
    one(std::integral_constant<int, 2>{}); one(std::integral_constant<int, 3>{});
    one(std::integral_constant<int, 4>{}); one(std::integral_constant<int, 5>{});
    one(std::integral_constant<int, 6>{}); one(std::integral_constant<int, 7>{});
  }
}

// Scores of one tile: S^T fragment (rows g, g+8; heads 2t, 2t+1), unscaled.
// `at` = address of the lane's D / 4 codes of token row g.  Even and odd
// contraction steps accumulate separately (two chains of dependent MMAs
// instead of one of twice the length).
template <int D, int BW>
__device__ __forceinline__ void key_mmas(uint32_t at, uint32_t sel, const uint32_t (&qf)[D / 16][2],
                                         float (&c)[4]) {
  constexpr int NB4 = D / 4 * BW / 8;               // bytes of D / 4 codes
  constexpr int NW = NB4 / 4, NB = D * BW / 8;
  uint32_t w0[NW], w1[NW];
  load_words<NB4>(at, w0);
  load_words<NB4>(at + 8 * NB, w1);
  constexpr int kChains = 2;
  float cc[kChains][4];
#pragma unroll
  for (int i = 0; i < kChains; ++i) cc[i][0] = cc[i][1] = cc[i][2] = cc[i][3] = 0.f;
  if constexpr (BW == 4) {
    // per word of the two rows: eight addresses, eight lookups, two MMAs
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      uint32_t ad[8], f[8];
      ad[0] = lut_addr<0>(w0[j], sel); ad[1] = lut_addr<0>(w1[j], sel);
      ad[2] = lut_addr<1>(w0[j], sel); ad[3] = lut_addr<1>(w1[j], sel);
      ad[4] = lut_addr<2>(w0[j], sel); ad[5] = lut_addr<2>(w1[j], sel);
      ad[6] = lut_addr<3>(w0[j], sel); ad[7] = lut_addr<3>(w1[j], sel);
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = lds32(ad[i]);
      mma16816(cc[0], f[0], f[1], f[2], f[3], qf[2 * j][0], qf[2 * j][1]);
      mma16816(cc[1], f[4], f[5], f[6], f[7], qf[2 * j + 1][0], qf[2 * j + 1][1]);
    }
  } else {
    auto one = [&](auto ksc) {
      constexpr int ks = decltype(ksc)::value;
      uint32_t a[4];
      key_fragment<BW, ks>(w0, w1, sel, a);
      mma16816(cc[ks % kChains], a[0], a[1], a[2], a[3], qf[ks][0], qf[ks][1]);
    };
    one(std::integral_constant<int, 0>{}); one(std::integral_constant<int, 1>{});
    one(std::integral_constant<int, 2>{}); one(std::integral_constant<int, 3>{});
    one(std::integral_constant<int, 4>{}); one(std::integral_constant<int, 5>{});
    one(std::integral_constant<int, 6>{}); one(std::integral_constant<int, 7>{});
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float v = cc[0][e];
#pragma unroll
    for (int i = 1; i < kChains; ++i) v += cc[i][e];
    c[e] = v;
  }
}

// fp32 scores of tile rows g and g+8 against two query rows (already rotated
// and scaled; any address space), times the key norms: {row g . qa, row g . qb,
// row g+8 . qa, row g+8 . qb}.  Kept out of line: it runs only for windows
// whose fp16 scores came out large, and must not cost the common path
// registers.
template <int D, int BW>
__device__ __noinline__ float4 precise_scores(uint32_t kbase, uint32_t nk_addr, int g,
                                              const float *qa, const float *qb,
                                              const float *centroids) {
  constexpr int NB = D * BW / 8;
  float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
  const uint32_t r0 = kbase + g * NB, r1 = kbase + (g + 8) * NB;
#pragma unroll 1
  for (int d = 0; d < D; ++d) {
    const int bit = d * BW, b0 = bit >> 3, sh = bit & 7;
    uint32_t x0 = lds_u8(r0 + b0), x1 = lds_u8(r1 + b0);
    if (sh + BW > 8) {
      x0 |= lds_u8(r0 + b0 + 1) << 8;
      x1 |= lds_u8(r1 + b0 + 1) << 8;
    }
    const float c0 = __ldg(centroids + ((x0 >> sh) & ((1u << BW) - 1u)));
    const float c1 = __ldg(centroids + ((x1 >> sh) & ((1u << BW) - 1u)));
    const float fa = qa[d], fb = qb[d];
    d0 = fmaf(fa, c0, d0); d1 = fmaf(fb, c0, d1);
    d2 = fmaf(fa, c1, d2); d3 = fmaf(fb, c1, d3);
  }
  const float nk0 = lds_half(nk_addr + g * 2), nk1 = lds_half(nk_addr + (g + 8) * 2);
  return make_float4(d0 * nk0, d1 * nk0, d2 * nk1, d3 * nk1);
}

// Flash-decoding state of one warp: query fragments (head g), un-normalised
// output fragments, and the softmax state of heads 2t, 2t+1: reference M (the
// probabilities are 2^(s - M), M >= every score seen), -M with -inf replaced
// by 0, the bound a window's scores (relative to M) must stay under to take
// the short path, and the sum of the probabilities.
template <int D> struct ScanState {
  uint32_t qf[D / 16][2];
  float acc[D / 16][4];
  float M0, M1, neg0, neg1, hi0, hi1, l0, l1;
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int j = 0; j < D / 16; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    M0 = M1 = hi0 = hi1 = -INFINITY;
    neg0 = neg1 = l0 = l1 = 0.f;
  }
};

// One window of two tiles at shared address `slot0` (first token `wtok`).  A
// window whose 32 tokens all exist on pages that were found needs no masks;
// MASKED is the form for the last window of a range (tokens from `tok1` on do
// not exist) and for refused page ids (`loaded`: one bit per tile).  `q0` =
// the group's `n_rep` rotated query rows in fp32.
template <class T, bool MASKED>
__device__ __forceinline__ void scan_window(ScanState<T::D> &st, uint32_t slot0, int wtok, int tok1,
                                            uint32_t loaded, int g, int t, uint32_t sel_k,
                                            uint32_t sel_v, const float *q0, int n_rep,
                                            const float *k_centroids) {
  constexpr uint32_t kFull = 0xffffffffu;
  constexpr int D = T::D;
  // ---- scores of the tiles --------------------------------------------
  float c[kTilesPerIter][4], a[kTilesPerIter][4], nk[kTilesPerIter][2];
  bool ok[kTilesPerIter][2];
#pragma unroll
  for (int u = 0; u < kTilesPerIter; ++u) {
    const uint32_t slot = slot0 + u * T::kSlot;
    key_mmas<D, T::BWK>(slot + g * T::NBK + t * (D / 4 * T::BWK / 8), sel_k, st.qf, c[u]);
    nk[u][0] = lds_half(slot + T::kOffNK + g * 2);
    nk[u][1] = lds_half(slot + T::kOffNK + (g + 8) * 2);
    ok[u][0] = ok[u][1] = true;
  }
  bool slow = true;
  if constexpr (!MASKED) {
    float top0 = -INFINITY, top1 = -INFINITY;
#pragma unroll
    for (int u = 0; u < kTilesPerIter; ++u) {
      a[u][0] = fmaf(c[u][0], nk[u][0], st.neg0); a[u][1] = fmaf(c[u][1], nk[u][0], st.neg1);
      a[u][2] = fmaf(c[u][2], nk[u][1], st.neg0); a[u][3] = fmaf(c[u][3], nk[u][1], st.neg1);
      top0 = max3(top0, a[u][0], a[u][2]);
      top1 = max3(top1, a[u][1], a[u][3]);
    }
    slow = __any_sync(kFull, top0 > st.hi0 || top1 > st.hi1);
  }
  if (slow) {
    // A score above the reference (or the first window, a large score, a
    // partly filled window): exact scores, fp32 rescoring when they are
    // large, new reference, state rescaled.
    float s[kTilesPerIter][4];
    float big = 0.f;
#pragma unroll
    for (int u = 0; u < kTilesPerIter; ++u) {
      s[u][0] = c[u][0] * nk[u][0]; s[u][1] = c[u][1] * nk[u][0];
      s[u][2] = c[u][2] * nk[u][1]; s[u][3] = c[u][3] * nk[u][1];
      if constexpr (MASKED) {
        const int tok = wtok + u * kTileTokens;
        const bool page_ok = (loaded >> u) & 1u;
        ok[u][0] = page_ok && tok + g < tok1;
        ok[u][1] = page_ok && tok + g + 8 < tok1;
      }
      if (ok[u][0]) big = fmaxf(big, fmaxf(fabsf(s[u][0]), fabsf(s[u][1])));
      if (ok[u][1]) big = fmaxf(big, fmaxf(fabsf(s[u][2]), fabsf(s[u][3])));
    }
    // fp16 operands carry about 2^-11.5 of the score scale as error; when
    // any score of this window is large (|s| > 8 in log2 units) its tiles
    // are scored again in fp32 on the CUDA cores, so that large logits
    // cost time, not accuracy.
    if (__any_sync(kFull, big > kPreciseAbove)) {
      const bool h0 = 2 * t < n_rep, h1 = 2 * t + 1 < n_rep;
      const float *qa = q0 + (h0 ? 2 * t : 0) * D, *qb = q0 + (h1 ? 2 * t + 1 : 0) * D;
#pragma unroll
      for (int u = 0; u < kTilesPerIter; ++u) {
        const uint32_t slot = slot0 + u * T::kSlot;
        const float4 d = precise_scores<D, T::BWK>(slot, slot + T::kOffNK, g, qa, qb, k_centroids);
        s[u][0] = h0 ? d.x : 0.f; s[u][1] = h1 ? d.y : 0.f;
        s[u][2] = h0 ? d.z : 0.f; s[u][3] = h1 ? d.w : 0.f;
      }
    }
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int u = 0; u < kTilesPerIter; ++u) {
      if (!ok[u][0]) s[u][0] = s[u][1] = -INFINITY;
      if (!ok[u][1]) s[u][2] = s[u][3] = -INFINITY;
      mx0 = fmaxf(mx0, fmaxf(s[u][0], s[u][2]));
      mx1 = fmaxf(mx1, fmaxf(s[u][1], s[u][3]));
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      mx0 = fmaxf(mx0, __shfl_xor_sync(kFull, mx0, o));
      mx1 = fmaxf(mx1, __shfl_xor_sync(kFull, mx1, o));
    }
    const float n0 = mx0 > st.M0 ? mx0 + kSlack : st.M0;
    const float n1 = mx1 > st.M1 ? mx1 + kSlack : st.M1;
    if (__any_sync(kFull, n0 != st.M0 || n1 != st.M1)) {
      // 2^(-inf - x) = 0 for the first window; an unchanged reference keeps 1
      const float alpha0 = n0 != st.M0 ? ex2(st.M0 - n0) : 1.f;
      const float alpha1 = n1 != st.M1 ? ex2(st.M1 - n1) : 1.f;
#pragma unroll
      for (int j = 0; j < D / 16; ++j) {
        st.acc[j][0] *= alpha0; st.acc[j][1] *= alpha1;
        st.acc[j][2] *= alpha0; st.acc[j][3] *= alpha1;
      }
      st.l0 *= alpha0;
      st.l1 *= alpha1;
      st.M0 = n0;
      st.M1 = n1;
    }
    // exp2(-inf - -inf) is defined as 0: with nothing seen the base is 0
    st.neg0 = st.M0 == -INFINITY ? 0.f : -st.M0;
    st.neg1 = st.M1 == -INFINITY ? 0.f : -st.M1;
    // short path while every score stays under the reference and under the
    // rescoring threshold; never when the running maximum is a large
    // negative number (all scores are large then)
    st.hi0 = (st.M0 == -INFINITY || st.M0 - kSlack < -kPreciseAbove) ? -INFINITY
                                                                     : fminf(0.f, kPreciseAbove - st.M0);
    st.hi1 = (st.M1 == -INFINITY || st.M1 - kSlack < -kPreciseAbove) ? -INFINITY
                                                                     : fminf(0.f, kPreciseAbove - st.M1);
#pragma unroll
    for (int u = 0; u < kTilesPerIter; ++u) {
      a[u][0] = s[u][0] + st.neg0; a[u][1] = s[u][1] + st.neg1;
      a[u][2] = s[u][2] + st.neg0; a[u][3] = s[u][3] + st.neg1;
    }
  }

  // ---- values of the tiles --------------------------------------------
#pragma unroll
  for (int u = 0; u < kTilesPerIter; ++u) {
    const uint32_t slot = slot0 + u * T::kSlot;
    const float nv0 = lds_half(slot + T::kOffNV + g * 2);
    const float nv1 = lds_half(slot + T::kOffNV + (g + 8) * 2);
    const float p0 = ex2(a[u][0]), p1 = ex2(a[u][1]);
    const float p2 = ex2(a[u][2]), p3 = ex2(a[u][3]);
    st.l0 += p0 + p2;
    st.l1 += p1 + p3;
    // rows g / g+8 of P' (token x head) -> B fragment (token pairs of head g)
    uint32_t r0 = pack_half2(p0 * nv0, p1 * nv0), r1 = pack_half2(p2 * nv1, p3 * nv1);
    if constexpr (MASKED) {
      r0 = ok[u][0] ? r0 : 0u;
      r1 = ok[u][1] ? r1 : 0u;
    }
    const uint32_t pb0 = movmatrix_trans(r0), pb1 = movmatrix_trans(r1);
    value_mmas<D, T::BWV, T::kVRow>(slot + T::kOffV + (2 * t) * T::kVRow, g, sel_v, pb0, pb1, st.acc);
  }
}

}  // namespace wtq
