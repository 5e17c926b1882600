// Decode attention in ONE launch: for calls whose work fits about one block per
// multiprocessor, where the split-K path (rotation, page scan, merge: three
// dependent kernels) is bound by the kernels' own latencies, and for head_dim
// 64, which the split-K tensor-core scan does not serve (in fp32: wtq_scan32.cuh).
//
// A cluster of c blocks (c = 1, 2, 4, 8) owns one (sequence, kv head) group.
// Every block rotates the group's query rows itself, each of its warps scans a
// contiguous share of the sequence's 32-token windows (head_dim 128 exactly as the
// split-K scan does, wtq_scan.cuh), the block merges its warps' states through shared
// memory, the blocks of the cluster exchange theirs through distributed shared
// memory, and each of them rotates 1/c of the output coordinates back and
// stores them.  Nothing goes through global memory but the inputs and the
// result, so the call needs no workspace.
//
// What does not depend on the kernel ahead of it in the stream (the lookup
// tables, this block's share of Pi_K) is fetched before griddepcontrol.wait, so
// after an append launched by this library it overlaps that kernel's tail.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "wtq_scan32.cuh"

namespace wtq {
namespace fused {

// Shared addresses below are offsets from an origin: the 64 KB boundary under the
// start of dynamic shared memory (in a cluster, a block's own addresses carry its
// rank in their upper bits), so that the tables start at origin + 0x10000 and the
// byte-permute that forms a table address takes its upper half from `sel`.
constexpr uint32_t kBase = 2048;            // dynamic shared memory must start at or below this offset
constexpr int kHeads = 8;                   // query heads of a group (MMA columns)
constexpr int kRotThreads = 256;            // threads of the two rotations

// Row stride of the value rows in a tile slot.  head_dim 128: padded so that the lanes'
// loads (group g: D/8 codes, t: two rows further) fall into different banks.
constexpr int vrow(int D, int bw) {
  return D == 128 ? (bw == 4 ? 80 : bw == 6 ? 112 : 144) : 8 * bw;
}

template <int D, int BWK, int BWV> struct Cfg : Slot<D, BWK, BWV, vrow(D, BWV)> {
  using Base = Slot<D, BWK, BWV, vrow(D, BWV)>;
  static constexpr int kPart = D * D / kRotThreads;             // coordinates per thread of the query rotation
  static constexpr int kQRow = D + 4 * (D / kPart);             // staged query row (4 words of pad per part)
  static constexpr uint32_t kQ = kBase;                         // staged queries; later the block's merged state
  static constexpr bool kFp32 = D == 64;                        // which scan: wtq_scan32.cuh or wtq_scan.cuh
  static constexpr uint32_t kQRot = kQ + kHeads * kQRow * 4;    // rotated queries; later the sums a
  static constexpr uint32_t kQRotBytes = 4 * (kFp32 ? scan32::kQueryWords : kHeads * D);
  static constexpr uint32_t kML = kQRot + kQRotBytes;           // the block's m[8], l[8]
  static constexpr uint32_t kRings = (kML + 2 * kHeads * 4 + 127) / 128 * 128;
  static constexpr int kRingWindows = 2 * kTilesPerIter * Base::kSlot;              // two windows per warp
  static constexpr int kRing = kRingWindows + (kFp32 ? (int)scan32::kWeights : 0);  // and the value weights
  static constexpr uint32_t kLutBytes =
      kFp32 ? scan32::table_bytes(BWK, BWV) : cmax(lut_entries(BWK), lut_entries(BWV)) * 256u;
  static constexpr int kRingsBelow = (int)((kLutAddr - kRings) / kRing);
  static constexpr int kRingsAbove = (int)((kSmemLimit - kLutAddr - kLutBytes) / kRing);
  static constexpr int kWarps = cmin(12, kRingsBelow + kRingsAbove);
  static constexpr int kThreads = 32 * kWarps;
  static constexpr uint32_t kDynamic =
      kLutAddr + kLutBytes + (uint32_t)cmax(kWarps - kRingsBelow, 0) * kRing;
  // a warp's state (acc [8][D], m, l) replaces its ring after the scan; the output
  // rotation's partial sums replace the rings below the tables after the merge
  static_assert(kRing >= kHeads * D * 4 + 2 * kHeads * 4 && kRing % 16 == 0, "state fits the ring");
  static_assert(kRings + kRotThreads * kHeads * 4 <= kLutAddr, "partial sums fit");
  static_assert(kThreads >= kRotThreads && kDynamic <= kSmemLimit, "shared memory budget");
  __device__ static uint32_t ring_address(int w) {
    return w < kRingsBelow ? kRings + (uint32_t)w * kRing
                           : kLutAddr + kLutBytes + (uint32_t)(w - kRingsBelow) * kRing;
  }
};

struct Params {
  DecodeSideDev k, v;
  const void *q;
  int dtype;
  int64_t qsb, qsh;
  float q_scale;             // scale * log2(e)
  void *out;
  int64_t osb, osh;
  const int32_t *page_table;
  int64_t table_stride;
  const int32_t *seq_lens;
  int n_rep, S, P, max_pages;
  int32_t *status;
};

__device__ __forceinline__ float lds_f(uint32_t a) { return __uint_as_float(lds32(a)); }
__device__ __forceinline__ void sts_f(uint32_t a, float v) { sts32(a, __float_as_uint(v)); }
__device__ __forceinline__ float4 lds_f4(uint32_t a) {
  const uint4 v = lds128(a);
  return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
// word at shared address `a` of block `rank` of the cluster
__device__ __forceinline__ float lds_peer(uint32_t a, int rank) {
  float v;
  asm volatile(
      "{\n\t.reg .b32 r;\n\tmapa.shared::cluster.u32 r, %1, %2;\n\tld.shared::cluster.f32 %0, [r];\n\t}\n"
      : "=f"(v) : "r"(a), "r"(rank) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_arrive() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

template <int D, int BWK, int BWV>
__global__ void __launch_bounds__(Cfg<D, BWK, BWV>::kThreads, 1) decode_fused_kernel(Params p) {
  using C = Cfg<D, BWK, BWV>;
  constexpr uint32_t kFull = 0xffffffffu;
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int rank = blockIdx.x, c = gridDim.x, kvh = blockIdx.y, b = blockIdx.z;
  const uint32_t smem = (uint32_t)__cvta_generic_to_shared(dyn_smem);
  const uint32_t origin = smem & ~0xffffu;
  if (smem > origin + kBase) {                                  // layout assumption broken: refuse
    if (p.status && tid == 0) atomicOr(p.status, WTQ_STATUS_LAYOUT);
    return;                                                     // (the same for every block of the cluster)
  }
  const uint32_t kq = origin + C::kQ, kqrot = origin + C::kQRot, kml = origin + C::kML, lut = origin + kLutAddr;
  // ---- constants: this thread's share of Pi_K, the lookup tables ---------------
  const int rc = tid / (D / C::kPart), rpart = tid % (D / C::kPart);   // output coordinate, part of the sum
  float4 w[C::kPart / 4];
  if (tid < kRotThreads) {
    const float4 *src = reinterpret_cast<const float4 *>(p.k.Pi + rc * D + rpart * C::kPart);
#pragma unroll
    for (int j = 0; j < C::kPart / 4; ++j) w[j] = __ldg(src + j);
  }
  // a lane makes the words of 32 (index, side) pairs at a time, the warp spreads each over its 32 banks
  constexpr int kPairs = (int)(C::kLutBytes / 128);
  for (int p0 = 32 * warp; p0 < kPairs; p0 += 32 * C::kWarps) {
    uint32_t word;
    if constexpr (C::kFp32) word = scan32::table_word(p0 + lane, BWK, BWV, p.k.centroids, p.v.centroids);
    else word = mma::lut_word((p0 + lane) * 32, BWK, BWV, p.k.centroids, p.v.centroids);
#pragma unroll
    for (int i = 0; i < 32; ++i) sts32(lut + 128u * (p0 + i) + 4u * lane, __shfl_sync(kFull, word, i));
  }

  griddep_wait();
  griddep_launch();
  // ---- this warp's tokens -------------------------------------------------------
  int L = p.seq_lens[b];
  L = L < 0 ? 0 : L;
  if (L > p.max_pages * p.S) {
    L = p.max_pages * p.S;
    if (p.status && tid == 0) atomicOr(p.status, WTQ_STATUS_BAD_POSITION);
  }
  const int windows = (L + kIterTokens - 1) / kIterTokens;
  const int worker = rank * C::kWarps + warp, workers = c * C::kWarps;
  const int tok0 = kIterTokens * (int)((int64_t)windows * worker / workers);
  const int tok1 = min(L, kIterTokens * (int)((int64_t)windows * (worker + 1) / workers));
  // ---- the group's queries -> shared memory (fp32) -------------------------------
  for (int e = tid; e < kHeads * D; e += C::kThreads) {
    const int h = e / D, d = e - h * D;
    float x = 0.f;
    if (h < p.n_rep)
      x = load_as_float(p.q, (int64_t)b * p.qsb + (int64_t)(kvh * p.n_rep + h) * p.qsh + d, p.dtype);
    sts_f(kq + 4u * (h * C::kQRow + d + 4 * (d / C::kPart)), x);
  }
  // ---- the copies: one window ahead of the arithmetic ----------------------------
  const uint32_t ring = origin + C::ring_address(warp);
  const int ts = 27 - __clz(p.S), tmask = (p.S >> 4) - 1;       // tiles per page as a shift and a mask
  const int tiles = tok1 > tok0 ? (tok1 - tok0 + kTileTokens - 1) / kTileTokens : 0;
  const int page0 = tok0 >> (ts + 4);
  int tile_at = (tok0 >> 4) - (page0 << ts);                    // tile relative to the first tile of page ids_first
  const int32_t *table_row = p.page_table + (int64_t)b * p.table_stride;
  int ids_first = page0, ids0, ids1;
  auto load_ids = [&]() {
    ids0 = ids_first + lane < p.max_pages ? table_row[ids_first + lane] : -1;
    ids1 = ids_first + 32 + lane < p.max_pages ? table_row[ids_first + 32 + lane] : -1;
  };
  ids0 = ids1 = -1;
  if (tiles > 0) load_ids();
  const uint8_t *src_k = p.k.pages + (int64_t)kvh * p.k.head_stride;
  const uint8_t *src_v = p.v.pages + (int64_t)kvh * p.v.head_stride;
  const bool n_is_v = lane >= 2;
  const __half *src_n = n_is_v ? p.v.norms + (int64_t)kvh * p.v.norm_head_stride + (lane - 2) * 8
                               : p.k.norms + (int64_t)kvh * p.k.norm_head_stride + lane * 8;
  const int64_t n_page = n_is_v ? p.v.norm_page_stride : p.k.norm_page_stride;
  const uint32_t n_dst = n_is_v ? C::kOffNV + (lane - 2) * 16 : C::kOffNK + lane * 16;
  int issued = 0;
  uint32_t bad = 0;                                             // refused tiles: bit 2 * half + tile
  auto issue_window = [&]() {                                   // window issued / 2, always one commit
    const int half = (issued >> 1) & 1;
    bad &= ~(3u << (2 * half));
#pragma unroll
    for (int u = 0; u < kTilesPerIter; ++u) {
      if (issued + u < tiles) {
        const int q = tile_at + u;
        int rel = q >> ts;
        const int sub = (q & tmask) << 4;                       // first token of the tile inside its page
        if (rel >= 64) {
          ids_first += rel & ~31;
          tile_at -= (rel & ~31) << ts;
          rel &= 31;
          load_ids();
        }
        const int pid = __shfl_sync(kFull, rel < 32 ? ids0 : ids1, rel);
        if ((uint32_t)pid < (uint32_t)p.P) {
          const uint32_t dst = ring + (uint32_t)(half * kTilesPerIter + u) * C::kSlot;
          const uint8_t *ks = src_k + (int64_t)pid * p.k.page_stride + sub * C::NBK;
          const uint8_t *vs = src_v + (int64_t)pid * p.v.page_stride + sub * C::NBV;
#pragma unroll
          for (int i = lane; i < C::NBK; i += 32) cp_async16(dst + i * 16, ks + i * 16);
          constexpr int kRowPieces = C::NBV / 16;
#pragma unroll
          for (int i = lane; i < C::NBV; i += 32) {
            const int row = i / kRowPieces, piece = i - row * kRowPieces;
            cp_async16(dst + C::kOffV + row * C::kVRow + piece * 16, vs + i * 16);
          }
          if (lane < 4) cp_async16(dst + n_dst, src_n + (int64_t)pid * n_page + sub);
        } else {
          bad |= 1u << (2 * half + u);
          if (p.status && lane == 0) atomicOr(p.status, WTQ_STATUS_BAD_PAGE);
        }
      }
    }
    tile_at += kTilesPerIter;
    issued += kTilesPerIter;
    cp_async_commit();
  };
  issue_window();
  __syncthreads();                                              // queries and tables are in place

  // ---- query rotation: q_rot[h][rc] = q_scale * sum_d q[h][d] Pi_K[rc][d] ---------
  if (tid < kRotThreads) {
    float acc[kHeads];
#pragma unroll
    for (int h = 0; h < kHeads; ++h) acc[h] = 0.f;
    const uint32_t at = kq + 4u * (rpart * (C::kPart + 4));
    auto heads = [&](auto first) {                              // four heads: independent chains
      constexpr int h0 = decltype(first)::value;
#pragma unroll
      for (int j = 0; j < C::kPart / 4; ++j)
#pragma unroll
        for (int h = h0; h < h0 + 4; ++h) {
          const float4 x = lds_f4(at + 4u * (h * C::kQRow + 4 * j));
          acc[h] = fmaf(x.x, w[j].x, acc[h]);
          acc[h] = fmaf(x.y, w[j].y, acc[h]);
          acc[h] = fmaf(x.z, w[j].z, acc[h]);
          acc[h] = fmaf(x.w, w[j].w, acc[h]);
        }
    };
    heads(std::integral_constant<int, 0>{});
    if (p.n_rep > 4) heads(std::integral_constant<int, 4>{});
#pragma unroll
    for (int h = 0; h < kHeads; ++h) {
#pragma unroll
      for (int o = 1; o < D / C::kPart; o <<= 1) acc[h] += __shfl_xor_sync(kFull, acc[h], o);
      if (rpart == 0)
        sts_f(kqrot + 4u * (C::kFp32 ? scan32::query_word(rc, h) : (uint32_t)(h * D + rc)), acc[h] * p.q_scale);
    }
  }
  __syncthreads();

  // ---- scan: this warp's windows; its state then replaces its ring -----------------
  const uint32_t sel_k = lut | (uint32_t)(lane << 2), sel_v = sel_k | 0x80u;
  const int n_full = tok1 > tok0 ? (tok1 - tok0) / kIterTokens : 0;
  const int n_iter = (tiles + kTilesPerIter - 1) / kTilesPerIter;
  auto walk = [&](auto window) {                                // window(slots, first token, refused tiles, whole)
    for (int it = 0; it < n_iter; ++it) {
      issue_window();
      cp_async_wait<1>();
      __syncwarp();
      const int half = it & 1;
      const uint32_t refused = (bad >> (2 * half)) & 3u;
      window(ring + (uint32_t)(half * kTilesPerIter) * C::kSlot, tok0 + it * kIterTokens, refused,
             it < n_full && refused == 0u);
      __syncwarp();
    }
    cp_async_wait<0>();
    __syncwarp();
  };
  if constexpr (C::kFp32) {
    scan32::State st;
    st.clear();
    walk([&](uint32_t slots, int first, uint32_t refused, bool) {
      scan32::window<typename C::Base>(st, slots, first, tok1, ~refused & 3u, lane, sel_k, sel_v, kqrot,
                                       ring + C::kRingWindows);
    });
    scan32::store_state(st, ring, lane);
  } else {
    ScanState<D> st;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {                       // head g, coordinates (D/4)t + 4ks ..
      const float4 x = lds_f4(kqrot + 4u * (g * D + (D / 4) * t + 4 * ks));
      st.qf[ks][0] = pack_half2(x.x, x.y);
      st.qf[ks][1] = pack_half2(x.z, x.w);
    }
    st.clear();
    const float *q0 = reinterpret_cast<const float *>(dyn_smem + (kqrot - smem));
    walk([&](uint32_t slots, int first, uint32_t refused, bool whole) {
      if (whole)
        scan_window<typename C::Base, false>(st, slots, 0, 0, 3u, g, t, sel_k, sel_v, q0, p.n_rep, p.k.centroids);
      else
        scan_window<typename C::Base, true>(st, slots, first, tok1, ~refused & 3u, g, t, sel_k, sel_v, q0, p.n_rep,
                                            p.k.centroids);
    });
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      st.l0 += __shfl_xor_sync(kFull, st.l0, o);
      st.l1 += __shfl_xor_sync(kFull, st.l1, o);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const uint32_t dst = ring + 4u * ((2 * t + e) * D + (D / 8) * g);
#pragma unroll
      for (int j = 0; j < D / 16; j += 2)
        asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(dst + 8u * j), "f"(st.acc[j][e]),
                     "f"(st.acc[j][2 + e]), "f"(st.acc[j + 1][e]), "f"(st.acc[j + 1][2 + e]) : "memory");
      if (g == 0) {
        sts_f(ring + 4u * (kHeads * D + 2 * t + e), e ? st.M1 : st.M0);
        sts_f(ring + 4u * (kHeads * D + kHeads + 2 * t + e), e ? st.l1 : st.l0);
      }
    }
  }

  // ---- merge of the block's warps -------------------------------------------------
  // this block's columns of Pi_V for the output rotation: requested now, used after the merge
  const int cols = D / c, parts = kRotThreads / cols, rows_of = D / parts;   // threads = (part, column)
  const int ocol = tid % cols, opart = tid / cols;
  constexpr int kMaxRows = D * D / kRotThreads;
  float pv[kMaxRows];
  if (tid < kRotThreads) {
    const float *src = p.v.Pi + (int64_t)opart * rows_of * D + rank * cols + ocol;
#pragma unroll
    for (int i = 0; i < kMaxRows; ++i) pv[i] = i < rows_of ? __ldg(src + i * D) : 0.f;
  }
  __syncthreads();
  const int elems = p.n_rep * D;
  for (int e = tid; e < elems; e += C::kThreads) {
    const int h = e / D, d = e - h * D;
    float mv[C::kWarps], m = -INFINITY;
#pragma unroll
    for (int i = 0; i < C::kWarps; ++i) {
      mv[i] = lds_f(origin + C::ring_address(i) + 4u * (kHeads * D + h));
      m = fmaxf(m, mv[i]);
    }
    float a = 0.f, l = 0.f;
#pragma unroll
    for (int i = 0; i < C::kWarps; ++i) {
      const float wt = mv[i] == -INFINITY ? 0.f : ex2(mv[i] - m);
      a = fmaf(wt, lds_f(origin + C::ring_address(i) + 4u * e), a);
      if (d == 0) l = fmaf(wt, lds_f(origin + C::ring_address(i) + 4u * (kHeads * D + kHeads + h)), l);
    }
    sts_f(kq + 4u * e, a);
    if (d == 0) {
      sts_f(kml + 4u * h, m);
      sts_f(kml + 4u * (kHeads + h), l);
    }
  }
  if (c > 1) {
    __syncwarp();
    cluster_arrive();                                           // (also orders the block's own threads)
    cluster_wait();
  } else {
    __syncthreads();
  }
  // ---- merge of the cluster's blocks, normalised: a[d][h] ---------------------------
  for (int e = tid; e < elems; e += C::kThreads) {
    const int h = e / D, d = e - h * D;
    float a, l;
    if (c == 1) {
      a = lds_f(kq + 4u * e);
      l = lds_f(kml + 4u * (kHeads + h));
    } else {
      float mr[8], lr[8], ar[8], m = -INFINITY;                 // all blocks' states in flight
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const bool on = r < c;
        mr[r] = on ? lds_peer(kml + 4u * h, r) : -INFINITY;
        lr[r] = on ? lds_peer(kml + 4u * (kHeads + h), r) : 0.f;
        ar[r] = on ? lds_peer(kq + 4u * e, r) : 0.f;
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) m = fmaxf(m, mr[r]);
      a = l = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const float wt = mr[r] == -INFINITY ? 0.f : ex2(mr[r] - m);
        a = fmaf(wt, ar[r], a);
        l = fmaf(wt, lr[r], l);
      }
    }
    sts_f(kqrot + 4u * (d * kHeads + h), l > 0.f ? a / fmaxf(l, 1e-30f) : 0.f);
  }
  __syncwarp();
  if (c > 1) cluster_arrive();                                  // this block no longer reads its peers
  __syncthreads();
  // ---- output rotation: out[h][col] = sum_d a[h][d] Pi_V[d][col] ---------------------
  if (tid < kRotThreads) {
    float o[kHeads];
#pragma unroll
    for (int h = 0; h < kHeads; ++h) o[h] = 0.f;
    const uint32_t at = kqrot + 4u * kHeads * (opart * rows_of);
    auto heads = [&](auto first) {
      constexpr int h0 = decltype(first)::value;
#pragma unroll
      for (int i = 0; i < kMaxRows; ++i) {
        if (i < rows_of) {
          const float4 x = lds_f4(at + 4u * (i * kHeads + h0));
          o[h0] = fmaf(x.x, pv[i], o[h0]);
          o[h0 + 1] = fmaf(x.y, pv[i], o[h0 + 1]);
          o[h0 + 2] = fmaf(x.z, pv[i], o[h0 + 2]);
          o[h0 + 3] = fmaf(x.w, pv[i], o[h0 + 3]);
        }
      }
    };
    heads(std::integral_constant<int, 0>{});
    if (p.n_rep > 4) heads(std::integral_constant<int, 4>{});
#pragma unroll
    for (int h = 0; h < kHeads; ++h)
      if (h < p.n_rep) sts_f(origin + C::kRings + 4u * ((opart * kHeads + h) * cols + ocol), o[h]);
  }
  __syncthreads();
  for (int e = tid; e < p.n_rep * cols; e += C::kThreads) {
    const int h = e / cols, col = e - h * cols;
    float v = 0.f;
    for (int i = 0; i < parts; ++i) v += lds_f(origin + C::kRings + 4u * ((i * kHeads + h) * cols + col));
    store_from_float(p.out, (int64_t)b * p.osb + (int64_t)(kvh * p.n_rep + h) * p.osh + rank * cols + col, v,
                     p.dtype);
  }
  __syncwarp();
  if (c > 1) cluster_wait();                                    // peers are done with this block's memory
}

// One-time set-up of an instantiation on the current device: its shared memory, and how
// many clusters of 1, 2, 4, 8 blocks can run at once (fewer than multiprocessors / size:
// a cluster lies within one GPC, and GPCs do not divide evenly).
struct Setup {
  std::atomic<int> state{0};                // 0: not done
  int clusters[4];
};
template <int D, int BWK, int BWV> int set_up(const Setup *&out) {
  using C = Cfg<D, BWK, BWV>;
  static Setup per_device[64];
  static std::mutex gate;
  int dev = 0;
  cudaGetDevice(&dev);
  Setup &s = per_device[dev & 63];
  out = &s;
  if (dev < 64 && s.state.load(std::memory_order_acquire)) return WTQ_OK;
  std::lock_guard<std::mutex> hold(gate);
  auto kernel = decode_fused_kernel<D, BWK, BWV>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::kDynamic);
  for (int i = 0; i < 4 && e == cudaSuccess; ++i) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1u << i;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1u << i);
    cfg.blockDim = dim3(C::kThreads);
    cfg.dynamicSmemBytes = C::kDynamic;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&s.clusters[i], kernel, &cfg);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();                     // the split-K path serves the call: its launches must not find this error
    return check_cuda(e, "wtq_decode: fused kernel set-up");
  }
  s.state.store(1, std::memory_order_release);
  return WTQ_OK;
}

template <int D, int BWK, int BWV>
int launch(const Params &p, int B, int Hkv, int cluster, cudaStream_t stream) {
  using C = Cfg<D, BWK, BWV>;
  const Setup *ready = nullptr;
  if (int rc = set_up<D, BWK, BWV>(ready)) return rc;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)cluster, (unsigned)Hkv, (unsigned)B);
  cfg.blockDim = dim3(C::kThreads);
  cfg.dynamicSmemBytes = C::kDynamic;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, decode_fused_kernel<D, BWK, BWV>, p);
  note_launches(1);
  return check_cuda(e, "wtq_decode fused launch");
}

template <int D> int set_up_widths(const DecodeParams &p, const Setup *&out) {
  if (p.k.bw == 4 && p.v.bw == 4) return set_up<D, 4, 4>(out);
  if (p.k.bw == 4 && p.v.bw == 6) return set_up<D, 4, 6>(out);
  if (p.k.bw == 6 && p.v.bw == 6) return set_up<D, 6, 6>(out);
  return set_up<D, 8, 8>(out);
}
template <int D> int launch_widths(const Params &p, int B, int Hkv, int cluster, cudaStream_t stream) {
  if (p.k.bw == 4 && p.v.bw == 4) return launch<D, 4, 4>(p, B, Hkv, cluster, stream);
  if (p.k.bw == 4 && p.v.bw == 6) return launch<D, 4, 6>(p, B, Hkv, cluster, stream);
  if (p.k.bw == 6 && p.v.bw == 6) return launch<D, 6, 6>(p, B, Hkv, cluster, stream);
  return launch<D, 8, 8>(p, B, Hkv, cluster, stream);
}

}  // namespace fused

// Blocks per group of the one-launch path; 0: the split-K path serves the call
// better.  Lengths are taken at the page table's full width.
//
// The cluster is the largest of 1, 2, 4, 8 with all groups resident at once and whose warps
// have about half a window each or more: at 1024 tokens
// and 2 groups 14.1 / 12.3 / 11.0 / 10.9 us with 1 / 2 / 4 / 8 blocks, at 200
// tokens and 8 groups 10.5 / 11.0 / 10.6 / 12.1; a second round of blocks costs
// more than it brings (32 groups of 8192 tokens: 22.4 us with 4, 49 with 8), and
// 16 was never better than 8.
//
// At head_dim 128 the table's width says how long a sequence may be, not how long the others
// are, and the two paths depend on that differently: one launch lasts as long as its longest
// group, `one` ns a token over the cluster's blocks; the split-K path deals chunks of all
// groups to the whole chip.  The line is drawn at the mix that favours split-K most, one
// sequence of the full width among short ones, for which its chunks still cost `split` ns a
// token x groups / multiprocessors: one launch where it saves more in fixed costs (`gap` us)
// than it then loses.  Measured (page pools in turn, larger than L2), one launch / split-K, us:
//   4/4 bits, 128 groups, one sequence of 2048 19.0 / 22.0, of 4096 28.4 / 27.1 (all of 4096
//   31.8 / 38.5), of 8192 47.5 / 37.1 (all 50.4 / 54.1); 64 groups 4096 19.8 / 21.8, 8192 29.6 / 27.2;
//   32 groups 8192 21.9 / 23.9, 16384 32.2 / 29.1; 144 groups 131072 575 / 66;
//   8/8 bits, 128 groups 2048 27.4 / 30.3, 4096 46.9 / 39.6; 32 groups 4096 20.8 / 23.3, 8192 31.3 / 29.7;
//   6/6 bits, 128 groups 1024 17.6 / 23.0, 2048 26.1 / 24.9; 64 groups 2048 18.1 / 22.7, 4096 27.2 / 25.2;
//   4/6 bits, 128 groups 2048 22.7 / 25.7, 4096 35.9 / 32.2; 64 groups 4096 23.8 / 25.4, 8192 36.7 / 31.8.
// One sequence alone has no others: its equal groups cost split-K 4.9 ns a token x groups /
// multiprocessors (times what a token of these widths costs to decode): 8 groups of 16384 21.4 /
// 24.0, of 32768 28.0 / 27.6, of 131072 89 / 55.
// With more groups than multiprocessors one launch would repeat its set-up in every round (320
// groups of 1000 tokens: 47.7 against 41.5).
int fused_cluster(const DecodeParams &p) {
  const int64_t groups = (int64_t)p.B * p.Hkv, sms = device_sms();
  const int64_t tokens = (int64_t)p.max_pages * p.S, windows = (tokens + kIterTokens - 1) / kIterTokens;
  const fused::Setup *ready = nullptr;
  if (p.D == 64 ? fused::set_up_widths<64>(p, ready) : fused::set_up_widths<128>(p, ready)) return 0;
  int c = 1;
  for (int i = 1; i < 4 && groups <= ready->clusters[i] && windows >= 4 << i; ++i) c = 1 << i;
  if (p.D == 64) return c;                  // (the alternative is the CUDA-core path)
  if (groups > sms) return 0;
  const double share = (double)groups / (double)sms;
  if (p.B == 1) {
    const double width = (p.k.bw + p.v.bw) / 8.0 * (p.k.bw + p.v.bw > 8 ? 1.25 : 1.0);
    return width * (double)tokens * (4.6 / c - 4.9 * share) <= 7500.0 ? c : 0;
  }
  struct Costs {
    double one, split, gap;
  };
  const Costs w = p.v.bw == 4 ? Costs{4.65, 2.8, 6.3} : p.k.bw == 4 ? Costs{6.4, 3.35, 8.0}
                  : p.k.bw == 6 ? Costs{7.9, 4.05, 7.0} : Costs{9.2, 5.4, 9.5};
  const double one = w.one / c * (c >= 4 ? 1.18 : 1.0);       // (short shares of a block: 32-token windows)
  return (double)tokens * (one - w.split * share) <= 1000.0 * w.gap ? c : 0;
}

bool fused_eligible(const DecodeParams &p) {
  auto aligned = [](const void *ptr) { return ((uintptr_t)ptr & 15) == 0; };
  return (p.D == 128 || p.D == 64) && mma_warps_per_sm(p.k.bw, p.v.bw) > 0 && p.S >= 16 &&
         (p.S & (p.S - 1)) == 0 && p.n_rep <= 8 && p.B <= 65535 && p.Hkv <= 65535 &&
         aligned(p.k.pages) && aligned(p.v.pages) && aligned(p.k.norms) && aligned(p.v.norms) &&
         aligned(p.k.Pi) && p.k.page_stride % 16 == 0 && p.k.head_stride % 16 == 0 &&
         p.v.page_stride % 16 == 0 && p.v.head_stride % 16 == 0 && p.k.norm_page_stride % 8 == 0 &&
         p.k.norm_head_stride % 8 == 0 && p.v.norm_page_stride % 8 == 0 && p.v.norm_head_stride % 8 == 0 &&
         // head_dim 128 rounds operands to 16 bits: only calls whose split-K scan does so too
         // (mma_eligible), none that the fp32 kernels serve
         (p.D == 64 || (p.k.page_stride < (int64_t)1 << 31 && p.v.page_stride < (int64_t)1 << 31 &&
                        p.k.norm_page_stride < (int64_t)1 << 30 && p.v.norm_page_stride < (int64_t)1 << 30));
}

int launch_decode_fused(const DecodeParams &p, const void *q, int dtype, const int64_t q_strides[2],
                        float q_scale, void *out, const int64_t out_strides[2], int cluster,
                        cudaStream_t stream) {
  fused::Params f;
  f.k = p.k; f.v = p.v; f.q = q; f.dtype = dtype; f.qsb = q_strides[0]; f.qsh = q_strides[1];
  f.q_scale = q_scale; f.out = out; f.osb = out_strides[0]; f.osh = out_strides[1];
  f.page_table = p.page_table; f.table_stride = p.table_stride; f.seq_lens = p.seq_lens;
  f.n_rep = p.n_rep; f.S = p.S; f.P = p.P; f.max_pages = p.max_pages; f.status = p.status;
  profile_mark_begin(stream);
  const int rc = p.D == 64 ? fused::launch_widths<64>(f, p.B, p.Hkv, cluster, stream)
                           : fused::launch_widths<128>(f, p.B, p.Hkv, cluster, stream);
  profile_mark_end(stream);
  return rc;
}

}  // namespace wtq
