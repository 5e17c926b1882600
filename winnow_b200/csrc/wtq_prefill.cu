// Chunked prefill straight from the packed pages: causal attention of a chunk
// of Q query tokens per sequence over that sequence's packed history, every
// page read and decoded once for all the query rows that share it.  Replaces
// the reference's prefill fallback, which dequantizes the whole history of
// each sequence to the model dtype and calls SDPA
// (turboquant_kv/packed_backend.py:192-226).
//
// Work is cut into items (sequence b, kv head, block of 256 query rows, range
// of the history); the query rows of a kv head are (token i, head r) pairs in
// token-major order, so the causal length never decreases along them.  Per item
// the 256 rotated query rows go to shared memory as fp16 once, as two M = 128
// operands; the range is then walked in tiles of 64 tokens by three groups of
// warps that meet only at mbarriers:
//
//   decode    seven warps: tasks of 16 tokens of one side (K or V), from packed codes
//             loaded into registers a task ahead to fp16 centroid x norm
//             through the per-lane lookup tables (wtq_lut.cuh) and stores them in
//             the canonical no-swizzle operand layout, two tiles deep;
//   multiply  one thread issues tcgen05.mma: S = Q K^T (N 64, K-major operands) one
//             tile ahead of O += P V (A = P from tensor memory, B = V with the
//             coordinates contiguous, i.e. MN-major: the same bytes as a K tile
//             read with the two strides exchanged);
//   softmax   two warpgroups, one per M tile, a thread per query row: scores from
//             tensor memory, causal mask, online softmax in the exp2 domain, the
//             probabilities back to tensor memory as fp16 over the scores they came
//             from.  The reference maximum is raised, and O rescaled, only when a
//             row's scores exceed it by 2^8, so almost no tile touches O.
//
// Tensor memory: S of two M tiles x two buffers x 64 columns, O of two M tiles x 128.
// fp16 scores are exact enough while they are small; a warp whose tile holds a row
// maximum beyond 8 (log2 domain) recomputes that tile's scores in fp32 from the
// packed codes.  At the end of the range every row that sees it writes its state
// (reference maximum, sum, un-normalised accumulator in the value basis) in the
// layout of the decode scan; a merge kernel combines the ranges, rotates back and
// stores.  Every wait is bounded; one that runs out raises a flag that ends all the others,
// and the status word says so.
//
// Measured, 16 sequences x 64 query tokens over 8k histories (137 GFLOP), call and kernel: as
// mma.sync (a warp per 32 rows decoding and multiplying in turn, accumulators and scores
// filling the register file, two warps a scheduler) 604 and 518 us; in this form 399 and 295;
// with the multiplying warp's control flow uniform 36 us less.  Bound now by the products:
// about 100 cycles each, 24 a tile, while the softmax warps wait 2.2 K of a tile's 3.9 K cycles.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "wtq_decode.cuh"
#include "wtq_lut.cuh"

namespace wtq {
namespace pf {

constexpr int kSoftWarps = 8, kDecodeWarps = 7, kMmaWarp = kSoftWarps + kDecodeWarps;   // 16 warps of 128 registers
constexpr int kThreads = 32 * (kMmaWarp + 1);
constexpr int kRows = 256;                      // query rows per item: two M = 128 operands
constexpr int kTile = 64;                       // tokens per tile
constexpr uint32_t kBase = 1024;                // dynamic shared memory is assumed to start at or below this
// mbarriers (8 bytes each).  All that can be up to two tiles apart exist per buffer, so
// that no side is ever two completions ahead of a phase another side still waits for.
constexpr uint32_t kKFull = kBase, kVFull = kBase + 16, kKFree = kBase + 32, kVFree = kBase + 48;   // [buffer]
constexpr uint32_t kSFull = kBase + 64;             // [M tile][buffer]: scores are in tensor memory
constexpr uint32_t kPFull = kBase + 96;             // [M tile][buffer]: probabilities are in tensor memory
constexpr uint32_t kODone = kBase + 128;            // [M tile][buffer]: the products of a tile into O are complete
constexpr uint32_t kTmemSlot = kBase + 160;         // tensor-memory address written by tcgen05.alloc
constexpr uint32_t kAbort = kBase + 164;            // a wait ran out
constexpr uint32_t kLast = kBase + 168;             // everything issued is complete
constexpr uint32_t kItem = kBase + 176;             // the item being worked on (8 words)
constexpr uint32_t kWalk = kItem + 32;              // balanced schedule: where this block stands (10 words)
constexpr uint32_t kTileBytes = kTile * 256;        // a decoded tile: [64 tokens][128] fp16
constexpr uint32_t kVTile = 2048;                   // two buffers
constexpr uint32_t kPlan = kVTile + 2 * kTileBytes; // balanced schedule: tiles of every (sequence, row block)
constexpr int kMaxPairs = 4096;                     // (sequence, row block) pairs the plan has room for
constexpr int kBalancedSlots = 3;                   // a group is cut by at most two block boundaries
static_assert(kWalk + 64 <= kVTile && kPlan + 4 * kMaxPairs <= mma::kLutAddr, "low region");
constexpr float kPreciseAbove = 8.f;            // |score| (log2 domain) beyond which fp16 is not trusted
constexpr float kSlack = 8.f;                   // how far scores may exceed the reference before it is raised
// tensor memory columns
constexpr uint32_t kColS = 0;                   // + 128 * (M tile) + 64 * buffer; P over the first 32 of each
constexpr uint32_t kColO = 256;                 // + 128 * (M tile)
constexpr uint32_t kCols = 512;
// instruction descriptors: dense, fp32 accumulator, fp16 A and B, M = 128
constexpr uint32_t kIdescQK = (1u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kIdescPV = (1u << 4) | (1u << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);   // B MN-major

struct Params {
  DecodeSideDev k, v;
  const float *q_rot;        // (B * Q, Hq, 128) fp32, times scale * log2(e)
  const int32_t *page_table;
  int64_t table_stride;
  const int32_t *seq_lens;   // (B)
  int32_t *row_lens;         // (B * Q) causal lengths, written here for the merge
  int B, Hq, Hkv, n_rep, Q, S, P, max_pages, max_tokens;
  int num_splits, chunk_tokens, row_blocks;
  int balanced;              // 1: tiles dealt evenly to the blocks (chunk_tokens unused), 0: equal chunks
  float *part_acc, *part_m, *part_l;
  int32_t *status, *work_counter;
  const uint32_t *lut;
};

template <int BWK, int BWV> struct Map {
  static constexpr uint32_t kLutBytes =
      (uint32_t)(mma::lut_entries(BWK) > mma::lut_entries(BWV) ? mma::lut_entries(BWK)
                                                                : mma::lut_entries(BWV)) * 256u;
  static constexpr uint32_t kQTile = mma::kLutAddr + kLutBytes;        // [256][128] fp16
  static constexpr uint32_t kKTile = kQTile + kRows * 256;             // two buffers
  static constexpr uint32_t kDynamic = kKTile + 2 * kTileBytes;
  static_assert(kDynamic <= 227u * 1024u, "shared memory budget");
};

__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
// ---- operand layout: core matrices of 8 rows x 16 bytes (128 bytes each); the 16 pieces
// of a group of eight rows follow one another (2 KB per group) --------------------------
__device__ __forceinline__ uint32_t operand_at(uint32_t tile, int row, int piece) {
  return tile + (uint32_t)(row >> 3) * 2048u + (uint32_t)piece * 128u + (uint32_t)(row & 7) * 16u;
}
__device__ __forceinline__ uint64_t descriptor(uint32_t start, uint32_t leading, uint32_t stride) {
  return (uint64_t)((start >> 4) & 0x3fffu) | ((uint64_t)(leading >> 4) << 16) |
         ((uint64_t)(stride >> 4) << 32) | ((uint64_t)1 << 46);          // version, no swizzle
}
// K-major operand (rows = M or N, contraction along a row): step ks takes pieces 2 ks, 2 ks + 1;
// leading offset: next piece, stride offset: next eight rows
__device__ __forceinline__ uint64_t desc_k_major(uint32_t tile, int ks) {
  return descriptor(tile + (uint32_t)ks * 256u, 128u, 2048u);
}
// MN-major operand (rows = contraction): step ks takes rows 16 ks .. 16 ks + 15; leading
// offset: next eight rows, stride offset: next piece
__device__ __forceinline__ uint64_t desc_mn_major(uint32_t tile, int ks) {
  return descriptor(tile + (uint32_t)ks * 4096u, 2048u, 128u);
}
__device__ __forceinline__ void umma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void umma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
      ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
// 1 in one lane of a converged warp, the same every time
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t r;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(r));
  return r;
}
constexpr int kWaitTries = 1 << 20;
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// Bounded wait for completion number `use` (0, 1, ..) of an mbarrier; false if it, or any
// other wait of the block, ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, int use) {
  for (int spin = 0; spin < kWaitTries; ++spin) {
    if (mbar_try(bar, (uint32_t)(use & 1))) return true;
    if ((spin & 255) == 255 && lds32(kAbort) != 0u) return false;
  }
  sts32(kAbort, 0x80000000u | (threadIdx.x >> 5) << 24 | ((uint32_t)use & 0xfffu) << 12 | (bar - kBase));   // who gave up on what
  return false;
}
template <int AT, int N> __device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&r)[N]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[AT + 0]), "=r"(r[AT + 1]), "=r"(r[AT + 2]), "=r"(r[AT + 3]),
        "=r"(r[AT + 4]), "=r"(r[AT + 5]), "=r"(r[AT + 6]), "=r"(r[AT + 7]),
        "=r"(r[AT + 8]), "=r"(r[AT + 9]), "=r"(r[AT + 10]), "=r"(r[AT + 11]),
        "=r"(r[AT + 12]), "=r"(r[AT + 13]), "=r"(r[AT + 14]), "=r"(r[AT + 15]),
        "=r"(r[AT + 16]), "=r"(r[AT + 17]), "=r"(r[AT + 18]), "=r"(r[AT + 19]),
        "=r"(r[AT + 20]), "=r"(r[AT + 21]), "=r"(r[AT + 22]), "=r"(r[AT + 23]),
        "=r"(r[AT + 24]), "=r"(r[AT + 25]), "=r"(r[AT + 26]), "=r"(r[AT + 27]),
        "=r"(r[AT + 28]), "=r"(r[AT + 29]), "=r"(r[AT + 30]), "=r"(r[AT + 31])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_store32(uint32_t addr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};\n"
      ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]),
        "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]),
        "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_store16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n"
      ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_wait_load() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_store() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }

// Eight consecutive centroid values (fp16) of a lane's share of a packed row:
// codes 8 J .. 8 J + 7 of the 32 the words hold.
template <int BW, int J, int NW>
__device__ __forceinline__ void decode_piece(const uint32_t (&w)[NW], uint32_t sel, uint32_t (&f)[4]) {
  if constexpr (BW == 4) {
    f[0] = lut_byte<0>(w[J], sel); f[1] = lut_byte<1>(w[J], sel);
    f[2] = lut_byte<2>(w[J], sel); f[3] = lut_byte<3>(w[J], sel);
  } else {
    f[0] = join(lut_code<BW, 8 * J>(w, sel), lut_code<BW, 8 * J + 1>(w, sel));
    f[1] = join(lut_code<BW, 8 * J + 2>(w, sel), lut_code<BW, 8 * J + 3>(w, sel));
    f[2] = join(lut_code<BW, 8 * J + 4>(w, sel), lut_code<BW, 8 * J + 5>(w, sel));
    f[3] = join(lut_code<BW, 8 * J + 6>(w, sel), lut_code<BW, 8 * J + 7>(w, sel));
  }
}
// The lane's quarter of a packed row in global memory.
template <int BW, int NW> __device__ __forceinline__ void load_quarter(const uint8_t *at, uint32_t (&w)[NW]) {
  if constexpr (BW == 6) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const uint2 v = __ldg(reinterpret_cast<const uint2 *>(at) + i);
      w[2 * i] = v.x; w[2 * i + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < BW / 4; ++i) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(at) + i);
      w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
  }
}

__device__ __forceinline__ uint32_t times(uint32_t c, __half2 n) {
  const __half2 y = __hmul2(*reinterpret_cast<const __half2 *>(&c), n);
  return *reinterpret_cast<const uint32_t *>(&y);
}
// Tokens 16 u .. 16 u + 15 of a tile: the lane (g, t) stores rows g and g + 8, coordinates
// 32 t .. 32 t + 31, as centroid x row norm rounded to fp16 (the scores and value sums then
// need no per-token scaling).
template <int BW, int NW>
__device__ __forceinline__ void decode_task(uint32_t tile, int u, int g, int t, uint32_t sel,
                                            const uint32_t (&w)[2][NW], const __half (&nrm)[2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = 16 * u + g + 8 * h;
    const __half2 n = __half2half2(nrm[h]);
    uint32_t f[4];
    decode_piece<BW, 0>(w[h], sel, f);
    sts128(operand_at(tile, row, 4 * t + 0), times(f[0], n), times(f[1], n), times(f[2], n), times(f[3], n));
    decode_piece<BW, 1>(w[h], sel, f);
    sts128(operand_at(tile, row, 4 * t + 1), times(f[0], n), times(f[1], n), times(f[2], n), times(f[3], n));
    decode_piece<BW, 2>(w[h], sel, f);
    sts128(operand_at(tile, row, 4 * t + 2), times(f[0], n), times(f[1], n), times(f[2], n), times(f[3], n));
    decode_piece<BW, 3>(w[h], sel, f);
    sts128(operand_at(tile, row, 4 * t + 3), times(f[0], n), times(f[1], n), times(f[2], n), times(f[3], n));
  }
}

// fp32 scores of this thread's query row against the 64 tokens of a tile, written over the
// tile's scores in tensor memory (`s_addr`, lane base included): the packed codes of its kv head are read
// from the pages (the same address for the whole warp) and the row of `q` along with them.
// Out of line: it runs only for tiles whose fp16 scores came out large.
template <int BW>
__device__ __noinline__ void precise_tile(const uint8_t *pages, int64_t page_stride, const __half *all_norms,
                                          int64_t norm_page_stride, const float *centroids, const int32_t *table,
                                          int P, int S, int tok0, int end, const float *q, uint32_t s_addr) {
  const int shift = 31 - __clz(S);
#pragma unroll 1
  for (int blk = 0; blk < kTile / 16; ++blk) {                // sixteen tokens of one page
    const int tok = tok0 + 16 * blk;
    const int page = tok < end ? table[tok >> shift] : -1;
    float acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    if (page >= 0 && page < P) {
      const int pos = tok & (S - 1);
      const uint8_t *row = pages + (int64_t)page * page_stride + (int64_t)pos * (16 * BW);
#pragma unroll 1
      for (int d = 0; d < 32; ++d) {                           // four coordinates: BW / 2 bytes of each row
        const float4 x = q ? __ldg(reinterpret_cast<const float4 *>(q) + d) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          uint32_t w = 0;
#pragma unroll
          for (int b = 0; b < BW / 2; ++b) w |= (uint32_t)__ldg(row + i * (16 * BW) + d * (BW / 2) + b) << (8 * b);
          constexpr uint32_t kMask = (1u << BW) - 1u;
          acc[i] = fmaf(x.x, __ldg(centroids + (w & kMask)), acc[i]);
          acc[i] = fmaf(x.y, __ldg(centroids + ((w >> BW) & kMask)), acc[i]);
          acc[i] = fmaf(x.z, __ldg(centroids + ((w >> (2 * BW)) & kMask)), acc[i]);
          acc[i] = fmaf(x.w, __ldg(centroids + ((w >> (3 * BW)) & kMask)), acc[i]);
        }
      }
      const __half *norms = all_norms + (int64_t)page * norm_page_stride + pos;
#pragma unroll
      for (int i = 0; i < 16; ++i) acc[i] *= __half2float(norms[i]);
    }
    uint32_t v[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __float_as_uint(acc[i]);
    __syncwarp();
    tmem_store16(s_addr + 16 * blk, v);
  }
  tmem_wait_store();
}

// Scores of the tokens from `seen` on become -inf (`masked`: some row of the warp has
// such); returns the row's maximum.
__device__ __forceinline__ float mask_and_maximum(uint32_t (&s)[64], bool masked, int seen) {
  if (masked) {
#pragma unroll
    for (int i = 0; i < 64; ++i) s[i] = i >= seen ? 0xff800000u : s[i];
  }
  float a = -INFINITY, c = -INFINITY;
#pragma unroll
  for (int i = 0; i < 64; i += 4) {
    a = max3(a, __uint_as_float(s[i]), __uint_as_float(s[i + 1]));
    c = max3(c, __uint_as_float(s[i + 2]), __uint_as_float(s[i + 3]));
  }
  return fmaxf(a, c);
}

template <int BWK, int BWV>
__global__ void __launch_bounds__(kThreads, 1) prefill_kernel(Params p) {
  using M = Map<BWK, BWV>;
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((uint32_t)__cvta_generic_to_shared(dyn_smem) > kBase) {   // layout assumption broken
    if (p.status && tid == 0) atomicOr(p.status, WTQ_STATUS_LAYOUT);
    return;
  }
  constexpr uint32_t kFull = 0xffffffffu;
  // causal length of every query row, for the merge
  for (int i = blockIdx.x * kThreads + tid; i < p.B * p.Q; i += gridDim.x * kThreads) {
    int L = p.seq_lens[i / p.Q];
    L = L < 0 ? 0 : (L > p.max_tokens ? p.max_tokens : L);
    const int len = L - p.Q + 1 + i % p.Q;
    p.row_lens[i] = len < 0 ? 0 : len;
  }
  // lookup tables (built by the rotation launch), tensor memory, barriers
  for (int i = tid; i < (int)(M::kLutBytes / 16); i += kThreads) {
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p.lut) + i);
    sts128(mma::kLutAddr + 16u * i, v.x, v.y, v.z, v.w);
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(kTmemSlot),
                 "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      mbar_init(kKFull + 8u * i, 4);                        // the four 16-token groups of a tile
      mbar_init(kVFull + 8u * i, 4);
      mbar_init(kKFree + 8u * i, 1);
      mbar_init(kVFree + 8u * i, 1);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      mbar_init(kSFull + 8u * i, 1);
      mbar_init(kODone + 8u * i, 1);
      mbar_init(kPFull + 8u * i, 4);                        // the four warps of an M tile
    }
    mbar_init(kLast, 1);
    sts32(kAbort, 0u);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  const int R = p.Q * p.n_rep;                              // query rows per (sequence, kv head)
  const int items = p.B * p.Hkv * p.row_blocks * p.num_splits;
  const int page_shift = 31 - __clz(p.S);
  // ---- balanced schedule ---------------------------------------------------------------
  // The 64-token tiles of all groups, laid end to end (sequence, row block, kv head), are
  // cut into one equal run per block, so every multiprocessor gets the same number of
  // tiles whatever the number of groups.  A run is at least half the longest group, hence a
  // group is cut at most twice and its pieces take chunk slots 0..2; the slot of a piece is
  // its block's distance from the block that holds the group's first tile.
  if (p.balanced) {
    const int pairs = p.B * p.row_blocks;
    for (int i = tid; i < pairs; i += kThreads) {
      const int b = i / p.row_blocks, rb = i - b * p.row_blocks;
      int L = p.seq_lens[b];
      L = L < 0 ? 0 : (L > p.max_tokens ? p.max_tokens : L);
      const int last = min(R, (rb + 1) * kRows) - 1;          // last row of the block
      const int len = L - p.Q + 1 + last / p.n_rep;
      sts32(kPlan + 4u * i, len > 0 ? (uint32_t)((len + kTile - 1) / kTile) : 0u);
    }
    __syncthreads();
    if (warp == 0) {
      long long total = 0;
      int longest = 0;
      for (int i = lane; i < pairs; i += 32) {
        const int n = (int)lds32(kPlan + 4u * i);
        total += n;
        longest = max(longest, n);
      }
#pragma unroll
      for (int d = 16; d; d >>= 1) {
        total += __shfl_xor_sync(kFull, total, d);
        longest = max(longest, __shfl_xor_sync(kFull, longest, d));
      }
      if (lane == 0) {
        total *= p.Hkv;
        long long share = (total + gridDim.x - 1) / gridDim.x;
        share = max(share, (long long)((longest + 1) / 2));
        share = max(share, 1LL);
        const long long lo = min(total, share * blockIdx.x), hi = min(total, lo + share);
        sts32(kWalk + 0, 0u);                                             // pair the walk stands in
        sts32(kWalk + 4, 0u); sts32(kWalk + 8, 0u);                       // tiles before that pair
        sts32(kWalk + 12, (uint32_t)lo); sts32(kWalk + 16, (uint32_t)(lo >> 32));   // next tile
        sts32(kWalk + 20, (uint32_t)hi); sts32(kWalk + 24, (uint32_t)(hi >> 32));   // end of the run
        sts32(kWalk + 28, (uint32_t)share); sts32(kWalk + 32, (uint32_t)(share >> 32));
      }
    }
  }
  auto walk64 = [&](uint32_t at) -> long long {
    return (long long)(((unsigned long long)lds32(at + 4) << 32) | lds32(at));
  };
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = lds32(kTmemSlot);
  // Tiles handled so far, over all items: buffers alternate and barrier phases count on.
  int tiles_all = 0, tiles_m[2] = {0, 0};

  for (;;) {
    fence_before();
    __syncthreads();                                        // everyone is done with the previous item
    fence_after();
    if (lds32(kAbort) != 0u) break;
    if (tid == 0) {
      if (!p.balanced) {
        sts32(kItem, (uint32_t)atomicAdd(p.work_counter, 1));
      } else {
        int i = (int)lds32(kWalk);
        long long pre = walk64(kWalk + 4), x = walk64(kWalk + 12);
        const long long hi = walk64(kWalk + 20), share = walk64(kWalk + 28);
        if (x >= hi) {
          sts32(kItem, 0xffffffffu);
        } else {
          int n = (int)lds32(kPlan + 4u * i);
          // ends before the last pair: x < hi <= all tiles (the bound on i only guards the plan)
          while (x >= pre + (long long)p.Hkv * n && i + 1 < p.B * p.row_blocks) {
            pre += (long long)p.Hkv * n;
            n = (int)lds32(kPlan + 4u * ++i);
          }
          const long long rel = x - pre;
          const int kvh = n > 0 ? (int)(rel / n) : p.Hkv, off = (int)(rel - (long long)kvh * n);
          const int take = (int)min(hi - x, (long long)(n - off));
          const long long slot = (long long)blockIdx.x - (pre + (long long)kvh * n) / share;
          if (slot < 0 || slot >= p.num_splits || kvh >= p.Hkv || take < 1) {   // cannot happen; never
            x = hi - take;                                                      // write outside the states
            if (p.status) atomicOr(p.status, WTQ_STATUS_LAYOUT);
            sts32(kItem, 0xffffffffu);
          } else {
            sts32(kItem, (uint32_t)i);
            sts32(kItem + 4, (uint32_t)kvh);
            sts32(kItem + 8, (uint32_t)off);
            sts32(kItem + 12, (uint32_t)(off + take));
            sts32(kItem + 16, (uint32_t)slot);
          }
          x += take;
          sts32(kWalk, (uint32_t)i);
          sts32(kWalk + 4, (uint32_t)pre); sts32(kWalk + 8, (uint32_t)(pre >> 32));
          sts32(kWalk + 12, (uint32_t)x); sts32(kWalk + 16, (uint32_t)(x >> 32));
        }
      }
    }
    __syncthreads();
    const int item = (int)lds32(kItem);
    int chunk, rb, kvh, b, start, cap;                       // cap: end of the item's token range
    if (!p.balanced) {
      if (item >= items) break;
      // chunks vary fastest, so blocks working at the same time share the query rows in L2
      chunk = item % p.num_splits;
      rb = (item / p.num_splits) % p.row_blocks;
      kvh = (item / (p.num_splits * p.row_blocks)) % p.Hkv;
      b = item / (p.num_splits * p.row_blocks * p.Hkv);
      start = chunk * p.chunk_tokens;
      cap = start + p.chunk_tokens;
    } else {
      if (item < 0) break;
      b = item / p.row_blocks;
      rb = item - b * p.row_blocks;
      kvh = (int)lds32(kItem + 4);
      start = (int)lds32(kItem + 8) * kTile;
      cap = (int)lds32(kItem + 12) * kTile;
      chunk = (int)lds32(kItem + 16);
    }
    int L = p.seq_lens[b];
    L = L < 0 ? 0 : (L > p.max_tokens ? p.max_tokens : L);
    const int row_lo = rb * kRows;
    const int row_hi = min(R, row_lo + kRows);             // rows [row_lo, row_hi) exist
    auto length_of = [&](int row) {                         // causal length of a row of this group
      const int len = L - p.Q + 1 + row / p.n_rep;
      return len < 0 ? 0 : len;
    };
    if (row_lo >= R) continue;
    // tiles each of the two M tiles sees (rows are in causal order: its last row sees most)
    int ntiles[2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int last = min(row_hi, row_lo + 128 * (m + 1)) - 1;
      const int limit = last >= row_lo + 128 * m ? min(length_of(last), cap) : 0;
      ntiles[m] = limit > start ? (limit - start + kTile - 1) / kTile : 0;
    }
    const int end = min(cap, length_of(row_hi - 1));
    const int nt = max(ntiles[0], ntiles[1]);
    if (nt == 0) continue;                                  // no row of the block sees this range
    const int32_t *table = p.page_table + (int64_t)b * p.table_stride;

    // ---- query rows -> fp16 operand (the softmax warps; the decode warps start at once) ----
    if (warp < kSoftWarps) {
      const int most = ntiles[1] > 0 ? 4096 : 2048;          // (row, piece) units
#pragma unroll 4
      for (int u = tid; u < most; u += 32 * kSoftWarps) {
        const int piece = (u >> 3) & 15, lr = (u & 7) + 8 * (u >> 7), row = row_lo + lr;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
        if (row < row_hi) {
          const int i = row / p.n_rep, r = row - i * p.n_rep;
          const float4 *src = reinterpret_cast<const float4 *>(
              p.q_rot + (((int64_t)b * p.Q + i) * p.Hq + kvh * p.n_rep + r) * 128 + 8 * piece);
          x = __ldg(src);
          y = __ldg(src + 1);
        }
        sts128(operand_at(M::kQTile, lr, piece), pack_half2(x.x, x.y), pack_half2(x.z, x.w), pack_half2(y.x, y.y),
               pack_half2(y.z, y.w));
      }
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp < kSoftWarps || warp == kMmaWarp)
      asm volatile("bar.sync 1, %0;\n" ::"r"(32 * (kSoftWarps + 1)) : "memory");

    if (warp < kSoftWarps) {
      // ================= softmax: M tile m, one query row per thread ====================
      const int m = warp >> 2;
      const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
      const int row = row_lo + 128 * m + 32 * (warp & 3) + lane;
      const int limit = row < row_hi ? min(length_of(row), cap) : 0;   // first token the row does NOT see
      int64_t qrow = -1;
      if (row < row_hi) {
        const int i = row / p.n_rep, r = row - i * p.n_rep;
        qrow = ((int64_t)b * p.Q + i) * p.Hq + kvh * p.n_rep + r;
      }
      const int all_see = __reduce_min_sync(kFull, limit);             // every row of the warp sees the tokens below
      const int n = ntiles[m];
      float ref = -INFINITY, sum = 0.f;
      bool ok = true;
      for (int j = 0; j < n && ok; ++j) {
        const int T = tiles_m[m] + j, buf = T & 1, tok0 = start + j * kTile;
        const uint32_t s_addr = tmem + lanes + kColS + 128u * m + 64u * buf;
        ok = mbar_wait(kSFull + 16u * m + 8u * buf, T >> 1);
        if (!__all_sync(kFull, ok)) { ok = false; break; }
        fence_after();
        uint32_t s[64];
        tmem_load32<0>(s_addr, s);
        tmem_load32<32>(s_addr + 32, s);
        tmem_wait_load();
        float mx = mask_and_maximum(s, tok0 + kTile > all_see, limit - tok0);
        // The fp16 error of a score grows with its size, and only scores near their row's
        // maximum carry weight: a tile is re-scored in fp32 when a row maximum lies beyond
        // +-8 (or is not a number).
        if (__any_sync(kFull, !(fabsf(mx) <= kPreciseAbove) && mx != -INFINITY)) {
          precise_tile<BWK>(p.k.pages + (int64_t)kvh * p.k.head_stride, p.k.page_stride,
                            p.k.norms + (int64_t)kvh * p.k.norm_head_stride, p.k.norm_page_stride, p.k.centroids, table,
                            p.P, p.S, tok0, end, qrow < 0 ? nullptr : p.q_rot + qrow * 128, s_addr);
          tmem_load32<0>(s_addr, s);
          tmem_load32<32>(s_addr + 32, s);
          tmem_wait_load();
          mx = mask_and_maximum(s, tok0 + kTile > all_see, limit - tok0);
        }
        if (__any_sync(kFull, mx > ref + kSlack || (ref == -INFINITY && mx != -INFINITY))) {
          const float now = mx > ref + kSlack || ref == -INFINITY ? mx : ref;
          if (j > 0) {                                                  // rescale what is accumulated
            const float scale = ref == now ? 1.f : ref == -INFINITY ? 0.f : ex2(ref - now);
            sum *= scale;
            ok = mbar_wait(kODone + 16u * m + 8u * (buf ^ 1), (T - 1) >> 1);
            if (!__all_sync(kFull, ok)) { ok = false; break; }
            fence_after();
#pragma unroll 1
            for (int c0 = 0; c0 < 128; c0 += 32) {
              uint32_t o[32];
              const uint32_t o_addr = tmem + lanes + kColO + 128u * m + c0;
              tmem_load32<0>(o_addr, o);
              tmem_wait_load();
#pragma unroll
              for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * scale);
              tmem_store32(o_addr, o);
            }
            tmem_wait_store();
          }
          ref = now;
        }
        const float base = ref == -INFINITY ? 0.f : ref;
        uint32_t pr[32];
        float sa = 0.f, sb = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          pr[i] = pack_half2(ex2(__uint_as_float(s[2 * i]) - base), ex2(__uint_as_float(s[2 * i + 1]) - base));
          // The sum takes the probabilities as the product has them: where a few keys carry the
          // row, their rounding then cancels in the quotient.
          const float2 pq = __half22float2(*reinterpret_cast<const __half2 *>(&pr[i]));
          sa += pq.x;
          sb += pq.y;
        }
        sum += sa + sb;
        tmem_store32(s_addr, pr);                                       // over the scores just read
        tmem_wait_store();
        fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(kPFull + 16u * m + 8u * buf);
      }
      // ---- the rows' states -----------------------------------------------------------
      if (ok && n > 0) {
        const int last = tiles_m[m] + n - 1;
        ok = mbar_wait(kODone + 16u * m + 8u * (last & 1), last >> 1);
        if (__all_sync(kFull, ok)) {
          fence_after();
          const bool keep = qrow >= 0 && limit > start;                 // the row exists and sees part of the range
          const int64_t state = qrow * p.num_splits + chunk;
#pragma unroll 1
          for (int c0 = 0; c0 < 128; c0 += 32) {
            uint32_t o[32];
            tmem_load32<0>(tmem + lanes + kColO + 128u * m + c0, o);
            tmem_wait_load();
            if (keep) {
              uint4 *dst = reinterpret_cast<uint4 *>(p.part_acc + state * 128 + c0);
#pragma unroll
              for (int i = 0; i < 8; ++i) dst[i] = make_uint4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
            }
          }
          if (keep) {
            p.part_m[state] = ref;
            p.part_l[state] = sum;
          }
        }
      }
    } else if (warp < kMmaWarp) {
      // ================= decode ==========================================================
      // Tasks of 16 tokens of one side, eight per tile (four of K, four of V), dealt round-robin;
      // the codes of a warp's next task are on their way while it decodes this one.
      constexpr int kMost = BWK > BWV ? BWK : BWV;
      const int g = lane & 7, t = lane >> 3;
      const uint32_t sel = mma::kLutAddr | (uint32_t)(lane << 2);
      const int tasks = 8 * nt;
      auto page_of = [&](int q) {                                       // -2: past the end of the range
        const int tok = start + (q >> 3) * kTile + 16 * (q & 3);
        return q < tasks && tok < end ? table[tok >> page_shift] : -2;
      };
      auto load = [&](int q, int page, uint32_t (&w)[2][kMost], __half (&nrm)[2]) {
        const bool is_v = (q & 4) != 0;
        const DecodeSideDev &sd = is_v ? p.v : p.k;
        const int tok = start + (q >> 3) * kTile + 16 * (q & 3);
        if ((uint32_t)page < (uint32_t)p.P) {
          const int pos = tok & (p.S - 1);
          const uint8_t *rows = sd.pages + (int64_t)page * sd.page_stride + (int64_t)kvh * sd.head_stride;
          const __half *norms = sd.norms + (int64_t)page * sd.norm_page_stride + (int64_t)kvh * sd.norm_head_stride + pos;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int r = g + 8 * h;
            if (BWK == BWV || !is_v) {
              load_quarter<BWK>(rows + (int64_t)(pos + r) * (16 * BWK) + t * (4 * BWK), w[h]);
            } else {
              load_quarter<BWV>(rows + (int64_t)(pos + r) * (16 * BWV) + t * (4 * BWV), w[h]);
            }
            nrm[h] = norms[r];
            if (tok + r >= end) nrm[h] = __ushort_as_half(0);
          }
        } else {
          if (page != -2 && p.status && lane == 0) atomicOr(p.status, WTQ_STATUS_BAD_PAGE);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int k = 0; k < kMost; ++k) w[h][k] = 0u;
            nrm[h] = __ushort_as_half(0);
          }
        }
      };
      uint32_t w[2][kMost], next[2][kMost];
      __half nrm[2], nrm_next[2];
      int q = warp - kSoftWarps;
      if (q < tasks) load(q, page_of(q), w, nrm);
      int page = page_of(q + kDecodeWarps);
      for (; q < tasks; q += kDecodeWarps) {
        if (q + kDecodeWarps < tasks) load(q + kDecodeWarps, page, next, nrm_next);
        page = page_of(q + 2 * kDecodeWarps);
        const bool is_v = (q & 4) != 0;
        const int T = tiles_all + (q >> 3), buf = T & 1, u = q & 3;
        if (T >= 2) {                                                   // the tile's last reader is done
          const bool ok = mbar_wait((is_v ? kVFree : kKFree) + 8u * buf, (T >> 1) - 1);
          if (!__all_sync(kFull, ok)) break;
        }
        if (!is_v) decode_task<BWK>(M::kKTile + (uint32_t)buf * kTileBytes, u, g, t, sel, w, nrm);
        else decode_task<BWV>(kVTile + (uint32_t)buf * kTileBytes, u, g, t, sel | 0x80u, w, nrm);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive((is_v ? kVFull : kKFull) + 8u * buf);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int k = 0; k < kMost; ++k) w[h][k] = next[h][k];
          nrm[h] = nrm_next[h];
        }
      }
    } else {
      // ================= multiply: the whole warp waits, one lane issues ======================
      // (Control flow stays uniform and the two M tiles are spelled out: with one lane in the
      // loop and the tile counts indexed, the code between the products took longer than
      // the products and was what everybody waited for.)
      const uint32_t issuer = elect_one();
      const uint64_t q_desc = desc_k_major(M::kQTile, 0);
      auto scores = [&](int j, auto m_) -> bool {                       // S of tile j, M tile m
        constexpr int m = decltype(m_)::value;
        const int T = tiles_all + j, buf = T & 1, Tm = tiles_m[m] + j, sb = Tm & 1;
        // the buffer's last probabilities have been consumed (those of an earlier item were
        // before its states were written)
        if (j >= 2 && !mbar_wait(kODone + 16u * m + 8u * sb, (Tm - 2) >> 1)) return false;
        fence_after();
        if (issuer) {
          const uint32_t d = tmem + kColS + 128u * m + 64u * sb;
          const uint64_t qa = q_desc + (uint64_t)m * (32768u >> 4);
          const uint64_t kb = desc_k_major(M::kKTile + (uint32_t)buf * kTileBytes, 0);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_ss(d, qa + 16u * ks, kb + 16u * ks, kIdescQK, ks > 0);
          umma_commit(kSFull + 16u * m + 8u * sb);
        }
        return true;
      };
      auto values = [&](int i, auto m_) -> bool {                       // O += P V of tile i, M tile m
        constexpr int m = decltype(m_)::value;
        const int T = tiles_all + i, buf = T & 1, Tm = tiles_m[m] + i, sb = Tm & 1;
        if (!mbar_wait(kPFull + 16u * m + 8u * sb, Tm >> 1)) return false;
        fence_after();
        if (issuer) {
          const uint32_t p_addr = tmem + kColS + 128u * m + 64u * sb, d = tmem + kColO + 128u * m;
          const uint64_t vb = desc_mn_major(kVTile + (uint32_t)buf * kTileBytes, 0);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            umma_ts(d, p_addr + 8u * ks, vb + 256u * ks, kIdescPV, i > 0 || ks > 0);
          umma_commit(kODone + 16u * m + 8u * sb);
        }
        return true;
      };
      constexpr std::integral_constant<int, 0> m0{};
      constexpr std::integral_constant<int, 1> m1{};
      for (int j = 0; j <= nt; ++j) {
        if (j < nt) {                                                   // scores of tile j
          const int T = tiles_all + j, buf = T & 1;
          bool ok = mbar_wait(kKFull + 8u * buf, T >> 1);
          if (ok && j < ntiles[0]) ok = scores(j, m0);
          if (ok && j < ntiles[1]) ok = scores(j, m1);
          if (!__all_sync(kFull, ok)) break;
          if (issuer) umma_commit(kKFree + 8u * buf);
        }
        if (j > 0) {                                                    // values of tile j - 1
          const int T = tiles_all + j - 1, buf = T & 1;
          bool ok = mbar_wait(kVFull + 8u * buf, T >> 1);
          if (ok && j - 1 < ntiles[0]) ok = values(j - 1, m0);
          if (ok && j - 1 < ntiles[1]) ok = values(j - 1, m1);
          if (!__all_sync(kFull, ok)) break;
          if (issuer) umma_commit(kVFree + 8u * buf);
        }
      }
    }
    __syncwarp();
    tiles_all += nt;
    tiles_m[0] += ntiles[0];
    tiles_m[1] += ntiles[1];
  }
  fence_before();
  __syncthreads();
  if (tid == 0 && lds32(kAbort) != 0u) {
    p.work_counter[1] = (int)lds32(kAbort);                 // (for whoever looks into the workspace)
    if (p.status) atomicOr(p.status, WTQ_STATUS_SCAN_TIMEOUT);
  }
  if (warp == kMmaWarp) {
    // A block that gave up may have products in flight: they end before their tensor memory
    // goes to somebody else (bounded, like every wait).
    fence_after();
    if (elect_one()) umma_commit(kLast);
    __syncwarp();
    for (int spin = 0; spin < kWaitTries && !mbar_try(kLast, 0u); ++spin) {
    }
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols) : "memory");
  }
}

template <int BWK, int BWV>
int launch(const Params &p, cudaStream_t stream) {
  using M = Map<BWK, BWV>;
  static std::atomic<bool> opted_in_dev[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !opted_in_dev[dev & 63].load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(prefill_kernel<BWK, BWV>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M::kDynamic);
    if (e != cudaSuccess) return check_cuda(e, "wtq_prefill: shared memory opt-in");
    opted_in_dev[dev & 63].store(true, std::memory_order_release);
  }
  const int64_t items = (int64_t)p.B * p.Hkv * p.row_blocks * p.num_splits;
  const int grid = p.balanced ? device_sms() : (int)std::min<int64_t>(items, device_sms());
  prefill_kernel<BWK, BWV><<<grid, kThreads, M::kDynamic, stream>>>(p);
  note_launches(1);
  return check_cuda(cudaGetLastError(), "wtq_prefill launch");
}

size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Tokens per chunk: a multiple of the tile, at least 256.
int chunk_tokens_for(int max_tokens, int splits) {
  int tokens = (max_tokens + splits - 1) / splits;
  tokens = (tokens + kTile - 1) / kTile * kTile;
  return tokens < 256 ? 256 : tokens;
}

// Shapes the balanced schedule serves: enough query rows for the tensor-core merge, at
// least half as many groups as multiprocessors (a run is never shorter than half a
// group, so fewer groups would leave blocks idle), and a plan that fits.
bool balanced_shape(int B, int Hq, int Hkv, int Q) {
  const int row_blocks = (Q * (Hq / Hkv) + kRows - 1) / kRows;
  const int64_t groups = (int64_t)B * Hkv * row_blocks;
  return (int64_t)B * Q * Hq >= 4096 && 2 * groups >= device_sms() &&
         (int64_t)B * row_blocks <= kMaxPairs;
}

// Equal chunks: items = groups x chunks run in waves of one per multiprocessor; every chunk
// beyond the first adds about 5 % (states to write and merge, queries to reload).  Both
// effects were measured at 16 x 8 kv heads x 8k tokens: 64 query tokens (128 groups) 690 /
// 726 / 769 us with 1 / 2 / 3 chunks, 256 query tokens (512 groups) 2549 / 2388 / 2633 us.
// Takes the count with the lowest modelled cost; chunks of at least 256 tokens.
int equal_chunks(int B, int Hq, int Hkv, int Q, int64_t max_tokens) {
  const int row_blocks = (Q * (Hq / Hkv) + kRows - 1) / kRows;
  const int64_t groups = (int64_t)B * Hkv * row_blocks;
  const int64_t sms = device_sms();
  const int64_t most = std::max<int64_t>(1, std::min<int64_t>(max_tokens / 256, 32));
  int64_t splits = 1;
  double best = 0.0;
  for (int64_t s = 1; s <= most; ++s) {
    const int64_t items = groups * s, waves = (items + sms - 1) / sms;
    const double cost = (1.0 + 0.05 * (double)(s - 1)) * (double)(waves * sms) / (double)items;
    if (s == 1 || cost < best - 1e-9) {
      best = cost;
      splits = s;
    }
  }
  // chunk sizes round up to whole tiles: drop chunks that would stay empty
  const int tokens = chunk_tokens_for((int)max_tokens, (int)splits);
  return (int)((max_tokens + tokens - 1) / tokens);
}

}  // namespace pf
}  // namespace wtq

using namespace wtq;

extern "C" int wtq_prefill_auto_splits(int B, int Hq, int Hkv, int Q, int max_pages, int S) {
  if (B < 1 || Hq < 1 || Hkv < 1 || Q < 1 || max_pages < 1 || S < 1 || Hq % Hkv) return 1;
  if (pf::balanced_shape(B, Hq, Hkv, Q)) return pf::kBalancedSlots;
  return pf::equal_chunks(B, Hq, Hkv, Q, (int64_t)max_pages * S);
}

static thread_local int g_last_schedule = -1;
extern "C" int wtq_prefill_last_schedule(void) { return g_last_schedule; }

extern "C" size_t wtq_prefill_workspace_bytes(int B, int Hq, int Hkv, int Q, int D, int num_splits) {
  if (B < 1 || Hq < 1 || Hkv < 1 || Q < 1 || D < 1 || num_splits < 1) return 0;
  const size_t rows = (size_t)B * Q * Hq;
  return 256 + pf::round_up((size_t)B * Q * sizeof(int32_t), 256) +
         pf::round_up(rows * D * sizeof(float), 256) +
         pf::round_up(rows * num_splits * D * sizeof(float), 256) +
         2 * pf::round_up(rows * num_splits * sizeof(float), 256) + 256 * 256;
}

extern "C" int wtq_prefill(const void *q, int dtype, const int64_t q_strides[2], void *out,
                           const int64_t out_strides[2], const wtq_side_t *k_side,
                           const wtq_side_t *v_side, const int32_t *page_table,
                           int64_t table_stride, const int32_t *seq_lens, float scale, int B, int Hq,
                           int Hkv, int Q, int D, int S, int P, int max_pages, int num_splits,
                           void *workspace, size_t workspace_bytes, int32_t *status, void *stream_) {
  cudaStream_t stream = (cudaStream_t)stream_;
  if (Q < 1) return fail(WTQ_ERR_ARG, "wtq_prefill: need Q >= 1");
  if (B > 0 && (int64_t)B * Q > (int64_t)1 << 24)
    return fail(WTQ_ERR_ARG, "wtq_prefill: B * Q is limited to 2^24 query tokens");
  // the rows of the call are the B * Q query tokens; everything the decode entry
  // checks about buffers, strides and shapes holds for them as for B sequences
  if (int rc = decode_validate(q, dtype, q_strides, out, out_strides, false, k_side, v_side,
                               page_table, seq_lens, B * Q, Hq, Hkv, D, S, P, max_pages))
    return rc;
  if (B == 0) return WTQ_OK;
  if (!workspace) return fail(WTQ_ERR_ARG, "wtq_prefill: null workspace");
  const int max_tokens = max_pages * S;
  const int64_t total_rows = (int64_t)B * Q * Hq;
  // Schedule.  An explicit num_splits cuts every history into that many equal chunks.
  // Left to the library (num_splits <= 0), shapes with enough groups and rows take the
  // balanced schedule (tiles dealt evenly to the blocks, three chunk slots per row) when
  // the output layout lets the tensor-core merge run; everything else takes equal chunks,
  // never more than wtq_prefill_auto_splits promised the caller's workspace.
  bool balanced = false;
  int splits = num_splits;
  if (num_splits <= 0) {
    splits = pf::equal_chunks(B, Hq, Hkv, Q, max_tokens);
    if (Hq % Hkv == 0 && pf::balanced_shape(B, Hq, Hkv, Q)) {
      MergeParams fit = {};
      fit.D = D; fit.Hq = Hq; fit.num_splits = pf::kBalancedSlots; fit.out = out;
      fit.osb = out_strides[0]; fit.osh = out_strides[1]; fit.Pi_v = v_side->Pi;
      fit.part_acc = (float *)workspace;                 // states start at a multiple of 256 bytes from here
      balanced = rows_mma_merge_eligible(fit, total_rows);
      splits = std::min(splits, pf::kBalancedSlots);
    }
  }
  splits = std::min(splits, std::max(1, max_tokens / pf::kTile));
  splits = std::min(splits, 256);
  const int chunk_tokens = pf::chunk_tokens_for(max_tokens, splits);
  splits = balanced ? pf::kBalancedSlots : (max_tokens + chunk_tokens - 1) / chunk_tokens;
  const size_t need = wtq_prefill_workspace_bytes(B, Hq, Hkv, Q, D, splits);
  if (workspace_bytes < need)
    return fail(WTQ_ERR_WORKSPACE, "wtq_prefill: workspace %zu < %zu bytes", workspace_bytes, need);

  pf::Params p;
  auto fill = [&](DecodeSideDev &d, const wtq_side_t &s) {
    d.pages = (const uint8_t *)s.pages; d.norms = (const __half *)s.norms;
    d.page_stride = s.page_stride; d.head_stride = s.head_stride;
    d.norm_page_stride = s.norm_page_stride; d.norm_head_stride = s.norm_head_stride;
    d.Pi = s.Pi; d.centroids = s.centroids; d.bw = s.bw; d.nb = D * s.bw / 8;
  };
  fill(p.k, *k_side);
  fill(p.v, *v_side);
  const size_t rows = (size_t)B * Q * Hq;
  char *ws = (char *)workspace;
  p.work_counter = (int32_t *)ws;
  ws += 256;
  p.row_lens = (int32_t *)ws;
  ws += pf::round_up((size_t)B * Q * sizeof(int32_t), 256);
  float *q_rot = (float *)ws;
  ws += pf::round_up(rows * D * sizeof(float), 256);
  p.part_acc = (float *)ws;
  ws += pf::round_up(rows * splits * D * sizeof(float), 256);
  p.part_m = (float *)ws;
  ws += pf::round_up(rows * splits * sizeof(float), 256);
  p.part_l = (float *)ws;
  ws += pf::round_up(rows * splits * sizeof(float), 256);
  p.lut = (const uint32_t *)ws;
  p.q_rot = q_rot;
  p.page_table = page_table; p.table_stride = table_stride; p.seq_lens = seq_lens;
  p.B = B; p.Hq = Hq; p.Hkv = Hkv; p.n_rep = Hq / Hkv; p.Q = Q; p.S = S; p.P = P;
  p.max_pages = max_pages; p.max_tokens = max_tokens; p.num_splits = splits;
  p.chunk_tokens = chunk_tokens;
  p.balanced = balanced ? 1 : 0;
  g_last_schedule = p.balanced;
  p.row_blocks = (Q * p.n_rep + pf::kRows - 1) / pf::kRows;
  p.status = status;
  if ((int64_t)B * Hkv * p.row_blocks * splits > (int64_t)1 << 30)
    return fail(WTQ_ERR_ARG, "wtq_prefill: too many work items; lower num_splits");

  // what the tensor-core kernels need of the layout (the same as the decode scan)
  DecodeParams probe = {};
  probe.k = p.k; probe.v = p.v; probe.D = D; probe.S = S; probe.n_rep = p.n_rep;
  probe.q_rot = q_rot; probe.part_acc = p.part_acc; probe.lut = p.lut;
  if (!mma_eligible(probe) || D != 128)
    return fail(WTQ_ERR_UNSUPPORTED, "wtq_prefill: needs head_dim 128, widths 4/4, 4/6, 6/6 or 8/8, "
                "a power-of-two page size >= 16, at most 8 query heads per kv head and 16-byte "
                "aligned pages");
  // balanced schedule: a row's slots that no piece writes must read as empty (l = 0)
  const int64_t zero_words = balanced ? (int64_t)rows * splits : 0;
  // rotation of the B * Q * Hq query rows (exp2 domain) and the lookup tables
  ScanSetup setup = {nullptr, (uint32_t *)p.lut, k_side->centroids, v_side->centroids, k_side->bw,
                     v_side->bw, mma_lut_words(k_side->bw, v_side->bw)};
  const float q_scale = scale * 1.4426950408889634f;
  if (rows_mma_rotate_eligible(q, q_strides[0], q_strides[1], Hq, D, total_rows, k_side->Pi, q_rot)) {
    if (int rc = launch_rotate_rows_mma(q, dtype, k_side->Pi, q_scale, total_rows, q_rot, setup, p.part_l,
                                        zero_words, p.work_counter, status, stream))
      return rc;
  } else {
    if (cudaMemsetAsync(p.work_counter, 0, 256, stream) != cudaSuccess)
      return check_cuda(cudaGetLastError(), "wtq_prefill: counter reset");
    if (zero_words && cudaMemsetAsync(p.part_l, 0, zero_words * sizeof(float), stream) != cudaSuccess)
      return check_cuda(cudaGetLastError(), "wtq_prefill: chunk state reset");
    if (int rc = launch_rotate_q(q, dtype, q_strides, k_side->Pi, q_scale, B * Q, Hq, D, q_rot,
                                 nullptr, chunk_tokens, max_tokens, setup, stream))
      return rc;
  }
  int rc = WTQ_ERR_UNSUPPORTED;
  if (p.k.bw == 4 && p.v.bw == 4) rc = pf::launch<4, 4>(p, stream);
  else if (p.k.bw == 4 && p.v.bw == 6) rc = pf::launch<4, 6>(p, stream);
  else if (p.k.bw == 6 && p.v.bw == 6) rc = pf::launch<6, 6>(p, stream);
  else if (p.k.bw == 8 && p.v.bw == 8) rc = pf::launch<8, 8>(p, stream);
  if (rc) return rc;
  MergeParams m = {};
  m.part_acc = p.part_acc; m.part_m = p.part_m; m.part_l = p.part_l;
  m.Pi_v = v_side->Pi; m.out = out; m.osb = out_strides[0]; m.osh = out_strides[1];
  m.dtype = dtype; m.Hq = Hq; m.D = D; m.num_splits = splits;
  m.work_counter = nullptr;
  // (balanced: slot c of a row is read when the row sees more than c tokens; a piece in
  // slot c starts at tile c or later, so no filled slot goes unread)
  if (balanced || rows_mma_merge_eligible(m, total_rows))
    return launch_merge_rows_mma(m, p.row_lens, total_rows, balanced ? 1 : chunk_tokens, max_tokens, status,
                                 stream);
  return launch_mma_merge(m, p.row_lens, B * Q, Hkv, p.n_rep, chunk_tokens, max_tokens, stream);
}
