// Fused dequantisation on the fifth-generation tensor cores (tcgen05): the
// same product as dequant_mma_kernel, out = (C Pi) * norm for head_dim 128 and
// widths 4/6/8, with the decoded operand and the 128 x 128 accumulator of a tile
// in tensor memory.
//
// A block takes tiles of 128 packed rows; three groups of warps meet only at mbarriers:
//   decode    eight warps, a thread per half row: 64 codes from the packed row become
//             fp16 centroid values through the per-lane lookup tables (wtq_lut.cuh) and go
//             to tensor memory as the A operand with tcgen05.st, no shared memory between;
//   multiply  one thread issues tcgen05.mma (M 128, N 128, K 16, fp16 in, fp32 out) for the
//             eight K steps of each product term; B is Pi with one row per output
//             coordinate, in shared memory in the canonical K-major layout without swizzle
//             (8-row x 16-byte core matrices); tcgen05.commit signals an mbarrier;
//   drain     eight warps read 32 lanes x 64 columns of the accumulator with tcgen05.ld,
//             scale by the row norm, convert, and pass the rows through a staging area so
//             that they leave as whole row segments.
// Operands and accumulators exist twice (512 columns in all), and the packed rows of the next
// two tiles are on their way into registers meanwhile.
// TERMS = 1: single fp16 operands.  TERMS = 3: centroids and Pi as fp16 high and
// low parts (times 2^8), the three significant products accumulated in the same
// tensor-memory tile.  Every wait is bounded; a wait that runs out marks the
// status word and the block leaves after freeing its tensor memory.
//
// Why tensor memory for A: an M 128, N 128, K 16 product with both operands in shared memory
// reads 8 KB of it in its 64 cycles, all that the SM's shared memory delivers, and the
// table lookups and the staging need as much again; and TMA stores, because plain ones back
// up the load/store pipes that lookups, staging and tcgen05.ld go through.  2^20 rows of 4 bits
// to bf16 (graph replay): 146 us with A in shared memory, 105 with A in tensor memory, 87 with
// TMA stores, of which the products take 45 at 1965 MHz; a plain fill of the output takes 73.
#include <cuda.h>

#include <atomic>
#include <cstring>
#include <mutex>

#include "wtq_common.cuh"
#include "wtq_lut.cuh"
#include "wtq_dequant.cuh"

namespace wtq {
namespace dq5 {

constexpr int kFeedWarps = 8, kDrainWarps = 8, kMmaWarp = kFeedWarps + kDrainWarps, kThreads = 32 * (kMmaWarp + 1);
constexpr int kSetupWarps = 16;                   // warps that lay out Pi and the tables
constexpr int kWarpCols = 128 / (kDrainWarps / 4); // accumulator columns a warp stores
constexpr uint32_t kBase = 1024;                  // dynamic shared memory is assumed to start at or below this
constexpr uint32_t kBarDone = kBase;              // 2 mbarriers: the products of operand b into accumulator b are complete
constexpr uint32_t kBarFree = kBase + 16;         // 2 mbarriers: accumulator b has been read out
constexpr uint32_t kBarFull = kBase + 32;         // 2 mbarriers: operand b is in tensor memory
constexpr uint32_t kTmemSlot = kBase + 48;        // tensor-memory address written by tcgen05.alloc
constexpr uint32_t kCent = kBase + 2048;          // 256 floats: the codebook while the tables are built
constexpr uint32_t kOperand = 128 * 128 * 2;      // one fp16 operand tile
constexpr uint32_t kBHi = 4096;
static_assert(kCent + 1024 <= kBHi && kBHi + kOperand <= mma::kLutAddr, "low region");
constexpr uint32_t kCols = 512;                   // tensor memory columns:
constexpr uint32_t kColD = 0;                     // + 128 * buffer: accumulators
constexpr uint32_t kColA = 256;                   // + 128 * buffer: operands, high parts then low parts
constexpr float kOperandScale = 256.f, kResultScale = 1.f / (256.f * 256.f);
// instruction descriptor: dense, fp32 accumulator, fp16 A and B, both K-major, N = 128, M = 128
constexpr uint32_t kIdesc = (1u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

constexpr uint32_t kBox = 32 * 128;
constexpr int kWaitTries = 1 << 20;               // polls of an mbarrier before a wait gives up (each suspends a while)

template <int BW, int TERMS, int DT> struct Map {
  static constexpr uint32_t kLutBytes = mma::lut_entries(BW) * 256u;
  static constexpr uint32_t kBLo = mma::kLutAddr + kLutBytes;
  // output staging: boxes of 32 rows x 128 bytes in the 128-byte swizzle (piece k of row r lies
  // at piece k ^ (r % 8)); a warp holds two: both of a tile (fp32), or of two tiles in turn
  static constexpr int kEsize = DT == WTQ_F32 ? 4 : 2;
  static constexpr int kBoxes = kWarpCols * kEsize / 128, kBoxCols = 128 / kEsize;
  static constexpr uint32_t kStage = kBLo + (TERMS == 3 ? kOperand : 0u), kStageBytes = 2 * kBox;
  static_assert(kStage % 1024 == 0, "swizzle atoms");
  static constexpr uint32_t kDynamic = kStage + kDrainWarps * kStageBytes;
  static_assert(kDynamic <= 227u * 1024u, "shared memory budget");
  // Table entries.  A 4-bit split table holds the high and the low pair of a byte's two codes
  // side by side (one 8-byte lookup); a 6/8-bit one holds both parts of a code in a word.
  static constexpr bool kPairEntries = BW == 4 && TERMS == 3;
  static constexpr int kLaneShift = kPairEntries ? 3 : 2;
};

// Element (row, piece) of an operand tile: 16-byte piece `piece` (8 values along K) of row `row`.
__device__ __forceinline__ uint32_t operand_at(uint32_t tile, int row, int piece) {
  return tile + (uint32_t)(row >> 3) * 2048u + (uint32_t)piece * 128u + (uint32_t)(row & 7) * 16u;
}
// Shared-memory descriptor of the two pieces (K = 16) starting at piece 2 * ks of a tile.
__device__ __forceinline__ uint64_t operand_desc(uint32_t tile, int ks) {
  const uint32_t start = tile + (uint32_t)ks * 256u;
  return (uint64_t)((start >> 4) & 0x3fffu) | ((uint64_t)(128u >> 4) << 16) |   // leading offset: next piece
         ((uint64_t)(2048u >> 4) << 32) |                                       // stride offset: next 8 rows
         ((uint64_t)1 << 46);                                                   // descriptor version, no swizzle
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w)
               : "memory");
}
__device__ __forceinline__ void umma(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b), "r"(kIdesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void tmem_store16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};\n"
      ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(addr)
      : "memory");
}
__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr));
}

// Codes 2 I, 2 I + 1, ... 31 of the 32 that the words hold, as fp16 pairs: high parts and
// (TERMS = 3) low parts.
template <int BW, int TERMS, int I>
__device__ __forceinline__ void decode_pairs(const uint32_t *w, uint32_t sel, uint32_t (&hi)[16], uint32_t (&lo)[16]) {
  if constexpr (I < 16) {
    if constexpr (BW == 4 && TERMS == 3) {
      const uint2 v = lds64(lut_addr<I & 3>(w[I >> 2], sel));
      hi[I] = v.x;
      lo[I] = v.y;
    } else if constexpr (BW == 4) {
      hi[I] = lut_byte<I & 3>(w[I >> 2], sel);
    } else {
      const uint32_t(&ws)[BW] = *reinterpret_cast<const uint32_t(*)[BW]>(w);
      const uint32_t a = lut_code<BW, 2 * I>(ws, sel), b = lut_code<BW, 2 * I + 1>(ws, sel);
      hi[I] = __byte_perm(a, b, 0x5410);
      if constexpr (TERMS == 3) lo[I] = __byte_perm(a, b, 0x7632);
    }
    decode_pairs<BW, TERMS, I + 1>(w, sel, hi, lo);
  }
}
// Half a packed row: 64 codes, 2 * BW words.
template <int BW>
__device__ __forceinline__ void load_half(const uint8_t *at, uint32_t (&w)[2 * BW]) {
  if constexpr (BW == 6) {                        // rows are 8-byte aligned at this width
#pragma unroll
    for (int i = 0; i < BW; ++i) {
      const uint2 v = __ldg(reinterpret_cast<const uint2 *>(at) + i);
      w[2 * i] = v.x; w[2 * i + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < BW / 2; ++i) {
      const uint4 v = __ldg(reinterpret_cast<const uint4 *>(at) + i);
      w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
  }
}

template <int DT> __device__ __forceinline__ uint32_t pack2(float x, float y) {
  if constexpr (DT == WTQ_BF16) {
    __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    return *reinterpret_cast<uint32_t *>(&h);
  } else {
    return pack_half2(x, y);
  }
}

// state (host memory): word 0 = 1 when the shared-memory layout assumption is broken, word
// 1 = 1 when a wait ran out and rows were left unwritten.
template <int BW, int TERMS, int DT>
__global__ void __launch_bounds__(kThreads, 1)
dequant_umma_kernel(DequantParams p, const __grid_constant__ CUtensorMap out_map,
                    const __grid_constant__ CUtensorMap out_map_b, int32_t *state) {
  using M = Map<BW, TERMS, DT>;
  extern __shared__ __align__(128) uint8_t dyn_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if ((uint32_t)__cvta_generic_to_shared(dyn_smem) > kBase) {
    if (tid == 0 && blockIdx.x == 0) state[0] = 1;
    return;
  }
  if (p.N == 0) return;                           // the set-up probe: nothing to read
  // ---- one-time: tensor memory, barriers, Pi, tables -------------------------------
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(kTmemSlot),
                 "r"(kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    if (lane == 0) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(kBarDone + 8u * b) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(kBarFree + 8u * b), "r"(kDrainWarps) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(kBarFull + 8u * b), "r"(kFeedWarps) : "memory");
      }
      asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
  }
  for (int e = tid; e < (1 << BW); e += kThreads)
    sts32(kCent + 4 * e, __float_as_uint(__ldg(p.centroids + e) * kOperandScale));
  // B[c][d] = Pi[d][c]: a lane takes column c = 8 cb + (lane & 7) and the rows d = 2 (4 db +
  // (lane >> 3)), d + 1 (sector-sized reads)
  if (warp < kSetupWarps) {
#pragma unroll 8
    for (int it = 0; it < 256 / kSetupWarps; ++it) {
      const int combo = it * kSetupWarps + warp, cb = combo & 15, db = combo >> 4;
      const int c = 8 * cb + (lane & 7), d = 2 * (4 * db + (lane >> 3));
      const float x0 = __ldg(p.Pi + d * 128 + c) * kOperandScale;
      const float x1 = __ldg(p.Pi + (d + 1) * 128 + c) * kOperandScale;
      const __half2 hi = __floats2half2_rn(x0, x1);
      const uint32_t off = operand_at(0, c, d >> 3) + (uint32_t)(d & 7) * 2u;
      sts32(kBHi + off, *reinterpret_cast<const uint32_t *>(&hi));
      if constexpr (TERMS == 3)
        sts32(M::kBLo + off, pack_half2(x0 - __low2float(hi), x1 - __high2float(hi)));
    }
  }
  __syncthreads();
  for (int idx = tid; idx < (int)(M::kLutBytes / 8); idx += kThreads) {     // entries x 32 lanes
    const int index = idx >> 5;
    float a, b;
    if constexpr (BW == 4) {
      a = __uint_as_float(lds32(kCent + 4 * (index & 15)));
      b = __uint_as_float(lds32(kCent + 4 * (index >> 4)));
    } else {
      a = b = __uint_as_float(lds32(kCent + 4 * index));
    }
    const __half2 hi = __floats2half2_rn(a, b);
    const uint32_t h = *reinterpret_cast<const uint32_t *>(&hi);
    const uint32_t l = pack_half2(a - __low2float(hi), b - __high2float(hi));
    const uint32_t at = mma::kLutAddr | (uint32_t)index << 8 | (uint32_t)(idx & 31) << M::kLaneShift;
    if constexpr (M::kPairEntries) {
      sts32(at, h);
      sts32(at + 4u, l);
    } else {
      sts32(at, BW == 4 ? h : __byte_perm(h, l, 0x5410));
    }
  }
  // what the tensor cores will read was written with ordinary stores
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = lds32(kTmemSlot);
  // The set-up above read the codebook and Pi only (which no kernel that lets its successor
  // in early writes) and ran under the tail of the kernel ahead; codes, norms and outputs are
  // touched after all earlier kernels.  The next kernel's blocks may move in as ours leave.
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

  // a call over two tensors (K and V of a layer): the second one's tiles follow the first's
  const int64_t tiles_each = (p.N + 127) >> 7, tiles = tiles_each * p.tensors;
  const uint32_t L32 = (uint32_t)p.L;
  const bool dense = p.L == p.MAXLEN;                       // source row = logical row: no plane arithmetic
  // source row of row lr of a tile of one tensor (rows past the end re-read the last one)
  auto source_of = [&](int64_t tile, int lr) -> int64_t {
    const int64_t row0 = tile << 7;
    lr = min(lr, (int)min((int64_t)127, p.N - 1 - row0));
    if (dense) return row0 + lr;
    const int64_t plane0 = row0 / p.L;
    const uint32_t pos = (uint32_t)(row0 - plane0 * p.L) + (uint32_t)lr, wrap = pos / L32;
    return (plane0 + wrap) * p.MAXLEN + (pos - wrap * L32);
  };
  // Bounded wait for completion number `use` (0, 1, ...) of an mbarrier; false if it ran out.
  auto wait_tries = [&](uint32_t bar, int use, int tries) -> bool {
    uint32_t done = 0;
    for (int spin = 0; spin < tries && !done; ++spin) {
      asm volatile(
          "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, q;\n\t}\n"
          : "=r"(done) : "r"(bar), "r"((uint32_t)(use & 1)) : "memory");
    }
    return done != 0;
  };
  auto wait_for = [&](uint32_t bar, int use) -> bool { return wait_tries(bar, use, p.wait_tries); };

  // Tile i of this block uses operand and accumulator i & 1.  What orders the groups:
  //   full[b]  arrives (once per decode warp) when operand b is in tensor memory;
  //   done[b]  arrives (tcgen05.commit) when the products of operand b into accumulator b are
  //            complete: the drain warps may read it, the decode warps overwrite the operand;
  //   free[b]  arrives (once per drain warp) when accumulator b is in registers.
  // Nobody is ever two completions ahead of a phase another group still waits for: operand b
  // is filled again only after done[b], accumulator b multiplied into only after free[b].
  // Every wait is bounded; whoever runs out of patience marks the state word and leaves its
  // loop, and the others then run out of patience too.
  if (warp < kFeedWarps) {
    // ---- decode: row 32 (warp % 4) + lane of the tile, codes 64 (warp / 4) .. + 63 -----------
    const int lr = 32 * (warp & 3) + lane, half = warp >> 2;
    const uint32_t sel = mma::kLutAddr | (uint32_t)(lane << M::kLaneShift);
    const uint32_t a_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + kColA + 32u * half;
    auto fetch = [&](int64_t tile, uint32_t (&w)[2 * BW]) {
      const bool second = tile >= tiles_each;
      load_half<BW>((second ? p.packed_b : p.packed) + source_of(tile - (second ? tiles_each : 0), lr) * (16 * BW) +
                        half * (8 * BW), w);
    };
    // one tile: codes in w to operand buf; then w is refilled for the tile after next
    auto feed = [&](int64_t tile, int i, int buf, uint32_t (&w)[2 * BW]) -> bool {
      if (i > 1) {
        const bool ok = wait_for(kBarDone + 8u * buf, (i - 2) >> 1);
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) state[1] = 1;
          return false;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t hi[16], lo[16];
        decode_pairs<BW, TERMS, 0>(w + c * BW, sel, hi, lo);
        tmem_store16(a_addr + 128u * buf + 16u * c, hi);
        if constexpr (TERMS == 3) tmem_store16(a_addr + 128u * buf + 64u + 16u * c, lo);
      }
      if (tile + 2 * (int64_t)gridDim.x < tiles) fetch(tile + 2 * (int64_t)gridDim.x, w);
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(kBarFull + 8u * buf) : "memory");
      return true;
    };
    uint32_t w0[2 * BW], w1[2 * BW];
    int64_t tile = blockIdx.x;
    if (tile < tiles) fetch(tile, w0);
    if (tile + gridDim.x < tiles) fetch(tile + gridDim.x, w1);
    for (int i = 0; tile < tiles; i += 2) {
      if (!feed(tile, i, 0, w0)) break;
      tile += gridDim.x;
      if (tile >= tiles || !feed(tile, i + 1, 1, w1)) break;
      tile += gridDim.x;
    }
  } else if (warp < kMmaWarp) {
    // ---- drain: row 32 (dw % 4) + lane, columns kWarpCols (dw / 4) .. -------------------------
    // (a warp may read the tensor-memory lanes 32 (warp % 4) ..; kFeedWarps is a multiple of 4)
    const int dw = warp - kFeedWarps, lr = 32 * (dw & 3) + lane;
    const uint32_t d_addr = tmem + ((uint32_t)(32 * (dw & 3)) << 16) + kColD + (uint32_t)(kWarpCols * (dw >> 2));
    const uint32_t stage = M::kStage + (uint32_t)dw * M::kStageBytes;
    constexpr int kRowBytes = kWarpCols * M::kEsize;
    int64_t tile = blockIdx.x;
    auto norm_at = [&](int64_t at) {
      const bool second = at >= tiles_each;
      return (second ? p.norms_b : p.norms)[source_of(at - (second ? tiles_each : 0), lr)];
    };
    __half nrm16 = __ushort_as_half(0);
    if (tile < tiles) nrm16 = norm_at(tile);
    for (int i = 0; tile < tiles; tile += gridDim.x, ++i) {
      const int buf = i & 1;
      const float nrm = __half2float(nrm16) * kResultScale;
      if (tile + gridDim.x < tiles) nrm16 = norm_at(tile + gridDim.x);
      const bool ok = wait_for(kBarDone + 8u * buf, i >> 1);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) state[1] = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      uint32_t v[kWarpCols / 32][32];
#pragma unroll
      for (int j = 0; j < kWarpCols / 32; ++j) tmem_load32(d_addr + 128u * buf + 32u * j, v[j]);
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      // the accumulator is in registers: hand the buffer back
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(kBarFree + 8u * buf) : "memory");
      // The thread holds consecutive columns of ONE row; stored as they are, every store
      // instruction of the warp would touch 32 rows.  They go through shared memory instead
      // (the swizzle puts the eight lanes that store together into different banks) and leave
      // as boxes by TMA, which keeps the stores out of the load/store pipes that the lookups,
      // the staging and the tensor-memory loads share.
      uint32_t q[kRowBytes / 4];                            // the row segment, converted
#pragma unroll
      for (int j = 0; j < kWarpCols / 32; ++j) {
        if constexpr (M::kEsize == 4) {
#pragma unroll
          for (int k = 0; k < 32; ++k) q[32 * j + k] = __float_as_uint(__uint_as_float(v[j][k]) * nrm);
        } else {
#pragma unroll
          for (int k = 0; k < 16; ++k)
            q[16 * j + k] = pack2<DT>(__uint_as_float(v[j][2 * k]) * nrm, __uint_as_float(v[j][2 * k + 1]) * nrm);
        }
      }
      const uint32_t box = stage + (M::kBoxes == 1 ? (uint32_t)buf * kBox : 0u);
      if (lane == 0) {                                       // the box written before is read out
        if constexpr (M::kBoxes == 1) asm volatile("cp.async.bulk.wait_group.read 1;\n" ::: "memory");
        else asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
      }
      __syncwarp();
#pragma unroll
      for (int k = 0; k < kRowBytes / 16; ++k)
        sts128(box + (uint32_t)(k >> 3) * kBox + (uint32_t)lane * 128u + (uint32_t)((k & 7) ^ (lane & 7)) * 16u,
               q[4 * k], q[4 * k + 1], q[4 * k + 2], q[4 * k + 3]);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      const bool second = tile >= tiles_each;
      const int64_t n0 = ((tile - (second ? tiles_each : 0)) << 7) + 32 * (dw & 3);
      if (lane == 0) {
        if (n0 < p.N) {                                      // (rows past the end are clipped by the map)
#pragma unroll
          for (int h = 0; h < M::kBoxes; ++h)
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];\n"
                         ::"l"(second ? &out_map_b : &out_map), "r"(kWarpCols * (dw >> 2) + M::kBoxCols * h), "r"((int)n0),
                         "r"(box + (uint32_t)h * kBox) : "memory");
        }
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
  } else if (lane == 0) {
    // ---- multiply: one thread ----------------------------------------------------------------
    int i = 0;
    for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++i) {
      const int buf = i & 1;
      bool ok = wait_for(kBarFull + 8u * buf, i >> 1);
      if (ok && i >= 2) ok = wait_for(kBarFree + 8u * buf, (i - 2) >> 1);
      if (!ok) {                 // nothing is issued: every later wait on done[] runs out as well
        state[1] = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t d = tmem + kColD + 128u * buf, a = tmem + kColA + 128u * buf;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        if constexpr (TERMS == 3) {
          umma(d, a + 64u + 8u * ks, operand_desc(kBHi, ks), ks > 0);
          umma(d, a + 8u * ks, operand_desc(M::kBLo, ks), 1u);
          umma(d, a + 8u * ks, operand_desc(kBHi, ks), 1u);
        } else {
          umma(d, a + 8u * ks, operand_desc(kBHi, ks), ks > 0);
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                   ::"r"(kBarDone + 8u * buf) : "memory");
    }
    // nothing is in flight when the tensor memory is freed, also where the others gave up
    if (i > 0) wait_tries(kBarDone + 8u * ((i - 1) & 1), (i - 1) >> 1, kWaitTries);
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kCols) : "memory");
}

}  // namespace dq5

namespace {

template <int BW, int TERMS, int DT> std::atomic<int> &variant_state(int dev) {
  static std::atomic<int> state[64];
  return state[dev & 63];
}

// The state words of every device, in pinned host memory so that a kernel which gave up is
// seen without asking the device.
std::atomic<int32_t *> g_words{nullptr};
int32_t *state_words(int dev) {                    // null where there is no memory to be had
  int32_t *words = g_words.load(std::memory_order_acquire);
  if (!words) {
    static std::mutex gate;
    std::lock_guard<std::mutex> hold(gate);
    words = g_words.load(std::memory_order_acquire);
    if (!words) {
      void *p = nullptr;
      if (cudaHostAlloc(&p, 64 * 2 * sizeof(int32_t), cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
      }
      memset(p, 0, 64 * 2 * sizeof(int32_t));
      words = (int32_t *)p;
      g_words.store(words, std::memory_order_release);
    }
  }
  return words + 2 * (dev & 63);
}
thread_local int t_wait_tries = dq5::kWaitTries;

}  // namespace

bool dequant_umma_gave_up() {
  int32_t *words = g_words.load(std::memory_order_acquire);
  if (!words) return false;
  int dev = 0;
  cudaGetDevice(&dev);
  words += 2 * (dev & 63) + 1;
  return __atomic_load_n(words, __ATOMIC_RELAXED) && __atomic_exchange_n(words, 0, __ATOMIC_ACQ_REL);
}
void dequant_umma_wait_tries(int tries) { t_wait_tries = tries < 0 ? dq5::kWaitTries : tries; }

// Tensor map of an output, (N, 128) elements, boxes of 32 rows x 128 bytes; false where the
// driver has no such call or refuses the tensor.
template <int DT> static bool output_map(CUtensorMap *map, void *out, int64_t N) {
  using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static const Encode encode = [] {
    void *f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      f = nullptr;
    return (Encode)f;
  }();
  if (!encode || N >= (int64_t)1 << 31) return false;
  constexpr int kEsize = DT == WTQ_F32 ? 4 : 2;
  const cuuint64_t dims[2] = {128, (cuuint64_t)N}, strides[1] = {128 * kEsize};
  const cuuint32_t box[2] = {128 / kEsize, 32}, steps[2] = {1, 1};
  const CUtensorMapDataType type = DT == WTQ_F32   ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : DT == WTQ_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                   : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  return encode(map, type, 2, out, dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Runs the tcgen05 kernel.  `*usable` comes back false (and nothing was
// launched for the call) when the kernel cannot be used here: the stream is
// capturing and the variant has not been set up yet, or the device places
// dynamic shared memory where the fixed addresses do not work.
template <int BW, int TERMS, int DT>
static int launch_variant(const DequantParams &p, cudaStream_t stream, bool *usable) {
  using M = dq5::Map<BW, TERMS, DT>;
  *usable = false;
  int dev = 0;
  cudaGetDevice(&dev);
  std::atomic<int> &state = variant_state<BW, TERMS, DT>(dev);
  auto kernel = dq5::dequant_umma_kernel<BW, TERMS, DT>;
  int s = state.load(std::memory_order_acquire);
  if (s == 0) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
      return WTQ_OK;
    static std::mutex gate;
    std::lock_guard<std::mutex> hold(gate);
    if ((s = state.load(std::memory_order_acquire)) == 0) {
      int32_t *const flag = state_words(dev);
      if (!flag) return WTQ_OK;
      cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)M::kDynamic);
      if (e == cudaSuccess) {
        DequantParams none = {};
        none.L = none.MAXLEN = 1;
        kernel<<<1, dq5::kThreads, M::kDynamic, stream>>>(none, CUtensorMap{}, CUtensorMap{}, flag);
        note_launches(1);
        e = cudaGetLastError();
      }
      if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
      if (e != cudaSuccess) return check_cuda(e, "wtq_dequant: tensor-memory kernel set-up");
      s = __atomic_load_n(flag, __ATOMIC_ACQUIRE) ? 2 : 1;
      state.store(s, std::memory_order_release);
    }
  }
  if (s != 1) return WTQ_OK;
  const int64_t tiles = (p.N + 127) / 128 * p.tensors;
  const int grid = (int)std::min<int64_t>(tiles, device_sms());
  CUtensorMap map, map_b;
  if (!output_map<DT>(&map, p.out, p.N) || !output_map<DT>(&map_b, p.tensors == 2 ? p.out_b : p.out, p.N))
    return WTQ_OK;
  cudaLaunchAttribute pdl;
  pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(dq5::kThreads);
  cfg.dynamicSmemBytes = M::kDynamic;
  cfg.stream = stream;
  cfg.attrs = &pdl;
  cfg.numAttrs = 1;
  DequantParams job = p;
  job.wait_tries = t_wait_tries;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, job, map, map_b, state_words(dev));
  note_launches(1);
  *usable = true;
  return check_cuda(e, "wtq_dequant tensor-memory launch");
}

template <int BW, int TERMS>
static int launch_dtype(const DequantParams &p, cudaStream_t stream, bool *usable) {
  if (p.out_dtype == WTQ_F32) return launch_variant<BW, TERMS, WTQ_F32>(p, stream, usable);
  if (p.out_dtype == WTQ_F16) return launch_variant<BW, TERMS, WTQ_F16>(p, stream, usable);
  return launch_variant<BW, TERMS, WTQ_BF16>(p, stream, usable);
}

int launch_dequant_umma(const DequantParams &p, int terms, cudaStream_t stream, bool *usable) {
  if (terms == 3) {
    if (p.bw == 4) return launch_dtype<4, 3>(p, stream, usable);
    if (p.bw == 6) return launch_dtype<6, 3>(p, stream, usable);
    return launch_dtype<8, 3>(p, stream, usable);
  }
  if (p.bw == 4) return launch_dtype<4, 1>(p, stream, usable);
  if (p.bw == 6) return launch_dtype<6, 1>(p, stream, usable);
  return launch_dtype<8, 1>(p, stream, usable);
}

}  // namespace wtq
