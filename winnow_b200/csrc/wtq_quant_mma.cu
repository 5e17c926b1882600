// Rotation + Lloyd-Max quantisation at head_dim 128 with the tensor cores doing
// the bulk of the arithmetic and the result still bit-exact.
//
// The contract (wtq_append.cu) fixes every rounding: a coordinate is ONE fp32 FMA
// chain over the 128 inputs in order.  Chains are slow (128 dependent FMAs and as
// many shared-memory reads for every coordinate: 64 K vectors took 414 us), and
// only matter where the last bits decide on which side of a bucket boundary the
// value falls.  So a warp takes 16 vectors and, without a barrier to any other:
//
//   1. reads them straight into the layout of the MMA's A fragments, which also
//      gives each lane whole partial sums of the norm (d = 2t, 2t + 1 mod 8);
//      norm and division exactly as the contract says;
//   2. y' = (x / |x|) Pi^T on mma.m16n8k16, both operands split into fp16 high and
//      low parts, high x high and the two cross terms in accumulators of their own;
//   3. bucket of y' from a table of cells.  |y' - y| <= kMargin, so the bucket is
//      y's own unless a boundary lies within kMargin of y';
//   4. the coordinates with a boundary that near (0.25 % at 4 bits, 3 % at 8) get
//      their chain, one lane each;
//   5. codes are packed eight at a time and stored.
//
// Measured, appends of K and V at 4 bits (8 bits): 512 tokens x 8 heads 16.8 us (20.6),
// before 150; 4 x 8 heads x 1999 tokens 88 us (152), before 830.  What bounds it is
// the latency of a pass (14 warps of 128 registers a multiprocessor, issue slots a
// third used): dependent divisions, MMA chains, one round of FMA chains; a form with
// block-wide phases and barriers took 130 us (268).
//
// kMargin is for rows of Pi no longer than 1, as a rotation's are; longer ones (any matrix
// is accepted) scale it, since every term below grows with |Pi_c|.  With sum_d |x_d| |Pi_cd| <= |x| |Pi_c| = 1, the chain is within
// 128 * 2^-24 = 7.6e-6 of the exact sum; the split operands leave out 3 * 2^-22
// = 7e-7; each of the 8 accumulating high x high MMAs adds 17 terms aligned to the
// largest (below 1) and cut at 24 bits, at most 17 * 2^-24 = 1.0e-6 each, and the
// cross terms 2^-11 of that.  2^-15 = 3.05e-5 is 1.8 times the sum.  (A NaN fails
// the comparison and takes the chain.)
#include <algorithm>
#include <atomic>

#include "wtq_lut.cuh"
#include "wtq_quant.cuh"

namespace wtq {
namespace qm {

constexpr int kWarps = 14, kThreads = 32 * kWarps;
constexpr int kVectors = 16;                          // a warp's pass
constexpr float kMargin = 3.0517578125e-5f;           // 2^-15
constexpr float kScale = 256.f, kUnscale = 1.f / 65536.f;   // operands times 2^8: low parts stay normal
constexpr int kXRow = 132;                            // floats per row of the normalised vectors
constexpr int kNearMost = 256;                        // list entries; a pass with more runs every chain

// A bucket is found by the cell of width 1 / kCells that y' falls into ([-1/2, 1/2); the end
// cells reach to infinity): the bucket of the cell's lower end, or the next one.
constexpr int kCells = 1024;

struct alignas(16) WarpSmem {
  float x[kVectors][kXRow];                           // normalised vectors, for the chains
  uint8_t idx[kVectors][128];
  uint16_t near[kNearMost];                           // coordinates that need their chain: v * 128 + c
};
struct Smem {
  uint4 pi[16][8][32];                                // B fragments: [8 coordinates][step][lane] {high, high, low, low}
  float2 around[256];                                 // boundaries below and above bucket k (-inf, +inf at the ends)
  uint8_t cell[kCells];                               // bucket of the lower end of each cell
  int crowded;                                        // a cell holds more than one boundary: search instead
  int longest;                                        // the largest |Pi_c|^2, as bits
  WarpSmem warp[kWarps];
};

__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo) {
  const __half2 h = __floats2half2_rn(a, b);
  hi = *reinterpret_cast<const uint32_t *>(&h);
  lo = pack_half2(a - __low2float(h), b - __high2float(h));
}
// number of boundaries strictly below y, by binary search
__device__ __forceinline__ int bucket(const Smem &s, int n, float y) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (s.around[mid].y < y) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}
__device__ __forceinline__ uint32_t nibbles(uint32_t x) {            // four codes of 4 bits -> 16 bits
  x |= x >> 4;
  return __byte_perm(x, 0, 0x4420);
}
__device__ __forceinline__ uint32_t sixes(uint32_t x) {              // four codes of 6 bits -> 24 bits
  return (x & 0x3fu) | ((x >> 2) & 0xfc0u) | ((x >> 4) & 0x3f000u) | ((x >> 6) & 0xfc0000u);
}
// codes 8 i .. 8 i + 7 of a row -> bytes bw i .. bw i + bw - 1 of the packed row
__device__ __forceinline__ void store_codes(uint8_t *row, int i, uint2 codes, int bw, bool words) {
  uint8_t *at = row + bw * i;
  if (words && bw == 4) {
    *reinterpret_cast<uint32_t *>(at) = nibbles(codes.x) | nibbles(codes.y) << 16;
    return;
  }
  if (words && bw == 8) {
    *reinterpret_cast<uint2 *>(at) = codes;
    return;
  }
  if (words && bw == 6) {
    const uint32_t lo = sixes(codes.x), hi = sixes(codes.y);
    uint16_t *h = reinterpret_cast<uint16_t *>(at);
    h[0] = (uint16_t)lo;
    h[1] = (uint16_t)(lo >> 16 | hi << 8);
    h[2] = (uint16_t)(hi >> 8);
    return;
  }
  uint64_t v = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v |= (uint64_t)((codes.x >> (8 * j)) & 255u) << (bw * j);
    v |= (uint64_t)((codes.y >> (8 * j)) & 255u) << (bw * (j + 4));
  }
  for (int j = 0; j < bw; ++j) at[j] = (uint8_t)(v >> (8 * j));
}

// Elements off, off + 1 of the source as floats.
__device__ __forceinline__ float2 load_pair(const void *src, int64_t off, int dtype, bool words) {
  if (words) {
    if (dtype == WTQ_F32) return *reinterpret_cast<const float2 *>((const float *)src + off);
    const uint32_t w = *reinterpret_cast<const uint32_t *>((const uint16_t *)src + off);
    if (dtype == WTQ_F16) return __half22float2(*reinterpret_cast<const __half2 *>(&w));
    return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
  }
  return make_float2(load_as_float(src, off, dtype), load_as_float(src, off + 1, dtype));
}

// Element offset of vector `vec` in the source; for an append also its place in the batch.
struct Source {
  int64_t from;
  int b, h, i;
};
template <bool APPEND> __device__ __forceinline__ Source source_of(const QuantJob &job, const QuantJobSide &a, int64_t vec) {
  Source r = {};
  if (APPEND) {                                                   // (a call's vectors number less than 2^32: see the launch)
    const uint32_t v = (uint32_t)vec, bh = v / (uint32_t)job.n;
    r.i = (int)(v - bh * (uint32_t)job.n);
    r.b = (int)(bh / (uint32_t)job.Hkv);
    r.h = (int)(bh - (uint32_t)r.b * (uint32_t)job.Hkv);
    r.from = (int64_t)r.b * a.sb + (int64_t)r.h * a.sh + (int64_t)r.i * a.st;
  } else {
    r.from = vec * a.st;
  }
  return r;
}

// Blocks blockIdx.x walk the passes of side blockIdx.y.
template <bool APPEND>
__global__ void __launch_bounds__(kThreads, 1) quant_mma_kernel(QuantJob job) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Smem &s = *reinterpret_cast<Smem *>(smem_raw);
  const QuantJobSide &a = job.side[blockIdx.y];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nbounds = a.q.nbounds, bw = a.q.bw;
  constexpr uint32_t kFull = 0xffffffffu;
  WarpSmem &w = s.warp[warp];
  // ---- constants: Pi as B fragments (n = output coordinate, k = input coordinate),
  // boundaries, cells ------------------------------------------------------------------
  float *squares = reinterpret_cast<float *>(s.warp);  // of each fragment, until the warps' tiles are used
#pragma unroll 4
  for (int e = warp; e < 128; e += kWarps) {
    const int nt = e >> 3, ks = e & 7;
    const float *row = a.q.Pi + (8 * nt + g) * 128 + 16 * ks + 2 * t;
    const float2 p = __ldg(reinterpret_cast<const float2 *>(row)), q = __ldg(reinterpret_cast<const float2 *>(row + 8));
    uint4 f;
    split2(p.x * kScale, p.y * kScale, f.x, f.z);
    split2(q.x * kScale, q.y * kScale, f.y, f.w);
    s.pi[nt][ks][lane] = f;
    squares[e * 32 + lane] = fmaf(p.x, p.x, fmaf(p.y, p.y, fmaf(q.x, q.x, q.y * q.y)));
  }
  for (int e = tid; e <= nbounds; e += kThreads)
    s.around[e] = make_float2(e > 0 ? __ldg(a.q.bounds + e - 1) : -INFINITY, e < nbounds ? __ldg(a.q.bounds + e) : INFINITY);
  if (tid == 0) s.crowded = s.longest = 0;
  __syncthreads();
  if (tid >= kThreads - 128) {                        // (the threads with fewest cells)
    const int c = tid - (kThreads - 128);
    float sum = 0.f;
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const float4 v = *reinterpret_cast<const float4 *>(squares + ((c >> 3) * 8 + ks) * 32 + (c & 7) * 4);
      sum += (v.x + v.y) + (v.z + v.w);
    }
    const int most = __reduce_max_sync(kFull, __float_as_int(fabsf(sum)));       // (a NaN beats every number)
    if (lane == 0) atomicMax(&s.longest, most);
  }
  // (cells start at multiples of 2^-10, exact in fp32)
  for (int e = tid; e < kCells; e += kThreads)
    s.cell[e] = (uint8_t)(e == 0 ? 0 : bucket(s, nbounds, (float)e * (1.f / kCells) - 0.5f));
  __syncthreads();
  for (int e = tid; e < kCells; e += kThreads)
    if ((e == kCells - 1 ? nbounds : s.cell[e + 1]) - s.cell[e] > 1) s.crowded = 1;
  __syncthreads();
  const bool crowded = s.crowded != 0;
  const float longest = __int_as_float(s.longest);
  const float margin = longest <= 1.0001f ? kMargin : kMargin * sqrtf(longest);   // (NaN stays: every chain runs)
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

  // A team of 2^ts warps takes a pass, each of them 128 / 2^ts of the output coordinates
  // (and all of the normalisation): unit = pass * 2^ts + part.
  const int ts = job.team_shift;
  const int64_t vectors = job.vectors, units = (vectors + kVectors - 1) / kVectors << ts;
  for (int64_t unit = blockIdx.x + (int64_t)gridDim.x * warp; unit < units; unit += (int64_t)gridDim.x * kWarps) {
    const int64_t v0 = (unit >> ts) * kVectors;
    const int part = (int)(unit & ((1 << ts) - 1));
    // ---- where vector `lane` (of 16) comes from and goes -----------------------------
    const int64_t vec = min(v0 + (lane & 15), vectors - 1);       // (vectors past the end repeat the last one)
    const bool mine = lane < 16 && v0 + lane < vectors;
    const Source at_v = source_of<APPEND>(job, a, vec);
    const int64_t from = at_v.from;
    {                                                             // the rows of this warp's next pass -> L2
      const int64_t next = ((unit + (int64_t)gridDim.x * kWarps) >> ts) * kVectors + (lane & 15);
      if (next < vectors) {
        const int el = job.dtype == WTQ_F32 ? 4 : 2;
        const char *p = (const char *)a.src + source_of<APPEND>(job, a, next).from * el + (lane >> 4) * 128;
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
        if (el == 4) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p + 256));
      }
    }
    int64_t code_off = -1, norm_off = -1;
    if (APPEND && mine) {
      const int pos = job.seq_lens[at_v.b] - job.n + at_v.i;
      const int slot_page = pos >= 0 ? pos / job.S : -1;
      if (pos < 0 || slot_page >= job.max_pages) {
        if (job.status) atomicOr(job.status, WTQ_STATUS_BAD_POSITION);
      } else {
        const int pid = job.page_table[(int64_t)at_v.b * job.table_stride + slot_page];
        if (pid < 0 || pid >= job.P) {
          if (job.status) atomicOr(job.status, WTQ_STATUS_BAD_PAGE);
        } else {
          const int slot = pos - slot_page * job.S;
          code_off = (int64_t)pid * a.page_stride + (int64_t)at_v.h * a.head_stride + (int64_t)slot * a.q.nb;
          norm_off = (int64_t)pid * a.norm_page_stride + (int64_t)at_v.h * a.norm_head_stride + slot;
        }
      }
    } else if (!APPEND && mine) {
      code_off = vec * a.q.nb;
      norm_off = vec;
    }
    // ---- rows g and g + 8: norm, division, A fragments ---------------------------------
    uint32_t ah[8][4], al[8][4];
    float norm[2], near_by[2];                                    // near_by: how near a boundary asks for the chain
    float2 x[2][16];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int64_t off = __shfl_sync(kFull, from, g + 8 * r) + 2 * t;
#pragma unroll
      for (int m = 0; m < 16; ++m) x[r][m] = load_pair(a.src, off + 8 * m, job.dtype, a.vec_src);
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float s0 = 0.f, s1 = 0.f;                                   // partial sums d = 2t and 2t + 1 mod 8
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        s0 = __fadd_rn(s0, __fmul_rn(x[r][m].x, x[r][m].x));
        s1 = __fadd_rn(s1, __fmul_rn(x[r][m].y, x[r][m].y));
      }
      float total = __fadd_rn(__shfl_sync(kFull, s0, lane & 28), __shfl_sync(kFull, s1, lane & 28));
#pragma unroll
      for (int k = 1; k < 4; ++k) {
        total = __fadd_rn(total, __shfl_sync(kFull, s0, (lane & 28) + k));
        total = __fadd_rn(total, __shfl_sync(kFull, s1, (lane & 28) + k));
      }
      norm[r] = fmaxf(__fsqrt_rn(total), 1e-10f);
      near_by[r] = margin;
      // A vector of zeros (padding) gives y = y' = 0 exactly, and a boundary is often there:
      // no chains for it.  (A NaN among the products still fails the comparison.)
      if (__any_sync(kFull, total == 0.f)) {
        bool zero = total == 0.f;
#pragma unroll
        for (int m = 0; m < 16; ++m) zero = zero && x[r][m].x == 0.f && x[r][m].y == 0.f;
        if ((__ballot_sync(kFull, zero) >> (lane & 28) & 15u) == 15u) near_by[r] = -1.f;
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        const float2 y = make_float2(__fdiv_rn(x[r][m].x, norm[r]), __fdiv_rn(x[r][m].y, norm[r]));
        *reinterpret_cast<float2 *>(&w.x[g + 8 * r][8 * m + 2 * t]) = y;
        split2(y.x * kScale, y.y * kScale, ah[m >> 1][r + 2 * (m & 1)], al[m >> 1][r + 2 * (m & 1)]);
      }
    __syncwarp();
    // ---- products, buckets: sixteen output coordinates at a time ---------------------------
    int near = 0;
#pragma unroll 1
    for (int np = part << (3 - ts); np < (part + 1) << (3 - ts); ++np) {
      float hh[2][4], lh[2][4], hl[2][4];                        // six independent chains of MMAs
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) hh[i][e] = lh[i][e] = hl[i][e] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 8; ++ks)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint4 f = s.pi[2 * np + i][ks][lane];
          mma16816_free(lh[i], al[ks][0], al[ks][1], al[ks][2], al[ks][3], f.x, f.y);
          mma16816_free(hl[i], ah[ks][0], ah[ks][1], ah[ks][2], ah[ks][3], f.z, f.w);
          mma16816_free(hh[i], ah[ks][0], ah[ks][1], ah[ks][2], ah[ks][3], f.x, f.y);
        }
      int k[8];
      bool doubt[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float y = (hh[e >> 2][e & 3] + (lh[e >> 2][e & 3] + hl[e >> 2][e & 3])) * kUnscale;
        float2 edge;
        if (!crowded) {
          k[e] = s.cell[min(__float2uint_rz(fmaf(y, (float)kCells, 0.5f * kCells)), kCells - 1u)];
          edge = s.around[k[e]];
          if (edge.y < y) edge = s.around[++k[e]];
        } else {
          k[e] = bucket(s, nbounds, y);
          edge = s.around[k[e]];
        }
        doubt[e] = !(y - edge.x > near_by[(e >> 1) & 1]) || !(edge.y - y > near_by[(e >> 1) & 1]);
      }
#pragma unroll
      for (int e = 0; e < 8; e += 2)                             // rows g, g + 8; coordinates 2t, 2t + 1
        *reinterpret_cast<uint16_t *>(&w.idx[g + 8 * ((e >> 1) & 1)][16 * np + 8 * (e >> 2) + 2 * t]) =
            (uint16_t)(k[e] | k[e + 1] << 8);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const uint32_t votes = __ballot_sync(kFull, doubt[e]);
        if (votes) {
          const int at = near + __popc(votes & ((1u << lane) - 1u));
          if (doubt[e] && at < kNearMost)
            w.near[at] = (uint16_t)((g + 8 * ((e >> 1) & 1)) * 128 + 16 * np + 8 * (e >> 2) + 2 * t + (e & 1));
          near += __popc(votes);
        }
      }
    }
    __syncwarp();
    // ---- the chains of the coordinates near a boundary --------------------------------------
    const bool all = near > kNearMost;
    const int chains = all ? kVectors * 128 : near;
#pragma unroll 1
    for (int e = lane; e < chains; e += 32) {
      const int at = all ? e : w.near[e], v = at >> 7, c = at & 127;
      if (all && (c >> (7 - ts)) != part) continue;
      const float4 *row = reinterpret_cast<const float4 *>(a.q.Pi + c * 128);
      const float4 *x = reinterpret_cast<const float4 *>(&w.x[v][0]);
      float acc = 0.f;
#pragma unroll 16
      for (int d = 0; d < 32; ++d) {
        const float4 p = __ldg(row + d), z = x[d];
        acc = __fmaf_rn(z.x, p.x, acc);
        acc = __fmaf_rn(z.y, p.y, acc);
        acc = __fmaf_rn(z.z, p.z, acc);
        acc = __fmaf_rn(z.w, p.w, acc);
      }
      w.idx[v][c] = (uint8_t)bucket(s, nbounds, acc);
    }
    __syncwarp();
    // ---- pack and store: a lane packs eight codes --------------------------------------------
#pragma unroll 1
    for (int e = lane; e < kVectors * 16 >> ts; e += 32) {
      const int v = e >> (4 - ts), i = (part << (4 - ts)) + (e & ((16 >> ts) - 1));
      const int64_t to = __shfl_sync(kFull, code_off, v);
      if (to < 0) continue;
      const uint2 codes = *reinterpret_cast<const uint2 *>(&w.idx[v][8 * i]);
      if (!APPEND && a.idx) {
        uint8_t *dst = a.idx + (v0 + v) * 128 + 8 * i;
        if (a.vec_dst) *reinterpret_cast<uint2 *>(dst) = codes;
        else
          for (int j = 0; j < 8; ++j) dst[j] = w.idx[v][8 * i + j];
      }
      if (APPEND || a.pages) store_codes(a.pages + to, i, codes, bw, a.vec_dst);
    }
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int64_t to = __shfl_sync(kFull, norm_off, g + 8 * r);
      if (t == 0 && part == 0 && to >= 0) {
        if (APPEND) a.norms[to] = __float2half_rn(norm[r]);
        else if (a.norms32) a.norms32[to] = norm[r];
      }
    }
    __syncwarp();                                                // the warp's tiles are reused by its next pass
  }
}

template <bool APPEND>
int launch(const QuantJob &job, int sides, int blocks, cudaStream_t stream, const char *what) {
  auto kernel = quant_mma_kernel<APPEND>;
  const int bytes = (int)sizeof(Smem);
  static_assert(sizeof(Smem) <= 227 * 1024 && offsetof(Smem, warp) % 16 == 0 && sizeof(WarpSmem) % 16 == 0, "shared memory plan");
  static std::atomic<bool> opted_in_dev[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !opted_in_dev[dev & 63].load(std::memory_order_acquire)) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return check_cuda(e, what);
    opted_in_dev[dev & 63].store(true, std::memory_order_release);
  }
  cudaLaunchAttribute pdl;
  pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  pdl.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, (unsigned)sides);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = stream;
  cfg.attrs = &pdl;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, job);
  note_launches(1);
  return check_cuda(e, what);
}

}  // namespace qm

bool quant_mma_eligible(int D, int order, const QuantJob &job, int sides) {
  if (D != 128 || order != WTQ_ORDER_SEQUENTIAL || job.vectors >= (int64_t)1 << 32) return false;
  for (int i = 0; i < sides; ++i)
    if (((uintptr_t)job.side[i].q.Pi & 15) != 0) return false;
  return true;
}

// Passes of sixteen vectors, dealt to the blocks first and to their warps second.  A
// pass takes one warp about 10 us whatever runs beside it, so where passes are fewer
// than warps a team of up to eight shares each.
int launch_quant_mma(QuantJob job, bool append, int sides, cudaStream_t stream, const char *what) {
  const int64_t passes = (job.vectors + qm::kVectors - 1) / qm::kVectors;
  const int most = std::max(1, device_sms() / sides);
  job.team_shift = 0;
  while (job.team_shift < 3 && (passes << (job.team_shift + 1)) <= (int64_t)most * qm::kWarps) ++job.team_shift;
  const int blocks = (int)std::min<int64_t>(passes << job.team_shift, most);
  return append ? qm::launch<true>(job, sides, blocks, stream, what)
                : qm::launch<false>(job, sides, blocks, stream, what);
}

}  // namespace wtq
