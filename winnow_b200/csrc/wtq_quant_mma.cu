// Rotation + Lloyd-Max quantisation at head_dim 128 with the tensor cores doing
// the bulk of the arithmetic and the result still bit-exact.
//
// The contract (wtq_append.cu) fixes every rounding: a coordinate is ONE fp32 FMA
// chain over the 128 inputs in order.  Chains are slow (a block's 128 threads
// spent 128 dependent FMAs and as many shared-memory reads on every vector:
// 64 K vectors took 414 us), and only matter where the last bits decide on which
// side of a bucket boundary the value falls.  So:
//
//   1. norm and division exactly as the contract says (8 partial sums per vector,
//      eight lanes per vector);
//   2. y' = (x / |x|) Pi^T on mma.m16n8k16 with both operands split into fp16 high
//      and low parts (three products, fp32 accumulation);
//   3. bucket of y' by binary search.  |y' - y| <= kMargin, so the bucket is y's own
//      unless a boundary lies within kMargin of y';
//   4. the few coordinates with a boundary that near (0.5 % at 4 bits, 6 % at 8) go
//      on a list and get their chain, one thread each;
//   5. codes are packed eight at a time and stored.
//
// kMargin: with sum_d |x_d| |Pi_cd| <= |x| |Pi_c| = 1, the chain is within
// 128 * 2^-24 = 7.6e-6 of the exact sum; the split operands leave out 3 * 2^-22
// = 7e-7; and 24 accumulating MMAs that each keep at least 24 bits below the
// largest term add at most 24 * 4 * 2^-22 = 2.3e-5.  2^-14 = 6.1e-5 covers twice
// their sum.  (A NaN fails the comparison and takes the chain.)
#include <algorithm>
#include <atomic>

#include "wtq_lut.cuh"
#include "wtq_quant.cuh"

namespace wtq {
namespace qm {

constexpr int kThreads = 256, kWarps = 8;
constexpr float kMargin = 6.103515625e-5f;            // 2^-14
constexpr float kScale = 256.f, kUnscale = 1.f / 65536.f;   // operands times 2^8: low parts stay normal
// row strides: consecutive rows start 8 banks apart in both tiles
constexpr int kXRow = 136;                            // floats per row of the fp32 tile
constexpr int kHRow = 144;                            // halves per row of an fp16 tile

template <int VB> struct Smem {
  float x[VB][kXRow];                                 // normalised vectors
  __half hi[VB][kHRow], lo[VB][kHRow];                // the same times 2^8, split
  uint8_t idx[VB][128];
  float bounds[257];                                  // -inf, boundaries, +inf
  float norm[VB];
  int64_t code_off[VB], norm_off[VB];                 // append: where the vector goes, -1: nowhere
  int near_count;
  uint16_t near[VB * 128];                            // coordinates that need their chain: v * 128 + c
};

__device__ __forceinline__ void split2(float a, float b, uint32_t &hi, uint32_t &lo) {
  const __half2 h = __floats2half2_rn(a, b);
  hi = *reinterpret_cast<const uint32_t *>(&h);
  lo = pack_half2(a - __low2float(h), b - __high2float(h));
}
// bucket of y among the boundaries b[1 .. n]: how many lie strictly below it
__device__ __forceinline__ int bucket(const float *b, int n, float y) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (b[mid + 1] < y) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}
// codes 8 i .. 8 i + 7 of a row -> bytes bw i .. bw i + bw - 1 of the packed row
__device__ __forceinline__ void store_codes(uint8_t *row, int i, uint2 codes, int bw, bool words) {
  uint64_t v = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v |= (uint64_t)((codes.x >> (8 * j)) & 255u) << (bw * j);
    v |= (uint64_t)((codes.y >> (8 * j)) & 255u) << (bw * (j + 4));
  }
  uint8_t *at = row + bw * i;
  if (words && bw == 4) {
    *reinterpret_cast<uint32_t *>(at) = (uint32_t)v;
  } else if (words && bw == 8) {
    *reinterpret_cast<uint2 *>(at) = make_uint2((uint32_t)v, (uint32_t)(v >> 32));
  } else if (words && bw == 6) {
    uint16_t *h = reinterpret_cast<uint16_t *>(at);
    h[0] = (uint16_t)v; h[1] = (uint16_t)(v >> 16); h[2] = (uint16_t)(v >> 32);
  } else {
    for (int j = 0; j < bw; ++j) at[j] = (uint8_t)(v >> (8 * j));
  }
}

// VB vectors per pass; grid.x blocks walk the vectors of side blockIdx.y.
template <int VB, bool APPEND>
__global__ void __launch_bounds__(kThreads, 2) quant_mma_kernel(QuantJob job) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  Smem<VB> &s = *reinterpret_cast<Smem<VB> *>(smem_raw);
  const QuantJobSide &a = job.side[blockIdx.y];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int nbounds = a.q.nbounds, bw = a.q.bw;
  // ---- constants: fragments of this warp's 16 output coordinates, boundaries ------
  // B operand, n = output coordinate, k = input coordinate.  The contraction order is
  // free: the lane's four values of step ks are d = 16 ks + 4 t .. 4 t + 3.
  uint32_t bh[2][8][2], bl[2][8][2];
#pragma unroll
  for (int nt = 0; nt < 2; ++nt) {
    const float4 *row = reinterpret_cast<const float4 *>(a.q.Pi + (16 * warp + 8 * nt + g) * 128);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const float4 w = __ldg(row + 4 * ks + t);
      split2(w.x * kScale, w.y * kScale, bh[nt][ks][0], bl[nt][ks][0]);
      split2(w.z * kScale, w.w * kScale, bh[nt][ks][1], bl[nt][ks][1]);
    }
  }
  for (int e = tid; e < nbounds; e += kThreads) s.bounds[e + 1] = __ldg(a.q.bounds + e);
  if (tid == 0) {
    s.bounds[0] = -INFINITY;
    s.bounds[nbounds + 1] = INFINITY;
    s.near_count = 0;
  }
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");

  const int64_t vectors = job.vectors;
  for (int64_t v0 = (int64_t)blockIdx.x * VB; v0 < vectors; v0 += (int64_t)gridDim.x * VB) {
    // ---- where the vectors come from and go ---------------------------------------
    if (APPEND && tid < VB) {
      const int64_t vec = v0 + tid;
      int64_t code_off = -1, norm_off = -1;
      if (vec < vectors) {
        const int i = (int)(vec % job.n);
        const int h = (int)((vec / job.n) % job.Hkv);
        const int b = (int)(vec / ((int64_t)job.n * job.Hkv));
        const int pos = job.seq_lens[b] - job.n + i;
        const int slot_page = pos >= 0 ? pos / job.S : -1;
        if (pos < 0 || slot_page >= job.max_pages) {
          if (job.status) atomicOr(job.status, WTQ_STATUS_BAD_POSITION);
        } else {
          const int pid = job.page_table[(int64_t)b * job.table_stride + slot_page];
          if (pid < 0 || pid >= job.P) {
            if (job.status) atomicOr(job.status, WTQ_STATUS_BAD_PAGE);
          } else {
            const int slot = pos - slot_page * job.S;
            code_off = (int64_t)pid * a.page_stride + (int64_t)h * a.head_stride + (int64_t)slot * a.q.nb;
            norm_off = (int64_t)pid * a.norm_page_stride + (int64_t)h * a.norm_head_stride + slot;
          }
        }
      }
      s.code_off[tid] = code_off;
      s.norm_off[tid] = norm_off;
    }
    // ---- load: a warp takes rows warp, warp + 8, ..; a lane four coordinates ---------
#pragma unroll
    for (int r = warp; r < VB; r += kWarps) {
      const int64_t vec = v0 + r;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (vec < vectors) {
        int64_t off;
        if (APPEND) {
          const int i = (int)(vec % job.n);
          const int h = (int)((vec / job.n) % job.Hkv);
          const int b = (int)(vec / ((int64_t)job.n * job.Hkv));
          off = (int64_t)b * a.sb + (int64_t)h * a.sh + (int64_t)i * a.st;
        } else {
          off = vec * a.st;
        }
        off += 4 * lane;
        if (a.vec_src) {
          if (job.dtype == WTQ_F32) {
            x = *reinterpret_cast<const float4 *>((const float *)a.src + off);
          } else {
            const uint2 w = *reinterpret_cast<const uint2 *>((const uint16_t *)a.src + off);
            if (job.dtype == WTQ_F16) {
              const float2 p = __half22float2(*reinterpret_cast<const __half2 *>(&w.x));
              const float2 q = __half22float2(*reinterpret_cast<const __half2 *>(&w.y));
              x = make_float4(p.x, p.y, q.x, q.y);
            } else {
              x = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u),
                              __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
            }
          }
        } else {
          x = make_float4(load_as_float(a.src, off, job.dtype), load_as_float(a.src, off + 1, job.dtype),
                          load_as_float(a.src, off + 2, job.dtype), load_as_float(a.src, off + 3, job.dtype));
        }
      }
      *reinterpret_cast<float4 *>(&s.x[r][4 * lane]) = x;
    }
    __syncthreads();
    // ---- norm and division: eight lanes per vector, lane j the partial sum d = j mod 8 --
#pragma unroll 1
    for (int r = tid >> 3; r < VB; r += kThreads / 8) {
      const int j = tid & 7;
      float x[16], acc = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = s.x[r][j + 8 * i];
#pragma unroll
      for (int i = 0; i < 16; ++i) acc = __fadd_rn(acc, __fmul_rn(x[i], x[i]));
      float total = __shfl_sync(0xffffffffu, acc, lane & 24);
#pragma unroll
      for (int k = 1; k < 8; ++k) total = __fadd_rn(total, __shfl_sync(0xffffffffu, acc, (lane & 24) + k));
      const float norm = fmaxf(__fsqrt_rn(total), 1e-10f);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float y = __fdiv_rn(x[i], norm);
        s.x[r][j + 8 * i] = y;
        const __half h = __float2half_rn(y * kScale);
        s.hi[r][j + 8 * i] = h;
        s.lo[r][j + 8 * i] = __float2half_rn(y * kScale - __half2float(h));
      }
      if (j == 0) s.norm[r] = norm;
    }
    __syncthreads();
    // ---- products, buckets ------------------------------------------------------------
#pragma unroll 1
    for (int mt = 0; mt < VB / 16; ++mt) {
      float acc[2][4];
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) acc[nt][0] = acc[nt][1] = acc[nt][2] = acc[nt][3] = 0.f;
      // A fragments (rows g, g + 8; the lane's four coordinates of a step are adjacent)
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t ah[4], al[4];
        const int r0 = 16 * mt + g, d = 16 * ks + 4 * t;
        const uint2 h0 = *reinterpret_cast<const uint2 *>(&s.hi[r0][d]), h1 = *reinterpret_cast<const uint2 *>(&s.hi[r0 + 8][d]);
        const uint2 l0 = *reinterpret_cast<const uint2 *>(&s.lo[r0][d]), l1 = *reinterpret_cast<const uint2 *>(&s.lo[r0 + 8][d]);
        ah[0] = h0.x; ah[1] = h1.x; ah[2] = h0.y; ah[3] = h1.y;
        al[0] = l0.x; al[1] = l1.x; al[2] = l0.y; al[3] = l1.y;
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          mma16816_free(acc[nt], al[0], al[1], al[2], al[3], bh[nt][ks][0], bh[nt][ks][1]);
          mma16816_free(acc[nt], ah[0], ah[1], ah[2], ah[3], bl[nt][ks][0], bl[nt][ks][1]);
          mma16816_free(acc[nt], ah[0], ah[1], ah[2], ah[3], bh[nt][ks][0], bh[nt][ks][1]);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int v = 16 * mt + g + 8 * h, c = 16 * warp + 8 * nt + 2 * t;
          uint16_t pair = 0;
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float y = acc[nt][2 * h + e] * kUnscale;
            const int k = bucket(s.bounds, nbounds, y);
            if (!(y - s.bounds[k] > kMargin) || !(s.bounds[k + 1] - y > kMargin)) {
              if (v0 + v < vectors) s.near[atomicAdd(&s.near_count, 1)] = (uint16_t)(v * 128 + c + e);
            }
            pair |= (uint16_t)(k << (8 * e));
          }
          *reinterpret_cast<uint16_t *>(&s.idx[v][c]) = pair;
        }
    }
    __syncthreads();
    // ---- the chains of the coordinates near a boundary -----------------------------------
    const int near = s.near_count;
#pragma unroll 1
    for (int e = tid; e < near; e += kThreads) {
      const int v = s.near[e] >> 7, c = s.near[e] & 127;
      const float4 *row = reinterpret_cast<const float4 *>(a.q.Pi + c * 128);
      const float4 *x = reinterpret_cast<const float4 *>(&s.x[v][0]);
      float acc = 0.f;
#pragma unroll 8
      for (int d = 0; d < 32; ++d) {
        const float4 w = __ldg(row + d), z = x[d];
        acc = __fmaf_rn(z.x, w.x, acc);
        acc = __fmaf_rn(z.y, w.y, acc);
        acc = __fmaf_rn(z.z, w.z, acc);
        acc = __fmaf_rn(z.w, w.w, acc);
      }
      s.idx[v][c] = (uint8_t)bucket(s.bounds, nbounds, acc);
    }
    __syncthreads();
    if (tid == 0) s.near_count = 0;
    // ---- pack and store: a thread packs eight codes -----------------------------------------
    for (int e = tid; e < VB * 16; e += kThreads) {
      const int v = e >> 4, i = e & 15;
      const int64_t vec = v0 + v;
      if (vec >= vectors) break;
      const uint2 codes = *reinterpret_cast<const uint2 *>(&s.idx[v][8 * i]);
      if (APPEND) {
        if (s.code_off[v] >= 0) store_codes(a.pages + s.code_off[v], i, codes, bw, a.vec_dst);
      } else {
        if (a.idx) {
          if (a.vec_dst) *reinterpret_cast<uint2 *>(a.idx + vec * 128 + 8 * i) = codes;
          else
            for (int j = 0; j < 8; ++j) a.idx[vec * 128 + 8 * i + j] = s.idx[v][8 * i + j];
        }
        if (a.pages) store_codes(a.pages + vec * a.q.nb, i, codes, bw, a.vec_dst);
      }
    }
    if (tid < VB && v0 + tid < vectors) {
      if (APPEND) {
        if (s.code_off[tid] >= 0) a.norms[s.norm_off[tid]] = __float2half_rn(s.norm[tid]);
      } else if (a.norms32) {
        a.norms32[v0 + tid] = s.norm[tid];
      }
    }
    __syncthreads();                                   // the tiles are reused by the next pass
  }
}

template <int VB, bool APPEND>
int launch(const QuantJob &job, int sides, int blocks, cudaStream_t stream, const char *what) {
  auto kernel = quant_mma_kernel<VB, APPEND>;
  const int bytes = (int)sizeof(Smem<VB>);
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
  if (D != 128 || order != WTQ_ORDER_SEQUENTIAL) return false;
  for (int i = 0; i < sides; ++i)
    if (((uintptr_t)job.side[i].q.Pi & 15) != 0) return false;
  return true;
}

// Sixteen vectors per block while that leaves at most two blocks per multiprocessor
// (a decode step's append: latency counts), 64 above (bulk fills: the chains of a
// pass are one round for the block, whatever their number).
int launch_quant_mma(const QuantJob &job, bool append, int sides, cudaStream_t stream, const char *what) {
  const int64_t slots = 2 * (int64_t)device_sms() / sides;
  const int64_t small = (job.vectors + 15) / 16;
  if (small <= slots)
    return append ? qm::launch<16, true>(job, sides, (int)small, stream, what)
                  : qm::launch<16, false>(job, sides, (int)small, stream, what);
  const int blocks = (int)std::min<int64_t>((job.vectors + 63) / 64, slots);
  return append ? qm::launch<64, true>(job, sides, blocks, stream, what)
                : qm::launch<64, false>(job, sides, blocks, stream, what);
}

}  // namespace wtq
