// Parameter blocks of the quantisation kernels (wtq_append.cu, wtq_quant_mma.cu).
#pragma once

#include "wtq_common.cuh"

namespace wtq {

struct QuantSideDev {
  const float *Pi;
  const float *bounds;
  int bw, nb, nbounds;
  bool vec4;      // Pi is 16-byte aligned and D a multiple of 4: rows can be read as float4
};

// One side of a call of the tensor-core kernel: K or V of an append, or the rows
// of wtq_quantize.
struct QuantJobSide {
  QuantSideDev q;
  const void *src;
  int64_t sb, sh, st;         // element strides: batch, head, token (quantize: st = row stride)
  bool vec_src, vec_dst;      // rows can be read / written in words of four or eight elements
  uint8_t *pages;             // append: the pages; quantize: packed rows or null
  __half *norms;              // append
  int64_t page_stride, head_stride, norm_page_stride, norm_head_stride;
  uint8_t *idx;               // quantize: unpacked codes or null
  float *norms32;             // quantize
};

struct QuantJob {
  QuantJobSide side[2];
  int64_t vectors;
  int dtype;
  const int32_t *page_table;
  int64_t table_stride;
  const int32_t *seq_lens;
  int Hkv, n, S, P, max_pages;
  int32_t *status;
  int team_shift;             // set by launch_quant_mma
};

bool quant_mma_eligible(int D, int order, const QuantJob &job, int sides);
int launch_quant_mma(QuantJob job, bool append, int sides, cudaStream_t stream, const char *what);

}  // namespace wtq
