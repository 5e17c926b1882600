// Parameter block and launchers shared by the dequantisation kernels.
#pragma once

#include "wtq_common.cuh"

namespace wtq {

struct DequantParams {
  const uint8_t *packed;
  const __half *norms;
  const float *centroids, *Pi;
  void *out;
  int out_dtype, bw, D, nb;
  int64_t N, L, MAXLEN;
  // a second tensor of the same shape, widths and quantizer (tcgen05 kernel only)
  int tensors = 1;
  const uint8_t *packed_b = nullptr;
  const __half *norms_b = nullptr;
  void *out_b = nullptr;
  int wait_tries = 0;           // set by launch_dequant_umma
};

// tcgen05 kernel (wtq_dequant_umma.cu); `terms` = 1 or 3.  *usable = false and
// nothing launched when the kernel cannot serve this call here.
int launch_dequant_umma(const DequantParams &p, int terms, cudaStream_t stream, bool *usable);
// Whether a wait ran out in it on the current device since this was last asked.
bool dequant_umma_gave_up();
// Polls a wait of the calls of this thread makes before it gives up; negative: the default.
void dequant_umma_wait_tries(int tries);

}  // namespace wtq
