// Fourier filter of small 3-D arrays in shared memory (fftfilter.cu).
#pragma once

#include <cuda_runtime.h>

namespace tmb {

// Whether items of shape n[3] take this path: even n[0]; n[0] / 2, n[1] and n[2] products of
// two factors of at most 16; 220 KiB of shared memory, 140 for fewer than 64 items.
bool fft_filter_supported(const int* n, int batch);
// x = irfftn(rfftn(x) * filter) in place for `batch` items.
int fft_filter(float* x, const float* filter, const int* n, int batch, cudaStream_t stream);

}  // namespace tmb
