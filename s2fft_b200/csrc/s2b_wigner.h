// Wigner (SO(3)) stage launchers (wigner.cu).
#pragma once

#include <cuda_runtime.h>

namespace s2b {

// slices n = n0 .. n0 + K - 1, slice k at tmp + k stride (complex elements); real0: slice n = 0
// is that of a real signal (orders weighted 0 / 1 / 2 for m < 0 / = 0 / > 0)
cudaError_t launch_gather_slices(bool fp64, const void* flmn, void* tmp, long stride, int B, int N,
                                 int L, int n0, int K, int real0, cudaStream_t s);
cudaError_t launch_scatter_slices(bool fp64, const void* tmp, long stride, void* flmn, int B, int N,
                                  int L, int n0, int K, int L0, cudaStream_t s);
cudaError_t launch_wigner_mirror(bool fp64, void* flmn, int B, int N, int L, cudaStream_t s);
cudaError_t launch_gamma_inverse(bool fp64, const void* fban, void* f, int B, int N, long npix,
                                 int reality, cudaStream_t s);
cudaError_t launch_gamma_forward(bool fp64, const void* f, void* fban, int B, int N, long npix,
                                 int reality, cudaStream_t s);

}  // namespace s2b
