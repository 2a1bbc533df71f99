// Transforms along an axis whose length has one prime factor p from 37 to 251:
// n = q p (q <= 13, tiles of up to 256 threads: n to about 510), as q-point butterflies and a direct p-point DFT that is a
// small matrix product in shared memory (prime_pass.cu).
#pragma once

#include <cuda_runtime.h>

#include "cbs_kernels.cuh"

namespace odt {

struct PrimePlan {
  int n = 0, q = 0, p = 0;       // n = q p; q == 0: no plan
  int h = 0, kp = 0;             // h = (p - 1) / 2; table pitch, 8 ceil((h + 1) / 8)
  int w = 0;                     // pencils per tile
  const float2* tw = nullptr;    // [n] exp(-2 pi i k / n), device
  // [2][h][kp] cos, sin (2 pi j k / p), j = 1 .. h, k = 0 .. h, and one more
  // row that is read ahead but not used; device
  const float* tab = nullptr;
};

// Host part of a plan (no device pointers); q == 0 where the kernel does not
// apply (no such factorisation, or a tile of 16 pencils exceeds the threads or
// max_smem).
PrimePlan prime_plan(int n, size_t max_smem);
// Host tables of a plan: [2][h][kp] and a row of zeros.
inline size_t prime_table_size(const PrimePlan& p) { return (2 * (size_t)p.h + 1) * p.kp; }
void prime_table(const PrimePlan& p, float* tab);

// DFT along the middle axis of x [n0, n, n2] in place (n0 == 1: contiguous
// lines), index shift sh on input and output, result times scale.
cudaError_t launch_prime_axis(float2* x, int n0, long long n2, bool inv, int sh, float scale, const PrimePlan& f,
                              cudaStream_t s);
// z-pass of iteration jj: forward z-FFT, Green's multiply, inverse z-FFT of a.T.
cudaError_t launch_prime_z(const BornArgs& a, int jj, const PrimePlan& f, cudaStream_t s);

}  // namespace odt
