// The 32-bit count at which thread blocks meet (host and device).
#pragma once

#ifdef __CUDACC__
#define TF_COUNT_FN __host__ __device__ __forceinline__
#else
#define TF_COUNT_FN inline
#endif

namespace tf {

// Whether a count that only grows has come to `goal`.  Both wrap, so what counts
// is their difference: less than 2^31 either way while blocks wait.
TF_COUNT_FN bool count_reached(unsigned seen, unsigned goal) { return static_cast<int>(seen - goal) >= 0; }

}  // namespace tf
