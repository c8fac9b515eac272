// A ring of R stages that bulk copies fill in turn: where the i-th copy goes, which phase of the stage's
// barrier it completes, and which copies may still be in flight when `issued` have been issued.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define NOMAD_RING_FN __host__ __device__ constexpr
#else
#define NOMAD_RING_FN constexpr
#endif

template <int R>
struct BulkRing {
  static NOMAD_RING_FN int stage(int i) { return i % R; }
  static NOMAD_RING_FN uint32_t parity(int i) { return (uint32_t)(i / R) & 1u; }
  static NOMAD_RING_FN int first_open(int issued) { return issued > R ? issued - R : 0; }
};
