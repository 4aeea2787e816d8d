// Position in a ring of pipeline stages, each with an mbarrier whose phases alternate.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define CHORD_RING_FN __host__ __device__ __forceinline__
#else
#define CHORD_RING_FN inline
#endif

namespace chord {

// Ring position advanced without divisions (a lone issuing thread pays ~100
// cycles for an integer division).
struct StageCursor {
  uint32_t s = 0, ph = 0;
  CHORD_RING_FN void advance(uint32_t stages) {
    if (++s == stages) {
      s = 0;
      ph ^= 1u;
    }
  }
  // Any distance, without a division (a few subtractions per tile at most).
  CHORD_RING_FN void advance_by(uint32_t n, uint32_t stages) {
    s += n;
    while (s >= stages) {
      s -= stages;
      ph ^= 1u;
    }
  }
  // Parity of the phase that the latest use of stage `i` before this position completes.  A stage
  // without a use yet: 1, for which a wait on a fresh barrier returns at once.
  CHORD_RING_FN uint32_t last_phase(uint32_t i) const { return i < s ? ph : ph ^ 1u; }
};

}  // namespace chord
