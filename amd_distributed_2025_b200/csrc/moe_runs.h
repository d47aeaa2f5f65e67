// How the one-rank MoE dispatch deals its items (a token's row in pieces: tokens x pieces of them, in order) out to the
// CTAs.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define B200_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define B200_HOST_DEVICE inline
#endif

namespace b200 {

// CTA b's run is [start(b), start(b + 1)): equal shares, and with a `slope` longer ones for the first CTAs than for the
// last.  Whole numbers throughout: the end of a run and the start of the next one are worked out by different CTAs, and
// must be the same number whatever the compiler makes of the expression; the longest run is known to the unit, because the
// CTAs' shared memory is cut to it.
struct MoeRuns {
  int32_t ctas, mean, rest;  // items = mean * ctas + rest
  int32_t slope;             // 2^20 times what the first of very many runs gains, over `ctas`

  // (Made anew by every CTA: a launch costs the host 0.3 us more with 168 bytes of parameters than with 152.)
  B200_HOST_DEVICE MoeRuns(int32_t items, int32_t n, int32_t s) : ctas(n), mean(items / n), rest(items % n), slope(s) {}
  B200_HOST_DEVICE int32_t start(int32_t b) const {
    return b * mean + (b < rest ? b : rest) + (int32_t)(((int64_t)slope * b * (ctas - b)) >> 20);
  }
  B200_HOST_DEVICE int32_t longest() const { return mean + 2 + (int32_t)(((int64_t)slope * (ctas - 1)) >> 20); }
};

// The slope at which the first run gains the fraction `lean` (up to a half) of the mean, and the last one loses it.  None
// for runs of fewer than four items, the last of which could end before it starts.
inline int32_t moe_run_slope(int32_t items, int32_t ctas, double lean) {
  const int32_t mean = items / ctas;
  const double slope = mean < 4 ? 0.0 : lean * 1048576.0 * mean / ctas;
  return slope < 2147483647.0 ? (int32_t)slope : 2147483647;  // (less of a lean beyond 2^27 items)
}

// Entries of the tokens that a run of `longest` items may touch: the first and the last token may be shared with neighbours.
inline int64_t moe_run_entries(int64_t longest, int64_t pieces, int64_t topk) {
  return ((longest + pieces - 2) / pieces + 1) * topk;
}

}  // namespace b200
