// tracks.cuh -- track blocks: the direct sums with most exponentials replaced
// by interpolation along smooth runs of samples (tracks.cu).
#pragma once

#include "visibility.cuh"

namespace viss {

// What the plan has staged; all pointers are device memory.
struct TrackInputs {
  const double4 *pix;      // [Jpad] sorted pixel records
  const float4 *cones;     // cone_count layout
  const int *perm;         // [J] caller's pixel of a record
  long long J, Jpad;
  int ntiles;
  const double4 *samp;     // [K] caller's order, channel-major
  const int4 *refs;        // [K] or null
  const double4 *occ;
  const float4 *occ32;
  long long K, Kc;
  int channels;
  int nsm;
  double max_turns;        // bound on |u.s + off|
};

// Builds the track blocks of the staged samples into *state (allocated on
// first use, buffers kept).  *usable = false when the samples are not smooth
// enough to gain, or memory is short; the direct kernels take the call then.
// Waits for `st` a few times; must not run under stream capture.
int tracks_build(void **state, const TrackInputs &in, cudaStream_t st, bool *usable);
void tracks_free(void *state);

// Modelled time of one call with the built blocks, in seconds (an occulted call
// also evaluates the pairs at the rims): 3.2e-14 s per (sample, pixel) and
// modelled issue slot, and 7e-14 s per occulted pair, from the adjoint at Nside 256 x
// 388,800 samples, 1 and 10 MHz (20.8 / 41.5 ms and 54.8 / 66.8 ms).
double tracks_seconds(const void *state, const TrackInputs &in, bool masked);

// V (channel-major, caller's order) and images of the built blocks.  pixsky:
// the staged pixel + sky records of every channel; coef: the caller's
// coefficients.  masked selects the occulted or the unmasked pair bits.
int tracks_forward(void *state, const TrackInputs &in, const double4 *pixsky, float2 *V, bool masked,
                   bool use_off, bool accumulate, unsigned long long *counter, int *err, int drop_tile,
                   cudaStream_t st);
int tracks_adjoint(void *state, const TrackInputs &in, const float2 *coef, float *image, float scale,
                   bool masked, bool use_off, bool accumulate, unsigned long long *counter, int *err,
                   int drop_tile, cudaStream_t st);

}  // namespace viss
