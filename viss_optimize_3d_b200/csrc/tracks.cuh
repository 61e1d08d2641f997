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

// Modelled time of one call with the built blocks, in seconds: per (sample, pixel)
// and modelled issue slot 3.1e-14 (forward) or 3.3e-14 s (adjoint), and in an
// occulted call 0.85 of that, for what is hidden, plus the pairs at the rims, whose
// share goes with the width of a tile: 4.3e-11 or 5.5e-11 / sqrt(J).  Within 10 %
// of nine calls of 1e10 to 3e11 terms at Nside 128 and 256, 1 to 10 MHz, occulted
// and not (9.6e-14 to 3.4e-13 s per term).
double tracks_seconds(const void *state, const TrackInputs &in, bool masked, bool adjoint);

// drop_tile from here on: the interpolation's first product instead of a tile's copy.
constexpr int kDropProduct = 1 << 30;

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
