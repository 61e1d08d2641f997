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
  long long pix_version;   // another one for newly staged pixels
  void *work;              // a call's sums go there if they fit
  size_t work_bytes;
};

// Looks at a few blocks of the staged samples (*state: allocated on first use,
// buffers kept).  *promising = false when the samples are not smooth enough for
// nodes to pay, or memory is short; the direct kernels take the calls then.  Waits
// for `st` a few times; must not run under stream capture.
int tracks_try(void **state, const TrackInputs &in, cudaStream_t st, bool *promising);
// Builds the blocks of the samples that tracks_try found promising; likewise.
int tracks_build(void *state, const TrackInputs &in, cudaStream_t st, bool *usable);
void tracks_free(void *state);

// Modelled time of one call through the blocks, in seconds, from what tracks_try
// counted in its blocks.  Fitted to 200 observations of 1e10 to 7e11 terms (Nside 48
// to 512, 500 to 8,640 snapshots, 4 to 10 satellites, 0.3 to 10 MHz), each occulted and
// not: where the blocks take more than .6 of the direct kernels' time, 17 % below to 36 %
// above what was measured (forward), 17 % below to 28 % above (adjoint).
double tracks_seconds(const void *state, const TrackInputs &in, bool masked, bool adjoint);
// Shares of the (sample, tile) pairs that an occulted call sees, and sees in part.
void tracks_shares(const void *state, double *seen, double *mixed);

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
