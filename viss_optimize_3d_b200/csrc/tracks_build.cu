// tracks_build.cu -- the track blocks of newly staged samples: which samples form
// a block, its nodes and weights, and its pair bits (tracks.cu has the method).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <new>

#include "tracks_impl.cuh"

namespace viss {

namespace {

constexpr double kNodeNoise2 = 4e-14;            // kNodeNoise^2
constexpr int kLagMax = 1024;                    // tracks interleaved in the caller's order, at most
constexpr int kLagSamples = 128;
constexpr int kBuckets = kTrackRankMax / 16 + 1; // blocks of similar rank are stored together
constexpr int kRankSamples = 48;                 // blocks that decide whether nodes pay
// Node sums of one slab of blocks: large enough that a slab's kernels fill the
// device several times over.
constexpr size_t kSlabBytes = 1ull << 28;

// Pixel groups of gp pixels: centre (normalised mean direction) and the largest
// chord from it to a pixel, rounded up; +inf with a pixel that is NaN or longer
// than 2 (its phases could reach 2^19 turns: tracks_build bounds those of unit
// vectors by 2^18).
__global__ void k_track_groups(int ng, int gp, long long Jpad, const double4 *pix, double4 *gcen, float *radius) {
  const int g = static_cast<int>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32, lane = threadIdx.x & 31;
  if (g >= ng) return;
  const long long p0 = static_cast<long long>(g) * gp, p1 = min(p0 + gp, Jpad);
  double x = 0, y = 0, z = 0;
  for (long long i = p0 + lane; i < p1; i += 32) {
    const double4 p = pix[i];
    x += p.x; y += p.y; z += p.z;
  }
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
    z += __shfl_xor_sync(0xffffffffu, z, o);
  }
  const double n = sqrt(x * x + y * y + z * z);
  double4 c = make_double4(1.0, 0.0, 0.0, 0.0);
  if (n > 1e-6) c = make_double4(x / n, y / n, z / n, 0.0);
  double r = 0;
  bool bad = !(n == n);
  for (long long i = p0 + lane; i < p1; i += 32) {
    const double4 p = pix[i];
    const double dx = p.x - c.x, dy = p.y - c.y, dz = p.z - c.z;
    const double d = sqrt(dx * dx + dy * dy + dz * dz);
    bad = bad || !(d == d) || !(p.x * p.x + p.y * p.y + p.z * p.z <= 4.0);
    r = fmax(r, d);
  }
  for (int o = 16; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(0xffffffffu, r, o));
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) {
    gcen[g] = c;
    radius[g] = bad ? __int_as_float(0x7f800000) : __double2float_ru(r);
  }
}

// score[B - 1]: how far apart, in phase turns across a group, samples k and
// k + B of one channel are on average, capped at 4; the same kLagSamples spread
// samples k for every lag B, so that the lags compare.
__global__ void k_track_lags(long long Kc, int channels, const double4 *samp, double rho, float *score) {
  const long long B = blockIdx.x + 1;
  const int t = threadIdx.x;
  const long long span = Kc - gridDim.x;           // k + B < Kc for the largest lag
  double v = 4.0;
  if (span > 0) {
    const long long at = (span - 1) * t / (kLagSamples - 1);
    const long long k = static_cast<long long>(t * 7 % channels) * Kc + at;
    const double4 a = samp[k], b = samp[k + B];
    const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    v = fmin(2.0 * rho * sqrt(dx * dx + dy * dy + dz * dz), 4.0);
    if (!(v == v)) v = 4.0;
  }
  __shared__ double red[kLagSamples / 32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((t & 31) == 0) red[t / 32] = v;
  __syncthreads();
  if (t == 0) {
    double s = 0;
    for (int w = 0; w < kLagSamples / 32; ++w) s += red[w];
    score[blockIdx.x] = static_cast<float>(s / kLagSamples);
  }
}

// Sample i of natural block b, -1 for none.
__device__ __forceinline__ long long block_sample(const TrackShape &s, int b, int i) {
  const int nbc = s.blocks_per_channel();
  const int ch = b / nbc, in = b - ch * nbc, tb = in / s.lag, track = in - tb * s.lag;
  const long long k = (static_cast<long long>(tb) * s.len + i) * s.lag + track;
  return (i < s.len && k < s.Kc) ? ch * s.Kc + k : -1;
}

// Slots of the stored blocks: block b is natural block order[b].
__global__ void k_track_slots(TrackShape s, long long Ks, const int *order, const double4 *samp, const int4 *refs,
                              int *slot, double4 *samp_s, int4 *refs_s) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= Ks) return;
  const long long k = block_sample(s, order[i / kTrackT], static_cast<int>(i % kTrackT));
  slot[i] = static_cast<int>(k);
  samp_s[i] = k >= 0 ? samp[k] : make_double4(0, 0, 0, 0);
  if (refs) refs_s[i] = k >= 0 ? refs[k] : make_int4(-1, -1, -1, -1);
}

// Pivoted Cholesky factorisation of a block's correlation matrix (file
// comment): thread = sample; column j of the factor at L[j * kTrackT + k].
// Returns the rank (0: not worth it), the pivots in piv and the pivots'
// diagonal entries in ld.
// RM: ranks up to it; 48 leave room for twice the CTAs per SM.
template <int RM>
struct TrackFactor {
  double L[RM * kTrackT];
  double u[3][kTrackT];
  double ld[RM], diag[kTrackT];
  unsigned long long best[kTrackT / 32];
  double sum[kTrackT / 32], top[kTrackT / 32];
  unsigned char piv[RM];
};
constexpr int kSmallRank = kTrackRankMax / 2;

template <int RM>
__device__ int track_factor(TrackFactor<RM> &f, bool valid, const double4 &u, double rho, int rank_max) {
  const int k = threadIdx.x, lane = k & 31, w = k >> 5;
  f.u[0][k] = u.x;
  f.u[1][k] = u.y;
  f.u[2][k] = u.z;
  double diag = valid ? 1.0 : 0.0;
  bool used = !valid;
  const int nvalid = __syncthreads_count(valid);
  const int cap = min(rank_max, nvalid * 3 / 4);
  for (int r = 0;; ++r) {
    // the worst predicted unused sample (its low bits carry the index), and how well all are
    unsigned long long key = used ? 0ull : (static_cast<unsigned long long>(__double_as_longlong(diag)) & ~127ull) | k;
    double sum = diag, top = diag;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      key = max(key, __shfl_xor_sync(0xffffffffu, key, o));
      sum += __shfl_xor_sync(0xffffffffu, sum, o);
      top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    f.diag[k] = diag;
    if (lane == 0) f.best[w] = key, f.sum[w] = sum, f.top[w] = top;
    __syncthreads();
    key = max(max(f.best[0], f.best[1]), max(f.best[2], f.best[3]));
    sum = (f.sum[0] + f.sum[1]) + (f.sum[2] + f.sum[3]);
    top = fmax(fmax(f.top[0], f.top[1]), fmax(f.top[2], f.top[3]));
    if (top <= 4.5 * kNodeNoise2 && sum <= 1.8 * kNodeNoise2 * nvalid) return r;
    if (r >= cap || key == 0) return 0;
    const int p = static_cast<int>(key & 127u);
    const double dx = u.x - f.u[0][p], dy = u.y - f.u[1][p], dz = u.z - f.u[2][p];
    const double x = 2.0 * rho * sqrt(dx * dx + dy * dy + dz * dz);     // half-turns of the sinc's argument
    double c = x > 1e-9 ? sinpi(x) / (3.14159265358979323846 * x) : 1.0;
    for (int j = 0; j < r; ++j) c = fma(-f.L[j * kTrackT + k], f.L[j * kTrackT + p], c);
    const double d = f.diag[p];                    // the pivot's own residual
    const double ld = sqrt(d + kNodeNoise2);
    const double l = valid ? c / ld : 0.0;
    f.L[r * kTrackT + k] = l;
    if (r == 0 && __syncthreads_and(!valid || x <= 1e-9)) {
      // one point (zero baselines): one node, whose weights are one exactly
      if (k == p) f.piv[0] = static_cast<unsigned char>(p), f.ld[0] = ld;
      __syncthreads();
      return 1;
    }
    diag = fmax(fma(-l, l, diag), 0.0);
    if (k == p) {
      used = true;
      f.piv[r] = static_cast<unsigned char>(p);
      f.ld[r] = ld;
    }
    __syncthreads();
  }
}

// Ranks of natural blocks (which: of all, if null) for group radius rho[blockIdx.y]
// and at most most[blockIdx.y] nodes, as rank[blockIdx.y][block] (0: more).
template <int RM>
__global__ void __launch_bounds__(kTrackT) k_track_ranks(TrackShape s, const int *which, const double4 *samp,
                                                         RadiusSet radii, int *rank) {
  extern __shared__ __align__(128) unsigned char smem[];
  TrackFactor<RM> &f = *reinterpret_cast<TrackFactor<RM> *>(smem);
  const int b = which ? which[blockIdx.x] : static_cast<int>(blockIdx.x);
  const long long k = block_sample(s, b, threadIdx.x);
  const double4 u = k >= 0 ? samp[k] : make_double4(0, 0, 0, 0);
  const int r = track_factor(f, k >= 0, u, radii.rho[blockIdx.y], radii.most[blockIdx.y]);
  if (threadIdx.x == 0) rank[blockIdx.y * gridDim.x + blockIdx.x] = r;
}

// Nodes and weights of every block: node n of block b is record noff[b] + n,
// its weights for the block's 128 slots P[(noff[b] + n) * 128 + k].  The factorisation
// is k_track_ranks's; should it ever end at another rank, *differ says so and the
// blocks are not used.  Blocks of ranks in (above, RM].
template <int RM>
__global__ void __launch_bounds__(kTrackT) k_track_weights(int above, const int *slot, const double4 *samp_s, RadiusSet radii,
                                                           const int *cls, const int *rank, const int *noff, double4 *node,
                                                           int *nodeblk, float *P, unsigned long long *differ) {
  extern __shared__ __align__(128) unsigned char smem[];
  TrackFactor<RM> &f = *reinterpret_cast<TrackFactor<RM> *>(smem);
  const int b = blockIdx.x, k = threadIdx.x;
  if (rank[b] <= above || rank[b] > RM) return;
  const long long i = static_cast<long long>(b) * kTrackT + k;
  const double4 u = samp_s[i];
  const bool valid = slot[i] >= 0;
  const int r = track_factor(f, valid, u, radii.rho[cls[b]], min(radii.most[cls[b]], RM));
  if (r != rank[b]) {
    if (k == 0) atomicOr(differ, 1ull);
    return;
  }
  const long long n0 = noff[b];
  if (k < r) {
    const int p = f.piv[k];
    node[n0 + k] = make_double4(f.u[0][p], f.u[1][p], f.u[2][p], 0.0);
    nodeblk[n0 + k] = b;
  }
  // x L11 = l_k from the last column back, L11[j][q] = L[q][piv j] (q < j), ld[j] on
  // the diagonal.  The pivots' rows are read by all, so x goes to registers first.
  double x[RM];
#pragma unroll 1
  for (int j = r - 1; j >= 0; --j) {
    double v = f.L[j * kTrackT + k];
    for (int q = j + 1; q < r; ++q) v = fma(-x[q], f.L[j * kTrackT + f.piv[q]], v);
    x[j] = v / f.ld[j];
  }
  for (int j = 0; j < r; ++j) P[(n0 + j) * kTrackT + k] = valid ? static_cast<float>(x[j]) : 0.f;
}

// A tile is merged with the others of its group of class c (2 or 3) when all
// of them are in `full`.
__device__ __forceinline__ unsigned merged_tiles(unsigned full, unsigned valid, int c) {
  if (c == 2) {
    const unsigned g = full & (full >> 1) & 0x55555555u;
    return g | (g << 1);
  }
  if (c == 3) {
    unsigned g = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const unsigned b = 0xffu << (8 * q);
      if ((full & b) == (valid & b)) g |= valid & b;
    }
    return g;
  }
  return 0;
}

__device__ __forceinline__ unsigned valid_tiles(int w, int ntiles) {
  const int left = ntiles - 32 * w;
  return left >= 32 ? 0xffffffffu : (left > 0 ? (1u << left) - 1u : 0u);
}

// Rows of class c (kClasses: blocks without nodes) for unocculted sums: the
// tiles whose group is within the class's radius (radius: per class, its
// groups', concatenated from at[c]), merged tiles, and the others.  left: bit c
// set where class c leaves a tile.
__global__ void k_track_class_rows(int W, int ntiles, const float *radius, ClassSet cs, unsigned *full,
                                   unsigned *merged, unsigned *rest, unsigned long long *left) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
  if (w >= W) return;
  const unsigned valid = valid_tiles(w, ntiles);
  unsigned ok = 0;
  if (c < kClasses) {
    const float rho = static_cast<float>(cs.rho[c]);
    for (int i = 0; i < 32; ++i) {
      const int t = 32 * w + i;
      if (t >= ntiles) break;
      const float *r = radius + cs.at[c];
      bool in;
      if (c == kHalf) in = r[2 * t] <= rho && r[2 * t + 1] <= rho;
      else in = r[t * kTilePix / group_pix(c)] <= rho && radius[cs.at[kTile] + t] <= rho;   // a tile may stand alone
      ok |= static_cast<unsigned>(in) << i;
    }
  }
  full[c * W + w] = ok;
  merged[c * W + w] = merged_tiles(ok, valid, c);
  rest[c * W + w] = valid & ~ok;
  if (valid & ~ok) atomicOr(left, 1ull << c);
}

// A sample's three classification rows (absent: sees everything), and its
// state on a cone: 2 sees all of it, 0 none, 1 part.
struct SampleRows {
  float4 r[3];
  bool has[3];
};
__device__ __forceinline__ SampleRows sample_rows(const int4 &rf, const float4 *occ32) {
  SampleRows s;
  s.has[0] = rf.x >= 0;
  s.has[1] = rf.y >= 0;
  s.has[2] = rf.z >= 0;
  const float4 pass = make_float4(0.f, 0.f, 0.f, -4.f);
  s.r[0] = s.has[0] ? occ32[rf.x] : pass;
  s.r[1] = s.has[1] ? occ32[rf.y] : pass;
  s.r[2] = s.has[2] ? occ32[rf.z] : pass;
  return s;
}
__device__ __forceinline__ int cone_rows_state(const float4 &cone, const SampleRows &s) {
  int st = 2;
#pragma unroll
  for (int c = 0; c < 3; ++c)
    if (s.has[c]) st = min(st, cone_state32(cone, s.r[c]));
  return st;
}

// Occulted pair bits, one warp per block and 32-tile word, of the tiles of the
// class rows: full (every sample of the block sees the tile), part (not all,
// but some do), merged, and rest (a sample needs the remainder kernel: on a
// tile with nodes one that sees part of it, elsewhere one that sees any of it).
// count: rest pairs, part pairs.
__global__ void k_track_bits(int W, int ntiles, const int *slot, const int4 *refs, const float4 *occ32,
                             const float4 *cones, const int *cls, const unsigned *crow, unsigned *full_out,
                             unsigned *part_out, unsigned *merged_out, unsigned *rest_out,
                             unsigned long long *count) {
  const int b = static_cast<int>(blockIdx.x), lane = threadIdx.x & 31;
  const int warps = blockDim.x / 32 * gridDim.y, w0 = blockIdx.y * (blockDim.x / 32) + threadIdx.x / 32;
  SampleRows rows[4];
  bool val[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const long long i = static_cast<long long>(b) * kTrackT + 32 * s + lane;
    val[s] = slot[i] >= 0;
    rows[s] = sample_rows(val[s] ? refs[i] : make_int4(-1, -1, -1, -1), occ32);
  }
  // bit 0: some sample is hidden, 1: some sees part, 2: some sees all
  auto states = [&](const float4 &cone) {
    unsigned m = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (val[s]) m |= 1u << cone_rows_state(cone, rows[s]);
    return __reduce_or_sync(0xffffffffu, m);
  };
  const int c = cls[b];
  unsigned long long nrest = 0, npart = 0;
  for (int w = w0; w < W; w += warps) {
    unsigned all = 0, any = 0, mix = 0;
    const unsigned valid = valid_tiles(w, ntiles);
    for (int q = 0; q < 32 / kSuperTiles; ++q) {
      const int t0 = 32 * w + q * kSuperTiles;
      if (t0 >= ntiles) break;
      unsigned m = states(cones[5LL * ntiles + t0 / kSuperTiles]);
      unsigned a8 = m == 4u ? 0xffu : 0u, y8 = (m & 4u) ? 0xffu : 0u, x8 = 0;   // without bit 1 true of every tile
      if (m & 2u) {
        a8 = y8 = 0;
        for (int i = 0; i < kSuperTiles && t0 + i < ntiles; ++i) {
          const unsigned n = states(cones[t0 + i]);
          a8 |= static_cast<unsigned>(n == 4u) << i;
          y8 |= static_cast<unsigned>((n & 4u) != 0) << i;
          x8 |= static_cast<unsigned>((n & 2u) != 0) << i;
        }
      }
      all |= a8 << (q * kSuperTiles);
      any |= y8 << (q * kSuperTiles);
      mix |= x8 << (q * kSuperTiles);
    }
    const unsigned ok = crow[c * W + w];
    const unsigned full = all & ok & valid, part = any & ~all & ok & valid;
    const unsigned rest = valid & ((mix & ok) | ((mix | any) & ~ok));
    if (lane == 0) {
      const long long at = static_cast<long long>(b) * W + w;
      full_out[at] = full;
      part_out[at] = part;
      merged_out[at] = merged_tiles(full, valid, c);
      rest_out[at] = rest;
    }
    nrest += __popc(rest);
    npart += __popc(part);
  }
  if (lane == 0 && nrest) atomicAdd(count, nrest);
  if (lane == 0 && npart) atomicAdd(count + 1, npart);
}

// Sums over the blocks' tiles of a call's work (TrackEstimate's members in order;
// refs null: an unocculted call), as k_track_bits classifies them.
constexpr int kEstimates = 8;
__global__ void k_track_estimate(int W, int ntiles, const int *slot, const int4 *refs, const float4 *occ32,
                                 const float4 *cones, const int *cls, const int *rank, const unsigned *crow,
                                 unsigned long long *sums) {
  const int b = static_cast<int>(blockIdx.x), lane = threadIdx.x & 31;
  const int warps = blockDim.x / 32 * gridDim.y, w0 = blockIdx.y * (blockDim.x / 32) + threadIdx.x / 32;
  SampleRows rows[4];
  bool val[4];
  int nvalid = 0;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const long long i = static_cast<long long>(b) * kTrackT + 32 * s + lane;
    val[s] = slot[i] >= 0;
    rows[s] = sample_rows(val[s] && refs ? refs[i] : make_int4(-1, -1, -1, -1), occ32);
    nvalid += __popc(__ballot_sync(0xffffffffu, val[s]));
  }
  // samples that see part of a cone, and all of it
  auto count = [&](const float4 &cone, int &part, int &all) {
    part = all = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int st = val[s] ? cone_rows_state(cone, rows[s]) : 0;
      part += __popc(__ballot_sync(0xffffffffu, st == 1));
      all += __popc(__ballot_sync(0xffffffffu, st == 2));
    }
  };
  const int c = cls[b], r = rank[b];
  unsigned long long sum[kEstimates] = {};
  for (int w = w0; w < W; w += warps) {
    const unsigned ok = crow[c * W + w], valid = valid_tiles(w, ntiles);
    unsigned full = 0, taken = 0;
    for (int q = 0; q < 32 / kSuperTiles; ++q) {
      const int t0 = 32 * w + q * kSuperTiles;
      if (t0 >= ntiles) break;
      int part, all;
      count(cones[5LL * ntiles + t0 / kSuperTiles], part, all);
      const bool refine = part > 0;
      for (int i = 0; i < kSuperTiles && t0 + i < ntiles; ++i) {
        const int bit = q * kSuperTiles + i;
        if (refine) count(cones[t0 + i], part, all);
        const bool in = (ok >> bit) & 1u;
        const int rest = part + (in ? 0 : all);
        full |= static_cast<unsigned>(in && all == nvalid) << bit;
        taken |= static_cast<unsigned>(in && all > 0) << bit;
        sum[3] += rest > 0;
        sum[4] += rest;
        sum[5] += part + all;
        sum[6] += part;
      }
    }
    const unsigned first = c == 2 ? 0x55555555u : 0x01010101u;
    const unsigned units = __popc(taken & ~(merged_tiles(full, valid, c) & ~first)) * (c == kHalf ? 2 : 1);
    sum[0] += static_cast<unsigned long long>(__popc(taken)) * kTilePix * r;
    sum[1] += static_cast<unsigned long long>(units) * kTrackT;
    sum[2] += static_cast<unsigned long long>(units) * kTrackT * r;
    if (r > kOneCtaRank) sum[7] += static_cast<unsigned long long>(units) * kTrackT;
  }
  if (lane == 0)
    for (int i = 0; i < kEstimates; ++i)
      if (sum[i]) atomicAdd(sums + i, sum[i]);
}

// Sample masks of the part tiles: a word's masks stand together, in the order
// of its tiles, wherever `next` had room (mask_at).
__global__ void k_track_masks(int W, const int *slot, const int4 *refs, const float4 *occ32, const float4 *cones,
                              const unsigned *part, int *mask_at, uint4 *mask, unsigned long long *next) {
  const int b = static_cast<int>(blockIdx.x), lane = threadIdx.x & 31;
  const int warps = blockDim.x / 32 * gridDim.y, w0 = blockIdx.y * (blockDim.x / 32) + threadIdx.x / 32;
  SampleRows rows[4];
  bool val[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    const long long i = static_cast<long long>(b) * kTrackT + 32 * s + lane;
    val[s] = slot[i] >= 0;
    rows[s] = sample_rows(val[s] ? refs[i] : make_int4(-1, -1, -1, -1), occ32);
  }
  for (int w = w0; w < W; w += warps) {
    const long long word = static_cast<long long>(b) * W + w;
    unsigned m = part[word];
    if (m == 0) continue;
    int at = 0;
    if (lane == 0) at = static_cast<int>(atomicAdd(next, static_cast<unsigned long long>(__popc(m))));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (lane == 0) mask_at[word] = at;
    for (; m; m &= m - 1, ++at) {
      const float4 cone = cones[32 * w + __ffs(m) - 1];
      unsigned seen[4];
#pragma unroll
      for (int s = 0; s < 4; ++s)
        seen[s] = __ballot_sync(0xffffffffu, val[s] && cone_rows_state(cone, rows[s]) == 2);
      if (lane == 0) mask[at] = make_uint4(seen[0], seen[1], seen[2], seen[3]);
    }
  }
}

}  // namespace

void tracks_free(void *state) { delete static_cast<TrackState *>(state); }

namespace {

// Modelled time of a block's nodes and interpolation per (sample, pixel), in issue
// slots of a scheduler, by which classes are chosen: an evaluated exponential term
// takes 21, an interpolated (sample, unit) about r + 100 (both measured on the 1 and
// 10 MHz Nside 256 observations), and a term left to the remainder kernels 1.5 times
// that of k_forward / k_adjoint (one sample per lane, no shared staging).
constexpr double kTermSlots = 21.0, kLeftSlots = 1.5 * kTermSlots;
double block_slots(int c, int r, int len) {
  return r ? kTermSlots * r / len + (r + 100.0) / group_pix(c) : kLeftSlots;
}

}  // namespace

double tracks_seconds(const void *state, const TrackInputs &in, bool masked, bool adjoint) {
  const TrackState &S = *static_cast<const TrackState *>(state);
  const TrackEstimate &e = S.est[masked];
  if (!adjoint)                                    // few blocks: short slabs, whose last waves are mostly empty
    return (4.68e-13 * e.nodes + 2.45e-12 * e.units + 1.95e-11 * e.wide_units + 1.12e-8 * e.rest_blocks +
            1.44e-4 * S.slab_count) * (1.0 + 30.0 / S.nb);
  if (masked)
    return 2.23e-13 * e.nodes + 8.92e-12 * e.units + 5.4e-14 * e.unit_nodes + 1.85e-10 * e.rest_samples +
           1.5e-4 * S.slab_count + 1.66e-4;
  return 4.99e-13 * e.nodes + 3.95e-12 * e.units + 9.6e-14 * e.unit_nodes + 1.22e-10 * e.rest_samples +
         (S.leaves_tiles ? 5.8e-9 * static_cast<double>(in.K) : 0.0) + 3.2e-5 * S.slab_count + 1.23e-4;
}

void tracks_shares(const void *state, double *seen, double *mixed) {
  const TrackState &S = *static_cast<const TrackState *>(state);
  *seen = S.est[1].seen;
  *mixed = S.est[1].mixed;
}

namespace {

// Pixel groups of newly staged pixels: centres, radii and the radii to try, kept until
// pixels are staged again.  S.pix_version stays behind if memory is short.
int track_pixels(TrackState &S, const TrackInputs &in, cudaStream_t st) {
  if (S.pix_version == in.pix_version) return 0;
  S.pix_version = -1;
  int ngs[kClasses], total = 0;
  for (int c = 0; c < kClasses; ++c) {
    ngs[c] = static_cast<int>((in.Jpad + group_pix(c) - 1) / group_pix(c));
    S.gat[c] = total;
    total += ngs[c];
  }
  if (!S.pixels.reset(TrackArena::bytes<double4>(total) + TrackArena::bytes<float>(total))) return 0;
  S.pixels.take(S.gcen, total);
  S.pixels.take(S.radius, total);
  for (int c = 0; c < kClasses; ++c) {
    k_track_groups<<<blks(ngs[c], 8), 256, 0, st>>>(ngs[c], group_pix(c), in.Jpad, in.pix, S.gcen + S.gat[c],
                                                    S.radius + S.gat[c]);
    TRACK_CUDA(cudaGetLastError(), "groups");
  }
  std::vector<float> radius(total);
  TRACK_CUDA(cudaMemcpyAsync(radius.data(), S.radius, sizeof(float) * total, cudaMemcpyDeviceToHost, st), "radii");
  TRACK_CUDA(cudaStreamSynchronize(st), "groups");
  // A class's radius: a percentile of its groups' (wider groups are left) with
  // the least time over some blocks.  On a power-of-two HEALPix grid all groups
  // are alike and the largest wins; elsewhere a few are far wider than the rest.
  // A group of more than 64 pixels is only worth it with few nodes.  A share that
  // takes in a group that has none (radius +inf) is no radius: nothing within it.
  const double share[kShares] = {1.0, 0.99, 0.97, 0.9};
  RadiusSet &trial = S.shares;
  for (int c = 0; c < kClasses; ++c) {
    auto b = radius.begin() + S.gat[c], e = b + ngs[c];
    for (int q = 0; q < kShares; ++q) {
      const int i = std::min(ngs[c] - 1, static_cast<int>(share[q] * ngs[c])), at = c * kShares + q;
      std::nth_element(b, b + i, e);
      S.within[at] = 0;
      if (!std::isfinite(b[i])) continue;            // at most 0 nodes: every block's rank is 0
      trial.rho[at] = b[i] * (1.0 + 1e-6);
      trial.most[at] = c == kHalf ? kTrackRankMax : kSmallRank;
      S.within[at] = std::count_if(b, e, [&](float v) { return v <= static_cast<float>(trial.rho[at]); }) /
                   static_cast<double>(ngs[c]);
    }
  }
  S.pix_version = in.pix_version;
  return 0;
}

// n natural blocks to look at, spread evenly over tracks and time together (the R2
// sequence, M. Roberts 2018: multiples of 1/g and 1/g^2, g^3 = g + 1) and the
// channels in turn: a baseline's length decides its ranks, and 48 blocks picked at
// random of 200 misjudged some calls by a fifth.
std::vector<int> spread_blocks(const TrackShape &s, int nb, int n) {
  std::vector<int> at(n);
  const int nbc = s.blocks_per_channel();
  auto part = [](double x, int m) { return std::min(m - 1, static_cast<int>((x - std::floor(x)) * m)); };
  for (int i = 0; i < n; ++i)
    at[i] = n == nb ? i
                    : i % s.channels * nbc + part(0.5 + 0.5698402909980532 * i, s.nbt) * s.lag +
                          part(0.5 + 0.7548776662466927 * i, s.lag);
  return at;
}

}  // namespace

int tracks_try(void **statep, const TrackInputs &in, cudaStream_t st, bool *promising) {
  *promising = false;
  if (!*statep) *statep = new (std::nothrow) TrackState();
  if (!*statep) return 0;
  TrackState &S = *static_cast<TrackState *>(*statep);
  if (!(in.max_turns < 262144.0)) return 0;        // fine_cis: |u.s + off| < 2^19 turns, |s| <= 2
  if (in.K > INT_MAX / 2 || in.ntiles < 8 || in.ntiles > INT_MAX / 16) return 0;
  const int lags = static_cast<int>(std::min<long long>(kLagMax, in.Kc / 32));
  if (lags < 1) return 0;
  TRACK_CUDA(cudaFuncSetAttribute(k_track_ranks<kTrackRankMax>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(sizeof(TrackFactor<kTrackRankMax>))), "attributes");
  TRACK_CUDA(cudaFuncSetAttribute(k_track_ranks<kSmallRank>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(sizeof(TrackFactor<kSmallRank>))), "attributes");
  if (int s = track_pixels(S, in, st)) return s;
  if (S.pix_version != in.pix_version) return 0;   // no memory
  // how far samples a lag apart are
  float *score_d;
  int *trial_rank_d, *order_d, *cls_d, *slot_d;
  double4 *samp_d;
  int4 *refs_d;
  unsigned long long *sums_d;
  const size_t slots = static_cast<size_t>(kRankSamples) * kTrackT, crows = static_cast<size_t>(kClasses + 1) * ((in.ntiles + 31) / 32);
  if (!S.trial.reset(TrackArena::bytes<float>(lags) +
                     TrackArena::bytes<int>(kRadii * kRankSamples) + 2 * TrackArena::bytes<int>(2 * kRankSamples) +
                     TrackArena::bytes<int>(slots) + TrackArena::bytes<double4>(slots) + TrackArena::bytes<int4>(slots) +
                     3 * TrackArena::bytes<unsigned>(crows) + TrackArena::bytes<unsigned long long>(1 + 2 * kEstimates)))
    return 0;
  S.trial.take(score_d, lags);
  S.trial.take(trial_rank_d, kRadii * kRankSamples);
  S.trial.take(order_d, 2 * kRankSamples);
  S.trial.take(cls_d, 2 * kRankSamples);           // classes, then ranks
  S.trial.take(slot_d, slots);
  S.trial.take(samp_d, slots);
  S.trial.take(refs_d, slots);
  for (auto &row : S.crow) S.trial.take(row, crows);
  S.trial.take(sums_d, 1 + 2 * kEstimates);        // classes that leave tiles, unocculted, occulted
  const double rho_lag = 2.0 / std::sqrt(static_cast<double>(in.ntiles));   // about one tile's radius
  k_track_lags<<<lags, kLagSamples, 0, st>>>(in.Kc, in.channels, in.samp, rho_lag, score_d);
  TRACK_CUDA(cudaGetLastError(), "lags");
  std::vector<float> score(lags);
  TRACK_CUDA(cudaMemcpyAsync(score.data(), score_d, sizeof(float) * lags, cudaMemcpyDeviceToHost, st), "lags");
  TRACK_CUDA(cudaStreamSynchronize(st), "lags");
  // the tracks: the shortest lag whose samples lie about as close as any lag's
  const float best = *std::min_element(score.begin(), score.end());
  if (!(best < 1.0f)) return 0;                    // neighbours a turn apart: nothing to interpolate
  TrackShape sh;
  sh.Kc = in.Kc;
  sh.channels = in.channels;
  sh.lag = 1;
  while (score[sh.lag - 1] > 1.05f * best + 1e-7f) ++sh.lag;
  const long long steps = (in.Kc + sh.lag - 1) / sh.lag;
  sh.nbt = static_cast<int>((steps + kTrackT - 1) / kTrackT);
  sh.len = static_cast<int>((steps + sh.nbt - 1) / sh.nbt);
  const long long nbl = static_cast<long long>(sh.channels) * sh.nbt * sh.lag;
  if (nbl * kTrackT > INT_MAX / 2 || nbl * kTrackT > 2 * in.K + 65536) return 0;
  const int nb = static_cast<int>(nbl);
  S.W = (in.ntiles + 31) / 32;
  if (static_cast<double>(nb) * S.W > INT_MAX) return 0;
  const RadiusSet &trial = S.shares;
  const double *within = S.within;
  const int nsamp = std::min(nb, kRankSamples);
  const std::vector<int> order = spread_blocks(sh, nb, nsamp);
  TRACK_CUDA(cudaMemcpyAsync(order_d, order.data(), sizeof(int) * nsamp, cudaMemcpyHostToDevice, st), "order");
  std::vector<int> rk(static_cast<size_t>(kRadii) * nsamp);
  auto block_cost = [&](int at, int i) {
    return within[at] * block_slots(at / kShares, rk[static_cast<size_t>(at) * nsamp + i], sh.len) + (1.0 - within[at]) * kLeftSlots;
  };
  // first the smallest groups alone: samples too sparse for those end here
  auto ranks_of = [&](int first, int n) -> cudaError_t {
    RadiusSet some{};
    for (int q = 0; q < n; ++q) some.rho[q] = trial.rho[first + q], some.most[q] = trial.most[first + q];
    if (first == kHalf)
      k_track_ranks<kTrackRankMax><<<dim3(nsamp, n), kTrackT, sizeof(TrackFactor<kTrackRankMax>), st>>>(
          sh, order_d, in.samp, some, trial_rank_d);
    else
      k_track_ranks<kSmallRank><<<dim3(nsamp, n), kTrackT, sizeof(TrackFactor<kSmallRank>), st>>>(
          sh, order_d, in.samp, some, trial_rank_d);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(rk.data() + static_cast<size_t>(first) * nsamp, trial_rank_d, sizeof(int) * n * nsamp,
                        cudaMemcpyDeviceToHost, st);
    return e != cudaSuccess ? e : cudaStreamSynchronize(st);
  };
  int pick_q[kClasses];
  std::vector<double> least(nsamp, kLeftSlots);    // a block's best class so far
  std::vector<int> least_cls(2 * nsamp, kClasses); // that class, and the rank
  std::fill(least_cls.begin() + nsamp, least_cls.end(), 0);
  for (bool &c : S.chosen) c = false;
  for (int pass = 0; pass < 2; ++pass) {
    TRACK_CUDA(ranks_of(pass ? kShares : 0, pass ? kRadii - kShares : kShares), "ranks");
    for (int c = pass ? 1 : 0; c < (pass ? kClasses : 1); ++c) {
      double best_sum = 1e300;
      for (int q = 0; q < kShares; ++q) {
        double sum = 0;
        for (int i = 0; i < nsamp; ++i) sum += block_cost(c * kShares + q, i);
        // an unocculted adjoint's few tiles that are left are walked by a few warps alone, about
        // 1 ms at 360 blocks (7.5 against 6.4 ms at Nside 256 x 45,720 samples, 1 MHz): not for
        // what the shares of a power-of-two grid differ by; on others they differ severalfold
        if (within[c * kShares + q] < 1.0) sum *= 1.1;
        if (sum < best_sum) best_sum = sum, pick_q[c] = c * kShares + q;
      }
      for (int i = 0; i < nsamp; ++i) {
        const double v = block_cost(pick_q[c], i);
        if (v < least[i]) {
          least[i] = v, least_cls[i] = c, least_cls[nsamp + i] = rk[static_cast<size_t>(pick_q[c]) * nsamp + i];
          S.chosen[c] = true;
        }
      }
    }
    // the smallest groups alone: samples that even those leave near the cost of a
    // call without track blocks end here (larger groups only help where those do)
    double mean = 0;
    for (double v : least) mean += v / nsamp;
    if (!(mean < 0.82 * kTermSlots)) return 0;
  }
  S.chosen[kHalf] = true;
  ClassSet cs{};
  for (int c = 0; c < kClasses; ++c) {
    cs.rho[c] = S.radii.rho[c] = trial.rho[pick_q[c]];
    S.radii.most[c] = trial.most[pick_q[c]];
    cs.at[c] = S.gat[c];
  }
  S.nb = nb;
  S.shape = sh;
  S.Ks = nbl * kTrackT;
  // those blocks' share of a call's work
  TRACK_CUDA(cudaMemcpyAsync(cls_d, least_cls.data(), sizeof(int) * 2 * nsamp, cudaMemcpyHostToDevice, st), "classes");
  TRACK_CUDA(cudaMemsetAsync(sums_d, 0, (1 + 2 * kEstimates) * sizeof(unsigned long long), st), "sums");
  k_track_class_rows<<<dim3(blks(S.W, 128), kClasses + 1), 128, 0, st>>>(S.W, in.ntiles, S.radius, cs, S.crow[0],
                                                                         S.crow[1], S.crow[2], sums_d);
  TRACK_CUDA(cudaGetLastError(), "class rows");
  k_track_slots<<<blks(nsamp * kTrackT, 256), 256, 0, st>>>(sh, nsamp * kTrackT, order_d, in.samp, in.refs, slot_d,
                                                            samp_d, refs_d);
  TRACK_CUDA(cudaGetLastError(), "slots");
  const unsigned by = static_cast<unsigned>(std::max(1, std::min((S.W + 3) / 4, (8 * in.nsm + nsamp - 1) / nsamp)));
  for (int m = 0; m < (in.refs ? 2 : 1); ++m) {
    k_track_estimate<<<dim3(nsamp, by), 128, 0, st>>>(S.W, in.ntiles, slot_d, m ? refs_d : nullptr, in.occ32, in.cones,
                                                      cls_d, cls_d + nsamp, S.crow[0], sums_d + 1 + m * kEstimates);
    TRACK_CUDA(cudaGetLastError(), "estimate");
  }
  unsigned long long sums[1 + 2 * kEstimates] = {};
  TRACK_CUDA(cudaMemcpyAsync(sums, sums_d, sizeof(sums), cudaMemcpyDeviceToHost, st), "estimate");
  TRACK_CUDA(cudaStreamSynchronize(st), "estimate");
  const double all = static_cast<double>(nb) / nsamp;
  for (int m = 0; m < 2; ++m) {
    const unsigned long long *v = sums + 1 + m * kEstimates;
    TrackEstimate &e = S.est[m];
    e.nodes = all * v[0], e.units = all * v[1], e.unit_nodes = all * v[2];
    e.rest_blocks = all * v[3], e.rest_samples = all * v[4];
    const double pairs = static_cast<double>(in.K) * in.ntiles;
    e.seen = all * v[5] / pairs, e.mixed = all * v[6] / pairs;
    e.wide_units = all * v[7];
  }
  S.class_rest = sums[0];
  S.leaves_tiles = false;
  bool bucket[kClasses * kBuckets] = {};           // classes and similar ranks that blocks have
  for (int i = 0; i < nsamp; ++i) {
    const int c = least_cls[i], r = least_cls[nsamp + i];
    if (c < kClasses) bucket[c * kBuckets + (r + 15) / 16] = true;
    S.leaves_tiles = S.leaves_tiles || (S.class_rest >> c & 1u);
  }
  S.slab_count = static_cast<double>(sh.channels) * std::count(bucket, bucket + kClasses * kBuckets, true);
  *promising = true;
  return 0;
}

int tracks_build(void *state, const TrackInputs &in, cudaStream_t st, bool *usable) {
  *usable = false;
  TrackState &S = *static_cast<TrackState *>(state);
  const TrackShape sh = S.shape;
  const int nb = S.nb;
  // every block's ranks in the classes some block looked at takes (the smallest always)
  RadiusSet some{};
  int nclass = 0, class_of[kClasses];
  for (int c = 0; c < kClasses; ++c) {
    if (!S.chosen[c]) continue;
    some.rho[nclass] = S.radii.rho[c];
    some.most[nclass] = S.radii.most[c];
    class_of[nclass++] = c;
  }
  // a block's class, and the stored order: by channel, class, similar rank, then as they come
  const bool masked = in.refs != nullptr;
  const size_t pairs = static_cast<size_t>(nb) * S.W;
  int *all_ranks_d;
  if (!S.masks.reset(TrackArena::bytes<int>(static_cast<size_t>(nclass) * nb))) return 0;
  S.masks.take(all_ranks_d, static_cast<size_t>(nclass) * nb);
  k_track_ranks<kTrackRankMax><<<nb, kTrackT, sizeof(TrackFactor<kTrackRankMax>), st>>>(sh, nullptr, in.samp, some,
                                                                                     all_ranks_d);
  TRACK_CUDA(cudaGetLastError(), "ranks");
  if (nclass > 1) {                                // the first is kHalf
    for (int i = 0; i + 1 < nclass; ++i) some.rho[i] = some.rho[i + 1], some.most[i] = some.most[i + 1];
    k_track_ranks<kSmallRank><<<dim3(nb, nclass - 1), kTrackT, sizeof(TrackFactor<kSmallRank>), st>>>(
        sh, nullptr, in.samp, some, all_ranks_d + nb);
    TRACK_CUDA(cudaGetLastError(), "ranks");
  }
  std::vector<int> rk(static_cast<size_t>(nclass) * nb);
  TRACK_CUDA(cudaMemcpyAsync(rk.data(), all_ranks_d, sizeof(int) * rk.size(), cudaMemcpyDeviceToHost, st), "ranks");
  TRACK_CUDA(cudaStreamSynchronize(st), "ranks");
  const int nbc = sh.blocks_per_channel();
  std::vector<int> pick(nb, kClasses), pick_rank(nb, 0);
  for (int b = 0; b < nb; ++b) {
    double m = kLeftSlots;
    for (int i = 0; i < nclass; ++i) {
      const int r = rk[static_cast<size_t>(i) * nb + b];
      const double v = block_slots(class_of[i], r, sh.len);
      if (v < m) m = v, pick[b] = class_of[i], pick_rank[b] = r;
    }
  }
  std::vector<std::vector<int>> piles(static_cast<size_t>(sh.channels) * (kClasses + 1) * kBuckets);
  for (int b = 0; b < nb; ++b)
    piles[(static_cast<size_t>(b / nbc) * (kClasses + 1) + pick[b]) * kBuckets + (pick_rank[b] + 15) / 16].push_back(b);
  std::vector<int> order, cls, rank, noff;
  S.slabs.clear();
  S.ld_max = 0;
  long long n = 0;
  for (size_t i = 0; i < piles.size(); ++i) {
    const int c = static_cast<int>(i / kBuckets % (kClasses + 1)), ch = static_cast<int>(i / kBuckets / (kClasses + 1));
    // slabs of whole blocks whose node sums fit kSlabBytes; node ranges start at multiples of 32
    const double units = static_cast<double>(in.ntiles) * (c == kHalf ? 2 : 1);
    const long long slab_nodes = std::max<long long>(512, static_cast<long long>(kSlabBytes / (8.0 * units)));
    bool fresh = true;
    for (int b : piles[i]) {
      const int r = pick_rank[b], at = static_cast<int>(order.size());
      if (fresh || n + r - S.slabs.back().n0 > slab_nodes) {
        n = (n + 31) / 32 * 32;
        S.slabs.push_back({ch, c, at, at, static_cast<int>(n), static_cast<int>(n), 0});
        fresh = false;
      }
      order.push_back(b);
      cls.push_back(c);
      rank.push_back(r);
      noff.push_back(static_cast<int>(n));
      n += r;
      if (n > INT_MAX / 4) return 0;
      TrackSlab &sl = S.slabs.back();
      sl.b1 = at + 1;
      sl.n1 = static_cast<int>(n);
      sl.rank = std::max(sl.rank, r);
      S.ld_max = std::max<long long>(S.ld_max, (n - sl.n0 + 31) / 32 * 32 * (c == kHalf ? 2 : 1));
    }
  }
  if (n == 0) return 0;
  const size_t nodes = (n + 31) / 32 * 32, rows = masked ? pairs : 0;
  const size_t sums = static_cast<size_t>(in.ntiles) * S.ld_max;
  // four sample masks per (block, word) are more than most observations need
  const size_t room = 4 * rows;
  if (!S.plan.reset(TrackArena::bytes<uint4>(room) + TrackArena::bytes<int>(S.Ks) + 4 * TrackArena::bytes<int>(nb) + TrackArena::bytes<int>(nodes) +
                    TrackArena::bytes<double4>(S.Ks) + TrackArena::bytes<double4>(nodes) +
                    TrackArena::bytes<int4>(masked ? S.Ks : 0) + TrackArena::bytes<float>(nodes * kTrackT) +
                    4 * TrackArena::bytes<unsigned>(rows) + TrackArena::bytes<int>(rows) +
                    TrackArena::bytes<float2>(sums) + TrackArena::bytes<unsigned long long>(4) + TrackArena::bytes<unsigned>(1)))
    return 0;
  S.plan.take(S.mask, room);
  S.plan.take(S.slot, S.Ks);
  for (int **p : {&S.order, &S.cls, &S.rank, &S.noff}) S.plan.take(*p, nb);
  S.plan.take(S.nodeblk, nodes);
  S.plan.take(S.samp, S.Ks);
  S.plan.take(S.node, nodes);
  S.plan.take(S.refs, masked ? S.Ks : 0);
  S.plan.take(S.P, nodes * kTrackT);
  for (auto &row : S.brow) S.plan.take(row, rows);
  S.plan.take(S.mask_at, rows);
  S.plan.take(S.sums, sums);
  unsigned long long *counts_d;                    // rest pairs, part pairs, ranks that differ; masks taken
  S.plan.take(counts_d, 4);
  S.plan.take(S.peak, 1);
  auto up = [&](int *dst, const std::vector<int> &v) {
    return cudaMemcpyAsync(dst, v.data(), sizeof(int) * v.size(), cudaMemcpyHostToDevice, st);
  };
  TRACK_CUDA(up(S.order, order), "order");
  TRACK_CUDA(up(S.cls, cls), "classes");
  TRACK_CUDA(up(S.rank, rank), "ranks");
  TRACK_CUDA(up(S.noff, noff), "offsets");
  k_track_slots<<<blks(S.Ks, 256), 256, 0, st>>>(sh, S.Ks, S.order, in.samp, in.refs, S.slot, S.samp, S.refs);
  TRACK_CUDA(cudaGetLastError(), "slots");
  TRACK_CUDA(cudaMemsetAsync(S.node, 0, sizeof(double4) * nodes, st), "nodes");
  TRACK_CUDA(cudaMemsetAsync(S.nodeblk, 0xff, sizeof(int) * nodes, st), "nodes");
  TRACK_CUDA(cudaMemsetAsync(counts_d, 0, 4 * sizeof(unsigned long long), st), "counts");
  TRACK_CUDA(cudaFuncSetAttribute(k_track_weights<kTrackRankMax>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(sizeof(TrackFactor<kTrackRankMax>))), "attributes");
  TRACK_CUDA(cudaFuncSetAttribute(k_track_weights<kSmallRank>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(sizeof(TrackFactor<kSmallRank>))), "attributes");
  k_track_weights<kSmallRank><<<nb, kTrackT, sizeof(TrackFactor<kSmallRank>), st>>>(
      0, S.slot, S.samp, S.radii, S.cls, S.rank, S.noff, S.node, S.nodeblk, S.P, counts_d + 2);
  TRACK_CUDA(cudaGetLastError(), "weights");
  if (*std::max_element(rank.begin(), rank.end()) > kSmallRank) {
    k_track_weights<kTrackRankMax><<<nb, kTrackT, sizeof(TrackFactor<kTrackRankMax>), st>>>(
        kSmallRank, S.slot, S.samp, S.radii, S.cls, S.rank, S.noff, S.node, S.nodeblk, S.P, counts_d + 2);
    TRACK_CUDA(cudaGetLastError(), "weights");
  }
  const unsigned by = static_cast<unsigned>(std::max(1, std::min(S.W / 8, (4 * in.nsm * 8) / nb + 1)));
  if (masked) {
    k_track_bits<<<dim3(nb, by), 128, 0, st>>>(S.W, in.ntiles, S.slot, S.refs, in.occ32, in.cones, S.cls, S.crow[0],
                                               S.brow[0], S.brow[1], S.brow[2], S.brow[3], counts_d);
    TRACK_CUDA(cudaGetLastError(), "pair bits");
  }
  unsigned long long pairs_of[3] = {0, 0, 0};
  TRACK_CUDA(cudaMemcpyAsync(pairs_of, counts_d, sizeof(pairs_of), cudaMemcpyDeviceToHost, st), "counts");
  TRACK_CUDA(cudaStreamSynchronize(st), "build");
  if (pairs_of[2]) return 0;
  if (masked) {
    if (pairs_of[1] > INT_MAX) return 0;
    if (pairs_of[1] > room) {
      if (!S.masks.reset(TrackArena::bytes<uint4>(pairs_of[1]))) return 0;
      S.masks.take(S.mask, pairs_of[1]);
    }
    k_track_masks<<<dim3(nb, by), 128, 0, st>>>(S.W, S.slot, S.refs, in.occ32, in.cones, S.brow[1], S.mask_at, S.mask,
                                                counts_d + 3);
    TRACK_CUDA(cudaGetLastError(), "sample masks");
    TRACK_CUDA(cudaStreamSynchronize(st), "build");  // later calls may come on other streams
  }
  S.has_rest[1] = pairs_of[0] != 0;
  S.has_rest[0] = false;                           // unocculted: tiles a used class leaves
  for (const TrackSlab &sl : S.slabs) S.has_rest[0] = S.has_rest[0] || (S.class_rest >> sl.cls & 1u);
  *usable = true;
  return 0;
}

}  // namespace viss
