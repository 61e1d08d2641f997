// tracks_impl.cuh -- what the track blocks' build (tracks_build.cu) and their
// sums (tracks.cu) share.
#pragma once

#include <string>
#include <vector>

#include "tracks.cuh"

namespace viss {

int record_error(int status, const std::string &msg);

constexpr int kTrackRankMax = 96;                // nodes of a block at most
constexpr int kClasses = 4;                      // group sizes; class kClasses: no nodes
constexpr int kHalf = 0, kTile = 1;              // 64 pixels: half a tile; 128: one
__host__ __device__ constexpr int group_pix(int c) { return c == 0 ? 64 : (c == 1 ? 128 : (c == 2 ? 256 : 1024)); }
__host__ __device__ constexpr int group_tiles(int c) { return c < 2 ? 1 : group_pix(c) / kTilePix; }

// The blocks of the caller's order: channel-major; per channel nbt x lag blocks,
// block (tb, b) holds the samples (t lag + b) of steps t in [tb len, tb len + len).
struct TrackShape {
  long long Kc;
  int channels, lag, len, nbt;
  __host__ __device__ int blocks_per_channel() const { return nbt * lag; }
};

// Pair bits of a set of blocks: row b of each (occulted) or row cls[b].
struct TrackBits {
  const unsigned *full, *part, *merged, *rest;   // part null: none
  const int *mask_at;                            // occulted: a word's first sample mask (of its part tiles)
  const uint4 *mask;                             // the samples that see all of a part tile
  const int *cls;                                // null: rows are per block
  int W;
  __device__ __forceinline__ long long row(int b) const { return static_cast<long long>(cls ? cls[b] : b) * W; }
};

// Blocks [b0, b1) of one channel and class, of similar rank; nodes [n0, n1).
struct TrackSlab {
  int ch, cls, b0, b1, n0, n1, rank;   // rank: the largest of its blocks
};

// One device allocation that buffers are cut from (an allocation call costs a
// third of a millisecond, whatever its size).
struct TrackArena {
  char *base = nullptr;
  size_t cap = 0, used = 0;
  ~TrackArena() {
    if (base) cudaFree(base);
  }
  // Room for `bytes` (256 per buffer for alignment included), emptied.
  bool reset(size_t bytes) {
    used = 0;
    if (base && bytes <= cap) return true;
    if (base) cudaFree(base);
    base = nullptr;
    cap = 0;
    void *p = nullptr;
    if (cudaMalloc(&p, bytes ? bytes : 256) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    base = static_cast<char *>(p);
    cap = bytes ? bytes : 256;
    return true;
  }
  template <class T>
  static size_t bytes(size_t n) {
    return (n * sizeof(T) + 255) / 256 * 256;
  }
  template <class T>
  void take(T *&p, size_t n) {
    p = reinterpret_cast<T *>(base + used);
    used += bytes<T>(n);
  }
};

// What a call has to do, estimated from a few blocks: node exponentials, (sample,
// unit) pairs and those times the rank, (block, tile) and (sample, tile) pairs of
// the remainder; the share of (sample, tile) pairs that are seen at all and in part;
// (sample, unit) pairs of ranks whose interpolation leaves room for one CTA per SM.
struct TrackEstimate {
  double nodes = 0, units = 0, unit_nodes = 0, rest_blocks = 0, rest_samples = 0, seen = 0, mixed = 0, wide_units = 0;
};
constexpr int kOneCtaRank = 52;

constexpr int kShares = 4;                       // radii tried per class
constexpr int kRadii = kClasses * kShares;
struct RadiusSet {
  double rho[kRadii];
  int most[kRadii];
};
struct ClassSet {
  double rho[kClasses];
  int at[kClasses];
};

struct TrackState {
  TrackArena pixels, trial, plan, masks, call;
  long long pix_version = -1;              // of the pixels that `pixels` and `shares` are of
  RadiusSet shares{};                      // radii to try, and the share of groups within each
  double within[kRadii] = {};
  float *radius = nullptr;                 // groups', class after class from gat[c]
  TrackEstimate est[2];                    // unocculted, occulted
  double slab_count = 0;                   // slabs, but for those that a class of one rank is cut into by memory
  unsigned long long class_rest = 0;       // bit c: class c leaves tiles
  bool leaves_tiles = false;               // a class that blocks take does
  RadiusSet radii{};                       // per class
  bool chosen[kClasses] = {};
  int *slot = nullptr, *order = nullptr, *cls = nullptr, *rank = nullptr, *noff = nullptr, *nodeblk = nullptr;
  double4 *samp = nullptr, *node = nullptr, *gcen = nullptr;
  int4 *refs = nullptr;
  float *P = nullptr;
  unsigned *crow[3] = {};                  // class rows: full, merged, rest (in `trial`)
  unsigned *brow[4] = {};                  // occulted: full, part, merged, rest per block
  int *mask_at = nullptr;
  uint4 *mask = nullptr;
  float2 *sums = nullptr;
  unsigned *peak = nullptr;                // a call's largest finite sky or coefficient, as float bits
  TrackShape shape{};
  int nb = 0, W = 0;
  int gat[kClasses] = {0, 0, 0, 0};        // a class's first centre in gcen
  long long Ks = 0, ld_max = 0;
  bool has_rest[2] = {false, false};       // unocculted, occulted
  std::vector<TrackSlab> slabs;

  TrackBits bits(bool occulted) const {
    TrackBits t{};
    t.W = W;
    t.full = occulted ? brow[0] : crow[0];
    t.part = occulted ? brow[1] : nullptr;
    t.merged = occulted ? brow[2] : crow[1];
    t.rest = occulted ? brow[3] : crow[2];
    t.mask_at = occulted ? mask_at : nullptr;
    t.mask = occulted ? mask : nullptr;
    t.cls = occulted ? nullptr : cls;
    return t;
  }
};

inline unsigned blks(long long n, int bs) { return static_cast<unsigned>((n + bs - 1) / bs); }

inline int track_cuda_err(cudaError_t e, const char *where) {
  return record_error(-2, std::string("track blocks: ") + where + ": " + cudaGetErrorString(e));
}

#define TRACK_CUDA(call, where)                                \
  do {                                                         \
    const cudaError_t e_ = (call);                             \
    if (e_ != cudaSuccess) return track_cuda_err(e_, where);   \
  } while (0)

}  // namespace viss
