// tracks.cu -- the direct sums of visibility.cu when the samples lie on smooth
// tracks (the baselines of a formation, sampled along its orbit).
//
// Against a compact group g of pixels (centre s_g, radius rho) the sum of one
// sample, with the phase of the centre taken out, is
//
//   G(u) = sum_{j in g} I_j e^{-2 pi i u.(s_j - s_g)},
//
// a function of u whose "frequencies" s_j - s_g all lie within rho.  Over a
// block of kTrackT = 128 successive samples of one track u moves by a few
// 1 / rho, so G at all of them follows from G at r << 128 of them (the nodes):
// G(u_k) = sum_n P_kn G(u_n) with real weights P that do not depend on the
// pixels.  Per (block, group) the kernels therefore evaluate r exponentials
// per pixel instead of 128, plus one phase per (sample, group):
//
//   forward  V_k  = sum_g e^{-2 pi i (u_k.s_g + off_k)} sum_n P_kn G_g(u_n)
//   adjoint  the transpose: b_n = sum_k P_kn a_k e^{2 pi i (u_k.s_g + off_k)}, and
//            C_j += Re(sum_n b_n e^{2 pi i u_n.(s_j - s_g)})
//
// Nodes and weights.  With directions s - s_g spread evenly over a sphere of
// radius rho the functions e^{-2 pi i u.(s - s_g)} of two samples correlate as
// sinc(2 rho |u - u'|).  A Cholesky factorisation of that matrix, pivoted on
// the sample that the nodes so far predict worst, picks the nodes; P is the
// least-squares predictor for node values that carry an independent relative
// error of kNodeNoise = 2e-7 (1.7e-7 of one node exponential, and FP32 sums).  A
// block stops when its mean squared prediction error, node errors included, is
// below 1.8 kNodeNoise^2 (no sample above 4.5): (2.7e-7)^2, where a term that
// k_forward evaluates is off by 3.7e-7 (a phase of 23 bits).  Measured against
// FP64 on four inputs each of 1 to 10 MHz observations at Nside 128 and 256: V 2.0e-7 -
// 3.2e-7, images of random coefficients 2.8e-7 - 3.0e-7 and of the observations 2.3e-7
// - 3.2e-7; the direct kernels 2.5e-7 - 4.6e-7, 5.0e-7 and 2.6e-7 - 5.4e-7.
// Stopping at 0.85 (3e-7)^2 with the same node error costs 25 % more nodes
// for 8 % less error, stopping at 2.5 saves 1 %.  Blocks that need more than
// kTrackRankMax nodes, or three quarters of their samples, are left to the
// remainder kernels.
//
// Group size.  Long baselines turn faster: every block takes the group size
// (64, 128, 256 or 1024 pixels) with the least modelled time, and blocks of one
// size (a class) are stored together, so that a launch has one size.
//
// Occultation.  The node sums of a 128-pixel tile are of all its pixels, so a
// sample that sees the whole tile (the conservative FP32 test of the direct
// kernels on the same cones and rows) takes its interpolated value whatever
// the block's other samples see.  Tiles that every sample of the block sees are
// merged into their group; samples that see part of a tile are evaluated by the
// remainder kernels with the exact predicate; both sides classify a (sample,
// tile) pair by the same function of the same inputs, so each is counted once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "direct.cuh"
#include "tcgen05.cuh"
#include "tracks_impl.cuh"

namespace viss {

namespace {

constexpr int kChunkTiles = 256;                 // most tiles of one interpolation chunk

}  // namespace

struct TrackNodeParams {
  const double4 *pix;          // forward: the channel's pixel + sky records; adjoint: pixel records
  const double4 *node;         // the slab's first node
  const int *nodeblk;
  TrackBits bits;
  int cls, ntiles;
  int nn;                      // nodes in the slab
  int per_chunk;               // forward: tiles (whole groups), adjoint: nodes (a multiple of 128)
  long long ld;                // node sums: value of (unit, node n) at unit * ld + n
  float2 *sums;
  double *part;                // adjoint: [chunk][Jpad], added to
  long long Jpad;
  unsigned long long *counter;
  int *err;
  int drop_tile;
  const unsigned *peak;        // forward
};

// Node sums are stored per unit: a half tile (2 t + h) in the 64-pixel class, else
// a tile; a merged group's sum stands at its first tile.
namespace {

// Angle of t = kTurn32 + phase, |phase| < 2^19 turns: its low 32 bits are the
// phase's fraction in 2^-32 turn, as a signed integer in [-1/2, 1/2) turn, so the
// conversion and one product give the angle to FP32 rounding, in as many
// instructions as turn_angle (whose 23-bit fraction covers 2^28 turns) and in the
// same time: exponentials 1.7e-7 off instead of 3.7e-7, so fewer nodes will do
// (with turn_angle the 10 MHz forward took 68.4 ms and the adjoint 78.7 ms
// instead of 54 and 67).
constexpr double kTurn32 = 1572864.0;            // 1.5 * 2^20
__device__ __forceinline__ float turn_angle32(double t) {
  return static_cast<float>(__double2loint(t)) * 1.46291807926716e-9f;
}

// The tensor cores take operands below 2^-126 for zero, and the low half of a split
// value is 2^-12 of it: skies below 1e-36 and coefficients below 1e-35 lost up to all
// their accuracy.  A call's operands are scaled by the power of two that brings its
// largest finite value to [1, 2), and the sums back in FP64; both are exact.
__global__ void k_track_peak(long long n, const double4 *pixsky, const float2 *coef, unsigned *peak) {
  unsigned top = 0;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const float2 v = pixsky ? make_float2(sky_of(pixsky[i]), 0.f) : coef[i];
    if (isfinite(v.x)) top = max(top, __float_as_uint(fabsf(v.x)));
    if (isfinite(v.y)) top = max(top, __float_as_uint(fabsf(v.y)));
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0 && top) atomicMax(peak, top);
}
__device__ __forceinline__ int peak_exponent(const unsigned *peak) {
  const unsigned bits = *peak;
  return bits ? min(max(static_cast<int>(bits >> 23) - 127, -126), 126) : 0;
}
__device__ __forceinline__ float scale_of(int e) { return __int_as_float((127 - e) << 23); }
__device__ __forceinline__ double unscale_of(int e) { return __hiloint2double((1023 + e) << 20, 0); }

constexpr int kNodeNT = 256;
constexpr int kNodeR = 4;
// Terms added in plain FP32 before a run's sum joins the others: pixels in the
// forward, nodes (two additions each) in the adjoint.  Runs of 128 left 1.9e-7 and
// 2.7e-7 of the sum's own size.  Images of random coefficients went from 3.75e-7 to
// 2.85e-7 of error at 1 MHz in the same time.  In the forward at 10 MHz runs of 32 took V
// from 3.0e-7 to 2.75e-7 for 1.2 % of the time, runs of 64 to 2.9e-7 for none (53.3 and
// 52.6 ms; its images are at 3.1e-7 with either).
constexpr int kFwdRun = 64, kNodeRun = 32;

// G of the slab's nodes (R per thread) over a chunk of tiles: the inner loop
// and the stage ring of k_forward, a value written per (unit, node) instead of
// one sum over all tiles.  Bound by the SFU and the FP64 phase like k_forward;
// it evaluates r / 128 of its terms.
template <bool HALF>
__global__ void __launch_bounds__(kNodeNT, 2) k_track_fwd_nodes(const TrackNodeParams p) {
  constexpr int S = kFwdStages, R = kNodeR, NT = kNodeNT;
  __shared__ __align__(128) double4 s_pix[S][kTilePix];
  __shared__ __align__(8) uint64_t s_full[S], s_empty[S];
  __shared__ int s_abort;
  volatile int *abort_flag = &s_abort;
  const int tid = threadIdx.x, lane = tid & 31;
  const int nb = blockIdx.x * (NT * R);
  double ux[R], uy[R], uz[R];
  int row[R];                                        // offset of the node's pair bits, -1 no node
  unsigned word[R], merged[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int n = nb + r * NT + tid;
    const int blk = n < p.nn ? p.nodeblk[n] : -1;
    const double4 u = blk >= 0 ? p.node[n] : make_double4(0, 0, 0, 0);
    ux[r] = u.x; uy[r] = u.y; uz[r] = u.z;
    row[r] = blk >= 0 ? static_cast<int>(p.bits.row(blk)) : -1;
    word[r] = merged[r] = 0;
  }
  const int t0 = blockIdx.y * p.per_chunk, ntile = max(0, min(t0 + p.per_chunk, p.ntiles) - t0);
  const int gt = group_tiles(p.cls);
  const int drop = (blockIdx.x == 0 && blockIdx.y == 0) ? min(p.drop_tile, ntile - 1) : -1;   // test hook (k_forward)
  constexpr uint32_t kTileBytes = kTilePix * sizeof(double4);
  auto issue = [&](int i, int stage) {
    if (i == drop) return;
    mbar_expect_tx(&s_full[stage], kTileBytes);
    bulk_g2s(s_pix[stage], p.pix + static_cast<long long>(t0 + i) * kTilePix, kTileBytes, &s_full[stage]);
  };
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], NT / 32);
    }
    fence_mbar_init();
    s_abort = 0;
  }
  __syncthreads();

  float g_re[R], g_im[R];
#pragma unroll
  for (int r = 0; r < R; ++r) g_re[r] = g_im[r] = 0.f;
  const float scale = scale_of(peak_exponent(p.peak));
  unsigned long long evaluated = 0;
  int next = 0;
  for (int it = 0; it < ntile; ++it) {
    const int t = t0 + it, stage = it % S;
    if (tid == 0 && !ring_refill<S>(s_empty, next, it, ntile, issue)) {
      atomicOr(p.err, kErrTimeout);
      *abort_flag = 1;
    }
    if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
    if (it == 0 || (t & 31) == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (row[r] < 0) continue;
        word[r] = p.bits.full[row[r] + (t >> 5)] | (p.bits.part ? p.bits.part[row[r] + (t >> 5)] : 0u);
        merged[r] = p.bits.merged[row[r] + (t >> 5)];
      }
    }
    unsigned rows = 0;                               // rows any lane of the warp needs
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const unsigned b = __ballot_sync(0xffffffffu, (word[r] >> (t & 31)) & 1u);
      rows |= static_cast<unsigned>(b != 0) << r;
      evaluated += static_cast<unsigned>(__popc(b)) * static_cast<unsigned>(kTilePix);
    }
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&s_full[stage], static_cast<uint32_t>(it / S) & 1u))) {
      if (lane == 0) atomicOr(p.err, kErrTimeout);
      *abort_flag = 1;
      break;
    }
    if (rows) {
#pragma unroll 1
      for (int h = 0; h < (HALF ? 2 : 1); ++h) {
        constexpr int kSpan = HALF ? kTilePix / 2 : kTilePix;
        const double4 *tp = s_pix[stage] + h * kSpan;
        float t_re[R], t_im[R];
#pragma unroll
        for (int r = 0; r < R; ++r) t_re[r] = t_im[r] = 0.f;
        auto term = [&](int r, const double4 &q, float I, double magic, float &re, float &im) {
          float sn, cs;
          sfu_sincos(turn_angle32(fma(uz[r], q.z, fma(uy[r], q.y, fma(ux[r], q.x, magic)))), sn, cs);
          re = fmaf(I, cs, re);
          im = fmaf(-I, sn, im);
        };
        if (rows == (1u << R) - 1) {
          for (int j0 = 0; j0 < kSpan; j0 += kFwdRun) {
            float re[R], im[R];
#pragma unroll
            for (int r = 0; r < R; ++r) re[r] = im[r] = 0.f;
#pragma unroll 4
            for (int j = j0; j < j0 + kFwdRun; j += 2) {
              const double4 q0 = tp[j], q1 = tp[j + 1];
              const float I0 = sky_of(q0), I1 = -sky_of(q1);
#pragma unroll
              for (int r = 0; r < R; ++r) {
                term(r, q0, I0, kTurn32, re[r], im[r]);
                term(r, q1, I1, kTurn32 + 0.5, re[r], im[r]);   // odd records half a turn on (k_forward)
              }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) t_re[r] += re[r], t_im[r] += im[r];
          }
        } else {
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (!((rows >> r) & 1u)) continue;
            for (int j0 = 0; j0 < kSpan; j0 += kFwdRun) {
              float re = 0.f, im = 0.f;
#pragma unroll 4
              for (int j = j0; j < j0 + kFwdRun; j += 2) {
                const double4 q0 = tp[j], q1 = tp[j + 1];
                term(r, q0, sky_of(q0), kTurn32, re, im);
                term(r, q1, -sky_of(q1), kTurn32 + 0.5, re, im);
              }
              t_re[r] += re;
              t_im[r] += im;
            }
          }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if (!((word[r] >> (t & 31)) & 1u)) continue;
          const int n = nb + r * NT + tid;
          if (HALF) {
            p.sums[(2LL * t + h) * p.ld + n] = make_float2(scale * t_re[r], scale * t_im[r]);
          } else if (!((merged[r] >> (t & 31)) & 1u)) {
            p.sums[static_cast<long long>(t) * p.ld + n] = make_float2(scale * t_re[r], scale * t_im[r]);
          } else {
            g_re[r] += t_re[r];
            g_im[r] += t_im[r];
            if (t % gt == gt - 1 || t == p.ntiles - 1) {   // the chunk holds whole groups
              p.sums[static_cast<long long>(t / gt * gt) * p.ld + n] = make_float2(scale * g_re[r], scale * g_im[r]);
              g_re[r] = g_im[r] = 0.f;
            }
          }
        }
      }
    }
    ring_release(s_empty, stage);
  }
  if (tid == 0) ring_drain<S>(s_full, next);
  if (lane == 0 && evaluated) atomicAdd(p.counter, evaluated);
}

struct TrackInterpParams {
  const double4 *samp;         // slots
  const int *slot;
  const int4 *refs;            // slots, null: unocculted
  const float4 *occ32;
  const float4 *cones;
  const double4 *node;         // all nodes
  const int *rank, *noff;
  const float *P;
  TrackBits bits;
  const double4 *gcen[3];      // centres of the half tiles, the tiles, the class's groups
  int cls, ntiles;
  int b0;                      // the slab's first block; every block of it has nodes
  int n0;                      // and node
  int per_chunk;               // tiles per blockIdx.y, a multiple of 32, at most kChunkTiles
  long long ld;
  float2 *sums;
  int use_off;
  double2 *vacc;               // forward: [chunk][slots of the slab]
  long long vstride;
  const float2 *coef;          // adjoint: slots
  int *err;
  bool drop;                   // test hook: block (0, 0) never signals its first product
  const unsigned *peak;        // forward
};

// A wait that gave up ends an interpolation block at its next barrier (all threads
// together, `broken`); before its tensor memory is freed, the products issued and
// not waited for get another bounded wait.
__device__ __forceinline__ bool broken(bool ok) { return __syncthreads_or(!ok) != 0; }
__device__ __forceinline__ void drain_products(uint64_t *done, int issued) {
  for (int i = max(issued - 2, 0); i < issued; ++i) mbar_wait_bounded(&done[i & 1], static_cast<uint32_t>(i >> 1) & 1u);
}

// A unit of one pass: its group's centre, its row of node sums, and which of
// the block's samples see it (bit k mod 32 of word k / 32).
struct __align__(16) PassUnit {
  double x, y, z;
  int row, pad;
  unsigned seen[kTrackT / 32];
};

// The units of block b in tiles [t0, t1) (t0 a multiple of 32): entries
// (tile * 8 + flags, index of its sample mask).  Written by the first warp;
// returns the count to all.
constexpr int kUnitPart = 1, kUnitMerged = 2, kUnitUpper = 4;   // upper: second half of the tile
__device__ int list_units(const TrackBits &bits, int b, int cls, int t0, int t1, int2 *list) {
  __shared__ int s_count;
  const int lane = threadIdx.x;
  if (lane < 32) {
    const int nw = (t1 - t0 + 31) / 32;            // at most 32
    const long long at = bits.row(b) + t0 / 32 + lane;
    unsigned full = 0, part = 0, merged = 0;
    int mask = 0;
    if (lane < nw) {
      full = bits.full[at];
      part = bits.part ? bits.part[at] : 0u;
      merged = bits.merged[at];
      if (part) mask = bits.mask_at[at];
    }
    const unsigned first = cls == 2 ? 0x55555555u : 0x01010101u;
    const unsigned start = (full | part) & ~(merged & ~first);
    const int each = cls == kHalf ? 2 : 1;
    int n = __popc(start) * each;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, n, o);
      if (lane >= o) n += v;
    }
    if (lane == 31) s_count = n;
    n -= __popc(start) * each;
    for (unsigned m = start; m; m &= m - 1) {
      const int i = __ffs(m) - 1;
      int2 e = make_int2((t0 + 32 * lane + i) * 8 + ((part >> i) & 1u ? kUnitPart : 0) +
                             ((merged >> i) & 1u ? kUnitMerged : 0),
                         mask + __popc(part & ((1u << i) - 1u)));
      list[n++] = e;
      e.x += kUnitUpper;
      if (cls == kHalf) list[n++] = e;
    }
  }
  __syncthreads();
  return s_count;
}

// Entry e as a pass unit.
__device__ __forceinline__ PassUnit pass_unit(const TrackInterpParams &p, int2 e) {
  PassUnit v;
  const int t = e.x >> 3;
  v.row = p.cls == kHalf ? 2 * t + ((e.x & kUnitUpper) ? 1 : 0) : t;
  const double4 c = p.cls == kHalf ? p.gcen[0][v.row] : ((e.x & kUnitMerged) ? p.gcen[2][t / group_tiles(p.cls)] : p.gcen[1][t]);
  v.x = c.x; v.y = c.y; v.z = c.z;
  uint4 m = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
  if (e.x & kUnitPart) m = p.bits.mask[e.y];
  v.seen[0] = m.x; v.seen[1] = m.y; v.seen[2] = m.z; v.seen[3] = m.w;
  return v;
}

// t = kFine + phase holds the phase's fraction in its low 32 bits, in units of
// 2^-32 turn, for |phase| < 2^19 turns.  fine_cis gives (cos, sin) of it to a
// few 1e-8 (the phases of whole partial sums): 23 bits of the distance to the
// nearest quarter turn, read as a float (the half unit in kFine centres the
// truncation), and least-squares polynomials at Chebyshev nodes (max error 9e-8).
constexpr double kFine = 1572864.0 + 1.4901161193847656e-08;    // 1.5 * 2^20 + 2^-26
__device__ __forceinline__ float2 fine_cis(double t) {
  const unsigned lo = static_cast<unsigned>(__double2loint(t));
  const unsigned q = lo + 0x20000000u;                           // quadrant in bits 30, 31
  const float x = __uint_as_float(((lo >> 7) & 0x7fffffu) ^ 0x3fc00000u) - 1.5f;   // quarter turns, |x| <= 1/2
  const float z = x * x;
  const float s0 = x * fmaf(z, fmaf(z, fmaf(z, -4.59227756e-3f, 7.96759945e-2f), -6.45962939e-1f), 1.57079631f);
  const float c0 = fmaf(z, fmaf(z, fmaf(z, -2.04244194e-2f, 2.53605679e-1f), -1.23369793f), 1.0f);
  const bool odd = q & 0x40000000u;
  const float s1 = odd ? c0 : s0, c1 = odd ? s0 : c0;
  // sin negative in quadrants 2, 3; cos in 1, 2
  return make_float2(__uint_as_float(__float_as_uint(c1) ^ ((q ^ (q << 1)) & 0x80000000u)),
                     __uint_as_float(__float_as_uint(s1) ^ (q & 0x80000000u)));
}
__device__ __forceinline__ double fine_phase(double ux, double uy, double uz, const PassUnit &g, double init) {
  return fma(uz, g.z, fma(uy, g.y, fma(ux, g.x, init)));
}

// The interpolation kernels' matrix products run on the tensor cores: TF32
// operands, each FP32 value split in two (22 bits), and the three products that
// matter -- hi lo, lo hi, hi hi -- accumulated in FP32, the small ones first
// (the accumulator truncates, so it should be small while they are added).
// Measured against FP64 on random 128 x K by K x 64 products: 1.1e-7 at K = 32,
// 1.8e-7 at K = 64, where FP32 multiply-adds give 1.0e-7 and 1.5e-7.
//
// What that leaves out in scale, on average, is put back (interp_scale; not for one
// node: identical samples, whose sums stay exact).  The SFU's sine and cosine are
// 7.6e-8 short over a turn.  Every product added into an accumulator truncates it:
// with the kernels' own order of products and the weights of 1 and 10 MHz
// observations, sums of n = ceil(r / 8) steps (forward) came out 3.8, 5.7, 7.4,
// 10.1, 12.9, 14.3e-8 short for n = 1 to 6, those of the adjoint's runs of 6 steps
// 1.04e-7 to 1.16e-7 at ranks of 10 to 37.  One factor of 1.5e-7 for all of them left
// V up to 5.8e-8 too large and images 3.0e-8 to 4.2e-8 too small; now 1.4e-8 of
// incoherent sums at most either way.
__device__ __forceinline__ float interp_scale(int r, bool adjoint) {
  if (r == 1) return 0.f;
  return 7.6e-8f + (adjoint ? 1.1e-7f : 1.7e-8f + 2.1e-8f * static_cast<float>((r + 7) / 8));
}

constexpr int kInterpNT = 256;
constexpr int kFwdUnits = 32;          // units per pass, forward: 64 columns of the product
constexpr int kFwdLboA = 2048, kFwdLboB = 2 * kFwdUnits * 16 + 16;

__host__ __device__ constexpr int round_up(int x, int m) { return (x + m - 1) / m * m; }

// Shared memory of the forward interpolation for blocks of rank r.
struct FwdInterpSmem {
  int a, b, un, units, list, total;
  __host__ __device__ explicit FwdInterpSmem(int r) {
    const int kc = round_up(r, 8) / 4;
    a = 0;                                           // P: hi, lo
    b = a + 2 * kc * kFwdLboA;                       // node sums: [2 buffers] hi, lo
    un = b + 4 * kc * kFwdLboB;
    units = un + r * static_cast<int>(sizeof(double4));
    list = units + 4 * kFwdUnits * static_cast<int>(sizeof(PassUnit));
    total = list + 2 * kChunkTiles * static_cast<int>(sizeof(int2));
  }
};

// V of one block's samples from its node sums over a chunk of tiles, kFwdUnits
// units a pass: node sums times e^{2 pi i u_n.s_g}, split, into shared memory;
// the product with P (split once, in shared memory for the whole launch) on the
// tensor core into tensor memory, double buffered, so it runs behind the next
// pass's preparation; then every thread takes its sample's row for half of the
// units, times e^{-2 pi i (u_k.s_g + off)}.  Bound by FP32 and integer issue, about
// 50 slots per (sample, unit), most of them the phase (the product in FP32
// multiply-adds took another 2 r + LDS).
template <bool PART>
__global__ void __launch_bounds__(kInterpNT, 3) k_track_fwd_interp(const TrackInterpParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t s_done[2];
  __shared__ double2 s_meet[kTrackT];
  const int b = p.b0 + blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = p.rank[b];
  const int kp = round_up(r, 8), kc = kp / 4, n0 = p.noff[b];
  const FwdInterpSmem at(r);
  unsigned char *A = smem + at.a, *B = smem + at.b;
  double4 *un = reinterpret_cast<double4 *>(smem + at.un);
  PassUnit *units = reinterpret_cast<PassUnit *>(smem + at.units);          // [4][kFwdUnits]
  int2 *list = reinterpret_cast<int2 *>(smem + at.list);
  if (warp == 0) tmem_alloc(&s_tmem, 128);
  if (tid == 0) {
    mbar_init(&s_done[0], 1);
    mbar_init(&s_done[1], 1);
    fence_mbar_init();
  }
  for (int n = tid; n < r; n += kInterpNT) un[n] = p.node[n0 + n];
  for (int i = tid; i < kp * kTrackT; i += kInterpNT) {
    const int n = i / kTrackT, k = i % kTrackT, o = umma_offset(k, n, kFwdLboA);
    float hi = 0.f, lo = 0.f;
    if (n < r) split_tf32(p.P[static_cast<long long>(n0 + n) * kTrackT + k], hi, lo);
    *reinterpret_cast<float *>(A + o) = hi;
    *reinterpret_cast<float *>(A + kc * kFwdLboA + o) = lo;
  }
  const int t0 = blockIdx.y * p.per_chunk, t1 = min(t0 + p.per_chunk, p.ntiles);
  const int count = list_units(p.bits, b, p.cls, t0, t1, list);             // synchronises
  const int passes = (count + kFwdUnits - 1) / kFwdUnits;
  const float2 *sums = p.sums + (n0 - p.n0);
  auto prepare = [&](int pass) {
    const int i = pass * kFwdUnits + tid;
    if (tid < kFwdUnits) units[(pass & 3) * kFwdUnits + tid] = i < count ? pass_unit(p, list[i]) : PassUnit{};
  };
  // this thread's node sums of a pass: one unit, nodes tid mod 8, + 8, ...
  const int own = tid >> 3, own_n = tid & 7, own_o = umma_offset(2 * own, own_n, kFwdLboB);
  // (the first 8 fetched a pass ahead)
  constexpr int kAhead = 8;
  float2 pre[kAhead];
  auto fetch = [&](int pass) {
    if (pass * kFwdUnits + own >= count) return;
    const float2 *src = sums + units[(pass & 3) * kFwdUnits + own].row * p.ld;
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      if (own_n + 8 * j < r) pre[j] = src[own_n + 8 * j];
  };
  // sample of this thread: row (warp mod 4) 32 + lane; half of the units
  const int half = warp >> 2, row = (warp & 3) * 32 + lane;
  const long long slot = static_cast<long long>(b) * kTrackT + row;
  double4 u = p.samp[slot];
  u.w = kFine + (p.use_off ? u.w : 0.0);
  prepare(0);
  prepare(1);
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  const uint32_t tmem = s_tmem;
  if (passes > 0) fetch(0);
  const bool drop = p.drop && blockIdx.x == 0 && blockIdx.y == 0;
  double vre = 0.0, vim = 0.0;
  bool ok = true;
  int pass = -1;
  for (; pass < passes; ++pass) {
    const int next = pass + 1;
    if (next < passes) {
      // the next pass's operand; its buffer was read by the product before the last one
      unsigned char *Bn = B + (next & 1) * 2 * kc * kFwdLboB;
      const bool have = next * kFwdUnits + own < count;
      const PassUnit g = units[(next & 3) * kFwdUnits + own];
      auto put = [&](int j, const float2 &sum) {
        const int n = own_n + 8 * j;
        float2 v = make_float2(0.f, 0.f);
        if (have && n < r) {
          const double4 w = un[n];
          const float2 c = fine_cis(fine_phase(w.x, w.y, w.z, g, kFine));
          v = make_float2(sum.x * c.x - sum.y * c.y, sum.x * c.y + sum.y * c.x);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          unsigned char *o = Bn + own_o + j * 2 * kFwdLboB + q * 16;   // row 2 own + q, column n
          float hi, lo;
          split_tf32(q ? v.y : v.x, hi, lo);
          *reinterpret_cast<float *>(o) = hi;
          *reinterpret_cast<float *>(o + kc * kFwdLboB) = lo;
        }
      };
#pragma unroll
      for (int j = 0; j < kAhead; ++j)
        if (8 * j < kp) put(j, pre[j]);
      for (int j = kAhead; 8 * j < kp; ++j)
        put(j, have && own_n + 8 * j < r ? sums[g.row * p.ld + own_n + 8 * j] : make_float2(0.f, 0.f));
      fence_async_smem();
      umma_fence_before();
    }
    if (broken(ok)) {
      ok = false;
      break;
    }
    umma_fence_after();
    prepare(pass + 3);                             // over the units every thread is done with
    if (next < passes && tid == 0) {
      const uint32_t a = smem_addr(A), bn = smem_addr(B + (next & 1) * 2 * kc * kFwdLboB);
      const uint32_t idesc = umma_idesc_tf32(2 * kFwdUnits), d = tmem + (next & 1) * 2 * kFwdUnits;
      bool add = false;
      for (int q = 0; q < 3; ++q)                  // hi lo, lo hi, hi hi
        for (int ks = 0; ks < kc; ks += 2, add = true)
          umma_tf32(d, umma_desc(a + ((q == 1 ? kc : 0) + ks) * kFwdLboA, kFwdLboA),
                    umma_desc(bn + ((q == 0 ? kc : 0) + ks) * kFwdLboB, kFwdLboB), idesc, add);
      if (next > 0 || !drop) umma_commit(&s_done[next & 1]);
    }
    if (pass + 2 < passes) fetch(pass + 2);
    if (pass < 0) continue;
    ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&s_done[pass & 1], (pass >> 1) & 1));
    umma_fence_after();
    const PassUnit *pu = units + (pass & 3) * kFwdUnits + half * (kFwdUnits / 2);
    float sre = 0.f, sim = 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float d[16];
      tmem_load16(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (pass & 1) * 2 * kFwdUnits +
                      half * kFwdUnits + 16 * h, d);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const PassUnit &g = pu[8 * h + q];         // past the last unit: a zero sum
        const float2 w = fine_cis(fine_phase(u.x, u.y, u.z, g, u.w));
        const bool on = !PART || ((g.seen[warp & 3] >> lane) & 1u);
        sre += on ? fmaf(d[2 * q], w.x, d[2 * q + 1] * w.y) : 0.f;
        sim += on ? fmaf(d[2 * q + 1], w.x, -d[2 * q] * w.y) : 0.f;
      }
    }
    vre += static_cast<double>(sre);
    vim += static_cast<double>(sim);
    umma_fence_before();                           // the next product but one writes these columns
  }
  if (!ok) {
    if (lane == 0) atomicOr(p.err, kErrTimeout);
    drain_products(s_done, min(pass + 1, passes));
  }
  // the two halves of the units meet
  if (half == 1) s_meet[row] = make_double2(vre, vim);
  umma_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, 128);
  if (half == 0) {
    const double2 o = s_meet[row];
    const double scale = unscale_of(peak_exponent(p.peak)) * (1.0 + static_cast<double>(interp_scale(r, false)));
    p.vacc[blockIdx.y * p.vstride + static_cast<long long>(blockIdx.x) * kTrackT + row] =
        make_double2(scale * (vre + o.x), scale * (vim + o.y));
  }
}

// V[slot[i]] = the slab's interpolated sums + the remainder's chunks (FP64).
__global__ void k_track_reduce_fwd(long long n, long long first, const int *slot, int nv, const double2 *vacc,
                                   long long vstride, int nchunk, const double2 *part, long long Ks, float2 *V,
                                   int accumulate) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long k = slot[first + i];
  if (k < 0) return;
  double re = 0, im = 0;
  for (int c = 0; c < nchunk; ++c) {
    const double2 v = part[static_cast<long long>(c) * Ks + first + i];
    re += v.x;
    im += v.y;
  }
  unbias(re, im);                                  // evaluated terms; the interpolated ones are
  for (int c = 0; c < nv; ++c) {
    const double2 v = vacc[c * vstride + i];
    re += v.x;
    im += v.y;
  }
  if (accumulate) {
    const float2 o = V[k];
    re += o.x;
    im += o.y;
  }
  V[k] = make_float2(static_cast<float>(re), static_cast<float>(im));
}

// -------------------------------------------------------------- remainder
struct TrackRestParams {
  const double4 *samp;         // slots
  const int *slot;
  const int4 *refs;            // null: unocculted
  const double4 *occ;
  const float4 *occ32;
  const double4 *pix;          // forward: pixel + sky records of channel 0; adjoint: pixel records
  const float4 *cones;
  TrackBits bits;
  int ntiles, use_off;
  long long pix_stride;        // forward: records per channel
  int nbc;                     // blocks per channel
  int len;                     // slots of a block that can hold a sample (the first ones)
  int per_chunk;               // forward: tiles, adjoint: blocks (a multiple of 32)
  int nchunk;
  long long Ks, Jpad;
  double2 *part_fwd;           // [chunk][Ks]
  double *part_adj;            // [channel][chunk][Jpad]
  const float2 *coef;          // adjoint: slots
  unsigned long long *counter;
};

constexpr int kRestNT = 128;

// Forward remainder: a warp owns 32 slots of one block (a CTA the block's
// four), walks the tiles its rest row names, and evaluates for each the
// 32-pixel sub-tiles that any of its samples needs, as the mixed path of
// k_forward does.  Warps are independent (no stage ring): which tiles a warp
// needs differs from warp to warp, so shared staging made each wait for all.
template <bool MASKED>
__global__ void __launch_bounds__(kRestNT, 8) k_track_fwd_rest(const TrackRestParams p) {
  __shared__ double4 s_pix[kRestNT / 32][kSubPix];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, b = blockIdx.x;
  double4 *px = s_pix[warp];
  const long long i = static_cast<long long>(b) * kTrackT + threadIdx.x;
  const bool valid = p.slot[i] >= 0;
  const double4 u = p.samp[i];
  const double off = p.use_off ? u.w : 0.0, mk = kMagic + off, mk2 = kMagic + 0.5 + off;
  int4 rf = make_int4(-1, -1, -1, -1);
  if (MASKED) rf = p.refs[i];
  const double4 *pix = p.pix + static_cast<long long>(b / p.nbc) * p.pix_stride;
  const long long row = p.bits.row(b);
  const int t0 = blockIdx.y * p.per_chunk, t1 = min(t0 + p.per_chunk, p.ntiles);
  float sr = 0.f, cr = 0.f, si = 0.f, ci = 0.f;    // Kahan sums
  double d0 = 0, d1 = 0;
  unsigned long long evaluated = 0, mixed = 0;
  if (__any_sync(0xffffffffu, valid)) {
    for (int w = t0 / 32; w * 32 < t1; ++w) {
      const unsigned taken = p.bits.full[row + w] | (p.bits.part ? p.bits.part[row + w] : 0u);
      for (unsigned todo = p.bits.rest[row + w]; todo; todo &= todo - 1) {
        const int bit = __ffs(todo) - 1, t = 32 * w + bit;
        int code = 0;
        if (valid) {
          code = MASKED ? sample_state(rf, p.cones[t], p.occ32) : 2;
          if ((taken >> bit) & 1u && (code & 3) == 2) code = 0;      // interpolated
        }
        if (__all_sync(0xffffffffu, (code & 3) == 0)) continue;
        double4 q0, q1, q2;
        unsigned ss = (code & 3) == 2 ? 0xAAu : 0u;  // 2 bits per sub-tile, as the state
        int nr = 0;
        if (MASKED) {
          float4 f0, f1, f2;
          nr = needed_rows(rf, (code & 3) == 1 ? code : 0, p.occ, p.occ32, q0, q1, q2, f0, f1, f2);
          if ((code & 3) == 1) {
            const float4 *sub = p.cones + p.ntiles + 4LL * t;
#pragma unroll
            for (int s = 0; s < 4; ++s) ss |= static_cast<unsigned>(rows_state(sub[s], nr, f0, f1, f2)) << (2 * s);
          }
        }
        float re = 0.f, im = 0.f;
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
          const unsigned st = (ss >> (2 * s)) & 3u;
          const unsigned seen = __ballot_sync(0xffffffffu, st != 0);
          if (seen == 0) continue;
          const int wn = MASKED ? __reduce_max_sync(0xffffffffu, st == 1 ? nr : 0) : 0;
          __syncwarp();
          px[lane] = pix[static_cast<long long>(t) * kTilePix + s * kSubPix + lane];
          __syncwarp();
          evaluated += static_cast<unsigned>(__popc(seen) * kSubPix);
          if (wn) mixed += static_cast<unsigned>(__popc(seen) * kSubPix);
          if (st == 0) continue;
          if (wn == 0) fwd_span<0, false>(px, u.x, u.y, u.z, mk, mk2, q0, q1, q2, re, im, d0, d1);
          else if (wn == 1) fwd_span<1, false>(px, u.x, u.y, u.z, mk, mk2, q0, q1, q2, re, im, d0, d1);
          else if (wn == 2) fwd_span<2, false>(px, u.x, u.y, u.z, mk, mk2, q0, q1, q2, re, im, d0, d1);
          else fwd_span<3, false>(px, u.x, u.y, u.z, mk, mk2, q0, q1, q2, re, im, d0, d1);
        }
        kahan_add(sr, cr, re);
        kahan_add(si, ci, im);
      }
    }
  }
  if (lane == 0) {
    if (evaluated) atomicAdd(p.counter, evaluated);
    if (mixed) atomicAdd(p.counter + 2, mixed);
  }
  p.part_fwd[blockIdx.y * p.Ks + i] = make_double2(static_cast<double>(sr) - static_cast<double>(cr),
                                                   static_cast<double>(si) - static_cast<double>(ci));
}

// Adjoint remainder: a warp owns one pixel tile (4 pixels per lane) and walks
// the blocks whose rest row names it.  Its lanes classify 32 samples at a time
// and put those the tile needs, with their exact rows, into the warp's list in
// shared memory (so 32 row fetches overlap); the list is then processed sample
// by sample, as the mixed path of k_adjoint does.
struct AdjRestList {
  double4 u[32];               // .w: phase constant
  double4 q[3][32];
  float2 c[32];
  unsigned meta[32];           // hidden sub-tiles | rows to test << 8
};

template <bool MASKED>
__global__ void __launch_bounds__(kRestNT, 6) k_track_adj_rest(const TrackRestParams p) {
  constexpr int P = 4;
  __shared__ AdjRestList s_list[kRestNT / 32];
  __shared__ float4 s_sub[kRestNT / 32][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  AdjRestList &L = s_list[warp];
  const int t = static_cast<int>(blockIdx.x) * (kRestNT / 32) + warp;
  if (t >= p.ntiles) return;                       // no block-wide synchronisation below
  const long long pbase = static_cast<long long>(t) * kTilePix;
  double sx[P], sy[P], sz[P];
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const double4 v = p.pix[pbase + q * 32 + lane];
    sx[q] = v.x; sy[q] = v.y; sz[q] = v.z;
  }
  const float4 cone = p.cones[t];
  if (lane < 4) s_sub[warp][lane] = p.cones[p.ntiles + 4LL * t + lane];
  __syncwarp();
  const int ch = blockIdx.y / p.nchunk, chunk = blockIdx.y - ch * p.nchunk;
  const int b0 = ch * p.nbc + chunk * p.per_chunk, b1 = min(b0 + p.per_chunk, (ch + 1) * p.nbc);
  const bool odd_lane = (lane & 1) != 0;
  const double half = odd_lane ? 0.5 : 0.0;
  float ks[P], kc[P];
#pragma unroll
  for (int q = 0; q < P; ++q) ks[q] = kc[q] = 0.f;
  double dacc[P];
  unsigned long long evaluated = 0, mixed = 0;
  for (int base = b0; base < b1; base += 32) {
    bool need = false, took = false;
    if (base + lane < b1) {
      const long long at = p.bits.row(base + lane) + (t >> 5);
      need = (p.bits.rest[at] >> (t & 31)) & 1u;
      took = need && (((p.bits.full[at] | (p.bits.part ? p.bits.part[at] : 0u)) >> (t & 31)) & 1u);
    }
    const unsigned taken = __ballot_sync(0xffffffffu, took);
    for (unsigned todo = __ballot_sync(0xffffffffu, need); todo; todo &= todo - 1) {
      const int bi = __ffs(todo) - 1;
      float acc[P];
#pragma unroll
      for (int q = 0; q < P; ++q) acc[q] = 0.f;
#pragma unroll 1
      for (int g = 0; g < p.len; g += 32) {
        const long long i = static_cast<long long>(base + bi) * kTrackT + g + lane;
        int code = 0;
        int4 rf = make_int4(-1, -1, -1, -1);
        if (p.slot[i] >= 0) {
          code = 2;
          if (MASKED) {
            rf = p.refs[i];
            code = sample_state(rf, cone, p.occ32);
          }
          if ((taken >> bi) & 1u && (code & 3) == 2) code = 0;      // interpolated
        }
        unsigned meta = 0;
        int i0 = -1, i1 = -1, i2 = -1;
        if (MASKED && (code & 3) == 1) {
          const int nr = needed_idx(rf, code, i0, i1, i2);
          float4 f0, f1, f2;
          class_rows(p.occ32, i0, i1, i2, f0, f1, f2);
          unsigned hid = 0, mix = 0;
#pragma unroll
          for (int q = 0; q < P; ++q) {
            const int ss = rows_state(s_sub[warp][q], nr, f0, f1, f2);
            hid |= static_cast<unsigned>(ss == 0) << q;
            mix |= static_cast<unsigned>(ss == 1) << q;
          }
          if (hid == (1u << P) - 1) code = 0;
          meta = hid | (mix ? static_cast<unsigned>(nr) << 8 : 0u);
        }
        const unsigned live = __ballot_sync(0xffffffffu, (code & 3) != 0);
        if (live == 0) continue;
        if ((code & 3) != 0) {
          const int at = __popc(live & ((1u << lane) - 1u));
          double4 u = p.samp[i];
          u.w = kMagic + (p.use_off ? u.w : 0.0);
          L.u[at] = u;
          L.c[at] = unbias_coef(p.coef[i]);
          L.meta[at] = meta;
          if (meta >> 8) exact_rows(p.occ, i0, i1, i2, L.q[0][at], L.q[1][at], L.q[2][at]);
        }
        const int n = __popc(live);
        evaluated += static_cast<unsigned>(n * kTilePix);
        mixed += static_cast<unsigned>(__popc(__ballot_sync(0xffffffffu, (code & 3) != 0 && (meta >> 8))) * kTilePix);
        __syncwarp();
        for (int e = 0; e < n; ++e) {
          const double4 u = L.u[e];
          const float2 c = L.c[e];
          const unsigned m = L.meta[e], hid = m & 0xffu, nr = m >> 8;
          const double mm = u.w + half;
          if (nr == 0)
            adj_sample<P, 0, false>(u, mm, c, sx, sy, sz, u, u, u, hid, acc, dacc);
          else if (nr == 1)
            adj_sample<P, 1, false>(u, mm, c, sx, sy, sz, L.q[0][e], u, u, hid, acc, dacc);
          else if (nr == 2)
            adj_sample<P, 2, false>(u, mm, c, sx, sy, sz, L.q[0][e], L.q[1][e], u, hid, acc, dacc);
          else
            adj_sample<P, 3, false>(u, mm, c, sx, sy, sz, L.q[0][e], L.q[1][e], L.q[2][e], hid, acc, dacc);
        }
        __syncwarp();
      }
#pragma unroll
      for (int q = 0; q < P; ++q) kahan_add(ks[q], kc[q], acc[q]);
    }
  }
  if (lane == 0) {
    if (evaluated) atomicAdd(p.counter, evaluated);
    if (mixed) atomicAdd(p.counter + 2, mixed);
  }
  double *out = p.part_adj + static_cast<long long>(blockIdx.y) * p.Jpad + pbase;
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const double sum = static_cast<double>(ks[q]) - static_cast<double>(kc[q]);
    out[q * 32 + lane] = odd_lane ? -sum : sum;
  }
}

// ---------------------------------------------------------------- adjoint
__global__ void k_track_coef(long long Ks, const int *slot, const float2 *coef, const unsigned *peak, float2 *out) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= Ks) return;
  const int k = slot[i];
  const float scale = scale_of(peak_exponent(peak));
  out[i] = k >= 0 ? make_float2(scale * coef[k].x, scale * coef[k].y) : make_float2(0.f, 0.f);
}

constexpr int kAdjUnits = 64;          // units per pass, adjoint: 128 rows of the product (re, then im)
constexpr int kAdjStep = 16;           // samples staged at a time
constexpr int kAdjLboA = 2 * kAdjUnits * 16 + 16;

// Shared memory of the adjoint interpolation for blocks of rank r, and its
// tensor memory: the hi hi products of three runs of samples (the accumulator
// truncates: 48 samples at most in one), and the small products.
constexpr int kAdjRuns = 3, kAdjRun = 3;    // runs; steps per run
struct AdjInterpSmem {
  int np, lbo_b, a, b, un, units, list, total;
  uint32_t cols;
  __host__ __device__ explicit AdjInterpSmem(int r) {
    np = round_up(r, 16);
    lbo_b = np * 16 + 16;
    cols = np <= 16 ? 64 : (np <= 32 ? 128 : (np <= 64 ? 256 : 512));
    a = 0;                                           // [2 buffers] hi, lo; the sums of a pass after it
    const int sa = 4 * (kAdjStep / 4) * kAdjLboA, sd = 2 * kAdjUnits * (np + 1) * static_cast<int>(sizeof(float));
    b = a + round_up(sa > sd ? sa : sd, 128);        // P^T: hi, lo
    un = b + 2 * (kTrackT / 4) * lbo_b;
    units = un + r * static_cast<int>(sizeof(double4));
    list = units + 2 * kAdjUnits * static_cast<int>(sizeof(PassUnit));
    total = list + 2 * kChunkTiles * static_cast<int>(sizeof(int2));
  }
};

// Node coefficients b_n of one block for a chunk of tiles, kAdjUnits units a
// pass: kAdjStep samples at a time, their coefficients times e^{2 pi i (u_k.s_g +
// off_k)}, split, into shared memory (double buffered) and through the tensor core
// into (unit, node) sums; at the end of the pass those times e^{-2 pi i u_n.s_g}.
// Bound like the forward by the phases, about 60 slots per (sample, unit).
template <bool PART>
__global__ void __launch_bounds__(kInterpNT, 3) k_track_adj_interp(const TrackInterpParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) uint64_t s_done[2];
  const int b = p.b0 + blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = p.rank[b];
  const int n0 = p.noff[b];
  const AdjInterpSmem at(r);
  unsigned char *A = smem + at.a, *B = smem + at.b;
  double4 *un = reinterpret_cast<double4 *>(smem + at.un);
  PassUnit *units = reinterpret_cast<PassUnit *>(smem + at.units);          // [2][kAdjUnits]
  int2 *list = reinterpret_cast<int2 *>(smem + at.list);
  const int sb = (kTrackT / 4) * at.lbo_b;
  if (warp == 0) tmem_alloc(&s_tmem, at.cols);
  if (tid == 0) {
    mbar_init(&s_done[0], 1);
    mbar_init(&s_done[1], 1);
    fence_mbar_init();
  }
  for (int n = tid; n < r; n += kInterpNT) un[n] = p.node[n0 + n];
  for (int i = tid; i < at.np * kTrackT; i += kInterpNT) {
    const int n = i / kTrackT, k = i % kTrackT, o = umma_offset(n, k, at.lbo_b);
    float hi = 0.f, lo = 0.f;
    if (n < r) split_tf32(p.P[static_cast<long long>(n0 + n) * kTrackT + k], hi, lo);
    *reinterpret_cast<float *>(B + o) = hi;
    *reinterpret_cast<float *>(B + sb + o) = lo;
  }
  const int t0 = blockIdx.y * p.per_chunk, t1 = min(t0 + p.per_chunk, p.ntiles);
  const int count = list_units(p.bits, b, p.cls, t0, t1, list);             // synchronises
  auto prepare = [&](int base, int buf) {
    if (tid < kAdjUnits)
      units[buf * kAdjUnits + tid] = base + tid < count ? pass_unit(p, list[base + tid]) : PassUnit{};
  };
  prepare(0, 0);
  umma_fence_before();
  __syncthreads();
  umma_fence_after();
  const uint32_t tmem = s_tmem, idesc = umma_idesc_tf32(at.np);
  // four units (rows unit0 + j of the operand, and kAdjUnits further for im), one sample of the step
  const int unit0 = warp * 8 + 4 * (lane >> 4), ks = lane & (kAdjStep - 1), own_o = umma_offset(unit0, ks, kAdjLboA);
  const long long slot0 = static_cast<long long>(b) * kTrackT + ks;
  double4 u = p.samp[slot0];
  float2 a = p.coef[slot0];
  const bool drop = p.drop && blockIdx.x == 0 && blockIdx.y == 0;
  int step = 0;                                    // products issued
  bool ok = true;
  for (int base = 0, buf = 0; base < count; base += kAdjUnits, buf ^= 1) {
    const int nu = min(kAdjUnits, count - base);
    const PassUnit *pu = units + buf * kAdjUnits;
    for (int s = 0; s < kTrackT / kAdjStep; ++s, ++step) {
      unsigned char *An = A + (step & 1) * 2 * (kAdjStep / 4) * kAdjLboA;
      // the buffer's last product (two steps ago)
      if (s >= 2) ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&s_done[step & 1], ((step >> 1) + 1) & 1));
      const int k = s * kAdjStep + ks;
      const double phase0 = kFine + (p.use_off ? u.w : 0.0);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const PassUnit &g = pu[unit0 + j];
        const float2 c = fine_cis(fine_phase(u.x, u.y, u.z, g, phase0));
        float2 v = make_float2(a.x * c.x - a.y * c.y, a.x * c.y + a.y * c.x);
        if (PART && !((g.seen[k >> 5] >> (k & 31)) & 1u)) v = make_float2(0.f, 0.f);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned char *o = An + own_o + j * 16 + h * (kAdjUnits / 8) * 128;
          float hi, lo;
          split_tf32(h ? v.y : v.x, hi, lo);
          *reinterpret_cast<float *>(o) = hi;
          *reinterpret_cast<float *>(o + (kAdjStep / 4) * kAdjLboA) = lo;
        }
      }
      // the next step's sample (cyclic: the next pass starts over)
      const long long ahead = slot0 + ((s + 1) & (kTrackT / kAdjStep - 1)) * kAdjStep;
      u = p.samp[ahead];
      a = p.coef[ahead];
      if (s == 0) prepare(base + kAdjUnits, buf ^ 1);
      fence_async_smem();
      umma_fence_before();
      if (broken(ok)) {
        ok = false;
        break;
      }
      umma_fence_after();
      if (tid == 0) {
        const uint32_t ah = smem_addr(An), al = ah + (kAdjStep / 4) * kAdjLboA;
        const uint32_t bh = smem_addr(B) + s * (kAdjStep / 4) * at.lbo_b, bl = bh + sb;
        const uint32_t dh = tmem + s / kAdjRun * at.np, dl = tmem + kAdjRuns * at.np;
        const bool first = s % kAdjRun == 0;
#pragma unroll
        for (int q = 0; q < kAdjStep / 8; ++q) {
          const uint64_t dah = umma_desc(ah + 2 * q * kAdjLboA, kAdjLboA), dal = umma_desc(al + 2 * q * kAdjLboA, kAdjLboA);
          const uint64_t dbh = umma_desc(bh + 2 * q * at.lbo_b, at.lbo_b), dbl = umma_desc(bl + 2 * q * at.lbo_b, at.lbo_b);
          umma_tf32(dl, dah, dbl, idesc, s > 0 || q > 0);
          umma_tf32(dl, dal, dbh, idesc, true);
          umma_tf32(dh, dah, dbh, idesc, !first || q > 0);
        }
        if (step > 0 || !drop) umma_commit(&s_done[step & 1]);
      }
    }
    if (!ok) break;                                // at a barrier of the steps: the same for all
    // the pass's last two products (the commit of the last covers both buffers' reads)
    ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&s_done[step & 1], ((step >> 1) + 1) & 1));
    ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&s_done[(step + 1) & 1], (((step + 1) >> 1) + 1) & 1));
    umma_fence_after();
    // rows (re of unit q, im of unit q at kAdjUnits + q) to shared memory, over the operand
    float *red = reinterpret_cast<float *>(A);       // [2 kAdjUnits][np + 1]
    const int row = (warp & 3) * 32 + lane;
    const uint32_t my = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    if (broken(ok)) {
      ok = false;
      break;
    }
    for (int c = (warp >> 2) * 16; c < at.np; c += 32) {
      float sum[16], d[16];
      tmem_load16(my + c, sum);
#pragma unroll
      for (int q = 1; q <= kAdjRuns; ++q) {
        tmem_load16(my + q * at.np + c, d);
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] += d[i];
      }
#pragma unroll
      for (int i = 0; i < 16; ++i) red[row * (at.np + 1) + c + i] = sum[i];
    }
    umma_fence_before();
    __syncthreads();
    umma_fence_after();
    // thread = unit and every fourth node: four neighbours write one 32-byte sector
    const int q = tid >> 2;
    if (q < nu) {
      const PassUnit &g = pu[q];
      const double gx = g.x, gy = g.y, gz = g.z;
      float2 *out = p.sums + g.row * p.ld + (n0 - p.n0);
      const float *sre = red + q * (at.np + 1), *sim = red + (kAdjUnits + q) * (at.np + 1);
      const float scale = interp_scale(r, true);
      for (int n = tid & 3; n < r; n += 4) {
        const double4 w = un[n];
        const float2 c = fine_cis(fma(w.z, gz, fma(w.y, gy, fma(w.x, gx, kFine))));
        const float re = sre[n] * c.x + sim[n] * c.y, im = sim[n] * c.x - sre[n] * c.y;
        const float sign = ((n0 - p.n0 + n) & 32) ? -1.f : 1.f;   // half a turn on (k_track_adj_nodes)
        out[n] = make_float2(sign * fmaf(scale, re, re), sign * fmaf(scale, im, im));
      }
    }
    __syncthreads();
  }
  if (!ok) {
    if (lane == 0) atomicOr(p.err, kErrTimeout);
    drain_products(s_done, step);
  }
  umma_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free(tmem, at.cols);
}

// Images of the node coefficients: the fast loop and the stage ring of
// k_adjoint.  A warp owns two tiles (8 pixels per lane), a CTA eight; beside
// the node records a stage holds their coefficients for the CTA's units.
constexpr int kAdjNodeNT = 128;
constexpr int kAdjNodeTile = 128;    // nodes per stage

template <bool HALF>
struct AdjNodeStage {
  double4 node[kAdjNodeTile];
  float2 coef[HALF ? 16 : 8][kAdjNodeTile];
};

template <bool HALF>
__global__ void __launch_bounds__(kAdjNodeNT, 4) k_track_adj_nodes(const TrackNodeParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int S = HALF ? 2 : 3, P = 8, NT = kAdjNodeNT, U = HALF ? 16 : 8;
  AdjNodeStage<HALF> *stages = reinterpret_cast<AdjNodeStage<HALF> *>(smem);
  __shared__ float s_kahan[2][P][NT];
  __shared__ __align__(8) uint64_t s_full[S], s_empty[S];
  __shared__ int s_abort;
  volatile int *abort_flag = &s_abort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ctile = static_cast<int>(blockIdx.x) * 8, t = ctile + 2 * warp;   // Jpad: an even tile count
  const bool tile_ok = t < p.ntiles;
  const long long pbase = static_cast<long long>(t) * kTilePix;
  double sx[P], sy[P], sz[P];
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const double4 v = tile_ok ? p.pix[pbase + q * 32 + lane] : make_double4(0, 0, 1, 0);
    sx[q] = v.x; sy[q] = v.y; sz[q] = v.z;
    s_kahan[0][q][tid] = s_kahan[1][q][tid] = 0.f;
  }
  const int n0 = blockIdx.y * p.per_chunk, n1 = min(n0 + p.per_chunk, p.nn);
  const int ntile = max(0, (n1 - n0 + kAdjNodeTile - 1) / kAdjNodeTile);
  const int unit0 = HALF ? 2 * ctile : ctile, units = min(U, (HALF ? 2 : 1) * (p.ntiles - ctile));
  const int group_unit = p.cls == 2 ? 2 * warp : 0;   // a merged group's unit, for both of the warp's tiles
  const int drop = (blockIdx.x == 0 && blockIdx.y == 0) ? min(p.drop_tile, ntile - 1) : -1;   // test hook (k_forward)
  auto issue = [&](int i, int stage) {
    if (i == drop) return;
    const int at = n0 + i * kAdjNodeTile, n = min(kAdjNodeTile, n1 - at), ne = (n + 1) & ~1;   // ld is even
    mbar_expect_tx(&s_full[stage], n * 32u + units * ne * 8u);
    bulk_g2s(stages[stage].node, p.node + at, n * 32u, &s_full[stage]);
    for (int g = 0; g < units; ++g)
      bulk_g2s(stages[stage].coef[g], p.sums + static_cast<long long>(unit0 + g) * p.ld + at, ne * 8u, &s_full[stage]);
  };
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < S; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], NT / 32);
    }
    fence_mbar_init();
    s_abort = 0;
  }
  __syncthreads();
  const bool odd_lane = (lane & 1) != 0;             // half a turn on, negated at the end (k_adjoint)
  const double magic = odd_lane ? kTurn32 + 0.5 : kTurn32;
  static_assert(kNodeRun == 32, "a run is a group of nodes below");
  unsigned long long evaluated = 0;
  int next = 0;
  for (int it = 0; it < ntile; ++it) {
    const int buf = it % S;
    if (tid == 0 && !ring_refill<S>(s_empty, next, it, ntile, issue)) {
      atomicOr(p.err, kErrTimeout);
      *abort_flag = 1;
    }
    if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
    const int at = n0 + it * kAdjNodeTile, n = min(kAdjNodeTile, n1 - at);
    // per node (lane of group g): bits 0, 1 the warp's two tiles have nodes, bit 2 both in a merged group
    unsigned three[kAdjNodeTile / 32];
#pragma unroll
    for (int g = 0; g < kAdjNodeTile / 32; ++g) {
      const int i = 32 * g + lane;
      const int blk = (tile_ok && i < n) ? p.nodeblk[at + i] : -1;
      three[g] = 0;
      if (blk >= 0) {
        const long long w = p.bits.row(blk) + (t >> 5);
        const unsigned on = p.bits.full[w] | (p.bits.part ? p.bits.part[w] : 0u);
        three[g] = ((on >> (t & 31)) & 3u) | (((p.bits.merged[w] >> (t & 31)) & 1u) << 2);
      }
    }
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&s_full[buf], static_cast<uint32_t>(it / S) & 1u))) {
      if (lane == 0) atomicOr(p.err, kErrTimeout);
      *abort_flag = 1;
      break;
    }
    const AdjNodeStage<HALF> &st = stages[buf];
    float acc[P], sum[P];
#pragma unroll
    for (int q = 0; q < P; ++q) sum[q] = 0.f;
    double from = magic;
    auto term = [&](int q, const double4 &u, const float2 &c) {
      float sn, cs;
      sfu_sincos(turn_angle32(fma(u.z, sz[q], fma(u.y, sy[q], fma(u.x, sx[q], from)))), sn, cs);
      acc[q] = fmaf(-c.y, sn, fmaf(c.x, cs, acc[q]));
    };
#pragma unroll 1
    for (int g = 0; g < kAdjNodeTile / 32; ++g) {
      unsigned b3 = three[0];
#pragma unroll
      for (int q = 1; q < kAdjNodeTile / 32; ++q) b3 = g == q ? three[q] : b3;
      const unsigned m0 = __ballot_sync(0xffffffffu, b3 & 1u), m1 = __ballot_sync(0xffffffffu, b3 & 2u);
      const unsigned mg = HALF ? 0u : __ballot_sync(0xffffffffu, b3 & 4u);
      // every other 32 nodes half a turn on, their coefficients negated: an SFU error that
      // the terms of a coherent sum share cancels (as k_forward's over pixels; odd lanes alone
      // do not do it for one pixel's sum).  Images of 1 MHz observations: 3.7-4.2e-7 of error
      // -> 2.2-2.5e-7, for 1.3 % of the 10 MHz adjoint's time.
      from = (g & 1) ? magic + 0.5 : magic;
#pragma unroll
      for (int q = 0; q < P; ++q) acc[q] = 0.f;
      evaluated += static_cast<unsigned>(__popc(m0) + __popc(m1)) * static_cast<unsigned>(kTilePix);
      for (unsigned m = m0 & m1; m; m &= m - 1) {
        const int j = __ffs(m) - 1, i = 32 * g + j;
        const double4 u = st.node[i];
        if (HALF) {
          const float2 c0 = st.coef[4 * warp][i], c1 = st.coef[4 * warp + 1][i], c2 = st.coef[4 * warp + 2][i],
                       c3 = st.coef[4 * warp + 3][i];
#pragma unroll
          for (int q = 0; q < P; ++q) term(q, u, q < 2 ? c0 : (q < 4 ? c1 : (q < 6 ? c2 : c3)));
        } else {
          const bool grp = (mg >> j) & 1u;
          const float2 c0 = st.coef[grp ? group_unit : 2 * warp][i], c1 = st.coef[grp ? group_unit : 2 * warp + 1][i];
#pragma unroll
          for (int q = 0; q < P; ++q) term(q, u, q < 4 ? c0 : c1);
        }
      }
      for (unsigned m = m0 & ~m1; m; m &= m - 1) {   // the first tile only
        const int j = __ffs(m) - 1, i = 32 * g + j;
        const double4 u = st.node[i];
        const float2 c0 = st.coef[HALF ? 4 * warp : ((mg >> j) & 1u ? group_unit : 2 * warp)][i];
        const float2 c1 = HALF ? st.coef[4 * warp + 1][i] : c0;
#pragma unroll
        for (int q = 0; q < 4; ++q) term(q, u, q < 2 ? c0 : c1);
      }
      for (unsigned m = m1 & ~m0; m; m &= m - 1) {   // the second
        const int i = 32 * g + __ffs(m) - 1;
        const double4 u = st.node[i];
        const float2 c0 = st.coef[HALF ? 4 * warp + 2 : 2 * warp + 1][i];
        const float2 c1 = HALF ? st.coef[4 * warp + 3][i] : c0;
#pragma unroll
        for (int q = 4; q < 8; ++q) term(q, u, q < 6 ? c0 : c1);
      }
#pragma unroll
      for (int q = 0; q < P; ++q) sum[q] += acc[q];
    }
#pragma unroll
    for (int q = 0; q < P; ++q) {
      float s = s_kahan[0][q][tid], c = s_kahan[1][q][tid];
      kahan_add(s, c, sum[q]);
      s_kahan[0][q][tid] = s;
      s_kahan[1][q][tid] = c;
    }
    ring_release(s_empty, buf);
  }
  if (tid == 0) ring_drain<S>(s_full, next);
  if (lane == 0 && evaluated) atomicAdd(p.counter, evaluated);
  if (!tile_ok) return;
  double *out = p.part + static_cast<long long>(blockIdx.y) * p.Jpad;
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const double sum = static_cast<double>(s_kahan[0][q][tid]) - static_cast<double>(s_kahan[1][q][tid]);
    out[pbase + q * 32 + lane] += odd_lane ? -sum : sum;
  }
}

// One channel's image: node chunks + remainder chunks (FP64).
__global__ void k_track_reduce_adj(long long J, long long Jpad, int nnode, const double *node, int nrest,
                                   const double *rest, const int *perm, const unsigned *peak, float scale, float *img,
                                   int accumulate) {
  const long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= J) return;
  double s = 0;
  for (int c = 0; c < nnode; ++c) s += node[static_cast<long long>(c) * Jpad + i];
  for (int c = 0; c < nrest; ++c) s += rest[static_cast<long long>(c) * Jpad + i];
  s *= static_cast<double>(scale) * unscale_of(peak_exponent(peak));
  const long long j = perm[i];
  if (accumulate) s += static_cast<double>(img[j]);
  img[j] = static_cast<float>(s);
}

}  // namespace

namespace {

TrackRestParams rest_params(const TrackState &S, const TrackInputs &in, bool masked, bool use_off,
                            unsigned long long *counter) {
  TrackRestParams rp{};
  rp.samp = S.samp;
  rp.slot = S.slot;
  rp.refs = masked ? S.refs : nullptr;
  rp.occ = in.occ;
  rp.occ32 = in.occ32;
  rp.cones = in.cones;
  rp.bits = S.bits(masked);
  rp.ntiles = in.ntiles;
  rp.use_off = use_off;
  rp.pix_stride = in.Jpad;
  rp.nbc = S.shape.blocks_per_channel();
  rp.len = S.shape.len;
  rp.Ks = S.Ks;
  rp.Jpad = in.Jpad;
  rp.counter = counter;
  return rp;
}

TrackInterpParams interp_params(const TrackState &S, const TrackInputs &in, const TrackSlab &sl, bool masked,
                                bool use_off, int &drop_tile) {
  TrackInterpParams ip{};
  ip.drop = drop_tile >= kDropProduct;
  if (ip.drop) drop_tile = -1;
  ip.samp = S.samp;
  ip.slot = S.slot;
  ip.refs = masked ? S.refs : nullptr;
  ip.occ32 = in.occ32;
  ip.cones = in.cones;
  ip.node = S.node;
  ip.rank = S.rank;
  ip.noff = S.noff;
  ip.P = S.P;
  ip.bits = S.bits(masked);
  ip.gcen[0] = S.gcen + S.gat[kHalf];
  ip.gcen[1] = S.gcen + S.gat[kTile];
  ip.gcen[2] = S.gcen + S.gat[sl.cls];
  ip.cls = sl.cls;
  ip.ntiles = in.ntiles;
  ip.b0 = sl.b0;
  ip.n0 = sl.n0;
  ip.ld = S.ld_max / (sl.cls == kHalf ? 2 : 1);
  ip.sums = S.sums;
  ip.peak = S.peak;
  ip.use_off = use_off;
  return ip;
}

// Tiles per interpolation chunk: about 16 CTAs per SM in all.
int interp_tiles(const TrackInputs &in, int nblk) {
  const int y = std::max(1, (16 * in.nsm + nblk - 1) / nblk);
  return std::min(kChunkTiles, std::max(64, (in.ntiles + y - 1) / y + 31) / 32 * 32);
}

TrackNodeParams node_params(const TrackState &S, const TrackInputs &in, const TrackSlab &sl, bool masked,
                            unsigned long long *counter, int *err, int &drop_tile) {
  TrackNodeParams np{};
  np.node = S.node + sl.n0;
  np.nodeblk = S.nodeblk + sl.n0;
  np.bits = S.bits(masked);
  np.cls = sl.cls;
  np.ntiles = in.ntiles;
  np.nn = sl.n1 - sl.n0;
  np.ld = S.ld_max / (sl.cls == kHalf ? 2 : 1);
  np.sums = S.sums;
  np.peak = S.peak;
  np.Jpad = in.Jpad;
  np.counter = counter;
  np.err = err;
  if (drop_tile < kDropProduct) {
    np.drop_tile = drop_tile;
    drop_tile = -1;
  } else {
    np.drop_tile = -1;
  }
  return np;
}

}  // namespace

namespace {

// A call's sums: in the caller's workspace if they fit, else in the blocks' own (at:
// null without memory).
struct TrackCut {
  char *at;
  template <class T>
  void take(T *&p, size_t n) {
    p = reinterpret_cast<T *>(at);
    at += TrackArena::bytes<T>(n);
  }
};
TrackCut call_sums(TrackState &S, const TrackInputs &in, size_t bytes) {
  if (in.work && bytes <= in.work_bytes) return {static_cast<char *>(in.work)};
  return {S.call.reset(bytes) ? S.call.base : nullptr};
}

int find_peak(const TrackState &S, long long n, const double4 *pixsky, const float2 *coef, int nsm, cudaStream_t st) {
  TRACK_CUDA(cudaMemsetAsync(S.peak, 0, sizeof(unsigned), st), "peak");
  k_track_peak<<<std::min<long long>(blks(n, 256), 8LL * nsm), 256, 0, st>>>(n, pixsky, coef, S.peak);
  TRACK_CUDA(cudaGetLastError(), "peak");
  return 0;
}

}  // namespace

int tracks_forward(void *state, const TrackInputs &in, const double4 *pixsky, float2 *V, bool masked,
                   bool use_off, bool accumulate, unsigned long long *counter, int *err, int drop_tile,
                   cudaStream_t st) {
  TrackState &S = *static_cast<TrackState *>(state);
  size_t vacc = 0;
  for (const TrackSlab &sl : S.slabs)
    vacc = std::max(vacc, static_cast<size_t>(blks(in.ntiles, interp_tiles(in, sl.b1 - sl.b0))) * (sl.b1 - sl.b0) * kTrackT);
  // the remainder: CTAs of one block and a chunk of tiles, small enough that a
  // block without nodes (every tile) does not outlast the others
  const int y = std::max(8, std::min((16 * in.nsm + S.nb - 1) / S.nb, S.W));
  const int per = ((in.ntiles + y - 1) / y + 31) / 32 * 32;
  const int nrest = S.has_rest[masked] ? static_cast<int>(blks(in.ntiles, per)) : 0;
  double2 *vacc_d, *rest_d;
  TrackCut sums = call_sums(S, in, TrackArena::bytes<double2>(vacc) +
                                       TrackArena::bytes<double2>(static_cast<size_t>(nrest) * S.Ks));
  if (!sums.at) return record_error(-3, "viss_forward: device allocation failed (track block sums)");
  sums.take(vacc_d, vacc);
  sums.take(rest_d, static_cast<size_t>(nrest) * S.Ks);
  if (int e = find_peak(S, in.channels * in.Jpad, pixsky, nullptr, in.nsm, st)) return e;
  if (nrest) {
    TrackRestParams rp = rest_params(S, in, masked, use_off, counter);
    rp.pix = pixsky;
    rp.per_chunk = per;
    rp.part_fwd = rest_d;
    if (masked) k_track_fwd_rest<true><<<dim3(S.nb, nrest), kRestNT, 0, st>>>(rp);
    else k_track_fwd_rest<false><<<dim3(S.nb, nrest), kRestNT, 0, st>>>(rp);
    TRACK_CUDA(cudaGetLastError(), "remainder");
  }
  const auto interp = masked ? k_track_fwd_interp<true> : k_track_fwd_interp<false>;
  TRACK_CUDA(cudaFuncSetAttribute(interp, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  FwdInterpSmem(kTrackRankMax).total), "attributes");
  for (const TrackSlab &sl : S.slabs) {
    const int nblk = sl.b1 - sl.b0;
    const long long slots = static_cast<long long>(nblk) * kTrackT;
    int nv = 0;
    if (sl.cls < kClasses) {
      TrackNodeParams np = node_params(S, in, sl, masked, counter, err, drop_tile);
      np.pix = pixsky + static_cast<long long>(sl.ch) * in.Jpad;
      const unsigned gx = blks(np.nn, kNodeNT * kNodeR);
      const int want = std::max(1, static_cast<int>(10LL * 2 * in.nsm / gx));
      np.per_chunk = ((in.ntiles + want - 1) / want + 7) / 8 * 8;            // whole groups
      const dim3 grid(gx, blks(in.ntiles, np.per_chunk));
      if (sl.cls == kHalf) k_track_fwd_nodes<true><<<grid, kNodeNT, 0, st>>>(np);
      else k_track_fwd_nodes<false><<<grid, kNodeNT, 0, st>>>(np);
      TRACK_CUDA(cudaGetLastError(), "node sums");
      TrackInterpParams ip = interp_params(S, in, sl, masked, use_off, drop_tile);
      ip.per_chunk = interp_tiles(in, nblk);
      nv = static_cast<int>(blks(in.ntiles, ip.per_chunk));
      ip.vacc = vacc_d;
      ip.vstride = slots;
      ip.err = err;
      interp<<<dim3(nblk, nv), kInterpNT, FwdInterpSmem(sl.rank).total, st>>>(ip);
      TRACK_CUDA(cudaGetLastError(), "interpolation");
    }
    k_track_reduce_fwd<<<blks(slots, 256), 256, 0, st>>>(slots, static_cast<long long>(sl.b0) * kTrackT, S.slot, nv,
                                                         vacc_d, slots, nrest, rest_d, S.Ks, V, accumulate);
    TRACK_CUDA(cudaGetLastError(), "reduce");
  }
  return 0;
}

int tracks_adjoint(void *state, const TrackInputs &in, const float2 *coef, float *image, float scale, bool masked,
                   bool use_off, bool accumulate, unsigned long long *counter, int *err, int drop_tile,
                   cudaStream_t st) {
  TrackState &S = *static_cast<TrackState *>(state);
  const int nbc = S.shape.blocks_per_channel();
  // the remainder: CTAs of four tiles and a chunk of blocks.  The tiles that a limb
  // grazes for a whole orbit have several times the others' work, so a chunk is a
  // 32nd of the blocks at most (8, 16, 32, 48 chunks of 3,038 blocks at Nside 256:
  // 23.2, 20.7, 18.5, 17.9 ms); channels divide them too, down to an eighth.  Each
  // costs 8 bytes per pixel.
  const unsigned rx = blks(in.ntiles, kRestNT / 32);
  const long long rwant = std::max({8LL, 32LL / in.channels, 24LL * in.nsm / (static_cast<long long>(rx) * in.channels)});
  int per = static_cast<int>((nbc + rwant - 1) / rwant + 31) / 32 * 32;
  int nrest = S.has_rest[masked] ? static_cast<int>(blks(nbc, per)) : 0;
  if (static_cast<long long>(nrest) * in.channels > 65535) {
    per = (nbc + 31) / 32 * 32;
    nrest = 1;
  }
  // node chunks of a slab: about 8 waves of four CTAs per SM, at least two stages each
  const unsigned gx = blks(in.ntiles, 8);
  const int ny = static_cast<int>(std::max<long long>(
      1, std::min<long long>((8LL * 4 * in.nsm + gx - 1) / gx, S.ld_max / (2 * kAdjNodeTile))));
  const size_t nodes = static_cast<size_t>(ny) * in.Jpad, rests = static_cast<size_t>(nrest) * in.channels * in.Jpad;
  float2 *coef_d;
  double *node_d, *rest_d;
  TrackCut sums = call_sums(S, in, TrackArena::bytes<float2>(S.Ks) + TrackArena::bytes<double>(nodes) +
                                       TrackArena::bytes<double>(rests));
  if (!sums.at) return record_error(-3, "viss_adjoint: device allocation failed (track block sums)");
  sums.take(coef_d, S.Ks);
  sums.take(node_d, nodes);
  sums.take(rest_d, rests);
  if (int e = find_peak(S, in.K, nullptr, coef, in.nsm, st)) return e;
  k_track_coef<<<blks(S.Ks, 256), 256, 0, st>>>(S.Ks, S.slot, coef, S.peak, coef_d);
  TRACK_CUDA(cudaGetLastError(), "coefficients");
  if (nrest) {
    TrackRestParams rp = rest_params(S, in, masked, use_off, counter);
    rp.pix = in.pix;
    rp.per_chunk = per;
    rp.nchunk = nrest;
    rp.part_adj = rest_d;
    rp.coef = coef_d;
    const dim3 grid(rx, nrest * in.channels);
    if (masked) k_track_adj_rest<true><<<grid, kRestNT, 0, st>>>(rp);
    else k_track_adj_rest<false><<<grid, kRestNT, 0, st>>>(rp);
    TRACK_CUDA(cudaGetLastError(), "remainder");
  }
  const size_t smem_half = 2 * sizeof(AdjNodeStage<true>), smem_tile = 3 * sizeof(AdjNodeStage<false>);
  const auto interp = masked ? k_track_adj_interp<true> : k_track_adj_interp<false>;
  TRACK_CUDA(cudaFuncSetAttribute(interp, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  AdjInterpSmem(kTrackRankMax).total), "attributes");
  TRACK_CUDA(cudaFuncSetAttribute(k_track_adj_nodes<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem_half)), "attributes");
  TRACK_CUDA(cudaFuncSetAttribute(k_track_adj_nodes<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(smem_tile)), "attributes");
  size_t si = 0;
  for (int ch = 0; ch < in.channels; ++ch) {
    TRACK_CUDA(cudaMemsetAsync(node_d, 0, sizeof(double) * ny * in.Jpad, st), "node images");
    for (; si < S.slabs.size() && S.slabs[si].ch == ch; ++si) {
      const TrackSlab &sl = S.slabs[si];
      if (sl.cls == kClasses) continue;
      const int nblk = sl.b1 - sl.b0;
      TrackInterpParams ip = interp_params(S, in, sl, masked, use_off, drop_tile);
      ip.coef = coef_d;
      ip.per_chunk = interp_tiles(in, nblk);
      ip.err = err;
      interp<<<dim3(nblk, blks(in.ntiles, ip.per_chunk)), kInterpNT, AdjInterpSmem(sl.rank).total, st>>>(ip);
      TRACK_CUDA(cudaGetLastError(), "interpolation");
      TrackNodeParams np = node_params(S, in, sl, masked, counter, err, drop_tile);
      np.pix = in.pix;
      np.per_chunk = ((np.nn + ny - 1) / ny + kAdjNodeTile - 1) / kAdjNodeTile * kAdjNodeTile;
      np.part = node_d;
      const dim3 grid(gx, blks(np.nn, np.per_chunk));
      if (sl.cls == kHalf) k_track_adj_nodes<true><<<grid, kAdjNodeNT, smem_half, st>>>(np);
      else k_track_adj_nodes<false><<<grid, kAdjNodeNT, smem_tile, st>>>(np);
      TRACK_CUDA(cudaGetLastError(), "node images");
    }
    k_track_reduce_adj<<<blks(in.J, 256), 256, 0, st>>>(
        in.J, in.Jpad, ny, node_d, nrest, rest_d + static_cast<long long>(ch) * nrest * in.Jpad, in.perm,
        S.peak, scale, image + static_cast<long long>(ch) * in.J, accumulate);
    TRACK_CUDA(cudaGetLastError(), "reduce");
  }
  return 0;
}

}  // namespace viss