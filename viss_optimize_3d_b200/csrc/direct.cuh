// direct.cuh -- device code of the direct sums: a sample's classification
// against pixel cones, the exact occultation test and the exponential terms.
// Shared by the direct kernels (visibility.cu) and the track blocks' remainder
// (tracks.cu).
#pragma once

#include "viss_common.cuh"

namespace viss {

// Classification of a sample (3 occulter refs) against one tile cone, packed:
// bits 0-1 state (2 every pixel visible, 0 none, 1 mixed), bits 2-4 which
// refs are mixed on this tile (only those need the per-pixel test).
__device__ __forceinline__ int sample_state(const int4 &rf, const float4 &cone,
                                            const float4 *occ32) {
  int st = 2, need = 0;
  const int r3[3] = {rf.x, rf.y, rf.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (r3[c] < 0) continue;
    const int s = cone_state32(cone, occ32[r3[c]]);
    st = min(st, s);
    if (s == 1) need |= 1 << c;
  }
  return st == 1 ? (1 | (need << 2)) : st;
}

// The same against the union of two tiles (a warp tile of 256 pixels): hidden
// only if hidden on both; all visible only if all visible on both; otherwise
// every ref that is not all-visible on both tiles is tested per pixel.
__device__ __forceinline__ int sample_state2(const int4 &rf, const float4 &c0, const float4 &c1,
                                             const float4 *occ32) {
  const int a = sample_state(rf, c0, occ32), b = sample_state(rf, c1, occ32);
  const int sa = a & 3, sb = b & 3;
  if (sa == 0 && sb == 0) return 0;
  if (sa == 2 && sb == 2) return 2;
  int need = 0;
  const int r3[3] = {rf.x, rf.y, rf.z};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    if (r3[c] < 0) continue;
    const bool full0 = (sa == 2) || (sa == 1 && !((a >> (2 + c)) & 1));
    const bool full1 = (sb == 2) || (sb == 1 && !((b >> (2 + c)) & 1));
    if (!(full0 && full1)) need |= 1 << c;
  }
  return need ? (1 | (need << 2)) : 2;
}

// The occulter rows a mixed sample must test (need bits 2-4 of its state
// code), compacted to the front: their indices (-1 past the count) and the
// count.
__device__ __forceinline__ int needed_idx(const int4 &rf, int code, int &i0, int &i1, int &i2) {
  i0 = i1 = i2 = -1;
  if (code & 4) i0 = rf.x;
  if (code & 8) {
    if (i0 < 0) i0 = rf.y;
    else i1 = rf.y;
  }
  if (code & 16) {
    if (i0 < 0) i0 = rf.z;
    else if (i1 < 0) i1 = rf.z;
    else i2 = rf.z;
  }
  return (i0 >= 0) + (i1 >= 0) + (i2 >= 0);
}

// Exact rows for those indices; absent rows pass every direction (thr = -4
// is below any dot product of unit vectors).
__device__ __forceinline__ void exact_rows(const double4 *occ, int i0, int i1, int i2,
                                           double4 &q0, double4 &q1, double4 &q2) {
  const double4 pass = make_double4(0.0, 0.0, 0.0, -4.0);
  q0 = i0 >= 0 ? occ[i0] : pass;
  q1 = i1 >= 0 ? occ[i1] : pass;
  q2 = i2 >= 0 ? occ[i2] : pass;
}

// Classification rows for those indices.
__device__ __forceinline__ void class_rows(const float4 *occ32, int i0, int i1, int i2,
                                           float4 &f0, float4 &f1, float4 &f2) {
  const float4 pass32 = make_float4(0.f, 0.f, 0.f, -4.f);
  f0 = i0 >= 0 ? occ32[i0] : pass32;
  f1 = i1 >= 0 ? occ32[i1] : pass32;
  f2 = i2 >= 0 ? occ32[i2] : pass32;
}

// Both, for one sample; returns how many rows need the test.
__device__ __forceinline__ int needed_rows(const int4 &rf, int code, const double4 *occ,
                                           const float4 *occ32, double4 &q0, double4 &q1,
                                           double4 &q2, float4 &f0, float4 &f1, float4 &f2) {
  int i0, i1, i2;
  const int n = needed_idx(rf, code, i0, i1, i2);
  exact_rows(occ, i0, i1, i2, q0, q1, q2);
  class_rows(occ32, i0, i1, i2, f0, f1, f2);
  return n;
}

// State of one cone against the first n classification rows (2 visible, 0
// hidden, 1 mixed).
__device__ __forceinline__ int rows_state(const float4 &cone, int n, const float4 &f0,
                                          const float4 &f1, const float4 &f2) {
  int st = 2;
  if (n > 0) st = min(st, cone_state32(cone, f0));
  if (n > 1) st = min(st, cone_state32(cone, f1));
  if (n > 2) st = min(st, cone_state32(cone, f2));
  return st;
}

// Exact visibility of direction s against the first NROWS rows (the same IEEE
// operations as the CPU oracle's predicate).
template <int NROWS>
__device__ __forceinline__ bool visible_rows(const double4 &q0, const double4 &q1,
                                             const double4 &q2, double s0, double s1, double s2) {
  bool v = true;
  if (NROWS > 0) v = dot_exact(s0, s1, s2, q0) >= q0.w;
  if (NROWS > 1) v = v & (dot_exact(s0, s1, s2, q1) >= q1.w);
  if (NROWS > 2) v = v & (dot_exact(s0, s1, s2, q2) >= q2.w);
  return v;
}

// FP64 reference term: (sin, cos) of 2 pi (phase mod 1), phase in FP64.
__device__ __forceinline__ void sincos_turns_fp64(double t, double &sn, double &cs) {
  const double f = t - rint(t);
  sincospi(2.0 * f, &sn, &cs);
}

// One forward term into (re, im): sky I at phase t.
template <bool FP64>
__device__ __forceinline__ void fwd_term(double t, float I, float &re, float &im, double &dre,
                                         double &dim) {
  if (FP64) {
    double sn, cs;
    sincos_turns_fp64(t, sn, cs);
    dre = fma(static_cast<double>(I), cs, dre);
    dim = fma(-static_cast<double>(I), sn, dim);
  } else {
    float sn, cs;
    sfu_sincos(turn_angle(t), sn, cs);
    re = fmaf(I, cs, re);
    im = fmaf(-I, sn, im);
  }
}

// The same for NS skies (split precision): one exponential, NS sums.
template <int NS>
__device__ __forceinline__ void fwd_term_skies(double t, const float (&I)[NS], float (&re)[NS], float (&im)[NS]) {
  float sn, cs;
  sfu_sincos(turn_angle(t), sn, cs);
#pragma unroll
  for (int c = 0; c < NS; ++c) {
    re[c] = fmaf(I[c], cs, re[c]);
    im[c] = fmaf(-I[c], sn, im[c]);
  }
}

// A pixel's NS sky values, zero where it is hidden; odd records negated.
template <int NS>
__device__ __forceinline__ void skies_of(const float4 &w, bool seen, bool odd, float (&I)[NS]) {
  const float v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int c = 0; c < NS; ++c) I[c] = seen ? (odd ? -v[c] : v[c]) : 0.f;
}

// Pixels per forward sub-tile (the span a mixed sample row is refined to).
constexpr int kSubPix = 32;

// One sample over kSubPix staged records, in pairs (even record at mk, odd
// record half a turn on at mk2 and negated), testing the first NROWS
// occulter rows per term (NROWS = 0: every pixel visible).
template <int NROWS, bool FP64>
__device__ __forceinline__ void fwd_span(const double4 *tp, double ux, double uy, double uz,
                                         double mk, double mk2, const double4 &q0,
                                         const double4 &q1, const double4 &q2, float &re,
                                         float &im, double &dre, double &dim) {
#pragma unroll 2
  for (int j = 0; j < kSubPix; j += 2) {
    const double4 a = tp[j], b = tp[j + 1];
    float Ia = sky_of(a), Ib = FP64 ? sky_of(b) : -sky_of(b);
    if (NROWS > 0) {
      Ia = visible_rows<NROWS>(q0, q1, q2, a.x, a.y, a.z) ? Ia : 0.f;
      Ib = visible_rows<NROWS>(q0, q1, q2, b.x, b.y, b.z) ? Ib : 0.f;
    }
    const double ta = fma(uz, a.z, fma(uy, a.y, fma(ux, a.x, mk)));
    fwd_term<FP64>(ta, Ia, re, im, dre, dim);
    const double tb = fma(uz, b.z, fma(uy, b.y, fma(ux, b.x, mk2)));
    fwd_term<FP64>(tb, Ib, re, im, dre, dim);
  }
}

// fwd_span for NS skies, whose values stand beside the records.
template <int NROWS, int NS>
__device__ __forceinline__ void fwd_span_skies(const double4 *tp, const float4 *wp, double ux, double uy, double uz,
                                               double mk, double mk2, const double4 &q0, const double4 &q1,
                                               const double4 &q2, float (&re)[NS], float (&im)[NS]) {
#pragma unroll 2
  for (int j = 0; j < kSubPix; j += 2) {
    const double4 a = tp[j], b = tp[j + 1];
    float Ia[NS], Ib[NS];
    skies_of<NS>(wp[j], visible_rows<NROWS>(q0, q1, q2, a.x, a.y, a.z), false, Ia);
    skies_of<NS>(wp[j + 1], visible_rows<NROWS>(q0, q1, q2, b.x, b.y, b.z), true, Ib);
    fwd_term_skies<NS>(fma(uz, a.z, fma(uy, a.y, fma(ux, a.x, mk))), Ia, re, im);
    fwd_term_skies<NS>(fma(uz, b.z, fma(uy, b.y, fma(ux, b.x, mk2))), Ib, re, im);
  }
}

// One sample into a lane's P pixels (pixel q of every lane lies in the warp's
// 32-pixel sub-tile q).  Bit q of the warp-uniform `hid` zeroes sub-tile q
// (none of it visible); NROWS > 0 tests the first NROWS occulter rows on
// every term.  The P terms stay one branch-free block: splitting them by
// sub-tile would serialise their DFMA -> MUFU latency chains, which costs more
// than evaluating a hidden term.
template <int P, int NROWS, bool FP64>
__device__ __forceinline__ void adj_sample(const double4 &u, double m, const float2 &a,
                                           const double (&sx)[P], const double (&sy)[P],
                                           const double (&sz)[P], const double4 &q0,
                                           const double4 &q1, const double4 &q2, unsigned hid,
                                           float (&acc)[P], double (&dacc)[P]) {
#pragma unroll
  for (int q = 0; q < P; ++q) {
    const double t = fma(u.z, sz[q], fma(u.y, sy[q], fma(u.x, sx[q], m)));
    bool vis = ((hid >> q) & 1u) == 0;
    if (NROWS > 0) vis = vis & visible_rows<NROWS>(q0, q1, q2, sx[q], sy[q], sz[q]);
    const float ar = vis ? a.x : 0.f, ai = vis ? a.y : 0.f;
    if (FP64) {
      double sn, cs;
      sincos_turns_fp64(t, sn, cs);
      dacc[q] += fma(static_cast<double>(ar), cs, -static_cast<double>(ai) * sn);
    } else {
      float sn, cs;
      sfu_sincos(turn_angle(t), sn, cs);
      acc[q] = fmaf(ar, cs, acc[q]);
      acc[q] = fmaf(-ai, sn, acc[q]);
    }
  }
}

}  // namespace viss
