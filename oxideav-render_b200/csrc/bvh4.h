// The quantised four-child node (Bvh4Node): how the builders and the refit
// write one, on the host and on the device.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include <vector_functions.h>

#include "dev_types.h"

#ifdef __CUDACC__
#define PT_HD __host__ __device__ __forceinline__
#else
#define PT_HD inline
#endif

namespace ptd {

// Packing is on the path of every refit (a small scene's is one chain of
// nodes from a leaf to the root) and of every host build: no divisions, no
// library calls and few branches. Refit of a 4,616-triangle scene, device
// part, with frexp, ldexp and 24 divisions a node / without: 0.23 / 0.22 ms
// (full-precision nodes 0.20; larger scenes within noise); a host build's
// time per node 205 / 129 ns.

// x = m * 2^e with m in [1/2, 1): e, for a normal x; and 2^e.
PT_HD int exponent_of(double x) {
  uint64_t b;
  memcpy(&b, &x, 8);
  return (int)(b >> 52 & 0x7ffu) - 1022;
}
PT_HD double power_of_two(int e) {
  const uint64_t b = (uint64_t)(e + 1023) << 52;
  double x;
  memcpy(&x, &b, 8);
  return x;
}
// The largest float at most x, for x zero or of a normal float's magnitude.
PT_HD float float_below(double x) {
  uint64_t b;
  memcpy(&b, &x, 8);
  b += (uint64_t)((int64_t)b >> 63) & 0x1fffffffu;  // magnitudes of negative values go up
  b &= ~(uint64_t)0x1fffffffu;
  memcpy(&x, &b, 8);
  return (float)x;
}

// The last plane of the grid origin + k * s on or below v, and the first on
// or above it, for v in [origin, origin + 2^30 s]; s is a power of two and
// `inv` its reciprocal, so the product is the quotient. The planes are exact
// in f64 (k is small, origin and s span fewer than 53 bits), v - origin need
// not be: a plane that its rounding put on the wrong side of v moves by one.
PT_HD int lower_plane(double v, double origin, double s, double inv) {
  const int k = (int)((v - origin) * inv);
  return k - (int)(origin + k * s > v);
}
PT_HD int upper_plane(double v, double origin, double s, double inv) {
  int k = (int)((v - origin) * inv);
  k += (int)(origin + k * s < v);
  return k + (int)(origin + k * s < v);
}

// Fills `out` from the boxes of up to four children (lo[axis][child],
// hi[axis][child]; used for refs other than kEmptyChild). Every stored plane
// lies on or outside the box it stands for: the lower ones are rounded down
// and the upper ones up, in f64, against the plane positions the node
// decodes to. An axis whose extent has no finite grid (infinite or huge
// coordinates, every child's box empty) decodes to NaN planes, which bound
// nothing; a child whose own box is empty (NaN corners) spans the node's.
PT_HD void pack_bvh4(const float lo[3][4], const float hi[3][4], const int ref[4], Bvh4Node &out) {
  float base[3], step[3];
  uint32_t qlo[3], qhi[3];
  for (int a = 0; a < 3; ++a) {
    float l = INFINITY, h = -INFINITY;
    for (int i = 0; i < 4; ++i)
      if (ref[i] != kEmptyChild) {
        l = lo[a][i] < l ? lo[a][i] : l;  // NaN corners are passed over
        h = hi[a][i] > h ? hi[a][i] : h;
      }
    int e = -100;
    const double range = (double)h - (double)l;
    bool grid = range >= 0.0 && range < 1.0e38;
    if (grid) {
      // The extent in 126 to 253 quanta.
      if (range > 0.0) {
        e = exponent_of(range) - 8;
        if (range >= 253.0 * power_of_two(e)) ++e;
      }
      // Not finer than the coordinates can resolve: the planes stay exact in
      // f64, and a box without extent gets a grid all the same.
      int least = -100;
      const double most = -(double)l > (double)h ? -(double)l : (double)h;  // the larger magnitude, as l <= h
      if (most > 0.0) {
        least = exponent_of(most) - 30;
        if (least < -100) least = -100;
      }
      if (range == 0.0 || e < least) e = least;
    }
    double s = 1.0, inv = 1.0, origin = 0.0;
    for (; grid; ++e) {
      s = power_of_two(e);
      inv = power_of_two(-e);
      const double wide = s * 32768.0;
      if (!(wide < 1.0e38)) {
        grid = false;
        break;
      }
      // The first plane, base + wide: on or below l. Where l is tiny against
      // the grid, l - wide rounds to -wide, which would place it at zero.
      float b = float_below((double)l - wide);
      if ((double)b + wide > (double)l) b = nextafterf(b, -INFINITY);
      if (!(fabsf(b) < 1.0e38f)) {
        grid = false;
        break;
      }
      origin = (double)b + wide;
      base[a] = b;
      step[a] = (float)wide;
      if (upper_plane((double)h, origin, s, inv) <= 255) break;
    }
    qlo[a] = 0u;
    qhi[a] = 0u;
    if (!grid) {
      base[a] = -INFINITY;
      step[a] = INFINITY;
    }
    for (int i = 0; i < 4; ++i) {
      uint32_t l8 = 255u, h8 = 0u;
      if (ref[i] != kEmptyChild) {
        l8 = 0u;
        h8 = 255u;
        if (grid && lo[a][i] <= hi[a][i]) {
          l8 = (uint32_t)lower_plane((double)lo[a][i], origin, s, inv);
          h8 = (uint32_t)upper_plane((double)hi[a][i], origin, s, inv);
        }
      }
      qlo[a] |= l8 << (8 * i);
      qhi[a] |= h8 << (8 * i);
    }
  }
  out.base = make_float4(base[0], base[1], base[2], step[0]);
  out.mid = make_uint4(0, 0, qlo[0], qhi[0]);
  memcpy(&out.mid.x, &step[1], 4);
  memcpy(&out.mid.y, &step[2], 4);
  out.planes = make_uint4(qlo[1], qhi[1], qlo[2], qhi[2]);
  out.child = make_int4(ref[0], ref[1], ref[2], ref[3]);
}

}  // namespace ptd
