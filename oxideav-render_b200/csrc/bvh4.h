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

// x = m * 2^e with m in [1/2, 1): e, for a normal x; and 2^e. A refit of a
// small scene is one chain of nodes from a leaf to the root, whose length is
// the latency of this file's arithmetic: no divisions and no library calls
// (with them the device part of refitting a 4,616-triangle scene took 0.23 ms,
// without 0.22, over full-precision nodes 0.20; larger scenes within noise).
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

// The last plane of the grid origin + k * s on or below v, and the first on
// or above it; s is a power of two and `inv` its reciprocal, so the product
// is the quotient. The planes are exact in f64 (k is at most 2^8, origin and s
// span fewer than 53 bits), v - origin need not be: a plane that its rounding
// put on the wrong side of v moves by one.
PT_HD double lower_plane(double v, double origin, double s, double inv) {
  const double k = floor((v - origin) * inv);
  return origin + k * s > v ? k - 1.0 : k;
}
PT_HD double upper_plane(double v, double origin, double s, double inv) {
  const double k = ceil((v - origin) * inv);
  return origin + k * s < v ? k + 1.0 : k;
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
        l = fminf(l, lo[a][i]);
        h = fmaxf(h, hi[a][i]);
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
      const double most = fmax(fabs((double)l), fabs((double)h));
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
      float b = (float)((double)l - wide);
      while ((double)b + wide > (double)l) b = nextafterf(b, -INFINITY);
      if (!(fabsf(b) < 1.0e38f)) {
        grid = false;
        break;
      }
      origin = (double)b + wide;
      base[a] = b;
      step[a] = (float)wide;
      if (upper_plane((double)h, origin, s, inv) <= 255.0) break;
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
