// cos and sin of a fixed-point phase, in fixed point.
//
// DFT matrices and phasors need cosines and sines of phases that are exact
// 64-bit fractions of a cycle (phase_fixed, common.cuh; x mod 2).  Double-
// precision sincospi holds this part's FP64 pipe (17 clocks a value per SM
// measured in the phasor kernel); the integer pipes give the same in about five:
// the nearest of 512 points of the circle from a table, and a rotation by the
// rest, |d| < 2^-7.3, with the Taylor series of cos d and sin d in 64-bit fixed
// point, cut where the terms fall below 2^-63.  The error is below 2^-60 (2.4 units of 2^-62 at most over
// thousands of phases against 60-digit values).
#pragma once

#include <stdint.h>

#include "common.cuh"

namespace lgb {

// round(2^62 cos(2 pi i / 512)), i = 0 .. 128
__device__ static const unsigned long long COS_TABLE[129] = {
    0x4000000000000000, 0x3ffec42d3725b6af, 0x3ffb10c1099a1976, 0x3ff4e5dffdeeb93a,
    0x3fec43c6f2dafbc7, 0x3fe12acb1ce35a81, 0x3fd39b5a0310742a, 0x3fc395f97ab61234,
    0x3fb11b47a24a4b3c, 0x3f9c2bfadb4cf5a9, 0x3f84c8e1c33fa68f, 0x3f6af2e32bae8247,
    0x3f4eaafe114a2d43, 0x3f2ff2499213350f, 0x3f0ec9f4e297526b, 0x3eeb33474240eec2,
    0x3ec52f9feeb96056, 0x3e9cc076165e599c, 0x3e71e758c9cb118a, 0x3e44a5eeec75b370,
    0x3e14fdf72461ae55, 0x3de2f147c8e784b2, 0x3dae81ced092c67a, 0x3d77b191be16e872,
    0x3d3e82ad8c5bb4bb, 0x3d02f75699a2198c, 0x3cc511d891c223dd, 0x3c84d4965782fcd4,
    0x3c424209ed0dc97f, 0x3bfd5cc45b7c5557, 0x3bb6276d998478c2, 0x3b6ca4c471413595,
    0x3b20d79e651a8c51, 0x3ad2c2e793cd1586, 0x3a8269a29b927359, 0x3a2fcee87c6bb7ef,
    0x39daf5e8798ee5e2, 0x3983e1e7f9f8b879, 0x392a96426823e9ed, 0x38cf166910e7363b,
    0x387165e3017b61a4, 0x3811884ce4aa921b, 0x37af8158df2a533f, 0x374b54ce6b21a4bf,
    0x36e5068a32dc7b22, 0x367c9a7deaae230a, 0x361214b02a03ff37, 0x35a5793c43aa215c,
    0x3536cc521d434606, 0x34c6123605f5c386, 0x34534f408c4f03bb, 0x33de87de535f286c,
    0x3367c08fe70e8168, 0x32eefde98fae8375, 0x3274449324c7f69f, 0x31f79947df2819d2,
    0x317900d62a2e816a, 0x30f8801f745d7d69, 0x30761c17ff2edba4, 0x2ff1d9c6ae2ee132,
    0x2f6bbe44d55f5dbc, 0x2ee3cebe06e4c257, 0x2e5a106fdfff2c87, 0x2dce88a9d5515d12,
    0x2d413cccfe779921, 0x2cb2324be0f07ae2, 0x2c216eaa3a59bdb7, 0x2b8ef77cca031883,
    0x2afad26919d93f45, 0x2a65052546ab2b98, 0x29cd9577c7cbd228, 0x293489373612716c,
    0x2899e64a123bac30, 0x27fdb2a68aada89b, 0x275ff45240a17279, 0x26c0b1620cb3e570,
    0x261feff9c2e069c2, 0x257db64bf5e7d3ef, 0x24da0a99ba25bd51, 0x2434f33267d6b163,
    0x238e76735cd190d9, 0x22e69ac7bdb69141, 0x223d66a836964508, 0x2192e09abb131d39,
    0x20e70f3245ffdb2d, 0x2039f90e987d6db3, 0x1f8ba4dbf89ab9fb, 0x1edc1952ef78d589,
    0x1e2b5d3806f63b1e, 0x1d79775b86e38955, 0x1cc66e9931c45e17, 0x1c1249d8011ee6a0,
    0x1b5d1009e15cc02b, 0x1aa6c82b6d3fc98b, 0x19ef7943a8ed8a2e, 0x19372a63bc93d72d,
    0x187de2a6aea962d2, 0x17c3a9311dcce702, 0x17088530fa459eaf, 0x164c7ddd3f27c611,
    0x158f9a75ab1fdcfe, 0x14d1e24278e76a25, 0x14135c9417660143, 0x135410c2e18151b1,
    0x1294062ed59f05a9, 0x11d3443f4cdb3dd2, 0x1111d262b1f67761, 0x104fb80e37fdadff,
    0x0f8cfcbd90af8d58, 0x0ec9a7f2a2a188af, 0x0e05c1353f27b17e, 0x0d415012d802284f,
    0x0c7c5c1e34d3055b, 0x0bb6ecef285f98a4, 0x0af10a22459fe32a, 0x0a2abb58949f2ced,
    0x0964083747309d11, 0x089cf8676d7abb56, 0x07d59395aa5cc38d, 0x070de171e7b0b53d,
    0x0645e9af0a6d0af8, 0x057db402a6a90630, 0x04b54824b3867d73, 0x03ecadcf3f041bfe,
    0x0323ecbe21bb027d, 0x025b0caeb28ab9a3, 0x0192155f7a3667e0, 0x00c90e8fe6f63c23,
    0x0000000000000000,
};

// The nearest of the table's points to a phase, and the rest |r| <= 2^54.
struct TablePoint {
  uint32_t at;
  bool neg;
  uint64_t ar;
};
__device__ __forceinline__ TablePoint table_point(uint64_t ph) {
  const uint32_t at = (uint32_t)((ph + (1ull << 54)) >> 55) & 511u;
  const int64_t r = (int64_t)(ph - ((uint64_t)at << 55));
  return TablePoint{at, r < 0, (uint64_t)(r < 0 ? -r : r)};
}

// (cos, sin) of a phase's angle less its quadrant (at & 384), in units of
// 2^-62, and u = 1 - sin d / d of the rest d, Q72.
__device__ __forceinline__ longlong2 first_quadrant_q62(const TablePoint& p, const unsigned long long* table,
                                                        uint64_t& u) {
  const uint64_t d = __umul64hi(p.ar << 8, 7244019458077122842ull);                    // |d|, Q68, < 2^60.7
  const uint64_t d2 = __umul64hi(d << 1, d << 1);                        // d^2, Q74, < 2^59.4
  const uint32_t y = (uint32_t)(d2 >> 28);                               // d^2, Q46
  // 1 - cos d = d^2 (1/2 - d^2/24 + d^4/720)
  const uint32_t w = 2863311531u - __umulhi(y, 5825u);         // 1/24 - d^2/720, Q36
  const uint64_t a = __umul64hi(d2, (1ull << 61) - ((uint64_t)__umulhi(y, w) << 12));   // Q72, < 2^56.4
  // sin d = d (1 - d^2 (1/6 - d^2/120))
  const uint64_t q6 = 768614336404564650ull - ((uint64_t)__umulhi(y, 2290649225u) << 10); // Q62
  u = __umul64hi(d2, q6);                                                // Q72, < 2^54.8
  const uint64_t sd = (d << 2) - (__umul64hi(d, u << 8) >> 14);          // Q70, < 2^62.7
  const int j = p.at & 127;
  const uint64_t c = table[j], s = table[128 - j];
  const int64_t ca = (int64_t)(__umul64hi(c, a << 6) >> 14), sa = (int64_t)(__umul64hi(s, a << 6) >> 14);
  int64_t cs = (int64_t)(__umul64hi(c, sd) >> 6), ss = (int64_t)(__umul64hi(s, sd) >> 6);
  if (p.neg) { cs = -cs; ss = -ss; }
  return make_longlong2((int64_t)c - ca - ss, (int64_t)s - sa + cs);
}

// (cos, sin)(2 pi ph / 2^64) in units of 2^-62; table: COS_TABLE or a copy.
__device__ __forceinline__ longlong2 cossin_q62(uint64_t ph, const unsigned long long* table) {
  const TablePoint p = table_point(ph);
  uint64_t u;
  longlong2 z = first_quadrant_q62(p, table, u);
  if (p.at & 128) z = make_longlong2(-z.y, z.x);
  return p.at & 256 ? make_longlong2(-z.x, -z.y) : z;
}

// v 2^e, or its negative
struct FixedValue {
  uint64_t v;
  int e;
  bool neg;
};

// cos and sin of pi x, x finite: x 2^63 mod 2^64 is the phase, exactly (below
// |x| = 2^-11 up to its last place).  Next to an axis (at & 127 = 0) the small
// one of the two is sin d from d's leading 64 bits, wherever they lie.
__device__ __forceinline__ void cossinpi(double x, const unsigned long long* table, FixedValue& c, FixedValue& s) {
  const uint64_t bits = (uint64_t)__double_as_longlong(x);
  int E = (int)(bits >> 52) & 0x7FF;
  uint64_t m = bits & 0xFFFFFFFFFFFFFull;
  if (E == 0) E = 1; else m |= 1ull << 52;
  const int sh = E - 1012;                                               // x 2^63 = m 2^sh
  uint64_t ph = sh >= 64 || sh <= -64 ? 0 : sh >= 0 ? m << sh : m >> -sh;
  if (bits >> 63) ph = 0 - ph;
  TablePoint p = table_point(ph);
  if (sh < 0) p.neg = bits >> 63;
  uint64_t u;
  const longlong2 z = first_quadrant_q62(p, table, u);
  c = FixedValue{(uint64_t)z.x, -62, false};                             // of the first quadrant's angle
  s = FixedValue{(uint64_t)z.y, -62, false};
  if ((p.at & 127) == 0) {
    const uint64_t r = sh < 0 ? m : p.ar;
    const int lz = __clzll((long long)r);
    const uint64_t dn = __umul64hi(lz < 64 ? r << lz : 0, 14488038916154245685ull);    // d 2^(61 + lz)
    s = FixedValue{dn - __umul64hi(dn, u >> 8), -61 - lz + (sh < 0 ? sh : 0), p.neg};
  }
  if (p.at & 128) {
    const FixedValue t = c;
    c = FixedValue{s.v, s.e, !s.neg};
    s = t;
  }
  if (p.at & 256) {
    c.neg = !c.neg;
    s.neg = !s.neg;
  }
}

// a exp(i pi x), each component within 1.3 units of its last place.  The
// product with the amplitude is taken in integers too: a double-precision
// multiply holds the FP64 pipe 16 clocks a warp.
__device__ __forceinline__ double2 phasor_f64(double a, double x, const unsigned long long* table) {
  if (((uint32_t)__double2hiint(x) & 0x7FF00000u) == 0x7FF00000u) return make_double2(x - x, x - x);   // NaN
  const uint64_t bits = (uint64_t)__double_as_longlong(a);
  if (bits << 1 == 0) return make_double2(0.0, 0.0);                     // outside the pupil
  FixedValue c, s;
  cossinpi(x, table, c, s);
  const int E = (int)(bits >> 52) & 0x7FF;
  if (E == 0 || E == 0x7FF) {                                            // subnormal, not finite
    const double cv = assembled(c.v, c.e), sv = assembled(s.v, s.e);
    return make_double2(a * (c.neg ? -cv : cv), a * (s.neg ? -sv : sv));
  }
  const uint64_t ma = bits << 11 | 1ull << 63;                           // |a| = ma 2^(E - 1086)
  auto times = [&](const FixedValue& q) {
    const int lz = __clzll((long long)q.v);
    const double r = q.v ? assembled(__umul64hi(q.v << lz, ma), q.e - lz + E - 1022) : 0.0;
    return q.neg != (bool)(bits >> 63) ? -r : r;
  };
  return make_double2(times(c), times(s));
}

}  // namespace lgb
