// FP64 Gaussians of the fragment-memory term: device code, and host code for
// its test (the same operations, so the same bits).
//
// e^x for x <= 0 by the table method of P. T. P. Tang ("Table-driven
// implementation of the exponential function in IEEE floating-point
// arithmetic", ACM TOMS 15 (1989)) in units of ln2 / 32: z = 32 x / ln2 = 32 m
// + j + f with |f| <= 1/2, e^x = 2^m 2^(j/32) (1 + p(f)), p the Taylor
// polynomial of 2^(f/32) - 1 to f^6 (remainder below 4e-18).  The row's factor
// carries the 32 / ln2, so z - (32 m + j) is exact.  2^(j/32) is a double and
// what that leaves, relative to it, which joins p(f) in the polynomial's last
// step.  Arguments below -708 (the padding's -1e59 among them) give 0.
//
// Error of a Gaussian, in units of 2^-53 (2^20 of separations 3 to 8, dr of
// 1.6 A; rms, absolute / relative): 0.29 / 1.05, by CUDA's exp() 0.30 / 1.12,
// with the table's doubles alone 0.38 / 1.16.  The low parts cost a third
// shuffle: 80 -> 84 us for the kernel on 61 chains (16,000 residues), 218 -> 230
// on 240; packed into the spare exponent bits of the doubles, 87 and 240.
#pragma once

#ifndef __CUDACC__
#include <cmath>
#include <cstring>
#endif

#ifndef AWSEM_HD
#ifdef __CUDACC__
#define AWSEM_HD __host__ __device__ __forceinline__
#else
#define AWSEM_HD inline
#endif
#endif

namespace awsem {
namespace dev {

#define AWSEM_EXP2_OF_32NDS \
  0x1.0000000000000p+0, 0x1.059b0d3158574p+0, 0x1.0b5586cf9890fp+0, 0x1.11301d0125b51p+0, \
  0x1.172b83c7d517bp+0, 0x1.1d4873168b9aap+0, 0x1.2387a6e756238p+0, 0x1.29e9df51fdee1p+0, \
  0x1.306fe0a31b715p+0, 0x1.371a7373aa9cbp+0, 0x1.3dea64c123422p+0, 0x1.44e086061892dp+0, \
  0x1.4bfdad5362a27p+0, 0x1.5342b569d4f82p+0, 0x1.5ab07dd485429p+0, 0x1.6247eb03a5585p+0, \
  0x1.6a09e667f3bcdp+0, 0x1.71f75e8ec5f74p+0, 0x1.7a11473eb0187p+0, 0x1.82589994cce13p+0, \
  0x1.8ace5422aa0dbp+0, 0x1.93737b0cdc5e5p+0, 0x1.9c49182a3f090p+0, 0x1.a5503b23e255dp+0, \
  0x1.ae89f995ad3adp+0, 0x1.b7f76f2fb5e47p+0, 0x1.c199bdd85529cp+0, 0x1.cb720dcef9069p+0, \
  0x1.d5818dcfba487p+0, 0x1.dfc97337b9b5fp+0, 0x1.ea4afa2a490dap+0, 0x1.f50765b6e4540p+0
// ... and the high words of 2^(j/32) / (the double above) - 1
#define AWSEM_EXP2_OF_32NDS_LOW \
  0x00000000u, 0x3c8cd252u, 0x3c979aa6u, 0xbc955652u, 0xbc801b16u, 0x3c9aecf7u, 0x3c968efeu, 0x3c82f7e1u, \
  0x3c834d75u, 0xbc924aeeu, 0x3c859f49u, 0x3c4363edu, 0x3c7690cfu, 0xbc78dec7u, 0x3c9063e2u, 0xbc8c33c5u, \
  0xbc93b3f0u, 0xbc781f64u, 0xbc7b32ddu, 0xbc9369b7u, 0x3c8db730u, 0xbc5da9b9u, 0x3c71affcu, 0xbc91bbd2u, \
  0x3c8c1a78u, 0xbc68d6f4u, 0x3c736eaeu, 0x3c676b2cu, 0x3c74a386u, 0xbc82d521u, 0xbc8ff713u, 0x3c8a64a9u

// -(32 / ln2) / (2 s2), rounded once: 32 / ln2 is a double and a rest
AWSEM_HD double gauss_factor(double s2)
{
  const double c = 0x1.71547652b82fep+5, rest = 0x1.777d0ffda0d24p-51, t = 2.0 * s2, q = -c / t;
  const double low = (fma(-q, t, -c) - rest) * q * -0x1.62e42fefa39efp-6;  // (what q leaves) / t, as 1 / t = -q ln2 / 32
  return low - low == 0.0 ? q + low : q;  // q where it has overflowed
}

// the nearest integer to z, in the low word of the result
constexpr double kGaussRound = 6755399441055744.0;  // 1.5 * 2^52
// the steps of 2^(f/32) - 1 + low, f = z less that integer, from kGaussTop:
// q = q f + each of AWSEM_GAUSS_POLY, then q f + low
constexpr double kGaussTop = 0x1.430912f86c787p-43;
#define AWSEM_GAUSS_POLY                                                                                            \
  0x1.5d87fe78a6731p-35, 0x1.3b2ab6fba4e77p-27, 0x1.c6b08d704a0c0p-20, 0x1.ebfbdff82c58fp-13, 0x1.62e42fefa39efp-6
constexpr double kGaussLeast = -708.0 * 0x1.71547652b82fep+5;

#ifndef __CUDACC__
// one Gaussian, by the kernel's operations
inline double gauss_host(double z)
{
  static const double table[32] = {AWSEM_EXP2_OF_32NDS}, poly[5] = {AWSEM_GAUSS_POLY};
  static const unsigned lows[32] = {AWSEM_EXP2_OF_32NDS_LOW};
  if (z < kGaussLeast) return 0.0;
  const double y = z + kGaussRound, f = z - (y - kGaussRound);
  long long bits;
  std::memcpy(&bits, &y, 8);
  const int n = (int) bits;
  const unsigned long long word = (unsigned long long) lows[n & 31] << 32;
  double low, q = kGaussTop;
  std::memcpy(&low, &word, 8);
  for (double c : poly) q = fma(f, q, c);
  const double s = std::ldexp(table[n & 31], n >> 5);
  return fma(s, fma(f, q, low), s);
}
#endif

}  // namespace dev
}  // namespace awsem
