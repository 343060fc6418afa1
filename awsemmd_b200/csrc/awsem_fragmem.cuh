// Fragment-memory term (fix_backbone.cpp:4079-4177, fragment_memory.cpp:
// 190-202) on a sliced, lane-interleaved memory table.
//
// Table layout.  A row is one target pair (i, j = i + min_sep + d) with the
// records of every memory covering it; a record holds the four memory
// distances of the atom pairs CA-CA, CA-CB, CB-CA, CB-CB.  Residues are
// taken 32 at a time (group g = residues 32g .. 32g+31).  Block (g, d) holds
// the rows (32g + l, d) of the group's 32 residues as `len` stripes; stripe
// m carries record m of each of the 32 rows side by side, lane l's record
// at [stripe][l].  Rows shorter than `len` are padded with records whose
// distances are 1e30 and whose coefficient is 0: their Gaussian is exactly
// zero, so padding never changes a sum.  Block lengths are even, so every
// block starts on an even stripe.  Blocks are stored g-major (block =
// g * nd + d), so the data of one group is contiguous.
//
// Kernel mapping.  One warp per (group, chunk of separations); lane l owns
// residue i = 32g + l and streams its rows stripe by stripe: every load of
// the warp is 32 consecutive records (512 B FP32, 1 KiB FP64) and each lane
// keeps its own sums, so no cross-lane reduction is needed.  A row's even
// and odd records go to two sets of sums, added at the row's end: two
// independent dependency chains per lane, and the same sums in every path
// that reads the table (the records pair up the same way in each).  Forces are
// converted to 64-bit fixed point (2^-32) per (row, atom pair) and added to
// the accumulator of j with integer atomics; i's forces are summed in
// registers over the chunk first.  Everything is order independent, so a
// residue's result does not depend on its group mates or on the chunking.
//
// FP64 rows are summed in pieces of kFmPiece records, a piece's sums from zero
// and added to the row's in order, so that the warps of a block can take the
// pieces of one row and give the bits of one warp alone.  A record is four
// FP64 exponentials (about 0.35 us for a warp that has its scheduler to
// itself): on one chain of 100 residues the 24 (group, separation) units took
// 46 us, the longest row's 120 records in series, while most of the chip was
// idle.  FP32 rows keep two running sums (pieces would round differently) and
// take 15 us on 2,000 residues.
#pragma once

#include "awsem_device.cuh"
#include "awsem_gauss.h"

namespace awsem {
namespace dev {

template <typename R> struct FMSlices {
  const int *soff;  // [G * nd] first stripe of block (g, d)
  const int *slen;  // [G * nd] stripes of block (g, d)
  const R *rf;      // [stripes][32][4] memory distances
  const R *coef;    // [stripes][32] eps * k_fm * weight * gamma, or nullptr when all equal `uniform`
  double uniform;
  int nd, min_sep;  // separations min_sep .. min_sep + nd - 1
  int groups;       // G = ceil(n_res / 32)
  int dsplit;       // separation chunks per group (warps per group)
  int psplit;       // warps per unit: 4 (FP64, one separation a chunk, rows of at most 4 pieces: a block
                    // takes a unit, a warp each piece of its row), 2 (FP32 without a copy ring: a warp
                    // each set of sums) or 1
  long long wait_limit;  // SM clock cycles a warp waits for one stage's copies before it gives up
  unsigned hold_tx;      // bytes each stage expects beyond its copies: 0, or (tests of the give-up
                         // path) 16, which never arrive, so every stage wait runs out
};

// One memory record: 16 bytes (FP32) or 32 bytes (FP64)
__device__ __forceinline__ void load_record(const float *rf, size_t rec, float m[4])
{
  float4 v = __ldg(reinterpret_cast<const float4 *>(rf) + rec);
  m[0] = v.x, m[1] = v.y, m[2] = v.z, m[3] = v.w;
}
__device__ __forceinline__ void load_record(const double *rf, size_t rec, double m[4])
{
  const double2 *q = reinterpret_cast<const double2 *>(rf) + 2 * rec;
  double2 u = __ldg(q), v = __ldg(q + 1);
  m[0] = u.x, m[1] = u.y, m[2] = v.x, m[3] = v.y;
}

__device__ __forceinline__ void red_add3(unsigned long long *p, const long long f[3])
{
#pragma unroll
  for (int c = 0; c < 3; c++)
    if (f[c]) atomicAdd(p + c, (unsigned long long) f[c]);
}

// Per-record arithmetic, shared by both load paths (so they agree bit for
// bit).  The Gaussian of a row with variance s^2 is exp(-dr^2 / (2 s^2)):
// FP32 evaluates it as 2^(k2 dr^2) with k2 = -log2(e) / (2 s^2) on the ex2
// unit, FP64 as e^x with z = 32 x / ln2 = k2 dr^2.
__device__ __forceinline__ float fm_gauss(float x)
{
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// FP64 Gaussians (awsem_gauss.h).  Lane j of the warp holds 2^(j/32), read by
// shuffles.  No branches and no calls: the exponentials of a record pair are
// formed side by side.  Every lane of the warp takes part.
__device__ const double kExp2Of32nds[32] = {AWSEM_EXP2_OF_32NDS};
__device__ const unsigned kExp2Of32ndsLow[32] = {AWSEM_EXP2_OF_32NDS_LOW};
template <typename R> struct GaussTable {};
template <> struct GaussTable<double> {
  double t = kExp2Of32nds[threadIdx.x & 31];
  unsigned low = kExp2Of32ndsLow[threadIdx.x & 31];
};
template <int N> __device__ __forceinline__ void fm_gauss(const double (&z)[N], const GaussTable<double> &tab, double (&g)[N])
{
  constexpr double poly[5] = {AWSEM_GAUSS_POLY};
  double y[N], f[N], q[N];
#pragma unroll
  for (int k = 0; k < N; k++) y[k] = __dadd_rn(z[k], kGaussRound);
#pragma unroll
  for (int k = 0; k < N; k++) f[k] = __dsub_rn(z[k], __dsub_rn(y[k], kGaussRound)), q[k] = kGaussTop;
#pragma unroll
  for (int c = 0; c < 5; c++)
#pragma unroll
    for (int k = 0; k < N; k++) q[k] = __fma_rn(f[k], q[k], poly[c]);
#pragma unroll
  for (int k = 0; k < N; k++)
    q[k] = __fma_rn(f[k], q[k], __hiloint2double((int) __shfl_sync(0xffffffffu, tab.low, __double2loint(y[k]) & 31), 0));
#pragma unroll
  for (int k = 0; k < N; k++) {
    const int n = __double2loint(y[k]);
    const double t = __shfl_sync(0xffffffffu, tab.t, n & 31);
    const double s = __hiloint2double(__double2hiint(t) + ((n >> 5) << 20), __double2loint(t));
    g[k] = z[k] < kGaussLeast ? 0.0 : __fma_rn(s, q[k], s);
  }
}
__device__ __forceinline__ float fm_k2(float s2) { return -1.4426950408889634f / (2.f * s2); }
__device__ __forceinline__ double fm_k2(double s2) { return gauss_factor(s2); }

// One record's four Gaussians g_k (times the record's coefficient when the
// coefficients are not uniform): es += sum g_k, fs_k += g_k dr_k.  The row's
// energy and radial force sums are scale * es and scale * fs_k, with scale =
// -coefficient (uniform) or -1.
// FP32 operand pairs for Blackwell's paired FP32 instructions (f32x2): each
// element is rounded as the scalar operation rounds it.
__device__ __forceinline__ unsigned long long f2_pack(float a, float b)
{
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ void f2_unpack(unsigned long long d, float &a, float &b)
{
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(d));
}
__device__ __forceinline__ unsigned long long f2_sub(unsigned long long a, unsigned long long b)
{
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b)
{
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c)
{
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

template <bool COEF, typename R>
__device__ __forceinline__ void fm_record(const GaussTable<R> &tab, const R rec[4], R cc, const R r[4], R k2, R &es, R fs[4])
{
  if constexpr (sizeof(R) == 4) {
    // atom pairs (0, 1) and (2, 3) as f32x2 pairs: the same operations in
    // the same order as the scalar loop below, half the instructions
    const unsigned long long k22 = f2_pack(k2, k2);
#pragma unroll
    for (int h = 0; h < 4; h += 2) {
      const unsigned long long dr = f2_sub(f2_pack(r[h], r[h + 1]), f2_pack(rec[h], rec[h + 1]));
      float x0, x1;
      f2_unpack(f2_mul(f2_mul(dr, dr), k22), x0, x1);
      float g0 = fm_gauss(x0), g1 = fm_gauss(x1);
      if (COEF) f2_unpack(f2_mul(f2_pack(g0, g1), f2_pack(cc, cc)), g0, g1);
      es = es + g0;
      es = es + g1;
      f2_unpack(f2_fma(f2_pack(g0, g1), dr, f2_pack(fs[h], fs[h + 1])), fs[h], fs[h + 1]);
    }
  } else {
    double dr[4], z[4], g[4];
#pragma unroll
    for (int k = 0; k < 4; k++) dr[k] = r[k] - rec[k], z[k] = dr[k] * dr[k] * k2;
    fm_gauss(z, tab, g);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (COEF) g[k] = g[k] * cc;
      es = es + g[k];
      fs[k] = madd(g[k], dr[k], fs[k]);
    }
  }
}

// Records of an FP64 piece (a multiple of the copy stages' stripes); FP32 rows are one piece.
constexpr int kFmPiece = 32, kFmBlockPieces = 4;
template <typename R> __host__ __device__ constexpr int fm_piece() { return sizeof(R) == 8 ? kFmPiece : 1 << 30; }

// Work unit w: chunk c (separations d0 <= d < d1) of group g; the stripes
// [lo, hi) of its row when a block shares it, whole rows otherwise.
struct FMUnit {
  int g, d0, d1, lo, hi;
};
template <typename R> __device__ __forceinline__ FMUnit fm_unit(int w, const FMSlices<R> &t)
{
  const int g = w / t.dsplit, c = w - g * t.dsplit;
  FMUnit q{g, c * t.nd / t.dsplit, (c + 1) * t.nd / t.dsplit, 0, 1 << 30};
  if (sizeof(R) == 8 && t.psplit > 1) {
    q.lo = kFmPiece * (threadIdx.x >> 5);
    q.hi = q.lo + kFmPiece;
  }
  return q;
}

// Geometry of row (i, j): the four atom-pair differences and distances
template <typename R, class Pos>
__device__ __forceinline__ void fm_row_geometry(const Pos &pos, int i, int j, V3<R> dv[4], R r[4])
{
  const V3<double> ca_i = pos(i, 0), cb_i = pos(i, 1), ca_j = pos(j, 0), cb_j = pos(j, 1);
  dv[0] = diff<R>(ca_i, ca_j);
  dv[1] = diff<R>(ca_i, cb_j);
  dv[2] = diff<R>(cb_i, ca_j);
  dv[3] = diff<R>(cb_i, cb_j);
#pragma unroll
  for (int k = 0; k < 4; k++) r[k] = m_sqrt(norm2(dv[k]));
}

// Where energies go: per residue (stride 1) or all to one total (stride 0),
// in fixed point (2^-32), and apart from it what rounding the rows to that
// left (2^-52), so that an energy is as good as its rows' sums and still the
// same however the rows are spread over units.  (FP64, nine to fourteen
// residues: 5e-10 off with rows in 2^-32 alone, below 7e-12 now.)
struct FMEnergy {
  unsigned long long *high, *low;
  int stride;
};
__device__ __forceinline__ int fix_low(double v, long long high)
{
  return __double2int_rn((v * F_SCALE - (double) high) * F_LOW_SCALE);
}

// Sums of the rows of one unit: the running sums of the current piece, in FP64
// the row's, and in FP32 the unit's forces on residue i in fixed point.  FP64
// rows add their forces on i to memory as they end, from differences formed
// again there: what the record loop holds then fits 12 warps per
// multiprocessor without spills (162 registers).
template <typename R> struct FMSums {
  R es = 0, fs[4] = {0, 0, 0, 0}, es1 = 0, fs1[4] = {0, 0, 0, 0};  // even and odd records
  R et = 0, ft[4] = {0, 0, 0, 0};                                  // FP64: the row's pieces so far
  long long fca[3] = {0, 0, 0}, fcb[3] = {0, 0, 0};
  long long e = 0;  // the rows' energies in fixed point, the same whatever rows share a unit ...
  int e_low = 0;    // ... and what their roundings left

  // a piece ends
  __device__ __forceinline__ void end_piece()
  {
    if constexpr (sizeof(R) == 8) {
      et = et + (es + es1);
#pragma unroll
      for (int k = 0; k < 4; k++) ft[k] = ft[k] + (fs[k] + fs1[k]);
    } else {
      et = es + es1;
#pragma unroll
      for (int k = 0; k < 4; k++) ft[k] = fs[k] + fs1[k];
    }
    es = es1 = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) fs[k] = fs1[k] = 0;
  }
  // the row (i, j) ends: its sums to fixed point
  template <class Pos>
  __device__ __forceinline__ void end_row(R scale, R s2, const R r[4], const V3<R> dv[4], const Pos &pos, int ii,
                                          bool live, int j, unsigned long long *facc)
  {
    const double er = (double) (scale * et);
    const long long ef = fix_force(er);
    e += ef;
    e_low += fix_low(er, ef);
    long long fja[3] = {0, 0, 0}, fjb[3] = {0, 0, 0};
    if constexpr (sizeof(R) == 8) {
      V3<R> dp[4];
      R rp[4];
      fm_row_geometry(pos, ii, j, dp, rp);
      split(scale, s2, rp, dp, fca, fcb, fja, fjb);
      if (live) {
        red_add3(facc + (size_t) 9 * ii, fca);
        red_add3(facc + (size_t) 9 * ii + 3, fcb);
      }
#pragma unroll
      for (int q = 0; q < 3; q++) fca[q] = fcb[q] = 0;
    } else {
      split(scale, s2, r, dv, fca, fcb, fja, fjb);
    }
    red_add3(facc + (size_t) 9 * j, fja);
    red_add3(facc + (size_t) 9 * j + 3, fjb);
    et = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) ft[k] = 0;
  }
  // atom pair k acts on CA(i) (k < 2) or CB(i), and on CA(j) (k even) or CB(j)
  __device__ __forceinline__ void split(R scale, R s2, const R r[4], const V3<R> dv[4], long long ga[3], long long gb[3],
                                        long long ha[3], long long hb[3]) const
  {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const R fc = ft[k] != R(0) ? (scale * ft[k]) / (s2 * r[k]) : R(0);
      const long long v[3] = {fix_force((double) (fc * dv[k].x)), fix_force((double) (fc * dv[k].y)),
                              fix_force((double) (fc * dv[k].z))};
#pragma unroll
      for (int q = 0; q < 3; q++) {
        if (k < 2)
          ga[q] += v[q];
        else
          gb[q] += v[q];
        if (k & 1)
          hb[q] -= v[q];
        else
          ha[q] -= v[q];
      }
    }
  }
  // the unit ends
  __device__ __forceinline__ void end_unit(bool live, int i, unsigned long long *facc, const FMEnergy &to)
  {
    if (sizeof(R) == 4 && live) {
      red_add3(facc + (size_t) 9 * i, fca);
      red_add3(facc + (size_t) 9 * i + 3, fcb);
    }
    long long en = live ? e : 0;
    int lo = live ? e_low : 0;
    size_t at = i;
    if (to.stride == 0) {  // one total: the warp's first
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        en += __shfl_xor_sync(0xffffffffu, en, o);
        lo += __shfl_xor_sync(0xffffffffu, lo, o);
      }
      if ((threadIdx.x & 31) != 0) en = lo = 0;
      at = 0;
    }
    if (en) atomicAdd(to.high + at, (unsigned long long) en);
    if (lo) atomicAdd(to.low + at, (unsigned long long) (long long) lo);
  }
};

// The pieces of a block's row meet (psplit > 1; every thread of the block
// takes part): warp p has piece p's sums (zero where the row has none), and
// warp 0 adds them in order, as one warp alone does.  Returns whether this
// warp now holds the row.
__device__ __forceinline__ bool fm_join_pieces(FMSums<double> &s)
{
  __shared__ double xch[kFmBlockPieces - 1][5][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp) {
    xch[warp - 1][4][lane] = s.et;
#pragma unroll
    for (int k = 0; k < 4; k++) xch[warp - 1][k][lane] = s.ft[k];
  }
  __syncthreads();
  if (warp) return false;
#pragma unroll
  for (int p = 0; p < kFmBlockPieces - 1; p++) {
    s.et = s.et + xch[p][4][lane];
#pragma unroll
    for (int k = 0; k < 4; k++) s.ft[k] = s.ft[k] + xch[p][k][lane];
  }
  return true;
}
__device__ __forceinline__ bool fm_join_pieces(FMSums<float> &) { return true; }

// Work unit w of the fragment-memory term, records loaded into registers.  `pos(r, b)` returns the FP64
// position of residue r's CA (b = 0) or CB (b = 1); forces go to `facc`
// ([atom][3], atom = 3 r + b, fixed point).  Energies are added in fixed
// point to `en`.  sig[s] is the Gaussian variance of sequence
// separation s, |s|^(2 * sigma_exp) (fix_backbone.cpp:4126).
template <bool COEF, typename R, class Pos>
__device__ __forceinline__ void fragmem_unit_reg_t(int w, const FMSlices<R> &t, const double *sig, int n,
                                                   const Pos &pos, unsigned long long *facc,
                                                   const FMEnergy &en)
{
  const int lane = threadIdx.x & 31;
  const FMUnit u = fm_unit(w, t);
  const int i = u.g * 32 + lane;
  const bool live = i < n;
  const int ii = live ? i : n - 1;
  const R scale = COEF ? R(-1) : -R(t.uniform);
  FMSums<R> sum;
  const GaussTable<R> tab;
  for (int d = u.d0; d < u.d1; d++) {
    const int blk = u.g * t.nd + d;
    const int hi = min(u.hi, t.slen[blk]);
    if (t.slen[blk] == 0) continue;
    const size_t base = (size_t) t.soff[blk] * 32 + lane;
    // rows past the end carry padding only; any valid partner index will do
    const int j = min(ii + t.min_sep + d, n - 1);
    V3<R> dv[4];
    R r[4];
    fm_row_geometry(pos, ii, j, dv, r);
    const R s2 = R(sig[t.min_sep + d]);
    const R k2 = fm_k2(s2);
    for (int p0 = u.lo; p0 < hi; p0 += fm_piece<R>()) {
      const int p1 = min(hi - p0, fm_piece<R>()) + p0;
#pragma unroll 2
      for (int m = p0; m < p1; m += 2) {  // block lengths and pieces are even
        const size_t at = base + (size_t) m * 32;
        R rec[4], rec1[4];
        load_record(t.rf, at, rec);
        load_record(t.rf, at + 32, rec1);
        fm_record<COEF>(tab, rec, COEF ? t.coef[at] : R(1), r, k2, sum.es, sum.fs);
        fm_record<COEF>(tab, rec1, COEF ? t.coef[at + 32] : R(1), r, k2, sum.es1, sum.fs1);
      }
      sum.end_piece();
    }
    if (sizeof(R) == 8 && t.psplit > 1 && !fm_join_pieces(sum)) return;
    sum.end_row(scale, s2, r, dv, pos, ii, live, j, facc);
  }
  sum.end_unit(live, i, facc, en);
}

template <typename R, class Pos>
__device__ __forceinline__ void fragmem_unit_reg(int w, const FMSlices<R> &t, const double *sig, int n, const Pos &pos,
                                                 unsigned long long *facc, const FMEnergy &en)
{
  if (t.coef)
    fragmem_unit_reg_t<true>(w, t, sig, n, pos, facc, en);
  else
    fragmem_unit_reg_t<false>(w, t, sig, n, pos, facc, en);
}

// FP32 rows by two warps: warp h (0, 1) of the pair takes a row's even or odd
// records, one of the row's two sets of sums, so the sums are a single warp's
// bit for bit.  Eight records are loaded ahead of their arithmetic.  The odd
// warp hands its sums over in shared memory (xch: two buffers of 5 x 32
// floats, used in turn, so one barrier a row suffices; `bar` is the pair's
// named barrier).  For callers with a warp per unit and no copy ring: on 8,000
// residues with weighted memories (66 MB) a single warp's 120 records in
// series, four loads in flight, held the call at 36 us.
template <bool COEF, class Pos>
__device__ __forceinline__ void fragmem_unit_pair(int w, int h, const FMSlices<float> &t, const double *sig, int n,
                                                  const Pos &pos, unsigned long long *facc, const FMEnergy &en, float *xch, int bar)
{
  constexpr int kAhead = 8;
  const int lane = threadIdx.x & 31;
  const FMUnit u = fm_unit(w, t);
  const int i = u.g * 32 + lane;
  const bool live = i < n;
  const int ii = live ? i : n - 1;
  const float scale = COEF ? -1.f : -(float) t.uniform;
  FMSums<float> sum;
  const GaussTable<float> tab;
  int turn = 0;
  for (int d = u.d0; d < u.d1; d++) {
    const int blk = u.g * t.nd + d, len = t.slen[blk];
    if (len == 0) continue;
    const size_t base = ((size_t) t.soff[blk] + h) * 32 + lane;
    const int j = min(ii + t.min_sep + d, n - 1), half = len / 2;  // len is even
    float rec[kAhead][4], cf[kAhead];
    auto load = [&](int k, int m) {
      const size_t at = base + (size_t) m * 64;
      load_record(t.rf, at, rec[k]);
      cf[k] = COEF ? t.coef[at] : 1.f;
    };
#pragma unroll
    for (int k = 0; k < kAhead; k++)
      if (k < half) load(k, k);
    V3<float> dv[4];
    float r[4];
    fm_row_geometry(pos, ii, j, dv, r);
    const float s2 = (float) sig[t.min_sep + d], k2 = fm_k2(s2);
    for (int m0 = 0; m0 < half; m0 += kAhead) {
#pragma unroll
      for (int k = 0; k < kAhead; k++) {
        if (m0 + k < half) fm_record<COEF>(tab, rec[k], cf[k], r, k2, sum.es, sum.fs);
        if (m0 + k + kAhead < half) load(k, m0 + k + kAhead);
      }
    }
    float *buf = xch + turn * 160 + lane;
    turn ^= 1;
    if (h) {
      buf[0] = sum.es;
#pragma unroll
      for (int k = 0; k < 4; k++) buf[32 * (k + 1)] = sum.fs[k];
    }
    asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
    if (!h) {
      sum.es1 = buf[0];
#pragma unroll
      for (int k = 0; k < 4; k++) sum.fs1[k] = buf[32 * (k + 1)];
      sum.end_piece();
      sum.end_row(scale, s2, r, dv, pos, ii, live, j, facc);
    } else {
      sum.es = 0.f;
#pragma unroll
      for (int k = 0; k < 4; k++) sum.fs[k] = 0.f;
    }
  }
  if (!h) sum.end_unit(live, i, facc, en);
}

// A launch with one warp per work unit, 128 threads a block; a block where
// psplit says so (FP64, sharing a row), a warp pair with PAIR (FP32: kernels of
// their own, in one the pair form was 5% slower)
template <bool PAIR, typename R, class Pos>
__device__ __forceinline__ void fragmem_warp(const FMSlices<R> &t, const double *sig, int n, const Pos &pos,
                                             unsigned long long *facc, const FMEnergy &en)
{
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if constexpr (PAIR) {
    __shared__ float xch[2][320];
    const int pair = (threadIdx.x >> 6) & 1;
    if (w / 2 >= t.groups * t.dsplit) return;  // both warps of the pair
    if (t.coef)
      fragmem_unit_pair<true>(w / 2, w & 1, t, sig, n, pos, facc, en, xch[pair], 1 + pair);
    else
      fragmem_unit_pair<false>(w / 2, w & 1, t, sig, n, pos, facc, en, xch[pair], 1 + pair);
  } else {
    const int u = t.psplit > 1 ? (int) blockIdx.x : w;
    if (u < t.groups * t.dsplit) fragmem_unit_reg(u, t, sig, n, pos, facc, en);
  }
}

// ---------------------------------------------------------------------------
// Bulk-copy pipeline.  A group's blocks are contiguous stripes, so a warp's
// whole share is one contiguous run of stripes: lane 0 streams it into a
// ring of kFmStages shared-memory stages of kFmStripes<R> stripes with 1-D bulk
// copies (cp.async.bulk, the TMA engine) completing on one mbarrier per
// stage, and the 32 lanes read their records from shared memory.  Up to
// kFmStages stages are in flight per warp with no register cost, which is
// what the register-load version lacks at full size.  Per lane the records
// are consumed in the same order, so the sums equal the register version's
// bit for bit.
// A stage is 4 KiB of distances in both forms: eight FP32 stripes (bandwidth
// bound: 3 x 4 KiB in flight a warp) or four FP64 ones (arithmetic bound; with
// eight, 25 KiB a warp left room for 8 warps per SM).
constexpr int kFmStages = 3;
template <typename R> constexpr int kFmStripes = sizeof(R) == 4 ? 8 : 4;

template <typename R> __host__ __device__ constexpr int fm_stage_bytes(bool coef)
{
  return kFmStripes<R> * 32 * (int) sizeof(R) * (coef ? 5 : 4);
}
// shared memory of one warp: 128 bytes of mbarriers, then the stages
template <typename R> __host__ __device__ constexpr int fm_warp_smem(bool coef)
{
  return 128 + kFmStages * fm_stage_bytes<R>(coef);
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// Wait for phase `parity` of an mbarrier, giving up after `limit` clock
// cycles (false: timed out).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, long long limit)
{
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > limit) return false;
  }
}

constexpr long long kFmWaitLimit = 4000000000LL;  // about two seconds at 2 GHz

__device__ __forceinline__ void load_record_shared(const float *rf, int rec, float m[4])
{
  const float4 v = reinterpret_cast<const float4 *>(rf)[rec];
  m[0] = v.x, m[1] = v.y, m[2] = v.z, m[3] = v.w;
}
__device__ __forceinline__ void load_record_shared(const double *rf, int rec, double m[4])
{
  const double2 *q = reinterpret_cast<const double2 *>(rf) + 2 * rec;
  const double2 u = q[0], v = q[1];
  m[0] = u.x, m[1] = u.y, m[2] = v.x, m[3] = v.y;
}

// One work unit (group g, chunk c of its separations) of a warp.  The warp's
// mbarriers keep counting phases across its units: chunk k of this unit is
// the warp's chunk kbase + k (stage (kbase + k) % kFmStages).  Returns false
// when a wait gave up.
template <bool COEF, typename R, class Pos>
__device__ __forceinline__ bool fragmem_unit_bulk_t(int w, const FMSlices<R> &t, const double *sig, int n,
                                                    const Pos &pos, unsigned long long *facc,
                                                    const FMEnergy &en, int *timed_out,
                                                    unsigned char *wsm, unsigned &kbase)
{
  const int lane = threadIdx.x & 31;
  const FMUnit u = fm_unit(w, t);
  const int g = u.g, d1 = u.d1;
  const int i = g * 32 + lane;
  const bool live = i < n;
  const int ii = live ? i : n - 1;
  const bool coef = COEF;
  const int stage_bytes = fm_stage_bytes<R>(coef);
  const uint32_t bars = smem_addr(wsm), data = bars + 128;
  // the warp's run of stripes: its non-empty blocks, contiguous from the first
  int first = -1, total = 0;
  for (int dd = u.d0; dd < d1; dd++) {
    const int len = min(u.hi, t.slen[g * t.nd + dd]) - u.lo;
    if (len <= 0) continue;
    if (first < 0) first = t.soff[g * t.nd + dd] + u.lo;
    total += len;
  }
  FMSums<R> sum;
  if (total <= 0) {
    // a block's warp without a piece still joins the others
    if (sizeof(R) == 8 && t.psplit > 1 && t.slen[g * t.nd + u.d0] > 0) fm_join_pieces(sum);
    return true;
  }
  const int last = first + total, nchunks = (total + kFmStripes<R> - 1) / kFmStripes<R>;
  auto issue = [&](int k) {  // lane 0: chunk k into stage (kbase + k) % kFmStages
    const int st = (kbase + k) % kFmStages, s0 = first + k * kFmStripes<R>, ns = min(kFmStripes<R>, last - s0);
    const uint32_t bar = bars + 8 * st, dst = data + st * stage_bytes;
    const uint32_t rb = ns * 32 * 4 * sizeof(R), cb = coef ? ns * 32 * sizeof(R) : 0;
    // the stage was last read through the generic proxy: order that before the async-proxy write
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect(bar, rb + cb + t.hold_tx);
    bulk_load(dst, t.rf + (size_t) s0 * 32 * 4, rb, bar);
    if (coef) bulk_load(dst + kFmStripes<R> * 32 * 4 * sizeof(R), t.coef + (size_t) s0 * 32, cb, bar);
  };
  if (lane == 0)
    for (int k = 0; k < kFmStages && k < nchunks; k++) issue(k);

  const R scale = COEF ? R(-1) : -R(t.uniform);
  const GaussTable<R> tab;
  // current row (block d): geometry, its end and its current piece's end
  int d = u.d0, row_end = 0, piece_end = 0, j = 0;
  V3<R> dv[4];
  R r[4], s2 = 1, k2 = -1;
  auto begin_row = [&]() {  // d: the next non-empty block at or after d
    while (d < d1 && t.slen[g * t.nd + d] == 0) d++;
    if (d >= d1) return;
    const int row0 = t.soff[g * t.nd + d] + u.lo - first;
    row_end = row0 + min(u.hi, t.slen[g * t.nd + d]) - u.lo;
    piece_end = min(row_end - row0, fm_piece<R>()) + row0;
    j = min(ii + t.min_sep + d, n - 1);
    fm_row_geometry(pos, ii, j, dv, r);
    s2 = R(sig[t.min_sep + d]);
    k2 = fm_k2(s2);
  };
  begin_row();
  bool ok = true;
  int fail_k = 0;
  for (int k = 0; k < nchunks; k++) {
    const int st = (kbase + k) % kFmStages;
    // the warp gives up together (every lane polls the same barrier)
    if (!__all_sync(0xffffffffu, mbar_wait(bars + 8 * st, ((kbase + k) / kFmStages) & 1, t.wait_limit))) {
      ok = false;
      fail_k = k;
      break;
    }
    const unsigned char *sd = wsm + 128 + st * stage_bytes;
    const R *srf = reinterpret_cast<const R *>(sd);
    const R *scf = reinterpret_cast<const R *>(sd + kFmStripes<R> * 32 * 4 * sizeof(R));
    const int s0 = k * kFmStripes<R>, ns = min(kFmStripes<R>, total - s0);
    for (int q = 0; q < ns;) {
      while (s0 + q >= piece_end && d < d1) {  // pieces and rows end on stripe boundaries
        sum.end_piece();
        if (sizeof(R) == 8 && piece_end < row_end) {  // FP32 rows are one piece
          piece_end = min(row_end - piece_end, fm_piece<R>()) + piece_end;
        } else {
          sum.end_row(scale, s2, r, dv, pos, ii, live, j, facc);
          d++;
          begin_row();
        }
      }
      // the stripes of this chunk that belong to the current piece (pieces,
      // chunks and their ends fall on even stripes: records pair up as in
      // the register path)
      const int run = max(q + 2, min(ns, piece_end - s0));
#pragma unroll(sizeof(R) == 4 ? 2 : 1)
      for (; q < run; q += 2) {
        R rec[4], rec1[4];
        load_record_shared(srf, q * 32 + lane, rec);
        load_record_shared(srf, (q + 1) * 32 + lane, rec1);
        fm_record<COEF>(tab, rec, COEF ? scf[q * 32 + lane] : R(1), r, k2, sum.es, sum.fs);
        fm_record<COEF>(tab, rec1, COEF ? scf[(q + 1) * 32 + lane] : R(1), r, k2, sum.es1, sum.fs1);
      }
    }
    __syncwarp();  // every lane has read the stage
    if (lane == 0 && k + kFmStages < nchunks) issue(k + kFmStages);
  }
  if (!ok) {
    // record the failure, let the copies in flight land (bounded), skip the sums
    if (lane == 0) atomicExch(timed_out, 1);
    for (int k = fail_k; k < nchunks && k < fail_k + kFmStages; k++)
      mbar_wait(bars + 8 * ((kbase + k) % kFmStages), ((kbase + k) / kFmStages) & 1, kFmWaitLimit / 8);
    if (sizeof(R) == 8 && t.psplit > 1) fm_join_pieces(sum);  // the block's other warps wait there
    return false;
  }
  kbase += nchunks;
  sum.end_piece();
  if (sizeof(R) == 8 && t.psplit > 1 && !fm_join_pieces(sum)) return true;
  sum.end_row(scale, s2, r, dv, pos, ii, live, j, facc);
  sum.end_unit(live, i, facc, en);
  return true;
}

template <typename R, class Pos>
__device__ __forceinline__ bool fragmem_unit_bulk(int w, const FMSlices<R> &t, const double *sig, int n,
                                                  const Pos &pos, unsigned long long *facc,
                                                  const FMEnergy &en, int *timed_out,
                                                  unsigned char *wsm, unsigned &kbase)
{
  return t.coef ? fragmem_unit_bulk_t<true>(w, t, sig, n, pos, facc, en, timed_out, wsm, kbase)
                : fragmem_unit_bulk_t<false>(w, t, sig, n, pos, facc, en, timed_out, wsm, kbase);
}

// A warp's copy ring: its stage mbarriers, initialised once (the phase
// count then runs on across the warp's units through kbase).
__device__ __forceinline__ void fragmem_ring_init(unsigned char *wsm)
{
  const uint32_t bars = smem_addr(wsm);
  if ((threadIdx.x & 31) == 0)
    for (int s = 0; s < kFmStages; s++) mbar_init(bars + 8 * s, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncwarp();
}

// The kernel body: each warp takes work units one at a time from a counter
// (zero at launch), so a grid smaller than the number of units (a few blocks
// per SM) still streams at full bandwidth and leaves the rest of each SM to
// the concurrent pair passes; warps that get more of their SM take more
// units, and the launch ends within one unit of balance.
template <typename R, class Pos>
__device__ __forceinline__ void fragmem_warp_take(const FMSlices<R> &t, const double *sig, int n, const Pos &pos,
                                                  unsigned long long *facc, const FMEnergy &en, int *timed_out, unsigned char *wsm, int *next)
{
  const int units = t.groups * t.dsplit, lane = threadIdx.x & 31;
  fragmem_ring_init(wsm);
  unsigned kbase = 0;
  if (sizeof(R) == 8 && t.psplit > 1) {  // a block takes a unit (both barriers: its warps stay together, also when one's wait gave up)
    __shared__ int s_u;
    while (true) {
      if (threadIdx.x == 0) s_u = atomicAdd(next, 1);
      __syncthreads();
      const int u = s_u;
      if (u >= units) return;
      const bool ok = fragmem_unit_bulk(u, t, sig, n, pos, facc, en, timed_out, wsm, kbase);
      if (!__syncthreads_and(ok)) return;
    }
  }
  while (true) {
    int u = 0;
    if (lane == 0) u = atomicAdd(next, 1);
    u = __shfl_sync(0xffffffffu, u, 0);
    if (u >= units) return;
    if (!fragmem_unit_bulk(u, t, sig, n, pos, facc, en, timed_out, wsm, kbase)) return;
  }
}

}  // namespace dev

// A handle's resident fragment-memory table, for entry points outside the
// engine: the slices with the element type erased, plus the variance table.
struct FMView {
  const int *soff, *slen;
  const void *rf, *coef;  // double (FP64 form) or float (mixed form) elements
  double uniform;
  int nd, min_sep, groups, dsplit, psplit, n_res, is_double;
  const double *sigma_sq;  // host table [64]
};

}  // namespace awsem
