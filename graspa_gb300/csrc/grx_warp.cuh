// grx_warp.cuh -- the trial-bead pair engine: tile culling, FP32 screening, warp
// compaction of in-cutoff pairs and dense evaluation.
//
// A work item is (one trial bead, one range of host units [+ the guest atoms]) and is
// processed by one warp. A host unit is a 32-entry chunk of the bead's voxel list or a 32-atom
// tile, whose bounds are tested against the cutoff first; the 32 pairs of a unit are screened
// in FP32 (in the FP64 form only where FP32 decides, see pair_screen). Pairs inside the
// screening radius are appended to a per-warp ring buffer in shared memory; every 32 queued
// pairs are evaluated by all 32 lanes together, so the costly part (displacement, LJ,
// real-space Coulomb) runs without idle lanes. The order of every sum is fixed by the ballot
// order, so results are deterministic.
#pragma once

#include <limits.h>

#include "grx_internal.cuh"
#include "grx_df.cuh"

namespace grx {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kQueue = 64;  // ring buffer entries per warp

// The mixed form of the single-molecule delta: split FP32 screening and FP32 LJ outside 1.1
// sigma as in GRX_MIXED, displacement, LJ inside and real-space Coulomb in FP64. A move's two
// configurations share nearly all of their energy, so the double-float Coulomb of the trial
// passes would show in their difference.
constexpr int kMixed64 = 3;

// Round to the nearest integer with two FP32 instructions (|x| < 2^22): adding
// 1.5*2^23 moves the fraction out of the mantissa. Differs from the reference's
// int-cast rounding only at exact half-cell ties, which lie beyond the cutoff.
__device__ __forceinline__ float rnd(float x) {
  return __fsub_rn(__fadd_rn(x, 12582912.0f), 12582912.0f);
}

// Minimum-image displacement on split coordinates: the image shift is applied to the
// hi part with the grid-exact cell (exact) and to the lo part with the remainder.
__device__ __forceinline__ void image_split(const BoxDev& b, float3& dh, float3& dl) {
  const float x = dh.x + dl.x, y = dh.y + dl.y, z = dh.z + dl.z;
  if (b.cubic) {
    const float nx = rnd(x * b.invf[0]), ny = rnd(y * b.invf[4]), nz = rnd(z * b.invf[8]);
    dh.x = __fmaf_rn(-nx, b.cell_hi[0], dh.x); dl.x = __fmaf_rn(-nx, b.cell_lo[0], dl.x);
    dh.y = __fmaf_rn(-ny, b.cell_hi[4], dh.y); dl.y = __fmaf_rn(-ny, b.cell_lo[4], dl.y);
    dh.z = __fmaf_rn(-nz, b.cell_hi[8], dh.z); dl.z = __fmaf_rn(-nz, b.cell_lo[8], dl.z);
  } else {
    const float nx = rnd(b.invf[0] * x + b.invf[3] * y + b.invf[6] * z);
    const float ny = rnd(b.invf[1] * x + b.invf[4] * y + b.invf[7] * z);
    const float nz = rnd(b.invf[2] * x + b.invf[5] * y + b.invf[8] * z);
    dh.x = __fmaf_rn(-nz, b.cell_hi[6], __fmaf_rn(-ny, b.cell_hi[3], __fmaf_rn(-nx, b.cell_hi[0], dh.x)));
    dh.y = __fmaf_rn(-nz, b.cell_hi[7], __fmaf_rn(-ny, b.cell_hi[4], __fmaf_rn(-nx, b.cell_hi[1], dh.y)));
    dh.z = __fmaf_rn(-nz, b.cell_hi[8], __fmaf_rn(-ny, b.cell_hi[5], __fmaf_rn(-nx, b.cell_hi[2], dh.z)));
    dl.x -= nx * b.cell_lo[0] + ny * b.cell_lo[3] + nz * b.cell_lo[6];
    dl.y -= nx * b.cell_lo[1] + ny * b.cell_lo[4] + nz * b.cell_lo[7];
    dl.z -= nx * b.cell_lo[2] + ny * b.cell_lo[5] + nz * b.cell_lo[8];
  }
}

// Screening test of one pair (true when it may lie inside a cutoff): FP32 on the hi parts alone
// (16 bytes per atom), against a radius padded for the hi rounding. The FP64 form tests every
// pair again exactly in its dense evaluation, so it screens in FP32 as well and lets through
// what FP32 cannot decide: far coordinates (kNearCoord) and, in triclinic cells, fractions next
// to a tie, where the two images differ in length. (An FP64 screen costs about 20 FP64
// operations per candidate, as much as the dense evaluation of a pair inside the cutoff.)
template <int PREC>
__device__ __forceinline__ bool screen_hi(const BoxDev& b, float4 ah, const Bead& bd) {
  float x = ah.x - bd.h.x, y = ah.y - bd.h.y, z = ah.z - bd.h.z;
  bool open = false;
  if (PREC == GRX_FP64)
    open = !(bd.unit & 2) || !(fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z)) < kNearCoord);
  if (b.cubic) {
    x = __fmaf_rn(-rnd(x * b.invf[0]), b.cellf[0], x);
    y = __fmaf_rn(-rnd(y * b.invf[4]), b.cellf[4], y);
    z = __fmaf_rn(-rnd(z * b.invf[8]), b.cellf[8], z);
  } else {
    const float sx = b.invf[0] * x + b.invf[3] * y + b.invf[6] * z;
    const float sy = b.invf[1] * x + b.invf[4] * y + b.invf[7] * z;
    const float sz = b.invf[2] * x + b.invf[5] * y + b.invf[8] * z;
    const float nx = rnd(sx), ny = rnd(sy), nz = rnd(sz);
    if (PREC == GRX_FP64) open = open || fmaxf(fmaxf(fabsf(sx - nx), fabsf(sy - ny)), fabsf(sz - nz)) > b.tie;
    x -= nx * b.cellf[0] + ny * b.cellf[3] + nz * b.cellf[6];
    y -= nx * b.cellf[1] + ny * b.cellf[4] + nz * b.cellf[7];
    z -= nx * b.cellf[2] + ny * b.cellf[5] + nz * b.cellf[8];
  }
  return x * x + y * y + z * z < b.screen2 || open;
}

template <int PREC, bool HOST>
__device__ __forceinline__ bool pair_screen(const BoxDev& b, int i, const Bead& bd) {
  return screen_hi<PREC>(b, HOST ? b.hrec[2 * i] : b.hi[i], bd);
}

// 32 read-only bytes in one load. The gathers of the pair evaluation go to a different line for
// most lanes, so their cost is line lookups, one per lane and load: a record or table piece of
// two float4 in one 256-bit load takes half of them.
__device__ __forceinline__ void load32(const float4* p, float4& a, float4& c) {
  unsigned long long q0, q1, q2, q3;
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(q0), "=l"(q1), "=l"(q2), "=l"(q3) : "l"(p));
  a = make_float4(__uint_as_float((unsigned)q0), __uint_as_float((unsigned)(q0 >> 32)), __uint_as_float((unsigned)q1),
                  __uint_as_float((unsigned)(q1 >> 32)));
  c = make_float4(__uint_as_float((unsigned)q2), __uint_as_float((unsigned)(q2 >> 32)), __uint_as_float((unsigned)q3),
                  __uint_as_float((unsigned)(q3 >> 32)));
}

// ---------------------------------------------------------------- FP64 pairs
// An SM retires two FP64 lanes per clock, so a warp's FP64 instruction takes 16 cycles of the
// SM and the FP64 form is bound by how many a pair needs. Images come from FP32 fractions and
// a table of lattice vectors (6 subtractions instead of about 15 operations of the rounded
// fractions), g and h from tables, LJ from one reciprocal, and the cutoff and overlap
// tests from integer comparisons of the words: 28 FP64 operations for a charged pair where the
// library form took about 150, and none per screened candidate where it took 20. CO2 in silica:
// 1500 Widom insertions 6.04 -> 1.40 ms, 10 steps of 152 GCMC chains 5.93 -> 1.77 ms.

// Minimum image of (x, y, z), whose hi parts differ by (fx, fy, fz): the reference's rounded
// fractions where FP32 decides them (pbc64 near a tie, for far coordinates and far images).
__device__ __forceinline__ void image64(const BoxDev& b, bool near, float fx, float fy, float fz, double& x, double& y,
                                        double& z) {
  float sx, sy, sz;
  if (b.cubic) {
    sx = fx * b.invf[0]; sy = fy * b.invf[4]; sz = fz * b.invf[8];
  } else {
    sx = b.invf[0] * fx + b.invf[3] * fy + b.invf[6] * fz;
    sy = b.invf[1] * fx + b.invf[4] * fy + b.invf[7] * fz;
    sz = b.invf[2] * fx + b.invf[5] * fy + b.invf[8] * fz;
  }
  const float nx = rnd(sx), ny = rnd(sy), nz = rnd(sz);
  const float off = fmaxf(fmaxf(fabsf(sx - nx), fabsf(sy - ny)), fabsf(sz - nz));
  const float top = fmaxf(fmaxf(fabsf(nx), fabsf(ny)), fabsf(nz));
  if (near && off < b.tie && top <= 1.0f && fmaxf(fmaxf(fabsf(fx), fabsf(fy)), fabsf(fz)) < kNearCoord) {
    const float idx = __fmaf_rn(9.0f, nz, __fmaf_rn(3.0f, ny, nx + 13.0f));
    const double2* v = reinterpret_cast<const double2*>(b.img) + 2 * (__float_as_int(idx + 12582912.0f) & 31);
    const double2 v0 = __ldg(v), v1 = __ldg(v + 1);
    x -= v0.x; y -= v0.y; z -= v1.x;
  } else {
    pbc64(b, x, y, z);
  }
}

// One piecewise quintic of grx_table.cu; k: the piece of s.
template <int SHIFT>
__device__ __forceinline__ int table64_piece(double s, int base) { return (__double2hiint(s) >> SHIFT) - base; }
template <int SHIFT>
__device__ __forceinline__ double table64(const double2* t, int k, double s) {
  const double2 a = __ldg(t + 3 * k), c = __ldg(t + 3 * k + 1), e = __ldg(t + 3 * k + 2);
  const int centre = (__double2hiint(s) & -(1 << SHIFT)) | (1 << (SHIFT - 1));
  const double u = s - __hiloint2double(centre, 0);
  return fma(u, fma(u, fma(u, fma(u, fma(u, e.y, e.x), c.y), c.x), a.y), a.x);
}

// 1/x for a normal x: the hardware's 20-bit estimate y refined by the third-order iteration
// y (1 + e + e^2), e = 1 - x y (Householder), to about one rounding.
__device__ __forceinline__ double recip64(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// 4 eps [(sigma^2/r^2)^6 - (sigma^2/r^2)^3] - shift in double-float (full molecules),
// used by the mixed form inside 1.1 sigma where FP32 rounding of the steep repulsion
// would exceed the error budget.
__device__ __forceinline__ df lj_df(const BoxDev& b, int row, df rr) {
  const float4 f = b.ffdf[row];
  const float2 sh = b.ffdf2[row];
  const df t = df_mul(rr, df{f.z, f.w});
  const df t3 = df_mul(df_mul(t, t), t);
  const df rri3 = df_recip(t3);
  const df term = df_mul(df{f.x, f.y}, df_mul(rri3, df_add_f(rri3, -1.0f)));
  return df_add(term, df{-sh.x, -sh.y});
}

// g(s) = erfc(alpha sqrt s)/sqrt s in double-float from piece k of the table. The piece's start
// s0 is s with the low 17 bits cleared and its width a power of two, so t = (s - s0)/width is
// formed exactly from the two halves of s, without loading either. Over one piece the terms of
// order >= 2 are ~1e-4 of g, so they are summed in FP32; the first two orders keep their low
// parts, not renormalised in between (|c0| > |c1 t| and |c1| > |t tail| hold on every piece).
// 26 instructions and two 16-byte loads; the normalised form took 44 and four. On the CO2-silica
// batch of 456 chains x 50 steps, with the accumulation below: 7.16 -> 6.79 ms, 20,000 Widom
// insertions 6.60 -> 5.79 ms.
__device__ __forceinline__ df coul_table_df(const BoxDev& b, int k, df s) {
  float4 c0, c1;
  load32(b.ctabf + 2 * k, c0, c1);
  const int bits = __float_as_int(s.hi);
  const float inv = __int_as_float((260 << 23) - (bits & 0x7f800000));  // 64 / 2^exponent
  const float t = __fmul_rn(__fsub_rn(s.hi, __int_as_float(bits & ~0x1ffff)), inv), tl = __fmul_rn(s.lo, inv);
  const float tail = __fmaf_rn(__fmaf_rn(__fmaf_rn(c1.w, t, c1.z), t, c1.y), t, c1.x);
  df p = two_prod(t, tail);
  p.lo = __fmaf_rn(tl, tail, p.lo);
  const df q = fast_two_sum(c0.z, p.hi);
  const float ql = __fadd_rn(q.lo, __fadd_rn(p.lo, c0.w));
  df m = two_prod(t, q.hi);
  m.lo = __fmaf_rn(t, ql, __fmaf_rn(tl, q.hi, m.lo));
  const df g = fast_two_sum(c0.x, m.hi);
  return {g.hi, __fadd_rn(g.lo, __fadd_rn(m.lo, c0.y))};
}

// Cold paths of the mixed-precision pair evaluation, kept out of line so the inlined copies of
// pair_dense stay small: LJ inside 1.1 sigma (double-float), LJ with a non-unit scaling or the
// 12-6-4 form, and g(s) outside the Coulomb table's range.
static __device__ __noinline__ float2 lj_df_cold(const BoxDev& b, int row, float rhi, float rlo) {
  const df e = lj_df(b, row, df{rhi, rlo});
  return make_float2(e.hi, e.lo);
}
static __device__ __noinline__ double vdw64_cold(const BoxDev& b, int row, double rr, double scaling) {
  return vdw64(b, row, rr, scaling);
}
static __device__ __noinline__ double coul_g_cold(const BoxDev& b, double rr) {
  const double r = sqrt(rr);
  return erfc(b.alpha * r) / r;
}

// Accumulators of one lane: FP64 for the FP64 and FP32 forms, double-float for mixed.
template <int PREC> struct LaneAcc { double v = 0.0, r = 0.0; };
template <> struct LaneAcc<GRX_MIXED> { df v = {0.f, 0.f}, r = {0.f, 0.f}; };

// Dense evaluation of one screened pair in the split forms, from its displacement (dh, dl): exact
// cutoff tests, LJ, real Coulomb, overlap flag (VDW_Coulomb.cu:1287-1322). row: type pair; sc1: the
// atom's scale is 1; qa: its charge as a float pair.
template <int PREC>
__device__ __forceinline__ void pair_core(const BoxDev& b, bool host, int i, const Bead& bd, float3 dh, float3 dl,
                                          int row, bool sc1, float2 qa, LaneAcc<PREC>& acc, int& flag) {
  if constexpr (PREC == kMixed64) {
    const double x = (double)dh.x + (double)dl.x;
    const double y = (double)dh.y + (double)dl.y;
    const double z = (double)dh.z + (double)dl.z;
    const double rr = x * x + y * y + z * z;
    if (rr < b.cut_vdw2) {
      const float4 f = b.ff32[row];
      const bool unit = sc1 && (bd.unit & 1) && !b.use_1264;
      double e;
      if (unit && (float)rr > f.w) e = (double)vdw32(f, (float)rr);
      else e = vdw64_cold(b, row, rr, (host ? b.hscale : b.scale)[i] * bd.scale);
      if (e > b.overlap) flag = 1;
      if (rr < 0.01) flag = 1;
      acc.v += e;
    }
    if (!b.no_charges && rr < b.cut_coul2) {
      const int k = table64_piece<kShiftG64>(rr, b.g64_base);
      double g;
      if ((unsigned)k < (unsigned)b.g64_n) g = table64<kShiftG64>(b.g64, k, rr);
      else g = coul_g_cold(b, rr);
      acc.r = fma((host ? b.hpos64 : b.pos64)[i].w, g, acc.r);
    }
  } else if constexpr (PREC == GRX_MIXED) {
    const df s = df_norm2_split(dh, dl);
    if (df_lt(s, df{b.cut_vdw2_df.x, b.cut_vdw2_df.y})) {
      const float4 f = b.ff32[row];
      const bool unit = sc1 && (bd.unit & 1) && !b.use_1264;
      df e;
      if (unit && s.hi > f.w) e = df{vdw32(f, s.hi), 0.0f};
      else if (unit) {
        const float2 c = lj_df_cold(b, row, s.hi, s.lo);
        e = df{c.x, c.y};
      }
      else e = df_from(vdw64_cold(b, row, df_to(s), (host ? b.hscale : b.scale)[i] * bd.scale));
      if (e.hi > b.overlapf) flag = 1;
      if (s.hi < 0.01f) flag = 1;
      df_accumulate(acc.v, e.hi, e.lo);
    }
    if (!b.no_charges && df_lt(s, df{b.cut_coul2_df.x, b.cut_coul2_df.y})) {
      df g;
      const int k = (__float_as_int(s.hi) >> 17) - b.ctab_base;
      if ((unsigned)k < (unsigned)b.ctab_n) g = coul_table_df(b, k, s);
      else g = df_from(coul_g_cold(b, df_to(s)));
      const df e = two_prod(g.hi, qa.x);  // prefactor * q_bead applied once per item
      df_accumulate(acc.r, e.hi, __fmaf_rn(g.hi, qa.y, __fmaf_rn(g.lo, qa.x, e.lo)));
    }
  } else {  // GRX_FP32
    const float fx = dh.x + dl.x, fy = dh.y + dl.y, fz = dh.z + dl.z;
    const float rr32 = fx * fx + fy * fy + fz * fz;
    if (rr32 < b.cut_vdw2f) {
      const float sc = (sc1 ? 1.0f : (float)(host ? b.hscale : b.scale)[i]) * (float)bd.scale;
      float e;
      if (sc == 1.0f && !b.use_1264) e = vdw32(b.ff32[row], rr32);
      else e = (float)vdw64(b, row, (double)rr32, (double)sc);
      if (e > b.overlapf) flag = 1;
      if (rr32 < 0.01f) flag = 1;
      acc.v += (double)e;
    }
    if (!b.no_charges && rr32 < b.cut_coul2f) acc.r += (double)coul32(b, qa.x * (float)bd.q, rr32);
  }
}

// The same in FP64 (host: atom i is a framework atom, else a guest).
__device__ __forceinline__ void pair_fp64(const BoxDev& b, bool host, int i, const Bead& bd, LaneAcc<GRX_FP64>& acc,
                                          int& flag) {
  float4 ah;
  double4 p;
  int ty;
  bool sc1;
  if (host) {
    ah = b.hrec[2 * i];
    p = b.hpos64[i];
    const unsigned t = b.htype[i];
    ty = (int)(t & 0x7fffu);
    sc1 = !(t & 0x8000u);
  } else {
    ah = b.hi[i];
    p = b.pos64[i];
    ty = b.meta[i].x;
    sc1 = __double_as_longlong(b.scale[i]) == 0x3ff0000000000000ll;
  }
  double x = p.x - bd.x, y = p.y - bd.y, z = p.z - bd.z;
  image64(b, (bd.unit & 2) != 0, ah.x - bd.h.x, ah.y - bd.h.y, ah.z - bd.h.z, x, y, z);
  const double rr = x * x + y * y + z * z;
  // non-negative doubles (and NaN above all of them) order as their words do
  const unsigned long long rb = (unsigned long long)__double_as_longlong(rr);
  const int rh = __double2hiint(rr);
  if (rb < (unsigned long long)__double_as_longlong(b.cut_vdw2)) {
    const int row = ty * b.ntypes + bd.type;
    double e;
    if (sc1 && (bd.unit & 1) && !b.use_1264 && rh >= 0x3fd00000) {  // full molecules, r >= 0.5 A
      const double2* f = reinterpret_cast<const double2*>(b.ff64 + row);
      const double2 f0 = __ldg(f), f1 = __ldg(f + 1);  // {4 eps, sigma}, {sigma^2, shift}
      const double r = recip64(rr);
      double u = f1.x * r;
      u = fma(fma(-rr, u, f1.x), r, u);  // sigma^2 / r^2, the rounding of the product taken out
      const double u3 = u * u * u;
      e = fma(f0.x, fma(u3, u3, -u3), -f1.y);
    } else {
      e = vdw64_cold(b, row, rr, (host ? b.hscale : b.scale)[i] * bd.scale);
    }
    if (__double2hiint(e) >= b.overlap_hi && e > b.overlap) flag = 1;
    if (rh <= 0x3f847ae1 && rr < 0.01) flag = 1;
    acc.v += e;
  }
  if (!b.no_charges && rb < (unsigned long long)__double_as_longlong(b.cut_coul2)) {
    const int k = table64_piece<kShiftG64>(rr, b.g64_base);
    double g;
    if ((unsigned)k < (unsigned)b.g64_n) g = table64<kShiftG64>(b.g64, k, rr);
    else g = coul_g_cold(b, rr);
    acc.r = fma(p.w, g, acc.r);  // prefactor * q_bead applied once per item
  }
}

// Atom i with the image of rounded fractions: framework atoms of the tile path, guests.
template <int PREC>
__device__ __forceinline__ void pair_dense(const BoxDev& b, bool host, int i, const Bead& bd, LaneAcc<PREC>& acc,
                                           int& flag) {
  if constexpr (PREC == GRX_FP64) {
    pair_fp64(b, host, i, bd, acc, flag);
  } else {
    // host atoms from their records (one 32-byte sector: split position and charge, plus the
    // 2-byte type); guest atoms from the per-field arrays
    float4 ah, al;
    int ty;
    bool sc1;  // the atom's scale is 1
    float2 qa;
    if (host) {
      load32(b.hrec + 2 * i, ah, al);
      const unsigned t = __ldg(b.htype + i);
      ty = (int)(t & 0x7fffu);
      sc1 = !(t & 0x8000u);
      qa = make_float2(ah.w, al.w);
    } else {
      ah = b.hi[i];
      al = b.lo[i];
      ty = b.meta[i].x;
      sc1 = al.w == 1.0f;
      qa = b.qdf[i];
    }
    float3 dh = make_float3(ah.x - bd.h.x, ah.y - bd.h.y, ah.z - bd.h.z);
    float3 dl = make_float3(al.x - bd.l.x, al.y - bd.l.y, al.z - bd.l.z);
    image_split(b, dh, dl);
    pair_core<PREC>(b, host, i, bd, dh, dl, ty * b.ntypes + bd.type, sc1, qa, acc, flag);
  }
}

// One work item: bead `bd` against host units [t0, t1) (tiles, or with VOX 32-entry chunks
// of the bead's voxel list) and, when g1 > g0, the live guest atoms [g0, g1). hacc / gacc =
// {vdw, real} of the host and the guest atoms (valid on every lane, summed later); flag is
// per lane.
//
// Candidates are screened 32 at a time (host, then guests) and the ones inside the screening
// radius appended to the warp's ring buffer; whenever 32 are queued, or the phase has no
// candidates left, the warp evaluates the next batch at the phase's one dense site. Whole
// chunks of voxel-list entries that lie inside the cutoff for the whole voxel (half of a
// silica bead's list) go to the dense site directly. Batches come in list order, so the sums
// do not depend on how the candidates were produced.
//
// Early overlap rejection: with `dead` (the bead's trial's flag in shared memory, null
// when the trial must be evaluated in full) the warp stops as soon as the trial is known
// to overlap: after a dense batch that set an overlap flag (it then marks the trial), or
// when another warp has marked it. An overlapping trial takes no part in the Rosenbluth
// weight, and its flag is still raised by the warp that found the overlap, so the trial
// flags (and every used energy) are the same as without the early exit.
template <int PREC, bool VOX>
__device__ __forceinline__ void warp_item(const BoxDev& b, const Bead& bd, int t0, int t1, int g0, int g1,
                                          int component, int newmol, int excl_comp, int excl_mol, int* q,
                                          LaneAcc<PREC>& hacc, LaneAcc<PREC>& gacc, int& flag,
                                          volatile int* dead) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  unsigned head = 0, tail = 0;
  // the trial is dead: marked by another warp, or an overlap found by this one (which marks it).
  // One vote, so the warp stays converged.
  auto stop = [&]() {
    if (!dead || !__any_sync(kFull, flag != 0 || *dead > 0)) return false;
    if (lane == 0) *dead = 1;
    return true;
  };
  auto push = [&](bool in, int i) {
    const unsigned m = __ballot_sync(kFull, in);
    if (in) q[(tail + __popc(m & lt)) & (kQueue - 1)] = i;
    tail += __popc(m);
  };
  // the next queued batch: entry of this lane (stale past n), n taken
  auto pop = [&](int& n) {
    n = (int)min(tail - head, 32u);
    __syncwarp();
    const int j = q[(head + lane) & (kQueue - 1)];
    __syncwarp();
    head += (unsigned)n;
    return j;
  };
  if (stop()) return;
  const float bx = bd.h.x + bd.l.x, by = bd.h.y + bd.l.y, bz = bd.h.z + bd.l.z;
  if constexpr (VOX) {
    if (t1 > t0) {
      const float fx = b.invf[0] * bx + b.invf[3] * by + b.invf[6] * bz;
      const float fy = b.invf[1] * bx + b.invf[4] * by + b.invf[7] * bz;
      const float fz = b.invf[2] * bx + b.invf[5] * by + b.invf[8] * bz;
      const float mx = floorf(fx), my = floorf(fy), mz = floorf(fz);
      const int ix = min(b.vn[0] - 1, max(0, (int)((fx - mx) * (float)b.vn[0])));
      const int iy = min(b.vn[1] - 1, max(0, (int)((fy - my) * (float)b.vn[1])));
      const int iz = min(b.vn[2] - 1, max(0, (int)((fz - mz) * (float)b.vn[2])));
      const int4 vm = b.vmeta[(iz * b.vn[1] + iy) * b.vn[0] + ix];
      // the bead in the home cell, for the screen, by whole cell vectors. (Their hi parts alone, exact in
      // FP32, leave out up to 1.2e-4 A a cell and vector against a guard band of 2e-3 A: silica beads 40
      // cells away were 3.4e-3 A off and lost pairs at the cutoff. So they are 4e-4 A off there and
      // 1e-3 A at 200 cells; hi and low parts apart would give 5e-4 A there, for 9 FMAs and 9 loads an
      // item more.)
      const float3 wh = make_float3(bd.h.x - (mx * b.cellf[0] + my * b.cellf[3] + mz * b.cellf[6]),
                                    bd.h.y - (mx * b.cellf[1] + my * b.cellf[4] + mz * b.cellf[7]),
                                    bd.h.z - (mx * b.cellf[2] + my * b.cellf[5] + mz * b.cellf[8]));
      const bool hcheck = component < b.nhost || (excl_comp >= 0 && excl_comp < b.nhost);
      int ch = t0;
      const int cend = min(t1, (vm.z + 31) >> 5);
      const int sure_end = hcheck ? t0 : min(cend, vm.y >> 5);  // chunks of entries inside the cutoff
      const unsigned* list = b.vlist + vm.x + lane;
      auto load = [&](int c) { return c < cend && 32 * c + lane < vm.z ? __ldg(list + 32 * c) : 0u; };
      unsigned next = load(ch);  // one chunk ahead: the list load is off the gather's path
      for (;;) {
        unsigned w;
        int n;
        if (ch < sure_end) {
          w = next;
          n = 32;
          next = load(++ch);
        } else {
          while (tail - head < 32u && ch < cend) {  // screen at the stored image
            const int j = (ch << 5) + lane;
            const unsigned c = next;
            next = load(++ch);
            bool in = j < vm.z;
            if (in && (j >= vm.y || hcheck)) {
              const int i = (int)(c & 0xFFFFFu);
              if (j >= vm.y) {
                const float4 ah = b.hrec[2 * i];
                if (b.vox == 2) {
                  in = screen_hi<PREC>(b, ah, bd);
                } else {
                  const float4 sh = __ldg(b.vshift + (c >> 20));
                  const float x = (ah.x - wh.x) - sh.x, y = (ah.y - wh.y) - sh.y, z = (ah.z - wh.z) - sh.z;
                  in = x * x + y * y + z * z < b.screen2 || (PREC == GRX_FP64 && !(bd.unit & 2));
                }
              }
              if (in && hcheck) {  // a host component is moved or excluded: skip its molecule
                int tz = 0;
                while (tz + 1 < b.nhost && i >= b.comp_off[tz + 1]) ++tz;
                const int mol = b.hmeta[i].y;
                if ((tz == excl_comp && mol == excl_mol) || (tz == component && mol == newmol)) in = false;
              }
            }
            push(in, (int)c);
          }
          if (tail == head) break;
          w = (unsigned)pop(n);
        }
        if (lane < n) pair_dense<PREC>(b, true, (int)(w & 0xFFFFFu), bd, hacc, flag);
        if (stop()) return;
      }
    }
  } else {
    // Groups of 32 tiles from `base`, culled one per lane; `mask` holds the group's surviving tiles.
    int base = t0;
    unsigned mask = 0;
    float sx = 0.f, sy = 0.f, sz = 0.f;  // this lane's tile: image shift of the bead
    bool one_image = false;
    int4 trl = make_int4(0, 0, -1, 0);   // this lane's tile range, shuffled to the warp below
    // screen the next surviving tile; false when none is left
    auto host_step = [&]() -> bool {
      // Tiles are tested 32 at a time, one per lane; survivors are then screened one tile at
      // a time by the whole warp. When a tile lies inside one periodic image of the bead
      // (stored positions compact, the tile sphere clear of the rounding boundaries), the
      // image shift is applied once to the bead instead of per atom.
      while (mask == 0) {
        if (base >= t1) return false;
        const int tl = base + lane;
        base += 32;
        bool pass = tl < t1;
        sx = sy = sz = 0.f;
        one_image = false;
        trl = make_int4(0, 0, -1, 0);
        if (pass) trl = b.tile_r[tl];
        if (pass && b.cull) {
          const float4 tc = b.tile_c[2 * tl];
          float dx = tc.x - bx, dy = tc.y - by, dz = tc.z - bz;
          // FP64: the hi parts of bead and tile hold their coordinates to 2^-13 A (below 2 kNearCoord)
          const bool exact = (bd.unit & 2) && fmaxf(fmaxf(fabsf(dx), fabsf(dy)), fabsf(dz)) + tc.w < kNearCoord;
          bool near4;
          const float lim = b.cull_r + tc.w;
          const float m = tc.w + 1e-2f;
          if (b.cubic) {
            // Bounding box of the tile at the centre's rounded image. Per axis the distance to
            // the box bounds every atom's rounded-image distance from below: an atom whose
            // rounding differs from the centre's lies at least half a cell minus the half
            // extent away on that axis.
            const float4 th = b.tile_c[2 * tl + 1];
            const float nx = rnd(dx * b.invf[0]), ny = rnd(dy * b.invf[4]), nz = rnd(dz * b.invf[8]);
            dx = __fmaf_rn(-nx, b.cellf[0], dx);
            dy = __fmaf_rn(-ny, b.cellf[4], dy);
            dz = __fmaf_rn(-nz, b.cellf[8], dz);
            const float qx = fmaxf(fabsf(dx) - th.x, 0.f), qy = fmaxf(fabsf(dy) - th.y, 0.f),
                        qz = fmaxf(fabsf(dz) - th.z, 0.f);
            pass = qx * qx + qy * qy + qz * qz <= b.cull_r * b.cull_r;
            one_image = trl.w != 0 && fabsf(dx) + th.x + 1e-2f < 0.5f * b.cellf[0] &&
                        fabsf(dy) + th.y + 1e-2f < 0.5f * b.cellf[4] && fabsf(dz) + th.z + 1e-2f < 0.5f * b.cellf[8];
            // the whole edges: n times their low parts alone would pass the screen's guard band
            sx = nx * b.cellf[0]; sy = ny * b.cellf[4]; sz = nz * b.cellf[8];
            near4 = fmaxf(fmaxf(fabsf(nx), fabsf(ny)), fabsf(nz)) <= 4.0f;
          } else {
            const float fx = b.invf[0] * dx + b.invf[3] * dy + b.invf[6] * dz;
            const float fy = b.invf[1] * dx + b.invf[4] * dy + b.invf[7] * dz;
            const float fz = b.invf[2] * dx + b.invf[5] * dy + b.invf[8] * dz;
            const float nx = rnd(fx), ny = rnd(fy), nz = rnd(fz);
            sx = nx * b.cellf[0] + ny * b.cellf[3] + nz * b.cellf[6];
            sy = nx * b.cellf[1] + ny * b.cellf[4] + nz * b.cellf[7];
            sz = nx * b.cellf[2] + ny * b.cellf[5] + nz * b.cellf[8];
            dx -= sx; dy -= sy; dz -= sz;
            const float d2 = dx * dx + dy * dy + dz * dz;
            const float rx = fabsf(fx - nx), ry = fabsf(fy - ny), rz = fabsf(fz - nz);
            if (d2 <= b.half_wmin2) {
              pass = d2 <= lim * lim;
            } else {
              const float lb = fmaxf(fmaxf(rx * b.wperp[0], ry * b.wperp[1]), rz * b.wperp[2]);
              pass = lb - 1e-3f <= lim;
            }
            one_image = trl.w != 0 && rx + m / b.wperp[0] < 0.5f - 1e-4f &&
                        ry + m / b.wperp[1] < 0.5f - 1e-4f && rz + m / b.wperp[2] < 0.5f - 1e-4f;
            near4 = fmaxf(fmaxf(fabsf(nx), fabsf(ny)), fabsf(nz)) <= 4.0f;
          }
          if (PREC == GRX_FP64) one_image = one_image && near4 && exact;
        }
        mask = __ballot_sync(kFull, pass);
      }
      const int src = __ffs(mask) - 1;
      mask &= mask - 1;
      const int i = __shfl_sync(kFull, trl.x, src) + lane, tz = __shfl_sync(kFull, trl.z, src);
      const bool oi = __shfl_sync(kFull, one_image, src);
      const float tsx = __shfl_sync(kFull, sx, src), tsy = __shfl_sync(kFull, sy, src),
                  tsz = __shfl_sync(kFull, sz, src);
      bool in = false;
      if (i < __shfl_sync(kFull, trl.y, src)) {
        bool skip = false;
        if (tz == component || tz == excl_comp) {
          const int mol = b.hmeta[i].y;
          skip = (tz == excl_comp && mol == excl_mol) || (tz == component && mol == newmol);
        }
        if (!skip) {
          if (oi) {
            const float4 ah = b.hrec[2 * i];
            const float x = ah.x - (bd.h.x + tsx);
            const float y = ah.y - (bd.h.y + tsy);
            const float z = ah.z - (bd.h.z + tsz);
            in = x * x + y * y + z * z < b.screen2;
          } else {
            in = pair_screen<PREC, true>(b, i, bd);
          }
        }
      }
      push(in, i);
      return true;
    };
    bool more = t1 > t0;
    for (;;) {
      while (more && tail - head < 32u) more = host_step();
      if (tail == head) break;
      int n;
      const int j = pop(n);
      if (lane < n) pair_dense<PREC>(b, true, j, bd, hacc, flag);
      if (stop()) return;
    }
  }
  if (g1 <= g0) return;
  // guest atoms [g0, g1) of the concatenated adsorbate components: component gc, its atoms
  // [gi, ghi) still to screen (indices within the component), gbase = the first concatenated
  // guest index after gc
  int gc = b.nhost, gbase = 0, gi = 0, ghi = 0;
  for (;;) {
    while (tail - head < 32u) {
      while (gi >= ghi && gc < b.ncomp && gbase < g1) {  // next component overlapping [g0, g1)
        const int n = b.comp_size[gc];
        gi = max(g0 - gbase, 0);
        ghi = min(g1 - gbase, n);
        gbase += n;
        ++gc;
      }
      if (gi >= ghi) break;
      const int c = gc - 1;
      const int i = b.comp_off[c] + gi + lane;
      bool in = false;
      if (gi + lane < ghi) {
        bool skip = false;
        if (c == component || c == excl_comp) {
          const int mol = b.meta[i].y;
          skip = (c == excl_comp && mol == excl_mol) || (c == component && mol == newmol);
        }
        if (!skip) in = pair_screen<PREC, false>(b, i, bd);
      }
      gi += 32;
      push(in, i);
    }
    if (tail == head) return;
    int n;
    const int j = pop(n);
    if (lane < n) pair_dense<PREC>(b, false, j, bd, gacc, flag);
    if (stop()) return;
  }
}

// Fixed-order warp sums (lane 0 receives the total). The double-float form keeps the
// reduction on the FP32 pipe; one conversion to FP64 happens on lane 0 only.
__device__ __forceinline__ double warp_sum(double x) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(kFull, x, o);
  return x;
}

// Out of line: called once per Ewald delta, so one copy serves them all.
static __device__ __noinline__ float2 warp_sum_df_out(float hi, float lo) {
  df x = {hi, lo};
  for (int o = 16; o > 0; o >>= 1) {
    const df y = {__shfl_down_sync(kFull, x.hi, o), __shfl_down_sync(kFull, x.lo, o)};
    x = df_add(x, y);
  }
  return make_float2(x.hi, x.lo);
}

__device__ __forceinline__ df warp_sum_df(df x) {
  const float2 r = warp_sum_df_out(x.hi, x.lo);
  return df{r.x, r.y};
}

__device__ __forceinline__ df lane_add(df a, df b) { return df_add(a, b); }
__device__ __forceinline__ double lane_add(double a, double b) { return a + b; }
__device__ __forceinline__ df lane_xor(df x, int o) {
  return {__shfl_xor_sync(kFull, x.hi, o), __shfl_xor_sync(kFull, x.lo, o)};
}
__device__ __forceinline__ double lane_xor(double x, int o) { return __shfl_xor_sync(kFull, x, o); }

// One exchange of a transposed sum: lanes with bit `o` clear keep a, the others b, and each
// receives its partner's share of what it keeps.
template <class T>
__device__ __forceinline__ T lane_fold(T a, T b, int o) {
  const bool up = (threadIdx.x & o) != 0;
  const T keep = up ? b : a, send = up ? a : b;
  return lane_add(keep, lane_xor(send, o));
}

// Warp sums of a work item's four accumulators: host vdw and real on lanes 0 and 16, guest vdw
// and real on lanes 8 and 24. Folding two sums into one register per exchange takes 7 additions
// (5 without guests) where four separate trees take 20. Out of line: one copy per form.
template <class T>
static __device__ __noinline__ T item_sums(T hv, T hr, T gv, T gr, bool guests) {
  T x = lane_fold(hv, hr, 16);
  if (guests) x = lane_fold(x, lane_fold(gv, gr, 16), 8);
  else x = lane_add(x, lane_xor(x, 8));
  for (int o = 4; o > 0; o >>= 1) x = lane_add(x, lane_xor(x, o));
  return x;
}

// The sums of one work item into its slot {hg_vdw, hg_real, gg_vdw, gg_real}. The mixed and FP64
// forms accumulate sum q_atom * g(r); the bead factor prefactor * q_bead is applied here, once.
template <int PREC>
__device__ __forceinline__ void warp_store(const LaneAcc<PREC>& h, const LaneAcc<PREC>& g, double* out4, df pq,
                                           double pq64, bool with_guests) {
  const int lane = threadIdx.x & 31;
  const bool real = lane >= 16, guest = (lane & 8) != 0;
  const auto x = item_sums(h.v, h.r, g.v, g.r, with_guests);
  if ((lane & 7) != 0) return;
  const int k = (real ? 1 : 0) + (guest ? 2 : 0);
  if constexpr (PREC == GRX_MIXED) {  // stored as float pairs in the 8-byte slots (item_get converts)
    const df v = real ? df_mul(x, pq) : x;
    reinterpret_cast<float2*>(out4)[k] = guest && !with_guests ? make_float2(0.f, 0.f) : make_float2(v.hi, v.lo);
  } else {
    const double f = real && (PREC == GRX_FP64 || PREC == kMixed64) ? pq64 : 1.0;
    out4[k] = guest && !with_guests ? 0.0 : x * f;
  }
}

// ---------------------------------------------------------------- Rosenbluth step
// Selection and weight of one CBMC step over nt <= 64 trials by one warp (SelectTrialPosition,
// mc_widom.h:14-39, and the sums of CBMC_FirstBead_Finish, :330-376): the trial without overlap
// that the uniform u picks from the shifted weights (with `retrace` the first one), the number of
// trials without overlap and the unshifted weight sum. Every trial is
// two lanes' worth at most, the cumulative sum a warp scan and the unshifted sum the shifted
// one times exp(max), so a step is one exp and five additions deep; a serial walk over the trials
// took two exps and three additions per trial, each a full FP64 latency on one lane.
struct StepChoice {
  int sel, nok;
  double w;
};

// The exponent of trial t.
__device__ __forceinline__ double trial_exponent(const double* te, int t, double beta, int bias) {
  double tot = te[4 * t] + te[4 * t + 2];
  if (bias) tot += te[4 * t + 1] + te[4 * t + 3];
  return __dmul_rn(-beta, tot);
}

static __device__ __noinline__ StepChoice choose_trial(const double* te, const int* tflag, int nt, double beta, int bias,
                                                       double u, bool retrace) {
  const int lane = threadIdx.x & 31;
  double lw[2], e[2] = {0.0, 0.0};
  bool ok[2];
  // order-preserving words: an integer maximum instead of FP64 comparisons
  long long top = LLONG_MIN;
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int t = lane + 32 * r;
    ok[r] = t < nt && !tflag[t];
    lw[r] = 0.0;
    if (ok[r]) {
      lw[r] = trial_exponent(te, t, beta, bias);
      const long long w = __double_as_longlong(lw[r]);
      top = max(top, w ^ ((w >> 63) & 0x7fffffffffffffffll));
    }
  }
  const unsigned ok0 = __ballot_sync(kFull, ok[0]), ok1 = __ballot_sync(kFull, ok[1]);
  StepChoice c;
  c.nok = __popc(ok0) + __popc(ok1);
  c.sel = -1;
  c.w = 0.0;
  if (c.nok == 0) return c;
  for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(kFull, top, o));
  const double mx = __longlong_as_double(top ^ ((top >> 63) & 0x7fffffffffffffffll));
  double scale;
  if (nt < 32) {  // the last lane is free for exp(max)
    const double x = exp_move(lane == 31 ? mx : (ok[0] ? __dsub_rn(lw[0], mx) : 0.0));
    scale = __shfl_sync(kFull, x, 31);
    e[0] = ok[0] ? x : 0.0;
  } else {
    scale = exp_move(mx);
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
      const double x = exp_move(ok[r] ? __dsub_rn(lw[r], mx) : 0.0);
      e[r] = ok[r] ? x : 0.0;
    }
  }
  double c0 = e[0], c1 = 0.0;
  for (int o = 1; o < 32; o <<= 1) {
    const double v = __shfl_up_sync(kFull, c0, o);
    if (lane >= o) c0 += v;
  }
  double sum = __shfl_sync(kFull, c0, 31);
  if (nt > 32) {
    c1 = e[1];
    for (int o = 1; o < 32; o <<= 1) {
      const double v = __shfl_up_sync(kFull, c1, o);
      if (lane >= o) c1 += v;
    }
    c1 += sum;
    sum = __shfl_sync(kFull, c1, 31);
  }
  const double wsel = u * sum;
  const unsigned m0 = __ballot_sync(kFull, ok[0] && (retrace || !(c0 < wsel))),
                 m1 = __ballot_sync(kFull, ok[1] && (retrace || !(c1 < wsel)));
  if (m0) c.sel = __ffs(m0) - 1;
  else if (m1) c.sel = 31 + __ffs(m1);
  else c.sel = ok1 ? 63 - __clz(ok1) : 31 - __clz(ok0);  // rounding left the sum below u * sum: the last one
  c.w = mx > -INFINITY || mx != mx ? scale * sum : 0.0;  // every energy +inf: no weight
  return c;
}

// The weights of a step as they are, by one warp: {their sum in the order of the trials, what it leaves
// over the weight of trial sel}. Where a trial outweighs the rest by 1e15 that remainder is roundings of the
// sum, and a reinsertion's retrace weight (StoredR) is made of it: it has to come from this order, as
// the oracle's and the host layer's do, and not from the shifted sum, which rounds elsewhere (5 of 60
// chains of 40 reinsertions beside charged atoms took other decisions). A chain of nt FP64 additions:
// 2.6 % of a pass of 64 CH4/Xe boxes. Also the sum beyond the range of exp, where exp of the maximum
// times the shifted sum is no number.
static __device__ __noinline__ double2 plain_weights(const double* te, const int* tflag, int nt, double beta, int bias,
                                                     int sel) {
  const int lane = threadIdx.x & 31;
  double x[2] = {0.0, 0.0};
#pragma unroll 1
  for (int r = 0; r < 2; ++r) {
    const int t = lane + 32 * r;
    if (t < nt && !tflag[t]) x[r] = exp_move(trial_exponent(te, t, beta, bias));
  }
  double w = 0.0, ws = 0.0;
#pragma unroll 1
  for (int t = 0; t < nt; ++t) {
    const double v = __shfl_sync(kFull, t < 32 ? x[0] : x[1], t & 31);
    w += v;
    if (t == sel) ws = v;
  }
  return make_double2(w, w - ws);
}

// Live adsorbate atoms of the box, and the 32-atom work units a bead pass covers
// (host tiles plus guest atoms in groups of 32).
__device__ __forceinline__ int guest_atoms(const BoxDev& b) {
  int g = 0;
  for (int c = b.nhost; c < b.ncomp; ++c) g += b.comp_size[c];
  return g;
}
__device__ __forceinline__ int host_units(const BoxDev& b) { return b.vox ? b.vchunks : b.ntiles; }
__device__ __forceinline__ int work_tiles(const BoxDev& b) { return host_units(b) + (guest_atoms(b) + 31) / 32; }

// Work split of one bead pass. The flattened space of nb beads x nu work units (host
// tiles, then guest atoms in groups of 32) is cut into `items` contiguous ranges of equal
// size, so every warp gets the same share whatever nb is. An item that crosses a bead
// boundary stores one partial per bead it touches, in slot item + bead; these slots are
// distinct (a later item cannot reach an earlier bead), so a pass uses at most
// items + nb - 1 slots.
struct PassSplit {
  unsigned nu, items, q, r;  // units per bead, items, and T = items * q + r with T = nb * nu
  __device__ __forceinline__ void range(unsigned item, unsigned& lo, unsigned& hi) const {
    lo = item * q + min(item, r);
    hi = lo + q + (item < r ? 1u : 0u);
  }
  __device__ __forceinline__ unsigned item_of(unsigned p) const {  // the item holding unit p
    const unsigned big = r * (q + 1);
    return p < big ? p / (q + 1) : r + (p - big) / q;
  }
};

// Items of a pass: mult per warp, never more than the units of the pass (at least 1).
__device__ __forceinline__ PassSplit pass_split(const BoxDev& b, int nb, int nwarps, int mult) {
  PassSplit s;
  s.nu = (unsigned)work_tiles(b);
  const unsigned T = (unsigned)nb * s.nu;
  s.items = max(1u, min((unsigned)(mult * nwarps), T));
  s.q = T / s.items;
  s.r = T - s.q * s.items;
  return s;
}

constexpr int kMaxItems = 320;

// One pass of `nb` beads (shared memory) over every atom by a whole block. Items
// [item0, item1) (all of them when item1 < 0) are taken dynamically by warps; the partial
// of bead `bead` within item `item` lands in ipart[(item + bead)*4 + q] and
// iflag[item + bead]. Caller syncs before reading them.
template <int PREC, bool VOX>
__device__ __noinline__ void block_bead_pass_impl(const BoxDev& b, const Bead* beads, int nb, int component,
                                                     int newmol, int excl_comp, int excl_mol, int* qbuf,
                                                     double* ipart, int* iflag, int* counter, PassSplit sp,
                                                     int item0, int item1, int chain, int* dead) {
  if (item1 < 0) item1 = (int)sp.items;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int* q = qbuf + warp * kQueue;
  const int nt = VOX ? b.vchunks : b.ntiles;
  const int ng = guest_atoms(b);
  if (sp.nu == 0) {  // nothing to interact with: zero partials, one item per bead slot
    for (int k = threadIdx.x; k < nb * 4; k += blockDim.x) ipart[k] = 0.0;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) iflag[k] = 0;
    return;
  }
  for (;;) {
    int item = 0;
    if (lane == 0) item = item0 + atomicAdd(counter, 1);
    item = __shfl_sync(kFull, item, 0);
    if (item >= item1) break;
    unsigned lo, hi;
    sp.range((unsigned)item, lo, hi);
    while (lo < hi) {
      const int bead = (int)(lo / sp.nu);
      const int u0 = (int)(lo - (unsigned)bead * sp.nu);
      const int u1 = (int)min(sp.nu, (unsigned)u0 + (hi - lo));
      // only the ranges reaching past the host tiles touch guest atoms
      const int t0 = min(u0, nt), t1 = min(u1, nt);
      const int g0 = min(32 * max(u0 - nt, 0), ng), g1 = min(32 * max(u1 - nt, 0), ng);
      // the bead is read from shared memory where it is used (fewer live registers around
      // the inlined dense evaluations: no spills in either pass)
      const Bead& bd = beads[bead];
      LaneAcc<PREC> hacc, gacc;
      int flag = 0;
      // trials of `chain` beads; dead[t] < 0: evaluated in full, else the early-exit flag
      volatile int* dt = nullptr;
      if (dead && dead[bead / chain] >= 0) dt = dead + bead / chain;
      warp_item<PREC, VOX>(b, bd, t0, t1, g0, g1, component, newmol, excl_comp, excl_mol, q, hacc, gacc, flag, dt);
      const unsigned fm = __ballot_sync(kFull, flag != 0);
      warp_store<PREC>(hacc, gacc, ipart + (item + bead) * 4, df{bd.pq.x, bd.pq.y},
                       b.prefactor * bd.q, g1 > g0);
      if (lane == 0) iflag[item + bead] = fm ? 1 : 0;
      lo += (unsigned)(u1 - u0);
    }
  }
}

// The pass through voxel lists or through tiles: two instantiations, so each keeps its own
// register allocation (the box decides, uniformly for the whole block).
// dead: per trial of `chain` beads, 0 for early overlap rejection, -1 to evaluate the trial
// in full (set by the caller before the pass; null: every trial in full).
template <int PREC>
__device__ __forceinline__ void block_bead_pass(const BoxDev& b, const Bead* beads, int nb, int component, int newmol,
                                                int excl_comp, int excl_mol, int* qbuf, double* ipart, int* iflag,
                                                int* counter, PassSplit sp, int item0 = 0, int item1 = -1,
                                                int chain = 1, int* dead = nullptr) {
  if (b.vox)
    block_bead_pass_impl<PREC, true>(b, beads, nb, component, newmol, excl_comp, excl_mol, qbuf, ipart, iflag,
                                     counter, sp, item0, item1, chain, dead);
  else
    block_bead_pass_impl<PREC, false>(b, beads, nb, component, newmol, excl_comp, excl_mol, qbuf, ipart, iflag,
                                      counter, sp, item0, item1, chain, dead);
}

// ---------------------------------------------------------------- thread-block clusters
// A cluster of CTAs may share one chain: each CTA evaluates a contiguous share of a pass's
// items and writes its partial slots into every peer's shared memory (PTX mapa + generic
// stores), so all CTAs reduce identical slots in identical order. barrier.cluster with
// release / acquire semantics orders those stores and the CTAs' global writes.
__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
template <class T>
__device__ __forceinline__ T* cluster_map(T* p, unsigned rank) {  // the same shared variable in CTA `rank`
  uint64_t out;
  asm volatile("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
  return reinterpret_cast<T*>(out);
}

// Items of a pass for CTA `rank` of a CL-CTA cluster: [i0, i1), contiguous.
__device__ __forceinline__ void cluster_items(const PassSplit& sp, int cl, unsigned rank, int& i0, int& i1) {
  const unsigned per = (sp.items + (unsigned)cl - 1u) / (unsigned)cl;
  i0 = (int)min(sp.items, rank * per);
  i1 = (int)min(sp.items, (unsigned)i0 + per);
}

// Active k vectors of CTA `rank` of a CL-CTA cluster: [k0, k1), contiguous.
__device__ __forceinline__ void cluster_k_range(int nact, int cl, unsigned rank, int& k0, int& k1) {
  const int per = (nact + cl - 1) / cl;
  k0 = min(nact, (int)rank * per);
  k1 = min(nact, k0 + per);
}

// Item partials: FP64 in the FP64 / FP32 forms, a float pair in the mixed form.
template <int PREC>
__device__ __forceinline__ double item_get(const double* ipart, int idx) {
  if constexpr (PREC == GRX_MIXED) {
    const float2 v = reinterpret_cast<const float2*>(ipart)[idx];
    return (double)v.x + (double)v.y;
  } else {
    return ipart[idx];
  }
}

// Slots of bead `bead`: [first, last] (slot = item + bead), in unit order.
__device__ __forceinline__ void bead_slots(const PassSplit& sp, int bead, int& first, int& last) {
  if (sp.nu == 0) { first = last = bead; return; }
  const unsigned p0 = (unsigned)bead * sp.nu;
  first = (int)sp.item_of(p0) + bead;
  last = (int)sp.item_of(p0 + sp.nu - 1) + bead;
}

// Per-trial sums of one pass: trial t = beads [t*chain, (t+1)*chain), partials in order.
template <int PREC>
__device__ __forceinline__ void reduce_items(const double* ipart, const int* iflag, int ntr, int chain,
                                             const PassSplit& sp, double* te, int* tflag) {
  for (int w = threadIdx.x; w < ntr * 4; w += blockDim.x) {
    const int t = w >> 2, k = w & 3;
    int f = 0;
    if constexpr (PREC == GRX_MIXED) {
      df s = {0.f, 0.f};
#pragma unroll 1
      for (int a = 0; a < chain; ++a) {
        int s0, s1;
        bead_slots(sp, t * chain + a, s0, s1);
#pragma unroll 1
        for (int c = s0; c <= s1; ++c) {
          const float2 v = reinterpret_cast<const float2*>(ipart)[c * 4 + k];
          s = df_add(s, df{v.x, v.y});
          f |= iflag[c];
        }
      }
      te[4 * t + k] = df_to(s);
    } else {
      double s = 0.0;
#pragma unroll 1
      for (int a = 0; a < chain; ++a) {
        int s0, s1;
        bead_slots(sp, t * chain + a, s0, s1);
#pragma unroll 1
        for (int c = s0; c <= s1; ++c) {
          s += ipart[c * 4 + k];
          f |= iflag[c];
        }
      }
      te[4 * t + k] = s;
    }
    if (k == 0) tflag[t] = f;
  }
}

// ---------------------------------------------------------------- single passes
// One trial (`chain` beads in shared memory) against every atom by a cluster of kTrialCtas CTAs
// of kTrialWarps warps. A host-driven call has 1 to 64 trials and its time is latency, so the
// pass is cut into 32 items spread over eight SMs (one block per bead left 142 of 152 SMs idle
// on a ten-trial step); the split depends on the chain length alone, so a trial's sums are the
// same whatever else the call holds. The CTAs write their partial slots into CTA 0, whose warp q
// adds quantity q over the slots.
constexpr int kTrialCtas = 8;
constexpr int kTrialWarps = 4;
constexpr int kTrialItems = kTrialCtas * kTrialWarps;
constexpr int kTrialSlots = kTrialItems + GRX_MAX_TRIAL_BEADS;

// One block copies a descriptor (a kernel parameter) into shared memory, where the out-of-line
// pass reads it through a pointer. The caller synchronises.
template <class T>
__device__ __forceinline__ void copy_words(T* dst, const T* src) {
  static_assert(sizeof(T) % 8 == 0, "copied in 8-byte words");
  for (int k = threadIdx.x; k < (int)(sizeof(T) / 8); k += blockDim.x)
    reinterpret_cast<unsigned long long*>(dst)[k] = reinterpret_cast<const unsigned long long*>(src)[k];
}

struct TrialWork {
  double ipart[kTrialSlots * 4];
  int iflag[kTrialSlots];
  int qbuf[kTrialWarps * kQueue];
  int counter;
};

// Called by every thread of the cluster after `beads` is filled and before any barrier that
// publishes it. In CTA 0, lane 0 of warp q < 4 returns quantity q (hg_vdw, hg_real, gg_vdw,
// gg_real) in `sum` and the overlap flag in `flag`.
template <int PREC>
__device__ __forceinline__ void trial_cluster_pass(const BoxDev& b, const Bead* beads, TrialWork& W, int chain,
                                                   int component, int newmol, int excl_comp, int excl_mol, double& sum,
                                                   int& flag) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned rank = cluster_rank();
  const PassSplit sp = pass_split(b, chain, kTrialItems, 1);
  const int nslot = (int)sp.items + chain;
  if (rank == 0) {  // a slot between two beads may stay unwritten
    for (int k = tid; k < nslot * 4; k += blockDim.x) W.ipart[k] = 0.0;
    for (int k = tid; k < nslot; k += blockDim.x) W.iflag[k] = 0;
  }
  if (tid == 0) W.counter = 0;
  __syncthreads();
  cluster_sync_all();
  int i0, i1;
  cluster_items(sp, kTrialCtas, rank, i0, i1);
  if (i0 < i1 && sp.nu > 0) {
    block_bead_pass<PREC>(b, beads, chain, component, newmol, excl_comp, excl_mol, W.qbuf, W.ipart, W.iflag, &W.counter,
                          sp, i0, i1);
    __syncthreads();
    if (rank != 0) {
      unsigned lo, hi;
      double* dst = cluster_map(W.ipart, 0);
      int* df = cluster_map(W.iflag, 0);
      for (int item = i0; item < i1; ++item) {  // the slots this CTA wrote, gaps left out
        sp.range((unsigned)item, lo, hi);
        const int b0 = (int)(lo / sp.nu), b1 = (int)((hi - 1u) / sp.nu);
        for (int k = tid; k < 5 * (b1 - b0 + 1); k += blockDim.x) {
          const int slot = item + b0 + k / 5, f = k % 5;
          if (f < 4) dst[slot * 4 + f] = W.ipart[slot * 4 + f];
          else df[slot] = W.iflag[slot];
        }
      }
    }
  }
  __syncthreads();
  cluster_sync_all();
  sum = 0.0;
  flag = 0;
  if (rank == 0 && warp < 4) {
    for (int s = lane; s < nslot; s += 32) {
      sum += item_get<PREC>(W.ipart, s * 4 + warp);
      flag |= W.iflag[s];
    }
    sum = warp_sum(sum);
    flag = __any_sync(kFull, flag != 0) ? 1 : 0;
  }
}

// Trial energies behind grx_trial_energies, grx_trial_energies_noalloc and
// grx_single_body_energy (they run this one kernel, so they give the same sums): one cluster
// per trial; trial t leaves out the atoms of (component, mol[t < split ? 0 : 1]).
struct TrialArgs {
  const Bead* beads;
  int chain;
  int component;
  int mol[2];
  int split;
  int excl_comp;
  int excl_mol;
  double* out;          // 4 per trial
  unsigned char* over;  // 1 per trial
};

template <int PREC>
__global__ void __cluster_dims__(kTrialCtas, 1, 1) __launch_bounds__(kTrialWarps * 32)
    trial_kernel(const __grid_constant__ BoxDev box, const __grid_constant__ TrialArgs a) {
  extern __shared__ double2 trial_smem[];
  Bead* beads = reinterpret_cast<Bead*>(trial_smem);
  __shared__ TrialWork W;
  __shared__ BoxDev b;
  copy_words(&b, &box);
  const int t = (int)blockIdx.x / kTrialCtas;
  const int nw = a.chain * (int)(sizeof(Bead) / 8);
  const double* src = reinterpret_cast<const double*>(a.beads + (size_t)t * a.chain);
  for (int k = threadIdx.x; k < nw; k += blockDim.x) reinterpret_cast<double*>(beads)[k] = src[k];
  __syncthreads();
  double sum;
  int flag;
  trial_cluster_pass<PREC>(b, beads, W, a.chain, a.component, a.mol[t < a.split ? 0 : 1], a.excl_comp, a.excl_mol, sum,
                           flag);
  const int warp = threadIdx.x >> 5;
  if (cluster_rank() == 0 && warp < 4 && (threadIdx.x & 31) == 0) {
    a.out[4 * t + warp] = sum;
    if (warp == 0) a.over[t] = (unsigned char)flag;
  }
}

static_assert(sizeof(Bead) % 8 == 0, "beads are staged in 8-byte words");

// Enqueues the pass over ntrials trials (ntrials >= 1).
template <int PREC>
static inline void launch_trials(const BoxDev& b, const TrialArgs& a, int ntrials, cudaStream_t s) {
  trial_kernel<PREC><<<ntrials * kTrialCtas, kTrialWarps * 32, a.chain * sizeof(Bead), s>>>(b, a);
}

// Rotate_Quaternions (mc_utilities.h:423-457) in FP64: df_quaternion_half and df_rotated with the
// uniforms u and v (half 0) or u and w (half 1).
__device__ __forceinline__ double2 quaternion_half(double u, double angle, int half) {
  double s, c;
  sincos(2 * 3.14159265358979323846 * angle, &s, &c);
  const double m = sqrt(half ? u : 1 - u);
  return make_double2(m * s, m * c);
}

__device__ __forceinline__ double rotated(double2 qa, double2 qb, int d, double x, double y, double z) {
  auto pick3 = [d](double a, double b, double c) { return d == 0 ? a : (d == 1 ? b : c); };
  const double ei = pick3(qa.y, qb.x, qb.y), ej = pick3(qb.x, qb.y, qa.y), ek = pick3(qb.y, qa.y, qb.x);
  const double ri = 1.0 - 2.0 * (ej * ej + ek * ek), rj = 2.0 * (ei * ej - qa.x * ek), rk = 2.0 * (ei * ek + qa.x * ej);
  return x * pick3(ri, rk, rj) + y * pick3(rj, ri, rk) + z * pick3(rk, rj, ri);
}

// make_bead by three lanes, 3 k + d of a warp the coordinate c of bead k along d (the whole warp
// calls; live: the lane has a coordinate). FP64 issues once for the three coordinates.
__device__ __forceinline__ void put_bead(const BoxDev& b, Bead& bd, int lane, int d, bool live, double c, double q,
                                         double scale, int type) {
  float h = 0.0f, l;
  if (live) {
    split_coord(c, h, l);
    (&bd.x)[d] = c;
    (&bd.h.x)[d] = h;
    (&bd.l.x)[d] = l;
    if (d == 0) {
      const df pq = df_from(b.prefactor * q);
      bd.q = q;
      bd.scale = scale;
      bd.type = type;
      bd.pq = make_float2(pq.hi, pq.lo);
    }
  }
  const unsigned near = __ballot_sync(kFull, fabsf(h) < kNearCoord);
  if (live && d == 0) bd.unit = (scale == 1.0 ? 1 : 0) | (((near >> lane) & 7u) == 7u ? 2 : 0);
}

// First-bead trials of a growth, the whole block: cell diagonal x Philox uniforms
// (mc_widom.h:133-139), a lane per coordinate. retrace: trial 0 is the bead (ox, oy, oz).
template <class Draw>
__device__ __forceinline__ void first_beads(const BoxDev& b, Bead* beads, Draw draw, int nt, double q, double scale,
                                            int type, bool retrace, double ox, double oy, double oz) {
  const int lane = threadIdx.x & 31, k = lane / 3, d = lane - 3 * k;
  for (int base = 10 * (int)(threadIdx.x >> 5); base < nt; base += 10 * (int)(blockDim.x >> 5)) {
    const int t = base + k;
    const bool live = k < 10 && t < nt;
    double c = 0.0;
    if (live) {
      if (retrace && t == 0) {
        c = d == 0 ? ox : (d == 1 ? oy : oz);
      } else {
        uint32_t r[4];
        draw(t, r);
        c = b.cell[4 * d] * u01(d == 0 ? r[0] : (d == 1 ? r[1] : r[2]));
      }
    }
    put_bead(b, beads[live ? t : 0], lane, d, live, c, q, scale, type);
  }
}

// Beads of trial orientations, the whole block: no lane pairs form the quaternions (one sine and
// cosine each, in `quat`, 2 per orientation), then a warp takes ten beads, a lane one coordinate of
// one. The mixed and FP32 forms rotate in double-float on the FP32 pipe, the FP64 form in FP64 (the
// oracle's arithmetic). The stage runs once per move on few lanes, so the length of a lane's chain
// is its time: with a bead's three coordinates and both sines on one lane it took 17 k of the 205 k
// cycles of a CO2 move (456 mixed chains 5.70 ms a pass, 5.47 ms so). retrace: orientation 0 is the
// existing chain ox / oy / oz.
// draw(o, r): the Philox words of orientation o.
template <int PREC, class Draw>
__device__ __forceinline__ void orientation_beads(const BoxDev& b, Bead* beads, float4* quat, Draw draw, int no,
                                                  int chain, int off, double scale_coul, double scale, double fx,
                                                  double fy, double fz, bool retrace, const double* ox,
                                                  const double* oy, const double* oz) {
  for (int t = threadIdx.x; t < 2 * no; t += blockDim.x) {
    uint32_t r[4];
    draw(t >> 1, r);
    const uint32_t angle = t & 1 ? r[2] : r[1];
    if constexpr (PREC == GRX_FP64) reinterpret_cast<double2*>(quat)[t] = quaternion_half(u01(r[0]), u01(angle), t & 1);
    else quat[t] = df_quaternion_half(r[0], angle, t & 1);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, k = lane / 3, d = lane - 3 * k, nb = no * chain;
  for (int base = 10 * (int)(threadIdx.x >> 5); base < nb; base += 10 * (int)(blockDim.x >> 5)) {
    const int t = base + k;
    const bool live = k < 10 && t < nb;
    double c = 0.0, q = 0.0;
    int type = 0;
    if (live) {
      const int o = t / chain, at = t - o * chain;
      if (retrace && o == 0) {
        c = d == 0 ? ox[at] : (d == 1 ? oy[at] : oz[at]);
      } else {
        const double4 t0 = b.pos64[off], pa = b.pos64[off + 1 + at];
        const double x = pa.x - t0.x, y = pa.y - t0.y, z = pa.z - t0.z;
        if constexpr (PREC == GRX_FP64) {
          const double2* p = reinterpret_cast<const double2*>(quat) + 2 * o;
          c = rotated(p[0], p[1], d, x, y, z);
        } else {
          c = df_to(df_rotated(quat[2 * o], quat[2 * o + 1], d, df_from(x), df_from(y), df_from(z)));
        }
        c += d == 0 ? fx : (d == 1 ? fy : fz);
      }
      q = b.charge[off + 1 + at] * scale_coul;
      type = b.meta[off + 1 + at].x;
    }
    put_bead(b, beads[live ? t : 0], lane, d, live, c, q, scale, type);
  }
}

}  // namespace grx
