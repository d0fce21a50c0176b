// grx_ewcol.cuh -- Fourier delta of a few moved atoms by columns of the active k.
//
// A column (kx, ky, |kz|) carries the k with +|kz| and -|kz|. With P = q X(kx) Y(ky) of an atom
// and Z = Z(|kz|), the four real sums over atoms
//   A = sum Re P Re Z,  B = sum Im P Im Z,  C = sum Re P Im Z,  D = sum Im P Re Z
// give dS(+|kz|) = (A - B) + i (C + D) and dS(-|kz|) = (A + B) + i (D - C): half the products of
// the per-k form, and P once for two k. The charge sits in the X table, and sums stay
// unnormalised pairs, so a (k, atom) takes about 45 FP32 instructions in double-float (156 in the
// per-k normalised form) and 4 operations in FP64 (12). With ROWS, P comes from a (kx, ky) table.
#pragma once

#include "grx_df.cuh"
#include "grx_internal.cuh"

namespace grx {

// Tables of the na moved atoms, [k][atom]: X carries the (signed) charge, Y and Z do not.
// `tid` of `nthreads` threads fill them; at: the atoms' positions and charges.
template <bool F64>
__device__ __forceinline__ void eik_fill(const BoxDev& b, int na, const double* mx, const double* my, const double* mz,
                                         const double* mq, void* tables, int tid, int nthreads) {
  const int k0 = (b.kmax[0] + 1) * na, k1 = k0 + (b.kmax[1] + 1) * na;
  if constexpr (F64) {  // one thread per atom and axis: the recurrence of Initialize_Vectors_thread
    double2* tab = static_cast<double2*>(tables);
    for (int t = tid; t < 3 * na; t += nthreads) {
      const int at = t % na, d = t / na;
      const double f = b.inv[d] * mx[at] + b.inv[3 + d] * my[at] + b.inv[6 + d] * mz[at];
      double2* o = tab + (d == 0 ? 0 : (d == 1 ? k0 : k1)) + at;
      const int km = b.kmax[d];
      double2 e = make_double2(d == 0 ? mq[at] : 1.0, 0.0);
      o[0] = e;
      if (km >= 1) {
        double sn, cs;
        sincos(f * (2.0 * 3.14159265358979323846), &sn, &cs);
        const double2 e1 = make_double2(cs, sn);
        for (int k = 1; k <= km; ++k) {
          e = cmul(e, e1);
          o[k * na] = e;
        }
      }
    }
  } else {  // one thread per entry
    float4* tab = static_cast<float4*>(tables);
    const int n = k1 + (b.kmax[2] + 1) * na;
    for (int t = tid; t < n; t += nthreads) {
      const int d = t < k0 ? 0 : (t < k1 ? 1 : 2);
      const int r = t - (d == 0 ? 0 : (d == 1 ? k0 : k1));
      const int k = r / na, at = r - k * na;
      const double f = b.inv[d] * mx[at] + b.inv[3 + d] * my[at] + b.inv[6 + d] * mz[at];
      // without the whole cells, whose phase is a multiple of 2 pi: the roundings of k f grow with f, and
      // with them left in the error of dS was 1.4 times that of the chain of products (7e-15 so, 9e-15
      // there, of charges of order 1)
      tab[t] = df_eik(f - rint(f), k, d == 0 ? df_from(mq[at]) : df{1.0f, 0.0f});
    }
  }
}

// Sums of one thread over columns first, first + stride, ... below end.
struct EwSums64 { double same = 0.0, cross = 0.0; };
struct EwSumsDf { df a = {0.f, 0.f}, n = {0.f, 0.f}, c = {0.f, 0.f}; };  // A.dS, temp |dS|^2, F.dS

__device__ __forceinline__ df df_neg(df a) { return {-a.hi, -a.lo}; }

// FP64: same = sum temp (|S + dS|^2 - |S|^2) = sum temp dS.(2 S + dS), cross = sum temp Re(S_cross dS*), S + dS to s_out.
__device__ __forceinline__ void ewald_columns(const BoxDev& b, int na, const double2* tab, int first, int end, int stride,
                                              const double2* s_same, const double2* s_cross, double2* s_out, EwSums64& e) {
  const double2* ey = tab + (b.kmax[0] + 1) * na;
  const double2* ez = ey + (b.kmax[1] + 1) * na;
  for (int col = first; col < end; col += stride) {
    const int4 c = b.kcol[col];
    const int kx = c.x & 0xff, ky = ((c.x >> 8) & 0xff) - 128, az = c.x >> 16;
    const double2 *X = tab + na * kx, *Y = ey + na * abs(ky), *Z = ez + na * az;
    double sa = 0.0, sb = 0.0, sc = 0.0, sd = 0.0;
    for (int at = 0; at < na; ++at) {
      double2 y = Y[at];
      if (ky < 0) y.y = -y.y;
      const double2 p = cmul(X[at], y), z = Z[at];
      sa = fma(p.x, z.x, sa);
      sb = fma(p.y, z.y, sb);
      sc = fma(p.x, z.y, sc);
      sd = fma(p.y, z.x, sd);
    }
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const int j = h ? c.z : c.y;
      if (j < 0) continue;
      const int slot = h ? c.w - az : c.w + az;
      const double2 ds = h ? make_double2(sa + sb, sd - sc) : make_double2(sa - sb, sc + sd);
      const double t = b.ktemp[j];
      const double2 ov = s_same[slot], xv = s_cross[slot];
      const double2 nv = make_double2(ov.x + ds.x, ov.y + ds.y);
      // |S + dS|^2 - |S|^2 without the cancellation of the two squares
      e.same = fma(t, fma(ds.x, ov.x + nv.x, ds.y * (ov.y + nv.y)), e.same);
      e.cross = fma(t, fma(xv.x, ds.x, xv.y * ds.y), e.cross);
      if (s_out) s_out[slot] = nv;
    }
  }
}

// Double-float: the sums against the temp * S tables (ewA, ewF, ewT); dS as a float pair per part to
// ds_out by slot (only an accepted move needs S + dS, and its FP64 additions cost as much as all
// the rest of a k). rows: the (kx, ky) products of ROWS.
template <bool ROWS>
__device__ __forceinline__ void ewald_columns(const BoxDev& b, int na, const float4* tab, const float4* rows, int first,
                                              int end, int stride, float4* ds_out, EwSumsDf& e) {
  const float4* fy = tab + (b.kmax[0] + 1) * na;
  const float4* fz = fy + (b.kmax[1] + 1) * na;
  for (int col = first; col < end; col += stride) {
    const int4 c = b.kcol[col];
    const int kx = c.x & 0xff, ky = ((c.x >> 8) & 0xff) - 128, az = c.x >> 16;
    const float4 *X = tab + na * kx, *Y = fy + na * abs(ky), *Z = fz + na * az;
    const float4* P = ROWS ? rows + (kx * (2 * b.kmax[1] + 1) + ky + b.kmax[1]) * na : nullptr;
    const float sy = ky < 0 ? -1.f : 1.f;
    df sa = {0.f, 0.f}, sb = sa, sc = sa, sd = sa;
#pragma unroll 1
    for (int at = 0; at < na; ++at) {
      df pr = {0.f, 0.f}, pi = pr;
      if constexpr (ROWS) {
        const float4 r = P[at];
        pr = df{r.x, r.y};
        pi = df{r.z, r.w};
      } else {
        const float4 x = X[at], y = Y[at];
        const df yi = {sy * y.z, sy * y.w};
        df_mac(pr, df{x.x, x.y}, df{y.x, y.y});
        df_mac(pr, df{-x.z, -x.w}, yi);
        df_mac(pi, df{x.x, x.y}, yi);
        df_mac(pi, df{x.z, x.w}, df{y.x, y.y});
      }
      const float4 z = Z[at];
      df_mac(sa, pr, df{z.x, z.y});
      df_mac(sb, pi, df{z.z, z.w});
      df_mac(sc, pr, df{z.z, z.w});
      df_mac(sd, pi, df{z.x, z.y});
    }
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const int j = h ? c.z : c.y;
      if (j < 0) continue;
      const df re = df_add(sa, h ? sb : df_neg(sb)), im = df_add(sd, h ? df_neg(sc) : sc);
      const float4 A = b.ewA[j], F = b.ewF[j];
      const float2 T = b.ewT[j];
      df_mac(e.a, df{A.x, A.y}, re);
      df_mac(e.a, df{A.z, A.w}, im);
      df n2 = {0.f, 0.f};
      df_mac(n2, re, re);
      df_mac(n2, im, im);
      df_mac(e.n, df{T.x, T.y}, n2);
      // the largest terms of a move, and they cancel: kept normalised (unnormalised pairs were off by a
      // fifth to two fifths more)
      e.c = df_add(e.c, df_add(df_mul(df{F.x, F.y}, re), df_mul(df{F.z, F.w}, im)));
      if (ds_out) ds_out[h ? c.w - az : c.w + az] = make_float4(re.hi, re.lo, im.hi, im.lo);
    }
  }
}

// same = 2 A.dS + temp |dS|^2 of one thread.
__device__ __forceinline__ df ew_same(const EwSumsDf& e) { return df_add(df{2.f * e.a.hi, 2.f * e.a.lo}, e.n); }

}  // namespace grx
