// grx_ewald.cu -- Ewald Fourier-space kernels (structure factors, move delta,
// commit) and the FP64 totals used for drift checks.
#include <algorithm>
#include <cmath>
#include <vector>

#include "grx_ewcol.cuh"
#include "grx_host.h"
#include "grx_warp.cuh"

namespace grx {

constexpr int kBigMolecule = 64;  // molecules above this size get the pair-parallel exclusion

struct CompRanges {  // live atoms of every component, compact numbering
  int n;                                // total live atoms
  int ncomp, nhost;
  int off[GRX_MAX_COMPONENTS];          // storage offset
  int base[GRX_MAX_COMPONENTS + 1];     // compact offset
  int molsize[GRX_MAX_COMPONENTS];
};

__device__ __forceinline__ int comp_of(const CompRanges& r, int j, int& local) {
  int c = 0;
  while (c + 1 < r.ncomp && j >= r.base[c + 1]) ++c;
  local = j - r.base[c];
  return c;
}

// eik tables of the live atoms [r.first, r.n): e^{i k s} for k = 0..kmax per axis by the
// recurrence of Initialize_Vectors (Ewald_Energy_Functions.h:42-95). x tables carry the charge
// (q e^{i kx s}); x and y are [k][atom], z is [atom][k], as sk_kernel reads them.
__global__ void eik_tables_kernel(BoxDev b, CompRanges r, int first, double2* ex, double2* ey, double2* ez) {
  const int j = first + blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= r.n) return;
  int local;
  const int c = comp_of(r, j, local);
  const double4 p = atom_pos64(b, r.off[c] + local);
  const double PI2 = 2.0 * 3.14159265358979323846;
  const int d = blockIdx.y;  // one axis per thread: the recurrence is a serial chain
  const double s = (b.inv[d] * p.x + b.inv[3 + d] * p.y + b.inv[6 + d] * p.z) * PI2;
  const int km = b.kmax[d];
  const size_t n = r.n;
  double2* t = d == 0 ? ex + j : (d == 1 ? ey + j : ez + (size_t)j * (km + 1));
  const size_t stride = d == 2 ? 1 : n;
  double2 e = d == 0 ? make_double2(p.w, 0.0) : make_double2(1.0, 0.0);
  t[0] = e;
  if (km >= 1) {
    double sn, cs;
    sincos(s, &sn, &cs);
    const double2 e1 = make_double2(cs, sn);
    for (int k = 1; k <= km; ++k) {
      e = cmul(e, e1);
      t[k * stride] = e;
    }
  }
}

// Structure factors (Ewald_Total, ewald_preparation.h:128-147). A block holds the columns
// (kx, ky, |kz|) of a few (kx, ky) rows, one per thread, and walks one chunk of atoms in tiles
// of 32: the tile's q X Y products are formed once per row in shared memory, and a column's
// four real sums with Re Z and Im Z give both +kz and -kz, two FP64 FMAs per (k, atom) where
// the direct product of three factors takes ten. FP64 issue (two lanes per SM and clock)
// bounds it. Chunks hold framework or adsorbate atoms only; their partial S(k) go to `part`
// [chunk][active k].
constexpr int kSkCols = 128;
constexpr int kSkRows = 32;
constexpr int kSkTile = 32;

struct SkChunks {
  int n, nhost, n_host_chunks, n_chunks;  // atoms, framework atoms, chunks of them (0 when the framework's S is a parent's), all chunks
  int host_len, guest_len;                // atoms per chunk
  __device__ __forceinline__ void range(int k, int& a0, int& a1) const {
    const bool host = k < n_host_chunks;
    a0 = host ? k * host_len : nhost + (k - n_host_chunks) * guest_len;
    a1 = host ? min(a0 + host_len, nhost) : min(a0 + guest_len, n);
  }
};
constexpr int kSkSums = GRX_THREADS / 32;  // sums per k that the chunks are spread over (the warps of sk_reduce_kernel)

// The rows of the block's group in R, the row of this thread's column; returns |kz| of the column.
__device__ __forceinline__ int sk_column(const KRow* rows, int2 g, KRow* R, int& row) {
  const int tid = threadIdx.x, nr = g.y - g.x;
  for (int k = tid; k < nr; k += blockDim.x) R[k] = rows[g.x + k];
  __syncthreads();
  row = 0;
  while (row + 1 < nr && tid >= R[row + 1].col) ++row;
  return tid - R[row].col;
}

// S(+kz) and S(-kz) of this thread's column over the atoms [a0, a1), by the whole block.
__device__ __forceinline__ void sk_sums(const BoxDev& b, int n, double2 (*P)[kSkTile + 1], const KRow* R, int nr, int row,
                                        int az, bool live, int a0, int a1, const double2* ex, const double2* ey,
                                        const double2* ez, double2& plus, double2& minus) {
  const int tid = threadIdx.x, kz1 = b.kmax[2] + 1;
  const double2* z = ez + (live ? az : 0);
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  for (int t0 = a0; t0 < a1; t0 += kSkTile) {
    for (int e = tid; e < nr * kSkTile; e += blockDim.x) {
      const int k = e / kSkTile, at = e % kSkTile, j = t0 + at;
      double2 v = make_double2(0.0, 0.0);
      if (j < a1) {
        double2 y = ey[(size_t)abs(R[k].ky) * n + j];
        if (R[k].ky < 0) y.y = -y.y;
        v = cmul(ex[(size_t)R[k].kx * n + j], y);
      }
      P[k][at] = v;
    }
    __syncthreads();
    if (live) {
      const int m = min(kSkTile, a1 - t0);
      const double2* zt = z + (size_t)t0 * kz1;
#pragma unroll 4
      for (int at = 0; at < m; ++at) {
        const double2 v = P[row][at], w = zt[(size_t)at * kz1];
        s0 = fma(v.x, w.x, s0);
        s1 = fma(v.y, w.y, s1);
        s2 = fma(v.x, w.y, s2);
        s3 = fma(v.y, w.x, s3);
      }
    }
    __syncthreads();
  }
  plus = make_double2(s0 - s1, s2 + s3);
  minus = make_double2(s0 + s1, s3 - s2);
}

__global__ void __launch_bounds__(kSkCols) sk_kernel(BoxDev b, SkChunks c, const KRow* rows, const int2* groups,
                                                     const double2* ex, const double2* ey, const double2* ez,
                                                     double2* part) {
  __shared__ double2 P[kSkRows][kSkTile + 1];
  __shared__ KRow R[kSkRows];
  const int2 g = groups[blockIdx.x];
  int row;
  const int az = sk_column(rows, g, R, row);
  const bool live = az < R[row].ncol;
  const int chunk = blockIdx.y;
  int a0, a1;
  c.range(chunk, a0, a1);
  double2 plus, minus;
  sk_sums(b, c.n, P, R, g.y - g.x, row, az, live, a0, a1, ex, ey, ez, plus, minus);
  if (!live) return;
  double2* out = part + (size_t)chunk * b.nact;
  const int jp = R[row].index(az), jm = az ? R[row].index(-az) : -1;
  if (jp >= 0) out[jp] = plus;
  if (jm >= 0) out[jm] = minus;
}

// Without room for the chunks' partial sums: a block walks the chunks of one kind (blockIdx.y 0 the
// framework's, 1 the adsorbates') behind one another and adds them up as sk_reduce_kernel does,
// every eighth chunk to one of eight sums, so that S(k) is the same to the last bit whatever the
// memory has room for.
__global__ void __launch_bounds__(kSkCols) sk_in_place_kernel(BoxDev b, SkChunks c, const KRow* rows,
                                                              const int2* groups, const double2* ex, const double2* ey,
                                                              const double2* ez) {
  __shared__ double2 P[kSkRows][kSkTile + 1];
  __shared__ KRow R[kSkRows];
  const int2 g = groups[blockIdx.x];
  int row;
  const int az = sk_column(rows, g, R, row);
  const bool live = az < R[row].ncol;
  const bool host = blockIdx.y == 0;
  const int first = host ? 0 : c.n_host_chunks, end = host ? c.n_host_chunks : c.n_chunks;
  if (first == end) return;
  double2 sp[kSkSums], sm[kSkSums];
  for (int w = 0; w < kSkSums; ++w) sp[w] = sm[w] = make_double2(0.0, 0.0);
  for (int k0 = first; k0 < end; k0 += kSkSums)
#pragma unroll
    for (int w = 0; w < kSkSums; ++w) {
      if (k0 + w >= end) break;
      int a0, a1;
      c.range(k0 + w, a0, a1);
      double2 plus, minus;
      sk_sums(b, c.n, P, R, g.y - g.x, row, az, live, a0, a1, ex, ey, ez, plus, minus);
      sp[w].x += plus.x; sp[w].y += plus.y;
      sm[w].x += minus.x; sm[w].y += minus.y;
    }
  if (!live) return;
  for (int w = 1; w < kSkSums; ++w) {
    sp[0].x += sp[w].x; sp[0].y += sp[w].y;
    sm[0].x += sm[w].x; sm[0].y += sm[w].y;
  }
  double2* out = host ? b.s_fw : b.s_ads;
  const int jp = R[row].index(az), jm = az ? R[row].index(-az) : -1;
  if (jp >= 0) out[b.kact[jp].w] = sp[0];
  if (jm >= 0) out[b.kact[jm].w] = sm[0];
}

// Sums the chunks of every active k, writes S(k) and adds the Fourier energies (Ewald_Total,
// ewald_preparation.h:150-161): epart per block {gg, hh, hg}. Bound by the latency of the chunk
// reads (the sums are in L2): a block takes one k per lane and every eighth chunk per warp, in a
// fixed order, so there are eight reads in flight for one and eight times the blocks (one k per
// thread and all chunks behind one another, 110 of them for the 3456-atom silica: 357 us for its
// totals, 332 us so).
constexpr int kSkReduceK = 32;
__global__ void __launch_bounds__(GRX_THREADS) sk_reduce_kernel(BoxDev b, const double2* part, int nh, int ng,
                                                                double* epart) {
  constexpr int W = kSkSums;
  __shared__ double2 F[W][32], G[W][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = blockIdx.x * kSkReduceK + lane;
  if (part) {
    double2 f = make_double2(0.0, 0.0), a = f;
    if (j < b.nact) {
#pragma unroll 4
      for (int k = w; k < nh; k += W) {
        const double2 v = part[(size_t)k * b.nact + j];
        f.x += v.x; f.y += v.y;
      }
#pragma unroll 4
      for (int k = nh + w; k < nh + ng; k += W) {
        const double2 v = part[(size_t)k * b.nact + j];
        a.x += v.x; a.y += v.y;
      }
    }
    F[w][lane] = f;
    G[w][lane] = a;
    __syncthreads();
  }
  if (w != 0) return;
  double gg = 0.0, hh = 0.0, hg = 0.0;
  if (j < b.nact) {
    const int slot = b.kact[j].w;
    double2 f, a;
    if (part) {
      f = F[0][lane];
      a = G[0][lane];
      for (int k = 1; k < W; ++k) {
        f.x += F[k][lane].x; f.y += F[k][lane].y;
        a.x += G[k][lane].x; a.y += G[k][lane].y;
      }
      if (b.shared_host) f = b.s_fw[slot];  // a replica reads its parent's
      else b.s_fw[slot] = f;
      b.s_ads[slot] = a;
    } else {
      f = b.s_fw[slot];
      a = b.s_ads[slot];
    }
    b.s_tmp[slot] = a;
    const double t = b.ktemp[j];
    gg = t * (a.x * a.x + a.y * a.y);
    hh = t * (f.x * f.x + f.y * f.y);
    hg = t * (f.x * a.x + f.y * a.y) * 2.0;
  }
  gg = warp_sum(gg);
  hh = warp_sum(hh);
  hg = warp_sum(hg);
  if (lane == 0) {
    epart[3 * blockIdx.x] = gg;
    epart[3 * blockIdx.x + 1] = hh;
    epart[3 * blockIdx.x + 2] = hg;
  }
}

// h(s) = erf(alpha sqrt s) / sqrt s from the table, by the library outside it.
static __device__ __noinline__ double excl_h_cold(const BoxDev& b, double s) {
  const double r = sqrt(s);
  return erf(b.alpha * r) / r;
}
__device__ __forceinline__ double excl_h(const BoxDev& b, double s) {
  const int k = table64_piece<kShiftH64>(s, b.h64_base);
  return (unsigned)k < (unsigned)b.h64_n ? table64<kShiftH64>(b.h64, k, s) : excl_h_cold(b, s);
}

// Self energy and intramolecular erf exclusion per atom (ewald_preparation.h:189-249),
// partial sums per block: [self_all, self_host, excl_all, excl_host].
__global__ void __launch_bounds__(GRX_THREADS) self_excl_kernel(BoxDev b, CompRanges r, double* part) {
  __shared__ double sbuf[32];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  double sa = 0, sh = 0, ea = 0, eh = 0;
  if (j < r.n) {
    int local;
    const int c = comp_of(r, j, local);
    const double4 p = atom_pos64(b, r.off[c] + local);
    const double pself = b.prefactor * b.alpha / sqrt(3.14159265358979323846);
    const double v = pself * p.w * p.w;
    sa = v;
    if (c < r.nhost) sh = v;
    const int ms = r.molsize[c];
    const int mol0 = (local / ms) * ms;
    const int lend = ms > kBigMolecule ? local + 1 : min(mol0 + ms, r.base[c + 1] - r.base[c]);
    for (int l2 = local + 1; l2 < lend; ++l2) {
      const double4 q = atom_pos64(b, r.off[c] + l2);
      double x = p.x - q.x, y = p.y - q.y, z = p.z - q.z;
      pbc64(b, x, y, z);
      const double e = b.prefactor * p.w * q.w * excl_h(b, x * x + y * y + z * z);
      ea += e;
      if (c < r.nhost) eh += e;
    }
  }
  sa = block_sum(sa, sbuf);
  sh = block_sum(sh, sbuf);
  ea = block_sum(ea, sbuf);
  eh = block_sum(eh, sbuf);
  if (threadIdx.x == 0) {
    part[4 * blockIdx.x + 0] = sa;
    part[4 * blockIdx.x + 1] = sh;
    part[4 * blockIdx.x + 2] = ea;
    part[4 * blockIdx.x + 3] = eh;
  }
}

// Intramolecular erf exclusion of the molecules of one component with more than
// kBigMolecule atoms (a framework is one such molecule): the pairs i < j of each molecule in
// 64 x 64 tiles, atoms of the j tile in shared memory. FP64 issue bounds it, so a pair takes
// its image from FP32 fractions (image64) and erf(alpha r) / r from the table: 16 FP64
// operations where sqrt, erf and the division took about 100.
// part per block: [excl_all, excl_host].
constexpr int kExclTile = 64;

__global__ void __launch_bounds__(GRX_THREADS) big_excl_kernel(BoxDev b, CompRanges r, int c, double* part) {
  __shared__ double sbuf[32];
  __shared__ double4 J[kExclTile];
  __shared__ float4 H[kExclTile];
  const int tid = threadIdx.x;
  const int ms = r.molsize[c];
  const int n = r.base[c + 1] - r.base[c];
  const long long nmol = (n + ms - 1) / ms;
  const long long T = (ms + kExclTile - 1) / kExclTile, per = T * (T + 1) / 2;
  const float4* hi = c < r.nhost ? b.hhi : b.hi;
  constexpr int kParts = GRX_THREADS / kExclTile, kSpan = kExclTile / kParts;
  double ea = 0.0;
  for (long long p = blockIdx.x; p < nmol * per; p += gridDim.x) {
    const long long m = p / per;
    const long long t = p - m * per;  // row-major upper triangle, counted from its last row
    const long long u = per - 1 - t;
    long long k = (long long)((sqrtf(8.0f * (float)u + 1.0f) - 1.0f) * 0.5f);
    while (k * (k + 1) / 2 > u) --k;
    while ((k + 1) * (k + 2) / 2 <= u) ++k;
    const int ti = (int)(T - 1 - k), tj = (int)(T - 1 - (u - k * (k + 1) / 2));
    const int m0 = (int)(m * ms), mend = min(m0 + ms, n);
    const int i0 = m0 + ti * kExclTile, j0 = m0 + tj * kExclTile;
    __syncthreads();
    if (tid < kExclTile) {
      const int j = j0 + tid;
      const bool in = j < mend;
      J[tid] = in ? atom_pos64(b, r.off[c] + j) : make_double4(0.0, 0.0, 0.0, 0.0);
      H[tid] = in ? hi[r.off[c] + j] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    const int i = i0 + tid % kExclTile, s0 = tid / kExclTile * kSpan;
    if (i < mend) {
      const double4 a = atom_pos64(b, r.off[c] + i);
      const float4 ah = hi[r.off[c] + i];
      const bool near = fabsf(ah.x) < kNearCoord && fabsf(ah.y) < kNearCoord && fabsf(ah.z) < kNearCoord;
      double e = 0.0;
      for (int s = s0; s < s0 + kSpan; ++s) {
        const int j = j0 + s;
        if (j <= i || j >= mend) continue;
        const double4 q = J[s];
        const float4 qh = H[s];
        double x = a.x - q.x, y = a.y - q.y, z = a.z - q.z;
        image64(b, near, ah.x - qh.x, ah.y - qh.y, ah.z - qh.z, x, y, z);
        e = fma(q.w, excl_h(b, x * x + y * y + z * z), e);
      }
      ea = fma(a.w, e, ea);
    }
  }
  ea = block_sum(ea * b.prefactor, sbuf);
  if (tid == 0) {
    part[2 * blockIdx.x + 0] = ea;
    part[2 * blockIdx.x + 1] = c < r.nhost ? ea : 0.0;
  }
}

// VDW + real Coulomb of one adsorbate atom per cluster against every atom outside its
// molecule, through the trial pass (VDWReal_Total_CPU, VDW_Coulomb.cu:34-226; device form
// Total_VDW_Coulomb_Energy :1580-1665): hg sums as they are, gg sums count every pair twice.
// part per atom: hg_v hg_r gg_v gg_r and the overlap flag (a pair above the overlap criterion
// or closer than 0.1 A, VDWCoulEnergy_Total :1385-1386) as the fifth value.
__global__ void __cluster_dims__(kTrialCtas, 1, 1) __launch_bounds__(kTrialWarps * 32)
    guest_total_kernel(const __grid_constant__ BoxDev box, const __grid_constant__ CompRanges r, double* part) {
  __shared__ TrialWork W;
  __shared__ BoxDev b;
  __shared__ Bead bead;
  __shared__ int who[2];
  copy_words(&b, &box);
  __syncthreads();
  const int t = (int)blockIdx.x / kTrialCtas;
  if (threadIdx.x == 0) {
    int local;
    const int c = comp_of(r, r.base[r.nhost] + t, local);
    const int i = r.off[c] + local;
    const double4 p = b.pos64[i];
    const int2 m = b.meta[i];
    make_bead(bead, p.x, p.y, p.z, p.w, b.scale[i], m.x, b.prefactor);
    who[0] = c;
    who[1] = m.y;
  }
  __syncthreads();
  double sum;
  int flag;
  trial_cluster_pass<GRX_FP64>(b, &bead, W, 1, who[0], who[1], -1, -1, sum, flag);
  const int warp = threadIdx.x >> 5;
  if (cluster_rank() == 0 && warp < 4 && (threadIdx.x & 31) == 0) {
    part[5 * t + warp] = warp < 2 ? sum : 0.5 * sum;
    if (warp == 0) part[5 * t + 4] = flag ? 1.0 : 0.0;
  }
}

// VDW + real Coulomb between framework atoms of different molecules or components (ordered
// pairs, factor 0.5); launched only when there are such pairs. Thread i, blockIdx.y a slice of
// the j atoms. part per block: hh_v hh_r.
__global__ void __launch_bounds__(GRX_THREADS) host_total_kernel(BoxDev b, CompRanges r, double* part) {
  __shared__ double sbuf[32];
  const int nh = r.base[r.nhost];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  LaneAcc<GRX_FP64> acc;
  double q = 0.0;
  int flag = 0;
  if (j < nh) {
    int li;
    const int ci = comp_of(r, j, li);
    const int ii = r.off[ci] + li;
    const double4 p = atom_pos64(b, ii);
    const int2 mi = atom_meta(b, ii);
    Bead bd;
    make_bead(bd, p.x, p.y, p.z, p.w, atom_scale(b, ii), mi.x, b.prefactor);
    q = b.prefactor * p.w;
    const int per = (nh + gridDim.y - 1) / gridDim.y;
    const int j1 = min(nh, (int)(blockIdx.y + 1) * per);
    for (int jc = blockIdx.y * per; jc < j1; ++jc) {
      int lj;
      const int cj = comp_of(r, jc, lj);
      const int jj = r.off[cj] + lj;
      if (ci == cj && atom_meta(b, jj).y == mi.y) continue;
      if (pair_screen<GRX_FP64, true>(b, jj, bd)) pair_dense<GRX_FP64>(b, true, jj, bd, acc, flag);
    }
  }
  const double v = block_sum(0.5 * acc.v, sbuf), e = block_sum(0.5 * q * acc.r, sbuf);
  if (threadIdx.x == 0) {
    const int k = blockIdx.y * gridDim.x + blockIdx.x;
    part[2 * k] = v;
    part[2 * k + 1] = e;
  }
}

// Fourier delta of one move (Fourier_Ewald_Diff, Ewald_Energy_Functions.h:280-397) by columns of
// k (grx_ewcol.cuh): every block rebuilds the eik tables of the few moved atoms in shared
// memory, then takes a strided subset of the columns. A call is latency, so the blocks are small
// (two warps, at most two blocks an SM): 12 on the silica box, where one thread per k made 6.
// at: x, y, z, q of the moved atoms (the old ones with their charges negated), in pinned host
// memory, as is part, per block {same, cross}.
constexpr int kDeltaThreads = 64;

__global__ void __launch_bounds__(kDeltaThreads) ewald_delta_kernel(const __grid_constant__ BoxDev b, const double* at,
                                                                    int na, const double2* s_same,
                                                                    const double2* s_cross, double2* s_out, double* part) {
  extern __shared__ double2 eik_s[];
  __shared__ double sbuf[32];
  eik_fill<true>(b, na, at, at + na, at + 2 * na, at + 3 * na, eik_s, threadIdx.x, blockDim.x);
  __syncthreads();
  EwSums64 e;
  ewald_columns(b, na, eik_s, blockIdx.x * blockDim.x + threadIdx.x, b.ncol, gridDim.x * blockDim.x, s_same, s_cross, s_out,
                e);
  const double same = block_sum(e.same, sbuf), cross = block_sum(e.cross, sbuf);
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = same;
    part[2 * blockIdx.x + 1] = cross;
  }
}

__global__ void commit_kernel(BoxDev b, double2* dst, const double2* src) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < b.nact; j += gridDim.x * blockDim.x) {
    const int slot = b.kact[j].w;
    dst[slot] = src[slot];
  }
}

static CompRanges ranges(grx_box* b) {
  CompRanges r{};
  r.ncomp = b->ncomp;
  r.nhost = b->nhost;
  int acc = 0;
  for (int c = 0; c < b->ncomp; ++c) {
    r.off[c] = (int)b->off[c];
    r.base[c] = acc;
    r.molsize[c] = (int)b->molsize[c];
    acc += b->size[c];
  }
  r.base[b->ncomp] = acc;
  r.n = acc;
  return r;
}

static grx_status sync_sizes(grx_box* b) {
  GRX_CHECK_CUDA(cudaMemcpyAsync(b->size, b->d_size, GRX_MAX_COMPONENTS * sizeof(int),
                                 cudaMemcpyDeviceToHost, b->stream), "read sizes");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "sync sizes");
  return GRX_OK;
}

// Structure factors and Fourier totals (out8), and with `pairs` the VDW + real Coulomb totals
// {hh_v, hh_r, hg_v, hg_r, gg_v, gg_r} and the overlap flag: every kernel enqueued, one read back.
static grx_status totals(grx_box* b, double* out8, double* pairs, uint8_t* overlap) {
  grx_status st = sync_sizes(b);
  if (st) return st;
  refresh_dev(b);
  const CompRanges r = ranges(b);
  const size_t n = std::max(r.n, 1);
  const size_t ntab = (size_t)(b->dev.kmax[0] + b->dev.kmax[1] + b->dev.kmax[2] + 3) * n;
  const int sms = sm_count(b);
  const int nhost = r.base[r.nhost], nguest = r.n - nhost;
  const int nblk_atoms = (r.n + GRX_THREADS - 1) / GRX_THREADS;
  const int nblk_big = 4 * sms;
  const int nblk_k = (b->nact + kSkReduceK - 1) / kSkReduceK;
  // framework pairs count only between molecules or components
  int host_comps = 0;
  bool host_pairs = false;
  for (int c = 0; c < r.nhost; ++c) {
    if (b->size[c] > 0) ++host_comps;
    host_pairs = host_pairs || b->many_mols[c];
  }
  host_pairs = pairs && (host_pairs || host_comps > 1);
  const int hx = (nhost + GRX_THREADS - 1) / GRX_THREADS;
  const int hy = host_pairs ? std::max(1, std::min(64, 4 * sms / std::max(hx, 1))) : 0;
  std::vector<int> big;
  for (int c = 0; c < r.ncomp; ++c)
    if (r.molsize[c] > kBigMolecule && r.base[c + 1] - r.base[c] >= 2) big.push_back(c);
  // result doubles: self + small exclusions, large exclusions, Fourier energies, pair totals
  const size_t o_big = 4 * (size_t)std::max(nblk_atoms, 1), o_k = o_big + 2 * (size_t)nblk_big * big.size(),
               o_pair = o_k + 3 * (size_t)nblk_k, o_host = o_pair + (pairs ? 5 * (size_t)nguest : 0),
               n_out = o_host + 2 * (size_t)hx * hy;
  // chunks of atoms: about eight blocks of sk_kernel per SM, at least one tile each
  SkChunks ck{};
  ck.n = (int)n;
  ck.nhost = nhost;
  const int fw_atoms = b->parent ? 0 : nhost;
  const bool sums = b->nact > 0 && r.n > 0;
  auto split = [&](int want) {
    auto len = [&](int atoms) {
      const int per = (int)(((int64_t)(fw_atoms + nguest) + want - 1) / want);
      return std::max(kSkTile, std::min((per + kSkTile - 1) / kSkTile * kSkTile, (std::max(atoms, 1) + kSkTile - 1) / kSkTile * kSkTile));
    };
    ck.host_len = len(fw_atoms);
    ck.guest_len = len(nguest);
    ck.n_host_chunks = fw_atoms ? (fw_atoms + ck.host_len - 1) / ck.host_len : 0;
    return ck.n_host_chunks + (nguest ? (nguest + ck.guest_len - 1) / ck.guest_len : 0);
  };
  int nchunks = 0;
  size_t part_bytes = 0;
  if (sums) {
    nchunks = split(std::max(1, 8 * sms / std::max(b->n_kgroups, 1)));
    part_bytes = (size_t)nchunks * b->nact * sizeof(double2);
  }
  const size_t fixed = ntab * sizeof(double2) + n_out * sizeof(double);
  st = ensure_scratch(b, fixed + part_bytes);
  if (st == GRX_ERR_OUT_OF_MEMORY && part_bytes) {  // the same sums, written in place chunk after chunk
    part_bytes = 0;
    st = ensure_scratch(b, fixed);
  }
  if (st) return st;
  double2* ex = (double2*)b->scratch;
  double2* ey = ex + (size_t)(b->dev.kmax[0] + 1) * n;
  double2* ez = ey + (size_t)(b->dev.kmax[1] + 1) * n;
  double* out = (double*)(ex + ntab);
  double2* part = part_bytes ? (double2*)(out + (n_out + 1) / 2 * 2) : nullptr;
  cudaStream_t s = b->stream;
  if (!b->parent)  // a replica's framework structure factor is its parent's, shared by every replica
    GRX_CHECK_CUDA(cudaMemsetAsync(b->s_fw, 0, b->nvec * sizeof(double2), s), "clear S_fw");
  GRX_CHECK_CUDA(cudaMemsetAsync(b->s_ads, 0, b->nvec * sizeof(double2), s), "clear S_ads");
  GRX_CHECK_CUDA(cudaMemsetAsync(b->s_tmp, 0, b->nvec * sizeof(double2), s), "clear S_tmp");
  std::vector<double> h(n_out, 0.0);
  if (sums) {
    const int first = b->parent ? nhost : 0;
    if (r.n > first)
      eik_tables_kernel<<<dim3((r.n - first + 127) / 128, 3), 128, 0, s>>>(b->dev, r, first, ex, ey, ez);
    ck.n_chunks = nchunks;
    if (part)
      sk_kernel<<<dim3(b->n_kgroups, nchunks), kSkCols, 0, s>>>(b->dev, ck, b->krow, b->kgroup, ex, ey, ez, part);
    else if (nchunks)
      sk_in_place_kernel<<<dim3(b->n_kgroups, 2), kSkCols, 0, s>>>(b->dev, ck, b->krow, b->kgroup, ex, ey, ez);
    count_launch((r.n > first) + (nchunks > 0));
  }
  if (b->nact > 0) {
    sk_reduce_kernel<<<nblk_k, GRX_THREADS, 0, s>>>(b->dev, part, ck.n_host_chunks, nchunks - ck.n_host_chunks, out + o_k);
    count_launch();
  }
  if (r.n > 0) {
    self_excl_kernel<<<nblk_atoms, GRX_THREADS, 0, s>>>(b->dev, r, out);
    count_launch();
    for (size_t g = 0; g < big.size(); ++g) {
      big_excl_kernel<<<nblk_big, GRX_THREADS, 0, s>>>(b->dev, r, big[g], out + o_big + 2 * (size_t)nblk_big * g);
      count_launch();
    }
  }
  if (pairs && nguest > 0) {
    guest_total_kernel<<<nguest * kTrialCtas, kTrialWarps * 32, 0, s>>>(b->dev, r, out + o_pair);
    count_launch();
  }
  if (host_pairs && nhost > 0) {
    host_total_kernel<<<dim3(hx, hy), GRX_THREADS, 0, s>>>(b->dev, r, out + o_host);
    count_launch();
  }
  GRX_CHECK_CUDA(cudaGetLastError(), "totals launch");
  if (r.n > 0 || b->nact > 0)
    GRX_CHECK_CUDA(cudaMemcpyAsync(h.data(), out, n_out * sizeof(double), cudaMemcpyDeviceToHost, s), "read totals");
  GRX_CHECK_CUDA(cudaStreamSynchronize(s), "totals");
  double gg = 0, hh = 0, hg = 0;
  for (int k = 0; k < nblk_k; ++k) {
    gg += h[o_k + 3 * k]; hh += h[o_k + 3 * k + 1]; hg += h[o_k + 3 * k + 2];
  }
  double sa = 0, sh = 0, ea = 0, eh = 0;
  for (int k = 0; k < nblk_atoms; ++k) {
    sa += h[4 * k]; sh += h[4 * k + 1]; ea += h[4 * k + 2]; eh += h[4 * k + 3];
  }
  if (r.n > 0)
    for (size_t k = 0; k < (size_t)nblk_big * big.size(); ++k) {
      ea += h[o_big + 2 * k];
      eh += h[o_big + 2 * k + 1];
    }
  out8[0] = gg; out8[1] = hh; out8[2] = hg;
  out8[3] = sa; out8[4] = sh; out8[5] = -ea; out8[6] = -eh;
  out8[7] = (double)b->nact;
  b->sk_valid = true;
  b->ewdf_valid = false;
  if (pairs) {
    for (int q = 0; q < 6; ++q) pairs[q] = 0.0;
    *overlap = 0;
    for (int t = 0; t < nguest; ++t) {
      for (int q = 0; q < 4; ++q) pairs[2 + q] += h[o_pair + 5 * (size_t)t + q];
      if (h[o_pair + 5 * (size_t)t + 4] != 0.0) *overlap = 1;
    }
    if (host_pairs)
      for (int k = 0; k < hx * hy; ++k) {
        pairs[0] += h[o_host + 2 * (size_t)k];
        pairs[1] += h[o_host + 2 * (size_t)k + 1];
      }
  }
  return GRX_OK;
}

}  // namespace grx

using namespace grx;

extern "C" {

grx_status grx_ewald_total(grx_box* b, double* out8) {
  GRX_REQUIRE(b && out8, "grx_ewald_total: null argument");
  return totals(b, out8, nullptr, nullptr);
}

grx_status grx_total_energy(grx_box* b, grx_energy* out) { return grx_total_energy_overlap(b, out, nullptr); }

grx_status grx_total_energy_overlap(grx_box* b, grx_energy* out, uint8_t* overlap) {
  GRX_REQUIRE(b && out, "grx_total_energy: null argument");
  double ew[8], e[6];
  uint8_t ovl = 0;
  grx_status st = totals(b, ew, e, &ovl);
  if (st) return st;
  if (overlap) *overlap = ovl;
  out->hh_vdw = e[0]; out->hh_real = e[1];
  out->hg_vdw = e[2]; out->hg_real = e[3];
  out->gg_vdw = e[4]; out->gg_real = e[5];
  // Ewald blocks as Ewald_Total combines them (ewald_preparation.h:170-249)
  out->hh_ewald = ew[1] - ew[4] + ew[6];
  out->hg_ewald = ew[2];
  out->gg_ewald = ew[0] + ew[1] - ew[3] + ew[5];
  return GRX_OK;
}

}  // extern "C"

namespace grx {

// Runs the Fourier delta of the staged old / new atoms (ewald_delta_kernel) against
// `same` (its S + dS staged into s_tmp) and `cross`; returns the two sums.
static grx_status ewald_delta_run(grx_box* b, const double* old_pos, const double* old_qs, size_t n_old,
                                  const double* new_pos, const double* new_qs, size_t n_new, const double2* same,
                                  const double2* cross, double& s_same, double& s_cross) {
  s_same = s_cross = 0.0;
  const size_t na = n_old + n_new;
  std::vector<double> pos(3 * na), q(na);
  grx_status st = fetch(pos.data(), old_pos, 3 * n_old * sizeof(double), "read old pos");
  if (!st) st = fetch(q.data(), old_qs, n_old * sizeof(double), "read old q");
  if (!st) st = fetch(pos.data() + 3 * n_old, new_pos, 3 * n_new * sizeof(double), "read new pos");
  if (!st) st = fetch(q.data() + n_old, new_qs, n_new * sizeof(double), "read new q");
  if (st) return st;
  refresh_dev(b);
  const int nblk = std::max(1, std::min((b->ncol + kDeltaThreads - 1) / kDeltaThreads, 2 * sm_count(b)));
  st = ensure_pinned(b, (4 * na + 2 * (size_t)nblk) * sizeof(double));
  if (st) return st;
  double* at = (double*)b->pinned;
  double* part = at + 4 * na;
  for (size_t a = 0; a < na; ++a) {
    for (int k = 0; k < 3; ++k) at[k * na + a] = pos[3 * a + k];
    at[3 * na + a] = a < n_old ? -q[a] : q[a];
  }
  if (b->nact > 0 && na > 0) {
    const size_t smem = (size_t)(b->dev.kmax[0] + b->dev.kmax[1] + b->dev.kmax[2] + 3) * na * sizeof(double2);
    ewald_delta_kernel<<<nblk, kDeltaThreads, smem, b->stream>>>(b->dev, at, (int)na, same, cross, b->s_tmp, part);
    count_launch();
    GRX_CHECK_CUDA(cudaGetLastError(), "ewald delta launch");
  }
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "ewald delta");
  if (b->nact > 0 && na > 0)
    for (int k = 0; k < nblk; ++k) { s_same += part[2 * k]; s_cross += part[2 * k + 1]; }
  return GRX_OK;
}

}  // namespace grx

extern "C" {

grx_status grx_ewald_delta(grx_box* b, int32_t comp, int32_t move_type, const double* old_pos,
                           const double* old_qs, size_t n_old, const double* new_pos,
                           const double* new_qs, size_t n_new, double scale_coul_new,
                           double* out2) {
  GRX_REQUIRE(b && out2, "grx_ewald_delta: null argument");
  GRX_REQUIRE(comp >= 0 && comp < b->ncomp, "grx_ewald_delta: component out of range");
  GRX_REQUIRE(n_old <= GRX_MAX_MOLSIZE && n_new <= GRX_MAX_MOLSIZE, "grx_ewald_delta: too many atoms");
  GRX_REQUIRE((n_old == 0 || (old_pos && old_qs)) && (n_new == 0 || (new_pos && new_qs)),
              "grx_ewald_delta: atom arrays missing");
  out2[0] = out2[1] = 0.0;
  if (b->dev.no_charges && !b->has_charge[comp]) return GRX_OK;
  const bool host_comp = comp < b->nhost;
  double s_same = 0, s_cross = 0;
  grx_status st = ewald_delta_run(b, old_pos, old_qs, n_old, new_pos, new_qs, n_new, host_comp ? b->s_fw : b->s_ads,
                                  host_comp ? b->s_ads : b->s_fw, s_same, s_cross);
  if (st) return st;
  // rigid exclusion correction of GPU_EwaldDifference_General (:548-574)
  if (b->rigid[comp]) {
    const double ex = b->excl_intra[comp] + b->excl_self[comp];
    if (move_type == GRX_MOVE_INSERTION || move_type == GRX_MOVE_SINGLE_INSERTION)
      s_same -= ex * (scale_coul_new * scale_coul_new - 0.0);
    else if (move_type == GRX_MOVE_DELETION || move_type == GRX_MOVE_SINGLE_DELETION)
      s_same -= ex * (0.0 - 1.0);
  }
  out2[0] = s_same;
  out2[1] = 2.0 * s_cross;
  return GRX_OK;
}

grx_status grx_ewald_delta_lambda(grx_box* b, int32_t comp, const double* pos, const double* charge, size_t n,
                                  double scale_coul_old, double scale_coul_new, int32_t use_staged, double* out2) {
  GRX_REQUIRE(b && out2, "grx_ewald_delta_lambda: null argument");
  GRX_REQUIRE(comp >= b->nhost && comp < b->ncomp, "grx_ewald_delta_lambda: component must be an adsorbate");
  GRX_REQUIRE(n >= 1 && n <= GRX_MAX_MOLSIZE && pos && charge, "grx_ewald_delta_lambda: bad atom arrays");
  out2[0] = out2[1] = 0.0;
  if (b->dev.no_charges && !b->has_charge[comp]) return GRX_OK;
  std::vector<double> hq(n), qo(n), qn(n);
  grx_status st = fetch(hq.data(), charge, n * sizeof(double), "read charges");
  if (st) return st;
  for (size_t a = 0; a < n; ++a) {  // Fourier_Ewald_Diff_LambdaChange: the same atoms, old and new scaleCoul
    qo[a] = hq[a] * scale_coul_old;
    qn[a] = hq[a] * scale_coul_new;
  }
  double s_same = 0, s_cross = 0;
  st = ewald_delta_run(b, pos, qo.data(), n, pos, qn.data(), n, use_staged ? b->s_tmp : b->s_ads, b->s_fw,
                                  s_same, s_cross);
  if (st) return st;
  // GPU_EwaldDifference_LambdaChange (:782-785): exclusion times the change of scaleCoul^2
  s_same -= (b->excl_intra[comp] + b->excl_self[comp]) *
            (scale_coul_new * scale_coul_new - scale_coul_old * scale_coul_old);
  out2[0] = s_same;
  out2[1] = 2.0 * s_cross;
  return GRX_OK;
}

grx_status grx_ewald_delta_identity_swap(grx_box* b, int32_t old_comp, int32_t new_comp, const double* old_pos,
                                         const double* old_qs, size_t n_old, const double* new_pos,
                                         const double* new_qs, size_t n_new, double* out2) {
  GRX_REQUIRE(b && out2, "grx_ewald_delta_identity_swap: null argument");
  GRX_REQUIRE(old_comp >= b->nhost && old_comp < b->ncomp && new_comp >= b->nhost && new_comp < b->ncomp,
              "grx_ewald_delta_identity_swap: both components must be adsorbates");
  GRX_REQUIRE(n_old <= GRX_MAX_MOLSIZE && n_new <= GRX_MAX_MOLSIZE, "grx_ewald_delta_identity_swap: too many atoms");
  GRX_REQUIRE((n_old == 0 || (old_pos && old_qs)) && (n_new == 0 || (new_pos && new_qs)),
              "grx_ewald_delta_identity_swap: atom arrays missing");
  out2[0] = out2[1] = 0.0;
  const bool q_old = b->has_charge[old_comp] != 0, q_new = b->has_charge[new_comp] != 0;
  if (b->dev.no_charges && !q_old && !q_new) return GRX_OK;
  // atoms of an uncharged side do not enter (Ewald_Energy_Functions.h:588-597)
  const size_t no = q_old ? n_old : 0, nn = q_new ? n_new : 0;
  if (no + nn == 0) return GRX_OK;
  double s_same = 0, s_cross = 0;
  grx_status st = ewald_delta_run(b, old_pos, old_qs, no, new_pos, new_qs, nn, b->s_ads, b->s_fw, s_same, s_cross);
  if (st) return st;
  if (b->rigid[new_comp] && q_new) s_same -= (b->excl_intra[new_comp] + b->excl_self[new_comp]) * 1.0;
  if (b->rigid[old_comp] && q_old) s_same -= (b->excl_intra[old_comp] + b->excl_self[old_comp]) * -1.0;
  out2[0] = s_same;
  out2[1] = 2.0 * s_cross;
  return GRX_OK;
}

grx_status grx_ewald_commit(grx_box* b, int32_t comp) {
  GRX_REQUIRE(b && comp >= 0 && comp < b->ncomp, "grx_ewald_commit: bad argument");
  if (b->nact == 0) return GRX_OK;
  refresh_dev(b);
  GRX_REQUIRE(comp >= b->nhost || !b->parent, "grx_ewald_commit: a replica cannot move its shared framework");
  double2* dst = comp < b->nhost ? b->s_fw : b->s_ads;
  commit_kernel<<<std::max(1, std::min((b->nact + 255) / 256, sm_count(b))), 256, 0, b->stream>>>(b->dev, dst, b->s_tmp);
  count_launch();
  b->ewdf_valid = false;
  GRX_CHECK_CUDA(cudaGetLastError(), "commit launch");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "commit");
  return GRX_OK;
}

}  // extern "C"
