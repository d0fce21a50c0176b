// grx_cbmc.cuh -- block-level CBMC stages shared by the Widom and GCMC kernels.
//
// Every function here is called by all threads of a block (NW warps) with the same
// arguments; each ends with the block synchronised and its results in the
// shared-memory workspace CbmcWork<NW>. The stages restate gRASPA's CBMC move pieces:
//   gen_first_trials  get_random_trial_position      mc_widom.h:122-213
//   gen_orientations  get_random_trial_orientation   mc_widom.h:215-303
//   trial_pass        Calculate_Multiple_Trial_Energy_VDWReal + host sums
//                     (VDW_Coulomb.cu:1183-1352, mc_widom.h:42-87)
//   step_weight       SelectTrialPosition + CBMC_FirstBead_Finish / chain finish
//                     (mc_widom.h:14-39, 305-383, 568-611)
//   ewald_move        Initialize_WaveVector_General + Fourier_Ewald_Diff
//                     (Ewald_Energy_Functions.h:162-185, 280-397)
#pragma once

#include "grx_ewcol.cuh"
#include "grx_warp.cuh"

namespace grx {

constexpr int kMaxTrials = 64;
constexpr int kMolWork = 32;      // atoms of one molecule held in shared memory
constexpr int kCbmcBeads = 128;   // trial beads of one pass
constexpr int kCbmcMaxMult = 8;   // items per warp of a bead pass, at most
constexpr int kEwRowBytes = 96 * 1024;  // largest (kx, ky) row-product table of a move
constexpr int kEwRowReuse = 16;         // active k per row at which the row products pay

// Entries of the row-product table of the double-float Ewald delta: one per (kx, ky) row and
// moved atom. The host enables it for a box (BoxDev::ew_rows) when the table for 2 * molsize
// atoms (a translation) fits kEwRowBytes and the box has at least kEwRowReuse active k per
// row, and sizes dynamic shared memory for it; the kernels read the flag.
__host__ __device__ __forceinline__ int ew_rows(const int* kmax) { return (kmax[0] + 1) * (2 * kmax[1] + 1); }
__host__ __device__ __forceinline__ bool ew_rows_worth(const int* kmax, int nact, int molsize) {
  return (size_t)ew_rows(kmax) * 2 * molsize * 16 <= (size_t)kEwRowBytes && nact >= kEwRowReuse * ew_rows(kmax);
}

// Workspace of a block of NW warps. A pass uses at most items + beads - 1 partial
// slots, items = mult * NW.
template <int NW>
struct CbmcWork {
  static constexpr int kItems = kCbmcBeads + kCbmcMaxMult * NW;
  Bead beads[kCbmcBeads];
  double ipart[kItems * 4];
  int iflag[kItems];
  int tdead[kCbmcBeads];  // per trial of a pass: early overlap rejection flag (-1: evaluated in full)
  alignas(16) int qbuf[NW * kQueue];  // the warps' pair queues; between passes the quaternions of gen_orientations
  double te[kMaxTrials * 4];
  int tflag[kMaxTrials];
  // moved atoms of the Ewald delta: [0, n_old) leave (charge stored negated),
  // [n_old, n_old + n_new) arrive
  double mx[2 * kMolWork], my[2 * kMolWork], mz[2 * kMolWork], mq[2 * kMolWork];
  double sbuf[32];
  double ewx[8][2];  // per-CTA Fourier partials {same, cross} of a cluster
  double wsum[2][NW];
  int counter;
  int staged;             // s_tmp holds the dS of a charged move: 1 not committed, 2 committed (0: none yet)
  long long cfg;    // trial configurations evaluated since the caller last cleared it
  long long cbeads; // their beads
  int ok;       // step constructed
  int big;      // and its weight (times that of the steps before it) above 1e-150
  int sel;      // chosen (or retraced) trial index
  int nok;      // trials without overlap
  double w;     // averaged weight of the step
};

// ---------------------------------------------------------------- trials
// First-bead trial positions: Cell diagonal x Philox uniforms (mc_widom.h:133-139);
// with `retrace`, trial 0 is the existing bead (deletion, mc_widom.h:141-156).
template <class WK>
__device__ __noinline__ void gen_first_trials(const BoxDev& b, WK& W, uint64_t seed, uint32_t stream,
                                                 uint64_t move, int nt, double q, double scale, int type,
                                                 bool retrace, double ox, double oy, double oz) {
  auto draw = [&](int t, uint32_t* r) { draw4_dev(seed, stream, move, SLOT_FIRST + t, r); };
  first_beads(b, W.beads, draw, nt, q, scale, type, retrace, ox, oy, oz);
  __syncthreads();
}

// Trial orientations about the chosen first bead (fx, fy, fz): the vectors from the
// component's slot-0 atom to its chain atoms, rotated by Philox quaternions. With
// `retrace`, orientation 0 is the existing chain (ox/oy/oz arrays, chain atoms).
template <int PREC, class WK>
__device__ __noinline__ void gen_orientations(const BoxDev& b, WK& W, uint64_t seed, uint32_t stream,
                                                 uint64_t move, int no, int chain, int off, double scale_coul,
                                                 double scale, double fx, double fy, double fz, bool retrace,
                                                 const double* ox, const double* oy, const double* oz,
                                                 uint32_t slot_base = SLOT_ORIENT) {
  static_assert(sizeof(W.qbuf) >= 2 * kMaxTrials * sizeof(float4), "quaternions in the pair queues");
  auto draw = [&](int o, uint32_t* r) { draw4_dev(seed, stream, move, slot_base + o, r); };
  orientation_beads<PREC>(b, W.beads, reinterpret_cast<float4*>(W.qbuf), draw, no, chain, off, scale_coul, scale, fx, fy,
                          fz, retrace, ox, oy, oz);
  __syncthreads();
}

// Energies of ntr = nb / chain trials of `chain` beads each (W.beads) against every
// atom, with the atoms of (comp, newmol) and of (excl_comp, excl_mol) excluded (the
// ExcludeList of an identity swap): W.te[4 t + k], W.tflag[t]. The first `early` trials
// (all of them when early < 0) stop at their first overlap (early overlap rejection):
// their flags are exact, their energies are not computed in full and must not be used
// when flagged, which is how every CBMC step treats a flagged trial.
// With CL > 1 the block is one CTA of a cluster that shares the chain: the pass is split
// over the cluster's warps (items per warp capped so the slots fit the workspace), each
// CTA copies its slots into its peers' workspaces, and every CTA reduces all slots. The
// second cluster barrier keeps a CTA from writing the next pass's slots into a peer that
// is still reducing this one.
template <int PREC, int CL, class WK>
__device__ __forceinline__ void trial_pass_body(const BoxDev& b, WK& W, int nb, int chain, int comp, int newmol,
                                                int excl_comp, int excl_mol, int early) {
  if (threadIdx.x == 0) {
    W.counter = 0;
    W.cfg += nb / chain;
    W.cbeads += nb;
  }
  for (int t = threadIdx.x; t < nb / chain; t += blockDim.x) W.tdead[t] = (early < 0 || t < early) ? 0 : -1;
  __syncthreads();
  const int nw = (int)(blockDim.x >> 5);
  if constexpr (CL == 1) {
    const PassSplit sp = pass_split(b, nb, nw, b.chunk_mult);
    block_bead_pass<PREC>(b, W.beads, nb, comp, newmol, excl_comp, excl_mol, W.qbuf, W.ipart, W.iflag, &W.counter, sp,
                          0, -1, chain, W.tdead);
    __syncthreads();
    reduce_items<PREC>(W.ipart, W.iflag, nb / chain, chain, sp, W.te, W.tflag);
    __syncthreads();
  } else {
    const PassSplit sp = pass_split(b, nb, nw * CL, max(1, min(b.chunk_mult, kCbmcMaxMult / CL)));
    const unsigned rank = cluster_rank();
    int i0, i1;
    cluster_items(sp, CL, rank, i0, i1);
    block_bead_pass<PREC>(b, W.beads, nb, comp, newmol, excl_comp, excl_mol, W.qbuf, W.ipart, W.iflag, &W.counter, sp,
                          i0, i1, chain, W.tdead);
    __syncthreads();
    if (sp.nu > 0 && i0 < i1) {  // this CTA's slots [s0, s0 + n): item + bead, increasing
      unsigned lo, hi;
      sp.range((unsigned)i0, lo, hi);
      const int s0 = i0 + (int)(lo / sp.nu);
      sp.range((unsigned)(i1 - 1), lo, hi);
      const int n = (i1 - 1) + (int)((hi - 1u) / sp.nu) - s0 + 1;
      const unsigned long long* src = reinterpret_cast<const unsigned long long*>(W.ipart);
      for (int k = threadIdx.x; k < (CL - 1) * n * 5; k += blockDim.x) {
        const int j = k / (n * 5), e = k - j * (n * 5);
        const unsigned peer = (unsigned)j + ((unsigned)j >= rank ? 1u : 0u);
        const int slot = s0 + e / 5, f = e % 5;
        if (f < 4) {
          cluster_map(reinterpret_cast<unsigned long long*>(W.ipart), peer)[slot * 4 + f] = src[slot * 4 + f];
        } else {
          cluster_map(W.iflag, peer)[slot] = W.iflag[slot];
        }
      }
    }
    cluster_sync_all();
    reduce_items<PREC>(W.ipart, W.iflag, nb / chain, chain, sp, W.te, W.tflag);
    __syncthreads();
    cluster_sync_all();
  }
}

template <int PREC, int CL = 1, class WK>
__device__ __noinline__ void trial_pass(const BoxDev& b, WK& W, int nb, int chain, int comp, int newmol,
                                          int early = -1) {
  trial_pass_body<PREC, CL>(b, W, nb, chain, comp, newmol, -1, -1, early);
}
// The same with a second excluded molecule (excl_comp, excl_mol).
template <int PREC, int CL = 1, class WK>
__device__ __noinline__ void trial_pass_excl(const BoxDev& b, WK& W, int nb, int chain, int comp, int newmol,
                                               int excl_comp, int excl_mol) {
  trial_pass_body<PREC, CL>(b, W, nb, chain, comp, newmol, excl_comp, excl_mol, -1);
}

// CBMC weight of one growth step (warp 0 computes, results in W.ok/big/sel/w/nok).
// Insertion: log-sum-exp selection with the uniform of word uw (SelectTrialPosition) and the
// 1e-150 failure test. Retrace (deletion): the first trial without overlap is the
// existing configuration and no selection is drawn. `stored` is added to the sum
// before averaging over 1 / inv trials (the reinsertion retrace's StoredR, mc_widom.h:363-366).
// chain: the weight of the steps before, multiplied by this one's. FP64 stays on warp 0: an FP64
// instruction takes 16 cycles of the SM per warp that issues it, whatever its lanes do.
template <class WK>
__device__ __noinline__ void step_weight(WK& W, int nt, double beta, int bias, uint32_t uw, double inv,
                                            bool retrace, double stored = 0.0, double* chain = nullptr) {
  if (threadIdx.x < 32) {
    StepChoice c = choose_trial(W.te, W.tflag, nt, beta, bias, u01(uw), retrace);
    if (c.w != c.w) c.w = plain_weights(W.te, W.tflag, nt, beta, bias, -1).x;
    if (threadIdx.x == 0) {
      W.nok = c.nok;
      W.ok = 0;
      W.big = 0;
      if (c.nok > 0) {
        if (retrace || !(c.w < 1e-150)) {
          double avg = (c.w + stored) * inv;
          if (!bias) avg *= exp_move(-beta * (W.te[4 * c.sel + 1] + W.te[4 * c.sel + 3]));
          W.ok = 1;
          W.sel = c.sel;
          W.w = avg;
          const double all = chain ? *chain * avg : avg;
          if (chain) *chain = all;
          W.big = chain ? !(all <= 1e-150) : all > 1e-150;  // apart for NaN: recorded when it is the chain's
        }
      }
    }
  }
  __syncthreads();
}

// ---------------------------------------------------------------- Ewald
// Fourier delta of the na moved atoms in W.mx/my/mz/mq (old atoms carry -q):
// dS(k) = sum q e^{ik.r}; same = sum temp (|S + dS|^2 - |S|^2), cross = sum temp
// Re(S_cross dS*), S_same = adsorbate block (guest moves), by columns of k (grx_ewcol.cuh). The
// FP64 form keeps the reference arithmetic; the other forms evaluate dS and both sums in
// double-float on the FP32 pipe against temp*S tables (ewA, ewF). In s_out (by slot) the FP64
// form stages S_same + dS, the others dS as float pairs, for a later commit. Results on thread 0.
// With CL > 1 each CTA of the cluster takes a contiguous range of the columns; the CTAs' partial
// sums are exchanged through distributed shared memory and added in rank order by every CTA, and
// the cluster barriers before a commit publish the staged S.
template <int PREC, class WK, bool ROWS = false, int CL = 1>
__device__ __noinline__ void ewald_move(const BoxDev& b, WK& W, int na, double2* eik, double2* s_out,
                                           double& same, double& cross) {
  const int tid = threadIdx.x;
  int c0 = 0, c1 = b.ncol;
  if constexpr (CL > 1) cluster_k_range(b.ncol, CL, cluster_rank(), c0, c1);
  eik_fill<PREC == GRX_FP64>(b, na, W.mx, W.my, W.mz, W.mq, eik, tid, blockDim.x);
  __syncthreads();
  same = 0.0;
  cross = 0.0;
  if constexpr (PREC == GRX_FP64) {
    EwSums64 e;
    ewald_columns(b, na, eik, c0 + tid, c1, blockDim.x, b.s_ads, b.s_fw, s_out, e);
    same = block_sum(e.same, W.sbuf);
    cross = block_sum(e.cross, W.sbuf);
  } else {
    const float4* fx = reinterpret_cast<const float4*>(eik);
    float4* rxy = nullptr;
    if constexpr (ROWS) {  // q X(kx) Y(ky) per (kx, ky) row and atom
      rxy = reinterpret_cast<float4*>(eik) + (b.kmax[0] + b.kmax[1] + b.kmax[2] + 3) * na;
      const float4* fy = fx + (b.kmax[0] + 1) * na;
      const int ny = 2 * b.kmax[1] + 1, nrow = ew_rows(b.kmax);
      for (int e = tid; e < nrow * na; e += blockDim.x) {
        const int row = e / na, at = e - row * na;
        const int kx = row / ny, ky = row - kx * ny - b.kmax[1];
        const float s = ky < 0 ? -1.f : 1.f;
        const float4 X = fx[at + na * kx], Y = fy[at + na * abs(ky)];
        const df xr = {X.x, X.y}, xi = {X.z, X.w};
        const df yr = {Y.x, Y.y}, yi = {s * Y.z, s * Y.w};
        const df pr = df_add(df_mul(xr, yr), df_mul(df{-xi.hi, -xi.lo}, yi));
        const df pi = df_add(df_mul(xr, yi), df_mul(xi, yr));
        rxy[e] = make_float4(pr.hi, pr.lo, pi.hi, pi.lo);
      }
      __syncthreads();
    }
    EwSumsDf e;
    ewald_columns<ROWS>(b, na, fx, rxy, c0 + tid, c1, blockDim.x, reinterpret_cast<float4*>(s_out), e);
    if (tid == 0) W.staged = 1;
    df sm = ew_same(e), cr = e.c;
    sm = warp_sum_df(sm);
    cr = warp_sum_df(cr);
    if ((tid & 31) == 0) { W.wsum[0][tid >> 5] = df_to(sm); W.wsum[1][tid >> 5] = df_to(cr); }
    __syncthreads();
    if (tid < 32) {  // one tree instead of a serial FP64 chain over the warps
      const bool in = tid < (int)(blockDim.x >> 5);
      same = warp_sum(in ? W.wsum[0][tid] : 0.0);
      cross = warp_sum(in ? W.wsum[1][tid] : 0.0);
    }
  }
  if constexpr (CL > 1) {
    const unsigned rank = cluster_rank();
    if (tid == 0)
      for (unsigned p = 0; p < (unsigned)CL; ++p) {
        double* dst = cluster_map(&W.ewx[0][0], p);
        dst[2 * rank] = same;
        dst[2 * rank + 1] = cross;
      }
    cluster_sync_all();
    if (tid < 32) {
      same = warp_sum(tid < CL ? W.ewx[tid][0] : 0.0);
      cross = warp_sum(tid < CL ? W.ewx[tid][1] : 0.0);
    }
  }
  __syncthreads();
}

// S + dS of one slot from a staged dS (FP64).
__device__ __forceinline__ double2 staged_sum(double2 v, float4 d) {
  return make_double2(v.x + (wide(d.x) + wide(d.y)), v.y + (wide(d.z) + wide(d.w)));
}

// Make the staged structure factor current and refresh its double-float table (in a
// cluster, the CTA's own range of k). staged: the workspace's mark of a staged dS.
template <int PREC, int CL = 1>
__device__ __noinline__ void commit_sk(const BoxDev& b, const double2* s_tmp, int* staged) {
  float4* ewA = const_cast<float4*>(b.ewA);
  int k0 = 0, k1 = b.nact;
  if constexpr (CL > 1) cluster_k_range(b.nact, CL, cluster_rank(), k0, k1);
  for (int j = k0 + threadIdx.x; j < k1; j += blockDim.x) {
    const int slot = b.kact[j].w;
    double2 v;
    if constexpr (PREC == GRX_FP64) v = s_tmp[slot];
    else v = staged_sum(b.s_ads[slot], reinterpret_cast<const float4*>(s_tmp)[slot]);
    b.s_ads[slot] = v;
    const double t = b.ktemp[j];
    const df ar = df_from(t * v.x), ai = df_from(t * v.y);
    ewA[j] = make_float4(ar.hi, ar.lo, ai.hi, ai.lo);
  }
  if (threadIdx.x == 0) *staged = 2;
  __syncthreads();
}

// After the last step: the staged vector as the box's callers know it, S of the last move evaluated
// (its S + dS when it was rejected). Called with the block (in a cluster, the cluster) synchronised.
template <int PREC, int CL>
__device__ __forceinline__ void settle_staged(const BoxDev& b, int staged) {
  if (PREC == GRX_FP64 || staged == 0) return;
  int k0 = 0, k1 = b.nact;
  if constexpr (CL > 1) cluster_k_range(b.nact, CL, cluster_rank(), k0, k1);
  for (int j = k0 + threadIdx.x; j < k1; j += blockDim.x) {
    const int slot = b.kact[j].w;
    const double2 v = b.s_ads[slot];
    b.s_tmp[slot] = staged == 2 ? v : staged_sum(v, reinterpret_cast<const float4*>(b.s_tmp)[slot]);
  }
}

// Write one atom into the box storage (all representations).
static __device__ __noinline__ void store_atom(const BoxDev& b, int idx, double x, double y, double z, double charge,
                                           double scale_coul, double scale, int type, int molid) {
  const double qe = charge * scale_coul;
  const_cast<double4*>(b.pos64)[idx] = make_double4(x, y, z, qe);
  float hx, lx, hy, ly, hz, lz;
  split_coord(x, hx, lx);
  split_coord(y, hy, ly);
  split_coord(z, hz, lz);
  const_cast<float4*>(b.hi)[idx] = make_float4(hx, hy, hz, (float)qe);
  const_cast<float4*>(b.lo)[idx] = make_float4(lx, ly, lz, (float)scale);
  const_cast<int2*>(b.meta)[idx] = make_int2(type, molid);
  const_cast<double*>(b.scale)[idx] = scale;
  const_cast<double*>(b.charge)[idx] = charge;
  const df q = df_from(qe);
  const_cast<float2*>(b.qdf)[idx] = make_float2(q.hi, q.lo);
}

}  // namespace grx
