// grx_widom.cu -- batched CBMC Widom insertions, fully on the device, and the
// stand-alone Rosenbluth selection entry point.
//
// One block per insertion (persistent grid-stride loop). Per insertion:
//   1. first-bead trial positions from Philox (get_random_trial_position),
//   2. pair energies of all trials against every atom (bead_pass),
//   3. Rosenbluth selection of the first bead (SelectTrialPosition),
//   4. trial orientations about the chosen bead (get_random_trial_orientation),
//   5. pair energies of the orientations, selection,
//   6. Ewald Fourier delta of the chosen molecule (Fourier_Ewald_Diff) and the
//      exclusion / tail factors of Insertion_Body (mc_swap_utilities.h:94-108).
#include <algorithm>
#include <cmath>
#include <vector>

#include "grx_ewcol.cuh"
#include "grx_host.h"
#include "grx_warp.cuh"

namespace grx {

constexpr int kMaxTrials = 64;
constexpr int kWidomItemsPerWarp = 1;  // work split of a bead pass (items per warp)

struct WidomArgs {
  int comp;
  int ntrials;
  int norient;
  int molsize;
  int newmol;
  int rigid;
  int charged;
  int pad_;
  double scale;
  double scale_coul;
  double beta;
  double tail;
  double excl;  // ExclusionIntra + ExclusionAtom of the component
  uint64_t seed;
  uint64_t first_move;
  int64_t n;
  uint32_t stream;
};

// choose_trial with the weights beyond the range of exp, out of line: the rare branch inlined into the
// kernel's two steps spilled registers of its body.
static __device__ __noinline__ StepChoice choose_step(const double* te, const int* tflag, int nt, double beta, int bias,
                                                      double u) {
  StepChoice c = choose_trial(te, tflag, nt, beta, bias, u, false);
  if (c.w != c.w) c.w = plain_weights(te, tflag, nt, beta, bias, -1).x;
  return c;
}

// Weight of one CBMC step by one warp (insertion branch); true when a trial was chosen.
__device__ bool select_trial_warp(const double* te, const int* tflag, int nt, double beta, int bias,
                                  double u, double navg, int& sel, double& wavg, int& nok) {
  const StepChoice c = choose_step(te, tflag, nt, beta, bias, u);
  nok = c.nok;
  if ((threadIdx.x & 31) != 0 || c.nok == 0 || c.w < 1e-150) return false;
  sel = c.sel;
  double avg = c.w / navg;
  if (!bias) avg *= exp(-beta * (te[4 * c.sel + 1] + te[4 * c.sel + 3]));
  wavg = avg;
  return true;
}

template <int PREC>
__global__ void __launch_bounds__(GRX_THREADS, 3) widom_kernel(BoxDev b, WidomArgs a, grx_widom_result* out) {
  __shared__ Bead beads[GRX_MAX_TRIAL_BEADS];
  __shared__ double ipart[kMaxItems * 4];
  __shared__ int iflag[kMaxItems];
  __shared__ alignas(16) int qbuf[(GRX_THREADS / 32) * kQueue];
  __shared__ int counter;
  __shared__ double te[kMaxTrials * 4];
  __shared__ int tflag[kMaxTrials];
  __shared__ int tdead[kMaxTrials];  // early overlap rejection flags of a pass's trials
  __shared__ double sbuf[32];
  __shared__ double newx[GRX_MAX_MOLSIZE], newy[GRX_MAX_MOLSIZE], newz[GRX_MAX_MOLSIZE], newq[GRX_MAX_MOLSIZE];
  __shared__ grx_widom_result res;
  __shared__ int s_ok;
  extern __shared__ double2 eik_s[];

  const int tid = threadIdx.x;
  const int off = b.comp_off[a.comp];
  const int ms = a.molsize, chain = ms - 1;
  for (int64_t m = blockIdx.x; m < a.n; m += gridDim.x) {
    const uint64_t move = a.first_move + (uint64_t)m;
    uint32_t selw[4];
    draw4(a.seed, a.stream, move, SLOT_SELECT, selw);
    if (tid == 0) {
      res = grx_widom_result{};
      res.sel_first = -1;
      res.sel_orient = -1;
      s_ok = 0;
      counter = 0;
    }
    // 1. first-bead trials (mc_widom.h:133-139)
    const int nt = a.ntrials;
    if (tid < nt) tdead[tid] = 0;
    auto draw_first = [&](int t, uint32_t* r) { draw4(a.seed, a.stream, move, SLOT_FIRST + t, r); };
    first_beads(b, beads, draw_first, nt, b.charge[off] * a.scale_coul, a.scale, b.meta[off].x, false, 0.0, 0.0, 0.0);
    __syncthreads();
    // 2. pair energies of the first-bead trials
    {
      const PassSplit sp = pass_split(b, nt, GRX_THREADS / 32, kWidomItemsPerWarp);
      block_bead_pass<PREC>(b, beads, nt, a.comp, a.newmol, -1, -1, qbuf, ipart, iflag, &counter, sp, 0, -1, 1,
                            tdead);
      __syncthreads();
      reduce_items<PREC>(ipart, iflag, nt, 1, sp, te, tflag);
      __syncthreads();
    }
    // 3. select the first bead
    if (tid < 32) {
      int sel = -1, nok = 0;
      double w = 0.0;
      const bool ok = select_trial_warp(te, tflag, nt, a.beta, b.vdw_real_bias, u01(selw[0]), (double)nt, sel, w,
                                        nok);
      if (tid == 0) res.n_ok_first = nok;
      if (ok && w > 1e-150) {
        s_ok = 1;
        res.sel_first = sel;
        res.w_first = w;
        res.rosenbluth = w;
        for (int q = 0; q < 4; ++q) res.e_first[q] = te[4 * sel + q];
        newx[0] = beads[sel].x; newy[0] = beads[sel].y; newz[0] = beads[sel].z;
        newq[0] = beads[sel].q;
      }
    }
    __syncthreads();
    if (s_ok && chain > 0) {
      // 4. orientations about the chosen first bead (mc_widom.h:255-276)
      const int no = a.norient, nb = no * chain;
      const double fx = newx[0], fy = newy[0], fz = newz[0];
      static_assert(sizeof(qbuf) >= 2 * kMaxTrials * sizeof(float4), "quaternions in the pair queues");
      auto draw = [&](int o, uint32_t* r) { draw4(a.seed, a.stream, move, SLOT_ORIENT + o, r); };
      orientation_beads<PREC>(b, beads, reinterpret_cast<float4*>(qbuf), draw, no, chain, off, a.scale_coul, a.scale, fx,
                              fy, fz, false, nullptr, nullptr, nullptr);
      if (tid == 0) counter = 0;
      if (tid < no) tdead[tid] = 0;
      __syncthreads();
      // 5. pair energies of the orientations
      const PassSplit sp = pass_split(b, nb, GRX_THREADS / 32, kWidomItemsPerWarp);
      block_bead_pass<PREC>(b, beads, nb, a.comp, a.newmol, -1, -1, qbuf, ipart, iflag, &counter, sp, 0, -1, chain,
                            tdead);
      __syncthreads();
      reduce_items<PREC>(ipart, iflag, no, chain, sp, te, tflag);
      __syncthreads();
      if (tid < 32) {
        int sel = -1, nok = 0;
        double w = 0.0;
        const bool ok = select_trial_warp(te, tflag, no, a.beta, b.vdw_real_bias, u01(selw[1]), (double)no, sel, w,
                                          nok);
        if (tid == 0) res.n_ok_orient = nok;
        if (tid == 0 && ok) {
          res.sel_orient = sel;
          res.w_chain = w;
          for (int q = 0; q < 4; ++q) res.e_chain[q] = te[4 * sel + q];
          res.rosenbluth *= w;
          if (res.rosenbluth <= 1e-150) s_ok = 0;
          for (int at = 0; at < chain; ++at) {
            const Bead& bd = beads[sel * chain + at];
            newx[1 + at] = bd.x; newy[1 + at] = bd.y; newz[1 + at] = bd.z; newq[1 + at] = bd.q;
          }
        } else if (tid == 0) {
          s_ok = 0;
        }
      }
      __syncthreads();
    }
    // 6. Ewald delta of the chosen molecule (insertion: no old atoms)
    if (s_ok && a.charged && !b.no_charges && b.nact > 0) {
      eik_fill<PREC == GRX_FP64>(b, ms, newx, newy, newz, newq, eik_s, tid, blockDim.x);
      __syncthreads();
      double same = 0.0, cross = 0.0;
      if constexpr (PREC == GRX_FP64) {
        EwSums64 e;
        ewald_columns(b, ms, eik_s, tid, b.ncol, blockDim.x, b.s_ads, b.s_fw, nullptr, e);
        same = block_sum(e.same, sbuf);
        cross = block_sum(e.cross, sbuf);
      } else {
        EwSumsDf e;
        ewald_columns<false>(b, ms, reinterpret_cast<const float4*>(eik_s), nullptr, tid, b.ncol, blockDim.x, nullptr, e);
        df sm = ew_same(e), cr = e.c;
        // block sums: warp tree in double-float, then FP64 over the 8 warp partials
        sm = warp_sum_df(sm);
        cr = warp_sum_df(cr);
        __shared__ double wsum[2][GRX_THREADS / 32];
        if ((tid & 31) == 0) { wsum[0][tid >> 5] = df_to(sm); wsum[1][tid >> 5] = df_to(cr); }
        __syncthreads();
        if (tid == 0) {
          for (int w = 0; w < GRX_THREADS / 32; ++w) { same += wsum[0][w]; cross += wsum[1][w]; }
        }
      }
      if (tid == 0) {
        if (a.rigid) same -= a.excl * (a.scale_coul * a.scale_coul - 0.0);
        res.ewald[0] = same;
        res.ewald[1] = 2.0 * cross;
        res.rosenbluth *= exp(-a.beta * (res.ewald[0] + res.ewald[1]));
      }
    }
    if (tid == 0) {
      if (s_ok) {
        res.rosenbluth *= exp(-a.beta * a.tail);
        res.success = 1;
      } else {
        res.rosenbluth = 0.0;
        res.success = 0;
      }
      out[m] = res;
    }
    __syncthreads();
  }
}

// temp * S(k) of both blocks in double-float, per active k (the box's static part of
// the Fourier delta: dE_same = sum 2 Re(A dS*) + temp |dS|^2, dE_cross = sum Re(F dS*)).
__global__ void ewald_df_refresh_kernel(BoxDev b, float4* ewA, float4* ewF, float2* ewT) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < b.nact; j += gridDim.x * blockDim.x) {
    const int slot = b.kact[j].w;
    const double t = b.ktemp[j];
    const double2 sa = b.s_ads[slot], sf = b.s_fw[slot];
    const df ar = df_from(t * sa.x), ai = df_from(t * sa.y), fr = df_from(t * sf.x), fi = df_from(t * sf.y);
    ewA[j] = make_float4(ar.hi, ar.lo, ai.hi, ai.lo);
    if (b.shared_host) continue;  // a replica's framework tables are its parent's
    ewF[j] = make_float4(fr.hi, fr.lo, fi.hi, fi.lo);
    const df tt = df_from(t);
    ewT[j] = make_float2(tt.hi, tt.lo);
  }
}

__global__ void select_kernel(const double* logw, int n, double u, int* sel, double* sum) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double mx = logw[0];
  for (int i = 1; i < n; ++i) mx = fmax(mx, logw[i]);
  double s = 0.0;
  for (int i = 0; i < n; ++i) s += exp(logw[i] - mx);
  const double ws = u * s;
  int k = 0;
  double cum = exp(logw[0] - mx);
  while (cum < ws && k + 1 < n) cum += exp(logw[++k] - mx);
  double w = 0.0;
  for (int i = 0; i < n; ++i) w += exp(logw[i]);
  *sel = k;
  *sum = w;
}

static grx_status widom_launch(grx_box* b, const grx_widom_desc* d, uint64_t first_move, size_t n,
                               grx_precision prec, grx_widom_result* dev_results) {
  GRX_REQUIRE(d->component >= b->nhost && d->component < b->ncomp,
              "grx_widom_insertions: component must be an adsorbate component");
  GRX_REQUIRE(d->ntrials >= 1 && d->ntrials <= kMaxTrials, "grx_widom_insertions: ntrials out of range (1..64)");
  const int ms = (int)b->molsize[d->component];
  GRX_REQUIRE(ms >= 1 && ms <= GRX_MAX_MOLSIZE, "grx_widom_insertions: molecule size out of range");
  if (ms > 1)
    GRX_REQUIRE(d->norient >= 1 && d->norient <= kMaxTrials && d->norient * (ms - 1) <= GRX_MAX_TRIAL_BEADS,
                "grx_widom_insertions: norient out of range");
  GRX_REQUIRE(prec == GRX_FP64 || prec == GRX_MIXED || prec == GRX_FP32, "grx_widom_insertions: bad precision");
  if (n == 0) return GRX_OK;
  refresh_dev(b);
  WidomArgs a{};
  a.comp = d->component;
  a.ntrials = d->ntrials;
  a.norient = ms > 1 ? d->norient : 0;
  a.molsize = ms;
  a.newmol = b->size[d->component] / ms;
  a.rigid = b->rigid[d->component];
  a.charged = b->has_charge[d->component];
  a.scale = d->scale;
  a.scale_coul = d->scale_coul;
  a.beta = d->beta;
  a.tail = d->tail_delta;
  a.excl = b->excl_intra[d->component] + b->excl_self[d->component];
  a.seed = d->seed;
  a.stream = d->stream;
  a.first_move = first_move;
  a.n = (int64_t)n;
  const size_t smem = (size_t)(b->dev.kmax[0] + b->dev.kmax[1] + b->dev.kmax[2] + 3) * ms * sizeof(double2);
  static_assert(sizeof(double2) == sizeof(float4), "eik entries of both forms");
  if (!b->ewdf_valid && b->nact > 0) {
    ewald_df_refresh_kernel<<<std::max(1, std::min((b->nact + 255) / 256, sm_count(b))), 256, 0, b->stream>>>(
        b->dev, b->ewA, b->ewF, b->ewT);
    count_launch();
    b->ewdf_valid = true;
  }
  const int grid = (int)std::min<size_t>(n, (size_t)sm_count(b) * 3);
  if (prec == GRX_FP64) widom_kernel<GRX_FP64><<<grid, GRX_THREADS, smem, b->stream>>>(b->dev, a, dev_results);
  else if (prec == GRX_MIXED) widom_kernel<GRX_MIXED><<<grid, GRX_THREADS, smem, b->stream>>>(b->dev, a, dev_results);
  else widom_kernel<GRX_FP32><<<grid, GRX_THREADS, smem, b->stream>>>(b->dev, a, dev_results);
  count_launch();
  GRX_CHECK_CUDA(cudaGetLastError(), "widom launch");
  return GRX_OK;
}

}  // namespace grx

using namespace grx;

extern "C" {

grx_status grx_widom_insertions_async(grx_box* b, const grx_widom_desc* d, uint64_t first_move, size_t n,
                                      grx_precision prec, grx_widom_result* results) {
  GRX_REQUIRE(b && d && (results || n == 0), "grx_widom_insertions_async: null argument");
  return widom_launch(b, d, first_move, n, prec, results);
}

grx_status grx_widom_insertions(grx_box* b, const grx_widom_desc* d, uint64_t first_move, size_t n,
                                grx_precision prec, grx_widom_result* results) {
  GRX_REQUIRE(b && d && (results || n == 0), "grx_widom_insertions: null argument");
  if (n == 0) return GRX_OK;
  grx_status st = ensure_results(b, n);
  if (st) return st;
  st = widom_launch(b, d, first_move, n, prec, b->d_results);
  if (st) return st;
  GRX_CHECK_CUDA(cudaMemcpyAsync(results, b->d_results, n * sizeof(grx_widom_result), cudaMemcpyDefault, b->stream),
                 "read widom results");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "widom insertions");
  return GRX_OK;
}

grx_status grx_cbmc_select(const double* logw, int32_t n, uint64_t seed, uint32_t stream, uint64_t move,
                           int32_t word, int32_t* selected, double* sum) {
  GRX_REQUIRE(logw && selected && sum && n >= 1 && n <= 4096 && word >= 0 && word < 4,
              "grx_cbmc_select: bad argument");
  uint32_t w[4];
  draw4(seed, stream, move, SLOT_SELECT, w);
  double* d_lw = nullptr;
  GRX_CHECK_CUDA(cudaMalloc(&d_lw, n * sizeof(double) + 2 * sizeof(double)), "select scratch");
  int* d_sel = (int*)(d_lw + n);
  double* d_sum = d_lw + n + 1;
  cudaError_t e = cudaMemcpy(d_lw, logw, n * sizeof(double), cudaMemcpyDefault);
  if (e == cudaSuccess) {
    select_kernel<<<1, 32>>>(d_lw, n, u01(w[word]), d_sel, d_sum);
    count_launch();
    e = cudaGetLastError();
  }
  int s = 0;
  double sm = 0.0;
  if (e == cudaSuccess) e = cudaMemcpy(&s, d_sel, sizeof(int), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(&sm, d_sum, sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d_lw);
  if (e != cudaSuccess) return cuda_status(e, "grx_cbmc_select");
  *selected = s;
  *sum = sm;
  return GRX_OK;
}

}  // extern "C"
