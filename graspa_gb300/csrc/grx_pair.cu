// grx_pair.cu -- stand-alone pair-energy entry points: CBMC trial energies and the
// single-molecule move delta (the reference's per-move kernels, one call each). Both run
// trial_kernel (grx_warp.cuh); a move delta is two trials, the new molecule and the old one.
#include <algorithm>
#include <cmath>
#include <vector>

#include "grx_host.h"
#include "grx_warp.cuh"

namespace grx {

static void host_split(double x, float& h, float& l) {
  const double hd = std::nearbyint(x * GRX_GRID_COORD) / GRX_GRID_COORD;
  h = (float)hd;
  l = (float)(x - hd);
}

static grx_status stage_beads(const grx_trials* t, size_t first_bead, size_t nbeads, double prefactor,
                              std::vector<Bead>& out) {
  const size_t nall = t->ntrials * t->chainsize;
  std::vector<double> pos(3 * nall), sc(nall, 1.0), q(nall, 0.0), scc(nall, 1.0);
  std::vector<size_t> ty(nall, 0);
  if (nall) {
    GRX_CHECK_CUDA(cudaMemcpy(pos.data(), t->pos, 3 * nall * sizeof(double), cudaMemcpyDefault), "read bead pos");
    if (t->scale) GRX_CHECK_CUDA(cudaMemcpy(sc.data(), t->scale, nall * sizeof(double), cudaMemcpyDefault), "read bead scale");
    if (t->charge) GRX_CHECK_CUDA(cudaMemcpy(q.data(), t->charge, nall * sizeof(double), cudaMemcpyDefault), "read bead charge");
    if (t->scale_coul) GRX_CHECK_CUDA(cudaMemcpy(scc.data(), t->scale_coul, nall * sizeof(double), cudaMemcpyDefault), "read bead scaleCoul");
    GRX_CHECK_CUDA(cudaMemcpy(ty.data(), t->type, nall * sizeof(size_t), cudaMemcpyDefault), "read bead type");
  }
  out.resize(nbeads);
  for (size_t k = 0; k < nbeads; ++k) {
    const size_t j = first_bead + k;
    Bead& bd = out[k];
    bd.x = pos[3 * j]; bd.y = pos[3 * j + 1]; bd.z = pos[3 * j + 2];
    host_split(bd.x, bd.h.x, bd.l.x);
    host_split(bd.y, bd.h.y, bd.l.y);
    host_split(bd.z, bd.h.z, bd.l.z);
    bd.q = q[j] * scc[j];
    bd.scale = sc[j];
    bd.type = (int)ty[j];
    const double pq = prefactor * bd.q;
    const float ph = (float)pq;
    bd.pq = make_float2(ph, (float)(pq - (double)ph));
    bd.unit = bead_unit(bd.scale, bd.h);
  }
  return GRX_OK;
}

static void run_trials(grx_box* b, const TrialArgs& a, int ntrials, int prec) {
  if (prec == GRX_FP64) launch_trials<GRX_FP64>(b->dev, a, ntrials, b->stream);
  else if (prec == GRX_MIXED) launch_trials<GRX_MIXED>(b->dev, a, ntrials, b->stream);
  else if (prec == kMixed64) launch_trials<kMixed64>(b->dev, a, ntrials, b->stream);
  else launch_trials<GRX_FP32>(b->dev, a, ntrials, b->stream);
  count_launch();
}

}  // namespace grx

using namespace grx;

extern "C" {

grx_status grx_trial_energies(grx_box* b, const grx_trials* t, int32_t component, int64_t exclude_comp,
                              int64_t exclude_molid, grx_precision prec, grx_trial_energy* out,
                              uint8_t* overlap) {
  GRX_REQUIRE(b && t && out && overlap, "grx_trial_energies: null argument");
  GRX_REQUIRE(t->chainsize >= 1 && t->chainsize <= GRX_MAX_TRIAL_BEADS,
              "grx_trial_energies: chainsize out of range");
  GRX_REQUIRE(t->ntrials == 0 || (t->pos && t->type), "grx_trial_energies: bead arrays missing");
  GRX_REQUIRE(prec == GRX_FP64 || prec == GRX_MIXED || prec == GRX_FP32, "grx_trial_energies: bad precision");
  GRX_REQUIRE(component >= 0 && component < b->ncomp, "grx_trial_energies: component out of range");
  if (t->ntrials == 0) return GRX_OK;
  refresh_dev(b);
  const size_t ch = t->chainsize;
  const size_t per_chunk = std::max<size_t>(1, GRX_MAX_TRIAL_BEADS / ch);
  std::vector<double> eo(4 * t->ntrials);
  std::vector<uint8_t> fo(t->ntrials);
  for (size_t t0 = 0; t0 < t->ntrials; t0 += per_chunk) {
    const size_t ntr = std::min(per_chunk, t->ntrials - t0);
    const int nb = (int)(ntr * ch);
    std::vector<Bead> beads;
    grx_status st = stage_beads(t, t0 * ch, nb, b->dev.prefactor, beads);
    if (st) return st;
    const size_t bead_bytes = (nb * sizeof(Bead) + 255) / 256 * 256;
    const size_t out_bytes = (ntr * 4 * sizeof(double) + 255) / 256 * 256;
    st = ensure_scratch(b, bead_bytes + out_bytes + ntr);
    if (st) return st;
    char* base = (char*)b->scratch;
    TrialArgs a{};
    a.beads = (Bead*)base;
    a.chain = (int)ch;
    a.component = component;
    a.mol[0] = (int)t->molid;
    a.split = (int)ntr;
    a.excl_comp = (int)exclude_comp;
    a.excl_mol = (int)exclude_molid;
    a.out = (double*)(base + bead_bytes);
    a.over = (unsigned char*)(base + bead_bytes + out_bytes);
    GRX_CHECK_CUDA(cudaMemcpyAsync(base, beads.data(), nb * sizeof(Bead), cudaMemcpyHostToDevice, b->stream), "upload beads");
    run_trials(b, a, (int)ntr, prec);
    GRX_CHECK_CUDA(cudaGetLastError(), "trial energy launch");
    GRX_CHECK_CUDA(cudaMemcpyAsync(eo.data() + 4 * t0, a.out, ntr * 4 * sizeof(double), cudaMemcpyDeviceToHost, b->stream), "read energies");
    GRX_CHECK_CUDA(cudaMemcpyAsync(fo.data() + t0, a.over, ntr, cudaMemcpyDeviceToHost, b->stream), "read flags");
    GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "trial energies");
  }
  GRX_CHECK_CUDA(cudaMemcpy(out, eo.data(), t->ntrials * sizeof(grx_trial_energy), cudaMemcpyDefault), "write energies");
  GRX_CHECK_CUDA(cudaMemcpy(overlap, fo.data(), t->ntrials, cudaMemcpyDefault), "write flags");
  return GRX_OK;
}

grx_status grx_single_body_energy(grx_box* b, const grx_trials* old_mol, const grx_trials* new_mol,
                                  int32_t component, int32_t do_new, int32_t do_old, grx_precision prec,
                                  double* out6, uint8_t* overlap) {
  GRX_REQUIRE(b && old_mol && new_mol && out6 && overlap, "grx_single_body_energy: null argument");
  GRX_REQUIRE(component >= 0 && component < b->ncomp, "grx_single_body_energy: component out of range");
  const size_t ms = new_mol->chainsize;
  GRX_REQUIRE(ms >= 1 && 2 * ms <= GRX_THREADS && old_mol->chainsize == ms,
              "grx_single_body_energy: molecule size out of range");
  GRX_REQUIRE(do_new || do_old, "grx_single_body_energy: nothing to do");
  refresh_dev(b);
  std::vector<Bead> nb_, ob_;
  grx_status st = stage_beads(new_mol, 0, ms, b->dev.prefactor, nb_);
  if (st) return st;
  st = stage_beads(old_mol, 0, ms, b->dev.prefactor, ob_);
  if (st) return st;
  nb_.insert(nb_.end(), ob_.begin(), ob_.end());
  const size_t bead_bytes = (2 * ms * sizeof(Bead) + 255) / 256 * 256;
  st = ensure_scratch(b, bead_bytes + 256);
  if (st) return st;
  // two trials: the new molecule and the old one, each without the atoms of its own molecule id
  TrialArgs a{};
  a.beads = (Bead*)b->scratch;
  a.chain = (int)ms;
  a.component = component;
  a.mol[0] = (int)new_mol->molid;
  a.mol[1] = (int)old_mol->molid;
  a.split = 1;
  a.excl_comp = -1;
  a.excl_mol = -1;
  a.out = (double*)((char*)b->scratch + bead_bytes);
  a.over = (unsigned char*)(a.out + 8);
  GRX_CHECK_CUDA(cudaMemcpyAsync(b->scratch, nb_.data(), 2 * ms * sizeof(Bead), cudaMemcpyHostToDevice, b->stream), "upload beads");
  run_trials(b, a, 2, prec == GRX_MIXED ? kMixed64 : (int)prec);
  GRX_CHECK_CUDA(cudaGetLastError(), "single body launch");
  struct { double e[8]; unsigned char over[8]; } r;
  GRX_CHECK_CUDA(cudaMemcpyAsync(&r, a.out, sizeof(r), cudaMemcpyDeviceToHost, b->stream), "read energies");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "single body");
  // HH / HG / GG by the atom's component and the moved one (mc_single_particle.h:142-170)
  double e[6] = {0, 0, 0, 0, 0, 0};
  const int host_slot = component < b->nhost ? 0 : 2;
  for (int q = 0; q < 4; ++q) {
    double d = 0.0;
    if (do_new) d += r.e[q];
    if (do_old) d -= r.e[4 + q];
    e[host_slot + q] = d;
  }
  const int flag = do_new && r.over[0];
  GRX_CHECK_CUDA(cudaMemcpy(out6, e, 6 * sizeof(double), cudaMemcpyDefault), "write energies");
  uint8_t f8 = flag ? 1 : 0;
  GRX_CHECK_CUDA(cudaMemcpy(overlap, &f8, 1, cudaMemcpyDefault), "write flag");
  return GRX_OK;
}

}  // extern "C"
