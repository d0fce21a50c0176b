// grx_pair.cu -- stand-alone pair-energy entry points: CBMC trial energies and the
// single-molecule move delta (the reference's per-move kernels, one call each). Both run
// trial_kernel (grx_warp.cuh); a move delta is two trials, the new molecule and the old one.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "grx_host.h"
#include "grx_warp.cuh"

namespace grx {

static void host_split(double x, float& h, float& l) {
  const double hd = std::nearbyint(x * GRX_GRID_COORD) / GRX_GRID_COORD;
  h = (float)hd;
  l = (float)(x - hd);
}

// The caller's bead arrays [0, nall) on the host.
struct HostBeads {
  std::vector<double> pos, scale, charge, scale_coul;
  std::vector<size_t> type;
};

static grx_status read_beads(const grx_trials* t, size_t nall, HostBeads& h) {
  h.pos.resize(3 * nall);
  h.scale.assign(nall, 1.0);
  h.charge.assign(nall, 0.0);
  h.scale_coul.assign(nall, 1.0);
  h.type.resize(nall);
  grx_status st = fetch(h.pos.data(), t->pos, 3 * nall * sizeof(double), "read bead pos");
  if (!st && t->scale) st = fetch(h.scale.data(), t->scale, nall * sizeof(double), "read bead scale");
  if (!st && t->charge) st = fetch(h.charge.data(), t->charge, nall * sizeof(double), "read bead charge");
  if (!st && t->scale_coul) st = fetch(h.scale_coul.data(), t->scale_coul, nall * sizeof(double), "read bead scaleCoul");
  if (!st) st = fetch(h.type.data(), t->type, nall * sizeof(size_t), "read bead type");
  return st;
}

static void make_beads(const HostBeads& h, size_t first, size_t n, double prefactor, Bead* out) {
  for (size_t k = 0; k < n; ++k) {
    const size_t j = first + k;
    Bead& bd = out[k];
    bd.x = h.pos[3 * j]; bd.y = h.pos[3 * j + 1]; bd.z = h.pos[3 * j + 2];
    host_split(bd.x, bd.h.x, bd.l.x);
    host_split(bd.y, bd.h.y, bd.l.y);
    host_split(bd.z, bd.h.z, bd.l.z);
    bd.q = h.charge[j] * h.scale_coul[j];
    bd.scale = h.scale[j];
    bd.type = (int)h.type[j];
    const double pq = prefactor * bd.q;
    const float ph = (float)pq;
    bd.pq = make_float2(ph, (float)(pq - (double)ph));
    bd.unit = bead_unit(bd.scale, bd.h);
  }
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
  HostBeads h;
  grx_status st = read_beads(t, t->ntrials * ch, h);
  if (st) return st;
  for (size_t t0 = 0; t0 < t->ntrials; t0 += per_chunk) {
    const size_t ntr = std::min(per_chunk, t->ntrials - t0);
    const int nb = (int)(ntr * ch);
    // the kernel reads the beads from and writes the sums to pinned host memory: one launch, no copies
    const size_t bead_bytes = nb * sizeof(Bead);
    st = ensure_pinned(b, bead_bytes + ntr * (4 * sizeof(double) + 1));
    if (st) return st;
    char* base = (char*)b->pinned;
    make_beads(h, t0 * ch, nb, b->dev.prefactor, (Bead*)base);
    TrialArgs a{};
    a.beads = (Bead*)base;
    a.chain = (int)ch;
    a.component = component;
    a.mol[0] = (int)t->molid;
    a.split = (int)ntr;
    a.excl_comp = (int)exclude_comp;
    a.excl_mol = (int)exclude_molid;
    a.out = (double*)(base + bead_bytes);
    a.over = (unsigned char*)(a.out + 4 * ntr);
    run_trials(b, a, (int)ntr, prec);
    GRX_CHECK_CUDA(cudaGetLastError(), "trial energy launch");
    GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "trial energies");
    std::memcpy(eo.data() + 4 * t0, a.out, ntr * 4 * sizeof(double));
    std::memcpy(fo.data() + t0, a.over, ntr);
  }
  st = deliver(out, eo.data(), t->ntrials * sizeof(grx_trial_energy), "write energies");
  if (!st) st = deliver(overlap, fo.data(), t->ntrials, "write flags");
  return st;
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
  HostBeads hn, ho;
  grx_status st = read_beads(new_mol, ms, hn);
  if (!st) st = read_beads(old_mol, ms, ho);
  const size_t bead_bytes = 2 * ms * sizeof(Bead);
  if (!st) st = ensure_pinned(b, bead_bytes + 8 * sizeof(double) + 8);
  if (st) return st;
  Bead* beads = (Bead*)b->pinned;
  // up to two trials, the new molecule and the old one, each without the atoms of its own molecule id.
  // Only what is asked for runs: the other side may hold anything (its types index the pair tables).
  const int nconf = (do_new ? 1 : 0) + (do_old ? 1 : 0);
  if (do_new) make_beads(hn, 0, ms, b->dev.prefactor, beads);
  if (do_old) make_beads(ho, 0, ms, b->dev.prefactor, beads + (nconf - 1) * ms);
  TrialArgs a{};
  a.beads = beads;
  a.chain = (int)ms;
  a.component = component;
  a.mol[0] = (int)(do_new ? new_mol->molid : old_mol->molid);
  a.mol[1] = (int)old_mol->molid;
  a.split = 1;
  a.excl_comp = -1;
  a.excl_mol = -1;
  a.out = (double*)((char*)b->pinned + bead_bytes);
  a.over = (unsigned char*)(a.out + 8);
  run_trials(b, a, nconf, prec == GRX_FP64 ? (int)GRX_FP64 : (prec == GRX_MIXED ? kMixed64 : (int)GRX_FP32));
  GRX_CHECK_CUDA(cudaGetLastError(), "single body launch");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "single body");
  const double* r = a.out;
  // HH / HG / GG by the atom's component and the moved one (mc_single_particle.h:142-170)
  double e[6] = {0, 0, 0, 0, 0, 0};
  const int host_slot = component < b->nhost ? 0 : 2;
  for (int q = 0; q < 4; ++q) {
    double d = 0.0;
    if (do_new) d += r[q];
    if (do_old) d -= r[4 * (nconf - 1) + q];
    e[host_slot + q] = d;
  }
  const int flag = do_new && a.over[0];
  st = deliver(out6, e, 6 * sizeof(double), "write energies");
  const uint8_t f8 = flag ? 1 : 0;
  if (!st) st = deliver(overlap, &f8, 1, "write flag");
  return st;
}

}  // extern "C"
