// grx_host.h -- host-side box object shared by the libgrx translation units.
#pragma once

#include <memory>
#include <vector>
#include <string>

#include "grx_internal.cuh"

namespace grx {
// Device copy of the FP64 tables of one (device, arena, alpha, range of g, range of h), shared by the
// boxes that use them and given back (to the arena, which costs the device no wait) with the last one.
struct Tables64 {
  int device = 0;
  grx_arena* arena = nullptr;
  double2* g = nullptr;  // g's pieces, h's behind them
  double2* h = nullptr;
  int g_base = 0, g_n = 0, h_base = 0, h_n = 0;
  ~Tables64();
};
}  // namespace grx

struct grx_box {
  grx::BoxDev dev{};
  grx_arena* arena = nullptr;  // device memory comes from here when set (else cudaMalloc)
  grx_box* parent = nullptr;   // a replica shares its parent's framework atoms, tiles and tables
  int replicas = 0;            // live replicas of this box
  cudaStream_t stream = nullptr;
  int device = 0;
  int num_sms = 0;

  // layout
  int ncomp = 0, nhost = 0;
  size_t cap[GRX_MAX_COMPONENTS] = {};
  size_t molsize[GRX_MAX_COMPONENTS] = {};
  size_t off[GRX_MAX_COMPONENTS + 1] = {};
  int size[GRX_MAX_COMPONENTS] = {};
  int rigid[GRX_MAX_COMPONENTS] = {};
  int has_charge[GRX_MAX_COMPONENTS] = {};
  int many_mols[GRX_MAX_COMPONENTS] = {};  // host components: live atoms of more than one molecule id
  size_t stored[GRX_MAX_COMPONENTS] = {};  // atoms written to storage (template included)
  double excl_intra[GRX_MAX_COMPONENTS] = {};
  double excl_self[GRX_MAX_COMPONENTS] = {};
  size_t total_cap = 0;

  // host mirrors (FP64) of the component data, for exclusion constants
  std::vector<double> h_pos, h_charge, h_scale_coul;

  // device allocations
  double4* pos64 = nullptr;
  float4* hi = nullptr;
  float4* lo = nullptr;
  int2* meta = nullptr;
  double* scale = nullptr;
  double* charge = nullptr;
  int* d_size = nullptr;
  grx::FFPair64* ff64 = nullptr;
  double* ffc10 = nullptr;
  float4* ff32 = nullptr;
  int4* kact = nullptr;
  double* ktemp = nullptr;
  double2* s_fw = nullptr;
  double2* s_ads = nullptr;
  double2* s_tmp = nullptr;
  int nvec = 0, nact = 0;
  grx::KRow* krow = nullptr;   // (kx, ky) rows of the active k, and groups of rows for sk_kernel
  int2* kgroup = nullptr;
  int n_kgroups = 0;
  int4* kcol = nullptr;        // columns (kx, ky, |kz|) of the active k
  int ncol = 0;
  std::vector<int4> h_kcol;
  std::vector<grx::KRow> h_krow;
  std::vector<int2> h_kgroup;
  std::vector<int4> h_kact;
  std::vector<double> h_ktemp;
  bool sk_valid = false;

  // spatial tiles of host atoms and the storage permutation of host components
  std::vector<float4> h_tile_c;
  std::vector<int4> h_tile_r;
  float4* tile_c = nullptr;
  int4* tile_r = nullptr;
  size_t tile_cap = 0;
  int ntiles = 0;
  std::vector<int> perm[GRX_MAX_COMPONENTS];  // storage slot -> caller index
  // candidate lists of host atoms per voxel (grx_voxel.cu); a replica uses its parent's
  int vox_mode = 1;          // 1: build them when they fit, 0: tile path only
  size_t vox_max_bytes = 32u << 20;  // byte cap of the lists (coarser voxels to stay below it)
  double sigma_max = 0.0;    // largest sigma of the type pairs (0: 12-6-4 tables)
  int vox_on = 0;            // 0 no lists, 1 entries with their image, 2 images by rounded fractions
  int vn[3] = {0, 0, 0};
  int vchunks = 0;
  size_t vox_entries = 0;
  int4* vmeta = nullptr;
  uint32_t* vlist = nullptr;
  // double-float copies for the mixed-precision pair path
  float2* qdf = nullptr;     // q * scaleCoul per atom as hi/lo floats
  // host (framework) atoms [0, off[nhost]) as the pair engine reads them: two float4 per atom,
  // {x_hi, y_hi, z_hi, q_hi} {x_lo, y_lo, z_lo, q_lo}, and the type with bit 15 set when the
  // atom's scale is not 1 (replicas use the parent's)
  float4* hrec = nullptr;
  uint16_t* htype = nullptr;
  float4* ffdf = nullptr;    // per type pair {4eps hi, lo, 1/sigma^2 hi, lo}
  float2* ffdf2 = nullptr;   // per type pair {shift hi, lo}
  float4* ctabf = nullptr;   // Coulomb table, 2 float4 per piece
  float4* ewA = nullptr;     // per active k: temp * S_ads as double-float complex
  float4* ewF = nullptr;     // per active k: temp * S_fw
  float2* ewT = nullptr;     // per active k: temp
  bool ewdf_valid = false;
  int ctab_n = 0, ctab_base = 0;
  std::shared_ptr<const grx::Tables64> t64;  // FP64 Coulomb tables, shared by boxes of equal parameters

  // scratch (grown on demand)
  double* scratch = nullptr;
  size_t scratch_bytes = 0;
  void* pinned = nullptr;
  size_t pinned_bytes = 0;
  grx_widom_result* d_results = nullptr;
  size_t results_cap = 0;
};

namespace grx {
grx_status ensure_scratch(grx_box* b, size_t bytes);
grx_status ensure_pinned(grx_box* b, size_t bytes);
grx_status ensure_results(grx_box* b, size_t n);
// Between a caller's array and host memory of ours: plain host memory by memcpy, anything the
// CUDA runtime knows (device, managed, pinned) through it.
grx_status fetch(void* dst, const void* src, size_t bytes, const char* what);
grx_status deliver(void* dst, const void* src, size_t bytes, const char* what);
// A cudaMemcpy from pageable memory may return with its last part still on the way to the device, and
// a non-blocking stream is not ordered behind the default stream that carries it: what uploads this
// way ends with this wait, since the calls that follow start their kernels with no copy before them.
cudaError_t uploads_done();
void refresh_dev(grx_box* b);
int sm_count(grx_box* b);
void* arena_alloc(grx_arena* a, size_t bytes);
void arena_free(grx_arena* a, void* p);
// Device allocation of a box: from its arena when it has one, else cudaMalloc.
cudaError_t dev_alloc(grx_box* b, void** p, size_t bytes);
// Builds the double-float S(k) tables of a box on its stream (framework tables skipped
// for replicas) and marks them valid.
grx_status ewald_df_refresh(grx_box* b);
void dev_free(grx_box* b, void* p);
// The FP64 Coulomb tables of the box (grx_table.cu). In an arena they are part of the box
// (tables64_bytes of its footprint); elsewhere, without device memory for them, the box runs on the
// library functions.
grx_status attach_tables64(grx_box* b, double alpha, double cut2, const double* cell);
size_t tables64_bytes(double alpha, double cut2, const double* cell);
// Voxel candidate lists of the machine's host atoms (grx_voxel.cu), rebuilt after the tiles.
grx_status build_voxels(grx_box* b);
}  // namespace grx

#define GRX_CHECK_CUDA(call, what)                                    \
  do {                                                                \
    cudaError_t e_ = (call);                                          \
    if (e_ != cudaSuccess) return grx::cuda_status(e_, what);         \
  } while (0)

#define GRX_REQUIRE(cond, msg)                                        \
  do {                                                                \
    if (!(cond)) {                                                    \
      grx::set_error("%s", msg);                                      \
      return GRX_ERR_INVALID_ARG;                                     \
    }                                                                 \
  } while (0)
