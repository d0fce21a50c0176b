// grx_voxel.cu -- candidate lists of framework (host) atoms per voxel of the cell.
//
// The cell is cut into nv[0] x nv[1] x nv[2] voxels, parallelepipeds in fractional
// coordinates with edges near g angstrom. A voxel's list holds every host atom whose
// nearest periodic image lies within r_list = (screening radius) + (voxel bounding
// radius) + margin of the voxel centre, with the lattice shift of that image. For any
// bead inside the voxel the list therefore holds every atom within the cutoff, at the
// image the bead sees it (the cell is wider than 2 r_list, so that image is unique).
// Atoms whose image lies within (screening radius - bounding radius) of the centre are
// inside the cutoff for every bead of the voxel: they come first in the list and go to
// the dense evaluation without the FP32 screen, the ones near the centre (1.1 sigma from some
// bead of the voxel) ahead of the rest: the pairs that take the out-of-line LJ then share a batch
// or two instead of falling into half of them, and an overlap shows at once. The others are
// screened with the stored shift. A bead pass walks its voxel's list in 32-atom chunks instead of culling the
// box's 32-atom tiles; the dense evaluation still applies the exact cutoff tests, so the
// lists change which pairs are screened, never which pairs count.
//
// A cell narrower than 2 r_list (or host atoms stored cells away from the home cell) has no such
// unique image. Its lists (mode 2) hold an atom once, whenever the image that rounded fractions pick for
// some bead of the voxel may lie within the screening radius; "sure" atoms are those whose picked
// image is the same for every bead of the voxel and inside the cutoff, and the others are
// screened with the rounded fractions, as the tile path does.
//
// Entry: bits 0-19 the atom's storage index, bits 20-28 the shift (nx + 4) | (ny + 4) << 3
// | (nz + 4) << 6, n in [-4, 3], the image being r - nx a - ny b - nz c. Lists are built on
// the device when the host atoms change (a warp per voxel counts, the host sums, the warp writes;
// host threads took 10 to 20 ms a box), and shared with the box's replicas.
#include <algorithm>
#include <cmath>
#include <vector>

#include "grx_host.h"

namespace grx {

namespace {

struct Geo {
  double inv[9], w[3];
};

constexpr double kMargin = 0.02;                  // A, on the voxel bounding radius
constexpr double kTieMargin = 1e-3;               // fractional, on a voxel's half extent (mode 2)
constexpr size_t kArenaHeadroom = 4u << 20;       // arena bytes left free for the box's other buffers

}  // namespace

// Voxel grid of a cell: the finest edge g in {1.5, 2, 2.5, 3, 4} A whose lists fit the byte
// cap max_bytes (estimated from the host-atom density). unique: only grids that leave the cell wider
// than 2 r_list. Returns false when none does.
static bool choose_voxels(const double* C, double volume, int nh_atoms, double r_screen, size_t max_bytes, bool unique,
                          Geo& G, double& half_wmin, int nv[3], double& h, double& est_bytes) {
  const double av[3] = {C[0], C[1], C[2]}, bv[3] = {C[3], C[4], C[5]}, cv[3] = {C[6], C[7], C[8]};
  auto cross_norm = [](const double* u, const double* v) {
    const double x = u[1] * v[2] - u[2] * v[1], y = u[2] * v[0] - u[0] * v[2], z = u[0] * v[1] - u[1] * v[0];
    return std::sqrt(x * x + y * y + z * z);
  };
  const double V = std::fabs(volume);
  G.w[0] = V / cross_norm(bv, cv);
  G.w[1] = V / cross_norm(cv, av);
  G.w[2] = V / cross_norm(av, bv);
  half_wmin = 0.5 * std::min(G.w[0], std::min(G.w[1], G.w[2]));
  const double len[3] = {std::sqrt(av[0] * av[0] + av[1] * av[1] + av[2] * av[2]),
                         std::sqrt(bv[0] * bv[0] + bv[1] * bv[1] + bv[2] * bv[2]),
                         std::sqrt(cv[0] * cv[0] + cv[1] * cv[1] + cv[2] * cv[2])};
  const double dens = (double)nh_atoms / V;
  for (double g : {1.5, 2.0, 2.5, 3.0, 4.0}) {
    int n[3];
    for (int k = 0; k < 3; ++k) n[k] = std::max(1, (int)std::ceil(len[k] / g));
    double hm = 0.0;  // half the longest body diagonal of a voxel
    for (int sy = -1; sy <= 1; sy += 2)
      for (int sz = -1; sz <= 1; sz += 2) {
        double x[3];
        for (int j = 0; j < 3; ++j) x[j] = av[j] / n[0] + sy * bv[j] / n[1] + sz * cv[j] / n[2];
        hm = std::max(hm, 0.5 * std::sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]));
      }
    hm += kMargin;
    if (unique && r_screen + hm + kMargin >= half_wmin) return false;  // coarser voxels only make the bound worse
    const double rl = r_screen + hm;
    const double per = unique ? dens * 4.18879 * rl * rl * rl * 1.25 : std::min((double)nh_atoms, dens * 4.18879 * rl * rl * rl * 1.5);
    const double est = (double)n[0] * n[1] * n[2] * (per + 32.0) * 4.0 +
                       (double)n[0] * n[1] * n[2] * 16.0;
    if (est <= (double)max_bytes) {
      for (int k = 0; k < 3; ++k) nv[k] = n[k];
      h = hm;
      est_bytes = est;
      return true;
    }
  }
  return false;
}

struct VoxelScan {
  int mode;
  int nv[3];
  float tie[3];  // mode 2: |fraction| of the centre above which the voxel reaches across the tie
  float r_list, r_sure, r_near;
};

constexpr int kVoxelWarps = 8;

// One warp per voxel walks the framework atoms in storage order, one per lane. Without `list` it
// counts: meta {0, sure, all, near}. With it, meta holds the first entry too, and the warp
// writes the groups near, sure and the rest behind each other. FP32 on the hi parts: its errors
// (1e-3 A and 1e-5 of a fraction) stay inside the margins of the radii and of the ties.
__global__ void __launch_bounds__(32 * kVoxelWarps) voxel_scan_kernel(const __grid_constant__ BoxDev b,
                                                                      const __grid_constant__ VoxelScan p, int4* meta,
                                                                      unsigned* list) {
  const int v = blockIdx.x * kVoxelWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (v >= p.nv[0] * p.nv[1] * p.nv[2]) return;
  const unsigned lt = (1u << lane) - 1u;
  const float fx = ((v % p.nv[0]) + 0.5f) / p.nv[0], fy = ((v / p.nv[0] % p.nv[1]) + 0.5f) / p.nv[1],
              fz = ((v / (p.nv[0] * p.nv[1])) + 0.5f) / p.nv[2];
  const float cx = b.cellf[0] * fx + b.cellf[3] * fy + b.cellf[6] * fz;
  const float cy = b.cellf[1] * fx + b.cellf[4] * fy + b.cellf[7] * fz;
  const float cz = b.cellf[2] * fx + b.cellf[5] * fy + b.cellf[8] * fz;
  const int4 m = list ? meta[v] : make_int4(0, 0, 0, 0);
  int at[3] = {m.x, m.x + m.w, m.x + m.y};  // next entry of near, sure, the rest
  int n[3] = {0, 0, 0};
  for (int c = 0; c < b.nhost; ++c) {
    const int end = b.comp_off[c] + b.comp_size[c];
    for (int i0 = b.comp_off[c]; i0 < end; i0 += 32) {
      const int i = i0 + lane;
      int group = -1;
      unsigned code = 4u | 4u << 3 | 4u << 6;
      if (i < end) {
        const float4 a = b.hhi[i];
        const float x = a.x - cx, y = a.y - cy, z = a.z - cz;
        float sx = b.invf[0] * x + b.invf[3] * y + b.invf[6] * z;
        float sy = b.invf[1] * x + b.invf[4] * y + b.invf[7] * z;
        float sz = b.invf[2] * x + b.invf[5] * y + b.invf[8] * z;
        const float nx = rintf(sx), ny = rintf(sy), nz = rintf(sz);
        sx -= nx; sy -= ny; sz -= nz;
        auto norm2 = [&](float u, float w, float t) {
          const float dx = b.cellf[0] * u + b.cellf[3] * w + b.cellf[6] * t;
          const float dy = b.cellf[1] * u + b.cellf[4] * w + b.cellf[7] * t;
          const float dz = b.cellf[2] * u + b.cellf[5] * w + b.cellf[8] * t;
          return dx * dx + dy * dy + dz * dz;
        };
        float r2 = norm2(sx, sy, sz);
        bool one = true;
        if (p.mode == 1) {
          code = (unsigned)((int)nx + 4) | (unsigned)((int)ny + 4) << 3 | (unsigned)((int)nz + 4) << 6;
        } else {  // the images that rounded fractions may pick for a bead of the voxel
          const bool tx = fabsf(sx) > p.tie[0], ty = fabsf(sy) > p.tie[1], tz = fabsf(sz) > p.tie[2];
          one = !(tx || ty || tz);
          const float ux = sx - copysignf(1.0f, sx), uy = sy - copysignf(1.0f, sy), uz = sz - copysignf(1.0f, sz);
          for (int k = 1; k < 8 && !one; ++k) {
            if ((k & 1 && !tx) || (k & 2 && !ty) || (k & 4 && !tz)) continue;
            r2 = fminf(r2, norm2(k & 1 ? ux : sx, k & 2 ? uy : sy, k & 4 ? uz : sz));
          }
        }
        if (r2 <= p.r_list * p.r_list) {
          const bool sure = one && p.r_sure > 0.0f && r2 <= p.r_sure * p.r_sure;
          group = !sure ? 2 : (p.r_near > 0.0f && r2 <= p.r_near * p.r_near ? 0 : 1);
        }
      }
#pragma unroll
      for (int g = 0; g < 3; ++g) {
        const unsigned k = __ballot_sync(0xffffffffu, group == g);
        if (list && group == g) list[at[g] + __popc(k & lt)] = (unsigned)i | code << 20;
        at[g] += __popc(k);
        n[g] += __popc(k);
      }
    }
  }
  if (!list && lane == 0) meta[v] = make_int4(0, n[0] + n[1], n[0] + n[1] + n[2], n[0]);
}

grx_status build_voxels(grx_box* b) {
  dev_free(b, b->vmeta);
  dev_free(b, b->vlist);
  b->vmeta = nullptr;
  b->vlist = nullptr;
  b->vox_on = 0;
  b->vchunks = 0;
  b->vox_entries = 0;
  const int nh_atoms = (int)b->off[b->nhost];
  if (b->vox_mode == 0 || b->nhost == 0 || nh_atoms == 0 || b->ntiles == 0 || nh_atoms >= (1 << 20)) {
    refresh_dev(b);
    return GRX_OK;
  }
  const BoxDev& d = b->dev;
  Geo G;
  for (int k = 0; k < 9; ++k) G.inv[k] = d.inv[k];
  const double* C = d.cell;
  const double r_screen = std::sqrt((double)d.screen2);
  int nv[3] = {0, 0, 0};
  double h = 0.0, half_wmin = 0.0, est = 0.0;
  // host atoms must lie within four cells of the home cell for the 3-bit shifts of mode 1
  bool near_home = true;
  for (int i = 0; i < nh_atoms; ++i)
    for (int k = 0; k < 3; ++k) {
      const double f = G.inv[k] * b->h_pos[3 * i] + G.inv[3 + k] * b->h_pos[3 * i + 1] + G.inv[6 + k] * b->h_pos[3 * i + 2];
      if (!(f >= -2.5 && f <= 2.5)) near_home = false;
      // coordinates that the hi parts do not hold exactly: the tile path serves the box
      if (!(std::fabs(b->h_pos[3 * i + k]) < (double)kNearCoord)) {
        refresh_dev(b);
        return GRX_OK;
      }
    }
  int mode = 0;
  if (near_home && choose_voxels(C, d.volume, nh_atoms, r_screen, b->vox_max_bytes, true, G, half_wmin, nv, h, est)) mode = 1;
  // not in an arena: its users size it by the footprints of their boxes, and such cells have never
  // taken lists on top of theirs
  else if (!b->arena &&
           choose_voxels(C, d.volume, nh_atoms, r_screen, b->vox_max_bytes, false, G, half_wmin, nv, h, est))
    mode = 2;
  if (!mode) {
    refresh_dev(b);
    return GRX_OK;
  }
  VoxelScan v{};
  v.mode = mode;
  for (int k = 0; k < 3; ++k) {
    v.nv[k] = nv[k];
    v.tie[k] = (float)(0.5 - (0.5 / nv[k] + kTieMargin));
  }
  v.r_list = (float)(r_screen + h);
  v.r_sure = (float)(r_screen - 2e-3 - h);  // inside the largest cutoff for every bead of the voxel
  v.r_near = (float)std::min((double)v.r_sure, 1.1 * b->sigma_max + h);
  const int nvox = nv[0] * nv[1] * nv[2];
  const int grid = (nvox + kVoxelWarps - 1) / kVoxelWarps;
  std::vector<int4> meta(nvox);
  grx_status st = ensure_scratch(b, nvox * sizeof(int4));
  if (st) {  // no room to count: the tile path serves the box
    refresh_dev(b);
    return GRX_OK;
  }
  int4* counts = (int4*)b->scratch;
  voxel_scan_kernel<<<grid, 32 * kVoxelWarps, 0, b->stream>>>(b->dev, v, counts, nullptr);
  count_launch();
  GRX_CHECK_CUDA(cudaGetLastError(), "voxel count launch");
  GRX_CHECK_CUDA(cudaMemcpyAsync(meta.data(), counts, nvox * sizeof(int4), cudaMemcpyDeviceToHost, b->stream),
                 "read voxel counts");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "voxel counts");
  size_t total = 0;
  int maxn = 0;
  for (int k = 0; k < nvox; ++k) {  // {first entry, sure, all, near}
    meta[k].x = (int)total;
    total += (size_t)meta[k].z;
    maxn = std::max(maxn, meta[k].z);
  }
  const size_t list_bytes = std::max<size_t>(total, 1) * sizeof(uint32_t);
  // the lattice vectors of the 512 shift codes follow the voxel records
  meta.resize(nvox + 512);
  static_assert(sizeof(int4) == sizeof(float4), "shift vectors share the voxel records' allocation");
  float4* shift = reinterpret_cast<float4*>(meta.data() + nvox);
  for (int c = 0; c < 512; ++c) {
    const double n[3] = {(c & 7) - 4.0, ((c >> 3) & 7) - 4.0, (c >> 6) - 4.0};
    float v[3];
    for (int k = 0; k < 3; ++k) v[k] = (float)(n[0] * d.cell[k] + n[1] * d.cell[3 + k] + n[2] * d.cell[6 + k]);
    shift[c] = make_float4(v[0], v[1], v[2], 0.0f);
  }
  if (b->arena) {  // in an arena the lists are optional: take them only with room to spare
    size_t used = 0, largest = 0;
    grx_arena_usage(b->arena, &used, &largest, nullptr);
    if (largest < meta.size() * sizeof(int4) + list_bytes + kArenaHeadroom) {
      refresh_dev(b);
      return GRX_OK;
    }
  }
  if (dev_alloc(b, (void**)&b->vmeta, meta.size() * sizeof(int4)) != cudaSuccess ||
      dev_alloc(b, (void**)&b->vlist, list_bytes) != cudaSuccess) {
    cudaGetLastError();  // no room: the tile path serves the box
    dev_free(b, b->vmeta);
    dev_free(b, b->vlist);
    b->vmeta = nullptr;
    b->vlist = nullptr;
    refresh_dev(b);
    return GRX_OK;
  }
  // on the box's stream: the kernel takes its write offsets from these records
  GRX_CHECK_CUDA(cudaMemcpyAsync(b->vmeta, meta.data(), meta.size() * sizeof(int4), cudaMemcpyHostToDevice, b->stream),
                 "upload voxels");
  voxel_scan_kernel<<<grid, 32 * kVoxelWarps, 0, b->stream>>>(b->dev, v, b->vmeta, b->vlist);
  count_launch();
  GRX_CHECK_CUDA(cudaGetLastError(), "voxel list launch");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "voxel lists");
  for (int k = 0; k < 3; ++k) b->vn[k] = nv[k];
  b->vchunks = (maxn + 31) / 32;
  b->vox_on = mode;
  b->vox_entries = total;
  refresh_dev(b);
  return GRX_OK;
}

}  // namespace grx

using namespace grx;

extern "C" grx_status grx_box_set_voxel_lists(grx_box* b, int32_t mode) {
  GRX_REQUIRE(b, "grx_box_set_voxel_lists: null box");
  GRX_REQUIRE(mode == 0 || mode == 1, "grx_box_set_voxel_lists: mode must be 0 or 1");
  GRX_REQUIRE(!b->parent && b->replicas == 0,
              "grx_box_set_voxel_lists: the lists are shared with replicas (set them on a box without any)");
  GRX_CHECK_CUDA(cudaStreamSynchronize(b->stream), "grx_box_set_voxel_lists");
  b->vox_mode = mode;
  return build_voxels(b);
}

extern "C" grx_status grx_box_get_voxel_lists(grx_box* b, int32_t* on, int32_t* dims, int64_t* entries) {
  GRX_REQUIRE(b && on, "grx_box_get_voxel_lists: null argument");
  const grx_box* h = b->parent ? b->parent : b;
  *on = h->vox_on ? 1 : 0;
  if (dims)
    for (int k = 0; k < 3; ++k) dims[k] = h->vox_on ? h->vn[k] : 0;
  if (entries) *entries = h->vox_on ? (int64_t)h->vox_entries : 0;
  return GRX_OK;
}
