// grx_table.cu -- FP64 tables of the real-space Coulomb functions
//   g(s) = erfc(alpha sqrt s) / sqrt s   (pairs inside the cutoff)
//   h(s) = erf(alpha sqrt s) / sqrt s    (intramolecular exclusions, any image distance)
// as piecewise quintics in s = r^2: 512 (g) or 256 (h) pieces per octave, indexed by the high
// word of the FP64 s, expanded about the piece's centre. An evaluation is one FP64 subtraction and five
// FMAs instead of a square root, an erfc and a division (about 80 FP64 operations, which the
// two FP64 lanes of an SM per clock make the whole cost of an FP64 pair).
//
// Both functions satisfy s f' = -f/2 -+ (alpha/sqrt pi) exp(-alpha^2 s), which gives every
// Taylor coefficient at the centre from f and the exponential. The sixth-order term is folded
// into the lower ones with the Chebyshev polynomial T6, so that truncation stays below a
// rounding of f: 0.23 (1/512)^6 / 32 at short range, (alpha^2 s / 1024)^6 / 720 / 32 in the
// Gaussian tail of g, which is why g has the finer pieces. The centre value is formed with the
// rounding error of the argument taken out, so an evaluation carries about one rounding where
// erfc(alpha sqrt s) / sqrt s amplifies that of alpha sqrt s by 2 alpha^2 s. Against 80-bit
// values over 0.26 A^2 to the cutoff (alpha 0.265, 12 A): rms 1.0e-16, library form 4.5e-16.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <utility>
#include <vector>

#include "grx_host.h"

namespace grx {

namespace {

constexpr double kTableMin = 0.25;  // A^2: shorter distances take the library functions

int32_t high_word(double x) {
  int64_t bits;
  std::memcpy(&bits, &x, 8);
  return (int32_t)(bits >> 32);
}

double from_high_word(int32_t h) {
  const int64_t bits = (int64_t)h << 32;
  double x;
  std::memcpy(&x, &bits, 8);
  return x;
}

// Value of erfc(x)/r (or erf(x)/r) for r = sqrt s, x = alpha r: r and x as unevaluated
// double sums, the low parts applied through the first derivative.
double centre_value(double alpha, double s, bool complement, double ex) {
  const double r = std::sqrt(s);
  const double dr = std::fma(-r, r, s) / (2.0 * r);
  const double x = alpha * r;
  const double dx = std::fma(alpha, r, -x) + alpha * dr;
  const double slope = 1.1283791670955126 * ex;  // 2/sqrt pi exp(-x^2)
  const double f = complement ? std::erfc(x) : std::erf(x);
  const double df = (complement ? -slope : slope) * dx;
  const double q = f / r;
  // q + (f - q r + df - q dr) / r
  return q + (std::fma(-q, r, f) + df - q * dr) / r;
}

int pieces(double smax, int shift) { return (high_word(smax) >> shift) - (high_word(kTableMin) >> shift) + 1; }

void fit(double alpha, double smax, bool complement, int shift, int& base, int& n, std::vector<double>& tab) {
  base = high_word(kTableMin) >> shift;
  n = pieces(smax, shift);
  tab.assign(6 * (size_t)n, 0.0);
  const double a2 = alpha * alpha, K = alpha / std::sqrt(3.14159265358979323846) * (complement ? 1.0 : -1.0);
  for (int k = 0; k < n; ++k) {
    const int32_t h = (base + k) << shift;
    const double s = from_high_word(h | (1 << (shift - 1)));  // centre
    const double w = 0.5 * (from_high_word((base + k + 1) << shift) - from_high_word(h));
    const double e = std::exp(-a2 * s);
    double c[7];
    c[0] = centre_value(alpha, s, complement, e);
    double p = K * e;  // K e^{-a2 s} (-a2)^m / m!
    for (int m = 0; m < 6; ++m) {
      c[m + 1] = (-(m + 0.5) * c[m] - p) / (s * (m + 1));
      p *= -a2 / (m + 1);
    }
    // u^6 -> (48 w^2 u^4 - 18 w^4 u^2 + w^6) / 32 on |u| <= w
    const double w2 = w * w;
    c[4] += 1.5 * w2 * c[6];
    c[2] -= 0.5625 * w2 * w2 * c[6];
    c[0] += 0.03125 * w2 * w2 * w2 * c[6];
    for (int m = 0; m < 6; ++m) tab[6 * (size_t)k + m] = c[m];
  }
}

// Ranges of g and h for a box, 0 where it has no tables (it runs on the library functions then).
struct Range64 {
  double g = 0.0, h = 0.0;
  bool any() const { return g > 0.0; }
};

Range64 range64(double alpha, double cut2, const double* cell) {
  double diag = 0.0;  // no image picked by rounded fractions is longer than half the summed edges
  for (int k = 0; k < 3; ++k)
    diag += 0.5 * std::sqrt(cell[3 * k] * cell[3 * k] + cell[3 * k + 1] * cell[3 * k + 1] + cell[3 * k + 2] * cell[3 * k + 2]);
  const double smax = diag * diag;
  if (!(alpha > 0.0) || !(cut2 > kTableMin) || !std::isfinite(smax) || smax > 1e12) return {};
  // whole octaves of h, so that cells of similar size share a table
  double top = kTableMin;
  while (top <= smax * (1.0 + 1e-6)) top *= 2.0;
  // g to the cutoff, or to the longest image distance (the cutoff may be infinite). Past alpha^2 s = 20
  // (erfc below 3e-10) the Gaussian tail would need finer pieces: library functions
  const double gtop = std::min({cut2 * (1.0 + 1e-9), top, 20.0 / (alpha * alpha)});
  if (!(gtop > kTableMin)) return {};
  return {gtop, top};
}

constexpr size_t kPieceBytes = 6 * sizeof(double);

// The fitted pieces, g then h, of the last few ranges: a serving process creates boxes of few kinds
// over and over, and a fit evaluates some 8,000 pieces on the host.
using Fitted = std::shared_ptr<const std::vector<double>>;
using FitKey = std::tuple<double, double, double>;
constexpr size_t kFits = 16;

std::mutex g_mutex;
std::map<std::tuple<int, const grx_arena*, double, double, double>, std::weak_ptr<const Tables64>> g_live;
std::vector<std::pair<FitKey, Fitted>> g_fits;  // at most kFits, the oldest first

Fitted fitted(double alpha, const Range64& r) {
  const FitKey key(alpha, r.g, r.h);
  for (const auto& f : g_fits)
    if (f.first == key) return f.second;
  int base, n;
  std::vector<double> g, h;
  fit(alpha, r.g, true, kShiftG64, base, n, g);
  fit(alpha, r.h, false, kShiftH64, base, n, h);
  g.insert(g.end(), h.begin(), h.end());
  if (g_fits.size() >= kFits) g_fits.erase(g_fits.begin());
  g_fits.emplace_back(key, std::make_shared<const std::vector<double>>(std::move(g)));
  return g_fits.back().second;
}

}  // namespace

Tables64::~Tables64() {
  if (arena) {
    arena_free(arena, g);
    return;
  }
  int prev = -1;
  cudaGetDevice(&prev);
  if (prev != device) cudaSetDevice(device);
  cudaFree(g);
  if (prev >= 0 && prev != device) cudaSetDevice(prev);
}

size_t tables64_bytes(double alpha, double cut2, const double* cell) {
  const Range64 r = range64(alpha, cut2, cell);
  return r.any() ? (size_t)(pieces(r.g, kShiftG64) + pieces(r.h, kShiftH64)) * kPieceBytes : 0;
}

grx_status attach_tables64(grx_box* b, double alpha, double cut2, const double* cell) {
  b->t64.reset();
  const Range64 r = range64(alpha, cut2, cell);
  if (!r.any()) return GRX_OK;
  std::lock_guard<std::mutex> lock(g_mutex);
  for (auto it = g_live.begin(); it != g_live.end();) it = it->second.expired() ? g_live.erase(it) : std::next(it);
  std::weak_ptr<const Tables64>& live = g_live[std::make_tuple(b->device, (const grx_arena*)b->arena, alpha, r.g, r.h)];
  b->t64 = live.lock();
  if (b->t64) return GRX_OK;
  const Fitted tab = fitted(alpha, r);
  auto n = std::make_shared<Tables64>();
  n->device = b->device;
  n->arena = b->arena;
  n->g_base = high_word(kTableMin) >> kShiftG64;
  n->g_n = pieces(r.g, kShiftG64);
  n->h_base = high_word(kTableMin) >> kShiftH64;
  n->h_n = pieces(r.h, kShiftH64);
  const size_t bytes = tab->size() * sizeof(double);
  if (dev_alloc(b, (void**)&n->g, bytes) != cudaSuccess) {
    n->g = nullptr;
    if (b->arena) {  // counted in grx_box_footprint; a box's arithmetic must not depend on its neighbours
      set_error("FP64 tables: %zu bytes do not fit the arena", bytes);
      return GRX_ERR_OUT_OF_MEMORY;
    }
    cudaGetLastError();
    return GRX_OK;  // the library functions serve the box
  }
  n->h = n->g + 3 * (size_t)n->g_n;
  GRX_CHECK_CUDA(cudaMemcpy(n->g, tab->data(), bytes, cudaMemcpyHostToDevice), "upload FP64 tables");
  b->t64 = n;
  live = b->t64;
  return GRX_OK;
}

}  // namespace grx
