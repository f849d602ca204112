// Analytic irradiance fields evaluated on the device in place of BallaSim's renderer (the render hook of
// src/engine/window.h:69-84 on this path): a moving tanh edge and a sum of moving Gaussian blobs, fp32 in a
// fixed operation order (bit-identical to any CPU evaluation compiled without contraction).
//
// Blob table rows (kBlobWords floats): a, cx0, cy0, vx, vy, 1/(2 r^2), (6 r)^2, (3 r)^2, |v|, pad. A blob adds
// exactly 0 where d^2 >= (6 r)^2. Per window a warp lists, in shared memory and in blob order, the blobs whose 6 r
// disc can reach its pixels during the window; every lane then runs one loop over that list with a branch-free
// term (a listed blob out of reach adds +0). Skipped and zero terms leave the fp32 sum's bits unchanged, so the
// result is the full definition's.
#pragma once

#include "bs_math.cuh"

namespace bs {

constexpr int kFieldTanhEdge = 1;
constexpr int kFieldBlobs = 2;
constexpr int kBlobWords = 10;
constexpr int kMaxListed = 256;  // tables of up to 256 blobs are culled per warp; larger ones evaluate every blob

struct FieldDev {
  int32_t kind;
  uint32_t width, height;
  float base, amp, nx, ny, c, speed, width_px;
  int32_t n_blobs;
  const float* blobs;  // device memory, n_blobs x kBlobWords
  // Set by field_bounds: no value of the field lies outside [lo, hi]; listable: at most 65,535 blobs, each term's
  // exponent in [-80, 0].
  float lo, hi;
  int32_t listable;
};

// The candidate blobs of one warp and window (indices in blob order), or all blobs (idx null).
struct BlobList {
  const uint16_t* idx;
  int32_t n;
};

// Bounds of the field's values over all pixels and times, from the parameters and the blob table in host memory: the
// base with every term of either sign, widened by the sums' rounding. tanh lies between -1 and 1, and a blob's term
// between 0 and its amplitude where that is finite and 1 / (2 r^2) is neither negative (the exponential would grow with
// the distance) nor infinite (infinity times the 0 at the centre). Anything else gives the widest bounds.
inline void field_bounds(FieldDev& f, const float* blobs_host) {
  const float inf = __builtin_huge_valf();
  double lo = f.base, hi = f.base, mag = lo < 0 ? -lo : lo;
  bool known = true, falling = true;  // falling: some term may be below 0 (terms >= 0 never round below the base)
  const auto span = [&](double below, double above) {
    lo -= below;
    hi += above;
    mag += below + above;
  };
  f.listable = f.n_blobs <= 65535 ? 1 : 0;
  if (f.kind == kFieldTanhEdge) {
    const double a = f.amp < 0 ? -f.amp : f.amp;
    span(a, a);
  } else {
    falling = false;
    for (int32_t k = 0; k < f.n_blobs; ++k) {
      const float* b = blobs_host + static_cast<size_t>(k) * kBlobWords;
      known = known && b[0] > -inf && b[0] < inf && b[5] >= 0.0f && b[5] < inf;
      falling = falling || b[0] < 0.0f;
      span(b[0] < 0.0f ? -b[0] : 0.0f, b[0] > 0.0f ? b[0] : 0.0f);
      if (!(b[5] >= 0.0f && b[5] * b[6] <= 79.0f)) f.listable = 0;
    }
  }
  const double rounding = 1e-7 * (64.0 + f.n_blobs);  // each sum rounds by at most 2^-24 of the terms so far
  if (falling) lo -= rounding * mag;
  hi += rounding * mag;
  if (!(known && lo > -3e38 && hi < 3e38 && mag < 3e38)) {
    lo = -3e38;
    hi = 3e38;
  }
  f.lo = static_cast<float>(lo);
  f.hi = static_cast<float>(hi);
}

BS_HD float t_seconds(int64_t t_ns) { return static_cast<float>(static_cast<double>(t_ns) * 1e-9); }

BS_HD float tanh_det(float u) {
  const float a = fabs_f(u);
  float r = 1.0f;
  if (a <= 9.0f) {
    const float e = exp_f(2.0f * a);
    r = 1.0f - 2.0f / (e + 1.0f);
  }
  return u < 0.0f ? -r : r;
}

BS_HD float edge_eval(const FieldDev& f, float xc, float yc, float ts) {
  const float u = (((f.nx * xc + f.ny * yc) - f.speed * ts) - f.c) / f.width_px;
  return f.base + f.amp * tanh_det(u);
}

// One blob's term, branch-free: A exp(-d^2 / (2 r^2)) inside 6 r, else +0 (the exp then sees a harmless 0).
BS_HD float blob_term(const float* b, float xc, float yc, float ts) {
  const float cx = b[1] + b[3] * ts, cy = b[2] + b[4] * ts;
  const float dx = xc - cx, dy = yc - cy;
  const float d2 = dx * dx + dy * dy;
  const bool in = d2 < b[6];
  const float term = b[0] * exp_f(in ? -(d2 * b[5]) : 0.0f);
  return in ? term : 0.0f;
}

// E(x, y, t) over every blob (the definition).
BS_HD float field_eval_all(const FieldDev& f, uint32_t x, uint32_t y, int64_t t_ns) {
  const float ts = t_seconds(t_ns);
  const float xc = static_cast<float>(x) + 0.5f, yc = static_cast<float>(y) + 0.5f;
  if (f.kind == kFieldTanhEdge) return edge_eval(f, xc, yc, ts);
  float e = f.base;
  for (int32_t k = 0; k < f.n_blobs; ++k) e = e + blob_term(f.blobs + static_cast<size_t>(k) * kBlobWords, xc, yc, ts);
  return e;
}

// E(x, y, t) over a warp's candidate list (bitwise field_eval_all when the list holds every blob in reach). One
// out-of-line copy serves the sampler's render sites (a smaller kernel for the instruction cache); blobs go in
// pairs whose exp chains are independent, summed in list order.
static __host__ __device__ __noinline__ float field_eval(const FieldDev& f, const BlobList& l, uint32_t x, uint32_t y,
                                                         int64_t t_ns) {
  if (f.kind != kFieldBlobs || l.idx == nullptr) return field_eval_all(f, x, y, t_ns);
  const float ts = t_seconds(t_ns);
  const float xc = static_cast<float>(x) + 0.5f, yc = static_cast<float>(y) + 0.5f;
  float e = f.base;
  int32_t i = 0;
  for (; i + 1 < l.n; i += 2) {
    const float t0 = blob_term(f.blobs + static_cast<size_t>(l.idx[i]) * kBlobWords, xc, yc, ts);
    const float t1 = blob_term(f.blobs + static_cast<size_t>(l.idx[i + 1]) * kBlobWords, xc, yc, ts);
    e = e + t0;
    e = e + t1;
  }
  if (i < l.n) e = e + blob_term(f.blobs + static_cast<size_t>(l.idx[i]) * kBlobWords, xc, yc, ts);
  return e;
}

// The lattice level of a pixel under a blob of speed v (0: none): clamp(ceil(log2(v W / 0.25 px)), l_min, l_max).
BS_HD int32_t level_of_speed(float v, int32_t l_min, int32_t l_max) {
  if (!(v > 0.0f)) return l_min;
  const float q = v * 0.033554432f;  // v W / 0.25 px with W = 2^23 ns
  const uint32_t bq = f2u(q);
  const int e = static_cast<int>((bq >> 23) & 0xffu) - 126;  // q = m 2^e, m in [0.5, 1) (q is normal)
  const bool half = (bq & 0x7fffffu) == 0u;                    // m == 0.5: log2 q = e - 1 exactly
  int32_t level = half ? e - 1 : e;
  if (level < l_min) level = l_min;
  if (level > l_max) level = l_max;
  return level;
}

// The level rule at the window start: clamp(ceil(log2(v W / 0.25 px)), l_min, l_max), v the speed of the fastest
// blob whose 3 r support covers the pixel (none, or the tanh edge: l_min).
BS_HD int32_t field_level(const FieldDev& f, const BlobList& l, uint32_t x, uint32_t y, int64_t t_w, int32_t l_min,
                          int32_t l_max) {
  if (f.kind != kFieldBlobs) return l_min;
  const float ts = t_seconds(t_w);
  const float xc = static_cast<float>(x) + 0.5f, yc = static_cast<float>(y) + 0.5f;
  float v = 0.0f;
  const int32_t n = l.idx != nullptr ? l.n : f.n_blobs;
  for (int32_t i = 0; i < n; ++i) {
    const int32_t k = l.idx != nullptr ? l.idx[i] : i;
    const float* b = f.blobs + static_cast<size_t>(k) * kBlobWords;
    const float cx = b[1] + b[3] * ts, cy = b[2] + b[4] * ts;
    const float dx = xc - cx, dy = yc - cy;
    const float d2 = dx * dx + dy * dy;
    v = (d2 <= b[7] && b[8] > v) ? b[8] : v;
  }
  return level_of_speed(v, l_min, l_max);
}

// The lattice level at which the chord over a step deviates by no more than the sampler's tolerance: a quarter of
// `deviation` (at `level`) per halving, at most max_refine of them; past most_log2 only that it is.
inline int32_t refined_level(int32_t level, double deviation, float tol, int32_t max_refine, int most_log2) {
  for (int32_t i = 0; i < max_refine && level <= most_log2 && deviation > tol; ++i) {
    deviation *= 0.25;
    ++level;
  }
  return level;
}
// A speed's way in a step of the lattice, px.
inline double lattice_step(float speed, int32_t level) {
  return static_cast<double>(speed) * 1e-9 * static_cast<double>(kWindowNs >> level);
}
// How many of a field's blobs are expected to take some window past 2^most_log2 samples by their motion: the lattice level
// of their speed refined to the tolerance (the chord deviates by step^2 / (8 r^2) of the value). Host side; parameters that
// are not numbers count as still.
inline int32_t blobs_expected_past(const FieldDev& f, const float* blobs_host, int32_t l_min, int32_t l_max, bool midpoint,
                                   float tol, int32_t max_refine, int most_log2) {
  int32_t past = 0;
  for (int32_t k = 0; k < f.n_blobs; ++k) {
    const float* b = blobs_host + static_cast<size_t>(k) * kBlobWords;
    const int32_t level = level_of_speed(b[8], l_min, l_max);
    const double dx = lattice_step(b[3], level), dy = lattice_step(b[4], level);
    const double deviation = 0.25 * (dx * dx + dy * dy) * b[5];
    if (refined_level(level, deviation, tol, midpoint ? max_refine : 0, most_log2) > most_log2) ++past;
  }
  return past;
}
// Whether the windows of a field are expected to hold at most 2^most_log2 samples: no such blob, or an edge that crosses
// no more than its width per step (its refined windows are few whatever the tolerance).
inline bool windows_expected_within(const FieldDev& f, const float* blobs_host, int32_t l_min, int32_t l_max, bool midpoint,
                                    float tol, int32_t max_refine, int most_log2) {
  if (l_min > most_log2) return false;
  if (f.kind == kFieldTanhEdge) {
    const double step = lattice_step(f.speed, l_min);
    return !((step < 0 ? -step : step) > f.width_px) || !midpoint;
  }
  return blobs_expected_past(f, blobs_host, l_min, l_max, midpoint, tol, max_refine, most_log2) == 0;
}
// The same for the windows at an edge, refined to the tolerance (step^2 / (8 width^2)).
inline bool edge_expected_within(const FieldDev& f, int32_t l_min, float tol, int32_t max_refine, int most_log2) {
  const double step = lattice_step(f.speed, l_min) / f.width_px;
  return refined_level(l_min, 0.125 * step * step, tol, max_refine, most_log2) <= most_log2;
}

#if defined(__CUDACC__)
// Builds the calling warp's candidate list for [t_a, t_b] in `list` (kMaxListed entries of shared memory): blob k
// is listed when its 6 r disc, swept from t_a to t_b, can reach the bounding box of the active lanes' pixel
// centres (a 1 px margin covers the fp32 rounding of the per-sample test). All 32 lanes call it together.
__device__ inline BlobList warp_blob_list(const FieldDev& f, bool have, uint32_t x, uint32_t y, int64_t t_a,
                                          int64_t t_b, uint16_t* list) {
  if (f.kind != kFieldBlobs || f.n_blobs > kMaxListed) return BlobList{nullptr, f.n_blobs};
  float x0 = have ? static_cast<float>(x) + 0.5f : 3.0e38f, x1 = have ? static_cast<float>(x) + 0.5f : -3.0e38f;
  float y0 = have ? static_cast<float>(y) + 0.5f : 3.0e38f, y1 = have ? static_cast<float>(y) + 0.5f : -3.0e38f;
  for (int o = 16; o > 0; o >>= 1) {
    x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
    y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
  }
  const float ta = t_seconds(t_a), tb = t_seconds(t_b);
  const uint32_t lane = threadIdx.x & 31u;
  int32_t n = 0;
  for (int32_t base = 0; base < f.n_blobs; base += 32) {
    const int32_t k = base + static_cast<int32_t>(lane);
    bool keep = false;
    if (k < f.n_blobs) {
      const float* b = f.blobs + static_cast<size_t>(k) * kBlobWords;
      const float cxa = b[1] + b[3] * ta, cxb = b[1] + b[3] * tb;
      const float cya = b[2] + b[4] * ta, cyb = b[2] + b[4] * tb;
      const float reach = sqrtf(b[6]) + 1.0f;
      const float bx0 = fminf(cxa, cxb) - reach, bx1 = fmaxf(cxa, cxb) + reach;
      const float by0 = fminf(cya, cyb) - reach, by1 = fmaxf(cya, cyb) + reach;
      keep = !(bx1 < x0 || bx0 > x1 || by1 < y0 || by0 > y1);
    }
    const uint32_t bits = __ballot_sync(0xffffffffu, keep);
    if (keep) list[n + __popc(bits & ((1u << lane) - 1u))] = static_cast<uint16_t>(k);
    n += __popc(bits);
  }
  __syncwarp();
  return BlobList{list, n};
}
#endif

}  // namespace bs
