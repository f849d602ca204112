// field_bounds (ballasim_b200/csrc/fields.cuh) on the CPU: over random fields, their blob tables now and then holding a
// value out of the ordinary, no sample lies outside [lo, hi], and one that is not finite comes with the widest bounds
// only. Exits 0 where that holds, else prints the first sample for which it does not.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#define __host__
#define __device__
#define __noinline__
#include "fields.cuh"

int main() {
  std::mt19937_64 rng(11);
  const auto uni = [&](double a, double b) { return static_cast<float>(std::uniform_real_distribution<double>(a, b)(rng)); };
  const float odd[] = {NAN, INFINITY, -INFINITY, 0.0f, -0.0f, -1.0f, 1e30f, -1e30f, 3e38f, 1e-40f};
  long strange = 0;
  for (int trial = 0; trial < 20000; ++trial) {
    bs::FieldDev f{};
    f.kind = trial % 4 == 0 ? bs::kFieldTanhEdge : bs::kFieldBlobs;
    f.width = 40;
    f.height = 30;
    f.base = trial % 3 == 0 ? uni(-80, 80) : uni(0, 80);
    f.amp = uni(-60, 60);
    f.nx = uni(-1, 1);
    f.ny = uni(-1, 1);
    f.c = uni(0, 40);
    f.speed = uni(-300, 300);
    f.width_px = uni(0.1, 4);
    const int n = f.kind == bs::kFieldBlobs ? trial % 9 : 0;
    std::vector<float> b(static_cast<size_t>(n) * bs::kBlobWords, 0.0f);
    for (int k = 0; k < n; ++k) {
      float* r = &b[static_cast<size_t>(k) * bs::kBlobWords];
      const float rad = uni(1, 12);
      r[0] = trial % 2 ? uni(0, 90) : uni(-60, 90);
      r[1] = uni(0, 40);
      r[2] = uni(0, 30);
      r[3] = uni(-90, 90);
      r[4] = uni(-90, 90);
      r[5] = 1.0f / (2.0f * rad * rad);
      r[6] = 36.0f * rad * rad;
      r[7] = 9.0f * rad * rad;
      r[8] = std::sqrt(r[3] * r[3] + r[4] * r[4]);
    }
    if (trial % 5 == 1) {  // one value out of the ordinary
      const float v = odd[rng() % (sizeof(odd) / sizeof(odd[0]))];
      if (n > 0) b[(rng() % n) * bs::kBlobWords + rng() % 9] = v;
      else if (f.kind == bs::kFieldTanhEdge) (rng() % 2 ? f.amp : f.width_px) = v;
      else f.base = v;
    }
    f.n_blobs = n;
    f.blobs = b.data();
    bs::field_bounds(f, b.data());
    const bool widest = f.lo == -3e38f && f.hi == 3e38f;
    for (int i = 0; i < 200; ++i) {
      const auto x = static_cast<uint32_t>(rng() % f.width), y = static_cast<uint32_t>(rng() % f.height);
      const float e = bs::field_eval_all(f, x, y, static_cast<int64_t>(rng() % 600) * 1000003);
      const bool finite = std::isfinite(e) && std::fabs(e) < 3e38f;
      strange += !finite;
      if (finite ? !(e >= f.lo && e <= f.hi) : !widest) {
        std::printf("trial %d: sample %g outside [%g, %g]\n", trial, e, f.lo, f.hi);
        return 1;
      }
    }
  }
  if (strange < 100) std::printf("only %ld samples were not finite\n", strange);
  return strange < 100;
}
