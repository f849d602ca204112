// The split engine (stage 1): per window, every pixel's common path in one kernel and the rare ones in another.
//
// A pixel-window is nearly always quiet: the sampler takes the lattice alone (no midpoint test fails) and the
// comparator's Delta stays between its levels. The window kernel decides that from the window's extreme samples
// against two precomputed bounds, without the model's state, its logarithms or the noise chains; the others (about 2 %:
// a crossing may occur, a noise candidate that may be accepted, the refractory interval) are posted to a list, and the
// rest kernel runs each of them through the full pixel model, one thread per pixel. Per call:
//
//  - split_begin_kernel (once): gathers every pixel's state and map from their planes into one 128-byte record, which
//    the rest kernel updates in place (a trial or a re-run starts again from the call's input); walks the noise chains to
//    the call's end, noting the candidates that some irradiance of the call may accept; and writes the quick records.
//  - split_window_kernel (per window): one warp per tile. Reads the quick records (28 B a pixel, in tile order, against
//    112 B of state and map), samples the lattice, and keeps the quiet pixels' carried samples; their state changes by
//    the search time and the held sample only, which the end kernel fills in.
//  - split_rest_kernel (per window): the posted pixels.
//  - split_end_kernel (once): the records back into the call's output planes.
//
// The quick test is sound, not exact: with I the photocurrent at the samples' extremes, widened by the rounding of the
// interpolation, ln(I / i_scale) - s3 - n3 + dl must stay off both levels by more than a slack that covers every
// rounding in Delta and in the bound itself. Where it answers "quiet", no integer of the window fires and the model
// would only move its search time to the window's end; where it does not, the model decides. So the events and the
// state are those of the other engines, bit for bit.
//
// Measured on five sensors of 4.3 Mpx with noise, 60 windows: the window kernels 14.1 ms, the rest kernels 8.8, begin
// 1.5, end 0.16; a form whose window kernel ran the model's clean segments in registers (one logarithm a sample, the
// noise chains met window by window, the full state through HBM) took 53.0 and 10.0 ms. Issue bounds the window kernel
// (61 % of its slots), the length of one pixel's chain the rest kernel.
#include "engine_dev.cuh"

namespace bs {

namespace {

constexpr int kSplitStage = 1 << kSplitStageLog2;  // samples after slot 0 that a posted pixel takes along
constexpr uint32_t kRestWhole = 0xFF;  // the samples of a window that has more: walked again by the rest kernel
constexpr int kCentres = 64;          // blobs a warp holds, and centres (one blob at two lattice slots) at a time
constexpr int kTile0Args = 16;        // sensors whose first tiles travel as kernel arguments

// The quick record of lane l of tile t, entry 32 t + l of each plane (tile order: a warp's loads are whole lines).
//   a: the bounds of log2 I at the call's start (upper, lower), their fall per second (the leak), and the first window
//      of the call that the pixel must be posted in (a noise candidate that may be accepted; INT_MIN: now);
//   b: the photocurrent's dark term and scale; c: the carried sample.
struct QuickPlanes {
  float4* a;
  float2* b;
  float* c;
};

// A pixel's state and map while a call runs, one cache line, entry 32 t + l as the quick record's: the posted pixels are
// few and scattered, and reading theirs from the 21 planes of the model took longer than the work on them. t_shot,
// n_shot: the shot chain's first candidate that may be accepted (skip_rejected), or its first at or after the call's
// end; later[]: the stops after it, as far as they fit (t < 0: not known).
struct alignas(128) SplitPixel {
  int64_t t_ref, t_search, blind_until, t_shot, t_ba;
  float s3_ref, n3_ref, dr_ref, i_scale;
  uint32_t flags, n_shot, n_ba;
  float theta_on, theta_off, leak, dark, scale;
  double ba_rate_hz, shot_max_hz;
  int64_t later_t[2];
  uint32_t later_n[2];
};
static_assert(sizeof(SplitPixel) == 128, "one line");

// A posted pixel: its slot (the entry above), pixel, a tag (sensor, samples left or kRestWhole, level, whether the times
// are staged too) and samples; the times of a refined window's samples, in an array of their own.
struct RestRecord {
  uint32_t slot, pixel, tag, pad;
  float v[kSplitStage];
};
struct RestTimes {
  uint32_t dt[kSplitStage];
};
struct RestList {
  RestRecord* rec;
  RestTimes* times;
  unsigned int* count;
  unsigned int* taken;  // the records that warps have taken after their first ones
  unsigned int capacity;
};

struct SplitArgs {
  const EngineSensor* sensors;
  int n_sensors;
  uint32_t total_tiles;
  const int64_t* t0;  // the model time, in device memory (a captured launch replays at any time)
  int32_t w, windows;
  SamplerRules r;
  uint32_t tile_lw;
  unsigned long long minus_zero2;  // two fp32 -0 (mul2)
  uint32_t block_tiles;  // split_solo_kernel: the tiles of a block
  QuickPlanes q;
  SplitPixel* px;
  uint16_t* lists;   // of a tile with pixels posted whole: its blob list (kMaxListed entries a tile) and
  int32_t* list_n;   // that list's length (< 0: none)
  float4* boxes;  // this window's blob boxes (total_blobs), and the next one's (written by the rest kernel)
  float4* boxes_next;
  uint32_t tile0[kTile0Args];
};

// Window w of the call: its start, and its start and end since the call's start in seconds.
struct WindowTimes {
  int32_t w;
  int64_t T0, T_end, t_w;
  float tau_a, tau_b;
  __device__ __forceinline__ WindowTimes(const SplitArgs& a, int32_t w_) : w(w_) {
    T0 = *a.t0;
    T_end = T0 + static_cast<int64_t>(a.windows) * kWindowNs;
    t_w = T0 + static_cast<int64_t>(w) * kWindowNs;
    tau_a = static_cast<float>(static_cast<double>(t_w - T0) * 1e-9);
    tau_b = static_cast<float>(static_cast<double>(t_w - T0 + kWindowNs) * 1e-9);
  }
};

__device__ __forceinline__ int sensor_of(const SplitArgs& a, uint32_t tile) {
  int si = 0;
  if (a.n_sensors <= kTile0Args) {
    while (si + 1 < a.n_sensors && a.tile0[si + 1] <= tile) ++si;
  } else {
    int lo = 0, hi = a.n_sensors - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (a.sensors[mid].tile0 <= tile) lo = mid;
      else hi = mid - 1;
    }
    si = lo;
  }
  return si;
}

// A blob's box for the window at t_w: where its 6 r disc, swept over the window, can be (a 1 px margin covers the fp32
// rounding of the per-sample test): x from .x to .y, y from .z to .w.
__device__ __forceinline__ float4 blob_box(const FieldDev& f, uint32_t k, float ta, float tb) {
  const float* b = f.blobs + static_cast<size_t>(k) * kBlobWords;
  const float cxa = b[1] + b[3] * ta, cxb = b[1] + b[3] * tb;
  const float cya = b[2] + b[4] * ta, cyb = b[2] + b[4] * tb;
  const float reach = sqrtf(b[6]) + 1.0f;
  return make_float4(fminf(cxa, cxb) - reach, fmaxf(cxa, cxb) + reach, fminf(cya, cyb) - reach, fmaxf(cya, cyb) + reach);
}
// All sensors' boxes, over the launch's threads.
__device__ __forceinline__ void write_boxes(const SplitArgs& a, int64_t t_w, float4* boxes) {
  const float ta = t_seconds(t_w), tb = t_seconds(t_w + kWindowNs);
  for (int si = 0; si < a.n_sensors; ++si) {
    const EngineSensor& S = a.sensors[si];
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < static_cast<uint32_t>(S.field.n_blobs);
         k += gridDim.x * blockDim.x) {
      boxes[S.blob0 + k] = blob_box(S.field, k, ta, tb);
    }
  }
}

// The records of one tile.
__device__ __forceinline__ void begin_tile(const SplitArgs& a, uint32_t tile, uint32_t lane) {
  const int64_t T0 = *a.t0, T_end = T0 + static_cast<int64_t>(a.windows) * kWindowNs;
  const EngineSensor& S = a.sensors[sensor_of(a, tile)];
  uint32_t x, y;
  tile_xy(tile - S.tile0, S.tiles_x, a.tile_lw, lane, x, y);
  const uint32_t slot = tile * 32u + lane;
  float4 qa = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float2 qb = make_float2(0.0f, 0.0f);
  float qc = 0.0f;
  uint32_t skipped = 0;
  if (x < S.width && y < S.height) {
    const uint32_t p = y * S.width + x;
    const bool noise = S.consts.noise != 0;
    PixelRegs s;
    PixelMapRegs m;
    load_state(S.in, p, noise, s);
    load_map(S.map, p, m);
    qc = S.carried_in[p];
    int64_t later_t[2] = {-1, -1};
    uint32_t later_n[2] = {0u, 0u};
    if (noise && m.shot_max_hz > 0.0 && s.t_shot < T_end) {
      const uint32_t limit = accept_limit(m, S.consts, S.field, qc);
      int64_t t = s.t_shot;
      uint32_t n = s.n_shot;
      U4 w = draw(S.consts.seed, kPurposeShot, S.consts.camera, p, n);
      // One candidate a turn, noted where the chain stops, so that the lanes' chains run together whatever their stops.
      for (int stops = 0;;) {
        if (t >= T_end || w.v[1] <= limit) {
          if (stops == 0) {
            s.t_shot = t;
            s.n_shot = n;
          } else {
            later_t[1] = t;
            later_n[1] = n;
            if (stops == 1) {
              later_t[0] = t;
              later_n[0] = n;
              later_t[1] = -1;
            }
          }
          ++stops;
          if (t >= T_end || stops == 3) break;
        } else {
          ++skipped;  // the stops are counted where the rest kernel meets them
        }
        ++n;
        w = draw(S.consts.seed, kPurposeShot, S.consts.camera, p, n);
        t = noise_after(w, t, m.shot_max_hz);
      }
    }
    SplitPixel r{s.t_ref, s.t_search, s.blind_until, s.t_shot, s.t_ba, s.s3_ref, s.n3_ref, s.dr_ref, s.i_scale, s.flags,
                 s.n_shot, s.n_ba, m.theta_on, m.theta_off, m.leak, m.dark, m.scale, m.ba_rate_hz, m.shot_max_hz,
                 {later_t[0], later_t[1]}, {later_n[0], later_n[1]}};
    a.px[slot] = r;
    qa = quick_record(s, m, noise, T0, T_end);
    qb = make_float2(m.dark, m.scale);
  }
  a.q.a[slot] = qa;
  a.q.b[slot] = qb;
  a.q.c[slot] = qc;
  const uint32_t sum = __reduce_add_sync(0xffffffffu, skipped);
  if (lane == 0u && sum != 0u) atomicAdd(&S.counters[kCntNoise], static_cast<unsigned long long>(sum));
}

// The output of one tile: every pixel's state, its search at least at the call's end (a quiet window moves it to its
// own), the held and the carried sample.
__device__ __forceinline__ void end_tile(const SplitArgs& a, uint32_t tile, uint32_t lane) {
  const EngineSensor& S = a.sensors[sensor_of(a, tile)];
  uint32_t x, y;
  tile_xy(tile - S.tile0, S.tiles_x, a.tile_lw, lane, x, y);
  if (x >= S.width || y >= S.height) return;
  const uint32_t p = y * S.width + x, slot = tile * 32u + lane;
  const SplitPixel r = a.px[slot];
  const float carried = a.q.c[slot];
  PixelRegs s;
  s.t_ref = r.t_ref;
  s.t_search = maxi(r.t_search, *a.t0 + static_cast<int64_t>(a.windows) * kWindowNs);
  s.blind_until = r.blind_until;
  s.s3_ref = r.s3_ref;
  s.n3_ref = r.n3_ref;
  s.dr_ref = r.dr_ref;
  s.i_scale = r.i_scale;
  s.held = clamp_irr(carried, S.consts.irr_max);
  s.flags = r.flags;
  s.t_shot = r.t_shot;
  s.t_ba = r.t_ba;
  s.n_shot = r.n_shot;
  s.n_ba = r.n_ba;
  store_state(S.out, p, S.consts.noise != 0, s);
  S.carried_out[p] = carried;
}

__global__ void __launch_bounds__(128) split_begin_kernel(const __grid_constant__ SplitArgs a) {
  const uint32_t tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  write_boxes(a, *a.t0, a.boxes);
  if (tile < a.total_tiles) begin_tile(a, tile, threadIdx.x & 31u);
}
__global__ void __launch_bounds__(128) split_end_kernel(const __grid_constant__ SplitArgs a) {
  const uint32_t tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (tile < a.total_tiles) end_tile(a, tile, threadIdx.x & 31u);
}

// Two fp32 values in one register pair, added and multiplied by one instruction each (the same roundings; 73.7 against
// 36.1 T operations a second in a loop of both). The assembler contracts a packed product and sum into one rounding even
// where both ask for theirs, so a product is formed as a fused one plus -0 (which changes nothing), with the -0s (z) read
// from the launch's arguments, where it cannot see them.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 x, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b, F2 z) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(z.v));
  return r;
}
__device__ __forceinline__ F2 both(float a) { return pack2(a, a); }

// exp_f of two values in [-80, 0] (no range test, one exact scaling step): the same operations, so the same bits (x - y
// is x + -y). The rounding to an integer adds and takes off 1.5 2^23, whose sum also holds the integer in its low bits.
__device__ __forceinline__ F2 exp_neg2(F2 x, F2 z) {
  const F2 t = add2(mul2(x, both(0x1.715476p+0f), z), both(12582912.0f));
  const F2 k = add2(t, both(-12582912.0f));
  const F2 r = add2(add2(x, mul2(k, both(-0x1.62e400p-1f), z)), mul2(k, both(-0x1.7f7d1cp-20f), z));
  F2 p = both(1.0f / 5040.0f);
  p = add2(mul2(p, r, z), both(1.0f / 720.0f));
  p = add2(mul2(p, r, z), both(1.0f / 120.0f));
  p = add2(mul2(p, r, z), both(1.0f / 24.0f));
  p = add2(mul2(p, r, z), both(1.0f / 6.0f));
  p = add2(mul2(p, r, z), both(0.5f));
  p = add2(mul2(p, r, z), both(1.0f));
  p = add2(mul2(p, r, z), both(1.0f));
  float p0, p1, t0, t1;
  unpack2(p, p0, p1);
  unpack2(t, t0, t1);
  return pack2(__uint_as_float(__float_as_uint(p0) + (__float_as_uint(t0) << 23)),
               __uint_as_float(__float_as_uint(p1) + (__float_as_uint(t1) << 23)));
}

// exceeds() with the quotient formed only near the tolerance (tol_lo: the tolerance less 2^-20 of it, below which the
// rounded quotient cannot exceed it; a NaN or a denominator that is not positive takes the quotient).
__device__ __forceinline__ bool exceeds_fast(const SamplerRules& r, float tol_lo, float a, float m, float b) {
  const float num = fabs_f((a + b) * -0.5f + m);
  const float low = fminf(fminf(a, m), b);
  const float den = r.dark + low;
  if (den > 0.0f && num < tol_lo * den) return false;
  return exceeds(r, a, m, b);
}

struct WarpShared {
  float4 centre[kCentres];  // a blob at two lattice slots: -cx, -cx', -cy, -cy'; first, at the window's start: cx, cy, (3 r)^2
  float4 blob[kCentres];    // -1 / (2 r^2), (6 r)^2, the amplitude; the speed
  uint16_t list[kMaxListed];
  float v[kSplitStage][32];
  uint32_t dt[kSplitStage][32];
};

// The general walk of a window some of whose intervals refine, out of line: stages the first kSplitStage samples.
__device__ __noinline__ uint32_t walk_refined(const SamplerRules* r, const FieldDev* f, const uint16_t* list, int n_list,
                                              uint32_t x, uint32_t y, int64_t t_w, int level, float carried, float* v,
                                              uint32_t* dt) {
  const BlobList bl{n_list >= 0 ? list : nullptr, n_list >= 0 ? n_list : f->n_blobs};
  uint32_t k = 0;
  return sample_pixel_window(*r, level, carried, false, [&](uint32_t d) { return field_eval(*f, bl, x, y, t_w + d); },
                             [&](uint32_t d, float val) {
                               if (k < static_cast<uint32_t>(kSplitStage)) {
                                 dt[k * 32u] = d;
                                 v[k * 32u] = val;
                               }
                               ++k;
                             });
}

// One window of one tile, by a warp: the quiet pixels' carried samples, the others' records in rl. n_samples, n_clean:
// the lane's samples staged and its clean segments. kBoxes: the blobs' boxes of the window are in a.boxes; else they are
// formed here.
template <bool kBoxes>
__device__ __forceinline__ void window_tile(const SplitArgs& a, const RestList& rl, const WindowTimes& wt, WarpShared& w,
                                            const EngineSensor& S, int si, uint32_t tile, uint32_t lane,
                                            unsigned long long& n_samples, unsigned long long& n_clean) {
  const unsigned full = 0xffffffffu;
  const int64_t t_w = wt.t_w;
  const float tol_lo = a.r.tol - 0x1p-20f * fabs_f(a.r.tol);
  uint32_t x, y;
  tile_xy(tile - S.tile0, S.tiles_x, a.tile_lw, lane, x, y);
  const bool have = x < S.width && y < S.height;
  const uint32_t slot = tile * 32u + lane;
  const float4 qa = a.q.a[slot];
  const float2 qb = a.q.b[slot];
  const float carried = a.q.c[slot];
  const FieldDev& f = S.field;
  const float xc = static_cast<float>(x) + 0.5f, yc = static_cast<float>(y) + 0.5f;
  // The blobs in reach of the tile during the window, in blob order; n_list < 0: no list (a tanh edge, more than
  // kMaxListed, or a table whose 1 / (2 r^2) and (6 r)^2 leave exp_neg's range).
  int n_list = f.kind == kFieldBlobs && f.listable ? 0 : -1;
  if (n_list == 0) {
    const uint32_t tx = __shfl_sync(full, x, 0), ty = __shfl_sync(full, y, 0);
    const float bx0 = static_cast<float>(tx) + 0.5f, bx1 = static_cast<float>(tx + (1u << a.tile_lw)) - 0.5f;
    const float by0 = static_cast<float>(ty) + 0.5f, by1 = static_cast<float>(ty + (32u >> a.tile_lw)) - 0.5f;
    const float ta = t_seconds(t_w), tb = t_seconds(t_w + kWindowNs);
    for (int32_t base = 0; base < f.n_blobs; base += 32) {
      const int32_t k = base + static_cast<int32_t>(lane);
      bool keep = false;
      if (k < f.n_blobs) {
        const float4 b = kBoxes ? a.boxes[S.blob0 + k] : blob_box(f, static_cast<uint32_t>(k), ta, tb);
        keep = !(b.y < bx0 || b.x > bx1 || b.w < by0 || b.z > by1);
      }
      const uint32_t bits = __ballot_sync(full, keep);
      if (n_list + __popc(bits) > kMaxListed) {
        n_list = -1;
        break;
      }
      if (keep) w.list[n_list + __popc(bits & ((1u << lane) - 1u))] = static_cast<uint16_t>(k);
      n_list += __popc(bits);
    }
    __syncwarp();
  }
  const bool listed = n_list >= 0 && n_list <= kCentres;  // else each lane evaluates its own samples
  // The listed blobs, one a lane; and the level rule (field_level) from their centres at the window's start.
  if (listed) {
    const float ts = t_seconds(t_w);
    for (int i = static_cast<int>(lane); i < n_list; i += 32) {
      const float* b = f.blobs + static_cast<size_t>(w.list[i]) * kBlobWords;
      w.blob[i] = make_float4(-b[5], b[6], b[0], b[8]);
      w.centre[i] = make_float4(b[1] + b[3] * ts, b[2] + b[4] * ts, b[7], 0.0f);
    }
    __syncwarp();
  }
  int level = a.r.l_min;
  if (listed) {
    float v = 0.0f;
    for (int i = 0; i < n_list; ++i) {
      const float4 c = w.centre[i];
      const float dx = xc - c.x, dy = yc - c.y;
      const float d2 = dx * dx + dy * dy, speed = w.blob[i].w;
      v = (d2 <= c.z && speed > v) ? speed : v;
    }
    level = level_of_speed(v, a.r.l_min, a.r.l_max);
  } else if (f.kind == kFieldBlobs) {
    level = field_level(f, BlobList{n_list > 0 ? w.list : nullptr, n_list > 0 ? n_list : f.n_blobs}, x, y, t_w,
                        a.r.l_min, a.r.l_max);
  }
  // The lattice: slot j of the tile's finest level, at every lane whose own level has it. A lane whose level holds
  // more than kSplitStage samples is posted whole.
  const bool fits = have && (1 << level) <= kSplitStage;
  const int fine = static_cast<int>(__reduce_max_sync(full, static_cast<unsigned>(fits ? level : 0)));
  const int slots = 1 << fine;
  const int skip = fits ? (1 << (fine - level)) - 1 : -1;  // a slot is the lane's own where (j & skip) == 0
  float p2 = carried, p1 = carried, v_lo = carried, v_hi = carried;
  bool flagged = false;
  uint32_t n = 1;
  const auto take = [&](int j, float e) {  // the field at slot j, where the lane has it
    if (!fits || (j & skip) != 0) return;
    if (n >= 2u) flagged = flagged || (a.r.midpoint != 0 && exceeds_fast(a.r, tol_lo, p2, p1, e));
    w.v[n - 1u][lane] = e;
    ++n;
    p2 = p1;
    p1 = e;
    v_lo = min_nan(v_lo, e);
    v_hi = max_nan(v_hi, e);
  };
  if (listed) {
    // Slots in pairs (1, 2), (3, 4), ..., each blob's term at both in one run of packed operations.
    const int shift = n_list > 1 ? 32 - __clz(n_list - 1) : 0;  // lanes per pair: the next power of two
    const int pairs = (slots + 1) / 2, group = n_list > 0 ? kCentres / n_list : pairs;
    const F2 xc2 = both(xc), yc2 = both(yc), z{a.minus_zero2};
    for (int g0 = 0; g0 < pairs; g0 += group) {
      const int g1 = g0 + group < pairs ? g0 + group : pairs;
      __syncwarp();
      for (int q = static_cast<int>(lane); q < (g1 - g0) << shift; q += 32) {
        const int i = q & ((1 << shift) - 1), g = g0 + (q >> shift);
        if (i < n_list) {
          const float* b = f.blobs + static_cast<size_t>(w.list[i]) * kBlobWords;
          const float ta = t_seconds(t_w + (static_cast<int64_t>(2 * g + 1) << (kWindowLog2 - fine)));
          const float tb = t_seconds(t_w + (static_cast<int64_t>(2 * g + 2) << (kWindowLog2 - fine)));
          w.centre[(g - g0) * n_list + i] = make_float4(-(b[1] + b[3] * ta), -(b[1] + b[3] * tb), -(b[2] + b[4] * ta),
                                                        -(b[2] + b[4] * tb));
        }
      }
      __syncwarp();
      for (int g = g0; g < g1; ++g) {
        F2 e = both(f.base);
        const float4* centre = w.centre + (g - g0) * n_list;
        for (int i = 0; i < n_list; ++i) {
          const float4 c = centre[i], b = w.blob[i];
          const F2 dx = add2(xc2, pack2(c.x, c.y)), dy = add2(yc2, pack2(c.z, c.w));
          const F2 d2 = add2(mul2(dx, dx, z), mul2(dy, dy, z));
          float da, db, xa, xb, ta, tb;
          unpack2(d2, da, db);
          unpack2(mul2(d2, both(b.x), z), xa, xb);
          const bool ina = da < b.y, inb = db < b.y;
          unpack2(mul2(both(b.z), exp_neg2(pack2(ina ? xa : 0.0f, inb ? xb : 0.0f), z), z), ta, tb);
          e = add2(e, pack2(ina ? ta : 0.0f, inb ? tb : 0.0f));
        }
        float ea, eb;
        unpack2(e, ea, eb);
        take(2 * g + 1, ea);
        if (2 * g + 2 <= slots) take(2 * g + 2, eb);
      }
    }
  } else {
    for (int j = 1; j <= slots; ++j) {
      float e = 0.0f;
      if (fits && (j & skip) == 0) {
        e = field_eval(f, BlobList{n_list > 0 ? w.list : nullptr, n_list > 0 ? n_list : f.n_blobs}, x, y,
                       t_w + (static_cast<int64_t>(j) << (kWindowLog2 - fine)));
      }
      take(j, e);
    }
  }
  float last = p1;
  // A flagged interval refines where it can still be split: such lanes walk the window in the general form.
  const bool refine = fits && flagged && (static_cast<uint32_t>(kWindowNs) >> level) >= a.r.min_split &&
                      a.r.max_refine_levels > 0;
  bool staged = fits;
  if (refine) {
    n = walk_refined(&a.r, &f, w.list, n_list, x, y, t_w, level, carried, &w.v[0][lane], &w.dt[0][lane]);
    staged = n - 1u <= static_cast<uint32_t>(kSplitStage);
    if (staged) {
      for (uint32_t q = 0; q + 1u < n; ++q) {
        const float e = w.v[q][lane];
        v_lo = min_nan(v_lo, e);
        v_hi = max_nan(v_hi, e);
        last = e;
      }
    }
  }
  if (staged) n_samples += n;
  // Quiet: the whole window clean by the bounds (NaN answers no); segments of one or two ns count no node in the
  // model, so a refined window that can hold them is posted.
  const float I_hi = qb.x + qb.y * v_hi, I_lo = qb.x + qb.y * v_lo;
  const float pad = 0x1p-21f * I_hi;
  const bool quiet = staged && wt.w < __float_as_int(qa.w) && v_lo >= 0.0f && v_hi <= S.consts.irr_max &&
                     __log2f(I_hi + pad) < qa.x - qa.z * wt.tau_b && __log2f(I_lo - pad) > qa.y - qa.z * wt.tau_a &&
                     !(refine && a.r.min_split <= 4u);
  if (quiet) {
    n_clean += n - 1u;
    a.q.c[slot] = last;
  }
  // One record per posted pixel, the warp's records reserved together; with a pixel posted whole, the tile's blob list.
  const bool post = have && !quiet;
  const unsigned posting = __ballot_sync(full, post);
  if (posting != 0u) {
    if (__any_sync(full, post && !staged)) {
      for (int i = static_cast<int>(lane); i < n_list; i += 32) a.lists[static_cast<size_t>(tile) * kMaxListed + i] = w.list[i];
      if (lane == 0u) a.list_n[tile] = n_list;
    }
    const int leader = __ffs(posting) - 1;
    unsigned int base = 0;
    if (static_cast<int>(lane) == leader) base = atomicAdd(rl.count, static_cast<unsigned int>(__popc(posting)));
    base = __shfl_sync(full, base, leader);
    if (post) {
      const unsigned int i = base + static_cast<unsigned int>(__popc(posting & ((1u << lane) - 1u)));
      if (i >= rl.capacity) {
        atomicOr(&S.counters[kCntErrors], kErrRestList);
      } else {
        const uint32_t left = staged ? n - 1u : kRestWhole;
        RestRecord& rec = rl.rec[i];
        rec.slot = slot;
        rec.pixel = y * S.width + x;
        rec.tag = static_cast<uint32_t>(si) | left << 16 | static_cast<uint32_t>(level) << 24 |
                  (refine ? 0x80000000u : 0u);
        if (staged) {
          for (uint32_t u = 0; u < left; ++u) {
            rec.v[u] = w.v[u][lane];
            if (refine) rl.times[i].dt[u] = w.dt[u][lane];
          }
        }
      }
    }
  }
  __syncwarp();
}

// A block's samples and clean segments per sensor, added to the sensors' counters once at the end (one atomic per warp
// and sensor would take longer than the kernel: atomics on one address pass one at a time).
struct SplitSums {
  unsigned long long v[kTile0Args][2];
  __device__ __forceinline__ void clear() {
    for (int q = static_cast<int>(threadIdx.x); q < 2 * kTile0Args; q += static_cast<int>(blockDim.x)) v[q / 2][q % 2] = 0ull;
  }
  __device__ __forceinline__ void add(const SplitArgs& a) const {
    if (static_cast<int>(threadIdx.x) >= a.n_sensors || a.n_sensors > kTile0Args) return;
    const unsigned long long n = v[threadIdx.x][0], clean = v[threadIdx.x][1];
    unsigned long long* cnt = a.sensors[threadIdx.x].counters;
    if (n) atomicAdd(&cnt[kCntSamples], n);
    if (clean) {
      atomicAdd(&cnt[kCntPieces], clean);
      atomicAdd(&cnt[kCntLeaves], clean);
    }
  }
};
// A warp's share of them, for the sensor it is at.
struct WarpSums {
  int counted = -1;
  unsigned long long samples = 0, clean = 0;
  __device__ __forceinline__ void flush(const SplitArgs& a, SplitSums& sums) {
    if (counted >= 0) {
      if (a.n_sensors <= kTile0Args) {
        warp_add(&sums.v[counted][0], samples);
        warp_add(&sums.v[counted][1], clean);
      } else {
        unsigned long long* cnt = a.sensors[counted].counters;
        warp_add(&cnt[kCntSamples], samples);
        warp_add(&cnt[kCntPieces], clean);
        warp_add(&cnt[kCntLeaves], clean);
      }
    }
    samples = clean = 0;
  }
  __device__ __forceinline__ void of(const SplitArgs& a, SplitSums& sums, int si) {
    if (si == counted) return;
    flush(a, sums);
    counted = si;
  }
};

// Window a.w of every tile. 6 blocks per SM (80 registers): 11.1 ms of engine time on 1280x720 with noise, 23.9 on the
// five sensors; 11.3 and 24.3 at 7, 11.5 and 24.7 at 8 (11.8 and 24.9 with the field's terms one slot at a time).
__global__ void __launch_bounds__(128, 6) split_window_kernel(const __grid_constant__ SplitArgs a, RestList rl) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  __shared__ WarpShared sh[4];
  __shared__ SplitSums sums;
  sums.clear();
  __syncthreads();
  const WindowTimes wt(a, a.w);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  WarpSums mine;
  for (uint32_t tile = blockIdx.x * (blockDim.x >> 5) + warp; tile < a.total_tiles; tile += warps) {
    const int si = sensor_of(a, tile);
    mine.of(a, sums, si);
    window_tile<true>(a, rl, wt, sh[warp], a.sensors[si], si, tile, lane, mine.samples, mine.clean);
  }
  mine.flush(a, sums);
  __syncthreads();
  sums.add(a);
}

// A window posted whole (more samples than the stage holds), out of line: walked from its start over the tile's blob
// list (every blob where it has none) and fed to the general pixel model. Returns the samples. (Walked by the tile's own
// warp in the window kernel instead, its 80 registers cost the other windows 9 %.)
__device__ __noinline__ uint32_t rest_whole(const SplitArgs* a, const EngineSensor* S, uint32_t tile, uint32_t pixel,
                                            int level, int64_t t_w, PixelRegs* s, const PixelMapRegs* m, PixelCounters* c,
                                            float* carried) {
  const FieldDev& f = S->field;
  const int32_t n_list = a->list_n[tile];
  const BlobList list{n_list >= 0 ? a->lists + static_cast<size_t>(tile) * kMaxListed : nullptr,
                      n_list >= 0 ? n_list : f.n_blobs};
  const uint32_t x = pixel % S->width, y = pixel / S->width;
  const ThreadSink sink{S->ev, &S->counters[kCntEvents]};
  PixelRegs sl = *s;
  const PixelMapRegs ml = *m;
  PixelCounters cl = *c;
  RegFeed<true, ThreadSink> feed{sl, ml, cl, S->consts, &S->consts, pixel, sink, t_w, t_w, sl.held, *carried, 0.0f};
  feed.start(*carried);
  const uint32_t n = sample_pixel_window(a->r, level, *carried, false,
                                         [&](uint32_t dt) { return field_eval(f, list, x, y, t_w + dt); }, feed);
  sl.held = feed.prev_v;
  *carried = feed.last_raw;
  *s = sl;
  *c = cl;
  return n;
}

// The earliest noise candidate: dropped, or tested by thinning against the photocurrent I at its time, and (step) its
// chain's next one (PixelProc::noise_candidate without the event). Out of line: few posted pixels come here.
struct CandidateOut {
  int64_t next;
  bool accepted, on;
};
__device__ __noinline__ void candidate_step(const SensorConsts* k, uint32_t pixel, bool shot, uint32_t n, int64_t tn,
                                            double rate, bool blind, bool step, float dark, float I,
                                            CandidateOut* out) {
  const uint32_t purpose = shot ? kPurposeShot : kPurposeBackground;
  out->accepted = out->on = false;
  if (!blind) {
    const U4 w = draw(k->seed, purpose, k->camera, pixel, n);
    const double accept = shot ? sqrt(static_cast<double>(dark) / static_cast<double>(I)) : 1.0;
    out->on = (w.v[2] & 1u) != 0u;
    out->accepted = open_uniform_d(w.v[1]) < accept;
  }
  out->next = step ? noise_after(draw(k->seed, purpose, k->camera, pixel, n + 1u), tn, rate) : 0;
}

// One pixel's comparator over the segments of one window, the times as offsets from the window's start. The steps and
// their order are PixelProc::piece's; the crossing search differs in which integers it looks at, not in the one it
// finds. Segments are dyadic (a lattice step or a half of one), so the interpolation's division by their length is
// exact as a product.
struct RestPixel {
  const PixelMapRegs& m;
  float s3, dn, dr, i_scale;  // dn = 0 - n3_ref
  int64_t since;              // t_w - t_ref
  uint32_t d0, d1;            // the segment, its values, 1 / length
  float v0, v1, inv;

  __device__ __forceinline__ float current(uint32_t d) const {
    return m.dark + m.scale * (v0 + (v1 - v0) * (static_cast<float>(d - d0) * inv));
  }
  __device__ __forceinline__ float x_of(float I) const { return log_f(I / i_scale); }
  // leak (t - t_ref) 1e-9 + dr; without leak the product is 0.
  __device__ __forceinline__ float dl(uint32_t d) const {
    if (m.leak == 0.0f) return dr;
    return m.leak * static_cast<float>(static_cast<double>(since + static_cast<int64_t>(d)) * 1e-9) + dr;
  }
  __device__ __forceinline__ float delta(float x, float l) const { return ((x - s3) + dn) + l; }

  // The first integer of (a, end) where Delta fires, given that Delta at a (where x is xa) does not; x at it. x is
  // monotone along the segment and dl never falls (PixelProc::may_fire_exact), so for any a < b
  //  - rising input: Delta never falls, so only theta_on can be met, at the first integer of a bisection;
  //  - falling input: Delta over (a, b] is at least x(b) with dl(a) and at most x(a) with dl(b). The first integer q
  //    where the former is at or below -theta_off (or the latter at or above theta_on) bounds the crossing from below;
  //    Delta at q decides, or the search goes on from q with dl and x taken there. Without leak q is the crossing.
  // The bisections start where the line (and the leak) reach the level in real arithmetic and widen from there by the
  // size of x's own rounding, so most take 6 to 8 evaluations of x where halving the segment takes up to 22.
  // x_end, exact_end: x at the segment's end, which bounds x before it where the line meets it exactly. hard: nothing
  // decided (both levels in reach on a falling segment, or Delta lingers at one): the general search takes those.
  __device__ __forceinline__ bool search(uint32_t a, float xa, uint32_t end, float x_start, float x_end, bool exact_end,
                                         uint32_t& hit, float& x_hit, bool& on, bool& hard, uint32_t& evals) const {
    const float len = static_cast<float>(d1 - d0);
    const float I0 = m.dark + m.scale * v0, dI = (m.dark + m.scale * v1) - I0;
    const bool up = v1 >= v0, leak = m.leak != 0.0f;
    const float drift = m.leak * 1.0e-9f;  // dl's rise per ns
    // c: the end of the search, met in the predicate's sense; the segment's end itself where x is known there.
    const uint32_t c_end = exact_end ? end : end - 1u;
    float xc_end = x_end;
    if (!exact_end) {
      xc_end = x_of(current(c_end));
      ++evals;
    }
    const float lc = dl(c_end);
    float la = dl(a);
    on = up;
    if (!up) {
      const bool off_may = delta(xc_end, la) <= -m.theta_off, on_may = leak && delta(xa, lc) >= m.theta_on;
      hard = off_may && on_may;
      if (off_may == on_may) return false;
      on = on_may;
    } else if (!(delta(xc_end, lc) >= m.theta_on)) {
      return false;
    }
    const float level = on ? m.theta_on : -m.theta_off;
    const float slope = (x_end - x_start) / len;
    const float unit = 1.0e-7f * (1.0f + fabs_f(x_start) + fabs_f(s3));
    for (int round = 0; round < 8; ++round) {
      uint32_t c = c_end;
      float xc = xc_end;
      const bool by_leak = !up && on;  // a falling segment met from above: only dl's rise counts
      if (by_leak ? !(delta(xa, lc) >= level) : !up && !(delta(xc, la) <= level)) return false;
      // Where the level is reached, from the segment's start: x = xt there, plus the leak's rise since a (up).
      float g;
      if (by_leak) {
        g = static_cast<float>(a - d0) + (level - delta(xa, la)) / drift;
      } else {
        const float xt = ((level - la) - dn) + s3;
        g = fabs_f(dI) > 1.0e-6f * I0 ? (i_scale * __expf(xt) - I0) / dI * len : (xt - x_start) / slope;
        if (up && leak) {
          const float da = static_cast<float>(a - d0);
          if (!(fabs_f(slope) > 1.0e-3f * drift)) {
            g = da + (level - delta(xa, la)) / drift;
          } else {
            g = da + (g - da) * (slope / (slope + drift));
          }
        }
      }
      const float per_ns = by_leak || (up && !(slope > drift)) ? drift : fabs_f(slope);
      int64_t band = 1 + static_cast<int64_t>(fminf(unit / per_ns, 4.0e6f));
      const int64_t gi = static_cast<int64_t>(d0) + static_cast<int64_t>(fminf(fmaxf(g, 0.0f), len));
      // A falling segment met at -theta_off under a leak: sound steps up to the guess first, each with dl taken where
      // the last one stood (dl at a alone puts q far ahead of the crossing).
      if (!up && !on && leak && round < 7) {
        const int64_t p = gi - band;
        if (p > static_cast<int64_t>(a) + 2 * band && p < static_cast<int64_t>(c)) {
          const float xp = x_of(current(static_cast<uint32_t>(p)));
          ++evals;
          if (delta(xp, la) > level) {
            a = static_cast<uint32_t>(p);
            xa = xp;
            la = dl(a);
            continue;
          }
          c = static_cast<uint32_t>(p);
          xc = xp;
        }
      }
      // (a, c]: not met at a, met at c. Probes either side of the guess, widening, until it is bracketed; then halves.
      uint32_t lo = a, hi = c;
      float xh = xc;
      bool below = false, above = false;
      while (hi - lo > 1u) {
        uint32_t t = lo + (hi - lo) / 2u;
        if (!(below && above)) {
          const int64_t p = !below ? gi - band : gi + band;
          if (p > static_cast<int64_t>(lo) && p < static_cast<int64_t>(hi)) {
            t = static_cast<uint32_t>(p);
          } else {  // outside what is left: this side needs no probe
            if (!below) below = true;
            else above = true;
            continue;
          }
        }
        float xt = xa;
        if (!by_leak) {
          xt = x_of(current(t));
          ++evals;
        }
        const float l = up || by_leak ? dl(t) : la;
        const bool met = on ? delta(xt, l) >= level : delta(xt, l) <= level;
        if (met) {
          hi = t;
          xh = xt;
          above = true;
          if (!below) band *= 8;
        } else {
          lo = t;
          if (below && !above) band *= 8;
          below = true;
        }
      }
      if (hi >= end) return false;  // met at the segment's end only
      if (by_leak) {
        xh = x_of(current(hi));
        ++evals;
      }
      const float lh = dl(hi);
      if (up || (on ? delta(xh, lh) >= level : delta(xh, lh) <= level)) {
        hit = hi;
        x_hit = xh;
        return true;
      }
      a = hi;  // Delta there is off the level: on from it, with x and dl there
      xa = xh;
      la = lh;
      if (a + 1u >= end) return false;
    }
    hard = true;
    return false;
  }
};

// Record i of the posted pixels of a window, by one thread. A lane steps through its window (quiet segments by the quick
// bounds, the refractory release, noise candidates) until it needs a crossing search or is done; the warp's lanes then
// search together (a loop that searched inside the step, at each lane's own segment, took 15.1 ms of rest kernels on
// 346x260, 239 windows, against 4.1).
__device__ __forceinline__ void rest_pixel(const SplitArgs& a, const RestList& rl, const WindowTimes& wt, unsigned int i,
                                           unsigned int lane) {
  const int64_t T0 = wt.T0, T_end = wt.T_end, t_w = wt.t_w;
  const float tau_a = wt.tau_a, tau_b = wt.tau_b;
  const RestRecord& rec = rl.rec[i];
  const uint32_t tag = rec.tag, pixel = rec.pixel, slot = rec.slot;
  const uint32_t left = tag >> 16 & 0xFFu;
  const int level = static_cast<int>(tag >> 24 & 0x7Fu);
  const bool timed = (tag & 0x80000000u) != 0u;
  const EngineSensor& S = a.sensors[tag & 0xFFFFu];
  const SensorConsts& k = S.consts;
  const bool noise = k.noise != 0;
  float raw = a.q.c[slot];
  const SplitPixel px = a.px[slot];
  // Quiet windows moved the search to their ends; the held sample is the carried one.
  PixelRegs s{px.t_ref, maxi(px.t_search, t_w), px.blind_until, px.s3_ref, px.n3_ref, px.dr_ref, px.i_scale,
              clamp_irr(raw, k.irr_max), px.flags, px.t_shot, px.t_ba, px.n_shot, px.n_ba};
  const PixelMapRegs m{px.theta_on, px.theta_off, px.leak, px.dark, px.scale, px.ba_rate_hz, px.shot_max_hz};
  int64_t later_t0 = px.later_t[0], later_t1 = px.later_t[1];
  uint32_t later_n0 = px.later_n[0], later_n1 = px.later_n[1];
  PixelCounters c;
  if (left == kRestWhole) {
    PixelRegs st = s;  // copies, so that the state itself stays in registers
    PixelMapRegs mt = m;
    PixelCounters ct = c;
    float rt = raw;
    const uint32_t n = rest_whole(&a, &S, slot >> 5, pixel, level, t_w, &st, &mt, &ct, &rt);
    s = st;
    c = ct;
    raw = rt;
    if (s.n_shot != px.n_shot) later_t0 = later_t1 = -1;
    atomicAdd(&S.counters[kCntSamples], static_cast<unsigned long long>(n));
  } else {
    ThreadSink sink{S.ev, &S.counters[kCntEvents]};
    RestPixel r{m, s.s3_ref, 0.0f - s.n3_ref, s.dr_ref, s.i_scale, t_w - s.t_ref, 0u, 0u, 0.0f, 0.0f, 0.0f};
    r.v1 = clamp_irr(raw, k.irr_max);
    float4 bounds = a.q.a[slot];
    float x0 = 0.0f, x1 = 0.0f;  // x at the segment's ends, where have_x
    bool have_x = false;
    uint32_t q = 0;
    bool next = true, done = false;
    for (;;) {
      // Steps until a search is needed: from `da` (Delta there does not fire) to before `stop`.
      bool need = false, found = false, on = false;
      uint32_t da = 0, hit = 0;
      float xa = 0.0f, x_hit = 0.0f;
      int64_t stop = 0;
      int label = -1;
      while (!done && !need && !found) {
        if (next) {  // the next sample's segment
          if (q == left) {
            done = true;
            break;
          }
          raw = rec.v[q];
          r.d0 = r.d1;
          r.v0 = r.v1;
          r.d1 = timed ? rl.times[i].dt[q]
                       : (q + 1u) << (static_cast<uint32_t>(kWindowLog2) - static_cast<uint32_t>(level));
          r.v1 = clamp_irr(raw, k.irr_max);
          r.inv = __uint_as_float((127u - (31u - static_cast<uint32_t>(__clz(static_cast<int>(r.d1 - r.d0))))) << 23);
          ++q;
          ++c.pieces;
          next = false;
          have_x = false;
        }
        const int64_t t0 = t_w + r.d0, e = t_w + r.d1;
        const int64_t tn = noise ? mini(s.t_shot, s.t_ba) : kForever;
        bool cand = false, drop = false;
        if (s.blind_until != kNotBlind) {
          cand = drop = s.blind_until >= e ? tn < e : tn <= s.blind_until;
          if (!cand) {
            if (s.blind_until >= e) {
              next = true;
            } else {  // the release: a new reference at x(t_rel) - eps_ci
              const uint32_t db = static_cast<uint32_t>(s.blind_until - t_w);
              r.s3 = r.x_of(r.current(db));
              r.dn = 0.0f;
              r.dr = -k.eps_ci;
              r.since = t_w - s.blind_until;
              s.t_ref = s.blind_until;
              s.blind_until = kNotBlind;
              s.s3_ref = r.s3;
              s.n3_ref = 0.0f;
              s.dr_ref = r.dr;
              bounds = quick_record(s, m, false, T0, T_end);
            }
          }
        } else {
          const int64_t lo = maxi(s.t_search, t0);
          stop = mini(e, tn);
          if (lo < stop) {
            // Quiet by the bounds (split_window_kernel's test on this segment alone), or by Delta at lo and the
            // segment's ends (PixelProc::segment_fast's).
            const float Ia = m.dark + m.scale * r.v0, Ib = m.dark + m.scale * r.v1;
            const float I_hi = fmaxf(Ia, Ib), I_lo = fminf(Ia, Ib);
            const float pad = 0x1p-21f * I_hi;
            bool quiet = __log2f(I_hi + pad) < bounds.x - bounds.z * tau_b &&
                         __log2f(I_lo - pad) > bounds.y - bounds.z * tau_a;
            ++c.leaves;
            if (!quiet) {
              if (!have_x) {
                x0 = r.x_of(Ia);
                x1 = r.x_of(Ib);
                have_x = true;
              }
              da = static_cast<uint32_t>(lo - t_w);
              xa = lo == t0 ? x0 : r.x_of(r.current(da));
              const float la = r.dl(da), D = r.delta(xa, la);
              if (D >= m.theta_on || D <= -m.theta_off) {
                found = true;
                hit = da;
                x_hit = xa;
                on = D >= m.theta_on;
              } else if (stop - lo == 1) {
                quiet = true;
              } else {
                if (r.v0 + (r.v1 - r.v0) == r.v1) {
                  const float top = r.delta(maxr(xa, x1), r.dl(r.d1)), low = r.delta(minr(xa, x1), la);
                  quiet = top < m.theta_on && low > -m.theta_off;
                }
                need = !quiet;
              }
            }
            if (quiet) s.t_search = maxi(s.t_search, stop);
          } else if (tn >= e) {
            next = true;
          } else {
            cand = true;
            drop = tn < s.t_search;
          }
        }
        if (cand) {
          const bool shot = s.t_shot <= s.t_ba;
          const uint32_t dc = static_cast<uint32_t>(tn - t_w);
          const float I = drop ? 0.0f : r.current(dc);
          CandidateOut o;
          candidate_step(&k, pixel, shot, shot ? s.n_shot : s.n_ba, tn, shot ? m.shot_max_hz : m.ba_rate_hz, drop,
                         !shot || later_t0 < 0, m.dark, I, &o);
          ++c.noise_candidates;
          if (shot && later_t0 >= 0) {  // the chain's next stop
            s.t_shot = later_t0;
            s.n_shot = later_n0;
            later_t0 = later_t1;
            later_n0 = later_n1;
            later_t1 = -1;
          } else if (shot) {  // more stops than the record holds: one candidate on
            ++s.n_shot;
            s.t_shot = o.next;
          } else {
            ++s.n_ba;
            s.t_ba = o.next;
          }
          if (o.accepted) {
            found = true;
            hit = dc;
            x_hit = r.x_of(I);
            on = o.on;
            label = kLabelNoise;
          }
        }
      }
      if (done) break;
      if (need) {
        bool hard = false;
        const uint32_t end = static_cast<uint32_t>(stop - t_w);
        found = r.search(da, xa, end, x0, x1, end == r.d1 && r.v0 + (r.v1 - r.v0) == r.v1, hit, x_hit, on, hard,
                         c.leaves);
        if (hard) {
          PixelRegs st = s;
          st.s3_ref = r.s3;
          st.n3_ref = 0.0f - r.dn;
          st.dr_ref = r.dr;
          NullSink none;
          PixelMapRegs mt = m;
          PixelCounters ct;
          PixelProc<NullSink> proc{st, mt, k, pixel, none, ct};
          int64_t th = t_w;
          bool up = false;
          float xt = 0.0f;
          found = proc.search(Segment{t_w + r.d0, t_w + r.d1, r.v0, r.v1}, t_w + da, stop, th, up, xt);
          hit = static_cast<uint32_t>(th - t_w);
          on = up;
          x_hit = xt;
          c.leaves += ct.leaves;
        }
        if (!found) s.t_search = maxi(s.t_search, stop);
      }
      if (found) {  // the event and the reset (PixelProc::fire)
        const int64_t t = t_w + hit;
        const float ds = x_hit - r.s3;
        const float l = m.leak * static_cast<float>(static_cast<double>(t - s.t_ref) * 1e-9);
        const float dl = l + r.dr;
        const float D = ds + r.dn + dl;
        const bool first = (s.flags & kFlagFirstAfterInit) != 0u;
        RawEvent ev;
        ev.pixel = pixel;
        ev.polarity = on ? 1 : 0;
        ev.label = label >= 0 ? static_cast<uint8_t>(label)
                   : first    ? first_label(on, ds, r.dn, l, k.label_cut)
                              : split_label(ds, dl, D, k.label_cut);
        ev.flags = static_cast<uint16_t>(s.flags);
        ev.t_cross = t;
        ev.ds = ds;
        ev.dn = r.dn;
        ev.dl = dl;
        ev.l_first = first ? l : 0.0f;
        sink.push(ev);
        s.flags = 0;
        if (k.ideal_reset || k.refractory_ns == 0) {
          s.t_ref = t;
          r.since = t_w - t;
          r.s3 = x_hit;
          r.dn = 0.0f;
          r.dr = k.ideal_reset ? D - (on ? m.theta_on : -m.theta_off) : -k.eps_ci;
          s.t_search = t + 1 + (k.ideal_reset ? k.refractory_ns : 0);
          s.s3_ref = r.s3;
          s.n3_ref = 0.0f;
          s.dr_ref = r.dr;
          bounds = quick_record(s, m, false, T0, T_end);
        } else {
          s.blind_until = t + k.refractory_ns;
          s.t_search = s.blind_until + 1;
        }
      }
    }
  }
  if (s.n_shot != px.n_shot && later_t0 < 0 && s.t_shot < T_end) {  // no stop noted: on to the next one
    const uint32_t from = s.n_shot;
    U4 w = draw(k.seed, kPurposeShot, k.camera, pixel, s.n_shot);
    skip_rejected(k, pixel, accept_limit(m, k, S.field, raw), m.shot_max_hz, T_end, w, s.t_shot, s.n_shot);
    c.noise_candidates += s.n_shot - from;
  }
  SplitPixel& out = a.px[slot];
  out.t_ref = s.t_ref;
  out.t_search = s.t_search;
  out.blind_until = s.blind_until;
  out.t_shot = s.t_shot;
  out.t_ba = s.t_ba;
  out.s3_ref = s.s3_ref;
  out.n3_ref = s.n3_ref;
  out.dr_ref = s.dr_ref;
  out.flags = s.flags;
  out.n_shot = s.n_shot;
  out.n_ba = s.n_ba;
  if (s.n_shot != px.n_shot) {
    out.later_t[0] = later_t0;
    out.later_t[1] = later_t1;
    out.later_n[0] = later_n0;
  }
  a.q.a[slot] = quick_record(s, m, noise, T0, T_end);
  a.q.c[slot] = raw;
  // The counters, one atomic per sensor among the lanes that are here (an atomic per pixel on the few counters would
  // bound the kernel).
  for (unsigned todo = __activemask();;) {
    const int lead = __ffs(static_cast<int>(todo)) - 1;
    const uint32_t si = __shfl_sync(todo, tag & 0xFFFFu, lead);
    const bool same = (tag & 0xFFFFu) == si;
    const unsigned group = __ballot_sync(todo, same);
    if (same) {
      const uint32_t pieces = __reduce_add_sync(group, c.pieces), leaves = __reduce_add_sync(group, c.leaves);
      const uint32_t cands = __reduce_add_sync(group, c.noise_candidates);
      if (static_cast<int>(lane) == lead) {
        atomicAdd(&S.counters[kCntPieces], static_cast<unsigned long long>(pieces));
        atomicAdd(&S.counters[kCntLeaves], static_cast<unsigned long long>(leaves));
        if (cands) atomicAdd(&S.counters[kCntNoise], static_cast<unsigned long long>(cands));
      }
      break;
    }
    todo &= ~group;
  }
}

// The posted pixels of window a.w. Where the list is shorter than the launch, each warp takes fewer records (a power of
// two of its lanes), since what one pixel does hardly ever falls together with what its neighbour does. A longer list's
// warps take their next records as they get to them: a window past the stage can have a hundred times its neighbour's
// samples (1280x720, 200 blobs of 400 px/s: 20.3 ms of engine time against 49.6 by a fixed stride, and 396 with every
// blob evaluated for those windows instead of the tile's list). 128 registers (4 blocks per SM): 5.90 ms of engine time
// on 346x260, 239 windows; 6.17 at 5 blocks, 6.58 at 6.
__global__ void __launch_bounds__(128, 4) split_rest_kernel(const __grid_constant__ SplitArgs a, RestList rl) {
  const WindowTimes wt(a, a.w);
  if (a.w + 1 < a.windows) write_boxes(a, wt.t_w + kWindowNs, a.boxes_next);
  const unsigned int count = min(*rl.count, rl.capacity);
  const unsigned int warps = gridDim.x * (blockDim.x >> 5);
  const unsigned int warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
  unsigned int share = 32u;
  while (share > 1u && static_cast<uint64_t>(share / 2u) * warps >= count) share /= 2u;
  if (lane >= share) return;
  const unsigned lanes = share == 32u ? 0xffffffffu : (1u << share) - 1u;
  for (unsigned int first = warp * share; first < count;) {
    if (first + lane < count) rest_pixel(a, rl, wt, first + lane, lane);
    if (warps * share >= count) break;
    __syncwarp(lanes);
    unsigned int next = 0;
    if (lane == 0u) next = atomicAdd(rl.taken, share);
    first = warps * share + __shfl_sync(lanes, next, 0);
  }
}

// The whole call in one launch, for few tiles: a block keeps its tiles through all windows, and each window's posted
// pixels stay in the block, spread over its warps. Nothing passes between blocks, so no window waits for the slowest
// pixel of another block's, and none of the two launches per window is paid.
__global__ void __launch_bounds__(128, 4) split_solo_kernel(const __grid_constant__ SplitArgs a, RestList rl) {
  const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  __shared__ WarpShared sh[4];
  __shared__ SplitSums sums;
  __shared__ unsigned int posted;
  sums.clear();
  // This block's tiles, and its part of the list.
  const uint32_t first = blockIdx.x * a.block_tiles;
  const uint32_t end = first + a.block_tiles < a.total_tiles ? first + a.block_tiles : a.total_tiles;
  RestList mine_list = rl;
  mine_list.rec += static_cast<size_t>(first) * 32u;
  mine_list.times += static_cast<size_t>(first) * 32u;
  mine_list.count = &posted;
  mine_list.capacity = a.block_tiles * 32u;
  for (uint32_t tile = first + warp; tile < end; tile += warps) begin_tile(a, tile, lane);
  if (threadIdx.x == 0) posted = 0;
  __syncthreads();
  WarpSums mine;
  for (int32_t w = 0; w < a.windows; ++w) {
    const WindowTimes wt(a, w);
    for (uint32_t tile = first + warp; tile < end; tile += warps) {
      const int si = sensor_of(a, tile);
      mine.of(a, sums, si);
      window_tile<false>(a, mine_list, wt, sh[warp], a.sensors[si], si, tile, lane, mine.samples, mine.clean);
    }
    __syncthreads();
    const unsigned int count = posted;
    __syncthreads();
    if (threadIdx.x == 0) posted = 0;
    for (unsigned int i = warp + warps * lane; i < count; i += warps * 32u) rest_pixel(a, mine_list, wt, i, lane);
    __syncthreads();
  }
  for (uint32_t tile = first + warp; tile < end; tile += warps) end_tile(a, tile, lane);
  mine.flush(a, sums);
  __syncthreads();
  sums.add(a);
}

}  // namespace

size_t split_scratch_bytes(uint32_t total_tiles, size_t total_blobs) {
  const size_t slots = static_cast<size_t>(total_tiles) * 32u;
  return slots * (sizeof(SplitPixel) + sizeof(float4) + sizeof(float2) + sizeof(float)) +
         total_tiles * (kMaxListed * sizeof(uint16_t) + sizeof(int32_t)) + 2u * total_blobs * sizeof(float4);
}
size_t split_record_bytes() { return sizeof(RestRecord) + sizeof(RestTimes); }

void launch_engine_split(const EngineSensor* sensors_dev, const uint32_t* tile0, int n_sensors, uint32_t total_tiles,
                         size_t total_blobs, const int64_t* t0, int32_t windows, const SamplerRules& r, void* scratch,
                         void* rest, unsigned int* rest_counts, unsigned int rest_capacity, int blocks,
                         int warps_per_block, int tile_lw, int rest_blocks, bool solo, cudaStream_t stream) {
  const size_t slots = static_cast<size_t>(total_tiles) * 32u;
  SplitArgs a{};
  a.sensors = sensors_dev;
  a.n_sensors = n_sensors;
  a.total_tiles = total_tiles;
  a.t0 = t0;
  a.windows = windows;
  a.r = r;
  a.tile_lw = static_cast<uint32_t>(tile_lw);
  a.minus_zero2 = 0x8000000080000000ull;
  a.px = static_cast<SplitPixel*>(scratch);
  float4* boxes = reinterpret_cast<float4*>(a.px + slots);
  a.q.a = boxes + 2u * total_blobs;
  a.q.b = reinterpret_cast<float2*>(a.q.a + slots);
  a.q.c = reinterpret_cast<float*>(a.q.b + slots);
  a.list_n = reinterpret_cast<int32_t*>(a.q.c + slots);
  a.lists = reinterpret_cast<uint16_t*>(a.list_n + total_tiles);
  RestRecord* records = static_cast<RestRecord*>(rest);
  RestTimes* times = reinterpret_cast<RestTimes*>(records + rest_capacity);
  for (int i = 0; i < n_sensors && i < kTile0Args; ++i) a.tile0[i] = tile0[i];
  a.boxes = boxes;
  if (solo) {
    const uint32_t most = static_cast<uint32_t>(blocks);
    a.block_tiles = (total_tiles + most - 1) / most;
    const RestList rl{records, times, nullptr, nullptr, rest_capacity};
    split_solo_kernel<<<(total_tiles + a.block_tiles - 1) / a.block_tiles, warps_per_block * 32, 0, stream>>>(a, rl);
    return;
  }
  split_begin_kernel<<<(total_tiles + 3) / 4, 128, 0, stream>>>(a);
  for (int32_t w = 0; w < windows; ++w) {
    a.w = w;
    a.boxes = boxes + (w & 1) * total_blobs;
    a.boxes_next = boxes + (1 - (w & 1)) * total_blobs;
    const RestList rl{records, times, rest_counts + 2 * w, rest_counts + 2 * w + 1, rest_capacity};
    split_window_kernel<<<blocks, warps_per_block * 32, 0, stream>>>(a, rl);
    split_rest_kernel<<<rest_blocks, 128, 0, stream>>>(a, rl);
  }
  split_end_kernel<<<(total_tiles + 3) / 4, 128, 0, stream>>>(a);
}

int split_rest_blocks_per_sm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, split_rest_kernel, 128, 0);
  return n;
}
int split_solo_blocks_per_sm(int warps_per_block) {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, split_solo_kernel, warps_per_block * 32, 0);
  return n;
}
int split_window_blocks_per_sm(int warps_per_block) {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, split_window_kernel, warps_per_block * 32, 0);
  return n;
}

}  // namespace bs
