// Device helpers that the engine kernels share: event sinks, a pixel's state and map loads, warp sums, the in-place test
// of a clean segment, the noise candidates of a stretch, the out-of-line pixel model, and an engine launch's arguments.
#pragma once

#include <cooperative_groups.h>

#include "device.h"

namespace bs {

namespace cg = cooperative_groups;

namespace {  // each including file's own: the compiler fits an internal function's calls to it

// Appends events to one sensor's buffer; the lanes of a warp that push together share one atomic, so every lane of
// the warp must push to the same buffer (a warp works on one tile of one sensor).
struct GlobalSink {
  EventBuf ev;
  unsigned long long* count;
  __device__ __forceinline__ void push(const RawEvent& e) {
    cg::coalesced_group g = cg::coalesced_threads();
    unsigned long long base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(count, static_cast<unsigned long long>(g.size()));
    base = g.shfl(base, 0);
    const unsigned long long i = base + g.thread_rank();
    if (i < ev.capacity) {
      const uint4* src = reinterpret_cast<const uint4*>(&e);
      uint4* dst = reinterpret_cast<uint4*>(ev.data + i);
      dst[0] = src[0];
      dst[1] = src[1];
    }
  }
};

// Appends each event with the pushing thread's own atomic: for a kernel whose lanes serve pixels of different
// sensors (split_rest_kernel).
struct ThreadSink {
  EventBuf ev;
  unsigned long long* count;
  __device__ __forceinline__ void push(const RawEvent& e) {
    const unsigned long long i = atomicAdd(count, 1ull);
    if (i < ev.capacity) {
      const uint4* src = reinterpret_cast<const uint4*>(&e);
      uint4* dst = reinterpret_cast<uint4*>(ev.data + i);
      dst[0] = src[0];
      dst[1] = src[1];
    }
  }
};

__device__ __forceinline__ void load_state(const StateSoA& a, uint32_t p, bool noise, PixelRegs& s) {
  s.t_ref = a.t_ref[p];
  s.t_search = a.t_search[p];
  s.blind_until = a.blind_until[p];
  s.s3_ref = a.s3_ref[p];
  s.n3_ref = a.n3_ref[p];
  s.dr_ref = a.dr_ref[p];
  s.i_scale = a.i_scale[p];
  s.held = a.held[p];
  s.flags = a.flags[p];
  if (noise) {
    s.t_shot = a.t_shot[p];
    s.t_ba = a.t_ba[p];
    s.n_shot = a.n_shot[p];
    s.n_ba = a.n_ba[p];
  } else {
    s.t_shot = s.t_ba = kForever;
    s.n_shot = s.n_ba = 0;
  }
}

__device__ __forceinline__ void store_state(const StateSoA& a, uint32_t p, bool noise, const PixelRegs& s) {
  a.t_ref[p] = s.t_ref;
  a.t_search[p] = s.t_search;
  a.blind_until[p] = s.blind_until;
  a.s3_ref[p] = s.s3_ref;
  a.n3_ref[p] = s.n3_ref;
  a.dr_ref[p] = s.dr_ref;
  a.i_scale[p] = s.i_scale;
  a.held[p] = s.held;
  a.flags[p] = s.flags;
  if (noise) {
    a.t_shot[p] = s.t_shot;
    a.t_ba[p] = s.t_ba;
    a.n_shot[p] = s.n_shot;
    a.n_ba[p] = s.n_ba;
  }
}

__device__ __forceinline__ void load_cascade(const StateSoA& a, uint32_t p, CascadeRegs& q) {
  q.z = a.z[p];
  q.x1 = a.x1[p];
  q.s2 = a.s2[p];
  q.s3 = a.s3[p];
  q.tv = a.tv[p];
}

__device__ __forceinline__ void store_cascade(const StateSoA& a, uint32_t p, const CascadeRegs& q) {
  a.z[p] = q.z;
  a.x1[p] = q.x1;
  a.s2[p] = q.s2;
  a.s3[p] = q.s3;
  a.tv[p] = q.tv;
}

__device__ __forceinline__ void load_lattice(const StateSoA& a, uint32_t p, uint32_t n, LatticeRegs& L) {
  for (int i = 0; i < 3; ++i) {
    L.nk[i] = a.lat[static_cast<size_t>(i) * n + p];
    L.nk1[i] = a.lat[static_cast<size_t>(3 + i) * n + p];
  }
  L.ln_a1 = a.lat[static_cast<size_t>(6) * n + p];
  L.rho = a.lat[static_cast<size_t>(7) * n + p];
  L.cell = a.cell[p];
  L.have_k1 = a.have_k1[p];
}

__device__ __forceinline__ void store_lattice(const StateSoA& a, uint32_t p, uint32_t n, const LatticeRegs& L) {
  for (int i = 0; i < 3; ++i) {
    a.lat[static_cast<size_t>(i) * n + p] = L.nk[i];
    a.lat[static_cast<size_t>(3 + i) * n + p] = L.nk1[i];
  }
  a.lat[static_cast<size_t>(6) * n + p] = L.ln_a1;
  a.lat[static_cast<size_t>(7) * n + p] = L.rho;
  a.cell[p] = L.cell;
  a.have_k1[p] = L.have_k1;
}

// Drops events (the init of the noise lattice fires nothing).
struct NullSink {
  __device__ void push(const RawEvent&) {}
};

__device__ __forceinline__ void load_map(const MapSoA& m, uint32_t p, PixelMapRegs& r) {
  r.theta_on = m.theta_on[p];
  r.theta_off = m.theta_off[p];
  r.leak = m.leak[p];
  r.dark = m.dark[p];
  r.scale = m.scale[p];
  r.ba_rate_hz = m.ba_rate[p];
  r.shot_max_hz = m.shot_max[p];
}

// Sums a value over the warp and adds it to a counter from lane 0 (all 32 lanes must call).
__device__ __forceinline__ void warp_add(unsigned long long* dst, unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v != 0ull) atomicAdd(dst, v);
}
__device__ __forceinline__ void warp_or(unsigned long long* dst, unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v != 0ull) atomicOr(dst, v);
}

// Would PixelProc::segment_fast pass segment [t0, e) with nothing but its clean effects (the piece counted, the
// search moved to e, a node counted when e - t0 > 2)? Only where it takes that branch: one 2^23 ns piece, the pixel
// not blind, its search armed at or before t0, no noise candidate before e, Delta(t0) below both levels, and the
// node (t0, e - 1] a single integer or excluded. Inline code on the caller's registers.
__device__ __forceinline__ bool clean_segment(const PixelRegs& s, const PixelMapRegs& m, const SensorConsts& k,
                                              int64_t t0, int64_t e, float v0, float v1, float x0, float x1) {
  if (((e - 1) >> kWindowLog2) != (t0 >> kWindowLog2)) return false;
  if (s.blind_until != kNotBlind || s.t_search > t0) return false;
  const int64_t tn = k.noise ? mini(s.t_shot, s.t_ba) : kForever;
  if (tn < e) return false;
  NullSink ns;
  PixelCounters nc;
  const PixelProc<NullSink> hp{const_cast<PixelRegs&>(s), m, k, 0u, ns, nc};
  const float D0 = hp.delta(t0, x0);
  if (D0 >= m.theta_on || D0 <= -m.theta_off) return false;
  if (e - t0 == 1) return true;
  return hp.excluded(Segment{t0, e, v0, v1}, t0, e, x0, x1);
}

// clean_segment's other case, for a segment it refused: the search armed after t0 (the first segment after init, or
// the segment of an event), where PixelProc::piece searches [t_search, e) alone, without Delta(t0); clean when
// nothing is left to search or the node (t0, e - 1] around it is excluded (the same effects).
__device__ __forceinline__ bool clean_after_start(const PixelRegs& s, const PixelMapRegs& m, const SensorConsts& k,
                                                  int64_t t0, int64_t e, float v0, float v1, float x0, float x1) {
  if (((e - 1) >> kWindowLog2) != (t0 >> kWindowLog2)) return false;
  if (s.blind_until != kNotBlind || s.t_search <= t0) return false;
  const int64_t tn = k.noise ? mini(s.t_shot, s.t_ba) : kForever;
  if (tn < e) return false;
  if (s.t_search >= e) return true;
  NullSink ns;
  PixelCounters nc;
  const PixelProc<NullSink> hp{const_cast<PixelRegs&>(s), m, k, 0u, ns, nc};
  return hp.excluded(Segment{t0, e, v0, v1}, t0, e, x0, x1);
}

// The noise candidates of a stretch [t_from, t_end) of every lane's pixel, computed with all 32 lanes together.
// A candidate that thinning rejects changes nothing but its chain (PixelProc::noise_candidate), and its acceptance
// depends only on its draw and the irradiance at its time, which the stretch's samples give: so each lane's chains
// move past their rejected candidates here, and stop at their first accepted candidate in the stretch (or at their
// first candidate after it). The pixel model then meets only accepted candidates, at which it runs its own noise
// path (the draw and the thinning test again, the refractory drop, the event) and follows the chains from there as
// usual. Events and the chains' end state are those of the pixel model meeting every candidate; only the count of
// the crossing search's nodes differs, since the search is no longer cut at rejected candidates (the first crossing
// is the same: a time-ordered search over [lo, e) finds what searches over [lo, tn) then [tn, e) find).
// active: this lane's stretch is in `run` (run.n samples after the one held at t_from, run.t(j) / run.v_at(j), raw
// values clamped here as the pixel model clamps them). All lanes of the warp call it.
template <class Run>
__device__ __forceinline__ void noise_ahead(PixelRegs& s, const PixelMapRegs& m, const SensorConsts& k,
                                            uint32_t pixel, bool active, int64_t t_from, float v_held,
                                            int64_t t_end, const Run& run, PixelCounters& c) {
  bool done_shot = !active, done_ba = !active;
  for (;;) {
    const bool p_shot = !done_shot && s.t_shot < t_end, p_ba = !done_ba && s.t_ba < t_end;
    if (!__any_sync(0xffffffffu, p_shot || p_ba)) break;
    if (!(p_shot || p_ba)) continue;
    const bool shot = p_shot && (!p_ba || s.t_shot <= s.t_ba);
    const int64_t tn = shot ? s.t_shot : s.t_ba;
    const uint32_t purpose = shot ? kPurposeShot : kPurposeBackground;
    const uint32_t nidx = shot ? s.n_shot : s.n_ba;
    // The segment holding tn: [t_a, t_b) between consecutive samples, or held after the last one.
    int64_t ta = t_from;
    float va = v_held;
    int64_t tb = kForever;
    float vb = va;
    for (int j = 0; j < run.n; ++j) {
      const int64_t tj = run.t(j);
      const float vj = clamp_irr(run.v_at(j), k.irr_max);
      if (tj > tn) {
        tb = tj;
        vb = vj;
        break;
      }
      ta = tj;
      va = vj;
    }
    if (tb == kForever) vb = va;
    const U4 w = draw(k.seed, purpose, k.camera, pixel, nidx);
    NullSink ns;
    PixelCounters nc;
    const PixelProc<NullSink> hp{s, m, k, pixel, ns, nc};
    const float I = hp.current(Segment{ta, tb, va, vb}, tn);
    const double accept = shot ? sqrt(static_cast<double>(m.dark) / static_cast<double>(I)) : 1.0;
    if (open_uniform_d(w.v[1]) < accept) {
      if (shot) done_shot = true;
      else done_ba = true;
      continue;
    }
    ++c.noise_candidates;
    const int64_t next = noise_next(k.seed, purpose, k.camera, pixel, nidx + 1, tn, shot ? m.shot_max_hz : m.ba_rate_hz);
    if (shot) {
      s.n_shot = nidx + 1;
      s.t_shot = next;
    } else {
      s.n_ba = nidx + 1;
      s.t_ba = next;
    }
  }
}

// A lane's window staged in shared memory (dt / v strided by 32 lanes) as noise_ahead's run.
struct StagedRun {
  int64_t t_w;
  const uint32_t* dt;
  const float* v;
  int n;
  __device__ __forceinline__ int64_t t(int j) const { return t_w + dt[j * 32]; }
  __device__ __forceinline__ float v_at(int j) const { return v[j * 32]; }
};
// A CSR run in device memory as noise_ahead's run.
struct GlobalRun {
  const int64_t* tp;
  const float* vp;
  int n;
  __device__ __forceinline__ int64_t t(int j) const { return __ldg(tp + j); }
  __device__ __forceinline__ float v_at(int j) const { return __ldg(vp + j); }
};

// x = ln(I / i_scale) at a sample of value v (PixelProc::x_at_sample on the caller's registers).
__device__ __forceinline__ float x_sample(const PixelRegs& s, const PixelMapRegs& m, float v) {
  return log_f((m.dark + m.scale * v) / s.i_scale);
}

// The pixel model's full path on a state in memory, out of line: the hot loops keep the state in registers and copy
// it here only for a segment that is not clean. fast: PixelProc::segment_fast with x at both ends; else
// PixelProc::segment over [from, to).
// kFlat: the processor's rare paths inline here, on copies the compiler can keep in registers (one large function:
// the CSR kernel and the streaming engine); else they stay separate out-of-line functions working on the state in
// memory (smaller code: the staged engine, whose instruction footprint sets its speed).
template <class Sink, bool kFlat>
__device__ __noinline__ void cold_segment(PixelRegs* s, const PixelMapRegs* m, const SensorConsts* k, uint32_t pixel,
                                          Sink sink, PixelCounters* c, Segment g, int64_t from, int64_t to, bool fast,
                                          float x0, float x1) {
  PixelRegs sl = *s;
  const PixelMapRegs ml = *m;
  PixelCounters cl = *c;
  PixelProc<Sink, kFlat> proc{sl, ml, *k, pixel, sink, cl};
  if (fast) proc.segment_fast(g, x0, x1);
  else proc.segment(g, from, to);
  *s = sl;
  *c = cl;
}

// One segment [t0, t1) of a pixel whose state is in registers: the clean outcome in place, anything else out of line.
template <bool kFlat = true, class Sink>
__device__ __forceinline__ void feed_segment(PixelRegs& s, const PixelMapRegs& m, const SensorConsts& k,
                                             const SensorConsts* kd, uint32_t pixel, const Sink& sink,
                                             PixelCounters& c, int64_t t0, int64_t t1, float v0, float v1, float x0,
                                             float x1) {
  if (clean_segment(s, m, k, t0, t1, v0, v1, x0, x1)) {
    ++c.pieces;
    if (t1 - t0 > 2) ++c.leaves;
    s.t_search = maxi(s.t_search, t1);
    return;
  }
  const Segment g{t0, t1, v0, v1};
  const bool fast = ((t1 - 1) >> kWindowLog2) == (t0 >> kWindowLog2);
  PixelRegs ts = s;
  PixelMapRegs tm = m;
  PixelCounters tc = c;
  cold_segment<Sink, kFlat>(&ts, &tm, kd, pixel, sink, &tc, g, t0, t1, fast, x0, x1);
  s = ts;
  c = tc;
}

// The held sample from t_from to t_end (the end of a call), out of line where there is such a stretch.
template <class Sink>
__device__ __forceinline__ void feed_held(PixelRegs& s, const PixelMapRegs& m, const SensorConsts* kd, uint32_t pixel,
                                          const Sink& sink, PixelCounters& c, int64_t t_from, float v,
                                          int64_t t_end) {
  if (t_from >= t_end) return;
  PixelRegs ts = s;
  PixelMapRegs tm = m;
  PixelCounters tc = c;
  cold_segment<Sink, true>(&ts, &tm, kd, pixel, sink, &tc, Segment{t_from, kForever, v, v}, t_from, t_end, false, 0.0f,
                           0.0f);
  s = ts;
  c = tc;
}

struct EngineArgs {
  const EngineSensor* sensors;
  int n_sensors;
  uint32_t total_tiles;
  const int64_t* t0;  // the model time, in device memory (a captured launch replays at any time)
  int32_t w0, w1;
  SamplerRules r;
  unsigned int* tile_counter;
  uint32_t tile_lw;   // log2 of the tile width: tiles of 2^lw x 2^(5 - lw) pixels, one warp each
};

// The pixel of `lane` in tile `local` of a sensor with tiles_x tiles per row.
__device__ __forceinline__ void tile_xy(uint32_t local, uint32_t tiles_x, uint32_t lw, uint32_t lane, uint32_t& x,
                                        uint32_t& y) {
  x = (local % tiles_x) * (1u << lw) + (lane & ((1u << lw) - 1u));
  y = (local / tiles_x) * (32u >> lw) + (lane >> lw);
}

// Feeds a window's samples, in time order, to the pixel model: every segment lies inside the window, so each
// takes the fast path with x at both ends, each x computed once.
struct WindowFeed {
  PixelProc<GlobalSink>* proc;
  int64_t t_w;
  float irr_max;
  int64_t prev_t;
  float prev_v;
  float last_raw;
  float x_prev;
  // Slot 0, the carried sample, sits at the model time: it replaces the held one.
  __device__ __forceinline__ void start(float carried) {
    last_raw = carried;
    prev_v = clamp_irr(carried, irr_max);
    x_prev = proc->x_at_sample(prev_v);
  }
  __device__ __forceinline__ void operator()(uint32_t dt, float v) {
    last_raw = v;
    const float vc = clamp_irr(v, irr_max);
    const int64_t t = t_w + dt;
    const float x1 = proc->x_at_sample(vc);
    proc->segment_fast(Segment{prev_t, t, prev_v, vc}, x_prev, x1);
    prev_t = t;
    prev_v = vc;
    x_prev = x1;
  }
};

// WindowFeed for a pixel whose state stays in the caller's registers (s, m, c): each segment's clean outcome is taken
// in place, anything else out of line (feed_segment<kFlat>); the same samples and state as WindowFeed's.
template <bool kFlat, class Sink = GlobalSink>
struct RegFeed {
  PixelRegs& s;
  const PixelMapRegs& m;
  PixelCounters& c;
  const SensorConsts& k;
  const SensorConsts* kd;
  uint32_t pixel;
  Sink sink;
  int64_t t_w;
  int64_t prev_t;
  float prev_v;
  float last_raw;
  float x_prev;
  __device__ __forceinline__ void start(float carried) {
    last_raw = carried;
    prev_v = clamp_irr(carried, k.irr_max);
    x_prev = x_sample(s, m, prev_v);
  }
  __device__ __forceinline__ void operator()(uint32_t dt, float v) {
    last_raw = v;
    const float vc = clamp_irr(v, k.irr_max);
    const int64_t t = t_w + dt;
    const float x1 = x_sample(s, m, vc);
    feed_segment<kFlat>(s, m, k, kd, pixel, sink, c, prev_t, t, prev_v, vc, x_prev, x1);
    prev_t = t;
    prev_v = vc;
    x_prev = x1;
  }
};

// ---------------------------------------------------------------------------------------------
// Quiet windows and noise stops (the split engine's header comment says what they are for)
// ---------------------------------------------------------------------------------------------
// The extremes of a window's samples: a NaN stays in both, so no bound holds for it.
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// The quick record's bounds from the state. Delta = ln(I / i_scale) - s3 - n3 + (leak (t - t_ref) 1e-9 + dr), so it
// stays below theta_on while log2 I < upper - leak log2(e) (t - T0), and above -theta_off alike. The slack, 2e-5 of the
// sum of the terms' magnitudes, is over 20 times what the roundings of Delta (four fp32 operations, log_f, the
// division) and of this evaluation (lg2.approx: 2^-22) add up to.
__device__ __forceinline__ float4 quick_record(const PixelRegs& s, const PixelMapRegs& m, bool noise, int64_t T0,
                                               int64_t T_end) {
  const float log2e = 1.4426950408889634f;
  const float drift = m.leak * since_ref(T0, s.t_ref);
  const float span = m.leak * static_cast<float>(static_cast<double>(T_end - T0) * 1e-9);
  const float c = ((s.s3_ref + s.n3_ref) - s.dr_ref) - drift;
  const float mag = 4.0f + fabs_f(s.s3_ref) + fabs_f(s.n3_ref) + fabs_f(s.dr_ref) + fabs_f(drift) + fabs_f(span) +
                    m.theta_on + m.theta_off;
  const float slack = 2.0e-5f * mag;
  const float li = __log2f(s.i_scale);
  float4 q;
  q.x = (c + m.theta_on - slack) * log2e + li - 1.0e-6f * fabs_f(li);
  q.y = (c - m.theta_off + slack) * log2e + li + 1.0e-6f * fabs_f(li);
  q.z = m.leak * log2e;
  int32_t gate = INT32_MAX;
  if (noise) {
    const int64_t tn = mini(s.t_shot, s.t_ba);
    if (tn < T_end) gate = static_cast<int32_t>((tn - T0) >> kWindowLog2);
  }
  if (s.blind_until != kNotBlind || !(mag < 1.0e3f)) gate = INT32_MIN;
  q.w = __int_as_float(gate);
  return q;
}

// Shot candidate n is accepted when its u1 < sqrt(I_dk / I) (PixelProc::candidate_accepted). Every photocurrent of the
// pixel in the call is at least that of the least sample (the field's lower bound or the carried sample; the
// interpolation's rounding, relative to the largest sample, taken off), so a candidate whose u1 is at or above the root
// there is rejected whenever it comes, and changes nothing but its chain. The largest word of u1 that may be accepted:
__device__ __forceinline__ uint32_t accept_limit(const PixelMapRegs& m, const SensorConsts& k, const FieldDev& f,
                                                 float carried) {
  const float v0 = clamp_irr(carried, k.irr_max);
  const float lo = minr(v0, clamp_irr(f.lo, k.irr_max)), hi = maxr(v0, clamp_irr(f.hi, k.irr_max));
  const float v = maxr(0.0f, lo - 0x1p-21f * hi);
  const float I = m.dark + m.scale * v;
  const double root = sqrt(static_cast<double>(m.dark) / static_cast<double>(I));
  const double bound = root * 0x1p32 + 2.0;  // u1 = (word + 1/2) 2^-32 < root only where word < bound
  return bound < 0x1p32 - 1.0 ? static_cast<uint32_t>(bound) : 0xFFFFFFFFu;
}
// From the chain's candidate n at t (w its draw) to its next stop: the first candidate that may be accepted, or the
// first at or after t_end.
__device__ __forceinline__ void skip_rejected(const SensorConsts& k, uint32_t pixel, uint32_t limit, double rate_hz,
                                              int64_t t_end, U4& w, int64_t& t, uint32_t& n) {
  while (t < t_end && w.v[1] > limit) {
    ++n;
    w = draw(k.seed, kPurposeShot, k.camera, pixel, n);
    t = noise_after(w, t, rate_hz);
  }
}

}  // namespace

}  // namespace bs
