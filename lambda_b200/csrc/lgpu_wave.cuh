// lgpu_wave.cuh — streaming wavefront path tracing.
//
// Paths in flight live in queue order: path i of the current queue keeps
// its state at index i of the `in` buffers (field-major, so a warp's access
// to one field is one coalesced transaction).  Each iteration
//
//   wf_plan               how many new paths fit behind the queue
//   wf_generate_stream<K> camera ray + hero wavelengths of the new paths,
//                         appended to the queue
//   wf_trace_*            closest hit of every queued path
//   wf_shade<K>           adds the last vertex's light sample if its shadow
//                         ray got through; emitters, light sample -> shadow
//                         ray, material sample -> next ray; a continuing
//                         path is written to the next position of the `out`
//                         queue, an ended one to the ended list
//   wf_shadow / wf_trace_persistent<true>
//                         any-hit test of the shadow rays: one visibility
//                         byte per ray
//   wf_finish<K>          ended paths (with the light sample of their last
//                         vertex if its shadow ray got through) -> XYZ of
//                         their (sample, pixel) film entry
//
// the last two on a second stream, beside the next iteration's plan, new
// paths and closest hits (its shading waits for them);
// then the host swaps `in` and `out`.  No path keeps a fixed slot, so no
// access is scattered.  Each path draws its random numbers from its own
// counter-based stream in the order of Renderer::tracePath
// (src/renderer.cpp:64-146), and each (sample, pixel) result has its own
// film entry summed in sample order, so the image does not depend on how
// paths are scheduled.  Queue appends take one atomic per warp (ballot +
// popc).
#pragma once

#include "lgpu_counters.cuh"
#include "lgpu_path.cuh"
#include "lgpu_traverse.cuh"

namespace lgpu {

__device__ __forceinline__ uint32_t warp_append(uint32_t* counter, bool pred) {
  unsigned const mask = __activemask();
  unsigned const b = __ballot_sync(mask, pred);
  int const lane = threadIdx.x & 31;
  int const leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader && b) base = atomicAdd(counter, __popc(b));
  base = __shfl_sync(mask, base, leader);
  return base + __popc(b & ((1u << lane) - 1u));
}

// The ray of path or shadow ray i from its two words (its second word's
// other half: hero wavelength and depth, or distance bound and object to skip).
__device__ __forceinline__ Ray make_ray(float4 a, float4 b) {
  return make_ray(f3{a.x, a.y, a.z}, f3{a.w, b.x, b.y});
}
__device__ __forceinline__ Ray load_ray(const float4* ra, const float4* rb, uint32_t i) {
  return make_ray(ra[i], rb[i]);
}
// Hit records: the object (UINT32_MAX on a miss) and, for a hit, two
// 16-byte words, so that a closer hit is recorded by two stores and read
// back by two loads wherever the path lies in the queue.
__device__ __forceinline__ void store_hit_point(const WaveState& w, uint32_t p, uint32_t face, float b0, float b1,
                                                float b2, f3 pl, float z) {
  w.hita[p] = make_float4(__uint_as_float(face), b0, b1, b2);
  w.hitb[p] = make_float4(pl.x, pl.y, pl.z, z);
}
__device__ __forceinline__ void store_hit(const WaveState& w, uint32_t p, const HitRec& h) {
  w.hobj[p] = h.obj;
  if (h.obj != UINT32_MAX) store_hit_point(w, p, h.face, h.b0, h.b1, h.b2, h.pl, h.z);
}
// the record of a path that hit object `obj`
__device__ __forceinline__ HitRec load_hit(const float4* hita, const float4* hitb, size_t p, uint32_t obj) {
  float4 const a = hita[p], b = hitb[p];
  HitRec h;
  h.obj = obj;
  h.z = b.w;
  h.face = __float_as_uint(a.x);
  h.b0 = a.y;
  h.b1 = a.z;
  h.b2 = a.w;
  h.pl = f3{b.x, b.y, b.z};
  return h;
}

__device__ __forceinline__ void clear_hit(HitRec& h, float z) {
  h.z = z;
  h.obj = UINT32_MAX;
  h.face = UINT32_MAX;
  h.b0 = h.b1 = h.b2 = 0.f;
  h.pl = f3{0.f, 0.f, 0.f};
}

// The non-template kernels get internal linkage: every translation unit
// that instantiates the renderer carries its own copy.
namespace {

// ---- streaming scheduler ------------------------------------------------------------

// Empty queue, no work handed out, nothing ended.
__global__ void wf_stream_init(WaveState w) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *w.n_in = 0;
    *w.n_out = 0;
    w.ctl[kCtlNext] = 0;
  }
}

// Plans the next generate (as many new paths as fit behind the queue, up to
// the remaining work items) and clears the iteration's counters.  The other
// counters of the pairs may still be in use by the last iteration.
__global__ void wf_plan(WaveState w, uint32_t total) {
  uint32_t const n_in = *w.n_in, next = w.ctl[kCtlNext];
  uint32_t const room = w.cap - n_in;
  uint32_t const left = total - next;
  uint32_t const n_new = room < left ? room : left;
  w.ctl[kCtlNew] = n_new;
  w.ctl[kCtlFirst] = next;
  w.ctl[kCtlPos] = n_in;
  w.ctl[kCtlNext] = next + n_new;
  *w.n_in = n_in + n_new;
  *w.n_out = 0;
  w.ctl[kCtlShadow + w.par] = 0;
  w.ctl[kCtlFetch] = 0;
  w.ctl[kCtlSFetch + w.par] = 0;
  w.ctl[kCtlFallback] = 0;
  w.ctl[kCtlLoopFetch] = 0;
  w.ctl[kCtlEnded + w.par] = 0;
  w.ctl[kCtlListB] = 0;
  w.ctl[kCtlListT] = 0;
  w.ctl[kCtlListL] = 0;
}

// Starts the planned paths at the end of the queue: work item q is sample
// q / npix of pixel q % npix (all pixels of one sample before the next).
// Camera ray and hero wavelength as sample::camera and sample::spectrum
// (cg.hpp:1534-1542, 1517-1531), random numbers drawn in the order of
// Renderer::render (src/renderer.cpp:33-41).
template <int K, class J>
__global__ void __launch_bounds__(256) wf_generate_stream(J jobs, WaveState w, DevCounters* cnt) {
  uint32_t const n_new = w.ctl[kCtlNew], first = w.ctl[kCtlFirst], pos = w.ctl[kCtlPos];
  uint32_t paths = 0;
  PathBuf const& in = w.in;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_new; k += gridDim.x * blockDim.x) {
    uint32_t const q = first + k;
    uint64_t const g = w.c0 + q;
    uint32_t const jb = jobs.job_of_item(g);
    const DevScene& S = jobs.scene(jb);
    const RenderArgs& a = jobs.args(jb);
    uint32_t const npix = jobs.npix_of(jb);
    uint64_t const l = g - jobs.item_base(jb);
    uint32_t const sample = uint32_t(l / npix);
    uint32_t const pix = jobs.frame_pixel(jb, uint32_t(l - uint64_t(sample) * npix));
    uint32_t const p = pos + k;
    float const omega = S.lambda_sup - S.lambda_inf;
    const lgpu_camera& C = S.cam;
    uint32_t const W = uint32_t(C.width);
    uint32_t const i = pix / W, j = pix - i * W;
    uint64_t rng = lgpu_path_state(a.seed, (uint64_t(a.stream_tag) << 32) | pix,
                                   uint64_t(a.spp_offset) + sample);
    float const u = float(j) + lgpu_flt(&rng);
    float const v = float(i) + lgpu_flt(&rng);
    f3 const Fx = f3{C.base_x[0], C.base_x[1], C.base_x[2]};
    f3 const Fy = f3{C.base_y[0], C.base_y[1], C.base_y[2]};
    f3 const Fz = f3{C.base_z[0], C.base_z[1], C.base_z[2]};
    f3 const P = f3{C.pos[0], C.pos[1], C.pos[2]};
    float const cu = -0.5f * C.w + C.delta * u;
    float const cv = -0.5f * C.h + C.delta * v;
    f3 const wij = f3{P.x + Fx.x * cu + Fy.x * cv - C.D * Fz.x, P.y + Fx.y * cu + Fy.y * cv - C.D * Fz.y,
                      P.z + Fx.z * cu + Fy.z * cv - C.D * Fz.z};
    float const la = lgpu_flt(&rng) - 0.5f;
    float const lb = lgpu_flt(&rng) - 0.5f;
    float const dd = 2.f * C.dof;
    f3 const wkl = f3{P.x + dd * (Fx.x * la + Fy.x * lb), P.y + dd * (Fx.y * la + Fy.y * lb),
                      P.z + dd * (Fx.z * la + Fy.z * lb)};
    f3 const dir = fnorm(f3{wij.x - wkl.x, wij.y - wkl.y, wij.z - wkl.z});
    float const hero = S.lambda_inf + omega * lgpu_flt(&rng);
    in.ra[p] = make_float4(wkl.x, wkl.y, wkl.z, dir.x);
    in.rb[p] = make_float4(dir.y, dir.z, hero, __uint_as_float(0u));
    in.rc[p] = make_uint4(uint32_t(rng), uint32_t(rng >> 32), q, kNoShadow);
    if (J::kMulti) in.job[p] = jb;
    if (w.vis) w.vis[q] = 0;
    // no spectral state: a path at depth 0 has throughput 1 and no
    // radiance, which the shading kernel supplies (frame +1.8 % measured)
    paths++;
  }
  TravStats const ts{0u, 0u, 0u, 0u};
  flush_counters(cnt, 0u, paths, ts, 0u);
}

// Ended paths: radiance splatted to XYZ (addHeroλ(λ, Li/prob),
// src/renderer.cpp:44) into the path's (sample, pixel) film entry.  Bound by
// issue (62 %): four wavelengths per word and loop body (40 registers; all
// 16 unrolled took 64 and 23 % more time), divisions by the two constants as
// div_by.  Benchmark frame: 16.0 -> 11.2 ms.
template <int K, class J>
__global__ void __launch_bounds__(256) wf_finish(J jobs, WaveState w, DevCounters* cnt) {
  uint32_t const n = w.ctl[kCtlEnded + w.par];
  uint32_t const cap = w.cap;
  uint32_t nonfinite = 0;
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    uint4 const rec = w.e_rec[e];
    const DevScene& S = jobs.scene(J::kMulti ? rec.w : 0u);
    float const omega = S.lambda_sup - S.lambda_inf;
    float const step = omega / float(K);
    float const prob_l = 1.f / omega;
    float const hero = __uint_as_float(rec.x);
    // the light sample of the path's last vertex, if its shadow ray got through
    uint32_t const sx_i = rec.z;
    bool const lit = sx_i != kNoShadow && w.s_vis[sx_i];
    float sx = 0.f, sy = 0.f, sz = 0.f;
    bool finite = true;
#pragma unroll 1
    for (int q = 0; q < K / 4; q++) {
      float4 const a4 = w.e_acc[q * cap + e];
      float4 const p4 = lit ? w.s_contrib[q * cap + sx_i] : make_float4(0.f, 0.f, 0.f, 0.f);
      float acc[4] = {a4.x, a4.y, a4.z, a4.w};
      float const pend[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (lit) acc[j] += pend[j];
        float const val = div_by_guarded(acc[j], prob_l, S.prob_lambda_rcp);
        finite = finite && isfinite(val);
        splat_xyz(S, hero_lambda(S, hero, step, 4 * q + j), val, sx, sy, sz);
      }
      if (w.ltot) w.ltot[size_t(rec.y) * (K / 4) + q] = make_float4(acc[0], acc[1], acc[2], acc[3]);
    }
    nonfinite += finite ? 0u : 1u;
    size_t const o = 3 * size_t(rec.y);
    w.sbuf[o] = sx;
    w.sbuf[o + 1] = sy;
    w.sbuf[o + 2] = sz;
  }
  TravStats const ts{0u, 0u, 0u, 0u};
  flush_counters(cnt, 0u, 0u, ts, nonfinite);
}

// Film: per pixel, the (sample, pixel) entries of the chunk [w.c0, c1)
// added in sample order.
template <class J>
__global__ void __launch_bounds__(256) wf_reduce(J jobs, WaveState w, uint64_t c1) {
  for (uint32_t gp = blockIdx.x * blockDim.x + threadIdx.x; gp < w.npix; gp += gridDim.x * blockDim.x) {
    uint32_t const jb = jobs.job_of_pixel(gp);
    uint32_t const npix = jobs.npix_of(jb);
    uint64_t const base = jobs.item_base(jb) + (gp - jobs.pix_base(jb));
    uint32_t const spp = jobs.args(jb).spp;
    // samples s with w.c0 <= base + s * npix < c1
    uint64_t const lo = w.c0 > base ? (w.c0 - base + npix - 1) / npix : 0;
    uint64_t hi = c1 > base ? (c1 - base + npix - 1) / npix : 0;
    if (hi > spp) hi = spp;
    if (lo >= hi) continue;
    if (w.film64) {
      // the FP64 film: the same samples in the same order, summed in double
      double* const f = w.film64 + 3 * size_t(gp);
      double X = f[0], Y = f[1], Z = f[2];
      for (uint64_t s = lo; s < hi; s++) {
        size_t const o = 3 * size_t(base + s * npix - w.c0);
        X += double(w.sbuf[o]);
        Y += double(w.sbuf[o + 1]);
        Z += double(w.sbuf[o + 2]);
      }
      f[0] = X;
      f[1] = Y;
      f[2] = Z;
      continue;
    }
    float X = w.film[3 * size_t(gp)], Y = w.film[3 * size_t(gp) + 1], Z = w.film[3 * size_t(gp) + 2];
    for (uint64_t s = lo; s < hi; s++) {
      size_t const o = 3 * size_t(base + s * npix - w.c0);
      X += w.sbuf[o];
      Y += w.sbuf[o + 1];
      Z += w.sbuf[o + 2];
    }
    w.film[3 * size_t(gp)] = X;
    w.film[3 * size_t(gp) + 1] = Y;
    w.film[3 * size_t(gp) + 2] = Z;
  }
}

// XYZ film / (spp * K) * Δ -> linear BT.709 RGB in the reference's layout
// (row 0 at the top), src/renderer.cpp:52-56, cg.hpp:144-148, 340-341.
template <int K, class J>
__global__ void __launch_bounds__(256) wf_finalize(J jobs, WaveState w) {
  for (uint32_t gp = blockIdx.x * blockDim.x + threadIdx.x; gp < w.npix; gp += gridDim.x * blockDim.x) {
    uint32_t const jb = jobs.job_of_pixel(gp);
    const DevScene& S = jobs.scene(jb);
    uint32_t const pix = jobs.frame_pixel(jb, gp - jobs.pix_base(jb));
    uint32_t const W = uint32_t(S.cam.width), H = uint32_t(S.cam.height);
    uint32_t const i = pix / W, j = pix - i * W;
    if (w.film64) {
      // double throughout, into an output of doubles
      double const nd = double(jobs.args(jb).spp) * double(K);
      double const X = w.film64[3 * size_t(gp)] / nd * double(S.lambda_delta);
      double const Y = w.film64[3 * size_t(gp) + 1] / nd * double(S.lambda_delta);
      double const Z = w.film64[3 * size_t(gp) + 2] / nd * double(S.lambda_delta);
      double* o = reinterpret_cast<double*>(jobs.out_of(jb)) + (size_t(H - i - 1) * W + j) * 3;
      o[0] = 3.2404542 * X - 1.5371385 * Y - 0.4985314 * Z;
      o[1] = -0.9692660 * X + 1.8760108 * Y + 0.0415560 * Z;
      o[2] = 0.0556434 * X - 0.2040259 * Y + 1.0572252 * Z;
      continue;
    }
    float const norm = float(jobs.args(jb).spp) * float(K);
    float const X = (w.film[3 * size_t(gp)] / norm) * S.lambda_delta;
    float const Y = (w.film[3 * size_t(gp) + 1] / norm) * S.lambda_delta;
    float const Z = (w.film[3 * size_t(gp) + 2] / norm) * S.lambda_delta;
    float* out = jobs.out_of(jb) + (size_t(H - i - 1) * W + j) * 3;
    out[0] = 3.2404542f * X - 1.5371385f * Y - 0.4985314f * Z;
    out[1] = -0.9692660f * X + 1.8760108f * Y + 0.0415560f * Z;
    out[2] = 0.0556434f * X - 0.2040259f * Y + 1.0572252f * Z;
  }
}

// ---- trace ------------------------------------------------------------------------

// Closest hit of every queued path with one thread per ray (the reference's
// linear object loop, or the instance BVH).
template <class J>
__global__ void __launch_bounds__(128) wf_trace(J jobs, WaveState w, DevCounters* cnt) {
  extern __shared__ StackEntry smem_stack[];
  StackEntry lm[kLocalStack];
  StackEntry lstack[kStackCap];
  StackEntry ltstack[kTlasStackCap];
  SplitStack st{smem_stack + threadIdx.x, blockDim.x, lm, 0, 0u};
  TravStats ts{0u, 0u, 0u, 0u};
  uint32_t rays = 0;
  uint32_t const n = *w.n_in;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t const jb = J::kMulti ? w.in.job[i] : 0u;
    const DevScene& S = jobs.scene(jb);
    bool const ref_order = (jobs.args(jb).flags & LGPU_FLAG_REFERENCE_ORDER) != 0;
    Ray const r = load_ray(w.in.ra, w.in.rb, i);
    HitRec h;
    clear_hit(h, kFltMax);
    scene_trace<false>(S, r, h, UINT32_MAX, ref_order, st, lstack, ltstack, ts);
    rays++;
    store_hit(w, i, h);
  }
  ts.flags |= st.flags;
  flush_counters(cnt, rays, 0u, ts, 0u);
}

// Records whether shadow ray s reached its light.  Its radiance is added
// to the path by the next iteration's shading (or by wf_finish for an ended
// path), which reads the path's contributions in queue order, coalesced.
__device__ __forceinline__ void shadow_done(const WaveState& w, uint32_t s, bool unoccluded) {
  w.s_vis[s] = unoccluded ? 1 : 0;
  if (unoccluded && w.vis) w.vis[w.s_item[s]] |= 1ull << w.s_depth[s];
}

// Persistent instance-BVH traversal of the extension rays (ANY = false,
// the `in` queue, hit records out) or the shadow rays (ANY = true, one
// visibility byte each).
//
// Bound by instruction issue (70 % of the slots; the scene's nodes are in
// L2 and L1): what counts is how many of a warp's lanes share each
// instruction.  The lanes of a warp are at nodes (12 to 13 of 32 at a time),
// leaves and objects; a warp that ran all three every time round executed
// the leaf and object code for two or three lanes.  So nodes are tested every
// time, and lanes at a leaf or an object wait until kTriLanes / kObjLanes of
// them are there (or as many as at nodes; 4, 8 and 12 were within 1 %, 2 %
// and 4 %).  Finished lanes wait too: with kRefill of them (8 and 16 were
// slower) their results are written and new rays fetched with one atomic.
// Benchmark frame (1920x1080, 64 spp, 288 M closest-hit and 194 M shadow
// rays): closest-hit 179 -> 120 ms, shadow 104 -> 82 ms against one loop in
// which each lane popped, sorted and pushed by itself.
constexpr int kRefill = 12;
constexpr int kTriLanes = 6, kObjLanes = 6;
// A launch with fewer rays than lanes is as long as its longest warp, and a
// warp with fewer rays takes fewer and shorter steps: closest-hit rays are
// then spread over all warps, 8 to each at least (131,072 rays of the
// inverse-rendering scene: 185 -> 165 us a launch, 16: 175 us; shadow rays
// gain 10 % there but the kernel then spills and loses 4 % on full queues).
constexpr uint32_t kMinShare = 8;

// Occupancy (measured best): 7 blocks of 128 per SM (72 registers) for
// any-hit queries (6: +11 %, 8: the same), 6 (80 registers) for closest-hit
// queries (5: +9 %, 7: +1 %).
template <bool ANY, int K, class J>
__global__ void __launch_bounds__(128, ANY ? 7 : 6) wf_trace_persistent(J jobs, WaveState w, DevCounters* cnt) {
  constexpr int Q = ANY ? kQueryAny : kQueryClosest;
  extern __shared__ StackEntry smem_stack[];
  StackEntry lm[kLocalStack];
  SplitStack st{smem_stack + threadIdx.x, blockDim.x, lm, 0, 0u};
  __shared__ float wsave[9 * 128];  // launched with 128 threads
  st.ws = wsave + threadIdx.x;
  uint32_t rays = 0, nodes = 0;  // of the warp
  uint32_t tris = 0, insts = 0;
  uint32_t const n = ANY ? w.ctl[kCtlShadow + w.par] : *w.n_in;
  uint32_t* fetch = w.ctl + (ANY ? kCtlSFetch + w.par : uint32_t(kCtlFetch));
  unsigned const FULL = 0xFFFFFFFFu;
  int const lane = threadIdx.x & 31;
  TraceState t;
  t.kind = kLaneIdle;
  // lanes without work that make the warp stop for new rays; once there are
  // none left, any lane that finishes
  int wait = kRefill;
  // Fewer closest-hit rays than lanes: each warp takes its share of them, at
  // least kMinShare, at once.
  uint32_t const warps = gridDim.x * (blockDim.x >> 5);
  uint32_t const share = ANY ? 32u : max(kMinShare, min(32u, (n + warps - 1u) / warps));
  bool const on = uint32_t(lane) < share;
  uint32_t idx = 0, jb = 0;
  auto accept = [&](uint32_t face, float b0, float b1, float b2, f3 pl, float z) {
    if (!ANY) store_hit_point(w, idx, face, b0, b1, b2, pl, z);
  };
  while (true) {
    // one warp sum counts the lanes of each kind
    uint32_t const sum = __reduce_add_sync(FULL, t.kind);
    int const n_tri = int((sum >> 8) & 0xFFu), n_obj = int((sum >> 16) & 0xFFu);
    if (int((sum >> 24) & 0x3Fu) >= wait) {
      if (t.kind == kLaneDone) {
        t.kind = kLaneIdle;
        if (ANY) {
          shadow_done(w, idx, t.obj == UINT32_MAX);
        } else {
          // The winner W of phase 1 may be a mesh whose bounds contain the ray
          // origin and which the ray leaves after the hit.  The reference
          // skips W if an object tested before it (lower index) was hit before
          // that exit (cg.hpp:1393, 1414).  If W is the only such mesh, an
          // any-hit query over the lower-index objects up to the exit (phase
          // 2; nothing to ask for object 0) decides it: without a hit W
          // stands, with one the answer is the closest hit without W (phase
          // 3).  If there are more, whether each counts depends on the
          // others, and the reference's loop answers (wf_trace_fallback).
          //
          // Asking first in that case too would leave 1 in 50 to 120 of those
          // rays for the loop (box room 1.86 instead of 1.91 ms, 14 box rooms
          // with instances 8.9 instead of 10.5 ms), but gives other answers:
          // the loop's exact box tests in the reference's trees reject
          // triangles that a ray grazes and that this search finds (one batch
          // in 75 of such rooms had a different image).
          bool const order = t.phase == 1 && t.exit > t.z, alone = t.n_inside == 1;
          bool const ask = order && alone && t.obj != 0u, again = t.phase == 2 && t.obj != UINT32_MAX;
          if (order && !alone) w.fb_queue[atomicAdd(w.ctl + kCtlFallback, 1u)] = idx;
          if (t.phase != 2) w.hobj[idx] = t.obj;
          if (ask || again) {
            t.w = load_ray(w.in.ra, w.in.rb, idx);
            if (ask) {
              t.z = prev_float(t.exit);
              t.wobj = t.obj;
              t.phase = 2;
            } else {
              t.z = kFltMax;
              t.phase = 3;
            }
            trace_begin(jobs.scene(jb), t, st);
          }
        }
      }
      unsigned idle = __ballot_sync(FULL, t.kind == kLaneIdle && on);
      if (wait == kRefill && idle) {
        uint32_t const want = uint32_t(__popc(idle));
        int const leader = __ffs(idle) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(fetch, want);
        base = __shfl_sync(FULL, base, leader);
        uint32_t const got = min(base < n ? n - base : 0u, want);
        uint32_t const k = uint32_t(__popc(idle & ((1u << lane) - 1u)));
        if (t.kind == kLaneIdle && on && k < got) {
          idx = base + k;
          if (J::kMulti) jb = ANY ? w.s_job[idx] : w.in.job[idx];
          if (ANY) {
            float4 const b = w.sb[idx];
            t.w = make_ray(w.sa[idx], b);
            t.z = b.z;
            t.wobj = __float_as_uint(b.w);
          } else {
            t.w = load_ray(w.in.ra, w.in.rb, idx);
            t.z = kFltMax;
          }
          t.phase = 1;
          trace_begin(jobs.scene(jb), t, st);
        }
        rays += got;
        if (base + want >= n || share < 32u) wait = 0;
      }
      idle = __ballot_sync(FULL, t.kind == kLaneIdle);
      if (wait != kRefill) {
        if (idle == FULL) break;
        wait = __popc(idle) + 1;
      }
      continue;
    }
    const DevScene& S = jobs.scene(jb);
    uint32_t todo = 0xFFu;
    if (t.kind == kLanePop) trace_pop<Q>(S, t, st, todo);
    int const n_node = __popc(__ballot_sync(FULL, t.kind == kLaneNode));
    nodes += n_node;
    if (t.kind == kLaneNode) trace_node<Q>(S, t, st, todo);
    if ((n_tri >= kTriLanes || n_tri >= n_node) && t.kind == kLaneTri) trace_leaf<Q>(S, t, tris, accept);
    if ((n_obj >= kObjLanes || n_obj >= n_node) && t.kind == kLaneObj) trace_object<Q>(S, t, st, insts, accept);
  }
  TravStats const ts{st.flags, lane == 0 ? nodes : 0u, tris, insts};
  flush_counters(cnt, lane == 0 ? rays : 0u, 0u, ts, 0u);
}

// Extension rays whose closest hit depends on the reference's object order
// (see scene_hit): the reference's loop over the objects, in its trees, with
// its tests and its order.  The objects that a ray cannot hit at any distance
// drop out first, 32 at a time by all lanes of a warp (every test of the loop
// only gets stricter as the distance bound shrinks).
//
// Few rays, whose time is the latency of one ray's loop: one warp per ray,
// whose first lane runs the loop over the remaining objects.  From kManyLoop
// rays on, the steps of wf_trace_persistent with the loop's tests (kQueryLoop),
// shared by the lanes whatever object each ray is at; the remaining objects
// wait on the stack of the ray's lane, the lowest indices on top, which holds
// those of kMaxLoopObjects objects (`steps`: no scene has more).
// Ray queries, closest-hit kernel included: 144,091 such rays among 40
// overlapping objects 5.4 ms with a warp per ray, 2.8 with steps; 116,177 among
// 1,000 objects 8.0, 5.5; 9,458 among 40 0.80, 0.75; 4,239 among 150 0.455,
// 0.469.  Box room 256x256, 16 spp (90,378 in 10 launches) 2.34, 2.18 ms; 64x64,
// 4 spp (1,490) 0.806, 0.846.  As a phase of the closest-hit kernel the steps
// spilled registers there (benchmark frame +3.5 %).
constexpr uint32_t kManyLoop = 8192;

template <class J>
__global__ void __launch_bounds__(128, 6) wf_trace_fallback(J jobs, WaveState w, bool steps, DevCounters* cnt) {
  extern __shared__ StackEntry smem_stack[];
  StackEntry lm[kLocalStack];
  static_assert(kLocalStack >= kStackCap, "a mesh's entries");
  uint32_t const n = w.ctl[kCtlFallback];
  unsigned const FULL = 0xFFFFFFFFu;
  int const lane = threadIdx.x & 31;
  uint32_t const warps = gridDim.x * (blockDim.x >> 5);
  if (n < kManyLoop || !steps) {
    TravStats ts{0u, 0u, 0u, 0u};
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
      uint32_t const p = w.fb_queue[i];
      const DevScene& S = jobs.scene(J::kMulti ? w.in.job[p] : 0u);
      Ray const r = load_ray(w.in.ra, w.in.rb, p);
      HitRec h;
      clear_hit(h, kFltMax);
      h.inside = false;
      for (uint32_t base = 0; base < S.n_objects; base += 32) {
        uint32_t const o = base + uint32_t(lane);
        unsigned m = __ballot_sync(FULL, o < S.n_objects && object_may_hit(S, o, r));
        if (lane == 0)
          while (m) {
            uint32_t const b = uint32_t(__ffs(m) - 1);
            m &= m - 1u;
            object_hit<false>(S, base + b, r, h, lm, ts, kRefOrder);
          }
        __syncwarp();
      }
      if (lane == 0) {
        store_hit(w, p, h);
        atomicAdd(&cnt->ordered, 1ull);
      }
    }
    flush_counters(cnt, 0u, 0u, ts, 0u);
    return;
  }
  SplitStack st{smem_stack + threadIdx.x, blockDim.x, lm, 0, 0u};
  __shared__ float wsave[9 * 128];  // launched with 128 threads
  st.ws = wsave + threadIdx.x;
  uint32_t rays = 0, nodes = 0;  // of the warp
  uint32_t tris = 0, insts = 0;
  TraceState t;
  t.kind = kLaneIdle;
  int wait = kRefill;
  // (32 except where n is below the number of lanes)
  uint32_t const share = min(32u, (n + warps - 1u) / warps);
  bool const on = uint32_t(lane) < share;
  uint32_t idx = 0, jb = 0;
  auto accept = [&](uint32_t face, float b0, float b1, float b2, f3 pl, float z) {
    store_hit_point(w, idx, face, b0, b1, b2, pl, z);
  };
  while (true) {
    uint32_t const sum = __reduce_add_sync(FULL, t.kind);
    int const n_tri = int((sum >> 8) & 0xFFu), n_obj = int((sum >> 16) & 0xFFu);
    if (int((sum >> 24) & 0x3Fu) >= wait) {
      if (t.kind == kLaneDone) {
        t.kind = kLaneIdle;
        w.hobj[idx] = t.obj;
      }
      unsigned idle = __ballot_sync(FULL, t.kind == kLaneIdle && on);
      if (wait == kRefill && idle) {
        uint32_t const want = uint32_t(__popc(idle));
        int const leader = __ffs(idle) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(w.ctl + kCtlLoopFetch, want);
        base = __shfl_sync(FULL, base, leader);
        uint32_t const got = min(base < n ? n - base : 0u, want);
        uint32_t const k = uint32_t(__popc(idle & ((1u << lane) - 1u)));
        bool const fresh = t.kind == kLaneIdle && on && k < got;
        if (fresh) {
          idx = w.fb_queue[base + k];
          if (J::kMulti) jb = w.in.job[idx];
          t.w = load_ray(w.in.ra, w.in.rb, idx);
          t.z = kFltMax;
          t.obj = UINT32_MAX;
          t.base = -1;
          t.kind = kLanePop;
          st.sp = 0;
        }
        for (unsigned m = __ballot_sync(FULL, fresh); m; m &= m - 1u) {
          int const src = __ffs(m) - 1;
          const DevScene& S = jobs.scene(__shfl_sync(FULL, jb, src));
          Ray r;
          r.p = f3{__shfl_sync(FULL, t.w.p.x, src), __shfl_sync(FULL, t.w.p.y, src), __shfl_sync(FULL, t.w.p.z, src)};
          r.u = f3{__shfl_sync(FULL, t.w.u.x, src), __shfl_sync(FULL, t.w.u.y, src), __shfl_sync(FULL, t.w.u.z, src)};
          r.inv = f3{0.f, 0.f, 0.f};  // the tests below use the local rays' own
          for (uint32_t b = (S.n_objects + 31u) / 32u; b-- > 0u;) {
            uint32_t const o = 32u * b + uint32_t(lane);
            unsigned const may = __ballot_sync(FULL, o < S.n_objects && object_may_hit(S, o, r));
            if (lane == src && may) st.push(StackEntry{kGroupBit | (32u * b), __uint_as_float(may)});
          }
        }
        rays += got;
        if (base + want >= n || share < 32u) wait = 0;
      }
      idle = __ballot_sync(FULL, t.kind == kLaneIdle);
      if (wait != kRefill) {
        if (idle == FULL) break;
        wait = __popc(idle) + 1;
      }
      continue;
    }
    const DevScene& S = jobs.scene(jb);
    uint32_t todo = 0;
    if (t.kind == kLanePop) trace_pop<kQueryLoop>(S, t, st, todo);
    int const n_node = __popc(__ballot_sync(FULL, t.kind == kLaneNode));
    nodes += n_node;
    if (t.kind == kLaneNode) trace_node<kQueryLoop>(S, t, st, todo);
    if ((n_tri >= kTriLanes || n_tri >= n_node) && t.kind == kLaneTri) trace_leaf<kQueryLoop>(S, t, tris, accept);
    if ((n_obj >= kObjLanes || n_obj >= n_node) && t.kind == kLaneObj) trace_object<kQueryLoop>(S, t, st, insts, accept);
  }
  if (lane == 0 && rays) atomicAdd(&cnt->ordered, static_cast<unsigned long long>(rays));
  TravStats const ts{st.flags, lane == 0 ? nodes : 0u, tris, insts};
  flush_counters(cnt, 0u, 0u, ts, 0u);
}

}  // namespace

// ---- shade ------------------------------------------------------------------------

// Material sort within a block: the block's queue entries [base, base +
// blockDim.x) are handed to its threads grouped by what the shading kernel
// will do with them (miss, then material type, then past the queue end), so
// a warp's lanes take the same branch of the BSDF code.  A counting sort:
// per warp one ballot per group, a shared table of the warps' counts, and
// each thread's rank within its group.  Returns the entry for this thread.
constexpr int kSortGroups = LGPU_MAT_DIREMITTER + 3;

// obj_of(q) is the object that entry q hit (UINT32_MAX: none).
template <class J, class O>
__device__ __forceinline__ uint32_t material_order(const J& jobs, const WaveState& w, uint32_t base, uint32_t n,
                                                   uint32_t* group, O obj_of) {
  __shared__ uint32_t counts[kSortGroups][kMaxShadeBlock / 32];
  __shared__ uint16_t perm[kMaxShadeBlock];
  __shared__ uint8_t groups[kMaxShadeBlock];
  uint32_t const t = threadIdx.x, lane = t & 31u, wid = t >> 5, nw = blockDim.x >> 5;
  uint32_t const q = base + t;
  uint32_t key = kSortGroups - 1;
  if (q < n) {
    uint32_t const obj = obj_of(q);
    if (obj == UINT32_MAX) {
      key = 0;
    } else {
      const DevScene& S = jobs.scene(J::kMulti ? w.in.job[q] : 0u);
      uint32_t type = uint32_t(S.mats[S.objects[obj].mat].type);
      // unshaded materials scatter in the Lambertian hits' code
      if (type == LGPU_MAT_MICROFACET || type > LGPU_MAT_DIREMITTER) type = LGPU_MAT_LAMBERTIAN;
      key = 1u + type;
    }
  }
  unsigned mine = 0;
#pragma unroll
  for (int b = 0; b < kSortGroups; b++) {
    unsigned const m = __ballot_sync(0xFFFFFFFFu, key == uint32_t(b));
    if (key == uint32_t(b)) mine = m;
    if (lane == 0) counts[b][wid] = __popc(m);
  }
  __syncthreads();
  uint32_t pos = __popc(mine & ((1u << lane) - 1u));
  for (uint32_t b = 0; b < key; b++)
    for (uint32_t v = 0; v < nw; v++) pos += counts[b][v];
  for (uint32_t v = 0; v < wid; v++) pos += counts[key][v];
  perm[pos] = uint16_t(t);
  groups[pos] = uint8_t(key);
  __syncthreads();
  uint32_t const r = base + perm[t];
  *group = groups[t];
  __syncthreads();  // counts and perm are reused by the block's next chunk
  return r;
}

// After material_order: the block's Blinn entries are appended to the list
// at the front of w.shade_list, its thin-film entries to the list growing
// down from its end (both lists hold queue positions, together at most the
// queue's length), and its Lambertian ones to w.shade_list2.  A group is a
// contiguous range of the block's threads, so one atomic per list and block
// places it.
__device__ __forceinline__ void list_material_groups(const WaveState& w, uint32_t i, uint32_t group) {
  __shared__ uint32_t lbase[3];
  uint32_t const gl = 1u + LGPU_MAT_LAMBERTIAN, gb = 1u + LGPU_MAT_BLINN, gt = 1u + LGPU_MAT_THINFILM;
  uint32_t const below_l = uint32_t(__syncthreads_count(group < gl));
  uint32_t const below_b = uint32_t(__syncthreads_count(group < gb));
  uint32_t const cnt_b = uint32_t(__syncthreads_count(group == gb));
  uint32_t const below_t = uint32_t(__syncthreads_count(group < gt));
  uint32_t const cnt_t = uint32_t(__syncthreads_count(group == gt));
  if (threadIdx.x == 0) {
    lbase[0] = cnt_b ? atomicAdd(w.ctl + kCtlListB, cnt_b) : 0u;
    lbase[1] = cnt_t ? atomicAdd(w.ctl + kCtlListT, cnt_t) : 0u;
    lbase[2] = below_b > below_l ? atomicAdd(w.ctl + kCtlListL, below_b - below_l) : 0u;
  }
  __syncthreads();
  if (group == gl) w.shade_list2[lbase[2] + threadIdx.x - below_l] = i;
  if (group == gb) w.shade_list[lbase[0] + threadIdx.x - below_b] = i;
  if (group == gt) w.shade_list[w.cap - 1u - (lbase[1] + threadIdx.x - below_t)] = i;
  __syncthreads();  // lbase is reused by the block's next chunk
}

// One vertex of Renderer::tracePath (src/renderer.cpp:64-146) for every
// queued path: emitter hit (73-84), light importance sample with the MIS
// power heuristic (87-113, its visibility left to the shadow kernel),
// material importance sample with Russian roulette (115-143).
// The launches of an iteration, by what their paths hit (MT), shade every
// path once; each has the code of its materials alone.
//   scenes without Blinn and thin film: LGPU_MAT_LAMBERTIAN (all paths, the
//     block's entries sorted by material);
//   others: kShadeRest (sorts, shades misses and emitters, and lists the
//     rest), then LGPU_MAT_BLINN, LGPU_MAT_THINFILM and kShadeLamb (Lambertian
//     and unshaded materials) over their lists, every warp full.
// The first kind stays for its scenes because a launch more costs them more
// than full warps give: a 64x64 thumbnail 472 against 508 us with lists, the
// Lambertian box room 1.85 against 1.90 ms.  The second, against one launch for
// all but the Blinn and thin-film lists: benchmark frame 277.2 -> 270.2 ms
// (39.1 ms of shading become 10.8 + 21.5), mixed materials 8.18 -> 7.78 ms.
// Without scattering code kShadeRest fits 6 blocks of 256 threads on an SM
// (4 blocks for the others): 10.8 ms against 14.0 with 8 and 11.9 with 5.
// REC: the primal pass of an adjoint, which records what the replay reads.
constexpr int kShadeLamb = 10, kShadeRest = 11;
template <int MT>
constexpr bool kShadeLists = MT == LGPU_MAT_BLINN || MT == LGPU_MAT_THINFILM || MT == kShadeLamb;
template <int MT>
__device__ __forceinline__ bool shade_group(uint32_t group) {
  return MT != kShadeRest || group < 1u + LGPU_MAT_LAMBERTIAN || group > 1u + LGPU_MAT_THINFILM;
}
// Entry j of a list launch (UINT32_MAX past its end) and the list's length.
template <int MT>
__device__ __forceinline__ uint32_t shade_list_length(const WaveState& w) {
  return w.ctl[MT == LGPU_MAT_BLINN ? kCtlListB : (MT == LGPU_MAT_THINFILM ? kCtlListT : kCtlListL)];
}
template <int MT>
__device__ __forceinline__ uint32_t shade_list_entry(const WaveState& w, uint32_t j, uint32_t n) {
  if (j >= n) return UINT32_MAX;
  if (MT == kShadeLamb) return w.shade_list2[j];
  return w.shade_list[MT == LGPU_MAT_BLINN ? j : w.cap - 1u - j];
}
// A material as a launch sees it: the types it cannot meet are ruled out for
// the compiler.
template <int MT>
__device__ __forceinline__ DevMaterial shade_material(const DevScene& S, uint32_t idx) {
  DevMaterial x = S.mats[idx];
  if (MT == LGPU_MAT_BLINN || MT == LGPU_MAT_THINFILM) x.type = MT;
  if (MT == kShadeLamb) x.type = x.type == LGPU_MAT_LAMBERTIAN ? LGPU_MAT_LAMBERTIAN : LGPU_MAT_MICROFACET;
  if (MT == kShadeRest) x.type = x.type == LGPU_MAT_DIREMITTER ? LGPU_MAT_DIREMITTER : LGPU_MAT_EMITTER;
  if (MT == LGPU_MAT_LAMBERTIAN && (x.type == LGPU_MAT_BLINN || x.type == LGPU_MAT_THINFILM))
    x.type = LGPU_MAT_MICROFACET;
  return x;
}
// What a launch's materials leave of the BSDF cases and lobes.
template <int MT>
__device__ __forceinline__ void shade_cases(BsdfScalars& bl, MatSample& ms) {
  if (MT == LGPU_MAT_LAMBERTIAN || MT == kShadeLamb) {
    bl.kind = bl.kind ? 1 : 0;
    ms.lobe = ms.lobe ? 1 : 0;
  } else if (MT == LGPU_MAT_BLINN) {
    bl.kind = bl.kind == 2 ? 2 : 3;
  } else if (MT == LGPU_MAT_THINFILM) {
    bl.kind = bl.kind ? 4 : 0;
    ms.lobe = ms.lobe ? 4 : 0;
  }
}

// Bound by memory latency (35 % of the issue slots, 2.4 TB/s of path state)
// and by what the geometry part spills.  So each launch's code knows which
// materials it can meet, the path's records are written before the
// wavelength loop (which then keeps only its scalars), and that loop moves
// 16-byte words of four wavelengths but computes one at a time: unrolled by
// four, its code overflowed the instruction cache (8 of 23 stalls) and was
// 17 % slower than 4-byte accesses.  4 blocks of 256 per SM (64 registers)
// where scattering is evaluated: 5 are 2 % faster for the benchmark frame's
// Lambertian hits but 7 % slower for the box room; 6 and 5 before.
// Benchmark frame: misses, emitters and Lambertian hits 48.2 -> 32.3 ms, Blinn
// list 16.5 -> 14.9, thin-film list 16.3 -> 14.3; box room 605 -> 472 us.
template <int K, class J, int MT, bool REC>
__global__ void __launch_bounds__(kMaxShadeBlock, MT == kShadeRest ? 6 : 4) wf_shade(J jobs, WaveState w, DevCounters* cnt) {
  uint32_t const n = *w.n_in;
  uint32_t const cap = w.cap;
  PathBuf const& in = w.in;
  PathBuf const& out = w.out;
  enum : int { kEnd = 0, kEmit = 1, kScatter = 2 };
  constexpr bool kList = kShadeLists<MT>;
  uint32_t const n_loop = kList ? shade_list_length<MT>(w) : n;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n_loop; base += gridDim.x * blockDim.x) {
    uint32_t group = 0, i;
    if (kList) {
      i = shade_list_entry<MT>(w, base + threadIdx.x, n_loop);
    } else {
      i = material_order(jobs, w, base, n, &group, [&](uint32_t q) { return w.hobj[q]; });
      if (MT == kShadeRest) list_material_groups(w, i, group);
    }
    bool const live = i < n && shade_group<MT>(group);
    uint32_t const jb = (J::kMulti && live) ? in.job[i] : 0u;
    const DevScene& S = jobs.scene(jb);
    const RenderArgs& a = jobs.args(jb);
    float const omega = S.lambda_sup - S.lambda_inf;
    float const step = omega / float(K);
    auto material = [&](uint32_t idx) { return shade_material<MT>(S, idx); };
    int kind = kEnd;
    bool cont = false, shadow = false, needs_test = false;
    f3 sp = f3{0.f, 0.f, 0.f}, sd = f3{0.f, 0.f, 1.f};
    float stmax = 0.f;
    uint32_t sskip = UINT32_MAX;
    f3 np = f3{0.f, 0.f, 0.f}, nd = f3{0.f, 0.f, 1.f};
    float lis_scale = 0.f, m_scale = 0.f, g_emit = 1.f, hero = 0.f;
    uint64_t rng = 0;
    uint32_t mat = 0, light = 0;
    bool front = true;
    MatSample ms;
    ms.ok = false;
    BsdfScalars bl{};
    uint32_t depth = 0, item = 0, prev_s = kNoShadow;
    if (live) {
      float4 const rb = in.rb[i];
      uint4 const rc = in.rc[i];
      hero = rb.z;
      depth = __float_as_uint(rb.w);
      item = rc.z;
      prev_s = rc.w;
      uint32_t const obj = w.hobj[i];
      size_t const v_at = size_t(depth) * w.v_items + item;
      if (REC && w.v_obj) w.v_obj[v_at] = UINT32_MAX;
      if (obj != UINT32_MAX) {
        HitRec const h = load_hit(w.hita, w.hitb, i, obj);
        Ray const r = make_ray(in.ra[i], rb);
        HitInfo const H = finalize_hit(S, r, h);
        f3 const un = fnorm(r.u);
        f3 const o = f3{-un.x, -un.y, -un.z};
        f3 const nn = H.front ? H.F.z : neg3(H.F.z);
        mat = H.mat;
        front = H.front;
        DevMaterial const m = material(mat);
        if (m.type == LGPU_MAT_EMITTER || m.type == LGPU_MAT_DIREMITTER) {
          kind = kEmit;
          if (m.type == LGPU_MAT_DIREMITTER) {
            float const c = fdot(o, H.F.z);
            g_emit = powf(c >= 0.f ? c : 0.f, m.specular);
          }
        } else if (depth <= a.max_scatter) {
          kind = kScatter;
          if (REC && w.v_obj) {
            w.v_obj[v_at] = obj;
            w.v_hita[v_at] = make_float4(__uint_as_float(h.face), h.b0, h.b1, h.b2);
            w.v_hitb[v_at] = make_float4(h.pl.x, h.pl.y, h.pl.z, h.z);
          }
          rng = (uint64_t(rc.y) << 32) | rc.x;
          light = uint32_t(lgpu_u64(&rng) % uint64_t(S.n_lights));
          float const prob_l = 1.f / float(S.n_lights);
          const lgpu_light& L = S.lights[light];
          // light sample without its visibility (the shadow kernel applies it)
          LightSample ls = sample_light_unoccluded(S, L, H, rng, stmax, sskip);
          float const x0 = lam_coord(S, hero);
          bl = bsdf_scalars(S, m, x0, ls.dir, o, nn, H.front);
          ms = sample_material(S, m, x0, H, o, a.sample_p, rng);
          float w_L = 1.f, w_mat = 0.f;
          if (ms.ok) {
            float const p_L_mati = prob_for_light(S, L, H.p, ms.dir) * prob_l;
            float const p_mat_Li = prob_for_material(S, m, x0, H, ls.dir, o, a.sample_p);
            float const p_L_i = ls.prob * prob_l;
            w_L = p_L_i * p_L_i / (p_L_i * p_L_i + p_mat_Li * p_mat_Li);
            w_mat = ms.prob * ms.prob / (ms.prob * ms.prob + p_L_mati * p_L_mati);
          }
          lis_scale = ls.scale / (ls.prob * prob_l) * w_L;
          m_scale = ms.ok ? w_mat / ms.prob : 0.f;
          needs_test = stmax >= 0.f;
          shadow = needs_test && lis_scale != 0.f;
          sp = H.p;
          sd = ls.dir;
          cont = ms.ok;
          if (cont) {
            np = H.p;
            nd = ms.dir;
          }
        }
      }
    }
    shade_cases<MT>(bl, ms);
    // compacted appends: next queue, ended list, shadow queue
    bool const ended = live && !cont;
    uint32_t const o_pos = warp_append(w.n_out, cont);
    uint32_t const e_pos = warp_append(w.ctl + kCtlEnded + w.par, ended);
    uint32_t const s_pos = warp_append(w.ctl + kCtlShadow + w.par, shadow);
    if (!live) continue;
    // the path's records first: the wavelength loop below then has only the
    // scalars of its spectra to keep in registers
    uint32_t const s_ref = shadow ? s_pos : kNoShadow;
    if (cont) {
      out.ra[o_pos] = make_float4(np.x, np.y, np.z, nd.x);
      out.rb[o_pos] = make_float4(nd.y, nd.z, hero, __uint_as_float(depth + 1));
      out.rc[o_pos] = make_uint4(uint32_t(rng), uint32_t(rng >> 32), item, s_ref);
      if (J::kMulti) out.job[o_pos] = jb;
    } else {
      w.e_rec[e_pos] = make_uint4(__float_as_uint(hero), item, s_ref, jb);
    }
    if (shadow) {
      if (J::kMulti) w.s_job[s_pos] = jb;
      if (REC) {
        w.s_item[s_pos] = item;
        w.s_depth[s_pos] = depth;
      }
      w.sa[s_pos] = make_float4(sp.x, sp.y, sp.z, sd.x);
      w.sb[s_pos] = make_float4(sd.y, sd.z, stmax, __uint_as_float(sskip));
    }
    float4* const acc_dst = cont ? out.acc + o_pos : w.e_acc + e_pos;
    DevMaterial const m = material(mat);
    // the light sample of the path's previous vertex, if its shadow ray got
    // through (recorded by the shadow kernel of the last iteration)
    const float4* const pend = (prev_s != kNoShadow && w.s_vis[prev_s]) ? w.s_prev + prev_s : nullptr;
    // a path at depth 0 starts with throughput 1 and no radiance (the
    // generate kernel writes neither)
    bool const fresh = depth == 0;
    auto load_beta = [&](int q) { return fresh ? make_float4(1.f, 1.f, 1.f, 1.f) : in.beta[q * cap + i]; };
    // the radiance so far, with that light sample
    auto load_acc = [&](int q) {
      float4 const v = fresh ? make_float4(0.f, 0.f, 0.f, 0.f) : in.acc[q * cap + i];
      float4 const p = pend ? pend[q * cap] : make_float4(0.f, 0.f, 0.f, 0.f);
      return make_float4(v.x + p.x, v.y + p.y, v.z + p.z, v.w + p.w);
    };
    if (kind == kScatter) {
      const lgpu_light& L = S.lights[light];
      float4 bt = make_float4(0.f, 0.f, 0.f, 0.f), acc = bt, con = bt;
#pragma unroll 1
      for (int k = 0; k < K; k++) {
        if ((k & 3) == 0) {
          bt = load_beta(k >> 2);
          acc = load_acc(k >> 2);
        }
        float const l = hero_lambda(S, hero, step, k);
        float const x = lam_coord(S, l);
        float const coef = bsdf_k(S, m, bl, x, l, front);
        float const rad = spec_at(S, L.spectrum, x);
        float const contrib = bt.x * (rad * coef * lis_scale);
        float const a_k = needs_test ? acc.x : acc.x + contrib;
        float const b_k = cont ? bt.x * (mat_mult_k(S, m, ms, x, l, front) * m_scale) : 0.f;
        // the words turn by one wavelength, so one loop body serves all four
        acc = make_float4(acc.y, acc.z, acc.w, a_k);
        bt = make_float4(bt.y, bt.z, bt.w, b_k);
        con = make_float4(con.y, con.z, con.w, contrib);
        if ((k & 3) == 3) {
          uint32_t const at = uint32_t(k >> 2) * cap;
          if (shadow) w.s_contrib[at + s_pos] = con;
          if (cont) out.beta[at + o_pos] = bt;
          acc_dst[at] = acc;
        }
      }
    } else if (kind == kEmit) {
      float4 bt = make_float4(0.f, 0.f, 0.f, 0.f), acc = bt;
#pragma unroll 1
      for (int k = 0; k < K; k++) {
        if ((k & 3) == 0) {
          bt = load_beta(k >> 2);
          acc = load_acc(k >> 2);
        }
        float const x = lam_coord(S, hero_lambda(S, hero, step, k));
        float const a_k = acc.x + bt.x * (spec_at(S, m.spectrum[0], x) * g_emit);
        acc = make_float4(acc.y, acc.z, acc.w, a_k);
        bt = make_float4(bt.y, bt.z, bt.w, 0.f);
        if ((k & 3) == 3) acc_dst[uint32_t(k >> 2) * cap] = acc;
      }
    } else {
#pragma unroll
      for (int q = 0; q < K / 4; q++) acc_dst[q * cap] = load_acc(q);
    }
  }
  (void)cnt;
}

// ---- shadow -----------------------------------------------------------------------

// Any-hit test of every shadow ray with one thread per ray.
template <int K, class J>
__global__ void __launch_bounds__(128) wf_shadow(J jobs, WaveState w, DevCounters* cnt) {
  extern __shared__ StackEntry smem_stack[];
  StackEntry lm[kLocalStack];
  StackEntry lstack[kStackCap];
  StackEntry ltstack[kTlasStackCap];
  SplitStack st{smem_stack + threadIdx.x, blockDim.x, lm, 0, 0u};
  TravStats ts{0u, 0u, 0u, 0u};
  uint32_t rays = 0;
  uint32_t const n = w.ctl[kCtlShadow + w.par];
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t const jb = J::kMulti ? w.s_job[i] : 0u;
    const DevScene& S = jobs.scene(jb);
    bool const ref_order = (jobs.args(jb).flags & LGPU_FLAG_REFERENCE_ORDER) != 0;
    float4 const b = w.sb[i];
    Ray const r = make_ray(w.sa[i], b);
    HitRec h;
    clear_hit(h, b.z);
    uint32_t const skip = __float_as_uint(b.w);
    bool const occ = scene_trace<true>(S, r, h, skip, ref_order, st, lstack, ltstack, ts);
    rays++;
    shadow_done(w, i, !occ);
  }
  ts.flags |= st.flags;
  flush_counters(cnt, rays, 0u, ts, 0u);
}

}  // namespace lgpu
