// lgpu_adjoint.cuh — path-replay backpropagation of the image loss to the
// material parameters (the reference has no derivative code; this is the
// adjoint of Renderer::tracePath, src/renderer.cpp:64-146).
//
// A path's radiance per hero wavelength is
//     L = Σ_v β_v (E_v + N_v),   β_{v+1} = β_v f_v / q_v,
// with E_v the emission found at vertex v, N_v its light sample (the BSDF
// value f(light dir) times the light's weighted radiance, if the shadow ray
// is unoccluded) and f_v / q_v the material sample's BSDF value over its
// (MIS-weighted) density.  For a parameter π of the material at vertex v,
// with sampling decisions and MIS weights held fixed,
//     dL/dπ = β_v ∂N_v/∂π + L_after_v ∂ln f_v/∂π,
// where L_after_v = Σ_{w>v} β_w (E_w + N_w) is the radiance the path
// gathers after v.  Two passes per chunk of work items:
//   primal  the wavefront render, which also stores every path's L and a bit
//           per vertex telling whether its shadow ray reached the light;
//   replay  the same paths again from their random streams (no shadow rays:
//           visibility comes from the bits), starting from L and subtracting
//           each vertex's contribution to get L_after_v, accumulating
//           dL/dπ · dLoss/dL into the gradients.  Where they fit in memory
//           the primal pass also records the vertices' hits, and the replay
//           traces no rays at all.
// Parameters: the bins of Lambertian albedo spectra and of thin-film IOR
// spectra, thin-film thickness, and the exponent α of Blinn and thin-film
// lobes.
#pragma once

#include "lgpu_render.cuh"

namespace lgpu {

// ---- derivatives of thinfilm::BRDFcosθ --------------------------------------------

// thinfilm_k (lgpu_path.cuh, cg.hpp:1001-1051), by the same operations, with
// its derivatives with respect to the film IOR n1 and the thickness d.  With
// q = sqrt(1 - 1/n1²), c = 1 - cos_i², φ = 4π n1 d q c / λ, and a, b the
// difference and sum of the IORs at an interface (R0 = a²/b²):
//     ∂φ/∂n1 = 4π d c / (λ q)    (n1 q = sqrt(n1² - 1)),   ∂φ/∂d = φ / d,
//     ∂R0_01/∂n1 = -4 (1 - n1) / (1 + n1)³,   ∂R0_12/∂n1 = 4 (n1 - n2) n2 / (n1 + n2)³.
// About 11 divisions where forward-mode dual numbers took 35, at the same
// error (2-norm over 400,000 random films against double precision: ∂n1
// 7.299e-3 with both, ∂d 9.416e-3; the rounding of φ makes it).
struct FilmGrad {
  float v, dn, dd;
};
__device__ __forceinline__ FilmGrad thinfilm_grad(float n1, float n2, float d, float alpha, float l, float cos_i,
                                                  float pow5, float pow_hn) {
  float const n01 = 1.f / n1;
  float const q = sqrtf(1.f - n01 * n01), c = 1.f - cos_i * cos_i;
  float const cos_l = q * c;
  float sn, cs;
  sincosf(4.f * kPi * n1 * d * cos_l / l, &sn, &cs);
  float const a01 = (1.f - n1), b01 = (1.f + n1);
  float const R0_01 = a01 * a01 / (b01 * b01);
  float const a12 = (n1 - n2), b12 = (n1 + n2);
  float const R0_12 = a12 * a12 / (b12 * b12);
  float const R01 = R0_01 + (1.f - R0_01) * pow5;
  float const R12 = R0_12 + (1.f - R0_12) * pow5;
  float const P = R01 * R12, root = sqrtf(P), Ravg = 2.f * root;
  float const den = 1.f + P + Ravg * cs;
  float const Rt = (R01 + R12 + Ravg * cs) / den;
  // derivatives
  float const k4 = 4.f * kPi / l, i01 = 1.f / b01, i12 = 1.f / b12, iden = 1.f / den;
  float const phi_n = q > 0.f ? k4 * d * c / q : 0.f, phi_d = k4 * n1 * cos_l;
  float const keep = 1.f - pow5;
  float const R01n = -4.f * a01 * (i01 * i01 * i01) * keep, R12n = 4.f * a12 * n2 * (i12 * i12 * i12) * keep;
  float const Pn = R01n * R12 + R01 * R12n;
  float const avg_n = root > 0.f ? Pn / root : 0.f;
  float const Xn = avg_n * cs - Ravg * sn * phi_n, Xd = -Ravg * sn * phi_d;
  float const s = (alpha + 2.f) * 0.125f * kInvPi * pow_hn;
  FilmGrad f;
  f.v = (alpha + 2.f) * 0.125f * kInvPi * Rt * pow_hn;
  f.dn = s * (((R01n + R12n + Xn) - Rt * (Pn + Xn)) * iden);
  f.dd = s * (Xd * (1.f - Rt) * iden);
  return f;
}

// ---- accumulation ---------------------------------------------------------------

// v * d spec_at(S, s, x) / d bins of spectrum s (the lerp of spec_at)
__device__ __forceinline__ void spec_grad(const DevScene& S, float* g_spec, int32_t s, float x, float v) {
  if (v == 0.f || !isfinite(v)) return;
  float* g = g_spec + size_t(s) * S.n_bins;
  uint32_t const n = S.n_bins;
  if (x < 0.f) {
    atomicAdd(g, v);
    return;
  }
  if (x >= 1e29f) {
    atomicAdd(g + n - 1, v);
    return;
  }
  uint32_t const i = min(uint32_t(x), n - 2);
  float const t = x - float(i);
  atomicAdd(g + i, v * (1.f - t));
  atomicAdd(g + i + 1, v * t);
}

// d ln(pow(hn, α) (α+2)) / dα, or 0 where the lobe value is 0
__device__ __forceinline__ float dlog_lobe_dalpha(float alpha, float c, float lnhn) {
  return c > 0.f ? 1.f / (alpha + 2.f) + lnhn : 0.f;
}

// v * d BxDFcosθ(light dir) / dα for the NEE term of a Blinn lobe (bsdf_k's
// cases 2 and 3)
__device__ __forceinline__ float grad_blinn(const DevScene& S, const DevMaterial& m, const BsdfScalars& r, float x,
                                            bool front, float v) {
  float const ior = spec_at(S, m.spectrum[4], x);
  float const eta = front ? 1.f / ior : ior;
  float const F0 = schlick_F0(eta);
  float const F = F0 + (1.f - F0) * r.b;
  float const gl = (m.alpha + 2.f) * 0.125f * kInvPi * r.c;
  float const spec = r.kind == 2 ? (spec_at(S, m.spectrum[1], x) + F * spec_at(S, m.spectrum[2], x)) * gl
                                 : spec_at(S, m.spectrum[2], x) * (1.f - F) * gl;
  return v * spec * dlog_lobe_dalpha(m.alpha, r.c, r.lnhn);
}

__device__ __forceinline__ float finite_or_zero(float x) { return isfinite(x) ? x : 0.f; }

namespace {

// Replay: the chunk's paths restart from their random streams with the
// radiance the primal pass recorded and their dLoss/dL weights:
//     dLoss/dL_k = Σ_c dLoss/dRGB_c (M_XYZ→RGB · w_XYZ(λ_k))_c Δ / (spp K p(λ))
// with w_XYZ(λ) the XYZ of addHeroλ(λ, 1) (cg.hpp:306-320, 283-288).
template <int K>
__global__ void __launch_bounds__(256) wf_replay_generate(OneJob jobs, WaveState w, AdjointArgs g) {
  uint32_t const n_new = w.ctl[kCtlNew], first = w.ctl[kCtlFirst], pos = w.ctl[kCtlPos];
  uint32_t const cap = w.cap;
  const DevScene& S = jobs.S;
  const RenderArgs& a = jobs.a;
  PathBuf const& in = w.in;
  float const omega = S.lambda_sup - S.lambda_inf;
  float const step = omega / float(K);
  const lgpu_camera& C = S.cam;
  uint32_t const W = uint32_t(C.width), H = uint32_t(C.height);
  float const scale = S.lambda_delta / (float(a.spp) * float(K)) * omega;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n_new; k += gridDim.x * blockDim.x) {
    uint32_t const q = first + k;
    uint64_t const gq = w.c0 + q;
    uint32_t const sample = uint32_t(gq / jobs.npix);
    uint32_t const pix = uint32_t(gq - uint64_t(sample) * jobs.npix);
    uint32_t const p = pos + k;
    uint32_t const i = pix / W, j = pix - i * W;
    uint64_t rng = lgpu_path_state(a.seed, (uint64_t(a.stream_tag) << 32) | pix, uint64_t(a.spp_offset) + sample);
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
    const float* dI = g.dimg + (size_t(H - i - 1) * W + j) * 3;
    float const dR = dI[0], dG = dI[1], dB = dI[2];
    // dLoss/dXYZ through the XYZ -> linear RGB matrix of finalize
    float const dX = 3.2404542f * dR - 0.9692660f * dG + 0.0556434f * dB;
    float const dY = -1.5371385f * dR + 1.8760108f * dG - 0.2040259f * dB;
    float const dZ = -0.4985314f * dR + 0.0415560f * dG + 1.0572252f * dB;
#pragma unroll
    for (int kq = 0; kq < K / 4; kq++) {
      float gw[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        float X = 0.f, Y = 0.f, Z = 0.f;
        splat_xyz(S, hero_lambda(S, hero, step, 4 * kq + j), 1.f, X, Y, Z);
        gw[j] = (dX * X + dY * Y + dZ * Z) * scale;
      }
      in.beta[kq * cap + p] = make_float4(1.f, 1.f, 1.f, 1.f);
      in.acc[kq * cap + p] = w.ltot[size_t(q) * (K / 4) + kq];
      in.gw[kq * cap + p] = make_float4(gw[0], gw[1], gw[2], gw[3]);
    }
  }
}

// One vertex of the replay: the same random decisions as wf_shade, the
// visibility recorded by the primal pass, gradients accumulated.  The
// launches by material are wf_shade's (MT); kShadeRest only fills the lists.
//
// Bound by issue and by instruction fetch (5 of 16 stalls in one launch for
// all materials, with the gradient code of each in every block).  64x64
// thin-film tiles under 64 spheres, 512x512, 32 spp: one launch with
// forward-mode dual numbers 18.8 ms, closed-form thin-film derivatives 10.7
// ms, launches by material 6.6 ms (4 blocks of 256 per SM; 3 and 5: +5 %),
// Lambertian hits in a list 6.4 ms; the bins' atomics are no bound (without
// them 18.4 of the 18.8 ms).
template <int K, int MT>
__global__ void __launch_bounds__(kMaxShadeBlock, 4) wf_shade_adjoint(OneJob jobs, WaveState w, AdjointArgs g) {
  uint32_t const n = *w.n_in;
  uint32_t const cap = w.cap;
  const DevScene& S = jobs.S;
  const RenderArgs& a = jobs.a;
  PathBuf const& in = w.in;
  PathBuf const& out = w.out;
  float const omega = S.lambda_sup - S.lambda_inf;
  float const step = omega / float(K);
  constexpr bool kList = kShadeLists<MT>;
  uint32_t const n_loop = kList ? shade_list_length<MT>(w) : n;
  for (uint32_t base = blockIdx.x * blockDim.x; base < n_loop; base += gridDim.x * blockDim.x) {
    uint32_t group = 0, i;
    if (kList) {
      i = shade_list_entry<MT>(w, base + threadIdx.x, n_loop);
    } else {
      i = material_order(jobs, w, base, n, &group, [&](uint32_t q) {
        return w.v_obj ? w.v_obj[size_t(__float_as_uint(in.rb[q].w)) * w.v_items + in.rc[q].z] : w.hobj[q];
      });
      if (MT == kShadeRest) {
        // misses and emitters end their paths without a gradient
        list_material_groups(w, i, group);
        continue;
      }
    }
    bool const live = i < n;
    auto material = [&](uint32_t idx) { return shade_material<MT>(S, idx); };
    bool cont = false, scatter = false, visible = false;
    f3 np = f3{0.f, 0.f, 0.f}, nd = f3{0.f, 0.f, 1.f};
    float lis_scale = 0.f, m_scale = 0.f, hero = 0.f;
    // d ln w_L / dα and d ln w_mat / dα of the MIS weights (below)
    float dlw_L = 0.f, dlw_mat = 0.f;
    uint64_t rng = 0;
    uint32_t mat = 0, light = 0, depth = 0, item = 0;
    bool front = true;
    MatSample ms;
    ms.ok = false;
    BsdfScalars bl{};
    if (live) {
      float4 const rb = in.rb[i];
      uint4 const rc = in.rc[i];
      hero = rb.z;
      depth = __float_as_uint(rb.w);
      item = rc.z;
      size_t const v_at = size_t(depth) * w.v_items + item;
      uint32_t const obj = w.v_obj ? w.v_obj[v_at] : w.hobj[i];
      if (obj != UINT32_MAX) {
        HitRec const h = w.v_obj ? load_hit(w.v_hita, w.v_hitb, v_at, obj) : load_hit(w.hita, w.hitb, i, obj);
        Ray const r = make_ray(in.ra[i], rb);
        HitInfo const H = finalize_hit(S, r, h);
        f3 const un = fnorm(r.u);
        f3 const o = f3{-un.x, -un.y, -un.z};
        f3 const nn = H.front ? H.F.z : neg3(H.F.z);
        mat = H.mat;
        front = H.front;
        DevMaterial const m = material(mat);
        // an emitter ends the path; its radiance is not a parameter
        if (m.type != LGPU_MAT_EMITTER && m.type != LGPU_MAT_DIREMITTER && depth <= a.max_scatter) {
          scatter = true;
          rng = (uint64_t(rc.y) << 32) | rc.x;
          light = uint32_t(lgpu_u64(&rng) % uint64_t(S.n_lights));
          float const prob_l = 1.f / float(S.n_lights);
          const lgpu_light& L = S.lights[light];
          float stmax = 0.f;
          uint32_t sskip = UINT32_MAX;
          LightSample ls = sample_light_unoccluded(S, L, H, rng, stmax, sskip);
          float const x0 = lam_coord(S, hero);
          bl = bsdf_scalars(S, m, x0, ls.dir, o, nn, H.front);
          ms = sample_material(S, m, x0, H, o, a.sample_p, rng);
          float w_L = 1.f, w_mat = 0.f;
          if (ms.ok) {
            float const p_L_mati = prob_for_light(S, L, H.p, ms.dir) * prob_l;
            float dlp_Li = 0.f;
            float const p_mat_Li = prob_for_material(S, m, x0, H, ls.dir, o, a.sample_p, &dlp_Li);
            float const p_L_i = ls.prob * prob_l;
            w_L = p_L_i * p_L_i / (p_L_i * p_L_i + p_mat_Li * p_mat_Li);
            w_mat = ms.prob * ms.prob / (ms.prob * ms.prob + p_L_mati * p_L_mati);
            // The power-heuristic weights depend on α through the material
            // pdf (at the light sample's direction for w_L, at the material
            // sample's for w_mat).  In a proper MIS their derivatives would
            // cancel in expectation; here they do not, because the
            // reference applies w_L only when a material sample exists
            // (src/renderer.cpp:120) and w_mat to the whole recursive
            // radiance (src/renderer.cpp:145), so the gradient of its
            // expected image carries them:
            //   d ln w_L / dα   = -2 (1 - w_L) d ln p_mat(ω_L) / dα
            //   d ln w_mat / dα =  2 (1 - w_mat) d ln p_mat(ω_mat) / dα
            // (the sample's own 1/pdf needs no term: its α-derivative equals
            // the score of the density the direction was drawn from).
            dlw_L = -2.f * (1.f - w_L) * dlp_Li;
            dlw_mat = 2.f * (1.f - w_mat) * ms.dlnprob;
          }
          lis_scale = ls.scale / (ls.prob * prob_l) * w_L;
          m_scale = ms.ok ? w_mat / ms.prob : 0.f;
          bool const needs_test = stmax >= 0.f;
          visible = !needs_test || ((w.vis[item] >> depth) & 1ull);
          cont = ms.ok;
          if (cont) {
            np = H.p;
            nd = ms.dir;
          }
        }
      }
    }
    shade_cases<MT>(bl, ms);
    uint32_t const o_pos = warp_append(w.n_out, cont);
    if (!scatter) continue;
    if (cont) {
      out.ra[o_pos] = make_float4(np.x, np.y, np.z, nd.x);
      out.rb[o_pos] = make_float4(nd.y, nd.z, hero, __uint_as_float(depth + 1));
      out.rc[o_pos] = make_uint4(uint32_t(rng), uint32_t(rng >> 32), item, kNoShadow);
    }
    DevMaterial const m = material(mat);
    const lgpu_light& L = S.lights[light];
    float g_d = 0.f, g_alpha = 0.f;
    float4 bt = make_float4(0.f, 0.f, 0.f, 0.f), gws = bt, rems = bt;
#pragma unroll 1
    for (int k = 0; k < K; k++) {
      uint32_t const at = uint32_t(k >> 2) * cap;
      if ((k & 3) == 0) {
        bt = in.beta[at + i];
        gws = in.gw[at + i];
        rems = in.acc[at + i];
      }
      float const l = hero_lambda(S, hero, step, k);
      float const x = lam_coord(S, l);
      float const gw = gws.x;
      float b = bt.x, rem = rems.x;
      // the spectrum the material's gradient goes to (Lambertian albedo or
      // film IOR): the light sample's and the material sample's part together
      float g_bin = 0.f;
      float n1 = 0.f, n2 = 0.f;
      if (m.type == LGPU_MAT_THINFILM) {
        n1 = spec_at(S, m.spectrum[0], x);
        n2 = spec_at(S, m.spectrum[1], x);
      }
      if (visible && lis_scale != 0.f) {
        float const rad = spec_at(S, L.spectrum, x);
        float const v = gw * b * rad * lis_scale;
        float coef;
        if (bl.kind == 4) {
          FilmGrad const f = thinfilm_grad(n1, n2, m.d, m.alpha, l, bl.a, bl.b, bl.c);
          coef = f.v;
          g_bin += finite_or_zero(v * f.dn);
          g_d += v * f.dd;
          g_alpha += v * f.v * dlog_lobe_dalpha(m.alpha, bl.c, bl.lnhn);
        } else {
          coef = bsdf_k(S, m, bl, x, l, front);
          if (bl.kind == 1) g_bin += finite_or_zero(v * kInvPi * bl.a);
          else if (bl.kind != 0) g_alpha += grad_blinn(S, m, bl, x, front, v);
        }
        float const nee = b * (rad * coef * lis_scale);
        g_alpha += gw * nee * dlw_L;
        rem -= nee;
      }
      if (cont) {
        // u * d ln f / dπ of the material sample's BSDF value f
        float const u = gw * rem;
        float f;
        if (ms.lobe == 4) {
          FilmGrad const t = thinfilm_grad(n1, n2, m.d, m.alpha, l, ms.a, ms.b, ms.c);
          f = t.v;
          if (f != 0.f && u != 0.f) {
            float const uf = u / f;
            g_bin += finite_or_zero(uf * t.dn);
            g_d += uf * t.dd;
            g_alpha += u * dlog_lobe_dalpha(m.alpha, ms.c, ms.lnhn);
          }
        } else {
          f = mat_mult_k(S, m, ms, x, l, front);
          if (f != 0.f && u != 0.f) {
            if (ms.lobe == 1) {
              float const alb = m.type == LGPU_MAT_LAMBERTIAN ? spec_at(S, m.spectrum[0], x) : 0.f;
              if (alb != 0.f) g_bin += finite_or_zero(u / alb);
            } else {
              g_alpha += u * dlog_lobe_dalpha(m.alpha, ms.c, ms.lnhn);
            }
          }
        }
        g_alpha += u * dlw_mat;
        b = b * (f * m_scale);
      }
      if (g_bin != 0.f) spec_grad(S, g.g_spec, m.spectrum[0], x, g_bin);
      // the words turn by one wavelength (see wf_shade)
      bt = make_float4(bt.y, bt.z, bt.w, b);
      gws = make_float4(gws.y, gws.z, gws.w, gw);
      rems = make_float4(rems.y, rems.z, rems.w, rem);
      if (cont && (k & 3) == 3) {
        out.beta[at + o_pos] = bt;
        out.acc[at + o_pos] = rems;
        out.gw[at + o_pos] = gws;
      }
    }
    // one number per material takes a term of every vertex on it: in 32 bits
    // two orders of 10^7 terms differed by 2e-5 of their sum
    if (g_d != 0.f && isfinite(g_d)) atomicAdd(g.g_mat_sum + 2 * size_t(mat), double(g_d));
    if (g_alpha != 0.f && isfinite(g_alpha)) atomicAdd(g.g_mat_sum + 2 * size_t(mat) + 1, double(g_alpha));
  }
}

__global__ void wf_material_grads(AdjointArgs g, uint32_t n_materials) {
  uint32_t const m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= n_materials) return;
  g.g_mat[4 * size_t(m)] = float(g.g_mat_sum[2 * size_t(m)]);
  g.g_mat[4 * size_t(m) + 1] = float(g.g_mat_sum[2 * size_t(m) + 1]);
  g.g_mat[4 * size_t(m) + 2] = 0.f;
  g.g_mat[4 * size_t(m) + 3] = 0.f;
}

}  // namespace

// The replay pass over work items [c0, c0 + total).
template <int K>
cudaError_t replay_chunk(const OneJob& jobs, WaveState& w, uint64_t c0, uint32_t total, bool linear,
                         const AdjointArgs& g, DevCounters* d_cnt, cudaStream_t st, WaveLaunch* run) {
  static uint32_t gen_per_sm = 0;
  if (!gen_per_sm) gen_per_sm = blocks_per_sm(wf_replay_generate<K>, 256, 0);
  WaveGrids const gr = wave_grids<K, OneJob>(run->cfg);
  uint32_t const sms = wave_occupancy<K, OneJob>().sms;
  DevCounters* const c_closest = run->on ? d_cnt + 1 : d_cnt;
  w.c0 = c0;
  wf_stream_init<<<1, 32, 0, st>>>(w);
  run->total++;
  return run_iterations(w, total, jobs.max_scatter(), st, run, [&](const WaveState& wi, bool generate) {
    wf_plan<<<1, 1, 0, st>>>(wi, total);
    if (generate) wf_replay_generate<K><<<sms * gen_per_sm, 256, 0, st>>>(jobs, wi, g);
    if (!wi.v_obj) {
      run->begin(0, st);
      launch_closest<K>(jobs, wi, gr, linear, c_closest, st);
      run->end(0, st);
      run->total += closest_launches(linear);
    }
    run->begin(2, st);
    // one block per queue chunk (see wave_chunk)
    uint32_t const sg = (wi.cap + gr.shade_block - 1) / gr.shade_block;
    bool const blinn = jobs.has_material(LGPU_MAT_BLINN), film = jobs.has_material(LGPU_MAT_THINFILM);
    bool const lists = blinn || film;
    if (!lists) {
      wf_shade_adjoint<K, LGPU_MAT_LAMBERTIAN><<<sg, gr.shade_block, 0, st>>>(jobs, wi, g);
    } else {
      wf_shade_adjoint<K, kShadeRest><<<sg, gr.shade_block, 0, st>>>(jobs, wi, g);
      cudaStream_t const fs = run->fork_side(st);
      if (film) wf_shade_adjoint<K, LGPU_MAT_THINFILM><<<sg, gr.shade_block, 0, fs>>>(jobs, wi, g);
      if (blinn) wf_shade_adjoint<K, LGPU_MAT_BLINN><<<sg, gr.shade_block, 0, film ? st : fs>>>(jobs, wi, g);
      run->end_side();
      wf_shade_adjoint<K, kShadeLamb><<<sg, gr.shade_block, 0, st>>>(jobs, wi, g);
    }
    run->wait_side(st);
    run->end(2, st);
    // plan, shade
    run->total += 2 + (generate ? 1 : 0) + (lists ? 1 : 0) + (blinn ? 1 : 0) + (film ? 1 : 0);
  });
}

// Primal render (image into d_img when not null) and gradients, chunk by
// chunk: the primal pass records, the replay pass differentiates.
template <int K>
cudaError_t launch_adjoint_k(const DevScene& S, const RenderArgs& a, WaveState* wave, uint64_t chunk_items,
                             float* d_img, const AdjointArgs& g, DevCounters* d_cnt, cudaStream_t st,
                             WaveLaunch* run) {
  OneJob const jobs{S, a, wave->npix, d_img};
  WaveState w = *wave;
  bool const linear = (a.flags & LGPU_FLAG_REFERENCE_ORDER) || S.n_objects <= 4;
  uint64_t const n_items = uint64_t(wave->npix) * a.spp;
  cudaError_t e = cudaMemsetAsync(w.film, 0, sizeof(float) * 3 * size_t(w.npix), st);
  for (uint64_t c0 = 0; c0 < n_items && e == cudaSuccess; c0 += chunk_items) {
    uint32_t const total = uint32_t(n_items - c0 < chunk_items ? n_items - c0 : chunk_items);
    e = wave_chunk<K, true>(jobs, w, c0, total, linear, d_cnt, st, run);
    if (e == cudaSuccess) e = replay_chunk<K>(jobs, w, c0, total, linear, g, d_cnt, st, run);
  }
  if (e == cudaSuccess && S.n_materials) {
    wf_material_grads<<<(S.n_materials + 255) / 256, 256, 0, st>>>(g, S.n_materials);
    run->total++;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && d_img) e = finalize_film<K>(jobs, w, st, run);
  return e;
}

}  // namespace lgpu
