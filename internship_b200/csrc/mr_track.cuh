// Woodcock delta tracking on a raw fp32 density grid: free flight, NEE
// transmittance and the path estimator (core/render.cuh:93-258).
#pragma once
#include "mr_device.cuh"

namespace mr {

struct Medium {
  const float* __restrict__ density;  // res^3, x-major
  int res;
  float max_density;  // global majorant (before alpha)
  float tr_scale;
  cudaTextureObject_t tex;  // layered copy of density read by texture gathers, or 0: texel loads
};

struct TrackStats {
  unsigned fetches;
  unsigned caps;
};

__device__ __forceinline__ float fetch_density(const Medium& m, F3 pos, TrackStats& st) {
  ++st.fetches;
  return m.tex ? tri_border_tex(m.tex, m.res, pos + 0.5f) : tri_border(m.density, m.res, pos + 0.5f);
}

// DeterminateNextVertex (core/render.cuh:138-172). R is Rng or RngRing;
// prime() keeps the lanes' Philox calls at the same iterations.
template <class R>
__device__ __forceinline__ bool next_vertex(const Medium& m, R& rng, float alpha, float g, F3 pos, F3 dir,
                                            float dis, F3& npos, F3& ndir, TrackStats& st) {
  const DivBy over_smax(m.max_density * alpha);
  float t = 0;
  int loop = 0;
  bool capped = true;
  while (loop++ < 10000) {
    if (loop & 1) rng.prime();
    float rk = rng.take();
    t -= over_smax(logf(1 - rk));
    if (t > dis) { npos = f3(0, 0, 0); ndir = f3(0, 0, 0); return false; }
    rk = rng.take();
    float d = fetch_density(m, pos + (dir * t), st);
    if (over_smax(d * alpha) > rk) { capped = false; break; }
    if (d < 0) t -= d;
  }
  if (capped) ++st.caps;
  float e0 = rng.next();
  float e1 = rng.next();
  ndir = hg_sample_dir(e0, e1, dir, g);
  npos = (dir * t) + pos;
  return true;
}

// Tr (core/render.cuh:93-136): ratio tracking while tr > 0.5, then delta tracking.
template <class R>
__device__ __forceinline__ float transmittance(const Medium& m, R& rng, F3 pos, F3 dir, float dis, float alpha,
                                               TrackStats& st) {
  const DivBy over_smax(m.max_density * alpha);
  float tr = 1, t = 0;
  int loop = 0;
  while (loop++ < 10000 && tr > 0.5f) {
    if (loop & 1) rng.prime();
    float rk = rng.take();
    t -= over_smax(logf(1 - rk)) * m.tr_scale;
    if (t > dis) break;
    float d = fetch_density(m, pos + (dir * t), st);
    tr *= 1 - fmaxf(0.0f, over_smax(d * alpha));
    if (d < 0) t -= d;
  }
  while (loop++ < 10000 && tr > 0.001f) {
    rng.prime();
    float rk = rng.take();
    t -= over_smax(logf(1 - rk)) * m.tr_scale;
    if (t > dis) break;
    float d = fetch_density(m, pos + (dir * t), st);
    if (rng.take() < fmaxf(0.0f, over_smax(d * alpha))) { tr = 0; break; }
    if (d < 0) t -= d;
  }
  if (loop > 10000) ++st.caps;
  return tr;
}

// GetMatrixFromNormal (core/render.cuh:355-369), rejection capped at 64 tries.
template <class R>
__device__ __forceinline__ void frame_from(R& rng, F3 v1, F3& a, F3& b, F3& c) {
  v1 = normalize(v1);
  for (int tries = 0; tries < 64; ++tries) {
    float ex = rng.next();
    float ey = rng.next();
    F3 r = uniform_sphere(ex, ey);
    if (fabsf(dot(r, v1)) < 0.01f) continue;
    F3 v2 = normalize(cross(v1, r));
    a = v1; b = v2; c = cross(v2, v1);
    return;
  }
  F3 r = fabsf(v1.x) < 0.5f ? f3(1, 0, 0) : f3(0, 1, 0);
  F3 v2 = normalize(cross(v1, r));
  a = v1; b = v2; c = cross(v2, v1);
}

struct PathScene {
  F3 L;            // normalized light direction
  F3 light_color;
  F3 scatter;      // albedo per channel
  F3 env;          // radiance of escaped rays, or the scale of the environment map
  float alpha, g;
  int max_bounces;
  const float4* env_map;  // SetHDRI image (w x h, row 0 = straight up), or null
  int env_w, env_h;
};

// Environment radiance seen along dir: SkyBox (core/render.cuh:57-61), the
// environment map at u = atan2(-d.z, d.x) / 2 pi + 1/2, v = acos(d.y) / pi,
// bilinear with wrap addressing as the reference's texture filter reads it
// (here in fp32), times the env scale (SetEnvExp); without a map, the
// constant env colour.
__device__ __forceinline__ F3 env_lookup(const float4* __restrict__ map, int w, int h, F3 scale, F3 d) {
  const float u = atan2f(-d.z, d.x) * (float)(0.5 / 3.1415926) + 0.5f;
  const float v = acosf(fmaxf(fminf(d.y, 1.0f), -1.0f)) * (float)(1.0 / 3.1415926);
  const float x = u * (float)w - 0.5f, y = v * (float)h - 0.5f;
  const float x0 = floorf(x), y0 = floorf(y);
  const float fx = x - x0, fy = y - y0;
  int i0 = (int)x0 % w, j0 = (int)y0 % h;
  if (i0 < 0) i0 += w;
  if (j0 < 0) j0 += h;
  const int i1 = i0 + 1 == w ? 0 : i0 + 1, j1 = j0 + 1 == h ? 0 : j0 + 1;
  const float4 a = __ldg(map + (size_t)j0 * w + i0), b = __ldg(map + (size_t)j0 * w + i1);
  const float4 c = __ldg(map + (size_t)j1 * w + i0), e = __ldg(map + (size_t)j1 * w + i1);
  const float r = lerpf(lerpf(a.x, b.x, fx), lerpf(c.x, e.x, fx), fy);
  const float g = lerpf(lerpf(a.y, b.y, fx), lerpf(c.y, e.y, fx), fy);
  const float bl = lerpf(lerpf(a.z, b.z, fx), lerpf(c.z, e.z, fx), fy);
  return f3(r * scale.x, g * scale.y, bl * scale.z);
}
__device__ __forceinline__ F3 sky(const PathScene& sc, F3 d) {
  return sc.env_map ? env_lookup(sc.env_map, sc.env_w, sc.env_h, sc.env, d) : sc.env;
}

struct CameraModel {
  F3 ori, fwd, up, right;
  int width, height;
};

// Camera ray of pixel (row, col) (core/volume.cu:155-163, row-major W x H).
__device__ __forceinline__ F3 camera_dir(const CameraModel& c, int row, int col, float jx, float jy) {
  float u = 1.0f - ((float)col + jx) / (float)c.width;
  float v = 1.0f - ((float)row + jy) / (float)c.height;
  F3 d = c.fwd + (c.right * (u * 2 - 1)) + (c.up * (v * 2 - 1));
  return normalize(d);
}

// Warp-aggregated claim of one work item per calling lane.
__device__ __forceinline__ unsigned long long claim_work(unsigned long long* counter) {
  unsigned mask = __activemask();
  int lane = threadIdx.x & 31;
  int leader = __ffs(mask) - 1;
  unsigned lt = mask & ((1u << lane) - 1u);
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(counter, (unsigned long long)__popc(mask));
  base = __shfl_sync(mask, base, leader);
  return base + __popc(lt);
}


// ---- path machine -------------------------------------------------------------
// The path estimator (free flight, then NEE transmittance at each vertex) as
// one step per loop iteration: a draw, a step length and one density fetch,
// whether a lane is in free flight (next_vertex), ratio tracking or delta
// tracking (transmittance). Lanes of a warp then share the expensive part of
// an iteration although their loops have different lengths (a ray beside the
// medium rejects tens of collisions while one inside it scatters at once).
// What only some lanes need, a collision's new direction or the next path,
// waits until kWaitCollide or kWaitNext lanes of the warp need it, or no lane
// can step. Every
// path draws the same numbers in the same order, with the same arithmetic, as
// next_vertex and transmittance do.
//
// P supplies the path: rng (RngRing); begin(pos, rd) starts the next one or
// returns false; escape(rd) adds the environment; scatter() applies the
// albedo at a collision; light(x) adds the light's term at the current
// vertex, x = transmittance * phase; finish() takes the path's result.
// Sphere scene / cloud labels at (collide, next) lanes waited for: (4, 8) 2.57
// / 7.42 ms, (2, 8) 2.55 / 7.45, (4, 4) 2.71 / 7.21, (8, 8) 2.79 / 8.08,
// (12, 16) 3.09 / 9.04; one threshold of 12 for both 3.30 / 9.22.
constexpr int kWaitCollide = 4, kWaitNext = 8;

// dot(a, b) with its two fused steps in a fixed order (which of the three
// products is rounded first is otherwise the compiler's choice, and changes
// the last bit of a path's phase value with the code around it).
__device__ __forceinline__ float dot_yxz(F3 a, F3 b) {
  return __fmaf_rn(a.z, b.z, __fmaf_rn(a.x, b.x, __fmul_rn(a.y, b.y)));
}

// ray_box_distance with its fused steps spelled out, for the same reason: a
// last bit of the distance decides, in one path of 1e8, whether a collision
// next to the box's face counts.
__device__ __forceinline__ float box_exit_path(F3 p, F3 dir) {
  const F3 d = inv3(dir);
  auto axis = [](float p, float d) {
    const float face = __fmul_rn(0.5f, d);
    return fmaxf(__fmaf_rn(-p, d, face), __fmaf_rn(-p, d, -face));
  };
  return fminf(axis(p.x, d.x), fminf(axis(p.y, d.y), axis(p.z, d.z)));
}

template <class P>
__device__ __forceinline__ void run_paths(P& p, const Medium& m, float alpha, float g, F3 L, int max_bounces,
                                          TrackStats& st) {
  enum { FLIGHT = 0, RATIO = 1, DELTA = 2, COLLIDE = 3, ESCAPED = 4, ENDED = 5, IDLE = 6, DONE = 7 };
  const DivBy over_smax(m.max_density * alpha);
  int mode = IDLE, loop = 0, bounce = 0;
  F3 pos = f3(0, 0, 0), rd = f3(0, 0, 0);
  float t = 0, dis = 0, dis_next = 0, tr = 0, ph = 0;

  auto step = [&] {
    const bool flight = mode == FLIGHT, ratio = mode == RATIO;
    const float r0 = p.rng.take();
    t -= over_smax(logf(1 - r0)) * (flight ? 1.0f : m.tr_scale);
    const bool out = t > dis;
    float d = 0;
    if (!out) d = fetch_density(m, pos + ((flight ? rd : L) * t), st);
    const float q = over_smax(d * alpha);
    const float qc = fmaxf(0.0f, q);
    const bool two = !out && !ratio;  // free flight and delta tracking draw again
    const float rk = p.rng.take_if(two);
    const bool hit = two && (flight ? q > rk : rk < qc);
    if (d < 0 && !hit) t -= d;
    if (flight) {
      if (hit) mode = COLLIDE;
      if (out) mode = ESCAPED;
      if (++loop >= 10000 && mode == FLIGHT) {
        ++st.caps;
        mode = COLLIDE;
      }
    } else {
      if (ratio) tr *= 1 - qc;
      else if (hit) tr = 0;
      bool stay = false;
      if (ratio && !out) {
        stay = loop < 10000 && tr > 0.5f;
        ++loop;
      }
      if (!stay) {
        bool end = !ratio && (out || hit);
        if (!end) {  // entry test of the delta-tracking loop
          end = !(loop < 10000 && tr > 0.001f);
          ++loop;
          mode = DELTA;
        }
        if (end) {
          if (loop > 10000) ++st.caps;
          p.light(tr * ph);
          ++bounce;
          mode = bounce >= max_bounces ? ENDED : FLIGHT;
          t = 0;
          loop = 0;
          dis = dis_next;
        }
      }
    }
  };

  int nc = 0, ne = 32;
  bool any = false;
  for (;;) {
    if ((ne >= kWaitNext || !any) && mode >= ESCAPED && mode != DONE) {
      if (mode == ESCAPED) p.escape(rd);
      if (mode != IDLE) p.finish();
      if (p.begin(pos, rd)) {
        t = 0;
        loop = 0;
        bounce = 0;
        dis = box_exit_path(pos, rd);
        mode = FLIGHT;
      } else {
        mode = DONE;
      }
    }
    if ((nc >= kWaitCollide || !any) && mode == COLLIDE) {
      const float e0 = p.rng.next(), e1 = p.rng.next();
      const F3 nd = hg_sample_dir(e0, e1, rd, g);
      pos = (rd * t) + pos;
      p.scatter();
      dis = box_exit_path(pos, L);
      ph = hg_phase(dot_yxz(rd, L), g);
      rd = nd;
      dis_next = box_exit_path(pos, rd);
      t = 0;
      tr = 1;
      loop = 1;
      mode = RATIO;
    }
    if (__all_sync(0xffffffffu, mode == DONE)) break;
    do {
#pragma unroll 1  // one copy of the step: the loop stays in the instruction cache
      for (int j = 0; j < 2; ++j) {
        if (mode <= DELTA) {
          if (j == 0) p.rng.prime();
          step();
        }
      }
      any = __any_sync(0xffffffffu, mode <= DELTA);
      nc = __popc(__ballot_sync(0xffffffffu, mode == COLLIDE));
      ne = __popc(__ballot_sync(0xffffffffu, mode >= ESCAPED && mode != DONE));
    } while (any && nc < kWaitCollide && ne < kWaitNext);
  }
}

}  // namespace mr
