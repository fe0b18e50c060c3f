// Delta-tracking path tracer (render type PT): a persistent kernel whose
// threads claim (pixel, sample) work items from a global queue with
// warp-aggregated atomics and start a new path as soon as theirs ends, so that
// lanes stay busy however long individual paths run. Replaces the
// one-launch-per-spp RenderCamera<false> loop of core/volume.cu:147-179,415-459.
#include <algorithm>
#include <cmath>

#include "mr_internal.h"
#include "mr_track.cuh"

namespace mr {

struct DTArgs {
  Medium m;
  PathScene sc;
  CameraModel cam;
  uint32_t seed, sample_offset;
  int spp;
  int row0, rows;                   // the rendered rows
  unsigned long long total;         // their pixels*spp (half the pixels with checker)
  unsigned long long* queue;        // work counter (zeroed before launch)
  unsigned long long* counters;     // [0] fetches, [1] paths, [2] loop caps
  float* store;                     // W*H*3 (nullable): one path per pixel, its radiance written, no sums
  int checker, flip;                // store only: half the pixels, those with (row + flip) & 1 == col & 1
  double* sum64;                    // (unless store) indexed by the frame's pixels, the rendered rows used
  double* sumsq64;                  // likewise (nullable)
};

// Per-pixel sums of one finished path's radiance (clamped at 0).
__device__ __forceinline__ void add_path(const DTArgs& a, unsigned pix, F3 L) {
  L = vmax(L, f3(0, 0, 0));
  size_t o = (size_t)pix * 3;
  if (a.store) {
    a.store[o] = L.x;
    a.store[o + 1] = L.y;
    a.store[o + 2] = L.z;
    return;
  }
  if (L.x == 0.0f && L.y == 0.0f && L.z == 0.0f) return;  // nothing to add (a ray beside the volume)
  atomicAdd(a.sum64 + o, (double)L.x);
  atomicAdd(a.sum64 + o + 1, (double)L.y);
  atomicAdd(a.sum64 + o + 2, (double)L.z);
  if (a.sumsq64) {
    atomicAdd(a.sumsq64 + o, (double)L.x * L.x);
    atomicAdd(a.sumsq64 + o + 1, (double)L.y * L.y);
    atomicAdd(a.sumsq64 + o + 2, (double)L.z * L.z);
  }
}

// CalculateRadiance (core/render.cuh:200-258) as paths of run_paths: a lane
// takes (pixel, sample) items from the global queue until one enters the
// volume. Bound by instruction issue (75 % of the issue slots busy). 128^3
// sphere, 256 x 256 x 64 spp: 5.03 ms with whole loops of next_vertex and
// transmittance per bounce (6.1 lanes active per instruction), 2.51 ms as
// run_paths (15.7 lanes).
struct PixelPaths {
  const DTArgs& a;
  unsigned long long P;
  RngRing rng;
  F3 rate, res;
  unsigned pix, paths;

  __device__ __forceinline__ bool begin(F3& pos, F3& rd) {
    for (;;) {
      const unsigned long long w = claim_work(a.queue);
      if (w >= a.total) return false;
      // sample-major order: concurrently traced paths are neighbouring pixels.
      const unsigned s = (unsigned)(w / P);
      pix = (unsigned)(w - (unsigned long long)s * P);
      const int per_row = a.checker ? (a.cam.width + 1) / 2 : a.cam.width;
      int row = pix / per_row;
      int col = pix - row * per_row;
      if (a.row0) {
        row += a.row0;
        pix += a.row0 * a.cam.width;
      }
      if (a.checker) {
        col = 2 * col + ((row + a.flip) & 1);
        if (col >= a.cam.width) continue;
        pix = row * a.cam.width + col;
      }
      rng.init(a.seed, pix, a.sample_offset + s, TAG_PT);
      const float jx = rng.next(), jy = rng.next();
      const F3 dir = normalize(camera_dir(a.cam, row, col, jx, jy));
      const float dis = ray_box_offset(a.cam.ori, dir);
      ++paths;
      if (dis < 0) { add_path(a, pix, sky(a.sc, dir)); continue; }
      if (a.sc.max_bounces <= 0) { add_path(a, pix, f3(0, 0, 0)); continue; }
      pos = a.cam.ori + dir * dis;
      rd = dir;
      rate = f3(1, 1, 1);
      res = f3(0, 0, 0);
      return true;
    }
  }
  __device__ __forceinline__ void escape(F3 rd) { res = res + sky(a.sc, rd) * rate; }
  __device__ __forceinline__ void scatter() { rate = rate * a.sc.scatter; }
  __device__ __forceinline__ void light(float x) { res = res + (a.sc.light_color * rate) * x; }
  __device__ __forceinline__ void finish() { add_path(a, pix, res); }
};

__global__ void __launch_bounds__(128) k_delta_track(const __grid_constant__ DTArgs a) {
  __shared__ uint32_t ring[kRingWords * 128];
  TrackStats st{0, 0};
  const int per_row = a.checker ? (a.cam.width + 1) / 2 : a.cam.width;
  PixelPaths pp{a, (unsigned long long)per_row * a.rows, {}, {}, {}, 0, 0};
  pp.rng.attach(ring);
  run_paths(pp, a.m, a.sc.alpha, a.sc.g, a.sc.L, a.sc.max_bounces, st);
  const unsigned paths = pp.paths;
  if (!a.counters) return;
  // one atomic per warp for the statistics
  unsigned f = st.fetches, c = st.caps, p = paths;
  for (int o = 16; o; o >>= 1) {
    f += __shfl_xor_sync(0xffffffffu, f, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
    p += __shfl_xor_sync(0xffffffffu, p, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(a.counters + 0, (unsigned long long)f);
    atomicAdd(a.counters + 1, (unsigned long long)p);
    if (c) atomicAdd(a.counters + 2, (unsigned long long)c);
  }
}

// The mean of spp samples from their FP64 sum.
__global__ void k_mean(const double* __restrict__ sum, float* __restrict__ x, size_t n, double spp) {
  size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
  if (i < n) x[i] = (float)(sum[i] / spp);
}

// SM count of the current device.
int sm_count() {
  static DeviceCache cache;
  return cache.get([] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
  });
}

// Resident grid of the delta tracker on the current device.
static int dt_grid() {
  static DeviceCache cache;
  return cache.get([] {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_delta_track, 128, 0);
    if (per_sm <= 0) per_sm = 1;
    return per_sm * sm_count();
  });
}

CameraModel make_camera(const mr_render_params* p) {
  CameraModel c;
  c.ori = to_f3(p->ori);
  c.fwd = normalize(-c.ori);
  c.up = to_f3(p->up);
  c.right = to_f3(p->right);
  c.width = p->width;
  c.height = p->height;
  return c;
}

PathScene make_path_scene(const mr_render_params* p) {
  PathScene sc;
  sc.L = normalize(to_f3(p->light_dir));
  sc.light_color = to_f3(p->light_color);
  sc.scatter = to_f3(p->scatter_rate);
  sc.env = to_f3(p->env_color);
  sc.alpha = p->alpha;
  sc.g = p->g;
  sc.max_bounces = p->max_bounces;
  sc.env_map = nullptr;
  sc.env_w = sc.env_h = 0;
  return sc;
}

void attach_env(PathScene& sc, const Volume* v) {
  sc.env_map = v->env_dev;
  sc.env_w = v->env_w;
  sc.env_h = v->env_h;
}

// Image_host::Sample (core/volume.hpp:22-42): bilinear with clamped texel
// indices at pos = uv * size - 1/2.
static F3 env_sample_host(const Volume* v, float u, float vv) {
  const int w = v->env_w, h = v->env_h;
  auto at = [&](int x, int y) {
    x = std::min(std::max(x, 0), w - 1);
    y = std::min(std::max(y, 0), h - 1);
    const float* q = &v->env_host[((size_t)y * w + x) * 4];
    return f3(q[0], q[1], q[2]);
  };
  const float px = u * (float)w - 0.5f, py = vv * (float)h - 0.5f;
  const int x = (int)std::floor(px), y = (int)std::floor(py);
  const float wx = px - (float)x, wy = py - (float)y;
  auto lerp3 = [](F3 a, F3 b, float t) { return a * (1.0f - t) + b * t; };
  return lerp3(lerp3(at(x, y), at(x + 1, y), wx), lerp3(at(x, y + 1), at(x + 1, y + 1), wx), wy);
}

// One light per neural pass (core/volume.cu:417-432): with probability
// rate = 4e / (4e + max(light colour)), e the environment scale, the light
// comes from the map: direction = the uniform sphere point of the R2
// sequence (Roberts2, core/vector.cu:174-178) at the pass index, colour =
// map(direction) * env * 4 / rate; otherwise the directional light with
// colour / (1 - rate). The coin is Philox (seed; pass, 0, 0, TAG_ENV) where
// the reference calls rand().
void select_env_light(const Volume* v, mr_render_params* q) {
  if (!v->env_dev || v->env_host.empty()) return;
  const F3 env = to_f3(q->env_color), lc = to_f3(q->light_color);
  const float e = std::max(env.x, std::max(env.y, env.z));
  const float m = std::max(lc.x, std::max(lc.y, lc.z));
  if (!(e > 0.0f)) return;
  const float rate = e * 4.0f / (e * 4.0f + m);
  uint32_t o[4];
  philox4x32_10(q->sample_offset, 0u, 0u, TAG_ENV, q->seed, 0u, o);
  if (u01(o[0]) < rate) {
    const float g = 1.32471795724474602596f;
    const float ax = 1.0f / g, ay = 1.0f / (g * g);
    const float n = (float)q->sample_offset;
    float rx = ax * n + 0.5f, ry = ay * n + 0.5f;
    rx -= std::floor(rx);
    ry -= std::floor(ry);
    const F3 d = uniform_sphere(rx, ry);
    const float u = std::atan2(-d.z, d.x) * (float)(0.5 / 3.1415926) + 0.5f;
    const float vv = std::acos(std::max(std::min(d.y, 1.0f), -1.0f)) * (float)(1.0 / 3.1415926);
    const F3 c = env_sample_host(v, u, vv);
    const float k = 4.0f / rate;
    q->light_dir = mr_float3{d.x, d.y, d.z};
    q->light_color = mr_float3{c.x * env.x * k, c.y * env.y * k, c.z * env.z * k};
  } else {
    const float k = 1.0f / (1.0f - rate);
    q->light_color = mr_float3{lc.x * k, lc.y * k, lc.z * k};
  }
}

int check_params(const mr_render_params* p) {
  if (!p) return set_error(MR_ERR_ARG, "render params are NULL");
  if (p->width <= 0 || p->height <= 0 || (long long)p->width * p->height > (1ll << 28))
    return set_error(MR_ERR_ARG, "image size %dx%d invalid", p->width, p->height);
  if (p->spp <= 0) return set_error(MR_ERR_ARG, "spp must be positive (got %d)", p->spp);
  if (p->max_bounces < 0) return set_error(MR_ERR_ARG, "max_bounces must be >= 0");
  if (!(p->alpha > 0.0f)) return set_error(MR_ERR_ARG, "alpha must be > 0");
  if (!(p->g > -1.0f && p->g < 1.0f)) return set_error(MR_ERR_ARG, "g = %f outside (-1, 1)", p->g);
  F3 L = to_f3(p->light_dir);
  if (!(dot(L, L) > 0.0f)) return set_error(MR_ERR_ARG, "light direction must be non-zero");
  F3 o = to_f3(p->ori);
  if (!(dot(o, o) > 0.0f)) return set_error(MR_ERR_ARG, "camera position must not be the volume centre");
  return MR_OK;
}

// Launch the tracer over `rows` rows from row0 on: adds the samples' radiance
// to sum64 (of these rows) and, unless null, its square to sumsq64. The volume's
// counters start anew with row 0.
static int launch_delta_track(Volume* v, const mr_render_params* p, int row0, int rows, double* sum64, double* sumsq64,
                              cudaStream_t s) {
  if (!v->data_set) return set_error(MR_ERR_STATE, "render before mr_volume_set_data");
  if (!v->mips_valid) return set_error(MR_ERR_STATE, "render before mr_volume_update");
  DTArgs a;
  a.m = Medium{v->density, v->res, v->max_density, p->tr_scale, 0};
  {
    int rc = density_gather_texture(v, s, &a.m.tex);
    if (rc) return rc;
  }
  a.sc = make_path_scene(p);
  attach_env(a.sc, v);
  a.cam = make_camera(p);
  a.seed = p->seed;
  a.sample_offset = p->sample_offset;
  a.spp = p->spp;
  a.row0 = row0;
  a.rows = rows;
  a.total = (unsigned long long)p->width * rows * p->spp;
  a.queue = v->d_counters + 4;
  a.counters = v->d_counters;
  a.store = nullptr;
  a.checker = a.flip = 0;
  a.sum64 = sum64 - (size_t)row0 * p->width * 3;
  a.sumsq64 = sumsq64 ? sumsq64 - (size_t)row0 * p->width * 3 : nullptr;
  MR_CUDA(cudaMemsetAsync(row0 ? a.queue : v->d_counters, 0, (row0 ? 1 : kCounters) * sizeof(unsigned long long), s));
  v->timer.mark(ST_PT, s);
  k_delta_track<<<dt_grid(), 128, 0, s>>>(a);
  v->timer.mark(ST_PT, s);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}

// One path per pixel (half the pixels with checker), sample `sample` of each
// pixel's stream: the path's radiance, clamped at 0, into dev_rgb at the
// rendered pixels. Leaves the volume's statistics alone.
int launch_path_frame(Volume* v, const mr_render_params* p, uint32_t sample, int checker, int flip, float* dev_rgb,
                      cudaStream_t s) {
  DTArgs a;
  a.m = Medium{v->density, v->res, v->max_density, p->tr_scale, 0};
  int rc = density_gather_texture(v, s, &a.m.tex);
  if (rc) return rc;
  a.sc = make_path_scene(p);
  attach_env(a.sc, v);
  a.cam = make_camera(p);
  a.seed = p->seed;
  a.sample_offset = sample;
  a.spp = 1;
  a.row0 = 0;
  a.rows = p->height;
  a.total = (unsigned long long)(checker ? (p->width + 1) / 2 : p->width) * p->height;
  a.queue = v->d_counters + kCounters;
  a.counters = nullptr;
  a.store = dev_rgb;
  a.checker = checker;
  a.flip = flip;
  a.sum64 = a.sumsq64 = nullptr;
  MR_CUDA(cudaMemsetAsync(a.queue, 0, sizeof(unsigned long long), s));
  k_delta_track<<<dt_grid(), 128, 0, s>>>(a);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}

// A pixel's samples finish in any order. Their FP64 sum is exact for all but
// extreme ranges of radiance, so two renders of one request agree, which fp32
// sums in the order of the atomics did only by timing. Where the device is
// nearly full, fewer rows at a time: the same image.
int render_pt(Volume* v, const mr_render_params* p, float* dev_rgb, cudaStream_t s) {
  const size_t row = (size_t)p->width * 3;
  int rows = p->height;
  double* sum = nullptr;
  cudaError_t e = pool_alloc((void**)&sum, rows * row * sizeof(double), s);
  while (e == cudaErrorMemoryAllocation && rows > 1) {
    rows = (rows + 1) / 2;
    e = pool_alloc((void**)&sum, rows * row * sizeof(double), s);
  }
  if (e != cudaSuccess)
    return set_error(MR_ERR_NOMEM, "sample sums of %zu bytes: %s", rows * row * sizeof(double), cudaGetErrorString(e));
  int rc = MR_OK;
  for (int r0 = 0; r0 < p->height && rc == MR_OK; r0 += rows) {
    const int m = std::min(rows, p->height - r0);
    const size_t n = m * row;
    e = cudaMemsetAsync(sum, 0, n * sizeof(double), s);
    if (e != cudaSuccess) rc = cuda_error(e, "cudaMemsetAsync(sample sums)");
    if (rc == MR_OK) rc = launch_delta_track(v, p, r0, m, sum, nullptr, s);
    if (rc == MR_OK) {
      k_mean<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(sum, dev_rgb + r0 * row, n, (double)p->spp);
      e = cudaGetLastError();
      if (e != cudaSuccess) rc = cuda_error(e, "k_mean");
    }
  }
  MR_CUDA(cudaFreeAsync(sum, s));
  return rc;
}

}  // namespace mr

using namespace mr;

extern "C" int mr_render_accumulate_f64(mr_volume* h, const mr_render_params* p, double* dev_sum,
                                        double* dev_sumsq, void* stream) {
  clear_error();
  if (!h || !dev_sum) return set_error(MR_ERR_ARG, "mr_render_accumulate_f64: NULL argument");
  int rc = check_params(p);
  if (rc) return rc;
  return launch_delta_track(&h->v, p, 0, p->height, dev_sum, dev_sumsq, (cudaStream_t)stream);
}
