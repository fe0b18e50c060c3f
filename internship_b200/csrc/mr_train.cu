// The learned part: training data from the project's own delta tracker and
// hand-written forward / backward / Adam kernels for the radiance-predictor
// network.
//
//  * k_train_points: MeanFreePathSample + GetDesiredCountSample
//    (dataGen.cu:148-216) on the GPU: rays from a sphere of radius 0.5 towards
//    the volume, up to four Woodcock vertices each over the 256^3 mip level 0
//    (the density dataGen's host code samples), with the reference's jitter /
//    view-direction rules; compacted with a global counter.
//  * k_train_labels: GetSample / GetSamples (core/render.cuh:276-315,
//    core/volume.cu:550-626): multiple-scattering radiance at a point along
//    its view direction, FP64 accumulation over the samples of a label.
//  * k_train_frames: the two random frames NNPredict draws
//    (core/render.cuh:355-369,469-523) for the view and light directions.
//  * the step: the network of core/radiancePredict.cu:370-485 (first albedo
//    channel) forward, the loss (X - log(1 + label/srp))^2 on the head output
//    X, and the backward pass, in fp32 over tiles of rows (mr_train_tile.cu)
//    or with the head's products on the tensor cores (mr_train_tc.cu).
//  * k_adam: Adam with bias correction on the fp32 master weights.
#include <algorithm>
#include <cmath>

#include "mr_internal.h"
#include "mr_net_layout.cuh"
#include "mr_track.cuh"
#include "mr_train.cuh"

namespace mr {

// ---- training points --------------------------------------------------------------

// dataGen's host DeterminateNextVertex (dataGen.cu:148-172): Woodcock free
// flight in which one draw rk per tentative collision sets both the step
// (t -= log(1 - rk) / S_max) and the acceptance test (S / S_max > rk), unlike
// the renderer's DeterminateNextVertex (core/render.cuh:138-172), which draws
// a second number for the test; the correlation shapes where the training
// points fall, so it is kept.
__device__ __forceinline__ bool next_vertex_datagen(const Medium& m, Rng& rng, float alpha, float g, F3 pos, F3 dir,
                                                    float dis, F3& npos, F3& ndir, TrackStats& st) {
  const float smax = m.max_density * alpha;
  float t = 0;
  int loop = 0;
  bool capped = true;
  while (loop++ < 10000) {
    const float rk = rng.next();
    t -= logf(1 - rk) / smax;
    if (t > dis) { npos = f3(0, 0, 0); ndir = f3(0, 0, 0); return false; }
    const float d = fetch_density(m, pos + (dir * t), st);
    if (d * alpha / smax > rk) { capped = false; break; }
    if (d < 0) t -= d;
  }
  if (capped) ++st.caps;
  const float e0 = rng.next(), e1 = rng.next();
  ndir = hg_sample_dir(e0, e1, dir, g);
  npos = (dir * t) + pos;
  return true;
}

// Six draws per vertex (keep, jitter, 3 x jitter point, view), always taken so
// that a ray's stream does not depend on which branches ran. The jitter is a
// uniform point of the ball of radius 1/128 (hash3box, dataGen.cu:115-118).
__global__ void k_train_points(Medium m, float alpha, float g, uint32_t seed, int n_rays, int cap, float* pos,
                               float* dir, unsigned* count, unsigned* caps) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n_rays) return;
  TrackStats st{0, 0};
  Rng rng;
  rng.init(seed, (uint32_t)r, 0u, TAG_GEN);
  const float e0 = rng.next(), e1 = rng.next(), e2 = rng.next(), e3 = rng.next();
  const F3 ori = uniform_sphere(e0, e1) * 0.5f;
  const F3 d = normalize(uniform_sphere(e2, e3) + normalize(ori * -1.0f));
  const float dis = ray_box_offset(ori, d);
  if (dis >= 0) {
    F3 sp = ori + d * dis, rd = d;
    for (int i = 0; i < 4; ++i) {
      const float dd = ray_box_distance(sp, rd);
      F3 np, nd;
      if (!next_vertex_datagen(m, rng, alpha, g, sp, rd, dd, np, nd, st)) break;
      const float uk = rng.next(), uj = rng.next(), j0 = rng.next(), j1 = rng.next(), j2 = rng.next(),
                  uv = rng.next();
      const F3 dv = sp - np;
      if (i == 0 || dot(dv, dv) > 1.0f / 64.0f || uk > 0.9f) {
        F3 p = np;
        if (uj > 0.5f) p = p + uniform_sphere(j0, j1) * (cbrtf(j2) * (1.0f / 128.0f));
        const F3 v = uv > 0.25f ? d : rd;
        const unsigned k = atomicAdd(count, 1u);
        if (k < (unsigned)cap) {
          pos[3 * k] = p.x; pos[3 * k + 1] = p.y; pos[3 * k + 2] = p.z;
          dir[3 * k] = v.x; dir[3 * k + 1] = v.y; dir[3 * k + 2] = v.z;
        }
      }
      sp = np;
      rd = nd;
    }
  }
  if (st.caps) atomicAdd(caps, st.caps);
}

// ---- labels -----------------------------------------------------------------------

struct LabelArgs {
  Medium m;
  const float* pos;
  const float* dir;
  int n, spp, chunk, max_bounces;
  F3 L;
  float alpha, g, albedo;
  uint32_t seed;
  double* sum;
  unsigned long long* queue;  // work counter
  unsigned* caps;
  PathScene env;  // only the environment fields: map, size and scale (black without a map)
};

// Work item = (label k, chunk of `chunk` samples), claimed from a global queue
// so that long and short paths balance across the grid; a lane runs the
// samples of its item one after the other as paths of run_paths. Sample s of
// label k uses the stream (seed; k, s, ., TAG_LABEL).
// 4096 labels x 256 spp on a 256^3 cloud: 22.0 ms with a chunk of 64 samples a
// lane (16 k lanes at work on a GPU that holds 114 k) and whole paths in
// lockstep; 7.4 ms with run_paths; 1.03 ms with the chunk sized to the grid.
// Density through texture gathers instead of texel loads: within 2 %, so no
// layered copy of the grid is made for labels.
struct LabelPaths {
  const LabelArgs& a;
  unsigned long long per, total;
  RngRing rng;
  F3 p0, d0;
  double acc;
  float rate, res;
  int k, s, s1;  // label, next sample and end of the item (s == s1: no item)

  __device__ __forceinline__ bool begin(F3& pos, F3& rd) {
    if (s == s1) {
      if (k >= 0) atomicAdd(a.sum + k, acc);
      const unsigned long long w = claim_work(a.queue);
      if (w >= total) return false;
      k = (int)(w / per);
      s = (int)(w % per) * a.chunk;
      s1 = min(a.spp, s + a.chunk);
      p0 = f3(a.pos[3 * k], a.pos[3 * k + 1], a.pos[3 * k + 2]);
      d0 = f3(a.dir[3 * k], a.dir[3 * k + 1], a.dir[3 * k + 2]);
      acc = 0.0;
    }
    rng.init(a.seed, (uint32_t)k, (uint32_t)s, TAG_LABEL);
    ++s;
    const float e0 = rng.next(), e1 = rng.next();
    rd = hg_sample_dir(e0, e1, d0, a.g);
    pos = p0;
    rate = 1.0f;
    res = 0.0f;
    return true;
  }
  // SkyBox(dir) * rate (core/render.cuh:294-296), channel 0
  __device__ __forceinline__ void escape(F3 rd) {
    if (a.env.env_map) res = res + rate * sky(a.env, rd).x;
  }
  __device__ __forceinline__ void scatter() { rate = rate * 1.001f * a.albedo; }
  __device__ __forceinline__ void light(float x) { res = res + rate * x; }
  __device__ __forceinline__ void finish() { acc += (double)res; }
};

__global__ void __launch_bounds__(128) k_train_labels(const __grid_constant__ LabelArgs a) {
  __shared__ uint32_t ring[kRingWords * 128];
  const unsigned long long per = (unsigned long long)((a.spp + a.chunk - 1) / a.chunk);
  TrackStats st{0, 0};
  LabelPaths lp{a, per, per * (unsigned long long)a.n, {}, {}, {}, 0.0, 0.0f, 0.0f, -1, 0, 0};
  lp.rng.attach(ring);
  run_paths(lp, a.m, a.alpha, a.g, a.L, a.max_bounces, st);
  if (st.caps) atomicAdd(a.caps, st.caps);
}

// Resident grid of the label kernel on the current device.
static int label_grid() {
  static DeviceCache cache;
  return cache.get([] {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_train_labels, 128, 0);
    return std::max(per_sm, 1) * sm_count();
  });
}

// Frames of NNPredict for view direction dir[k] and light L: stream
// (seed; k, 1, ., TAG_MISC).
__global__ void k_train_frames(const float* dir, int n, F3 L, uint32_t seed, float* frame) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  Rng rng;
  rng.init(seed, (uint32_t)k, 1u, TAG_MISC);
  F3 X, Y, Z, LX, ly, lz;
  frame_from(rng, f3(dir[3 * k], dir[3 * k + 1], dir[3 * k + 2]), X, Y, Z);
  frame_from(rng, L, LX, ly, lz);
  float* f = frame + 12 * (size_t)k;
  f[0] = X.x; f[1] = X.y; f[2] = X.z; f[3] = Y.x; f[4] = Y.y; f[5] = Y.z;
  f[6] = Z.x; f[7] = Z.y; f[8] = Z.z; f[9] = LX.x; f[10] = LX.y; f[11] = LX.z;
}

// ---- the training step -------------------------------------------------------------

__global__ void k_adam(float* w, float* m, float* v, float* grad, int n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = grad[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  grad[i] = 0.0f;
}

struct Trainer {
  float* w = nullptr;
  float* m = nullptr;
  float* v = nullptr;
  float* grad = nullptr;
  float* loss = nullptr;
  int step = 0;
  float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  int precision = MR_PREC_FP32;
  // The step's buffers (TrainWork) for up to `cap` rows, grown on demand to
  // at most kStepRows: larger batches run in pieces, and so do batches whose
  // buffers do not fit into the device's free memory.
  float* work = nullptr;
  size_t cap = 0;
  uint8_t* img = nullptr;  // BF16 head weights, rebuilt from w every step
  int* err = nullptr;      // set when a bounded wait of the head kernel gives up
};

// Rows of one pass of a step: 65,536 rows take 361 MB of buffers.
constexpr int kStepRows = 65536;
static_assert(kStepRows * kTrainWorkFloats * sizeof(float) == 360710144, "the figure above");

int launch_head_pack(const float* w, uint8_t* img, cudaStream_t s);
int launch_head_tc(const TrainArgs& a, const uint8_t* img, int* err, cudaStream_t s);
size_t head_image_bytes();

}  // namespace mr

using namespace mr;

struct mr_trainer { Trainer t; };

static int check_volume_ready(const mr_volume* h) {
  if (!h) return set_error(MR_ERR_ARG, "NULL volume");
  if (!h->v.data_set || !h->v.mips_valid) return set_error(MR_ERR_STATE, "volume needs mr_volume_set_data and _update");
  return MR_OK;
}

extern "C" int mr_train_points(mr_volume* h, float alpha, float g, uint32_t seed, int32_t n_rays, int32_t cap,
                               float* dev_pos, float* dev_dir, int32_t* host_count, void* stream) {
  clear_error();
  int rc = check_volume_ready(h);
  if (rc) return rc;
  if (!dev_pos || !dev_dir || !host_count) return set_error(MR_ERR_ARG, "mr_train_points: NULL argument");
  if (n_rays < 0 || cap < 0 || !(alpha > 0.0f)) return set_error(MR_ERR_ARG, "mr_train_points: bad n_rays/cap/alpha");
  Volume* v = &h->v;
  cudaStream_t s = (cudaStream_t)stream;
  MR_CUDA(cudaMemsetAsync(v->d_counters, 0, kCounters * sizeof(unsigned long long), s));
  unsigned* cnt = reinterpret_cast<unsigned*>(v->d_counters + 4);
  unsigned* caps = reinterpret_cast<unsigned*>(v->d_counters + 5);
  // dataGen's Woodcock steps read VolumeRender::DensityAtPosition(0, p): the
  // 256^3 level 0 of the mip pyramid, trilinear with a zero border
  // (core/volume.cu:1495-1497, 675-703), under the density grid's majorant.
  if (n_rays > 0)
    k_train_points<<<(n_rays + 127) / 128, 128, 0, s>>>(Medium{v->mips, 256, v->max_density, 1.0f, 0}, alpha, g,
                                                        seed, n_rays, cap, dev_pos, dev_dir, cnt, caps);
  MR_CUDA(cudaGetLastError());
  unsigned c = 0;
  MR_CUDA(cudaMemcpyAsync(&c, cnt, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
  MR_CUDA(cudaStreamSynchronize(s));
  *host_count = (int32_t)std::min<unsigned>(c, (unsigned)cap);
  return MR_OK;
}

extern "C" int mr_train_labels(mr_volume* h, const float* dev_pos, const float* dev_dir, int32_t n, mr_float3 light_dir,
                               float alpha, float g, float albedo, int32_t max_bounces, int32_t spp, uint32_t seed,
                               double* dev_sum, void* stream) {
  clear_error();
  int rc = check_volume_ready(h);
  if (rc) return rc;
  if (!dev_pos || !dev_dir || !dev_sum) return set_error(MR_ERR_ARG, "mr_train_labels: NULL argument");
  if (n < 0 || spp <= 0 || max_bounces < 0 || !(alpha > 0.0f))
    return set_error(MR_ERR_ARG, "mr_train_labels: bad n/spp/max_bounces/alpha");
  if (n == 0) return MR_OK;
  Volume* v = &h->v;
  cudaStream_t s = (cudaStream_t)stream;
  MR_CUDA(cudaMemsetAsync(v->d_counters, 0, kCounters * sizeof(unsigned long long), s));
  if (max_bounces == 0) return MR_OK;  // no vertex: every sum stays as it is
  LabelArgs a;
  a.m = Medium{v->density, v->res, v->max_density, 1.0f, 0};
  a.pos = dev_pos;
  a.dir = dev_dir;
  a.n = n;
  a.spp = spp;
  // Samples a lane runs per claimed item: enough items for eight per resident
  // lane, so that labels in small numbers still fill the GPU, and at most 64
  // samples per FP64 atomic.
  const int grid = label_grid();
  a.chunk = (int)std::min<long long>(64, std::max<long long>(1, (long long)n * spp / (8ll * 128 * grid)));
  a.chunk = std::min(a.chunk, spp);
  a.max_bounces = max_bounces;
  a.L = normalize(to_f3(light_dir));
  a.alpha = alpha;
  a.g = g;
  a.albedo = albedo;
  a.seed = seed;
  a.sum = dev_sum;
  a.queue = v->d_counters + 4;
  a.caps = reinterpret_cast<unsigned*>(v->d_counters + 2);
  a.env = PathScene{};
  a.env.env = f3(1.0f, 1.0f, 1.0f);  // the map at unit scale; black without one
  attach_env(a.env, v);
  k_train_labels<<<grid, 128, 0, s>>>(a);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}

extern "C" int mr_train_frames(const float* dev_dir, int32_t n, mr_float3 light_dir, uint32_t seed, float* dev_frame,
                               void* stream) {
  clear_error();
  if (!dev_dir || !dev_frame) return set_error(MR_ERR_ARG, "mr_train_frames: NULL argument");
  if (n < 0) return set_error(MR_ERR_ARG, "n < 0");
  if (n == 0) return MR_OK;
  k_train_frames<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(dev_dir, n, normalize(to_f3(light_dir)), seed,
                                                                   dev_frame);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}

extern "C" int mr_trainer_create(const float* host_weights, size_t count, mr_trainer** out) {
  clear_error();
  if (!out || !host_weights) return set_error(MR_ERR_ARG, "mr_trainer_create: NULL argument");
  *out = nullptr;
  if (count != MR_WEIGHT_TOTAL) return set_error(MR_ERR_ARG, "weight blob has %zu floats, expected %d", count, MR_WEIGHT_TOTAL);
  mr_trainer* h = new mr_trainer();
  Trainer& t = h->t;
  const size_t bytes = MR_WEIGHT_TOTAL * sizeof(float);
  cudaError_t e = cudaMalloc(&t.w, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&t.m, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&t.v, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&t.grad, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&t.loss, sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(t.w, host_weights, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(t.m, 0, bytes);
  if (e == cudaSuccess) e = cudaMemset(t.v, 0, bytes);
  if (e == cudaSuccess) e = cudaMemset(t.grad, 0, bytes);
  if (e != cudaSuccess) {
    mr_trainer_destroy(h);
    return set_error(MR_ERR_NOMEM, "mr_trainer_create: %s", cudaGetErrorString(e));
  }
  *out = h;
  return MR_OK;
}

extern "C" int mr_trainer_destroy(mr_trainer* h) {
  if (!h) return MR_OK;
  cudaFree(h->t.w);
  cudaFree(h->t.m);
  cudaFree(h->t.v);
  cudaFree(h->t.grad);
  cudaFree(h->t.loss);
  cudaFree(h->t.work);
  cudaFree(h->t.img);
  cudaFree(h->t.err);
  delete h;
  return MR_OK;
}

extern "C" int mr_trainer_set_precision(mr_trainer* h, int32_t precision) {
  clear_error();
  if (!h) return set_error(MR_ERR_ARG, "mr_trainer_set_precision: NULL trainer");
  if (precision != MR_PREC_FP32 && precision != MR_PREC_BF16)
    return set_error(MR_ERR_ARG, "training precision must be MR_PREC_FP32 or MR_PREC_BF16 (got %d)", precision);
  Trainer& t = h->t;
  if (precision == MR_PREC_BF16 && !t.img) {
    MR_CUDA(cudaMalloc(&t.img, head_image_bytes()));
    MR_CUDA(cudaMalloc(&t.err, sizeof(int)));
    MR_CUDA(cudaMemset(t.err, 0, sizeof(int)));
  }
  t.precision = precision;
  return MR_OK;
}

// MR_ERR_TIMEOUT (and a reset) when a bounded wait of the BF16 head gave up.
static int head_error(Trainer& t) {
  if (!t.err) return MR_OK;
  int e = 0;
  MR_CUDA(cudaMemcpy(&e, t.err, sizeof(int), cudaMemcpyDeviceToHost));
  if (!e) return MR_OK;
  MR_CUDA(cudaMemset(t.err, 0, sizeof(int)));
  return set_error(MR_ERR_TIMEOUT, "BF16 training head: an mbarrier wait timed out");
}

static int fwd_bwd(Trainer& t, const float* desc, const float* aux, const float* label, int n, cudaStream_t s) {
  MR_CUDA(cudaMemsetAsync(t.loss, 0, sizeof(float), s));
  const auto whole_tiles = [](size_t rows) { return (rows + kTrainRows - 1) / kTrainRows * kTrainRows; };
  const size_t need = whole_tiles(std::min(n, kStepRows));
  // Under a capture the buffers are nodes of the graph, also where t.work is
  // large enough: a later call with more rows frees t.work, and a replay must
  // not write there.
  float* temp = nullptr;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (s && cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusActive) {
    MR_CUDA(cudaMallocAsync(&temp, need * kTrainWorkFloats * sizeof(float), s));
  } else if (need > t.cap) {
    cudaFree(t.work);
    t.work = nullptr;
    t.cap = 0;
    // where the device is nearly full, buffers for fewer rows and smaller pieces
    size_t rows = need;
    cudaError_t e = cudaMalloc(&t.work, rows * kTrainWorkFloats * sizeof(float));
    while (e == cudaErrorMemoryAllocation && rows > kTrainRows) {
      rows = whole_tiles(rows / 2);
      e = cudaMalloc(&t.work, rows * kTrainWorkFloats * sizeof(float));
    }
    cudaGetLastError();  // the failed attempts'
    if (e != cudaSuccess) return set_error(MR_ERR_NOMEM, "training buffers for %zu rows: %s", rows, cudaGetErrorString(e));
    t.cap = rows;
  }
  TrainArgs a;
  a.w = t.w;
  a.grad = t.grad;
  a.inv_batch = 1.0f / (float)n;
  a.loss = t.loss;
  float* p = temp ? temp : t.work;
  a.wk.rows = temp ? need : t.cap;
  auto take = [&](size_t floats) {
    float* q = p;
    p += floats * a.wk.rows;
    return q;
  };
  a.wk.h0 = take(128);
  a.wk.dh0 = take(128);
  a.wk.pool = take(72);
  a.wk.gate = take(36);
  a.wk.sp = take(6);
  a.wk.dgate = take(72);
  a.wk.dsp = take(12);
  a.wk.a3 = take(32);
  a.wk.da3 = take(32);
  a.wk.xs = take(3 * kTrunkSaved);
  a.wk.mask = reinterpret_cast<uint16_t*>(take(kTrunkMaskFloats));
  const bool tc = t.precision == MR_PREC_BF16;
  int rc = tc ? launch_head_pack(t.w, t.img, s) : (int)MR_OK;
  const int piece = (int)std::min<size_t>(kStepRows, a.wk.rows);
  for (int r0 = 0; r0 < n && !rc; r0 += piece) {
    a.n = std::min(piece, n - r0);
    a.desc = desc + (size_t)r0 * 576;
    a.aux = aux + (size_t)r0 * 5;
    a.label = label + r0;
    rc = launch_train_trunk_fwd(a, s);
    if (!rc) rc = tc ? launch_head_tc(a, t.img, t.err, s) : launch_train_head(a, s);
    if (!rc) rc = launch_train_trunk_bwd(a, s);
  }
  if (temp) MR_CUDA(cudaFreeAsync(temp, s));
  return rc;
}

extern "C" int mr_trainer_gradient(mr_trainer* h, const float* dev_desc, const float* dev_aux, const float* dev_label,
                                   int32_t n, float* host_grad, float* host_loss, void* stream) {
  clear_error();
  if (!h || !dev_desc || !dev_aux || !dev_label || !host_grad) return set_error(MR_ERR_ARG, "mr_trainer_gradient: NULL argument");
  if (n <= 0) return set_error(MR_ERR_ARG, "n <= 0");
  cudaStream_t s = (cudaStream_t)stream;
  Trainer& t = h->t;
  MR_CUDA(cudaMemsetAsync(t.grad, 0, MR_WEIGHT_TOTAL * sizeof(float), s));
  int rc = fwd_bwd(t, dev_desc, dev_aux, dev_label, n, s);
  if (rc) return rc;
  MR_CUDA(cudaMemcpyAsync(host_grad, t.grad, MR_WEIGHT_TOTAL * sizeof(float), cudaMemcpyDeviceToHost, s));
  float l = 0.0f;
  MR_CUDA(cudaMemcpyAsync(&l, t.loss, sizeof(float), cudaMemcpyDeviceToHost, s));
  MR_CUDA(cudaMemsetAsync(t.grad, 0, MR_WEIGHT_TOTAL * sizeof(float), s));
  MR_CUDA(cudaStreamSynchronize(s));
  if (host_loss) *host_loss = l;
  return head_error(t);
}

extern "C" int mr_trainer_step(mr_trainer* h, const float* dev_desc, const float* dev_aux, const float* dev_label,
                               int32_t n, float lr, float* host_loss, void* stream) {
  clear_error();
  if (!h || !dev_desc || !dev_aux || !dev_label) return set_error(MR_ERR_ARG, "mr_trainer_step: NULL argument");
  if (n <= 0 || !(lr > 0.0f)) return set_error(MR_ERR_ARG, "mr_trainer_step: bad n / lr");
  cudaStream_t s = (cudaStream_t)stream;
  Trainer& t = h->t;
  int rc = fwd_bwd(t, dev_desc, dev_aux, dev_label, n, s);
  if (rc) return rc;
  ++t.step;
  const float c1 = 1.0f - std::pow(t.b1, (float)t.step), c2 = 1.0f - std::pow(t.b2, (float)t.step);
  k_adam<<<(MR_WEIGHT_TOTAL + 255) / 256, 256, 0, s>>>(t.w, t.m, t.v, t.grad, MR_WEIGHT_TOTAL, lr, t.b1, t.b2, t.eps,
                                                        c1, c2);
  MR_CUDA(cudaGetLastError());
  if (host_loss) {
    float l = 0.0f;
    MR_CUDA(cudaMemcpyAsync(&l, t.loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    MR_CUDA(cudaStreamSynchronize(s));
    *host_loss = l;
    return head_error(t);
  }
  return MR_OK;
}

extern "C" int mr_trainer_weights(const mr_trainer* h, float* host_out, size_t count) {
  clear_error();
  if (!h || !host_out) return set_error(MR_ERR_ARG, "mr_trainer_weights: NULL argument");
  if (count != MR_WEIGHT_TOTAL) return set_error(MR_ERR_ARG, "expected %d floats", MR_WEIGHT_TOTAL);
  MR_CUDA(cudaMemcpy(host_out, h->t.w, MR_WEIGHT_TOTAL * sizeof(float), cudaMemcpyDeviceToHost));
  return MR_OK;
}
