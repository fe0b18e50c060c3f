// The training step's fp32 kernels over tiles of 64 rows: forward and
// backward of the radiance-predictor network (core/radiancePredict.cu:370-485,
// first albedo channel) as block GEMMs in shared memory.
//
//   k_train_stats   pooled descriptor statistics, the squeeze-excitation
//                   gates of every block, the trunk-output gates and LGGS
//   k_train_trunk_fwd, k_train_trunk_bwd
//                   the trunks of one branch (density, transmittance or
//                   phase): forward to the head input, backward from its
//                   gradient
//   k_train_head    LC0 / LC1 / LC2, the tail and the loss, forward and
//                   backward (fp32 step)
//   k_train_tail    the tail and the loss alone (BF16 step, between the
//                   tensor-core head's halves in mr_train_tc.cu)
//   k_train_gates   backward of the squeeze-excitation and output gates
//
// The gates depend on descriptor statistics alone, so the three branches of
// the trunks are independent of one another given the gates, and each CTA
// runs one branch with its weights (25 KB) in shared memory.
//
// A tile's activations are stored feature-major, 64 rows padded to 68 floats:
// a thread's 4 x 4 (or 4 x 8) piece of a layer reads four rows of a feature
// with one 16-byte load, and the 16-byte loads of eight features at one row
// group (weight gradients) fall into distinct banks. Weight gradients are
// summed over the tile in registers and added to the global fp32 gradient
// with one atomic per tile and weight. (One thread per row with every
// activation in local memory and a warp reduction plus an atomic per weight,
// the form these kernels replace: 8.08 ms for 20,011 rows in fp32, 8.2 ms for
// 65,536 rows in BF16; bound by the shuffles and by local memory.)
#include <algorithm>

#include "mr_internal.h"
#include "mr_net_layout.cuh"
#include "mr_train.cuh"

namespace mr {

constexpr int kR = kTrainRows;  // rows of a tile
constexpr int kRS = kR + 4;     // padded feature stride (floats)

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float a, float b, float c, float d) {
  *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
}
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) { st4(p, v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
  acc = fmaf(a.x, b.x, acc);
  acc = fmaf(a.y, b.y, acc);
  acc = fmaf(a.z, b.z, acc);
  return fmaf(a.w, b.w, acc);
}
__device__ __forceinline__ void add_grad(float* g, float v) {
  if (v != 0.0f) atomicAdd(g, v);
}
// NC (1, 2 or 4) consecutive descriptor features. Descriptor rows are 2304
// bytes, so every piece is aligned to its size if the caller's table is to 16
// bytes (WIDE); any other table is read one feature at a time.
template <int NC, bool WIDE>
__device__ __forceinline__ void load_desc(const float* __restrict__ p, float (&v)[NC]) {
  if constexpr (NC == 4 && WIDE) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(p));
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else if constexpr (NC == 2 && WIDE) {
    const float2 q = __ldg(reinterpret_cast<const float2*>(p));
    v[0] = q.x; v[1] = q.y;
  } else {
#pragma unroll
    for (int i = 0; i < NC; ++i) v[i] = __ldg(p + i);
  }
}

// ---- statistics and gates ------------------------------------------------------
// Per-row layers of the gates, four rows (4 rg ..) per thread: a weight load
// serves four multiply-adds. (One row per thread: bound by those loads;
// 65,536 rows, k_train_stats 93 -> 67 us, k_train_gates 115 -> 91.)
__device__ __forceinline__ void fma4(float4& s, const float4 x, float w) {
  s.x = fmaf(x.x, w, s.x);
  s.y = fmaf(x.y, w, s.y);
  s.z = fmaf(x.z, w, s.z);
  s.w = fmaf(x.w, w, s.w);
}
__device__ __forceinline__ float4 relu4(const float4 s) { return make_float4(relu(s.x), relu(s.y), relu(s.z), relu(s.w)); }
__device__ __forceinline__ float4 sigmoid4(const float4 s) {
  return make_float4(sigmoid(s.x), sigmoid(s.y), sigmoid(s.z), sigmoid(s.w));
}
__device__ __forceinline__ void st4(float* p, const float4 v) { *reinterpret_cast<float4*>(p) = v; }

// Squeeze-excitation inputs of block b: means, maxima, g, gamma (P: 75 pooled features).
__device__ __forceinline__ void se_inputs(const float* P, int b, int rg, float4 (&t)[8]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    t[k] = ld4(P + (3 * b + k) * kRS + 4 * rg);
    t[3 + k] = ld4(P + (36 + 3 * b + k) * kRS + 4 * rg);
  }
  t[6] = ld4(P + 72 * kRS + 4 * rg);
  t[7] = ld4(P + 73 * kRS + 4 * rg);
}
// Hidden unit o, before its ReLU.
__device__ __forceinline__ float4 se_hidden(const float* __restrict__ W, const float4 (&t)[8], int o) {
  float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
  for (int j = 0; j < 8; ++j) fma4(s, t[j], __ldg(W + j + o * 8));
  return s;
}
// LSEFin1's 16 sums over the 75 features, after the ReLU, to SW: 256 threads,
// one output and four rows each.
__device__ __forceinline__ void fin1(const float* P, const float* __restrict__ W, float* SW) {
  const int rg = threadIdx.x & 15, o = threadIdx.x >> 4;
  float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 15
  for (int j = 0; j < 75; ++j) fma4(s, ld4(P + j * kRS + 4 * rg), __ldg(W + o * 75 + j));
  st4(SW + o * kRS + 4 * rg, relu4(s));
}

template <bool WIDE>
__global__ void __launch_bounds__(256) k_train_stats(TrainArgs a) {
  extern __shared__ __align__(16) float sm[];
  float* P = sm;             // 75 features: mean, max, g, gamma, srp
  float* SW = sm + 75 * kRS;  // 16
  const TrainTables& T = c_tt;
  const int r0 = blockIdx.x * kR;
  const float* __restrict__ W = a.w;
  // one (row, block, branch) segment of the descriptor at a time
  for (int i = threadIdx.x; i < kR * 36; i += 256) {
    const int row = i / 36, q = i - row * 36, b = q / 3, br = q - 3 * b, S = T.S[b];
    const float* d = a.desc + (size_t)min(r0 + row, a.n - 1) * 576 + br * 192 + T.from[b];
    float s = 0.0f, m = -10000.0f;
    for (int k = 0; k < S; k += 4) {
      float v[4];
      load_desc<4, WIDE>(d + k, v);
      s += v[0]; s += v[1]; s += v[2]; s += v[3];
      m = fmaxf(fmaxf(fmaxf(fmaxf(m, v[0]), v[1]), v[2]), v[3]);
    }
    P[q * kRS + row] = s / (float)S;
    P[(36 + q) * kRS + row] = m;
  }
  if (threadIdx.x < kR) {
    const float* x = a.aux + 5 * (size_t)min(r0 + (int)threadIdx.x, a.n - 1);
    for (int i = 0; i < 3; ++i) P[(72 + i) * kRS + threadIdx.x] = x[i];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 72 * kR; i += 256) {
    const int f = i / kR, row = i % kR;
    a.wk.pool[(size_t)f * a.wk.rows + r0 + row] = P[f * kRS + row];
  }
  if (threadIdx.x < 12 * 16) {
    const int b = threadIdx.x >> 4, rg = threadIdx.x & 15;
    float4 t[8], h[8];
    se_inputs(P, b, rg, t);
#pragma unroll
    for (int o = 0; o < 8; ++o) h[o] = relu4(se_hidden(W + T.se0[b], t, o));
#pragma unroll
    for (int o = 0; o < 3; ++o)
      st4(a.wk.gate + (size_t)(3 * b + o) * a.wk.rows + r0 + 4 * rg, sigmoid4(se_hidden(W + T.se1[b], h, o)));
  }
  fin1(P, W + T.f1, SW);
  __syncthreads();
  if (threadIdx.x < 6 * 16) {
    const int o = threadIdx.x >> 4, rg = threadIdx.x & 15;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < 16; ++j) fma4(s, ld4(SW + j * kRS + 4 * rg), __ldg(W + T.f2 + o * 16 + j));
    st4(a.wk.sp + (size_t)o * a.wk.rows + r0 + 4 * rg, sigmoid4(s));
  }
  for (int i = threadIdx.x; i < 8 * kR; i += 256) {
    const int row = i / 8, o = i % 8;
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < 3; ++j) s += P[(72 + j) * kRS + row] * __ldg(W + T.ggw + o * 3 + j);
    a.wk.h0[(size_t)(r0 + row) * 128 + 120 + o] = relu(s + __ldg(W + T.ggb + o));
  }
}

// ---- trunks --------------------------------------------------------------------
// Layers in order: blocks 0..7, L81, blocks 8..11, LD41. Shared memory holds
// each layer's weights, rows padded by 4 floats and stored in the order
// slot(o) = o / NC + 8 (o % NC) (NC = S / 8 columns per thread), which puts
// the rows that the four column groups of a warp read at once into distinct
// banks; and the input tiles of two layers in turn.
//
// The forward kernel writes every layer's input, the trunks' outputs and the
// signs of all outputs to memory (wk.xs, wk.mask); the backward kernel copies
// the inputs back one layer ahead. 65,536 rows: forward 226 -> 187 us and
// backward 502 -> 278 us against keeping a tile's 232 inputs in shared memory
// and running the forward again. A CTA has the weights once for two tiles,
// which go their own ways: 16 warps per SM for the backward where one tile per
// CTA allows 12 (20,011 rows: 110 us, with one tile 122). The forward gains
// nothing from more warps (three CTAs per SM: 192 us).
constexpr int kTrunkThreads = 128;
__host__ __device__ constexpr int layer_width(int l) {
  return l < 2 ? 8 : l < 5 ? 16 : l < 9 ? 32 : 8;
}
__host__ __device__ constexpr int layer_w(int l) {  // offset of layer l's weights
  int o = 0;
  for (int k = 0; k < l; ++k) o += layer_width(k) * (layer_width(k) + 4);
  return o;
}
__host__ __device__ constexpr int layer_x(int l) {  // first feature of layer l's input (and its biases)
  int o = 0;
  for (int k = 0; k < l; ++k) o += layer_width(k);
  return o;
}
constexpr int kLayers = 14, kTrunkW = layer_w(kLayers), kTrunkX = layer_x(kLayers);
static_assert(kTrunkX + 40 == kTrunkSaved && kLayers * kTrunkThreads * 2 == kTrunkMask, "the sizes in mr_train.cuh");
// forward: weights, biases, two input tiles of 32 features; backward: weights,
// two input tiles and two gradient buffers
constexpr int kTrunkTiles = 2;  // tiles of a CTA, 128 threads each
constexpr int kFwdSmem = (kTrunkW + kTrunkX + kTrunkTiles * 64 * kRS) * 4;
constexpr int kBwdSmem = (kTrunkW + kTrunkTiles * 128 * kRS) * 4;

// Blob offsets of layer l of branch br.
__device__ __forceinline__ int layer_wg(const TrainTables& T, int l, int br) {
  return l < 8 ? T.w[l][br] : l == 8 ? T.l81w[br] : l < 13 ? T.w[l - 1][br] : T.ld41w[br];
}
__device__ __forceinline__ int layer_bg(const TrainTables& T, int l, int br) {
  return l < 8 ? T.b[l][br] : l == 8 ? T.l81b[br] : l < 13 ? T.b[l - 1][br] : T.ld41b[br];
}

struct TrunkCtx {
  float *Ws, *Bs, *X, *D;  // weights, biases, input tiles, gradient buffers (two of 32 features each)
  float* xs;               // the tile's and branch's piece of wk.xs
  uint16_t* mask;          // and of wk.mask: [layer][thread], pre-activation > 0, bit 4 j + r
  const TrainArgs* a;
  int br, r0, rg, c, t, g;  // branch, first row, row and column group, thread of the tile, tile of the CTA
};

// Barrier of a tile's threads.
__device__ __forceinline__ void tile_sync(const TrunkCtx& k) {
  if (k.g == 0)
    asm volatile("bar.sync 1, %0;" ::"n"(kTrunkThreads) : "memory");
  else
    asm volatile("bar.sync 2, %0;" ::"n"(kTrunkThreads) : "memory");
}

__device__ __forceinline__ void trunk_ctx(TrunkCtx& k, const TrainArgs& a) {
  k.a = &a;
  k.br = blockIdx.x % 3;
  k.t = threadIdx.x % kTrunkThreads;
  k.g = threadIdx.x / kTrunkThreads;
  const int warp = k.t >> 5, lane = k.t & 31;
  k.rg = (lane & 7) + 8 * (warp & 1);
  k.c = (lane >> 3) + 4 * (warp >> 1);
}
__device__ __forceinline__ void trunk_tile(TrunkCtx& k, int tile) {
  k.r0 = tile * kR;
  const size_t q = (size_t)tile * 3 + k.br;
  k.xs = k.a->wk.xs + q * (kTrunkSaved * kR);
  k.mask = k.a->wk.mask + q * (kTrunkMask / 2);
}
__device__ __forceinline__ void trunk_weights(const TrunkCtx& k, bool biases) {
#pragma unroll 1
  for (int l = 0; l < kLayers; ++l) {
    const int S = layer_width(l), nc = S / 8, wg = layer_wg(c_tt, l, k.br), bg = layer_bg(c_tt, l, k.br);
    for (int i = threadIdx.x; i < S * S; i += blockDim.x) {
      const int o = i / S, c = i - o * S;
      k.Ws[layer_w(l) + (o / nc + 8 * (o % nc)) * (S + 4) + c] = __ldg(k.a->w + wg + i);
    }
    if (biases && threadIdx.x < S) k.Bs[layer_x(l) + threadIdx.x] = __ldg(k.a->w + bg + threadIdx.x);
  }
}

// The descriptor features of layer l (a block's) at the caller's rows and
// columns: s[r][j].
template <int NC, bool WIDE>
__device__ __forceinline__ void load_features(const TrunkCtx& k, int block, float (&s)[4][NC]) {
  const int f = k.br * 192 + c_tt.from[block] + k.c * NC;
#pragma unroll
  for (int r = 0; r < 4; ++r)
    load_desc<NC, WIDE>(k.a->desc + (size_t)min(k.r0 + 4 * k.rg + r, k.a->n - 1) * 576 + f, s[r]);
}

// Rows 4 rg .. 4 rg + 3, outputs c NC .. c NC + NC - 1 of layer l from the
// input tile x: bias after the sum over ascending inputs.
template <int NC>
__device__ __forceinline__ void tile_fwd(const TrunkCtx& k, int l, const float* x, float (&y)[NC][4]) {
  constexpr int S = 8 * NC;
  x += 4 * k.rg;
  const float* w = k.Ws + layer_w(l) + k.c * (S + 4);
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) y[j][r] = 0.0f;
#pragma unroll 2
  for (int q = 0; q < S / 4; ++q) {
    float4 wv[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) wv[j] = ld4(w + j * 8 * (S + 4) + 4 * q);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 v = ld4(x + (4 * q + u) * kRS);
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const float wj = (&wv[j].x)[u];
        y[j][0] = fmaf(v.x, wj, y[j][0]);
        y[j][1] = fmaf(v.y, wj, y[j][1]);
        y[j][2] = fmaf(v.z, wj, y[j][2]);
        y[j][3] = fmaf(v.w, wj, y[j][3]);
      }
    }
  }
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const float b = k.Bs[layer_x(l) + k.c * NC + j];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float v = y[j][r] + b;
      m |= (v > 0.0f ? 1u : 0u) << (4 * j + r);
      y[j][r] = relu(v);
    }
  }
  k.mask[l * kTrunkThreads + k.t] = (uint16_t)m;
}

// A layer's input, the caller's piece, to its tile and to memory.
template <int NC>
__device__ __forceinline__ void put_input(const TrunkCtx& k, int l, float* x, int j, float a, float b, float c, float d) {
  st4(x + (k.c * NC + j) * kRS + 4 * k.rg, a, b, c, d);
  st4(k.xs + (layer_x(l) + k.c * NC + j) * kR + 4 * k.rg, a, b, c, d);
}

// Blocks l .. l + count - 1 of one width (l counts layers; the block is
// l - shift). y: the running output, in and out; with `rep` the last block
// doubles the width (REP3) and leaves its output in the next input tile for
// take_wide. buf: the input tile to use, alternating (one barrier a layer).
template <int NC, bool WIDE>
__device__ __forceinline__ void blocks_fwd(const TrunkCtx& k, int l, int count, int shift, bool rep, int& buf,
                                           float (&y)[NC][4]) {
  constexpr int S = 8 * NC;
  auto gate = [&](int l) {
    return ld4(k.a->wk.gate + (size_t)(3 * (l - shift) + k.br) * k.a->wk.rows + k.r0 + 4 * k.rg);
  };
  float s[4][NC];
  load_features<NC, WIDE>(k, l - shift, s);
  float4 g = gate(l);
#pragma unroll 1
  for (int n = 0; n < count; ++n, ++l) {
    float* x = k.X + buf * 32 * kRS;
    buf ^= 1;
#pragma unroll
    for (int j = 0; j < NC; ++j)
      put_input<NC>(k, l, x, j, fmaf(s[0][j], g.x, y[j][0]), fmaf(s[1][j], g.y, y[j][1]), fmaf(s[2][j], g.z, y[j][2]),
                    fmaf(s[3][j], g.w, y[j][3]));
    tile_sync(k);
    float sn[4][NC];
    if (n + 1 < count) {  // lands during the products
      load_features<NC, WIDE>(k, l + 1 - shift, sn);
      g = gate(l + 1);
    }
    tile_fwd<NC>(k, l, x, y);
    if (rep && n == count - 1) {
      float* o = k.X + buf * 32 * kRS;
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        st4(o + (k.c * NC + j) * kRS + 4 * k.rg, y[j]);
        st4(o + (S + k.c * NC + j) * kRS + 4 * k.rg, s[0][j], s[1][j], s[2][j], s[3][j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < NC; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) y[j][r] += s[r][j];
    }
    if (n + 1 < count)
#pragma unroll
      for (int j = 0; j < NC; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r][j] = sn[r][j];
  }
}
// The wide output in the wider column split. The tile it sits in is the next
// layer's: every thread overwrites the piece it read.
template <int NC>
__device__ __forceinline__ void take_wide(const TrunkCtx& k, int buf, float (&y)[NC][4]) {
  tile_sync(k);
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const float4 v = ld4(k.X + buf * 32 * kRS + (k.c * NC + j) * kRS + 4 * k.rg);
    y[j][0] = v.x; y[j][1] = v.y; y[j][2] = v.z; y[j][3] = v.w;
  }
}
// L81 and LD41: y is the layer's input.
template <int NC>
__device__ __forceinline__ void last_fwd(const TrunkCtx& k, int l, int& buf, float (&y)[NC][4]) {
  float* x = k.X + buf * 32 * kRS;
  buf ^= 1;
#pragma unroll
  for (int j = 0; j < NC; ++j) put_input<NC>(k, l, x, j, y[j][0], y[j][1], y[j][2], y[j][3]);
  tile_sync(k);
  tile_fwd<NC>(k, l, x, y);
}

// Head-input columns of a trunk: y = relu(L81 or LD41) times its output gate.
// y itself is kept as feature kTrunkX + at + column, for the gate's gradient.
template <int NC>
__device__ __forceinline__ void put_h0(const TrunkCtx& k, int col, int at, const float4 sp, const float (&y)[NC][4]) {
#pragma unroll
  for (int j = 0; j < NC; ++j) st4(k.xs + (kTrunkX + at + k.c * NC + j) * kR + 4 * k.rg, y[j]);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    float* p = k.a->wk.h0 + (size_t)(k.r0 + 4 * k.rg + r) * 128 + col + k.c * NC;
    const float g = (&sp.x)[r];
    if constexpr (NC == 4)
      st4(p, y[0][r] * g, y[1][r] * g, y[2][r] * g, y[3][r] * g);
    else
      p[0] = y[0][r] * g;
  }
}

// CTA b: branch b % 3; its tiles g = 0 .. G - 1 at a time: b / 3 G + g, then
// gridDim / 3 G further on.
template <bool WIDE>
__global__ void __launch_bounds__(kTrunkTiles * kTrunkThreads, 2) k_train_trunk_fwd(const __grid_constant__ TrainArgs a) {
  extern __shared__ __align__(16) float sm[];
  TrunkCtx k;
  trunk_ctx(k, a);
  k.Ws = sm;
  k.Bs = k.Ws + kTrunkW;
  k.X = k.Bs + kTrunkX + k.g * 64 * kRS;
  trunk_weights(k, true);
  __syncthreads();
  const int tiles = (a.n + kR - 1) / kR;
  const size_t N = a.wk.rows;
  int buf = 0;
  for (int tile = blockIdx.x / 3 * kTrunkTiles + k.g; tile < tiles; tile += gridDim.x / 3 * kTrunkTiles) {
    trunk_tile(k, tile);
    {
      float y1[1][4] = {}, y2[2][4], y4[4][4];
      blocks_fwd<1, WIDE>(k, 0, 2, 0, true, buf, y1);
      take_wide<2>(k, buf, y2);
      blocks_fwd<2, WIDE>(k, 2, 3, 0, true, buf, y2);
      take_wide<4>(k, buf, y4);
      blocks_fwd<4, WIDE>(k, 5, 3, 0, false, buf, y4);
      last_fwd<4>(k, 8, buf, y4);
      put_h0<4>(k, 32 * k.br, 0, ld4(a.wk.sp + (size_t)k.br * N + k.r0 + 4 * k.rg), y4);
    }
    float yl[1][4] = {};
    blocks_fwd<1, WIDE>(k, 9, 4, 1, false, buf, yl);
    last_fwd<1>(k, 13, buf, yl);
    put_h0<1>(k, 96 + 8 * k.br, 32, ld4(a.wk.sp + (size_t)(3 + k.br) * N + k.r0 + 4 * k.rg), yl);
  }
}

// Weight gradient of layer l, dW[o][i] += sum over rows of D[o] x[i], and the
// bias gradient from the caller's own rows of D.
template <int NC>
__device__ __forceinline__ void tile_dw(const TrunkCtx& k, int l, const float* x, const float* D,
                                        const float (&dp)[NC][4]) {
  constexpr int S = 8 * NC;
  float* G = k.a->grad;
  const int wg = layer_wg(c_tt, l, k.br), bg = layer_bg(c_tt, l, k.br);
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    float s = (dp[j][0] + dp[j][1]) + (dp[j][2] + dp[j][3]);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((k.t & 7) == 0) add_grad(G + bg + k.c * NC + j, s);
  }
  const int ig = k.t & 7, og = k.t >> 3;
  x += ig * kRS;
  if constexpr (NC == 1) {  // 64 weights: each half of the threads sums half the rows
    const float* d = D + (og & 7) * kRS;
    const int k0 = (k.t >> 6) * (kR / 2);
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < kR / 2; q += 4) s = dot4(ld4(d + k0 + q), ld4(x + k0 + q), s);
    add_grad(G + wg + (og & 7) * S + ig, s);
  } else {
    constexpr int NO = NC / 2;
    float s[NO][NC];
#pragma unroll
    for (int u = 0; u < NO; ++u)
#pragma unroll
      for (int j = 0; j < NC; ++j) s[u][j] = 0.0f;
#pragma unroll 2
    for (int q = 0; q < kR; q += 4) {
      float4 dv[NO], xv[NC];
#pragma unroll
      for (int u = 0; u < NO; ++u) dv[u] = ld4(D + (og + 16 * u) * kRS + q);
#pragma unroll
      for (int j = 0; j < NC; ++j) xv[j] = ld4(x + 8 * j * kRS + q);
#pragma unroll
      for (int u = 0; u < NO; ++u)
#pragma unroll
        for (int j = 0; j < NC; ++j) s[u][j] = dot4(dv[u], xv[j], s[u][j]);
    }
#pragma unroll
    for (int u = 0; u < NO; ++u)
#pragma unroll
      for (int j = 0; j < NC; ++j) add_grad(G + wg + (og + 16 * u) * S + ig + 8 * j, s[u][j]);
  }
}

// The backward pass takes the layers in the order 8 (L81), 7 .. 0, 13 (LD41),
// 12 .. 9: step i is layer bwd_layer(i).
__device__ __forceinline__ int bwd_layer(int i) { return i < 9 ? 8 - i : 22 - i; }

struct BwdState {
  int step;       // layers of the tile done
  int buf;        // gradient buffer to use next
  int next;       // the CTA's next tile, or -1
  uint32_t mask;  // the next layer's signs
};

// Starts the copy of a step's layer inputs into input tile step & 1 and loads
// its signs; step kLayers is the next tile's first.
__device__ __forceinline__ void fetch_step(const TrunkCtx& k, BwdState& b, int step) {
  const float* xs = k.xs;
  const uint16_t* mask = k.mask;
  if (step == kLayers) {
    if (b.next < 0) return;
    const size_t q = (size_t)b.next * 3 + k.br;
    xs = k.a->wk.xs + q * (kTrunkSaved * kR);
    mask = k.a->wk.mask + q * (kTrunkMask / 2);
    step = 0;
  }
  const int l = bwd_layer(step), at = layer_x(l);
  const uint32_t dst = (uint32_t)__cvta_generic_to_shared(k.X + (step & 1) * 32 * kRS);
  for (int i = k.t; i < layer_width(l) * (kR / 4); i += kTrunkThreads) {
    const int f = i / (kR / 4), q = i % (kR / 4);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (f * kRS + 4 * q) * 4),
                 "l"(xs + (at + f) * kR + 4 * q)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  b.mask = mask[l * kTrunkThreads + k.t];
}

// Backward of the next layer in order (l): d = gradient of its ReLU output in,
// of its input out. One barrier: the gradient buffers and the input tiles
// alternate, and a tile is refilled only after the barrier behind its last
// reads.
template <int NC>
__device__ __forceinline__ void tile_bwd(const TrunkCtx& k, BwdState& b, int l, float (&d)[NC][4]) {
  constexpr int S = 8 * NC;
  const uint32_t m = b.mask;
  const int i = b.step++;
  float* D = k.D + b.buf * 32 * kRS;
  b.buf ^= 1;
#pragma unroll
  for (int j = 0; j < NC; ++j) {
#pragma unroll
    for (int r = 0; r < 4; ++r) d[j][r] = (m >> (4 * j + r)) & 1u ? d[j][r] : 0.0f;
    st4(D + (k.c * NC + j) * kRS + 4 * k.rg, d[j]);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  tile_sync(k);
  fetch_step(k, b, i + 1);
  tile_dw<NC>(k, l, k.X + (i & 1) * 32 * kRS, D, d);
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) d[j][r] = 0.0f;
  const float* w = k.Ws + layer_w(l) + k.c * NC;
#pragma unroll 2
  for (int q = 0; q < 8; ++q) {
#pragma unroll
    for (int u = 0; u < NC; ++u) {  // output q NC + u, stored at row q + 8 u
      const float4 v = ld4(D + (q * NC + u) * kRS + 4 * k.rg);
      float wv[NC];
      const float* wr = w + (q + 8 * u) * (S + 4);
      if constexpr (NC == 4) {
        const float4 f = ld4(wr);
        wv[0] = f.x; wv[1] = f.y; wv[2] = f.z; wv[3] = f.w;
      } else if constexpr (NC == 2) {
        const float2 f = *reinterpret_cast<const float2*>(wr);
        wv[0] = f.x; wv[1] = f.y;
      } else {
        wv[0] = wr[0];
      }
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        d[j][0] = fmaf(v.x, wv[j], d[j][0]);
        d[j][1] = fmaf(v.y, wv[j], d[j][1]);
        d[j][2] = fmaf(v.z, wv[j], d[j][2]);
        d[j][3] = fmaf(v.w, wv[j], d[j][3]);
      }
    }
  }
}

// Sum over the tile's columns (the four column groups of the warp; the two
// warps that share the rows write a half each).
__device__ __forceinline__ void row_sums(const TrunkCtx& k, float* half0, size_t half_stride, float (&s)[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 8);
    s[r] += __shfl_xor_sync(0xffffffffu, s[r], 16);
  }
  if ((k.t & 31) < 8) st4(half0 + (k.t >> 6) * half_stride + k.r0 + 4 * k.rg, s);
}

// Blocks l, l - 1, ..., l - count + 1 backward; d as in tile_bwd.
template <int NC, bool WIDE>
__device__ __forceinline__ void blocks_bwd(const TrunkCtx& k, BwdState& b, int l, int count, int shift, float (&d)[NC][4]) {
#pragma unroll 1
  for (int n = 0; n < count; ++n, --l) {
    float s[4][NC];
    load_features<NC, WIDE>(k, l - shift, s);  // for the gate's gradient; lands during the products
    tile_bwd<NC>(k, b, l, d);
    float dg[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < NC; ++j) dg[r] = fmaf(d[j][r], s[r][j], dg[r]);
    row_sums(k, k.a->wk.dgate + (size_t)(3 * (l - shift) + k.br) * k.a->wk.rows, (size_t)36 * k.a->wk.rows, dg);
  }
}

// The first half of a wide gradient (the ReLU part of REP3's output) in the
// narrower column split.
template <int NC>
__device__ __forceinline__ void narrow(const TrunkCtx& k, BwdState& b, const float (&w)[2 * NC][4], float (&d)[NC][4]) {
  float* D = k.D + b.buf * 32 * kRS;
  b.buf ^= 1;
#pragma unroll
  for (int j = 0; j < 2 * NC; ++j) st4(D + (k.c * 2 * NC + j) * kRS + 4 * k.rg, w[j]);
  tile_sync(k);
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const float4 v = ld4(D + (k.c * NC + j) * kRS + 4 * k.rg);
    d[j][0] = v.x; d[j][1] = v.y; d[j][2] = v.z; d[j][3] = v.w;
  }
}

// The head input's gradient at a trunk's columns: d = dh0 * gate, and the
// gate's own gradient sum(dh0 * y).
template <int NC>
__device__ __forceinline__ void take_dh0(const TrunkCtx& k, int col, int at, const float4 sp, float* dsp, float (&d)[NC][4]) {
  float y[NC][4];
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const float4 v = ld4(k.xs + (kTrunkX + at + k.c * NC + j) * kR + 4 * k.rg);
    y[j][0] = v.x; y[j][1] = v.y; y[j][2] = v.z; y[j][3] = v.w;
  }
  float s[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int row = k.r0 + 4 * k.rg + r;
    const float* p = k.a->wk.dh0 + (size_t)row * 128 + col + k.c * NC;
    float v[NC];
    if constexpr (NC == 4) {
      const float4 q = row < k.a->n ? ld4(p) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
      v[0] = row < k.a->n ? p[0] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      s[r] = fmaf(v[j], y[j][r], s[r]);
      d[j][r] = v[j] * (&sp.x)[r];
    }
  }
  row_sums(k, dsp, (size_t)6 * k.a->wk.rows, s);
}

template <bool WIDE>
__global__ void __launch_bounds__(kTrunkTiles * kTrunkThreads, 2) k_train_trunk_bwd(const __grid_constant__ TrainArgs a) {
  extern __shared__ __align__(16) float sm[];
  TrunkCtx k;
  trunk_ctx(k, a);
  k.Ws = sm;
  k.Bs = nullptr;
  k.X = k.Ws + kTrunkW + k.g * 128 * kRS;
  k.D = k.X + 64 * kRS;
  const int tiles = (a.n + kR - 1) / kR, stride = gridDim.x / 3 * kTrunkTiles;
  const int first = blockIdx.x / 3 * kTrunkTiles + k.g;
  const size_t N = a.wk.rows;
  BwdState b{0, 0, first, 0};
  if (b.next < tiles) fetch_step(k, b, kLayers);
  trunk_weights(k, false);
  __syncthreads();
  for (int tile = first; tile < tiles; tile += stride) {
    trunk_tile(k, tile);
    b.step = 0;
    b.next = tile + stride < tiles ? tile + stride : -1;
    {
      float d4[4][4], d2[2][4], d1[1][4];
      take_dh0<4>(k, 32 * k.br, 0, ld4(a.wk.sp + (size_t)k.br * N + k.r0 + 4 * k.rg), a.wk.dsp + (size_t)k.br * N, d4);
      tile_bwd<4>(k, b, 8, d4);
      blocks_bwd<4, WIDE>(k, b, 7, 3, 0, d4);
      narrow<2>(k, b, d4, d2);
      blocks_bwd<2, WIDE>(k, b, 4, 3, 0, d2);
      narrow<1>(k, b, d2, d1);
      blocks_bwd<1, WIDE>(k, b, 1, 2, 0, d1);
    }
    float dl[1][4];
    take_dh0<1>(k, 96 + 8 * k.br, 32, ld4(a.wk.sp + (size_t)(3 + k.br) * N + k.r0 + 4 * k.rg),
                a.wk.dsp + (size_t)(3 + k.br) * N, dl);
    tile_bwd<1>(k, b, 13, dl);
    blocks_bwd<1, WIDE>(k, b, 12, 4, 1, dl);
  }
}

// ---- head and tail ---------------------------------------------------------------
// 256 threads: thread (rg, c) owns rows 4 rg .. 4 rg + 3 and N / 16 columns of
// a layer of N outputs.
constexpr int kHeadThreads2 = 256;
// Tail weights in shared memory: LX (16 rows of 36), the 12 residual layers
// (16 rows of 20), LX12 (16), then the biases LXB, LX0B .. LX11B, LX12B.
constexpr int kTailR = 16 * 36, kTail12 = kTailR + 12 * 320, kTailB = kTail12 + 16, kTailW = kTailB + 13 * 16 + 4;
// Features of the tail's storage: AR[0..6], TT[0..5] (16 each), and its two
// gradient buffers.
constexpr int kTailTT = 7 * 16, kTailD = kTailTT + 6 * 16, kTailX = kTailD + 32;

struct HeadCtx {
  float* tw;  // tail weights
  float* T;   // tail storage, kTailX features
  const TrainArgs* a;
  int r0, rg, c, t;
};

__device__ __forceinline__ void load_tail_weights(const TrainArgs& a, float* tw) {
  const TrainTables& T = c_tt;
  for (int i = threadIdx.x; i < 512; i += kHeadThreads2) tw[(i / 32) * 36 + i % 32] = __ldg(a.w + T.lxw + i);
  for (int i = threadIdx.x; i < 12 * 256; i += kHeadThreads2) {
    const int l = i >> 8, e = i & 255;
    tw[kTailR + l * 320 + (e >> 4) * 20 + (e & 15)] = __ldg(a.w + T.lxrw[l] + e);
  }
  if (threadIdx.x < 16) {
    tw[kTail12 + threadIdx.x] = __ldg(a.w + T.lx12w + threadIdx.x);
    tw[kTailB + threadIdx.x] = __ldg(a.w + T.lxb + threadIdx.x);
  }
  for (int i = threadIdx.x; i < 12 * 16; i += kHeadThreads2) tw[kTailB + 16 + i] = __ldg(a.w + T.lxrb[i >> 4] + (i & 15));
  if (threadIdx.x == 0) tw[kTailB + 13 * 16] = __ldg(a.w + T.lx12b);
}

// Column c of a layer with 16 outputs and K inputs (rows of W padded to RW).
template <int K, int RW>
__device__ __forceinline__ void row16(const HeadCtx& k, const float* X, const float* W, float bias, float (&y)[4]) {
  y[0] = y[1] = y[2] = y[3] = 0.0f;
#pragma unroll
  for (int q = 0; q < K / 4; ++q) {
    const float4 w = ld4(W + k.c * RW + 4 * q);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 v = ld4(X + (4 * q + u) * kRS + 4 * k.rg);
      const float wu = (&w.x)[u];
      y[0] = fmaf(v.x, wu, y[0]);
      y[1] = fmaf(v.y, wu, y[1]);
      y[2] = fmaf(v.z, wu, y[2]);
      y[3] = fmaf(v.w, wu, y[3]);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) y[r] += bias;
}
// Input column i of the same layer's input gradient: sum over its 16 outputs.
template <int RW>
__device__ __forceinline__ void col16(const HeadCtx& k, const float* D, const float* W, int i, float (&y)[4]) {
  y[0] = y[1] = y[2] = y[3] = 0.0f;
#pragma unroll
  for (int o = 0; o < 16; ++o) {
    const float w = W[o * RW + i];
    const float4 v = ld4(D + o * kRS + 4 * k.rg);
    y[0] = fmaf(v.x, w, y[0]);
    y[1] = fmaf(v.y, w, y[1]);
    y[2] = fmaf(v.z, w, y[2]);
    y[3] = fmaf(v.w, w, y[3]);
  }
}
// dW[o][i] of NO x NI weights per thread: o = tid / 16 + 16 u, i = tid % 16 + 16 j.
template <int NO, int NI>
__device__ __forceinline__ void head_dw(const HeadCtx& k, const float* D, const float* X, float* G) {
  const int og = k.t >> 4, ig = k.t & 15;
  float s[NO][NI];
#pragma unroll
  for (int u = 0; u < NO; ++u)
#pragma unroll
    for (int j = 0; j < NI; ++j) s[u][j] = 0.0f;
#pragma unroll 1
  for (int q = 0; q < kR; q += 4) {
    float4 dv[NO];
#pragma unroll
    for (int u = 0; u < NO; ++u) dv[u] = ld4(D + (og + 16 * u) * kRS + q);
#pragma unroll
    for (int j = 0; j < NI; ++j) {
      const float4 x = ld4(X + (ig + 16 * j) * kRS + q);
#pragma unroll
      for (int u = 0; u < NO; ++u) s[u][j] = dot4(dv[u], x, s[u][j]);
    }
  }
#pragma unroll
  for (int u = 0; u < NO; ++u)
#pragma unroll
    for (int j = 0; j < NI; ++j) add_grad(G + (og + 16 * u) * (16 * NI) + ig + 16 * j, s[u][j]);
}
// dW[o][i] of a 16 x 16 NI layer: two outputs and 2 NI inputs per thread over a
// quarter of the rows (row quads k, k + 4, ... of lane k % 4), summed over the
// four lanes. A warp's lanes hold the inputs in an order that spreads the
// eight loads of a phase over all banks. (One weight per thread over all rows
// takes twice the shared-memory loads: k_train_tail, 65,536 rows, 143 -> 130
// us.)
template <int NI>
__device__ __forceinline__ void tail_dw(const HeadCtx& k, const float* D, const float* X, float* G) {
  const int warp = k.t >> 5, q0 = k.t & 3, m = (k.t & 31) >> 2, ig = (m & 1) * 4 + (m >> 1);
  float s[2][2 * NI];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int j = 0; j < 2 * NI; ++j) s[u][j] = 0.0f;
#pragma unroll
  for (int q = 4 * q0; q < kR; q += 16) {
    const float4 d0 = ld4(D + warp * kRS + q), d1 = ld4(D + (warp + 8) * kRS + q);
#pragma unroll
    for (int j = 0; j < 2 * NI; ++j) {
      const float4 x = ld4(X + (ig + 8 * j) * kRS + q);
      s[0][j] = dot4(d0, x, s[0][j]);
      s[1][j] = dot4(d1, x, s[1][j]);
    }
  }
  // lane bit 0 keeps one output, bit 1 one half of the inputs
  float h[2 * NI];
#pragma unroll
  for (int j = 0; j < 2 * NI; ++j) {
    const float mine = q0 & 1 ? s[1][j] : s[0][j], other = q0 & 1 ? s[0][j] : s[1][j];
    h[j] = mine + __shfl_xor_sync(0xffffffffu, other, 1);
  }
#pragma unroll
  for (int j = 0; j < NI; ++j) {
    const float mine = q0 & 2 ? h[NI + j] : h[j], other = q0 & 2 ? h[j] : h[NI + j];
    add_grad(G + (warp + 8 * (q0 & 1)) * (16 * NI) + ig + 8 * ((q0 & 2 ? NI : 0) + j),
             mine + __shfl_xor_sync(0xffffffffu, other, 2));
  }
}
// Bias gradient of column o from the caller's rows of it.
__device__ __forceinline__ void head_db(const HeadCtx& k, float* g, const float (&d)[4]) {
  float s = (d[0] + d[1]) + (d[2] + d[3]);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((k.t & 7) == 0) add_grad(g, s);
}

// The tail (LX, six residual pairs, LX12; radiancePredict.cu:454-473) from A3
// (32 features), the loss (X - log(1 + label / srp))^2 / batch added to
// *a.loss, and the backward pass: d[j] = dL/dA3 of columns 2 c + j.
__device__ __forceinline__ void tail_tile(const HeadCtx& k, const float* A3, float (&d)[2][4]) {
  const TrainArgs& a = *k.a;
  const TrainTables& T = c_tt;
  float *AR = k.T, *TT = k.T + kTailTT * kRS, *D1 = k.T + kTailD * kRS, *D2 = D1 + 16 * kRS;
  const float* tb = k.tw + kTailB;
  const int own = k.c * kRS + 4 * k.rg;
  float v[4], ar[4];
  uint32_t mu = 0;
  row16<32, 36>(k, A3, k.tw, tb[k.c], ar);
#pragma unroll
  for (int r = 0; r < 4; ++r) ar[r] = relu(ar[r]);
  st4(AR + own, ar);
  __syncthreads();
#pragma unroll 1
  for (int l = 0; l < 6; ++l) {
    const float* w = k.tw + kTailR + 640 * l;
    row16<16, 20>(k, AR + 16 * l * kRS, w, tb[16 + 32 * l + k.c], v);
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] = relu(v[r]);
    st4(TT + 16 * l * kRS + own, v);
    __syncthreads();
    row16<16, 20>(k, TT + 16 * l * kRS, w + 320, tb[32 + 32 * l + k.c], v);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      mu |= (v[r] > 0.0f ? 1u : 0u) << (4 * l + r);
      ar[r] += relu(v[r]);
    }
    st4(AR + 16 * (l + 1) * kRS + own, ar);
    __syncthreads();
  }
  // LX12, the loss and its gradient: one thread per row; dOP into D1's first feature
  const float* A6 = AR + 96 * kRS;
  if (k.t < kR) {
    float o = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) o = fmaf(A6[i * kRS + k.t], k.tw[kTail12 + i], o);
    o += tb[13 * 16];
    const int row = k.r0 + k.t;
    float err = 0.0f;
    if (row < a.n) {
      const float srp = a.aux[5 * (size_t)row + 2];
      err = relu(o) - log1pf(fmaxf(a.label[row], 0.0f) / srp);
    }
    float l = err * err * a.inv_batch;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) l += __shfl_xor_sync(0xffffffffu, l, s);
    if ((k.t & 31) == 0) atomicAdd(a.loss, l);
    D1[k.t] = 2.0f * err * a.inv_batch * (o > 0.0f ? 1.0f : 0.0f);
  }
  __syncthreads();
  {
    const float4 g = ld4(D1 + 4 * k.rg);
    const float w = k.tw[kTail12 + k.c];
    v[0] = g.x * w; v[1] = g.y * w; v[2] = g.z * w; v[3] = g.w * w;
    if (k.t < 17) {  // gradients of LX12: 16 weights and the bias
      float s = 0.0f;
      for (int q = 0; q < kR; q += 4) {
        const float4 e = ld4(D1 + q);
        s = k.t < 16 ? dot4(e, ld4(A6 + k.t * kRS + q), s) : s + ((e.x + e.y) + (e.z + e.w));
      }
      add_grad(a.grad + (k.t < 16 ? T.lx12w + k.t : T.lx12b), s);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int l = 5; l >= 0; --l) {  // v = dL/dAR[l + 1]
    const float* w = k.tw + kTailR + 640 * l;
    float e[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) e[r] = (mu >> (4 * l + r)) & 1u ? v[r] : 0.0f;
    st4(D1 + own, e);
    head_db(k, a.grad + T.lxrb[2 * l + 1] + k.c, e);
    __syncthreads();
    tail_dw<1>(k, D1, TT + 16 * l * kRS, a.grad + T.lxrw[2 * l + 1]);
    col16<20>(k, D1, w + 320, k.c, e);
    const float4 tt = ld4(TT + 16 * l * kRS + own);
    e[0] = tt.x > 0.0f ? e[0] : 0.0f;
    e[1] = tt.y > 0.0f ? e[1] : 0.0f;
    e[2] = tt.z > 0.0f ? e[2] : 0.0f;
    e[3] = tt.w > 0.0f ? e[3] : 0.0f;
    st4(D2 + own, e);
    head_db(k, a.grad + T.lxrb[2 * l] + k.c, e);
    __syncthreads();
    tail_dw<1>(k, D2, AR + 16 * l * kRS, a.grad + T.lxrw[2 * l]);
    col16<20>(k, D2, w, k.c, e);
#pragma unroll
    for (int r = 0; r < 4; ++r) v[r] += e[r];
  }
  {
    const float4 x = ld4(AR + own);
    v[0] = x.x > 0.0f ? v[0] : 0.0f;
    v[1] = x.y > 0.0f ? v[1] : 0.0f;
    v[2] = x.z > 0.0f ? v[2] : 0.0f;
    v[3] = x.w > 0.0f ? v[3] : 0.0f;
    st4(D1 + own, v);
    head_db(k, a.grad + T.lxb + k.c, v);
  }
  __syncthreads();
  tail_dw<2>(k, D1, A3, a.grad + T.lxw);
  col16<36>(k, D1, k.tw, 2 * k.c, d[0]);
  col16<36>(k, D1, k.tw, 2 * k.c + 1, d[1]);
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const float4 x = ld4(A3 + (2 * k.c + j) * kRS + 4 * k.rg);
    d[j][0] = x.x > 0.0f ? d[j][0] : 0.0f;
    d[j][1] = x.y > 0.0f ? d[j][1] : 0.0f;
    d[j][2] = x.z > 0.0f ? d[j][2] : 0.0f;
    d[j][3] = x.w > 0.0f ? d[j][3] : 0.0f;
  }
}

__device__ __forceinline__ void head_coords(HeadCtx& k) {
  k.t = threadIdx.x;
  const int warp = k.t >> 5, lane = k.t & 31;
  k.rg = (lane & 7) + 8 * (warp & 1);
  k.c = (lane >> 3) + 4 * (warp >> 1);
}

// The tail for the BF16 step: a3 (rows x 32) in, its gradient (masked by
// A3 > 0) out to da3.
constexpr int kTailSmem = (kTailW + (32 + kTailX) * kRS) * 4;
__global__ void __launch_bounds__(kHeadThreads2, 2) k_train_tail(const __grid_constant__ TrainArgs a) {
  extern __shared__ __align__(16) float sm[];
  HeadCtx k;
  head_coords(k);
  k.a = &a;
  k.tw = sm;
  float* A3 = sm + kTailW;
  k.T = A3 + 32 * kRS;
  load_tail_weights(a, k.tw);
  const int tiles = (a.n + kR - 1) / kR;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    k.r0 = tile * kR;
    __syncthreads();
    for (int i = k.t; i < 8 * 16; i += kHeadThreads2) {  // 4 x 4 pieces, transposed
      const int rg = i & 15, cg = i >> 4;
      float4 v[4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
        v[r] = reinterpret_cast<const float4*>(a.wk.a3 + (size_t)min(k.r0 + 4 * rg + r, a.n - 1) * 32)[cg];
      float* x = A3 + 4 * cg * kRS + 4 * rg;
      st4(x, v[0].x, v[1].x, v[2].x, v[3].x);
      st4(x + kRS, v[0].y, v[1].y, v[2].y, v[3].y);
      st4(x + 2 * kRS, v[0].z, v[1].z, v[2].z, v[3].z);
      st4(x + 3 * kRS, v[0].w, v[1].w, v[2].w, v[3].w);
    }
    __syncthreads();
    float d[2][4];
    tail_tile(k, A3, d);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int row = k.r0 + 4 * k.rg + r;
      if (row < a.n) *reinterpret_cast<float2*>(a.wk.da3 + (size_t)row * 32 + 2 * k.c) = make_float2(d[0][r], d[1][r]);
    }
  }
}

// The fp32 head. Layer weights stream through a two-slot ring of 16-wide
// pieces (cp.async): 16 inputs of every output row forward, 16 output rows
// backward.
constexpr int kPiece = 16 * 16 * 10;  // floats of a slot: 128 rows of 20, or 16 rows of 132
constexpr int kHeadX = 128 + 128 + 64 + 32 + 32 + kTailX;
constexpr int kHeadSmem2 = (kTailW + 2 * kPiece + kHeadX * kRS) * 4;
static_assert(kHeadSmem2 <= 232448, "shared memory budget");
static_assert(192 <= kTailD, "the LC gradients reuse the tail's storage");

__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Y = relu(W X + b): NC columns per thread, N = 16 NC outputs, K inputs.
template <int NC, int K>
__device__ __forceinline__ void head_fwd(const HeadCtx& k, float* ring, const float* X, const float* __restrict__ W,
                                         const float* __restrict__ B, float* Y) {
  constexpr int N = 16 * NC, P = K / 16;
  auto fetch = [&](int p) {
    float* s = ring + (p & 1) * kPiece;
    for (int i = k.t; i < N * 4; i += kHeadThreads2) {
      const int o = i >> 2, q = i & 3;
      cp16(s + (o / NC + 16 * (o % NC)) * 20 + 4 * q, W + o * K + 16 * p + 4 * q);
    }
    cp_commit();
  };
  float y[NC][4];
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) y[j][r] = 0.0f;
  fetch(0);
#pragma unroll 1
  for (int p = 0; p < P; ++p) {
    if (p + 1 < P) {
      fetch(p + 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    const float* s = ring + (p & 1) * kPiece + k.c * 20;
    const float* x = X + 16 * p * kRS + 4 * k.rg;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float4 xv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[u] = ld4(x + (4 * q + u) * kRS);
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const float4 w = ld4(s + 16 * j * 20 + 4 * q);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float wu = (&w.x)[u];
          y[j][0] = fmaf(xv[u].x, wu, y[j][0]);
          y[j][1] = fmaf(xv[u].y, wu, y[j][1]);
          y[j][2] = fmaf(xv[u].z, wu, y[j][2]);
          y[j][3] = fmaf(xv[u].w, wu, y[j][3]);
        }
      }
    }
    __syncthreads();  // the slot is free again
  }
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const float b = __ldg(B + k.c * NC + j);
    st4(Y + (k.c * NC + j) * kRS + 4 * k.rg, relu(y[j][0] + b), relu(y[j][1] + b), relu(y[j][2] + b),
        relu(y[j][3] + b));
  }
  __syncthreads();
}
// d = W^T D: NC input columns per thread (16 NC inputs), N outputs.
template <int NC, int N>
__device__ __forceinline__ void head_dx(const HeadCtx& k, float* ring, const float* D, const float* __restrict__ W,
                                        float (&y)[NC][4]) {
  constexpr int K = 16 * NC, P = N / 16;
  auto fetch = [&](int p) {
    float* s = ring + (p & 1) * kPiece;
    for (int i = k.t; i < 16 * (K / 4); i += kHeadThreads2) {
      const int o = i / (K / 4), q = i % (K / 4);
      cp16(s + o * (K + 4) + 4 * q, W + (16 * p + o) * K + 4 * q);
    }
    cp_commit();
  };
#pragma unroll
  for (int j = 0; j < NC; ++j)
#pragma unroll
    for (int r = 0; r < 4; ++r) y[j][r] = 0.0f;
  fetch(0);
#pragma unroll 1
  for (int p = 0; p < P; ++p) {
    if (p + 1 < P) {
      fetch(p + 1);
      cp_wait<1>();
    } else {
      cp_wait<0>();
    }
    __syncthreads();
    const float* s = ring + (p & 1) * kPiece + k.c * NC;
    const float* d = D + 16 * p * kRS + 4 * k.rg;
#pragma unroll 4
    for (int o = 0; o < 16; ++o) {
      const float4 v = ld4(d + o * kRS);
#pragma unroll
      for (int j4 = 0; j4 < NC / 4; ++j4) {
        const float4 w = ld4(s + o * (K + 4) + 4 * j4);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float wu = (&w.x)[u];
          float(&yj)[4] = y[4 * j4 + u];
          yj[0] = fmaf(v.x, wu, yj[0]);
          yj[1] = fmaf(v.y, wu, yj[1]);
          yj[2] = fmaf(v.z, wu, yj[2]);
          yj[3] = fmaf(v.w, wu, yj[3]);
        }
      }
    }
    __syncthreads();
  }
}
// y masked by A > 0 (columns c NC + j) into D, with the bias gradients.
template <int NC>
__device__ __forceinline__ void mask_store(const HeadCtx& k, const float* A, float* D, float* gb, float (&y)[NC][4]) {
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    const int o = (k.c * NC + j) * kRS + 4 * k.rg;
    const float4 x = ld4(A + o);
    y[j][0] = x.x > 0.0f ? y[j][0] : 0.0f;
    y[j][1] = x.y > 0.0f ? y[j][1] : 0.0f;
    y[j][2] = x.z > 0.0f ? y[j][2] : 0.0f;
    y[j][3] = x.w > 0.0f ? y[j][3] : 0.0f;
    st4(D + o, y[j]);
    head_db(k, gb + k.c * NC + j, y[j]);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kHeadThreads2, 1) k_train_head(const __grid_constant__ TrainArgs a) {
  extern __shared__ __align__(16) float sm[];
  HeadCtx k;
  head_coords(k);
  k.a = &a;
  k.tw = sm;
  float* ring = sm + kTailW;
  float* H0 = ring + 2 * kPiece;
  float *A1 = H0 + 128 * kRS, *A2 = A1 + 128 * kRS, *A3 = A2 + 64 * kRS, *D3 = A3 + 32 * kRS;
  k.T = D3 + 32 * kRS;
  float *D2 = k.T, *D1 = k.T + 64 * kRS;  // over the tail's storage, once it is done
  load_tail_weights(a, k.tw);
  const TrainTables& T = c_tt;
  const int tiles = (a.n + kR - 1) / kR;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    k.r0 = tile * kR;
    __syncthreads();
    for (int i = k.t; i < 32 * 16; i += kHeadThreads2) {  // 4 x 4 pieces, transposed
      const int rg = i & 15, cg = i >> 4;
      float4 v[4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
        v[r] = reinterpret_cast<const float4*>(a.wk.h0 + (size_t)(k.r0 + 4 * rg + r) * 128)[cg];
      float* x = H0 + 4 * cg * kRS + 4 * rg;
      st4(x, v[0].x, v[1].x, v[2].x, v[3].x);
      st4(x + kRS, v[0].y, v[1].y, v[2].y, v[3].y);
      st4(x + 2 * kRS, v[0].z, v[1].z, v[2].z, v[3].z);
      st4(x + 3 * kRS, v[0].w, v[1].w, v[2].w, v[3].w);
    }
    __syncthreads();
    head_fwd<8, 128>(k, ring, H0, a.w + T.lc0w, a.w + T.lc0b, A1);
    head_fwd<4, 128>(k, ring, A1, a.w + T.lc1w, a.w + T.lc1b, A2);
    head_fwd<2, 64>(k, ring, A2, a.w + T.lc2w, a.w + T.lc2b, A3);
    {
      float d[2][4];
      tail_tile(k, A3, d);
      mask_store<2>(k, A3, D3, a.grad + T.lc2b, d);
    }
    head_dw<2, 4>(k, D3, A2, a.grad + T.lc2w);
    {
      float d[4][4];
      head_dx<4, 32>(k, ring, D3, a.w + T.lc2w, d);
      mask_store<4>(k, A2, D2, a.grad + T.lc1b, d);
    }
    head_dw<4, 8>(k, D2, A1, a.grad + T.lc1w);
    float d[8][4];
    head_dx<8, 64>(k, ring, D2, a.w + T.lc1w, d);
    mask_store<8>(k, A1, D1, a.grad + T.lc0b, d);
    head_dw<8, 8>(k, D1, H0, a.grad + T.lc0w);
    head_dx<8, 128>(k, ring, D1, a.w + T.lc0w, d);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float* p = a.wk.dh0 + (size_t)(k.r0 + 4 * k.rg + r) * 128 + 8 * k.c;
      st4(p, d[0][r], d[1][r], d[2][r], d[3][r]);
      st4(p + 4, d[4][r], d[5][r], d[6][r], d[7][r]);
    }
  }
}

// ---- gates backward ----------------------------------------------------------------
// Features: the pool (75), per block H (8), DH (8), DG (3), then SW (16),
// DF (16), DS (6), DX (8).
constexpr int kGH = 75, kGDH = kGH + 96, kGDG = kGDH + 96, kGSW = kGDG + 36, kGDF = kGSW + 16, kGDS = kGDF + 16,
              kGDX = kGDS + 6, kGX = kGDX + 8;
constexpr int kGatesSmem = kGX * kRS * 4;
// One weight gradient: features a and b whose product is summed over the
// rows, and its place in the blob. b < 0: the sum of a alone (a bias).
struct GateGrad {
  short a, b;
  int g;
};
constexpr int kGateGrads = 12 * (24 + 64) + 1200 + 96 + 24 + 8;
struct GateTable {
  GateGrad e[kGateGrads];
};
constexpr GateTable make_gate_table() {
  GateTable t{};
  const TrainTables T = make_train_tables();
  int n = 0;
  for (int b = 0; b < 12; ++b) {
    for (int o = 0; o < 3; ++o)
      for (int j = 0; j < 8; ++j) t.e[n++] = {(short)(kGDG + 3 * b + o), (short)(kGH + 8 * b + j), T.se1[b] + 8 * o + j};
    for (int o = 0; o < 8; ++o)
      for (int j = 0; j < 8; ++j) {
        const int p = j < 3 ? 3 * b + j : j < 6 ? 36 + 3 * b + j - 3 : 72 + j - 6;
        t.e[n++] = {(short)(kGDH + 8 * b + o), (short)p, T.se0[b] + 8 * o + j};
      }
  }
  for (int o = 0; o < 16; ++o)
    for (int j = 0; j < 75; ++j) t.e[n++] = {(short)(kGDF + o), (short)j, T.f1 + 75 * o + j};
  for (int o = 0; o < 6; ++o)
    for (int j = 0; j < 16; ++j) t.e[n++] = {(short)(kGDS + o), (short)(kGSW + j), T.f2 + 16 * o + j};
  for (int o = 0; o < 8; ++o)
    for (int j = 0; j < 3; ++j) t.e[n++] = {(short)(kGDX + o), (short)(72 + j), T.ggw + 3 * o + j};
  for (int o = 0; o < 8; ++o) t.e[n++] = {(short)(kGDX + o), (short)-1, T.ggb + o};
  return t;
}
static __device__ const GateTable d_gate_table = make_gate_table();

__global__ void __launch_bounds__(256, 2) k_train_gates(const __grid_constant__ TrainArgs a) {
  extern __shared__ __align__(16) float F[];
  const TrainTables& T = c_tt;
  const float* __restrict__ W = a.w;
  const int t = threadIdx.x, r0 = blockIdx.x * kR;
  const size_t N = a.wk.rows;
  for (int i = t; i < 72 * 16; i += 256) {
    const int f = i >> 4, q = i & 15;
    *reinterpret_cast<float4*>(F + f * kRS + 4 * q) = ld4(a.wk.pool + (size_t)f * N + r0 + 4 * q);
  }
  if (t < kR) {
    const float* x = a.aux + 5 * (size_t)min(r0 + t, a.n - 1);
    for (int i = 0; i < 3; ++i) F[(72 + i) * kRS + t] = x[i];
  }
  __syncthreads();
  if (t < 12 * 16) {
    const int b = t >> 4, rg = t & 15;
    float4 x[8], dg[3];
    se_inputs(F, b, rg, x);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const size_t at = (size_t)(3 * b + k) * N + r0 + 4 * rg;
      const float4 g = ld4(a.wk.gate + at), d0 = ld4(a.wk.dgate + at), d1 = ld4(a.wk.dgate + 36 * N + at);
      dg[k] = make_float4((d0.x + d1.x) * g.x * (1.0f - g.x), (d0.y + d1.y) * g.y * (1.0f - g.y),
                          (d0.z + d1.z) * g.z * (1.0f - g.z), (d0.w + d1.w) * g.w * (1.0f - g.w));
      st4(F + (kGDG + 3 * b + k) * kRS + 4 * rg, dg[k]);
    }
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      const float4 s = se_hidden(W + T.se0[b], x, o);
      float4 dh = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
      for (int j = 0; j < 3; ++j) fma4(dh, dg[j], __ldg(W + T.se1[b] + j * 8 + o));
      st4(F + (kGH + 8 * b + o) * kRS + 4 * rg, relu4(s));
      st4(F + (kGDH + 8 * b + o) * kRS + 4 * rg, s.x > 0.0f ? dh.x : 0.0f, s.y > 0.0f ? dh.y : 0.0f,
          s.z > 0.0f ? dh.z : 0.0f, s.w > 0.0f ? dh.w : 0.0f);
    }
  }
  fin1(F, W + T.f1, F + kGSW * kRS);
  for (int i = t; i < 6 * kR; i += 256) {
    const int o = i / kR, row = i % kR;
    const size_t at = (size_t)o * N + r0 + row;
    const float g = a.wk.sp[at];
    F[(kGDS + o) * kRS + row] = (a.wk.dsp[at] + a.wk.dsp[6 * N + at]) * g * (1.0f - g);
  }
  for (int i = t; i < 8 * kR; i += 256) {
    const int row = i / 8, o = i % 8;
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < 3; ++j) s += F[(72 + j) * kRS + row] * __ldg(W + T.ggw + o * 3 + j);
    s += __ldg(W + T.ggb + o);
    F[(kGDX + o) * kRS + row] = s > 0.0f && r0 + row < a.n ? a.wk.dh0[(size_t)(r0 + row) * 128 + 120 + o] : 0.0f;
  }
  __syncthreads();
  for (int i = t; i < 16 * kR; i += 256) {
    const int o = i / kR, row = i % kR;
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < 6; ++j) s += __ldg(W + T.f2 + j * 16 + o) * F[(kGDS + j) * kRS + row];
    F[(kGDF + o) * kRS + row] = F[(kGSW + o) * kRS + row] > 0.0f ? s : 0.0f;
  }
  __syncthreads();
  for (int i = t; i < kGateGrads; i += 256) {
    const GateGrad e = d_gate_table.e[i];
    const float* pa = F + e.a * kRS;
    float s = 0.0f;
    if (e.b >= 0) {
      const float* pb = F + e.b * kRS;
#pragma unroll 4
      for (int q = 0; q < kR; q += 4) s = dot4(ld4(pa + q), ld4(pb + q), s);
    } else {
      for (int q = 0; q < kR; q += 4) {
        const float4 v = ld4(pa + q);
        s += (v.x + v.y) + (v.z + v.w);
      }
    }
    add_grad(a.grad + e.g, s);
  }
}

// ---- launches ------------------------------------------------------------------------

static int tile_attrs() {
  static DeviceCache attr;
  return attr.once([] {
    MR_CUDA(cudaFuncSetAttribute(k_train_trunk_fwd<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem));
    MR_CUDA(cudaFuncSetAttribute(k_train_trunk_fwd<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem));
    MR_CUDA(cudaFuncSetAttribute(k_train_trunk_bwd<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem));
    MR_CUDA(cudaFuncSetAttribute(k_train_trunk_bwd<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem));
    MR_CUDA(cudaFuncSetAttribute(k_train_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, kTailSmem));
    MR_CUDA(cudaFuncSetAttribute(k_train_head, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeadSmem2));
    MR_CUDA(cudaFuncSetAttribute(k_train_gates, cudaFuncAttributeMaxDynamicSharedMemorySize, kGatesSmem));
    return (int)MR_OK;
  });
}
static unsigned trunk_grid(int n) {  // two CTAs per SM
  const int ctas = ((n + kR - 1) / kR + kTrunkTiles - 1) / kTrunkTiles;
  return 3u * (unsigned)std::min(ctas, std::max(1, 2 * sm_count() / 3));
}
// The descriptors' 16-byte loads (load_desc).
static bool wide_rows(const TrainArgs& a) { return (reinterpret_cast<uintptr_t>(a.desc) & 15) == 0; }

// Statistics, gates and the trunks' forward: wk.h0 of the rows.
int launch_train_trunk_fwd(const TrainArgs& a, cudaStream_t s) {
  int rc = tile_attrs();
  if (rc) return rc;
  const auto stats = wide_rows(a) ? k_train_stats<true> : k_train_stats<false>;
  stats<<<(a.n + kR - 1) / kR, 256, (75 + 16) * kRS * 4, s>>>(a);
  MR_CUDA(cudaGetLastError());
  const auto trunk = wide_rows(a) ? k_train_trunk_fwd<true> : k_train_trunk_fwd<false>;
  trunk<<<trunk_grid(a.n), kTrunkTiles * kTrunkThreads, kFwdSmem, s>>>(a);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}
// The fp32 head: wk.h0 -> loss, gradients, wk.dh0.
int launch_train_head(const TrainArgs& a, cudaStream_t s) {
  k_train_head<<<std::min((a.n + kR - 1) / kR, sm_count()), kHeadThreads2, kHeadSmem2, s>>>(a);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}
// The tail alone: wk.a3 -> loss, gradients, wk.da3.
int launch_train_tail(const TrainArgs& a, cudaStream_t s) {
  k_train_tail<<<std::min((a.n + kR - 1) / kR, 2 * sm_count()), kHeadThreads2, kTailSmem, s>>>(a);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}
// The trunks and the gates backward from wk.dh0.
int launch_train_trunk_bwd(const TrainArgs& a, cudaStream_t s) {
  const auto trunk = wide_rows(a) ? k_train_trunk_bwd<true> : k_train_trunk_bwd<false>;
  trunk<<<trunk_grid(a.n), kTrunkTiles * kTrunkThreads, kBwdSmem, s>>>(a);
  MR_CUDA(cudaGetLastError());
  k_train_gates<<<(a.n + kR - 1) / kR, 256, kGatesSmem, s>>>(a);
  MR_CUDA(cudaGetLastError());
  return MR_OK;
}

}  // namespace mr
