// Training pieces shared by the trainer (mr_train.cu), the fp32 tile kernels
// (mr_train_tile.cu) and the BF16 tensor-core head (mr_train_tc.cu): the
// offsets of the network's weight arrays per block
// (core/radiancePredict.cu:370-485), the step's arguments and buffers.
#pragma once
#include "mr_internal.h"
#include "mr_net_layout.cuh"

namespace mr {

struct TrainTables {
  int S[12], from[12], se0[12], se1[12], w[12][3], b[12][3];
  int l81w[3], l81b[3], ld41w[3], ld41b[3];
  int f1, f2, ggw, ggb, lc0w, lc0b, lc1w, lc1b, lc2w, lc2b, lxw, lxb, lxrw[12], lxrb[12], lx12w, lx12b;
};
constexpr TrainTables make_train_tables() {
  TrainTables t{};
  const WeightTable wt = make_weight_table();
  const int S[12] = {8, 8, 16, 16, 16, 32, 32, 32, 8, 8, 8, 8};
  const int from[12] = {0, 8, 16, 32, 48, 64, 96, 128, 160, 168, 176, 184};
  const int se0[12] = {MR_W_LSE01W, MR_W_LSE11W, MR_W_LSE21W, MR_W_LSE31W, MR_W_LSE41W, MR_W_LSE51W,
                       MR_W_LSE61W, MR_W_LSE71W, MR_W_LDSE01W, MR_W_LDSE11W, MR_W_LDSE21W, MR_W_LDSE31W};
  const int se1[12] = {MR_W_LSE02W, MR_W_LSE12W, MR_W_LSE22W, MR_W_LSE32W, MR_W_LSE42W, MR_W_LSE52W,
                       MR_W_LSE62W, MR_W_LSE72W, MR_W_LDSE02W, MR_W_LDSE12W, MR_W_LDSE22W, MR_W_LDSE32W};
  const int lw[12][3] = {{MR_W_L01W, MR_W_L_Tr01W, MR_W_L_Hg01W}, {MR_W_L11W, MR_W_L_Tr11W, MR_W_L_Hg11W},
                         {MR_W_L21W, MR_W_L_Tr21W, MR_W_L_Hg21W}, {MR_W_L31W, MR_W_L_Tr31W, MR_W_L_Hg31W},
                         {MR_W_L41W, MR_W_L_Tr41W, MR_W_L_Hg41W}, {MR_W_L51W, MR_W_L_Tr51W, MR_W_L_Hg51W},
                         {MR_W_L61W, MR_W_L_Tr61W, MR_W_L_Hg61W}, {MR_W_L71W, MR_W_L_Tr71W, MR_W_L_Hg71W},
                         {MR_W_LD01W, MR_W_LD_Tr01W, MR_W_LD_Hg01W}, {MR_W_LD11W, MR_W_LD_Tr11W, MR_W_LD_Hg11W},
                         {MR_W_LD21W, MR_W_LD_Tr21W, MR_W_LD_Hg21W}, {MR_W_LD31W, MR_W_LD_Tr31W, MR_W_LD_Hg31W}};
  const int lb[12][3] = {{MR_W_L01B, MR_W_L_Tr01B, MR_W_L_Hg01B}, {MR_W_L11B, MR_W_L_Tr11B, MR_W_L_Hg11B},
                         {MR_W_L21B, MR_W_L_Tr21B, MR_W_L_Hg21B}, {MR_W_L31B, MR_W_L_Tr31B, MR_W_L_Hg31B},
                         {MR_W_L41B, MR_W_L_Tr41B, MR_W_L_Hg41B}, {MR_W_L51B, MR_W_L_Tr51B, MR_W_L_Hg51B},
                         {MR_W_L61B, MR_W_L_Tr61B, MR_W_L_Hg61B}, {MR_W_L71B, MR_W_L_Tr71B, MR_W_L_Hg71B},
                         {MR_W_LD01B, MR_W_LD_Tr01B, MR_W_LD_Hg01B}, {MR_W_LD11B, MR_W_LD_Tr11B, MR_W_LD_Hg11B},
                         {MR_W_LD21B, MR_W_LD_Tr21B, MR_W_LD_Hg21B}, {MR_W_LD31B, MR_W_LD_Tr31B, MR_W_LD_Hg31B}};
  for (int i = 0; i < 12; ++i) {
    t.S[i] = S[i]; t.from[i] = from[i];
    t.se0[i] = wt.off[se0[i]]; t.se1[i] = wt.off[se1[i]];
    for (int br = 0; br < 3; ++br) { t.w[i][br] = wt.off[lw[i][br]]; t.b[i][br] = wt.off[lb[i][br]]; }
  }
  const int l81w[3] = {MR_W_L81W, MR_W_L_Tr81W, MR_W_L_Hg81W}, l81b[3] = {MR_W_L81B, MR_W_L_Tr81B, MR_W_L_Hg81B};
  const int ld41w[3] = {MR_W_LD41W, MR_W_LD_Tr41W, MR_W_LD_Hg41W};
  const int ld41b[3] = {MR_W_LD41B, MR_W_LD_Tr41B, MR_W_LD_Hg41B};
  for (int br = 0; br < 3; ++br) {
    t.l81w[br] = wt.off[l81w[br]]; t.l81b[br] = wt.off[l81b[br]];
    t.ld41w[br] = wt.off[ld41w[br]]; t.ld41b[br] = wt.off[ld41b[br]];
  }
  t.f1 = wt.off[MR_W_LSEFin1W]; t.f2 = wt.off[MR_W_LSEFin2W];
  t.ggw = wt.off[MR_W_LGGSW]; t.ggb = wt.off[MR_W_LGGSB];
  t.lc0w = wt.off[MR_W_LC0W]; t.lc0b = wt.off[MR_W_LC0B]; t.lc1w = wt.off[MR_W_LC1W]; t.lc1b = wt.off[MR_W_LC1B];
  t.lc2w = wt.off[MR_W_LC2W]; t.lc2b = wt.off[MR_W_LC2B]; t.lxw = wt.off[MR_W_LXW]; t.lxb = wt.off[MR_W_LXB];
  const int rw[12] = {MR_W_LX0W, MR_W_LX1W, MR_W_LX2W, MR_W_LX3W, MR_W_LX4W, MR_W_LX5W,
                      MR_W_LX6W, MR_W_LX7W, MR_W_LX8W, MR_W_LX9W, MR_W_LX10W, MR_W_LX11W};
  const int rb[12] = {MR_W_LX0B, MR_W_LX1B, MR_W_LX2B, MR_W_LX3B, MR_W_LX4B, MR_W_LX5B,
                      MR_W_LX6B, MR_W_LX7B, MR_W_LX8B, MR_W_LX9B, MR_W_LX10B, MR_W_LX11B};
  for (int i = 0; i < 12; ++i) { t.lxrw[i] = wt.off[rw[i]]; t.lxrb[i] = wt.off[rb[i]]; }
  t.lx12w = wt.off[MR_W_LX12W]; t.lx12b = wt.off[MR_W_LX12B];
  return t;
}
static __constant__ TrainTables c_tt = make_train_tables();

__device__ __forceinline__ float relu(float x) { return x > 0.0f ? x : 0.0f; }
__device__ __forceinline__ float sigmoid(float x) { return 1.0f / (1.0f + expf(-x)); }

// Rows of a tile of the training kernels (mr_train_tile.cu).
constexpr int kTrainRows = 64;

// Buffers of a training step, `rows` rows each (a multiple of kTrainRows).
// Feature-major ones hold feature f of row r at [f * rows + r].
struct TrainWork {
  size_t rows;
  float* h0;     // head input, rows x 128
  float* dh0;    // its gradient, rows x 128
  float* pool;   // 72 features: segment means, then maxima
  float* gate;   // 36: squeeze-excitation gates
  float* sp;     // 6: gates of the trunk outputs
  float* dgate;  // 2 x 36: gradients of the gates, two partial sums
  float* dsp;    // 2 x 6: gradients of the output gates, two partial sums
  float* a3;     // BF16 step: LC2 output after ReLU, rows x 32
  float* da3;    // BF16 step: its gradient, 0 where a3 is 0
  // For the trunks' backward, per tile of kTrainRows rows and branch:
  float* xs;       // [kTrunkSaved][kTrainRows]: every layer's input, then the two outputs
  uint16_t* mask;  // kTrunkMask bytes: the signs of every layer's outputs
};
constexpr int kTrunkSaved = 232 + 40;         // features
constexpr int kTrunkMask = 14 * 128 * 2;      // bytes: layers, threads
static_assert(3 * kTrunkMask % (4 * kTrainRows) == 0, "whole floats per row");
constexpr size_t kTrunkMaskFloats = 3 * kTrunkMask / (4 * kTrainRows);  // per row
constexpr size_t kTrainWorkFloats =           // per row
    128 + 128 + 72 + 36 + 6 + 72 + 12 + 32 + 32 + 3 * kTrunkSaved + kTrunkMaskFloats;

struct TrainArgs {
  const float* w;       // fp32 master weights (blob layout)
  float* grad;          // fp32 gradient accumulator (blob layout)
  const float* desc;    // n x 576, row-major
  const float* aux;     // n x 5 (g, gamma, srp.xyz)
  const float* label;   // n radiance labels
  int n;
  float inv_batch;      // loss weight: 1 / rows of the whole batch
  float* loss;          // sum of (X - T)^2 / batch, added to
  TrainWork wk;
};

int launch_train_trunk_fwd(const TrainArgs& a, cudaStream_t s);
int launch_train_head(const TrainArgs& a, cudaStream_t s);
int launch_train_tail(const TrainArgs& a, cudaStream_t s);
int launch_train_trunk_bwd(const TrainArgs& a, cudaStream_t s);

}  // namespace mr
