// Parameter block of the two-SM GEMM (kernel in gemm_pair_tcgen05.cu).
#pragma once
#include "gemm_tcgen05.cuh"

namespace swb {

struct PairParams {
  int M, N;
  int tiles_m, tiles_n;               // tiles of 256 rows x BN columns (grouped: tiles_m bounds the list)
  int kblocks, kblocks_per_split, splits;
  void* out;
  int ldd, out_fp32;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;      // D = act(acc + bias) * gate + residual
  int ld_res;
  const __nv_bfloat16* gate;          // one row of N factors for each rows_per_gate rows
  int ld_gate, rows_per_gate;
  int act;
  float act_a, act_b;
  int first_n;                        // > 0: columns from here on (a multiple of the tile width) go to out2 and take act2
  void* out2;
  int ldd2, act2;
  float* workspace;                   // [tile][CTA of the pair][split][BN][128] fp32
  int* counters;                      // [tile][CTA of the pair][epilogue warp], zero between launches
  const int4* group_tiles;            // grouped rows: (first row, rows of the group from there on, group, -)
  const int* group_count;             // entries of the list, on the device
  // 3x3 convolution (conv_c > 0): a CTA's 128 rows are a box of 2^box_w_log x 2^box_h_log pixels, boxes run row by row
  int conv_n, conv_h, conv_w, conv_c;
  int box_w_log, box_h_log, boxes_x, boxes_y;
  float* stats;                       // optional [conv_n][N / group_channels][2]: sums and sums of squares of what is stored are added
  int group_channels;                 // 4, 8, 16 or 32
};

bool gemm_pair_accepts(const GemmArgs& a);
// Tile width and number of k-splits for a plain product whose partial sums may take sum_bytes. Returns its estimated microseconds.
// multiple > 0: only widths that divide it.
double gemm_pair_plan(int T, int N, int K, size_t sum_bytes, int* block_n, int* splits, int multiple = 0);
// Bytes of partial sums of a product (block_n, splits: 0 = by the plan); 0 = no k-splits.
size_t gemm_pair_split_bytes(int T, int N, int K, int block_n, int splits);
constexpr size_t GEMM_SPLIT_BYTES_MAX = (size_t)96 << 20;
// block_n, splits: 0 = by the plan.
int gemm_pair_launch(const GemmArgs& a, int block_n, int splits, cudaStream_t stream);

}  // namespace swb
