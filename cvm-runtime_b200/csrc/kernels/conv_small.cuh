// The small-launch form of the tensor-core convolution (conv_small.cu), chosen and prepared by
// cvmk_conv2d_tc_prepare().
#pragma once
#include "tc_common.cuh"

namespace cvmk {

struct SmallConvParams {
  void* y;
  int y_dtype;
  int m_total, oc, oh, ow;
  int c, kw, cblocks;             // cblocks: K blocks per filter tap
  int stride_h, stride_w, pad_h, pad_w, dil_h, dil_w;
  int a_mode;                     // 0 plain 2-D tiles (1x1, dense), 1 im2col-mode TMA, 2 spatial patches
  int patch_w, patch_h, patch_n, patch_w_log2, patch_h_log2, tiles_w, tiles_h;
  int block_k, block_n, stages;
  int group;                      // units that share a ring stage and its barrier
  int swap;                       // dense: the weights are the 128-row operand, the activations the block_n-row one
  int num_n_tiles, images;
  int units;                      // (filter tap, channel block) pairs of the whole reduction
  int split, split_log2;          // CTAs of a cluster, each reducing units / split of them
  int tmem_cols;
  tc::FastDiv fd_n_tiles, fd_tiles_w, fd_tiles_h, fd_ohow, fd_ow, fd_cblocks, fd_kw;
  int* status;
  const int32_t* bias;
  int bias_static, first_step;
  const int8_t* res;              // int8 operand of a fused tensor add / subtract, or nullptr
  int pad_;                       // what follows lies better this way (without it 57 launches of ResNet-50, 13 images: 313.0 -> 314.1 us)
  int fast_variant;               // -1: the chain step by step; else as in conv_tc.cu (+ 8: wide)
  int f_mul, f_add, f_pre_lo, f_pre_hi;
  tc::FastQ fq;
  DevChain chain;
};

constexpr int SMALL_MAX_STAGES = 12;

// Dynamic shared memory of a launch: the operand ring (which also holds the partial sums this CTA sends
// when the reduction is cut, or else the tile's packed results on their way out: more than the ring where
// that is a single unit of 32 channels) and, behind it, the partial sums it receives.
__host__ __device__ inline int small_ring_bytes(int block_k, int block_n, int units, int split) {   // units in the ring
  const int ring = units * (tc::BLOCK_M + block_n) * block_k, sums = tc::BLOCK_M * block_n * (split > 1 ? 4 : 1);
  return ring > sums ? ring : sums;
}
inline int small_smem_bytes(int block_k, int block_n, int units, int split) {
  const int rows = split > 1 ? tc::BLOCK_M / split * (split - 1) : 0;   // received from the other ranks, split 2, 4 or 8
  return 1024 + small_ring_bytes(block_k, block_n, units, split) + rows * block_n * 4;
}
int launch_conv_small(const CUtensorMap& a, const CUtensorMap& b, const SmallConvParams& p, int grid, int smem, cudaStream_t stream);

}  // namespace cvmk
