// Depthwise 3 x 3 convolutions, stride 1 and 2, on the sm_100a tensor cores.
//
// A depthwise layer is 9 multiplies an output element; on the CUDA cores it is bound by the instructions around
// them (about 23 an element), at a third of the memory rate.  Here a group of 32 channels is multiplied by
// block-diagonal weights: D[pixel, o] = sum_t A_t[pixel, 32 channels] x diag(w_t), one tcgen05.mma kind::i8 of K = 32
// a filter tap, whose A operand is a window of the staged input.  Such a product reads 4 KB of A and 32 bytes for each
// column from shared memory, at 128 bytes a cycle: 40 cycles with 32 columns, 48 with 64 and 64 with 128.  So, with stride 1, a row
// of the tile is not one output pixel but a block of 2 x 2, whose 4 x 4 input pixels are multiplied once each, by the
// weights of the up to four outputs that they belong to side by side: 16 products where four times nine were.  With
// stride 2 a row is one output pixel, and the input, four times the output, sets the time.
//
// In both, A's rows are two input pixels apart, so the input is staged as two planes, of every second pixel each (TMA
// boxes with a traversal stride of two), P = 32 or 64 channels a pixel: a tap is a window of one of the planes, and its
// 8-row groups are two lines apart.  Where the image has just these P channels, pairs of pixels are staged instead, in
// half as many rows of twice the bytes (a box's rows cost the TMA engine the same, be they 32 or 128 bytes), and a tap
// is a half of the pairs.  A tile is 8 x 16 rows (blocks or pixels) of one image, or of several images with few lines
// stacked on top of each other, each with the extra line that its last taps read.
//
// Persistent CTAs of one channel block each; its weights are laid out once in shared memory by the CTA itself, while
// the kernel before it still runs.  Warp 0 loads the input of the next tiles (zero fill outside the image), warp 1
// issues the products, eight or sixteen warps requantise and write the tile as it will lie in memory, the last one
// stores it.  Two accumulators, so that the requantisation of a tile runs beside the products of the next.
//
// One B200, 256 images, launched between events (some 6 us of it the launch), the kernels before -> this one: 32
// channels at 112 x 112 78 -> 47 us (210 MB, 32 us at the copy rate), 128 at 56 x 56 76 -> 52 (32), 256 at 28 x 28
// 47 -> 30 (16), 512 at 14 x 14 29 -> 20 (8); stride 2: 64 at 112 x 112 86 -> 51 (40), 128 at 56 x 56 47 -> 33 (20).  No one
// thing bounds stride 1: 128 channels at 56 x 56 take 47 us without the products, 49 without the input, 51 without the
// requantisation, all of them 53; a quarter of the rows of such tiles lies outside the images.
//
// Any chain behind the products: [bias] shift clamp has forms of its own; a wide sum, and the sum with another tensor (whose
// tile TMA brings into the output buffer before the result), run packed too, everything else step by step.  128 channels at
// 28 x 28, 150 images, in a chain of such layers: 9.1 us with shift and clamp, 14.5 with a wide sum or a clip alone, 15.3 with a
// tensor (depthwise3x3_kernel 39.0, 34.8, 57.2; the clip step by step 18.9; the tensor loaded by the threads that need it 18.4:
// a row's 32 bytes lie in a cache line of their own).  The wide sum's clamp is three more integer instructions an element, the
// tensor waits in one of the two output buffers, which it takes from the tile two before.
//
// Reproduces groupwise_conv2d with groups = C (src/runtime/cpu/ops/ops.cc:333-366) and the chain behind it.
// Every wait is bounded, as in conv_tc.cu.
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>
#include <algorithm>
#include "common.cuh"
#include "conv_dw.cuh"
#include "tc_common.cuh"

namespace cvmk {
namespace {

using namespace tc;

constexpr int TILE_X = 8, TILE_Y = 16;     // rows of a tile: TILE_X neighbours are one 8-row group of the operand
constexpr int BOX_H = 2 * (TILE_Y + 1);    // lines
constexpr int MAX_UNITS = 8;
constexpr int SMEM_MAX = 227 * 1024 - 1024;   // less the static part

struct DwParams {
  const int8_t* w;        // [3, 3, C]
  const int32_t* bias;
  int* status;
  int C, images;
  int rows_x, rows_y;     // operand rows of an image: 2 x 2 blocks of output pixels (stride 1) or output pixels
  int pad_h, pad_w;
  int per_tile;           // images of a tile
  int pitch_y;            // operand lines from one image of a tile to the next
  int band;               // operand lines of an image in a tile
  int tiles_x, tiles_y, c_tiles, num_tiles;
  FastDiv fd_c, fd_x, fd_y, fd_pitch;
  int units, box_bytes;    // of the ring; bytes of a box
  int pairs, out_pairs;    // the input is staged, the output stored as pairs of pixels
  uint32_t out_mask;       // the output tile's swizzle: address bits 4.. ^= bits 7.. & out_mask
  int mul, add;
  uint32_t lo, hi;
  int bias_static;
  // chains that are not just [bias] shift clamp
  int out_w, out_h;        // of an image, in pixels
  int kind;                // of the packed form (PackedChain), or -1: step by step
  int out_box_bytes;       // of one image's part of an output tile
  int wide, pre_lo, pre_hi;
  uint32_t lo2, hi2;
  DevChain chain;
};

// How the sums become bytes: shift and clamp with a lower bound of any kind, or of 0, or any other chain.
enum { PACKED = 0, PACKED_RELU = 1, OTHER = 2 };

// The products of one channel group: the input pixel of the block, the columns and the first of them, and where their
// weights begin in a row of blocks of 32 x 32 bytes, each with one filter tap on its diagonal (9: none).  Stride 1: the
// outputs of a block are 32 columns each, in the order (0,0), (0,1), (1,1), (1,0); a product of an edge has a zero
// block where it meets an output that it does not belong to.  There are three shapes only, and the rows
// of blocks that the products need overlap, 35 KB where 48 blocks would stand alone: what shared memory has left is
// the ring's.
struct Product { int iy, ix, n, col, first; };
constexpr int NUM_PRODUCTS1 = 16, NUM_BLOCKS1 = 35;
__host__ __device__ constexpr Product product1(int i) {
  constexpr Product list[NUM_PRODUCTS1] = {
      {1, 1, 128, 0, 15}, {1, 2, 128, 0, 4}, {2, 1, 128, 0, 12}, {2, 2, 128, 0, 1}, {1, 0, 128, 0, 31}, {2, 0, 128, 0, 28},
      {1, 3, 128, 0, 23}, {2, 3, 128, 0, 20},
      {0, 0, 64, 0, 19}, {0, 1, 64, 0, 18}, {0, 2, 64, 0, 7}, {0, 3, 64, 0, 26},
      {3, 0, 64, 64, 10}, {3, 1, 64, 64, 11}, {3, 2, 64, 64, 0}, {3, 3, 64, 64, 9}};
  return list[i];
}
__host__ __device__ constexpr int block_tap1(int b) {
  constexpr int list[NUM_BLOCKS1] = {7, 8, 7, 4, 5, 4, 1, 2, 1, 8, 9, 6, 7, 6, 3, 4, 3, 0, 1, 0, 9, 8, 5, 9, 5, 2, 9, 2, 6, 9, 9, 3, 9, 9, 0};
  return list[b];
}
// Every output of a block gets each of its nine taps once, from the input pixel it belongs to.
constexpr bool products1_complete() {
  constexpr int out_y[4] = {0, 0, 1, 1}, out_x[4] = {0, 1, 1, 0};
  int seen[4][9] = {};
  for (int i = 0; i < NUM_PRODUCTS1; ++i) {
    const Product p = product1(i);
    for (int j = 0; j < p.n / 32; ++j) {
      const int q = p.col / 32 + j, tap = block_tap1(p.first + j);
      if (tap == 9) continue;
      if (out_y[q] + tap / 3 != p.iy || out_x[q] + tap % 3 != p.ix) return false;
      ++seen[q][tap];
    }
  }
  for (int q = 0; q < 4; ++q)
    for (int t = 0; t < 9; ++t)
      if (seen[q][t] != 1) return false;
  return true;
}
static_assert(products1_complete(), "taps of a block");
constexpr int NUM_PRODUCTS2 = 9, NUM_BLOCKS2 = 9;   // stride 2: one output, nine taps
__host__ __device__ constexpr Product product2(int i) { return Product{i / 3, i % 3, 32, 0, i}; }
struct BlockTaps { int8_t t[NUM_BLOCKS1]; };
constexpr BlockTaps make_taps() {
  BlockTaps b = {};
  for (int i = 0; i < NUM_BLOCKS1; ++i) b.t[i] = (int8_t)block_tap1(i);
  return b;
}
__constant__ BlockTaps block_taps1 = make_taps();

template <int S>
struct Shape {
  static constexpr int PRODUCTS = S == 1 ? NUM_PRODUCTS1 : NUM_PRODUCTS2;
  static constexpr int BLOCKS = S == 1 ? NUM_BLOCKS1 : NUM_BLOCKS2;
  static constexpr int OUT = S == 1 ? 2 : 1;              // output pixels of a row, in each direction
  static constexpr int COLS = 32 * OUT * OUT;             // accumulator columns of a channel group
  static constexpr int EPI_WARPS = S == 1 ? 16 : 8;       // warps that requantise
  static constexpr int IO_WARP = 2 + EPI_WARPS, THREADS = 32 * (3 + EPI_WARPS);
};

// G: channel groups of a tile, 1 or 2 (P = 32 G channels).  PAIRS: a tile's input is one box of pixel pairs, not two
// planes; where an image has P channels, an even width and padding 1.
template <int S, int G, int PAIRS, int FORM>
__global__ void __launch_bounds__(Shape<S>::THREADS, 1)
conv_dw_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_y, const __grid_constant__ CUtensorMap tmap_r,
               const __grid_constant__ DwParams p) {
  using Sh = Shape<S>;
  constexpr int P = 32 * G;                               // bytes of a staged pixel
  constexpr int ROW = PAIRS ? 2 * P : P, LINE = (PAIRS ? TILE_X + 2 : TILE_X + 1) * ROW;   // a row of the operand, a line of them
  constexpr int UNIT = (LINE * BOX_H + 1023) & ~1023, UNITS = PAIRS ? 1 : 2;               // units of the ring: boxes of a tile
  constexpr int OUT_LINE = TILE_X * Sh::OUT * P, OUT_BYTES = TILE_Y * Sh::OUT * OUT_LINE;
  constexpr int W_BYTES = G * Sh::BLOCKS * 1024;
  constexpr int ACC_COLS = G * Sh::COLS;
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[MAX_UNITS], bar_empty[MAX_UNITS];
  __shared__ uint64_t bar_acc_full[2], bar_acc_empty[2], bar_staged[2], bar_out_free[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ __align__(16) int32_t bias_s[P];   // (other chains; the two others keep it in registers)
  uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* const ring = smem + W_BYTES;
  uint8_t* const out = ring + p.units * UNIT;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int c_tile = (int)blockIdx.x - fdiv((int)blockIdx.x, p.fd_c) * p.c_tiles;   // (the grid is a multiple of c_tiles)
  const int c0 = c_tile * P;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.units; ++s) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bar_acc_full[a], 1);
      mbar_init(&bar_acc_empty[a], Sh::EPI_WARPS);
      mbar_init(&bar_staged[a], Sh::EPI_WARPS);
      mbar_init(&bar_out_free[a], 1);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 512);
    pdl_trigger();   // (not before this CTA has its columns)
  }
  int32_t bias[32];
  uint32_t tmem_base = 0;
  if (warp == 0) {   // its loads need the barriers only, which it has set up itself
    __syncwarp();
    __threadfence_block();
    asm volatile("bar.arrive 1, %0;" ::"n"(Sh::THREADS) : "memory");
  } else {
    if (warp >= 2 && warp < Sh::IO_WARP) {
      // all of a thread's weights and its bias set out before anything is stored, behind which ordinary loads would stay
      constexpr int WORKERS = 32 * Sh::EPI_WARPS, MINE = (G * Sh::BLOCKS * 32 + WORKERS - 1) / WORKERS;
      const int t = (int)threadIdx.x - 64;
      const int g = G == 2 ? (warp - 2) >> (S == 1 ? 3 : 2) : 0;
      if (!p.bias_static) pdl_wait();
      const int32_t my_bias = !p.bias ? 0 : (FORM == OTHER ? (t < P ? p.bias[c0 + t] : 0) : p.bias[c0 + g * 32 + lane]);
      uint8_t w[MINE];
#pragma unroll
      for (int k = 0; k < MINE; ++k) {
        const int i = t + k * WORKERS, c = i & 31, blk = i >> 5, bg = blk / Sh::BLOCKS, b = blk - bg * Sh::BLOCKS;
        const int tap = blk < G * Sh::BLOCKS ? (S == 1 ? block_taps1.t[b] : b) : 9;
        w[k] = tap == 9 ? (uint8_t)0 : (uint8_t)p.w[(size_t)tap * p.C + c0 + bg * 32 + c];
      }
      for (int i = t; i < W_BYTES / 16; i += WORKERS) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
      asm volatile("bar.sync 2, %0;" ::"n"(WORKERS) : "memory");
#pragma unroll
      for (int k = 0; k < MINE; ++k) {
        const int i = t + k * WORKERS;
        const uint32_t at = (uint32_t)((i & 31) * 33);   // row c, byte c
        if ((i >> 5) < G * Sh::BLOCKS) smem[(size_t)(i >> 5) * 1024 + (at ^ (((at >> 7) & 1u) << 4))] = w[k];
      }
      fence_async_smem();
      if (FORM == OTHER && t < P) bias_s[t] = p.wide ? my_bias : (int32_t)((uint32_t)(my_bias + p.add) * (uint32_t)p.mul);
#pragma unroll
      for (int j = 0; j < (FORM == OTHER ? 0 : 32); ++j)
        bias[j] = (int32_t)((uint32_t)(__shfl_sync(0xffffffffu, my_bias, j) + p.add) * (uint32_t)p.mul);
    }
    if (warp == Sh::IO_WARP && lane < 2)
      asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(lane ? &tmap_y : &tmap_x)) : "memory");
    tc_fence_before();
    asm volatile("bar.sync 1, %0;" ::"n"(Sh::THREADS) : "memory");
    tc_fence_after();
    tmem_base = tmem_slot;
  }

  // Tile t: x fastest after the channel block, then y, then images.
  auto origin = [&](int tile, int* x0, int* y0, int* n0) {
    const int m = fdiv(tile, p.fd_c), r = fdiv(m, p.fd_x), i = fdiv(r, p.fd_y);
    *x0 = (m - r * p.tiles_x) * TILE_X;
    *y0 = (r - i * p.tiles_y) * p.band;
    *n0 = i * p.per_tile;
  };
  const int step = (int)gridDim.x;
  const bool has_operand = FORM == OTHER && p.kind > 0;   // its tile lies in the output buffer before the result does

  if (warp == 0) {
    // ---------------------------------------------------------------- input
    const bool leader = elect_one();
    int unit = 0;
    uint32_t phase = 0;
    bool live = true;
    pdl_wait();
    for (int tile = blockIdx.x; live && tile < p.num_tiles; tile += step) {
      int x0, y0, n0;
      origin(tile, &x0, &y0, &n0);
#pragma unroll
      for (int u = 0; u < UNITS; ++u) {
        if (!mbar_wait(&bar_empty[unit], phase ^ 1, &abort_flag, 1)) { live = false; break; }
        if (leader) {
          mbar_expect_tx(&bar_full[unit], (uint32_t)p.box_bytes);
          tma_load_4d(ring + unit * UNIT, &tmap_x, &bar_full[unit], c0, PAIRS ? x0 - 1 : 2 * x0 - p.pad_w + u, 2 * y0 - p.pad_h, n0);
        }
        __syncwarp();
        if (++unit == p.units) { unit = 0; phase ^= 1; }
      }
    }
    // nothing else waits for the last commits of the units, which must not come when the CTA has gone
    for (int u = 0; live && u < p.units; ++u) {
      live = mbar_wait(&bar_empty[unit], phase ^ 1, &abort_flag, 1);
      if (++unit == p.units) { unit = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- products
    const bool leader = elect_one();
    // rows of the operand in groups of 8, groups two lines apart
    const uint64_t desc_a = (umma_desc(smem_u32(ring), ROW) & ~((uint64_t)0x3FFF << 32)) | ((uint64_t)(2 * LINE / 16) << 32);
    const uint64_t desc_w = umma_desc(smem_u32(smem), 32);
    const uint32_t a_lo = (uint32_t)desc_a, a_hi = (uint32_t)(desc_a >> 32), w_lo = (uint32_t)desc_w, w_hi = (uint32_t)(desc_w >> 32);
    int unit = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    bool live = true;
    // A commit holds this thread until the products before it have left the queue, so the commits that a tile owes
    // follow the first products of the next, as in conv_tc.cu; before the thread waits it pays them.
    int owed_unit = -1, owed_acc = -1;
    auto flush = [&]() {
      if (leader) {
        if (owed_unit >= 0) mma_commit(&bar_empty[owed_unit]);
        if (owed_acc >= 0) mma_commit(&bar_acc_full[owed_acc]);
      }
      owed_unit = owed_acc = -1;
    };
    auto ensure = [&](uint64_t* bar, uint32_t parity, int code) -> bool {
      if (mbar_test(bar, parity)) return true;
      flush();
      return mbar_wait(bar, parity, &abort_flag, code);
    };
    pdl_wait();
    for (int tile = blockIdx.x; live && tile < p.num_tiles; tile += step) {
      if (!ensure(&bar_acc_empty[acc], acc_phase ^ 1, 2)) break;
      const uint32_t d = tmem_base + (uint32_t)(acc * ACC_COLS);
#pragma unroll
      for (int u = 0; u < UNITS; ++u) {
        if (!ensure(&bar_full[unit], phase, 3)) { live = false; break; }
        tc_fence_after();
        const uint32_t al = a_lo + (uint32_t)(unit * (UNIT / 16));
#pragma unroll
        for (int g = 0; g < G; ++g) {
          int issued = 0;
#pragma unroll
          for (int i = 0; i < Sh::PRODUCTS; ++i) {
            const Product q = S == 1 ? product1(i) : product2(i);
            if (!PAIRS && (q.ix & 1) != u) continue;   // a tap of the other plane
            const int at = PAIRS ? ((q.ix + 1) >> 1) * ROW + ((q.ix + 1) & 1) * P : (q.ix >> 1) * P;
            mma_i8_if(leader, d + (uint32_t)(g * Sh::COLS + q.col), al + (uint32_t)((q.iy * LINE + at + g * 32) >> 4), a_hi,
                      w_lo + (uint32_t)((g * Sh::BLOCKS + q.first) * 64), w_hi, umma_idesc_i8(q.n), u == 0 && issued == 0 ? 0u : 1u);
            if (g == 0 && issued == 2) flush();
            ++issued;
          }
        }
        owed_unit = unit;
        if (u == UNITS - 1) owed_acc = acc;
        if (++unit == p.units) { unit = 0; phase ^= 1; }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (live) flush();
  } else if (warp < Sh::IO_WARP) {
    // ---------------------------------------------------------------- requantisation
    // A warp has the 32 rows of its TMEM lanes, and of their output pixels (32 columns a channel group) one or two: there
    // are four warps for each quarter of the lanes with stride 1, two with stride 2.
    const int quarter = warp & 3, sub = (warp - 2) >> 2;
    constexpr int CHUNKS = S == 1 && G == 2 ? 2 : 1;
    const int g = G == 2 ? sub >> (S == 1 ? 1 : 0) : 0, first = S == 1 ? (G == 2 ? 2 * (sub & 1) : sub) : 0;
    const bool works = !(G == 1 && S == 2 && sub == 1);
    const int bx = lane & 7, by = quarter * 4 + (lane >> 3);
    const int img = p.per_tile > 1 ? fdiv(by, p.fd_pitch) : 0, ly = by - img * p.pitch_y;
    const FastQ fq = {p.lo, p.hi, FORM == OTHER ? p.lo2 : 0, FORM == OTHER ? p.hi2 : 0};
    const int mul = p.mul;
    const uint32_t base = smem_u32(out);
    int k = 0;
    pdl_wait();
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += step, ++k) {
      int x0, y0, n0;
      origin(tile, &x0, &y0, &n0);
      const int acc = k & 1;
      const uint32_t use = (uint32_t)(k >> 1) & 1u;
      // (a warp whose 32 rows all lie outside the images has nothing to write)
      const bool any = __any_sync(0xffffffffu, x0 + bx < p.rows_x && ly < p.band && y0 + ly < p.rows_y && img < p.per_tile && n0 + img < p.images);
      if (!mbar_wait(&bar_out_free[acc], has_operand ? use : use ^ 1u, &abort_flag, 5)) break;
      if (!mbar_wait(&bar_acc_full[acc], use, &abort_flag, 4)) break;
      tc_fence_after();
      if (works && any) {
        const uint32_t t0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * ACC_COLS + g * Sh::COLS + first * 32);
#pragma unroll
        for (int c = 0; c < CHUNKS; ++c) {
          int32_t v[32];
          tmem_ld32(t0 + (uint32_t)(c * 32), v);
          const int q = first + c, oy = S == 1 ? q >> 1 : 0, ox = S == 1 ? (q ^ (q >> 1)) & 1 : 0;   // (0,0), (0,1), (1,1), (1,0)
          // the output tile lies as the store takes it: lines of pixels, swizzled
          const uint32_t lin = base + (uint32_t)(acc * OUT_BYTES + (by * Sh::OUT + oy) * OUT_LINE + (bx * Sh::OUT + ox) * P + g * 32);
          const uint32_t key = ((lin >> 7) & p.out_mask) << 4, at0 = lin ^ key, at1 = (lin + 16u) ^ key;
          uint4 a, b;
          const uint4 none = make_uint4(0, 0, 0, 0);
          if (FORM == OTHER) {
            if (p.kind < 0) {
              const int x = (x0 + bx) * Sh::OUT + ox, y = (y0 + ly) * Sh::OUT + oy;
              const bool inside = img < p.per_tile && ly < p.band && n0 + img < p.images && x < p.out_w && y < p.out_h;
              const size_t at = (((size_t)(n0 + img) * p.out_h + y) * p.out_w + x) * p.C + c0 + g * 32;
#pragma unroll
              for (int h = 0; h < 2; ++h) {   // (16 columns at a time: with a tensor operand 32 do not fit the registers)
                int32_t u[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) u[j] = v[16 * h + j];
                if (inside) apply_chain<16>(p.chain, u, at + 16 * h, c0 + g * 32 + 16 * h);
                (h ? b : a) = make_uint4(pack4(u[0], u[1], u[2], u[3]), pack4(u[4], u[5], u[6], u[7]), pack4(u[8], u[9], u[10], u[11]), pack4(u[12], u[13], u[14], u[15]));
              }
            } else {
              const int4* bp = reinterpret_cast<const int4*>(bias_s + g * 32);
              if (p.wide) {   // (two loops: a choice an element costs both)
                const int am = p.add * mul;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const int4 b4 = bp[j];
                  const int32_t bj[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                  for (int i = 0; i < 4; ++i) v[4 * j + i] = min(max(v[4 * j + i] + bj[i], p.pre_lo), p.pre_hi) * mul + am;
                }
              } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                  const int4 b4 = bp[j];
                  const int32_t bj[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
                  for (int i = 0; i < 4; ++i) v[4 * j + i] = v[4 * j + i] * mul + bj[i];
                }
              }
              uint4 r0 = none, r1 = none;
              if (has_operand) {
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r0.x), "=r"(r0.y), "=r"(r0.z), "=r"(r0.w) : "r"(at0));
                asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r1.x), "=r"(r1.y), "=r"(r1.z), "=r"(r1.w) : "r"(at1));
              }
              if (p.kind == 0) fast_requant<0, 0>(fq, v, none, none, &a, &b);
              else if (p.kind == 2) fast_requant<0, 2>(fq, v, r0, r1, &a, &b);
              else fast_requant<0, 3>(fq, v, r0, r1, &a, &b);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = v[j] * mul + bias[j];
            fast_requant<FORM == PACKED_RELU, 0>(fq, v, none, none, &a, &b);
          }
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at0), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at1), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w) : "memory");
        }
      }
      tc_fence_before();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&bar_acc_empty[acc]);
        mbar_arrive(&bar_staged[acc]);
      }
    }
  } else {
    // ---------------------------------------------------------------- output
    const bool leader = elect_one();
    int k = 0;
    auto hand_back = [&](int buf, int tile) {   // buffer `buf`, to the requantisation of tile `tile`
      if (FORM == OTHER && has_operand) {
        if (tile >= p.num_tiles) return;
        int x0, y0, n0;
        origin(tile, &x0, &y0, &n0);
        const int count = min(p.per_tile, p.images - n0);
        mbar_expect_tx(&bar_out_free[buf], (uint32_t)(count * p.out_box_bytes));
        for (int i = 0; i < count; ++i)
          tma_load_4d(out + buf * OUT_BYTES + (size_t)(i * p.pitch_y * Sh::OUT) * OUT_LINE, &tmap_r, &bar_out_free[buf], c0,
                      p.out_pairs ? x0 * Sh::OUT / 2 : x0 * Sh::OUT, y0 * Sh::OUT, n0 + i);
      } else {
        mbar_arrive(&bar_out_free[buf]);
      }
    };
    pdl_wait();
    if (has_operand && leader) { hand_back(0, blockIdx.x); hand_back(1, blockIdx.x + step); }
    for (int tile = blockIdx.x; tile < p.num_tiles; tile += step, ++k) {
      int x0, y0, n0;
      origin(tile, &x0, &y0, &n0);
      const int buf = k & 1;
      if (!mbar_wait(&bar_staged[buf], (uint32_t)(k >> 1) & 1u, &abort_flag, 6)) break;
      if (leader) {
        const uint8_t* src = out + buf * OUT_BYTES;
        for (int i = 0; i < p.per_tile && n0 + i < p.images; ++i)
          tma_store_4d(&tmap_y, src + (size_t)(i * p.pitch_y * Sh::OUT) * OUT_LINE, c0, p.out_pairs ? x0 * Sh::OUT / 2 : x0 * Sh::OUT, y0 * Sh::OUT, n0 + i);
        tma_store_commit();
        tma_store_wait_read();
        hand_back(buf, tile + 2 * step);
      }
      __syncwarp();
    }
  }

  __syncwarp();
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);   // copies that may still be in flight land before shared memory is released
    if (lane == 0 && p.status) atomicOr(p.status, 0x800 | abort_flag);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

CUresult encode(EncodeTiledFn enc, CUtensorMap* map, const void* base, int64_t n, int64_t h, int64_t w, int64_t c, int box_c, int box_w,
                int box_h, int box_n, int step_w, CUtensorMapL2promotion promo) {
  cuuint64_t dims[4] = {(cuuint64_t)c, (cuuint64_t)w, (cuuint64_t)h, (cuuint64_t)n};
  cuuint64_t strides[3] = {(cuuint64_t)c, (cuuint64_t)(w * c), (cuuint64_t)(h * w * c)};
  cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)box_w, (cuuint32_t)box_h, (cuuint32_t)box_n};
  cuuint32_t estr[4] = {1, (cuuint32_t)step_w, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             box_c == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (box_c == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B), promo, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

template <int S, int G, int PAIRS, int FORM>
int launch(const CUtensorMap& tx, const CUtensorMap& ty, const CUtensorMap& tr, const DwParams& p, int grid, int smem, int dev, cudaStream_t stream) {
  static bool attr_set_dev[64] = {false};
  bool& attr_set = attr_set_dev[dev & 63];
  if (!attr_set) {
    if (check_cuda(cudaFuncSetAttribute(conv_dw_kernel<S, G, PAIRS, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX), "cudaFuncSetAttribute(conv_dw_kernel)"))
      return CVMK_ERR_CUDA;
    attr_set = true;
  }
  launch_pdl(conv_dw_kernel<S, G, PAIRS, FORM>, dim3((unsigned)grid), dim3(Shape<S>::THREADS), smem, stream, tx, ty, tr, p);
  return check_cuda(cudaGetLastError(), "conv_dw_kernel launch");
}

typedef int (*LaunchFn)(const CUtensorMap&, const CUtensorMap&, const CUtensorMap&, const DwParams&, int, int, int, cudaStream_t);
template <int S, int G, int PAIRS>
LaunchFn of_form(int form) { return form == OTHER ? launch<S, G, PAIRS, OTHER> : (form == PACKED ? launch<S, G, PAIRS, PACKED> : launch<S, G, PAIRS, PACKED_RELU>); }
template <int S>
LaunchFn of_shape(int groups, bool pairs, int form) {
  if (groups == 1) return pairs ? of_form<S, 1, 1>(form) : of_form<S, 1, 0>(form);
  return pairs ? of_form<S, 2, 1>(form) : of_form<S, 2, 0>(form);
}

// The shape and the tiles of a layer, or false when it is not one for this kernel.
bool plan_tiles(const cvmk_conv_direct_desc& d, DwParams* params, int* sm_count) {
  const int S = d.stride_h;
  if (d.C % 32 != 0 || d.x_dtype != CVMK_I8 || d.y_dtype != CVMK_I8 || d.KH != 3 || d.KW != 3 || d.dil_h != 1 || d.dil_w != 1 ||
      (S != 1 && S != 2) || d.stride_w != S || d.pad_h > 1 || d.pad_w > 1 || d.N < 1 || d.OH < 1 || d.OW < 1)
    return false;
  const int P = d.C % 64 == 0 ? 64 : 32, out = S == 1 ? 2 : 1;
  int dev = 0, sms = 148;   // (without a device, of the part this library is built for)
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  else cudaGetLastError();
  DwParams& p = *params;
  memset(&p, 0, sizeof(p));
  p.C = d.C; p.images = d.N;
  p.pad_h = d.pad_h; p.pad_w = d.pad_w;
  p.rows_x = (d.OW + out - 1) / out;
  p.rows_y = (d.OH + out - 1) / out;
  p.c_tiles = d.C / P;
  if (p.c_tiles > sms) return false;
  // A tile holds TILE_Y operand lines of one image, or as many of several as are stacked in it, each with one line more
  // (what its last taps read), rounded up so that its part of the output tile starts on a multiple of 1024 bytes.  Images
  // of at most seven lines are stacked whole; higher ones in bands of fewer lines where that takes fewer rounds of
  // tiles (a band's last line is loaded again with the next, 16 % more input at seven lines).  Stride 1, in a chain of such
  // layers, whole images -> bands: 256 channels at 16 x 16, 256 images 12.4 -> 10.0 us; 128 at 38 x 38, 128 images 24.3 ->
  // 13.5 (on the CUDA cores before), 256 at 36 x 36, 128 images 39.5 -> 22.1 (likewise).
  const int whole = std::max(1, 1024 / (8 * out * out * P));
  p.tiles_x = (p.rows_x + TILE_X - 1) / TILE_X;
  const int64_t grid_max = sms / p.c_tiles * p.c_tiles;
  int64_t tiles = 0, rounds = 0, of_images = 0;
  for (int band = std::min(p.rows_y, TILE_Y); band >= 1; --band) {
    int pitch = (band + 1 + whole - 1) / whole * whole, images = TILE_Y / pitch;
    if (images < 2) { pitch = TILE_Y; images = 1; }
    if (images == 1 && band < std::min(p.rows_y, TILE_Y)) continue;
    const int bands = (p.rows_y + band - 1) / band;
    const int64_t t = (int64_t)p.tiles_x * bands * ((d.N + images - 1) / images) * p.c_tiles, r = (t + grid_max - 1) / grid_max;
    if (!tiles) of_images = t;
    else if (r >= rounds) continue;
    tiles = t; rounds = r;
    p.band = band; p.pitch_y = pitch; p.per_tile = images; p.tiles_y = bands;
  }
  if (tiles > INT32_MAX / 2) return false;
  // One box of pixel pairs has half the rows of twice the bytes, and a store of pairs too, where the two pixels lie
  // side by side (C channels a tile).
  p.pairs = d.C == P && d.W % 2 == 0 && d.pad_w == 1;
  p.out_pairs = d.C == P && d.OW % 2 == 0;
  // The CUDA-core kernel stays the better one where whole images do not give every SM a tile, and where five eighths of their
  // rows lie outside the images.  Device time with the line at 0, 96, 150, 296 and 592 tiles: MobileNet, one image 123, 99,
  // 99, 99, 99 us; 20 images 182, 172, 170, 170, 176; 256 images 692 each (of 828 with none); SSD-512 on 3 images 328, 328,
  // 329, 339, 350; on 8 images 450, 449, 440, 444, 455.  Pairs of pixels are worth it from half as many tiles on (SSD-512, one
  // image: 293 -> 276 us).  By the share of rows inside the images, a layer on the CUDA cores -> here: 0.47, 256 channels at 15 x
  // 20, 256 images 23.8 -> 14.9 us; 0.42, 256 at 18 x 18, 128 images 14.0 -> 10.3; 0.39, 128 at 19 x 19, 128 images 10.0 -> 8.5,
  // but 40 images of 20 x 20 5.4 -> 5.9, so the rows inside have to fill tiles for half of the SMs; 0.375, 512 at 8 x 8, 256
  // images 9.6 -> 10.0, 1024 at 7 x 7 16.6 -> 15.1.
  const int64_t least = p.pairs ? sms / 2 : sms, used = (int64_t)p.rows_x * p.rows_y * d.N * p.c_tiles;
  if (of_images < least || 2 * used < least * TILE_X * TILE_Y || 8 * used <= 3 * tiles * TILE_X * TILE_Y) return false;
  p.num_tiles = (int)tiles;
  *sm_count = sms;
  return true;
}

}  // namespace

int launch_conv_dw(const cvmk_conv_direct_desc& d, const DevChain& chain, cudaStream_t stream) {
  DwParams p;
  int sms = 0;
  if (!plan_tiles(d, &p, &sms)) return -1;
  const int S = d.stride_h, G = d.C % 64 == 0 ? 2 : 1, P = 32 * G, out = S == 1 ? 2 : 1;
  const bool pairs = p.pairs, out_pairs = p.out_pairs;
  p.w = d.w; p.status = d.status;
  p.fd_c = make_fastdiv(p.c_tiles); p.fd_x = make_fastdiv(p.tiles_x); p.fd_y = make_fastdiv(p.tiles_y); p.fd_pitch = make_fastdiv(p.pitch_y);
  const int box_h = p.per_tile > 1 ? 2 * p.pitch_y : std::min(BOX_H, 2 * (p.band + 1));
  const int row = pairs ? 2 * P : P, box_w = pairs ? TILE_X + 2 : TILE_X + 1;
  p.box_bytes = box_w * row * box_h * p.per_tile;
  const int unit_bytes = (box_w * row * BOX_H + 1023) & ~1023;   // (rows of a tile outside its images read the rest of a unit)
  const int w_bytes = G * (S == 1 ? NUM_BLOCKS1 : NUM_BLOCKS2) * 1024;
  const int out_bytes = TILE_X * TILE_Y * out * out * P;
  p.units = std::min(MAX_UNITS, (SMEM_MAX - 1024 - w_bytes - 2 * out_bytes) / unit_bytes);
  p.out_mask = (uint32_t)((out_pairs ? 2 * P : P) / 16 - 1);
  const int first = chain.n > 0 && chain.s[0].op == K_ADD_C;
  PackedChain pc;
  memset(&pc, 0, sizeof(pc));
  bool packed = pack_chain(chain, first, d.acc_bound, &pc) && (!pc.kind || ((uintptr_t)chain.s[pc.step].ptr & 15) == 0);
  if (chain.n - first == 1 && chain.s[first].op == K_CLIP && chain.s[first].a >= -32767 && chain.s[first].b <= 32767) {   // a shift by 0
    packed = true;
    pc.wide = 1; pc.mul = 1 << 16;
    pc.pre_lo = pc.lo = chain.s[first].a;
    pc.pre_hi = pc.hi = chain.s[first].b;
  }
  p.bias = first ? reinterpret_cast<const int32_t*>(chain.s[0].ptr) : nullptr;
  p.mul = pc.mul; p.add = pc.add;
  p.lo = both_halves(pc.lo); p.hi = both_halves(pc.hi);
  p.kind = packed ? pc.kind : -1;
  p.wide = pc.wide; p.pre_lo = pc.pre_lo; p.pre_hi = pc.pre_hi;
  p.lo2 = both_halves(pc.lo2); p.hi2 = both_halves(pc.hi2);
  p.bias_static = d.bias_static;
  p.out_w = d.OW; p.out_h = d.OH;
  p.chain = chain;
  // (206 KB and more: beside a CTA of this kernel, which has all TMEM columns of its SM, no CTA of conv_tc_kernel starts)
  const int smem = std::max(1024 + w_bytes + p.units * unit_bytes + 2 * out_bytes, 206 * 1024);

  static EncodeTiledFn enc = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    const cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    return e == cudaSuccess && q == cudaDriverEntryPointSuccess ? (EncodeTiledFn)fn : (EncodeTiledFn) nullptr;
  }();
  if (!enc) { set_error("conv_dw: cuTensorMapEncodeTiled not found"); return CVMK_ERR_CUDA; }
  CUtensorMap tx, ty, tr;
  const int f = pairs ? 2 : 1, fo = out_pairs ? 2 : 1, out_h = p.band * out;
  p.out_box_bytes = TILE_X * out * P * out_h;
  auto encode_out = [&](CUtensorMap* map, const void* base, CUtensorMapL2promotion promo) {
    return encode(enc, map, base, d.N, d.OH, d.OW / fo, d.C * fo, P * fo, TILE_X * out / fo, out_h, 1, 1, promo);
  };
  if (encode(enc, &tx, d.x, d.N, d.H, d.W / f, d.C * f, row, pairs ? box_w : 2 * box_w, box_h, p.per_tile, pairs ? 1 : 2, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) != CUDA_SUCCESS ||
      encode_out(&ty, d.y, CU_TENSOR_MAP_L2_PROMOTION_NONE) != CUDA_SUCCESS ||
      encode_out(&tr, p.kind > 0 ? chain.s[pc.step].ptr : d.y, CU_TENSOR_MAP_L2_PROMOTION_L2_128B) != CUDA_SUCCESS) {
    set_error("conv_dw: tensor map rejected");
    return CVMK_ERR_CUDA;
  }
  const int grid = std::min(p.num_tiles, sms) / p.c_tiles * p.c_tiles;
  const int form = p.kind != 0 || p.wide ? OTHER : (pc.lo == 0 ? PACKED_RELU : PACKED);
  int dev = 0;
  cudaGetDevice(&dev);
  const LaunchFn launch_form = S == 1 ? of_shape<1>(G, pairs, form) : of_shape<2>(G, pairs, form);
  return launch_form(tx, ty, tr, p, grid, smem, dev, stream);
}

bool conv_dw_takes(const cvmk_conv_direct_desc& d) {
  DwParams p;
  int sms = 0;
  return plan_tiles(d, &p, &sms);
}

}  // namespace cvmk
