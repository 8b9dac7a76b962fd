// conv2d (groups = 1) and dense for launches that do not fill the GPU.
//
// The persistent kernel of conv_tc.cu gives a CTA whole 128 x 256 tiles; a layer over one image has
// a handful of them, so most SMs idle while a few walk the whole reduction block by block (a 3 x 3
// layer over 512 channels is 36 dependent K blocks, 10 us), and its set-up and hand-overs between
// eight epilogue warps, staging buffers and the store engine cost several microseconds a launch.
// What bounds such a layer is latency, so here
//   - a tile is 128 x 64 or 128 x 32, one CTA each, and the reduction is cut over a CLUSTER of up
//     to eight CTAs, each of which multiplies its share of the (filter tap, channel block) units;
//   - the partial sums (int32: exact in any order) are exchanged through distributed shared memory:
//     every rank finishes a run of the tile's rows and receives that run from the others by bulk
//     copies (8 KB each; written element by element with st.shared::cluster the exchange ran at 16
//     bytes a clock, 1.2 us), so every CTA of the cluster has the same share of the
//     requantisation and of the stores, eight columns a thread;
//   - the weights of the first ring stages are requested BEFORE griddepcontrol.wait (they are model
//     parameters), i.e. while the previous layer still runs, and so is the bias.  How much shared memory
//     the ring takes is choose_small()'s decision (conv_tc.cu): all of a reduction in flight is worth
//     more than two layers side by side on an SM.
//
// Dense layers of at most 128 rows swap the operands: the weights are the 128-row operand (tile rows are
// output channels) and the activations the narrow one.  Such a layer is a stream of weights, and this
// way a tensor instruction takes 4 KB of it and shared memory holds little else.
//
// Measured (B200): ResNet-50, one image, 415 -> 192 us on the device; VGG-19, one image, 318 -> 164;
// ResNet-50, 13 images of 197 x 197, 539 -> 312; 25088 -> 4096 in a chain of layers whose weights come
// from HBM 22 us at 64 rows (4.6 TB/s), 32 at 128.
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>
#include "conv_small.cuh"

namespace cvmk {
namespace {

using namespace tc;

constexpr int THREADS = 320;   // warp 0: TMA, warp 1: MMA + TMEM, warps 2..9: epilogue

// (relaxed: the barriers' initialisation is released by its own fence, and the second use only says that
//  memory is no longer read; an arrive with release semantics waited half a microsecond for earlier stores)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// A value that is the same for the whole warp, out of a shuffle: the compiler then keeps it (and what is
// computed from it) in uniform registers, where TMA and tensor instructions take their operands.
__device__ __forceinline__ int uniform(int v) { return __shfl_sync(0xffffffffu, v, 0); }
// Copies `bytes` of this CTA's shared memory to `dst` (an address of the cluster window) and reports them
// to the mbarrier `bar` of the receiving CTA.
__device__ __forceinline__ void bulk_to_rank(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src),
               "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

// Packed requantisation of V columns of one row (see fast_requant): OC is a multiple of 32 and the
// output int8 on this path.  `res`: the tensor operand's bytes.
template <int V>
__device__ __forceinline__ void requant(const SmallConvParams& p, const int32_t* v, const int32_t* bias_s, const uint32_t* res, uint32_t* w) {
  const int4* bp = reinterpret_cast<const int4*>(bias_s);
  const int mul = p.f_mul;
  const int kind = (p.fast_variant & 7) >> 1;   // 0 no tensor step, 1 and 2 add, 3 subtract
  const bool wide = p.fast_variant >= 8;
#pragma unroll
  for (int q = 0; q < V / 4; ++q) {
    const int4 t = bp[q];
    int a = v[4 * q], b = v[4 * q + 1], c = v[4 * q + 2], d = v[4 * q + 3];
    if (wide) {
      const int lo = p.f_pre_lo, hi = p.f_pre_hi, am = p.f_add * mul;
      a = min(max(a + t.x, lo), hi) * mul + am;
      b = min(max(b + t.y, lo), hi) * mul + am;
      c = min(max(c + t.z, lo), hi) * mul + am;
      d = min(max(d + t.w, lo), hi) * mul + am;
    } else {
      a = a * mul + t.x;
      b = b * mul + t.y;
      c = c * mul + t.z;
      d = d * mul + t.w;
    }
    uint32_t h0 = __byte_perm((uint32_t)a, (uint32_t)b, 0x7632);
    uint32_t h1 = __byte_perm((uint32_t)c, (uint32_t)d, 0x7632);
    h0 = __vmaxs2(__vmins2(h0, p.fq.f_hi1), p.fq.f_lo1);
    h1 = __vmaxs2(__vmins2(h1, p.fq.f_hi1), p.fq.f_lo1);
    if (kind != 0) {
      const uint32_t ra = prmt(res[q], 0, 0x9180), rb = prmt(res[q], 0, 0xB3A2);
      h0 = kind == 3 ? __vsub2(h0, ra) : __vadd2(h0, ra);
      h1 = kind == 3 ? __vsub2(h1, rb) : __vadd2(h1, rb);
      h0 = __vmaxs2(__vmins2(h0, p.fq.f_hi2), p.fq.f_lo2);
      h1 = __vmaxs2(__vmins2(h1, p.fq.f_hi2), p.fq.f_lo2);
    }
    w[q] = __byte_perm(h0, h1, 0x6420);
  }
}

// Bias, chain step by step and store of 8 columns of one output row (OC is a multiple of 8: all of them
// or none exist).
template <int V>
__device__ __forceinline__ void by_steps(const SmallConvParams& p, const int32_t* v, int row, int col0, const int32_t* bias_s) {
  if (col0 >= p.oc) return;
  const size_t lin = (size_t)row * p.oc + col0;
  int32_t t[V];
#pragma unroll
  for (int j = 0; j < V; ++j) t[j] = v[j] + bias_s[j];   // zeros without a bias
  apply_chain<V>(p.chain, t, lin, col0, 1, nullptr, -1, p.first_step);
  if (p.y_dtype == CVMK_I8) {
    *reinterpret_cast<uint2*>(reinterpret_cast<int8_t*>(p.y) + lin) = make_uint2(pack4(t[0], t[1], t[2], t[3]), pack4(t[4], t[5], t[6], t[7]));
  } else {
    int4* dst = reinterpret_cast<int4*>(reinterpret_cast<int32_t*>(p.y) + lin);
    dst[0] = make_int4(t[0], t[1], t[2], t[3]);
    dst[1] = make_int4(t[4], t[5], t[6], t[7]);
  }
}

// Swapped operands: 8 output rows (row0 ..) of output channel `ch`.
__device__ __forceinline__ void store_swapped(const SmallConvParams& p, const int32_t* v, int ch, int row0, int32_t bias) {
  if (ch >= p.oc) return;
  int32_t t[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) t[j] = v[j] + bias;
  apply_chain<8>(p.chain, t, 0, ch, 0, nullptr, -1, p.first_step);   // (no tensor operands: see choose_small)
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (row0 + j < p.m_total) {
      const size_t lin = (size_t)(row0 + j) * p.oc + ch;
      if (p.y_dtype == CVMK_I8) reinterpret_cast<int8_t*>(p.y)[lin] = (int8_t)t[j];
      else reinterpret_cast<int32_t*>(p.y)[lin] = t[j];
    }
}

// The products of G units of NK K-steps each, in one straight line behind one predicate: 50 cycles an
// instruction (its own run time); with a loop in the elected lane's branch it was 80.
template <int G, int NK>
__device__ __forceinline__ void issue_steps(bool leader, uint32_t d, uint32_t al, uint32_t hi, uint32_t a_q, uint32_t unit_q, uint32_t idesc,
                                            uint32_t first) {
#pragma unroll
  for (int k = 0; k < G; ++k) {
    if (leader) mma_i8_k<NK>(d, al, hi, al + a_q, hi, idesc, k == 0 ? first : 1u);
    al += unit_q;
  }
}
template <int G>
__device__ __forceinline__ void issue_units(bool leader, int nk, uint32_t d, uint32_t al, uint32_t hi, uint32_t a_q, uint32_t unit_q,
                                            uint32_t idesc, uint32_t first) {
  if (nk == 4) issue_steps<G, 4>(leader, d, al, hi, a_q, unit_q, idesc, first);
  else if (nk == 2) issue_steps<G, 2>(leader, d, al, hi, a_q, unit_q, idesc, first);
  else issue_steps<G, 1>(leader, d, al, hi, a_q, unit_q, idesc, first);
}

// SWAP: operands swapped (dense).  Whether the reduction is cut stays a run-time choice: with an instance
// each, consecutive layers alternate between two kernels, and code the SM has not cached costs more than
// the branches (ResNet-50 batch 1: 213 against 205 us).
template <bool SWAP>
__global__ void __launch_bounds__(THREADS)
conv_small_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ SmallConvParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[SMALL_MAX_STAGES];
  __shared__ uint64_t bar_empty[SMALL_MAX_STAGES];
  __shared__ uint64_t bar_acc;
  __shared__ uint64_t bar_part;   // this CTA's rows of every rank's partial sums have landed
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ __align__(16) int32_t bias_s[BLOCK_M];

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int split = p.split;
  const bool SPLIT = split > 1;
  const int rank = uniform(SPLIT ? (int)cluster_rank() : 0);
  const int tile = (int)blockIdx.x >> p.split_log2;
  const int a_bytes = BLOCK_M * p.block_k, b_bytes = p.block_n * p.block_k;
  const int unit_bytes = a_bytes + b_bytes, stage_bytes = p.group * unit_bytes;   // a ring stage is `group` units: one barrier
  const int u0 = (rank * p.units) >> p.split_log2;
  const int mine = (((rank + 1) * p.units) >> p.split_log2) - u0;
  // tile origin
  const int mt = uniform(fdiv(tile, p.fd_n_tiles));
  const int n0 = (tile - mt * p.num_n_tiles) * p.block_n;
  const int m0 = mt * BLOCK_M;
  // a channel's bias a thread (warps 2 and on), if it is a parameter as early as its place is known
  static_assert(THREADS - 64 >= BLOCK_M, "a thread for every channel");
  const int ch0 = SWAP ? m0 : n0, channels = SWAP ? BLOCK_M : p.block_n, bias_at = (int)threadIdx.x - 64;
  int32_t bias = 0;
  auto load_bias = [&]() { if (p.bias && bias_at < channels && ch0 + bias_at < p.oc) bias = p.bias[ch0 + bias_at]; };
  if (warp >= 2 && p.bias_static) load_bias();
  int cw = 0, ch = 0, cn = 0;
  if (p.a_mode == 2) {
    const int r = uniform(fdiv(mt, p.fd_tiles_w));
    cw = (mt - r * p.tiles_w) * p.patch_w;
    cn = uniform(fdiv(r, p.fd_tiles_h));
    ch = (r - cn * p.tiles_h) * p.patch_h;
    cn *= p.patch_n;
  }
  int img = 0, base_w = 0, base_h = 0;
  if (p.a_mode == 1) {
    img = uniform(fdiv(m0, p.fd_ohow));
    const int rem = m0 - img * (p.oh * p.ow);
    const int oy = uniform(fdiv(rem, p.fd_ow));
    base_w = (rem - oy * p.ow) * p.stride_w - p.pad_w;
    base_h = oy * p.stride_h - p.pad_h;
  }

  touch_params(p);
  const bool leader = elect_one();
  const uint32_t ring = smem_u32(smem), full0 = smem_u32(&bar_full[0]);
  const int groups = (mine + p.group - 1) / p.group;
  // announces the bytes of group `g` in ring stage `s` and requests its weights (the elected lane)
  auto load_b = [&](int s, int g) {
    const int i0 = g * p.group, n = min(p.group, mine - i0);
    uint32_t sb = ring + (uint32_t)(s * stage_bytes + (SWAP ? 0 : a_bytes));
    const int wrow = SWAP ? m0 : n0;
    const uint32_t bar = full0 + 8u * (uint32_t)s;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((uint32_t)(n * unit_bytes)) : "memory");
    int col = (u0 + i0) * p.block_k;
    for (int k = 0; k < n; ++k, sb += (uint32_t)unit_bytes, col += p.block_k)
      asm volatile(
          "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
          " [%0], [%1, {%3, %4}], [%2];" ::"r"(sb), "l"(reinterpret_cast<uint64_t>(&tmap_b)), "r"(bar), "r"(col), "r"(wrow)
          : "memory");
  };
  if (warp == 0) {
    if (leader) {
      for (int s = 0; s < p.stages; ++s) {
        mbar_init(&bar_full[s], 1);
        mbar_init(&bar_empty[s], 1);
      }
      mbar_init(&bar_acc, 1);
      mbar_init(&bar_part, 1 + (THREADS - 64) / 32);
      abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (leader) asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap_a)) : "memory");
    // the weights of the first stages: parameters, no kernel writes them
    const int first = min(p.stages, groups);
    if (leader)
      for (int i = 0; i < first; ++i) load_b(i, i);
    __syncwarp();
  } else if (warp == 1) {
    // (the next kernel may start only once this CTA has its TMEM columns: it could take them, and then
    //  wait for this kernel's end)
    tmem_alloc(&tmem_slot, (uint32_t)p.tmem_cols);
    pdl_trigger();
  } else {
    if (!p.bias_static) {
      pdl_wait();
      load_bias();
    }
    // packed requantisation: (bias + rounding addend) pre-multiplied, see fast_requant()
    if (bias_at < channels) bias_s[bias_at] = (p.fast_variant >= 0 && p.fast_variant < 8) ? (int32_t)((uint32_t)(bias + p.f_add) * (uint32_t)p.f_mul) : bias;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = (uint32_t)uniform((int)tmem_slot);
  if (SPLIT) cluster_arrive();   // this CTA's barriers exist (waited for before anything is sent to it)

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA
    // Units in weight-matrix order: channel blocks, filter columns, filter rows.  The first lap of the
    // ring, whose stages are free, is a loop of the elected lane with nothing in it but the
    // load and three counters (about 20 cycles a load; with waits, divisions and the choice of
    // the load's kind in the loop it took 350, more than the loads themselves).
    const int tap = fdiv(u0, p.fd_cblocks);
    int cc = (u0 - tap * p.cblocks) * p.block_k;
    int fy = fdiv(tap, p.fd_kw), fx = tap - fy * p.kw;
    const int lap0 = min(p.stages * p.group, mine);
    auto step = [&]() {
      cc += p.block_k;
      if (cc >= p.c) { cc = 0; if (++fx == p.kw) { fx = 0; ++fy; } }
    };
    auto patch = [&](uint32_t sa, uint32_t bar) {
      asm volatile(
          "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
          " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(sa), "l"(reinterpret_cast<uint64_t>(&tmap_a)), "r"(bar), "r"(cc),
          "r"(cw + fx * p.dil_w - p.pad_w), "r"(ch + fy * p.dil_h - p.pad_h), "r"(cn)
          : "memory");
    };
    auto im2col = [&](uint32_t sa, uint32_t bar) {
      asm volatile(
          "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
          " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};" ::"r"(sa), "l"(reinterpret_cast<uint64_t>(&tmap_a)), "r"(bar), "r"(cc),
          "r"(base_w), "r"(base_h), "r"(img), "h"((uint16_t)(fx * p.dil_w)), "h"((uint16_t)(fy * p.dil_h))
          : "memory");
    };
    const int xrow = SWAP ? n0 : m0;
    const uint32_t xoff = SWAP ? (uint32_t)a_bytes : 0u;
    auto plain = [&](uint32_t sa, uint32_t bar) {
      asm volatile(
          "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
          " [%0], [%1, {%3, %4}], [%2];" ::"r"(sa + xoff), "l"(reinterpret_cast<uint64_t>(&tmap_a)), "r"(bar), "r"(cc), "r"(xrow)
          : "memory");
    };
    pdl_wait();
    if (leader) {
      uint32_t sa = ring, bar = full0;
      int k = 0;
      auto next = [&]() {
        sa += (uint32_t)unit_bytes;
        if (++k == p.group) { k = 0; bar += 8; }
        step();
      };
      if (p.a_mode == 2) for (int i = 0; i < lap0; ++i, next()) patch(sa, bar);
      else if (p.a_mode == 1) for (int i = 0; i < lap0; ++i, next()) im2col(sa, bar);
      else for (int i = 0; i < lap0; ++i, next()) plain(sa, bar);
      int stage = 0;
      uint32_t phase = 0;
      for (int g = p.stages; g < groups; ++g) {
        if (!mbar_wait(&bar_empty[stage], phase, &abort_flag, 1)) break;
        load_b(stage, g);
        sa = ring + (uint32_t)(stage * stage_bytes);
        bar = full0 + 8u * (uint32_t)stage;
        for (int i = g * p.group; i < min(mine, (g + 1) * p.group); ++i, sa += (uint32_t)unit_bytes, step()) {
          if (p.a_mode == 2) patch(sa, bar);
          else if (p.a_mode == 1) im2col(sa, bar);
          else plain(sa, bar);
        }
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA
    const uint32_t idesc = umma_idesc_i8(p.block_n);
    const uint64_t desc0 = umma_desc(ring, p.block_k);
    const uint32_t lo0 = (uint32_t)desc0, hi = (uint32_t)(desc0 >> 32);
    const uint32_t stage_q = (uint32_t)stage_bytes >> 4, unit_q = (uint32_t)unit_bytes >> 4, a_q = (uint32_t)a_bytes >> 4;
    const int nk = p.block_k / 32;
    int stage = 0;
    uint32_t phase = 0;
    // All lanes run this loop, in uniform registers, and one executes the instructions (alone in its
    // branch); no tcgen05 fence is needed between a TMA load's barrier and the products of its bytes.
    for (int g = 0, i = 0; g < groups; ++g) {
      if (!mbar_wait(&bar_full[stage], phase, &abort_flag, 3)) break;
      const int n = min(p.group, mine - i);
      const uint32_t al = lo0 + stage_q * (uint32_t)stage;
      if (n == 3) issue_units<3>(leader, nk, tmem_base, al, hi, a_q, unit_q, idesc, (uint32_t)i);
      else if (n == 2) issue_units<2>(leader, nk, tmem_base, al, hi, a_q, unit_q, idesc, (uint32_t)i);
      else issue_units<1>(leader, nk, tmem_base, al, hi, a_q, unit_q, idesc, (uint32_t)i);
      i += n;
      if (g + p.stages < groups) {   // (nobody waits for the last ones)
        if (leader) mma_commit(&bar_empty[stage]);
      }
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    if (leader) mma_commit(&bar_acc);
  }
  __syncwarp();

  // ------------------------------------------------------------------ epilogue
  // Warps 2..9: two per quarter of the TMEM lanes, each with half of the tile's columns.
  const int quarter = warp & 3, half = warp >= 6 ? 1 : 0;
  const int row_in_tile = quarter * 32 + lane;
  const int half_n = p.block_n >> 1, c_first = half * half_n;
  const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c_first;
  auto out_row = [&](int r) {                    // linear output row of tile row r; -1 outside the tensor
    if (p.a_mode != 2) return m0 + r < p.m_total ? m0 + r : -1;
    const int ow = cw + (r & (p.patch_w - 1)), q = r >> p.patch_w_log2;
    const int oh = ch + (q & (p.patch_h - 1)), on = cn + (q >> p.patch_h_log2);
    return (ow < p.ow && oh < p.oh && on * p.oh * p.ow < p.m_total) ? (on * p.oh + oh) * p.ow + ow : -1;
  };
  const bool with_res = p.res != nullptr;
  // The epilogue warps report their last TMEM load; the MMA warp then frees the columns while they go on.
  auto tmem_done = [&]() {
    tc_fence_before();
    asm volatile("bar.arrive 1, %0;" ::"r"(THREADS - 32) : "memory");
  };
  auto tmem_free = [&]() {
    asm volatile("bar.sync 1, %0;" ::"r"(THREADS - 32) : "memory");
    tc_fence_after();
    tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  };
  if (warp >= 2) pdl_wait();
  if (!SPLIT && SWAP) {
    if (warp >= 2) {
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar_acc, 0u, &abort_flag, 4));
      tc_fence_after();
      const int ch = m0 + row_in_tile;
      for (int c = 0; ok && c < half_n; c += 16) {
        int32_t v[16];
        tmem_ld16(tbase + (uint32_t)c, v);
        store_swapped(p, v, ch, n0 + c_first + c, bias_s[row_in_tile]);
        store_swapped(p, v + 8, ch, n0 + c_first + c + 8, bias_s[row_in_tile]);
      }
      tmem_done();
    } else if (warp == 1) {
      tmem_free();
    }
  } else if (!SPLIT) {
    if (warp >= 2) {
      const int row = out_row(row_in_tile);
      const bool packed = p.fast_variant >= 0;
      // Packed results are turned through the idle operand ring so that a store instruction covers whole
      // rows of the tile: each warp stores 16 rows of its quarter, `cpr` 16-byte chunks a row.
      const int cpr_log2 = p.block_n == 64 ? 2 : 1, chunk = lane & ((1 << cpr_log2) - 1);
      const int st0 = quarter * 32 + half * 16 + (lane >> cpr_log2), st1 = st0 + 8;   // (16 rows: two turns of 8 with 64 columns)
      const int out0 = out_row(st0), out1 = cpr_log2 == 2 ? out_row(st1) : -1;
      auto slot = [&](int r, int c) { return smem + r * p.block_n + ((c ^ ((r >> 1) & ((1 << cpr_log2) - 1))) << 4); };
      // the tensor operand travels while the products are computed
      uint32_t res[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (with_res && row >= 0 && n0 + c_first < p.oc) {
        const uint4* q = reinterpret_cast<const uint4*>(p.res + (size_t)row * p.oc + n0 + c_first);
        const uint4 t = q[0];
        res[0] = t.x; res[1] = t.y; res[2] = t.z; res[3] = t.w;
        if (half_n == 32) {
          const uint4 u = q[1];
          res[4] = u.x; res[5] = u.y; res[6] = u.z; res[7] = u.w;
        }
      }
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar_acc, 0u, &abort_flag, 4));
      tc_fence_after();
      if (ok) {
        int32_t v[32];
        if (half_n == 32) tmem_ld32(tbase, v);
        else {
          int32_t t[16];
          tmem_ld16(tbase, t);
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = t[j];
        }
        tmem_done();
        const int32_t* bp = bias_s + c_first;
        if (packed) {
          uint32_t w[8];
          requant<16>(p, v, bp, res, w);
          const int c0 = c_first >> 4;
          *reinterpret_cast<uint4*>(slot(row_in_tile, c0)) = make_uint4(w[0], w[1], w[2], w[3]);
          if (half_n == 32) {
            requant<16>(p, v + 16, bp + 16, res + 4, w + 4);
            *reinterpret_cast<uint4*>(slot(row_in_tile, c0 + 1)) = make_uint4(w[4], w[5], w[6], w[7]);
          }
          asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
          const int col = n0 + chunk * 16;
          if (col < p.oc) {
            int8_t* y = reinterpret_cast<int8_t*>(p.y) + col;
            if (out0 >= 0) *reinterpret_cast<uint4*>(y + (size_t)out0 * p.oc) = *reinterpret_cast<const uint4*>(slot(st0, chunk));
            if (out1 >= 0) *reinterpret_cast<uint4*>(y + (size_t)out1 * p.oc) = *reinterpret_cast<const uint4*>(slot(st1, chunk));
          }
        } else if (row >= 0) {
          by_steps<8>(p, v, row, n0 + c_first, bp);
          by_steps<8>(p, v + 8, row, n0 + c_first + 8, bp + 8);
          if (half_n == 32) {
            by_steps<8>(p, v + 16, row, n0 + c_first + 16, bp + 16);
            by_steps<8>(p, v + 24, row, n0 + c_first + 24, bp + 24);
          }
        }
      } else {
        tmem_done();
      }
    } else if (warp == 1) {
      tmem_free();
    }
  } else {
    // The tile's rows up to the last one inside the tensor are dealt to the ranks in runs of rows_per.
    // Each CTA writes its partial sums of all rows into its (now idle) operand ring and sends every
    // other rank its run; `part` of the receiver holds one block of its rows from each of them.  16-byte
    // chunks of a row are XORed with the low bits of its number in the run (lanes hold different rows).
    // All index arithmetic (divisions among it) is done before the waits it would otherwise follow.
    int rows = min(BLOCK_M, (SWAP ? p.oc : p.m_total) - m0);
    if (p.a_mode == 2) {
      const int images = p.images - cn;
      rows = images >= p.patch_n ? BLOCK_M : images << (p.patch_w_log2 + p.patch_h_log2);
    }
    const int rows_per = (rows + split - 1) >> p.split_log2;
    const int row_bytes = p.block_n * 4;
    uint8_t* part = smem + small_ring_bytes(p.block_k, p.block_n, p.stages * p.group, split);
    const int mine_rows = max(0, min(rows_per, rows - rank * rows_per));
    if (warp == 1 && leader) mbar_expect_tx(&bar_part, (uint32_t)((split - 1) * mine_rows * row_bytes));
    if (warp >= 2) {
      const int rl = row_in_tile % rows_per;
      uint8_t* const stage_row = smem + row_in_tile * row_bytes;
      // the runs (one to five) that the quarter's rows belong to
      const int r_end = min(rows, quarter * 32 + 32), dest0 = (quarter * 32) / rows_per;
      // this CTA's rows: eight columns a thread and turn
      const int t = (int)threadIdx.x - 64, per_row_log2 = 31 - __clz(p.block_n >> 3), per_row = 1 << per_row_log2;
      const int jobs = mine_rows << per_row_log2;
      // (swapped operands: rows are output channels, so neighbouring threads take neighbouring rows)
      int job_rl = t >> per_row_log2, job_q = t & (per_row - 1);
      if (SWAP && mine_rows > 0) { job_q = t / mine_rows; job_rl = t - job_q * mine_rows; }
      int row = -1;
      uint32_t res[2] = {0, 0};
      auto job_row = [&]() {
        const int col = n0 + job_q * 8;
        if (SWAP) { row = m0 + rank * rows_per + job_rl; return; }
        row = out_row(rank * rows_per + job_rl);
        if (col >= p.oc) row = -1;
        if (!with_res || row < 0) return;
        const uint2 q = *reinterpret_cast<const uint2*>(p.res + (size_t)row * p.oc + col);
        res[0] = q.x; res[1] = q.y;
      };
      if (t < jobs) job_row();
      cluster_wait();   // every CTA of the cluster has started and initialised its barriers
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar_acc, 0u, &abort_flag, 4));
      tc_fence_after();
      if (ok) {
        for (int c = 0; c < half_n; c += 16) {
          int32_t v[16];
          tmem_ld16(tbase + (uint32_t)c, v);
          if (row_in_tile < rows) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
              *reinterpret_cast<int4*>(stage_row + (((((c_first + c) >> 2) + j) ^ (rl & 7)) << 4)) = make_int4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
        fence_async_smem();
      }
      tmem_done();
      // both warps of a quarter have written its 32 rows: one of them sends the runs they belong to
      asm volatile("bar.sync %0, 64;" ::"r"(2 + quarter) : "memory");
      if (lane == 0) mbar_arrive(&bar_part);   // (this CTA's own run is read where it lies)
      if (half == 0 && ok && leader) {
        int r = quarter * 32;
        for (int dest = dest0; r < r_end; ++dest) {
          const int run = min(r_end, (dest + 1) * rows_per) - r;
          const int theirs = min(rows_per, rows - dest * rows_per), block = rank - (rank > dest ? 1 : 0);
          if (dest != rank)
            bulk_to_rank(map_rank(smem_u32(part) + (uint32_t)((block * theirs + r - dest * rows_per) * row_bytes), (uint32_t)dest),
                         smem_u32(smem + r * row_bytes), (uint32_t)(run * row_bytes), map_rank(smem_u32(&bar_part), (uint32_t)dest));
          r += run;
        }
      }
      __syncwarp();
      const bool landed = mbar_wait(&bar_part, 0u, &abort_flag, 5);
      __syncwarp();
      cluster_arrive();   // what was sent here has left its senders' memory
      if (landed) {
        for (int k = t; k < jobs; k += THREADS - 64) {
          if (k != t) {
            job_rl = k >> per_row_log2; job_q = k & (per_row - 1);
            if (SWAP) { job_q = k / mine_rows; job_rl = k - job_q * mine_rows; }
            job_row();
          }
          if (row < 0) continue;
          const int o0 = ((2 * job_q) ^ (job_rl & 7)) << 4, o1 = ((2 * job_q + 1) ^ (job_rl & 7)) << 4;
          const uint8_t* src = smem + (rank * rows_per + job_rl) * row_bytes;
          int4 a = *reinterpret_cast<const int4*>(src + o0), b = *reinterpret_cast<const int4*>(src + o1);
          int32_t v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
          src = part + job_rl * row_bytes;
#pragma unroll 7
          for (int s = 1; s < split; ++s, src += mine_rows * row_bytes) {
            a = *reinterpret_cast<const int4*>(src + o0);
            b = *reinterpret_cast<const int4*>(src + o1);
            v[0] += a.x; v[1] += a.y; v[2] += a.z; v[3] += a.w;
            v[4] += b.x; v[5] += b.y; v[6] += b.z; v[7] += b.w;
          }
          if (SWAP) {
            store_swapped(p, v, row, n0 + job_q * 8, bias_s[rank * rows_per + job_rl]);
          } else if (p.fast_variant >= 0) {
            uint32_t w[2];
            requant<8>(p, v, bias_s + job_q * 8, res, w);
            *reinterpret_cast<uint2*>(reinterpret_cast<int8_t*>(p.y) + (size_t)row * p.oc + n0 + job_q * 8) = make_uint2(w[0], w[1]);
          } else {
            by_steps<8>(p, v, row, n0 + job_q * 8, bias_s + job_q * 8);
          }
        }
      }
    } else {
      cluster_wait();
      cluster_arrive();
      if (warp == 1) tmem_free();
    }
    __syncwarp();
    cluster_wait();   // nobody still reads this CTA's memory
  }

  // Every warp leaves on its own; the TMEM columns have gone back already (tmem_free above).
  __syncwarp();
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);   // copies in flight land before shared memory is released
    if (lane == 0 && p.status) atomicOr(p.status, 0x200 | abort_flag);
  }
}

}  // namespace

int launch_conv_small(const CUtensorMap& a, const CUtensorMap& b, const SmallConvParams& p, int grid, int smem, cudaStream_t stream) {
  static void (*const kernels[2])(CUtensorMap, CUtensorMap, SmallConvParams) = {conv_small_kernel<false>, conv_small_kernel<true>};
  static bool attr_of_device[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_of_device[dev & 63]) {
    for (auto k : kernels) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
      if (check_cuda(e, "cudaFuncSetAttribute(conv_small_kernel)")) return CVMK_ERR_CUDA;
    }
    attr_of_device[dev & 63] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (!dev_env("CVM_B200_NO_PDL")) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (p.split > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)p.split;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = (unsigned)n;
  return check_cuda(cudaLaunchKernelEx(&cfg, kernels[p.swap ? 1 : 0], a, b, p), "conv_small_kernel launch");
}

}  // namespace cvmk
