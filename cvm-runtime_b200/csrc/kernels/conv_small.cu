// conv2d (groups = 1) and dense for launches that do not fill the GPU.
//
// The persistent kernel of conv_tc.cu gives a CTA whole 128 x 256 tiles; a layer over one image has
// a handful of them, so most SMs idle while a few walk the whole reduction block by block (a 3 x 3
// layer over 512 channels is 36 dependent K blocks, 10 us), and its set-up and hand-overs between
// eight epilogue warps, staging buffers and the store engine cost several microseconds a launch.
// What bounds such a layer is latency, so here
//   - a tile is 128 x 64 (or 32 / 128), one CTA each, and the reduction is cut over a CLUSTER of up
//     to eight CTAs, each of which multiplies its share of the (filter tap, channel block) units;
//   - the partial sums (int32: exact in any order) are exchanged through distributed shared memory:
//     rank r of the cluster finishes rows [r * 128 / split, ...) of the tile, so every CTA of the
//     cluster has the same share of the requantisation and of the stores;
//   - the weights of the first ring stages are requested BEFORE griddepcontrol.wait (they are model
//     parameters), i.e. while the previous layer still runs, and so is the bias; a CTA takes at most
//     half of an SM's shared memory so that two layers fit beside each other;
//   - results are stored straight from registers.
#include <cuda.h>
#include <cuda_runtime.h>
#include <string.h>
#include "conv_small.cuh"

namespace cvmk {
namespace {

using namespace tc;

constexpr int THREADS = 192;   // warp 0: TMA, warp 1: MMA + TMEM, warps 2..5: epilogue

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The address, in the cluster's shared window, of `addr` in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
  return d;
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, int a, int b, int c, int d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

template <int RELU1, int KIND>
__device__ __forceinline__ void requant_case(const SmallConvParams& p, const int32_t (&v)[32], const uint4& r0, const uint4& r1,
                                             uint4* a, uint4* b) {
  fast_requant<RELU1, KIND>(p.fq, v, r0, r1, a, b);
}

// Bias, chain and store of 32 columns of one output row.  `row` is a linear output row inside the
// tensor; columns past OC (a multiple of 8) are left alone.  r0, r1: the tensor operand's 32 bytes.
__device__ __forceinline__ void finish_chunk(const SmallConvParams& p, int32_t (&v)[32], int row, int col0, const int32_t* bias_s,
                                             const uint4& r0, const uint4& r1) {
  const size_t lin = (size_t)row * p.oc + col0;
  const int4* bp = reinterpret_cast<const int4*>(bias_s);
  if (p.fast_variant >= 0) {   // OC is a multiple of 32 and the output int8 on this path
    if (p.fast_variant >= 8) {
      const int lo = p.f_pre_lo, hi = p.f_pre_hi, mul = p.f_mul, am = p.f_add * p.f_mul;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int4 t = bp[j];
        v[4 * j] = min(max(v[4 * j] + t.x, lo), hi) * mul + am;
        v[4 * j + 1] = min(max(v[4 * j + 1] + t.y, lo), hi) * mul + am;
        v[4 * j + 2] = min(max(v[4 * j + 2] + t.z, lo), hi) * mul + am;
        v[4 * j + 3] = min(max(v[4 * j + 3] + t.w, lo), hi) * mul + am;
      }
    } else {
      const int mul = p.f_mul;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int4 t = bp[j];
        v[4 * j] = v[4 * j] * mul + t.x;
        v[4 * j + 1] = v[4 * j + 1] * mul + t.y;
        v[4 * j + 2] = v[4 * j + 2] * mul + t.z;
        v[4 * j + 3] = v[4 * j + 3] * mul + t.w;
      }
    }
    uint4 a, b;
    switch (p.fast_variant & 7) {
      case 0: requant_case<0, 0>(p, v, r0, r1, &a, &b); break;
      case 1: requant_case<1, 0>(p, v, r0, r1, &a, &b); break;
      case 2: requant_case<0, 1>(p, v, r0, r1, &a, &b); break;
      case 3: requant_case<1, 1>(p, v, r0, r1, &a, &b); break;
      case 4: requant_case<0, 2>(p, v, r0, r1, &a, &b); break;
      case 5: requant_case<1, 2>(p, v, r0, r1, &a, &b); break;
      case 6: requant_case<0, 3>(p, v, r0, r1, &a, &b); break;
      default: requant_case<1, 3>(p, v, r0, r1, &a, &b); break;
    }
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<int8_t*>(p.y) + lin);
    dst[0] = a;
    dst[1] = b;
    return;
  }
  if (p.bias) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int4 t = bp[j];
      v[4 * j] += t.x; v[4 * j + 1] += t.y; v[4 * j + 2] += t.z; v[4 * j + 3] += t.w;
    }
  }
  // step by step, eight columns at a time (OC is a multiple of 8: all of them or none exist)
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    if (col0 + g * 8 >= p.oc) break;
    int32_t t[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) t[j] = v[g * 8 + j];
    apply_chain<8>(p.chain, t, lin + g * 8, col0 + g * 8, 1, nullptr, -1, p.first_step);
    if (p.y_dtype == CVMK_I8) {
      uint2 o;
      o.x = pack4(t[0], t[1], t[2], t[3]);
      o.y = pack4(t[4], t[5], t[6], t[7]);
      *reinterpret_cast<uint2*>(reinterpret_cast<int8_t*>(p.y) + lin + g * 8) = o;
    } else {
      int4* dst = reinterpret_cast<int4*>(reinterpret_cast<int32_t*>(p.y) + lin + g * 8);
      dst[0] = make_int4(t[0], t[1], t[2], t[3]);
      dst[1] = make_int4(t[4], t[5], t[6], t[7]);
    }
  }
}

__global__ void __launch_bounds__(THREADS)
conv_small_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ SmallConvParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t bar_full[SMALL_MAX_STAGES];
  __shared__ uint64_t bar_empty[SMALL_MAX_STAGES];
  __shared__ uint64_t bar_acc;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_flag;
  __shared__ __align__(16) int32_t bias_s[SMALL_MAX_N];

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int split = p.split;
  const int rank = split > 1 ? (int)cluster_rank() : 0;
  const int tile = split > 1 ? (int)blockIdx.x / split : (int)blockIdx.x;
  const int a_bytes = BLOCK_M * p.block_k, b_bytes = p.block_n * p.block_k;
  const int stage_bytes = a_bytes + b_bytes;
  const int u0 = rank * p.units / split, u1 = (rank + 1) * p.units / split;
  const int mine = u1 - u0;
  // tile origin
  const int mt = fdiv(tile, p.fd_n_tiles);
  const int n0 = (tile - mt * p.num_n_tiles) * p.block_n;
  const int m0 = mt * BLOCK_M;
  int cw = 0, ch = 0, cn = 0;
  if (p.a_mode == 2) {
    const int r = fdiv(mt, p.fd_tiles_w);
    cw = (mt - r * p.tiles_w) * p.patch_w;
    cn = fdiv(r, p.fd_tiles_h);
    ch = (r - cn * p.tiles_h) * p.patch_h;
    cn *= p.patch_n;
  }

  if (split > 1) cluster_arrive();   // (waited for before anything is written into another CTA)
  const bool leader = elect_one();
  const uint32_t ring = smem_u32(smem);
  if (warp == 0) {
    if (leader) {
      for (int s = 0; s < p.stages; ++s) {
        mbar_init(&bar_full[s], 1);
        mbar_init(&bar_empty[s], 1);
      }
      mbar_init(&bar_acc, 1);
      abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    // the weights of the first stages: parameters, no kernel writes them
    const int first = min(p.stages, mine);
    for (int i = 0; i < first; ++i)
      if (leader) {
        mbar_expect_tx(&bar_full[i], (uint32_t)stage_bytes);
        tma_load_2d(smem + i * stage_bytes + a_bytes, &tmap_b, &bar_full[i], (u0 + i) * p.block_k, n0);
      }
  } else if (warp == 1) {
    // (the next kernel may start only once this CTA has its TMEM columns: it could take them, and then
    //  wait for this kernel's end)
    tmem_alloc(&tmem_slot, (uint32_t)p.tmem_cols);
    pdl_trigger();
  } else {
    const bool early = p.bias_static != 0;
    if (!early) pdl_wait();
    for (int i = (int)threadIdx.x - 64; i < p.block_n; i += 128) {
      const int32_t b = (p.bias && n0 + i < p.oc) ? __ldg(p.bias + n0 + i) : 0;
      // packed requantisation: (bias + rounding addend) pre-multiplied, see fast_requant()
      bias_s[i] = (p.fast_variant >= 0 && p.fast_variant < 8) ? (int32_t)((uint32_t)(b + p.f_add) * (uint32_t)p.f_mul) : b;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA
    int img = 0, base_w = 0, base_h = 0;
    if (p.a_mode == 1) {
      img = fdiv(m0, p.fd_ohow);
      const int rem = m0 - img * (p.oh * p.ow);
      const int oy = fdiv(rem, p.fd_ow);
      base_w = (rem - oy * p.ow) * p.stride_w - p.pad_w;
      base_h = oy * p.stride_h - p.pad_h;
    }
    // first unit: filter tap and channel block
    int tap = fdiv(u0, p.fd_cblocks);
    int cc = (u0 - tap * (p.c / p.block_k)) * p.block_k;
    int fy = fdiv(tap, p.fd_kw), fx = tap - fy * p.kw;
    pdl_wait();
    int stage = 0;
    uint32_t phase = 0;
    for (int i = 0; i < mine; ++i) {
      uint8_t* sa = smem + stage * stage_bytes;
      uint64_t* bar = &bar_full[stage];
      if (i >= p.stages) {
        if (!mbar_wait(&bar_empty[stage], phase ^ 1, &abort_flag, 1)) break;
        if (leader) {
          mbar_expect_tx(bar, (uint32_t)stage_bytes);
          tma_load_2d(sa + a_bytes, &tmap_b, bar, (u0 + i) * p.block_k, n0);
        }
      }
      if (leader) {
        const int off_w = fx * p.dil_w, off_h = fy * p.dil_h;
        if (p.a_mode == 2) tma_load_4d(sa, &tmap_a, bar, cc, cw + off_w - p.pad_w, ch + off_h - p.pad_h, cn);
        else if (p.a_mode == 1) tma_load_im2col_4d(sa, &tmap_a, bar, cc, base_w, base_h, img, (uint16_t)off_w, (uint16_t)off_h);
        else tma_load_2d(sa, &tmap_a, bar, cc, m0);
      }
      cc += p.block_k;
      if (cc >= p.c) { cc = 0; if (++fx == p.kw) { fx = 0; ++fy; } }
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA
    const uint32_t idesc = umma_idesc_i8(p.block_n);
    const uint64_t desc0 = umma_desc(ring, p.block_k);
    const uint32_t lo0 = (uint32_t)desc0, hi = (uint32_t)(desc0 >> 32);
    const uint32_t stage_q = (uint32_t)stage_bytes >> 4, a_q = (uint32_t)a_bytes >> 4;
    const int nk = p.block_k / 32;
    int stage = 0;
    uint32_t phase = 0;
    for (int i = 0; i < mine; ++i) {
      if (!mbar_wait(&bar_full[stage], phase, &abort_flag, 3)) break;
      tc_fence_after();
      const uint32_t al = lo0 + stage_q * (uint32_t)stage;
      if (leader) {
        if (nk == 4) mma_i8_k<4>(tmem_base, al, hi, al + a_q, hi, idesc, (uint32_t)i);
        else if (nk == 2) mma_i8_k<2>(tmem_base, al, hi, al + a_q, hi, idesc, (uint32_t)i);
        else mma_i8_k<1>(tmem_base, al, hi, al + a_q, hi, idesc, (uint32_t)i);
        if (i + p.stages < mine) mma_commit(&bar_empty[stage]);   // (nobody waits for the last ones)
        if (i + 1 == mine) mma_commit(&bar_acc);
      }
      if (++stage == p.stages) { stage = 0; phase ^= 1; }
    }
    __syncwarp();
  }

  __syncwarp();

  // ------------------------------------------------------------------ epilogue
  const int quarter = warp & 3;
  const int row_in_tile = quarter * 32 + lane;   // epilogue warps 2..5: TMEM lanes of the warp's quarter
  const int rows_per = BLOCK_M / split;          // rows this CTA finishes
  auto out_row = [&](int r) {                    // linear output row of tile row r; -1 outside the tensor
    if (p.a_mode != 2) return m0 + r < p.m_total ? m0 + r : -1;
    const int ow = cw + (r & (p.patch_w - 1)), q = r >> p.patch_w_log2;
    const int oh = ch + (q & (p.patch_h - 1)), on = cn + (q >> p.patch_h_log2);
    return (ow < p.ow && oh < p.oh && on * p.oh * p.ow < p.m_total) ? (on * p.oh + oh) * p.ow + ow : -1;
  };
  const uint4 none = make_uint4(0, 0, 0, 0);
  auto operand = [&](int row, int col, uint4* r0, uint4* r1) {
    if (p.res == nullptr || p.fast_variant < 0 || row < 0 || col >= p.oc) return;
    const uint4* q = reinterpret_cast<const uint4*>(p.res + (size_t)row * p.oc + col);
    *r0 = q[0];
    *r1 = q[1];
  };
  const int chunks = p.block_n >> 5;
  if (warp >= 2) pdl_wait();
  if (split == 1) {
    if (warp >= 2) {
      const int row = out_row(row_in_tile);
      uint4 r0 = none, r1 = none;
      operand(row, n0, &r0, &r1);   // the tensor operand travels while the products are computed
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar_acc, 0u, &abort_flag, 4));
      tc_fence_after();
      if (ok) {
        const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16);
        for (int c = 0; c < chunks; ++c) {
          const int col = n0 + c * 32;
          if (col >= p.oc) break;
          int32_t v[32];
          tmem_ld32(tbase + (uint32_t)(c * 32), v);
          uint4 q0 = r0, q1 = r1;
          if (c + 1 < chunks) operand(row, col + 32, &r0, &r1);
          if (row >= 0) finish_chunk(p, v, row, col, bias_s + c * 32, q0, q1);
        }
      }
    }
  } else {
    cluster_wait();   // every CTA of the cluster has started
    // Partial sums: tile row r goes to rank r / rows_per, as row r % rows_per of its block from
    // this rank.  16-byte chunks of a row are XORed with its low bits: lanes hold different rows.
    uint8_t* part = smem + p.stages * stage_bytes;
    if (warp >= 2) {
      const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar_acc, 0u, &abort_flag, 4));
      tc_fence_after();
      if (ok) {
        const int dest = row_in_tile / rows_per, rl = row_in_tile - dest * rows_per;
        const uint32_t base = map_rank(smem_u32(part) + (uint32_t)((rank * rows_per + rl) * p.block_n * 4), (uint32_t)dest);
        const uint32_t tbase = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const bool live = out_row(row_in_tile) >= 0;
        for (int c = 0; c < chunks; ++c) {
          int32_t v[32];
          tmem_ld32(tbase + (uint32_t)(c * 32), v);
          if (live) {
#pragma unroll
            for (int j = 0; j < 8; ++j)
              st_cluster_v4(base + (uint32_t)(((c * 8 + j) ^ (rl & 7)) << 4), v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          }
        }
      }
    }
    __syncwarp();
    cluster_arrive();
    uint4 r0 = none, r1 = none;
    const int t = (int)threadIdx.x - 64;
    const int jobs = rows_per * chunks;
    auto job_row = [&](int k) { return rank * rows_per + k / chunks; };
    if (warp >= 2 && t < jobs) operand(out_row(job_row(t)), n0 + (t % chunks) * 32, &r0, &r1);
    cluster_wait();
    if (warp >= 2 && !abort_flag) {
      for (int k = t; k < jobs; k += 128) {
        const int rl = k / chunks, c = k - rl * chunks, col = n0 + c * 32;
        const int row = out_row(rank * rows_per + rl);
        if (row < 0 || col >= p.oc) continue;
        if (k != t) operand(row, col, &r0, &r1);
        int32_t v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0;
        for (int s = 0; s < split; ++s) {
          const uint8_t* src = part + (size_t)(s * rows_per + rl) * p.block_n * 4;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int4 q = *reinterpret_cast<const int4*>(src + (((c * 8 + j) ^ (rl & 7)) << 4));
            v[4 * j] += q.x; v[4 * j + 1] += q.y; v[4 * j + 2] += q.z; v[4 * j + 3] += q.w;
          }
        }
        finish_chunk(p, v, row, col, bias_s + c * 32, r0, r1);
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);   // copies in flight land before shared memory is released
    if (threadIdx.x == 0 && p.status) atomicOr(p.status, 0x200 | abort_flag);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
  }
}

}  // namespace

int launch_conv_small(const CUtensorMap& a, const CUtensorMap& b, const SmallConvParams& p, int grid, int smem, cudaStream_t stream) {
  static bool attr_of_device[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_of_device[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(conv_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(conv_small_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (check_cuda(e, "cudaFuncSetAttribute(conv_small_kernel)")) return CVMK_ERR_CUDA;
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
  return check_cuda(cudaLaunchKernelEx(&cfg, conv_small_kernel, a, b, p), "conv_small_kernel launch");
}

}  // namespace cvmk
