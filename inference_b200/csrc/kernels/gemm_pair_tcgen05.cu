// bf16 GEMM for sm_100a on pairs of SMs: D[T, N] = epilogue(A[T, K] * W[N, K]^T), for token counts above the decode kernels'.
//
// A cluster of two CTAs computes a 256 x BN tile (BN = 32 .. 256) with tcgen05.mma.cta_group::2: each CTA brings its own 128 rows
// of A and half of the tile's weight rows, so a k-block of 64 costs an SM 32 KB of operands (BN = 256) instead of the 48 KB
// of a 128 x 256 tile on one SM. That traffic out of L2 is what bounded the one-SM kernel at prompt sizes
// (gemm_tcgen05.cu, which keeps the peer-scatter epilogues, the shapes without 16-byte rows and those where 128-row tiles fill the
// chip better: gemm_bf16_takes_pairs).
//   warp 0      TMA producer of this CTA; all copies of a stage complete on the even CTA's barrier
//   warp 1      TMEM owner; in the even CTA it issues the MMAs of the pair
//   warps 2..9  epilogue: warp = (32 TMEM lanes, half of the columns); two accumulators, so it overlaps the next tile's
//               main loop. Rows leave through a 4 KB slab of shared memory per warp as whole 128-byte lines.
// Persistent clusters walk (tile, k-split) items. With k-splits every warp parks its fp32 part of the tile in the workspace and the
// last one to arrive sums the parts in split order: the result does not depend on timing.
// Two more layouts of A and D share the kernel: an implicit 3x3 convolution (a CTA's 128 rows are a box of pixels behind a 4-D tensor
// map) and grouped rows (mixture of experts: a device list of row ranges, each with its own weight).
// Every wait is bounded; on expiry the CTA raises its abort flag, lets its copies land, frees TMEM and returns.
#include "common.cuh"
#include "gemm_pair.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

namespace swb {

SWB_REGISTER_STATUS_UNIT(gemm_pair);

namespace {

constexpr int BM = 128;                 // rows of one CTA (256 of the pair)
constexpr int BK = 64;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int GROUP_M = 8;              // row tiles walked before the next column of tiles: their A stays in L2

template <int BN>
struct PairCfg {
  static constexpr int STAGES = BN >= 192 ? 6 : 8;
  static constexpr uint32_t A_BYTES = BM * BK * 2;
  static constexpr uint32_t B_BYTES = BN / 2 * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr uint32_t TMEM_COLS = BN > 128 ? 512 : 2 * BN;
  static constexpr uint32_t SLAB_BYTES = 32 * 128;
  static constexpr uint32_t SMEM_SLABS = STAGES * STAGE_BYTES;
  static constexpr uint32_t SMEM_BARS = SMEM_SLABS + EPI_WARPS * SLAB_BYTES;
  static constexpr size_t SMEM_BYTES = SMEM_BARS + 256 + 1024 /*align slack*/;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same shared-memory address in the even CTA of the pair.
__device__ __forceinline__ uint32_t in_even_cta(uint32_t addr) { return addr & 0xFEFFFFFFu; }

// Copies whose completion is counted on the even CTA's barrier.
__device__ __forceinline__ void tma_pair_2d(uint32_t dst, const void* tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_pair_4d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void umma_pair_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on the barrier at this address in both CTAs once every MMA issued so far has completed.
__device__ __forceinline__ void umma_pair_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_even(uint32_t bar) {
  asm volatile(
      "{\n"
      ".reg .b32 remote;\n"
      "mapa.shared::cluster.u32 remote, %0, 0;\n"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [remote];\n"
      "}\n" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void tmem_ld_32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
      "%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// One (tile, k-range) item. Every role walks the same sequence.
struct Item {
  int tm, tn, tile, split, kb0, kb1;
  int row0, rows, weight_row;          // rows of the pair's tile that exist, first weight row
};
struct ItemIter {
  const PairParams& p;
  int next_item, total, tiles_m;
  __device__ explicit ItemIter(const PairParams& pp) : p(pp) {
    next_item = (int)blockIdx.x >> 1;
    tiles_m = p.group_tiles ? __ldg(p.group_count) : p.tiles_m;
    total = tiles_m * p.tiles_n * p.splits;
  }
  __device__ __forceinline__ bool next(Item& s) {
    if (next_item >= total) return false;
    s.tile = next_item / p.splits;
    s.split = next_item - s.tile * p.splits;
    next_item += (int)gridDim.x >> 1;
    const int per_group = GROUP_M * p.tiles_n;
    const int g = s.tile / per_group, first_m = g * GROUP_M, r = s.tile - g * per_group;
    const int gsize = min(GROUP_M, tiles_m - first_m);
    s.tm = first_m + r % gsize;
    s.tn = r / gsize;
    s.kb0 = s.split * p.kblocks_per_split;
    s.kb1 = min(p.kblocks, s.kb0 + p.kblocks_per_split);
    if (p.group_tiles) {
      const int4 t = __ldg(p.group_tiles + s.tm);
      s.row0 = t.x;
      s.rows = t.y;
      s.weight_row = t.z * p.N;
    } else {
      s.row0 = s.tm * 2 * BM;
      s.rows = p.M - s.row0;
      s.weight_row = 0;
    }
    return true;
  }
};

// Pixel box of a convolution's CTA tile.
struct Box {
  int img, y0, x0;
};
__device__ __forceinline__ Box box_of(const PairParams& p, int index) {
  const int per_img = p.boxes_x * p.boxes_y;
  Box b;
  b.img = index / per_img;
  const int r = index - b.img * per_img, by = r / p.boxes_x;
  b.y0 = by << p.box_h_log;
  b.x0 = (r - by * p.boxes_x) << p.box_w_log;
  return b;
}

__device__ __forceinline__ float pair_act(float x, const PairParams& p, int act) {
  switch (act) {
    case SWB_ACT_SILU: return silu_f(x);
    case SWB_ACT_GELU_TANH: return gelu_tanh_f(x);
    case SWB_ACT_RELU2: return relu2_f(x);
    case SWB_ACT_XIELU: return xielu_f(x, p.act_a, p.act_b);
    default: return x;
  }
}
// The same for 32 values: one choice for all of them. Looked up for every element it was half of the time of short products: 897 x 14336 x 1152 with bias and GELU 93 us
// (107 with the output chosen at run time too) and 52.7 so, 722 x 15360 x 5120 108 and 90, two outputs of 9216 and 12288 columns of 3072 at 4608 rows 628 and 443.
__device__ __forceinline__ void pair_act_all(float* v, const PairParams& p, int act) {
  auto all = [&](auto f) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = f(v[j]);
  };
  switch (act) {
    case SWB_ACT_SILU: all([](float x) { return silu_f(x); }); break;
    case SWB_ACT_GELU_TANH: all([](float x) { return gelu_tanh_f(x); }); break;
    case SWB_ACT_RELU2: all([](float x) { return relu2_f(x); }); break;
    case SWB_ACT_XIELU: all([&](float x) { return xielu_f(x, p.act_a, p.act_b); }); break;
    default: break;
  }
}
__device__ __forceinline__ void add_bf16x8(float* v, const uint4 u) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) v[2 * i] += __uint_as_float(w[i] << 16), v[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
}
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ void copy_async16(void* smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Where the columns of a tile go. TWO: there is a second output, an instantiation of its own.
template <bool TWO>
struct OutSel {
  void* out;
  int ldd, act, first;       // first accumulator column of this output
  __device__ __forceinline__ OutSel(const PairParams& p, int col0) {
    const bool second = TWO && col0 >= p.first_n;
    out = second ? p.out2 : p.out, ldd = second ? p.ldd2 : p.ldd, act = second ? p.act2 : p.act, first = second ? p.first_n : 0;
  }
};

// Where the rows of this warp's 32 TMEM lanes lie in D (and in the residual): -1 = no such row.
struct RowMap {
  const PairParams& p;
  int first, valid;      // plain and grouped rows: first row of the warp, how many of its 32 exist
  Box box;
  int lane0;             // convolution: first of the warp's rows within the CTA's box
  __device__ __forceinline__ long long operator()(int r) const {
    if (p.conv_c == 0) return r < valid ? (long long)(first + r) : -1;
    const int i = lane0 + r, y = box.y0 + (i >> p.box_w_log), x = box.x0 + (i & ((1 << p.box_w_log) - 1));
    if (box.img >= p.conv_n || y >= p.conv_h || x >= p.conv_w) return -1;
    return ((long long)box.img * p.conv_h + y) * p.conv_w + x;
  }
};

// Sums for the group norm that reads a convolution's output. Lanes 0..7 have the warp's first 64 columns, lanes 8..15 the next ones (eight columns each,
// in two halves); the sums stay in registers over the tiles of an image's column block and go to memory when that changes. (A pass of its own
// over the output took 107 us for 128 channels at 1216 x 832, behind a convolution of 337 us; with the sums it takes 351.)
struct GroupSums {
  float sum[2], sq[2];
  int img, col0;
  __device__ __forceinline__ void clear() { sum[0] = sum[1] = sq[0] = sq[1] = 0.f; }
  template <int COLS>
  __device__ __forceinline__ void flush(const PairParams& p, int lane) {
    const int gc = p.group_channels;
    if (img >= 0) {
      float s0 = sum[0], s1 = sum[1], q0 = sq[0], q1 = sq[1];
      if (gc >= 8) s0 += s1, q0 += q1;
      for (int o = 1; o < gc / 8; o <<= 1) {
        s0 += __shfl_xor_sync(0xffffffffu, s0, o);
        q0 += __shfl_xor_sync(0xffffffffu, q0, o);
      }
      const int chunk = lane & 7, in_warp = (lane >> 3) * 64 + chunk * 8, c = col0 + in_warp;
      if (in_warp < COLS && c < p.N && (gc < 8 || chunk % (gc / 8) == 0)) {
        float* at = p.stats + ((size_t)img * (p.N / gc) + c / gc) * 2;
        atomicAdd(at, s0);
        atomicAdd(at + 1, q0);
        if (gc == 4) {
          atomicAdd(at + 2, s1);
          atomicAdd(at + 3, q1);
        }
      }
    }
    clear();
  }
};

// cols accumulator columns of this warp's 32 rows (thread = row) -> D. `load(c, v)` gives columns c .. c + 31.
template <bool STATS, bool TWO, typename Load>
__device__ __forceinline__ void store_columns(int cols, const PairParams& p, const RowMap& rows, int col0, uint8_t* slab, int lane, GroupSums& sums, Load load) {
  const OutSel<TWO> to(p, col0);
  const bool pairs = gemm_act_pairs(p.act);
  const long long my_row = rows(lane);
  const int swz = lane & 7;
  const int sub = lane >> 3, chunk = lane & 7;           // coalesced phases: four rows at a time, eight lanes each
  if (p.out_fp32) {      // a slab holds 32 rows x 32 fp32 of D, 16-byte chunk c of row r at c ^ (r & 7)
#pragma unroll 1
    for (int c = 0; c < cols; c += 32) {
      const int a0 = col0 + c;
      if (a0 >= p.N) break;
      float v[32];
      __syncwarp();
      load(c, v);
      if (p.bias) {
#pragma unroll
        for (int j = 0; j < 32; j += 8)
          if (a0 + j < p.N) add_bf16x8(v + j, __ldg(reinterpret_cast<const uint4*>(p.bias + a0 + j)));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float4 f = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        if (p.act != SWB_ACT_NONE) f = make_float4(pair_act(f.x, p, p.act), pair_act(f.y, p, p.act), pair_act(f.z, p, p.act), pair_act(f.w, p, p.act));
        *reinterpret_cast<float4*>(slab + lane * 128 + ((j ^ swz) << 4)) = f;
      }
      __syncwarp();
      const int d = a0 + chunk * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + sub;
        const long long row = rows(r);
        if (row < 0 || d >= p.N) continue;
        float4 f = *reinterpret_cast<const float4*>(slab + r * 128 + ((chunk ^ (r & 7)) << 4));
        if (p.residual) {
          const uint2 u = *reinterpret_cast<const uint2*>(p.residual + row * p.ld_res + d);
          f.x += __uint_as_float(u.x << 16), f.y += __uint_as_float(u.x & 0xffff0000u);
          f.z += __uint_as_float(u.y << 16), f.w += __uint_as_float(u.y & 0xffff0000u);
        }
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + row * p.ldd + d) = f;
      }
    }
    return;
  }
  // A slab holds 32 rows x 64 bf16 of D; its 16-byte chunk c of row r lies at c ^ (r & 7).
  uint8_t* my_slab = slab + lane * 128;
  const int step = pairs ? 128 : 64;
  const int width = pairs ? p.N / 2 : p.N;              // columns of D
  const bf16* gate = p.gate ? p.gate + (long long)(my_row < 0 ? 0 : (int)my_row / p.rows_per_gate) * p.ld_gate : nullptr;
#pragma unroll 1
  for (int s = 0; s < cols; s += step) {
    const int d0 = pairs ? (col0 + s) >> 1 : col0 + s;   // first column of D in this slab
    if (d0 >= width) break;
    const bool in = d0 + chunk * 8 < width && chunk * 8 < (pairs ? (cols - s) / 2 : cols - s);
    if (p.residual) {      // copies straight to the slab: all on their way at a time, without registers
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + sub;
        const long long row = rows(r);
        if (row >= 0 && in) copy_async16(slab + r * 128 + ((chunk ^ (r & 7)) << 4), p.residual + row * p.ld_res + d0 + chunk * 8);
      }
      copy_async_wait();
      __syncwarp();
    }
#pragma unroll 1
    for (int c = s; c < min(s + step, cols); c += 32) {
      float v[32];
      load(c, v);
      const int a0 = col0 + c;                           // first accumulator column
      if (a0 >= p.N) break;
      if (p.bias) {
#pragma unroll
        for (int j = 0; j < 32; j += 8)
          if (a0 + j < p.N) add_bf16x8(v + j, __ldg(reinterpret_cast<const uint4*>(p.bias + a0 + j)));
      }
      if (pairs) {
        float o[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float g = v[2 * j], u = v[2 * j + 1];
          o[j] = p.act == SWB_ACT_CLAMPED_PAIRS ? clamped_gate_f<false>(g, u, p.act_a)
                                                : (p.act == SWB_ACT_GEGLU_PAIRS ? gelu_tanh_f(g) : silu_f(g)) * u;
        }
        const int k = (c - s) >> 4;                      // 16 columns of D = two chunks
        *reinterpret_cast<uint4*>(my_slab + ((k ^ swz) << 4)) = pack8(o);
        *reinterpret_cast<uint4*>(my_slab + (((k + 1) ^ swz) << 4)) = pack8(o + 8);
      } else {
        pair_act_all(v, p, to.act);
        const int k0 = (c - s) >> 3;
        if (gate) {
#pragma unroll
          for (int j = 0; j < 32; j += 8) {
            if (a0 + j >= p.N) continue;
            float f[8];
            load_row8(gate + a0 + j, f);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[j + i] *= f[i];
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4* at = reinterpret_cast<uint4*>(my_slab + (((k0 + j) ^ swz) << 4));
          if (p.residual) add_bf16x8(v + 8 * j, *at);
          *at = pack8(v + 8 * j);
        }
      }
    }
    __syncwarp();
    bf16* out = reinterpret_cast<bf16*>(to.out) + (d0 - to.first) + chunk * 8;
    int first = sub;
    asm volatile("" : "+r"(first));      // places of rows are computed again: kept from the residual's copies they would spill
    float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i * 4 + first;
      const long long row = rows(r);
      if (row >= 0 && in) {
        const uint4 u = *reinterpret_cast<const uint4*>(slab + r * 128 + ((chunk ^ (r & 7)) << 4));
        *reinterpret_cast<uint4*>(out + row * to.ldd) = u;
        if constexpr (STATS) {
          const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float a = __uint_as_float(w[j] << 16), b = __uint_as_float(w[j] & 0xffff0000u);
            t[j >> 1] += a + b;
            t[2 + (j >> 1)] = fmaf(a, a, fmaf(b, b, t[2 + (j >> 1)]));
          }
        }
      }
    }
    if constexpr (STATS) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        t[j] += __shfl_xor_sync(0xffffffffu, t[j], 8);
        t[j] += __shfl_xor_sync(0xffffffffu, t[j], 16);
      }
      if (sub == s >> 6) sums.sum[0] += t[0], sums.sum[1] += t[1], sums.sq[0] += t[2], sums.sq[1] += t[3];
    }
    __syncwarp();
  }
}

template <int BN, bool STATS, bool TWO>
__global__ void __launch_bounds__(THREADS, 1) __cluster_dims__(2, 1, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const PairParams p) {
  using Cfg = PairCfg<BN>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw_addr = smem_u32(smem_raw);
  uint8_t* smem = smem_raw + ((1024u - (raw_addr & 1023u)) & 1023u);
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(smem + Cfg::SMEM_BARS);   // used in the even CTA: a stage of both CTAs is there
  uint64_t* bar_empty = bar_full + STAGES;
  uint64_t* bar_tfull = bar_empty + STAGES;
  uint64_t* bar_tempty = bar_tfull + 2;                                      // used in the even CTA: 2 x EPI_WARPS arrivals
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_tempty + 2);
  volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta = cluster_rank();

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&bar_full[s], 1);
      mbar_init(&bar_empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&bar_tfull[a], 1);
      mbar_init(&bar_tempty[a], 2 * EPI_WARPS);
    }
    *s_abort = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(Cfg::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();        // both CTAs' barriers exist before either signals the other's
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  // The issuing warps run whole, with one elected lane for the instruction itself: descriptors and addresses stay in uniform registers.
  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    pdl_wait(TL_GEMM);
    ItemIter iter(p);
    Item c;
    while (ok && iter.next(c)) {
      const int b_row = c.weight_row + c.tn * BN + (int)cta * (BN / 2);
      const int a_row = c.row0 + (int)cta * BM;
      Box box{};
      if (p.conv_c) box = box_of(p, 2 * c.tm + (int)cta);
      for (int kb = c.kb0; kb < c.kb1; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bar_empty[stage], phase ^ 1, s_abort, 100 + stage));
        if (!ok) break;
        const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
        const uint32_t bar = in_even_cta(smem_u32(&bar_full[stage]));
        if (elect_one()) {
          if (cta == 0) mbar_arrive_expect_tx(&bar_full[stage], 2 * Cfg::STAGE_BYTES);
          if (p.conv_c) {
            const int slabs = p.conv_c / BK, tap = kb / slabs, c0 = (kb - tap * slabs) * BK;
            tma_pair_4d(sa, &tmap_a, bar, c0, box.x0 + tap % 3 - 1, box.y0 + tap / 3 - 1, box.img);
          } else {
            tma_pair_2d(sa, &tmap_a, bar, kb * BK, a_row);
          }
          tma_pair_2d(sa + Cfg::A_BYTES, &tmap_b, bar, kb * BK, b_row);
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
    // Not earlier: blocks of the next kernel that wait on an SM during the main loop cost more than their early start gives
    // (a prompt step of an 8B decoder, 8000 tokens: 115 ms with the trigger at the start of every kernel, 107 ms without).
    pdl_launch_dependents();
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (even CTA) ------------------------------
    if (cta == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16_f32(2 * BM, BN);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      pdl_wait();
      ItemIter iter(p);
      Item c;
      while (ok && iter.next(c)) {
        ok = __all_sync(0xffffffffu, mbar_wait(&bar_tempty[acc], acc_phase ^ 1, s_abort, 200 + acc));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + (uint32_t)(acc * BN);
        for (int kb = c.kb0; kb < c.kb1; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&bar_full[stage], phase, s_abort, 300 + stage));
          if (!ok) break;
          tc_fence_after_sync();
          const uint32_t sa = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint64_t adesc = umma_desc_kmajor_sw128(sa);
          const uint64_t bdesc = umma_desc_kmajor_sw128(sa + Cfg::A_BYTES);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_pair_f16(tmem_d, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k), idesc, (kb > c.kb0 || k > 0) ? 1u : 0u);
            umma_pair_commit(smem_u32(&bar_empty[stage]));
          }
          __syncwarp();
          if (++stage == STAGES) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        if (elect_one()) umma_pair_commit(smem_u32(&bar_tfull[acc]));
        __syncwarp();
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    // columns of one warp, in slabs of 64 where there are as many; with BN = 32 the second half's warps idle, with 224 they have one load less
    constexpr int COLS = BN / 2 < 32 ? 32 : BN == 224 ? 128 : BN / 2;
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int cols = BN == 224 && half ? BN - COLS : COLS;
    const bool idle = BN < 64 && half == 1;
    uint8_t* slab = smem + Cfg::SMEM_SLABS + (warp - 2) * Cfg::SLAB_BYTES;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    pdl_wait();
    ItemIter iter(p);
    Item c;
    GroupSums sums;
    sums.clear();
    sums.img = -1, sums.col0 = 0;
    while (ok && iter.next(c)) {
      // one answer for the warp: what follows (tcgen05.ld, __syncwarp, the split counter) takes all of its lanes
      ok = __all_sync(0xffffffffu, mbar_wait(&bar_tfull[acc], acc_phase, s_abort, 400 + acc));
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN + half * COLS);
      const int col0 = c.tn * BN + half * COLS;
      const int row_in_tile = (int)cta * BM + quarter * 32;
      RowMap rows{p, c.row0 + row_in_tile, c.rows - row_in_tile, p.conv_c ? box_of(p, 2 * c.tm + (int)cta) : Box{}, quarter * 32};
      if (STATS && !idle && rows.box.img < p.conv_n && (rows.box.img != sums.img || col0 != sums.col0)) {
        sums.flush<COLS>(p, lane);
        sums.img = rows.box.img, sums.col0 = col0;
      }
      if (p.splits == 1) {
        if (!idle) store_columns<STATS, TWO>(cols, p, rows, col0, slab, lane, sums, [&](int cc, float* v) { tmem_ld_32(taddr + cc, v); });
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_even(smem_u32(&bar_tempty[acc]));
      } else {
        constexpr size_t SLOT = (size_t)BN * BM;
        const size_t tile_slot = ((size_t)c.tile * 2 + cta) * p.splits;
        const size_t mine = (size_t)half * COLS * BM + quarter * 32 + lane;
        if (!idle) {
          float* ws = p.workspace + (tile_slot + c.split) * SLOT + mine;
#pragma unroll 1
          for (int cc = 0; cc < cols; cc += 32) {
            float v[32];
            tmem_ld_32(taddr + cc, v);
#pragma unroll
            for (int j = 0; j < 32; ++j) __stcg(ws + (size_t)(cc + j) * BM, v[j]);
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_even(smem_u32(&bar_tempty[acc]));
        // each warp's part of the tile is reduced by the last such warp to arrive: no barrier among the warps
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) {
          int* counter = p.counters + (c.tile * 2 + (int)cta) * EPI_WARPS + (warp - 2);
          last = atomicAdd(counter, 1) == p.splits - 1;
          if (last) *counter = 0;                        // ready for the next launch
        }
        last = __shfl_sync(0xffffffffu, last, 0);
        if (last && !idle) {
          __threadfence();
          const float* ws = p.workspace + tile_slot * SLOT + mine;
          store_columns<false, TWO>(cols, p, rows, col0, slab, lane, sums, [&](int cc, float* v) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __ldcg(ws + (size_t)(cc + j) * BM);
            for (int s = 1; s < p.splits; ++s) {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] += __ldcg(ws + (size_t)s * SLOT + (size_t)(cc + j) * BM);
            }
          });
        }
      }
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (STATS && !idle) sums.flush<COLS>(p, lane);
  }

  __syncwarp();
  if (*s_abort) {   // copies and MMAs in flight finish within microseconds; nothing is released before
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 1000000ull) {
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();        // neither CTA leaves while the other's MMAs read its operands or its warps signal its barriers
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::TMEM_COLS) : "memory");
  }
}

template <int BN, bool STATS, bool TWO>
int launch_pair_as(const CUtensorMap& ta, const CUtensorMap& tb, const PairParams& p, int clusters, cudaStream_t stream) {
  auto kern = gemm_pair_kernel<BN, STATS, TWO>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairCfg<BN>::SMEM_BYTES);
    if (e != cudaSuccess) return -(int)e;
    configured[dev] = true;
  }
  return launch_kernel(kern, dim3(2 * clusters), dim3(THREADS), PairCfg<BN>::SMEM_BYTES, stream, ta, tb, p);
}

template <int BN>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const PairParams& p, int clusters, cudaStream_t stream) {
  // sums: tiles whose warps' columns do not differ; two outputs: widths that divide the first one's 64-column pieces, as the plan gives them
  if constexpr (BN != 224) {
    if (p.stats) return launch_pair_as<BN, true, false>(ta, tb, p, clusters, stream);
  }
  if constexpr (BN != 32) {
    if (p.first_n > 0) return launch_pair_as<BN, false, true>(ta, tb, p, clusters, stream);
  }
  return p.stats || p.first_n > 0 ? -4 : launch_pair_as<BN, false, false>(ta, tb, p, clusters, stream);
}

// Estimated microseconds of a plan, without what gemm_pair_plan adds to the best one. Fitted to sweeps of every tile width and up to six splits over
// token counts 100..8000 and the projections of an 8B decoder and a 12B image transformer. A k-block costs more the fuller the chip
// is (operand traffic, power): 0.29 us at BN = 256 on half of the pairs, 0.35 us on all of them. Narrower tiles move the same A for less
// work but fill a last wave better: 975 x 9216 x 3072 takes 41.8 us at 256, 45.9 at 192, 52.3 at 128; 700 x 4096 x 4096 takes 27.2, 22.5, 32.1.
// 224 is for counts of row tiles that leave a wave of 256 partly empty without filling two of 192 (1231 x 3072 x 15360: 85.3 us at 256, 82.5 at 224, 118.5 at
// 192; 1231 x 9216 x 3072: 54.5, 51.7, 57.7; 975 x 12288 x 3072: 56.1, 54.2, 59.3); with k-splits the other widths fill the chip as well.
// k-splits pay for parking and reading back partial sums: 100 x 3072 x 12288 takes 43.4 us at 128, 25.3 in three splits, 33.5 in four.
double plan_cost(int bn, int splits, long tiles, int kblocks, int pairs) {
  const long items = tiles * splits, waves = (items + pairs - 1) / pairs;
  const int per = (kblocks + splits - 1) / splits;
  const double fill = (double)items / (double)(waves * pairs);
  const double t = bn == 256 ? 0.22 + 0.14 * fill : bn == 224 ? 0.195 + 0.125 * fill : bn == 192 ? 0.17 + 0.11 * fill : bn == 128 ? 0.15 + 0.085 * fill : 0.13 + 0.1 * fill;
  return waves * (per * t + 0.5) + (splits > 1 ? bn / 256.0 * (2.0 + 2.0 * splits) : 0.0);
}

}  // namespace

namespace {

size_t split_bytes(int T, int N, int bn, int splits) {
  const size_t tiles = (size_t)((T + 2 * BM - 1) / (2 * BM)) * ((N + bn - 1) / bn);
  return tiles * 2 * splits * BM * bn * sizeof(float);
}
bool counters_suffice(long tiles) { return tiles * 2 * EPI_WARPS * (long)sizeof(int) <= (long)SWB_GEMM_COUNTER_BYTES; }

}  // namespace

double gemm_pair_plan(int T, int N, int K, size_t sum_bytes, int* block_n, int* splits, int multiple) {
  const int pairs = device_sm_count() / 2;
  const int kblocks = (K + BK - 1) / BK;
  const long tm = (T + 2 * BM - 1) / (2 * BM);
  double best = 1e30;
  for (int bn : {256, 224, 192, 128, 64}) {
    if ((bn > 64 && bn >= 2 * N) || multiple % bn) continue;
    const long tiles = tm * ((N + bn - 1) / bn);
    for (int s = 1; s <= 8; ++s) {
      if (s > 1 && (bn == 224 || kblocks / s < 8 || sum_bytes < split_bytes(T, N, bn, s) || !counters_suffice(tiles) || tiles > pairs)) break;
      const double c = plan_cost(bn, s, tiles, kblocks, pairs);
      if (c < best) best = c, *block_n = bn, *splits = s;
    }
  }
  return best + 3.35 + 2.89 * *block_n / 256.0;      // launch, first loads and the last tile's epilogue
}

size_t gemm_pair_split_bytes(int T, int N, int K, int block_n, int splits) {
  if (block_n <= 0 && N > 32) {
    int s = 1;
    gemm_pair_plan(T, N, K, GEMM_SPLIT_BYTES_MAX, &block_n, &s);
    if (splits <= 0) splits = s;
  }
  return splits > 1 ? split_bytes(T, N, block_n, splits) : 0;
}

bool gemm_pair_accepts(const GemmArgs& a) {
  if (a.scatter || a.group_of_mtile || a.ssq_in || a.ssq_out || (a.peer && a.peer->mode)) return false;
  const bool pairs = gemm_act_pairs(a.act);
  const size_t esz = a.out_fp32 ? 4 : 2;
  if (pairs && (a.out_fp32 || a.residual || a.N % 16)) return false;
  if (a.gate && (a.out_fp32 || pairs)) return false;
  if (a.D2 && (a.first_n <= 0 || a.first_n >= a.N || a.first_n % 64 || a.conv_c || a.group_tiles || a.out_fp32 || pairs || gemm_act_pairs(a.act2) || a.residual || a.gate ||
               a.ldd2 % 8 || (reinterpret_cast<uintptr_t>(a.D2) & 15)))
    return false;
  if (a.conv_stats) {
    const int gc = a.stats_groups > 0 && a.N % a.stats_groups == 0 ? a.N / a.stats_groups : 0;
    if (!a.conv_c || a.out_fp32 || pairs || (gc != 4 && gc != 8 && gc != 16 && gc != 32)) return false;
  }
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (a.N % 8 || (a.ldd * esz) % 16 || !aligned(a.D) || (a.bias && !aligned(a.bias))) return false;
  if (a.residual && (!aligned(a.residual) || a.ld_res % 8)) return false;
  if (a.gate && (!aligned(a.gate) || a.ld_gate % 8 || a.rows_per_gate <= 0)) return false;
  return true;
}

int gemm_pair_launch(const GemmArgs& a, int block_n, int splits, cudaStream_t stream) {
  if (!gemm_pair_accepts(a)) return -3;
  PairParams p{};
  p.M = a.T;
  p.N = a.N;
  p.kblocks = (a.K + BK - 1) / BK;
  p.out = a.D;
  p.ldd = a.ldd;
  p.out_fp32 = a.out_fp32;
  p.bias = reinterpret_cast<const bf16*>(a.bias);
  p.residual = reinterpret_cast<const bf16*>(a.residual);
  p.ld_res = a.ld_res;
  p.gate = reinterpret_cast<const bf16*>(a.gate);
  p.ld_gate = a.ld_gate;
  p.rows_per_gate = a.rows_per_gate;
  p.act = a.act;
  p.act_a = a.act_a;
  p.act_b = a.act_b;
  if (a.D2) p.first_n = a.first_n, p.out2 = a.D2, p.ldd2 = a.ldd2, p.act2 = a.act2;
  p.tiles_m = (a.T + 2 * BM - 1) / (2 * BM);
  CUtensorMap ta, tb;
  int r;
  if (a.conv_c > 0) {
    if (a.conv_n <= 0 || a.conv_h <= 0 || a.conv_w <= 0 || a.conv_c % BK || a.K != 9 * a.conv_c || (long)a.T != (long)a.conv_n * a.conv_h * a.conv_w) return -3;
    // the box of 128 pixels that covers an image with the fewest boxes
    long best = -1;
    for (int wl = 7; wl >= 3; --wl) {
      const int bw = 1 << wl, bh = BM / bw;
      const long boxes = (long)((a.conv_w + bw - 1) / bw) * ((a.conv_h + bh - 1) / bh);
      if (best < 0 || boxes < best) {
        best = boxes;
        p.box_w_log = wl;
        p.box_h_log = 7 - wl;
        p.boxes_x = (a.conv_w + bw - 1) / bw;
        p.boxes_y = (a.conv_h + bh - 1) / bh;
      }
    }
    p.conv_n = a.conv_n;
    p.conv_h = a.conv_h;
    p.conv_w = a.conv_w;
    p.conv_c = a.conv_c;
    p.stats = a.conv_stats;
    p.group_channels = a.conv_stats ? a.N / a.stats_groups : 0;
    p.tiles_m = (int)((best * a.conv_n + 1) / 2);
    r = make_tmap_bf16_nhwc(&ta, a.A, a.conv_n, a.conv_h, a.conv_w, a.conv_c, 1 << p.box_w_log, 1 << p.box_h_log);
  } else {
    r = make_tmap_bf16_2d(&ta, a.A, a.T, a.K, a.lda, BM);
  }
  if (r) return r;
  if (a.group_tiles) {
    p.group_tiles = reinterpret_cast<const int4*>(a.group_tiles);
    p.group_count = a.group_count;
    p.tiles_m = a.group_max_tiles;
  }
  const int pairs = device_sm_count() / 2;
  void *counters = a.split_counters, *sums = a.split_sums;
  size_t sum_bytes = a.split_counters ? a.split_bytes : 0;
  if (!counters && a.workspace && a.workspace_bytes > SWB_GEMM_COUNTER_BYTES && !a.gate && (a.T <= 256 || a.force_mode == 3)) {
    counters = a.workspace;
    sums = reinterpret_cast<uint8_t*>(a.workspace) + SWB_GEMM_COUNTER_BYTES;
    sum_bytes = std::min(a.workspace_bytes - SWB_GEMM_COUNTER_BYTES, GEMM_SPLIT_BYTES_MAX);
  }
  if (a.conv_c || a.group_tiles) sum_bytes = 0;
  if (block_n <= 0) {
    if (a.N <= 32 && !gemm_act_pairs(a.act)) {      // a gated pair's epilogue takes 64 accumulator columns or more
      block_n = 32;
      splits = 1;
    } else {
      int s = 1;
      // a convolution's and a group list's rows are not T: plan with the row tiles they have. 768: all widths whose warps' columns do not differ (the
      // group sums of a convolution take them for equal; the number of a list's tiles is a bound, so how full its last wave is is not known)
      gemm_pair_plan(a.conv_c || a.group_tiles ? p.tiles_m * 2 * BM : a.T, a.N, a.K, sum_bytes, &block_n, &s, a.D2 ? a.first_n : a.conv_c || a.group_tiles ? 768 : 0);
      splits = splits > 0 ? splits : s;
    }
  }
  splits = std::max(1, splits);
  if (block_n != 256 && block_n != 224 && block_n != 192 && block_n != 128 && block_n != 64 && block_n != 32) return -4;
  if (gemm_act_pairs(a.act) && block_n < 64) return -4;
  r = make_tmap_bf16_2d(&tb, a.W, a.group_tiles ? a.groups * a.N : a.N, a.K, a.ldw, block_n / 2);
  if (r) return r;
  p.tiles_n = (a.N + block_n - 1) / block_n;
  const int per = (p.kblocks + splits - 1) / splits;
  splits = (p.kblocks + per - 1) / per;
  p.splits = splits;
  p.kblocks_per_split = per;
  const long tiles = (long)p.tiles_m * p.tiles_n;
  if (splits > 1) {
    if (!counters || !sums || sum_bytes < split_bytes(a.T, a.N, block_n, splits) || !counters_suffice(tiles)) return -4;
    p.counters = reinterpret_cast<int*>(counters);
    p.workspace = reinterpret_cast<float*>(sums);
  }
  const int clusters = (int)std::min<long>(tiles * splits, pairs);
  switch (block_n) {
    case 32: return launch_pair<32>(ta, tb, p, clusters, stream);
    case 64: return launch_pair<64>(ta, tb, p, clusters, stream);
    case 128: return launch_pair<128>(ta, tb, p, clusters, stream);
    case 224: return launch_pair<224>(ta, tb, p, clusters, stream);
    case 192: return launch_pair<192>(ta, tb, p, clusters, stream);
    default: return launch_pair<256>(ta, tb, p, clusters, stream);
  }
}

}  // namespace swb
