// Q4_K products of a decode step that are chained: D[T <= 8, N] = epilogue(A[T, K] * dequant(Wq)[N, K]^T).
//
// At this size the packed weights are the only stream that matters (4.5 bits per weight), and the arithmetic must not cost more than
// their arrival. A step of it is 16 weight rows x one super-block of 256 x 8 tokens, in a warp of its own: mma.sync.m16n8k16 in f16
// on operands that are exact.
//   weights      a 4-bit code as the bits of an f16 is code * 2^-24, a subnormal number that the tensor cores multiply exactly: two masks and a shift per word and
//                no conversion. High nibbles are 16 times too large, their activations 16 times too small. Block scales (6 bits, the same way) multiply the
//                fp32 sums of the 32 weights of a block. (Scales multiplied into f16 codes, which is exact too, kept the half-rate FMA pipe busy
//                with 64 packed multiply-adds per step: 23.1 us where this takes 21.0 for 28672 x 4096 at 4 tokens.)
//   activations  bf16 times a power of two of the (token, super-block) that takes the largest to 2^9 .. 2^10: f16 holds them exactly down to 2^-19 of
//                that one, and below it to 2^-35 of it. Those of an fp32 stream are rounded to 11 bits.
//   minima       sum over blocks of m * (sum of the block's activations): one more MMA per super-block, the sums as two f16 parts.
// The order of the reduction index is free as long as both operands agree. d and dmin are applied to the fp32 result of each super-block.
// A step does the same for any number of tokens; what grows with them is the conversion of the activations and the passes over a long reduction that they
// need. 28672 x 4096 takes 19.6 / 21.0 / 22.6 us at 1 / 4 / 8 tokens, 4096 x 14336 13.6 / 17.8 / 25.9; the kernel of single products (gemv_q4k.cu: dp4a on
// activations that are rounded to int8) 23.5 / 34.2 / 50.4 and 13.5 / 21.6 / 32.2. What is left above the weights' arrival (10.2 and 5.1 us): about 5 us of
// a launch before the first and behind the last weight, shared memory (activations 4 KB and weights 2.3 KB per step) and
// latency with four warps to a scheduler. A decode step of 4 tokens of an 8B decoder went from 3.27 to 2.50 ms, its error against 64 bits from 0.029 to 0.004.
// Small models gain from 4 tokens on; at 1 and 2 a step of 8 layers of 2048 takes 320 and 343 us where nine kernels a layer took 304 and 341.
//
// One CTA of 16 warps per SM. A CTA has every gridDim-th tile of 16 rows; the (tile, super-block) steps of its tiles lie on one line that is cut
// into 16 equal parts, one per warp, so that few warps meet in a tile and none is idle. Packed bytes come through a ring of
// cp.async stages per warp, requested before the activations exist. Parts meet in shared memory and are summed in the order of the
// reduction index. The epilogue may scale by 1 / rms of the token, add bias and residual, gate pairs of rows and add up the squares of what it
// stores, so that a decode step of packed projections runs without norm, activation or addition kernels.
//
// Super-block (144 bytes, 256 weights): fp16 d, fp16 dmin, 12 bytes of 6-bit scales / mins for 8 sub-blocks of 32,
// 128 bytes of nibbles in four 32-byte chunks; in chunk j the low nibbles are weights 64j .. 64j+31 (sub-block 2j) and
// the high nibbles weights 64j+32 .. 64j+63 (sub-block 2j+1). w = d * sc * q - dmin * m.
#include "common.cuh"
#include "gemm_tcgen05.cuh"

#include <cuda_fp16.h>

#include <algorithm>
#include <cstdlib>

namespace swb {

SWB_REGISTER_STATUS_UNIT(gemv_q4k_chain);

namespace {

constexpr int GV_THREADS = 512;
constexpr int GV_WARPS = GV_THREADS / 32;
constexpr int GV_ROWS = 16;                    // weight rows of a tile
constexpr int GV_ROUND = 16;                   // tiles of a CTA whose sums are in shared memory at a time
constexpr int GV_TOK_STRIDE = 20;              // floats between the tokens of a part: keeps the banks of a fragment's four columns apart
constexpr int GV_PART = 8 * GV_TOK_STRIDE;
constexpr int GV_STAGE = 8 * 336;              // 16 rows of 144 bytes, an odd row 192 bytes behind its even one: eight lanes' reads meet no bank twice
constexpr int GV_SMEM_MAX = 226 * 1024;

struct GvParams {
  const uint8_t* w;
  const void* a;                               // bf16, or fp32 (a_f32)
  void* out;                                   // bf16, or fp32 (out_f32) as the residual
  const bf16* bias;
  const void* residual;
  const unsigned long long* ssq_in;
  unsigned long long *ssq_out, *ssq_zero;
  float norm_scale, norm_eps;                  // 2^-24 / width of the norm
  long long row_bytes;
  int lda, ldd, ld_res, N, K, act, a_f32, out_f32;
  int stages, passes, kb_pass;                 // passes over the reduction index, super-blocks of one
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void mma_f16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same onto zeros
__device__ __forceinline__ void mma_f16_first(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }

// A row's super-block header: block scales as fp32 and the lane's two minima as f16, both times 2^-24.
struct RowScales {
  float sc[8], d, dmin;
  uint32_t mins;
};
// msel: bytes 2 (tig mod 2) and the next one, each under a zero byte
__device__ __forceinline__ RowScales decode_header(const uint4 h, uint32_t msel, bool upper) {
  RowScales r;
  const float2 dd = __half22float2(bits_h2(h.x));
  r.d = dd.x * 281474976710656.f, r.dmin = dd.y * 16777216.f;      // takes the 2^-48 of code and scale, and the 2^-24 of a minimum, away again
  const uint32_t s_lo = h.y & 0x3f3f3f3fu, s_hi = (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u);
  const uint32_t m = upper ? ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u) : h.z & 0x3f3f3f3fu;
  const uint32_t two[4] = {__byte_perm(s_lo, 0, 0x4140), __byte_perm(s_lo, 0, 0x4342), __byte_perm(s_hi, 0, 0x4140), __byte_perm(s_hi, 0, 0x4342)};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(bits_h2(two[i]));
    r.sc[2 * i] = f.x, r.sc[2 * i + 1] = f.y;
  }
  r.mins = __byte_perm(m, 0, msel);
  return r;
}

// Shared memory: activations [super-block of the pass][T][8 blocks][4 lanes] uint4, blocks of odd tokens swapped pairwise (eight lanes read two
// tokens: other banks), their block sums [super-block][T][4] uint2, powers of two
// [super-block][8] float, parts [GV_ROUND + GV_WARPS][8][GV_TOK_STRIDE] float, stages [warp][stages][GV_STAGE].
size_t gv_act_bytes(int T, int kb) { return (size_t)kb * (512 * T + 32 * T + 32); }
constexpr size_t GV_PART_BYTES = (size_t)(GV_ROUND + GV_WARPS) * GV_PART * 4;

template <int T>
__global__ void __launch_bounds__(GV_THREADS, 1) gemv_q4k_chain_kernel(const GvParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint4* act = reinterpret_cast<uint4*>(smem);
  uint2* sums = reinterpret_cast<uint2*>(act + (size_t)p.kb_pass * 32 * T);
  float* pow2 = reinterpret_cast<float*>(sums + (size_t)p.kb_pass * 4 * T);
  float* parts = pow2 + p.kb_pass * 8;
  uint8_t* ring = reinterpret_cast<uint8_t*>(parts + (GV_ROUND + GV_WARPS) * GV_PART);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
  const int kb = p.K / 256, tiles = (p.N + GV_ROWS - 1) / GV_ROWS;
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;      // tiles of this CTA, every gridDim-th
  const int rounds = (mine + GV_ROUND - 1) / GV_ROUND, per_round = (mine + rounds - 1) / rounds;

  // ---- the copies of a step: 144 pieces of 16 bytes, lane i takes pieces i, i + 32, .. ----
  const uint32_t my_ring = smem_u32(ring) + (uint32_t)(warp * p.stages * GV_STAGE);
  uint32_t dst[5], src[5];      // 16 rows are less than 4 GB
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    const int i = lane + 32 * j, r = i / 9;
    dst[j] = my_ring + (uint32_t)((r >> 1) * 336 + (r & 1) * 192 + (i - r * 9) * 16);
    src[j] = (uint32_t)(r * p.row_bytes) + (uint32_t)(i - r * 9) * 16;
  }
  auto request = [&](int tile_local, int sb, int slot) {
    const int row0 = ((int)blockIdx.x + tile_local * (int)gridDim.x) * GV_ROWS, left = p.N - 1 - row0;
    const uint8_t* base = p.w + (long long)row0 * p.row_bytes + (long long)sb * 144;
    const uint32_t at = (uint32_t)(slot * GV_STAGE);
    if (left >= GV_ROWS - 1) {
#pragma unroll
      for (int j = 0; j < 5; ++j)
        if (j < 4 || lane < 16) cp_async16(dst[j] + at, base + src[j]);
    } else {                         // rows past the last one repeat it (their results are not stored)
      for (int j = 0; j < 5; ++j) {
        const int i = lane + 32 * j, r = i / 9;
        if (i < 144) cp_async16(my_ring + (uint32_t)((r >> 1) * 336 + (r & 1) * 192 + (i - r * 9) * 16) + at, base + (long long)min(r, left) * p.row_bytes + (i - r * 9) * 16);
      }
    }
  };

  // ---- fragment constants of this lane ----
  const int tok = min(g, T - 1);                          // column of B; columns past T repeat the last token
  const uint32_t m2 = (uint32_t)(tig & 1) * 2, msel = m2 | (4u << 4) | ((m2 + 1) << 8) | (4u << 12);
  const bool upper = tig >= 2;
  const uint8_t* rows_at = ring + (size_t)warp * p.stages * GV_STAGE + (g >> 1) * 336 + (g & 1) * 192;     // row g; row g + 8 is 4 * 336 further

  bool waited = false;
  for (int round = 0; round < rounds; ++round) {
    const int t0 = round * per_round, nt = min(per_round, mine - t0);
    // results of a round: a thread per (tile, token, pair of rows), eight neighbours have a tile's token
    constexpr int ITEMS = (GV_ROUND * T * 8 + GV_THREADS - 1) / GV_THREADS;
    float y[ITEMS][2] = {}, rms[ITEMS];
    for (int pass = 0; pass < p.passes; ++pass) {
      const int k0 = pass * p.kb_pass, nk = min(p.kb_pass, kb - k0);
      const int total = nt * nk, u0 = total * warp / GV_WARPS, u1 = total * (warp + 1) / GV_WARPS;
      int rt = u0 / nk, rs = u0 - rt * nk;                // next step to request
      int ru = u0;
      auto request_next = [&](int slot) {
        if (ru < u1) {
          request(t0 + rt, k0 + rs, slot);
          ++ru;
          if (++rs == nk) rs = 0, ++rt;
        }
        cp_async_commit();                                // a group per step, empty ones too: the count of groups in flight stays fixed
      };
      for (int s = 0; s < p.stages; ++s) request_next(s);

      if (!waited) {
        pdl_wait(TL_GEMM_QUANT);
        pdl_launch_dependents();
        waited = true;
        if (p.ssq_zero && blockIdx.x == 0 && threadIdx.x < 64) p.ssq_zero[threadIdx.x] = 0ull;
      }
      // ---- activations of this pass: a warp per (token, super-block), a lane has eight neighbours ----
      if (round == 0 || p.passes > 1) {
        constexpr int AHEAD = 4;                          // units of a warp whose loads are on their way together: one by one each waits for L2
        for (int i0 = warp; i0 < T * nk; i0 += AHEAD * GV_WARPS) {
          uint4 raw[AHEAD][2];
#pragma unroll
          for (int n = 0; n < AHEAD; ++n) {
            const int i = min(i0 + n * GV_WARPS, T * nk - 1);
            const size_t at = (size_t)(i % T) * p.lda + (size_t)(k0 + i / T) * 256 + lane * 8;
            if (p.a_f32) {
              raw[n][0] = *reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(p.a) + at);
              raw[n][1] = *reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(p.a) + at + 4);
            } else {
              raw[n][0] = *reinterpret_cast<const uint4*>(reinterpret_cast<const bf16*>(p.a) + at);
            }
          }
#pragma unroll
          for (int n = 0; n < AHEAD; ++n) {
          const int i = i0 + n * GV_WARPS, t = i % T, sb = i / T;
          if (i >= T * nk) break;                         // the whole warp
          const uint4 r0 = raw[n][0], r1 = raw[n][1];
          float v[8];
          if (p.a_f32) {
            v[0] = __uint_as_float(r0.x), v[1] = __uint_as_float(r0.y), v[2] = __uint_as_float(r0.z), v[3] = __uint_as_float(r0.w);
            v[4] = __uint_as_float(r1.x), v[5] = __uint_as_float(r1.y), v[6] = __uint_as_float(r1.z), v[7] = __uint_as_float(r1.w);
          } else {
            const uint32_t w[4] = {r0.x, r0.y, r0.z, r0.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) v[2 * e] = __uint_as_float(w[e] << 16), v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
          }
          float top = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) top = fmaxf(top, fabsf(v[e]));
          top = warp_max(top);
          const int exp = min(9 - ((int)(__float_as_uint(top) >> 23) - 127), 126);
          const int block = lane >> 2, high = block & 1;
          const float put = __uint_as_float((uint32_t)(127 + exp) << 23) * (high ? 0.0625f : 1.f);
          float sum = 0.f;                                // of what the product sees
          uint32_t f[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {                   // elements as the nibbles of a word pair up: (0, 2), (1, 3), (4, 6), (5, 7)
            const int e = (q >> 1) * 4 + (q & 1);
            const __half2 h = __floats2half2_rn(v[e] * put, v[e + 2] * put);
            const float2 seen = __half22float2(h);
            sum += seen.x + seen.y;
            f[q] = h2_bits(h);
          }
          act[(sb * T + t) * 32 + (lane ^ ((t & 1) << 2))] = make_uint4(f[0], f[1], f[2], f[3]);
          sum += __shfl_xor_sync(0xffffffffu, sum, 1);
          sum += __shfl_xor_sync(0xffffffffu, sum, 2);
          if ((lane & 3) == 0) {
            sum *= high ? 16.f : 1.f;
            const __half s_hi = __float2half_rn(sum), s_lo = __float2half_rn(sum - __half2float(s_hi));
            __half* to = reinterpret_cast<__half*>(sums + (size_t)(sb * T + t) * 4 + (block >> 1)) + (block & 1);
            to[0] = s_hi, to[2] = s_lo;
          }
          if (lane == 0) pow2[sb * 8 + t] = __uint_as_float((uint32_t)(127 - exp) << 23);
          }
        }
      }
      __syncthreads();

      // ---- the steps of this warp ----
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
      int lt = u0 / nk, ls = u0 - lt * nk, slot = 0;
      for (int u = u0; u < u1; ++u) {
        if (p.stages == 4) cp_async_wait<3>();
        else if (p.stages == 3) cp_async_wait<2>();
        else cp_async_wait<1>();
        __syncwarp();
        const uint8_t* at = rows_at + slot * GV_STAGE;
        uint4 h[2];                                       // [row g | row g + 8]
        uint2 q[2][4];                                    // eight bytes of each chunk of 32
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          h[r] = *reinterpret_cast<const uint4*>(at + r * 4 * 336);
#pragma unroll
          for (int j = 0; j < 4; ++j) q[r][j] = *reinterpret_cast<const uint2*>(at + r * 4 * 336 + 16 + j * 32 + tig * 8);
        }
        __syncwarp();                                     // all lanes have read the stage
        request_next(slot);
        if (++slot == p.stages) slot = 0;

        const RowScales s0 = decode_header(h[0], msel, upper), s1 = decode_header(h[1], msel, upper);
        float sum[4] = {0.f, 0.f, 0.f, 0.f}, low[4];
        const uint4 *b_low = act + (ls * T + tok) * 32 + tig + ((tok & 1) << 2), *b_high = act + (ls * T + tok) * 32 + tig + ((~tok & 1) << 2);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 bl = b_low[j * 8], bh = b_high[j * 8];
          const uint32_t x = q[0][j].x, y = q[1][j].x, u0 = q[0][j].y, u1 = q[1][j].y;
          const uint32_t x8 = x >> 8, y8 = y >> 8, u08 = u0 >> 8, u18 = u1 >> 8;
          constexpr uint32_t LO = 0x000f000fu, HI = 0x00f000f0u;
          float a[4], b[4];
          mma_f16_first(a, x & LO, y & LO, x8 & LO, y8 & LO, bl.x, bl.y);
          mma_f16_first(b, x & HI, y & HI, x8 & HI, y8 & HI, bh.x, bh.y);
          mma_f16(a, u0 & LO, u1 & LO, u08 & LO, u18 & LO, bl.z, bl.w);
          mma_f16(b, u0 & HI, u1 & HI, u08 & HI, u18 & HI, bh.z, bh.w);
          sum[0] = fmaf(s0.sc[2 * j], a[0], fmaf(s0.sc[2 * j + 1], b[0], sum[0]));
          sum[1] = fmaf(s0.sc[2 * j], a[1], fmaf(s0.sc[2 * j + 1], b[1], sum[1]));
          sum[2] = fmaf(s1.sc[2 * j], a[2], fmaf(s1.sc[2 * j + 1], b[2], sum[2]));
          sum[3] = fmaf(s1.sc[2 * j], a[3], fmaf(s1.sc[2 * j + 1], b[3], sum[3]));
        }
        const uint2 bs = sums[(size_t)(ls * T + tok) * 4 + tig];
        mma_f16_first(low, s0.mins, s1.mins, s0.mins, s1.mins, bs.x, bs.y);
        const float2 e2 = *reinterpret_cast<const float2*>(pow2 + ls * 8 + tig * 2);
        acc[0] = fmaf(e2.x, s0.d * sum[0] - s0.dmin * low[0], acc[0]);
        acc[1] = fmaf(e2.y, s0.d * sum[1] - s0.dmin * low[1], acc[1]);
        acc[2] = fmaf(e2.x, s1.d * sum[2] - s1.dmin * low[2], acc[2]);
        acc[3] = fmaf(e2.y, s1.d * sum[3] - s1.dmin * low[3], acc[3]);
        if (++ls == nk || u + 1 == u1) {                  // the end of this warp's part of the tile: part number tile + warp, in order along the line
          float* part = parts + (size_t)(lt + warp) * GV_PART;
          part[tig * 2 * GV_TOK_STRIDE + g] = acc[0];
          part[(tig * 2 + 1) * GV_TOK_STRIDE + g] = acc[1];
          part[tig * 2 * GV_TOK_STRIDE + g + 8] = acc[2];
          part[(tig * 2 + 1) * GV_TOK_STRIDE + g + 8] = acc[3];
          acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
          ls = 0, ++lt;
        }
      }
      cp_async_wait<0>();
      __syncthreads();
#pragma unroll
      for (int it = 0; it < ITEMS; ++it) {
        const int i = it * GV_THREADS + threadIdx.x, rest = i >> 3, t = rest % T, first = rest / T * nk, end = first + nk;
        if (rest / T >= nt) continue;
        // warps whose parts of the line meet this tile: warp w has [total w / 16, total (w + 1) / 16)
        int w = first * GV_WARPS / total;
        while (total * (w + 1) / GV_WARPS <= first) ++w;
        for (; w < GV_WARPS && total * w / GV_WARPS < end; ++w) {
          if (total * w / GV_WARPS == total * (w + 1) / GV_WARPS) continue;      // fewer steps than warps: this one had none
          const float2 f = *reinterpret_cast<const float2*>(parts + (size_t)(rest / T + w) * GV_PART + t * GV_TOK_STRIDE + (i & 7) * 2);
          y[it][0] += f.x, y[it][1] += f.y;
        }
      }
    }

#pragma unroll
    for (int it = 0; it < ITEMS; ++it)
      rms[it] = p.ssq_in ? rsqrtf((float)__ldcg(p.ssq_in + ((it * GV_THREADS + threadIdx.x) >> 3) % T) * p.norm_scale + p.norm_eps) : 1.f;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      const int i = it * GV_THREADS + threadIdx.x, pair = i & 7, t = (i >> 3) % T, lt = (i >> 3) / T;
      const int n = ((int)blockIdx.x + (t0 + lt) * (int)gridDim.x) * GV_ROWS + pair * 2;
      float y0 = y[it][0], y1 = y[it][1], ss = 0.f;
      if (lt < nt && n < p.N) {
        const bool two = n + 1 < p.N;
        if (p.ssq_in) y0 *= rms[it], y1 *= rms[it];
        if (p.bias) y0 += __bfloat162float(p.bias[n]), y1 += two ? __bfloat162float(p.bias[n + 1]) : 0.f;
        if (gemm_act_pairs(p.act)) {                       // N is even
          reinterpret_cast<bf16*>(p.out)[(size_t)t * p.ldd + (n >> 1)] = __float2bfloat16((p.act == SWB_ACT_GEGLU_PAIRS ? gelu_tanh_f(y0) : silu_f(y0)) * y1);
        } else {
          const size_t from = (size_t)t * p.ld_res + n, to = (size_t)t * p.ldd + n;
          if (p.out_f32) {
            const float* res = reinterpret_cast<const float*>(p.residual);
            float* out = reinterpret_cast<float*>(p.out);
            if (res) y0 += res[from], y1 += two ? res[from + 1] : 0.f;
            out[to] = y0;
            if (two) out[to + 1] = y1;
          } else {
            const bf16* res = reinterpret_cast<const bf16*>(p.residual);
            bf16* out = reinterpret_cast<bf16*>(p.out);
            if (res) y0 += __bfloat162float(res[from]), y1 += two ? __bfloat162float(res[from + 1]) : 0.f;
            const bf16 o0 = __float2bfloat16(y0), o1 = __float2bfloat16(y1);
            out[to] = o0;
            if (two) out[to + 1] = o1;
            y0 = __bfloat162float(o0), y1 = __bfloat162float(o1);
          }
          ss = y0 * y0 + (two ? y1 * y1 : 0.f);
        }
      }
      if (p.ssq_out) {      // sum of squares of exactly what was stored, 2^-24 fixed point: the order of the CTAs does not matter
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lt < nt && pair == 0) atomicAdd(p.ssq_out + t, __float2ull_rn(fminf(ss, 5.0e11f) * 16777216.f));
      }
    }
  }
}

// Passes over the reduction index and stages of a ring for T tokens of K: the fewest passes that leave two stages, then as many stages as fit, up to four.
bool gv_plan(int T, int K, int* passes, int* kb_pass, int* stages) {
  const int kb = K / 256;
  for (int n = 1; n <= 4; ++n) {
    const int per = (kb + n - 1) / n;
    if ((long long)per * (n - 1) >= kb) continue;         // no empty pass
    const size_t fixed = gv_act_bytes(T, per) + GV_PART_BYTES;
    for (int s = 4; s >= 2; --s) {
      if (fixed + (size_t)s * GV_WARPS * GV_STAGE <= GV_SMEM_MAX) {
        *passes = n, *kb_pass = per, *stages = s;
        return true;
      }
    }
  }
  return false;
}

template <int T>
int launch_gv(const GvParams& p, cudaStream_t stream) {
  auto kern = gemv_q4k_chain_kernel<T>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GV_SMEM_MAX);
    if (e != cudaSuccess) return -(int)e;
    configured[dev] = true;
  }
  const size_t smem = gv_act_bytes(T, p.kb_pass) + GV_PART_BYTES + (size_t)p.stages * GV_WARPS * GV_STAGE;
  const int ctas = std::min(device_sm_count(), (p.N + GV_ROWS - 1) / GV_ROWS);
  return launch_kernel(kern, dim3(ctas), dim3(GV_THREADS), smem, stream, p);
}

int launch_any(GvParams& p, int T, cudaStream_t stream) {
  if (!gv_plan(T, p.K, &p.passes, &p.kb_pass, &p.stages)) return -3;
  switch (T) {
    case 1: return launch_gv<1>(p, stream);
    case 2: return launch_gv<2>(p, stream);
    case 3: return launch_gv<3>(p, stream);
    case 4: return launch_gv<4>(p, stream);
    case 5: return launch_gv<5>(p, stream);
    case 6: return launch_gv<6>(p, stream);
    case 7: return launch_gv<7>(p, stream);
    case 8: return launch_gv<8>(p, stream);
    default: return -3;
  }
}

GvParams gv_params(const void* A, int lda, const void* Wq, void* D, int ldd, int N, int K, const void* bias) {
  GvParams p{};
  p.w = reinterpret_cast<const uint8_t*>(Wq);
  p.a = A;
  p.out = D;
  p.bias = reinterpret_cast<const bf16*>(bias);
  p.row_bytes = (long long)K / 256 * 144;
  p.lda = lda;
  p.ldd = ldd;
  p.N = N;
  p.K = K;
  return p;
}

}  // namespace

// Whether this kernel takes the problem: T in 1..8, K a multiple of 256 up to what at most four passes hold (28 672 at eight tokens),
// 16-byte aligned operands.
static bool gemv_q4k_chain_accepts(int T, int K, int lda, const void* A, const void* Wq) {
  static const bool off = [] { const char* e = getenv("SWB_Q4K_GEMV"); return e && e[0] == '0'; }();
  if (off || T < 1 || T > 8 || K <= 0 || K % 256 != 0 || lda % 8 != 0) return false;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(Wq) & 15)) return false;
  int passes, kb_pass, stages;
  return gv_plan(T, K, &passes, &kb_pass, &stages);
}

}  // namespace swb

extern "C" {

// 1 when swb_gemv_q4k_normed takes T tokens of K.
int swb_gemv_q4k_supported(int T, int K) { return swb::gemv_q4k_chain_accepts(T, K, 8, nullptr, nullptr) ? 1 : 0; }

// One link of a folded-norm chain (see swb_gemm_bf16_normed) with packed Q4_K weights: D[T <= 8, N] = act(rms * A Wq^T + bias) + residual.
// ssq_in: u64 [64] sums of squares of A's rows in 2^-24 fixed point (rms = 1 / sqrt(sum / norm_dim + eps)); ssq_out: those of what is stored,
// zero at launch; ssq_zero: cleared. act: none or a gated pair (rows in (gate, up) pairs, D [T, N / 2]); residual and ssq_out only without one.
// A is bf16 or (a_f32) fp32, D and the residual bf16 or (out_f32) fp32.
int swb_gemv_q4k_normed(const void* A, int lda, int a_f32, const void* Wq, void* D, int ldd, int out_f32, int T, int N, int K, const void* bias,
                        const void* residual, int ld_res, int act, const void* ssq_in, void* ssq_out, void* ssq_zero, int norm_dim, float eps, void* stream) {
  using namespace swb;
  if (T <= 0 || N <= 0) return 0;
  const bool pairs = act == SWB_ACT_SWIGLU_PAIRS || act == SWB_ACT_GEGLU_PAIRS;
  if (!gemv_q4k_chain_accepts(T, K, lda, A, Wq) || !D || (act != SWB_ACT_NONE && !pairs) || (pairs && (residual || ssq_out || out_f32 || (N & 1))) ||
      (ssq_in && norm_dim <= 0))
    return -3;
  GvParams p = gv_params(A, lda, Wq, D, ldd, N, K, bias);
  p.residual = residual;
  p.a_f32 = a_f32;
  p.out_f32 = out_f32;
  p.ld_res = ld_res;
  p.act = act;
  p.ssq_in = reinterpret_cast<const unsigned long long*>(ssq_in);
  p.ssq_out = reinterpret_cast<unsigned long long*>(ssq_out);
  p.ssq_zero = reinterpret_cast<unsigned long long*>(ssq_zero);
  p.norm_scale = ssq_in ? 1.f / 16777216.f / (float)norm_dim : 0.f;
  p.norm_eps = eps;
  return launch_any(p, T, reinterpret_cast<cudaStream_t>(stream));
}

}  // extern "C"
