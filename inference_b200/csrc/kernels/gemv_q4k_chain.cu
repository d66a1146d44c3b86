// Q4_K products of a decode step that are chained: D[T <= 8, N] = epilogue(A[T, K] * dequant(Wq)[N, K]^T).
//
// At this size the packed weights are the only stream that matters (4.5 bits per weight), and the arithmetic must not cost more than
// their arrival. A step of it is 16 weight rows x one super-block of 256 x 8 tokens, in a warp of its own: mma.sync.m16n8k16 in f16
// on operands that are exact.
//   weights      q * sc (4-bit code times 6-bit block scale, at most 945) is a whole number that f16 holds exactly. A code becomes f16 by
//                or-ing it under the exponent of 1024; one packed multiply-add takes the 1024 away again and applies the scale. High nibbles
//                stay 16 times too large, their activations are 16 times too small.
//   activations  bf16 times a power of two of the (token, super-block) that takes the largest to 2^9 .. 2^10: f16 holds them exactly down to 2^-19 of
//                that one, and below it to 2^-35 of it. Those of an fp32 stream are rounded to 11 bits.
//   minima       sum over blocks of m * (sum of the block's activations): one more MMA per super-block, the sums as two f16 parts.
// The order of the reduction index is free as long as both operands agree, so a lane multiplies the 16-byte pieces of a row as they lie
// and has four block scales to decode per row and super-block. d and dmin are applied to the fp32 result of each super-block.
// The cost per weight does not depend on T. 28672 x 4096 takes 21.1 / 23.3 / 25.2 us at 1 / 4 / 8 tokens, 4096 x 14336 14.7 / 20.0 / 29.0; the kernel of single
// products (gemv_q4k.cu: dp4a on activations that are rounded to int8) 23.5 / 34.2 / 50.4 and 13.5 / 21.6 / 32.2. What is left above the weights' arrival
// (10.2 and 5.1 us) is latency: half of the issue slots are idle with four warps to a scheduler, and about 5 us of a launch lie before the
// first and behind the last weight. A decode step of 4 tokens of an 8B decoder went from 3.26 to 2.55 ms, its error against 64 bits from 0.029 to 0.004.
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
__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2*>(&u); }
// (v & mask) | 0x6400 in both halves: whole numbers on top of 1024
__device__ __forceinline__ uint32_t on_1024(uint32_t v, uint32_t mask) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, 0x64006400, 0xEA;" : "=r"(r) : "r"(v), "r"(mask));
  return r;
}

// What a lane needs of one row's super-block header.
struct RowScales {
  __half2 sc[4], off[4];       // [set * 2 + (low | high nibbles)]: block scale, -1024 times it
  uint32_t mins;               // two minima as f16
  float d, dmin;
};
// sel0 / sel1: byte 2 (tig / 2) and the next one, each twice under 0x64; msel: bytes 2 (tig mod 2) and the next one.
__device__ __forceinline__ RowScales decode_header(const uint4 h, uint32_t sel0, uint32_t sel1, uint32_t msel, bool upper) {
  RowScales r;
  const float2 dd = __half22float2(bits_h2(h.x));
  r.d = dd.x, r.dmin = dd.y;
  const uint32_t s_lo = h.y & 0x3f3f3f3fu, m_lo = h.z & 0x3f3f3f3fu;
  const uint32_t s_hi = (h.w & 0x0f0f0f0fu) | ((h.y >> 2) & 0x30303030u), m_hi = ((h.w >> 4) & 0x0f0f0f0fu) | ((h.z >> 2) & 0x30303030u);
  const __half2 base = bits_h2(0x64006400u), minus = bits_h2(0xE400E400u);      // 1024, -1024
  const uint32_t w[4] = {__byte_perm(s_lo, 0x64646464u, sel0), __byte_perm(s_lo, 0x64646464u, sel1), __byte_perm(s_hi, 0x64646464u, sel0),
                         __byte_perm(s_hi, 0x64646464u, sel1)};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    r.sc[i] = __hsub2(bits_h2(w[i]), base);
    r.off[i] = __hmul2(r.sc[i], minus);
  }
  r.mins = h2_bits(__hsub2(bits_h2(__byte_perm(upper ? m_hi : m_lo, 0x64646464u, msel)), base));
  return r;
}

// Shared memory: activations [super-block of the pass][T][8 parts][4 lanes] uint4, parts of odd tokens swapped pairwise (eight lanes read two
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
  const uint32_t b2 = (uint32_t)(tig >> 1) * 2, m2 = (uint32_t)(tig & 1) * 2;
  const uint32_t sel0 = b2 | (4u << 4) | (b2 << 8) | (4u << 12), sel1 = (b2 + 1) | (4u << 4) | ((b2 + 1) << 8) | (4u << 12);
  const uint32_t msel = m2 | (4u << 4) | ((m2 + 1) << 8) | (4u << 12);
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
        for (int i = warp; i < T * nk; i += GV_WARPS) {
          const int t = i % T, sb = i / T;
          float v[8];
          const size_t at = (size_t)t * p.lda + (size_t)(k0 + sb) * 256 + lane * 8;
          if (p.a_f32) load_row8(reinterpret_cast<const float*>(p.a) + at, v);
          else load_row8(reinterpret_cast<const bf16*>(p.a) + at, v);
          float top = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) top = fmaxf(top, fabsf(v[e]));
          top = warp_max(top);
          const int exp = min(9 - ((int)(__float_as_uint(top) >> 23) - 127), 126);
          const int block = lane >> 2, piece = (block >> 1) * 2 + ((lane >> 1) & 1), high = block & 1;
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
          act[((sb * T + t) * 8 + (((piece >> 2) * 4 + high * 2 + (lane & 1)) ^ (t & 1))) * 4 + (piece & 3)] = make_uint4(f[0], f[1], f[2], f[3]);
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
        uint4 h[2], q[2][2];                              // [row g | row g + 8][pieces tig | tig + 4]
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint4* row = reinterpret_cast<const uint4*>(at + r * 4 * 336);
          h[r] = row[0];
          q[r][0] = row[1 + tig];
          q[r][1] = row[5 + tig];
        }
        __syncwarp();                                     // all lanes have read the stage
        request_next(slot);
        if (++slot == p.stages) slot = 0;

        const RowScales s0 = decode_header(h[0], sel0, sel1, msel, upper), s1 = decode_header(h[1], sel0, sel1, msel, upper);
        float sum[4] = {0.f, 0.f, 0.f, 0.f}, sum2[4] = {0.f, 0.f, 0.f, 0.f}, low[4] = {0.f, 0.f, 0.f, 0.f};
        const uint4* bp = act + (ls * T + tok) * 32 + tig;
#pragma unroll
        for (int set = 0; set < 2; ++set) {
          const uint32_t w0[4] = {q[0][set].x, q[0][set].y, q[0][set].z, q[0][set].w};
          const uint32_t w1[4] = {q[1][set].x, q[1][set].y, q[1][set].z, q[1][set].w};
          const __half2 scl0 = s0.sc[set * 2], scl1 = s1.sc[set * 2], sch0 = s0.sc[set * 2 + 1], sch1 = s1.sc[set * 2 + 1];
          const __half2 ofl0 = s0.off[set * 2], ofl1 = s1.off[set * 2], ofh0 = s0.off[set * 2 + 1], ofh1 = s1.off[set * 2 + 1];
#pragma unroll
          for (int v = 0; v < 2; ++v) {
            const uint4 bl = bp[((set * 4 + v) ^ (tok & 1)) * 4], bh = bp[((set * 4 + 2 + v) ^ (tok & 1)) * 4];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const uint32_t x = w0[v * 2 + e], y = w1[v * 2 + e], x8 = x >> 8, y8 = y >> 8;
              auto scaled = [](uint32_t w, uint32_t mask, __half2 sc, __half2 off) { return h2_bits(__hfma2(bits_h2(on_1024(w, mask)), sc, off)); };
              mma_f16(sum, scaled(x, 0x000f000fu, scl0, ofl0), scaled(y, 0x000f000fu, scl1, ofl1), scaled(x8, 0x000f000fu, scl0, ofl0),
                      scaled(y8, 0x000f000fu, scl1, ofl1), e ? bl.z : bl.x, e ? bl.w : bl.y);
              mma_f16(sum2, scaled(x, 0x00f000f0u, sch0, ofh0), scaled(y, 0x00f000f0u, sch1, ofh1), scaled(x8, 0x00f000f0u, sch0, ofh0),
                      scaled(y8, 0x00f000f0u, sch1, ofh1), e ? bh.z : bh.x, e ? bh.w : bh.y);
            }
          }
        }
        const uint2 bs = sums[(size_t)(ls * T + tok) * 4 + tig];
        mma_f16(low, s0.mins, s1.mins, s0.mins, s1.mins, bs.x, bs.y);
        const float2 e2 = *reinterpret_cast<const float2*>(pow2 + ls * 8 + tig * 2);
        acc[0] += e2.x * (s0.d * (sum[0] + sum2[0]) - s0.dmin * low[0]);
        acc[1] += e2.y * (s0.d * (sum[1] + sum2[1]) - s0.dmin * low[1]);
        acc[2] += e2.x * (s1.d * (sum[2] + sum2[2]) - s1.dmin * low[2]);
        acc[3] += e2.y * (s1.d * (sum[3] + sum2[3]) - s1.dmin * low[3]);
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
        if (p.bias) y0 += __bfloat162float(p.bias[n]), y1 += two ? __bfloat162float(p.bias[n + 1]) : 0.f;
        if (p.ssq_in) y0 *= rms[it], y1 *= rms[it];
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

// Whether this kernel takes the problem: T in 1..8, K a multiple of 256 up to what at most four passes hold (29 184 at eight tokens),
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
