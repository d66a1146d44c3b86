// Q4_K matrix-vector kernel for 1..8 tokens: D[T, N] = A[T, K] * dequant(Wq)[N, K]^T (+ bias).
//
// At this size the packed weights are the only stream that matters (4.5 bits per weight) and the arithmetic must not
// cost more than their arrival. The weights are therefore never expanded: the activations are quantised to int8 per
// 32-element block inside the kernel (each CTA does all of them: K * T elements, a few microseconds at most, after
// the first weight loads have been issued), stored in shared memory in the order in which a super-block's nibbles lie,
// and the dot products run on packed-byte integer multiply-adds (dp4a), eight weights per instruction pair. This is the
// numerical scheme of the llama.cpp-derived kernels the reference uses (candle-kernels/src/mmvq_gguf.cu: q8_1
// activations against Q4_K weights), laid out for this machine: one persistent 512-thread CTA per SM, two output rows
// per warp at a time (one for small matrices), every lane owning one 16-byte piece of four super-blocks of them, the loads of the next
// slice in flight while the current one is consumed.
//
// From two tokens on the kernel is bound by shared memory and instruction issue, not by the weights' arrival: a warp-step of four
// super-blocks reads 3 x 16 bytes of activations per lane and token. Two rows share these reads; block scales and sums lie beside
// each other (one load instead of four); dot products start at 1.5 * 2^23 as a bit pattern, so that a subtraction makes them float
// (they stay below 2^22, hence exactly) without the conversion unit. Row pairs go to the SMs in turn, so that all have the same number
// to within one. 6144 + 4096 + 28672 rows of 4096 and 4096 of 14336 at four tokens, 32 times over: an
// 8B decoder's step of 4 tokens went from 3.69 to 3.27 ms.
//
// Super-block (144 bytes, 256 weights): fp16 d, fp16 dmin, 12 bytes of 6-bit scales / mins for 8 sub-blocks of 32,
// 128 bytes of nibbles in four 32-byte chunks; in chunk j the low nibbles are weights 64j .. 64j+31 (sub-block 2j) and
// the high nibbles weights 64j+32 .. 64j+63 (sub-block 2j+1). w = d * sc * q - dmin * m.
#include "common.cuh"

#include <cuda_fp16.h>

#include <algorithm>

namespace swb {

int device_sm_count();   // gemm_tcgen05.cu

SWB_REGISTER_STATUS_UNIT(gemv_q4k);

namespace {

constexpr int GV_THREADS = 512;
constexpr int GV_WARPS = GV_THREADS / 32;

struct GvParams {
  const uint8_t* w;
  const bf16* a;
  bf16* out;
  const bf16* bias;
  long long row_bytes;
  int lda, ldd, N, K, kblocks;
};

__device__ __forceinline__ uint4 ld_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ int dp4a_us(uint32_t u, int s, int acc) {   // unsigned bytes of u times signed bytes of s
  int r;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(u), "r"(s), "r"(acc));
  return r;
}

// Shared memory, per token t:
//   q_lo / q_hi  [K / 2] int8   quantised activations that meet low / high nibbles: super-block sb, piece i -> sb * 128 + i * 16
//   blk          [K / 32] float4  for piece i of super-block sb (chunk j = i / 2), at sb * 8 + i: block scales of sub-blocks 2j and
//                2j + 1, then scale * sum of the 16 quantised activations of the piece among the low and among the high ones
constexpr int GV_FLOAT_BIAS = 0x4B400000;      // 1.5 * 2^23
// GV_ROWS: rows of a warp that share its reads of the activations.
template <int T, int GV_ROWS>
__global__ void __launch_bounds__(GV_THREADS, 1) gemv_q4k_kernel(const GvParams p) {
  constexpr int GV_STEPS = 4 / GV_ROWS;      // warp-steps (of 4 super-blocks) of each row loaded before any is consumed
  extern __shared__ __align__(16) uint8_t smem[];
  const int K = p.K, kb = p.kblocks;
  int8_t* q_lo = reinterpret_cast<int8_t*>(smem);
  int8_t* q_hi = q_lo + (size_t)T * (K / 2);
  float* blk = reinterpret_cast<float*>(q_hi + (size_t)T * (K / 2));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane >> 3, piece = lane & 7;          // super-block within the warp-step, 16-byte piece within it
  const int total_warps = gridDim.x * GV_WARPS;
  const int groups = (p.N + GV_ROWS - 1) / GV_ROWS;
  int row = blockIdx.x + gridDim.x * warp;              // group of rows

  // Work items are (group of rows, slice of 16 / GV_ROWS super-blocks); two register buffers alternate so that the next item's bytes are
  // in flight while the current one is consumed. The first item starts moving before the activations exist.
  const int spr = (kb + GV_STEPS * 4 - 1) / (GV_STEPS * 4);
  uint4 hdrA[GV_ROWS][GV_STEPS], qsA[GV_ROWS][GV_STEPS], hdrB[GV_ROWS][GV_STEPS], qsB[GV_ROWS][GV_STEPS];
  auto issue = [&](uint4 (*hdr)[GV_STEPS], uint4 (*qs)[GV_STEPS], int r, int sl) {
#pragma unroll
    for (int e = 0; e < GV_ROWS; ++e) {      // a row past the last one repeats it (its result is not stored)
      const uint8_t* rp = p.w + (size_t)min(r * GV_ROWS + e, p.N - 1) * p.row_bytes;
#pragma unroll
      for (int s = 0; s < GV_STEPS; ++s) {
        const int b = sl * (GV_STEPS * 4) + s * 4 + sub;
        if (b < kb) {
          const uint8_t* at = rp + (size_t)b * 144;
          hdr[e][s] = ld_stream(at);
          qs[e][s] = ld_stream(at + 16 + piece * 16);
        }
      }
    }
  };
  if (row < groups) issue(hdrA, qsA, row, 0);

  pdl_wait(TL_GEMM_QUANT);
  // ---- quantise the activations: one thread per (token, 32-element block) ----
  const int nblk = K / 32;
  for (int idx = threadIdx.x; idx < T * nblk; idx += GV_THREADS) {
    const int t = idx / nblk, b = idx - t * nblk;
    const uint4* src = reinterpret_cast<const uint4*>(p.a + (size_t)t * p.lda + b * 32);
    float v[32];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const uint4 x = src[c];
      const uint32_t wds[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[c * 8 + e * 2] = __uint_as_float(wds[e] << 16);
        v[c * 8 + e * 2 + 1] = __uint_as_float(wds[e] & 0xFFFF0000u);
      }
    }
    float amax = 0.f;
#pragma unroll
    for (int e = 0; e < 32; ++e) amax = fmaxf(amax, fabsf(v[e]));
    const float d = amax * (1.f / 127.f), inv = amax > 0.f ? 127.f / amax : 0.f;
    // block b = sb * 8 + 2j + h: h = 0 meets low nibbles, h = 1 high nibbles of chunk j
    const int sb = b >> 3, j = (b >> 1) & 3, h = b & 1;
    int8_t* qd = (h ? q_hi : q_lo) + (size_t)t * (K / 2) + sb * 128 + j * 32;
    uint32_t packed[8];
    int sums[2] = {0, 0};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint32_t wd = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int q = __float2int_rn(v[c * 4 + e] * inv);
        sums[c >> 2] += q;
        wd |= (uint32_t)(q & 0xFF) << (8 * e);
      }
      packed[c] = wd;
    }
    reinterpret_cast<uint4*>(qd)[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    reinterpret_cast<uint4*>(qd)[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    float* at = blk + ((size_t)t * (K / 32) + sb * 8 + j * 2) * 4 + h;
    at[0] = at[4] = d;
    at[2] = d * (float)sums[0];
    at[6] = d * (float)sums[1];
  }
  __syncthreads();
  pdl_launch_dependents();

  const int j = piece >> 1;   // chunk of this lane's piece: sub-blocks 2j (low nibbles) and 2j + 1 (high)
  float acc[GV_ROWS][T];
  auto consume = [&](const uint4 (*hdr)[GV_STEPS], const uint4 (*qs)[GV_STEPS], int r, int sl) {
    if (sl == 0) {
#pragma unroll
      for (int e = 0; e < GV_ROWS; ++e)
#pragma unroll
        for (int t = 0; t < T; ++t) acc[e][t] = 0.f;
    }
#pragma unroll
    for (int s = 0; s < GV_STEPS; ++s) {
      const int b = sl * (GV_STEPS * 4) + s * 4 + sub;
      if (b < kb) {
        float sc[GV_ROWS][2], mn[GV_ROWS][2];
        uint32_t lo[GV_ROWS][4], hi[GV_ROWS][4];
#pragma unroll
        for (int w = 0; w < GV_ROWS; ++w) {
          const uint4 h4 = hdr[w][s], q = qs[w][s];
          const __half2 dd = *reinterpret_cast<const __half2*>(&h4.x);
          const float d = __low2float(dd), dmin = __high2float(dd);
          auto sbyte = [&](int i) -> uint32_t {
            const uint32_t wv = i < 4 ? h4.y : (i < 8 ? h4.z : h4.w);
            return (wv >> ((i & 3) * 8)) & 0xFFu;
          };
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int k = j * 2 + e;
            uint32_t scv, mv;
            if (j < 2) {
              scv = sbyte(k) & 63u;
              mv = sbyte(k + 4) & 63u;
            } else {
              scv = (sbyte(k + 4) & 0xFu) | ((sbyte(k - 4) >> 6) << 4);
              mv = (sbyte(k + 4) >> 4) | ((sbyte(k) >> 6) << 4);
            }
            sc[w][e] = d * (float)scv;
            mn[w][e] = dmin * (float)mv;
          }
          const uint32_t wq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            lo[w][c] = wq[c] & 0x0F0F0F0Fu;
            hi[w][c] = (wq[c] >> 4) & 0x0F0F0F0Fu;
          }
        }
#pragma unroll
        for (int t = 0; t < T; ++t) {
          const int4 a0 = *reinterpret_cast<const int4*>(q_lo + (size_t)t * (K / 2) + b * 128 + piece * 16);
          const int4 a1 = *reinterpret_cast<const int4*>(q_hi + (size_t)t * (K / 2) + b * 128 + piece * 16);
          const float4 f = *reinterpret_cast<const float4*>(blk + ((size_t)t * (K / 32) + b * 8 + piece) * 4);
#pragma unroll
          for (int w = 0; w < GV_ROWS; ++w) {
            const int s0 = dp4a_us(lo[w][3], a0.w, dp4a_us(lo[w][2], a0.z, dp4a_us(lo[w][1], a0.y, dp4a_us(lo[w][0], a0.x, GV_FLOAT_BIAS))));
            const int s1 = dp4a_us(hi[w][3], a1.w, dp4a_us(hi[w][2], a1.z, dp4a_us(hi[w][1], a1.y, dp4a_us(hi[w][0], a1.x, GV_FLOAT_BIAS))));
            const float bias = __int_as_float(GV_FLOAT_BIAS);
            acc[w][t] = fmaf(sc[w][0] * f.x, __int_as_float(s0) - bias, acc[w][t]);
            acc[w][t] = fmaf(sc[w][1] * f.y, __int_as_float(s1) - bias, acc[w][t]);
            acc[w][t] = fmaf(-mn[w][0], f.z, acc[w][t]);
            acc[w][t] = fmaf(-mn[w][1], f.w, acc[w][t]);
          }
        }
      }
    }
    if (sl == spr - 1) {
#pragma unroll
      for (int w = 0; w < GV_ROWS; ++w) {
        const int n = r * GV_ROWS + w;
#pragma unroll
        for (int t = 0; t < T; ++t) {
          float v = acc[w][t];
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
          if (lane == t && n < p.N) {
            if (p.bias) v += __bfloat162float(p.bias[n]);
            p.out[(size_t)t * p.ldd + n] = __float2bfloat16(v);
          }
        }
      }
    }
  };
  auto advance = [&](int& r, int& sl) {
    if (++sl == spr) {
      sl = 0;
      r += total_warps;
    }
  };
  int sl = 0;
  while (row < groups) {
    int rn = row, sn = sl;
    advance(rn, sn);
    if (rn < groups) issue(hdrB, qsB, rn, sn);
    consume(hdrA, qsA, row, sl);
    row = rn;
    sl = sn;
    if (row >= groups) break;
    advance(rn, sn);
    if (rn < groups) issue(hdrA, qsA, rn, sn);
    consume(hdrB, qsB, row, sl);
    row = rn;
    sl = sn;
  }
}

constexpr int GV_SMEM_MAX = 226 * 1024;
size_t gv_smem(int T, int K) { return (size_t)T * ((size_t)K + (size_t)(K / 32) * 16); }

template <int T, int GV_ROWS>
int launch_gv_rows(const GvParams& p, cudaStream_t stream) {
  const size_t smem = gv_smem(T, p.K);
  auto kern = gemv_q4k_kernel<T, GV_ROWS>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GV_SMEM_MAX);
    if (e != cudaSuccess) return -(int)e;
    configured[dev] = true;
  }
  if (smem > GV_SMEM_MAX) return -3;
  const int ctas = std::min(device_sm_count(), (p.N + GV_WARPS * GV_ROWS - 1) / (GV_WARPS * GV_ROWS));
  return launch_kernel(kern, dim3(ctas), dim3(GV_THREADS), smem, stream, p);
}

// Two rows a warp where there are more rows than warps on the chip. With fewer the second row only takes a warp's place: 2048 x 2048 at
// 4 tokens takes 3.7 us with a row per warp and 4.3 with two, 4096 x 4096 8.3 and 7.5.
template <int T>
int launch_gv(const GvParams& p, cudaStream_t stream) {
  return p.N <= device_sm_count() * GV_WARPS ? launch_gv_rows<T, 1>(p, stream) : launch_gv_rows<T, 2>(p, stream);
}

}  // namespace

// Whether the matrix-vector kernel takes this problem: T in 1..8, K a multiple of 256 whose activations fit in shared
// memory, 16-byte aligned operands.
bool gemv_q4k_accepts(int T, int K, int lda, const void* A, const void* Wq) {
  if (T < 1 || T > 8 || K <= 0 || K % 256 != 0 || lda % 8 != 0) return false;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(Wq) & 15)) return false;
  return gv_smem(T, K) <= GV_SMEM_MAX;
}

int gemv_q4k_launch(const void* A, int lda, const void* Wq, void* D, int ldd, int T, int N, int K, const void* bias,
                    cudaStream_t stream) {
  GvParams p{};
  p.w = reinterpret_cast<const uint8_t*>(Wq);
  p.a = reinterpret_cast<const bf16*>(A);
  p.out = reinterpret_cast<bf16*>(D);
  p.bias = reinterpret_cast<const bf16*>(bias);
  p.row_bytes = (long long)K / 256 * 144;
  p.lda = lda;
  p.ldd = ldd;
  p.N = N;
  p.K = K;
  p.kblocks = K / 256;
  cudaStream_t st = stream;
  switch (T) {
    case 1: return launch_gv<1>(p, st);
    case 2: return launch_gv<2>(p, st);
    case 3: return launch_gv<3>(p, st);
    case 4: return launch_gv<4>(p, st);
    case 5: return launch_gv<5>(p, st);
    case 6: return launch_gv<6>(p, st);
    case 7: return launch_gv<7>(p, st);
    case 8: return launch_gv<8>(p, st);
    default: return -3;
  }
}

}  // namespace swb
