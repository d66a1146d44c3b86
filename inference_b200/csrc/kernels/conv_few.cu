// The last step of an image decoder: group norm, SiLU and a 3x3 convolution to at most eight channels, in one pass over a bf16 NHWC activation
// (candle-gen-flux/src/vae/native.rs: norm_out, swish, conv_out).
//
// With eight output channels the convolution has no use for a large tile of products: as an implicit GEMM it fetches every activation nine times
// (315 us for 128 channels at 1216 x 832, bound by L2), behind a norm that reads and writes them all (128 us). Here a CTA brings a tile of 8 x 32 pixels
// and its border to shared memory once, normed and activated on the way and rounded to bf16 as the norm's own kernel stores it, and takes the nine
// shifted products from there (ldmatrix + mma.sync.m16n8k16, a warp per row of the tile). Two CTAs to an SM: one loads while the other multiplies. The
// pair takes 212 us (64 x 64 pixels: 15 against 16; 1024 x 1024 of 64 channels: 123 against 258). What is left of it: exponentials and reciprocals of the
// activation (about 80 us with the borders) and shared memory's reads (about 85).
#include "common.cuh"

#include <algorithm>

namespace swb {

int device_sm_count();   // gemm_tcgen05.cu

namespace {

constexpr int CF_THREADS = 256;
constexpr int CF_H = 8, CF_W = 32;                       // output pixels of a tile
constexpr int CF_PX_W = CF_W + 2, CF_PX = (CF_H + 2) * CF_PX_W;

struct FewParams {
  const bf16* x;
  const float* sums;                                     // [n][groups][2]
  const bf16 *gamma, *beta;
  const bf16* w;                                         // [8][9 C], columns (ky, kx, c)
  const bf16* bias;                                      // [8]
  bf16* out;                                             // [n, h, w, 8]
  int n, h, wd, groups;
  float eps;
};

template <int C>
constexpr size_t cf_smem() { return (size_t)CF_PX * C * 2 + (size_t)(9 * C / 16) * 32 * 8; }

template <int C>
__global__ void __launch_bounds__(CF_THREADS, 2) norm_silu_conv_few_kernel(const FewParams p) {
  constexpr int C8 = C / 8, AT_ONCE = CF_THREADS / C8;   // pixels that the CTA loads together
  extern __shared__ __align__(128) uint8_t smem[];
  uint2* frag = reinterpret_cast<uint2*>(smem + (size_t)CF_PX * C * 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int tiles_x = (p.wd + CF_W - 1) / CF_W, tiles_y = (p.h + CF_H - 1) / CF_H, per_image = tiles_x * tiles_y;
  const int total = per_image * p.n;

  pdl_launch_dependents();
  pdl_wait();
  // weights in the order in which the lanes of a product hold them
  for (int i = threadIdx.x; i < 9 * C / 16 * 32; i += CF_THREADS) {
    const int l = i & 31, k = (i >> 5) * 16 + (l & 3) * 2;
    const bf16* row = p.w + (size_t)(l >> 2) * 9 * C + k;
    frag[i] = make_uint2(*reinterpret_cast<const uint32_t*>(row), *reinterpret_cast<const uint32_t*>(row + 8));
  }
  const int v = threadIdx.x % C8, px0 = threadIdx.x / C8;
  float ga[8], be[8], sc[8], sh[8];
  load_row8(p.gamma + v * 8, ga);
  load_row8(p.beta + v * 8, be);
  const float b0 = __bfloat162float(p.bias[t4 * 2]), b1 = __bfloat162float(p.bias[t4 * 2 + 1]);
  int image = -1;
  for (int i = blockIdx.x; i < total; i += gridDim.x) {
    const int tile = total - 1 - i;                      // last pixels first: of what the kernel in front of this one wrote they are the part that L2 still holds
    const int n = tile / per_image, r = tile - n * per_image, ty = r / tiles_x * CF_H, tx = r % tiles_x * CF_W;
    if (n != image) {
      image = n;
      const int cpg = C / p.groups;
      const float cnt = (float)p.h * (float)p.wd * (float)cpg;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float* st = p.sums + ((size_t)n * p.groups + (v * 8 + j) / cpg) * 2;
        const float mean = st[0] / cnt, var = fmaxf(st[1] / cnt - mean * mean, 0.f);
        sc[j] = rsqrtf(var + p.eps) * ga[j];
        sh[j] = be[j] - mean * sc[j];
      }
    }
    __syncthreads();                                     // the products of the tile before have read its pixels
    const uint4* image_at = reinterpret_cast<const uint4*>(p.x + (size_t)n * p.h * p.wd * C) + v;
    constexpr int AHEAD = 4;
    for (int i0 = px0; i0 < CF_PX; i0 += AHEAD * AT_ONCE) {
      uint4 raw[AHEAD];
      bool in[AHEAD];
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int i = i0 + a * AT_ONCE, y = ty - 1 + i / CF_PX_W, x = tx - 1 + i % CF_PX_W;
        in[a] = i < CF_PX && y >= 0 && y < p.h && x >= 0 && x < p.wd;
        if (in[a]) raw[a] = image_at[((size_t)y * p.wd + x) * C8];
      }
#pragma unroll
      for (int a = 0; a < AHEAD; ++a) {
        const int i = i0 + a * AT_ONCE;
        if (i >= CF_PX) break;
        uint4 o = make_uint4(0u, 0u, 0u, 0u);            // the convolution's border is zero behind the activation
        if (in[a]) {
          const uint32_t u[4] = {raw[a].x, raw[a].y, raw[a].z, raw[a].w};
          float f[8];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            f[2 * j] = silu_f(fmaf(__uint_as_float(u[j] << 16), sc[2 * j], sh[2 * j]));
            f[2 * j + 1] = silu_f(fmaf(__uint_as_float(u[j] & 0xffff0000u), sc[2 * j + 1], sh[2 * j + 1]));
          }
          store_row8(reinterpret_cast<bf16*>(&o), f);
        }
        *reinterpret_cast<uint4*>(smem + (size_t)i * (C * 2) + ((v ^ (i & 7)) << 4)) = o;      // eight neighbouring pixels' pieces lie in eight banks' groups
      }
    }
    __syncthreads();

    float acc[2][4] = {};
    const uint32_t base = smem_u32(smem);
    const int a_px = lane & 15, a_chunk = lane >> 4;
#pragma unroll 1
    for (int tap = 0; tap < 9; ++tap) {
      const int first = (warp + tap / 3) * CF_PX_W + tap % 3 + a_px;
      const uint2* b_at = frag + tap * (C / 16) * 32 + lane;
#pragma unroll
      for (int k = 0; k < C / 16; ++k) {
        const uint2 b = b_at[k * 32];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const int px = first + m * 16;
          uint32_t a0, a1, a2, a3;
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                       : "r"(base + (uint32_t)px * (C * 2) + (uint32_t)(((2 * k + a_chunk) ^ (px & 7)) << 4)));
          asm volatile(
              "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
              : "+f"(acc[m][0]), "+f"(acc[m][1]), "+f"(acc[m][2]), "+f"(acc[m][3])
              : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
        }
      }
    }
    const int y = ty + warp;
    if (y < p.h) {
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int x = tx + m * 16 + half * 8 + g;
          if (x < p.wd)
            *reinterpret_cast<__nv_bfloat162*>(p.out + (((size_t)n * p.h + y) * p.wd + x) * 8 + t4 * 2) =
                __floats2bfloat162_rn(acc[m][half * 2] + b0, acc[m][half * 2 + 1] + b1);
        }
    }
  }
}

template <int C>
int launch_few(const FewParams& p, cudaStream_t stream) {
  auto kern = norm_silu_conv_few_kernel<C>;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cf_smem<C>());
    if (e != cudaSuccess) return -(int)e;
    configured[dev] = true;
  }
  const long long tiles = (long long)((p.wd + CF_W - 1) / CF_W) * ((p.h + CF_H - 1) / CF_H) * p.n;
  return launch_kernel(kern, dim3((unsigned)std::min<long long>(tiles, 2LL * device_sm_count())), dim3(CF_THREADS), cf_smem<C>(), stream, p);
}

}  // namespace
}  // namespace swb

extern "C" {

// out [n, h, w, 8] = conv3x3(silu(group_norm(x))) + bias for x [n, h, w, c] bf16, c 64 or 128: sums fp32 [n, groups, 2] of x (swb_conv3x3_nhwc_stats), W [8, (ky, kx,
// c)] and bias [8] bf16, stride 1, zero padding 1. 16-byte aligned pointers. -3 for other widths.
int swb_norm_silu_conv3x3_few(const void* x, int n, int h, int w, int c, const void* sums, int groups, const void* gamma, const void* beta, float eps, const void* W,
                              const void* bias, void* out, void* stream) {
  using namespace swb;
  if (n <= 0 || h <= 0 || w <= 0) return 0;
  for (const void* q : {x, sums, gamma, beta, W, bias, (const void*)out})
    if (!q || (reinterpret_cast<uintptr_t>(q) & 15)) return -3;
  if (groups <= 0 || c % groups || (long long)n * h * w > 0x7fffffffLL) return -3;
  const FewParams p{reinterpret_cast<const bf16*>(x), reinterpret_cast<const float*>(sums), reinterpret_cast<const bf16*>(gamma), reinterpret_cast<const bf16*>(beta),
                    reinterpret_cast<const bf16*>(W), reinterpret_cast<const bf16*>(bias), reinterpret_cast<bf16*>(out), n, h, w, groups, eps};
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return c == 128 ? launch_few<128>(p, s) : c == 64 ? launch_few<64>(p, s) : -3;
}

}  // extern "C"
