// The last step of an image decoder: group norm, SiLU and a 3x3 convolution to at most eight channels, in one pass over a bf16 NHWC activation
// (candle-gen-flux/src/vae/native.rs: norm_out, swish, conv_out).
//
// With eight output channels the convolution has no use for a large tile of products: as an implicit GEMM it fetches every activation nine times
// (315 us for 128 channels at 1216 x 832, bound by L2), behind a norm that reads and writes them all (128 us). Here a CTA brings a tile of 8 x 32 pixels
// and its border to shared memory, normed and activated on the way and rounded to bf16 as the norm's own kernel stores it, and takes the nine shifted
// products from there (ldmatrix + mma.sync.m16n8k16). Tiles are walked down a column, so that a tile norms eight rows and has two from the one above; a warp
// takes half of the channels for four rows, whose operands serve up to three products each. Two CTAs to an SM: one loads while the other multiplies. The pair takes
// 168 us (1024 x 1024 of 64 channels: 99 against 258; 64 x 64 of 128: 14 against 16). Ten rows for each tile and a warp for each row took 212; places divided out
// for each load 8 more, four loads on their way and no prefetch 10 more. Loads and activations alone take 135 (exponentials and reciprocals 66),
// products alone about 140.
#include "common.cuh"

#include <algorithm>

namespace swb {

int device_sm_count();   // gemm_tcgen05.cu

namespace {

constexpr int CF_AHEAD = 6;                              // loads of a thread on their way
constexpr int CF_THREADS = 256;
constexpr int CF_H = 8, CF_W = 32;                       // output pixels of a tile
constexpr int CF_ROWS = CF_H + 2, CF_PX_W = CF_W + 2, CF_PX = CF_ROWS * CF_PX_W;

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

// pixels, weights, sums on their way between the two halves of the channels
template <int C>
constexpr size_t cf_smem() { return (size_t)CF_PX * C * 2 + (size_t)(9 * C / 16) * 32 * 8 + CF_THREADS * 8 * 4; }

template <int C>
__global__ void __launch_bounds__(CF_THREADS, 2) norm_silu_conv_few_kernel(const FewParams p) {
  constexpr int C8 = C / 8, AT_ONCE = CF_THREADS / C8;   // pixels that the CTA loads together
  extern __shared__ __align__(128) uint8_t smem[];
  uint2* frag = reinterpret_cast<uint2*>(smem + (size_t)CF_PX * C * 2);
  float* parts = reinterpret_cast<float*>(frag + 9 * C / 16 * 32);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int tiles_x = (p.wd + CF_W - 1) / CF_W, tiles_y = (p.h + CF_H - 1) / CF_H;
  const int total = tiles_x * tiles_y * p.n;

  pdl_launch_dependents();
  pdl_wait();
  // weights in the order in which the lanes of a product hold them
  for (int i = threadIdx.x; i < 9 * C / 16 * 32; i += CF_THREADS) {
    const int l = i & 31, k = (i >> 5) * 16 + (l & 3) * 2;
    const bf16* row = p.w + (size_t)(l >> 2) * 9 * C + k;
    frag[i] = make_uint2(*reinterpret_cast<const uint32_t*>(row), *reinterpret_cast<const uint32_t*>(row + 8));
  }
  const int v = threadIdx.x % C8, px0 = threadIdx.x / C8;
  float sc[8], sh[8];
  const float b0 = __bfloat162float(p.bias[t4 * 2]), b1 = __bfloat162float(p.bias[t4 * 2 + 1]);
  int image = -1, above = -1;
  // a run of neighbouring tiles, down the columns of tiles
  const int last = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
  for (int tile = (int)((long long)total * blockIdx.x / gridDim.x); tile < last; ++tile) {
    const int column = tile / tiles_y, ty = (tile - column * tiles_y) * CF_H, n = column / tiles_x, tx = (column - n * tiles_x) * CF_W;
    if (n != image) {
      image = n;
      const int cpg = C / p.groups;
      const float cnt = (float)p.h * (float)p.wd * (float)cpg;
      float ga[8], be[8];
      load_row8(p.gamma + v * 8, ga);
      load_row8(p.beta + v * 8, be);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float* st = p.sums + ((size_t)n * p.groups + (v * 8 + j) / cpg) * 2;
        const float mean = st[0] / cnt, var = fmaxf(st[1] / cnt - mean * mean, 0.f);
        sc[j] = rsqrtf(var + p.eps) * ga[j];
        sh[j] = be[j] - mean * sc[j];
      }
    }
    // input row y lies in row (y + 1) % 10 of the ring; below another tile of the column its first two rows are there
    const uint4* image_at = reinterpret_cast<const uint4*>(p.x + (size_t)n * p.h * p.wd * C) + v;
    // (places move on by additions: dividing them out for each load took 8 us of 186)
    int row = column == above ? 2 : 0, col = px0;
    int px = (ty + row) % CF_ROWS * CF_PX_W + col;
    const uint4* from = image_at + ((long long)(ty - 1 + row) * p.wd + tx - 1 + col) * C8;
    while (row < CF_ROWS) {
      uint4 raw[CF_AHEAD];
      bool in[CF_AHEAD];
      int rows = row, left = (CF_ROWS - row) * CF_PX_W - col;      // pixels up to the tile's end
#pragma unroll
      for (int a = 0; a < CF_AHEAD; ++a) {
        in[a] = rows < CF_ROWS && (unsigned)(ty - 1 + rows) < (unsigned)p.h && (unsigned)(tx - 1 + col) < (unsigned)p.wd;
        if (in[a]) raw[a] = *from;
        col += AT_ONCE, from += AT_ONCE * C8;
        if (col >= CF_PX_W) col -= CF_PX_W, ++rows, from += (long long)(p.wd - CF_PX_W) * C8;
      }
      row = rows;
#pragma unroll
      for (int a = 0; a < CF_AHEAD; ++a) {
        if (left <= 0) break;
        left -= AT_ONCE;
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
        *reinterpret_cast<uint4*>(smem + (size_t)px * (C * 2) + ((v ^ (px & 7)) << 4)) = o;      // pieces of eight neighbouring pixels lie in different banks
        px += AT_ONCE;
        if (px >= CF_PX) px -= CF_PX;
      }
    }
    above = column;
    __syncthreads();

    // the next tile's rows on their way to L2 meanwhile
    if (threadIdx.x < CF_H && tile + 1 < last && ty + CF_H < p.h) {
      const int y = ty + CF_H + 1 + threadIdx.x, x = max(tx - 1, 0), px = min(tx + CF_W + 1, p.wd) - x;
      if (y < p.h)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p.x + (((size_t)n * p.h + y) * p.wd + x) * C), "r"(px * C * 2) : "memory");
    }
    // A warp has half of the channels for four rows of sixteen pixels: six rows of operands serve twelve products.
    const int part = warp >> 2, row0 = (warp >> 1 & 1) * 4, x0 = (warp & 1) * 16;
    float acc[4][4] = {};
    const uint32_t base = smem_u32(smem);
    int at[6];
#pragma unroll
    for (int r = 0; r < 6; ++r) at[r] = (ty + row0 + r) % CF_ROWS * CF_PX_W + x0 + (lane & 15);
#pragma unroll 1
    for (int dx = 0; dx < 3; ++dx) {
#pragma unroll
      for (int kk = 0; kk < C / 32; ++kk) {
        const int k = part * (C / 32) + kk;
        uint2 b[3];
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) b[dy] = frag[((dy * 3 + dx) * (C / 16) + k) * 32 + lane];
#pragma unroll
        for (int r = 0; r < 6; ++r) {
          const int px = at[r] + dx;
          uint32_t a0, a1, a2, a3;
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                       : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                       : "r"(base + (uint32_t)px * (C * 2) + (uint32_t)(((2 * k + (lane >> 4)) ^ (px & 7)) << 4)));
#pragma unroll
          for (int dy = 0; dy < 3; ++dy) {
            const int o = r - dy;
            if (o < 0 || o > 3) continue;
            asm volatile(
                "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                : "+f"(acc[o][0]), "+f"(acc[o][1]), "+f"(acc[o][2]), "+f"(acc[o][3])
                : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b[dy].x), "r"(b[dy].y));
          }
        }
      }
    }
    // each half finishes two of the rows
    float* give = parts + (size_t)warp * 8 * 32 + lane;
    const float* take = parts + (size_t)(warp ^ 4) * 8 * 32 + lane;
#pragma unroll
    for (int j = 0; j < 8; ++j) give[j * 32] = part ? acc[j >> 2][j & 3] : acc[2 + (j >> 2)][j & 3];
    __syncthreads();                                     // (and all products have read their pixels)
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      const int y = ty + row0 + part * 2 + o;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int x = tx + x0 + half * 8 + g, j = o * 4 + half * 2;
        const float s0 = (part ? acc[2 + o][half * 2] : acc[o][half * 2]) + take[j * 32];
        const float s1 = (part ? acc[2 + o][half * 2 + 1] : acc[o][half * 2 + 1]) + take[(j + 1) * 32];
        if (y < p.h && x < p.wd)
          *reinterpret_cast<__nv_bfloat162*>(p.out + (((size_t)n * p.h + y) * p.wd + x) * 8 + t4 * 2) = __floats2bfloat162_rn(s0 + b0, s1 + b1);
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
