// Image rebuild (createImage, cuda_svd_denoiser.cu:413-498).
//
// The reference forms all denoised patches D X with one SGEMM, copies them to
// the host and overlap-adds them in a single host thread.  Here:
//   col2im_kernel  one CTA per pixel tile (sides of 8 to 64; where that is
//                  slower, col2im_direct_kernel, one thread per pixel, with
//                  the same sums): the denoised patches that
//                  cover the tile (x_hat_p = sum_s x_s d_s from the compact
//                  codes) are formed in shared memory, then each pixel sums
//                  the covering patches in patch order (ix, then iy, the
//                  reference's order) and the tile's share of
//                  sum (img/w - y)^2 is reduced in FP64;
//   lambda_kernel  fixed-order sum of the tile partials ->
//                  lambda = |sqrt(sum / (sigma2 * P)) - 1|;
//   blend_kernel   out = (lambda y + img) / (lambda + w), exp2 for speckle.
// Pixels no patch covers (w = 0) are excluded from the lambda sum and come
// back as y (the reference would divide 0/0 there).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "device_util.cuh"
#include "ksvd_internal.cuh"

namespace ksvd {

// One CTA of 1024 threads per SM: its 63 registers a thread fill the register
// file, so the tile may have nearly all of the shared memory.  (2048 x 2048
// image, 12 x 12 patches at stride 3: 0.46 ms a rebuild with 64 x 32 tiles; with
// 110 KB, 32 x 16 tiles, 0.52; two CTAs of 512 threads, 24 x 32 tiles, 0.50; four
// of 256, 8 x 24 tiles, 0.78.)
constexpr size_t kCol2imSmemLimit = 220 * 1024;
constexpr int kCol2imThreads = 1024;
constexpr int kDirectThreads = 256;

static int ceil_div(int a, int b) { return (a + b - 1) / b; }
static int tile_patches_1d(int TS, int ext, int stride) { return (TS + ext - 1) / stride + 1; }

struct Tile {
  int x, y;
};

static size_t tile_bytes(const PatchGeom& g, Tile t) {
  return size_t(tile_patches_1d(t.x, g.ph, g.sh)) * tile_patches_1d(t.y, g.pw, g.sw) * g.n * sizeof(float);
}

// Modelled time (us) of a rebuild with tile t: waves of one CTA per SM, each
// forming its patches (rounds of a patch per warp, 160 features and 4 atoms at a
// time, and their shared-memory stores) and summing its pixels.
static double tile_us(const PatchGeom& g, int L, int num_sms, Tile t) {
  const int np = std::min(tile_patches_1d(t.x, g.ph, g.sh), g.nx) * std::min(tile_patches_1d(t.y, g.pw, g.sw), g.ny);
  const double waves = std::ceil(double(ceil_div(g.W, t.x)) * ceil_div(g.H, t.y) / num_sms);
  const double rounds = ceil_div(np, kCol2imThreads / 32);
  return 6.8 + waves * (rounds * (0.46 * ceil_div(g.n, 160) * ceil_div(L, 4) + 0.62) +
                        1.33 * ceil_div(t.x * t.y, kCol2imThreads) + 0.75 + 2.1e-5 * np * g.n * L);
}

// The same of the gather without tiles: a thread per pixel forms the elements it
// needs, lanes along x, so a warp's loads touch fewer lines with a larger step.
static double direct_us(const PatchGeom& g, int L) {
  const double sh = g.sh, cover = double(ceil_div(g.ph, g.sh)) * ceil_div(g.pw, g.sw);
  return 11.6 + 1e-6 * g.W * g.H * cover * (2.73 + L * (0.82 / sh + 7.7 / (sh * sh) + 0.045 * g.pw));
}

// Pixel tile of the shared-memory gather, or x = 0 for the gather without tiles:
// the one of the least modelled time.  Large tiles form fewer patches per pixel
// (each patch is formed once per tile it touches), small images want more CTAs;
// pixels that few patches cover, and patches of which few fit a tile, are faster
// gathered.  The constants are a least-squares fit (8% for tiles, 18% for the
// gather) to each tile's time on 20 geometries (patches of 4 x 4 to 22 x 22, steps
// 1 to 8, 128 x 128 to 2048 x 2048); its choice is within 15% of the fastest tile on
// all of them.  (2048 x 2048, 20 x 20 at stride 4: 2.92 ms with the largest tile in
// 110 KB, 1.20 with 24 x 24; 8 x 8 at stride 4: 0.20 with tiles, 0.16 without.)
static Tile pick_tile(const PatchGeom& g, int L, int num_sms) {
  const int sides[] = {64, 48, 32, 24, 16, 8};
  Tile best{0, 0};
  double least = direct_us(g, L);
  for (int tx : sides)
    for (int ty : sides) {
      const Tile t{tx, ty};
      if (tile_bytes(g, t) > kCol2imSmemLimit) continue;
      const double us = tile_us(g, L, num_sms, t);
      if (us < least) {
        best = t;
        least = us;
      }
    }
  return best;
}

int col2im_num_tiles(const PatchGeom& g, int L, int num_sms) {
  const Tile t = pick_tile(g, L, num_sms);
  if (t.x == 0) return int((int64_t(g.W) * g.H + kDirectThreads - 1) / kDirectThreads);
  return ceil_div(g.W, t.x) * ceil_div(g.H, t.y);
}

// ix range covering x: ix*sh <= x < ix*sh + ph, 0 <= ix < nx
__device__ __forceinline__ int cover_lo(int x, int ext, int stride) {
  int t = x - ext + 1;
  return t <= 0 ? 0 : (t + stride - 1) / stride;
}
__device__ __forceinline__ int cover_hi(int x, int stride, int npos) { return min(npos - 1, x / stride); }

__global__ void __launch_bounds__(kCol2imThreads)
    col2im_kernel(const float* __restrict__ noisy, PatchGeom g, int TX, int TY, const float* __restrict__ D, int K,
                  int L, const int32_t* __restrict__ idx, const float* __restrict__ coef,
                  float* __restrict__ acc_out, double* __restrict__ partials) {
  extern __shared__ float xs[];
  __shared__ double red[32];
  const int tx0 = blockIdx.x * TX, ty0 = blockIdx.y * TY;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int tx1 = min(g.W, tx0 + TX) - 1, ty1 = min(g.H, ty0 + TY) - 1;
  const int ixl = cover_lo(tx0, g.ph, g.sh), ixh = cover_hi(tx1, g.sh, g.nx);
  const int iyl = cover_lo(ty0, g.pw, g.sw), iyh = cover_hi(ty1, g.sw, g.ny);
  const int npx = max(0, ixh - ixl + 1), npy = max(0, iyh - iyl + 1);
  for (int q = warp; q < npx * npy; q += nwarps) {
    const int ix = ixl + q / npy, iy = iyl + q % npy;
    const int64_t p = int64_t(ix) * g.ny + iy;
    // the patch's code, one (atom, coefficient) pair per lane, broadcast below
    int a_l = -1;
    float x_l = 0.0f;
    if (lane < L) {
      a_l = __ldg(idx + p * L + lane);
      x_l = __ldg(coef + p * L + lane);
      if (a_l < 0 || a_l >= K) a_l = -1;
    }
    // features lane, lane + 32, ... in groups of kCF; per group the rows of
    // kCS atoms are loaded before their FMAs (sum over s ascending, as in a
    // plain loop)
    constexpr int kCF = 5, kCS = 4;
    for (int i0 = 0; i0 < g.n; i0 += 32 * kCF) {
      float v[kCF];
#pragma unroll
      for (int f = 0; f < kCF; ++f) v[f] = 0.0f;
      for (int s0 = 0; s0 < L; s0 += kCS) {  // L <= 32, the same trip count in every lane
        float dv[kCS][kCF];
        float xv[kCS];
        bool uv[kCS];
#pragma unroll
        for (int u = 0; u < kCS; ++u) {
          const int s = s0 + u;
          const int a = __shfl_sync(0xffffffffu, a_l, s & 31);
          const float x = __shfl_sync(0xffffffffu, x_l, s & 31);
          const bool use = s < L && a >= 0;
          uv[u] = use;
          xv[u] = x;
#pragma unroll
          for (int f = 0; f < kCF; ++f) {
            const int i = i0 + 32 * f + lane;
            dv[u][f] = (use && i < g.n) ? __ldg(D + int64_t(a) * g.n + i) : 0.0f;
          }
        }
#pragma unroll
        for (int u = 0; u < kCS; ++u) {
          if (uv[u])
#pragma unroll
            for (int f = 0; f < kCF; ++f) v[f] = fmaf(xv[u], dv[u][f], v[f]);
        }
      }
#pragma unroll
      for (int f = 0; f < kCF; ++f) {
        const int i = i0 + 32 * f + lane;
        if (i < g.n) xs[q * g.n + i] = v[f];
      }
    }
  }
  __syncthreads();
  double part = 0.0;
  for (int t = threadIdx.x; t < TX * TY; t += blockDim.x) {
    const int x = tx0 + t % TX, y = ty0 + t / TX;
    if (x >= g.W || y >= g.H) continue;
    const int ia = max(ixl, cover_lo(x, g.ph, g.sh)), ib = min(ixh, cover_hi(x, g.sh, g.nx));
    const int ja = max(iyl, cover_lo(y, g.pw, g.sw)), jb = min(iyh, cover_hi(y, g.sw, g.ny));
    float acc = 0.0f;
    int w = 0;
    for (int ix = ia; ix <= ib; ++ix)
      for (int iy = ja; iy <= jb; ++iy) {
        const int q = (ix - ixl) * npy + (iy - iyl);
        acc += xs[q * g.n + (x - ix * g.sh) * g.pw + (y - iy * g.sw)];
        ++w;
      }
    acc_out[size_t(y) * g.W + x] = acc;
    if (w > 0) {
      const double d = double(acc) / double(w) - double(noisy[size_t(y) * g.W + x]);
      part += d * d;
    }
  }
  part = block_sum(part, red);
  if (threadIdx.x == 0) partials[blockIdx.y * gridDim.x + blockIdx.x] = part;
}

// The same sums without shared memory, for patches too large for a tile's
// covering patches to fit it and for pixels that few patches cover: one thread per pixel forms the element of each
// covering patch it needs (x_hat_p[r] = sum_s x_s d_s[r], the same FMA order
// as col2im_kernel) and adds them in the same patch order, so the result is
// identical; each block reduces its share of the lambda sum.
__global__ void __launch_bounds__(kDirectThreads) col2im_direct_kernel(
    const float* __restrict__ noisy, PatchGeom g, const float* __restrict__ D, int K, int L,
    const int32_t* __restrict__ idx, const float* __restrict__ coef, float* __restrict__ acc_out,
    double* __restrict__ partials) {
  __shared__ double red[32];
  const int64_t P = int64_t(g.W) * g.H;
  const int64_t q = int64_t(blockIdx.x) * kDirectThreads + threadIdx.x;
  double part = 0.0;
  if (q < P) {
    const int y = int(q / g.W), x = int(q - int64_t(y) * g.W);
    const int ia = cover_lo(x, g.ph, g.sh), ib = cover_hi(x, g.sh, g.nx);
    const int ja = cover_lo(y, g.pw, g.sw), jb = cover_hi(y, g.sw, g.ny);
    float acc = 0.0f;
    int w = 0;
    for (int ix = ia; ix <= ib; ++ix)
      for (int iy = ja; iy <= jb; ++iy) {
        const int64_t p = int64_t(ix) * g.ny + iy;
        const int off = (x - ix * g.sh) * g.pw + (y - iy * g.sw);
        float v = 0.0f;
        for (int s = 0; s < L; ++s) {
          const int a = __ldg(idx + p * L + s);
          if (a < 0 || a >= K) continue;
          v = fmaf(__ldg(coef + p * L + s), __ldg(D + int64_t(a) * g.n + off), v);
        }
        acc += v;
        ++w;
      }
    acc_out[q] = acc;
    if (w > 0) {
      const double d = double(acc) / double(w) - double(noisy[q]);
      part = d * d;
    }
  }
  part = block_sum(part, red);
  if (threadIdx.x == 0) partials[blockIdx.x] = part;
}

__global__ void __launch_bounds__(1024) lambda_kernel(const double* __restrict__ partials, int np, double sigma2,
                                                      double pixels, double* __restrict__ lambda_dev) {
  __shared__ double red[32];
  double s = 0.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) s += partials[i];
  s = block_sum(s, red);
  if (threadIdx.x == 0) lambda_dev[0] = fabs(sqrt(s / (sigma2 * pixels)) - 1.0);
}

__global__ void blend_kernel(const float* __restrict__ noisy, PatchGeom g, const float* __restrict__ acc,
                             const double* __restrict__ lambda_dev, int speckle, float* __restrict__ out) {
  const double lam = lambda_dev[0];
  const float lamf = float(lam);
  const int64_t P = int64_t(g.W) * g.H;
  for (int64_t q = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; q < P; q += int64_t(gridDim.x) * blockDim.x) {
    const int y = int(q / g.W), x = int(q - int64_t(y) * g.W);
    const int cx = max(0, min(g.nx - 1, x / g.sh) - cover_lo(x, g.ph, g.sh) + 1);
    const int cy = max(0, min(g.ny - 1, y / g.sw) - cover_lo(y, g.pw, g.sw) + 1);
    const float w = float(cx * cy);
    const float yv = noisy[q];
    float v = (w > 0.0f) ? (lamf * yv + acc[q]) / (lamf + w) : yv;
    if (speckle) v = exp2f(v);
    out[q] = v;
  }
}

cudaError_t launch_col2im(const float* noisy, const PatchGeom& g, const float* dict, int K, int L,
                          const int32_t* idx, const float* coef, float* acc, double* partials, int* num_partials,
                          int num_sms, cudaStream_t s) {
  const Tile t = pick_tile(g, L, num_sms);
  if (t.x == 0) {
    const int64_t blocks = (int64_t(g.W) * g.H + kDirectThreads - 1) / kDirectThreads;
    col2im_direct_kernel<<<unsigned(blocks), kDirectThreads, 0, s>>>(noisy, g, dict, K, L, idx, coef, acc, partials);
    *num_partials = int(blocks);
    return cudaGetLastError();
  }
  const size_t smem = tile_bytes(g, t);
  if (smem > 47 * 1024) {  // with the static part beyond the default limit of 48 KB
    cudaError_t e = cudaFuncSetAttribute(col2im_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
  }
  dim3 grid(ceil_div(g.W, t.x), ceil_div(g.H, t.y));
  col2im_kernel<<<grid, kCol2imThreads, smem, s>>>(noisy, g, t.x, t.y, dict, K, L, idx, coef, acc, partials);
  *num_partials = int(grid.x * grid.y);
  return cudaGetLastError();
}

cudaError_t launch_blend(const float* noisy, const PatchGeom& g, const float* acc, const double* partials,
                         int num_partials, double sigma2, int speckle, float* out, double* lambda_dev,
                         cudaStream_t s) {
  lambda_kernel<<<1, 1024, 0, s>>>(partials, num_partials, sigma2, double(g.W) * double(g.H), lambda_dev);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int64_t P = int64_t(g.W) * g.H;
  const int blocks = int(std::min<int64_t>((P + 255) / 256, 148 * 16));
  blend_kernel<<<blocks, 256, 0, s>>>(noisy, g, acc, lambda_dev, speckle, out);
  return cudaGetLastError();
}

}  // namespace ksvd
