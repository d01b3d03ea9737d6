// Pooling (channels-last), softmax, softmax cross-entropy (+ gradient).
//
// Pooling: one thread per (pixel, 4-channel vector), 16-byte accesses.  The max
// gradient is a gather over the windows containing an input pixel and gives the
// gradient to the FIRST maximum of each window (row-major), so it is
// deterministic, needs no atomics and no zero-fill pass.
// Softmax family: one warp per row for short rows (the row stays in registers), one
// CTA per row with 16-byte lanes and a one-pass running (max, sum) for long rows; the
// mean of the row losses is a fixed-order second stage.
//
// Roles in the reference: cudnnPoolingForward/Backward (src/ops/CudnnMaxPool.cu,
// CudnnAvgPool.cu) and the <<<1,1024>>> kernels of src/ops/Softmax.cu:3-22 and
// src/ops/SoftmaxCrossEntropy.cu:5-104.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include "scratch.h"
#include "launch.cuh"
#include <float.h>
#include <type_traits>
#include <limits.h>
#include <stdint.h>

#define TSB_OK 0
#define TSB_ERR_ARG 1
#define TSB_ERR_UNSUPPORTED 2
#define TSB_ERR_LAUNCH 3
#define TSB_ERR_OOM 5

namespace cg = cooperative_groups;

namespace {

using tsb_launch::load;
using tsb_launch::load_last;

int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}
int ew_grid(long long work) {
  long long blocks = (work + 255) / 256;
  const long long cap = (long long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  return blocks < 1 ? 1 : (int)blocks;
}
int done() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TSB_OK : (TSB_ERR_LAUNCH | ((int)e << 8));
}

struct PoolP {
  int n, c, h, w, oh, ow, kh, kw, pad, stride;
  long long xsn, xsh, xsw, ysn, ysh, ysw;
};

template <int KIND>
__global__ void pool_fwd(const float* x, float* __restrict__ y, const PoolP p) {
  tsb_launch::enter();
  const int C4 = p.c >> 2;
  const long long total = (long long)p.n * p.oh * p.ow * C4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C4) * 4;
    long long r = i / C4;
    const int ox = (int)(r % p.ow); r /= p.ow;
    const int oy = (int)(r % p.oh);
    const int n = (int)(r / p.oh);
    float4 acc = KIND == 0 ? make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX) : make_float4(0, 0, 0, 0);
    for (int a = 0; a < p.kh; ++a) {
      const int iy = oy * p.stride - p.pad + a;
      if ((unsigned)iy >= (unsigned)p.h) continue;
      for (int b = 0; b < p.kw; ++b) {
        const int ix = ox * p.stride - p.pad + b;
        if ((unsigned)ix >= (unsigned)p.w) continue;
        const float4 v = *reinterpret_cast<const float4*>(x + n * p.xsn + iy * p.xsh + ix * p.xsw + c);
        if (KIND == 0) {
          acc.x = fmaxf(acc.x, v.x); acc.y = fmaxf(acc.y, v.y); acc.z = fmaxf(acc.z, v.z); acc.w = fmaxf(acc.w, v.w);
        } else {
          acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
      }
    }
    if (KIND == 1) {
      const float s = 1.f / (float)(p.kh * p.kw);
      acc.x *= s; acc.y *= s; acc.z *= s; acc.w *= s;
    }
    *reinterpret_cast<float4*>(y + n * p.ysn + oy * p.ysh + ox * p.ysw + c) = acc;
  }
}

// Windows of K x K, K = 2 or 3, which is what networks pool with: one output of four channels per thread, its loads all in
// flight (positions outside are read inside and passed over), 32-bit index arithmetic.  Bound by DRAM.
// 32 x 112 x 112 x 64, 3 x 3 stride 2: 39.5 -> 23.0 us (5.6 TB/s); 16 x 224 x 224 x 64, 2 x 2: 51.0 -> 37.4 (6.9 TB/s).
template <int KIND, int K>
__global__ void __launch_bounds__(256) pool_fwd_small(const float* x, float* __restrict__ y, const PoolP p,
                                                      const unsigned total) {
  tsb_launch::enter();
  const unsigned i = blockIdx.x * 256u + threadIdx.x;
  if (i >= total) return;
  const unsigned C4 = (unsigned)p.c >> 2, r = i / C4, r2 = r / (unsigned)p.ow;
  const int c = (int)(i - r * C4) * 4, ox = (int)(r - r2 * (unsigned)p.ow);
  const int n = (int)(r2 / (unsigned)p.oh), oy = (int)(r2 - (unsigned)n * (unsigned)p.oh);
  const float* base = x + n * p.xsn + c;
  float4 v[K * K];
  bool inside[K * K];
#pragma unroll
  for (int a = 0; a < K; ++a)
#pragma unroll
    for (int b = 0; b < K; ++b) {
      const int iy = oy * p.stride - p.pad + a, ix = ox * p.stride - p.pad + b;
      inside[a * K + b] = (unsigned)iy < (unsigned)p.h && (unsigned)ix < (unsigned)p.w;
      v[a * K + b] = load(reinterpret_cast<const float4*>(base + min(max(iy, 0), p.h - 1) * p.xsh + min(max(ix, 0), p.w - 1) * p.xsw));
    }
  float4 acc = KIND == 0 ? make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX) : make_float4(0, 0, 0, 0);
#pragma unroll
  for (int q = 0; q < K * K; ++q)
    if (inside[q]) {
      if (KIND == 0) {
        acc.x = fmaxf(acc.x, v[q].x); acc.y = fmaxf(acc.y, v[q].y); acc.z = fmaxf(acc.z, v[q].z); acc.w = fmaxf(acc.w, v[q].w);
      } else {
        acc.x += v[q].x; acc.y += v[q].y; acc.z += v[q].z; acc.w += v[q].w;
      }
    }
  if (KIND == 1) {
    const float s = 1.f / (float)(K * K);
    acc.x *= s; acc.y *= s; acc.z *= s; acc.w *= s;
  }
  *reinterpret_cast<float4*>(y + n * p.ysn + oy * p.ysh + ox * p.ysw + c) = acc;
}

// Average pooling over large windows (the global pool in front of a classifier).  One thread per output and four
// channels leaves n * C / 1024 blocks that walk the window one load at a time; here a block of 32 pixel lanes x 8
// channel vectors (128-byte segments) reads the window with four loads in flight per thread, and a cluster of up to 8
// blocks shares one window, joined through distributed shared memory in a fixed order, so one launch both fills the
// chip and stays deterministic.  Bound by DRAM.  16 x 112 x 112 x 64: 3465 us with a thread per output, 20.6 now;
// 32 x 56 x 56 x 256: 794 and 32.4; 32 x 28 x 28 x 512: 195 and 20.5; 32 x 17 x 17 x 256: 83 and 7.2.
constexpr int WIN_COLS = 8, WIN_LANES = 32;
__global__ void __launch_bounds__(WIN_COLS * WIN_LANES) avg_pool_window(const float* x,
                                                                        float* __restrict__ y, const PoolP p) {
  tsb_launch::enter();
  cg::cluster_group cl = cg::this_cluster();
  __shared__ float4 sh[WIN_LANES][WIN_COLS];
  const int cx = threadIdx.x % WIN_COLS, lane = threadIdx.x / WIN_COLS;
  const int splits = (int)cl.num_blocks(), part = (int)cl.block_rank();
  const int c = (blockIdx.y * WIN_COLS + cx) * 4;
  long long r = blockIdx.x / splits;
  const int ox = (int)(r % p.ow); r /= p.ow;
  const int oy = (int)(r % p.oh);
  const int n = (int)(r / p.oh);
  const int y0 = max(oy * p.stride - p.pad, 0), y1 = min(oy * p.stride - p.pad + p.kh, p.h);
  const int x0 = max(ox * p.stride - p.pad, 0), x1 = min(ox * p.stride - p.pad + p.kw, p.w);
  const int ww = max(x1 - x0, 0), pixels = ww * max(y1 - y0, 0);
  const int per = (pixels + splits - 1) / splits, end = min(pixels, (part + 1) * per);
  float4 a[4] = {};
  if (c < p.c) {
    const float* base = x + n * p.xsn + c;
    for (int i = part * per + lane; i < end; i += 4 * WIN_LANES) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = i + u * WIN_LANES, qy = q / ww, qx = q - qy * ww;
        v[u] = q < end ? load_last(reinterpret_cast<const float4*>(base + (y0 + qy) * p.xsh + (x0 + qx) * p.xsw))
                       : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) { a[u].x += v[u].x; a[u].y += v[u].y; a[u].z += v[u].z; a[u].w += v[u].w; }
    }
  }
  sh[lane][cx] = make_float4((a[0].x + a[1].x) + (a[2].x + a[3].x), (a[0].y + a[1].y) + (a[2].y + a[3].y),
                             (a[0].z + a[1].z) + (a[2].z + a[3].z), (a[0].w + a[1].w) + (a[2].w + a[3].w));
  for (int o = WIN_LANES / 2; o > 0; o >>= 1) {
    __syncthreads();
    if (lane < o) {
      const float4 u = sh[lane][cx], v = sh[lane + o][cx];
      sh[lane][cx] = make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w);
    }
  }
  cl.sync();
  if (part == 0 && lane == 0 && c < p.c) {
    float4 t = sh[0][cx];
    for (int j = 1; j < splits; ++j) {
      const float4 u = *cl.map_shared_rank(&sh[0][cx], j);
      t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
    }
    const float s = 1.f / (float)(p.kh * p.kw);
    *reinterpret_cast<float4*>(y + n * p.ysn + oy * p.ysh + ox * p.ysw + c) =
        make_float4(t.x * s, t.y * s, t.z * s, t.w * s);
  }
  cl.sync();                       // a block's shared memory stays until block 0 has read it
}

// Blocks per window: doubled (up to the portable cluster size) while fewer than four blocks per SM are in flight and
// a block would still have two rounds of its four loads.
int window_splits(long long blocks, int pixels) {
  int s = 1;
  while (s < 8 && blocks * s < 4ll * sm_count() && pixels / (2 * s) >= 8 * WIN_LANES) s *= 2;
  return s;
}

__device__ __forceinline__ int ceil_div_pos(int a, int b) { return a <= 0 ? 0 : (a + b - 1) / b; }

template <int KIND>
__global__ void pool_bwd(const float* x, const float* y, const float* dy,
                         float* __restrict__ dx, const PoolP p) {
  tsb_launch::enter();
  const int C4 = p.c >> 2;
  const long long total = (long long)p.n * p.h * p.w * C4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C4) * 4;
    long long r = i / C4;
    const int ix = (int)(r % p.w); r /= p.w;
    const int iy = (int)(r % p.h);
    const int n = (int)(r / p.h);
    // output windows that contain (iy, ix)
    const int oy0 = ceil_div_pos(iy + p.pad - p.kh + 1, p.stride), oy1 = min(p.oh - 1, (iy + p.pad) / p.stride);
    const int ox0 = ceil_div_pos(ix + p.pad - p.kw + 1, p.stride), ox1 = min(p.ow - 1, (ix + p.pad) / p.stride);
    float4 acc = make_float4(0, 0, 0, 0);
    float4 me = make_float4(0, 0, 0, 0);
    if (KIND == 0) me = *reinterpret_cast<const float4*>(x + n * p.xsn + iy * p.xsh + ix * p.xsw + c);
    for (int oy = oy0; oy <= oy1; ++oy) {
      for (int ox = ox0; ox <= ox1; ++ox) {
        const float4 g = *reinterpret_cast<const float4*>(dy + n * p.ysn + oy * p.ysh + ox * p.ysw + c);
        if (KIND == 1) {
          acc.x += g.x; acc.y += g.y; acc.z += g.z; acc.w += g.w;
          continue;
        }
        const float4 m = *reinterpret_cast<const float4*>(y + n * p.ysn + oy * p.ysh + ox * p.ysw + c);
        // am I the first maximum of this window?  (scan the elements that precede me)
        bool fx = me.x == m.x, fy = me.y == m.y, fz = me.z == m.z, fw = me.w == m.w;
        if (fx | fy | fz | fw) {
          const int my_a = iy - (oy * p.stride - p.pad), my_b = ix - (ox * p.stride - p.pad);
          for (int a = 0; a <= my_a; ++a) {
            const int yy = oy * p.stride - p.pad + a;
            if ((unsigned)yy >= (unsigned)p.h) continue;
            const int bend = (a == my_a) ? my_b : p.kw;
            for (int b = 0; b < bend; ++b) {
              const int xx = ox * p.stride - p.pad + b;
              if ((unsigned)xx >= (unsigned)p.w) continue;
              const float4 v = *reinterpret_cast<const float4*>(x + n * p.xsn + yy * p.xsh + xx * p.xsw + c);
              fx = fx && v.x != m.x; fy = fy && v.y != m.y; fz = fz && v.z != m.z; fw = fw && v.w != m.w;
            }
          }
          if (fx) acc.x += g.x;
          if (fy) acc.y += g.y;
          if (fz) acc.z += g.z;
          if (fw) acc.w += g.w;
        }
      }
    }
    if (KIND == 1) {
      const float s = 1.f / (float)(p.kh * p.kw);
      acc.x *= s; acc.y *= s; acc.z *= s; acc.w *= s;
    }
    *reinterpret_cast<float4*>(dx + n * p.xsn + iy * p.xsh + ix * p.xsw + c) = acc;
  }
}

// Average-pool backward where no windows overlap (kernel <= stride, no padding): every pixel has one window or none, and
// the pass is a broadcast of dy, bound by the writes of dx.  A block owns one image row; a thread's next element is found
// by adding, not dividing, and its loads (L1 and L2) are issued four at a time before the stores.
// One window per image, 32 x 56 x 56 x 256: 65.0 us in the general form (a division per index and element) -> 16.8;
// 32 x 28 x 28 x 512: 33.4 -> 9.1; 32 x 17 x 17 x 256: 7.8 -> 3.0; 32 x 7 x 7 x 2048: 9.9 -> 3.7; windows of 4 x 4 in
// 32 x 56 x 56 x 64: 20.3 -> 7.2.
__global__ void __launch_bounds__(256) avg_pool_bwd_rows(const float* dy, float* __restrict__ dx, const PoolP p) {
  tsb_launch::enter();
  const unsigned C4 = (unsigned)p.c >> 2, row = blockIdx.x, n = row / (unsigned)p.h, iy = row - n * (unsigned)p.h;
  const unsigned oy = iy / (unsigned)p.stride;
  const bool row_in = (int)oy < p.oh && (int)(iy - oy * p.stride) < p.kh;
  const float* g = dy + n * p.ysn + oy * p.ysh;
  float* d = dx + n * p.xsn + iy * p.xsh;
  const float s = 1.f / (float)(p.kh * p.kw);
  unsigned ix = threadIdx.x / C4, c = threadIdx.x - ix * C4;
  const unsigned step_x = 256u / C4, step_c = 256u - step_x * C4;
  while (ix < (unsigned)p.w) {
    float4 v[4];
    unsigned xs[4], cs[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      xs[u] = ix; cs[u] = c;
      v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      const unsigned ox = p.ow == 1 ? 0u : ix / (unsigned)p.stride;
      if (row_in && ix < (unsigned)p.w && (int)ox < p.ow && (int)(ix - ox * p.stride) < p.kw)
        v[u] = load(reinterpret_cast<const float4*>(g + ox * p.ysw) + c);
      ix += step_x;
      c += step_c;
      if (c >= C4) { c -= C4; ++ix; }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (xs[u] < (unsigned)p.w)
        *(reinterpret_cast<float4*>(d + xs[u] * p.xsw) + cs[u]) = make_float4(v[u].x * s, v[u].y * s, v[u].z * s, v[u].w * s);
  }
}

// Backward for windows that tile the input exactly (kernel == stride, no padding, h = oh*stride):
// one thread owns one output window and four channels, reads its K x K inputs and one gradient,
// and writes the K x K input gradients -- x and dx cross HBM once each and y is not read at all.
// Ties go to the first maximum in scan order, as in the general kernel.
template <int KIND, int K>
__global__ void pool_bwd_tiled(const float* x, const float* dy, float* __restrict__ dx,
                               const PoolP p) {
  tsb_launch::enter();
  const int C4 = p.c >> 2;
  const long long total = (long long)p.n * p.oh * p.ow * C4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C4) * 4;
    long long r = i / C4;
    const int ox = (int)(r % p.ow); r /= p.ow;
    const int oy = (int)(r % p.oh);
    const int n = (int)(r / p.oh);
    const float4 g = *reinterpret_cast<const float4*>(dy + n * p.ysn + oy * p.ysh + ox * p.ysw + c);
    const long long base = n * p.xsn + (long long)(oy * K) * p.xsh + (long long)(ox * K) * p.xsw + c;
    if (KIND == 1) {
      const float s = 1.f / (float)(K * K);
      const float4 o = make_float4(g.x * s, g.y * s, g.z * s, g.w * s);
#pragma unroll
      for (int a = 0; a < K; ++a)
#pragma unroll
        for (int b = 0; b < K; ++b) *reinterpret_cast<float4*>(dx + base + a * p.xsh + b * p.xsw) = o;
      continue;
    }
    float4 v[K * K];
#pragma unroll
    for (int a = 0; a < K; ++a)
#pragma unroll
      for (int b = 0; b < K; ++b) v[a * K + b] = load_last(reinterpret_cast<const float4*>(x + base + a * p.xsh + b * p.xsw));
    int ax = 0, ay = 0, az = 0, aw = 0;          // index of the first maximum per channel
    float4 m = v[0];
#pragma unroll
    for (int q = 1; q < K * K; ++q) {
      if (v[q].x > m.x) { m.x = v[q].x; ax = q; }
      if (v[q].y > m.y) { m.y = v[q].y; ay = q; }
      if (v[q].z > m.z) { m.z = v[q].z; az = q; }
      if (v[q].w > m.w) { m.w = v[q].w; aw = q; }
    }
#pragma unroll
    for (int a = 0; a < K; ++a)
#pragma unroll
      for (int b = 0; b < K; ++b) {
        const int q = a * K + b;
        const float4 o = make_float4(ax == q ? g.x : 0.f, ay == q ? g.y : 0.f, az == q ? g.z : 0.f,
                                     aw == q ? g.w : 0.f);
        *reinterpret_cast<float4*>(dx + base + a * p.xsh + b * p.xsw) = o;
      }
  }
}

// Max-pool backward for windows that overlap (e.g. 3x3 stride 2), in two passes without scans:
//   pass 1, one thread per output window and four channels: position (a * kw + b) of the first
//           maximum inside the window, one byte per channel;
//   pass 2, one thread per input pixel and four channels: add dy of every window that contains the
//           pixel and whose recorded position is this pixel, in a fixed order.
// After a ReLU most windows tie at zero, which made the scan-for-earlier-maximum form of the general
// kernel expensive; here every tensor is read once.
__global__ void pool_argmax(const float* x, unsigned char* __restrict__ idx, const PoolP p) {
  tsb_launch::enter();
  const int C4 = p.c >> 2;
  const long long total = (long long)p.n * p.oh * p.ow * C4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % C4) * 4;
    long long r = i / C4;
    const int ox = (int)(r % p.ow); r /= p.ow;
    const int oy = (int)(r % p.oh);
    const int n = (int)(r / p.oh);
    float4 m = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX);
    uchar4 q = make_uchar4(255, 255, 255, 255);
    for (int a = 0; a < p.kh; ++a) {
      const int iy = oy * p.stride - p.pad + a;
      if ((unsigned)iy >= (unsigned)p.h) continue;
      for (int b = 0; b < p.kw; ++b) {
        const int ix = ox * p.stride - p.pad + b;
        if ((unsigned)ix >= (unsigned)p.w) continue;
        const float4 v = *reinterpret_cast<const float4*>(x + n * p.xsn + iy * p.xsh + ix * p.xsw + c);
        const unsigned char pos = (unsigned char)(a * p.kw + b);
        if (v.x > m.x || q.x == 255) { m.x = v.x; q.x = pos; }
        if (v.y > m.y || q.y == 255) { m.y = v.y; q.y = pos; }
        if (v.z > m.z || q.z == 255) { m.z = v.z; q.z = pos; }
        if (v.w > m.w || q.w == 255) { m.w = v.w; q.w = pos; }
      }
    }
    *reinterpret_cast<uchar4*>(idx + i * 4) = q;
  }
}

__global__ void pool_bwd_from_argmax(const unsigned char* idx, const float* dy,
                                     float* __restrict__ dx, const PoolP p) {
  tsb_launch::enter();
  const int C4 = p.c >> 2;
  const long long total = (long long)p.n * p.h * p.w * C4;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c4 = (int)(i % C4);
    const int c = c4 * 4;
    long long r = i / C4;
    const int ix = (int)(r % p.w); r /= p.w;
    const int iy = (int)(r % p.h);
    const int n = (int)(r / p.h);
    const int oy0 = ceil_div_pos(iy + p.pad - p.kh + 1, p.stride), oy1 = min(p.oh - 1, (iy + p.pad) / p.stride);
    const int ox0 = ceil_div_pos(ix + p.pad - p.kw + 1, p.stride), ox1 = min(p.ow - 1, (ix + p.pad) / p.stride);
    float4 acc = make_float4(0, 0, 0, 0);
    for (int oy = oy0; oy <= oy1; ++oy) {
      for (int ox = ox0; ox <= ox1; ++ox) {
        const int pos = (iy - (oy * p.stride - p.pad)) * p.kw + (ix - (ox * p.stride - p.pad));
        const uchar4 q = *reinterpret_cast<const uchar4*>(idx + ((((long long)n * p.oh + oy) * p.ow + ox) * C4 + c4) * 4);
        const float4 g = *reinterpret_cast<const float4*>(dy + n * p.ysn + oy * p.ysh + ox * p.ysw + c);
        if (q.x == pos) acc.x += g.x;
        if (q.y == pos) acc.y += g.y;
        if (q.z == pos) acc.z += g.z;
        if (q.w == pos) acc.w += g.w;
      }
    }
    *reinterpret_cast<float4*>(dx + n * p.xsn + iy * p.xsh + ix * p.xsw + c) = acc;
  }
}

// The same in one pass for windows small against a tile: a block owns T x T input pixels of 32 channels, finds the
// first maximum of every window that reaches into them (windows on the edge are found by both neighbours), keeps
// position and gradient in shared memory and gathers from there, in the order of pool_bwd_from_argmax.  x comes from
// DRAM once and its overlapping reads from L1, and the positions never leave the SM.
// 32 x 112 x 112 x 64, 3 x 3 stride 2: 180 us in two passes, 127 in one.
__global__ void __launch_bounds__(256) max_pool_bwd_tile(const float* x, const float* dy,
                                                         float* __restrict__ dx, const PoolP p, int tiles_x, int nw) {
  tsb_launch::enter();
  constexpr int T = 16;
  extern __shared__ float4 grad[];                                          // [window][8]
  uchar4* pos = reinterpret_cast<uchar4*>(grad + nw * nw * 8);
  const int kh = p.kh, kw = p.kw, stride = p.stride;
  const int lane = threadIdx.x & 7, c = (blockIdx.y * 8 + lane) * 4;
  const int y0 = (int)(blockIdx.x / tiles_x) * T, x0 = (int)(blockIdx.x % tiles_x) * T;
  const long long n = blockIdx.z;
  const int oy0 = ceil_div_pos(y0 + p.pad - kh + 1, stride), ox0 = ceil_div_pos(x0 + p.pad - kw + 1, stride);
  const int oy1 = min(p.oh - 1, (min(y0 + T, p.h) - 1 + p.pad) / stride);
  const int ox1 = min(p.ow - 1, (min(x0 + T, p.w) - 1 + p.pad) / stride);
  const int ny = oy1 - oy0 + 1, nx = ox1 - ox0 + 1;                          // may be <= 0: no window reaches here
  const bool live = c < p.c;
  for (int w = threadIdx.x >> 3; live && nx > 0 && w < ny * nx; w += 32) {
    const int oy = oy0 + w / nx, ox = ox0 + w % nx;
    grad[w * 8 + lane] = load(reinterpret_cast<const float4*>(dy + n * p.ysn + oy * p.ysh + ox * p.ysw + c));
    float4 m = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX);
    uchar4 q = make_uchar4(255, 255, 255, 255);
    auto take = [&](const float4& v, unsigned char at) {
      if (v.x > m.x || q.x == 255) { m.x = v.x; q.x = at; }
      if (v.y > m.y || q.y == 255) { m.y = v.y; q.y = at; }
      if (v.z > m.z || q.z == 255) { m.z = v.z; q.z = at; }
      if (v.w > m.w || q.w == 255) { m.w = v.w; q.w = at; }
    };
    const float* base = x + n * p.xsn + c;
    for (int a = 0; a < kh; ++a) {
      const int iy = oy * stride - p.pad + a;
      if ((unsigned)iy >= (unsigned)p.h) continue;
      for (int b = 0; b < kw; ++b) {
        const int ix = ox * stride - p.pad + b;
        if ((unsigned)ix >= (unsigned)p.w) continue;
        take(load(reinterpret_cast<const float4*>(base + iy * p.xsh + ix * p.xsw)), (unsigned char)(a * kw + b));
      }
    }
    pos[w * 8 + lane] = q;
  }
  __syncthreads();
  for (int i = threadIdx.x >> 3; live && i < T * T; i += 32) {
    const int iy = y0 + i / T, ix = x0 + i % T;
    if (iy >= p.h || ix >= p.w) continue;
    const int wy0 = ceil_div_pos(iy + p.pad - kh + 1, stride), wy1 = min(p.oh - 1, (iy + p.pad) / stride);
    const int wx0 = ceil_div_pos(ix + p.pad - kw + 1, stride), wx1 = min(p.ow - 1, (ix + p.pad) / stride);
    float4 acc = make_float4(0, 0, 0, 0);
    for (int oy = wy0; oy <= wy1; ++oy) {
      for (int ox = wx0; ox <= wx1; ++ox) {
        const int at = (iy - (oy * stride - p.pad)) * kw + (ix - (ox * stride - p.pad));
        const int w = ((oy - oy0) * nx + (ox - ox0)) * 8 + lane;
        const uchar4 q = pos[w];
        const float4 g = grad[w];
        if (q.x == at) acc.x += g.x;
        if (q.y == at) acc.y += g.y;
        if (q.z == at) acc.z += g.z;
        if (q.w == at) acc.w += g.w;
      }
    }
    *reinterpret_cast<float4*>(dx + n * p.xsn + iy * p.xsh + ix * p.xsw + c) = acc;
  }
}

// The same for 3 x 3 windows two apart with a padding of PAD, 0 or 1.  That kernel is bound by its instructions; here a
// pixel's windows are constants: 2 x 2 pixels lie in 2 x 2 windows, and which place of a window each of them is does not
// depend on where they are.  So a thread gathers four pixels from four windows, nine comparisons a channel with constants
// and no bounds (windows that do not exist have no position).  A window's maximum starts at its first place inside, which
// is where a position outside is read.
// 32 x 112 x 112 x 64: 127 us by the kernel above, 84 by it with the window as constants, 50 here (232 MB: 4.6 TB/s).
template <int PAD>
__global__ void __launch_bounds__(256) max_pool_bwd_3s2(const float* x, const float* dy, float* __restrict__ dx, const PoolP p,
                                                        int tiles_x) {
  tsb_launch::enter();
  constexpr int NW = 9;                                                     // windows of 16 pixels, per axis
  __shared__ float4 grad[NW * NW * 8];
  __shared__ uchar4 pos[NW * NW * 8];
  const int lane = threadIdx.x & 7, c = (blockIdx.y * 8 + lane) * 4;
  const bool live = c < p.c;
  const int y0 = (int)(blockIdx.x / tiles_x) * 16, x0 = (int)(blockIdx.x % tiles_x) * 16;
  const int oy0 = y0 / 2 - 1 + PAD, ox0 = x0 / 2 - 1 + PAD;
  x += blockIdx.z * p.xsn + c;
  dy += blockIdx.z * p.ysn + c;
  dx += blockIdx.z * p.xsn + c;
  for (int w = threadIdx.x >> 3; live && w < NW * NW; w += 32) {
    const int oy = oy0 + w / NW, ox = ox0 + w % NW, iy = oy * 2 - PAD, ix = ox * 2 - PAD;
    uchar4 q = make_uchar4(255, 255, 255, 255);
    if ((unsigned)oy < (unsigned)p.oh && (unsigned)ox < (unsigned)p.ow && iy < p.h && ix < p.w) {
      grad[w * 8 + lane] = load(reinterpret_cast<const float4*>(dy + oy * p.ysh + ox * p.ysw));
      float4 v[9];
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < 3; ++b)
          v[a * 3 + b] = load(reinterpret_cast<const float4*>(x + min(max(iy + a, 0), p.h - 1) * p.xsh + min(max(ix + b, 0), p.w - 1) * p.xsw));
      float4 m = v[0];
      const unsigned char first = (iy < 0 ? 3 : 0) + (ix < 0 ? 1 : 0);
      q = make_uchar4(first, first, first, first);
#pragma unroll
      for (int at = 1; at < 9; ++at) {
        const bool inside = (unsigned)(iy + at / 3) < (unsigned)p.h && (unsigned)(ix + at % 3) < (unsigned)p.w;
        if (inside && v[at].x > m.x) { m.x = v[at].x; q.x = at; }
        if (inside && v[at].y > m.y) { m.y = v[at].y; q.y = at; }
        if (inside && v[at].z > m.z) { m.z = v[at].z; q.z = at; }
        if (inside && v[at].w > m.w) { m.w = v[at].w; q.w = at; }
      }
    }
    pos[w * 8 + lane] = q;
  }
  __syncthreads();
  for (int i = threadIdx.x >> 3; live && i < 64; i += 32) {
    const int by = i >> 3, bx = i & 7, iy = y0 + 2 * by, ix = x0 + 2 * bx;
    if (iy >= p.h || ix >= p.w) continue;
    uchar4 q[4];
    float4 g[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int w = ((by + k / 2) * NW + bx + k % 2) * 8 + lane;
      q[k] = pos[w];
      g[k] = grad[w];
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int a = r / 2 + 2 - PAD - 2 * (k / 2), b = r % 2 + 2 - PAD - 2 * (k % 2), at = a * 3 + b;
        if (a < 0 || a > 2 || b < 0 || b > 2) continue;
        if (q[k].x == at) acc.x += g[k].x;
        if (q[k].y == at) acc.y += g[k].y;
        if (q[k].z == at) acc.z += g[k].z;
        if (q[k].w == at) acc.w += g[k].w;
      }
      if (iy + r / 2 < p.h && ix + r % 2 < p.w)
        *reinterpret_cast<float4*>(dx + (iy + r / 2) * p.xsh + (ix + r % 2) * p.xsw) = acc;
    }
  }
}

unsigned char* argmax_scratch(size_t bytes, cudaStream_t st) {
  return static_cast<unsigned char*>(tsb_scratch::get(st, tsb_scratch::POOL_ARGMAX, bytes, size_t(32) << 20));
}

// ------------------------------------------------------------------ softmax family
__device__ __forceinline__ float block_max(float v, float* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (lane == 0) sh[w] = v;
  __syncthreads();
  float r = sh[0];
  for (int i = 1; i < (blockDim.x >> 5); ++i) r = fmaxf(r, sh[i]);
  __syncthreads();
  return r;
}
__device__ __forceinline__ float block_sum(float v, float* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sh[w] = v;
  __syncthreads();
  float r = 0.f;
  for (int i = 0; i < (blockDim.x >> 5); ++i) r += sh[i];
  __syncthreads();
  return r;
}

__global__ void softmax_rows(const float* x, float* __restrict__ y, long long rows, long long cols) {
  tsb_launch::enter();
  __shared__ float sh[8];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float* xr = x + row * cols;
    float m = -FLT_MAX;
    for (long long i = threadIdx.x; i < cols; i += blockDim.x) m = fmaxf(m, xr[i]);
    m = block_max(m, sh);
    float s = 0.f;
    for (long long i = threadIdx.x; i < cols; i += blockDim.x) s += __expf(xr[i] - m);
    s = block_sum(s, sh);
    const float inv = 1.f / s;
    tsb_launch::read_then_write<4>((long long)threadIdx.x, cols, (long long)blockDim.x, [&](long long i) { return xr[i]; },
                                   [&](long long i, float v) { y[row * cols + i] = __expf(v - m) * inv; });
  }
}

// Short rows (cols <= 1024, a multiple of 4): one warp per row, the row held in registers between the
// maximum, the sum and the store, so it is read once and no block barrier is involved.
template <int NV>
__global__ void __launch_bounds__(256) softmax_warp_rows(const float4* x, float4* __restrict__ y,
                                                         long long rows, int nvec) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float4* xr = x + row * nvec;
    float4 v[NV];
    float m = -FLT_MAX;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      v[j] = i < nvec ? load(xr + i) : make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX);
      m = fmaxf(m, fmaxf(fmaxf(v[j].x, v[j].y), fmaxf(v[j].z, v[j].w)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      v[j].x = __expf(v[j].x - m); v[j].y = __expf(v[j].y - m);
      v[j].z = __expf(v[j].z - m); v[j].w = __expf(v[j].w - m);
      s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float inv = 1.f / s;
    float4* yr = y + row * nvec;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec) yr[i] = make_float4(v[j].x * inv, v[j].y * inv, v[j].z * inv, v[j].w * inv);
    }
  }
}

// The same for rows whose length is no multiple of 4 (or whose base is not 16-byte aligned): scalar,
// still coalesced, lanes; NE elements per lane.
template <int NE>
__global__ void __launch_bounds__(256, NE == 32 ? 4 : 1) softmax_warp_rows_scalar(const float* x, float* __restrict__ y,
                                                                long long rows, int cols) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float* xr = x + row * cols;
    float v[NE];
    float m = -FLT_MAX;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      v[j] = i < cols ? load(xr + i) : -FLT_MAX;
      m = fmaxf(m, v[j]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NE; ++j) { v[j] = __expf(v[j] - m); s += v[j]; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float inv = 1.f / s;
    float* yr = y + row * cols;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      if (i < cols) yr[i] = v[j] * inv;
    }
  }
}

template <int NE>
__global__ void __launch_bounds__(256) softmax_grad_warp_rows_scalar(const float* y,
                                                                     const float* dy,
                                                                     float* __restrict__ dx, long long rows,
                                                                     int cols) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float* yr = y + row * cols;
    const float* gr = dy + row * cols;
    float a[NE], g[NE];
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      a[j] = i < cols ? load(yr + i) : 0.f;
      g[j] = i < cols ? load(gr + i) : 0.f;
      s += a[j] * g[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    float* dr = dx + row * cols;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      if (i < cols) dr[i] = a[j] * (g[j] - s);
    }
  }
}

// Softmax backward, dx = y * (dy - sum(dy * y)): one warp per row, y and dy read once.
template <int NV>
__global__ void __launch_bounds__(256) softmax_grad_warp_rows(const float4* y,
                                                              const float4* dy,
                                                              float4* __restrict__ dx, long long rows, int nvec) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float4* yr = y + row * nvec;
    const float4* gr = dy + row * nvec;
    float4 a[NV], g[NV];
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      a[j] = i < nvec ? load(yr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      g[j] = i < nvec ? load(gr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      s += (a[j].x * g[j].x + a[j].y * g[j].y) + (a[j].z * g[j].z + a[j].w * g[j].w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    float4* dr = dx + row * nvec;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec)
        dr[i] = make_float4(a[j].x * (g[j].x - s), a[j].y * (g[j].y - s), a[j].z * (g[j].z - s),
                            a[j].w * (g[j].w - s));
    }
  }
}

// Attention soft-max: y = softmax(scale * x + mask) over rows of `cols` scores, one warp per row, the row held in
// registers, so the scaling, the key-padding mask and the causal mask cost no pass of their own.
//   key_tokens (optional) [batch][cols]: a key whose token is 0 is padding and gets -1e9 added
//   causal: column j of query row q (row % tq) is replaced by -1e9 when j > q
// Rows are [batch][rows_per_batch] with rows_per_batch = heads * tq.
template <int NE>
__global__ void __launch_bounds__(256) masked_softmax_warp_rows(const float* x,
                                                                const float* key_tokens,
                                                                float* __restrict__ y, long long rows, int cols,
                                                                long long rows_per_batch, int tq, float scale,
                                                                int causal) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float* xr = x + row * cols;
    // 32-bit index arithmetic (rows < 2^31, checked by the launcher): two 64-bit divisions per row would cost as much
    // as the row's loads
    const float* kt = key_tokens ? key_tokens + (long long)((unsigned)row / (unsigned)rows_per_batch) * cols : nullptr;
    const int q = (int)((unsigned)row % (unsigned)tq);
    float v[NE];
    float m = -FLT_MAX;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      float t = -FLT_MAX;
      if (i < cols) {
        t = load(xr + i) * scale;
        if (kt && load(kt + i) == 0.f) t += -1e9f;
        if (causal && i > q) t = -1e9f;
      }
      v[j] = t;
      m = fmaxf(m, t);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      v[j] = i < cols ? __expf(v[j] - m) : 0.f;
      s += v[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float inv = 1.f / s;
    float* yr = y + row * cols;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      if (i < cols) yr[i] = v[j] * inv;
    }
  }
}

// The same with 16-byte lanes (cols % 4 == 0, 16-byte aligned rows): NV float4 per lane.
template <int NV>
__global__ void __launch_bounds__(256) masked_softmax_warp_rows_v4(const float4* x,
                                                                   const float4* key_tokens,
                                                                   float4* __restrict__ y, long long rows, int nvec,
                                                                   long long rows_per_batch, int tq, float scale,
                                                                   int causal) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float4* xr = x + row * nvec;
    const float4* kt = key_tokens ? key_tokens + (long long)((unsigned)row / (unsigned)rows_per_batch) * nvec : nullptr;
    const int q = (int)((unsigned)row % (unsigned)tq);
    float4 v[NV], keys[NV];                     // all loads first
    float m = -FLT_MAX;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      v[j] = make_float4(-FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX);
      keys[j] = make_float4(1.f, 1.f, 1.f, 1.f);
      if (i < nvec) v[j] = load_last(xr + i);
      if (i < nvec && kt) keys[j] = load(kt + i);
    }
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      float4 t = v[j];
      if (i < nvec) {
        t.x *= scale; t.y *= scale; t.z *= scale; t.w *= scale;
        const float4 k = keys[j];
        if (k.x == 0.f) t.x += -1e9f;
        if (k.y == 0.f) t.y += -1e9f;
        if (k.z == 0.f) t.z += -1e9f;
        if (k.w == 0.f) t.w += -1e9f;
        if (causal) {
          const int c = 4 * i;
          if (c > q) t.x = -1e9f;
          if (c + 1 > q) t.y = -1e9f;
          if (c + 2 > q) t.z = -1e9f;
          if (c + 3 > q) t.w = -1e9f;
        }
      }
      v[j] = t;
      m = fmaxf(m, fmaxf(fmaxf(t.x, t.y), fmaxf(t.z, t.w)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec) {
        v[j].x = __expf(v[j].x - m); v[j].y = __expf(v[j].y - m);
        v[j].z = __expf(v[j].z - m); v[j].w = __expf(v[j].w - m);
      } else {
        v[j] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
      s += (v[j].x + v[j].y) + (v[j].z + v[j].w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float inv = 1.f / s;
    float4* yr = y + row * nvec;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec) yr[i] = make_float4(v[j].x * inv, v[j].y * inv, v[j].z * inv, v[j].w * inv);
    }
  }
}

// Its backward: dx = scale * y * (dy - sum(dy * y)) (masked positions have y = 0).
template <int NE>
__global__ void __launch_bounds__(256) scaled_softmax_grad_warp_rows(const float* y,
                                                                     const float* dy,
                                                                     float* __restrict__ dx, long long rows, int cols,
                                                                     float scale) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float* yr = y + row * cols;
    const float* gr = dy + row * cols;
    float a[NE], g[NE];
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      a[j] = i < cols ? load(yr + i) : 0.f;
      g[j] = i < cols ? load(gr + i) : 0.f;
      s += a[j] * g[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    float* dr = dx + row * cols;
#pragma unroll
    for (int j = 0; j < NE; ++j) {
      const int i = lane + 32 * j;
      if (i < cols) dr[i] = scale * a[j] * (g[j] - s);
    }
  }
}

template <int NV>
__global__ void __launch_bounds__(256) scaled_softmax_grad_warp_rows_v4(const float4* y,
                                                                        const float4* dy,
                                                                        float4* __restrict__ dx, long long rows,
                                                                        int nvec, float scale) {
  tsb_launch::enter();
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarp = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long row = warp0; row < rows; row += nwarp) {
    const float4* yr = y + row * nvec;
    const float4* gr = dy + row * nvec;
    float4 a[NV], g[NV];
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      a[j] = i < nvec ? load(yr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      g[j] = i < nvec ? load_last(gr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      s += (a[j].x * g[j].x + a[j].y * g[j].y) + (a[j].z * g[j].z + a[j].w * g[j].w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    float4* dr = dx + row * nvec;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = lane + 32 * j;
      if (i < nvec)
        dr[i] = make_float4(scale * a[j].x * (g[j].x - s), scale * a[j].y * (g[j].y - s),
                            scale * a[j].z * (g[j].z - s), scale * a[j].w * (g[j].w - s));
    }
  }
}

// Any row length: one CTA per row, the second pass finds the row in L2.
__global__ void softmax_grad_rows(const float* y, const float* dy, float* __restrict__ dx,
                                  long long rows, long long cols) {
  tsb_launch::enter();
  __shared__ float sh[8];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float* yr = y + row * cols;
    const float* gr = dy + row * cols;
    float s = 0.f;
    for (long long i = threadIdx.x; i < cols; i += blockDim.x) s += yr[i] * gr[i];
    s = block_sum(s, sh);
    tsb_launch::read_then_write<4>((long long)threadIdx.x, cols, (long long)blockDim.x,
                                   [&](long long i) { return make_float2(yr[i], gr[i]); },
                                   [&](long long i, float2 v) { dx[row * cols + i] = v.x * (v.y - s); });
  }
}

// Running (maximum, sum of exponentials) of a row in one pass: the sum is rescaled when the maximum moves.
struct MaxSum { float m, s; };
__device__ __forceinline__ MaxSum ms_join(MaxSum a, MaxSum b) {
  const float m = fmaxf(a.m, b.m);
  return {m, a.s * __expf(a.m - m) + b.s * __expf(b.m - m)};
}
__device__ __forceinline__ void ms_add4(MaxSum& a, const float4 v) {
  const float m4 = fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w));
  if (m4 > a.m) { a.s *= __expf(a.m - m4); a.m = m4; }
  a.s += (__expf(v.x - a.m) + __expf(v.y - a.m)) + (__expf(v.z - a.m) + __expf(v.w - a.m));
}
// Block-wide join; sh holds 2 floats per warp.
__device__ __forceinline__ MaxSum block_max_sum(MaxSum a, float* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    MaxSum b{__shfl_xor_sync(0xffffffffu, a.m, o), __shfl_xor_sync(0xffffffffu, a.s, o)};
    a = ms_join(a, b);
  }
  if (lane == 0) { sh[2 * w] = a.m; sh[2 * w + 1] = a.s; }
  __syncthreads();
  MaxSum r{sh[0], sh[1]};
  for (int i = 1; i < nw; ++i) r = ms_join(r, MaxSum{sh[2 * i], sh[2 * i + 1]});
  __syncthreads();
  return r;
}
template <bool STAGED>
__device__ __forceinline__ MaxSum row_max_sum(const float4* xr, int nvec, float* sh) {
  auto at = [&](int i) { return STAGED ? xr[i] : load(xr + i); };
  MaxSum a{-FLT_MAX, 0.f};
  int i = threadIdx.x;
  for (; i + 3 * (int)blockDim.x < nvec; i += 4 * blockDim.x) {
    const float4 v0 = at(i), v1 = at(i + blockDim.x), v2 = at(i + 2 * blockDim.x), v3 = at(i + 3 * blockDim.x);
    ms_add4(a, v0); ms_add4(a, v1); ms_add4(a, v2); ms_add4(a, v3);
  }
  for (; i < nvec; i += blockDim.x) ms_add4(a, at(i));
  return block_max_sum(a, sh);
}

// Where the labels of a row come from: an array, or class ids (one-hot rows scaled and shifted, as label smoothing
// makes them: `on` at the id and `off` elsewhere), which are worth a number a row instead of a pass over rows x classes.
struct DenseLabels {
  const float4* lab;
  const float4* r;
  __device__ __forceinline__ void row(long long i, int nvec) { r = lab + i * nvec; }
  __device__ __forceinline__ float4 at(int i) const { return __ldcs(r + i); }
};
struct SmoothLabels {
  const float* ids;
  float on, off;
  long long id;
  __device__ __forceinline__ void row(long long i, int) { id = (long long)ids[i]; }
  __device__ __forceinline__ float4 at(int i) const {
    const long long c = 4ll * i;
    return make_float4(id == c ? on : off, id == c + 1 ? on : off, id == c + 2 ? on : off, id == c + 3 ? on : off);
  }
};

// A row of logits in shared memory.  A thread reads only what it copied itself, in every pass, so its own wait is enough,
// and in the last pass it refills a place with the next row's value as soon as it has read it: the next row's loads run
// under this row's arithmetic and stores.
__device__ __forceinline__ void stage(float4* place, const float4* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(place)), "l"(from)
               : "memory");
}
__device__ __forceinline__ void staged() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Long rows, 16-byte lanes.  Two passes over the logits; rows of 32 to 200 KB wait for the second one in shared memory
// (STAGED): left to L2, most of a 128 KB row is gone by then, with some 600 rows in flight.  Bound by DRAM.
// 4096 x 32000 gradient with labels from ids: 278 us (dense labels, unstaged) -> 193 us.  The loss from ids takes one pass
// (below); the label tensors (one-hot, scaled, shifted) are not made at all.
template <class Labels, bool STAGED>
__global__ void __launch_bounds__(512) ce_rows_v4(const float4* x, Labels lab,
                                                  float* __restrict__ row_loss, long long rows, int nvec) {
  tsb_launch::enter();
  extern __shared__ float4 row_buf[];
  __shared__ float sh[64];
  if (STAGED)
    for (int i = threadIdx.x; blockIdx.x < rows && i < nvec; i += blockDim.x)
      stage(row_buf + i, x + (long long)blockIdx.x * nvec + i);
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float4* xr = STAGED ? row_buf : x + row * nvec;
    const float4* next = STAGED && row + gridDim.x < rows ? x + (row + gridDim.x) * nvec : nullptr;
    if (STAGED) staged();
    lab.row(row, nvec);
    const MaxSum ms = row_max_sum<STAGED>(xr, nvec, sh);
    const float lse = ms.m + logf(ms.s);
    float l = 0.f;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      const float4 t = lab.at(i);
      const float4 v = STAGED ? xr[i] : load(xr + i);
      if (next) stage(row_buf + i, next + i);
      l -= (t.x * (v.x - lse) + t.y * (v.y - lse)) + (t.z * (v.z - lse) + t.w * (v.w - lse));
    }
    l = block_sum(l, sh);
    if (threadIdx.x == 0) row_loss[row] = l;
  }
}

// The loss with labels from ids in one pass: sum t (x - lse) = sum t (x - c) - (lse - c) sum t over the labels t, for any
// c, so the row is read once.  With the labelled logit as c that class adds nothing, every other one has the weight `off`,
// and rounding is relative to lse - c, which the loss is made of: a common offset of the logits costs no digits.
// Every logit is weighed before it is added: logits at the lowest float (masked classes) under a label of 0 count as 0, as
// in the two-pass form.  No such c (an id outside the classes, a masked or infinite label): 0, and each class its own
// label.
struct SmoothSum {
  float c;
  bool inside, usual;
  MaxSum a;
  float d;
  __device__ __forceinline__ SmoothSum(const float* row, const SmoothLabels& lab, int nvec) : a{-FLT_MAX, 0.f}, d(0.f) {
    inside = lab.id >= 0 && lab.id < 4ll * nvec;
    const float at_id = inside ? load(row + lab.id) : FLT_MAX;
    usual = fabsf(at_id) < 1e30f;
    c = usual ? at_id : 0.f;
  }
  __device__ __forceinline__ void add(const float4 v, const float4 t) {
    ms_add4(a, v);
    d += (t.x * (v.x - c) + t.y * (v.y - c)) + (t.z * (v.z - c) + t.w * (v.w - c));
  }
  // Returns the maximum and sum of the row.
  __device__ __forceinline__ MaxSum finish(const SmoothLabels& lab, int nvec, float* sh, float* loss) {
    const MaxSum ms = block_max_sum(a, sh);
    d = block_sum(d, sh);
    if (threadIdx.x == 0) {
      const float ones = 4.f * (float)nvec * lab.off + (inside ? lab.on - lab.off : 0.f);
      *loss = ones * ((ms.m - c) + logf(ms.s)) - d;
    }
    return ms;
  }
};
// xr: the row x, or its copy in shared memory.
__device__ __forceinline__ MaxSum smooth_row_loss(const float4* x, const float4* xr, const SmoothLabels& lab, int nvec, float* sh,
                                                  float* loss) {
  SmoothSum sum(reinterpret_cast<const float*>(x), lab, nvec);
  int i = threadIdx.x;
  if (sum.usual) {
    const float4 off = make_float4(lab.off, lab.off, lab.off, lab.off);
    for (; i + 3 * (int)blockDim.x < nvec; i += 4 * blockDim.x) {
      const float4 v0 = load(xr + i), v1 = load(xr + i + blockDim.x), v2 = load(xr + i + 2 * blockDim.x),
                   v3 = load(xr + i + 3 * blockDim.x);
      sum.add(v0, off); sum.add(v1, off); sum.add(v2, off); sum.add(v3, off);
    }
    for (; i < nvec; i += blockDim.x) sum.add(load(xr + i), off);
  } else {
    for (; i < nvec; i += blockDim.x) sum.add(load(xr + i), lab.at(i));
  }
  return sum.finish(lab, nvec, sh, loss);
}
// 4096 x 32000 with the mean of the rows: 91 us, bound by DRAM.  (The row is walked here and not by the
// function above, whose code for it takes 3 to 5 % longer.)
__global__ void __launch_bounds__(512) ce_smooth_rows_v4(const float4* x, SmoothLabels lab,
                                                         float* __restrict__ row_loss, long long rows, int nvec) {
  tsb_launch::enter();
  __shared__ float sh[64];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float4* xr = x + row * nvec;
    lab.row(row, nvec);
    SmoothSum sum(reinterpret_cast<const float*>(xr), lab, nvec);
    int i = threadIdx.x;
    if (sum.usual) {
      const float4 off = make_float4(lab.off, lab.off, lab.off, lab.off);
      for (; i + 3 * (int)blockDim.x < nvec; i += 4 * blockDim.x) {
        const float4 v0 = load(xr + i), v1 = load(xr + i + blockDim.x), v2 = load(xr + i + 2 * blockDim.x),
                     v3 = load(xr + i + 3 * blockDim.x);
        sum.add(v0, off); sum.add(v1, off); sum.add(v2, off); sum.add(v3, off);
      }
      for (; i < nvec; i += blockDim.x) sum.add(load(xr + i), off);
    } else {
      for (; i < nvec; i += blockDim.x) sum.add(load(xr + i), lab.at(i));
    }
    sum.finish(lab, nvec, sh, row_loss + row);
  }
}

// row_loss (LOSS): the loss as well, as the kernels above make it; a training step that takes both reads its logits once.
// 4096 x 32000 with labels from ids, in one run: 91 us of loss, 198 of gradient, 297 of the two in turn
// -> 220 (the step that takes both 1187 -> 1127 us at the power cap).
template <class Labels, bool STAGED, bool LOSS>
__global__ void __launch_bounds__(512) ce_grad_rows_v4(const float4* x, Labels lab,
                                                       const float* g, float4* __restrict__ dx,
                                                       long long rows, int nvec, float* __restrict__ row_loss) {
  tsb_launch::enter();
  extern __shared__ float4 row_buf[];
  __shared__ float sh[64];
  const float scale = g[0] / (float)rows;
  if (STAGED)
    for (int i = threadIdx.x; blockIdx.x < rows && i < nvec; i += blockDim.x)
      stage(row_buf + i, x + (long long)blockIdx.x * nvec + i);
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float4* xr = STAGED ? row_buf : x + row * nvec;
    const float4* next = STAGED && row + gridDim.x < rows ? x + (row + gridDim.x) * nvec : nullptr;
    float4* dr = dx + row * nvec;
    if (STAGED) staged();
    lab.row(row, nvec);
    MaxSum ms;
    constexpr bool FROM_IDS = std::is_same<Labels, SmoothLabels>::value;
    if constexpr (LOSS && FROM_IDS) ms = smooth_row_loss(x + row * nvec, xr, lab, nvec, sh, row_loss + row);
    else ms = row_max_sum<STAGED>(xr, nvec, sh);
    const float inv = 1.f / ms.s, m = ms.m, lse = LOSS && !FROM_IDS ? m + logf(ms.s) : 0.f;
    float l = 0.f;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
      const float4 t = lab.at(i);
      const float4 v = STAGED ? xr[i] : load(xr + i);
      if (next) stage(row_buf + i, next + i);
      if (LOSS && !FROM_IDS) l -= (t.x * (v.x - lse) + t.y * (v.y - lse)) + (t.z * (v.z - lse) + t.w * (v.w - lse));
      float4 o;
      o.x = (__expf(v.x - m) * inv - t.x) * scale;
      o.y = (__expf(v.y - m) * inv - t.y) * scale;
      o.z = (__expf(v.z - m) * inv - t.z) * scale;
      o.w = (__expf(v.w - m) * inv - t.w) * scale;
      __stcs(dr + i, o);
    }
    if (LOSS && !FROM_IDS) {
      l = block_sum(l, sh);
      if (threadIdx.x == 0) row_loss[row] = l;
    }
  }
}

// Rows of up to KEPT values a thread stay in registers between the passes of the two kernels below.
constexpr int KEPT = 8;
__device__ __forceinline__ void keep_row(float (&v)[KEPT], const float* xr, int cols, float rest) {
#pragma unroll
  for (int u = 0; u < KEPT; ++u) {
    const int i = threadIdx.x + u * blockDim.x;
    v[u] = i < cols ? load(xr + i) : rest;
  }
}
__device__ __forceinline__ MaxSum kept_max_sum(const float (&v)[KEPT], int cols, float* sh) {
  float m = -FLT_MAX, s = 0.f;
#pragma unroll
  for (int u = 0; u < KEPT; ++u) m = fmaxf(m, v[u]);
  m = block_max(m, sh);
#pragma unroll
  for (int u = 0; u < KEPT; ++u)
    if (threadIdx.x + u * blockDim.x < cols) s += expf(v[u] - m);
  return {m, block_sum(s, sh)};
}

__global__ void ce_rows(const float* x, const float* lab, float* __restrict__ row_loss,
                        long long rows, long long cols) {
  tsb_launch::enter();
  __shared__ float sh[8];
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float* xr = x + row * cols;
    const float* lr = lab + row * cols;
    float l = 0.f;
    if (cols <= KEPT * (long long)blockDim.x) {
      float v[KEPT], t[KEPT];
      keep_row(v, xr, (int)cols, -FLT_MAX);
      keep_row(t, lr, (int)cols, 0.f);
      const MaxSum ms = kept_max_sum(v, (int)cols, sh);
      const float lse = ms.m + logf(ms.s);
#pragma unroll
      for (int u = 0; u < KEPT; ++u)
        if (threadIdx.x + u * blockDim.x < cols) l -= t[u] * (v[u] - lse);
    } else {
      float m = -FLT_MAX;
      for (long long i = threadIdx.x; i < cols; i += blockDim.x) m = fmaxf(m, xr[i]);
      m = block_max(m, sh);
      float s = 0.f;
      for (long long i = threadIdx.x; i < cols; i += blockDim.x) s += expf(xr[i] - m);
      s = block_sum(s, sh);
      const float lse = m + logf(s);
      for (long long i = threadIdx.x; i < cols; i += blockDim.x) l -= lr[i] * (xr[i] - lse);
    }
    l = block_sum(l, sh);
    if (threadIdx.x == 0) row_loss[row] = l;
  }
}

__global__ void mean_rows(const float* row_loss, float* __restrict__ out, long long rows) {
  tsb_launch::enter();
  __shared__ float sh[32];
  float s = 0.f;
  for (long long i = threadIdx.x; i < rows; i += blockDim.x) s += row_loss[i];
  s = block_sum(s, sh);
  if (threadIdx.x == 0) out[0] = s / (float)rows;
}

// row_loss (LOSS): where the loss of every row goes as well, as ce_rows makes it.  (A template: a test at run time cost the
// gradient alone its registers, 4096 x 33278 511 -> 598 us.)
template <bool LOSS>
__global__ void ce_grad_rows(const float* x, const float* lab, const float* g, float* __restrict__ dx, long long rows,
                             long long cols, float* __restrict__ row_loss) {
  tsb_launch::enter();
  __shared__ float sh[8];
  const float scale = g[0] / (float)rows;
  for (long long row = blockIdx.x; row < rows; row += gridDim.x) {
    const float* xr = x + row * cols;
    if (cols <= KEPT * (long long)blockDim.x) {
      float v[KEPT], t[KEPT];
      keep_row(v, xr, (int)cols, -FLT_MAX);
      keep_row(t, lab + row * cols, (int)cols, 0.f);
      const MaxSum ms = kept_max_sum(v, (int)cols, sh);
      const float inv = 1.f / ms.s;
#pragma unroll
      for (int u = 0; u < KEPT; ++u) {
        const int i = threadIdx.x + u * blockDim.x;
        if (i < cols) dx[row * cols + i] = (expf(v[u] - ms.m) * inv - t[u]) * scale;
      }
      if (LOSS) {
        const float lse = ms.m + logf(ms.s);
        float l = 0.f;
#pragma unroll
        for (int u = 0; u < KEPT; ++u)
          if (threadIdx.x + u * blockDim.x < cols) l -= t[u] * (v[u] - lse);
        l = block_sum(l, sh);
        if (threadIdx.x == 0) row_loss[row] = l;
      }
      continue;
    }
    float m = -FLT_MAX;
    for (long long i = threadIdx.x; i < cols; i += blockDim.x) m = fmaxf(m, xr[i]);
    m = block_max(m, sh);
    float s = 0.f;
    for (long long i = threadIdx.x; i < cols; i += blockDim.x) s += expf(xr[i] - m);
    s = block_sum(s, sh);
    const float inv = 1.f / s;
    if (LOSS) {
      const float lse = m + logf(s);
      float l = 0.f;
      for (long long i = threadIdx.x; i < cols; i += blockDim.x) l -= lab[row * cols + i] * (xr[i] - lse);
      l = block_sum(l, sh);
      if (threadIdx.x == 0) row_loss[row] = l;
    }
    tsb_launch::read_then_write<4>((long long)threadIdx.x, cols, (long long)blockDim.x,
                                   [&](long long i) { return make_float2(xr[i], lab[row * cols + i]); },
                                   [&](long long i, float2 v) { dx[row * cols + i] = (expf(v.x - m) * inv - v.y) * scale; });
  }
}

// Launch of a long-row kernel (`plain` / `staged`: its two forms): rows that fit are staged, by as many persistent
// blocks as have room for a row each.
template <class K, class... A>
int launch_rows(K plain, K staged, long long rows, int nvec, cudaStream_t st, A... args) {
  const int threads = nvec >= 2048 ? 512 : 256;
  const size_t row_bytes = (size_t)nvec * sizeof(float4);
  if (nvec >= 2048 && row_bytes <= 200 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(staged, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return TSB_ERR_LAUNCH | ((int)e << 8);
    long long per_sm = (long long)(224 * 1024 / (row_bytes + 2048));
    if (per_sm > 4) per_sm = 4;
    const long long grid = rows < per_sm * sm_count() ? rows : per_sm * sm_count();
    tsb_launch::launch(staged, dim3((unsigned)grid), dim3(threads), row_bytes, st, args...);
  } else {
    tsb_launch::launch(plain, dim3((unsigned)(rows < 148 * 16 ? rows : 148 * 16)), dim3(threads), 0, st, args...);
  }
  return done();
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

float* row_scratch(long long rows, cudaStream_t st) {
  return static_cast<float*>(tsb_scratch::get(st, tsb_scratch::LOSS_ROWS, (size_t)rows * sizeof(float),
                                              size_t(65536) * sizeof(float)));
}

// Gradient with dense labels, and the loss of every row where row_loss is given.
int ce_grad(const float* x, const float* labels, const float* g, float* dx, long long rows, long long cols, float* row_loss,
            cudaStream_t st) {
  const int grid = (int)(rows < 148 * 16 ? rows : 148 * 16), nvec = (int)(cols / 4);
  if (cols >= 512 && cols % 4 == 0 && cols / 4 < (1ll << 30) && aligned16(x) && aligned16(labels) && aligned16(dx)) {
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const DenseLabels lab{reinterpret_cast<const float4*>(labels), nullptr};
    float4* dx4 = reinterpret_cast<float4*>(dx);
    if (row_loss)
      return launch_rows(ce_grad_rows_v4<DenseLabels, false, true>, ce_grad_rows_v4<DenseLabels, true, true>, rows, nvec, st, x4,
                         lab, g, dx4, rows, nvec, row_loss);
    return launch_rows(ce_grad_rows_v4<DenseLabels, false, false>, ce_grad_rows_v4<DenseLabels, true, false>, rows, nvec, st, x4,
                       lab, g, dx4, rows, nvec, row_loss);
  }
  tsb_launch::launch(row_loss ? ce_grad_rows<true> : ce_grad_rows<false>, grid, cols >= 1024 ? 256 : 128, 0, st, x, labels, g, dx,
                     rows, cols, row_loss);
  return done();
}

}  // namespace

extern "C" {

int tsb_pool_fwd(int kind, const float* x, float* y, int n, int c, int h, int w, int oh, int ow, int kh, int kw,
                 int pad, int stride, long long xsn, long long xsh, long long xsw, long long ysn, long long ysh,
                 long long ysw, void* stream) {
  if ((c % 4) || (xsw % 4) || (ysw % 4)) return TSB_ERR_UNSUPPORTED;
  PoolP p{n, c, h, w, oh, ow, kh, kw, pad, stride, xsn, xsh, xsw, ysn, ysh, ysw};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Large windows whose outputs leave the one-thread-per-output form on less than a quarter of the SMs (8 x 8 windows:
  // 8 images of 1536 channels, 12 blocks: 10.3 -> 4.6 us; 32 of 2048, 64 blocks: 10.3 us and 12.7 us with a block per
  // window, and 28.7 against 89.7 us for 256 images).
  const long long outs = (long long)n * oh * ow;
  const int cblocks = (c / 4 + WIN_COLS - 1) / WIN_COLS;
  if (kind == 1 && kh * kw >= 2 * WIN_LANES && outs > 0 && outs * (c / 4) < 64ll * sm_count() && cblocks <= 65535) {
    const int splits = window_splits(outs * cblocks, kh * kw);
    tsb_launch::launch_cluster((unsigned)splits, avg_pool_window, dim3((unsigned)(outs * splits), (unsigned)cblocks),
                               dim3(WIN_COLS * WIN_LANES), 0, st, x, y, p);
    return done();
  }
  const long long work = outs * (c / 4);
  if (kh == kw && (kh == 2 || kh == 3) && work > 0 && work <= INT_MAX && h > 0 && w > 0) {
    const unsigned blocks = (unsigned)((work + 255) / 256), total = (unsigned)work;
    if (kind == 0 && kh == 2) tsb_launch::launch(pool_fwd_small<0, 2>, blocks, 256, 0, st, x, y, p, total);
    else if (kind == 0) tsb_launch::launch(pool_fwd_small<0, 3>, blocks, 256, 0, st, x, y, p, total);
    else if (kh == 2) tsb_launch::launch(pool_fwd_small<1, 2>, blocks, 256, 0, st, x, y, p, total);
    else tsb_launch::launch(pool_fwd_small<1, 3>, blocks, 256, 0, st, x, y, p, total);
    return done();
  }
  const int grid = ew_grid((long long)n * oh * ow * (c / 4));
  if (kind == 0) tsb_launch::launch(pool_fwd<0>, grid, 256, 0, st, x, y, p);
  else tsb_launch::launch(pool_fwd<1>, grid, 256, 0, st, x, y, p);
  return done();
}

int tsb_pool_bwd(int kind, const float* x, const float* y, const float* dy, float* dx, int n, int c, int h, int w,
                 int oh, int ow, int kh, int kw, int pad, int stride, long long xsn, long long xsh, long long xsw,
                 long long ysn, long long ysh, long long ysw, void* stream) {
  if ((c % 4) || (xsw % 4) || (ysw % 4)) return TSB_ERR_UNSUPPORTED;
  if (kind == 0 && (!x || !y)) return TSB_ERR_ARG;
  PoolP p{n, c, h, w, oh, ow, kh, kw, pad, stride, xsn, xsh, xsw, ysn, ysh, ysw};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (kh == stride && kw == stride && pad == 0 && oh * stride == h && ow * stride == w && (stride == 2 || stride == 3)) {
    const int tg = ew_grid((long long)n * oh * ow * (c / 4));
    if (kind == 0 && stride == 2) tsb_launch::launch(pool_bwd_tiled<0, 2>, tg, 256, 0, st, x, dy, dx, p);
    else if (kind == 0) tsb_launch::launch(pool_bwd_tiled<0, 3>, tg, 256, 0, st, x, dy, dx, p);
    else if (stride == 2) tsb_launch::launch(pool_bwd_tiled<1, 2>, tg, 256, 0, st, x, dy, dx, p);
    else tsb_launch::launch(pool_bwd_tiled<1, 3>, tg, 256, 0, st, x, dy, dx, p);
    return done();
  }
  if (kind == 1 && pad == 0 && kh <= stride && kw <= stride && n > 0 && h > 0 && (long long)n * h <= INT_MAX && c > 0) {
    tsb_launch::launch(avg_pool_bwd_rows, (unsigned)(n * h), 256, 0, st, dy, dx, p);
    return done();
  }
  const int grid = ew_grid((long long)n * h * w * (c / 4));
  if (kind == 0 && kh * kw < 255) {
    // windows that reach into 16 x 16 pixels, per axis; their gradients and positions in at most 48 KB
    const int nw = (16 + (kh > kw ? kh : kw) - 2) / stride + 1;
    const size_t smem = (size_t)nw * nw * 8 * (sizeof(float4) + sizeof(uchar4));
    const long long tiles_x = (w + 15) / 16, tiles = tiles_x * ((h + 15) / 16);
    if (smem <= 48 * 1024 && n <= 65535 && (c / 4 + 7) / 8 <= 65535 && tiles < (1ll << 31)) {
      const dim3 blocks((unsigned)tiles, (unsigned)((c / 4 + 7) / 8), (unsigned)n);
      if (kh == 3 && kw == 3 && stride == 2 && (pad == 0 || pad == 1))
        tsb_launch::launch(pad == 0 ? max_pool_bwd_3s2<0> : max_pool_bwd_3s2<1>, blocks, 256, 0, st, x, dy, dx, p, (int)tiles_x);
      else
        tsb_launch::launch(max_pool_bwd_tile, blocks, 256, smem, st, x, dy, dx, p, (int)tiles_x, nw);
      return done();
    }
    // overlapping windows: positions of the maxima first, then a gather per input pixel
    unsigned char* idx = argmax_scratch((size_t)n * oh * ow * c, st);
    if (idx) {
      tsb_launch::launch(pool_argmax, ew_grid((long long)n * oh * ow * (c / 4)), 256, 0, st, x, idx, p);
      tsb_launch::launch(pool_bwd_from_argmax, grid, 256, 0, st, idx, dy, dx, p);
      return done();
    }
  }
  if (kind == 0) tsb_launch::launch(pool_bwd<0>, grid, 256, 0, st, x, y, dy, dx, p);
  else tsb_launch::launch(pool_bwd<1>, grid, 256, 0, st, x, y, dy, dx, p);
  return done();
}

int tsb_softmax(const float* x, float* y, long long rows, long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cols <= 1024 && cols % 4 == 0 && aligned16(x) && aligned16(y)) {
    const int nvec = (int)(cols / 4);
    const long long blocks = (rows + 7) / 8;
    const int wgrid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
    const float4* xv = reinterpret_cast<const float4*>(x);
    float4* yv = reinterpret_cast<float4*>(y);
    if (nvec <= 32) tsb_launch::launch(softmax_warp_rows<1>, wgrid, 256, 0, st, xv, yv, rows, nvec);
    else if (nvec <= 64) tsb_launch::launch(softmax_warp_rows<2>, wgrid, 256, 0, st, xv, yv, rows, nvec);
    else if (nvec <= 128) tsb_launch::launch(softmax_warp_rows<4>, wgrid, 256, 0, st, xv, yv, rows, nvec);
    else tsb_launch::launch(softmax_warp_rows<8>, wgrid, 256, 0, st, xv, yv, rows, nvec);
    return done();
  }
  if (cols <= 1024) {
    const long long blocks = (rows + 7) / 8;
    const int wgrid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
    const int c = (int)cols;
    if (c <= 64) tsb_launch::launch(softmax_warp_rows_scalar<2>, wgrid, 256, 0, st, x, y, rows, c);
    else if (c <= 128) tsb_launch::launch(softmax_warp_rows_scalar<4>, wgrid, 256, 0, st, x, y, rows, c);
    else if (c <= 256) tsb_launch::launch(softmax_warp_rows_scalar<8>, wgrid, 256, 0, st, x, y, rows, c);
    else if (c <= 512) tsb_launch::launch(softmax_warp_rows_scalar<16>, wgrid, 256, 0, st, x, y, rows, c);
    else tsb_launch::launch(softmax_warp_rows_scalar<32>, wgrid, 256, 0, st, x, y, rows, c);
    return done();
  }
  const int grid = (int)(rows < 148 * 16 ? rows : 148 * 16);
  tsb_launch::launch(softmax_rows, grid, cols >= 1024 ? 256 : 128, 0, st, x, y, rows, cols);
  return done();
}

int tsb_softmax_grad(const float* y, const float* dy, float* dx, long long rows, long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cols <= 1024 && cols % 4 == 0 && aligned16(y) && aligned16(dy) && aligned16(dx)) {
    const int nvec = (int)(cols / 4);
    const long long blocks = (rows + 7) / 8;
    const int wgrid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
    const float4* yv = reinterpret_cast<const float4*>(y);
    const float4* gv = reinterpret_cast<const float4*>(dy);
    float4* dv = reinterpret_cast<float4*>(dx);
    if (nvec <= 32) tsb_launch::launch(softmax_grad_warp_rows<1>, wgrid, 256, 0, st, yv, gv, dv, rows, nvec);
    else if (nvec <= 64) tsb_launch::launch(softmax_grad_warp_rows<2>, wgrid, 256, 0, st, yv, gv, dv, rows, nvec);
    else if (nvec <= 128) tsb_launch::launch(softmax_grad_warp_rows<4>, wgrid, 256, 0, st, yv, gv, dv, rows, nvec);
    else tsb_launch::launch(softmax_grad_warp_rows<8>, wgrid, 256, 0, st, yv, gv, dv, rows, nvec);
    return done();
  }
  if (cols <= 1024) {
    const long long blocks = (rows + 7) / 8;
    const int wgrid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
    const int c = (int)cols;
    if (c <= 64) tsb_launch::launch(softmax_grad_warp_rows_scalar<2>, wgrid, 256, 0, st, y, dy, dx, rows, c);
    else if (c <= 128) tsb_launch::launch(softmax_grad_warp_rows_scalar<4>, wgrid, 256, 0, st, y, dy, dx, rows, c);
    else if (c <= 256) tsb_launch::launch(softmax_grad_warp_rows_scalar<8>, wgrid, 256, 0, st, y, dy, dx, rows, c);
    else if (c <= 512) tsb_launch::launch(softmax_grad_warp_rows_scalar<16>, wgrid, 256, 0, st, y, dy, dx, rows, c);
    else tsb_launch::launch(softmax_grad_warp_rows_scalar<32>, wgrid, 256, 0, st, y, dy, dx, rows, c);
    return done();
  }
  const int grid = (int)(rows < 148 * 16 ? rows : 148 * 16);
  tsb_launch::launch(softmax_grad_rows, grid, cols >= 1024 ? 256 : 128, 0, st, y, dy, dx, rows, cols);
  return done();
}

// y = softmax(scale * x + key-padding mask [+ causal mask]) row-wise; rows = batch * rows_per_batch, query index
// of a row = row % tq.  cols <= 1024 (TSB_ERR_UNSUPPORTED beyond: the caller composes the operators instead).
int tsb_masked_softmax(const float* x, const float* key_tokens, float* y, long long rows, long long cols,
                       long long rows_per_batch, int tq, float scale, int causal, void* stream) {
  if (rows <= 0 || cols <= 0 || rows_per_batch <= 0 || tq <= 0) return TSB_ERR_ARG;
  if (cols > 1024 || rows >= (1ll << 31) || rows_per_batch >= (1ll << 31)) return TSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long blocks = (rows + 7) / 8;
  const int wgrid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
  const int c = (int)cols;
  if (c % 4 == 0 && aligned16(x) && aligned16(y) && (!key_tokens || aligned16(key_tokens))) {
    const int nvec = c / 4;
    const float4* xv = reinterpret_cast<const float4*>(x);
    const float4* kv = reinterpret_cast<const float4*>(key_tokens);
    float4* yv = reinterpret_cast<float4*>(y);
#define TSB_MSV(NV) tsb_launch::launch(masked_softmax_warp_rows_v4<NV>, wgrid, 256, 0, st, xv, kv, yv, rows, nvec, \
                                       rows_per_batch, tq, scale, causal)
    if (nvec <= 32) TSB_MSV(1);
    else if (nvec <= 64) TSB_MSV(2);
    else if (nvec <= 128) TSB_MSV(4);
    else TSB_MSV(8);
#undef TSB_MSV
    return done();
  }
#define TSB_MSM(NE) tsb_launch::launch(masked_softmax_warp_rows<NE>, wgrid, 256, 0, st, x, key_tokens, y, rows, c, \
                                       rows_per_batch, tq, scale, causal)
  if (c <= 64) TSB_MSM(2);
  else if (c <= 128) TSB_MSM(4);
  else if (c <= 256) TSB_MSM(8);
  else if (c <= 512) TSB_MSM(16);
  else TSB_MSM(32);
#undef TSB_MSM
  return done();
}

int tsb_scaled_softmax_grad(const float* y, const float* dy, float* dx, long long rows, long long cols, float scale,
                            void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  if (cols > 1024) return TSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const long long blocks = (rows + 7) / 8;
  const int wgrid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
  const int c = (int)cols;
  if (c % 4 == 0 && aligned16(y) && aligned16(dy) && aligned16(dx)) {
    const int nvec = c / 4;
    const float4* yv = reinterpret_cast<const float4*>(y);
    const float4* gv = reinterpret_cast<const float4*>(dy);
    float4* dv = reinterpret_cast<float4*>(dx);
#define TSB_SSV(NV) tsb_launch::launch(scaled_softmax_grad_warp_rows_v4<NV>, wgrid, 256, 0, st, yv, gv, dv, rows, \
                                       nvec, scale)
    if (nvec <= 32) TSB_SSV(1);
    else if (nvec <= 64) TSB_SSV(2);
    else if (nvec <= 128) TSB_SSV(4);
    else TSB_SSV(8);
#undef TSB_SSV
    return done();
  }
#define TSB_SSG(NE) tsb_launch::launch(scaled_softmax_grad_warp_rows<NE>, wgrid, 256, 0, st, y, dy, dx, rows, c, scale)
  if (c <= 64) TSB_SSG(2);
  else if (c <= 128) TSB_SSG(4);
  else if (c <= 256) TSB_SSG(8);
  else if (c <= 512) TSB_SSG(16);
  else TSB_SSG(32);
#undef TSB_SSG
  return done();
}

int tsb_softmax_ce(const float* x, const float* labels, float* loss, long long rows, long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* rl = row_scratch(rows, st);
  if (!rl) return TSB_ERR_OOM;
  const int grid = (int)(rows < 148 * 16 ? rows : 148 * 16);
  if (cols >= 512 && cols % 4 == 0 && cols / 4 < (1ll << 30) && aligned16(x) && aligned16(labels)) {
    const int rc = launch_rows(ce_rows_v4<DenseLabels, false>, ce_rows_v4<DenseLabels, true>, rows, (int)(cols / 4), st,
                               reinterpret_cast<const float4*>(x),
                               DenseLabels{reinterpret_cast<const float4*>(labels), nullptr}, rl, rows, (int)(cols / 4));
    if (rc) return rc;
    tsb_launch::launch(mean_rows, 1, 1024, 0, st, rl, loss, rows);
    return done();
  }
  tsb_launch::launch(ce_rows, grid, cols >= 1024 ? 256 : 128, 0, st, x, labels, rl, rows, cols);
  tsb_launch::launch(mean_rows, 1, 1024, 0, st, rl, loss, rows);
  return done();
}

int tsb_softmax_ce_grad(const float* x, const float* labels, const float* g, float* dx, long long rows,
                        long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  return ce_grad(x, labels, g, dx, rows, cols, nullptr, static_cast<cudaStream_t>(stream));
}

// Loss (the mean of the rows) and gradient from one pass over the logits.
int tsb_softmax_ce_both(const float* x, const float* labels, const float* g, float* loss, float* dx, long long rows,
                        long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* rl = row_scratch(rows, st);
  if (!rl) return TSB_ERR_OOM;
  const int rc = ce_grad(x, labels, g, dx, rows, cols, rl, st);
  if (rc) return rc;
  tsb_launch::launch(mean_rows, 1, 1024, 0, st, rl, loss, rows);
  return done();
}

// The same with labels that are `on` at a row's class id and `off` elsewhere (an id outside the classes: `off`
// everywhere).  TSB_ERR_UNSUPPORTED where the dense entries would not take their long-row kernels.
int tsb_softmax_ce_smooth(const float* x, const float* ids, float on, float off, float* loss, long long rows,
                          long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  if (cols < 512 || cols % 4 || cols / 4 >= (1ll << 30) || !aligned16(x)) return TSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* rl = row_scratch(rows, st);
  if (!rl) return TSB_ERR_OOM;
  tsb_launch::launch(ce_smooth_rows_v4, dim3((unsigned)(rows < 148 * 16 ? rows : 148 * 16)),
                     dim3(cols >= 8192 ? 512 : 256), 0, st, reinterpret_cast<const float4*>(x),
                     SmoothLabels{ids, on, off, 0}, rl, rows, (int)(cols / 4));
  tsb_launch::launch(mean_rows, 1, 1024, 0, st, rl, loss, rows);
  return done();
}

int tsb_softmax_ce_grad_smooth(const float* x, const float* ids, float on, float off, const float* g, float* dx,
                               long long rows, long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  if (cols < 512 || cols % 4 || cols / 4 >= (1ll << 30) || !aligned16(x) || !aligned16(dx)) return TSB_ERR_UNSUPPORTED;
  return launch_rows(ce_grad_rows_v4<SmoothLabels, false, false>, ce_grad_rows_v4<SmoothLabels, true, false>, rows, (int)(cols / 4),
                     static_cast<cudaStream_t>(stream), reinterpret_cast<const float4*>(x),
                     SmoothLabels{ids, on, off, 0}, g, reinterpret_cast<float4*>(dx), rows, (int)(cols / 4), (float*)nullptr);
}

int tsb_softmax_ce_both_smooth(const float* x, const float* ids, float on, float off, const float* g, float* loss, float* dx,
                               long long rows, long long cols, void* stream) {
  if (rows <= 0 || cols <= 0) return TSB_ERR_ARG;
  if (cols < 512 || cols % 4 || cols / 4 >= (1ll << 30) || !aligned16(x) || !aligned16(dx)) return TSB_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* rl = row_scratch(rows, st);
  if (!rl) return TSB_ERR_OOM;
  const int rc = launch_rows(ce_grad_rows_v4<SmoothLabels, false, true>, ce_grad_rows_v4<SmoothLabels, true, true>, rows,
                             (int)(cols / 4), st, reinterpret_cast<const float4*>(x), SmoothLabels{ids, on, off, 0}, g,
                             reinterpret_cast<float4*>(dx), rows, (int)(cols / 4), rl);
  if (rc) return rc;
  tsb_launch::launch(mean_rows, 1, 1024, 0, st, rl, loss, rows);
  return done();
}

}  // extern "C"
