// Colour and light passes (the reference's setCell outputs other than the cell id),
// shaders/compute/operations.glsl:99-169 with math.glsl:40-44,82-106.
//
// Every float operation is an explicit round-to-nearest intrinsic in the shader's order, so
// nothing is contracted into FMAs: the light pass and the colour equal a strict-IEEE CPU
// evaluation bit for bit.  GLSL leaves the precision of sin to the driver; the colour's
// noise fixes it to se_sin (below), which the CPU oracle evaluates with the same binary64
// operations.
#include "noise_sin.cuh"
#include "render.hpp"

#include <algorithm>

namespace se::rt {
namespace {

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
// GLSL max / min / clamp as the spec defines them (max(a, b) = a < b ? b : a)
__device__ __forceinline__ float gmax(float a, float b) { return a < b ? b : a; }
__device__ __forceinline__ float gmin(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float gclamp(float x, float lo, float hi) { return gmin(gmax(x, lo), hi); }

// old_hash2 component: -1 + 2 * fract(sin(q) * 43758.5453123)
__device__ __forceinline__ float grad_component(float q) {
  const float v = fmul(se_sin_fast(q), 43758.5453123f);
  return fadd(-1.0f, fmul(2.0f, fsub(v, floorf(v))));
}
// old_hash2: the gradient at a lattice point
__device__ __forceinline__ float2 grad(float qx, float qy) {
  const float gx = grad_component(fadd(fmul(qx, 127.1f), fmul(qy, 311.7f)));
  const float gy = grad_component(fadd(fmul(qx, 269.5f), fmul(qy, 183.3f)));
  return make_float2(gx, gy);
}

// The lattice point below p in _noise's skewed grid.
__device__ __forceinline__ float2 simplex_base(float px, float py) {
  const float s = fmul(fadd(px, py), 0.366025404f);
  return make_float2(floorf(fadd(px, s)), floorf(fadd(py, s)));
}
// p relative to the point i, and _noise's choice of the second corner: i + (ox, 1 - ox)
__device__ __forceinline__ float simplex_offset(float px, float py, float2 i, float2& a) {
  const float t = fmul(fadd(i.x, i.y), 0.211324865f);
  a = make_float2(fadd(fsub(px, i.x), t), fadd(fsub(py, i.y), t));
  return a.x < a.y ? 0.0f : 1.0f;  // step(a.y, a.x)
}
// _noise: 2D simplex noise from p's offset a, ox and the gradients at the three corners
__device__ __forceinline__ float simplex(float2 a, float ox, float2 g0, float2 g1, float2 g2) {
  const float K2 = 0.211324865f;
  const float oy = fsub(1.0f, ox);
  const float bx = fadd(fsub(a.x, ox), K2), by = fadd(fsub(a.y, oy), K2);
  const float c2 = fmul(2.0f, K2);
  const float cx = fadd(fsub(a.x, 1.0f), c2), cy = fadd(fsub(a.y, 1.0f), c2);
  const float h0 = gmax(fsub(0.5f, fadd(fmul(a.x, a.x), fmul(a.y, a.y))), 0.0f);
  const float h1 = gmax(fsub(0.5f, fadd(fmul(bx, bx), fmul(by, by))), 0.0f);
  const float h2 = gmax(fsub(0.5f, fadd(fmul(cx, cx), fmul(cy, cy))), 0.0f);
  const float n0 = fmul(fmul(fmul(fmul(h0, h0), h0), h0), fadd(fmul(a.x, g0.x), fmul(a.y, g0.y)));
  const float n1 = fmul(fmul(fmul(fmul(h1, h1), h1), h1), fadd(fmul(bx, g1.x), fmul(by, g1.y)));
  const float n2 = fmul(fmul(fmul(fmul(h2, h2), h2), h2), fadd(fmul(cx, g2.x), fmul(cy, g2.y)));
  return fadd(0.25f, fmul(0.5f, fadd(fadd(fmul(n0, 70.0f), fmul(n1, 70.0f)), fmul(n2, 70.0f))));
}

// The 2D kernels take their row blocks from by0 + blockIdx.y: a tall world is covered by
// several launches, as a grid's y extent stops at 65535.
//
// noise(p, 3 octaves, lacunarity 2, frequency 0.25): octave o samples simplex noise at p 2^o / 4.
// Bound by the sines of the gradients, two a lattice point.  A 32 x 32 tile has 0.11, 0.43
// and 1.73 points a cell in its three octaves, which every cell would evaluate for its nine
// corners again; so the tile marks the points that its cells use, evaluates these once and
// keeps them in shared memory.  A world's first image, allocation included (nine points a cell in
// binary64 / this): 64 x 64 98 / 31 us, 1920 x 1080 4405 / 174, 3001 x 2003 12535 / 358,
// 8192 x 8192 138 ms / 3.2.
// The first cell's point bounds those of the others from below, as every operation on the way is
// monotone; sides of at most 2^20 cells keep the coordinates below 2^21, where they are off by less
// than 0.1, so 31 cells span at most 31 (1 + 2 * 0.366) 2^o / 4 + 0.2 points either way.
constexpr int kNoiseTile = 32;
// lattice points along a tile's side in octave o, skew and second corner included
__host__ __device__ constexpr int noise_side(int o) { return o == 0 ? 16 : o == 1 ? 30 : 56; }
// where octave o begins in the shared array
__host__ __device__ constexpr int noise_base(int o) {
  return o == 0 ? 0 : o == 1 ? 16 * 16 : o == 2 ? 16 * 16 + 30 * 30 : 16 * 16 + 30 * 30 + 56 * 56;
}
constexpr int kNoisePoints = noise_base(3);

__global__ void __launch_bounds__(256) se_noise_kernel(float* __restrict__ out, int W, int H, int by0) {
  __shared__ float2 val[kNoisePoints];
  __shared__ uint16_t list[kNoisePoints];  // octave << 12 | row << 6 | column
  __shared__ int count;
  const int x0 = blockIdx.x * kNoiseTile, y0 = (by0 + blockIdx.y) * kNoiseTile;
  const int lane = threadIdx.x & 31, x = x0 + lane;
  const int rows = x < W ? min(kNoiseTile, H - y0) : 0, row0 = threadIdx.x >> 5;
  float2 lo[3];
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    const float sc = 0.25f * (1 << o);
    lo[o] = simplex_base(fmul((float)x0, sc), fmul((float)y0, sc));
  }
  for (int i = threadIdx.x; i < kNoisePoints; i += 256) val[i].x = 0.0f;
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  // the first corner's place in val, the second's beside or below it, the third's across
  const auto corners = [&](int o, int y, float2& a, float& ox, int& c0, int& c1) {
    const float sc = 0.25f * (1 << o), px = fmul((float)x, sc), py = fmul((float)y, sc);
    const float2 i = simplex_base(px, py);
    ox = simplex_offset(px, py, i, a);
    c0 = noise_base(o) + (int)(i.y - lo[o].y) * noise_side(o) + (int)(i.x - lo[o].x);
    c1 = c0 + (ox != 0.0f ? 1 : noise_side(o));
  };
  for (int r = row0; r < rows; r += 8) {
    const int y = y0 + r;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      float2 a;
      float ox;
      int c0, c1;
      corners(o, y, a, ox, c0, c1);
      val[c0].x = 1.0f;
      val[c1].x = 1.0f;
      val[c0 + noise_side(o) + 1].x = 1.0f;
    }
  }
  __syncthreads();
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    for (int i = threadIdx.x; i < ((noise_base(o + 1) - noise_base(o) + 31) & ~31); i += 256) {
      const bool used = i < noise_base(o + 1) - noise_base(o) && val[noise_base(o) + i].x != 0.0f;
      const unsigned who = __ballot_sync(0xffffffffu, used);
      int at = 0;
      if (lane == 0 && who) at = atomicAdd(&count, __popc(who));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(who & ((1u << lane) - 1u));
      if (used) list[at] = (uint16_t)(o << 12 | (i / noise_side(o)) << 6 | i % noise_side(o));
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < count; i += 256) {
    const int p = list[i], o = p >> 12, row = p >> 6 & 63, col = p & 63;
    const float2 b = o == 0 ? lo[0] : o == 1 ? lo[1] : lo[2];
    const int at = noise_base(o) + row * noise_side(o) + col;
    val[at] = grad(fadd(b.x, (float)col), fadd(b.y, (float)row));
  }
  __syncthreads();
  for (int r = row0; r < rows; r += 8) {
    const int y = y0 + r;
    float f = 0.0f;
#pragma unroll
    for (int o = 0; o < 3; ++o) {
      float2 a;
      float ox;
      int c0, c1;
      corners(o, y, a, ox, c0, c1);
      f = fadd(f, fmul(__fdiv_rn(1.0f, (float)(o + 1)),
                       simplex(a, ox, val[c0], val[c1], val[c0 + noise_side(o) + 1])));
    }
    out[(size_t)y * W + x] = f;
  }
}

__device__ __forceinline__ uint32_t mat_index(uint32_t id, int nmat) { return id < (uint32_t)nmat ? id : 1u; }

// One cell per thread, grid-stride: id, cached noise -> RGBA32F.
__global__ void __launch_bounds__(256) se_color_kernel(const uint32_t* __restrict__ grid,
                                                       const float* __restrict__ noise, float4* __restrict__ out,
                                                       long long n, const RenderMat* __restrict__ mats, int nmat) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint32_t m = mat_index(__ldg(grid + i), nmat);
    float4 c = __ldg(reinterpret_cast<const float4*>(mats[m].color));
    if (m != 0u) {  // kRenderNoise: every material but EMPTY
      const float d = fmul(__ldg(noise + i), 0.25f);
      c.x = gclamp(fsub(c.x, d), 0.0f, 1.0f);
      c.y = gclamp(fsub(c.y, d), 0.0f, 1.0f);
      c.z = gclamp(fsub(c.z, d), 0.0f, 1.0f);
    }
    out[i] = c;
  }
}

// The colour of one cell and its alpha.
__device__ __forceinline__ float4 cell_color(uint32_t id, float nz, const RenderMat* __restrict__ mats, int nmat) {
  const uint32_t m = mat_index(id, nmat);
  float4 c = __ldg(reinterpret_cast<const float4*>(mats[m].color));
  if (m != 0u) {  // kRenderNoise: every material but EMPTY
    const float d = fmul(nz, 0.25f);
    c.x = gclamp(fsub(c.x, d), 0.0f, 1.0f);
    c.y = gclamp(fsub(c.y, d), 0.0f, 1.0f);
    c.z = gclamp(fsub(c.z, d), 0.0f, 1.0f);
  }
  return c;
}

// One texel of a pyramid level from its four sources; at a level one texel wide or high the
// second source index is clamped, as sampling is.
__device__ __forceinline__ float mip_texel(float a, float b, float c, float d, int sw, int sh) {
  if (sw == 1) b = a, d = c;
  if (sh == 1) c = a, d = b;
  return fmul(fadd(fadd(fadd(a, b), c), d), 0.25f);
}

__device__ __forceinline__ float cell_alpha(uint32_t id, const RenderMat* __restrict__ mats, int nmat) {
  return __ldg(&mats[mat_index(id, nmat)].color[3]);
}

// Levels 1 to 4 of the alpha pyramid in one pass over the ids: a cell's alpha is its material's.
// A thread takes 2 x 2 cells (a texel of level 1), a warp 16 x 8 cells, whose texels of levels 2 and 3
// it reduces by shuffles, and a CTA 64 x 16, whose texels of level 4 need one barrier;
// se_mip_tail_kernel makes levels 5 and 6 (no larger lod is sampled).  A launch per level cost 3-4 us
// each; with the colours written in the same pass 1920 x 1080 takes 20.4 us and 8192 x 8192 279, the
// pyramid alone (both kernels) 12.2 and 135.  64 x 64 cells a CTA with all six levels reduced in shared memory kept
// too few loads in flight between its barriers (8192 x 8192 with colours: 323 and 545 us with 256 and 1024
// threads, 283 so).
// Block (bx, by) of 64 x 16 cells by threads t = 0 .. 255 (whole CTAs take part; blocks beyond the world
// write nothing).
__device__ __forceinline__ void mip_block(const uint32_t* __restrict__ grid, const MipLevels& mip, int W, int H,
                                          const RenderMat* __restrict__ mats, int nmat, int bx, int by, int t,
                                          float (*s3)[8]) {
  const int lane = t & 31, wx = (t >> 5) & 3, wy = t >> 7;
  const int x = bx * 32 + wx * 8 + (lane & 7), y = by * 8 + wy * 4 + (lane >> 3);
  const int c0 = 2 * x, r0 = 2 * y;
  float v = 0.0f;
  if (c0 < W && r0 < H) {
    const bool pair = c0 + 1 < W;
    float a[2][2];
#pragma unroll
    for (int dr = 0; dr < 2; ++dr) {
      const int r = min(r0 + dr, H - 1);  // at an odd last row or column the pair's second index is clamped
      const size_t i = (size_t)r * W + c0;
      uint32_t id0, id1;
      if (pair && (W & 1) == 0) {  // 8-byte aligned pairs
        const uint2 g = __ldg(reinterpret_cast<const uint2*>(grid + i));
        id0 = g.x, id1 = g.y;
      } else {
        id0 = __ldg(grid + i);
        id1 = pair ? __ldg(grid + i + 1) : id0;
      }
      a[dr][0] = cell_alpha(id0, mats, nmat);
      a[dr][1] = cell_alpha(id1, mats, nmat);
    }
    if (mip.levels == 1) mip.level[1][0] = a[0][0];  // one cell
    v = fmul(fadd(fadd(fadd(a[0][0], a[0][1]), a[1][0]), a[1][1]), 0.25f);
    if (mip.levels > 1 && x < mip.w[1] && y < mip.h[1]) mip.level[1][(size_t)y * mip.w[1] + x] = v;
  }
  if (mip.levels <= 2) return;  // uniform
#pragma unroll
  for (int l = 2; l <= 3; ++l) {  // lanes whose column and row are multiples of 2^(l-1) hold a texel
    const int d = 1 << (l - 2), m = 2 * d - 1;
    const float b = __shfl_down_sync(0xffffffffu, v, d), c = __shfl_down_sync(0xffffffffu, v, 8 * d),
                e = __shfl_down_sync(0xffffffffu, v, 9 * d);
    v = mip_texel(v, b, c, e, mip.w[l - 1], mip.h[l - 1]);
    const int tx = x >> (l - 1), ty = y >> (l - 1);
    if (l < mip.levels && !(lane & m) && !((lane >> 3) & m) && tx < mip.w[l] && ty < mip.h[l])
      mip.level[l][(size_t)ty * mip.w[l] + tx] = v;
  }
  if (mip.levels <= 4) return;
  if (lane == 0 || lane == 4) s3[wy][wx * 2 + (lane >> 2)] = v;
  __syncthreads();
  if (t < 4) {
    const int i = t, tx = bx * 4 + i;
    if (tx < mip.w[4] && by < mip.h[4])
      mip.level[4][(size_t)by * mip.w[4] + tx] =
          mip_texel(s3[0][2 * i], s3[0][2 * i + 1], s3[1][2 * i], s3[1][2 * i + 1], mip.w[3], mip.h[3]);
  }
}

__global__ void __launch_bounds__(256) se_mip_kernel(const uint32_t* __restrict__ grid, const MipLevels mip, int W,
                                                     int H, const RenderMat* __restrict__ mats, int nmat, int by0) {
  __shared__ float s3[2][8];
  mip_block(grid, mip, W, H, mats, nmat, blockIdx.x, by0 + blockIdx.y, threadIdx.x, s3);
}

// A load: of what an earlier launch wrote, or (SAME) this launch itself, before a barrier.
template <bool SAME, class T>
__device__ __forceinline__ T load(const T* p) {
  if constexpr (SAME)
    return *p;
  else
    return __ldg(p);
}

// Levels 5 and 6 from level 4: thread t takes the 4 x 4 texels of level 4 under a texel of level 6.
template <bool SAME>
__device__ __forceinline__ void mip_tail(const MipLevels& mip, int t) {
  const int w4 = mip.w[4], h4 = mip.h[4], w5 = mip.w[5], h5 = mip.h[5];
  const int nx = (w5 + 1) / 2;
  const int X = t % nx, Y = t / nx;
  if (2 * Y >= h5) return;
  float a[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      a[j][i] = load<SAME>(mip.level[4] + (size_t)min(4 * Y + j, h4 - 1) * w4 + min(4 * X + i, w4 - 1));
  float b[2][2];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      b[j][i] = mip_texel(a[2 * j][2 * i], a[2 * j][2 * i + 1], a[2 * j + 1][2 * i], a[2 * j + 1][2 * i + 1], w4, h4);
      if (2 * X + i < w5 && 2 * Y + j < h5) mip.level[5][(size_t)(2 * Y + j) * w5 + 2 * X + i] = b[j][i];
    }
  if (mip.levels > 6 && X < mip.w[6] && Y < mip.h[6])
    mip.level[6][(size_t)Y * mip.w[6] + X] = mip_texel(b[0][0], b[0][1], b[1][0], b[1][1], w5, h5);
}
__global__ void __launch_bounds__(128) se_mip_tail_kernel(const MipLevels mip) {
  mip_tail<false>(mip, blockIdx.x * 128 + threadIdx.x);
}

// Light pass over a 64 x 4R tile per CTA.  The tile plus a one-cell ring is staged in
// shared memory as each cell's contribution to its neighbours' blend,
// (rgb * keep * a, a) for its previous light (rgb, a), where keep is 0 when its old cell is a
// light obstacle, else 1; plus a byte that marks cells outside the world.
// Thread t computes the cells (t % 64, t / 64 + 4 j), j < R: a warp touches 32 consecutive
// cells of a row, so shared-memory reads and global loads / stores are contiguous.
constexpr int LTW = 64, LSW = LTW + 2;

// GLSL max (a < b ? b : a).  CLEAN: neither argument is NaN or -0, where the hardware
// maximum returns the same value in one instruction instead of a compare and a select.
template <bool CLEAN>
__device__ __forceinline__ float lmax(float a, float b) {
  return CLEAN ? fmaxf(a, b) : gmax(a, b);
}

// The 8-neighbour blend for the staged cell s0.  INTERIOR: all 8 neighbours lie in the
// world (no checks; the mean's division by 8 is the product by 0.125, the same correctly
// rounded quotient).  CLEAN: every staged value is a non-negative number or +inf (so are
// the running maxima, which start at +0).
template <bool INTERIOR, bool CLEAN>
__device__ __forceinline__ float4 light_blend(const float4* sl, const uint8_t* sk, int s0) {
  // neighbours in getDiagonalNeighbours order: DOWN, UP, DOWNLEFT, UPLEFT, DOWNRIGHT,
  // UPRIGHT, RIGHT, LEFT (offsets in the staged array)
  constexpr int NOFF[8] = {LSW, -LSW, LSW - 1, -LSW - 1, LSW + 1, -LSW + 1, 1, -1};
  float a0 = 0.0f, a1 = 0.0f, a2 = 0.0f, a3 = 0.0f, m0 = 0.0f, m1 = 0.0f, m2 = 0.0f, maxf = 0.0f;
  int num = 0;
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const int s = s0 + NOFF[n];
    if (!INTERIOR && sk[s]) continue;  // outside the world
    const float4 c = sl[s];
    const float t0 = c.x, t1 = c.y, t2 = c.z, a = c.w;
    const float falloff = a == 0.0f ? maxf : a;
    a0 = fadd(a0, t0);
    a1 = fadd(a1, t1);
    a2 = fadd(a2, t2);
    a3 = fadd(a3, falloff);
    // clean: a == 0 leaves maxf (>= +0) as it is either way, so the running maximum need
    // not wait for the falloff select
    maxf = CLEAN ? fmaxf(a, maxf) : gmax(falloff, maxf);
    ++num;
    m0 = lmax<CLEAN>(m0, t0);  // the alpha of the maximum is not used (mix takes .rgb)
    m1 = lmax<CLEAN>(m1, t1);
    m2 = lmax<CLEAN>(m2, t2);
  }
  if (INTERIOR) {
    a0 = fmul(a0, 0.125f);
    a1 = fmul(a1, 0.125f);
    a2 = fmul(a2, 0.125f);
    a3 = fmul(a3, 0.125f);
  } else if (num > 0) {
    const float fn = (float)num;
    a0 = __fdiv_rn(a0, fn);
    a1 = __fdiv_rn(a1, fn);
    a2 = __fdiv_rn(a2, fn);
    a3 = __fdiv_rn(a3, fn);
  }
  // mix(avg.rgb, max.rgb, 0.5) = avg * (1 - 0.5) + max * 0.5
  return make_float4(fadd(fmul(a0, 0.5f), fmul(m0, 0.5f)), fadd(fmul(a1, 0.5f), fmul(m1, 0.5f)),
                     fadd(fmul(a2, 0.5f), fmul(m2, 0.5f)), a3);
}

// TALL: the row blocks start at by0 (a world with more than 65535 of them takes several
// launches); otherwise by0 is 0 and unused, which keeps the common kernel's code as tight
// as it measured best.
template <bool TALL, int R>
__global__ void __launch_bounds__(256, 5) se_light_kernel(const uint32_t* __restrict__ old_grid,
                                                       const uint32_t* __restrict__ new_grid,
                                                       const float4* __restrict__ lin, float4* __restrict__ lout,
                                                       int W, int H, const RenderMat* __restrict__ mats, int nmat,
                                                       int by0) {
  constexpr int LTH = 4 * R, NT = 256, NS = LSW * (LTH + 2), NU = (NS + NT - 1) / NT;
  __shared__ float4 sl[NS];  // contribution (rgb * keep * a, a) per staged cell
  __shared__ uint8_t sk[NS];  // 1: outside the world
  const int X0 = blockIdx.x * LTW, Y0 = (TALL ? by0 + (int)blockIdx.y : (int)blockIdx.y) * LTH;
  // Issue every global load of this thread first (staged ids and light, then the new ids
  // of its four cells), so that they are in flight together.
  uint32_t ids[NU];
  float4 ls[NU];
  bool in[NU];
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int i = threadIdx.x + u * NT;
    const int r = i / LSW, c = i - r * LSW;
    const int gx = X0 - 1 + c, gy = Y0 - 1 + r;
    in[u] = i < NS && gx >= 0 && gy >= 0 && gx < W && gy < H;
    if (in[u]) {
      const size_t q = (size_t)gy * W + gx;
      ids[u] = __ldg(old_grid + q);
      ls[u] = __ldg(lin + q);
    }
  }
  const int cx = threadIdx.x & 63;
  uint32_t nid[R];
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int x = X0 + cx, y = Y0 + (threadIdx.x >> 6) + 4 * j;
    nid[j] = (x < W && y < H) ? __ldg(new_grid + (size_t)y * W + x) : 0u;
  }
  uint32_t top = 0;  // the largest bit pattern staged by this thread
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    const int i = threadIdx.x + u * NT;
    if (i >= NS) break;
    if (in[u]) {
      const float keep = (__ldg(&mats[mat_index(ids[u], nmat)].flags) & kRenderObstacle) ? 0.0f : 1.0f;
      const float4 l = ls[u];
      // light_data = light * vec4(vec3(keep), 1.0); contribution = (light_data.rgb * a, a)
      const float4 c =
          make_float4(fmul(fmul(l.x, keep), l.w), fmul(fmul(l.y, keep), l.w), fmul(fmul(l.z, keep), l.w), l.w);
      sl[i] = c;
      sk[i] = 0;
      top = max(top, max(max(__float_as_uint(c.x), __float_as_uint(c.y)),
                         max(__float_as_uint(c.z), __float_as_uint(c.w))));
    } else {
      sl[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      sk[i] = 1;
    }
  }
  // Patterns up to 0x7f800000 are +0 .. +inf: no NaN, no -0 (nor any negative value).
  const bool clean = !__syncthreads_or(top > 0x7f800000u);
  const bool interior = X0 >= 1 && Y0 >= 1 && X0 + LTW + 1 <= W && Y0 + LTH + 1 <= H;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int cy = (threadIdx.x >> 6) + 4 * j;
    const int x = X0 + cx, y = Y0 + cy;
    if (x >= W || y >= H) continue;
    const RenderMat* nm = mats + mat_index(nid[j], nmat);
    float4 L;
    if (__ldg(&nm->flags) & kRenderEmits) {
      L = make_float4(__ldg(nm->emission + 0), __ldg(nm->emission + 1), __ldg(nm->emission + 2),
                      __ldg(nm->emission + 3));
    } else if (y == 0) {
      L = make_float4(1.0f, 1.0f, 1.0f, 0.999999f);
    } else {
      const int s0 = (cy + 1) * LSW + cx + 1;
      if (clean)
        L = interior ? light_blend<true, true>(sl, sk, s0) : light_blend<false, true>(sl, sk, s0);
      else
        L = interior ? light_blend<true, false>(sl, sk, s0) : light_blend<false, false>(sl, sk, s0);
    }
    lout[(size_t)y * W + x] = L;
  }
}

// ---- headless composite ---------------------------------------------------------------
__device__ __forceinline__ int mirror_index(int i, int n) {  // GL_MIRRORED_REPEAT on texel indices
  if ((unsigned)i < (unsigned)n) return i;  // almost every tap
  if (i == -1) return 0;
  if (i == n) return n - 1;
  const int p = 2 * n;
  int m = i % p;
  if (m < 0) m += p;
  return m >= n ? p - 1 - m : m;
}
__device__ __forceinline__ float4 tap(const float4* t, int w, int h, int i, int j) {
  return __ldg(t + (size_t)mirror_index(j, h) * w + mirror_index(i, w));
}
__device__ __forceinline__ float lerp4(float t00, float t10, float t01, float t11, float w00, float w10, float w01,
                                       float w11) {
  return fadd(fadd(fadd(fmul(t00, w00), fmul(t10, w10)), fmul(t01, w01)), fmul(t11, w11));
}
__device__ float4 sample_linear(const float4* t, int w, int h, float u, float v) {
  const float x = fsub(fmul(u, (float)w), 0.5f), y = fsub(fmul(v, (float)h), 0.5f);
  const float fx = floorf(x), fy = floorf(y);
  const float a = fsub(x, fx), b = fsub(y, fy);
  const int i = (int)fx, j = (int)fy;
  float4 t00, t10, t01, t11;
  if ((unsigned)i < (unsigned)(w - 1) && (unsigned)j < (unsigned)(h - 1)) {  // all four taps inside: no wrap
    const float4* p = t + (size_t)j * w + i;
    t00 = __ldg(p), t10 = __ldg(p + 1), t01 = __ldg(p + w), t11 = __ldg(p + w + 1);
  } else {
    t00 = tap(t, w, h, i, j), t10 = tap(t, w, h, i + 1, j), t01 = tap(t, w, h, i, j + 1),
    t11 = tap(t, w, h, i + 1, j + 1);
  }
  const float w00 = fmul(fsub(1.0f, a), fsub(1.0f, b)), w10 = fmul(a, fsub(1.0f, b)), w01 = fmul(fsub(1.0f, a), b),
              w11 = fmul(a, b);
  return make_float4(lerp4(t00.x, t10.x, t01.x, t11.x, w00, w10, w01, w11),
                     lerp4(t00.y, t10.y, t01.y, t11.y, w00, w10, w01, w11),
                     lerp4(t00.z, t10.z, t01.z, t11.z, w00, w10, w01, w11),
                     lerp4(t00.w, t10.w, t01.w, t11.w, w00, w10, w01, w11));
}
// sampleBlurred(tex, uv, radius, gamma).a with lod = log2(radius), from its three textureLod
// samples at lod - 1, lod, lod + 1: weights exp(-gamma * (lod - i)^2) = w_side, 1, w_side.
__device__ __forceinline__ float blurred_alpha(float lo, float mid, float hi, float w_side) {
  float acc = fadd(0.0f, fmul(lo, w_side));
  acc = fadd(acc, fmul(mid, 1.0f));
  acc = fadd(acc, fmul(hi, w_side));
  return __fdiv_rn(acc, fadd(fadd(fadd(0.0f, w_side), 1.0f), w_side));
}

// The part of a fragment that depends only on the pixelated coordinate (pu, pv): the
// clamped light and the occlusion.
struct Shared {
  float lr, lg, lb, occ;
};
__device__ __forceinline__ Taps axis_taps(float u, int n) {
  const float x = fsub(fmul(u, (float)n), 0.5f), f = floorf(x);
  const int i = (int)f;
  const float a = fsub(x, f);
  return Taps{mirror_index(i, n), mirror_index(i + 1, n), a, fsub(1.0f, a)};
}
struct Weights {
  float w00, w10, w01, w11;
};
__device__ __forceinline__ Weights tap_weights(const Taps& c, const Taps& r) {
  return Weights{fmul(c.ia, r.ia), fmul(c.a, r.ia), fmul(c.ia, r.a), fmul(c.a, r.a)};
}
__device__ __forceinline__ Taps load_taps(const Taps* p) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(p));
  return Taps{__float_as_int(v.x), __float_as_int(v.y), v.z, v.w};
}
// Column pair k and row r0.  IDX: the integer type that holds any texel's index.
template <class IDX, bool SAME>
__device__ __forceinline__ Shared shared_terms(const CompositeSrc& m, const CompositeCoords& cc,
                                               const float4* __restrict__ light, int k, int r0, float ws0, float ws1,
                                               float ws2) {
  Shared S{0.0f, 0.0f, 0.0f, 0.0f};
  if (light) {
    const Taps c = load_taps(cc.col + k), r = load_taps(cc.row + r0);
    const Weights k = tap_weights(c, r);
    const IDX p = (IDX)r.i0 * (IDX)m.w, q = (IDX)r.i1 * (IDX)m.w;
    const float4 t00 = __ldg(light + (p + (IDX)c.i0)), t10 = __ldg(light + (p + (IDX)c.i1)),
                 t01 = __ldg(light + (q + (IDX)c.i0)), t11 = __ldg(light + (q + (IDX)c.i1));
    S.lr = gclamp(lerp4(t00.x, t10.x, t01.x, t11.x, k.w00, k.w10, k.w01, k.w11), 0.0f, 1.0f);
    S.lg = gclamp(lerp4(t00.y, t10.y, t01.y, t11.y, k.w00, k.w10, k.w01, k.w11), 0.0f, 1.0f);
    S.lb = gclamp(lerp4(t00.z, t10.z, t01.z, t11.z, k.w00, k.w10, k.w01, k.w11), 0.0f, 1.0f);
  }
  // The three sampleBlurred calls (lod 1, 4, 5) take textureLod at lods 0..2, 3..5 and 4..6:
  // seven distinct samples.  lod 0 is a magnification (level 0, nearest); lod l >= 1 reads
  // the alpha level in slot l, bilinearly.
  float s[kOccLods];
  s[0] = cell_alpha(__ldg(m.grid + ((IDX)__ldg(cc.nrow + r0) * (IDX)m.w + (IDX)__ldg(cc.ncol + k))), m.mats, m.nmat);
#pragma unroll
  for (int l = 1; l < kOccLods; ++l) {
    const Taps c = load_taps(cc.col + (size_t)l * cc.lw + k), r = load_taps(cc.row + (size_t)l * cc.lh + r0);
    const Weights k = tap_weights(c, r);
    const IDX p = (IDX)r.i0 * (IDX)m.aw[l], q = (IDX)r.i1 * (IDX)m.aw[l];
    const float* A = m.alpha[l];
    s[l] = lerp4(load<SAME>(A + (p + (IDX)c.i0)), load<SAME>(A + (p + (IDX)c.i1)), load<SAME>(A + (q + (IDX)c.i0)),
                 load<SAME>(A + (q + (IDX)c.i1)), k.w00, k.w10, k.w01, k.w11);
  }
  const float occ = fsub(1.0f, blurred_alpha(s[0], s[1], s[2], ws0));
  const float occ2 = fsub(1.0f, blurred_alpha(s[3], s[4], s[5], ws1));
  const float occ3 = fsub(1.0f, blurred_alpha(s[4], s[5], s[6], ws2));
  S.occ = gclamp(fadd(occ, fadd(fmul(occ2, 0.4f), fmul(occ3, 0.25f))), 0.0f, 1.0f);
  return S;
}

__device__ __forceinline__ int coords_len(int n) { return (n + 4) & ~3; }  // round_up(n + 1, 4)

// The column and row tables: one thread per column / row.  d = 1 / pixelate with
// pixelate = W / 2, as the fragment computes them.
__global__ void __launch_bounds__(256) se_composite_coords_kernel(CompositeTable t, CompositeSrc m, int W, int H,
                                                                  float d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < coords_len(W)) {
    const float ut = __fdiv_rn(fadd((float)i, 0.5f), (float)W);
    t.u[i] = i < W ? ut : 0.0f;
    t.ix[i] = i < W ? mirror_index((int)floorf(fmul(ut, (float)W)), W) : 0;
    // column pair i: its even column 2i (column 2i + 1 pixelates to the same u)
    if (i < t.lw) {
      const float ue = __fdiv_rn(fadd((float)(2 * i), 0.5f), (float)W);
      const float p = 2 * i < W ? fmul(floorf(__fdiv_rn(ue, d)), d) : 0.0f;
      t.ncol[i] = mirror_index((int)floorf(fmul(p, (float)W)), W);
      for (int l = 0; l < kOccLods; ++l) t.col[(size_t)l * t.lw + i] = axis_taps(p, l == 0 ? W : m.aw[l]);
    }
  }
  if (i < coords_len(H)) {
    const float vt = __fdiv_rn(fadd((float)i, 0.5f), (float)H);
    t.v[i] = i < H ? vt : 0.0f;
    t.iy[i] = i < H ? mirror_index((int)floorf(fmul(vt, (float)H)), H) : 0;
    const float p = i < H ? fmul(floorf(__fdiv_rn(vt, d)), d) : 0.0f;
    t.pv[i] = p;
    t.nrow[i] = mirror_index((int)floorf(fmul(p, (float)H)), H);
    for (int l = 0; l < kOccLods; ++l) t.row[(size_t)l * t.lh + i] = axis_taps(p, l == 0 ? H : m.ah[l]);
  }
}

// Thread = 2 x 2 pixels: columns 2k, 2k + 1 share pu; rows share pv when W <= H, else the shared
// terms are computed per row (the choice is uniform in a warp).  The taps of every column pair and
// row along every sampled texture, their indices wrapped, come from tables made once per world: a
// sample is then two 16-byte loads, four taps and its weights, without the index arithmetic and
// the wrap branch of its own.  Bound by the latency of its ~32 taps at 32 warps an SM (with
// the tables 14.1 M warp instructions at 1920 x 1080 instead of 17.8 M, 36.6 -> 27.1 us).  Colours are made
// from ids and noise as they are needed, 40 B a pixel: reading a stored colour field took 32.7 us where
// this takes 30.6 (4096 x 4096 162 / 156, 8192 x 8192 604 / 588) and the field's own pass 8-144 us more.  Tables rebuilt per CTA in shared memory cost what they
// saved (35 and 189 us), as did one lane per pixel with the shared terms passed by shuffles.
template <class IDX, bool SAME>
__device__ __forceinline__ void composite_block(const CompositeSrc& m, const CompositeCoords& cc,
                                                const float4* __restrict__ light, const float4* __restrict__ bg, int bw,
                                                int bh, float ws0, float ws1, float ws2, float4* __restrict__ out,
                                                int bx, int by, int t) {
  const int W = m.w, H = m.h;
  const int k = bx * 32 + (t & 31), c0 = 2 * k, r0 = 2 * (by * 8 + (t >> 5));
  if (c0 >= W || r0 >= H) return;
  // c0 and r0 are even: 8-byte aligned pair loads, in bounds up to index W / H
  const float2 us = __ldg(reinterpret_cast<const float2*>(cc.u + c0));
  const int2 ixs = __ldg(reinterpret_cast<const int2*>(cc.ix + c0));
  const float2 vs = __ldg(reinterpret_cast<const float2*>(cc.v + r0));
  const int2 iys = __ldg(reinterpret_cast<const int2*>(cc.iy + r0));
  const float2 pvs = __ldg(reinterpret_cast<const float2*>(cc.pv + r0));
  // texture(color_tex, uv, 0.0): a magnification, the nearest texel
  const bool two = c0 + 1 < W, down = r0 + 1 < H;
  uint32_t ids[2][2];
  float nz[2][2];
#pragma unroll
  for (int dr = 0; dr < 2; ++dr) {
    const IDX p = (IDX)(dr && down ? iys.y : iys.x) * (IDX)W;
    const IDX i0 = p + (IDX)ixs.x, i1 = p + (IDX)(two ? ixs.y : ixs.x);
    ids[dr][0] = __ldg(m.grid + i0), nz[dr][0] = __ldg(m.noise + i0);
    ids[dr][1] = __ldg(m.grid + i1), nz[dr][1] = __ldg(m.noise + i1);
  }
  const float ambient = 0.1f;
  Shared S = shared_terms<IDX, SAME>(m, cc, light, k, r0, ws0, ws1, ws2);
#pragma unroll
  for (int dr = 0; dr < 2; ++dr) {
    if (dr == 1) {
      if (!down) break;
      if (pvs.y != pvs.x) S = shared_terms<IDX, SAME>(m, cc, light, k, r0 + 1, ws0, ws1, ws2);
    }
    const float v = dr ? vs.y : vs.x;
    const float sky = fmul(0.5f, fsub(1.0f, dr ? pvs.y : pvs.x));
    const float shade = fadd(ambient, fmul(S.occ, fsub(1.0f, ambient)));
    const float base = fadd(ambient, sky);
#pragma unroll
    for (int dc = 0; dc < 2; ++dc) {
      const int cx = c0 + dc;
      if (cx >= W) break;
      const float u = dc ? us.y : us.x;
      float4 col = cell_color(ids[dr][dc], nz[dr][dc], m.mats, m.nmat);
      col.x = gclamp(fmul(col.x, shade), 0.0f, 1.0f);
      col.y = gclamp(fmul(col.y, shade), 0.0f, 1.0f);
      col.z = gclamp(fmul(col.z, shade), 0.0f, 1.0f);
      const float4 b = bg ? sample_linear(bg, bw, bh, u, fsub(1.0f, v)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      const float ia = fsub(1.0f, col.w);
      float4 o;  // mix(bg, col, col.a) * vec4(ambient + sky + light, 1.0)
      o.x = fmul(fadd(fmul(b.x, ia), fmul(col.x, col.w)), fadd(base, S.lr));
      o.y = fmul(fadd(fmul(b.y, ia), fmul(col.y, col.w)), fadd(base, S.lg));
      o.z = fmul(fadd(fmul(b.z, ia), fmul(col.z, col.w)), fadd(base, S.lb));
      o.w = fmul(fadd(fmul(b.w, ia), fmul(col.w, col.w)), 1.0f);
      out[(size_t)(r0 + dr) * W + cx] = o;
    }
  }
}

template <class IDX>
__global__ void __launch_bounds__(256, 4) se_composite_kernel(const CompositeSrc m, const CompositeCoords cc,
                                                              const float4* __restrict__ light,
                                                              const float4* __restrict__ bg, int bw, int bh, float ws0,
                                                              float ws1, float ws2, float4* __restrict__ out,
                                                              int by0) {
  composite_block<IDX, false>(m, cc, light, bg, bw, bh, ws0, ws1, ws2, out, blockIdx.x, by0 + blockIdx.y, threadIdx.x);
}

// What the CTAs of the cluster wrote before it is seen by all of them after it.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}

// Pyramid and composite of a small world in one launch: one cluster, whose barriers stand
// between the steps.  A CTA takes blockDim.x / 256 of the blocks of 64 x 16 cells.  The three
// launches that it replaces are bound by their launching and by each other's ends (us, three / one
// launch: frame, light and image of one of three worlds in turn, and of one waited for; 64 x 64 11.3 / 8.2,
// 30.8 / 24.4; 128 x 128 12.0 / 8.1, 31.7 / 25.6; 180 x 180 11.9 / 8.8, 31.3 / 29.4).  Up to 48 blocks, three to
// a CTA: with four, 256 x 256, the wait is the longer one (30.4 / 31.6).  Where the device (or the part of it
// that the stream may use) has no room for such a cluster, the three launches stay.
constexpr int kImageCtas = 16;  // beyond the portable 8: half as many blocks to a CTA
__global__ void __launch_bounds__(768) se_image_kernel(const MipLevels mip, const CompositeSrc m,
                                                       const CompositeCoords cc, const float4* __restrict__ light,
                                                       const float4* __restrict__ bg, int bw, int bh, float ws0,
                                                       float ws1, float ws2, float4* __restrict__ out) {
  __shared__ float s3[3][2][8];
  const int sub = threadIdx.x >> 8, t = threadIdx.x & 255, b = blockIdx.x * (blockDim.x >> 8) + sub;
  const int nbx = (m.w + 63) / 64, bx = b % nbx, by = b / nbx;
  mip_block(m.grid, mip, m.w, m.h, m.mats, m.nmat, bx, by, t, s3[sub]);
  cluster_barrier();
  if (mip.levels > 5) {
    if (blockIdx.x == 0) mip_tail<true>(mip, threadIdx.x);  // at most 48 texels of level 6
    cluster_barrier();
  }
  composite_block<uint32_t, true>(m, cc, light, bg, bw, bh, ws0, ws1, ws2, out, bx, by, t);
}

// Launches fn(by0, n) for the row blocks [by0, by0 + n) of a 2D grid, n <= 65535.
template <class F>
void for_row_blocks(int blocks, F&& fn) {
  for (int by0 = 0; by0 < blocks; by0 += 65535) fn(by0, (unsigned)std::min(65535, blocks - by0));
}

}  // namespace

cudaError_t render_mips(const uint32_t* grid, const MipLevels& mip, int W, int H, const RenderMat* mats, int nmat,
                        cudaStream_t s) {
  for_row_blocks((H + 15) / 16, [&](int by0, unsigned n) {
    se_mip_kernel<<<dim3((unsigned)((W + 63) / 64), n), 256, 0, s>>>(grid, mip, W, H, mats, nmat, by0);
  });
  if (mip.levels > 5) {
    const long long n = (long long)((mip.w[5] + 1) / 2) * ((mip.h[5] + 1) / 2);
    se_mip_tail_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(mip);
  }
  return cudaGetLastError();
}

size_t composite_coords_bytes(int W, int H) {
  const size_t LW = (size_t)((W + 4) & ~3), LH = (size_t)((H + 4) & ~3), PW = ((size_t)W / 2 + 4) & ~(size_t)3;
  return sizeof(Taps) * kOccLods * (PW + LH) + 4 * (2 * LW + PW + 4 * LH);
}

cudaError_t render_composite_coords(void* buf, const CompositeSrc& src, CompositeCoords* out, cudaStream_t s) {
  const int W = src.w, H = src.h;
  CompositeTable t{};
  t.lw = (W / 2 + 4) & ~3;
  t.lh = (H + 4) & ~3;
  const size_t LW = (size_t)((W + 4) & ~3), LH = (size_t)t.lh;
  t.col = static_cast<Taps*>(buf);
  t.row = t.col + (size_t)kOccLods * t.lw;
  t.u = reinterpret_cast<float*>(t.row + (size_t)kOccLods * t.lh);
  t.ix = reinterpret_cast<int*>(t.u + LW);
  t.ncol = t.ix + LW;
  t.v = reinterpret_cast<float*>(t.ncol + t.lw);
  t.iy = reinterpret_cast<int*>(t.v + LH);
  t.pv = reinterpret_cast<float*>(t.iy + LH);
  t.nrow = reinterpret_cast<int*>(t.pv + LH);
  const float pixelate = (float)W / 2.0f;  // fragment140.glsl: pixelate = resolution.x / 2
  const float d = 1.0f / pixelate;
  const int n = (int)std::max(LW, LH);
  se_composite_coords_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(t, src, W, H, d);
  *out = CompositeCoords{t.u, t.ix, t.ncol, t.v, t.iy, t.pv, t.nrow, t.col, t.row, t.lw, t.lh};
  return cudaGetLastError();
}

cudaError_t render_composite(const CompositeSrc& src, const CompositeCoords& coords, const float4* light,
                             const float4* bg, int bw, int bh, const float w_side[3], float4* out, cudaStream_t s) {
  for_row_blocks((src.h + 15) / 16, [&](int by0, unsigned n) {
    const dim3 g((unsigned)((src.w + 63) / 64), n);
    if ((unsigned long long)src.w * src.h < 1ull << 32)
      se_composite_kernel<uint32_t><<<g, 256, 0, s>>>(src, coords, light, bg, bw, bh, w_side[0], w_side[1], w_side[2],
                                                      out, by0);
    else
      se_composite_kernel<uint64_t><<<g, 256, 0, s>>>(src, coords, light, bg, bw, bh, w_side[0], w_side[1], w_side[2],
                                                      out, by0);
  });
  return cudaGetLastError();
}

namespace {
// The launch of se_image_kernel for a world of at most 3 * kImageCtas blocks; `at` holds its attribute.
cudaError_t image_launch(int W, int H, cudaStream_t s, cudaLaunchConfig_t* c, cudaLaunchAttribute* at) {
  const int blocks = ((W + 63) / 64) * ((H + 15) / 16), sub = (blocks + kImageCtas - 1) / kImageCtas;
  *c = cudaLaunchConfig_t{};
  c->gridDim = dim3((unsigned)((blocks + sub - 1) / sub));
  c->blockDim = dim3((unsigned)(256 * sub));
  c->stream = s;
  *at = cudaLaunchAttribute{};
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = c->gridDim.x;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  c->attrs = at;
  c->numAttrs = 1;
  if (c->gridDim.x <= 8) return cudaSuccess;
  // beyond the portable cluster size; a setting of the current device's kernel
  return cudaFuncSetAttribute(se_image_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
}
}  // namespace

bool image_in_one_launch(int W, int H, cudaStream_t s) {
  if ((long long)((W + 63) / 64) * ((H + 15) / 16) > 3 * kImageCtas) return false;
  cudaLaunchConfig_t c;
  cudaLaunchAttribute at;
  int clusters = 0;
  if (image_launch(W, H, s, &c, &at) == cudaSuccess &&
      cudaOccupancyMaxActiveClusters(&clusters, se_image_kernel, &c) == cudaSuccess)
    return clusters > 0;
  cudaGetLastError();  // the answer is no, not a failure
  return false;
}

cudaError_t render_image(const MipLevels& mip, const CompositeSrc& src, const CompositeCoords& coords,
                         const float4* light, const float4* bg, int bw, int bh, const float w_side[3], float4* out,
                         cudaStream_t s) {
  cudaLaunchConfig_t c;
  cudaLaunchAttribute at;
  cudaError_t e = image_launch(src.w, src.h, s, &c, &at);
  if (e != cudaSuccess) return e;
  return cudaLaunchKernelEx(&c, se_image_kernel, mip, src, coords, light, bg, bw, bh, w_side[0], w_side[1], w_side[2],
                            out);
}

cudaError_t render_noise(float* noise, int W, int H, cudaStream_t s) {
  for_row_blocks((H + kNoiseTile - 1) / kNoiseTile, [&](int by0, unsigned n) {
    se_noise_kernel<<<dim3((unsigned)((W + kNoiseTile - 1) / kNoiseTile), n), 256, 0, s>>>(noise, W, H, by0);
  });
  return cudaGetLastError();
}

cudaError_t render_color(const uint32_t* grid, const float* noise, float4* out, int W, int H, const RenderMat* mats,
                         int nmat, cudaStream_t s) {
  const long long n = (long long)W * H;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long blocks = std::min<long long>((n + 255) / 256, (long long)sms * 8);
  se_color_kernel<<<(unsigned)(blocks > 0 ? blocks : 1), 256, 0, s>>>(grid, noise, out, n, mats, nmat);
  return cudaGetLastError();
}

namespace {
template <int R>
void launch_light(const uint32_t* old_grid, const uint32_t* new_grid, const float4* light_in, float4* light_out, int W,
                  int H, const RenderMat* mats, int nmat, cudaStream_t s) {
  const int rows = (H + 4 * R - 1) / (4 * R);
  const dim3 g((unsigned)((W + LTW - 1) / LTW), (unsigned)std::min(rows, 65535));
  if (rows <= 65535)
    se_light_kernel<false, R><<<g, 256, 0, s>>>(old_grid, new_grid, light_in, light_out, W, H, mats, nmat, 0);
  else
    for_row_blocks(rows, [&](int by0, unsigned n) {
      se_light_kernel<true, R><<<dim3(g.x, n), 256, 0, s>>>(old_grid, new_grid, light_in, light_out, W, H, mats, nmat,
                                                            by0);
    });
}
}  // namespace

cudaError_t light_pass(const uint32_t* old_grid, const uint32_t* new_grid, const float4* light_in, float4* light_out,
                       int W, int H, const RenderMat* mats, int nmat, cudaStream_t s) {
  // Worlds of up to 2^20 cells take tiles of 4 rows: with 16 a thread's four cells, one after the
  // other, are the pass's latency and few SMs have a CTA (4 / 16 rows: 64 x 64 4.2 / 8.3 us,
  // 640 x 400 8.3 / 12.4, 1280 x 800 14.4 / 18.1, 1920 x 1080 27.3 / 23.5, 4096 x 4096 212 / 131).
  if ((long long)W * H <= 1 << 20)
    launch_light<1>(old_grid, new_grid, light_in, light_out, W, H, mats, nmat, s);
  else
    launch_light<4>(old_grid, new_grid, light_in, light_out, W, H, mats, nmat, s);
  return cudaGetLastError();
}

}  // namespace se::rt
