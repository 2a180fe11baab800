// The colour and light outputs of the reference's setCell (shaders/compute/operations.glsl
// :99-169), as ahead-of-time sm_103a kernels that read a per-material table.  Plain C++
// declarations, shared by the kernels (render.cu) and the runtime.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace se::rt {

// One material's render data.  Ids >= the table size read entry 1 (NULL), as
// getMaterialFromID returns MAT_NULL for unknown ids.
struct alignas(16) RenderMat {
  float color[4];
  float emission[4];
  uint32_t flags;  // kRender* bits
  uint32_t pad[3];
};
enum : uint32_t {
  kRenderEmits = 1,     // emission.rgb != vec3(0): the cell's light is its emission
  kRenderObstacle = 2,  // isLightObstacle: emission.rgb == vec3(0) and not of type EMPTY
  kRenderNoise = 4,     // mat != MAT_EMPTY: the colour is darkened by the noise
};

// noise(vec2(x, y), 3, 2.0, 0.25) (math.glsl:98-106) for every cell of a W x H world.
cudaError_t render_noise(float* noise, int W, int H, cudaStream_t s);
// output_color (RGBA32F) of a grid, from the cached noise field.
cudaError_t render_color(const uint32_t* grid, const float* noise, float4* out, int W, int H, const RenderMat* mats,
                         int nmat, cudaStream_t s);
// output_light of the frame that took old_grid to new_grid, from the previous light field.
cudaError_t light_pass(const uint32_t* old_grid, const uint32_t* new_grid, const float4* light_in, float4* light_out,
                       int W, int H, const RenderMat* mats, int nmat, cudaStream_t s);

// Headless composite (shaders/fragment140.glsl:70-100): the colour field's box-filter
// pyramid, then one RGBA32F pixel per texel.  The colour field itself is not stored: a texel is
// its cell's id and noise (8 bytes instead of 16 written and 16 read).  GL filtering is fixed to the spec's formulas
// in binary32 (mirrored-repeat wrap, nearest / bilinear taps, LINEAR_MIPMAP_NEAREST level
// choice); the three blur weights exp(-gamma) for gamma 0.5, 0.35, 0.2 are passed in.
// The fragment reads levels above 0 only through their alpha (the occlusion's
// textureLod(...).a), so those levels are kept as alpha alone: the same box-filter sums of
// the alpha channel, a quarter of the bytes.
// The occlusion's textureLod calls use the integer lods 0 .. 6.
constexpr int kOccLods = 7;
// What the composite samples: the colour field (level 0), by ids and noise, and, for lod l = 1 .. 6, the alpha
// level textureLod reads at lod l.  With LINEAR_MIPMAP_NEAREST that is level
// ceil(l + 0.5) - 1 = l, or the last level of a shorter pyramid; a 1 x 1 field has no level
// 1, and its slots hold a copy of its own alpha.
struct CompositeSrc {
  const uint32_t* grid;
  const float* noise;
  const RenderMat* mats;
  int nmat;
  int w, h;
  const float* alpha[kOccLods];  // [0] is unused
  int aw[kOccLods], ah[kOccLods];
};
// exp(-gamma) for the three sampleBlurred calls (gamma 0.5, 0.35, 0.2), rounded to binary32.
constexpr float kBlurSideWeight[3] = {0.606530666f, 0.704688072f, 0.818730772f};
// Size of the next level: halved, at least 1.
inline int mip_next(int n) { return n > 1 ? n / 2 : 1; }
// The pyramid levels the composite reads (alpha only): levels 1 .. levels - 1, at most 6.
struct MipLevels {
  float* level[kOccLods];  // [0] is unused
  int w[kOccLods], h[kOccLods];
  int levels;
};
// The pyramid's alpha levels of a grid; levels == 1 (a single cell): its alpha in level[1].
cudaError_t render_mips(const uint32_t* grid, const MipLevels& mip, int W, int H, const RenderMat* mats, int nmat,
                        cudaStream_t s);
// A coordinate's two bilinear taps along one axis of a texture: the wrapped indices, and the
// weights of the second and of the first.
struct alignas(16) Taps {
  int i0, i1;
  float a, ia;
};
// Column and row tables of the composite, functions of the field's size only (built once):
// u = (c + 0.5) / W and the column of its nearest texel; per column pair the nearest column and
// the taps of its pixelated u (floor(u / d) * d at its even column, d = 1 / (W / 2)); per row v,
// its nearest row, the pixelated v and that one's nearest row and taps.  Taps [l * lw + pair] /
// [l * lh + row]: l = 0 along the light field, l >= 1 along the alpha level in slot l.  Column and
// row arrays hold round_up(n + 1, 4) entries, so that the pair loads of an odd last column or
// row stay in bounds.
struct CompositeCoords {
  const float* u;
  const int *ix, *ncol;
  const float* v;
  const int* iy;
  const float* pv;
  const int* nrow;
  const Taps *col, *row;
  int lw, lh;
};
struct CompositeTable {  // the same, to be filled
  float* u;
  int *ix, *ncol;
  float* v;
  int* iy;
  float* pv;
  int* nrow;
  Taps *col, *row;
  int lw, lh;
};
size_t composite_coords_bytes(int W, int H);
// Fills `buf` (composite_coords_bytes(W, H), 16-byte aligned) for src's sizes and points `out`
// into it.
cudaError_t render_composite_coords(void* buf, const CompositeSrc& src, CompositeCoords* out, cudaStream_t s);
cudaError_t render_composite(const CompositeSrc& src, const CompositeCoords& coords, const float4* light,
                             const float4* bg, int bw, int bh, const float w_side[3], float4* out, cudaStream_t s);
// Small worlds: render_mips and render_composite in one launch, where its cluster can run on the
// device and stream.
bool image_in_one_launch(int W, int H, cudaStream_t s);
cudaError_t render_image(const MipLevels& mip, const CompositeSrc& src, const CompositeCoords& coords,
                         const float4* light, const float4* bg, int bw, int bh, const float w_side[3], float4* out,
                         cudaStream_t s);

}  // namespace se::rt
