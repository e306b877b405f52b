// pbf_render.cu — screen-space fluid buffers as CUDA kernels: the particle
// sprites of ParicleRasterizer (src/renderer/filteredParticleFluid/
// paricleRasterizer.ts:170-204, shader/depthPassShader.ts,
// shader/volumePassShader.ts) and the narrow-range filter of TextureFilter
// (textureFilter.ts:129-160, shader/filterPassShader.ts).
//
// Rasterisation is restated for camera-facing sprites.  The view matrix is
// affine and the projection has no x/y shear, so a sprite (the particle's
// camera-space centre plus (+-hs, +-hs, 0, 0)) projects to an axis-aligned
// rectangle whose corners share clip z and w.  It is clipped away whole
// unless 0 <= z_clip <= w_clip with w_clip > 0.  A pixel is covered when its
// centre lies in the rectangle (left/top edges in, right/bottom out), and
// the sprite's uv there is the centre's position across the rectangle
// (perspective-correct interpolation reduces to linear at constant w).
//
// Depth pass: the fragment at uv has n.xy = 2 uv - 1, is discarded when
// |n.xy|^2 > 1, and otherwise lies on the sphere of radius R in front of the
// centre: z = c.z + sqrt(1 - |n.xy|^2) R.  Its depth (clip z / clip w,
// clamped to [0, 1]) must beat the depth buffer ('greater', reverse-Z) and
// all other fragments of the pixel; equal depths keep the first particle
// drawn, i.e. the lowest index.  One 64-bit atomicMax per fragment on
// (depth bits, ~index) decides it, so the result does not depend on thread
// order.  The winner's eye depth -z / w goes to the depth map (0 elsewhere)
// and its depth to the depth buffer.
//
// Fragment n.xy: uv is the pixel centre's position across the rectangle,
// n = 2 uv - 1, evaluated as one fused multiply-add per axis from per-sprite
// constants (sx = 2 / (x1 - x0), ox = (0.5 - x0) sx - 1; likewise in y from
// the bottom edge).  A sprite's fragments are skipped where a bound of its
// depths cannot beat the pixel's key, which changes nothing in the result.
//
// Volume pass: sprites of half-side R on the half-resolution target add
// exp(-2 |n.xy|^2), evaluated as the product exp(-2 nx^2) exp(-2 ny^2) of
// per-column and per-row factors.  The sum is kept in 64-bit fixed point
// with 40 fraction bits, where every float term in [2^-3, 2) is exact, so
// the sum is exact and order-free; it is rounded to float once.  The
// exponential is this file's own (splat_exp), so the CPU restatement can
// produce the same bits.
//
// Many particles on a large map are drawn in two phases: a share of the depth
// sprites, then everything else behind a depth test per 8 x 8 tile, with the
// small volume sprites sorted by tile and summed in shared memory.  Fewer are
// drawn at once, 1 to 32 of them a warp.  Neither changes a bit of the result.
//
// The filter is the reference's narrow-range filter, separable, x then y,
// with its sample window of 32 + 32 texels per 32-texel block: the centre it
// reads for texel p is p - (16 - filterSize/2), so filter sizes below 32
// shift the image as the reference's shader does.  Reads outside the image
// clamp to the edge (the robust-access behaviour of WGSL textureLoad under
// coordinate clamping).  The x pass writes a cleared temporary where its
// centre is positive; the y pass writes the depth map where the
// temporary's centre is positive and leaves the other texels as they were.
//
// This unit is compiled with -fmad=false: every float operation rounds as
// written, fused multiply-adds only where written (__fmaf_rn), which the CPU
// restatement reproduces with fmaf.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

#include "../../include/pbf_gb300.h"
#include "pbf_device.cuh"
#include "pbf_kernels.h"

namespace {

constexpr int kMaxHalf = 16;          // MaxFilterSize 32 >> 1
constexpr int kFilterX = 128;         // texels per block of the x pass
constexpr int kFilterYRows = 64;      // rows per block of the y pass, at most
constexpr double kFix = 1099511627776.0;  // 2^40

struct Gauss {
  float w[kMaxHalf + 1];  // the filter's weights by distance
};

struct Cam {
  float v[16];  // view, column-major
  float p[16];  // projection, column-major
};

// A sprite on one target: its covered pixels and the affine maps from pixel
// index to the fragment's n.xy = 2 uv - 1 (uv measured from the rectangle's
// left and bottom edges at the pixel centre): nx = i sx + ox, ny = j sy + oy.
struct Sprite {
  int i0, i1, j0, j1;  // covered pixels [i0, i1) x [j0, j1)
  float sx, ox, sy, oy;
  float cz, cw;        // camera-space z and w of the centre
  uint32_t dmax;       // bits of an upper bound of the fragment depths (depth sprites)
};

__device__ inline void mat_vec(const float* m, float x, float y, float z, float w, float o[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) o[r] = ((m[r] * x + m[4 + r] * y) + m[8 + r] * z) + m[12 + r] * w;
}

__device__ inline int pixel_edge(float f, int size) {
  // first pixel whose centre i + 0.5 is >= f, clamped to [0, size]
  const float e = fminf(fmaxf(f - 0.5f, -1.0f), (float)size);
  return min(max((int)ceilf(e), 0), size);
}

// The sprite of half-side hs around the camera-space centre c on a W x H
// target; false when it is clipped away or covers no pixel centre.
__device__ inline bool make_sprite(const Cam& C, const float c[4], float hs, int W, int H, Sprite& s) {
  float bl[4], tr[4];
  mat_vec(C.p, c[0] + (-hs), c[1] + (-hs), c[2], c[3], bl);
  mat_vec(C.p, c[0] + hs, c[1] + hs, c[2], c[3], tr);
  if (!(bl[3] > 0.0f) || !(bl[2] >= 0.0f) || !(bl[2] <= bl[3])) return false;
  const float fw = (float)W, fh = (float)H;
  const float fx0 = 0.5f * (bl[0] / bl[3] + 1.0f) * fw;
  const float fx1 = 0.5f * (tr[0] / tr[3] + 1.0f) * fw;
  const float fyb = 0.5f * (-(bl[1] / bl[3]) + 1.0f) * fh;
  const float fyt = 0.5f * (-(tr[1] / tr[3]) + 1.0f) * fh;
  if (!(fx1 != fx0) || !(fyb != fyt)) return false;
  s.i0 = pixel_edge(fminf(fx0, fx1), W);
  s.i1 = pixel_edge(fmaxf(fx0, fx1), W);
  s.j0 = pixel_edge(fminf(fyt, fyb), H);
  s.j1 = pixel_edge(fmaxf(fyt, fyb), H);
  const float ax = 2.0f / (fx1 - fx0), ay = 2.0f / (fyb - fyt);
  s.sx = ax;
  s.ox = __fmaf_rn(0.5f - fx0, ax, -1.0f);
  s.sy = -ay;
  s.oy = __fmaf_rn(fyb - 0.5f, ay, -1.0f);
  s.cz = c[2];
  s.cw = c[3];
  return s.i0 < s.i1 && s.j0 < s.j1;
}

// |n.xy|^2 of the sprite's fragment at pixel (i, j).
__device__ inline float sprite_r2(const Sprite& s, int i, int j) {
  const float nx = __fmaf_rn((float)i, s.sx, s.ox), ny = __fmaf_rn((float)j, s.sy, s.oy);
  return __fmaf_rn(nx, nx, ny * ny);
}

// [0, 1] depth of camera-space z (w = the centre's w).
__device__ inline float depth_of(const Cam& C, float z, float w) {
  const float d = __fmaf_rn(C.p[10], z, C.p[14] * w) / __fmaf_rn(C.p[11], z, C.p[15] * w);
  return d > 0.0f ? fminf(d, 1.0f) : 0.0f;
}

// Depth-pass fragment: camera z of the sphere point and its [0, 1] depth.
__device__ inline float sprite_depth(const Cam& C, const Sprite& s, float r2, float R, float& z) {
  z = __fmaf_rn(sqrtf(1.0f - r2), R, s.cz);
  return depth_of(C, z, s.cw);
}

// An upper bound of the depths of a depth sprite's fragments.  Their z lie
// in [c.z, zt = c.z + R] (sqrt(1 - r2) is in [0, 1] and the rounded fma is
// monotone in it).  With a positive denominator on that interval, a
// numerator that does not fall and a denominator that does not rise as z
// grows (p10 >= 0 >= p11: the reverse-Z perspective) make every rounded
// non-negative depth at most the depth at zt, and negative depths clamp to
// 0; the mirror case bounds them by the depth at c.z.  Otherwise there is no
// bound (all ones).
__device__ inline uint32_t depth_bound(const Cam& C, float cz, float cw, float R) {
  const float zt = __fmaf_rn(1.0f, R, cz);
  const float d0 = __fmaf_rn(C.p[11], cz, C.p[15] * cw), d1 = __fmaf_rn(C.p[11], zt, C.p[15] * cw);
  if (!(d0 > 0.0f && d1 > 0.0f)) return 0xffffffffu;
  if (C.p[10] >= 0.0f && C.p[11] <= 0.0f) return __float_as_uint(depth_of(C, zt, cw));
  if (C.p[10] <= 0.0f && C.p[11] >= 0.0f) return __float_as_uint(depth_of(C, cz, cw));
  return 0xffffffffu;
}

// v * 2^40 as an integer, exactly, for a float v in [2^-3, 2): its 24-bit
// significand shifted by (biased exponent - 110).
__device__ inline unsigned long long fix40(float v) {
  const uint32_t b = __float_as_uint(v);
  const uint32_t e = (b >> 23) & 0xffu;
  return (unsigned long long)((b & 0x7fffffu) | 0x800000u) << (e - 110u);
}

// exp(x) for x in [-2, 0]: Cody-Waite reduction x = k ln2 + r with ln 2 in
// two parts (the high part has 16 significant bits, so k * hi is exact for
// |k| <= 3), then exp(r) by its Taylor series to degree 8 in Horner form with
// fused multiply-adds (|r| <= 0.35: truncation below 3e-10), scaled by 2^k.
__device__ inline float splat_exp(float x) {
  const float k = floorf(__fmaf_rn(x, 1.44269502f, 0.5f));
  const float r = __fmaf_rn(-k, 1.42860677e-6f, __fmaf_rn(-k, 0.693145751953125f, x));
  float p = 2.48015873e-5f;              // 1/8!
  p = __fmaf_rn(p, r, 1.98412698e-4f);   // 1/7!
  p = __fmaf_rn(p, r, 1.38888889e-3f);   // 1/6!
  p = __fmaf_rn(p, r, 8.33333333e-3f);   // 1/5!
  p = __fmaf_rn(p, r, 4.16666667e-2f);   // 1/4!
  p = __fmaf_rn(p, r, 1.66666667e-1f);   // 1/3!
  p = __fmaf_rn(p, r, 0.5f);
  p = __fmaf_rn(p, r, 1.0f);
  p = __fmaf_rn(p, r, 1.0f);
  return p * __uint_as_float((uint32_t)((int)k + 127) << 23);   // 2^k (k in [-3, 0])
}

__device__ inline uint32_t depth_bits(float d) { return __float_as_uint(d); }

// Also clears the words of `zero` (the volume tiles' counts).
__global__ void k_init(const float* scene, unsigned long long* keys, unsigned long long* acc, int W, int H, int W2,
                       int H2, uint32_t* zero, uint32_t words) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  for (uint32_t q = y * gridDim.x * blockDim.x + x; q < words; q += gridDim.x * gridDim.y * blockDim.x) zero[q] = 0u;
  if (x >= W) return;
  const size_t p = (size_t)y * W + x;
  float s = scene ? scene[p] : 0.0f;
  s = s > 0.0f ? fminf(s, 1.0f) : 0.0f;
  keys[p] = ((unsigned long long)depth_bits(s) << 32) | 0xffffffffull;
  if (x < W2 && y < H2) acc[(size_t)y * W2 + x] = 0ull;
}

// Sprites are set up one per lane (32 particles per warp) in shared memory;
// the warp then walks them one by one with its lanes spread over each
// sprite's pixels: for sprites up to 32 pixels wide, floor(32 / width) rows
// per step (lane -> row lane / width by a 16-bit reciprocal, exact for lane
// and width up to 32), else 32 columns per step.  Every lane takes part in
// every step (frag receives whether its pixel is inside the sprite), so the
// fragment code may use warp-wide votes and shuffles.
struct SpriteSlot {
  Sprite s[2];   // depth, volume
  uint32_t ok;   // bit 0: depth sprite visible, bit 1: volume sprite visible
};

// ceil(2^16 / w) for w = 1 .. 32
__constant__ uint32_t c_recip16[33] = {0,    65536, 32768, 21846, 16384, 13108, 10923, 9363, 8192, 7282, 6554,
                                       5958, 5462,  5042,  4682,  4370,  4096,  3856,  3641, 3450, 3277, 3121,
                                       2979, 2850,  2731,  2622,  2521,  2428,  2341,  2260, 2185, 2115, 2048};

template <typename Frag>
__device__ inline void walk_sprite(const Sprite& s, uint32_t lane, Frag frag) {
  const int w = s.i1 - s.i0;
  if (w <= 32) {
    const uint32_t m = c_recip16[w];
    const int rows = (int)((32u * m) >> 16);
    const int lr = (int)((lane * m) >> 16), lc = (int)lane - lr * w;
    for (int jb = s.j0; jb < s.j1; jb += rows) {
      const int j = jb + lr;
      frag(s.i0 + lc, j, lr < rows && j < s.j1);
    }
  } else {
    for (int j = s.j0; j < s.j1; ++j)
      for (int ib = s.i0; ib < s.i1; ib += 32) frag(ib + (int)lane, j, ib + (int)lane < s.i1);
  }
}

// exp(-2 n^2) of a fragment coordinate n: the volume term exp(-2 |n|^2) is
// the product of the x and y factors.
__device__ inline float gauss_axis(float n) { return splat_exp((n * n) * -2.0f); }

// Depth test ahead of the fragments: the smallest depth that any pixel of an
// 8 x 8 tile holds.  Most sprites of a deep cloud lie behind the surface: at
// 2^20 particles every covered pixel has hundreds of fragments, and reading its
// key for each was half of the pass.  A share of the particles (one block of
// 32 in kFirstShare, spread over the index range) is drawn first; the tiles'
// smallest depths then reject a sprite whose bound is below them in all the
// tiles it touches, which changes nothing in the result.
constexpr int kTile = 8;
constexpr uint32_t kFirstShare = 16;
// The two phases and the volume sums by tile pay for their five extra launches
// (about 25 us) and for the particles' second reading where there are many
// fragments and many of them to a pixel: the square root of their product,
// particles times side^2 over the square root of the map's pixels, tells best
// where.  Sprites of 25 pixels and more are too large to be summed by tile.  A
// frame, all at once and tiled (us, both with the best number of particles a
// warp):
//   n          side  map          fill   all  tiled
//     500,000   1.6  1920 x 1080    931   184   215
//   1,048,576   1.6  1920 x 1080  1,953   299   332
//     700,000   1.4   320 x 180   5,433   193   189
//     900,000   2.7  1280 x 720   6,985   263   293
//     524,288   2.7   640 x 360   8,138   168   193
//     700,000   4.1  1920 x 1080  8,149   277   275
//     400,000   8.2  3840 x 2160  9,313   461   458
//     700,000   2.6   640 x 339   9,930   208   195
//     900,000   4.1  1920 x 1080 10,477   342   366
//     500,000   4.1   960 x 540  11,641   222   203
//   1,048,576   4.1  1920 x 1080 12,207   371   340
//     400,000   5.5  1280 x 720  12,417   207   204
//     500,000   8.2  1920 x 1080 23,282   481   387
//   1,048,576   8.2  1920 x 1080 48,826   792   530
//     620,000  16.4  3840 x 2160 57,740 1,567 1,363
//     620,000  32.8  1920 x 1080          7,135 7,363
// (Powers of two are worst for the first share in these clouds: the particles
// lie in index order on a lattice, and every 16th block falls on the same lines.)
// Below kTiledMin the first share is too small: 2^18 particles at 1920 x 1080
// with sides of 8.2 took 321 at once and 429 tiled.
constexpr uint32_t kTiledMin = 3u << 17;
constexpr double kTiledFill = 9.5e3, kTiledSide = 25.0;
inline bool takes_tiles(uint32_t n, double side, int W, int H) {
  return n >= kTiledMin && side < kTiledSide && n * side * side >= kTiledFill * std::sqrt((double)W * H);
}
constexpr int kMaxTiles = 16;                // larger sprites are not tested

__global__ void __launch_bounds__(256) k_tile_min(const unsigned long long* __restrict__ keys, int W, int H, int tw,
                                                  uint32_t* __restrict__ tile_min) {
  pbf::chain_begin(keys);
  // one warp per tile, two pixels a lane
  const uint32_t lane = threadIdx.x & 31u, tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int tx = (int)tile % tw, ty = (int)tile / tw;
  if (ty * kTile >= H) return;
  uint32_t m = 0xffffffffu;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = tx * kTile + (int)(lane & 7u), j = ty * kTile + (int)(lane >> 3) + 4 * h;
    if (i < W && j < H) m = min(m, (uint32_t)(keys[(size_t)j * W + i] >> 32));
  }
  m = __reduce_min_sync(0xffffffffu, m);
  if (lane == 0) tile_min[tile] = m;
}

// Whether a depth sprite may win a pixel in any of its tiles.
__device__ inline bool may_win(const Sprite& s, const uint32_t* __restrict__ tile_min, int tw) {
  const int x0 = s.i0 / kTile, x1 = (s.i1 - 1) / kTile, y0 = s.j0 / kTile, y1 = (s.j1 - 1) / kTile;
  if ((x1 - x0 + 1) * (y1 - y0 + 1) > kMaxTiles) return true;
  if (x1 - x0 <= 1 && y1 - y0 <= 1) {  // most sprites: the four loads at once
    const uint32_t *r0 = tile_min + (size_t)y0 * tw, *r1 = tile_min + (size_t)y1 * tw;
    const uint32_t a = __ldg(r0 + x0), b = __ldg(r0 + x1), c = __ldg(r1 + x0), d = __ldg(r1 + x1);
    return s.dmax >= min(min(a, b), min(c, d));
  }
  for (int y = y0; y <= y1; ++y)
    for (int x = x0; x <= x1; ++x)
      if (s.dmax >= __ldg(tile_min + (size_t)y * tw + x)) return true;
  return false;
}

// What a launch of the splat draws: all particles at once, or the first share's
// depth sprites, or everything else.
enum SplatPhase { kAll = 0, kFirst = 1, kRest = 2 };

constexpr int kQueue = 64;  // per-warp queue of depth fragments that pass the bound test

// Depth fragments that may win are queued (pixel, sprite) per warp and
// evaluated 32 at a time with all lanes busy: the full fragment (square root,
// division, key, atomicMax) runs only for them.
__device__ inline void depth_fragments(const Cam& C, const SpriteSlot* slots, const uint32_t* qij, const uint8_t* qk,
                                       uint32_t count, uint32_t lane, uint32_t base, float R, int W,
                                       unsigned long long* keys) {
  if (lane >= count) return;
  const uint32_t e = qij[lane], k = qk[lane];
  const int i = (int)(e & 0xffffu), j = (int)(e >> 16);
  const Sprite& s = slots[k].s[0];
  const float r2 = sprite_r2(s, i, j);
  if (r2 > 1.0f) return;
  float z;
  const float d = sprite_depth(C, s, r2, R, z);
  const unsigned long long key = ((unsigned long long)__float_as_uint(d) << 32) | (0xffffffffull - (base + k));
  unsigned long long* kp = keys + (size_t)j * W + i;
  if (key > *(volatile unsigned long long*)kp) atomicMax(kp, key);
}

// ---- volume sprites by tile ---------------------------------------------------------
// The sums of a deep cloud are some 60 M additions to 100 K pixels at 2^20
// particles; as 64-bit atomics on the map they took as long as all the rest of
// the pass.  Sprites of at most 2 kVolHalo pixels across are sorted by the 24 x
// 24 tile of their centre, and a CTA adds up a run of them in shared memory
// before it adds its window (the tile and kVolHalo pixels around) to the map.
// Integer sums: the result is the same in any order.
constexpr int kVolTile = 24;                 // (four CTAs' windows fit an SM)
constexpr int kVolHalo = 8;
constexpr int kVolWin = kVolTile + 2 * kVolHalo;
constexpr uint32_t kVolWarps = 8;
constexpr uint32_t kVolPer = 60;             // sprites of one tile a warp takes at most
constexpr uint32_t kVolRun = kVolWarps * kVolPer;  // sprites a CTA takes
constexpr uint32_t kVolFew = 24;             // runs of fewer in one tile go to the map directly
constexpr uint32_t kNoTile = 0xffffffffu;

__device__ inline bool by_tile(const Sprite& s) { return s.i1 - s.i0 <= 2 * kVolHalo && s.j1 - s.j0 <= 2 * kVolHalo; }
__device__ inline uint32_t tile_of(const Sprite& s, int vw) {
  return (uint32_t)(((s.j0 + s.j1) >> 1) / kVolTile * vw + ((s.i0 + s.i1) >> 1) / kVolTile);
}

// Volume fragments of one sprite, its lanes' axis factors computed once:
// add(i, j, term) for each pixel of the disc.
template <typename Add>
__device__ inline void volume_fragments(const Sprite& s, uint32_t lane, Add add) {
  // per-lane axis factors: this lane's column (narrow sprites) and row j0 + lane
  const int w = s.i1 - s.i0, h = s.j1 - s.j0;
  float ex = 0.0f, ey = 0.0f;
  if (w <= 32) {
    const uint32_t m = c_recip16[w];
    const int lc = (int)lane - (int)((lane * m) >> 16) * w;
    ex = gauss_axis(__fmaf_rn((float)(s.i0 + lc), s.sx, s.ox));
  }
  if (h <= 32) ey = gauss_axis(__fmaf_rn((float)(s.j0 + (int)lane), s.sy, s.oy));
  walk_sprite(s, lane, [&](int i, int j, bool in) {
    float fy = __shfl_sync(0xffffffffu, ey, (j - s.j0) & 31);
    if (!in) return;
    const float r2 = sprite_r2(s, i, j);
    if (r2 > 1.0f) return;
    if (h > 32) fy = gauss_axis(__fmaf_rn((float)j, s.sy, s.oy));
    const float fx = w <= 32 ? ex : gauss_axis(__fmaf_rn((float)i, s.sx, s.ox));
    add(i, j, fx * fy);
  });
}

// The tiles' first places: the exclusive scan of their counts by one CTA, which
// waits on no other, so a place is always that of its count: a look-back scan
// that gave up would leave entries of the order unwritten, which k_volume_sum
// takes for tiles and particles.  One round up to 1,024 tiles (1920 x 1080 has
// 920, 3840 x 2160 3,600); a frame of 2^20 particles takes 523 us at 1920 x 1080
// and 2,179 at 3840 x 2160, 524 and 2,180 with the look-back scan.
constexpr uint32_t kPlaceThreads = 1024;

__global__ void __launch_bounds__(kPlaceThreads) k_volume_places(const uint32_t* __restrict__ count, uint32_t m,
                                                                 uint32_t* __restrict__ place) {
  __shared__ uint32_t s_warp[32];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  pbf::chain_begin(count);
  uint32_t before = 0u;
  for (uint32_t b = 0; b < m; b += kPlaceThreads) {
    const uint32_t t = b + threadIdx.x, v = t < m ? count[t] : 0u;
    uint32_t x = v;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31u) s_warp[wib] = x;
    __syncthreads();
    uint32_t w = s_warp[lane];
    const uint32_t total = __reduce_add_sync(0xffffffffu, w);
    const uint32_t mine = __reduce_add_sync(0xffffffffu, lane < wib ? w : 0u);
    if (t < m) place[t] = before + mine + x - v;
    before += total;
    __syncthreads();
  }
}

// Particles in tile order (any order within a tile): place[t] is the tile's
// first place, and the splat's count of a tile gave each of its sprites a rank
// (2^20 particles: 6 us; 33 with the places counted up here).
__global__ void __launch_bounds__(256) k_volume_order(uint32_t n, const uint2* __restrict__ tile,
                                                      const uint32_t* __restrict__ place, uint2* __restrict__ order) {
  pbf::chain_begin(tile, place, order);
  const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  const uint2 t = tile[q];  // (tile, rank)
  if (t.x != kNoTile) order[__ldg(place + t.x) + t.y] = make_uint2(t.x, q);
}

// A CTA's run of kVolRun sorted sprites, tile by tile, the tile's sprites shared
// out among its warps.  A term exp(-2 |n|^2) is a float in [2^-3, 1], so in
// units of 2^-26 an integer of at most 2^26, and 32-bit sums hold the kVolPer
// sprites a warp takes.  Each warp has a window of its own, so its sums are
// plain shared-memory reads and writes: one window per CTA took shared atomics
// (four to five passes of the data path each) and barriers every 56 sprites.
// A sprite is at most 16 pixels wide and high here: lanes 0 to 15 evaluate the
// column factors and 16 to 31 the row factors at once.
constexpr uint32_t kVolThreads = 32 * kVolWarps;
constexpr size_t kVolSmem = sizeof(uint32_t) * kVolWarps * kVolWin * kVolWin;
static_assert(kVolPer < 64, "32-bit sums");

__global__ void __launch_bounds__(kVolThreads) k_volume_sum(Cam C, const float4* __restrict__ pos, float R, int W2,
                                                            int H2, int vw, const uint2* __restrict__ order,
                                                            const uint32_t* __restrict__ total,
                                                            unsigned long long* acc) {
  extern __shared__ uint32_t s_win[];
  __shared__ uint32_t s_end;
  constexpr uint32_t kPix = kVolWin * kVolWin;
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
  uint32_t* win = s_win + wib * kPix;
  pbf::chain_begin(pos, order, total, acc);
  const uint32_t first = blockIdx.x * kVolRun, last = min(first + kVolRun, *total);
  if (first >= last) return;
  for (uint32_t p = lane; p < kPix; p += 32u) win[p] = 0u;
  __syncwarp();
  uint32_t b = first;
  while (b < last) {  // one tile's sprites [b, e)
    const uint32_t t = order[b].x;
    if (threadIdx.x == 0) s_end = last;
    __syncthreads();
    for (uint32_t k = b + threadIdx.x; k < last; k += kVolThreads)
      if (order[k].x != t) {
        atomicMin(&s_end, k);
        break;
      }
    __syncthreads();
    const uint32_t e = s_end;
    const bool direct = e - b < kVolFew;
    const int wx = (int)(t % (uint32_t)vw) * kVolTile - kVolHalo, wy = (int)(t / (uint32_t)vw) * kVolTile - kVolHalo;
    const uint32_t per = (e - b + kVolWarps - 1u) / kVolWarps, g0 = b + wib * per, g1 = min(g0 + per, e);
    for (uint32_t g = g0; g < g1; g += 32u) {
      const uint32_t cnt = min(32u, g1 - g);
      Sprite mine{};
      if (lane < cnt) {
        const float4 x = __ldg(pos + order[g + lane].y);
        float c[4];
        mat_vec(C.v, x.x, x.y, x.z, 1.0f, c);
        make_sprite(C, c, R, W2, H2, mine);
      }
      for (int k = 0; k < (int)cnt; ++k) {
        const int i0 = __shfl_sync(0xffffffffu, mine.i0, k), w = __shfl_sync(0xffffffffu, mine.i1, k) - i0;
        const int j0 = __shfl_sync(0xffffffffu, mine.j0, k), h = __shfl_sync(0xffffffffu, mine.j1, k) - j0;
        const float sx = __shfl_sync(0xffffffffu, mine.sx, k), ox = __shfl_sync(0xffffffffu, mine.ox, k);
        const float sy = __shfl_sync(0xffffffffu, mine.sy, k), oy = __shfl_sync(0xffffffffu, mine.oy, k);
        // a column or row past the sprite's gets a coordinate outside the disc
        const bool row = lane >= 16u;
        const int q = (int)(lane & 15u);
        const float f = (float)((row ? j0 : i0) + q);
        float nn = __fmaf_rn(f, row ? sy : sx, row ? oy : ox);
        if (q >= (row ? h : w)) nn = 2.0f;
        const float n2 = nn * nn, gs = splat_exp(n2 * -2.0f);
        // lane -> (row of the step, column)
        const uint32_t m = c_recip16[w], rows = (32u * m) >> 16, lr = (lane * m) >> 16;
        const int col = (int)lane - (int)lr * w;
        float nx = __shfl_sync(0xffffffffu, nn, col);
        if (lr >= rows) nx = 2.0f;
        const float ex = __shfl_sync(0xffffffffu, gs, col) * 67108864.0f;  // in units of 2^-26, exact
        if (direct) {
          for (int r0 = 0; r0 < h; r0 += (int)rows) {
            const int r = r0 + (int)lr, src = min(16 + r, 31);
            const float ny2 = __shfl_sync(0xffffffffu, n2, src), ey = __shfl_sync(0xffffffffu, gs, src);
            if (r < h && __fmaf_rn(nx, nx, ny2) <= 1.0f)
              atomicAdd(acc + (size_t)(j0 + r) * W2 + i0 + col, (unsigned long long)__float2uint_rn(ex * ey) << 14);
          }
          continue;
        }
        uint32_t* at = win + (j0 - wy + (int)lr) * kVolWin + (i0 - wx) + col;
        for (int r = (int)lr; r < h + (int)lr; r += (int)rows, at += rows * kVolWin) {
          const int src = min(16 + r, 31);
          const float ny2 = __shfl_sync(0xffffffffu, n2, src), ey = __shfl_sync(0xffffffffu, gs, src);
          // (a step's pixels are distinct, and the next sprite's come after them)
          if (r < h && __fmaf_rn(nx, nx, ny2) <= 1.0f) *at += __float2uint_rn(ex * ey);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    if (!direct) {
      for (uint32_t p = threadIdx.x; p < kPix; p += kVolThreads) {
        unsigned long long v = 0ull;
#pragma unroll
        for (uint32_t k = 0; k < kVolWarps; ++k) {
          v += s_win[k * kPix + p];
          s_win[k * kPix + p] = 0u;
        }
        if (v) atomicAdd(acc + (size_t)(wy + (int)(p / kVolWin)) * W2 + wx + (int)(p % kVolWin), v << 14);
      }
    }
    b = e;
    __syncthreads();
  }
}

// kSteps: the keys of four steps of a depth sprite are read together.
template <bool kSteps>
__global__ void __launch_bounds__(256) k_splat(Cam C, const float4* __restrict__ pos, uint32_t n, float R, int W, int H,
                                               int W2, int H2, unsigned long long* keys, unsigned long long* acc,
                                               int phase, uint32_t per, const uint32_t* __restrict__ tile_min, int tw,
                                               uint2* __restrict__ vol_tile, uint32_t* __restrict__ vol_count) {
  __shared__ SpriteSlot slots[8][32];
  __shared__ uint32_t qij[8][kQueue];
  __shared__ uint8_t qk[8][kQueue];
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  pbf::chain_begin(pos, keys, acc, tile_min, vol_tile, vol_count);
  // `per` particles (a power of two) of a block of 32 a warp
  const uint32_t parts = 32u / per;
  const uint64_t stride = phase == kFirst ? kFirstShare * 32u : 32u;
  const uint64_t items = ((uint64_t)n + stride - 1u) / stride * parts;
  for (uint64_t it = warp; it < items; it += warps) {
    const uint64_t b = it / parts * stride + it % parts * per;
    if (b >= n) continue;
    const uint32_t base = (uint32_t)b, q = base + lane;
    const bool first = (base / 32u) % kFirstShare == 0u;  // drawn in the first phase
    SpriteSlot& mine = slots[wib][lane];
    mine.ok = 0;
    const uint32_t cnt = min(per, n - base);
    uint32_t vt = kNoTile;
    if (lane < cnt) {
      const float4 x = pos[q];
      float c[4];
      mat_vec(C.v, x.x, x.y, x.z, 1.0f, c);
      if (!(phase == kRest && first) && make_sprite(C, c, 0.5f * R, W, H, mine.s[0])) {
        mine.s[0].dmax = depth_bound(C, c[2], c[3], R);
        if (phase != kRest || may_win(mine.s[0], tile_min, tw)) mine.ok |= 1u;
      }
      if (phase != kFirst && make_sprite(C, c, R, W2, H2, mine.s[1])) {
        // with phases, small volume sprites are summed by tile
        if (phase == kRest && by_tile(mine.s[1]))
          vt = tile_of(mine.s[1], (W2 + kVolTile - 1) / kVolTile);
        else
          mine.ok |= 2u;
      }
    }
    if (phase == kRest) {  // the tiles' counts, one addition per warp and tile; the old counts give ranks
      const unsigned peers = __match_any_sync(0xffffffffu, vt);
      const int leader = __ffs(peers) - 1;
      uint32_t rank = 0u;
      if (vt != kNoTile && (int)lane == leader) rank = atomicAdd(vol_count + vt, (uint32_t)__popc(peers));
      rank = __shfl_sync(0xffffffffu, rank, leader) + (uint32_t)__popc(peers & lt);
      if (lane < cnt) vol_tile[q] = make_uint2(vt, rank);
    }
    __syncwarp();
    uint32_t qn = 0;  // queued depth fragments (warp-uniform)
    for (uint32_t k = 0; k < cnt; ++k) {
      const SpriteSlot& sl = slots[wib][k];
      const uint32_t ok = sl.ok;
      if (ok & 1u) {
        const Sprite s = sl.s[0];
        const unsigned long long bound = ((unsigned long long)s.dmax << 32) | (0xffffffffull - (base + k));
        // only fragments whose sprite bound beats the pixel's current key can win
        auto consider = [&](int i, int j, bool pass) {
          const unsigned m = __ballot_sync(0xffffffffu, pass);
          if (pass) {
            const uint32_t at = qn + __popc(m & lt);
            qij[wib][at] = ((uint32_t)j << 16) | (uint32_t)i;
            qk[wib][at] = (uint8_t)k;
          }
          qn += __popc(m);
          if (qn >= 32) {
            __syncwarp();
            depth_fragments(C, slots[wib], qij[wib], qk[wib], 32, lane, base, R, W, keys);
            __syncwarp();
            qn -= 32;
            if (lane < qn) {
              qij[wib][lane] = qij[wib][32 + lane];
              qk[wib][lane] = qk[wib][32 + lane];
            }
            __syncwarp();
          }
        };
        const int w = s.i1 - s.i0;
        const int rows1 = w <= 32 ? (int)((32u * c_recip16[w]) >> 16) : 0;
        if (!kSteps || w > 32 || s.j1 - s.j0 <= rows1) {  // one step, or rows of many
          walk_sprite(s, lane, [&](int i, int j, bool in) {
            consider(i, j, in && bound > *(volatile unsigned long long*)(keys + (size_t)j * W + i));
          });
        } else {
          // four steps' keys are read together: one at a time, each step of a
          // sprite waited for its read
          const uint32_t m = c_recip16[w];
          const int rows = (int)((32u * m) >> 16), lr = (int)((lane * m) >> 16), i = s.i0 + (int)lane - lr * w;
          for (int jb = s.j0 + lr; jb - lr < s.j1; jb += 4 * rows) {
            unsigned long long key[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const int j = jb + h * rows;
              key[h] = lr < rows && j < s.j1 ? *(volatile unsigned long long*)(keys + (size_t)j * W + i) : ~0ull;
            }
#pragma unroll
            for (int h = 0; h < 4; ++h)
              if (jb - lr + h * rows < s.j1) consider(i, jb + h * rows, bound > key[h]);
          }
        }
      }
      if (ok & 2u) {
        volume_fragments(sl.s[1], lane,
                         [&](int i, int j, float v) { atomicAdd(acc + (size_t)j * W2 + i, fix40(v)); });
      }
    }
    __syncwarp();
    depth_fragments(C, slots[wib], qij[wib], qk[wib], qn, lane, base, R, W, keys);
    __syncwarp();
  }
}

// Per pixel: the winning fragment's eye depth (recomputed from its index),
// the updated depth buffer, and the volume map.
__global__ void k_resolve(Cam C, const float4* __restrict__ pos, float R, int W, int H, int W2, int H2,
                          const unsigned long long* keys, const unsigned long long* acc, float* depth, float* scene,
                          float* volume) {
  pbf::chain_begin(pos, keys, acc, depth, scene, volume);
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
  if (x >= W) return;
  const size_t p = (size_t)y * W + x;
  const unsigned long long key = keys[p];
  float s0 = scene ? scene[p] : 0.0f;
  s0 = s0 > 0.0f ? fminf(s0, 1.0f) : 0.0f;
  float out = 0.0f;
  if ((uint32_t)(key >> 32) != depth_bits(s0)) {
    const uint32_t q = 0xffffffffu - (uint32_t)key;
    const float4 xq = pos[q];
    float c[4];
    mat_vec(C.v, xq.x, xq.y, xq.z, 1.0f, c);
    Sprite s;
    make_sprite(C, c, 0.5f * R, W, H, s);
    float z;
    sprite_depth(C, s, sprite_r2(s, x, y), R, z);
    out = -z / s.cw;
    if (scene) scene[p] = __uint_as_float((uint32_t)(key >> 32));
  }
  depth[p] = out;
  if (x < W2 && y < H2) {
    const size_t p2 = (size_t)y * W2 + x;
    volume[p2] = (float)((double)acc[p2] * (1.0 / kFix));
  }
}

// The narrow-range filter for one texel given its window v[0 .. 2 half]
// (centre v[half]); false when the centre is not positive (no write).
__device__ inline bool narrow_range(const Gauss& G, const float* v, int stride, int half, float threshold, float mu,
                                    float& result) {
  const float center = v[half * stride];
  if (!(center > 0.0f)) return false;
  float value_sum = center, weight_sum = 1.0f;
  float lo = center - threshold, hi = center + threshold;
  const float bound_high = center + mu;
  for (int i = 1; i <= half; ++i) {
    float a = v[(half - i) * stride], b = v[(half + i) * stride];
    const float g = G.w[i];
    if (a < lo || b < lo) continue;
    a = a > hi ? bound_high : a;
    b = b > hi ? bound_high : b;
    lo = fminf(lo, fminf(a, b) - threshold);
    hi = fmaxf(hi, fmaxf(a, b) + threshold);
    weight_sum += g * 2.0f;
    value_sum += (a + b) * g;
  }
  result = value_sum / weight_sum;
  return true;
}

__global__ void __launch_bounds__(kFilterX) k_filter_x(const __grid_constant__ Gauss G, const float* __restrict__ src,
                                                      float* __restrict__ dst, int W, int H, int half, float threshold,
                                                      float mu) {
  __shared__ float row[kFilterX + 2 * kMaxHalf];
  const int x0 = blockIdx.x * kFilterX, y = blockIdx.y;
  pbf::chain_begin(src, dst);
  const float* s = src + (size_t)y * W;
  for (int k = threadIdx.x; k < kFilterX + 2 * kMaxHalf; k += kFilterX)
    row[k] = s[min(max(x0 - kMaxHalf + k, 0), W - 1)];
  __syncthreads();
  const int x = x0 + threadIdx.x;
  if (x >= W) return;
  float r;
  dst[(size_t)y * W + x] = narrow_range(G, row + threadIdx.x, 1, half, threshold, mu, r) ? r : 0.0f;
}

__global__ void __launch_bounds__(256) k_filter_y(const __grid_constant__ Gauss G, const float* __restrict__ src,
                                                  float* __restrict__ dst, int W, int H, int rows, int half,
                                                  float threshold, float mu) {
  __shared__ float col[kFilterYRows + 2 * kMaxHalf][33];
  const int x = blockIdx.x * 32 + threadIdx.x, y0 = blockIdx.y * rows;
  const int xc = min(x, W - 1);
  pbf::chain_begin(src, dst);
  for (int k = threadIdx.y; k < rows + 2 * kMaxHalf; k += 8)
    col[k][threadIdx.x] = src[(size_t)min(max(y0 - kMaxHalf + k, 0), H - 1) * W + xc];
  __syncthreads();
  if (x >= W) return;
  for (int q = threadIdx.y; q < rows; q += 8) {
    const int y = y0 + q;
    if (y >= H) break;
    float r;
    if (narrow_range(G, &col[q][threadIdx.x], 33, half, threshold, mu, r)) dst[(size_t)y * W + x] = r;
  }
}

}  // namespace

struct pbf_renderer {
  int W = 0, H = 0, W2 = 0, H2 = 0;
  pbf_render_options opt{};
  pbf_camera cam{};
  bool has_cam = false;
  Gauss gauss{};
  float* depth = nullptr;
  float* temp = nullptr;
  float* volume = nullptr;
  unsigned long long* keys = nullptr;
  unsigned long long* acc = nullptr;
  uint32_t* tile_min = nullptr;
  // volume sprites by tile, for up to vol_cap particles: tile and rank in it
  // per particle, order, then the tiles' counts and places
  uint32_t vol_cap = 0;
  uint2* vol_tile = nullptr;
  uint2* vol_order = nullptr;  // behind vol_tile's in one allocation
  uint32_t* vol_count = nullptr;
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  float ms[2] = {0.0f, 0.0f};
};

namespace {

void release(pbf_renderer* r) {
  cudaFree(r->depth);
  cudaFree(r->temp);
  cudaFree(r->volume);
  cudaFree(r->keys);
  cudaFree(r->acc);
  cudaFree(r->tile_min);
  cudaFree(r->vol_tile);
  cudaFree(r->vol_count);
  for (auto& e : r->ev)
    if (e) cudaEventDestroy(e);
}

// Gaussian weights of filterPassShader.ts: sigma = (filterSize >> 1) / 2,
// weight_i = exp(-i^2 * 0.5 / sigma^2) with the argument formed in float.
void gauss_table(uint32_t filter_size, float* g) {
  const int half = (int)(filter_size >> 1);
  const float sigma = (float)half * 0.5f;
  const float k = 0.5f / (sigma * sigma);
  for (int i = 0; i <= kMaxHalf; ++i) {
    const float arg = -(float)(i * i) * k;
    g[i] = (i <= half && half > 0) ? (float)std::exp((double)arg) : 0.0f;
  }
}

// TextureFilter.execute: x pass img -> temp, y pass temp -> img.
cudaError_t launch_filter(const Gauss& gauss, float* img, float* temp, int W, int H, uint32_t filter_size, float R,
                          cudaStream_t st) {
  if (filter_size < 2) return cudaSuccess;
  const int half = (int)(filter_size >> 1);
  const dim3 segments((unsigned)((W + kFilterX - 1) / kFilterX), (unsigned)H);
  const cudaError_t e = pbf::launch_chain(true, k_filter_x, segments, dim3(kFilterX), 0, st, gauss, img, temp, W, H, half,
                                          R * 5.0f, R);
  if (e != cudaSuccess) return e;
  // 64 rows a block read 1.5 texels per texel written, 16 rows 3: worth it where
  // the blocks are too few for the device
  const int rows = (int64_t)W * H < (1 << 20) ? 16 : kFilterYRows;
  return pbf::launch_chain(true, k_filter_y, dim3((unsigned)((W + 31) / 32), (unsigned)((H + rows - 1) / rows)),
                           dim3(32, 8), 0, st, gauss, temp, img, W, H, rows, half, R * 5.0f, R);
}

// Pixels across a particle's sprites, the same number on both maps, if it is as
// far from the camera as the world's origin (the reference's camera looks at
// it): what the splat's division of the work goes by.
double sprite_side(const Cam& C, double R, int H) {
  const double x = C.v[12], y = C.v[13], z = C.v[14];
  return R * std::fabs((double)C.p[5]) * H / (2.0 * std::max(std::sqrt(x * x + y * y + z * z), R));
}

size_t volume_tiles(const pbf_renderer* r) {
  return (size_t)((r->W2 + kVolTile - 1) / kVolTile) * ((r->H2 + kVolTile - 1) / kVolTile);
}

// Words per renderer: the tiles' counts and a 0 after them, which k_init clears,
// then the places of both.
size_t volume_words(const pbf_renderer* r) { return 2 * (volume_tiles(r) + 1); }

// Workspace for n particles (16 bytes each), kept and grown by half as much
// again, so that a scene that emits particles allocates a few times and not on
// every frame.
cudaError_t volume_workspace(pbf_renderer* r, uint32_t n, cudaStream_t st) {
  if (n <= r->vol_cap) return cudaSuccess;
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  cudaFree(r->vol_tile);
  r->vol_tile = nullptr;
  r->vol_cap = 0;
  uint32_t cap = (uint32_t)std::min<uint64_t>((uint64_t)n + n / 2, 0xfffffffeu);
  e = cudaMalloc(&r->vol_tile, 2 * (size_t)cap * sizeof(uint2));
  if (e != cudaSuccess) {
    cudaGetLastError();
    cap = n;
    e = cudaMalloc(&r->vol_tile, 2 * (size_t)cap * sizeof(uint2));
  }
  if (e != cudaSuccess) return e;
  r->vol_order = r->vol_tile + cap;
  r->vol_cap = cap;
  return cudaSuccess;
}

// The volume sprites summed by tile, once the splat has found their tiles.
cudaError_t volume_by_tile(pbf_renderer* r, const Cam& C, const float4* pos, uint32_t n, float R, cudaStream_t st) {
  const size_t m = volume_tiles(r) + 1;
  uint32_t* place = r->vol_count + m;
  // (entry m - 1 of the counts is 0: its place is the total)
  cudaError_t e = pbf::launch_chain(true, k_volume_places, 1, kPlaceThreads, 0, st, r->vol_count, (uint32_t)m, place);
  if (e == cudaSuccess)
    e = pbf::launch_chain(true, k_volume_order, (n - 1u) / 256u + 1u, 256, 0, st, n, r->vol_tile, place, r->vol_order);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_volume_sum, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kVolSmem);
  if (e == cudaSuccess)
    e = pbf::launch_chain(true, k_volume_sum, (n - 1u) / kVolRun + 1u, kVolThreads, kVolSmem, st, C, pos, R, r->W2,
                          r->H2, (r->W2 + kVolTile - 1) / kVolTile, r->vol_order, place + (m - 1), r->acc);
  return e;
}

bool finite16(const float* m) {
  for (int q = 0; q < 16; ++q)
    if (!std::isfinite(m[q])) return false;
  return true;
}

}  // namespace

extern "C" {

int pbf_renderer_create(uint32_t width, uint32_t height, pbf_renderer** out) {
  if (!out || width < 2 || height < 2 || width > 16384 || height > 16384) return PBF_EINVAL;
  *out = nullptr;
  pbf_renderer* r = new pbf_renderer();
  r->W = (int)width;
  r->H = (int)height;
  r->W2 = (int)(width / 2);  // fluidVolumeMap: canvas size / 2
  r->H2 = (int)(height / 2);
  // RenderingOptions defaults of the reference (src/common/config.ts:14-20)
  r->opt.mode = 0;
  r->opt.filter_size = 32;
  r->opt.particle_radius = 0.02f;
  r->opt.opacity = 0.25f;
  r->opt.tint_color[0] = 6.0f / 255.0f;
  r->opt.tint_color[1] = 105.0f / 255.0f;
  r->opt.tint_color[2] = 217.0f / 255.0f;
  const size_t px = (size_t)width * height, px2 = (size_t)r->W2 * r->H2;
  cudaError_t e = cudaMalloc(&r->depth, px * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&r->temp, px * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&r->volume, px2 * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&r->keys, px * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMalloc(&r->acc, px2 * sizeof(unsigned long long));
  if (e == cudaSuccess)
    e = cudaMalloc(&r->tile_min, (size_t)((width + kTile - 1) / kTile) * ((height + kTile - 1) / kTile) * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMalloc(&r->vol_count, volume_words(r) * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemset(r->depth, 0, px * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(r->volume, 0, px2 * sizeof(float));
  for (auto& ev : r->ev)
    if (e == cudaSuccess) e = cudaEventCreate(&ev);
  if (e != cudaSuccess) {
    release(r);
    delete r;
    return PBF_ECUDA;
  }
  pbf_renderer_set_config(r, &r->opt);
  *out = r;
  return PBF_OK;
}

int pbf_renderer_destroy(pbf_renderer* r) {
  if (!r) return PBF_EINVAL;
  cudaDeviceSynchronize();
  release(r);
  delete r;
  return PBF_OK;
}

int pbf_renderer_set_config(pbf_renderer* r, const pbf_render_options* o) {
  if (!r || !o || o->filter_size > 2 * kMaxHalf || !(o->particle_radius > 0.0f) ||
      !std::isfinite(o->particle_radius))
    return PBF_EINVAL;
  r->opt = *o;
  gauss_table(o->filter_size, r->gauss.w);
  return PBF_OK;
}

int pbf_renderer_set_camera(pbf_renderer* r, const pbf_camera* c) {
  if (!r || !c || !finite16(c->view) || !finite16(c->projection)) return PBF_EINVAL;
  const float* v = c->view;
  const float* p = c->projection;
  if (v[3] != 0.0f || v[7] != 0.0f || v[11] != 0.0f || v[15] != 1.0f) return PBF_EINVAL;  // affine view
  // projection without x/y shear: x_clip from (x, z), y_clip from (y, z), z_clip and w_clip from z
  if (p[1] != 0.0f || p[2] != 0.0f || p[3] != 0.0f || p[4] != 0.0f || p[6] != 0.0f || p[7] != 0.0f) return PBF_EINVAL;
  r->cam = *c;
  r->has_cam = true;
  return PBF_OK;
}

int pbf_render(pbf_renderer* r, const float* d_positions, uint32_t n, float* d_scene_depth, void* stream) {
  if (!r || (!d_positions && n) || !r->has_cam || n > 0xfffffffeu) return PBF_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  Cam C;
  std::memcpy(C.v, r->cam.view, sizeof(C.v));
  std::memcpy(C.p, r->cam.projection, sizeof(C.p));
  const float R = r->opt.particle_radius;
  const float4* pos = (const float4*)d_positions;
  cudaEventRecord(r->ev[0], st);
  const dim3 rows((unsigned)((r->W + 255) / 256), (unsigned)r->H);
  const double side = sprite_side(C, R, r->H);
  bool tiled = takes_tiles(n, side, r->W, r->H);
  if (tiled && volume_workspace(r, n, st) != cudaSuccess) {
    cudaGetLastError();  // without the workspace, everything is drawn at once
    tiled = false;
  }
  k_init<<<rows, 256, 0, st>>>(d_scene_depth, r->keys, r->acc, r->W, r->H, r->W2, r->H2, r->vol_count,
                               tiled ? (uint32_t)volume_tiles(r) + 1u : 0u);
  cudaError_t e = cudaSuccess;
  if (n) {
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int tw = (r->W + kTile - 1) / kTile, th = (r->H + kTile - 1) / kTile;
    auto splat = [&](int phase, uint64_t particles) {
      // Few particles are spread over the device, as a warp walks its own one
      // after another (8000 at 1920 x 1080, a frame: 32 a warp 219 us, 2 a warp
      // 73).  Many with small sprites are taken in blocks that set their sprites
      // up with most lanes, with large ones fewer, which is more even (us with
      // 8 / 16 / 32 a warp, at once: 400,000 with sides of 1.6 175 / 165 / 170,
      // 700,000 251 / 231 / 225, 380,000 with 4.1 197 / 191 / 201, 400,000 with
      // 32.8 4,783 / 5,097 / 5,916; the rest of the tiled path: 400,000 with 8.2
      // 331 / 325 / 341, 1,048,576 580 / 540 / 530, 620,000 with 16.4 at 3840 x
      // 2160 1,363 / 1,400 / 1,535).
      uint32_t per = 4;  // the first share
      if (phase == kAll) {
        per = side < 4.0 && n >= 300000u ? 32 : side < 5.7 && n >= 150000u ? 16 : 8;
        while (per > 1 && particles < (uint64_t)sms * 32 * per) per /= 2;
      } else if (phase == kRest) {
        per = side >= 10.5 ? 8 : side >= 6.5 && n < 800000u ? 16 : 32;
      }
      const uint64_t warps = (particles + per - 1) / per;
      // sprites of a step or two have no keys to read ahead (620,000 with sides
      // of 1.6: 211 us without, 217 with; 380,000 with 8.2: 371 and 355)
      auto kernel = phase == kAll && side < 5.0 ? k_splat<false> : k_splat<true>;
      return pbf::launch_chain(true, kernel, (unsigned)((warps + 7) / 8), 256, 0, st, C, pos, n, R, r->W,
                               r->H, r->W2, r->H2, r->keys, r->acc, phase, per, r->tile_min, tw, r->vol_tile,
                               r->vol_count);
    };
    if (!tiled) {
      e = splat(kAll, n);
    } else {
      e = splat(kFirst, ((uint64_t)n + kFirstShare - 1) / kFirstShare);
      if (e == cudaSuccess)
        e = pbf::launch_chain(true, k_tile_min, (unsigned)(((uint64_t)tw * th + 7) / 8), 256, 0, st, r->keys, r->W,
                              r->H, tw, r->tile_min);
      if (e == cudaSuccess) e = splat(kRest, n);
      if (e == cudaSuccess) e = volume_by_tile(r, C, pos, n, R, st);
    }
  }
  if (e == cudaSuccess)
    e = pbf::launch_chain(true, k_resolve, rows, 256, 0, st, C, pos, R, r->W, r->H, r->W2, r->H2, r->keys, r->acc,
                          r->depth, d_scene_depth, r->volume);
  if (e != cudaSuccess) return PBF_ECUDA;
  cudaEventRecord(r->ev[1], st);
  if (launch_filter(r->gauss, r->depth, r->temp, r->W, r->H, r->opt.filter_size, R, st) != cudaSuccess)
    return PBF_ECUDA;
  cudaEventRecord(r->ev[2], st);
  if (cudaGetLastError() != cudaSuccess) return PBF_ECUDA;
  if (cudaEventSynchronize(r->ev[2]) != cudaSuccess) return PBF_ECUDA;
  cudaEventElapsedTime(&r->ms[0], r->ev[0], r->ev[1]);
  cudaEventElapsedTime(&r->ms[1], r->ev[1], r->ev[2]);
  return PBF_OK;
}

int pbf_texture_filter(const pbf_render_options* o, float* d_texture, uint32_t width, uint32_t height, void* stream) {
  if (!o || (!d_texture && width && height) || o->filter_size > 2 * kMaxHalf || !(o->particle_radius > 0.0f) ||
      !std::isfinite(o->particle_radius) || width > 65536 || height > 65536)
    return PBF_EINVAL;
  if (o->filter_size < 2 || width == 0 || height == 0) return PBF_OK;
  cudaStream_t st = (cudaStream_t)stream;
  Gauss g;
  gauss_table(o->filter_size, g.w);
  float* temp = nullptr;
  if (cudaMallocAsync(&temp, (size_t)width * height * sizeof(float), st) != cudaSuccess) return PBF_ECUDA;
  cudaError_t e = launch_filter(g, d_texture, temp, (int)width, (int)height, o->filter_size, o->particle_radius, st);
  cudaFreeAsync(temp, st);
  // the texture is filtered when the call returns
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? PBF_OK : PBF_ECUDA;
}

int pbf_render_simulation(pbf_renderer* r, pbf_handle* h, float* d_scene_depth) {
  if (!r || !h) return PBF_EINVAL;
  return pbf_render(r, pbf_position_device(h), pbf_particle_count(h), d_scene_depth, pbf_stream(h));
}

const float* pbf_renderer_map_device(const pbf_renderer* r, uint32_t which) {
  if (!r) return nullptr;
  return which == PBF_RENDER_DEPTH ? r->depth : which == PBF_RENDER_VOLUME ? r->volume : nullptr;
}

int pbf_renderer_map_size(const pbf_renderer* r, uint32_t which, uint32_t* width, uint32_t* height) {
  if (!r || !width || !height || which > PBF_RENDER_VOLUME) return PBF_EINVAL;
  *width = (uint32_t)(which == PBF_RENDER_DEPTH ? r->W : r->W2);
  *height = (uint32_t)(which == PBF_RENDER_DEPTH ? r->H : r->H2);
  return PBF_OK;
}

int pbf_renderer_copy_map(const pbf_renderer* r, uint32_t which, float* host, size_t bytes) {
  uint32_t w, h;
  if (!host || pbf_renderer_map_size(r, which, &w, &h)) return PBF_EINVAL;
  if (bytes != (size_t)w * h * sizeof(float)) return PBF_EINVAL;
  return cudaMemcpy(host, pbf_renderer_map_device(r, which), bytes, cudaMemcpyDeviceToHost) == cudaSuccess
             ? PBF_OK
             : PBF_ECUDA;
}

int pbf_renderer_timings(const pbf_renderer* r, float ms[2]) {
  if (!r || !ms) return PBF_EINVAL;
  ms[0] = r->ms[0];
  ms[1] = r->ms[1];
  return PBF_OK;
}

}  // extern "C"
