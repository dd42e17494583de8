// vox_raster.cu — headless rasteriser of emitted meshes (vertex layout): the reference's
// vertex stage (src/shaders/vertex.vert:22-27, gl_Position = global matrix * vertex) and
// pipeline state (src/renderer/pipeline.rs:36-45: counter-clockwise front faces, back
// faces culled, depth test Less; src/renderer/renderer.rs:92-105: clear colour
// (0.1, 0.2, 0.3), depth 1.0), with a procedural stand-in for the texture images
// (fragment.frag samples image files, which are not part of this path).
//
// Pass 1 (k_raster_faces, k_raster_tiles): every pixel centre that a triangle (two per face,
// indices [0,2,1] and [3,1,2]) covers with depth in [0, 1) takes the 64-bit minimum of
// (depth bits << 32 | triangle id), which equals draw-order Less testing whatever the
// order the threads run in. Pass 2 (k_raster_shade): one thread per pixel shades the
// winning triangle (perspective-correct texture coordinates). Every float operation is
// written out in the order the CPU oracle uses (the file is built with -fmad=false).
//
// Pass 1 spreads a triangle over as many threads as its box has work for: a lane takes boxes of
// up to kLanePixels by itself, its warp boxes of up to kWarpPixels, and larger boxes are
// cut into tiles of 32 x 32 that k_raster_tiles deals out to all warps. (One thread a triangle
// left the image to the threads of the few nearest ones.) The tile list is kept in the output
// image, which pass 2 overwrites. The minimum is a reduction whose old value nobody waits for:
// reading a key first, to spare hidden pixels the update, made a warp's box a chain of loads
// (k_raster_faces 190 us instead of 66). Measured, us an image: 1280 x 720 over 64 chunks of
// 32^3 67 -> 51, 1920 x 1080 over 256 chunks of 16^3 1236 -> 71, 3840 x 2160 over 200 chunks of
// 32^3 1718 -> 280. With 8/512 as the limits; 16/128 takes 54 and 263 to 372, 16/1024 53 and 198
// to 283 (720p and 2160p, four views). At 720p the four launches take 4, 20, 10 and 11 us, each
// bound by latency; at 2160p boxes and shading are bound by their arithmetic.
#include <cstdint>

#include "voxgpu.h"
#include "vox_kernels.h"
#include "vox_launch.h"
#include "vox_types.h"

namespace vox {
namespace {

constexpr unsigned long long kEmptyKey = 0xFFFFFFFFFFFFFFFFull;

struct ScreenVert {
  float x, y, z, w;  // screen x, y (pixels, y down), NDC depth, clip w
  float u, v;
};

// Vertex k of face g through the global matrix (column-major), perspective divide and
// viewport transform. Returns false when the vertex is not in front of the camera.
__device__ __forceinline__ bool to_screen(const RasterArgs& a, unsigned long long g, int k,
                                          ScreenVert& o) {
  const float* vx = reinterpret_cast<const float*>(
      reinterpret_cast<const unsigned char*>(a.vertices) + g * 96ull + (unsigned)k * 24u);
  const float px = vx[0], py = vx[1], pz = vx[2];
  const float* m = a.m;
  const float cx = ((m[0] * px + m[4] * py) + m[8] * pz) + m[12];
  const float cy = ((m[1] * px + m[5] * py) + m[9] * pz) + m[13];
  const float cz = ((m[2] * px + m[6] * py) + m[10] * pz) + m[14];
  const float cw = ((m[3] * px + m[7] * py) + m[11] * pz) + m[15];
  if (!(cw > 0.0f)) return false;
  const float nx = cx / cw, ny = cy / cw, nz = cz / cw;
  o.x = (nx + 1.0f) * 0.5f * (float)a.width;
  o.y = (1.0f - ny) * 0.5f * (float)a.height;
  o.z = nz;
  o.w = cw;
  o.u = vx[3];
  o.v = vx[4];
  return true;
}

__device__ __forceinline__ float edge(const ScreenVert& a, const ScreenVert& b, float px, float py) {
  return (b.x - a.x) * (py - a.y) - (b.y - a.y) * (px - a.x);
}

// Top-left rule for an edge a -> b of a triangle with positive area (y down).
__device__ __forceinline__ bool top_left(const ScreenVert& a, const ScreenVert& b) {
  const float dx = b.x - a.x, dy = b.y - a.y;
  return dy < 0.0f || (dy == 0.0f && dx > 0.0f);
}

// The three vertices of triangle t of face g in the face's index order; false if culled.
__device__ __forceinline__ bool setup(const RasterArgs& a, unsigned long long g, int t,
                                      ScreenVert& v0, ScreenVert& v1, ScreenVert& v2, float& area) {
  const uint32_t* ix = reinterpret_cast<const uint32_t*>(
      reinterpret_cast<const unsigned char*>(a.indices) + g * 24ull + (unsigned)t * 12u);
  // chunk-local indices 4f + k: the vertex of this face is k = index & 3
  if (!to_screen(a, g, (int)(ix[0] & 3u), v0) || !to_screen(a, g, (int)(ix[1] & 3u), v1) ||
      !to_screen(a, g, (int)(ix[2] & 3u), v2))
    return false;
  area = edge(v0, v1, v2.x, v2.y);
  // counter-clockwise in NDC (y up) is clockwise on screen (y down): negative area
  if (!(area < 0.0f)) return false;  // back face or degenerate
  const ScreenVert tmp = v1;         // reorder to positive area
  v1 = v2;
  v2 = tmp;
  area = -area;
  return true;
}

constexpr int kLanePixels = 8;
constexpr int kWarpPixels = 512;
constexpr int kTile = 32;

// The list of tiles in the image buffer: their number, then {triangle, tile x | tile y << 16}.
struct TileList {
  unsigned* count;
  uint2* tiles;
  unsigned cap;
};
constexpr unsigned kNoTriangle = 0xFFFFFFFFu;

// What the coverage test of a triangle needs: screen positions, depths, area, fill rule.
struct Tri {
  float x[3], y[3], z[3], area;
  unsigned tl;  // bit i: edge i (opposite vertex i) is top or left
};
struct Box {
  int x0, y0, x1, y1;
  __device__ int pixels() const { return x1 < x0 || y1 < y0 ? 0 : (x1 - x0 + 1) * (y1 - y0 + 1); }
};

__device__ __forceinline__ void finish_tri(Tri& t, const ScreenVert& v0, const ScreenVert& v1,
                                           const ScreenVert& v2, float area) {
  t.x[0] = v0.x, t.x[1] = v1.x, t.x[2] = v2.x;
  t.y[0] = v0.y, t.y[1] = v1.y, t.y[2] = v2.y;
  t.z[0] = v0.z, t.z[1] = v1.z, t.z[2] = v2.z;
  t.area = area;
  t.tl = (top_left(v1, v2) ? 1u : 0u) | (top_left(v2, v0) ? 2u : 0u) | (top_left(v0, v1) ? 4u : 0u);
}

// The pixels whose centres may be covered (the whole image's at most).
__device__ __forceinline__ Box tri_box(const Tri& t, int width, int height) {
  const float fx0 = fminf(fminf(t.x[0], t.x[1]), t.x[2]), fx1 = fmaxf(fmaxf(t.x[0], t.x[1]), t.x[2]);
  const float fy0 = fminf(fminf(t.y[0], t.y[1]), t.y[2]), fy1 = fmaxf(fmaxf(t.y[0], t.y[1]), t.y[2]);
  if (fx1 < 0.0f || fy1 < 0.0f || fx0 > (float)width || fy0 > (float)height) return Box{0, 0, -1, -1};
  return Box{max(0, (int)floorf(fx0)), max(0, (int)floorf(fy0)), min(width - 1, (int)ceilf(fx1)),
             min(height - 1, (int)ceilf(fy1))};
}

__device__ __forceinline__ float edge_at(const Tri& t, int i, int j, float px, float py) {
  return (t.x[j] - t.x[i]) * (py - t.y[i]) - (t.y[j] - t.y[i]) * (px - t.x[i]);
}

__device__ __forceinline__ void raster_pixel(const Tri& t, uint32_t id, int px, int py, int width,
                                             unsigned long long* keys) {
  const float sx = (float)px + 0.5f, sy = (float)py + 0.5f;
  const float w0 = edge_at(t, 1, 2, sx, sy), w1 = edge_at(t, 2, 0, sx, sy), w2 = edge_at(t, 0, 1, sx, sy);
  const bool in = (w0 > 0.0f || (w0 == 0.0f && (t.tl & 1u))) && (w1 > 0.0f || (w1 == 0.0f && (t.tl & 2u))) &&
                  (w2 > 0.0f || (w2 == 0.0f && (t.tl & 4u)));
  if (!in) return;
  float z = ((w0 * t.z[0] + w1 * t.z[1]) + w2 * t.z[2]) / t.area;
  if (!(z >= 0.0f && z < 1.0f)) return;
  z = z + 0.0f;  // -0 -> +0, so that the key order is the float order
  const unsigned long long key = ((unsigned long long)__float_as_uint(z) << 32) | (unsigned long long)id;
  atomicMin(keys + (size_t)py * width + px, key);
}

__global__ void k_raster_clear(unsigned long long* keys, long long n, unsigned* tiles) {
  pdl_trigger();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i == 0 && tiles) *tiles = 0u;
  // two keys a store where they are 16-byte aligned
  const long long head = (reinterpret_cast<uintptr_t>(keys) & 15u) && n > 0 ? 1 : 0, pairs = (n - head) >> 1;
  if (i < pairs)
    reinterpret_cast<ulonglong2*>(keys + head)[i] = make_ulonglong2(kEmptyKey, kEmptyKey);
  if (i == 0 && head) keys[0] = kEmptyKey;
  if (i == 0 && head + 2 * pairs < n) keys[n - 1] = kEmptyKey;
}

__device__ __forceinline__ float pick(const float v[4], uint32_t k) {
  return k == 0u ? v[0] : (k == 1u ? v[1] : (k == 2u ? v[2] : v[3]));
}

// One thread per face: its four vertices once, then its two triangles. A warp's faces lie far
// apart in the list, so that the near faces of one chunk, whose boxes take the longest, fall to
// many warps (with neighbours in a warp the last warps ran 66 us instead of 20 on a 720p view
// over 64 chunks of 32^3).
__global__ void __launch_bounds__(128)
k_raster_faces(RasterArgs a, unsigned long long* keys, TileList list) {
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  const unsigned long long warps = gridDim.x * (unsigned long long)(blockDim.x / 32);
  const unsigned long long g = lane * warps + blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const bool face = g < a.faces;
  float vx[4], vy[4], vz[4];
  bool front[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    ScreenVert v;
    front[k] = face && to_screen(a, g, k, v);
    vx[k] = front[k] ? v.x : 0.0f;
    vy[k] = front[k] ? v.y : 0.0f;
    vz[k] = front[k] ? v.z : 0.0f;
  }
  const unsigned behind = (front[0] ? 0u : 1u) | (front[1] ? 0u : 2u) | (front[2] ? 0u : 4u) | (front[3] ? 0u : 8u);
  const uint32_t* ix = reinterpret_cast<const uint32_t*>(
      reinterpret_cast<const unsigned char*>(a.indices) + g * 24ull);
  // the vertices are older than the clearing launch, the keys and the list are not
  pdl_wait();
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    const uint32_t id = (uint32_t)(2ull * g + (unsigned)half);
    Tri t;
    Box box{0, 0, -1, -1};
    if (face) {
      // chunk-local indices 4f + k: the vertex of this face is k = index & 3
      const uint32_t k0 = ix[3 * half] & 3u, k1 = ix[3 * half + 1] & 3u, k2 = ix[3 * half + 2] & 3u;
      if (((behind >> k0) & 1u) == 0u && ((behind >> k1) & 1u) == 0u && ((behind >> k2) & 1u) == 0u) {
        ScreenVert v0, v1, v2;
        v0.x = pick(vx, k0), v0.y = pick(vy, k0), v0.z = pick(vz, k0);
        v1.x = pick(vx, k1), v1.y = pick(vy, k1), v1.z = pick(vz, k1);
        v2.x = pick(vx, k2), v2.y = pick(vy, k2), v2.z = pick(vz, k2);
        const float area = edge(v0, v1, v2.x, v2.y);
        // counter-clockwise in NDC (y up) is clockwise on screen (y down): negative area; the
        // others are back faces or degenerate
        if (area < 0.0f) {
          finish_tri(t, v0, v2, v1, -area);  // reordered to positive area
          box = tri_box(t, a.width, a.height);
        }
      }
    }
    const int pixels = box.pixels();
    if (pixels <= kLanePixels) {
      for (int py = box.y0; py <= box.y1; ++py)
        for (int px = box.x0; px <= box.x1; ++px) raster_pixel(t, id, px, py, a.width, keys);
    }
    // places in the tile list for the warp's large boxes, with one update of its length (an
    // update per box made the warps of near faces wait for up to 64 in turn)
    const int tx0 = box.x0 / kTile, ty0 = box.y0 / kTile;
    const unsigned tw = pixels > kWarpPixels ? (unsigned)(box.x1 / kTile - tx0 + 1) : 0u;
    const unsigned tiles = tw * (unsigned)(box.y1 / kTile - ty0 + 1);
    unsigned place = tiles;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, place, off);
      if (lane >= off) place += v;
    }
    const unsigned all = __shfl_sync(0xffffffffu, place, 31);
    place -= tiles;
    if (all != 0u) {
      // The length may run past the room, but not around: no warp adds to a full list or more
      // than its room, which is at most 2^18 (times every resident warp: below 2^32).
      unsigned base = list.cap;
      if (lane == 0 && all <= list.cap && *const_cast<volatile unsigned*>(list.count) < list.cap) base = atomicAdd(list.count, all);
      place += __shfl_sync(0xffffffffu, base, 0);
    }
    // a box whose tiles do not all fit is done here, its places in the list left empty
    const bool listed = tiles != 0u && place <= list.cap && tiles <= list.cap - place;
    unsigned rest = __ballot_sync(0xffffffffu, pixels > kLanePixels);
    while (rest) {  // one box after the other, by the whole warp
      const int from = __ffs(rest) - 1;
      rest &= rest - 1u;
      const uint32_t wid = __shfl_sync(0xffffffffu, id, from);
      const unsigned wtiles = __shfl_sync(0xffffffffu, tiles, from);
      const bool wlisted = __shfl_sync(0xffffffffu, (int)listed, from) != 0;
      if (wtiles != 0u) {
        const unsigned at = __shfl_sync(0xffffffffu, place, from), ww = __shfl_sync(0xffffffffu, tw, from);
        const unsigned wx = (unsigned)__shfl_sync(0xffffffffu, tx0, from), wy = (unsigned)__shfl_sync(0xffffffffu, ty0, from);
        for (unsigned k = lane; k < wtiles; k += 32)
          if (at < list.cap && k < list.cap - at)
            list.tiles[at + k] = make_uint2(wlisted ? wid : kNoTriangle, (wx + k % ww) | ((wy + k / ww) << 16));
        if (wlisted) continue;
      }
      Tri w;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        w.x[k] = __shfl_sync(0xffffffffu, t.x[k], from);
        w.y[k] = __shfl_sync(0xffffffffu, t.y[k], from);
        w.z[k] = __shfl_sync(0xffffffffu, t.z[k], from);
      }
      w.area = __shfl_sync(0xffffffffu, t.area, from);
      w.tl = __shfl_sync(0xffffffffu, t.tl, from);
      Box b;
      b.x0 = __shfl_sync(0xffffffffu, box.x0, from), b.y0 = __shfl_sync(0xffffffffu, box.y0, from);
      b.x1 = __shfl_sync(0xffffffffu, box.x1, from), b.y1 = __shfl_sync(0xffffffffu, box.y1, from);
      // 8 x 4 pixels a step
      for (int py = b.y0 + (lane >> 3); py <= b.y1; py += 4)
        for (int px = b.x0 + (lane & 7); px <= b.x1; px += 8) raster_pixel(w, wid, px, py, a.width, keys);
      __syncwarp();
    }
  }
}

// The listed tiles, a warp each: 32 pixels of a row a step.
__global__ void __launch_bounds__(256)
k_raster_tiles(RasterArgs a, unsigned long long* keys, TileList list) {
  pdl_trigger();
  pdl_wait();
  const unsigned n = min(*list.count, list.cap);
  const int lane = threadIdx.x & 31;
  for (unsigned e = blockIdx.x * 8u + (threadIdx.x >> 5); e < n; e += gridDim.x * 8u) {
    const uint2 tile = list.tiles[e];
    if (tile.x == kNoTriangle) continue;
    ScreenVert v0, v1, v2;
    float area;
    setup(a, tile.x >> 1, (int)(tile.x & 1u), v0, v1, v2, area);  // listed: it is a front face
    Tri t;
    finish_tri(t, v0, v1, v2, area);
    const Box b = tri_box(t, a.width, a.height);
    const int px = (int)(tile.y & 0xFFFFu) * kTile + lane, ty = (int)(tile.y >> 16) * kTile;
    if (px >= b.x0 && px <= b.x1)
      for (int py = max(b.y0, ty); py <= min(b.y1, ty + kTile - 1); ++py)
        raster_pixel(t, tile.x, px, py, a.width, keys);
  }
}

// Procedural texture: a base colour per texture index and a 4x4 checker over (u, v).
__device__ __forceinline__ void shade(uint32_t tex, float u, float v, uint8_t* rgba) {
  const float pal[4][3] = {{0.45f, 0.55f, 0.25f}, {0.45f, 0.32f, 0.20f},
                           {0.30f, 0.70f, 0.25f}, {0.60f, 0.60f, 0.60f}};
  const float* c = pal[tex & 3u];
  const int cu = (int)floorf(u * 4.0f), cv = (int)floorf(v * 4.0f);
  const float f = ((cu + cv) & 1) ? 0.85f : 1.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) rgba[k] = (uint8_t)(c[k] * f * 255.0f + 0.5f);
  rgba[3] = 255;
}

__global__ void k_raster_shade(RasterArgs a, const unsigned long long* keys, uint8_t* rgba) {
  pdl_wait();
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)a.width * a.height) return;
  uint8_t* o = rgba + 4 * i;
  const unsigned long long key = keys[i];
  if (key == kEmptyKey) {  // clear colour (0.1, 0.2, 0.3, 1.0)
    o[0] = (uint8_t)(0.1f * 255.0f + 0.5f);
    o[1] = (uint8_t)(0.2f * 255.0f + 0.5f);
    o[2] = (uint8_t)(0.3f * 255.0f + 0.5f);
    o[3] = 255;
    return;
  }
  const unsigned long long tri = key & 0xFFFFFFFFull;
  const unsigned long long g = tri >> 1;
  ScreenVert v0, v1, v2;
  float area;
  setup(a, g, (int)(tri & 1ull), v0, v1, v2, area);  // the winning triangle was set up before
  const float sx = (float)(i % a.width) + 0.5f, sy = (float)(i / a.width) + 0.5f;
  const float w0 = edge(v1, v2, sx, sy), w1 = edge(v2, v0, sx, sy), w2 = edge(v0, v1, sx, sy);
  // perspective-correct interpolation: weights w_i / clip w_i
  const float b0 = w0 / v0.w, b1 = w1 / v1.w, b2 = w2 / v2.w;
  const float den = (b0 + b1) + b2;
  const float u = ((b0 * v0.u + b1 * v1.u) + b2 * v2.u) / den;
  const float v = ((b0 * v0.v + b1 * v1.v) + b2 * v2.v) / den;
  const uint32_t slot = *reinterpret_cast<const uint32_t*>(
      reinterpret_cast<const unsigned char*>(a.vertices) + g * 96ull + 20u);
  shade(a.tex[slot < 6u ? slot : 0u], u, v, o);
}

}  // namespace

cudaError_t launch_raster(const RasterArgs& a, unsigned long long* keys, uint8_t* rgba,
                          cudaStream_t st) {
  const long long px = (long long)a.width * a.height;
  // the tile list in the image buffer: its count at the first 8-byte boundary, then the tiles
  const uintptr_t base = (reinterpret_cast<uintptr_t>(rgba) + 7u) & ~(uintptr_t)7u;
  const long long room = (long long)(reinterpret_cast<uintptr_t>(rgba) + 4ull * px) - (long long)base - 8;
  TileList list{reinterpret_cast<unsigned*>(base), reinterpret_cast<uint2*>(base + 8),
                room > 0 ? (unsigned)(room / 8 < (1ll << 18) ? room / 8 : (1ll << 18)) : 0u};
  const bool tiled = room >= 8 && px > kWarpPixels;  // else no box is large, and there is no list
  k_raster_clear<<<(unsigned)((px / 2 + 256) / 256), 256, 0, st>>>(keys, px, tiled ? list.count : nullptr);
  void* with_list[] = {const_cast<RasterArgs*>(&a), &keys, &list};
  void* with_image[] = {const_cast<RasterArgs*>(&a), &keys, &rgba};
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && a.faces > 0) {
    e = launch_dependent((const void*)k_raster_faces, dim3((unsigned)((a.faces + 127) / 128)), dim3(128),
                         with_list, 0, st);
    if (e == cudaSuccess && tiled)
      e = launch_dependent((const void*)k_raster_tiles, dim3(a.num_sms * 8), dim3(256), with_list, 0, st);
  }
  if (e != cudaSuccess) return e;
  return launch_dependent((const void*)k_raster_shade, dim3((unsigned)((px + 255) / 256)), dim3(256),
                          with_image, 0, st);
}

}  // namespace vox
