// vox_misc.cu — small kernels around the hot path: the chunk-frustum test, the indirect
// draw list of the visible meshes, and the conversions between occupancy bitmasks and the
// reference's one-byte-per-voxel cubes.
#include <cstdint>

#include "voxgpu.h"
#include "vox_device.cuh"
#include "vox_kernels.h"
#include "vox_launch.h"
#include "vox_types.h"

namespace vox {

namespace {

constexpr uint8_t kGrass = 0;  // CubeType::GRASS (src/cube.rs:17-21)
constexpr uint8_t kAir = 2;    // CubeType::AIR

// The two conversions stream one byte a voxel past one bit a voxel and are bound by HBM. Both
// arrays hold the voxels of all chunks in one order (x, z, y, chunk), so a thread works on
// units of 16 voxels without any chunk arithmetic: 16 bytes of cubes, and half a row word
// (N >= 32), one row word (N = 16) or two (N = 8). Each thread has kUnits units in flight, one
// block stride apart, so that a warp access covers 512 contiguous bytes. kVec = false serves
// cube buffers that are not 16-byte aligned (byte accesses, same units).
// Measured: vox_generate + vox_occ_to_cubes of 1500 chunks of 32^3 221 -> 41 us (the conversion
// alone was 196 us with one thread a byte and 64-bit divisions per voxel: 178 M warp
// instructions); vox_cubes_to_occ of 2048 chunks of 32^3 59.4 -> 14.6 us, 5.2 TB/s (one thread a
// row word before: 32 byte loads, 32 bytes apart across a warp).
constexpr int kUnits = 4;
constexpr int kConvThreads = 256;

// Four voxel bits -> four cube bytes (bit set: GRASS = 0, clear: AIR = 2).
__device__ __forceinline__ uint32_t cubes_of_bits(uint32_t b) {
  static_assert(kGrass == 0 && kAir == 2, "the spread below writes 2 for a clear bit");
  return (((~b & 0xFu) * 0x00204081u) & 0x01010101u) << 1;
}
// Four cube bytes -> four voxel bits (a byte other than AIR is solid).
__device__ __forceinline__ uint32_t bits_of_cubes(uint32_t v) {
  const uint32_t x = v ^ (0x01010101u * kAir);
  const uint32_t nz = (((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u;  // byte != AIR
  return ((nz >> 7) * 0x01020408u) >> 24;
}

template <int N, bool kVec>
__global__ void __launch_bounds__(kConvThreads)
k_occ_to_cubes(const uint32_t* __restrict__ occ, long long units, uint8_t* __restrict__ cubes) {
  const long long q0 = blockIdx.x * (long long)(kConvThreads * kUnits) + threadIdx.x;
  uint32_t bits[kUnits];
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const long long q = q0 + u * kConvThreads;
    bits[u] = 0u;
    if (q < units) {
      if (N >= 32) bits[u] = occ[q >> 1] >> (16 * (int)(q & 1));
      else if (N == 16) bits[u] = occ[q];
      else bits[u] = (occ[2 * q] & 0xFFu) | (occ[2 * q + 1] << 8);
    }
  }
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const long long q = q0 + u * kConvThreads;
    if (q >= units) continue;
    const uint32_t w[4] = {cubes_of_bits(bits[u]), cubes_of_bits(bits[u] >> 4),
                           cubes_of_bits(bits[u] >> 8), cubes_of_bits(bits[u] >> 12)};
    if (kVec) {
      reinterpret_cast<uint4*>(cubes)[q] = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 16; ++k) cubes[16 * q + k] = (uint8_t)(w[k >> 2] >> (8 * (k & 3)));
    }
  }
}

// A voxel is solid iff its byte is not AIR (chunk.rs:71). units is a multiple of 32, so a
// warp's lanes are all inside or all outside (the exchange below needs both halves of a word).
template <int N, bool kVec>
__global__ void __launch_bounds__(kConvThreads)
k_cubes_to_occ(const uint8_t* __restrict__ cubes, long long units, uint32_t* __restrict__ occ) {
  const long long q0 = blockIdx.x * (long long)(kConvThreads * kUnits) + threadIdx.x;
  uint4 v[kUnits];
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const long long q = q0 + u * kConvThreads;
    v[u] = make_uint4(0u, 0u, 0u, 0u);
    if (q >= units) continue;
    if (kVec) {
      v[u] = reinterpret_cast<const uint4*>(cubes)[q];
    } else {
      uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int k = 0; k < 16; ++k) w[k >> 2] |= (uint32_t)cubes[16 * q + k] << (8 * (k & 3));
      v[u] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
#pragma unroll
  for (int u = 0; u < kUnits; ++u) {
    const long long q = q0 + u * kConvThreads;
    if (q >= units) continue;  // the same for every lane of the warp
    const uint32_t b = bits_of_cubes(v[u].x) | (bits_of_cubes(v[u].y) << 4) |
                       (bits_of_cubes(v[u].z) << 8) | (bits_of_cubes(v[u].w) << 12);
    if (N >= 32) {
      const uint32_t other = __shfl_xor_sync(0xffffffffu, b, 1);
      if ((threadIdx.x & 1) == 0) occ[q >> 1] = b | (other << 16);
    } else if (N == 16) {
      occ[q] = b;
    } else {
      occ[2 * q] = b & 0xFFu;
      occ[2 * q + 1] = b >> 8;
    }
  }
}

// Frustum::contains (src/frustum_culling.rs:16-40) per chunk: corners in the reference's
// order, planes near, far, left, right, top, bottom; dist = ((a*x + b*y) + c*z) + d with
// one rounding per operation (the file is built with -fmad=false).

// Whether corner k of the chunk is inside every plane.
__device__ __forceinline__ bool corner_inside(const Planes& pl, float px, float py, float pz, float e, int k) {
  const float x = (k & 1) ? px + e : px;
  const float z = (k & 2) ? pz + e : pz;
  const float y = (k & 4) ? py + e : py;
  bool inside = true;
#pragma unroll
  for (int j = 0; j < 6; ++j) {
    const float d = pl.p[4 * j] * x + pl.p[4 * j + 1] * y + pl.p[4 * j + 2] * z + pl.p[4 * j + 3];
    inside = inside & !(d < 0.0f);
  }
  return inside;
}
__device__ __forceinline__ bool frustum_contains(const Planes& pl, vox_chunk_coord c, int extent) {
  const float px = (float)(c.x * extent), py = (float)(c.y * extent), pz = (float)(c.z * extent);
  bool any = false;
#pragma unroll
  for (int k = 0; k < 8; ++k) any = any | corner_inside(pl, px, py, pz, (float)extent, k);
  return any;
}

// One lane per corner: the launch is as short as its longest chain of operations, and a lane
// of eight corners takes eight times as many.
__global__ void __launch_bounds__(256)
k_frustum(Planes pl, const vox_chunk_coord* coords, int n, int extent, uint8_t* visible) {
  pdl_trigger();
  pdl_wait();
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long i = t >> 3;
  bool in = false;
  if (i < n) {
    const vox_chunk_coord c = coords[i];
    in = corner_inside(pl, (float)(c.x * extent), (float)(c.y * extent), (float)(c.z * extent), (float)extent,
                       (int)(t & 7));
  }
  const unsigned b = __ballot_sync(0xffffffffu, in);
  if (i < n && (t & 7) == 0) visible[i] = ((b >> (threadIdx.x & 24)) & 0xFFu) ? 1 : 0;
}

// World::render (src/world.rs:24-40) as an indirect draw list: a CTA takes kDrawTile chunks (a
// ticket each, so that it waits only for tiles that running CTAs hold), tests each
// (Frustum::contains), compacts the visible chunks that have faces in chunk order (warp ballots,
// a scan of the warp totals) and takes the tile's place in the list by look-back over the
// tiles before it. Records whose counts or offsets do not fit the 32-bit fields latch
// ERR_CAPACITY and are zeroed. Frustum test and list of 50,000 chunks 91 -> 12.8 us, of 8,000 20.5
// -> 12.7 us with one CTA walking all tiles before; both are now bound by the two calls (up to
// 2,000 chunks they were before, too).
// Tickets and look-back words are the draw lists' own, and the epoch is the host's count of them
// (they are issued in stream order), so that a list is independent of batches: of one that a
// caller's graph replays on another stream, and of one that gave up with its queue words mid-way.
// Without words one CTA (of kDrawWalk threads) walks the tiles by itself: the form of a call that
// a caller's graph records, whose replays must not depend on scratch that a later call may move.
constexpr int kDrawTile = 256, kDrawWalk = 1024;
__global__ void __launch_bounds__(kDrawWalk)
k_draw_list(Planes pl, const vox_chunk_coord* coords, const unsigned long long* offs, int n, int extent,
            int instanced, DrawRecord* out, uint32_t* count, BatchCtl* ctl, unsigned long long* words,
            unsigned epoch, int spin_limit) {
  __shared__ uint32_t wsum[kDrawWalk / 32];
  __shared__ unsigned s_tile;
  __shared__ uint32_t s_base;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int warps = (int)blockDim.x >> 5;
  const bool walk = words == nullptr;
  pdl_wait();
  if (t == 0 && !walk) {
    unsigned* tickets = reinterpret_cast<unsigned*>(words);
    s_tile = atomicAdd(tickets, 1u);
    if (s_tile == gridDim.x - 1u) *tickets = 0u;  // the last one
  }
  __syncthreads();
  const int tiles = walk ? (int)(((long long)n + blockDim.x - 1) / blockDim.x) : 1;
  const int tile0 = walk ? 0 : (int)s_tile;
  uint32_t walked = 0;  // warp 0: records of the tiles that this CTA has walked
  if (tiles == 0 && t == 0) *count = 0u;
  for (int tile = tile0; tile < tile0 + tiles; ++tile) {
    const long long i = (long long)tile * blockDim.x + t;
    bool vis = false;
    unsigned long long f0 = 0, nf = 0;
    if (i < n) {
      f0 = offs[i];
      nf = offs[i + 1] - f0;
      vis = nf > 0 && frustum_contains(pl, coords[i], extent);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, vis);
    const uint32_t before = (uint32_t)__popc(bal & ((1u << lane) - 1u));
    if (lane == 0) wsum[warp] = (uint32_t)__popc(bal);
    __syncthreads();
    if (warp == 0) {
      const uint32_t v = lane < warps ? wsum[lane] : 0u;
      uint32_t incl = v;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += u;
      }
      if (lane < warps) wsum[lane] = incl - v;
      const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
      const uint32_t excl =
          walk ? walked : (uint32_t)lookback(words + 1, ctl, epoch, tile, total, spin_limit);
      walked += total;
      if (lane == 0) {
        s_base = excl;
        if (tile == (walk ? tiles : (int)gridDim.x) - 1) *count = excl + total;
      }
    }
    __syncthreads();
    if (vis) {
      DrawRecord r;
      bool fits;
      if (instanced) {  // the quad's 6 indices, one instance per face
        fits = f0 + nf <= 0xFFFFFFFFull;
        r.index_count = 6u;
        r.instance_count = (uint32_t)nf;
        r.first_index = 0u;
        r.base_vertex = 0;
        r.first_instance = (uint32_t)f0;
      } else {          // 6 indices per face, chunk-local indices over 4 vertices per face
        fits = 6ull * (f0 + nf) <= 0xFFFFFFFFull && 4ull * f0 <= 0x7FFFFFFFull;
        r.index_count = (uint32_t)(6ull * nf);
        r.instance_count = 1u;
        r.first_index = (uint32_t)(6ull * f0);
        r.base_vertex = (int32_t)(4ull * f0);
        r.first_instance = 0u;
      }
      if (!fits) {
        atomicOr(&ctl->err, ERR_CAPACITY);
        r = DrawRecord{0u, 0u, 0u, 0, 0u};
      }
      out[s_base + wsum[warp] + before] = r;
    }
    if (walk) __syncthreads();  // wsum and s_base are read before the next tile writes them
  }
}

// Units of 16 voxels of n chunks of n_size^3, and the blocks that cover them.
long long conv_units(int n, int n_size) { return (long long)n * n_size * n_size * n_size / 16; }
unsigned conv_blocks(long long units) {
  return (unsigned)((units + kConvThreads * kUnits - 1) / (kConvThreads * kUnits));
}

template <int N>
void occ_to_cubes_n(const uint32_t* occ, long long units, uint8_t* cubes, cudaStream_t st) {
  if ((reinterpret_cast<uintptr_t>(cubes) & 15u) == 0)
    k_occ_to_cubes<N, true><<<conv_blocks(units), kConvThreads, 0, st>>>(occ, units, cubes);
  else
    k_occ_to_cubes<N, false><<<conv_blocks(units), kConvThreads, 0, st>>>(occ, units, cubes);
}

template <int N>
void cubes_to_occ_n(const uint8_t* cubes, long long units, uint32_t* occ, cudaStream_t st) {
  if ((reinterpret_cast<uintptr_t>(cubes) & 15u) == 0)
    k_cubes_to_occ<N, true><<<conv_blocks(units), kConvThreads, 0, st>>>(cubes, units, occ);
  else
    k_cubes_to_occ<N, false><<<conv_blocks(units), kConvThreads, 0, st>>>(cubes, units, occ);
}

}  // namespace

cudaError_t launch_occ_to_cubes(const uint32_t* occ, int n, int n_size, uint8_t* cubes,
                                cudaStream_t st) {
  const long long units = conv_units(n, n_size);
  if (units == 0) return cudaSuccess;
  switch (n_size) {
    case 8: occ_to_cubes_n<8>(occ, units, cubes, st); break;
    case 16: occ_to_cubes_n<16>(occ, units, cubes, st); break;
    default: occ_to_cubes_n<32>(occ, units, cubes, st); break;  // 32^3 and 64^3: full row words
  }
  return cudaGetLastError();
}

cudaError_t launch_cubes_to_occ(const uint8_t* cubes, int n, int n_size, uint32_t* occ,
                                cudaStream_t st) {
  const long long units = conv_units(n, n_size);
  if (units == 0) return cudaSuccess;
  switch (n_size) {
    case 8: cubes_to_occ_n<8>(cubes, units, occ, st); break;
    case 16: cubes_to_occ_n<16>(cubes, units, occ, st); break;
    default: cubes_to_occ_n<32>(cubes, units, occ, st); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_frustum(const Planes& planes, const void* coords, int n, int extent,
                           uint8_t* visible, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const Planes* pl = &planes;
  const vox_chunk_coord* c = static_cast<const vox_chunk_coord*>(coords);
  void* params[] = {const_cast<Planes*>(pl), &c, &n, &extent, &visible};
  return launch_dependent((const void*)k_frustum, dim3((unsigned)((8ll * n + 255) / 256)), dim3(256), params,
                          0, st);
}

int draw_list_tiles(int n) { return n > 0 ? (int)(((long long)n + kDrawTile - 1) / kDrawTile) : 1; }

cudaError_t launch_draw_list(const Planes& planes, const void* coords,
                             const unsigned long long* offs, int n, int extent, int instanced,
                             DrawRecord* out, uint32_t* count, BatchCtl* ctl, unsigned long long* words,
                             unsigned epoch, int spin_limit, cudaStream_t st) {
  const Planes* pl = &planes;
  const vox_chunk_coord* c = static_cast<const vox_chunk_coord*>(coords);
  void* params[] = {const_cast<Planes*>(pl), &c, &offs, &n, &extent, &instanced, &out, &count, &ctl, &words,
                    &epoch, &spin_limit};
  return launch_dependent((const void*)k_draw_list, dim3(words ? (unsigned)draw_list_tiles(n) : 1u),
                          dim3(words ? kDrawTile : kDrawWalk), params, 0, st);
}

}  // namespace vox

// ---------------------------------------------------------------------------------------
// Bounded-wait self-test: the look-back of chunk 1 waits on chunk 0, which never
// publishes (its state word is zero). The wait must end after spin_limit polls with the
// timeout bit latched, leaving the context usable.
// ---------------------------------------------------------------------------------------

namespace vox {
namespace {
__global__ void k_lookback_probe(unsigned long long* state2, BatchCtl* ctl, int spin_limit) {
  if (threadIdx.x < 32) (void)lookback(state2, ctl, 0xABCDEFu, 1, 0ull, spin_limit);
}
}  // namespace

cudaError_t launch_lookback_probe(unsigned long long* state2, BatchCtl* ctl, int spin_limit,
                                  cudaStream_t st) {
  k_lookback_probe<<<1, 32, 0, st>>>(state2, ctl, spin_limit);
  return cudaGetLastError();
}
}  // namespace vox
