// vox_device.cuh — device code of the chunk generation + meshing path (sm_103a).
//
// One CTA owns one chunk at a time. The chunk's occupancy lives in shared memory as
// one N-bit row per (y, z) (bit x = voxel solid), plus six halo rows per side. Face
// masks of a row come from shifts of the row and its neighbours, counts from popc.
// A deterministic block scan over rows gives every row's first face, the rows that have
// faces and the voxels that have faces. Chunks of a batch get their global first face
// from a decoupled look-back over a device work queue (k_mesh_batch), from one scan
// behind a grid barrier (k_mesh_batch_phased), or from a look-back over totals published
// by separate generation items (k_mesh_batch_overlap). Each warp compacts the faces of a
// run of voxels, stages them 32 at a time in shared memory in their final byte layout,
// and sends each batch to global memory with a TMA bulk copy
// (cp.async.bulk.global.shared::cta), or stores them directly.
//
// Reference semantics restated here (Blatko1/wgpu-voxel-engine):
//   fill rule            src/chunk.rs:35-45     (solid -> GRASS, else AIR)
//   culling/emission     src/chunk.rs:59-245    (y -> z -> x order; L R Bk F D U per voxel;
//                                               lateral halo only; y borders always emitted)
//   face records         src/quad.rs:14-54      (T * R instance matrix, texture index)
//   vertex expansion     src/shaders/vertex.vert:22-27
//
// Compiled with -fmad=false: every float expression rounds once per operation in the
// written order, which is what makes the noise and vertex bits match the CPU oracle.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "voxgpu.h"
#include "vox_schedule.h"
#include "vox_types.h"

namespace vox {

template <int N>
struct Shape {
  using RowT = typename std::conditional<(N > 32), unsigned long long, uint32_t>::type;
  static constexpr int R = N * N;                 // rows per chunk
  static constexpr int W = N > 32 ? N / 32 : 1;   // u32 words per row
  // CTA sizes the kernels are instantiated for (rows split evenly over the threads)
  static constexpr int T0 = N == 8 ? 32 : (N == 16 ? 128 : (N == 32 ? 256 : 512));
  static constexpr int T1 = 2 * T0;
  static constexpr int LOG2N = N == 8 ? 3 : (N == 16 ? 4 : (N == 32 ? 5 : 6));
  // Capacity of the face-voxel list (voxels with at least one face, as (row << LOG2N) | x
  // in 16 bits); a chunk with more face voxels is emitted row by row instead.
  static constexpr int VCap = N > 32 ? 0 : (N * N * N < 8192 ? N * N * N : 8192);
};

__host__ __device__ constexpr int align16(int b) { return (b + 15) & ~15; }

// Per-octave lattice data of one column coordinate (heightmap generation).
struct AxisX {
  int px, px1;  // p[X], p[X + 1]
  float fr, u;  // fractional coordinate and its fade
};
struct AxisZ {
  int y;        // lattice Y & 255
  float fr, v;  // fractional coordinate and its fade
  int pad;
};

// Octaves whose per-axis lattice data are computed between one pair of barriers.
constexpr int kOctGroup = 8;

// Density generation from per-chunk lattice tables (see dens_tables): per octave and axis
// the lattice data of the N + 2 coordinates (local -1..N), and the gradient coefficients
// of every lattice corner the chunk's coordinates touch. Configurations beyond these
// limits (more octaves, more corners, frequencies <= 0) take the per-sample hash path.
struct __align__(16) DensAxis {
  float fr, fr1;  // fractional coordinate, fractional - 1 (one f32x2 operand)
  float fade;     // fade of the fractional coordinate
  int ci;         // lattice cell relative to the chunk's first cell on this axis
};
constexpr int kDensMaxOct = 4;
template <int N>
__host__ __device__ constexpr int dens_max_corners() { return N <= 8 ? 128 : (N <= 16 ? 256 : 1024); }
// Byte offsets of the density tables in the generation scratch: int hdr[16] (per octave:
// corner-table base, corners along y and along z), DensAxis axes[octave][axis][N + 2],
// then the corner-pair records: record i holds the gradients of corner i and of corner i + 1
// (its +z neighbour on the lattice) as {gx_i, gx_i+1, gy_i, gy_i+1} and {gz_i, gz_i+1}; then
// the coarse samples and the cells of 8 x 4 x 8 voxels they decide (gen_density): per (y, z)
// cell row and 32-bit row word, the solid bits and the bits still to be evaluated, the list of
// the words with any such bits, and its length.
template <int N>
struct DensPlan {
  static constexpr int kCells = N / 8;                       // cells along x and along z
  static constexpr int kCellsY = N / 4;                      // cells along y
  static constexpr int kPts = kCells + 1;                    // coarse samples along x and z
  static constexpr int kPtsY = kCellsY + 1;
  static constexpr int kSegs = N > 32 ? N / 32 : 1;          // 32-bit words per row
  static constexpr int kWords = kCellsY * kCells * kSegs;    // row words over all (y, z) cells
  static constexpr int kAxes = 64;
  static constexpr int kPairXY = kAxes + kDensMaxOct * 3 * (N + 2) * 16;
  static constexpr int kPairZ = kPairXY + dens_max_corners<N>() * 16;
  static constexpr int kCoarse = kPairZ + dens_max_corners<N>() * 8;
  static constexpr int kKnown = kCoarse + align16(kPtsY * kPts * kPts * 4);
  static constexpr int kMixed = kKnown + align16(kWords * 4);
  static constexpr int kList = kMixed + align16(kWords * 4);  // [0]: length, then word indices
  static constexpr int kBytes = kList + align16((kWords + 1) * 4);
};
template <int N>
__host__ __device__ constexpr int dens_scratch_bytes() {
  return DensPlan<N>::kBytes;
}
// A warp's face list: the faces of one group of 32 voxels (6 each) after fewer than one
// batch of faces carried over from the previous group.
constexpr int kWarpFaces = 32 * 6 + 32;
// Faces one warp stages at a time (each warp has two staging buffers of this many faces).
constexpr int kWarpBatch = 32;
// Bytes of one warp staging buffer (vertex records, then the index records shifted by up
// to 8 bytes; or instance records shifted by up to 12 bytes).
template <int LAYOUT>
__host__ __device__ constexpr int warp_buf_bytes() {
  return LAYOUT == VOX_LAYOUT_INSTANCED ? align16(kWarpBatch * 68 + 16)
                                        : kWarpBatch * 96 + align16(kWarpBatch * 24 + 16);
}

// Shared-memory carve-up; the same functions size the launch on the host.
template <int N, int LAYOUT>
struct SmemPlan {
  using RowT = typename Shape<N>::RowT;
  static constexpr int kTables = align16((int)sizeof(TablesDev));
  static constexpr int kOcc = align16(Shape<N>::R * (int)sizeof(RowT));
  static constexpr int kHalo = align16(6 * N * (int)sizeof(RowT));
  static constexpr int kRows = align16((Shape<N>::R + 1) * 4);
  static constexpr int kNz = align16(Shape<N>::R * 2);
  static constexpr int kVList = align16(Shape<N>::VCap * 2);
  static constexpr int kMisc = 64;
  static constexpr int kFixed0 = kTables + kOcc + kHalo + kRows + kNz + kVList + kMisc;
  // the chunk state from occ through misc (contiguous in shared memory), as spilled by the
  // phased and overlap kernels: occupancy, halo, row offsets, row and voxel lists, counts
  static constexpr int kSpill = kOcc + kHalo + kRows + kNz + kVList + kMisc;
  // per-warp face lists (face-parallel emission)
  __host__ __device__ static int list_bytes(int threads) { return (threads / 32) * kWarpFaces * 4; }
  __host__ __device__ static int fixed(int threads) { return kFixed0 + list_bytes(threads); }
  // generation scratch, aliased with the staging window
  static constexpr int kColK = align16((N + 2) * (N + 2) * 4);
  static constexpr int kAxisHalf = kOctGroup * align16((N + 2) * 16);
  static constexpr int kAxis = 2 * kAxisHalf;
  // heightmap corner tables: per-octave header, then the gradient coefficients (gx, gy)
  static constexpr int kHHdr = align16((4 * kOctGroup + 1) * 4);
  static constexpr int kHeight = kColK + kAxis + kHHdr + dens_max_corners<N>() * 8;
  // hashed heightmap columns (up to 32^3): the hashed gradients, then the lattice data
  static constexpr int kHashed = N > 32 ? 0 : kGrad2 * 8 + 2 * kOctGroup * (N + 2) * 16;
  static constexpr int kScratch0 = kHeight > kHashed ? kHeight : kHashed;
  static constexpr int kGenScratch = kScratch0 > dens_scratch_bytes<N>() ? kScratch0 : dens_scratch_bytes<N>();
  // staging area: stage_faces / kWarpBatch buffers per warp when staging (stage_faces
  // 32 or 64), else only the generation scratch
  __host__ __device__ static int stage_bytes(int threads, int stage_faces) {
    const int b = stage_faces > 0
                      ? (threads / 32) * (stage_faces / kWarpBatch) * warp_buf_bytes<LAYOUT>()
                      : 0;
    return b < kGenScratch ? kGenScratch : b;
  }
  __host__ __device__ static int total(int threads, int stage_faces) {
    return fixed(threads) + stage_bytes(threads, stage_faces);
  }
};

// ------------------------------------------------------------------------------------
// Noise (Perlin improved noise, 2002) — same operation order as the CPU oracle.
// ------------------------------------------------------------------------------------

__device__ __forceinline__ float d_fade(float t) {
  return t * t * t * (t * (t * 6.0f - 15.0f) + 10.0f);
}
__device__ __forceinline__ float d_lerp(float t, float a, float b) { return a + t * (b - a); }

// Packed FP32 pairs: one f32x2 instruction performs the operation on both halves, each
// rounded to nearest like the scalar add / sub / mul, so a pair of scalar expressions
// evaluated this way gives the same bits with half the instructions. The low half is the
// first element.
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2_pack(float lo, float hi) {
  f2_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(f2_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
  f2_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2_t f2_sub(f2_t a, f2_t b) {
  f2_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
  f2_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// d_lerp on both halves. nz holds {-0, -0} that the compiler does not know: a mul.f32x2 whose
// product only an add.f32x2 takes can come out as one fused operation, in spite of -fmad=false
// and .rn (a product that the gradients' coefficients 0 and +-1 make exact is the same either
// way). The single rounding turned 17 of the 8 * 10^8 voxels of 24,576 chunks of 32^3 around the
// cave surface against the oracle, and against the same world voxels in chunks of the other
// sizes. As an fma with -0 the product is rounded by itself, sign of zero included: none.
__device__ __forceinline__ f2_t f2_lerp(f2_t t, f2_t a, f2_t b, f2_t nz) {
  f2_t m;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(m) : "l"(t), "l"(f2_sub(b, a)), "l"(nz));
  return f2_add(a, m);
}
// Gradient dot products from the coefficient table (gx, gy, gz) of hash & 15.
__device__ __forceinline__ float d_grad3(const float4* gt, int h, float x, float y, float z) {
  const float4 g = gt[h & 15];
  return (g.x * x + g.y * y) + g.z * z;
}
__device__ __forceinline__ float d_grad2(const float4* gt, int h, float x, float y) {
  const float4 g = gt[h & 15];
  return g.x * x + g.y * y;
}

__device__ __forceinline__ float d_noise3(const uint8_t* p, const float4* gt, float x, float y,
                                          float z) {
  float fx = floorf(x), fy = floorf(y), fz = floorf(z);
  int X = (int)fx & 255, Y = (int)fy & 255, Z = (int)fz & 255;
  x = x - fx;
  y = y - fy;
  z = z - fz;
  float u = d_fade(x), v = d_fade(y), w = d_fade(z);
  int A = p[X] + Y, AA = p[A] + Z, AB = p[A + 1] + Z;
  int B = p[X + 1] + Y, BA = p[B] + Z, BB = p[B + 1] + Z;
  float x1 = x - 1.0f, y1 = y - 1.0f, z1 = z - 1.0f;
  float l00 = d_lerp(u, d_grad3(gt, p[AA], x, y, z), d_grad3(gt, p[BA], x1, y, z));
  float l10 = d_lerp(u, d_grad3(gt, p[AB], x, y1, z), d_grad3(gt, p[BB], x1, y1, z));
  float l01 = d_lerp(u, d_grad3(gt, p[AA + 1], x, y, z1), d_grad3(gt, p[BA + 1], x1, y, z1));
  float l11 = d_lerp(u, d_grad3(gt, p[AB + 1], x, y1, z1), d_grad3(gt, p[BB + 1], x1, y1, z1));
  return d_lerp(w, d_lerp(v, l00, l10), d_lerp(v, l01, l11));
}

// noise2 at a column whose per-axis lattice data were computed once per octave; the
// operations are those of the oracle's or_noise2_f32, minus the shared subexpressions.
__device__ __forceinline__ float d_noise2_axes(const uint8_t* p, const float4* gt, const AxisX& ax,
                                               const AxisZ& az) {
  const int A = ax.px + az.y, B = ax.px1 + az.y;
  const float x = ax.fr, y = az.fr;
  const float x1 = x - 1.0f, y1 = y - 1.0f;
  const float l0 = d_lerp(ax.u, d_grad2(gt, p[p[A]], x, y), d_grad2(gt, p[p[B]], x1, y));
  const float l1 =
      d_lerp(ax.u, d_grad2(gt, p[p[A + 1]], x, y1), d_grad2(gt, p[p[B + 1]], x1, y1));
  return d_lerp(az.v, l0, l1);
}

// The same with the gradients of the hashed corners in a table (entry A: gradient of p[p[A]]).
__device__ __forceinline__ float d_noise2_hashed(const float2* grad2, const AxisX& ax, const AxisZ& az) {
  const float2* A = grad2 + ax.px + az.y;
  const float2* B = grad2 + ax.px1 + az.y;
  const float2 g00 = A[0], g01 = A[1], g10 = B[0], g11 = B[1];
  const float x = ax.fr, y = az.fr;
  const float x1 = x - 1.0f, y1 = y - 1.0f;
  const float l0 = d_lerp(ax.u, g00.x * x + g00.y * y, g10.x * x1 + g10.y * y);
  const float l1 = d_lerp(ax.u, g01.x * x + g01.y * y1, g11.x * x1 + g11.y * y1);
  return d_lerp(az.v, l0, l1);
}

__device__ __forceinline__ float d_fbm3(const uint8_t* p, const float4* gt, float x, float y,
                                        float z, const GenDev& g) {
  float sum = 0.0f, amp = 1.0f, f = g.freq;
  for (int o = 0; o < g.octaves; ++o) {
    sum = sum + amp * d_noise3(p, gt, x * f, y * f, z * f);
    f = f * g.lac;
    amp = amp * g.gain;
  }
  return sum;
}

// Draw i (0-based) of splitmix64 seeded with s0 is mix(s0 + (i + 1) * gamma).
__device__ __forceinline__ unsigned long long d_splitmix_at(unsigned long long s0,
                                                            unsigned long long i) {
  unsigned long long z = s0 + (i + 1ull) * 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// ------------------------------------------------------------------------------------
// Small helpers
// ------------------------------------------------------------------------------------

__device__ __forceinline__ int popc_row(uint32_t v) { return __popc(v); }
__device__ __forceinline__ int popc_row(unsigned long long v) { return __popcll(v); }

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// TMA bulk copies shared -> global (cp.async.bulk, bulk-group completion).
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void bulk_s2g(void* gdst, const void* ssrc, uint32_t bytes) {
  const uint32_t s = (uint32_t)__cvta_generic_to_shared(ssrc);
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
               ::"l"(gdst), "r"(s), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read_all() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// Issues [src, src + bytes) -> dst in pieces of at most 32 KiB (16-byte multiples).
__device__ __forceinline__ void bulk_s2g_pieces(unsigned char* dst, const unsigned char* src,
                                                uint32_t bytes) {
  while (bytes > 0) {
    const uint32_t b = bytes > 32768u ? 32768u : bytes;
    bulk_s2g(dst, src, b);
    dst += b;
    src += b;
    bytes -= b;
  }
}

// Look-back state word: epoch (24 bits) | flag (2 bits) | value (38 bits).
constexpr unsigned long long kFlagAgg = 1ull;
constexpr unsigned long long kFlagIncl = 2ull;
__device__ __forceinline__ unsigned long long pack_state(unsigned epoch, unsigned long long flag,
                                                         unsigned long long value) {
  return ((unsigned long long)(epoch & 0xFFFFFFu) << 40) | (flag << 38) |
         (value & ((1ull << 38) - 1));
}

// ------------------------------------------------------------------------------------
// Shared-memory view of one chunk
// ------------------------------------------------------------------------------------

template <int N, int LAYOUT>
struct ChunkSmem {
  using RowT = typename Shape<N>::RowT;
  TablesDev* tab;
  RowT* occ;        // [R]
  RowT* halo;       // [6][N]: 0 -x (bits z, by y), 1 +x, 2 -z (bits x, by y), 3 +z, 4 -y (bits x, by z), 5 +y
  uint32_t* rows;   // [R + 1] exclusive face offsets per row
  uint16_t* nz;     // rows that have faces, ascending
  uint16_t* vlist;  // face voxels in emission order, (row << LOG2N) | x (Shape<N>::VCap)
  int* misc;        // [0] rows with faces; [1] face voxels listed in vlist, or -1
  uint32_t* lists;  // per-warp face lists (packed x, y, z, dir)
  unsigned char* stage;
  // generation scratch (aliased with the staging window)
  int* colk;        // heightmap column thresholds
  AxisX* ax;        // per-octave x-axis lattice data, [kOctGroup][N + 2]
  AxisZ* az;        // per-octave z-axis lattice data, [kOctGroup][N + 2]
  int* hhdr;        // heightmap corner tables: per octave base, corners along z, first x, first z;
                    // [4 * kOctGroup] = corner count, or -1 when the tables are not used
  float2* hcorner;  // heightmap corner gradient coefficients (gx, gy)
  // heightmap columns up to 32^3 (ColumnHash): lattice data per octave and coordinate (x, then z), and
  // the gradients of the hashed corners; unused otherwise
  AxisX* hax;
  const float2* grad2;

  __device__ void carve(unsigned char* base) { carve(base, SmemPlan<N, LAYOUT>::list_bytes(blockDim.x)); }
  __device__ void carve(unsigned char* base, int list_bytes) {
    using P = SmemPlan<N, LAYOUT>;
    unsigned char* q = base;
    tab = reinterpret_cast<TablesDev*>(q);
    q += P::kTables;
    occ = reinterpret_cast<RowT*>(q);
    q += P::kOcc;
    halo = reinterpret_cast<RowT*>(q);
    q += P::kHalo;
    rows = reinterpret_cast<uint32_t*>(q);
    q += P::kRows;
    nz = reinterpret_cast<uint16_t*>(q);
    q += P::kNz;
    vlist = reinterpret_cast<uint16_t*>(q);
    q += P::kVList;
    misc = reinterpret_cast<int*>(q);
    q += P::kMisc;
    lists = reinterpret_cast<uint32_t*>(q);
    q += list_bytes;
    scratch_at(q);
  }
  // The staging area, and the generation scratch in the same place, at q.
  __device__ void scratch_at(unsigned char* q) {
    using P = SmemPlan<N, LAYOUT>;
    stage = q;
    colk = reinterpret_cast<int*>(q);
    ax = reinterpret_cast<AxisX*>(q + P::kColK);
    az = reinterpret_cast<AxisZ*>(q + P::kColK + P::kAxisHalf);
    hhdr = reinterpret_cast<int*>(q + P::kColK + P::kAxis);
    hcorner = reinterpret_cast<float2*>(q + P::kColK + P::kAxis + P::kHHdr);
  }
};

template <int N, int LAYOUT>
__device__ __forceinline__ void load_tables(ChunkSmem<N, LAYOUT>& s, const TablesDev* g) {
  const int words = (int)sizeof(TablesDev) / 4;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(g);
  uint32_t* dst = reinterpret_cast<uint32_t*>(s.tab);
  for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = src[i];
}

// The hashed gradient table (MeshArgs::grad2, kGrad2 entries) into shared memory at dst, with the
// lattice data's place behind it.
template <int T, int N, int LAYOUT>
__device__ __forceinline__ void load_grad2(ChunkSmem<N, LAYOUT>& s, unsigned char* dst, const float2* src) {
  const float4* from = reinterpret_cast<const float4*>(src);
  for (int i = threadIdx.x; i < kGrad2 / 2; i += T) reinterpret_cast<float4*>(dst)[i] = __ldg(from + i);
  s.grad2 = reinterpret_cast<const float2*>(dst);
  s.hax = reinterpret_cast<AxisX*>(dst + kGrad2 * 8);
}

// Write one ballot word for the element run [e0, e0 + 32) of a row-major bit array
// whose rows are N bits wide, into 32-bit word storage `words` (row r, word r*W + x/32).
template <int N>
__device__ __forceinline__ void store_ballot(uint32_t* words, int e, bool pred) {
  const unsigned b = __ballot_sync(0xffffffffu, pred);
  const int x = e % N;
  if ((x & 31) == 0) {
    const int row = e / N;
    constexpr uint32_t kMask = N >= 32 ? 0xFFFFFFFFu : ((1u << (N & 31)) - 1u);
    const uint32_t v = N >= 32 ? b : ((b >> (threadIdx.x & 31)) & kMask);
    words[row * Shape<N>::W + (x >> 5)] = v;
  }
}

template <int N>
__device__ __forceinline__ typename Shape<N>::RowT full_row() {
  using RowT = typename Shape<N>::RowT;
  return N >= 64 ? (RowT)~0ull : (RowT)((1ull << (N & 63)) - 1ull);
}

// ------------------------------------------------------------------------------------
// Occupancy generation into shared memory
// ------------------------------------------------------------------------------------

// Halo element (h, a, b) -> local voxel coordinates (may be -1 or N).
template <int N>
__device__ __forceinline__ void halo_coord(int h, int a, int b, int& x, int& y, int& z) {
  switch (h) {
    case 0: x = -1; y = a; z = b; break;
    case 1: x = N; y = a; z = b; break;
    case 2: x = b; y = a; z = -1; break;
    case 3: x = b; y = a; z = N; break;
    case 4: x = b; y = -1; z = a; break;
    default: x = b; y = N; z = a; break;
  }
}

// k = ceil(base + amp * fbm) - oy clamped to [-1, N + 1] (-1 for NaN): voxel (x, y, z) of a
// column is solid iff y < k.
template <int N>
__device__ __forceinline__ int threshold(const GenDev& g, float fbm, int oy) {
  const float h = g.base + g.amp * fbm;
  const float cl = ceilf(h);
  long long kk = (long long)cl - (long long)oy;
  if (!(cl == cl)) kk = -1;
  return (int)(kk < -1 ? -1 : (kk > N + 1 ? N + 1 : kk));
}

// How heightmap columns up to 32^3 get their lattice data. kHashAll: also from shared tables.
enum ColumnHash : int { kHashNone = 0, kHashGrad = 1, kHashAll = 2 };

// Threshold of one column (local x, z in -1..N), computed by the calling lane alone: the
// fBm of the per-column path (d_noise2_axes with the lattice data of this column). The same
// operations, in the same order, as the shared-table paths below and as the oracle. With
// kHash, s.grad2 holds the gradients of the hashed corners (entry A: the gradient of p[p[A]]),
// so a corner is one load instead of a chain of three.
template <int N, int kHash = kHashNone, int LAYOUT>
__device__ __forceinline__ int column_k(const ChunkSmem<N, LAYOUT>& s, const GenDev& g, int ox,
                                        int oy, int oz, int x, int z) {
  const uint8_t* p = s.tab->perm;
  const float4* gt = reinterpret_cast<const float4*>(s.tab->grad);
  float f = g.freq, amp = 1.0f, sum = 0.0f;
  for (int o = 0; o < g.octaves; ++o) {
    const float cx = (float)(ox + x) * f, cz = (float)(oz + z) * f;
    const float flx = floorf(cx), flz = floorf(cz);
    const int lx = (int)flx & 255;
    AxisX ax;
    ax.px = p[lx];
    ax.px1 = p[lx + 1];
    ax.fr = cx - flx;
    ax.u = d_fade(ax.fr);
    AxisZ az;
    az.y = (int)flz & 255;
    az.fr = cz - flz;
    az.v = d_fade(az.fr);
    az.pad = 0;
    sum = sum + amp * (kHash != kHashNone ? d_noise2_hashed(s.grad2, ax, az) : d_noise2_axes(p, gt, ax, az));
    f = f * g.lac;
    amp = amp * g.gain;
  }
  return threshold<N>(g, sum, oy);
}

// The same from the lattice data of the chunk's x and z coordinates (hashed_axes) too: a column
// and octave is two axis entries and four gradients, without the two floors and fades.
template <int N, int LAYOUT>
__device__ __forceinline__ int column_k_hashed(const ChunkSmem<N, LAYOUT>& s, const GenDev& g, int oy,
                                               int x, int z) {
  constexpr int side = N + 2;
  const AxisX* pax = s.hax + x + 1;
  const AxisZ* paz = reinterpret_cast<const AxisZ*>(s.hax + kOctGroup * side) + z + 1;
  float amp = 1.0f, sum = 0.0f;
  for (int o = 0; o < g.octaves; ++o) {
    const AxisX ax = pax[o * side];
    const AxisZ az = paz[o * side];
    sum = sum + amp * d_noise2_hashed(s.grad2, ax, az);
    amp = amp * g.gain;
  }
  return threshold<N>(g, sum, oy);
}

// The lattice data that column_k_hashed reads, for every x and z coordinate and up to kOctGroup
// octaves (all threads; ends with a barrier).
template <int N, int T, int LAYOUT>
__device__ __forceinline__ void hashed_axes(const ChunkSmem<N, LAYOUT>& s, const GenDev& g, int ox, int oz) {
  constexpr int side = N + 2;
  const uint8_t* p = s.tab->perm;
  AxisX* pax = s.hax;
  AxisZ* paz = reinterpret_cast<AxisZ*>(s.hax + kOctGroup * side);
  for (int i = threadIdx.x; i < 2 * side * g.octaves; i += T) {
    const int o = i / (2 * side), r = i % (2 * side), k = r % side - 1;
    float fo = g.freq;
    for (int q = 0; q < o; ++q) fo = fo * g.lac;
    const float c = (float)((r < side ? ox : oz) + k) * fo;
    const float fl = floorf(c);
    const int L = (int)fl & 255;
    const float fr = c - fl;
    if (r < side) {
      AxisX v;
      v.px = p[L];
      v.px1 = p[L + 1];
      v.fr = fr;
      v.u = d_fade(fr);
      pax[o * side + k + 1] = v;
    } else {
      AxisZ v;
      v.y = L;
      v.fr = fr;
      v.v = d_fade(fr);
      v.pad = 0;
      paz[o * side + k + 1] = v;
    }
  }
  __syncthreads();
}

// Heightmap chunk. Column thresholds colk[(z+1)*(N+2) + (x+1)] = ceil(h(x, z)) - oy,
// clamped to [-1, N + 1], so that voxel (x, y, z), y in [-1, N], is solid iff
// y < colk (the same as (float)(oy + y) < h for the integer y). The fBm runs octave by
// octave: the lattice data of every x and z coordinate are computed once per octave,
// each thread accumulating its own columns in registers.
//
// Three ways to the thresholds. Up to 32^3 every lane of the row phase below computes the
// threshold of its own column, with no shared lattice data, so that generation needs no CTA
// barrier before the row ballots; the list kernel hashes corners by table (kHashGrad), and
// k_generate, which has no latency to hide behind a count, also reads the coordinates' lattice
// data from a table (kHashAll: cubes of 1500 terrain chunks of 32^3 37.0 -> 34.9 us; in the list
// kernel it gained nothing at 16^3 and cost 5 % with one octave). The shared-table path (larger chunks): the lattice data and corner tables are built once per octave in shared memory,
// every thread accumulates its columns, and the thresholds go through s.colk.
template <int N, int LAYOUT, int T, int kHash>
__device__ void gen_heightmap(ChunkSmem<N, LAYOUT>& s, const GenDev& g, int ox, int oy, int oz,
                              unsigned halo_mask, bool with_halo) {
  using RowT = typename Shape<N>::RowT;
  constexpr int side = N + 2;
  constexpr bool direct = N <= 32;
  const int t = threadIdx.x;
  // the lattice data are worth their barrier from three octaves on
  const bool axes = kHash == kHashAll && g.octaves >= 3 && g.octaves <= kOctGroup;
  if (axes) hashed_axes<N, T>(s, g, ox, oz);
  if (!direct) {
    constexpr int CPT = (side * side + T - 1) / T;
    const uint8_t* p = s.tab->perm;
    const float4* gt = reinterpret_cast<const float4*>(s.tab->grad);
    float acc[CPT];
  #pragma unroll
    for (int c = 0; c < CPT; ++c) acc[c] = 0.0f;
    // Corner tables (one octave group, positive frequencies, few enough corners): per octave
    // the gradient coefficients of every lattice corner the chunk's columns touch. A corner's
    // hash p[p[p[X] + Y]] depends only on its coordinates mod 256 (the permutation table is
    // doubled), so a column reads 4 table entries instead of 8 permutation bytes and 4
    // gradient entries; the arithmetic is the per-column path's, in the same order.
    bool tab = false;
    if (g.octaves <= kOctGroup) {
      if (t < 32) {
        constexpr int kCap = dens_max_corners<N>();
        int cnt = 0, ncz = 0, x0 = 0, z0 = 0;
        bool ok = true;
        if (t < g.octaves) {
          float fo = g.freq;
          for (int q = 0; q < t; ++q) fo = fo * g.lac;
          // positive, and small enough that every cell index fits an int
          ok = fo > 0.0f && fabsf((float)(ox - 1) * fo) < 1.0e9f &&
               fabsf((float)(ox + N) * fo) < 1.0e9f && fabsf((float)(oz - 1) * fo) < 1.0e9f &&
               fabsf((float)(oz + N) * fo) < 1.0e9f;
          if (ok) {
            // coordinates grow with the local index (fo > 0): local -1 has the first cell
            x0 = (int)floorf((float)(ox - 1) * fo);
            z0 = (int)floorf((float)(oz - 1) * fo);
            const int ncx = (int)floorf((float)(ox + N) * fo) - x0 + 2;
            ncz = (int)floorf((float)(oz + N) * fo) - z0 + 2;
            ok = ncx > 0 && ncz > 0 && ncx <= kCap && ncz <= kCap && ncx * ncz <= kCap;
            cnt = ok ? ncx * ncz : 0;
          }
        }
        int incl = cnt;
  #pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, incl, off);
          if (t >= off) incl += u;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const bool all_ok = __all_sync(0xffffffffu, ok);
        if (t < g.octaves) {
          s.hhdr[4 * t + 0] = incl - cnt;
          s.hhdr[4 * t + 1] = ncz;
          s.hhdr[4 * t + 2] = x0;
          s.hhdr[4 * t + 3] = z0;
        }
        if (t == 0) s.hhdr[4 * kOctGroup] = all_ok && total <= kCap ? total : -1;
      }
      __syncthreads();
      tab = s.hhdr[4 * kOctGroup] >= 0;
    }
    float f = g.freq, amp = 1.0f;
    for (int o0 = 0; o0 < g.octaves; o0 += kOctGroup) {
      const int no = g.octaves - o0 < kOctGroup ? g.octaves - o0 : kOctGroup;
      // lattice data of every x and z coordinate for the octaves [o0, o0 + no)
      for (int i = t; i < 2 * side * no; i += T) {
        const int o = i / (2 * side), r = i % (2 * side);
        const int a = r / side, k = r % side - 1;
        float fo = f;
        for (int q = 0; q < o; ++q) fo = fo * g.lac;
        const float c = (float)(a == 0 ? ox + k : oz + k) * fo;
        const float fl = floorf(c);
        const int L = (int)fl & 255;
        const float fr = c - fl;
        if (a == 0) {
          AxisX v;
          // tables: the cell relative to the table's first x; else p[X], p[X + 1]
          v.px = tab ? (int)fl - s.hhdr[4 * o + 2] : p[L];
          v.px1 = tab ? 0 : p[L + 1];
          v.fr = fr;
          v.u = d_fade(fr);
          s.ax[o * side + k + 1] = v;
        } else {
          AxisZ v;
          v.y = tab ? (int)fl - s.hhdr[4 * o + 3] : L;
          v.fr = fr;
          v.v = d_fade(fr);
          v.pad = 0;
          s.az[o * side + k + 1] = v;
        }
      }
      if (tab) {
        const int total = s.hhdr[4 * kOctGroup];
        for (int i = t; i < total; i += T) {
          int o = 0;
          for (int q = 1; q < no; ++q)
            if (i >= s.hhdr[4 * q]) o = q;
          const int jj = i - s.hhdr[4 * o], nz = s.hhdr[4 * o + 1];
          const int X = (s.hhdr[4 * o + 2] + jj / nz) & 255, Y = (s.hhdr[4 * o + 3] + jj % nz) & 255;
          const float4 gg = gt[p[p[p[X] + Y]] & 15];
          s.hcorner[i] = make_float2(gg.x, gg.y);
        }
      }
      __syncthreads();
  #pragma unroll
      for (int c = 0; c < CPT; ++c) {
        const int j = t + c * T;
        if (j < side * side) {
          const int zi = j / side, xi = j % side;
          const bool corner = (zi == 0 || zi == side - 1) && (xi == 0 || xi == side - 1);
          if (!corner) {
            float a = amp, sum = acc[c];
            if (tab) {
              for (int o = 0; o < no; ++o) {
                const AxisX ax = s.ax[o * side + xi];
                const AxisZ az = s.az[o * side + zi];
                const int nz = s.hhdr[4 * o + 1];
                const float2* C = s.hcorner + s.hhdr[4 * o] + ax.px * nz + az.y;
                const float2 g00 = C[0], g01 = C[1], g10 = C[nz], g11 = C[nz + 1];
                const float x = ax.fr, y = az.fr;
                const float x1 = x - 1.0f, y1 = y - 1.0f;
                const float l0 = d_lerp(ax.u, g00.x * x + g00.y * y, g10.x * x1 + g10.y * y);
                const float l1 = d_lerp(ax.u, g01.x * x + g01.y * y1, g11.x * x1 + g11.y * y1);
                sum = sum + a * d_lerp(az.v, l0, l1);
                a = a * g.gain;
              }
            } else {
              for (int o = 0; o < no; ++o) {
                sum = sum + a * d_noise2_axes(p, gt, s.ax[o * side + xi], s.az[o * side + zi]);
                a = a * g.gain;
              }
            }
            acc[c] = sum;
          }
        }
      }
      for (int o = 0; o < no; ++o) {
        f = f * g.lac;
        amp = amp * g.gain;
      }
      // the next group rewrites the lattice data; after the last group the thresholds
      // below use only this thread's sums
      if (o0 + kOctGroup < g.octaves) __syncthreads();
    }
  #pragma unroll
    for (int c = 0; c < CPT; ++c) {
      const int j = t + c * T;
      if (j < side * side) {
        s.colk[j] = threshold<N>(g, acc[c], oy);
      }
    }
    __syncthreads();
  }  // !direct
  // Rows from the column thresholds, one warp task per 32 columns: the own columns of a group of
  // z values, or the columns of the lateral halo strips (for N < 32 several side by side).
  // Lanes hold one column's threshold k each. Row y of the task is the ballot of y < k: full
  // below the task's smallest k, empty from its largest on, so only the rows in between are
  // voted on; lane y keeps row y, and one store per lane writes the rows.
  {
    constexpr int S = N > 32 ? N / 32 : 1;   // 32-bit words per row
    constexpr int LW = N >= 32 ? 32 : N;     // lanes per row word
    constexpr int G = 32 / LW;               // z values per own task
    constexpr int HP = G < 4 ? G : 4;        // halo strips per halo task
    constexpr int W = Shape<N>::W;
    constexpr int YP = N > 32 ? N / 32 : 1;  // rows a lane keeps
    constexpr uint32_t kWordFull = N >= 32 ? 0xFFFFFFFFu : ((1u << (N & 31)) - 1u);
    constexpr int kOwnTasks = (N / G) * S;
    const int tasks = kOwnTasks + (with_halo ? (4 / HP) * S : 0);
    const int lane = t & 31, warp = t >> 5;
    constexpr int nwarps = T / 32;
    uint32_t* occw = reinterpret_cast<uint32_t*>(s.occ);
    uint32_t* halow = reinterpret_cast<uint32_t*>(s.halo);
    const int sub = lane / LW, b = lane % LW;  // row word group and bit of this lane
    const bool vertical = with_halo && (halo_mask >> 4) != 0u;
    for (int task = warp; task < tasks; task += nwarps) {
      const bool own = task < kOwnTasks;
      const int seg = own ? task % S : (task - kOwnTasks) % S;
      const int xb = seg * 32 + b;  // bit position within the row
      const int z0 = (task / S) * G, h0 = own ? 0 : ((task - kOwnTasks) / S) * HP;
      int x = xb, z = z0 + sub;
      bool used = true;
      if (!own) {
        const int h = h0 + (sub < HP ? sub : HP - 1);
        used = ((halo_mask >> h) & 1u) != 0u;
        x = h == 0 ? -1 : (h == 1 ? N : xb);
        z = h == 2 ? -1 : (h == 3 ? N : xb);
      }
      int k = -1;
      if (used) {
        if (!direct) k = s.colk[(z + 1) * side + x + 1];
        else if (axes) k = column_k_hashed<N>(s, g, oy, x, z);
        else k = column_k<N, kHash>(s, g, ox, oy, oz, x, z);
      }
      const int kmin = __reduce_min_sync(0xffffffffu, k), kmax = __reduce_max_sync(0xffffffffu, k);
      uint32_t keep[YP];
#pragma unroll
      for (int j = 0; j < YP; ++j) keep[j] = lane + 32 * j < kmin ? 0xFFFFFFFFu : 0u;
      for (int y = kmin < 0 ? 0 : kmin; y < (kmax > N ? N : kmax); ++y) {
        const uint32_t bal = __ballot_sync(0xffffffffu, y < k);
#pragma unroll
        for (int j = 0; j < YP; ++j)
          if (lane + 32 * j == y) keep[j] = bal;
      }
#pragma unroll
      for (int j = 0; j < YP; ++j) {
        const int y = lane + 32 * j;
        if (y >= N) continue;
        if (!own) {
#pragma unroll
          for (int q = 0; q < HP; ++q)
            halow[((h0 + q) * N + y) * W + seg] = (keep[j] >> ((q * LW) & 31)) & kWordFull;
        } else if (N == 16) {
          *reinterpret_cast<uint2*>(occw + y * N + z0) = make_uint2(keep[j] & 0xFFFFu, keep[j] >> 16);
        } else if (N == 8) {
          *reinterpret_cast<uint4*>(occw + y * N + z0) = make_uint4(
              keep[j] & 0xFFu, (keep[j] >> 8) & 0xFFu, (keep[j] >> 16) & 0xFFu, keep[j] >> 24);
        } else {
          occw[(y * N + z0) * W + seg] = keep[j];
        }
      }
      if (own && with_halo) {
        // -y and +y halo rows of these z values (bits x): y = -1 and y = N
        uint32_t b4 = 0u, b5 = 0u;
        if (vertical) {
          b4 = __ballot_sync(0xffffffffu, ((halo_mask >> 4) & 1u) && -1 < k);
          b5 = __ballot_sync(0xffffffffu, ((halo_mask >> 5) & 1u) && N < k);
        }
        if (b == 0) {
          halow[(4 * N + z) * W + seg] = (b4 >> lane) & kWordFull;
          halow[(5 * N + z) * W + seg] = (b5 >> lane) & kWordFull;
        }
      }
    }
  }
  __syncthreads();
}

template <int N, int GM, int LAYOUT>
__device__ __forceinline__ bool gen_solid(const ChunkSmem<N, LAYOUT>& s, const GenDev& g, int x,
                                          int y, int z, int ox, int oy, int oz,
                                          unsigned long long s0) {
  if (GM == GM_DENSITY) {
    const int wy = oy + y;
    const float f = d_fbm3(s.tab->perm, reinterpret_cast<const float4*>(s.tab->grad),
                           (float)(ox + x), (float)wy, (float)(oz + z), g);
    const float d = f - ((float)wy - g.y_ref) * g.y_scale;
    return g.solid_below_zero ? (d < 0.0f) : (d > 0.0f);
  } else {  // GM_BERNOULLI
    const unsigned long long i = (unsigned long long)(x + N * z + N * N * y);
    return (d_splitmix_at(s0, i) & 1ull) != 0ull;
  }
}

// Builds the density lattice tables of a chunk in the generation scratch (all threads; ends
// with a barrier) and returns true, or returns false without a barrier when the
// configuration is beyond the table limits (the same answer in every thread). The layout
// is DensPlan's.
template <int N, int LAYOUT, int T>
__device__ bool dens_tables(ChunkSmem<N, LAYOUT>& s, const GenDev& g, int ox, int oy, int oz) {
  using P = DensPlan<N>;
  if (g.octaves > kDensMaxOct) return false;
  int* hdr = reinterpret_cast<int*>(s.stage);
  DensAxis* axes = reinterpret_cast<DensAxis*>(s.stage + P::kAxes);
  uint4* pair_xy = reinterpret_cast<uint4*>(s.stage + P::kPairXY);
  uint2* pair_z = reinterpret_cast<uint2*>(s.stage + P::kPairZ);
  const int org[3] = {ox, oy, oz};
  // corner counts (every thread computes them; cheap)
  int lo[kDensMaxOct][3], nc[kDensMaxOct][3], base[kDensMaxOct];
  int total = 0;
  float f = g.freq;
#pragma unroll
  for (int o = 0; o < kDensMaxOct; ++o) {
    if (o < g.octaves) {
      if (!(f > 0.0f)) return false;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        // coordinates grow with the local index (f > 0): local -1 has the first cell, N the last
        const int c0 = (int)floorf((float)(org[a] - 1) * f);
        const int c1 = (int)floorf((float)(org[a] + N) * f);
        lo[o][a] = c0;
        nc[o][a] = c1 - c0 + 2;  // corners along this axis
      }
      base[o] = total;
      total += nc[o][0] * nc[o][1] * nc[o][2];
      f = f * g.lac;
    }
  }
  if (total > dens_max_corners<N>()) return false;
  const int t = threadIdx.x;
  if (t < g.octaves) {
    hdr[4 * t + 0] = base[t];
    hdr[4 * t + 1] = nc[t][1];
    hdr[4 * t + 2] = nc[t][2];
  }
  // axis data: the oracle's per-sample operations, once per coordinate
  for (int i = t; i < g.octaves * 3 * (N + 2); i += T) {
    const int o = i / (3 * (N + 2)), r = i % (3 * (N + 2));
    const int a = r / (N + 2), k = r % (N + 2);
    float fo = g.freq;
    for (int q = 0; q < o; ++q) fo = fo * g.lac;
    const float c = (float)(org[a] + k - 1) * fo;
    const float fl = floorf(c);
    DensAxis v;
    v.fr = c - fl;
    v.fade = d_fade(v.fr);
    v.fr1 = v.fr - 1.0f;
    int c0 = 0;
#pragma unroll
    for (int q = 0; q < kDensMaxOct; ++q)
#pragma unroll
      for (int b = 0; b < 3; ++b)
        if (q == o && b == a) c0 = lo[q][b];
    v.ci = (int)fl - c0;
    axes[i] = v;
  }
  // corner gradients: hash p[p[p[X] + Y] + Z] of the corner's lattice coordinates mod 256
  // (the doubled permutation makes this the hash the per-sample chain computes)
  const uint8_t* p = s.tab->perm;
  const float4* gt = reinterpret_cast<const float4*>(s.tab->grad);
  for (int i = t; i < total; i += T) {
    int o = 0;
#pragma unroll
    for (int q = 1; q < kDensMaxOct; ++q)
      if (q < g.octaves && i >= base[q]) o = q;
    int ix = 0, iy = 0, iz = 0, l0 = 0, l1 = 0, l2 = 0, n1 = 1, n2 = 1, b0 = 0;
#pragma unroll
    for (int q = 0; q < kDensMaxOct; ++q)
      if (q == o) {
        b0 = base[q];
        n1 = nc[q][1];
        n2 = nc[q][2];
        l0 = lo[q][0];
        l1 = lo[q][1];
        l2 = lo[q][2];
      }
    const int j = i - b0;
    iz = j % n2;
    iy = (j / n2) % n1;
    ix = j / (n1 * n2);
    const int X = (l0 + ix) & 255, Y = (l1 + iy) & 255, Z = (l2 + iz) & 255;
    // corner i and its +z neighbour (the record of a chunk's last z corner is never read)
    const float4 g0 = gt[p[p[p[X] + Y] + Z] & 15];
    const float4 g1 = gt[p[p[p[X] + Y] + ((Z + 1) & 255)] & 15];
    pair_xy[i] = make_uint4(__float_as_uint(g0.x), __float_as_uint(g1.x), __float_as_uint(g0.y),
                            __float_as_uint(g1.y));
    pair_z[i] = make_uint2(__float_as_uint(g0.z), __float_as_uint(g1.z));
  }
  __syncthreads();
  return true;
}

// Density of local sample (x, y, z), -1 <= x, y, z <= N, from the lattice tables: the
// operations of the per-sample path (d_fbm3, then the height term), in the same order.
template <int N, int LAYOUT>
__device__ __forceinline__ float dens_value_tab(const ChunkSmem<N, LAYOUT>& s, const GenDev& g,
                                                int x, int y, int z, int oy) {
  using P = DensPlan<N>;
  const int* hdr = reinterpret_cast<const int*>(s.stage);
  const DensAxis* axes = reinterpret_cast<const DensAxis*>(s.stage + P::kAxes);
  const float4* pair_xy = reinterpret_cast<const float4*>(s.stage + P::kPairXY);
  const float2* pair_z = reinterpret_cast<const float2*>(s.stage + P::kPairZ);
  float sum = 0.0f, amp = 1.0f;
  for (int o = 0; o < g.octaves; ++o) {
    const DensAxis* ao = axes + o * 3 * (N + 2);
    const DensAxis ax = ao[x + 1], ay = ao[(N + 2) + y + 1], az = ao[2 * (N + 2) + z + 1];
    const int n1 = hdr[4 * o + 1], n2 = hdr[4 * o + 2];
    const int sx = n1 * n2;
    // the pair records of the four (x, y) corner columns: corners z and z + 1
    const int c = hdr[4 * o] + (ax.ci * n1 + ay.ci) * n2 + az.ci;
    const float4 q00 = pair_xy[c], q10 = pair_xy[c + sx], q01 = pair_xy[c + n2],
                 q11 = pair_xy[c + sx + n2];
    const float2 h00 = pair_z[c], h10 = pair_z[c + sx], h01 = pair_z[c + n2],
                 h11 = pair_z[c + sx + n2];
    const float3 g000 = make_float3(q00.x, q00.z, h00.x), g001 = make_float3(q00.y, q00.w, h00.y);
    const float3 g100 = make_float3(q10.x, q10.z, h10.x), g101 = make_float3(q10.y, q10.w, h10.y);
    const float3 g010 = make_float3(q01.x, q01.z, h01.x), g011 = make_float3(q01.y, q01.w, h01.y);
    const float3 g110 = make_float3(q11.x, q11.z, h11.x), g111 = make_float3(q11.y, q11.w, h11.y);
    const float xf = ax.fr, yf = ay.fr, zf = az.fr, x1 = ax.fr1, y1 = ay.fr1, z1 = az.fr1;
    const float u = ax.fade, v = ay.fade, w = az.fade;
    const float l00 = d_lerp(u, (g000.x * xf + g000.y * yf) + g000.z * zf,
                             (g100.x * x1 + g100.y * yf) + g100.z * zf);
    const float l10 = d_lerp(u, (g010.x * xf + g010.y * y1) + g010.z * zf,
                             (g110.x * x1 + g110.y * y1) + g110.z * zf);
    const float l01 = d_lerp(u, (g001.x * xf + g001.y * yf) + g001.z * z1,
                             (g101.x * x1 + g101.y * yf) + g101.z * z1);
    const float l11 = d_lerp(u, (g011.x * xf + g011.y * y1) + g011.z * z1,
                             (g111.x * x1 + g111.y * y1) + g111.z * z1);
    const float n = d_lerp(w, d_lerp(v, l00, l10), d_lerp(v, l01, l11));
    sum = sum + amp * n;
    amp = amp * g.gain;
  }
  return sum - ((float)(oy + y) - g.y_ref) * g.y_scale;
}

// What is known about a density chunk before any sample of it is evaluated (the same answer
// in every thread).
//
// Perlin's noise is bounded: a value is a convex combination of gradient dot products, and
// its largest magnitude over every choice of the corner gradients is 1.0364. And it is smooth:
// along an axis it is twice continuously differentiable, across lattice cells too, with a
// second derivative (per squared cell) below 12.1 for every choice of gradients (a test
// computes both from the formulas). So the density, the fBm minus a term linear in y, stays
// within 1.037 * sum|amp| of that term, and inside a cell of voxels of edge h it stays within
// `slack` = 13/8 * sum |amp| f^2 (h^2 + h^2 + hy^2) of the range of its values at the cell's eight
// corners (trilinear interpolation error). A cell whose corner densities all exceed the slack
// with one sign therefore needs no evaluation (the cells are h by h, and hy along y). `err` covers the rounding of the computed values
// against exact arithmetic: coordinates are off by up to 2^-24 of their size, which moves a
// value by less than 2e-6 * |c| (the slope of the noise is below 5 a cell on each axis); the
// arithmetic of one value rounds to less than 4e-5; the height term and the sum to less than
// 4e-6 of their size. Configurations outside these assumptions (coordinates of 2^24 and more,
// infinite or NaN parameters) make a comparison below false and are evaluated in full, as are
// frequencies so high that the slack exceeds the fBm's own range.
struct DensBounds {
  int known;    // 0: every sample is air, 1: every sample is solid, -1: not known
  float slack;  // a cell with corner densities beyond +-slack is known; infinite: none is
};
template <int N>
__device__ __forceinline__ DensBounds dens_bounds(const GenDev& g, int ox, int oy, int oz, float h,
                                                  float hy) {
  constexpr int kLim = (1 << 24) - 256;
  const bool exact = ox > -kLim && ox < kLim && oy > -kLim && oy < kLim && oz > -kLim && oz < kLim;
  const float cm = (float)(max(max(abs(ox), abs(oy)), abs(oz)) + N + 1);
  float A = 0.0f, S = 0.0f, err = 0.0f, f = g.freq, amp = 1.0f;
  for (int o = 0; o < g.octaves; ++o) {
    const float a = fabsf(amp);
    A = A + a;
    S = S + a * (f * f);
    err = err + a * (2e-6f * (cm * fabsf(f)) + 4e-5f);
    f = f * g.lac;
    amp = amp * g.gain;
  }
  const float t0 = ((float)(oy - 1) - g.y_ref) * g.y_scale;
  const float t1 = ((float)(oy + N) - g.y_ref) * g.y_scale;
  err = err + 4e-6f * (A + fmaxf(fabsf(t0), fabsf(t1)));
  const float b = 1.037f * A + err;
  DensBounds r;
  r.known = -1;
  if (exact && t0 > b && t1 > b) r.known = g.solid_below_zero ? 1 : 0;    // every d < 0
  if (exact && t0 < -b && t1 < -b) r.known = g.solid_below_zero ? 0 : 1;  // every d > 0
  const float slack = 1.625f * (2.0f * h * h + hy * hy) * S + 2.0f * err;
  r.slack = exact && slack < A ? slack : __int_as_float(0x7f800000);
  return r;
}

// Evaluation of the samples of one row word along x (lane = x; for N < 32 the lanes past N
// hold further y rows) at kDensB consecutive z from zs: lane i of the first kDensB gets the
// ballot of z = zs + i. Octave by octave, with the fBm sums in registers. Within an octave
// the lattice cell along z changes rarely (every 1 / frequency voxels), so the four
// corner-pair records the lane's samples read — columns x0 and x0 + 1 at y0 and y0 + 1, each
// the gradients of corners z and z + 1 — stay in registers until it does, as the sums
// g.x * x + g.y * y, which do not depend on z, and g.z. The two corners of a record are
// evaluated together as f32x2 pairs: a gradient dot product is then one multiply and one
// add per pair, the four x lerps two pairs, the two y lerps one, then the z lerp of the
// pair's halves. Every value is the result of the operations of dens_value_tab, in the same
// order. z is the inner axis because the dot product ends with g.z * z: with x or y inside,
// each pair costs a second addition (49 instead of 39 FP32 lane operations a sample and
// octave).
constexpr int kDensB = 8;
template <int N, int LAYOUT>
__device__ __forceinline__ uint32_t dens_block_z(const ChunkSmem<N, LAYOUT>& s, const GenDev& g, int oy,
                                                 int x, int y, int zs) {
  using P = DensPlan<N>;
  const int* hdr = reinterpret_cast<const int*>(s.stage);
  const ulonglong2* axes = reinterpret_cast<const ulonglong2*>(s.stage + P::kAxes);
  const ulonglong2* pair_xy = reinterpret_cast<const ulonglong2*>(s.stage + P::kPairXY);
  const f2_t* pair_z = reinterpret_cast<const f2_t*>(s.stage + P::kPairZ);
  const f2_t nz = f2_pack(g.neg_zero, g.neg_zero);
  float sum[kDensB];
#pragma unroll
  for (int i = 0; i < kDensB; ++i) sum[i] = 0.0f;
  float amp = 1.0f;
#pragma unroll 1
  for (int o = 0; o < g.octaves; ++o) {
    const DensAxis ax = reinterpret_cast<const DensAxis*>(axes)[o * 3 * (N + 2) + x + 1];
    const DensAxis ay = reinterpret_cast<const DensAxis*>(axes)[o * 3 * (N + 2) + (N + 2) + y + 1];
    const ulonglong2* za = axes + o * 3 * (N + 2) + 2 * (N + 2) + zs + 1;
    const int n1 = hdr[4 * o + 1], n2 = hdr[4 * o + 2];
    const int r00 = hdr[4 * o] + (ax.ci * n1 + ay.ci) * n2, r10 = r00 + n1 * n2;
    const f2_t uu = f2_pack(ax.fade, ax.fade), vv = f2_pack(ay.fade, ay.fade);
    int cur = -1;                             // cell of the records held (cells are >= 0)
    f2_t q00 = 0, q10 = 0, q01 = 0, q11 = 0;  // {gx * x + gy * y} of columns (x0|x1, y0|y1)
    f2_t z00 = 0, z10 = 0, z01 = 0, z11 = 0;  // {gz}
#pragma unroll
    for (int i = 0; i < kDensB; ++i) {
      const ulonglong2 zr = za[i];  // {zf, zf - 1}, {fade, cell}: the same in every lane
      const int ci = (int)(unsigned)(zr.y >> 32);
      if (ci != cur) {
        cur = ci;
        const f2_t xa = f2_pack(ax.fr, ax.fr), xb = f2_pack(ax.fr1, ax.fr1);
        const f2_t ya = f2_pack(ay.fr, ay.fr), yb = f2_pack(ay.fr1, ay.fr1);
        const ulonglong2 g00 = pair_xy[r00 + ci], g10 = pair_xy[r10 + ci];
        const ulonglong2 g01 = pair_xy[r00 + n2 + ci], g11 = pair_xy[r10 + n2 + ci];
        q00 = f2_add(f2_mul(g00.x, xa), f2_mul(g00.y, ya));
        q10 = f2_add(f2_mul(g10.x, xb), f2_mul(g10.y, ya));
        q01 = f2_add(f2_mul(g01.x, xa), f2_mul(g01.y, yb));
        q11 = f2_add(f2_mul(g11.x, xb), f2_mul(g11.y, yb));
        z00 = pair_z[r00 + ci], z10 = pair_z[r10 + ci];
        z01 = pair_z[r00 + n2 + ci], z11 = pair_z[r10 + n2 + ci];
      }
      // (g.x * x + g.y * y) + g.z * z of corners (x_, y_, z) and (x_, y_, z + 1)
      const f2_t d00 = f2_add(q00, f2_mul(z00, zr.x));
      const f2_t d10 = f2_add(q10, f2_mul(z10, zr.x));
      const f2_t d01 = f2_add(q01, f2_mul(z01, zr.x));
      const f2_t d11 = f2_add(q11, f2_mul(z11, zr.x));
      const f2_t l0 = f2_lerp(uu, d00, d10, nz);  // {l00, l01}
      const f2_t l1 = f2_lerp(uu, d01, d11, nz);  // {l10, l11}
      float m0, m1;
      f2_unpack(f2_lerp(vv, l0, l1, nz), m0, m1);
      sum[i] = sum[i] + amp * d_lerp(__uint_as_float((unsigned)zr.y), m0, m1);
    }
    amp = amp * g.gain;
  }
  const float ty = ((float)(oy + y) - g.y_ref) * g.y_scale;
  const int lane = threadIdx.x & 31;
  uint32_t keep = 0u;
#pragma unroll
  for (int i = 0; i < kDensB; ++i) {
    const float d = sum[i] - ty;
    const uint32_t b = __ballot_sync(0xffffffffu, g.solid_below_zero ? (d < 0.0f) : (d > 0.0f));
    if (lane == i) keep = b;
  }
  return keep;
}

// The same with kDensY samples along y, for the lateral halo planes (lane: a position along the
// plane, x or z; the other coordinate fixed): lane i of the first kDensY gets the ballot of
// y = ys + i. The records are held with g.x * x and g.z * z.
constexpr int kDensY = 4;
template <int N, int LAYOUT>
__device__ __forceinline__ uint32_t dens_block_y(const ChunkSmem<N, LAYOUT>& s, const GenDev& g, int oy,
                                                 int x, int ys, int z) {
  using P = DensPlan<N>;
  const int* hdr = reinterpret_cast<const int*>(s.stage);
  const DensAxis* axes = reinterpret_cast<const DensAxis*>(s.stage + P::kAxes);
  const ulonglong2* pair_xy = reinterpret_cast<const ulonglong2*>(s.stage + P::kPairXY);
  const f2_t* pair_z = reinterpret_cast<const f2_t*>(s.stage + P::kPairZ);
  const f2_t nz = f2_pack(g.neg_zero, g.neg_zero);
  float sum[kDensY];
#pragma unroll
  for (int i = 0; i < kDensY; ++i) sum[i] = 0.0f;
  float amp = 1.0f;
#pragma unroll 1
  for (int o = 0; o < g.octaves; ++o) {
    const DensAxis ax = axes[o * 3 * (N + 2) + x + 1];
    const DensAxis az = axes[o * 3 * (N + 2) + 2 * (N + 2) + z + 1];
    const DensAxis* ya = axes + o * 3 * (N + 2) + (N + 2) + ys + 1;
    const int n1 = hdr[4 * o + 1], n2 = hdr[4 * o + 2];
    const int c0 = hdr[4 * o] + ax.ci * n1 * n2 + az.ci, c1 = c0 + n1 * n2;
    const f2_t uu = f2_pack(ax.fade, ax.fade), zz = f2_pack(az.fr, az.fr1);
    int cur = -1;
    f2_t gy00 = 0, gy10 = 0, gy01 = 0, gy11 = 0;  // {gy} of columns (x0|x1, y0|y1)
    f2_t px00 = 0, px10 = 0, px01 = 0, px11 = 0;  // {gx * x}
    f2_t pz00 = 0, pz10 = 0, pz01 = 0, pz11 = 0;  // {gz * zf, gz' * (zf - 1)}
#pragma unroll
    for (int i = 0; i < kDensY; ++i) {
      const DensAxis ay = ya[i];  // the same in every lane
      if (ay.ci != cur) {
        cur = ay.ci;
        const f2_t xa = f2_pack(ax.fr, ax.fr), xb = f2_pack(ax.fr1, ax.fr1);
        const int r0 = cur * n2, r1 = r0 + n2;
        const ulonglong2 g00 = pair_xy[c0 + r0], g10 = pair_xy[c1 + r0];
        const ulonglong2 g01 = pair_xy[c0 + r1], g11 = pair_xy[c1 + r1];
        gy00 = g00.y, gy10 = g10.y, gy01 = g01.y, gy11 = g11.y;
        px00 = f2_mul(g00.x, xa), px10 = f2_mul(g10.x, xb);
        px01 = f2_mul(g01.x, xa), px11 = f2_mul(g11.x, xb);
        pz00 = f2_mul(pair_z[c0 + r0], zz), pz10 = f2_mul(pair_z[c1 + r0], zz);
        pz01 = f2_mul(pair_z[c0 + r1], zz), pz11 = f2_mul(pair_z[c1 + r1], zz);
      }
      const f2_t ya2 = f2_pack(ay.fr, ay.fr), yb2 = f2_pack(ay.fr1, ay.fr1);
      // (g.x * x + g.y * y) + g.z * z of corners (x_, y_, z) and (x_, y_, z + 1)
      const f2_t d00 = f2_add(f2_add(px00, f2_mul(gy00, ya2)), pz00);
      const f2_t d10 = f2_add(f2_add(px10, f2_mul(gy10, ya2)), pz10);
      const f2_t d01 = f2_add(f2_add(px01, f2_mul(gy01, yb2)), pz01);
      const f2_t d11 = f2_add(f2_add(px11, f2_mul(gy11, yb2)), pz11);
      const f2_t l0 = f2_lerp(uu, d00, d10, nz);  // {l00, l01}
      const f2_t l1 = f2_lerp(uu, d01, d11, nz);  // {l10, l11}
      float m0, m1;
      f2_unpack(f2_lerp(f2_pack(ay.fade, ay.fade), l0, l1, nz), m0, m1);
      sum[i] = sum[i] + amp * d_lerp(az.fade, m0, m1);
    }
    amp = amp * g.gain;
  }
  const int lane = threadIdx.x & 31;
  uint32_t keep = 0u;
#pragma unroll
  for (int i = 0; i < kDensY; ++i) {
    const float d = sum[i] - ((float)(oy + ys + i) - g.y_ref) * g.y_scale;
    const uint32_t b = __ballot_sync(0xffffffffu, g.solid_below_zero ? (d < 0.0f) : (d > 0.0f));
    if (lane == i) keep = b;
  }
  return keep;
}

// A density chunk and its halo planes, or false (without a barrier) when the configuration is
// beyond the lattice tables (the caller then evaluates sample by sample). Chunks whose bounds
// decide them (dens_bounds) cost neither tables nor noise. Else the density is sampled on a
// coarse grid, which decides most cells of 8 x 4 x 8 voxels (spacing 8 along x and z: points 0,
// 8, ..., N, with halos -1, 7, ..., N, so that the planes at -1 and N are inside too, one spacing
// of 9; along y the same with 4). The rest are evaluated, a warp taking one row word at 8
// consecutive z (dens_block_z), and the undecided parts of the lateral planes 4 rows at a time
// (dens_block_y). Work goes by rows, so cells flat in y leave less to evaluate: with cells of
// 8^3 a cave chunk at the surface evaluates 37 row words of 128, with 8 x 4 x 8 about 25.
// On the 4096-chunk 32^3 cave terrain (3 octaves at 1/96; 55 % of the chunks are decided by
// their bounds, about 9 % of all samples are evaluated) vox_generate went from 610 us, bound by
// the FP32 pipe with every sample evaluated and x as the inner axis, to 103 us; the fused
// launch with its halos from 916 to 285 us.
template <int N, int LAYOUT, int T>
__device__ bool gen_density(ChunkSmem<N, LAYOUT>& s, const GenDev& g, int ox, int oy, int oz,
                            unsigned halo_mask, bool with_halo) {
  using RowT = typename Shape<N>::RowT;
  using P = DensPlan<N>;
  constexpr int W = Shape<N>::W;
  constexpr int LX = N < 32 ? N : 32;       // lanes along a row word
  constexpr int kSub = 32 / LX;             // y rows a warp evaluates side by side
  constexpr uint32_t kWordFull = N >= 32 ? 0xFFFFFFFFu : ((1u << (N & 31)) - 1u);
  constexpr int C = P::kCells, CY = P::kCellsY;
  const int t = threadIdx.x;
  uint32_t* occw = reinterpret_cast<uint32_t*>(s.occ);
  uint32_t* halow = reinterpret_cast<uint32_t*>(s.halo);
  const DensBounds bd = dens_bounds<N>(g, ox, oy, oz, with_halo ? 9.0f : 8.0f, with_halo ? 5.0f : 4.0f);
  if (bd.known >= 0) {
    const RowT v = bd.known ? full_row<N>() : (RowT)0;
    for (int i = t; i < N * N; i += T) s.occ[i] = v;
    if (with_halo)
      for (int i = t; i < 6 * N; i += T) s.halo[i] = ((halo_mask >> (i / N)) & 1u) ? v : (RowT)0;
    __syncthreads();
    return true;
  }
  if (!dens_tables<N, LAYOUT, T>(s, g, ox, oy, oz)) return false;
  float* coarse = reinterpret_cast<float*>(s.stage + P::kCoarse);
  uint32_t* known = reinterpret_cast<uint32_t*>(s.stage + P::kKnown);
  uint32_t* mixed = reinterpret_cast<uint32_t*>(s.stage + P::kMixed);
  int* list = reinterpret_cast<int*>(s.stage + P::kList);
  const bool use_coarse = bd.slack < 3.0e38f;
  if (t == 0) list[0] = 0;
  if (use_coarse) {
    constexpr int Q = P::kPts, QY = P::kPtsY;
    for (int i = t; i < QY * Q * Q; i += T) {
      const int px = i % Q, pz = (i / Q) % Q, py = i / (Q * Q);
      auto at = [&](int p) { return with_halo ? (p == C ? N : 8 * p - 1) : 8 * p; };
      const int y = with_halo ? (py == CY ? N : 4 * py - 1) : 4 * py;
      coarse[i] = dens_value_tab<N, LAYOUT>(s, g, at(px), y, at(pz), oy);
    }
  }
  __syncthreads();
  // row words over the (y, z) cells: word index ((cy * C) + cz) * kSegs + seg
  for (int i = t; i < P::kWords; i += T) {
    uint32_t k = 0u, m = 0u;
    if (use_coarse) {
      constexpr int Q = P::kPts;
      const int seg = i % P::kSegs, cz = (i / P::kSegs) % C, cy = i / (P::kSegs * C);
      const float* p00 = coarse + (cy * Q + cz) * Q + seg * 4;
      const float* p10 = p00 + Q * Q;
      constexpr int kX = C < 4 ? C : 4;  // cells along x in one row word
      float mn = 0.0f, mx = 0.0f;        // over the four samples at x point j
#pragma unroll
      for (int j = 0; j <= kX; ++j) {
        const float a = p00[j], b = p00[Q + j], c = p10[j], d = p10[Q + j];
        const float n2 = fminf(fminf(a, b), fminf(c, d)), x2 = fmaxf(fmaxf(a, b), fmaxf(c, d));
        if (j > 0) {
          const bool pos = fminf(mn, n2) > bd.slack, neg = fmaxf(mx, x2) < -bd.slack;
          if (g.solid_below_zero ? neg : pos) k |= 0xFFu << (8 * (j - 1));
          else if (!pos && !neg) m |= 0xFFu << (8 * (j - 1));
        }
        mn = n2;
        mx = x2;
      }
    } else {
      m = kWordFull;
    }
    known[i] = k;
    mixed[i] = m;
    if (m != 0u) list[1 + atomicAdd(list, 1)] = i;
  }
  __syncthreads();
  // decided cell rows: their words at every voxel row
  for (int i = t; i < N * N * W; i += T) {
    const int seg = i % W, z = (i / W) % N, y = i / (W * N);
    const int c = ((y >> 2) * C + (z >> 3)) * P::kSegs + seg;
    if (mixed[c] == 0u) occw[i] = known[c];
  }
  // Work items of a warp: the undecided row words (kSub rows y, 8 z each), then the lateral
  // halo planes (kPl planes side by side, 4 rows y), then the -y and +y planes (8 rows z).
  constexpr int kPl = kSub < 2 ? 1 : 2;
  constexpr int kPerCell = 4 / kSub;
  const int own = list[0] * kPerCell;
  const int lateral = with_halo ? (4 / kPl) * CY * P::kSegs : 0;
  const int vertical = with_halo ? 2 * C * P::kSegs : 0;
  const int lane = t & 31, lx = lane % LX, sub = lane / LX;
  for (int it = t >> 5; it < own + lateral + vertical; it += T / 32) {
    if (it < own) {
      const int c = list[1 + it / kPerCell];
      const int seg = c % P::kSegs, cz = (c / P::kSegs) % C, cy = c / (P::kSegs * C);
      const int y = cy * 4 + (it % kPerCell) * kSub, zs = cz * 8;
      const uint32_t b = dens_block_z<N, LAYOUT>(s, g, oy, seg * 32 + lx, y + sub, zs);
      if (lane < kDensB) {
#pragma unroll
        for (int q = 0; q < kSub; ++q)
          occw[((y + q) * N + zs + lane) * W + seg] = (b >> ((q * LX) & 31)) & kWordFull;
      }
    } else if (it < own + lateral) {
      const int k = it - own;
      const int seg = k % P::kSegs, cy = (k / P::kSegs) % CY, h0 = (k / (P::kSegs * CY)) * kPl;
      const int pl = sub < kPl ? sub : kPl - 1;  // 8^3 chunks: the lanes past two planes repeat
      const int h = h0 + pl, ys = cy * 4;
      // decided bits and undecided bits of this lane's plane word (a decided cell is one byte)
      uint32_t kn = 0u, mi = 0u;
      if (h >= 2) {  // z planes: words along x of the first or last cell row
        const int c = (cy * C + (h == 2 ? 0 : C - 1)) * P::kSegs + seg;
        kn = known[c];
        mi = mixed[c];
      } else {       // x planes: the first or last cell of the words along z
        const int w = h == 0 ? 0 : P::kSegs - 1, sh = h == 0 ? 0 : 8 * ((C - 1) & 3);
#pragma unroll
        for (int j = 0; j < (C < 4 ? C : 4); ++j) {
          const int c = (cy * C + seg * 4 + j) * P::kSegs + w;
          kn |= ((known[c] >> sh) & 0xFFu) << (8 * j);
          mi |= ((mixed[c] >> sh) & 0xFFu) << (8 * j);
        }
      }
      const bool used = (halo_mask >> h) & 1u;
      uint32_t b;
      if (__any_sync(0xffffffffu, used && mi != 0u)) {
        const int p = seg * 32 + lx;
        b = dens_block_y<N, LAYOUT>(s, g, oy, h == 0 ? -1 : (h == 1 ? N : p), ys,
                                    h == 2 ? -1 : (h == 3 ? N : p));
      } else {
        b = 0u;
#pragma unroll
        for (int q = 0; q < kPl; ++q)
          b |= (__shfl_sync(0xffffffffu, kn, q * LX) & kWordFull) << ((q * LX) & 31);
      }
      if (lane < kDensY) {
#pragma unroll
        for (int q = 0; q < kPl; ++q)
          halow[((h0 + q) * N + ys + lane) * W + seg] =
              ((halo_mask >> (h0 + q)) & 1u) ? (b >> ((q * LX) & 31)) & kWordFull : 0u;
      }
    } else {
      const int k = it - own - lateral;
      const int seg = k % P::kSegs, cz = (k / P::kSegs) % C, h = 4 + k / (P::kSegs * C);
      const int c = ((h == 4 ? 0 : CY - 1) * C + cz) * P::kSegs + seg;
      const bool used = (halo_mask >> h) & 1u;
      uint32_t b = used ? known[c] : 0u;
      if (used && mixed[c] != 0u)
        b = dens_block_z<N, LAYOUT>(s, g, oy, seg * 32 + lx, h == 4 ? -1 : N, cz * 8) & kWordFull;
      if (lane < kDensB) halow[(h * N + cz * 8 + lane) * W + seg] = b;
    }
  }
  __syncthreads();
  return true;
}

// Fills s.occ (own rows) and, for every set bit of `halo_mask`, the halo rows; the other
// halo rows are zero (a neighbour that is not loaded counts as air, chunk.rs:102-107).
// kHash: where heightmap columns get their lattice data (see column_k).
template <int N, int GM, int LAYOUT, int T, int kHash = kHashNone>
__device__ void gen_chunk(ChunkSmem<N, LAYOUT>& s, const GenDev& g, vox_chunk_coord c,
                          long long chunk_index, unsigned halo_mask, bool with_halo) {
  using RowT = typename Shape<N>::RowT;
  const int ox = c.x * N, oy = c.y * N, oz = c.z * N;
  if (GM == GM_HEIGHT) {
    gen_heightmap<N, LAYOUT, T, kHash>(s, g, ox, oy, oz, halo_mask, with_halo);
    return;
  }
  if (GM == GM_DENSITY) {
    if (gen_density<N, LAYOUT, T>(s, g, ox, oy, oz, halo_mask, with_halo)) return;
  }
  const unsigned long long s0 = g.seed ^ (unsigned long long)chunk_index;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  uint32_t* occw = reinterpret_cast<uint32_t*>(s.occ);
  for (int base = warp * 32; base < N * N * N; base += nwarps * 32) {
    const int e = base + lane;
    const int row = e / N, x = e % N;
    const int y = row / N, z = row % N;
    store_ballot<N>(occw, e, gen_solid<N, GM, LAYOUT>(s, g, x, y, z, ox, oy, oz, s0));
  }
  if (with_halo) {
    uint32_t* halow = reinterpret_cast<uint32_t*>(s.halo);
    for (int h = 0; h < 6; ++h) {
      if ((halo_mask >> h) & 1u) {
        for (int base = warp * 32; base < N * N; base += nwarps * 32) {
          const int e = base + lane;
          int x, y, z;
          halo_coord<N>(h, e / N, e % N, x, y, z);
          store_ballot<N>(halow + h * N * Shape<N>::W, e,
                          gen_solid<N, GM, LAYOUT>(s, g, x, y, z, ox, oy, oz, s0));
        }
      } else {
        for (int i = threadIdx.x; i < N; i += blockDim.x) s.halo[h * N + i] = (RowT)0;
      }
    }
  }
  __syncthreads();
}

// Occupancy from global memory: own rows copied; halo rows taken from the neighbours'
// boundary planes (nbr[d] == nullptr: not loaded, zero halo). Every thread issues all its loads
// before it uses one, so the chunk costs one memory latency instead of one per plane. Plain loads:
// the launch that writes the occupancy may still run when this kernel starts (see vox_launch.h).
template <int N, int LAYOUT, int T>
__device__ __forceinline__ void load_chunk(ChunkSmem<N, LAYOUT>& s, const uint32_t* self,
                                           const uint32_t* const nbr[6], unsigned use_mask) {
  constexpr int W = Shape<N>::W;
  constexpr int kOwn = N * N * W / T, kPlane = N * N / T, kRow = N * W;
  static_assert(kPlane >= 1 && kPlane * T == N * N, "planes must split evenly over threads");
  constexpr int kMost = N > 32 ? 4 : kOwn;  // own words in flight (64^3: in turns)
  uint32_t* occw = reinterpret_cast<uint32_t*>(s.occ);
  uint32_t* halow = reinterpret_cast<uint32_t*>(s.halo);
  const int t = threadIdx.x;
  uint32_t own[kMost], px[2][kPlane], pr = 0u;
#pragma unroll
  for (int k = 0; k < kMost; ++k) own[k] = self[t + k * T];
  // x planes: bit (N - 1) (h = 0) or bit 0 (h = 1) of the neighbour's row (y, z)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t* nb = ((use_mask >> h) & 1u) ? nbr[h] : nullptr;
    constexpr int kLast = (N - 1) >> 5;
#pragma unroll
    for (int k = 0; k < kPlane; ++k)
      px[h][k] = nb ? nb[(t + k * T) * W + (h == 0 ? kLast : 0)] >> (h == 0 ? (N - 1) & 31 : 0) : 0u;
  }
  // whole rows: -z: (y, N-1); +z: (y, 0); -y: (N-1, z); +y: (0, z)
  auto row_word = [&](int i) {
    const int h = 2 + i / kRow, a = (i % kRow) / W, w = i % W;
    const uint32_t* nb = ((use_mask >> h) & 1u) ? nbr[h] : nullptr;
    const int r = h == 2 ? a * N + (N - 1) : (h == 3 ? a * N : (h == 4 ? (N - 1) * N + a : a));
    return nb ? nb[r * W + w] : 0u;
  };
  if (t < 4 * kRow) pr = row_word(t);
#pragma unroll
  for (int k = 0; k < kMost; ++k) occw[t + k * T] = own[k];
  for (int k = kMost; k < kOwn; k += kMost) {
#pragma unroll
    for (int j = 0; j < kMost; ++j) own[j] = self[t + (k + j) * T];
#pragma unroll
    for (int j = 0; j < kMost; ++j) occw[t + (k + j) * T] = own[j];
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int k = 0; k < kPlane; ++k)
      store_ballot<N>(halow + h * N * W, t + k * T, (px[h][k] & 1u) != 0u);
  if (t < 4 * kRow) halow[2 * kRow + t] = pr;
  for (int i = t + T; i < 4 * kRow; i += T) halow[2 * kRow + i] = row_word(i);
  __syncthreads();
}

// ------------------------------------------------------------------------------------
// Face masks, counts and emission
// ------------------------------------------------------------------------------------

template <int N, int LAYOUT>
__device__ __forceinline__ void row_masks(const ChunkSmem<N, LAYOUT>& s, int y, int z,
                                          typename Shape<N>::RowT m[6]) {
  using RowT = typename Shape<N>::RowT;
  const RowT row = s.occ[y * N + z];
  const RowT lb = (s.halo[0 * N + y] >> z) & (RowT)1;
  const RowT rb = (s.halo[1 * N + y] >> z) & (RowT)1;
  const RowT ln = (row << 1) | lb;
  const RowT rn = (row >> 1) | (rb << (N - 1));
  const RowT bn = z > 0 ? s.occ[y * N + z - 1] : s.halo[2 * N + y];
  const RowT fn = z < N - 1 ? s.occ[y * N + z + 1] : s.halo[3 * N + y];
  const RowT dn = y > 0 ? s.occ[(y - 1) * N + z] : s.halo[4 * N + z];
  const RowT un = y < N - 1 ? s.occ[(y + 1) * N + z] : s.halo[5 * N + z];
  m[0] = row & ~ln;
  m[1] = row & ~rn;
  m[2] = row & ~bn;
  m[3] = row & ~fn;
  m[4] = row & ~dn;
  m[5] = row & ~un;
}

// Per-row face counts -> exclusive offsets in s.rows[0..R], the face voxels in emission order
// in s.vlist when they fit (count in s.misc[1], else -1) and, for sizes whose voxels may not
// fit, the ascending list of the rows with faces in s.nz (count in s.misc[0], else 0); returns
// the chunk's face total.
template <int N, int LAYOUT, int T>
__device__ uint32_t count_and_scan(ChunkSmem<N, LAYOUT>& s) {
  using RowT = typename Shape<N>::RowT;
  constexpr int RPT = Shape<N>::R / T;
  constexpr int VCap = Shape<N>::VCap;
  static_assert(RPT >= 1 && RPT * T == Shape<N>::R, "rows must split evenly over threads");
  // One packed sum per thread. Where every voxel fits the list (up to 16^3) the rows are not
  // listed, and faces (at most 3 N^3 + 6 N^2, below 2^14) and face voxels (at most 2^12) fit 32
  // bits; else 64 bits hold faces, face voxels and rows with faces, 20 bits each.
  constexpr bool kSmall = VCap >= N * N * N;
  using SumT = typename std::conditional<kSmall, uint32_t, unsigned long long>::type;
  constexpr int kFaceShift = kSmall ? 16 : 40, kVoxShift = kSmall ? 0 : 20;
  constexpr uint32_t kMask = kSmall ? 0xFFFFu : 0xFFFFFu;
  const int t = threadIdx.x;
  uint32_t cnt[RPT];
  RowT any[RPT];
  uint32_t local = 0, vl = 0, nzl = 0;
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int r = t * RPT + k;
    uint32_t c = 0;
    any[k] = (RowT)0;
    if (s.occ[r] != (RowT)0) {
      RowT m[6];
      row_masks<N, LAYOUT>(s, r / N, r % N, m);
#pragma unroll
      for (int d = 0; d < 6; ++d) c += (uint32_t)popc_row(m[d]);
      any[k] = VCap > 0 ? (m[0] | m[1] | m[2] | m[3] | m[4] | m[5]) : (RowT)0;
    }
    cnt[k] = c;
    local += c;
    if (VCap > 0) vl += (uint32_t)popc_row(any[k]);
    nzl += c != 0u ? 1u : 0u;
  }
  // Deterministic block scan: warp inclusive scan, then a scan of the warp totals.
  const int lane = t & 31, warp = t >> 5, nwarps = T >> 5;
  const SumT mine = ((SumT)local << kFaceShift) | ((SumT)vl << kVoxShift) | (kSmall ? (SumT)0 : (SumT)nzl);
  SumT incl = mine;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const SumT v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  SumT* wsum = reinterpret_cast<SumT*>(s.stage);  // staging is free
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  // every warp scans the warp totals itself (no second barrier)
  SumT before = 0, tot = 0;
  {
    const SumT v = lane < nwarps ? wsum[lane] : (SumT)0;
    SumT vi = v;
#pragma unroll
    for (int off = 1; off < T / 32; off <<= 1) {
      const SumT u = __shfl_up_sync(0xffffffffu, vi, off);
      if (lane >= off) vi += u;
    }
    before = __shfl_sync(0xffffffffu, vi - v, warp);  // exclusive offset of this warp
    tot = __shfl_sync(0xffffffffu, vi, nwarps - 1);   // chunk totals
  }
  const SumT excl = before + incl - mine;
  const uint32_t nvox = (uint32_t)(tot >> kVoxShift) & kMask;
  const bool use_list = VCap > 0 && nvox <= (uint32_t)VCap;
  uint32_t run = (uint32_t)(excl >> kFaceShift);
  uint32_t vrun = (uint32_t)(excl >> kVoxShift) & kMask;
  uint32_t nzrun = (uint32_t)excl & kMask;
#pragma unroll
  for (int k = 0; k < RPT; ++k) {
    const int r = t * RPT + k;
    s.rows[r] = run;
    if (!kSmall && cnt[k] != 0u) s.nz[nzrun++] = (uint16_t)r;
    if (VCap > 0 && use_list) {
      RowT u = any[k];
      if (u == full_row<N>()) {  // a face of every voxel: most rows of the chunk's borders
#pragma unroll
        for (int x = 0; x < N; ++x) s.vlist[vrun + x] = (uint16_t)((r << Shape<N>::LOG2N) | x);
        vrun += N;
        u = (RowT)0;
      }
      while (u) {
        const int x = __ffs((uint32_t)u) - 1;
        u &= u - (RowT)1;
        s.vlist[vrun++] = (uint16_t)((r << Shape<N>::LOG2N) | x);
      }
    }
    run += cnt[k];
  }
  const uint32_t total = (uint32_t)(tot >> kFaceShift);
  if (t == 0) {
    s.rows[Shape<N>::R] = total;
    s.misc[0] = kSmall ? 0 : (int)(tot & kMask);
    s.misc[1] = use_list ? (int)nvox : -1;
  }
  __syncthreads();
  return total;
}

// Decoupled look-back (one warp): the sum of the published values of states 0 .. i - 1. Each
// poll reads a window of 128 predecessors (4 per lane, coalesced), walks back to the nearest
// inclusive prefix and sums the aggregates in between. Every wait is bounded (spin_limit
// polls); on timeout the error bit is set and what was summed so far is returned.
constexpr int kLookbackWindow = 128;
static __device__ unsigned long long lookback_sum(unsigned long long* state, BatchCtl* ctl,
                                                  unsigned epoch, int i, int spin_limit) {
  const int lane = threadIdx.x & 31;
  unsigned long long excl = 0;
  if (i == 0) return 0;
  const unsigned tag = epoch & 0xFFFFFFu;
  const unsigned long long vmask = (1ull << 38) - 1;
  int j = i - 1;
  int spins = 0;
  while (true) {
    // window position p = 32k + lane <-> chunk j - p (p = 0 is the nearest predecessor)
    unsigned long long sv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int idx = j - (32 * k + lane);
      sv[k] = idx >= 0 ? ld_relaxed_u64(&state[idx]) : pack_state(epoch, kFlagIncl, 0);
    }
    int first_incl = kLookbackWindow;
    unsigned bad[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const unsigned e = (unsigned)(sv[k] >> 40) & 0xFFFFFFu;
      const unsigned long long flag = (sv[k] >> 38) & 3ull;
      const bool valid = e == tag && flag != 0ull;
      const unsigned incl = __ballot_sync(0xffffffffu, valid && flag == kFlagIncl);
      bad[k] = __ballot_sync(0xffffffffu, !valid);
      if (first_incl == kLookbackWindow && incl) first_incl = 32 * k + __ffs(incl) - 1;
    }
    // every position up to and including first_incl must be published
    bool wait = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int hi = first_incl - 32 * k;  // positions 0..hi of this row are needed
      if (hi < 0) continue;
      const unsigned need = hi >= 31 ? 0xffffffffu : ((2u << hi) - 1u);
      if (bad[k] & need) wait = true;
    }
    if (wait) {
      if (++spins > spin_limit) {
        if (lane == 0) atomicOr(&ctl->err, ERR_TIMEOUT);
        break;
      }
      __nanosleep(spins < 8 ? 20 : 200);
      continue;
    }
    unsigned long long v = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (32 * k + lane <= first_incl) v += sv[k] & vmask;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    excl += v;
    if (first_incl < kLookbackWindow) break;
    j -= kLookbackWindow;
  }
  return excl;
}

// Look-back over chunks (warp 0 of the CTA): the exclusive prefix of chunk i, whose inclusive
// prefix is published. publish_agg = false: chunk i's aggregate is already published (overlap
// schedule).
static __device__ unsigned long long lookback(unsigned long long* state, BatchCtl* ctl,
                                              unsigned epoch, int i, unsigned long long total,
                                              int spin_limit, bool publish_agg = true) {
  const int lane = threadIdx.x & 31;
  if (lane == 0 && publish_agg && i > 0) st_relaxed_u64(&state[i], pack_state(epoch, kFlagAgg, total));
  const unsigned long long excl = lookback_sum(state, ctl, epoch, i, spin_limit);
  if (lane == 0) st_relaxed_u64(&state[i], pack_state(epoch, kFlagIncl, excl + total));
  return excl;
}

// Pulls the launch's per-chunk inputs (coordinates, neighbour masks) into L2 at the start,
// one 128-byte line per CTA and step of the grid, so that the chunks' first reads find them
// there instead of in DRAM.
__device__ __forceinline__ void prefetch_inputs(const MeshArgs& a) {
  const unsigned long long cbytes = 12ull * (unsigned long long)a.n;
  const unsigned long long mbytes = a.nbr_mask ? (unsigned long long)a.n : 0ull;
  const char* cp = reinterpret_cast<const char*>(a.coords);
  const char* mp = reinterpret_cast<const char*>(a.nbr_mask);
  for (unsigned long long off = 128ull * blockIdx.x; off < cbytes; off += 128ull * gridDim.x)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(cp + off));
  for (unsigned long long off = 128ull * blockIdx.x; off < mbytes; off += 128ull * gridDim.x)
    asm volatile("prefetch.global.L2 [%0];" ::"l"(mp + off));
}

// Global face index of the launch's first face (MeshArgs::base_ptr; one thread reads it).
__device__ __forceinline__ unsigned long long launch_base(const MeshArgs& a) {
  return a.base_ptr ? *reinterpret_cast<const volatile unsigned long long*>(a.base_ptr) : 0ull;
}

// Status mirror of a launch whose caller waits for it (outputs in host memory): the last
// CTA to finish copies the error word, with kMirrorValid set, into a page-locked host word,
// so that the host reads the status after the stream sync without a device-to-host copy.
// Every earlier launch on the stream has completed, so the word holds their bits too.
__device__ __forceinline__ void finish_launch(const MeshArgs& a) {
  if (a.err_mirror == nullptr) return;
  __syncthreads();  // this CTA's error bits are set
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.ctl->done, 1u) == gridDim.x - 1u) {
      __threadfence();
      const unsigned e = atomicOr(&a.ctl->err, 0u);
      a.ctl->done = 0u;
      *reinterpret_cast<volatile unsigned*>(a.err_mirror) = e | kMirrorValid;
    }
  }
}

// Staging-buffer placement of window records. The index records (vertex layout) and the
// instance records are shifted so that the bulk-copied part starts on a 16-byte boundary
// in shared and in global memory (global face g0 + l0 with (g0 + l0) even, resp. a
// multiple of 4).
template <int LAYOUT>
__device__ __forceinline__ int stage_shift(unsigned long long g) {
  if (LAYOUT == VOX_LAYOUT_INSTANCED) {
    const int l0 = (int)((4u - (unsigned)(g & 3ull)) & 3u);
    return (16 - 4 * l0) & 15;
  }
  return (g & 1ull) ? 8 : 0;
}

// Writes face l of the staging window (chunk-local index f_local) for voxel (x, y, z).
template <int LAYOUT>
__device__ __forceinline__ void stage_face(unsigned char* stage, int stage_faces, int shift, int l,
                                           int dir, float tx, float ty, float tz, uint32_t f_local,
                                           const TablesDev* tab) {
  if (LAYOUT == VOX_LAYOUT_INSTANCED) {
    uint32_t* o = reinterpret_cast<uint32_t*>(stage + shift + (size_t)l * 68);
    const float z0 = tx * 0.0f, z1 = ty * 0.0f, z2 = tz * 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      o[4 * c + 0] = __float_as_uint(tab->part[dir][0][c] + z0);
      o[4 * c + 1] = __float_as_uint(tab->part[dir][1][c] + z1);
      o[4 * c + 2] = __float_as_uint(tab->part[dir][2][c] + z2);
      o[4 * c + 3] = __float_as_uint(tab->row3[dir][c]);
    }
    o[12] = __float_as_uint(tx);
    o[13] = __float_as_uint(ty);
    o[14] = __float_as_uint(tz);
    o[15] = __float_as_uint(1.0f);
    o[16] = tab->tex[dir];
  } else {
    float4* v = reinterpret_cast<float4*>(stage + (size_t)l * 96);
    // rotated corners of the direction, 12 floats = 3 float4 (v0xyz v1xyz v2xyz v3xyz)
    const float4* C = reinterpret_cast<const float4*>(tab->corner[dir]);
    const float4 c0 = C[0], c1 = C[1], c2 = C[2];
    const float face = __uint_as_float(tab->slot[dir]);
    // tex coords of quad::VERTICES (src/quad.rs:66-87): (0,0) (1,0) (0,1) (1,1)
    v[0] = make_float4(c0.x + tx, c0.y + ty, c0.z + tz, 0.0f);
    v[1] = make_float4(0.0f, face, c0.w + tx, c1.x + ty);
    v[2] = make_float4(c1.y + tz, 1.0f, 0.0f, face);
    v[3] = make_float4(c1.z + tx, c1.w + ty, c2.x + tz, 0.0f);
    v[4] = make_float4(1.0f, face, c2.y + tx, c2.z + ty);
    v[5] = make_float4(c2.w + tz, 1.0f, 1.0f, face);
    uint2* ix = reinterpret_cast<uint2*>(stage + (size_t)stage_faces * 96 + shift + (size_t)l * 24);
    const uint32_t b = 4u * f_local;
    ix[0] = make_uint2(b + 0u, b + 2u);
    ix[1] = make_uint2(b + 1u, b + 3u);
    ix[2] = make_uint2(b + 1u, b + 2u);
  }
}

// Sends `nw` faces staged in one warp buffer to the global output starting at face
// index g: lane 0 issues the TMA bulk copies of the 16-byte aligned part and commits them
// as one bulk group; the few unaligned head/tail records are stored word by word by the
// other lanes. Call after fence.proxy.async + __syncwarp.
template <int LAYOUT>
__device__ __forceinline__ void flush_warp(const unsigned char* buf, int shift, int nw,
                                           unsigned long long g, void* out0, void* out1) {
  const int lane = threadIdx.x & 31;
  unsigned char* o0 = reinterpret_cast<unsigned char*>(out0);
  if (LAYOUT == VOX_LAYOUT_INSTANCED) {
    int l0 = (int)((4u - (unsigned)(g & 3ull)) & 3u);
    if (l0 > nw) l0 = nw;
    const int l1 = l0 + ((nw - l0) & ~3);
    const unsigned char* src = buf + shift;
    if (lane == 0) {
      if (l1 > l0)
        bulk_s2g(o0 + (g + l0) * 68ull, src + (size_t)l0 * 68, (uint32_t)(l1 - l0) * 68u);
      bulk_commit();
    }
    // head faces [0, l0) and tail faces [l1, nw), 17 words each
    const int head = l0 * 17, tail = (nw - l1) * 17;
    for (int q = lane - 1; q >= 0 && q < head + tail; q += 31) {
      const int w = q < head ? q : (l1 * 17 + (q - head));
      reinterpret_cast<uint32_t*>(o0 + g * 68ull)[w] = reinterpret_cast<const uint32_t*>(src)[w];
    }
  } else {
    unsigned char* o1 = reinterpret_cast<unsigned char*>(out1);
    const int l0 = (int)(g & 1ull) < nw ? (int)(g & 1ull) : nw;
    const int l1 = l0 + ((nw - l0) & ~1);
    const unsigned char* isrc = buf + kWarpBatch * 96 + shift;
    if (lane == 0) {
      bulk_s2g(o0 + g * 96ull, buf, (uint32_t)nw * 96u);
      if (l1 > l0)
        bulk_s2g(o1 + (g + l0) * 24ull, isrc + (size_t)l0 * 24, (uint32_t)(l1 - l0) * 24u);
      bulk_commit();
    }
    const int head = l0 * 6, tail = (nw - l1) * 6;
    for (int q = lane - 1; q >= 0 && q < head + tail; q += 31) {
      const int w = q < head ? q : (l1 * 6 + (q - head));
      reinterpret_cast<uint32_t*>(o1 + g * 24ull)[w] = reinterpret_cast<const uint32_t*>(isrc)[w];
    }
  }
}

// flush_warp with plain stores instead of bulk copies: the lanes copy the 16-byte aligned
// part in 16-byte units (each warp store writes 512 contiguous bytes), then the head/tail
// words. For outputs in host memory, where full-line writes matter most.
template <int LAYOUT>
__device__ __forceinline__ void flush_warp_lanes(const unsigned char* buf, int shift, int nw,
                                                 unsigned long long g, void* out0, void* out1) {
  const int lane = threadIdx.x & 31;
  unsigned char* o0 = reinterpret_cast<unsigned char*>(out0);
  if (LAYOUT == VOX_LAYOUT_INSTANCED) {
    int l0 = (int)((4u - (unsigned)(g & 3ull)) & 3u);
    if (l0 > nw) l0 = nw;
    const int l1 = l0 + ((nw - l0) & ~3);
    const unsigned char* src = buf + shift;
    const uint4* s16 = reinterpret_cast<const uint4*>(src + (size_t)l0 * 68);
    uint4* d16 = reinterpret_cast<uint4*>(o0 + (g + l0) * 68ull);
    for (int q = lane; q < (l1 - l0) * 68 / 16; q += 32) d16[q] = s16[q];
    const int head = l0 * 17, tail = (nw - l1) * 17;
    for (int q = lane; q < head + tail; q += 32) {
      const int w = q < head ? q : (l1 * 17 + (q - head));
      reinterpret_cast<uint32_t*>(o0 + g * 68ull)[w] = reinterpret_cast<const uint32_t*>(src)[w];
    }
  } else {
    unsigned char* o1 = reinterpret_cast<unsigned char*>(out1);
    const int l0 = (int)(g & 1ull) < nw ? (int)(g & 1ull) : nw;
    const int l1 = l0 + ((nw - l0) & ~1);
    const unsigned char* isrc = buf + kWarpBatch * 96 + shift;
    const uint4* v16 = reinterpret_cast<const uint4*>(buf);
    uint4* dv = reinterpret_cast<uint4*>(o0 + g * 96ull);
    for (int q = lane; q < nw * 6; q += 32) dv[q] = v16[q];
    const uint4* i16 = reinterpret_cast<const uint4*>(isrc + (size_t)l0 * 24);
    uint4* di = reinterpret_cast<uint4*>(o1 + (g + l0) * 24ull);
    for (int q = lane; q < (l1 - l0) * 24 / 16; q += 32) di[q] = i16[q];
    const int head = l0 * 6, tail = (nw - l1) * 6;
    for (int q = lane; q < head + tail; q += 32) {
      const int w = q < head ? q : (l1 * 6 + (q - head));
      reinterpret_cast<uint32_t*>(o1 + g * 24ull)[w] = reinterpret_cast<const uint32_t*>(isrc)[w];
    }
  }
}

// A face of a face list: local voxel (x, y, z) and emission direction, a byte each.
__device__ __forceinline__ uint32_t pack_face(int x, int y, int z, int d) {
  return (uint32_t)x | ((uint32_t)y << 8) | ((uint32_t)z << 16) | ((uint32_t)d << 24);
}

// Face compaction of one warp: lane l owns element base + l of the chunk's emission
// elements, the face voxels of s.vlist (use_list) or else every voxel of the rows with
// faces (rows nz[], N voxels each); either way the warp's voxels are consecutive in
// emission order. Each lane lists its voxel's faces in direction order; returns the warp's
// face count and, in `first`, the chunk-relative index of the warp's first face. Face i of
// the warp (index first + i) goes to list[i], or with kAbsolute to list[first + i].
template <int N, bool kAbsolute = false, int LAYOUT>
__device__ __forceinline__ int warp_faces(const ChunkSmem<N, LAYOUT>& s, bool use_list,
                                          int elems, int base, uint32_t* list, uint32_t& first) {
  using RowT = typename Shape<N>::RowT;
  const int lane = threadIdx.x & 31;
  const int e = base + lane;
  unsigned bits = 0;
  uint32_t mine = 0;
  int x = 0, y = 0, z = 0;
  if (e < elems) {
    int r;
    if (Shape<N>::VCap > 0 && use_list) {
      const uint32_t q = s.vlist[e];
      x = (int)(q & (uint32_t)(N - 1));
      r = (int)(q >> Shape<N>::LOG2N);
    } else {
      r = s.nz[e / N];
      x = e % N;
    }
    y = r / N;
    z = r % N;
    RowT m[6];
    row_masks<N, LAYOUT>(s, y, z, m);
#pragma unroll
    for (int d = 0; d < 6; ++d) bits |= (unsigned)((m[d] >> x) & (RowT)1) << d;
    // Only lane 0's position is needed (the warp scan places the others): the row's face
    // offset plus the faces of the voxels before x in the row.
    uint32_t pre = 0;
    if (lane == 0 && x != 0) {
      const RowT below = (RowT)(~(RowT)0) >> (sizeof(RowT) * 8 - x);
#pragma unroll
      for (int d = 0; d < 6; ++d) pre += (uint32_t)popc_row(m[d] & below);
    }
    mine = s.rows[r] + pre;
  }
  const int cnt = __popc(bits);
  int incl = cnt;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  first = __shfl_sync(0xffffffffu, mine, 0);  // lane 0's voxel starts the warp's range
  uint32_t* out = list + (incl - cnt) + (kAbsolute ? (int)first : 0);
  const uint32_t code = pack_face(x, y, z, 0);
  while (bits) {
    const int d = __ffs(bits) - 1;
    bits &= bits - 1u;
    *out++ = code | ((uint32_t)d << 24);
  }
  __syncwarp();
  return total;
}

// Emission elements of the chunk in shared memory: listed face voxels, or every voxel of
// the rows with faces.
template <int N, int LAYOUT>
__device__ __forceinline__ int emit_elems(const ChunkSmem<N, LAYOUT>& s) {
  return s.misc[1] >= 0 ? s.misc[1] : s.misc[0] * N;
}

// Emits the faces of the chunk in reference order: chunk-local face f goes to global
// face g0 + f. Every warp compacts the faces of its 32 voxels, stages them 32 at a time
// in one of its two shared-memory buffers (one face record per lane, final byte layout)
// and sends each batch to global memory with a TMA bulk copy issued by its lane 0. A
// warp has nbuf (1 or 2) such buffers. No CTA-wide barrier: a warp waits only until the
// bulk copy that last read a buffer is done before refilling it, and until all its
// copies have read shared memory at the end (the staging area is reused by the next
// chunk's generation).
// Faces per whole number of 128-byte output lines: 16 for the 96-byte vertex and 24-byte
// index records, 32 for the 68-byte instance records.
template <int LAYOUT>
__host__ __device__ constexpr unsigned line_faces() { return LAYOUT == VOX_LAYOUT_INSTANCED ? 32u : 16u; }

// Sends one batch of nw faces (lane l < nw holds face first + l of the chunk in q) to global
// faces g, g + 1, ...: staged in one of the warp's nbuf buffers (`bufs`, buffer index b
// carried across calls) and sent by a TMA bulk copy, or by coalesced lane stores when
// lane_flush.
template <int N, int LAYOUT>
__device__ __forceinline__ void warp_send_batch(const TablesDev* tab, uint32_t q, int nw, uint32_t first,
                                                vox_chunk_coord c, unsigned long long g, void* out0,
                                                void* out1, unsigned char* bufs, int nbuf,
                                                bool lane_flush, int& b) {
  constexpr int kBuf = warp_buf_bytes<LAYOUT>();
  const int lane = threadIdx.x & 31;
  unsigned char* buf = bufs + b * kBuf;
  // the copy issued nbuf batches ago read this buffer; wait until it is done reading
  if (lane == 0) {
    if (nbuf == 1) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    else asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
  }
  __syncwarp();
  const int shift = stage_shift<LAYOUT>(g);
  if (lane < nw) {
    const int x = q & 255, y = (q >> 8) & 255, z = (q >> 16) & 255, d = q >> 24;
    stage_face<LAYOUT>(buf, kWarpBatch, shift, lane, d, (float)(c.x * N + x), (float)(c.y * N + y),
                       (float)(c.z * N + z), first + (uint32_t)lane, tab);
  }
  if (lane_flush) {
    __syncwarp();
    flush_warp_lanes<LAYOUT>(buf, shift, nw, g, out0, out1);
  } else {
    fence_proxy_async_smem();
    __syncwarp();
    flush_warp<LAYOUT>(buf, shift, nw, g, out0, out1);
  }
  __syncwarp();
  b = nbuf == 2 ? b ^ 1 : 0;
}

// Faces of the batch that starts at global face g with `left` faces to go: a batch that starts
// off a line_faces boundary of the output ends on a later one, so that the batches after it
// cover whole 128-byte lines.
template <int LAYOUT>
__device__ __forceinline__ int batch_faces(unsigned long long g, int left) {
  return min(kWarpBatch - (int)(g & (unsigned long long)(line_faces<LAYOUT>() - 1u)), left);
}
// The faces of a batch of cnt faces at g that fit an output of cap faces.
__device__ __forceinline__ int faces_in(unsigned long long g, int cnt, unsigned long long cap) {
  return g >= cap ? 0 : (g + (unsigned long long)cnt > cap ? (int)(cap - g) : cnt);
}

// Sends the nwf faces of a warp's face list (chunk-local indices first, first + 1, ...) to
// global faces g0 + first + ..., a batch at a time.
template <int N, int LAYOUT>
__device__ __forceinline__ void warp_send_faces(const TablesDev* tab, const uint32_t* list, int nwf,
                                                uint32_t first, vox_chunk_coord c,
                                                unsigned long long g0, unsigned long long cap,
                                                void* out0, void* out1, unsigned char* bufs,
                                                int nbuf, bool lane_flush, int& b) {
  const int lane = threadIdx.x & 31;
  for (int r0 = 0, cnt = 0; r0 < nwf; r0 += cnt) {
    const unsigned long long g = g0 + first + (unsigned)r0;
    cnt = batch_faces<LAYOUT>(g, nwf - r0);
    const int nw = faces_in(g, cnt, cap);
    if (nw == 0) continue;
    warp_send_batch<N, LAYOUT>(tab, lane < nw ? list[r0 + lane] : 0u, nw, first + (uint32_t)r0, c, g,
                               out0, out1, bufs, nbuf, lane_flush, b);
  }
}

// Emission of elements [lo, hi): part w of `parts` (a warp each) takes the contiguous run
// [lo + w*per, ...) of whole groups of 32 elements, so consecutive groups' faces are adjacent
// in the output.
// Faces accumulate in the warp's list and leave once there are at least 32, up to the last
// line_faces boundary of the output (g0: the output index of chunk-local face 0); fewer
// than line_faces are carried to the next group, and the rest leave at the end. Batches
// that start and end on those boundaries write whole 128-byte lines, which matters most
// for outputs in host memory, where a partial line costs a slower write.
template <int N, int LAYOUT, typename Smem, typename Send>
__device__ __forceinline__ void emit_runs(const Smem& s, int lo, int hi, int part,
                                          int parts, unsigned long long g0, Send send) {
  constexpr unsigned kLine = line_faces<LAYOUT>();
  const unsigned phase = (unsigned)(g0 & (unsigned long long)(kLine - 1u));
  const bool use_list = s.misc[1] >= 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* list = s.lists + warp * kWarpFaces;
  const int groups = (hi - lo + 31) >> 5;
  const int gper = (groups + parts - 1) / parts;
  const int wlo = lo + part * gper * 32;
  const int whi = min(hi, wlo + gper * 32);
  int have = 0;             // faces waiting in list[0, have)
  uint32_t first_have = 0;  // chunk-local index of list[0]
  for (int base = wlo; base < whi; base += 32) {
    uint32_t first;
    const int nwf = warp_faces<N>(s, use_list, whi, base, list + have, first);
    if (have == 0) first_have = first;
    have += nwf;
    const int full = have >= 32 ? have - (int)((phase + first_have + (unsigned)have) & (kLine - 1u)) : 0;
    if (full > 0) {
      send(list, full, first_have);
      // move the remainder (< 32 faces) to the front of the list
      const uint32_t keep = lane < have - full ? list[full + lane] : 0u;
      __syncwarp();
      if (lane < have - full) list[lane] = keep;
      __syncwarp();
      first_have += (uint32_t)full;
      have -= full;
    }
  }
  if (have > 0) send(list, have, first_have);
}

// wait_read = false: the caller's next use of the staging area is another emit_chunk. With
// one buffer per warp its first send waits for every earlier copy's read of that buffer,
// so the warp need not wait for its last copies here (with two buffers it still does: the
// next call starts again at buffer 0, which the last copy may still be reading).
template <int N, int LAYOUT>
__device__ void emit_chunk(const ChunkSmem<N, LAYOUT>& s, vox_chunk_coord c, unsigned long long g0,
                           unsigned long long cap, void* out0, void* out1, int nbuf,
                           bool lane_flush, int lo, int hi, int part, int parts,
                           bool wait_read = true) {
  constexpr int kBuf = warp_buf_bytes<LAYOUT>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* bufs = s.stage + (size_t)warp * nbuf * kBuf;
  int b = 0;
  emit_runs<N, LAYOUT>(s, lo, hi, part, parts, g0, [&](const uint32_t* list, int nf, uint32_t first) {
    warp_send_faces<N, LAYOUT>(s.tab, list, nf, first, c, g0, cap, out0, out1, bufs, nbuf,
                               lane_flush, b);
  });
  if (wait_read || nbuf != 1) {
    if (lane == 0) bulk_wait_read_all();
    __syncwarp();
  }
}

// Writes one face record straight to global memory (face index g).
template <int LAYOUT>
__device__ __forceinline__ void store_face(void* out0, void* out1, unsigned long long g, int dir,
                                           float tx, float ty, float tz, uint32_t f_local,
                                           const TablesDev* tab) {
  if (LAYOUT == VOX_LAYOUT_INSTANCED) {
    uint32_t* o = reinterpret_cast<uint32_t*>(out0) + g * 17ull;
    const float z0 = tx * 0.0f, z1 = ty * 0.0f, z2 = tz * 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      o[4 * c + 0] = __float_as_uint(tab->part[dir][0][c] + z0);
      o[4 * c + 1] = __float_as_uint(tab->part[dir][1][c] + z1);
      o[4 * c + 2] = __float_as_uint(tab->part[dir][2][c] + z2);
      o[4 * c + 3] = __float_as_uint(tab->row3[dir][c]);
    }
    o[12] = __float_as_uint(tx);
    o[13] = __float_as_uint(ty);
    o[14] = __float_as_uint(tz);
    o[15] = __float_as_uint(1.0f);
    o[16] = tab->tex[dir];
  } else {
    float4* v = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(out0) + g * 96ull);
    const float4* C = reinterpret_cast<const float4*>(tab->corner[dir]);
    const float4 c0 = C[0], c1 = C[1], c2 = C[2];
    const float face = __uint_as_float(tab->slot[dir]);
    v[0] = make_float4(c0.x + tx, c0.y + ty, c0.z + tz, 0.0f);
    v[1] = make_float4(0.0f, face, c0.w + tx, c1.x + ty);
    v[2] = make_float4(c1.y + tz, 1.0f, 0.0f, face);
    v[3] = make_float4(c1.z + tx, c1.w + ty, c2.x + tz, 0.0f);
    v[4] = make_float4(1.0f, face, c2.y + tx, c2.z + ty);
    v[5] = make_float4(c2.w + tz, 1.0f, 1.0f, face);
    uint2* ix = reinterpret_cast<uint2*>(reinterpret_cast<unsigned char*>(out1) + g * 24ull);
    const uint32_t b = 4u * f_local;
    ix[0] = make_uint2(b + 0u, b + 2u);
    ix[1] = make_uint2(b + 1u, b + 3u);
    ix[2] = make_uint2(b + 1u, b + 2u);
  }
}

// The direct counterpart of warp_send_faces: lane l stores faces l, l + 32, ... of the
// list straight to global memory.
template <int N, int LAYOUT>
__device__ __forceinline__ void warp_store_faces(const TablesDev* tab, const uint32_t* list, int nwf,
                                                 uint32_t first, vox_chunk_coord c,
                                                 unsigned long long g0, unsigned long long cap,
                                                 void* out0, void* out1) {
  const int ox = c.x * N, oy = c.y * N, oz = c.z * N;
  for (int i = threadIdx.x & 31; i < nwf; i += 32) {
    const uint32_t q = list[i];
    const int x = q & 255, y = (q >> 8) & 255, z = (q >> 16) & 255, d = q >> 24;
    const uint32_t l = first + (uint32_t)i;
    const unsigned long long gg = g0 + l;
    if (gg < cap)
      store_face<LAYOUT>(out0, out1, gg, d, (float)(ox + x), (float)(oy + y), (float)(oz + z),
                         l, tab);
  }
  __syncwarp();
}

// Direct variant of emit_chunk: the same runs and compaction, then every lane writes one
// face record straight to global memory (32 consecutive faces per warp step).
template <int N, int LAYOUT>
__device__ void emit_chunk_direct(const ChunkSmem<N, LAYOUT>& s, vox_chunk_coord c,
                                  unsigned long long g0, unsigned long long cap, void* out0,
                                  void* out1, int lo, int hi, int part, int parts) {
  emit_runs<N, LAYOUT>(s, lo, hi, part, parts, g0, [&](const uint32_t* list, int nf, uint32_t first) {
    warp_store_faces<N, LAYOUT>(s.tab, list, nf, first, c, g0, cap, out0, out1);
  });
}

// A chunk's face list (overlap schedule): one packed face (pack_face) per face in emission
// order, in the chunk's spill slot, written by the generation item from the face voxels and
// read by the emission item, which then needs no chunk state in shared memory, no compaction
// and no barrier beyond the offset's. It takes 4 bytes a face next to the 68 or 120 it
// describes. Chunks with more faces than max_list_faces (3.7 N^2 at 64^3, whose slots hold no
// more) spill their occupancy and row lists instead and are compacted at emission.
//
// The most faces of a list in a slot of `bytes`: what fits, but no more than `most` N^2, from where its
// traffic costs more than the compaction: 9 at 16^3 (white-noise columns of 11 N^2 faces, 2000 chunks:
// 151 us a batch in one launch with lists of all that fits, 138 without; 155 and 137 in two) and in one
// launch 5 at 8^3 (8000 chunks of 6 N^2: 107 and 100 us; in two launches lists stay ahead, 50 us of
// 3000 chunks against 59). Terrain has 2 N^2 to 4 N^2 faces, random voxels 6 N^2 to 100 N^2.
template <int N>
__host__ __device__ constexpr uint32_t max_list_faces(int bytes, int most) {
  return (uint32_t)(bytes / 4 < most * N * N ? bytes / 4 : most * N * N);
}
// Position of set bit n (from 0) of m, which has more than n.
template <int N, typename RowT>
__device__ __forceinline__ int nth_bit(RowT m, int n) {
  int pos = 0;
#pragma unroll
  for (int w = N / 2; w > 0; w >>= 1) {
    const int c = popc_row((RowT)(m & (((RowT)1 << w) - (RowT)1)));
    if (n >= c) {
      n -= c;
      m >>= w;
      pos += w;
    }
  }
  return pos;
}

// 64^3 chunks have no voxel list: a warp takes 32 rows at a time, dealt out over the warps so
// that neighbouring rows (which have faces together) go to different ones, counts the face
// voxels of each, and then every lane finds its own voxel among them by search. (Going
// through all 64 voxels of every row with faces left nine lanes in ten idle: 30 terrain chunks
// of 64^3 took 380 us a batch, 127 us this way. Where the voxels are listed the search costs
// more than it saves: at 32^3 a batch of 777 cave chunks took 57 us instead of 45.)
template <int N, int LAYOUT>
__device__ __forceinline__ void write_face_rows(const ChunkSmem<N, LAYOUT>& s, uint32_t* dst) {
  using RowT = typename Shape<N>::RowT;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int r0 = 0; r0 < N * N; r0 += 32 * nwarps) {
    RowT m[6];
    const int mine = r0 + lane * nwarps + warp;
    const bool faces = s.rows[mine + 1] != s.rows[mine];
    if (__all_sync(0xffffffffu, !faces)) continue;
    int cnt = 0;
    if (faces) {
      row_masks<N, LAYOUT>(s, mine / N, mine % N, m);
      cnt = popc_row((RowT)(m[0] | m[1] | m[2] | m[3] | m[4] | m[5]));
    }
    int incl = cnt;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += v;
    }
    const int voxels = __shfl_sync(0xffffffffu, incl, 31);
    for (int base = 0; base < voxels; base += 32) {
      const int k = base + lane;
      int own = 0;  // the lane whose row holds voxel k: the first with incl > k
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, incl, own + step - 1) <= k) own += step;
      const int before = __shfl_sync(0xffffffffu, incl - cnt, own);
      if (k < voxels) {
        const int r = r0 + own * nwarps + warp, y = r / N, z = r % N;
        row_masks<N, LAYOUT>(s, y, z, m);
        const int x = nth_bit<N>((RowT)(m[0] | m[1] | m[2] | m[3] | m[4] | m[5]), k - before);
        const RowT below = ((RowT)1 << x) - (RowT)1;
        uint32_t* out = dst + s.rows[r];
        unsigned bits = 0;
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          out += popc_row((RowT)(m[d] & below));
          bits |= (unsigned)((m[d] >> x) & (RowT)1) << d;
        }
        const uint32_t code = pack_face(x, y, z, 0);
        while (bits) {
          const int d = __ffs(bits) - 1;
          bits &= bits - 1u;
          *out++ = code | ((uint32_t)d << 24);
        }
      }
      __syncwarp();
    }
  }
}

template <int N, int LAYOUT>
__device__ __forceinline__ void write_face_list(const ChunkSmem<N, LAYOUT>& s, uint32_t* dst) {
  if constexpr (Shape<N>::VCap == 0) {
    write_face_rows<N, LAYOUT>(s, dst);
  } else {
    const bool use_list = s.misc[1] >= 0;
    const int elems = emit_elems(s);
    for (int base = (int)(threadIdx.x & ~31u); base < elems; base += blockDim.x) {
      uint32_t first;
      warp_faces<N, true>(s, use_list, elems, base, dst, first);
    }
  }
}

// Emission of part `part` of `parts` (a warp each) of a chunk from its face list (`total` faces,
// the chunk's first at global face g0): the output lines that the chunk touches are cut
// evenly over the parts, so every batch but the chunk's first and last covers whole lines.
template <int N, int LAYOUT>
__device__ __forceinline__ void emit_list(const ChunkSmem<N, LAYOUT>& s, const uint32_t* codes,
                                          uint32_t total, unsigned part, unsigned parts,
                                          vox_chunk_coord c, unsigned long long g0,
                                          unsigned long long cap, void* out0, void* out1, int nbuf,
                                          bool lane_flush) {
  constexpr unsigned kLine = line_faces<LAYOUT>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned phase = (unsigned)(g0 & (unsigned long long)(kLine - 1u));
  const unsigned lines = (phase + total + kLine - 1u) / kLine;
  const unsigned la = lines * part / parts, lb = lines * (part + 1u) / parts;
  if (la == lb) return;
  const int lo = la == 0u ? 0 : (int)(la * kLine - phase);
  const int hi = (int)min(total, lb * kLine - phase);
  unsigned char* bufs = s.stage + (size_t)warp * nbuf * warp_buf_bytes<LAYOUT>();
  int b = 0;
  int cnt = batch_faces<LAYOUT>(g0 + (unsigned)lo, hi - lo);
  uint32_t q = lane < cnt ? __ldcg(codes + lo + lane) : 0u;
  for (int r = lo; r < hi;) {
    const unsigned long long g = g0 + (unsigned)r;
    const int r2 = r + cnt;
    const int cnt2 = r2 < hi ? batch_faces<LAYOUT>(g0 + (unsigned)r2, hi - r2) : 0;
    const uint32_t q2 = lane < cnt2 ? __ldcg(codes + r2 + lane) : 0u;  // the next batch's faces
    const int nw = faces_in(g, cnt, cap);
    if (nw == 0) break;
    if (nbuf > 0) {
      warp_send_batch<N, LAYOUT>(s.tab, q, nw, (uint32_t)r, c, g, out0, out1, bufs, nbuf, lane_flush, b);
    } else if (lane < nw) {
      const int x = q & 255, y = (q >> 8) & 255, z = (q >> 16) & 255, d = q >> 24;
      store_face<LAYOUT>(out0, out1, g + (unsigned)lane, d, (float)(c.x * N + x), (float)(c.y * N + y),
                         (float)(c.z * N + z), (uint32_t)(r + lane), s.tab);
    }
    r = r2;
    cnt = cnt2;
    q = q2;
  }
  if (nbuf > 1) {  // the next item starts at buffer 0 again (one buffer: its first send waits)
    if (lane == 0) bulk_wait_read_all();
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------------
// Kernels
// ------------------------------------------------------------------------------------

// Minimum resident CTAs per SM the fused kernels are compiled for, i.e. their register
// budget: 64 registers a thread in general (4 CTAs of 256 threads), which keeps the
// meshing paths at the occupancy their shared memory allows. The 3-D density generator
// needs more: 80 at 256 threads for 32^3 chunks (3 CTAs), 64 at 512 (2 CTAs); 16^3 and 8^3
// chunks keep the budgets the compiler chose for them unconstrained, and 64^3 density or
// heightmap chunks at 512 threads keep up to 128.
template <int N, int GM, int T>
__host__ __device__ constexpr int fused_min_ctas() {
  if (GM == GM_DENSITY) {
    if (N == 32) return T == 256 ? 3 : 2;
    if (N == 16) return T == 256 ? 3 : 7;
    if (N == 8) return T == 64 ? 14 : 25;
    return 1;
  }
  if (GM == GM_HEIGHT && N == 64 && T == 512) return 1;
  return 65536 / (T * 64) > 0 ? 65536 / (T * 64) : 1;
}

// Persistent fused generation + meshing over a device work queue (GM != GM_OCC), or
// meshing of resident occupancy (GM == GM_OCC). One chunk per CTA iteration; T threads.
// Occupancy and halo rows of chunk i in shared memory: loaded from the slot pool
// (GM_OCC) or generated from the noise field.
template <int N, int GM, int LAYOUT, int T, int kHash = kHashNone>
__device__ __forceinline__ void prepare_chunk(ChunkSmem<N, LAYOUT>& s, const MeshArgs& a, int i,
                                              vox_chunk_coord c) {
  if (GM == GM_OCC) {
    const unsigned long long words = (unsigned long long)N * N * Shape<N>::W;
    const int slot = a.slots[i];
    const uint32_t* nb[6];
    unsigned use = 0;
    bool bad = slot < 0 || slot >= a.pool_slots;
    for (int d = 0; d < 6; ++d) {
      const int ns = a.nbr_slots ? a.nbr_slots[6 * i + d] : -1;
      nb[d] = nullptr;
      if (d >= 4 && !a.full6) continue;
      if (ns >= a.pool_slots) bad = true;
      if (ns >= 0 && ns < a.pool_slots) {
        nb[d] = a.occ_pool + (unsigned long long)ns * words;
        use |= 1u << d;
      }
    }
    if (bad && threadIdx.x == 0) atomicOr(&a.ctl->err, ERR_BAD_INPUT);
    // An out-of-range slot reads slot 0 instead (the call then reports VOX_ERR_INVALID).
    const int sl = (slot >= 0 && slot < a.pool_slots) ? slot : 0;
    load_chunk<N, LAYOUT, T>(s, a.occ_pool + (unsigned long long)sl * words, nb, use);
  } else {
    unsigned m = a.nbr_mask ? a.nbr_mask[i] : 0u;
    if (GM == GM_BERNOULLI) m = 0u;
    if (!a.full6) m &= 0xFu;
    gen_chunk<N, GM, LAYOUT, T, kHash>(s, a.gen, c, a.index_base + i, m, true);
  }
}

template <int N, int GM, int LAYOUT, int T>
__global__ void __launch_bounds__(T, fused_min_ctas<N, GM, T>())
k_mesh_batch(const __grid_constant__ MeshArgs a, const __grid_constant__ TablesDev tab) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ChunkSmem<N, LAYOUT> s;
  s.carve(smem_raw);
  load_tables<N, LAYOUT>(s, &tab);  // the tables travel as a kernel parameter
  __shared__ int s_item;
  __shared__ unsigned long long s_base, s_base0;
  __shared__ unsigned s_epoch;
  if (threadIdx.x == 0) {
    s_epoch = ld_relaxed_u32(&a.ctl->epoch);
    s_base0 = launch_base(a);
    __threadfence();
    s_item = (int)atomicAdd(&a.ctl->next, 1u);
  }
  __syncthreads();
  const unsigned epoch = s_epoch;
  const unsigned long long base0 = s_base0;
  int i = s_item;
  while (true) {
    if (i >= a.n) {
      if (threadIdx.x == 0 && i == a.n + (int)gridDim.x - 1) {
        // The last ticket of this launch: reset the queue and advance the epoch.
        a.ctl->next = 0u;
        a.ctl->epoch = epoch + 1u;
      }
      break;
    }
    // The next ticket is drawn now and used after this chunk, so the atomic's latency
    // overlaps the chunk's work. A CTA reserves chunks in increasing order, so the
    // lowest unfinished chunk is always being processed and every look-back ends.
    int next_item = 0;
    if (threadIdx.x == 0) next_item = (int)atomicAdd(&a.ctl->next, 1u);
    const vox_chunk_coord c = a.coords[i];
    prepare_chunk<N, GM, LAYOUT, T>(s, a, i, c);
    const uint32_t total = count_and_scan<N, LAYOUT, T>(s);
    if (threadIdx.x < 32) {
      const unsigned long long excl =
          base0 + lookback(a.state, a.ctl, epoch, i, total, a.spin_limit);
      if (threadIdx.x == 0) {
        s_base = excl;
        a.face_offsets[i] = excl;
        if (i == a.n - 1) {
          a.face_offsets[a.n] = excl + total;
          if (excl + total > a.cap) atomicOr(&a.ctl->err, ERR_CAPACITY);
        }
      }
    }
    __syncthreads();
    if (a.stage_faces > 0)
      emit_chunk<N, LAYOUT>(s, c, s_base, a.cap, a.out0, a.out1, a.stage_faces / kWarpBatch,
                            a.lane_flush != 0, 0, emit_elems(s), threadIdx.x >> 5, T / 32);
    else emit_chunk_direct<N, LAYOUT>(s, c, s_base, a.cap, a.out0, a.out1, 0, emit_elems(s),
                                        threadIdx.x >> 5, T / 32);
    if (threadIdx.x == 0) s_item = next_item;
    __syncthreads();
    i = s_item;
  }
  if ((threadIdx.x & 31) == 0) bulk_wait_all();  // every lane 0 issued bulk copies
  finish_launch(a);
}

// ------------------------------------------------------------------------------------
// Phased schedule of the fused batch kernel (cooperative launch: the whole grid is
// resident, so CTAs may wait for one another).
//  A. CTAs take chunks from the work queue, prepare and count them, and spill the chunk
//     state (occupancy, halo, row offsets, row and voxel lists) to a per-chunk slot
//     (L2-resident) and the face total to counts[i].
//  B. Grid barrier (it also resets the queue). CTA 0 scans counts[] into face_offsets[]
//     and raises the scan flag.
//  C. CTAs take emission items (a chunk, or a segment of one) from the queue again,
//     reload the chunk state, wait for the scan flag once, and emit at face_offsets[i].
// There is no chunk-to-chunk dependency inside a phase. The output bytes are the same
// as the look-back schedule's.
// ------------------------------------------------------------------------------------

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_u32(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid barrier, called by thread 0 of every CTA after a __syncthreads. The last CTA to
// arrive resets the arrival count and the first work queue, then advances the
// generation; the others poll the generation at most spin_limit times. Returns the new
// generation, or 0xFFFFFFFF after a timeout (ERR_TIMEOUT is set).
static __device__ unsigned grid_barrier_t0(BatchCtl* ctl, unsigned nblocks, int spin_limit) {
  const unsigned gen = ld_acquire_u32(&ctl->bar_gen);
  __threadfence();  // this CTA's earlier writes are visible before its arrival
  const unsigned arrived = atomicAdd(&ctl->bar_count, 1u);
  if (arrived == nblocks - 1u) {
    ctl->bar_count = 0u;
    ctl->next = 0u;
    __threadfence();
    st_release_u32(&ctl->bar_gen, gen + 1u);
    return gen + 1u;
  }
  int spins = 0;
  while (ld_acquire_u32(&ctl->bar_gen) == gen) {
    if (++spins > spin_limit) {
      atomicOr(&ctl->err, ERR_TIMEOUT);
      return 0xFFFFFFFFu;
    }
    __nanosleep(spins < 8 ? 32 : 256);
  }
  __threadfence();
  return gen + 1u;
}

// Deterministic exclusive scan of counts[0, n) into offs[0, n) starting at `base`, base +
// total at offs[n] (one CTA of T threads, 8 counts per thread per tile). Returns base + total.
template <int T>
__device__ unsigned long long scan_counts(const uint32_t* counts, int n,
                                          unsigned long long* offs, unsigned long long* wsum,
                                          unsigned long long base) {
  constexpr int V = 8;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nwarps = T >> 5;
  unsigned long long carry = base;
  for (int base = 0; base < n; base += T * V) {
    uint32_t v[V];
    unsigned long long local = 0;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int idx = base + t * V + k;
      v[k] = idx < n ? __ldcg(counts + idx) : 0u;
      local += v[k];
    }
    unsigned long long incl = local;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long u = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += u;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const unsigned long long w = lane < nwarps ? wsum[lane] : 0ull;
      unsigned long long wi = w;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long u = __shfl_up_sync(0xffffffffu, wi, off);
        if (lane >= off) wi += u;
      }
      if (lane < nwarps) wsum[32 + lane] = wi - w;
      if (lane == nwarps - 1) wsum[64] = wi;
    }
    __syncthreads();
    unsigned long long run = carry + wsum[32 + warp] + incl - local;
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int idx = base + t * V + k;
      if (idx < n) offs[idx] = run;
      run += v[k];
    }
    carry += wsum[64];
    __syncthreads();  // wsum is reused by the next tile
  }
  if (t == 0) offs[n] = carry;
  return carry;
}

template <int N, int GM, int LAYOUT, int T>
__global__ void __launch_bounds__(T, fused_min_ctas<N, GM, T>())
k_mesh_batch_phased(const __grid_constant__ MeshArgs a, const __grid_constant__ TablesDev tab) {
  using P = SmemPlan<N, LAYOUT>;
  // spill slot of a chunk: [occ | halo | rows] [nz] [vlist] [misc], laid out as in shared
  // memory; the lists are copied only as far as they are used
  constexpr int kFixed16 = (P::kOcc + P::kHalo + P::kRows) / 16;
  constexpr int kNzOff = P::kOcc + P::kHalo + P::kRows;
  constexpr int kVlOff = kNzOff + P::kNz;
  constexpr int kMiscOff = kVlOff + P::kVList;
  static_assert(P::kSpill == kMiscOff + P::kMisc, "spill layout");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ChunkSmem<N, LAYOUT> s;
  s.carve(smem_raw);
  load_tables<N, LAYOUT>(s, &tab);  // the tables travel as a kernel parameter
  __shared__ int s_item;
  __shared__ unsigned s_gen;
  __shared__ unsigned long long s_base;
  unsigned char* const spill = reinterpret_cast<unsigned char*>(a.scratch);
  uint4* const fixed16 = reinterpret_cast<uint4*>(s.occ);  // s.halo, s.rows follow s.occ
  const int t = threadIdx.x;
  __syncthreads();

  // A. prepare + count + spill (the next ticket is drawn before the chunk's work)
  if (t == 0) s_item = (int)atomicAdd(&a.ctl->next, 1u);
  __syncthreads();
  for (int i = s_item; i < a.n;) {
    int next_item = 0;
    if (t == 0) next_item = (int)atomicAdd(&a.ctl->next, 1u);
    prepare_chunk<N, GM, LAYOUT, T>(s, a, i, a.coords[i]);
    const uint32_t total = count_and_scan<N, LAYOUT, T>(s);
    unsigned char* dst = spill + (unsigned long long)i * P::kSpill;
    for (int q = t; q < kFixed16; q += T) __stcg(reinterpret_cast<uint4*>(dst) + q, fixed16[q]);
    const int nzw = (s.misc[0] + 1) >> 1;                          // u32 words of nz used
    const int vlw = s.misc[1] > 0 ? (s.misc[1] + 1) >> 1 : 0;      // u32 words of vlist used
    for (int q = t; q < nzw; q += T)
      __stcg(reinterpret_cast<uint32_t*>(dst + kNzOff) + q, reinterpret_cast<const uint32_t*>(s.nz)[q]);
    for (int q = t; q < vlw; q += T)
      __stcg(reinterpret_cast<uint32_t*>(dst + kVlOff) + q,
             reinterpret_cast<const uint32_t*>(s.vlist)[q]);
    if (t == 0) {
      __stcg(reinterpret_cast<int2*>(dst + kMiscOff), make_int2(s.misc[0], s.misc[1]));
      __stcg(a.counts + i, total);
      s_item = next_item;
    }
    __syncthreads();
    i = s_item;
  }

  // B. barrier; CTA 0 scans the counts
  __syncthreads();
  if (t == 0) s_gen = grid_barrier_t0(a.ctl, gridDim.x, a.spin_limit);
  __syncthreads();
  const unsigned gen = s_gen;
  if (gen == 0xFFFFFFFFu) return;
  if (blockIdx.x == 0) {
    if (t == 0) s_base = launch_base(a);
    __syncthreads();
    const unsigned long long total = scan_counts<T>(a.counts, a.n, a.face_offsets,
                                                    reinterpret_cast<unsigned long long*>(s.stage),
                                                    s_base);
    __syncthreads();
    if (t == 0) {
      if (total > a.cap) atomicOr(&a.ctl->err, ERR_CAPACITY);
      __threadfence();
      st_release_u32(&a.ctl->scan_flag, gen);
    }
  }

  // C. emission items from the work queue: item k is segment k % split of chunk
  // k / split (the chunk's emission elements cut into split runs of whole warp batches).
  // The chunk state comes back from the spill slot, so nothing is counted twice.
  const int split = a.split > 0 ? a.split : 1;
  const int items = a.n * split;
  bool scanned = blockIdx.x == 0;  // thread 0's view: the scan flag has been seen
  if (t == 0) s_item = (int)atomicAdd(&a.ctl->next, 1u);
  __syncthreads();
  int k = s_item;
  while (true) {
    if (k >= items) {
      // The last ticket of this launch resets the queue.
      if (t == 0 && k == items + (int)gridDim.x - 1) a.ctl->next = 0u;
      break;
    }
    int next_item = 0;
    if (t == 0) next_item = (int)atomicAdd(&a.ctl->next, 1u);
    const int i = k / split, seg = k - i * split;
    const unsigned char* src = spill + (unsigned long long)i * P::kSpill;
    for (int q = t; q < kFixed16; q += T) fixed16[q] = __ldcg(reinterpret_cast<const uint4*>(src) + q);
    if (t == 0) {
      const int2 m = __ldcg(reinterpret_cast<const int2*>(src + kMiscOff));
      s.misc[0] = m.x;
      s.misc[1] = m.y;
    }
    __syncthreads();
    const bool use_list = s.misc[1] >= 0;
    const int elems = emit_elems(s);
    const int per = ((elems + split - 1) / split + 31) & ~31;
    const int lo = min(elems, seg * per), hi = min(elems, lo + per);
    if (lo < hi) {
      // the list entries that elements [lo, hi) read
      const int e0 = use_list ? lo : lo / N, e1 = use_list ? hi : (hi - 1) / N + 1;
      const uint32_t* lsrc = reinterpret_cast<const uint32_t*>(src + (use_list ? kVlOff : kNzOff));
      uint32_t* ldst = reinterpret_cast<uint32_t*>(use_list ? s.vlist : s.nz);
      for (int q = (e0 >> 1) + t; q < (e1 + 1) >> 1; q += T) ldst[q] = __ldcg(lsrc + q);
    }
    if (t == 0) {
      int spins = 0;
      while (!scanned) {
        if (ld_acquire_u32(&a.ctl->scan_flag) == gen) {
          scanned = true;
          break;
        }
        if (++spins > a.spin_limit) break;
        __nanosleep(spins < 8 ? 32 : 256);
      }
      if (scanned) {
        s_base = __ldcg(a.face_offsets + i);
      } else {
        atomicOr(&a.ctl->err, ERR_TIMEOUT);
        s_base = ~0ull;
      }
    }
    __syncthreads();
    if (s_base == ~0ull) break;  // the scan flag never came: give up (error reported)
    if (lo < hi) {
      const vox_chunk_coord c = a.coords[i];
      if (a.stage_faces > 0)
        emit_chunk<N, LAYOUT>(s, c, s_base, a.cap, a.out0, a.out1, a.stage_faces / kWarpBatch,
                              a.lane_flush != 0, lo, hi, t >> 5, T / 32, false);
      else emit_chunk_direct<N, LAYOUT>(s, c, s_base, a.cap, a.out0, a.out1, lo, hi, t >> 5, T / 32);
    }
    if (t == 0) s_item = next_item;
    __syncthreads();
    k = s_item;
  }
  if ((t & 31) == 0) bulk_wait_all();  // every lane 0 issued bulk copies
}

// ------------------------------------------------------------------------------------
// Overlap schedule of the fused batch kernel: the phases of k_mesh_batch_phased without
// the grid barrier, interleaved on one work queue. A generation item (A) prepares and
// counts a chunk, spills its state and publishes its face total as an epoch-tagged
// aggregate look-back state; an emission item (C) waits until its own chunk is published,
// takes the chunk's offset from a decoupled look-back over the published totals, reloads
// the chunk state and emits. Ticket order (overlap_ticket): A(0..L-1), then A(L+m) and
// C(m) alternately while generation items remain, then the remaining emission items.
// Every wait is for an item with a smaller ticket, which a running CTA holds or has
// finished, and generation items never wait, so every wait ends without co-residency:
// a normal launch. L = n (all generation first) suits launches bound by issue; a smaller L
// starts emission early, which hides generation behind a slow output (host memory).
// ------------------------------------------------------------------------------------

template <int N, int GM, int LAYOUT, int T>
__global__ void __launch_bounds__(T, fused_min_ctas<N, GM, T>())
k_mesh_batch_overlap(const __grid_constant__ MeshArgs a, const __grid_constant__ TablesDev tab) {
  using P = SmemPlan<N, LAYOUT>;
  constexpr int kFixed16 = (P::kOcc + P::kHalo + P::kRows) / 16;
  constexpr int kNzOff = P::kOcc + P::kHalo + P::kRows;
  constexpr int kVlOff = kNzOff + P::kNz;
  constexpr int kMiscOff = kVlOff + P::kVList;
  static_assert(P::kSpill == kMiscOff + P::kMisc, "spill layout");
  constexpr uint32_t kListCap = max_list_faces<N>(kMiscOff, N == 8 ? 5 : 9);  // faces of a face list
  constexpr int kListed = -2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ChunkSmem<N, LAYOUT> s;
  s.carve(smem_raw);
  load_tables<N, LAYOUT>(s, &tab);  // the tables travel as a kernel parameter
  __shared__ unsigned s_item;
  __shared__ unsigned s_epoch;
  __shared__ unsigned long long s_base, s_base0;
  unsigned char* const spill = reinterpret_cast<unsigned char*>(a.scratch);
  uint4* const fixed16 = reinterpret_cast<uint4*>(s.occ);  // s.halo, s.rows follow s.occ
  const int t = threadIdx.x;
  if (t == 0) {
    prefetch_inputs(a);
    s_epoch = ld_relaxed_u32(&a.ctl->epoch);
    s_base0 = launch_base(a);
    __threadfence();
    s_item = atomicAdd(&a.ctl->next, 1u);
  }
  __syncthreads();
  const unsigned epoch = s_epoch;
  const unsigned long long base0 = s_base0;
  const unsigned tag = epoch & 0xFFFFFFu;
  const unsigned n = (unsigned)a.n;
  const int split = a.split > 0 ? a.split : 1;
  const unsigned items = n * (unsigned)split;
  const unsigned lag = a.lag < 0 || (unsigned)a.lag > n ? n : (unsigned)a.lag;
  const unsigned last_ticket = n + items + gridDim.x - 1u;
  bool stage_busy = false;  // bulk copies of this CTA may still read the staging area
  unsigned tk = s_item;
  while (true) {
    unsigned idx;
    const int kind = overlap_ticket(tk, n, items, lag, idx);
    if (kind == 2) {
      // The last ticket of this launch resets the queue and advances the epoch.
      if (t == 0 && tk == last_ticket) {
        a.ctl->next = 0u;
        a.ctl->epoch = epoch + 1u;
      }
      break;
    }
    // the next ticket is drawn now and used after this item, so the atomic's latency
    // overlaps the item's work
    unsigned next_tk = 0;
    if (t == 0) next_tk = atomicAdd(&a.ctl->next, 1u);
    if (kind == 0) {
      // A. prepare + count + spill + publish the chunk's total. Generation reuses the
      // staging area as scratch: wait until the earlier copies have read it.
      if (stage_busy) {
        if ((t & 31) == 0) bulk_wait_read_all();
        __syncthreads();
        stage_busy = false;
      }
      const int i = (int)idx;
      prepare_chunk<N, GM, LAYOUT, T>(s, a, i, a.coords[i]);
      const uint32_t total = count_and_scan<N, LAYOUT, T>(s);
      unsigned char* dst = spill + (unsigned long long)i * P::kSpill;
      // the chunk's face list, or its state when the list does not fit the slot; an empty
      // chunk (no row with faces) spills only its counts
      const bool listed = total <= kListCap;
      if (listed) {
        write_face_list<N, LAYOUT>(s, reinterpret_cast<uint32_t*>(dst));
      } else {
        for (int q = t; q < kFixed16; q += T) __stcg(reinterpret_cast<uint4*>(dst) + q, fixed16[q]);
        const int nzw = (s.misc[0] + 1) >> 1;
        const int vlw = s.misc[1] > 0 ? (s.misc[1] + 1) >> 1 : 0;
        for (int q = t; q < nzw; q += T)
          __stcg(reinterpret_cast<uint32_t*>(dst + kNzOff) + q, reinterpret_cast<const uint32_t*>(s.nz)[q]);
        for (int q = t; q < vlw; q += T)
          __stcg(reinterpret_cast<uint32_t*>(dst + kVlOff) + q,
                 reinterpret_cast<const uint32_t*>(s.vlist)[q]);
      }
      __syncthreads();  // every store of the slot precedes the publication below
      if (t == 0) {
        // {faces, kListed} or {rows with faces, face voxels or -1}
        __stcg(reinterpret_cast<int2*>(dst + kMiscOff),
               listed ? make_int2((int)total, kListed) : make_int2(s.misc[0], s.misc[1]));
        __threadfence();
        st_relaxed_u64(&a.state[i], pack_state(epoch, i == 0 ? kFlagIncl : kFlagAgg, total));
      }
    } else {
      // C. emission item idx: segment idx % split of chunk idx / split
      const int c_i = (int)(idx / (unsigned)split), seg = (int)(idx % (unsigned)split);
      const unsigned char* src = spill + (unsigned long long)c_i * P::kSpill;
      // Every thread waits for the chunk's published state with an acquire load, so its
      // own reads of the spill slot below are ordered after the slot's stores (no fence
      // and no barrier before the reload). The waits are bounded; the barrier below
      // combines them.
      unsigned long long w = 0;
      int ok = 0;
      for (int spins = 0;;) {
        w = ld_acquire_u64(&a.state[c_i]);
        if (((unsigned)(w >> 40) & 0xFFFFFFu) == tag && ((w >> 38) & 3ull) != 0ull) {
          ok = 1;
          break;
        }
        if (++spins > a.spin_limit) break;
        __nanosleep(spins < 8 ? 32 : 256);
      }
      ok = __all_sync(0xffffffffu, ok);  // warp-uniform (warp 0's look-back needs every lane)
      if (!ok && (t & 31) == 0) atomicOr(&a.ctl->err, ERR_TIMEOUT);
      // Warp 0 takes the chunk's offset by look-back over the published totals while the
      // other warps reload the chunk's state if it has no face list (a one-warp CTA does
      // both, in turn).
      constexpr int TR = T > 32 ? T - 32 : 32;  // reloading threads
      const int tr = T > 32 ? t - 32 : t;
      int2 m = make_int2(0, kListed);
      if (ok) m = __ldcg(reinterpret_cast<const int2*>(src + kMiscOff));
      const bool listed = m.y == kListed;
      if (t < 32 && ok) {
        // the chunk's face total
        const unsigned long long total =
            listed ? (unsigned long long)m.x
                   : __ldcg(reinterpret_cast<const uint32_t*>(src + P::kOcc + P::kHalo) + Shape<N>::R);
        w = __shfl_sync(0xffffffffu, w, 0);
        // An inclusive state (chunk 0, or a segment of a chunk whose offset another item
        // has already found) gives the offset at once.
        const unsigned long long excl =
            base0 + (((w >> 38) & 3ull) == kFlagIncl
                         ? (w & ((1ull << 38) - 1)) - total
                         : lookback(a.state, a.ctl, epoch, c_i, total, a.spin_limit, false));
        if (t == 0) {
          s_base = excl;
          if (seg == 0) {
            a.face_offsets[c_i] = excl;
            if (c_i == a.n - 1) {
              a.face_offsets[a.n] = excl + total;
              if (excl + total > a.cap) atomicOr(&a.ctl->err, ERR_CAPACITY);
            }
          }
        }
      }
      if (ok && !listed && tr >= 0) {
        if (tr == 0) {
          s.misc[0] = m.x;
          s.misc[1] = m.y;
        }
        for (int q = tr; q < kFixed16; q += TR) fixed16[q] = __ldcg(reinterpret_cast<const uint4*>(src) + q);
        const bool use_list = m.y >= 0;
        const int elems = use_list ? m.y : m.x * N;
        const int per = ((elems + split - 1) / split + 31) & ~31;
        const int lo = min(elems, seg * per), hi = min(elems, lo + per);
        if (lo < hi) {
          const int e0 = use_list ? lo : lo / N, e1 = use_list ? hi : (hi - 1) / N + 1;
          const uint32_t* lsrc = reinterpret_cast<const uint32_t*>(src + (use_list ? kVlOff : kNzOff));
          uint32_t* ldst = reinterpret_cast<uint32_t*>(use_list ? s.vlist : s.nz);
          for (int q = (e0 >> 1) + tr; q < (e1 + 1) >> 1; q += TR) ldst[q] = __ldcg(lsrc + q);
        }
      }
      if (!__syncthreads_and(ok)) break;  // never published (error reported)
      const vox_chunk_coord c = a.coords[c_i];
      if (listed) {
        if (m.x > 0) {
          emit_list<N, LAYOUT>(s, reinterpret_cast<const uint32_t*>(src), (uint32_t)m.x,
                               (unsigned)(seg * (T / 32) + (t >> 5)), (unsigned)(split * (T / 32)), c,
                               s_base, a.cap, a.out0, a.out1, a.stage_faces / kWarpBatch,
                               a.lane_flush != 0);
          stage_busy = true;
        }
      } else {
        const int elems = emit_elems(s);
        const int per = ((elems + split - 1) / split + 31) & ~31;
        const int lo = min(elems, seg * per), hi = min(elems, lo + per);
        if (lo < hi) {
          if (a.stage_faces > 0) {
            emit_chunk<N, LAYOUT>(s, c, s_base, a.cap, a.out0, a.out1, a.stage_faces / kWarpBatch,
                                  a.lane_flush != 0, lo, hi, t >> 5, T / 32, false);
            stage_busy = true;
          } else {
            emit_chunk_direct<N, LAYOUT>(s, c, s_base, a.cap, a.out0, a.out1, lo, hi, t >> 5, T / 32);
          }
        }
      }
    }
    if (t == 0) s_item = next_tk;
    __syncthreads();
    tk = s_item;
  }
  if ((t & 31) == 0) bulk_wait_all();  // every lane 0 issued bulk copies
  finish_launch(a);
}

// Register budget of k_generate as resident CTAs per SM: 64 registers a thread for the 3-D
// density noise (dens_block_z holds a block of sums and four corner records), 32 for
// the heightmap columns up to 32^3 and for Bernoulli fills, whose occupancy then follows
// shared memory alone.
template <int N, int GM, int T>
__host__ __device__ constexpr int generate_min_ctas() {
  if (GM == GM_DENSITY || (GM == GM_HEIGHT && N > 32)) return 65536 / (T * 64) > 0 ? 65536 / (T * 64) : 1;
  return 65536 / (T * 32) > 32 ? 32 : 65536 / (T * 32);
}

// Chunk::new for n chunks, occupancy rows written to global memory. One CTA per chunk:
// chunk i at occ_out + i * words, or at slot a.slots[i] of a pool of a.pool_slots slots when
// a.slots is set (an out-of-range slot writes nothing and latches ERR_BAD_INPUT).
template <int N, int GM, int T>
__global__ void __launch_bounds__(T, generate_min_ctas<N, GM, T>())
k_generate(MeshArgs a, uint32_t* occ_out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ChunkSmem<N, VOX_LAYOUT_VERTEX> s;
  s.carve(smem_raw);
  constexpr int words = N * N * Shape<N>::W;
  const int i = blockIdx.x;
  long long slot = i;
  if (a.slots) {
    slot = a.slots[i];
    if (slot < 0 || slot >= a.pool_slots) {
      if (threadIdx.x == 0) atomicOr(&a.ctl->err, ERR_BAD_INPUT);
      return;  // uniform across the CTA: no barrier has been reached yet
    }
  }
  load_tables<N, VOX_LAYOUT_VERTEX>(s, a.tables);
  constexpr bool kHashed = GM == GM_HEIGHT && N <= 32;
  if (kHashed) load_grad2<T>(s, s.stage, a.grad2);
  __syncthreads();
  gen_chunk<N, GM, VOX_LAYOUT_VERTEX, T, kHashed ? kHashAll : kHashNone>(s, a.gen, a.coords[i],
                                                                         a.index_base + i, 0u, false);
  const uint32_t* src = reinterpret_cast<const uint32_t*>(s.occ);
  uint32_t* dst = occ_out + (size_t)slot * words;
  for (int q = threadIdx.x; q < words; q += blockDim.x) dst[q] = src[q];
}

// The halo planes of chunks outside a batch (the staged-halo path of the fused batch):
// for each listed chunk i below the count *a.n_dev (at most a.n), only the plane of its
// occupancy that the meshing of its neighbour in the batch reads — x = N - 1 or x = 0 for
// dirs[i] = 0 or 1 (the chunk is the batch chunk's -x or +x neighbour), z = N - 1 or 0 for
// 2 or 3, y = N - 1 or 0 for 4 or 5 — written to occ_out + i * words, every other bit zero.
// N * N samples instead of N^3; each is the sample the fused launch generates for that halo
// plane (generation is a function of the voxel's world position). A grid of a few CTAs per
// SM strides over the list, so the launch is sized before the count is known.
template <int N, int GM, int T>
__global__ void __launch_bounds__(T, 65536 / (T * 64))
k_generate_planes(MeshArgs a, const uint8_t* __restrict__ dirs, uint32_t* occ_out) {
  static_assert(GM == GM_HEIGHT || GM == GM_DENSITY, "planes of the noise generators only");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ChunkSmem<N, VOX_LAYOUT_VERTEX> s;
  s.carve(smem_raw);
  constexpr int W = Shape<N>::W;
  constexpr int words = N * N * W;
  const int count = (int)min((unsigned)a.n, *a.n_dev);
  if ((int)blockIdx.x >= count) return;  // uniform across the CTA
  load_tables<N, VOX_LAYOUT_VERTEX>(s, a.tables);
  uint32_t* occw = reinterpret_cast<uint32_t*>(s.occ);
  for (int i = blockIdx.x; i < count; i += gridDim.x) {
    for (int q = threadIdx.x; q < words; q += blockDim.x) occw[q] = 0u;
    __syncthreads();  // (the first pass: also the tables)
    const vox_chunk_coord c = a.coords[i];
    const int d = dirs[i];
    const int fix = (d & 1) ? 0 : N - 1;
    const int ox = c.x * N, oy = c.y * N, oz = c.z * N;
    for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
      const int p = e / N, q = e % N;
      const int x = d <= 1 ? fix : q;
      const int y = d <= 3 ? p : fix;
      const int z = d <= 1 ? q : (d <= 3 ? fix : p);
      bool solid;
      if constexpr (GM == GM_HEIGHT)
        solid = y < column_k<N>(s, a.gen, ox, oy, oz, x, z);
      else
        solid = gen_solid<N, GM, VOX_LAYOUT_VERTEX>(s, a.gen, x, y, z, ox, oy, oz, 0ull);
      if (solid) atomicOr(&occw[(y * N + z) * W + (x >> 5)], 1u << (x & 31));
    }
    __syncthreads();
    uint32_t* dst = occ_out + (size_t)i * words;
    for (int q = threadIdx.x; q < words; q += blockDim.x) dst[q] = occw[q];
    __syncthreads();  // the next plane clears s.occ
  }
}

}  // namespace vox
