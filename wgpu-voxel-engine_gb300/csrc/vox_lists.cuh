// vox_lists.cuh — the two launches of a batch under the overlap schedule with outputs in device
// memory: k_list_chunks generates (or loads) and counts one chunk per CTA and writes its faces
// as a list of 4-byte codes, k_emit_lists turns the lists into records.
//
// One persistent launch for both (k_mesh_batch_overlap) gives every CTA the registers and the
// shared memory of the hungrier half: 4 CTAs of 256 threads an SM for 16^3 terrain, whose chunks
// then need two waves and whose emission waits behind CTA barriers (a chunk in 6.4 us, twice, then
// as long for its emission). Split, generation runs at the occupancy of its own needs (8 CTAs,
// all 1024 chunks at once, the last done after 14 us), and emission has no CTA barriers: a
// warp takes a part of a chunk, reads its codes and writes whole 128-byte lines. The second
// launch is a programmatic dependent of the first (its CTAs start as soon as the last
// generation CTA has started, and wait for chunks, not for the kernel), so splitting costs no
// launch gap.
// Measured, us a batch, one launch -> two (both as they are now): 1024 terrain chunks of 16^3 33.7 ->
// 30.7, 64 start chunks of 32^3 as instances 37.2 -> 16.1, 777 cave chunks of 32^3 from occupancy
// 53.8 -> 35.4, 4096 cave chunks generated 301 -> 282. What bounds them: generation by its
// instructions (58 % of issue at 16^3), emission by the offsets' way (the slowest chunk of a group, its
// scan, the poll: about 4 us) and then the writes (61 MB in 11 us into L2, 4.7 TB/s into HBM).
// Figures beside single choices below were taken when the choice was made, each pair on one tree.
#pragma once

#include "vox_device.cuh"
#include "vox_launch.h"

namespace vox {

// Slot of a chunk in the scratch: its face list, or (more than kCap faces) the spilled chunk state of
// SmemPlan. 64^3 slots hold a list of 8 N^2 faces, the others the size of the chunk state (see
// max_list_faces).
template <int N>
struct ListSlot {
  using P = SmemPlan<N, VOX_LAYOUT_VERTEX>;
  static constexpr int kNzOff = P::kOcc + P::kHalo + P::kRows;
  static constexpr int kVlOff = kNzOff + P::kNz;
  static constexpr int kMiscOff = kVlOff + P::kVList;
  static constexpr int kBytes = N == 64 ? 8 * N * N * 4 : P::kSpill;
  static constexpr uint32_t kCap = max_list_faces<N>(kBytes, N == 8 ? 10 : 9);
  static_assert(kBytes >= P::kSpill, "the slot holds a spilled chunk state");
};

// a.counts[i] of a chunk that has no list counts the runs of it that emission warps have taken; all
// are taken once it is at least kTaken, as those of a listed chunk are from the start.
constexpr uint32_t kTaken = 1u << 30;

// CTA sizes of k_list_chunks: kBig = 0 for many chunks; kBig = 1, up to one thread a row, for
// batches of no more chunks than SMs, where a chunk's latency is the batch's.
template <int N>
__host__ __device__ constexpr int list_threads(int big) {
  return N == 8 ? 64 : (N == 16 ? 256 : (N == 32 ? (big ? 1024 : 256) : (big ? 1024 : 512)));
}

// Dynamic shared memory of k_list_chunks: tables, occupancy, halo and counts, then the row
// offsets, row and voxel lists and the count's warp totals, which take the place of the
// generator's scratch once the occupancy is there.
template <int N, int GM>
struct ListSmem {
  using P = SmemPlan<N, VOX_LAYOUT_VERTEX>;
  static constexpr int kRowsOff = P::kTables + P::kOcc + P::kHalo + P::kMisc;
  static constexpr int kLists = P::kRows + P::kNz + P::kVList;
  static constexpr int kScratch = GM == GM_DENSITY  ? dens_scratch_bytes<N>()
                                  : GM == GM_HEIGHT ? (N > 32 ? P::kHeight : kGrad2 * 8)
                                                    : 0;
  static constexpr int kBytes = kRowsOff + (kScratch > kLists + 256 ? kScratch : kLists + 256);
  // The generator's scratch is at lists(base); the count's is behind the lists.
  __device__ static unsigned char* lists(unsigned char* base) { return base + kRowsOff; }
  __device__ static void carve(ChunkSmem<N, VOX_LAYOUT_VERTEX>& s, unsigned char* base) {
    s.carve(base, 0);
    s.misc = reinterpret_cast<int*>(base + P::kTables + P::kOcc + P::kHalo);
    s.rows = reinterpret_cast<uint32_t*>(lists(base));
    s.nz = reinterpret_cast<uint16_t*>(lists(base) + P::kRows);
    s.vlist = reinterpret_cast<uint16_t*>(lists(base) + P::kRows + P::kNz);
    s.scratch_at(lists(base));
  }
};

// Resident CTAs per SM that k_list_chunks is compiled for (its register budget): 64 registers
// for the density evaluation and for 64^3 chunks, 32 otherwise.
template <int N, int GM, int kBig>
__host__ __device__ constexpr int list_min_ctas() {
  constexpr int kCtas = 65536 / (list_threads<N>(kBig) * (GM == GM_DENSITY || N == 64 ? 64 : 32));
  return kCtas < 32 ? kCtas : 32;
}

template <int N, int GM, int kBig>
__global__ void __launch_bounds__(list_threads<N>(kBig), list_min_ctas<N, GM, kBig>())
k_list_chunks(const __grid_constant__ MeshArgs a, const __grid_constant__ TablesDev tab) {
  using P = SmemPlan<N, VOX_LAYOUT_VERTEX>;
  using S = ListSlot<N>;
  constexpr int T = list_threads<N>(kBig);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  using M = ListSmem<N, GM>;
  ChunkSmem<N, VOX_LAYOUT_VERTEX> s;
  M::carve(s, smem_raw);
  unsigned char* const lists = M::lists(smem_raw);
  const int i = blockIdx.x, t = threadIdx.x;
  constexpr bool kHashed = GM == GM_HEIGHT && N <= 32;
  if (GM != GM_OCC) {  // the context's tables are older than any launch of the stream
    load_tables<N, VOX_LAYOUT_VERTEX>(s, &tab);
    if (kHashed) load_grad2<T>(s, lists, a.grad2);
  }
  pdl_wait();
  // Only now: k_emit_lists does not wait for earlier work itself, so it must not start, and read
  // the epoch, before the launches ahead of this one have ended.
  pdl_trigger();
  unsigned epoch = 0;
  if (t == 0) epoch = ld_relaxed_u32(&a.ctl->epoch);
  const vox_chunk_coord c = a.coords[i];
  if (GM != GM_OCC) __syncthreads();
  prepare_chunk<N, GM, VOX_LAYOUT_VERTEX, T, kHashed ? kHashGrad : kHashNone>(s, a, i, c);
  s.stage = lists + M::kLists;
  const uint32_t total = count_and_scan<N, VOX_LAYOUT_VERTEX, T>(s);
  unsigned char* dst = reinterpret_cast<unsigned char*>(a.scratch) + (unsigned long long)i * S::kBytes;
  if (t == 0) {
    __stcg(a.counts + i, total <= S::kCap ? kTaken : 0u);
    if (total > S::kCap) atomicAdd(&a.ctl->open, 1u);
  }
  if (total <= S::kCap) {
    write_face_list<N, VOX_LAYOUT_VERTEX>(s, reinterpret_cast<uint32_t*>(dst));
  } else {
    constexpr int kOccHalo = (P::kOcc + P::kHalo) / 16, kRows = P::kRows / 16;
    for (int q = t; q < kOccHalo + kRows; q += T)  // s.halo follows s.occ
      __stcg(reinterpret_cast<uint4*>(dst) + q,
             q < kOccHalo ? reinterpret_cast<const uint4*>(s.occ)[q]
                          : reinterpret_cast<const uint4*>(s.rows)[q - kOccHalo]);
    const int nzw = (s.misc[0] + 1) >> 1;
    const int vlw = s.misc[1] > 0 ? (s.misc[1] + 1) >> 1 : 0;
    for (int q = t; q < nzw; q += T)
      __stcg(reinterpret_cast<uint32_t*>(dst + S::kNzOff) + q, reinterpret_cast<const uint32_t*>(s.nz)[q]);
    for (int q = t; q < vlw; q += T)
      __stcg(reinterpret_cast<uint32_t*>(dst + S::kVlOff) + q,
             reinterpret_cast<const uint32_t*>(s.vlist)[q]);
    if (t == 0) __stcg(reinterpret_cast<int2*>(dst + S::kMiscOff), make_int2(s.misc[0], s.misc[1]));
  }
  __syncthreads();  // every store of the slot precedes the publication below
  if (t == 0) {
    __threadfence();
    st_relaxed_u64(&a.state[i], pack_state(epoch, i == 0 ? kFlagIncl : kFlagAgg, total));
  }
}

// Offsets. k_list_chunks publishes its chunks' totals as aggregate states. A scan item, one warp
// per group of kGroup chunks, waits for the group's totals, scans them, takes the group's base by
// look-back over the group states (behind the n chunk states) and upgrades the chunk states to
// inclusive prefixes, so that an emission item only waits for two neighbouring words. Letting
// each emission warp look back itself reads the same few words thousands of times (the
// 1024-chunk 16^3 terrain in one persistent launch: 42.6 us against 36.0 us).
constexpr int kGroup = 32;
static_assert(kGroup == kStateGroup, "the host sizes the states by groups");

__device__ __forceinline__ bool state_valid(unsigned long long w, unsigned tag) {
  return ((unsigned)(w >> 40) & 0xFFFFFFu) == tag && ((w >> 38) & 3ull) != 0ull;
}

// Scan item g (one warp). Returns false after a timeout (error bit set).
static __device__ bool scan_group(const MeshArgs& a, unsigned epoch, int g, unsigned long long base0) {
  const int lane = threadIdx.x & 31, i = g * kGroup + lane;
  const unsigned tag = epoch & 0xFFFFFFu;
  unsigned long long w = 0;
  for (int spins = 0;;) {
    if (i < a.n) w = ld_acquire_u64(&a.state[i]);
    if (__all_sync(0xffffffffu, i >= a.n || state_valid(w, tag))) break;
    if (++spins > a.spin_limit) {
      if (lane == 0) atomicOr(&a.ctl->err, ERR_TIMEOUT);
      return false;
    }
    __nanosleep(spins < 8 ? 32 : 128);
  }
  const unsigned total = i < a.n ? (unsigned)w : 0u;  // below 2^20; a group's below 2^25
  unsigned incl = total;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned v = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += v;
  }
  const unsigned sum = __shfl_sync(0xffffffffu, incl, 31);
  const unsigned long long excl = lookback(a.state + a.n, a.ctl, epoch, g, sum, a.spin_limit);
  __threadfence();  // the chunks' stores, seen by the acquire above, precede the upgrade
  if (i < a.n) {
    st_relaxed_u64(&a.state[i], pack_state(epoch, kFlagIncl, excl + incl));
    a.face_offsets[i] = base0 + excl + incl - total;
    if (i == a.n - 1) {
      const unsigned long long end = base0 + excl + incl;
      a.face_offsets[a.n] = end;
      if (end > a.cap) atomicOr(&a.ctl->err, ERR_CAPACITY);
    }
  }
  return true;
}

// Waits for chunk i's offset and total (one warp). Returns false after a timeout.
static __device__ bool chunk_offset(const MeshArgs& a, unsigned epoch, int i, unsigned long long& excl,
                                    unsigned& total) {
  const int lane = threadIdx.x & 31, idx = i - 1 + lane;  // lanes 0 and 1: chunks i - 1 and i
  const unsigned tag = epoch & 0xFFFFFFu;
  unsigned long long w = pack_state(epoch, kFlagIncl, 0);
  for (int spins = 0;;) {
    if (lane < 2 && idx >= 0) w = ld_acquire_u64(&a.state[idx]);
    const bool ready = state_valid(w, tag) && ((w >> 38) & 3ull) == kFlagIncl;
    if (__all_sync(0xffffffffu, ready)) break;
    if (++spins > a.spin_limit) {
      if (lane == 0) atomicOr(&a.ctl->err, ERR_TIMEOUT);
      return false;
    }
    __nanosleep(spins < 8 ? 32 : 256);
  }
  __syncwarp();
  const unsigned long long vmask = (1ull << 38) - 1;
  excl = __shfl_sync(0xffffffffu, w, 0) & vmask;
  total = (unsigned)((__shfl_sync(0xffffffffu, w, 1) & vmask) - excl);
  return true;
}

// ------------------------------------------------------------------------------------
// Records from face codes. A warp writes the records of up to 32 consecutive faces: lane l builds
// the record of its face in the warp's staging buffer, then the lanes copy the buffer to the
// output in 16-byte units, so that every store covers whole lines. Emission is short of warps
// as long as it waits for generation, so its time is the instructions of a batch: about 65
// this way. Building each 16-byte unit in the lane that stores it (no buffer; a shuffle, a
// table entry and the translation per unit) took 215, or 670 for instances, and sending the
// buffer with a TMA bulk copy waits about a microsecond for the copy to have read it.
// ------------------------------------------------------------------------------------

// CTA size of the emission grid, 32 warps an SM either way. From 32^3 on small CTAs fill the
// places that generation CTAs leave one by one (777 cave chunks 39.5 -> 37.8 us; the same at
// 16^3: 2000 chunks 51.6 -> 54.5 us). With 40 warps an SM (48 registers) the terrain batch took
// 37.3 instead of 33.5 us, with 24 warps 42.5.
template <int N>
__host__ __device__ constexpr int emit_threads() { return N <= 16 ? 256 : 128; }

// Translations of a chunk: local coordinate q_c of byte c of a face code -> world coordinate
// o_c + q_c as a float, rounded once. Origins below 2^23 - 64 in size take a shorter way with the
// same result: the byte in the low mantissa of 2^23 is exact, and so is every sum here.
struct Origin {
  int o[3];
  float f[3];  // (float)o - 2^23
  bool small;
  __device__ Origin(vox_chunk_coord c, int n) : o{c.x * n, c.y * n, c.z * n} {
    constexpr int kLim = (1 << 23) - 64;
    small = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      small = small && o[k] > -kLim && o[k] < kLim;
      f[k] = (float)o[k] - 8388608.0f;
    }
  }
  template <bool kSmall>
  __device__ __forceinline__ float at(uint32_t q, int k) const {
    return kSmall ? __uint_as_float(__byte_perm(q, 0x4B000000u, 0x7440u | (unsigned)k)) + f[k]
                  : (float)(o[k] + (int)((q >> (8 * k)) & 255u));
  }
};

// A store of records; kStream: as the first to leave L2, for outputs that do not fit there.
template <bool kStream, typename T>
__device__ __forceinline__ void put(T* p, T v) {
  if (kStream) __stcs(p, v);
  else *p = v;
}

// kPad: staging and table entries spread over the banks (41.2 -> 39.5 us on the cave chunks of
// 32^3; at 16^3 the shorter address arithmetic is worth more, 33.4 against 34.0 us).
template <int LAYOUT, bool kPad>
struct FaceStore;

template <bool kPad>
struct FaceStore<VOX_LAYOUT_VERTEX, kPad> {
  // Per direction 12 corner coordinates and the face; padded 80 bytes apart, so that the six
  // directions' entries lie in different banks.
  static constexpr int kEntry = kPad ? 5 : 4;  // 16-byte units
  static constexpr int kTableBytes = 6 * kEntry * 16;
  // A warp's buffer: 16-byte unit u at u, or padded at u + u / 24 (a gap behind every four
  // records), so that the eight lanes that store a unit together hit different banks.
  static constexpr int kBufBytes = (kWarpBatch * 6 + (kPad ? kWarpBatch / 4 : 0)) * 16;
  const float4* table;
  float4* buf;
  int lane;

  // Fills the table (all threads; the caller synchronises) and sets up the lane.
  __device__ void init(unsigned char* smem, unsigned char* bufs, const TablesDev& tab) {
    table = reinterpret_cast<const float4*>(smem);
    lane = threadIdx.x & 31;
    buf = reinterpret_cast<float4*>(bufs + (threadIdx.x >> 5) * kBufBytes);
    for (int i = threadIdx.x; i < 6 * 13; i += blockDim.x) {
      const int d = i / 13, k = i % 13;
      reinterpret_cast<float*>(smem)[d * kEntry * 4 + k] =
          k < 12 ? (&tab.corner[d][0][0])[k] : __uint_as_float(tab.slot[d]);
    }
  }

  // Writes nw faces (chunk-local indices first, first + 1, ...) at global face g.
  template <bool kSmall, bool kStream = false>
  __device__ __forceinline__ void batch(uint32_t q, int nw, uint32_t first, const Origin& org,
                                        unsigned long long g, void* out0, void* out1) const {
    const float4* C = table + (q >> 24) * (unsigned)kEntry;
    const float4 c0 = C[0], c1 = C[1], c2 = C[2];
    const float face = C[3].x;
    const float tx = org.at<kSmall>(q, 0), ty = org.at<kSmall>(q, 1), tz = org.at<kSmall>(q, 2);
    float4* v = buf + lane * 6 + (kPad ? lane >> 2 : 0);
    __syncwarp();  // the last batch has been copied out
    // position, tex coords (0,0) (1,0) (0,1) (1,1) (src/quad.rs:66-87) and face, 6 words a vertex
    v[0] = make_float4(c0.x + tx, c0.y + ty, c0.z + tz, 0.0f);
    v[1] = make_float4(0.0f, face, c0.w + tx, c1.x + ty);
    v[2] = make_float4(c1.y + tz, 1.0f, 0.0f, face);
    v[3] = make_float4(c1.z + tx, c1.w + ty, c2.x + tz, 0.0f);
    v[4] = make_float4(1.0f, face, c2.y + tx, c2.z + ty);
    v[5] = make_float4(c2.w + tz, 1.0f, 1.0f, face);
    __syncwarp();
    float4* o = reinterpret_cast<float4*>(reinterpret_cast<unsigned char*>(out0) + g * 96ull) + lane;
    const int units = nw * 6;
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (32 * k + lane < units) put<kStream>(o + 32 * k, buf[32 * k + lane + (kPad ? (32 * k + lane) / 24 : 0)]);
    // indices 4 f + {0, 2, 1, 3, 1, 2}: 8-byte pair j of face u / 3
    uint2* x = reinterpret_cast<uint2*>(reinterpret_cast<unsigned char*>(out1) + g * 24ull) + lane;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int u = 32 * k + lane, f = u / 3, j = u - 3 * f;
      const uint32_t b = 4u * (first + (uint32_t)f);
      if (f < nw) put<kStream>(x + 32 * k, make_uint2(b + (j == 0 ? 0u : 1u), b + (j == 1 ? 3u : 2u)));
    }
  }
};

template <bool kPad>
struct FaceStore<VOX_LAYOUT_INSTANCED, kPad> {
  static constexpr int kTableBytes = 6 * 80;  // per direction the 17 words of a record
  static constexpr int kBufBytes = kWarpBatch * 68;
  const float* table;
  float* buf;
  int lane;

  __device__ void init(unsigned char* smem, unsigned char* bufs, const TablesDev& tab) {
    table = reinterpret_cast<const float*>(smem);
    lane = threadIdx.x & 31;
    buf = reinterpret_cast<float*>(bufs + (threadIdx.x >> 5) * kBufBytes);
    for (int i = threadIdx.x; i < 6 * 17; i += blockDim.x) {
      const int d = i / 17, w = i % 17, c = w >> 2, r = w & 3;
      float v;
      if (w == 16) v = __uint_as_float(tab.tex[d]);
      else if (c == 3) v = 1.0f;
      else v = r == 3 ? tab.row3[d][c] : tab.part[d][r][c];
      reinterpret_cast<float*>(smem)[d * 20 + w] = v;
    }
  }

  template <bool kSmall, bool kStream = false>
  __device__ __forceinline__ void batch(uint32_t q, int nw, uint32_t, const Origin& org,
                                        unsigned long long g, void* out0, void*) const {
    const float4* M = reinterpret_cast<const float4*>(table + (q >> 24) * 20u);
    const float tx = org.at<kSmall>(q, 0), ty = org.at<kSmall>(q, 1), tz = org.at<kSmall>(q, 2);
    const float z0 = tx * 0.0f, z1 = ty * 0.0f, z2 = tz * 0.0f;
    const float tex = table[(q >> 24) * 20u + 16u];
    float* v = buf + lane * 17;
    __syncwarp();  // the last batch has been copied out
#pragma unroll
    for (int c = 0; c < 3; ++c) {  // column c of the matrix: t_r * 0 decides the sign of a zero
      const float4 m = M[c];
      v[4 * c + 0] = m.x + z0;
      v[4 * c + 1] = m.y + z1;
      v[4 * c + 2] = m.z + z2;
      v[4 * c + 3] = m.w;
    }
    v[12] = tx;
    v[13] = ty;
    v[14] = tz;
    v[15] = 1.0f;
    v[16] = tex;
    __syncwarp();
    unsigned char* o = reinterpret_cast<unsigned char*>(out0) + g * 68ull;
    if (((unsigned)g & 3u) == 0u) {  // 16-byte units, and the words of the last up to 3 faces
      const int units = nw * 17 >> 2;
#pragma unroll
      for (int k = 0; k < 5; ++k)
        if (32 * k + lane < units)
          put<kStream>(reinterpret_cast<float4*>(o) + 32 * k + lane, reinterpret_cast<const float4*>(buf)[32 * k + lane]);
      if (lane < (nw * 17 & 3))
        put<kStream>(reinterpret_cast<float*>(o) + 4 * units + lane, buf[4 * units + lane]);
    } else {
      for (int k = lane; k < nw * 17; k += 32) put<kStream>(reinterpret_cast<float*>(o) + k, buf[k]);
    }
  }
};

// A chunk without a list is emitted by compaction from its spilled state, in runs of run_groups()
// groups of 32 elements that warps take one at a time. Such chunks are dense, and a batch of them is
// bound by HBM writes and by its last wave: 2000 chunks of 16^3 in four parts are 1.6 waves of warps,
// which left a third of the warps idle in the second. So the warps of a chunk's parts share its runs,
// and a warp that has no part left, and has met such chunks, looks for others with runs left: chunk
// open_chunk() from `from` on, in steps of 32 counts (done: how many are behind it), or -1. Their
// records leave L2 first (__stcs), as their batches do not fit there. us a batch, one part a warp with
// plain stores -> now (one launch before the lists): random voxels from a pool, 2000 chunks of 16^3
// 332 -> 259 (269), 400 of 32^3 431 -> 382 (385); white-noise columns, 2000 of 16^3 171 -> 137 (138,
// with the shorter list below), 400 of 32^3 237 -> 210 (209); white-noise density, 2000 of 16^3 329 ->
// 288 (312), 400 of 32^3 515 -> 446 (473).
template <int N>
__host__ __device__ constexpr int run_groups() { return N <= 16 ? 4 : 8; }

static __device__ int open_chunk(const MeshArgs& a, int from, unsigned& done, unsigned turn) {
  const int lane = threadIdx.x & 31;
  for (; done < (unsigned)a.n && ld_relaxed_u32(&a.ctl->open) != 0u; done += 32u) {
    const long long at = (long long)from + done + lane;
    const int i = (int)(at < a.n ? at : at - a.n);
    const unsigned left =
        __ballot_sync(0xffffffffu, done + lane < (unsigned)a.n && ld_relaxed_u32(a.counts + i) < kTaken);
    if (left == 0u) continue;
    const unsigned ahead = left & (0xffffffffu << (turn & 31u));  // (warps begin at different ones)
    return __shfl_sync(0xffffffffu, i, __ffs(ahead != 0u ? ahead : left) - 1);
  }
  return -1;
}

template <int N, int LAYOUT>
__global__ void __launch_bounds__(emit_threads<N>(), 1024 / emit_threads<N>())
k_emit_lists(const __grid_constant__ MeshArgs a, const __grid_constant__ TablesDev tab) {
  using S = ListSlot<N>;
  constexpr unsigned kLine = line_faces<LAYOUT>();
  constexpr int kEmitThreads = emit_threads<N>();
  using Store = FaceStore<LAYOUT, (N > 16)>;
  __shared__ __align__(16) unsigned char s_table[Store::kTableBytes];
  __shared__ __align__(16) unsigned char s_bufs[kEmitThreads / 32 * Store::kBufBytes];
  __shared__ uint32_t s_lists[kEmitThreads / 32 * kWarpFaces];
  __shared__ unsigned long long s_base0;
  __shared__ unsigned s_epoch;
  pdl_trigger();  // (a launch behind this one waits for its end before it touches anything)
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  Store store;
  store.init(s_table, s_bufs, tab);
  if (t == 0) {
    s_epoch = ld_relaxed_u32(&a.ctl->epoch);
    s_base0 = launch_base(a);
  }
  __syncthreads();
  const unsigned epoch = s_epoch;
  const unsigned long long base0 = s_base0;
  bool ok = true;
  if (warp == 0) {  // scan items, in ticket order: a running warp holds every smaller ticket
    const unsigned scans = ((unsigned)a.n + kGroup - 1u) / kGroup;
    while (ok) {
      unsigned g = 0;
      if (lane == 0) g = atomicAdd(&a.ctl->next_scan, 1u);
      g = __shfl_sync(0xffffffffu, g, 0);
      if (g >= scans) break;
      ok = scan_group(a, epoch, (int)g, base0);
    }
  }
  // Emission items: part k % 2^split of chunk k >> split, dealt out to the warps of the grid in
  // chunk order; then runs of chunks without a list.
  // (32-bit: a chunk's scratch is more than 2 KB, so no launch has 2^32 items.)
  const unsigned parts = 1u << a.split;
  const unsigned items = (unsigned)a.n << a.split, stride = gridDim.x * (kEmitThreads / 32);
  unsigned k = blockIdx.x * (kEmitThreads / 32) + (unsigned)warp;
  int met = -1;  // the last chunk without a list that this warp has met
  unsigned done = 0;
  while (ok) {
    int i = (int)(k >> a.split);
    const unsigned part = k & (parts - 1u);
    const bool own = k < items;
    if (own) {
      k += stride;
    } else {
      if (met < 0) break;
      i = open_chunk(a, met, done, k);
      if (i < 0) break;
    }
    const vox_chunk_coord c = a.coords[i];
    unsigned long long g0;
    unsigned total;
    // (from 32^3 on epoch and base are read again for each item, which spares the registers: the
    // cave rebuild of 777 chunks 35.6 -> 35.0 us; at 16^3 it costs as much)
    ok = chunk_offset(a, N > 16 ? *const_cast<volatile unsigned*>(&s_epoch) : epoch, i, g0, total);
    if (!ok || total == 0u) continue;
    g0 += N > 16 ? *const_cast<volatile unsigned long long*>(&s_base0) : base0;
    const Origin org(c, N);
    auto send = [&](uint32_t q, int nw, uint32_t first, unsigned long long g) {
      if (org.small) store.template batch<true>(q, nw, first, org, g, a.out0, a.out1);
      else store.template batch<false>(q, nw, first, org, g, a.out0, a.out1);
    };
    unsigned char* src = reinterpret_cast<unsigned char*>(a.scratch) + (unsigned long long)i * S::kBytes;
    if (total <= S::kCap) {
      if (!own) continue;  // (its count was not there yet; it is now, and not open)
      // the output lines that the chunk touches, cut evenly over the parts
      const uint32_t* codes = reinterpret_cast<const uint32_t*>(src);
      const unsigned phase = (unsigned)(g0 & (unsigned long long)(kLine - 1u));
      const unsigned lines = (phase + total + kLine - 1u) / kLine;
      const unsigned la = (unsigned)(((unsigned long long)lines * part) >> a.split);
      const unsigned lb = (unsigned)(((unsigned long long)lines * (part + 1u)) >> a.split);
      if (la == lb) continue;
      const int lo = la == 0u ? 0 : (int)(la * kLine - phase);
      const int hi = (int)min(total, lb * kLine - phase);
      int cnt = batch_faces<LAYOUT>(g0 + (unsigned)lo, hi - lo);
      uint32_t q = lane < cnt ? __ldcg(codes + lo + lane) : 0u;
      for (int r = lo; r < hi;) {
        const unsigned long long g = g0 + (unsigned)r;
        const int r2 = r + cnt;
        const int cnt2 = r2 < hi ? batch_faces<LAYOUT>(g0 + (unsigned)r2, hi - r2) : 0;
        const uint32_t q2 = lane < cnt2 ? __ldcg(codes + r2 + lane) : 0u;  // the next batch
        const int nw = faces_in(g, cnt, a.cap);
        if (nw == 0) break;
        send(q, nw, (uint32_t)r, g);
        r = r2;
        cnt = cnt2;
        q = q2;
      }
    } else {
      met = i;
      ChunkSmem<N, LAYOUT> d;
      d.occ = reinterpret_cast<typename Shape<N>::RowT*>(src);
      d.halo = reinterpret_cast<typename Shape<N>::RowT*>(src + S::P::kOcc);
      d.rows = reinterpret_cast<uint32_t*>(src + S::P::kOcc + S::P::kHalo);
      d.nz = reinterpret_cast<uint16_t*>(src + S::kNzOff);
      d.vlist = reinterpret_cast<uint16_t*>(src + S::kVlOff);
      d.misc = reinterpret_cast<int*>(src + S::kMiscOff);
      d.lists = s_lists;
      const int elems = emit_elems(d);
      const unsigned runs = (unsigned)(elems + 32 * run_groups<N>() - 1) / (32u * run_groups<N>());
      bool took = false;
      for (;;) {
        unsigned run = 0;
        if (lane == 0) {
          run = atomicAdd(a.counts + i, 1u);
          if (run == runs - 1u) {
            atomicOr(a.counts + i, kTaken);
            atomicSub(&a.ctl->open, 1u);
          }
        }
        run = __shfl_sync(0xffffffffu, run, 0);
        if (run >= runs) {
          if (!own && !took) done += 32u;  // all taken meanwhile: go on behind it
          break;
        }
        took = true;
        const int lo = (int)run * 32 * run_groups<N>();
        emit_runs<N, LAYOUT>(d, lo, min(elems, lo + 32 * run_groups<N>()), 0, 1, g0,
                             [&](const uint32_t* list, int nf, uint32_t first) {
          for (int r = 0, cnt = 0; r < nf; r += cnt) {
            const unsigned long long g = g0 + first + (unsigned)r;
            cnt = batch_faces<LAYOUT>(g, nf - r);
            const int nw = faces_in(g, cnt, a.cap);
            if (nw == 0) continue;
            const uint32_t q = lane < nw ? list[r + lane] : 0u;
            store.template batch<false, true>(q, nw, first + (uint32_t)r, org, g, a.out0, a.out1);
          }
          __syncwarp();
        });
      }
    }
  }
  // The last CTA to finish resets the scan tickets and advances the epoch: every chunk of the
  // launch is published and emitted by then.
  __syncthreads();
  if (t == 0) {
    __threadfence();
    if (atomicAdd(&a.ctl->done, 1u) == gridDim.x - 1u) {
      a.ctl->done = 0u;
      a.ctl->next_scan = 0u;
      a.ctl->epoch = epoch + 1u;
    }
  }
  // the generation launch has completed too before this one does
  pdl_wait();
}

// ------------------------------------------------------------------------------------
// Plain per-chunk mesher: one chunk, one launch (no queue, no look-back). One CTA used to do
// it all, so a chunk's emission ran on one SM of 152. Now single_ctas CTAs each load and count
// the whole chunk (redundant, but the GPU has nothing else to do and the counts need no
// exchange) and emit their part of it: a few groups of 32 face voxels a warp. A call on a
// terrain chunk of 64^3 238 -> 17.8 us, a cave chunk of 64^3 as instances 139 -> 22.4 us; from
// 32^3 down a call is bound by the caller (16 us through Python either way; waiting for one
// chunk of 32^3 takes about 5 us less).
// ------------------------------------------------------------------------------------

template <int N>
__host__ __device__ constexpr int single_threads() {
  return N == 8 ? 64 : (N == 16 ? 256 : (N == 32 ? 512 : 1024));
}
template <int N>
__host__ __device__ constexpr int single_ctas() { return N == 8 ? 1 : (N == 16 ? 2 : (N == 32 ? 8 : 64)); }
template <int N, int LAYOUT>
__host__ __device__ constexpr int single_smem() {
  return ListSmem<N, GM_OCC>::kBytes +
         single_threads<N>() / 32 * (kWarpFaces * 4 + FaceStore<LAYOUT, false>::kBufBytes);
}

template <int N, int LAYOUT>
__global__ void __launch_bounds__(single_threads<N>())
k_mesh_single(const __grid_constant__ MeshArgs a, const __grid_constant__ TablesDev tab) {
  using M = ListSmem<N, GM_OCC>;
  constexpr int T = single_threads<N>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(16) unsigned char s_table[FaceStore<LAYOUT, false>::kTableBytes];
  ChunkSmem<N, VOX_LAYOUT_VERTEX> s;
  M::carve(s, smem_raw);
  s.lists = reinterpret_cast<uint32_t*>(smem_raw + M::kBytes);
  const int t = threadIdx.x, lane = t & 31;
  FaceStore<LAYOUT, false> store;
  store.init(s_table, smem_raw + M::kBytes + T / 32 * kWarpFaces * 4, tab);
  pdl_trigger();
  pdl_wait();
  unsigned use = 0;
  for (int d = 0; d < 6; ++d)
    if (a.occ_nbr[d] && (d < 4 || a.full6)) use |= 1u << d;
  load_chunk<N, VOX_LAYOUT_VERTEX, T>(s, a.occ_self, a.occ_nbr, use);
  s.stage = smem_raw + M::kRowsOff + M::kLists;
  const uint32_t total = count_and_scan<N, VOX_LAYOUT_VERTEX, T>(s);
  if (blockIdx.x == 0 && t == 0) {
    a.face_offsets[0] = total;
    if ((unsigned long long)total > a.cap) atomicOr(&a.ctl->err, ERR_CAPACITY);
  }
  const Origin org(a.coord_single, N);
  emit_runs<N, LAYOUT>(s, 0, emit_elems(s), (int)blockIdx.x * (T / 32) + (t >> 5),
                       (int)gridDim.x * (T / 32), 0ull, [&](const uint32_t* list, int nf, uint32_t first) {
    for (int r = 0, cnt = 0; r < nf; r += cnt) {
      const unsigned long long g = first + (unsigned)r;
      cnt = batch_faces<LAYOUT>(g, nf - r);
      const int nw = faces_in(g, cnt, a.cap);
      if (nw == 0) continue;
      const uint32_t q = lane < nw ? list[r + lane] : 0u;
      if (org.small) store.template batch<true>(q, nw, (uint32_t)g, org, g, a.out0, a.out1);
      else store.template batch<false>(q, nw, (uint32_t)g, org, g, a.out0, a.out1);
    }
    __syncwarp();
  });
}

}  // namespace vox
