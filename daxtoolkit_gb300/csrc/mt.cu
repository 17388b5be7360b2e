// Marching tetrahedra on an unstructured tetrahedral grid
// (dax/worklet/MarchingTetrahedra.h:49-161 driven by DispatcherMapCell and
// DispatcherGenerateInterpolatedCells).
//
// Layout: points float[P][3], field float[P], connectivity int32[C][4]
// (dax::cont::UnstructuredGrid<CellTagTetrahedron>), all caller-owned.
//
//   count   K1 k_mt_count: the case byte of every cell (4 field gathers
//           each), the triangle totals of every chunk of kMtChunk cells and
//           of every tile of kMtTile cells;
//           K2 k_mt_tile_scan: exclusive tile offsets and the total T.
//   emit    K3 k_mt_emit: one warp per chunk of kMtChunk cells, chunks
//           without triangles skipped; each lane takes 16 consecutive cells
//           (one 16-byte load of their cases) and a warp scan of the lanes'
//           triangle counts gives every cell its first output triangle; the
//           case's TriTable edges, lower point id
//           first, weight (iso - f[A]) / (f[B] - f[A]) and Lerp of the two
//           points (MarchingTetrahedra.h:117-161, GenerateWorklets.h:79-92).
//           Unmerged it writes vertices, connectivity and records directly;
//           merged it writes one key (A, B) per record.
//   merge   the reference's ResolveCoordinates on the device adapter's own
//           primitives: Sort and Unique of the keys (radix sort, 32- or
//           64-bit keys as P needs), LowerBounds of every record key
//           (k_mt_merged_conn), and the unique edges' vertices
//           (k_mt_merged_verts).
//
// Point ids outside [0, P) are not dereferenced: the cell counts as case 0
// and Info.error gets kErrBadIndex.
#include "common.cuh"
#include "kernels.cuh"
#include "mc_case.cuh"
#include "mt_tables.h"
#include "tma.cuh"

namespace daxgb {

// The tables are compile-time constants folded into instructions: lanes of a
// warp index them with different cases, which a constant-memory table would
// serve one address at a time.
constexpr uint32_t kMtWords[16] = DAX_GB300_MT_CASE_WORDS;
__constant__ uint32_t c_mt_case[16] = DAX_GB300_MT_CASE_WORDS;  // copied to shared memory

// NumFaces of case c in bits 2c .. 2c+1.
constexpr uint32_t mt_face_bits() {
  uint32_t b = 0;
  for (int c = 0; c < 16; ++c) b |= (kMtWords[c] >> 28) << (2 * c);
  return b;
}
constexpr uint32_t kMtFaceBits = mt_face_bits();

// cellVertEdges (MarchingTetrahedra.h:126-129), byte e = edge e: low nibble
// first corner, high nibble second.
constexpr unsigned long long kTetEdges = 0x231303022110ull;

__device__ __forceinline__ int mt_faces(int cs) { return (int)((kMtFaceBits >> (2 * cs)) & 3u); }

// GetTetrahedronClassification (MarchingTetrahedra.h:36-46).
__device__ __forceinline__ int mt_classify(const float v[4], float iso) {
  return (v[0] > iso ? 1 : 0) | (v[1] > iso ? 2 : 0) | (v[2] > iso ? 4 : 0) | (v[3] > iso ? 8 : 0);
}

// a[k] for k in 0..3 by selects, so the four values stay in registers.
template <typename T>
__device__ __forceinline__ T pick4(const T a[4], int k) {
  return k == 0 ? a[0] : (k == 1 ? a[1] : (k == 2 ? a[2] : a[3]));
}

// Point ids of cell c; false when one lies outside [0, P).
template <bool VEC>
__device__ __forceinline__ bool load_tet(const int32_t* __restrict__ conn, long long c,
                                         long long P, int id[4]) {
  if (VEC) {
    const int4 q = __ldg(reinterpret_cast<const int4*>(conn) + c);
    id[0] = q.x;
    id[1] = q.y;
    id[2] = q.z;
    id[3] = q.w;
  } else {
#pragma unroll
    for (int n = 0; n < 4; ++n) id[n] = __ldg(conn + 4 * c + n);
  }
  bool ok = true;
#pragma unroll
  for (int n = 0; n < 4; ++n) ok = ok && id[n] >= 0 && (long long)id[n] < P;
  return ok;
}

// Warp w of a tile takes the kMtChunk consecutive cells of chunk 8 * tile + w;
// the chunk's and the tile's triangle totals are stored.
//
// Bound by the connectivity's bytes (16 a cell): 83 million cells take 222 us,
// 1.44 GB at 6.5 TB/s.  A bulk copy brings the ids of kMtGroup cells into the
// warp's buffer, and as soon as they are in registers the next group's is issued,
// also over the end of a tile.  A lane takes kMtRun consecutive cells: in a mesh of
// tetrahedralized voxels, five cells each, the lanes then gather the same corner
// of consecutive voxels, one or two lines a load.  The twenty ids of a lane are
// checked by one unsigned maximum and their gathers issued together; a group that
// reaches past the end or lists a bad id goes cell by cell.
//
// If the lanes' runs lie apart, more than half of them over 32 ids from the run of
// two lanes before (neighbouring voxels list their corners in other orders), a
// lane takes one corner of eight cells instead: L1 looks up a line at a time, and
// the corners of a cell, asked for together, share lines where the points are in
// order, whatever the order of the cells.  A vote on the values is then eight
// cells' cases.  (A corner of 32 cells a load took 1240 us, count and scan, for
// cells in no order, now 995; voxels in random order 478 and 427.)
//
// Gathers in no order also need L1 as room for the lines on their way: the buffers
// of four blocks are held below 100 KB.  With 132 KB, 1057 and 454 us; points in no
// order either, 1290 and now 1203.
//
// (A cell a lane, with loads straight from global memory: 301 us in order, 1082 for
// cells and 552 for voxels in random order, 1211 for cells and points in none.
// Runs with a check a cell were issue bound, 81 instructions a row of 32 cells:
// 292.  Two buffers a warp took as long, but left the gathers half the L1: 2040 us
// for cells in no order.)
//
// Connectivity that is not 16-byte aligned is copied by plain loads: 387 us.
constexpr int kMtRun = 5;
constexpr int kMtGroup = 32 * kMtRun;
constexpr int kMtGroups = kMtChunk / kMtGroup;  // whole groups a chunk; the rest a cell a lane
static_assert(kMtGroups == 3 && kMtChunk - kMtGroups * kMtGroup == 32,
              "four groups a tile, the last of one cell a lane");

template <bool VEC>
__global__ void __launch_bounds__(kMtThreads, VEC ? 4 : 5)
    k_mt_count(const int32_t* __restrict__ conn, long long C, const float* __restrict__ f,
               long long P, float iso, uint8_t* __restrict__ cases, unsigned* __restrict__ tile_tot,
               unsigned* __restrict__ chunk_tot, Info* info, int tiles, unsigned polls) {
  constexpr int kWarps = kMtThreads / 32;
  __shared__ unsigned s_warp[2][kWarps];
  __shared__ __align__(16) int4 s_ids[kWarps][kMtGroup];
  __shared__ __align__(16) uint8_t s_case[kWarps][kMtGroups * kMtGroup];
  __shared__ uint64_t s_bar[kWarps];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint8_t* const cs_of = s_case[wid];
  if (VEC && lane == 0) {
    mbar_init(&s_bar[wid], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  bool bad = false, late = false;  // late: a copy did not land in time, and no other is issued
  int awaited = 0;                 // its group
  // an id is a point if it is below this as an unsigned: negative ones are not
  const unsigned points = (unsigned)min(P, 1ll << 31);
  unsigned long long policy = 0;
  if (VEC) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  // the ids of group g of a tile's chunk into the warp's buffer
  auto copy = [&](long long tile, int g) {
    if (tile >= tiles || late) return;
    const long long c = tile * kMtTile + (long long)wid * kMtChunk + g * kMtGroup;
    const int n = (int)min((long long)(g < kMtGroups ? kMtGroup : 32), max(C - c, 0ll));
    int4* dst = s_ids[wid];
    if (VEC) {
      if (lane == 0) {
        uint64_t* bar = &s_bar[wid];
        if (n > 0) {
          mbar_arrive_tx(bar, 16u * n);
          bulk_load(dst, conn + 4 * c, 16u * n, bar, policy);
        } else {
          mbar_arrive(bar);
        }
      }
    } else {
      for (int i = lane; i < n; i += 32) {
        const int32_t* q = conn + 4 * (c + i);
        dst[i] = make_int4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
      }
    }
  };
  auto landed = [&](int g) {  // four groups a tile: group g is of parity g & 1
    if (VEC && !late) {
      Spin sp(polls);
      bool ok = polls > 0 && mbar_test(&s_bar[wid], g & 1);
      while (!ok && sp.more()) ok = mbar_test(&s_bar[wid], g & 1);
      late = __any_sync(kFull, !ok);
      awaited = g;
    }
    __syncwarp();
  };
  // a cell whose ids need not be points
  auto classify = [&](const int4& q, bool& is) -> int {
    const bool ok = q.x >= 0 && (long long)q.x < P && q.y >= 0 && (long long)q.y < P && q.z >= 0 &&
                    (long long)q.z < P && q.w >= 0 && (long long)q.w < P;
    is = is && ok;
    if (!ok) return 0;
    const float v[4] = {__ldg(f + q.x), __ldg(f + q.y), __ldg(f + q.z), __ldg(f + q.w)};
    return mt_classify(v, iso);
  };
  copy(blockIdx.x, 0);
  int flip = 0;
#pragma unroll 1
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x, flip ^= 1) {
    unsigned sum = 0;
    const long long cb = tile * kMtTile + (long long)wid * kMtChunk;
#pragma unroll 1
    for (int g = 0; g < kMtGroups; ++g) {
      landed(g);
      if (late) break;
      const int4* ids = s_ids[wid];
      uint8_t* const out = cs_of + g * kMtGroup;
      const long long cg = cb + g * kMtGroup;
      int4 q[kMtRun];
      q[0] = ids[kMtRun * lane];
      const int before = __shfl_up_sync(kFull, q[0].x, 2);
      const bool apart =
          __popc(__ballot_sync(kFull, (unsigned)q[0].x - (unsigned)before + 32u > 64u)) > 16;
      if (apart) {
#pragma unroll
        for (int i = 0; i < kMtRun; ++i) {
          const int* const w = reinterpret_cast<const int*>(ids) + 128 * i + lane;
          q[i] = make_int4(w[0], w[32], w[64], w[96]);
        }
      } else {
#pragma unroll
        for (int i = 1; i < kMtRun; ++i) q[i] = ids[kMtRun * lane + i];
      }
      unsigned top = 0;
#pragma unroll
      for (int i = 0; i < kMtRun; ++i)
        top = max(top, max(max((unsigned)q[i].x, (unsigned)q[i].y),
                           max((unsigned)q[i].z, (unsigned)q[i].w)));
      // Whether every id is a point of the mesh.  The vote takes each lane's loaded
      // values, so all of the loads have returned before the buffer is filled
      // again (a barrier alone lets the copy pass loads that still wait); the fence
      // orders them before the copy's writes.
      const bool fast = __all_sync(kFull, top < points && cg + kMtGroup <= C);
      if (!fast) {
        bool is = true;
#pragma unroll 1
        for (int i = lane; i < kMtGroup; i += 32) {
          const int cs = cg + i < C ? classify(ids[i], is) : 0;
          out[i] = (uint8_t)cs;
          sum += (unsigned)mt_faces(cs);
        }
        bad = __any_sync(kFull, !is) || bad;  // as above, every load has returned
      }
      if (VEC) fence_proxy_async();
      __syncwarp();
      copy(tile, g + 1);
      if (!fast) continue;
      float v[kMtRun][4];
#pragma unroll
      for (int i = 0; i < kMtRun; ++i) {
        v[i][0] = __ldg(f + q[i].x);
        v[i][1] = __ldg(f + q[i].y);
        v[i][2] = __ldg(f + q[i].z);
        v[i][3] = __ldg(f + q[i].w);
      }
      if (apart) {
        // a vote is eight cells' cases: cell 32 i + lane is the lane's four bits of
        // vote lane / 8
#pragma unroll
        for (int i = 0; i < kMtRun; ++i) {
          unsigned b[4];
#pragma unroll
          for (int n = 0; n < 4; ++n) b[n] = __ballot_sync(kFull, v[i][n] > iso);
          const unsigned lo = lane & 8 ? b[1] : b[0], hi = lane & 8 ? b[3] : b[2];
          const int cs = (int)((lane & 16 ? hi : lo) >> (4 * (lane & 7)) & 15u);
          out[32 * i + lane] = (uint8_t)cs;
          sum += (unsigned)mt_faces(cs);
        }
      } else {
#pragma unroll
        for (int i = 0; i < kMtRun; ++i) {
          const int cs = mt_classify(v[i], iso);
          out[kMtRun * lane + i] = (uint8_t)cs;
          sum += (unsigned)mt_faces(cs);
        }
      }
    }
    landed(kMtGroups);
    if (!late) {
      const int at = kMtGroups * kMtGroup + lane;
      const int4 q = s_ids[wid][lane];
      bool is = (unsigned)q.x < points && (unsigned)q.y < points && (unsigned)q.z < points &&
                (unsigned)q.w < points;
      bad = __any_sync(kFull, cb + at < C && !is) || bad;  // as above, every load has returned
      if (VEC) fence_proxy_async();
      __syncwarp();
      copy(tile + gridDim.x, 0);
      is = is && cb + at < C;
      int cs = 0;
      if (is) {
        const float v[4] = {__ldg(f + q.x), __ldg(f + q.y), __ldg(f + q.z), __ldg(f + q.w)};
        cs = mt_classify(v, iso);
      }
      if (cb + at < C) cases[cb + at] = (uint8_t)cs;
      sum += (unsigned)mt_faces(cs);
    }
    __syncwarp();
    // the chunk's cases in whole lines
    constexpr int kStaged = kMtGroups * kMtGroup;
    if (cb + kStaged <= C && (reinterpret_cast<uintptr_t>(cases) & 15) == 0) {
      if (lane < kStaged / 16)
        reinterpret_cast<uint4*>(cases + cb)[lane] = reinterpret_cast<const uint4*>(cs_of)[lane];
    } else {
      for (int i = lane; i < kStaged && cb + i < C; i += 32) cases[cb + i] = cs_of[i];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(kFull, sum, d);
    if (lane == 0) {
      chunk_tot[tile * (kMtTile / kMtChunk) + wid] = sum;
      s_warp[flip][wid] = sum;
    }
    __syncthreads();  // one a tile: s_warp's other row is written before the next one
    if (threadIdx.x == 0) {
      unsigned t = 0;
      for (int w = 0; w < kWarps; ++w) t += s_warp[flip][w];
      tile_tot[tile] = t;
    }
  }
  if (bad) atomicOr(&info->error, kErrBadIndex);
  if (late) {
    atomicOr(&info->error, kErrTimeout);
    Spin sp;
    while (!mbar_test(&s_bar[wid], awaited & 1) && sp.more()) {
    }
  }
}

// One block: exclusive offsets of the tile totals (tile_off[tiles] = T) and
// the total into Info; more than 2^31 - 1 vertex records is an overflow.
// Warp w sums its own contiguous run of tiles, 32 at a time, the block scans
// the 32 run totals, then every warp scans its run.  (A run a thread, whose
// loads lay 80 bytes apart, took 19 us for 20 thousand tiles; 12 now.)
__global__ void __launch_bounds__(1024) k_mt_tile_scan(const unsigned* __restrict__ tile_tot,
                                                       int tiles,
                                                       unsigned long long* __restrict__ tile_off,
                                                       Info* info) {
  __shared__ unsigned long long s_warp[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int per = (tiles + 1023) / 1024 * 32;  // tiles a warp
  const int b = wid * per, e = min(b + per, tiles);
  unsigned long long v = 0;
#pragma unroll 4
  for (int i = b + lane; i < e; i += 32) v += tile_tot[i];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(kFull, v, d);
  if (lane == 0) s_warp[wid] = v;
  __syncthreads();
  unsigned long long run = 0, all = 0;
  for (int w = 0; w < 32; ++w) {
    const unsigned long long t = s_warp[w];
    run += w < wid ? t : 0ull;
    all += t;
  }
#pragma unroll 4
  for (int i0 = b; i0 < e; i0 += 32) {
    const int i = i0 + lane;
    const unsigned long long t = i < e ? tile_tot[i] : 0u;
    unsigned long long x = t;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned long long y = __shfl_up_sync(kFull, x, d);
      if (lane >= d) x += y;
    }
    if (i < e) tile_off[i] = run + x - t;
    run += __shfl_sync(kFull, x, 31);
  }
  if (threadIdx.x == 0) {
    tile_off[tiles] = all;
    info->total_a = (long long)all;
    info->total_b = 0;
    if (3ull * all > 2147483647ull) atomicOr(&info->error, kErrOverflow);
  }
}

// Output sinks of the emit pass.
struct MtOut {
  float* verts;       // unmerged: [3T][3]
  int32_t* tconn;     // unmerged: [3T]
  int32_t* ra;        // unmerged records (optional)
  int32_t* rb;
  float* rw;
  void* keys;         // merged: [3T] keys (A << kbits) | B
  int kbits;
  bool wide;          // 64-bit keys
  long long vcap, tcap;
};

// One warp per chunk; bound by latency: a chunk's totals, its cases, the ids of
// its cells with triangles, then their values follow each other.  So a warp looks
// up 32 chunk totals at once and the earlier totals of a tile in one load (a total
// at a time left 33 loads one behind the other), and a listed cell is 32 bits,
// which with six blocks an SM gives half as many warps again: the keys of 256^3
// points, 64 us before, take 49; the merged call went from 604 to 584 us, the
// unmerged one from 387 to 369.
// (Six spill 52 bytes in the unmerged form; eight, which spill in both, took 579
// and 367.)
template <bool VEC, bool KEYS>
__global__ void __launch_bounds__(kMtThreads, 6) k_mt_emit(const float* __restrict__ pts,
                                                        const int32_t* __restrict__ conn,
                                                        long long C,
                                                        const float* __restrict__ f, long long P,
                                                        float iso,
                                                        const uint8_t* __restrict__ cases,
                                                        const unsigned long long* __restrict__ tile_off,
                                                        const unsigned* __restrict__ chunk_tot,
                                                        Info* info, MtOut o, long long chunks) {
  // per warp: the chunk's cells with triangles, cell in chunk | case << 12 |
  // first triangle, relative to the chunk's, << 16
  __shared__ uint32_t s_act[kMtThreads / 32][kMtChunk];
  __shared__ uint32_t s_case[16];
  if (threadIdx.x < 16) s_case[threadIdx.x] = c_mt_case[threadIdx.x];
  __syncthreads();
  // nothing is written when an earlier pass failed or the outputs are short
  const long long T = info->total_a;
  if (info->error) return;
  if (!KEYS && (T > o.tcap || 3 * T > o.vcap)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&info->error, kErrCapacity);
    return;
  }
  constexpr int kPerTile = kMtTile / kMtChunk;
  static_assert(kPerTile <= 32 && kMtChunk <= 4096, "a chunk's entry and its tile's totals");
  const int lane = threadIdx.x & 31;
  uint32_t* act = s_act[threadIdx.x >> 5];
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  // The warp's next 32 chunks are looked up at once, a chunk a lane, and those
  // with triangles taken one after the other.
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  unsigned todo = 0;
  for (long long next = warp0, base = 0;;) {
    if (todo == 0) {
      if (next >= chunks) break;
      const long long mych = next + lane * nwarps;
      todo = __ballot_sync(kFull, mych < chunks && __ldg(chunk_tot + mych) != 0);
      base = next;
      next += 32 * nwarps;
      continue;
    }
    const long long ch = base + (__ffs(todo) - 1) * nwarps;
    todo &= todo - 1;
    // the chunk's first triangle: its tile's offset plus the earlier chunks
    const long long tile = ch / kPerTile;
    const unsigned before = lane < (int)(ch - tile * kPerTile)
                                ? __ldg(chunk_tot + tile * kPerTile + lane) : 0u;
    const unsigned long long t0 = tile_off[tile] + __reduce_add_sync(kFull, before);
    // lane l reads the cases of the kMtPerLane consecutive cells c0 .. c0 + 15
    const long long cbase = ch * kMtChunk;
    const long long c0 = cbase + (long long)lane * kMtPerLane;
    uint32_t cw[kMtPerLane / 4];
    if (c0 + kMtPerLane <= C) {
      const uint4 q = __ldg(reinterpret_cast<const uint4*>(cases + c0));
      cw[0] = q.x;
      cw[1] = q.y;
      cw[2] = q.z;
      cw[3] = q.w;
    } else {
#pragma unroll
      for (int q = 0; q < kMtPerLane / 4; ++q) {
        uint32_t w = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const long long c = c0 + 4 * q + b;
          if (c < C) w |= (uint32_t)cases[c] << (8 * b);
        }
        cw[q] = w;
      }
    }
    // (triangles << 16) | active cells of this lane, scanned over the warp
    unsigned mine = 0;
#pragma unroll
    for (int e = 0; e < kMtPerLane; ++e) {
      const int nf = mt_faces((cw[e >> 2] >> (8 * (e & 3))) & 0xF);
      mine += ((unsigned)nf << 16) | (nf ? 1u : 0u);
    }
    unsigned x = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const unsigned y = __shfl_up_sync(kFull, x, d);
      if (lane >= d) x += y;
    }
    const unsigned nact = __shfl_sync(kFull, x, 31) & 0xFFFFu;
    unsigned slot = (x - mine) & 0xFFFFu, tri = (x - mine) >> 16;
#pragma unroll
    for (int e = 0; e < kMtPerLane; ++e) {
      const int cs = (int)((cw[e >> 2] >> (8 * (e & 3))) & 0xF);
      const int nf = mt_faces(cs);
      if (nf) {
        act[slot++] = (unsigned)(lane * kMtPerLane + e) | ((unsigned)cs << 12) | (tri << 16);
        tri += (unsigned)nf;
      }
    }
    __syncwarp();
    // one active cell per lane
    for (unsigned a = lane; a < nact; a += 32) {
      const uint32_t ent = act[a];
      const long long c = cbase + (ent & 0xFFFu);
      const int cs = (int)((ent >> 12) & 0xFu);
      const int nf = mt_faces(cs);
      const unsigned long long tc = t0 + (ent >> 16);
      int id[4];
      if (!load_tet<VEC>(conn, c, P, id)) continue;  // the count pass saw it: case 0, error set
      const float v[4] = {__ldg(f + id[0]), __ldg(f + id[1]), __ldg(f + id[2]), __ldg(f + id[3])};
      const uint32_t word = s_case[cs];
      for (int m = 0; m < 3 * nf; ++m) {
        const int e = (int)((word >> (4 * m)) & 0xF);
        const int ed = (int)((kTetEdges >> (8 * e)) & 0xFF);
        const int e0 = ed & 0xF, e1 = ed >> 4;
        // the lower point id first (MarchingTetrahedra.h:142-151)
        const int i0 = pick4(id, e0), i1 = pick4(id, e1);
        const bool keep = i0 < i1;
        const int A = keep ? i0 : i1, B = keep ? i1 : i0;
        const long long rec = 3 * (long long)tc + m;
        if (KEYS) {
          if (o.wide)
            static_cast<unsigned long long*>(o.keys)[rec] =
                ((unsigned long long)A << o.kbits) | (unsigned long long)B;
          else
            static_cast<uint32_t*>(o.keys)[rec] = ((uint32_t)A << o.kbits) | (uint32_t)B;
        } else {
          const float fa = keep ? pick4(v, e0) : pick4(v, e1);
          const float fb = keep ? pick4(v, e1) : pick4(v, e0);
          const float w = __fdiv_rn(__fsub_rn(iso, fa), __fsub_rn(fb, fa));
          const float* pa = pts + 3 * (long long)A;
          const float* pb = pts + 3 * (long long)B;
#pragma unroll
          for (int q = 0; q < 3; ++q) o.verts[3 * rec + q] = lerp_rn(__ldg(pa + q), __ldg(pb + q), w);
          o.tconn[rec] = (int32_t)rec;
          if (o.ra) {
            o.ra[rec] = A;
            o.rb[rec] = B;
            o.rw[rec] = w;
          }
        }
      }
    }
    __syncwarp();
  }
}

// The merge scratch starts with a header: the number of unique keys and the
// byte offsets of the record keys and of the unique keys.
// magic marks a header written by dax_gb300_mt_merge; T is the triangle
// count of the count pass it merged.
struct MtMergeHeader {
  unsigned long long magic, V, keys, uniq, T;
};
constexpr unsigned long long kMtMergeMagic = 0x4d54204d45524745ull;

// The header describes keys of this count pass that lie inside the buffer.
template <typename U>
__device__ __forceinline__ bool merge_header_ok(const MtMergeHeader* h, long long T,
                                                unsigned long long mbytes) {
  const unsigned long long n = 3ull * (unsigned long long)T;
  return h->magic == kMtMergeMagic && h->T == (unsigned long long)T && h->V <= n &&
         h->keys <= mbytes && h->uniq <= mbytes && n * sizeof(U) <= mbytes - h->keys &&
         n * sizeof(U) <= mbytes - h->uniq;
}

// conn[r] = LowerBounds(unique keys, key of record r).  The first ten steps of
// the search run over 1023 of the keys, evenly spaced, that each block holds in
// shared memory: all 21 steps through L2 took 41 us for 2 M records of 1 M
// keys, now 32.
constexpr int kMtSamples = 1023;
template <typename U>
__global__ void __launch_bounds__(256) k_mt_merged_conn(const char* __restrict__ m,
                                                        unsigned long long mbytes, Info* info,
                                                        long long tcap, long long vcap,
                                                        int32_t* __restrict__ tconn) {
  const MtMergeHeader* hdr = reinterpret_cast<const MtMergeHeader*>(m);
  const long long T = info->total_a;
  if (info->error) return;
  if (!merge_header_ok<U>(hdr, T, mbytes)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&info->error, kErrState);
    return;
  }
  const long long V = (long long)hdr->V;
  if (T > tcap || V > vcap) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&info->error, kErrCapacity);
    return;
  }
  const U* __restrict__ keys = reinterpret_cast<const U*>(m + hdr->keys);
  const U* __restrict__ uniq = reinterpret_cast<const U*>(m + hdr->uniq);
  const long long n = 3 * T;
  __shared__ U s_key[kMtSamples];  // key at (i + 1) V / 1024
  for (int i = threadIdx.x; i < kMtSamples; i += blockDim.x) {
    const long long at = (i + 1) * V / (kMtSamples + 1);
    s_key[i] = at < V ? uniq[at] : ~(U)0;
  }
  __syncthreads();
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n;
       r += (long long)gridDim.x * blockDim.x) {
    const U k = keys[r];
    int below = 0;  // samples less than k
#pragma unroll
    for (int step = (kMtSamples + 1) / 2; step > 0; step >>= 1)
      if (s_key[below + step - 1] < k) below += step;
    long long lo = below * V / (kMtSamples + 1), hi = (below + 1) * V / (kMtSamples + 1);
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (__ldg(uniq + mid) < k) lo = mid + 1;
      else hi = mid;
    }
    tconn[r] = (int32_t)lo;
  }
}

// Vertex v of the merged output from unique key v: its two point ids, the
// weight from their field values, Lerp of their coordinates.
// (i, j, k) of point p of a uniform grid.
__device__ __forceinline__ void grid_ijk(const Grid& g, int p, int& i, int& j, int& k) {
  const unsigned row = (unsigned)p / (unsigned)g.nx;
  i = p - (int)(row * (unsigned)g.nx);
  split_row(g, row, j, k);
}

// GRID: the points are a uniform grid's (coordinates from the point id),
// else the explicit pts array.
template <typename U, bool GRID>
__global__ void __launch_bounds__(256) k_mt_merged_verts(const char* __restrict__ m,
                                                         unsigned long long mbytes, Grid g,
                                                         const Info* info, long long tcap,
                                                         long long vcap, int kbits,
                                                         const float* __restrict__ pts,
                                                         const float* __restrict__ f, float iso,
                                                         float* __restrict__ verts,
                                                         int32_t* __restrict__ ra,
                                                         int32_t* __restrict__ rb,
                                                         float* __restrict__ rw) {
  const MtMergeHeader* hdr = reinterpret_cast<const MtMergeHeader*>(m);
  const long long T = info->total_a;
  if (info->error || !merge_header_ok<U>(hdr, T, mbytes)) return;
  const long long V = (long long)hdr->V;
  if (T > tcap || V > vcap) return;
  const U* __restrict__ uniq = reinterpret_cast<const U*>(m + hdr->uniq);
  const U mask = (U)((((unsigned long long)1) << kbits) - 1ull);
  for (long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x; v < V;
       v += (long long)gridDim.x * blockDim.x) {
    const U k = uniq[v];
    const int A = (int)(k >> kbits), B = (int)(k & mask);
    const float fa = __ldg(f + A), fb = __ldg(f + B);
    const float w = __fdiv_rn(__fsub_rn(iso, fa), __fsub_rn(fb, fa));
    if (GRID) {
      int ia, ja, ka, ib, jb, kb;
      grid_ijk(g, A, ia, ja, ka);
      grid_ijk(g, B, ib, jb, kb);
      verts[3 * v + 0] = lerp_rn(coord(g.ox, g.sx, ia, g.mx), coord(g.ox, g.sx, ib, g.mx), w);
      verts[3 * v + 1] = lerp_rn(coord(g.oy, g.sy, ja, g.my), coord(g.oy, g.sy, jb, g.my), w);
      verts[3 * v + 2] = lerp_rn(coord(g.oz, g.sz, ka, g.mz), coord(g.oz, g.sz, kb, g.mz), w);
    } else {
      const float* pa = pts + 3 * (long long)A;
      const float* pb = pts + 3 * (long long)B;
#pragma unroll
      for (int a = 0; a < 3; ++a) verts[3 * v + a] = lerp_rn(__ldg(pa + a), __ldg(pb + a), w);
    }
    if (ra) {
      ra[v] = A;
      rb[v] = B;
      rw[v] = w;
    }
  }
}

// DispatcherMapCell<MarchingTetrahedraCount>: NumFaces of every cell as an
// int32 count array (cells with an id outside [0, P) count 0 and raise
// kErrBadIndex in *err).
__global__ void __launch_bounds__(256) k_mt_cell_count(const int32_t* __restrict__ conn,
                                                       long long C,
                                                       const float* __restrict__ f, long long P,
                                                       float iso, int32_t* __restrict__ count,
                                                       int* err) {
  bool bad = false;
  for (long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x; c < C;
       c += (long long)gridDim.x * blockDim.x) {
    int id[4];
    int nf = 0;
    if (load_tet<false>(conn, c, P, id)) {
      const float v[4] = {__ldg(f + id[0]), __ldg(f + id[1]), __ldg(f + id[2]), __ldg(f + id[3])};
      nf = mt_faces(mt_classify(v, iso));
    } else {
      bad = true;
    }
    count[c] = nf;
  }
  if (bad && err) atomicOr(err, kErrBadIndex);
}

__global__ void k_mt_set_header(MtMergeHeader* hdr, MtMergeHeader v) { *hdr = v; }

// ---- Marching cubes driven by an arbitrary count array ----------------------
// DispatcherGenerateInterpolatedCells<MarchingCubesGenerate> with any per-cell
// count array (DispatcherGenerateInterpolatedCells.h:158-231): the inclusive
// scan of the counts, UpperBounds(scan, t) for the input cell of output
// triangle t, visit index t - (scan[cell] - count[cell]), then the worklet's
// triangle (MarchingCubes.h:121-168).  A count of 0 drops a cell's
// triangles; a visit index at or beyond the cell's NumFaces (a count the
// worklet cannot honour) raises kErrBadCount and writes nothing for it.

// cellVertEdges (MarchingCubes.h:131-135): byte e = corners of edge e (low
// nibble, high nibble), bytes 0-7 in the first word, 8-11 in the second.
constexpr unsigned long long kHexEdgesLo = 0x7467655430232110ull;
constexpr unsigned int kHexEdgesHi = 0x73625140u;

__device__ __forceinline__ int hex_edge(int e) {
  return e < 8 ? (int)((kHexEdgesLo >> (8 * e)) & 0xFF) : (int)((kHexEdgesHi >> (8 * (e - 8))) & 0xFF);
}

// UpperBounds, the first cell whose scan exceeds t, for the first and the last
// of a warp's triangles: every lane receives both, between which the cells of
// the others lie.  Half the warp searches for each, 16 places a step (24 steps
// of one place, through L2, were most of the 78 us of 1.5 M triangles of 8 M
// cells; 61 now).
__device__ __forceinline__ void warp_cells(const int32_t* __restrict__ scan, unsigned C, int first,
                                           int last, unsigned& lo, unsigned& hi) {
  const unsigned lane = threadIdx.x & 31, half = lane >> 4, l = lane & 15;
  const int t = half ? last : first;
  unsigned a = 0, b = C;  // C < 2^31
  while (__any_sync(kFull, a < b)) {
    const unsigned step = (b - a + 15u) >> 4, at = a + step * (l + 1u) - 1u;
    // the last places may lie past b: they are past t
    const bool le = at < b && __ldg(scan + at) <= t;
    const unsigned n = __popc((__ballot_sync(kFull, le) >> (16 * half)) & 0xffffu);  // places not past t
    const unsigned past = a + step * (n + 1u) - 1u;  // the first place past t, if below b
    b = n < 16u && past < b ? past : b;
    a += step * n;
    if (a > b) a = b;
  }
  lo = __shfl_sync(kFull, a, 0);
  hi = __shfl_sync(kFull, a, 16);
}

template <bool KEYS>
__global__ void __launch_bounds__(256) k_mc_counted(Grid g, const float* __restrict__ f, float iso,
                                                    const int32_t* __restrict__ count,
                                                    const int32_t* __restrict__ scan, long long C,
                                                    unsigned long long mcx,
                                                    unsigned long long mcy, Info* info, MtOut o) {
  __shared__ uint64_t s_case[256];
  s_case[threadIdx.x] = kMcCase[threadIdx.x];
  __syncthreads();
  const long long T = info->total_a;
  if (info->error) return;
  if (!KEYS && (T > o.tcap || 3 * T > o.vcap)) {
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&info->error, kErrCapacity);
    return;
  }
  const unsigned cx = (unsigned)(g.nx - 1), cy = (unsigned)(g.ny - 1);
  const long long sy = g.nx, sz = (long long)g.nx * g.ny;
  bool bad = false;
  const int lane = threadIdx.x & 31;
  for (long long t0 = (long long)blockIdx.x * blockDim.x + (threadIdx.x & ~31); t0 < T;
       t0 += (long long)gridDim.x * blockDim.x) {
    const long long t = t0 + lane < T ? t0 + lane : T - 1;
    unsigned lo, hi;
    warp_cells(scan, (unsigned)C, (int)t0, (int)(t0 + 31 < T ? t0 + 31 : T - 1), lo, hi);
    while (lo < hi) {
      const unsigned mid = (lo + hi) >> 1;
      if (__ldg(scan + mid) <= (int)t) lo = mid + 1;
      else hi = mid;
    }
    if (t0 + lane >= T) continue;
    if (lo >= C) {
      bad = true;
      continue;
    }
    const long long c = lo;
    const long long visit = t - ((long long)__ldg(scan + c) - __ldg(count + c));
    const unsigned r = div_by((unsigned)c, mcx);
    const int i = (int)((unsigned)c - r * cx);
    const unsigned kk = div_by(r, mcy);
    const int k = (int)kk, j = (int)(r - kk * cy);
    const long long p0 = ((long long)k * g.ny + j) * g.nx + i;
    int cs = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int dx = (0x66 >> q) & 1, dy = (0xCC >> q) & 1, dz = q >> 2;
      cs |= (__ldg(f + p0 + dx + dy * sy + dz * sz) > iso ? 1 : 0) << q;
    }
    const uint64_t word = s_case[cs];
    if (visit < 0 || visit >= (long long)(word >> 60)) {
      bad = true;
      continue;
    }
    for (int m = 0; m < 3; ++m) {
      const int e = (int)((word >> (4 * (3 * visit + m))) & 0xF);
      const int ed = hex_edge(e);
      const int q0 = ed & 0xF, q1 = ed >> 4;
      const long long id0 = p0 + ((0x66 >> q0) & 1) + ((0xCC >> q0) & 1) * sy + (q0 >> 2) * sz;
      const long long id1 = p0 + ((0x66 >> q1) & 1) + ((0xCC >> q1) & 1) * sy + (q1 >> 2) * sz;
      // the lower point id first (MarchingCubes.h:148-157)
      const bool keep = id0 < id1;
      const int qa = keep ? q0 : q1, qb = keep ? q1 : q0;
      const int A = (int)(keep ? id0 : id1), B = (int)(keep ? id1 : id0);
      const long long rec = 3 * t + m;
      if (KEYS) {
        if (o.wide)
          static_cast<unsigned long long*>(o.keys)[rec] =
              ((unsigned long long)A << o.kbits) | (unsigned long long)B;
        else
          static_cast<uint32_t*>(o.keys)[rec] = ((uint32_t)A << o.kbits) | (uint32_t)B;
      } else {
        const float fa = __ldg(f + A), fb = __ldg(f + B);
        const float w = __fdiv_rn(__fsub_rn(iso, fa), __fsub_rn(fb, fa));
        const int ia = i + ((0x66 >> qa) & 1), ja = j + ((0xCC >> qa) & 1), ka = k + (qa >> 2);
        const int ib = i + ((0x66 >> qb) & 1), jb = j + ((0xCC >> qb) & 1), kb = k + (qb >> 2);
        o.verts[3 * rec + 0] = lerp_rn(coord(g.ox, g.sx, ia, g.mx), coord(g.ox, g.sx, ib, g.mx), w);
        o.verts[3 * rec + 1] = lerp_rn(coord(g.oy, g.sy, ja, g.my), coord(g.oy, g.sy, jb, g.my), w);
        o.verts[3 * rec + 2] = lerp_rn(coord(g.oz, g.sz, ka, g.mz), coord(g.oz, g.sz, kb, g.mz), w);
        o.tconn[rec] = (int32_t)rec;
        if (o.ra) {
          o.ra[rec] = A;
          o.rb[rec] = B;
          o.rw[rec] = w;
        }
      }
    }
  }
  if (bad) atomicOr(&info->error, kErrBadCount);
}

__global__ void k_set_total(Info* info, long long T, int error) {
  info->total_a = T;
  info->total_b = 0;
  info->total_c = 0;
  info->error = error;
}

void launch_set_total(Info* info, long long T, int error, cudaStream_t s) {
  k_set_total<<<1, 1, 0, s>>>(info, T, error);
}

void launch_mc_counted(const Grid& g, const float* f, float iso, const int32_t* count,
                       const int32_t* scan, Info* info, void* keys, float* verts, long long vcap,
                       int32_t* tconn, long long tcap, int32_t* ra, int32_t* rb, float* rw,
                       long long T_hint, int num_sms, cudaStream_t s) {
  const long long C = (long long)(g.nx - 1) * (g.ny - 1) * (g.nz - 1);
  MtOut o{};
  o.verts = verts;
  o.tconn = tconn;
  o.ra = ra;
  o.rb = rb;
  o.rw = rw;
  o.keys = keys;
  o.kbits = mt_key_bits(g.P);
  o.wide = 2 * o.kbits > 32;
  o.vcap = vcap;
  o.tcap = tcap;
  const unsigned long long mcx = div_multiplier((unsigned)(g.nx - 1));
  const unsigned long long mcy = div_multiplier((unsigned)(g.ny - 1));
  const long long want = (T_hint + 255) / 256;
  if (keys) {
    const int b = resident_blocks(k_mc_counted<true>, 256, 0, num_sms, want);
    k_mc_counted<true><<<b, 256, 0, s>>>(g, f, iso, count, scan, C, mcx, mcy, info, o);
  } else {
    const int b = resident_blocks(k_mc_counted<false>, 256, 0, num_sms, want);
    k_mc_counted<false><<<b, 256, 0, s>>>(g, f, iso, count, scan, C, mcx, mcy, info, o);
  }
}

// ---- Tetrahedralize (the upstream caller: uniform grid -> tetrahedra) -----
// PossibleTetraSplitCases (dax/worklet/Tetrahedralize.h:36-48): rows 0-4
// split even cell ids, rows 5-9 odd ones; entries are voxel corners in
// TopologyUniform order.
constexpr uint8_t kTetSplit[10][4] = {{2, 1, 5, 0}, {0, 2, 3, 7}, {2, 5, 6, 7}, {0, 7, 4, 5},
                                      {0, 2, 7, 5}, {1, 3, 6, 2}, {0, 1, 3, 4}, {1, 4, 5, 6},
                                      {3, 6, 7, 4}, {1, 4, 6, 3}};
// rows r0 .. r0+3 as 16-bit fields of corner nibbles
constexpr unsigned long long tet_split_word(int r0) {
  unsigned long long w = 0;
  for (int r = r0; r < r0 + 4 && r < 10; ++r)
    for (int t = 0; t < 4; ++t)
      w |= (unsigned long long)kTetSplit[r][t] << (16 * (r - r0) + 4 * t);
  return w;
}
constexpr unsigned long long kTetSplit0 = tet_split_word(0), kTetSplit1 = tet_split_word(4),
                             kTetSplit2 = tet_split_word(8);

// One thread per output tetrahedron o: cell o / 5, visit o % 5
// (Tetrahedralize.h:71-80); consecutive threads write consecutive 16 bytes.
template <bool VEC>
__global__ void __launch_bounds__(256) k_tetrahedralize(Grid g, unsigned long long mcx,
                                                        unsigned long long mcy, long long n_out,
                                                        int32_t* __restrict__ out) {
  const unsigned cx = (unsigned)(g.nx - 1), cy = (unsigned)(g.ny - 1);
  for (long long o = (long long)blockIdx.x * blockDim.x + threadIdx.x; o < n_out;
       o += (long long)gridDim.x * blockDim.x) {
    const unsigned c = (unsigned)(o / 5);
    const int visit = (int)(o - 5ll * c);
    const unsigned r = div_by(c, mcx);
    const unsigned i = c - r * cx;
    const unsigned k = div_by(r, mcy);
    const unsigned j = r - k * cy;
    const int first = (int)(i + (unsigned)g.nx * (j + (unsigned)g.ny * k));
    const int sy = g.nx, sz = g.nx * g.ny;
    const int sr = visit + 5 * (int)(c & 1);  // split row
    const unsigned long long sw = sr < 4 ? kTetSplit0 : (sr < 8 ? kTetSplit1 : kTetSplit2);
    const unsigned row = (unsigned)(sw >> (16 * (sr & 3))) & 0xFFFFu;
    // voxel corner n (TopologyUniform order) is +x for n in {1,2,5,6}
    // (0x66), +y for n in {2,3,6,7} (0xCC), +z for n >= 4
    int q4[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const int n = (int)((row >> (4 * t)) & 0xF);
      q4[t] = first + ((0x66 >> n) & 1) + sy * ((0xCC >> n) & 1) + sz * (n >> 2);
    }
    const int4 q = make_int4(q4[0], q4[1], q4[2], q4[3]);
    if (VEC) {
      reinterpret_cast<int4*>(out)[o] = q;
    } else {
      out[4 * o + 0] = q.x;
      out[4 * o + 1] = q.y;
      out[4 * o + 2] = q.z;
      out[4 * o + 3] = q.w;
    }
  }
}

// The implicit coordinates of a uniform grid as an explicit [P][3] array
// (UniformGrid::ComputePointCoordinates, dax/cont/UniformGrid.h:82-89).
__global__ void __launch_bounds__(256) k_point_coordinates(Grid g, float* __restrict__ out) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.P;
       p += (long long)gridDim.x * blockDim.x) {
    const unsigned row = (unsigned)(p / g.nx);
    const int i = (int)(p - (long long)row * g.nx);
    int j, k;
    split_row(g, row, j, k);
    out[3 * p + 0] = coord(g.ox, g.sx, i, g.mx);
    out[3 * p + 1] = coord(g.oy, g.sy, j, g.my);
    out[3 * p + 2] = coord(g.oz, g.sz, k, g.mz);
  }
}

void launch_tetrahedralize(const Grid& g, int32_t* out, int num_sms, cudaStream_t s) {
  const long long C = (long long)(g.nx - 1) * (g.ny - 1) * (g.nz - 1);
  const unsigned long long mcx = div_multiplier((unsigned)(g.nx - 1));
  const unsigned long long mcy = div_multiplier((unsigned)(g.ny - 1));
  const long long n_out = 5 * C;
  if ((reinterpret_cast<uintptr_t>(out) & 15) == 0) {
    const int b = resident_blocks(k_tetrahedralize<true>, 256, 0, num_sms, (n_out + 255) / 256);
    k_tetrahedralize<true><<<b, 256, 0, s>>>(g, mcx, mcy, n_out, out);
  } else {
    const int b = resident_blocks(k_tetrahedralize<false>, 256, 0, num_sms, (n_out + 255) / 256);
    k_tetrahedralize<false><<<b, 256, 0, s>>>(g, mcx, mcy, n_out, out);
  }
}

void launch_point_coordinates(const Grid& g, float* out, int num_sms, cudaStream_t s) {
  const int b = resident_blocks(k_point_coordinates, 256, 0, num_sms, (g.P + 255) / 256);
  k_point_coordinates<<<b, 256, 0, s>>>(g, out);
}

// ---- host side --------------------------------------------------------------

MtLayout mt_layout(long long C) {
  auto a256 = [](size_t x) { return (x + 255) & ~(size_t)255; };
  const long long tiles = (C + kMtTile - 1) / kMtTile;
  MtLayout L;
  L.tiles = (int)tiles;
  L.info = 0;
  L.tile_tot = a256(sizeof(Info));
  L.tile_off = a256(L.tile_tot + 4 * (size_t)(tiles + 1));
  L.chunk_tot = a256(L.tile_off + 8 * (size_t)(tiles + 1));
  L.cases = a256(L.chunk_tot + 4 * (size_t)tiles * (kMtTile / kMtChunk));
  L.total = a256(L.cases + (size_t)(C > 0 ? C : 1));
  return L;
}

int mt_key_bits(long long P) {
  int b = 1;
  while (b < 31 && (1ll << b) < P) ++b;
  return b;
}

void launch_mt_count(const int32_t* conn, long long C, const float* f, long long P, float iso,
                     char* scratch, int num_sms, cudaStream_t s, unsigned polls) {
  const MtLayout L = mt_layout(C);
  Info* info = reinterpret_cast<Info*>(scratch + L.info);
  cudaMemsetAsync(info, 0, sizeof(Info), s);
  const bool vec = (reinterpret_cast<uintptr_t>(conn) & 15) == 0;
  uint8_t* cases = reinterpret_cast<uint8_t*>(scratch + L.cases);
  unsigned* tot = reinterpret_cast<unsigned*>(scratch + L.tile_tot);
  unsigned* ctot = reinterpret_cast<unsigned*>(scratch + L.chunk_tot);
  if (vec) {
    // four blocks in 100 KB of shared memory, so that L1 keeps 156 KB (a hint; set
    // once per device): left to itself the driver takes 132 KB
    static int hinted[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !hinted[dev]) {
      cudaFuncSetAttribute(k_mt_count<true>, cudaFuncAttributePreferredSharedMemoryCarveout, 43);
      hinted[dev] = 1;
    }
    const int b = resident_blocks(k_mt_count<true>, kMtThreads, 0, num_sms, L.tiles);
    k_mt_count<true><<<b, kMtThreads, 0, s>>>(conn, C, f, P, iso, cases, tot, ctot, info, L.tiles,
                                              polls);
  } else {
    const int b = resident_blocks(k_mt_count<false>, kMtThreads, 0, num_sms, L.tiles);
    k_mt_count<false><<<b, kMtThreads, 0, s>>>(conn, C, f, P, iso, cases, tot, ctot, info,
                                               L.tiles, polls);
  }
  k_mt_tile_scan<<<1, 1024, 0, s>>>(tot, L.tiles,
                                    reinterpret_cast<unsigned long long*>(scratch + L.tile_off),
                                    info);
}

namespace {

template <bool KEYS>
void emit(const float* pts, const int32_t* conn, long long C, const float* f, long long P,
          float iso, char* scratch, const MtOut& o, int num_sms, cudaStream_t s) {
  const MtLayout L = mt_layout(C);
  Info* info = reinterpret_cast<Info*>(scratch + L.info);
  const uint8_t* cases = reinterpret_cast<const uint8_t*>(scratch + L.cases);
  const unsigned long long* off = reinterpret_cast<const unsigned long long*>(scratch + L.tile_off);
  const unsigned* ctot = reinterpret_cast<const unsigned*>(scratch + L.chunk_tot);
  const long long chunks = (C + kMtChunk - 1) / kMtChunk;
  const long long want = (chunks + kMtThreads / 32 - 1) / (kMtThreads / 32);
  if ((reinterpret_cast<uintptr_t>(conn) & 15) == 0) {
    const int b = resident_blocks(k_mt_emit<true, KEYS>, kMtThreads, 0, num_sms, want);
    k_mt_emit<true, KEYS><<<b, kMtThreads, 0, s>>>(pts, conn, C, f, P, iso, cases, off, ctot, info,
                                                   o, chunks);
  } else {
    const int b = resident_blocks(k_mt_emit<false, KEYS>, kMtThreads, 0, num_sms, want);
    k_mt_emit<false, KEYS><<<b, kMtThreads, 0, s>>>(pts, conn, C, f, P, iso, cases, off, ctot,
                                                    info, o, chunks);
  }
}

}  // namespace

void launch_mt_emit_direct(const float* pts, const int32_t* conn, long long C, const float* f,
                           long long P, float iso, char* scratch, float* verts, long long vcap,
                           int32_t* tconn, long long tcap, int32_t* ra, int32_t* rb, float* rw,
                           int num_sms, cudaStream_t s) {
  MtOut o{};
  o.verts = verts;
  o.tconn = tconn;
  o.ra = ra;
  o.rb = rb;
  o.rw = rw;
  o.vcap = vcap;
  o.tcap = tcap;
  emit<false>(pts, conn, C, f, P, iso, scratch, o, num_sms, s);
}

void launch_mt_emit_keys(const int32_t* conn, long long C, const float* f, long long P, float iso,
                         char* scratch, void* keys, int num_sms, cudaStream_t s) {
  MtOut o{};
  o.keys = keys;
  o.kbits = mt_key_bits(P);
  o.wide = 2 * o.kbits > 32;
  emit<true>(nullptr, conn, C, f, P, iso, scratch, o, num_sms, s);
}

void launch_mt_cell_count(const int32_t* conn, long long C, const float* f, long long P,
                          float iso, int32_t* count, int* err, int num_sms, cudaStream_t s) {
  const int b = resident_blocks(k_mt_cell_count, 256, 0, num_sms, (C + 255) / 256);
  k_mt_cell_count<<<b, 256, 0, s>>>(conn, C, f, P, iso, count, err);
}

void launch_mt_set_merged(void* merge, long long T, long long V, size_t keys_off,
                          size_t uniq_off, cudaStream_t s) {
  MtMergeHeader h{kMtMergeMagic, (unsigned long long)V, (unsigned long long)keys_off,
                  (unsigned long long)uniq_off, (unsigned long long)T};
  k_mt_set_header<<<1, 1, 0, s>>>(static_cast<MtMergeHeader*>(merge), h);
}

void launch_mt_merged(const float* pts, const Grid* grid, Info* info, const float* f,
                      long long P, float iso, const void* merge, size_t merge_bytes, float* verts,
                      long long vcap, int32_t* tconn, long long tcap, int32_t* ra, int32_t* rb,
                      float* rw, int num_sms, cudaStream_t s) {
  const Grid g = grid ? *grid : Grid{};
  const unsigned long long mb = (unsigned long long)merge_bytes;
  const char* m = static_cast<const char*>(merge);
  const int kbits = mt_key_bits(P);
  const long long want = (3 * tcap + 255) / 256;  // grid-stride: never more than resident
  if (2 * kbits > 32) {
    typedef unsigned long long U;
    const int b1 = resident_blocks(k_mt_merged_conn<U>, 256, 0, num_sms, want);
    k_mt_merged_conn<U><<<b1, 256, 0, s>>>(m, mb, info, tcap, vcap, tconn);
    if (grid) {
      const int b2 = resident_blocks(k_mt_merged_verts<U, true>, 256, 0, num_sms, want);
      k_mt_merged_verts<U, true><<<b2, 256, 0, s>>>(m, mb, g, info, tcap, vcap, kbits, pts, f, iso,
                                                    verts, ra, rb, rw);
    } else {
      const int b2 = resident_blocks(k_mt_merged_verts<U, false>, 256, 0, num_sms, want);
      k_mt_merged_verts<U, false><<<b2, 256, 0, s>>>(m, mb, g, info, tcap, vcap, kbits, pts, f,
                                                     iso, verts, ra, rb, rw);
    }
  } else {
    typedef uint32_t U;
    const int b1 = resident_blocks(k_mt_merged_conn<U>, 256, 0, num_sms, want);
    k_mt_merged_conn<U><<<b1, 256, 0, s>>>(m, mb, info, tcap, vcap, tconn);
    if (grid) {
      const int b2 = resident_blocks(k_mt_merged_verts<U, true>, 256, 0, num_sms, want);
      k_mt_merged_verts<U, true><<<b2, 256, 0, s>>>(m, mb, g, info, tcap, vcap, kbits, pts, f, iso,
                                                    verts, ra, rb, rw);
    } else {
      const int b2 = resident_blocks(k_mt_merged_verts<U, false>, 256, 0, num_sms, want);
      k_mt_merged_verts<U, false><<<b2, 256, 0, s>>>(m, mb, g, info, tcap, vcap, kbits, pts, f,
                                                     iso, verts, ra, rb, rw);
    }
  }
}

}  // namespace daxgb
