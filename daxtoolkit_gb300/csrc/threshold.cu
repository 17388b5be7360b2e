// Cell threshold on the in-range bit stream (bit = lo <= f <= hi), on the
// row-word pipeline marching cubes uses.
//
// K2a (k_thr_words): per row word w = (point row r = (j, k), word m)
//     kept[w] = cells 32m .. 32m+31 of cell row r whose 8 corners are all in
//               range (ThresholdFunction, dax/worklet/Threshold.h:30-66)
//     used[w] = points 32m .. 32m+31 of point row r that are a corner of a
//               kept cell (FillPointMask,
//               dax/cont/DispatcherGenerateTopology.h:206-227): the OR of the
//               kept masks of cell rows (j-1..j, k-1..k), each with its +x
//               neighbour cell
//     wc[w]   = popc(kept) << 16 | popc(used), and per-tile totals
// K2b (k_word_scan, shared with marching cubes): per-word exclusive offsets
//     wt (kept cells) and wv (used points), the compacted list act of the
//     words with either, and the totals.
// K3 (k_thr_emit): a warp loads kThrBatch active words at once (lane = word),
//     starts the copies of the field values of all their used points into
//     shared memory (cp.async, one wait per batch), then walks the words
//     with lane = bit: the word's used points (coordinates and field:
//     StreamCompact with the point mask, :237-239 and :98-113) and
//     its kept cells, whose 8 corner ids are each corner's rank among the
//     used points.  That equals the reference's Copy/Sort/Unique/LowerBounds
//     of the connectivity (:229-258), because the used ids sorted ascending
//     are exactly the used points in point order.
#include "common.cuh"
#include "kernels.cuh"

namespace daxgb {

// Pairs of a point row: bit x says whether points 32m + x and 32m + x + 1 are
// both in range.
__device__ __forceinline__ uint32_t row_pairs(const uint32_t* __restrict__ bits, unsigned pos) {
  const uint32_t* const s = bits + (pos >> 5);
  const uint32_t x0 = __ldg(s), x1 = __ldg(s + 1);
  return __funnelshift_r(x0, x1, pos) & __funnelshift_rc(x0, x1, (pos & 31u) + 1u);
}

// The pairs of a point row that the row one plane down (x) and up (y) has too;
// none across the grid's ends, nor for a row past its last.
__device__ __forceinline__ uint2 plane_pairs(const uint32_t* __restrict__ bits, unsigned pos,
                                             unsigned dz, int k, int nz) {
  uint2 q = make_uint2(0u, 0u);
  if (k < nz) {
    const uint32_t b = row_pairs(bits, pos);
    if (k > 0) q.x = b & row_pairs(bits, pos - dz);
    if (k + 1 < nz) q.y = b & row_pairs(bits, pos + dz);
  }
  return q;
}

// K2a: one block per tile of kScanTile words (grid-stride over tiles).  A lane
// walks down one word column over `depth` consecutive point rows: the pairs of
// a row, in its plane and combined with the planes below and above, serve the
// cells of the row and of the one before, and the kept cells between two rows
// the used points of both.  Consecutive lanes take consecutive words; lane 0
// repeats the word before lane 1's, whose last cell lane 1's first point may
// belong to, and writes nothing.  A grid has fewer than 2^31 points, so bit
// positions are 32-bit; rows are at most 8192 points, 256 words, long.  kept is
// written where a point is used.  (Kept masks and used masks in two passes, four
// words a lane: from the classification's end to the scan's 40 us at 512^3, 16
// at 200 x 180 x 150, 17 at 60^3; now 34, 10 and 11, and with two blocks an SM
// in place of four, which spill 12 bytes, 39, 9 and 11.)
constexpr int kThrThreads = 512;
__global__ void __launch_bounds__(kThrThreads, 4)
    k_thr_words(Grid g, const uint32_t* __restrict__ bits, uint32_t* __restrict__ kept,
                uint32_t* __restrict__ used, uint32_t* __restrict__ wc,
                uint32_t* __restrict__ tile_tot, int tiles) {
  constexpr unsigned kWarps = kThrThreads / 32, kCols = 31;
  __shared__ uint32_t s_sum[3];  // the tile's kept cells, used points and active words
  pdl_trigger();
  pdl_wait();  // the classification's bits
  const int lane = threadIdx.x & 31;
  const unsigned W = (unsigned)(g.R * g.wr), wr = (unsigned)g.wr, nx = (unsigned)g.nx;
  const unsigned dz = nx * (unsigned)g.ny;
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (threadIdx.x < 3) s_sum[threadIdx.x] = 0;
    __syncthreads();
    const unsigned lo = (unsigned)tile * kScanTile, n = min((unsigned)kScanTile, W - lo);
    const unsigned r0 = div_by(lo, g.mwr), rows = div_by(lo + n - 1u, g.mwr) - r0 + 1u;
    // the fewest rows a lane with which the block covers the tile at once
    const unsigned fit = kWarps * kCols / wr;
    const unsigned depth = (rows + fit - 1u) / fit;
    const unsigned items = (rows + depth - 1u) / depth * wr;
    uint32_t sk = 0, su = 0, sa = 0;
    for (unsigned q0 = (threadIdx.x >> 5) * kCols; q0 < items; q0 += kWarps * kCols) {
      const unsigned q1 = q0 + (unsigned)lane;  // the lane's item, plus one
      const bool mine = lane > 0 && q1 <= items;
      const unsigned q = q1 == 0u ? 0u : min(q1 - 1u, items - 1u);
      const unsigned chunk = div_by(q, g.mwr), m = q - chunk * wr;
      const unsigned r = r0 + chunk * depth;
      int j, k;
      split_row(g, r, j, k);
      unsigned pos = r * nx + 32u * m;
      unsigned w = mine ? r * wr + m - lo : 0x80000000u;  // the word's place in the tile; before it: above n
      const uint32_t cmask = low_mask(g.nx - 1 - 32 * (int)m), pmask = low_mask(g.nx - 32 * (int)m);
      uint2 cur = plane_pairs(bits, pos, dz, k, g.nz);
      uint32_t up = 0u;  // kept cells of cell row j - 1, of both planes
      if (j > 0) {
        const uint2 prev = plane_pairs(bits, pos - nx, dz, k, g.nz);
        up = ((prev.x & cur.x) | (prev.y & cur.y)) & cmask;
      }
#pragma unroll 2
      for (unsigned d = 0; d < depth; ++d) {
        const bool cells = j + 1 < g.ny;  // the row has cells in y
        j = cells ? j + 1 : 0;
        k += cells ? 0 : 1;
        pos += nx;
        const uint2 nxt = plane_pairs(bits, pos, dz, k, g.nz);
        const uint32_t own = cells ? nxt.y & cur.y & cmask : 0u;
        const uint32_t dp = cells ? own | (nxt.x & cur.x & cmask) : 0u;
        const uint32_t K = up | dp;
        const uint32_t before = __shfl_up_sync(kFull, K, 1) >> 31;
        const uint32_t U = (K | (K << 1) | (m > 0 ? before : 0u)) & pmask;
        if (w < n) {
          const uint32_t ck = __popc(own), cu = __popc(U);
          used[lo + w] = U;
          if (U) kept[lo + w] = own;
          wc[lo + w] = ck << 16 | cu;
          sk += ck;
          su += cu;
          sa += U ? 1u : 0u;
        }
        up = dp;
        cur = nxt;
        w += wr;
      }
    }
    sk = __reduce_add_sync(kFull, sk);
    su = __reduce_add_sync(kFull, su);
    sa = __reduce_add_sync(kFull, sa);
    if (lane == 0) {
      atomicAdd(&s_sum[0], sk);
      atomicAdd(&s_sum[1], su);
      atomicAdd(&s_sum[2], sa);
    }
    __syncthreads();
    if (threadIdx.x < 3) tile_tot[threadIdx.x * tiles + tile] = s_sum[threadIdx.x];
    __syncthreads();  // s_sum is free
  }
}

void launch_thr_count(const Grid& g, const uint32_t* bits, uint32_t* kept, uint32_t* used,
                      uint32_t* wc, uint32_t* tile_tot, int num_sms, cudaStream_t s) {
  (void)num_sms;
  const int tiles = word_scan_tiles(g.R * g.wr);  // a block a tile
  launch_pdl(k_thr_words, (unsigned)tiles, (unsigned)kThrThreads, 0, s, g, bits, kept, used, wc,
             tile_tot, tiles);
}

// Words a warp of the emit takes at a time.  Small batches even the warps out:
// 133, 139, 143 and 145 us with 8, 16, 24 and 32 at 512^3, 11 to 16 us at 200 x
// 180 x 150.
constexpr int kThrBatch = 8;

// Per active word, what the emit loop needs: its masks and offsets, and for
// kept cells the used masks and offsets of corner rows q = dj + 2 dk
// (q = 1..3) at word m, and the first used-point offsets of rows q = 0..3 at
// word m + 1 (the +x corner of a cell at bit 31 is that word's first point,
// always used).
struct ThrWord {
  uint32_t w, u, kw, v0, t0;
  uint32_t r, m, j, k;  // the word's point row (j, k) and word index in the row
  uint32_t cu[3], cv[7];
};

// Bound by its writes, 16 bytes a used point and 32 a kept cell, and by the
// latency of each word's chain: stores of whole sectors (a cell is one 32-byte
// store, a word's coordinates leave through shared memory) took the 13.5 M
// cells and 14 M points of a 512^3 threshold from 143 to 138 us, 655 MB at 4.7
// TB/s; batches of 8 words took that to 133.  (The words' data broadcast from shared memory in place of shuffles,
// and four words at a time with their values a group ahead, took a fifth off
// the instructions and no time.)
__global__ void __launch_bounds__(256) k_thr_emit(Grid g, const float* __restrict__ f,
                                                  const uint32_t* __restrict__ kept,
                                                  const uint32_t* __restrict__ used,
                                                  const uint32_t* __restrict__ wt,
                                                  const uint32_t* __restrict__ wv,
                                                  const uint32_t* __restrict__ act,
                                                  Info* __restrict__ info,
                                                  int32_t* __restrict__ conn, long long kcap,
                                                  float* __restrict__ coords,
                                                  float* __restrict__ fout, long long ucap) {
  const long long K = info->total_a, U = info->total_b, A = info->total_c;
  if (K > kcap || U > ucap || (info->error & (kErrOverflow | kErrTimeout))) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && (K > kcap || U > ucap))
      atomicOr(&info->error, kErrCapacity);
    return;
  }
  const int lane = threadIdx.x & 31;
  const uint32_t below = (1u << lane) - 1u;
  // a cell's connectivity leaves as one store of 32 bytes, two of 16 or eight of 4,
  // as the array's address allows (512^3 points, 13.5 M cells: 139, 152 and 213 us)
  const unsigned conn_at = (unsigned)reinterpret_cast<uintptr_t>(conn) & 31u;
  const unsigned wr = (unsigned)g.wr;
  __shared__ float s_field[8][kThrBatch][32];  // per warp: field value of bit `lane` of batch word s
  float (*const sf)[32] = s_field[threadIdx.x >> 5];
  __shared__ float s_coord[8][2][96];  // per warp, alternating words: the word's coordinates
  // the block's batches of words are every gridDim.x-th one; its warps take
  // them from a counter in shared memory (words differ widely in cost)
  __shared__ unsigned s_next;
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  while (true) {
    unsigned n = 0;
    if (lane == 0) n = atomicAdd(&s_next, 1u);
    const long long a0 =
        ((long long)__shfl_sync(kFull, n, 0) * gridDim.x + blockIdx.x) * kThrBatch;
    if (a0 >= A) break;
    // lane L gathers active word a0 + L
    ThrWord d{};
    const int cnt = (int)min((long long)kThrBatch, A - a0);
    if (lane < cnt) {
      d.w = __ldg(act + a0 + lane);
      d.u = __ldg(used + d.w);
      d.kw = __ldg(kept + d.w);
      d.v0 = __ldg(wv + d.w);
      d.t0 = __ldg(wt + d.w);
      int mi, ji, ki;
      d.r = split_word(g, d.w, mi);
      split_row(g, d.r, ji, ki);
      d.m = (uint32_t)mi;
      d.j = (uint32_t)ji;
      d.k = (uint32_t)ki;
      if (d.kw) {  // a kept cell implies rows j + 1 and k + 1 exist
        const unsigned m = d.m;
        const uint32_t rows[4] = {d.w, d.w + wr, d.w + (unsigned)g.ny * wr,
                                  d.w + (unsigned)(g.ny + 1) * wr};
#pragma unroll
        for (int q = 1; q < 4; ++q) {
          d.cu[q - 1] = __ldg(used + rows[q]);
          d.cv[q - 1] = __ldg(wv + rows[q]);
        }
        if (m + 1 < wr) {
#pragma unroll
          for (int q = 0; q < 4; ++q) d.cv[3 + q] = __ldg(wv + rows[q] + 1);
        }
      }
    }
    if (fout) {
      // the field values of the batch's used points, all copies in flight at
      // once (a field read is a DRAM round trip: K1 streamed it evict-first)
      for (int s = 0; s < cnt; ++s) {
        const uint32_t u = __shfl_sync(kFull, d.u, s);
        const uint32_t r = __shfl_sync(kFull, d.r, s), m = __shfl_sync(kFull, d.m, s);
        const bool on = (u >> lane) & 1u;
        const float* src = on ? f + ((long long)r * g.nx + 32 * m + lane) : f;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(&sf[s][lane]);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src),
                     "r"(on ? 4 : 0)
                     : "memory");
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    for (int s = 0; s < cnt; ++s) {
      const uint32_t u = __shfl_sync(kFull, d.u, s);
      const uint32_t kw = __shfl_sync(kFull, d.kw, s);
      const uint32_t m = __shfl_sync(kFull, d.m, s);
      const int j = (int)__shfl_sync(kFull, d.j, s), k = (int)__shfl_sync(kFull, d.k, s);
      const int i = 32 * (int)m + lane;
      const uint32_t v0 = __shfl_sync(kFull, d.v0, s);
      // the word's points leave through shared memory, so that each store of
      // the warp covers 128 consecutive bytes
      float* const sc = s_coord[threadIdx.x >> 5][s & 1];
      if ((u >> lane) & 1u) {
        const int rank = __popc(u & below);
        sc[3 * rank] = coord(g.ox, g.sx, i, g.mx);
        sc[3 * rank + 1] = coord(g.oy, g.sy, j, g.my);
        sc[3 * rank + 2] = coord(g.oz, g.sz, k, g.mz);
        if (fout) fout[(long long)v0 + rank] = sf[s][lane];
      }
      __syncwarp();
      const int nc = 3 * __popc(u);
      float* const c0 = coords + 3 * (long long)v0;
#pragma unroll
      for (int t = 0; t < 96; t += 32)
        if (t + lane < nc) c0[t + lane] = sc[t + lane];
      if (kw == 0u) continue;  // uniform across the warp
      const uint32_t t0 = __shfl_sync(kFull, d.t0, s);
      uint32_t cu[4], cv[8];  // corner rows q at word m (0..3); cv[4 + q]: at word m + 1
      cu[0] = u;
      cv[0] = v0;
#pragma unroll
      for (int e = 0; e < 3; ++e) cu[e + 1] = __shfl_sync(kFull, d.cu[e], s);
#pragma unroll
      for (int e = 0; e < 7; ++e) cv[e + 1] = __shfl_sync(kFull, d.cv[e], s);
      if ((kw >> lane) & 1u) {
        const long long cid = (long long)t0 + __popc(kw & below);
        // used-point ranks of the corners at i (lo) and i + 1 (hi) of corner
        // rows q = dj + 2 dk: hi = lo + the bit of point i, except on lane
        // 31, whose i + 1 is bit 0 of word m + 1
        int32_t lo[4], hi[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t b = cv[q] + (uint32_t)__popc(cu[q] & below);
          lo[q] = (int32_t)b;
          hi[q] = (int32_t)(lane == 31 ? cv[4 + q] : b + ((cu[q] >> lane) & 1u));
        }
        // v0..v7: (i,j,k) (i+1,j,k) (i+1,j+1,k) (i,j+1,k), then the same at k+1
        const int32_t ids[8] = {lo[0], hi[0], hi[1], lo[1], lo[2], hi[2], hi[3], lo[3]};
        if (conn_at == 0u) {  // a cell is one 32-byte sector
          asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(conn + 8 * cid),
                       "r"(ids[0]), "r"(ids[1]), "r"(ids[2]), "r"(ids[3]), "r"(ids[4]), "r"(ids[5]),
                       "r"(ids[6]), "r"(ids[7])
                       : "memory");
        } else if (conn_at == 16u) {
          int4* const dst = reinterpret_cast<int4*>(conn + 8 * cid);
          dst[0] = make_int4(ids[0], ids[1], ids[2], ids[3]);
          dst[1] = make_int4(ids[4], ids[5], ids[6], ids[7]);
        } else {
#pragma unroll
          for (int v = 0; v < 8; ++v) conn[8 * cid + v] = ids[v];
        }
      }
    }
  }
}

// CompactPointField of DispatcherGenerateTopology (:98-113): any point
// field of `comps` floats per point, compacted to the used points in point
// order -- the order of the threshold's output coordinates.  A warp per row
// word, lane = bit: a used point's output index is its word's used-point
// offset plus its rank in the word.  Needs the count pass (used masks, word
// offsets, totals) on the same scratch; writes nothing when the used points
// exceed `cap`.
__global__ void __launch_bounds__(256) k_thr_compact_field(Grid g, const uint32_t* __restrict__ used,
                                                           const uint32_t* __restrict__ wv,
                                                           Info* __restrict__ info,
                                                           const float* __restrict__ in, int comps,
                                                           float* __restrict__ out, long long cap) {
  const long long U = info->total_b;
  if (U > cap || (info->error & (kErrOverflow | kErrTimeout))) {
    if (blockIdx.x == 0 && threadIdx.x == 0 && U > cap) atomicOr(&info->error, kErrCapacity);
    return;
  }
  const int lane = threadIdx.x & 31;
  const long long W = g.R * g.wr;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long w = warp0; w < W; w += nwarps) {
    const uint32_t u = __ldg(used + w);
    if (!((u >> lane) & 1u)) continue;
    int m;
    const unsigned r = split_word(g, (unsigned)w, m);
    const long long p = (long long)r * g.nx + 32ll * m + lane;
    const long long id = (long long)__ldg(wv + w) + __popc(u & ((1u << lane) - 1u));
    for (int c = 0; c < comps; ++c) out[id * comps + c] = __ldg(in + p * comps + c);
  }
}

void launch_thr_compact_field(const Grid& g, const uint32_t* used, const uint32_t* wv, Info* info,
                              const float* in, int comps, float* out, long long cap, int num_sms,
                              cudaStream_t s) {
  const long long want = (g.R * g.wr + 7) / 8;  // a warp per word, 8 warps a block
  const int blocks = resident_blocks(k_thr_compact_field, 256, 0, num_sms, want);
  k_thr_compact_field<<<blocks, 256, 0, s>>>(g, used, wv, info, in, comps, out, cap);
}

void launch_thr_emit(const Grid& g, const float* f, const WordOffsets& o, const uint32_t* kept,
                     const uint32_t* used, Info* info, int32_t* conn, long long kcap,
                     float* coords, float* fout, long long ucap, int num_sms, cudaStream_t s) {
  // the active count lives on the device: one resident wave, grid-stride
  const long long want = (g.R * g.wr + 8 * kThrBatch - 1) / (8 * kThrBatch);
  const int blocks = resident_blocks(k_thr_emit, 256, 0, num_sms, want);
  // an ordinary launch: the blocks split the active words statically, so all
  // blocks should start together on an idle device (count and emit, launched
  // after and early into the SMs that the scan frees: 26.3 and 24.2 us at 100^3,
  // 42.7 and 40.6 at 200^3, 130.7 and 130.7 at 384^3, 265.9 and 269 at 512^3)
  k_thr_emit<<<blocks, 256, 0, s>>>(g, f, kept, used, o.wt, o.wv, o.act, info, conn, kcap, coords,
                                    fout, ucap);
}

}  // namespace daxgb
