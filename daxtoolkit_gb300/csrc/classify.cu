// K1: point classification into a bit stream, and the per-cell count kernels
// behind DispatcherMapCell<MarchingCubesCount | ThresholdCount>.
//
// K1 is the only kernel that reads the whole field.  It is a pure stream: each
// warp step loads 32 x float4 (512 B, fully coalesced, evict-first) and emits
// four 32-bit words of classification bits, so HBM traffic is 4 B/point read +
// 1/8 B/point written.  Everything downstream (counts, scans, generation)
// works on the 16x smaller bit stream, which stays resident in L2.
#include "common.cuh"
#include "kernels.cuh"
#include "mc_case.cuh"

namespace daxgb {

template <int MODE>
__device__ __forceinline__ uint32_t classify_point(float v, float a, float b) {
  // MODE 0: marching-cubes inside test, values[i] > iso (dax/worklet/MarchingCubes.h:40-47)
  // MODE 1: threshold test, min <= value <= max (dax/worklet/Threshold.h:40-43)
  if (MODE == 0) return v > a ? 1u : 0u;
  return (v >= a && v <= b) ? 1u : 0u;
}

// Each warp-chunk covers 128 points = 4 bit words.  UNROLL chunks per warp
// step keep several 512 B loads in flight per warp.  Chunks are global over
// the grid set; each grid's chunks start on a fresh chunk, so a chunk never
// straddles two grids and each grid's bits start on a word boundary.
//
// [c_begin, c_end) restricts a one-grid launch to a range of chunks (the
// slabs of the pipelined marching cubes); `init`, when not null, is the Info
// block whose error words and emit counters this launch clears (it runs
// before every other pass of its count pass).
//
// KEEP: the field is read with the default cache policy instead of
// evict-first, so that a slab's values can still be in L2 when the emit of
// that slab gathers its crossing-edge end points (pipelined calls).
template <typename T>
__device__ __forceinline__ T ld_field(const T* p, bool keep) {
  return keep ? __ldg(p) : __ldcs(p);
}

template <int MODE, bool VEC, bool KEEP>
__global__ void __launch_bounds__(256) k_classify_bits(GridSet S, uint32_t* __restrict__ bits,
                                                       long long nwords, long long c_begin,
                                                       long long c_end, Info* init) {
  constexpr int UNROLL = 4;
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  const long long nchunks = S.chunks;
  const float nan = __int_as_float(0x7fc00000);  // classifies as 0 in both modes
  __shared__ long long s_keys[kStagedSlots];
  const long long* keys =
      stage_slot_keys(S, s_keys, [](const GridSlot& sl) { return sl.chunk0; }) ? s_keys : nullptr;
  pdl_trigger();  // the count pass may launch into the SMs this grid frees
  if (init && blockIdx.x == 0 && threadIdx.x == 0) {
    init->error = 0;
    init->ticket = 0;
    init->done = 0;
  }
  if (S.count == 1) {
    // one grid: field pointer and thresholds are loop invariants
    const float* __restrict__ f = S.one.field;
    const long long P = S.one.g.P;
    const float a = S.one.iso, b = S.one.iso_hi;
    for (long long c0 = c_begin + warp * UNROLL; c0 < c_end; c0 += nwarps * UNROLL) {
      float4 v[UNROLL];
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const long long base = ((c0 + u) << 7) + lane * 4;
        if (c0 + u >= c_end) {
          v[u] = make_float4(nan, nan, nan, nan);
        } else if (VEC && base + 3 < P) {
          v[u] = ld_field(reinterpret_cast<const float4*>(f + base), KEEP);
        } else {
          v[u].x = base + 0 < P ? ld_field(f + base + 0, KEEP) : nan;
          v[u].y = base + 1 < P ? ld_field(f + base + 1, KEEP) : nan;
          v[u].z = base + 2 < P ? ld_field(f + base + 2, KEEP) : nan;
          v[u].w = base + 3 < P ? ld_field(f + base + 3, KEEP) : nan;
        }
      }
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const uint32_t nib = classify_point<MODE>(v[u].x, a, b) |
                             (classify_point<MODE>(v[u].y, a, b) << 1) |
                             (classify_point<MODE>(v[u].z, a, b) << 2) |
                             (classify_point<MODE>(v[u].w, a, b) << 3);
        uint32_t w = nib << (4 * (lane & 7));
        w |= __shfl_xor_sync(kFull, w, 1);
        w |= __shfl_xor_sync(kFull, w, 2);
        w |= __shfl_xor_sync(kFull, w, 4);
        if ((lane & 7) == 0 && c0 + u < c_end) bits[((c0 + u) << 2) + (lane >> 3)] = w;
      }
    }
  } else {
    // one search per warp step (the step's chunks are consecutive), then a
    // step forward where a chunk starts a later grid; the next step's search
    // runs while this step's loads are in flight
    const long long stride = nwarps * UNROLL;
    int snext = warp * UNROLL < nchunks
                    ? (keys ? slot_search(keys, S.count, warp * UNROLL) : slot_of_chunk(S, warp * UNROLL))
                    : 0;
    for (long long c0 = warp * UNROLL; c0 < nchunks; c0 += stride) {
      float4 v[UNROLL];
      float a[UNROLL], b[UNROLL];
      long long wout[UNROLL];
      int si = snext;
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const long long c = c0 + u;
        v[u] = make_float4(nan, nan, nan, nan);
        a[u] = b[u] = 0.0f;
        wout[u] = -1;
        if (c < nchunks) {
          while (si + 1 < S.count && (keys ? keys[si + 1] : __ldg(&S.slots[si + 1].chunk0)) <= c) ++si;
          const GridSlot& sl = S.slots[si];
          const long long lc = c - sl.chunk0;
          const long long base = (lc << 7) + lane * 4;
          const float* f = sl.field;
          const long long P = sl.g.P;
          a[u] = sl.iso;
          b[u] = sl.iso_hi;
          wout[u] = sl.word0 + (lc << 2);
          if (VEC && base + 3 < P) {
            v[u] = __ldcs(reinterpret_cast<const float4*>(f + base));
          } else {
            if (base + 0 < P) v[u].x = __ldcs(f + base + 0);
            if (base + 1 < P) v[u].y = __ldcs(f + base + 1);
            if (base + 2 < P) v[u].z = __ldcs(f + base + 2);
            if (base + 3 < P) v[u].w = __ldcs(f + base + 3);
          }
        }
      }
      if (c0 + stride < nchunks)
        snext = keys ? slot_search(keys, S.count, c0 + stride) : slot_of_chunk(S, c0 + stride);
#pragma unroll
      for (int u = 0; u < UNROLL; ++u) {
        const uint32_t nib = classify_point<MODE>(v[u].x, a[u], b[u]) |
                             (classify_point<MODE>(v[u].y, a[u], b[u]) << 1) |
                             (classify_point<MODE>(v[u].z, a[u], b[u]) << 2) |
                             (classify_point<MODE>(v[u].w, a[u], b[u]) << 3);
        uint32_t w = nib << (4 * (lane & 7));
        w |= __shfl_xor_sync(kFull, w, 1);
        w |= __shfl_xor_sync(kFull, w, 2);
        w |= __shfl_xor_sync(kFull, w, 4);
        if ((lane & 7) == 0 && wout[u] >= 0) bits[wout[u] + (lane >> 3)] = w;
      }
    }
  }
  // zero the padding words after the last chunk (read by unaligned fetches)
  if (blockIdx.x == 0 && threadIdx.x < 8 && c_end == nchunks) {
    const long long w = (nchunks << 2) + threadIdx.x;
    if (w < nwords) bits[w] = 0u;
  }
}

void launch_classify_bits(int mode, const GridSet& S, bool all_aligned, uint32_t* bits,
                          long long nwords, int num_sms, cudaStream_t s) {
  launch_classify_range(mode, S, all_aligned, bits, nwords, 0, S.chunks, nullptr, kPassClassify,
                        false, num_sms, s);
}

void launch_classify_range(int mode, const GridSet& S, bool all_aligned, uint32_t* bits,
                           long long nwords, long long c_begin, long long c_end, Info* init,
                           int pass, bool keep, int num_sms, cudaStream_t s) {
  // blocks of 8 warps x 4 chunks
  const long long want = (c_end - c_begin + 4 * 8 - 1) / (4 * 8);
#define DAXGB_K1(M, V, K)                                                      \
  {                                                                            \
    const int blocks = resident_blocks(k_classify_bits<M, V, K>, 256, 0, num_sms, want, pass); \
    k_classify_bits<M, V, K><<<blocks, 256, 0, s>>>(S, bits, nwords, c_begin, c_end, init); \
  }
  if (mode == 0 && keep) {
    if (all_aligned) DAXGB_K1(0, true, true) else DAXGB_K1(0, false, true)
  } else if (mode == 0) {
    if (all_aligned) DAXGB_K1(0, true, false) else DAXGB_K1(0, false, false)
  } else {
    if (all_aligned) DAXGB_K1(1, true, false) else DAXGB_K1(1, false, false)
  }
#undef DAXGB_K1
}

// ---- per-cell count arrays (the Dax count handles) ---------------------
// Bound by HBM (the field in, a count a cell out).  A warp takes 31 cells of
// a cell row and kCellRows rows after one another: lane l holds point i0 + l
// of the two planes of each row, so every point is loaded and tested once a
// plane pair, the tests of 32 points are one ballot, and a cell's case is two
// neighbouring bits of four ballots (31 cells, not 32, so that no lane needs a
// second point).  One thread a cell with eight loads, eight tests and 64-bit
// divisions took 70 us for the 15 M cells of 301 x 257 x 199, now 38.
//
// MODE 0: MarchingCubesCount.  MODE 1: ThresholdCount.  MODE 2: the Mandelbulb's
// MandlebulbClipCount (Benchmarks/Mandlebulb/Worklets.h:112-170), a cell's
// triangle count when one of its points lies beyond the plane,
// dot(N, p - O) > loc; otherwise 0.
constexpr int kCellRows = 8;

struct ClipPlane {
  float3 o, n;
  float loc;
};

template <int MODE>
__global__ void __launch_bounds__(256) k_cell_count(Grid g, const float* __restrict__ f, float a,
                                                    float b, ClipPlane pl, unsigned segs,
                                                    unsigned bands, unsigned items,
                                                    int32_t* __restrict__ count,
                                                    uint8_t* __restrict__ cases) {
  __shared__ unsigned char s_nf[256];
  if (MODE != 1) s_nf[threadIdx.x] = (unsigned char)mc_num_tris(threadIdx.x);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int cx = g.nx - 1, cy = g.ny - 1;
  const long long dz = (long long)g.nx * g.ny;
  for (unsigned it = blockIdx.x * 8u + (threadIdx.x >> 5); it < items; it += gridDim.x * 8u) {
    const unsigned row = it / segs, k = row / bands;
    const int i0 = 31 * (int)(it - row * segs), j0 = kCellRows * (int)(row - k * bands);
    const int i = i0 + lane, ir = i < g.nx ? i : g.nx - 1;
    const float* p = f + ir + (long long)g.nx * j0 + dz * k;
    float v[kCellRows + 1][2];
#pragma unroll
    for (int q = 0; q <= kCellRows; ++q) {
      v[q][0] = v[q][1] = 0.0f;
      if (j0 + q < g.ny) {
        v[q][0] = __ldg(p + (long long)q * g.nx);
        v[q][1] = __ldg(p + (long long)q * g.nx + dz);
      }
    }
    float tx = 0, tz0 = 0, tz1 = 0;
    if (MODE == 2) {
      tx = __fmul_rn(pl.n.x, __fsub_rn(coord(g.ox, g.sx, ir, g.mx), pl.o.x));
      tz0 = __fmul_rn(pl.n.z, __fsub_rn(coord(g.oz, g.sz, (int)k, g.mz), pl.o.z));
      tz1 = __fmul_rn(pl.n.z, __fsub_rn(coord(g.oz, g.sz, (int)k + 1, g.mz), pl.o.z));
    }
    // the previous row's tests: r0, r1 of the values, w0 | w1 of the plane
    unsigned r0 = 0, r1 = 0, w = 0;
    long long c = (long long)cx * (j0 - 1 + (long long)cy * k) + i;
#pragma unroll
    for (int q = 0; q <= kCellRows; ++q) {
      const unsigned s0 = __ballot_sync(kFull, classify_point<MODE == 1 ? 1 : 0>(v[q][0], a, b));
      const unsigned s1 = __ballot_sync(kFull, classify_point<MODE == 1 ? 1 : 0>(v[q][1], a, b));
      unsigned x = 0;
      if (MODE == 2) {
        const float ty = __fmul_rn(pl.n.y, __fsub_rn(coord(g.oy, g.sy, j0 + q, g.my), pl.o.y));
        const float t = __fadd_rn(tx, ty);
        x = __ballot_sync(kFull, __fadd_rn(t, tz0) > pl.loc || __fadd_rn(t, tz1) > pl.loc);
      }
      if (q > 0 && j0 + q < g.ny && lane < 31 && i < cx) {
        int out;
        if (MODE == 1) {
          const unsigned all = r0 & r1 & s0 & s1;
          out = (int)((all >> lane) & (all >> (lane + 1)) & 1u);
        } else {
          // vertex order (i, j) (i+1, j) (i+1, j+1) (i, j+1), then one plane up
          const unsigned n0 = (s0 >> lane) & 3u, n1 = (s1 >> lane) & 3u;
          const unsigned cs = ((r0 >> lane) & 3u) | ((n0 >> 1) | ((n0 & 1u) << 1)) << 2 |
                              ((r1 >> lane) & 3u) << 4 | ((n1 >> 1) | ((n1 & 1u) << 1)) << 6;
          out = s_nf[cs];
          if (MODE == 0 && cases) cases[c] = (uint8_t)cs;
          if (MODE == 2 && !(((w | x) >> lane) & 3u)) out = 0;
        }
        count[c] = out;
      }
      r0 = s0;
      r1 = s1;
      w = x;
      c += cx;
    }
  }
}

// A cell a thread, its eight loads served by L1: grids whose rows or bands leave
// many of a warp's 248 cells empty.  It takes 55, 71 and 100 us (modes 0, 1, 2)
// for 16 M cells of any shape; the kernel above 41, 35 and 51 with all 248 cells
// of a warp, the same with 171, 109 and 109 (64 x 64 and 33 x 33 cells in x and
// y), 5370, 5500 and 7390 with one (1 x 1).
template <int MODE>
__global__ void __launch_bounds__(256) k_cell_count_each(Grid g, const float* __restrict__ f,
                                                         float a, float b, ClipPlane pl,
                                                         unsigned long long mcx,
                                                         unsigned long long mcy, unsigned cells,
                                                         int32_t* __restrict__ count,
                                                         uint8_t* __restrict__ cases) {
  __shared__ unsigned char s_nf[256];
  if (MODE != 1) s_nf[threadIdx.x] = (unsigned char)mc_num_tris(threadIdx.x);
  __syncthreads();
  const unsigned cx = (unsigned)g.nx - 1u, cy = (unsigned)g.ny - 1u;
  const long long dz = (long long)g.nx * g.ny;
  for (unsigned c = blockIdx.x * 256u + threadIdx.x; c < cells; c += gridDim.x * 256u) {
    const unsigned r = div_by(c, mcx), i = c - r * cx, k = div_by(r, mcy), j = r - k * cy;
    const float* p = f + (long long)i + (long long)g.nx * j + dz * k;
    bool in = false;
    unsigned cs = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int qx = (0x66 >> q) & 1, qy = (0xCC >> q) & 1, qz = q >> 2;
      const float v = __ldg(p + qx + (qy ? g.nx : 0) + (qz ? dz : 0));
      cs |= (classify_point<MODE == 1 ? 1 : 0>(v, a, b) ? 1u : 0u) << q;
      if (MODE == 2)
        in = in || plane_value(g, pl.o, pl.n, (int)i + qx, (int)j + qy, (int)k + qz) > pl.loc;
    }
    if (MODE == 1) count[c] = cs == 255u;
    else count[c] = MODE == 0 || in ? s_nf[cs] : 0;
    if (MODE == 0 && cases) cases[c] = (uint8_t)cs;
  }
}

template <int MODE>
static void cell_count(const Grid& g, const float* f, float a, float b, const ClipPlane& pl,
                       int32_t* count, uint8_t* cases, int num_sms, cudaStream_t s) {
  const unsigned segs = ((unsigned)g.nx - 1 + 30) / 31;
  const unsigned bands = ((unsigned)g.ny - 1 + kCellRows - 1) / kCellRows;
  const unsigned items = segs * bands * ((unsigned)g.nz - 1);
  const unsigned cells = ((unsigned)g.nx - 1) * ((unsigned)g.ny - 1) * ((unsigned)g.nz - 1);
  constexpr long long kLeastCells = MODE == 0 ? 171 : 109;  // a warp, on average
  if (cells < kLeastCells * items) {
    const int blocks = resident_blocks(k_cell_count_each<MODE>, 256, 0, num_sms,
                                       ((long long)cells + 255) / 256);
    k_cell_count_each<MODE><<<blocks, 256, 0, s>>>(g, f, a, b, pl, div_multiplier((unsigned)g.nx - 1),
                                                   div_multiplier((unsigned)g.ny - 1), cells, count,
                                                   cases);
    return;
  }
  const int blocks = resident_blocks(k_cell_count<MODE>, 256, 0, num_sms, (items + 7) / 8);
  k_cell_count<MODE><<<blocks, 256, 0, s>>>(g, f, a, b, pl, segs, bands, items, count, cases);
}

void launch_cell_count(int mode, const Grid& g, const float* f, float a, float b, int32_t* count,
                       uint8_t* cases, int num_sms, cudaStream_t s) {
  if (mode == 0) cell_count<0>(g, f, a, b, ClipPlane{}, count, cases, num_sms, s);
  else cell_count<1>(g, f, a, b, ClipPlane{}, count, cases, num_sms, s);
}

void launch_mandelbulb_clip_count(const Grid& g, const float* f, float iso, float3 o, float3 n,
                                  float loc, int32_t* count, int num_sms, cudaStream_t s) {
  cell_count<2>(g, f, iso, 0.0f, ClipPlane{o, n, loc}, count, nullptr, num_sms, s);
}

}  // namespace daxgb
