// Generic data-parallel primitives of the device adapter
// (dax::cont::DeviceAdapterAlgorithm, dax/cont/internal/DeviceAdapterAlgorithm.h:44-331;
// the reference's generic versions are dax/cont/internal/DeviceAdapterAlgorithmGeneral.h):
// ScanInclusive / ScanExclusive, Sort / SortByKey, Unique, LowerBounds /
// UpperBounds and StreamCompact, on the element types the Dax pipelines use
// (dax::Id = int32, int64, unsigned, dax::Scalar = float) with values of up
// to 16 bytes (a dax::Vector3 is 12).
//
// Tiles: the float scan works on kPTile elements (256 threads x 16), the sort
// on kSweepTile, the integer scan and the compaction on kSElems:
//   scan     integers: one pass, each tile's prefix found by a decoupled
//            look-back over the tiles before it; floats: reduce-then-scan,
//            tile sums, one block scanning the sums, then each tile scanned
//            with its prefix, whose fixed order of additions gives the same
//            result on every run (in place allowed for both);
//   sort     LSD radix sort, 8-bit digits, stable, one read and one write of
//            the elements a pass: a tile ranks its keys by ballots, finds the
//            earlier tiles' digit counts by a look-back, and writes its digits'
//            runs; up to 8192 elements are sorted in one block;
//   compact  one pass on the integer scan's machinery: a tile's kept
//            elements are counted as it lands, its offset found by the
//            look-back, and the kept elements written at their places
//            (Unique = compact of "differs from the previous key", in place;
//            StreamCompact = compact of "stencil != 0").
#include <cstdint>
#include <cstring>
#include <string>

#include "../../include/dax_gb300.h"
#include "common.cuh"
#include "kernels.cuh"
#include "tma.cuh"

namespace daxgb {

namespace {

constexpr int kPT = 256;
constexpr int kPI = 16;
constexpr int kPTile = kPT * kPI;

int ptiles(long long n) { return (int)((n + kPTile - 1) / kPTile); }

// Integer sums wrap like the reference's dax::Id arithmetic: accumulate in
// the unsigned type of the same width.
template <typename T> struct Acc { typedef T type; };
template <> struct Acc<int32_t> { typedef uint32_t type; };
template <> struct Acc<int64_t> { typedef unsigned long long type; };

template <typename A>
__device__ __forceinline__ A block_exclusive(A v, A* s_warp, A* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  A x = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const A y = __shfl_up_sync(kFull, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  A base = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kPT / 32; ++w) {
    if (w < warp) base += s_warp[w];
    tot += s_warp[w];
  }
  __syncthreads();
  *total = tot;
  return base + x - v;
}

// ---- scan -----------------------------------------------------------------

template <typename T>
__global__ void __launch_bounds__(kPT) k_tile_sum(const T* __restrict__ in, long long n,
                                                  typename Acc<T>::type* __restrict__ sums,
                                                  int tiles) {
  typedef typename Acc<T>::type A;
  __shared__ A s_warp[kPT / 32];
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    A v = 0;
    const long long b = (long long)tile * kPTile;
#pragma unroll 4
    for (int e = 0; e < kPI; ++e) {
      const long long i = b + e * kPT + threadIdx.x;
      if (i < n) v += (A)in[i];
    }
    A tot;
    block_exclusive(v, s_warp, &tot);
    if (threadIdx.x == 0) sums[tile] = tot;
  }
}

// One block: exclusive scan of the tile sums in place; the grand total goes
// to sums[tiles].
template <typename A>
__global__ void __launch_bounds__(1024) k_scan_sums(A* __restrict__ sums, int tiles) {
  __shared__ A s_warp[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  A carry = 0;
  for (int c0 = 0; c0 < tiles; c0 += 1024) {
    const int i = c0 + threadIdx.x;
    const A v = i < tiles ? sums[i] : (A)0;
    A x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const A y = __shfl_up_sync(kFull, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    A base = 0, tot = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) base += s_warp[w];
      tot += s_warp[w];
    }
    if (i < tiles) sums[i] = carry + base + x - v;
    carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[tiles] = carry;
}

// A tile is loaded with coalesced (striped) loads into shared memory, each
// thread then scans 16 consecutive elements, and the results leave the same
// way.  The tile's prefix comes from the scanned sums.  Every element of a
// tile is read before any is written: in place is fine.
__device__ __forceinline__ int pad(int i) { return i + (i >> 5); }

template <typename T>
__global__ void __launch_bounds__(kPT) k_tile_scan(const T* __restrict__ in, T* out, long long n,
                                                   const typename Acc<T>::type* __restrict__ pre,
                                                   int tiles, int exclusive) {
  typedef typename Acc<T>::type A;
  __shared__ A s_warp[kPT / 32];
  __shared__ A s_t[kPTile + kPTile / 32];
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long b = (long long)tile * kPTile;
#pragma unroll
    for (int e = 0; e < kPI; ++e) {
      const int li = e * kPT + threadIdx.x;
      s_t[pad(li)] = b + li < n ? (A)in[b + li] : (A)0;
    }
    __syncthreads();
    A v[kPI];
    A sum = 0;
#pragma unroll
    for (int e = 0; e < kPI; ++e) {
      v[e] = s_t[pad(threadIdx.x * kPI + e)];
      sum += v[e];
    }
    A tot;
    A run = pre[tile] + block_exclusive(sum, s_warp, &tot);
#pragma unroll
    for (int e = 0; e < kPI; ++e) {
      const A next = run + v[e];
      s_t[pad(threadIdx.x * kPI + e)] = exclusive ? run : next;
      run = next;
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kPI; ++e) {
      const int li = e * kPT + threadIdx.x;
      if (b + li < n) out[b + li] = (T)s_t[pad(li)];
    }
    __syncthreads();
  }
}

// Two-level scan of many sums: chunks of 1024 scanned in parallel (each
// chunk's total to aux), the totals scanned by one block, then added back.
template <typename A>
__global__ void __launch_bounds__(1024) k_chunk_scan(A* __restrict__ v, int count,
                                                     A* __restrict__ aux) {
  __shared__ A s_warp[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = blockIdx.x * 1024 + threadIdx.x;
  const A x0 = i < count ? v[i] : (A)0;
  A x = x0;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const A y = __shfl_up_sync(kFull, x, d);
    if (lane >= d) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  A base = 0, tot = 0;
  for (int w = 0; w < 32; ++w) {
    if (w < warp) base += s_warp[w];
    tot += s_warp[w];
  }
  if (i < count) v[i] = base + x - x0;
  if (threadIdx.x == 0) aux[blockIdx.x] = tot;
}

template <typename A>
__global__ void __launch_bounds__(1024) k_chunk_add(A* __restrict__ v, int count,
                                                    const A* __restrict__ aux, int chunks) {
  const int i = blockIdx.x * 1024 + threadIdx.x;
  if (i < count) v[i] += aux[blockIdx.x];
  if (blockIdx.x == 0 && threadIdx.x == 0) v[count] = aux[chunks];
}

// Exclusive scan of v[0..count) in place, total to v[count]; aux holds
// count / 1024 + 2 entries.
template <typename A>
void scan_sums(A* v, int count, A* aux, cudaStream_t s) {
  if (count <= 8192) {
    k_scan_sums<A><<<1, 1024, 0, s>>>(v, count);
    return;
  }
  const int chunks = (count + 1023) / 1024;
  k_chunk_scan<A><<<chunks, 1024, 0, s>>>(v, count, aux);
  k_scan_sums<A><<<1, 1024, 0, s>>>(aux, chunks);
  k_chunk_add<A><<<chunks, 1024, 0, s>>>(v, count, aux, chunks);
}

int sum_slots(long long n) { return ptiles(n) + 1 + ptiles(n) / 1024 + 2; }

int resident(const void* kernel, int threads, int num_sms, long long want) {
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, 0) != cudaSuccess ||
      per < 1)
    per = 1;
  const long long cap = (long long)num_sms * per;
  return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}

template <typename T>
void scan_t(const T* in, T* out, long long n, bool exclusive, void* scratch, int num_sms,
            cudaStream_t s) {
  typedef typename Acc<T>::type A;
  const int tiles = ptiles(n);
  A* sums = static_cast<A*>(scratch);
  const int b = resident((const void*)k_tile_sum<T>, kPT, num_sms, tiles);
  k_tile_sum<T><<<b, kPT, 0, s>>>(in, n, sums, tiles);
  scan_sums<A>(sums, tiles, sums + tiles + 1, s);
  k_tile_scan<T><<<b, kPT, 0, s>>>(in, out, n, sums, tiles, exclusive ? 1 : 0);
}

// ---- single-pass scan of integer elements ---------------------------------
//
// One read and one write of every element, by one persistent block an SM, with
// the look-back of D. Merrill and M. Garland, "Single-pass Parallel Prefix Scan
// with Decoupled Look-back" (NVIDIA NVR-2016-002, 2016).  A copy warp takes tiles of kSElems elements from a ticket counter and keeps
// them in a ring of shared-memory stages (192 KB), each filled by one bulk TMA
// copy.  Sixteen compute warps reduce a tile as soon as it lands and publish
// its sum (AGG); a look-back warp then finds the tile's prefix over the
// published states of the tiles before it (32 a step, lane = tile) and
// publishes the inclusive prefix (INC), while the compute warps reduce the
// next Ring::ahead tiles; they then scan the tile in shared memory, and the
// copy warp writes it back with one bulk copy and fills the stage again.
//
// Why this shape: what limits it is how long a stage is held, mostly by its
// look-back (the prefix crosses the ~500 tiles in flight 32 a step, an L2 round
// trip each).  Summing three tiles ahead hides it where one did not, with half
// the ring still loading: 100 M int32 took 240, 179, 155 and 178 us with 1, 2, 3
// and 4 of six 32 KB stages ahead (120 at the copy bandwidth), and 182 with one
// of three 64 KB stages ahead and eight compute warps that also stored and
// refilled.  8-byte elements have room for three 64 KB stages, one ahead.
// Reading more states a step, 2 or 4 a lane, and shorter sleeps between polls
// measured no faster (183 to 200 us against 183).
//
// Tiles are taken in ticket order and each block's tickets increase in the
// order it processes them, so the smallest unfinished tile always has all
// its predecessors' sums published and its block working on it: no tile
// waits on a later one.  Every wait is still bounded (Spin).  A wait that runs
// out marks the scan failed (DAX_GB300_ERROR_TIMEOUT when the total is read),
// and nothing is written for a tile whose prefix is not known: the look-back
// warp publishes such a tile as BAD, which ends the look-back of every later
// tile that meets it, and compute warps without a prefix write no more tiles.
//
// Integer sums wrap, so any split of the look-back gives the same result;
// float scans keep the deterministic reduce-then-scan above.
//
// Shared-memory layout of a tile: warp w owns elements [w, w + 1) * kWarpElems;
// its lane reads and writes 16-byte chunk c at element c * 32 * E + lane * E
// of that range (E elements a chunk), so every access of a warp covers 512
// consecutive bytes and no two lanes share a bank.  The scan goes chunk by
// chunk: a lane's E elements, a warp scan of the chunk totals, and the carry
// of the chunks before.  Arrays that are not 16-byte aligned, and the ragged
// last tile, are loaded and stored element by element instead.
//
// Scratch (zeroed before the launch, the states included): ticket, error,
// total, then per tile its state: flag << 32 | sum in one 64-bit word for
// 32-bit sums, two such words (low and high halves) for 64-bit sums.
constexpr unsigned kStAgg = 1u, kStInc = 2u, kStBad = 3u;
constexpr size_t kScanHead = 64;
constexpr int kSThreads = 512;  // compute threads
constexpr int kSElems = 8192;   // elements a tile
constexpr unsigned kSRing = 192 * 1024;

template <typename Staged>
struct Ring {
  static constexpr unsigned bytes = kSElems * sizeof(Staged);      // a tile, a stage
  static constexpr int stages = (int)(kSRing / bytes);             // 6 or 3
  static constexpr int chunks = (int)(bytes / (16u * kSThreads));  // 16-byte chunks a thread
  static constexpr int ahead = stages / 2;  // tiles summed before the oldest is written
};

struct ScanCtl {
  unsigned ticket, error;
  unsigned long long total;
};

__device__ __forceinline__ unsigned long long ld_relaxed64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

template <typename A> struct TileStates;

template <> struct TileStates<uint32_t> {
  unsigned long long* word;
  __host__ __device__ static size_t bytes(int tiles) { return (size_t)tiles * 8; }
  __host__ __device__ static size_t clear_bytes(int tiles) { return (size_t)tiles * 8; }
  __host__ __device__ explicit TileStates(char* base, int) : word((unsigned long long*)base) {}
  __device__ void publish(int t, unsigned flag, uint32_t v) const {
    st_relaxed64(word + t, (unsigned long long)flag << 32 | v);
  }
  __device__ unsigned read(int t, uint32_t& v) const {
    const unsigned long long w = ld_relaxed64(word + t);
    v = (uint32_t)w;
    return (unsigned)(w >> 32);
  }
};

// 64-bit sums: two 64-bit words, each the flag above 32 bits of the sum,
// stored and loaded as one 16-byte access (each word is single-copy atomic,
// the pair need not be); words with different flags are a read that caught a
// publication half done, and count as not yet published.
template <> struct TileStates<unsigned long long> {
  unsigned long long* pair;
  __host__ __device__ static size_t bytes(int tiles) { return (size_t)tiles * 16; }
  __host__ __device__ static size_t clear_bytes(int tiles) { return (size_t)tiles * 16; }
  __host__ __device__ explicit TileStates(char* base, int) : pair((unsigned long long*)base) {}
  __device__ void publish(int t, unsigned flag, unsigned long long v) const {
    const unsigned long long f = (unsigned long long)flag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(pair + 2 * t),
                 "l"(f | (v & 0xffffffffull)), "l"(f | (v >> 32))
                 : "memory");
  }
  __device__ unsigned read(int t, unsigned long long& v) const {
    unsigned long long lo, hi;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                 : "=l"(lo), "=l"(hi)
                 : "l"(pair + 2 * t)
                 : "memory");
    const unsigned f = (unsigned)(lo >> 32);
    if (f != (unsigned)(hi >> 32)) return 0u;
    v = (lo & 0xffffffffull) | (hi << 32);
    return f;
  }
};

template <typename A>
__device__ __forceinline__ A warp_inclusive(A x, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const A y = __shfl_up_sync(kFull, x, d);
    if (lane >= d) x += y;
  }
  return x;
}

// The exclusive prefix of `tile` from the states of the tiles before it
// (one warp; every lane returns it).  A step reads the states of tiles
// top - lane, polls those not yet published (a short sleep between polls),
// and ends at the nearest inclusive prefix.  Sets `failed` (on every lane) if
// a wait ran out, here or before the nearest tile that knows.
template <typename A>
__device__ A look_back(const TileStates<A>& st, int tile, int lane, unsigned polls, bool& failed) {
  A prefix = 0;
  failed = false;
  for (int top = tile - 1; top >= 0; top -= 32) {
    const int t = top - lane;
    A x = 0;
    unsigned f = kStInc;  // before tile 0: an inclusive zero
    if (t >= 0) {
      Spin spin(polls);
      while ((f = st.read(t, x)) == 0u) {
        if (!spin.more()) {
          f = kStBad;
          break;
        }
        __nanosleep(300);
      }
    }
    // the nearest tile with its inclusive prefix (or none) ends the look-back
    const unsigned incl = __ballot_sync(kFull, f >= kStInc);
    const int last = incl ? __ffs(incl) - 1 : 31;
    A part = lane <= last ? x : (A)0;
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(kFull, part, d);
    prefix += part;
    if (incl) {
      failed = __shfl_sync(kFull, f, last) == kStBad;
      break;
    }
  }
  return prefix;
}

__device__ __forceinline__ void compute_sync() {  // the compute warps only
  asm volatile("bar.sync 1, %0;" ::"r"(kSThreads) : "memory");
}
// The same, and whether `ok` holds on every compute thread.
__device__ __forceinline__ bool compute_all(bool ok) {
  unsigned all;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n"
      " barrier.cta.red.and.pred q, 2, %2, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(all)
      : "r"((unsigned)ok), "r"(kSThreads)
      : "memory");
  return all != 0;
}

__device__ __forceinline__ bool wait_phase(uint64_t* bar, unsigned parity,
                                           unsigned polls = kSpinIters) {
  Spin sp(polls);
  while (!mbar_test(bar, parity))
    if (!sp.more()) return false;
  return true;
}

// A lane's first 16-byte chunk of a staged tile: warp w owns elements
// [w, w + 1) * (tile / warps); chunk c of the lane is 32 * c chunks further.
template <typename Staged>
__device__ __forceinline__ Staged* lane_chunk0(Staged* s_data, int warp, int lane) {
  constexpr int kWarpElems = kSElems / (kSThreads / 32);
  return s_data + warp * kWarpElems + lane * (16 / (int)sizeof(Staged));
}

// The single-pass driver the integer scan and the compaction share (run by
// one persistent block an SM: kSThreads compute threads, a look-back warp, and
// a copy warp that fills the stages and stores them).  Op is the pass's policy:
//   Staged, Sum        the ring's element type; the tile sums
//   Carry              what a compute thread keeps of a tile from its sum to
//                      its output
//   src                the staged array
//   on_take(t)         the copy warp, when it issues the bulk copy of whole tile t
//   on_land(k, b, aux) thread 0, when the tile of stage k (first element b)
//                      has landed, before it is summed; aux[k] is the pass's
//                      own per-stage word
//   thread_sum(...)    a compute thread's part of the tile's sum
//   finish(...)        the compute threads' output of the tile, given the
//                      sum of everything before the warp's first element
//   store(...)         the copy warp, once every compute warp has finished a
//                      whole tile: the stage's bytes out (the scan), or nothing
constexpr int kSBlock = kSThreads + 64;

template <class Op>
__device__ __forceinline__ void single_pass(const Op& op, long long n, int tiles, ScanCtl* ctl,
                                            char* states, int bulk, unsigned polls) {
  typedef typename Op::Staged Staged;
  typedef typename Op::Sum Sum;
  typedef typename Op::Carry Carry;
  constexpr int kTileElems = kSElems, kSStages = Ring<Staged>::stages, kAhead = Ring<Staged>::ahead;
  constexpr unsigned kSTileBytes = Ring<Staged>::bytes;
  constexpr int kWarps = kSThreads / 32;
  const TileStates<Sum> st(states, tiles);
  extern __shared__ __align__(128) unsigned char scan_smem[];
  // a stage's tile has landed (or is the compute warps' to load) / its sum is
  // known / its prefix is known / its output is done
  __shared__ __align__(8) uint64_t b_full[kSStages], b_agg[kSStages], b_pre[kSStages],
      b_done[kSStages];
  __shared__ int s_tile[kSStages];  // the stage's occupant
  __shared__ int s_seen[kSStages];  // the occupant as handed to the look-back warp
  __shared__ Sum s_tot[kSStages], s_pre[kSStages], s_wsum[kSStages][kWarps];
  __shared__ bool s_known[kSStages];  // whether s_pre is the tile's prefix
  __shared__ unsigned long long s_aux[kSStages];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a tile is copied in bulk when it is whole and the arrays are 16-byte aligned
  auto whole = [&](int t) { return bulk && (long long)(t + 1) * kTileElems <= n; };
  auto stage = [&](int k) { return reinterpret_cast<Staged*>(scan_smem + (size_t)k * kSTileBytes); };
  if (threadIdx.x == 0) {
    for (int k = 0; k < kSStages; ++k) {
      mbar_init(&b_full[k], 1);
      mbar_init(&b_agg[k], 1);
      mbar_init(&b_pre[k], 1);
      mbar_init(&b_done[k], kWarps);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == kWarps + 1) {
    // the copy warp (one lane): stage use i holds the block's i-th ticket
    if (lane != 0) return;
    unsigned long long policy;  // read once: evict first
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    bool ok = true;
    // waits for the output of use i and stores it
    auto retire = [&](int i) {
      const int k = i % kSStages, t = s_tile[k];
      ok = wait_phase(&b_done[k], (i / kSStages) & 1, polls);
      if (ok && whole(t)) op.store(stage(k), (long long)t * kTileElems);
    };
    int i = 0;
    for (;; ++i) {
      const int k = i % kSStages;
      if (i >= kSStages) retire(i - kSStages);
      if (!ok) break;
      const int t = (int)atomicAdd(&ctl->ticket, 1u);
      s_tile[k] = t;
      if (t < tiles && whole(t)) {
        mbar_arrive_tx(&b_full[k], kSTileBytes);
        bulk_load(stage(k), op.src + (long long)t * kTileElems, kSTileBytes, &b_full[k], policy);
        op.on_take(t);
      } else {
        mbar_arrive(&b_full[k]);
      }
      if (t >= tiles) break;
    }
    for (int r = i < kSStages ? 0 : i - kSStages + 1; ok && r < i; ++r) retire(r);
    if (!ok) {
      // the compute warps gave up: wait (bounded) for the copies still in
      // flight, so that none lands in shared memory after the block leaves
      atomicOr(&ctl->error, 1u);
      for (int r = i < kSStages ? 0 : i - kSStages; r < i; ++r)
        wait_phase(&b_full[r % kSStages], (r / kSStages) & 1);
    }
    return;
  }

  if (warp == kWarps) {
    // the look-back warp: the block's tiles in order
    for (int i = 0;; ++i) {
      const int k = i % kSStages;
      if (!__all_sync(kFull, wait_phase(&b_agg[k], (i / kSStages) & 1, polls))) {
        if (lane == 0) atomicOr(&ctl->error, 1u);
        break;
      }
      const int tile = s_seen[k];
      if (tile >= tiles) break;
      const Sum tot = s_tot[k];
      bool failed;
      const Sum prefix = look_back(st, tile, lane, polls, failed);
      if (lane == 0) {
        if (tile > 0) st.publish(tile, failed ? kStBad : kStInc, prefix + tot);
        if (failed) atomicOr(&ctl->error, 1u);
        if (tile == tiles - 1) ctl->total = (unsigned long long)(prefix + tot);
        s_pre[k] = prefix;
        s_known[k] = !failed;
        mbar_arrive(&b_pre[k]);
      }
      __syncwarp();
    }
    return;
  }

  // compute warps.  reduce(i): the tile of stage use i lands (bulk) or is
  // loaded here (elements), is summed, and its sum published and handed on;
  // returns the tile, `tiles` once they are done (the later uses hold later
  // tickets) or when the tile did not land in time
  auto reduce = [&](int i, Carry& carry) -> int {
    const int k = i % kSStages;
    int tile = tiles;
    if (compute_all(wait_phase(&b_full[k], (i / kSStages) & 1, polls)))
      tile = s_tile[k];
    else if (threadIdx.x == 0)
      atomicOr(&ctl->error, 1u);
    if (tile >= tiles) {
      if (threadIdx.x == 0) {
        s_seen[k] = tiles;
        mbar_arrive(&b_agg[k]);
      }
      return tiles;
    }
    Staged* s_data = stage(k);
    const long long b = (long long)tile * kTileElems;
    if (!whole(tile)) {
      const long long cnt = n - b < kTileElems ? n - b : kTileElems;
      for (int j = threadIdx.x; j < kTileElems; j += kSThreads)
        s_data[j] = j < cnt ? op.src[b + j] : (Staged)0;
      compute_sync();
    }
    if (threadIdx.x == 0) op.on_land(k, b, s_aux);
    Sum sum = op.thread_sum(s_data, k, b, warp, lane, s_aux, carry);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(kFull, sum, d);
    if (lane == 0) s_wsum[k][warp] = sum;
    compute_sync();
    if (threadIdx.x == 0) {
      Sum tot = 0;
      for (int w = 0; w < kWarps; ++w) tot += s_wsum[k][w];
      st.publish(tile, tile == 0 ? kStInc : kStAgg, tot);
      s_tot[k] = tot;
      s_seen[k] = tile;
      mbar_arrive(&b_agg[k]);
    }
    return tile;
  };

  // the tiles summed and not yet written, oldest first
  Carry carry[kAhead + 1];
  int tile[kAhead + 1];
#pragma unroll
  for (int d = 0; d < kAhead; ++d) {
    tile[d] = tiles;
    if (d == 0 || tile[d > 0 ? d - 1 : 0] < tiles) tile[d] = reduce(d, carry[d]);
  }
  bool lost = false;  // the warp got no prefix for a tile: it only sums, for the block's barriers,
                      // and the copy warp, whose stage does not come back, gives up
  for (int i = 0; tile[0] < tiles; ++i) {
    const int k = i % kSStages;
    tile[kAhead] = tile[kAhead - 1] < tiles ? reduce(i + kAhead, carry[kAhead]) : tiles;
    // the prefix is read before the votes on it, which its loads then hide (100 M
    // values compacted: 190 us, 195 in the other order, 185 without the votes)
    const bool ok = wait_phase(&b_pre[k], (i / kSStages) & 1, polls);
    const bool known = s_known[k];  // of use where every lane's wait ended
    Sum run = s_pre[k];
    for (int w = 0; w < warp; ++w) run += s_wsum[k][w];
    if (__any_sync(kFull, !ok) || !known) {
      lost = true;
      if (lane == 0) atomicOr(&ctl->error, 1u);
    }
    if (!lost) {
      op.finish(stage(k), (long long)tile[0] * kTileElems, run, warp, lane, carry[0], whole(tile[0]));
      // the warp's shared-memory writes before the bulk copy reads them (and
      // its reads before the stage's next bulk copy writes it)
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&b_done[k]);
    }
#pragma unroll
    for (int d = 0; d < kAhead; ++d) {
      tile[d] = tile[d + 1];
      carry[d] = carry[d + 1];
    }
  }
}

// The integer scan's policy: sums of the elements; the tile is scanned in
// shared memory chunk by chunk (a lane's E elements, a warp scan of the chunk
// totals, the carry of the chunks before) and written back whole, or, a ragged
// or unaligned tile, by each warp its own range.
template <typename T>
struct ScanPass {
  typedef typename Acc<T>::type Staged;
  typedef typename Acc<T>::type Sum;
  static constexpr int E = 16 / (int)sizeof(Staged);
  static constexpr int kSChunks = Ring<Staged>::chunks;
  struct Chunk { Staged e[E]; };
  struct Carry {};
  const Staged* src;
  T* out;
  long long n;
  int exclusive;
  __device__ void on_take(int) const {}
  __device__ void on_land(int, long long, unsigned long long*) const {}
  __device__ Sum thread_sum(Staged* s_data, int, long long, int warp, int lane,
                            const unsigned long long*, Carry&) const {
    const Chunk* sc = reinterpret_cast<const Chunk*>(lane_chunk0(s_data, warp, lane));
    Sum sum = 0;
#pragma unroll 4
    for (int c = 0; c < kSChunks; ++c) {
      const Chunk x = sc[32 * c];
#pragma unroll
      for (int e = 0; e < E; ++e) sum += x.e[e];
    }
    return sum;
  }
  __device__ void finish(Staged* s_data, long long b, Sum run, int warp, int lane, const Carry&,
                         bool whole) const {
    Chunk* sc = reinterpret_cast<Chunk*>(lane_chunk0(s_data, warp, lane));
#pragma unroll 4
    for (int c = 0; c < kSChunks; ++c) {
      Chunk x = sc[32 * c];
      Sum l[E];
      Sum acc = 0;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        l[e] = acc;  // exclusive within the lane's chunk
        acc += x.e[e];
      }
      const Sum ci = warp_inclusive(acc, lane);
      const Sum base = run + ci - acc;
#pragma unroll
      for (int e = 0; e < E; ++e) x.e[e] = base + l[e] + (exclusive ? (Sum)0 : x.e[e]);
      sc[32 * c] = x;
      run += __shfl_sync(kFull, ci, 31);
    }
    if (!whole) {
      __syncwarp();
      constexpr int kWarpElems = 32 * kSChunks * E;
      const int j0 = warp * kWarpElems;
      for (int j = j0 + lane; j < j0 + kWarpElems && b + j < n; j += 32) out[b + j] = (T)s_data[j];
    }
  }
  __device__ void store(Staged* s_data, long long b) const {
    bulk_store_and_wait_read(out + b, s_data, Ring<Staged>::bytes);
  }
};

template <typename T>
__global__ void __launch_bounds__(kSBlock, 1)
    k_scan_single(ScanPass<T> op, long long n, int tiles, ScanCtl* ctl, char* states, int bulk,
                  unsigned polls) {
  single_pass(op, n, tiles, ctl, states, bulk, polls);
}

int single_pass_tiles(long long n) { return (int)((n + kSElems - 1) / kSElems); }

template <typename T>
size_t single_scan_bytes(long long n) {
  typedef typename Acc<T>::type A;
  return kScanHead + TileStates<A>::bytes(single_pass_tiles(n));
}

// Clears the scratch's control words and tile states and launches one block
// an SM of `kernel` (the ring is above the 48 KB of shared memory a launch
// gets without opting in: set once per device and kernel; a failure shows
// as the launch's error).  The self-check of the waits: polls, the most polls
// of a wait; lost, whether no block takes tile 0, whose sum every other tile
// then waits for in vain.
template <class Op>
void launch_single_pass(void (*kernel)(Op, long long, int, ScanCtl*, char*, int, unsigned),
                        const Op& op, long long n, int bulk, char* scratch, int num_sms,
                        cudaStream_t s, unsigned polls = kSpinIters, bool lost = false) {
  typedef typename Op::Staged Staged;
  typedef typename Op::Sum Sum;
  const size_t smem = kSRing;
  static int opted[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !opted[dev]) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
            cudaSuccess &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared) == cudaSuccess)
      opted[dev] = 1;
  }
  const int tiles = single_pass_tiles(n);
  const int blocks = tiles < num_sms ? tiles : num_sms;
  cudaMemsetAsync(scratch, 0, kScanHead + TileStates<Sum>::clear_bytes(tiles), s);
  if (lost) cudaMemsetAsync(scratch, 1, 1, s);  // the first ticket is 1 (little-endian)
  kernel<<<blocks, kSBlock, smem, s>>>(op, n, tiles, reinterpret_cast<ScanCtl*>(scratch),
                                       scratch + kScanHead, bulk, polls);
}

template <typename T>
void scan_single(const T* in, T* out, long long n, bool exclusive, char* scratch, int num_sms,
                 cudaStream_t s, unsigned polls = kSpinIters, bool lost = false) {
  typedef typename Acc<T>::type A;
  const ScanPass<T> op{reinterpret_cast<const A*>(in), out, n, exclusive ? 1 : 0};
  const int bulk = ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  launch_single_pass(k_scan_single<T>, op, n, bulk, scratch, num_sms, s, polls, lost);
}

// ---- radix sort -------------------------------------------------------------

// Keys as unsigned integers whose order is the key type's order (ascending);
// descending order is the complement.  Floats: negative values have all bits
// flipped, the others only the sign bit (IEEE total order for non-NaN keys).
template <typename U> struct Bits;
template <> struct Bits<uint32_t> {
  static constexpr uint32_t sign = 0x80000000u;
};
template <> struct Bits<unsigned long long> {
  static constexpr unsigned long long sign = 0x8000000000000000ull;
};

// The ordering map of a sort pass: keys read from the caller's array are
// mapped to ordered bits as they are loaded (the first pass), and mapped back
// as the last pass stores them, so that no pass of its own goes over the keys
// for either.  Branch-free: x ^ (flip where the sign bit is set) ^ flop, with
// flip = all bits but the sign for floats, 0 otherwise, and flop = the sign
// bit for signed and float keys, complemented for descending order; both 0
// where a pass maps nothing.  flip leaves the sign bit, so the inverse is the
// same two steps in the other order.
template <typename U>
struct KeyOrder {
  U in_flip, in_flop, out_flip, out_flop;
  KeyOrder(int kind, bool desc, bool in, bool out) {
    const U flip = kind == 2 ? (U)~Bits<U>::sign : (U)0;
    const U flop = (U)((kind ? Bits<U>::sign : (U)0) ^ (desc ? ~(U)0 : (U)0));
    in_flip = in ? flip : 0;
    in_flop = in ? flop : 0;
    out_flip = out ? flip : 0;
    out_flop = out ? flop : 0;
  }
  static __device__ __forceinline__ U sign_mask(U x) {
    return sizeof(U) == 4 ? (U)((int32_t)x >> 31) : (U)((int64_t)x >> 63);
  }
  __device__ __forceinline__ U load(U x) const { return x ^ (sign_mask(x) & in_flip) ^ in_flop; }
  __device__ __forceinline__ U store(U t) const {
    t ^= out_flop;
    return t ^ (sign_mask(t) & out_flip);
  }
};

// One sweep per digit: the method of A. Adinets and D. Merrill, "Onesweep: A
// Faster Least Significant Digit Radix Sort for GPUs" (arXiv 2206.01784, 2022).
// A pass reads every key (and value) once and writes it
// once: a block takes a tile of kSweepTile elements from a ticket counter, ranks
// its keys, publishes its count of every digit, finds how many keys of each
// digit the earlier tiles hold by looking back over their published counts
// (thread = digit), and writes the tile out in digit order.  The digits'
// global starts come from one histogram of all passes' digits, since a pass
// only permutes the keys.
//
// Why this shape (100 M int32 pairs): a pass per tile histogram, scan of the
// histograms and scatter read the keys twice, and the scatter spent 11.7 of
// its 17 stall cycles an instruction on __match_any_sync (short scoreboard)
// and gathered its values from global memory in digit order: 1.31 ms a pass.
// Here equal digits are found by eight ballots, values pass through shared
// memory like the keys, and the look-back replaces histogram and scan:
// 0.49 ms a pass, against 0.24 ms for its 1.6 GB at the copy bandwidth.  What
// is left is 108 instructions a row of 32 keys (101 M for 30 M keys) and the random shared
// memory accesses of counters and places (63 % of that pipe), which 36 warps
// of 16 keys a thread cannot hide from one another.  (Finding equal digits by
// atomicOr of the lanes into a mask a digit, 16 instructions instead of 50 but
// three more random accesses, took 0.54.)
//
// State of (tile, digit), one 32-bit word, zeroed before the pass: 0 nothing
// yet; count + 1 (count <= kSweepTile) the tile's own count; bit 31 | sum the
// count over the tiles up to and including it (n < 2^31).
// Tickets go out in tile order, so a wait is only ever on a block that is
// running.  The wait is bounded all the same, and a thread whose wait runs out
// counts the missing tile's digit from the keys themselves (a pass never
// writes the array it reads), so the result does not depend on it.
constexpr int kSortThreads = 512;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kSortWarps = kSortThreads / 32;

// A sweep's blocks are smaller than the one that sorts alone, so that more of
// them, in different phases, share an SM: three of 4-byte keys with up to one
// word of values, two otherwise (by registers and shared memory).  100 M int32
// pairs: 2.14 ms with three of 384 threads, the same with two of 512, 2.36 with
// two of 384; 30 M int64 pairs: 1.72, 2.18 (one block fits) and 1.72 ms.  (At
// three blocks the form with one word of values spills 32 bytes, at two those
// with three and four words 8 to 16.)
constexpr int kSweepThreads = 384;
constexpr int kSweepTile = kSweepThreads * kSortItems;
constexpr int kSweepWarps = kSweepThreads / 32;
template <typename U, int VW>
constexpr int kSweepBlocks = sizeof(U) == 4 && VW <= 1 ? 3 : 2;
constexpr uint32_t kSortInc = 0x80000000u;

int sort_tiles(long long n) { return (int)((n + kSweepTile - 1) / kSweepTile); }

// Lanes whose digit (bits shift .. shift + 7 of the key) equals this lane's:
// a ballot per bit.
template <typename U>
__device__ __forceinline__ unsigned equal_digits(U key, int shift) {
  const unsigned d = (unsigned)(key >> shift);
  unsigned peers = kFull;
#pragma unroll
  for (int b = 0; b < 8; ++b)
    asm volatile("{\n .reg .pred p;\n .reg .b32 t, v;\n"
        " and.b32 t, %1, %2;\n setp.ne.u32 p, t, 0;\n"
        " vote.sync.ballot.b32 v, p, 0xffffffff;\n"
        " @!p not.b32 v, v;\n and.b32 %0, %0, v;\n}\n"
        : "+r"(peers)
        : "r"(d), "r"(1u << b));
  return peers;
}

// Places in a tile, below 2^16: two a register.
struct Places {
  uint32_t p[kSortItems / 2];
  __device__ __forceinline__ uint32_t get(int e) const { return (p[e / 2] >> (16 * (e & 1))) & 0xffffu; }
  __device__ __forceinline__ void set(int e, uint32_t v) {
    p[e / 2] = (e & 1) ? __byte_perm(p[e / 2], v, 0x5410) : __byte_perm(p[e / 2], v, 0x3254);
  }
};

// Ranks a warp's keys (rows of 32, in row then lane order) among its equal
// digits; cnt: the warp's 256 counters, zero before, its digit counts after.
// FULL: every row holds 32 keys; else the first `count` places do.
template <bool FULL, typename U>
__device__ __forceinline__ void warp_rank(const U (&key)[kSortItems], Places& rank,
                                          int shift, int count, int lane, uint32_t* cnt) {
  const unsigned lt = (1u << lane) - 1u;
  constexpr int kG = 4;  // rows whose masks, which do not depend on one another, come first
#pragma unroll
  for (int e0 = 0; e0 < kSortItems; e0 += kG) {
    unsigned peers[kG];
#pragma unroll
    for (int g = 0; g < kG; ++g)
      if (FULL || 32 * (e0 + g) < count) {
        peers[g] = equal_digits(key[e0 + g], shift);
        if (!FULL) peers[g] &= low_mask(count - 32 * (e0 + g));
      }
#pragma unroll
    for (int g = 0; g < kG; ++g)
      if (FULL || 32 * (e0 + g) < count) {
        uint32_t* c = cnt + ((unsigned)(key[e0 + g] >> shift) & 255u);
        const bool ok = FULL || lane < count - 32 * (e0 + g);
        const unsigned below = __popc(peers[g] & lt);
        const uint32_t before = ok ? *c : 0u;
        __syncwarp();
        if (ok && below == 0u) *c = before + __popc(peers[g]);
        __syncwarp();
        rank.set(e0 + g, before + below);
      }
  }
}

// Turns the warps' digit counts s_cnt[warp][256] into each (warp, digit)'s
// first place in the tile sorted by digit; threads 0..255 return their
// digit's count and, in *start, its first place.  s_warp: 8 words.
template <int WARPS>
__device__ __forceinline__ uint32_t place_digits(uint32_t* s_cnt, uint32_t* s_warp, uint32_t* start) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t tot = 0, x = 0;
  if (tid < 256) {
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const uint32_t c = s_cnt[w * 256 + tid];
      s_cnt[w * 256 + tid] = tot;
      tot += c;
    }
    x = tot;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
  }
  __syncthreads();
  if (tid < 256) {
    x -= tot;
    for (int w = 0; w < warp; ++w) x += s_warp[w];
    *start = x;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) s_cnt[w * 256 + tid] += x;
  }
  return tot;
}

// Digit counts of all keys for `npass` passes from digit `first`:
// hist[p * 256 + digit], zero before.  Bound by the shared-memory atomics,
// about eight lanes a cycle whether or not they collide (100 M int32 keys, four
// digits: 177 us; sixteen copies of every counter measured the same).
template <typename U>
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const U* __restrict__ keys, long long n,
                                                             int first, int npass,
                                                             uint32_t* __restrict__ hist,
                                                             KeyOrder<U> ord) {
  constexpr int kD = (int)sizeof(U);
  __shared__ uint32_t s_h[kD * 256];
  for (int i = threadIdx.x; i < kD * 256; i += kSortThreads) s_h[i] = 0;
  __syncthreads();
  const long long stride = (long long)gridDim.x * kSortThreads;
  for (long long i = (long long)blockIdx.x * kSortThreads + threadIdx.x; i < n; i += 4 * stride) {
    U k[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) k[u] = i + u * stride < n ? keys[i + u * stride] : (U)0;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i + u * stride < n) {
        const U x = ord.load(k[u]) >> (8 * first);
#pragma unroll
        for (int p = 0; p < kD; ++p)
          if (p < npass) atomicAdd(&s_h[p * 256 + ((unsigned)(x >> (8 * p)) & 255u)], 1u);
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < npass * 256; i += kSortThreads)
    if (s_h[i]) atomicAdd(hist + i, s_h[i]);
}

// Shared memory above 48 KB is opted into once per device and kernel; a
// failure shows as the launch's error.
void opt_in_smem(const void* kernel, size_t smem, int* done) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || done[dev]) return;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
      cudaSuccess)
    done[dev] = 1;
}

// Keys of `tile` whose digit is d, counted from the keys (a wait ran out).
template <typename U>
__device__ __forceinline__ uint32_t count_digit(const U* kin, long long n, int tile, int shift,
                                             unsigned d, KeyOrder<U> ord) {
  const long long b = (long long)tile * kSweepTile;
  const long long e = b + kSweepTile < n ? b + kSweepTile : n;
  uint32_t c = 0;
#pragma unroll 1
  for (long long i = b; i < e; ++i) c += ((unsigned)(ord.load(kin[i]) >> shift) & 255u) == d;
  return c;
}

// Keys of digit d in the tiles before `tile`.  kLook states are read at a time.
constexpr int kLook = 4;

template <typename U>
__device__ __forceinline__ uint32_t digit_look_back(const uint32_t* state, int tile, unsigned d,
                                                    const U* kin, long long n, int shift,
                                                    const KeyOrder<U>& ord, unsigned polls) {
  uint32_t prefix = 0;
  int t = tile - 1;
  Spin spin(polls);
  while (t >= 0) {
    uint32_t v[kLook];
#pragma unroll
    for (int q = 0; q < kLook; ++q)
      v[q] = t >= q ? ld_relaxed(state + (long long)(t - q) * 256 + d) : kSortInc;
    bool waiting = false;
#pragma unroll
    for (int q = 0; q < kLook; ++q) {
      if (t < 0 || waiting) continue;
      if (v[q] & kSortInc) {
        prefix += v[q] & ~kSortInc;
        t = -1;
      } else if (v[q]) {
        prefix += v[q] - 1u;
        --t;
      } else {
        waiting = true;
      }
    }
    if (waiting && !spin.more()) {
      prefix += count_digit(kin, n, t, shift, d, ord);
      --t;
    }
  }
  return prefix;
}

template <typename U>
constexpr size_t sweep_smem(int vwords) {
  return (size_t)kSweepTile * sizeof(U) + (vwords ? (size_t)kSweepTile * 4 : 0) +
         (size_t)kSweepWarps * 256 * 4 + 256 * 4 + 16 * 4;
}

// One tile of a pass.  VW: 32-bit words a value (0: keys only); FULL: the
// tile holds kSweepTile elements.
template <typename U, int VW, bool FULL>
__device__ __forceinline__ void sweep_tile(const U* __restrict__ kin, U* __restrict__ kout,
                                           const uint32_t* __restrict__ vin,
                                           uint32_t* __restrict__ vout, long long n, int shift,
                                           const uint32_t* __restrict__ hist,
                                           uint32_t* __restrict__ state, int tile,
                                           const KeyOrder<U>& ord, unsigned polls, U* s_key,
                                           uint32_t* s_val, uint32_t* s_cnt, uint32_t* s_dst,
                                           uint32_t* s_warp) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const long long tb = (long long)tile * kSweepTile;
  const int valid = FULL ? kSweepTile : (int)(n - tb);
  const int l0 = warp * (kSortItems * 32) + lane;  // the thread's first element of the tile
  const U* kt = kin + tb + l0;
  U key[kSortItems];
  Places rank;
#pragma unroll
  for (int e = 0; e < kSortItems; ++e)
    key[e] = FULL || l0 + 32 * e < valid ? __ldcs(kt + 32 * e) : (U)0;
#pragma unroll
  for (int e = 0; e < kSortItems; ++e) key[e] = ord.load(key[e]);
  uint32_t* cnt = s_cnt + warp * 256;
  warp_rank<FULL>(key, rank, shift, valid - (l0 - lane), lane, cnt);
  __syncthreads();
  uint32_t lstart = 0;
  const uint32_t tot = place_digits<kSweepWarps>(s_cnt, s_warp, &lstart);
  uint32_t* mine = state + (long long)tile * 256 + tid;
  if (tid < 256) st_relaxed(mine, tile == 0 ? kSortInc | tot : tot + 1u);
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kSortItems; ++e)
    if (FULL || l0 + 32 * e < valid) {
      const uint32_t at = rank.get(e) + cnt[(unsigned)(key[e] >> shift) & 255u];  // its place in the tile
      rank.set(e, at);
      s_key[at] = key[e];
    }
  uint32_t v[VW ? kSortItems : 1];
  auto load_values = [&](int q) {
    const uint32_t* vt = vin + (tb + l0) * VW + q;
#pragma unroll
    for (int e = 0; e < kSortItems; ++e)
      if (FULL || l0 + 32 * e < valid) v[e] = VW == 1 ? __ldcs(vt + 32 * e) : vt[32 * e * VW];
  };
  auto place_values = [&]() {
#pragma unroll
    for (int e = 0; e < kSortItems; ++e)
      if (FULL || l0 + 32 * e < valid) s_val[rank.get(e)] = v[e];
  };
  if constexpr (VW > 0) load_values(0);  // in flight during the look-back
  if (tid < 256) {
    // the digit's start over all keys: an exclusive scan of the 256 counts
    const uint32_t h = hist[tid];
    uint32_t x = h;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[8 + warp] = x;
    asm volatile("bar.sync 1, 256;" ::: "memory");  // the 256 digit threads
    x -= h;
    for (int w = 0; w < warp; ++w) x += s_warp[8 + w];
    const uint32_t before = digit_look_back(state, tile, (unsigned)tid, kin, n, shift, ord,
                                            polls);
    if (tile > 0) st_relaxed(mine, kSortInc | (before + tot));
    s_dst[tid] = x + before - lstart;
  }
  if constexpr (VW > 0) place_values();
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kSortItems; ++e) {
    const int j = tid + e * kSweepThreads;
    if (FULL || j < valid) {
      const U k = s_key[j];
      const uint32_t at = s_dst[(unsigned)(k >> shift) & 255u] + j;
      kout[at] = ord.store(k);
      if constexpr (VW > 0) vout[(long long)at * VW] = s_val[j];
    }
  }
  if constexpr (VW > 1) {
#pragma unroll 1
    for (int q = 1; q < VW; ++q) {
      load_values(q);
      __syncthreads();  // the previous word has left
      place_values();
      __syncthreads();
#pragma unroll
      for (int e = 0; e < kSortItems; ++e) {
        const int j = tid + e * kSweepThreads;
        if (FULL || j < valid) {
          const uint32_t at = s_dst[(unsigned)(s_key[j] >> shift) & 255u] + j;
          vout[(long long)at * VW + q] = s_val[j];
        }
      }
    }
  }
}

// One pass: hist: the digits' counts over all keys.
template <typename U, int VW>
__global__ void __launch_bounds__(kSweepThreads, (kSweepBlocks<U, VW>))
    k_radix_sweep(const U* __restrict__ kin, U* __restrict__ kout, const uint32_t* __restrict__ vin,
                  uint32_t* __restrict__ vout, long long n, int shift,
                  const uint32_t* __restrict__ hist, uint32_t* __restrict__ state,
                  unsigned* __restrict__ ticket, KeyOrder<U> ord, unsigned polls) {
  extern __shared__ unsigned long long s_dyn[];
  U* s_key = reinterpret_cast<U*>(s_dyn);                            // [kSweepTile]
  uint32_t* s_val = reinterpret_cast<uint32_t*>(s_key + kSweepTile);  // [kSweepTile] if VW
  uint32_t* s_cnt = s_val + (VW ? kSweepTile : 0);                    // [kSweepWarps][256]
  uint32_t* s_dst = s_cnt + kSweepWarps * 256;  // [256] global place of the run - its local start
  uint32_t* s_warp = s_dst + 256;              // [16]
  __shared__ int s_tile;
  if (threadIdx.x == 0) s_tile = (int)atomicAdd(ticket, 1u);
  for (int i = threadIdx.x; i < kSweepWarps * 256; i += kSweepThreads) s_cnt[i] = 0;
  __syncthreads();
  const int tile = s_tile;
  if ((long long)tile * kSweepTile >= n) return;
  if ((long long)(tile + 1) * kSweepTile <= n)
    sweep_tile<U, VW, true>(kin, kout, vin, vout, n, shift, hist, state, tile, ord, polls, s_key,
                            s_val, s_cnt, s_dst, s_warp);
  else
    sweep_tile<U, VW, false>(kin, kout, vin, vout, n, shift, hist, state, tile, ord, polls, s_key,
                             s_val, s_cnt, s_dst, s_warp);
}

// At most kSortTile elements: every pass in one block's shared memory, the
// elements' first places carried beside the keys; the values are moved once,
// at the end (each word of every row is read before any is written).
template <typename U>
constexpr size_t block_sort_smem() {
  return (size_t)kSortTile * (sizeof(U) + 2) + (size_t)kSortWarps * 256 * 4 + 16 * 4;
}

template <typename U>
__global__ void __launch_bounds__(kSortThreads, 1)
    k_sort_block(U* keys, uint32_t* vals, int vwords, int n, int passes, KeyOrder<U> ord) {
  extern __shared__ unsigned long long s_dyn[];
  U* s_key = reinterpret_cast<U*>(s_dyn);                            // [kSortTile]
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(s_key + kSortTile);  // [kSortWarps][256]
  uint32_t* s_warp = s_cnt + kSortWarps * 256;                       // [8]
  uint16_t* s_src = reinterpret_cast<uint16_t*>(s_warp + 16);        // [kSortTile]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rows = (n + kSortThreads - 1) / kSortThreads;  // rows of 32 a warp
  const int w0 = warp * rows * 32;
  const int count = min(n - w0, rows * 32);  // the warp's keys (<= 0: none)
  uint32_t* cnt = s_cnt + warp * 256;
  U key[kSortItems];
  Places rank;
  uint16_t src[kSortItems];
#pragma unroll
  for (int e = 0; e < kSortItems; ++e) {
    const int li = w0 + 32 * e + lane;
    if (e < rows && li < n) {
      key[e] = ord.load(keys[li]);
      src[e] = (uint16_t)li;
    }
  }
  for (int p = 0; p < passes; ++p) {
    const int shift = 8 * p;
    if (p > 0) {
#pragma unroll
      for (int e = 0; e < kSortItems; ++e) {
        const int li = w0 + 32 * e + lane;
        if (e < rows && li < n) {
          key[e] = s_key[li];
          src[e] = s_src[li];
        }
      }
    }
    for (int i = tid; i < kSortWarps * 256; i += kSortThreads) s_cnt[i] = 0;
    __syncthreads();
    warp_rank<false>(key, rank, shift, count, lane, cnt);
    __syncthreads();
    uint32_t start;
    place_digits<kSortWarps>(s_cnt, s_warp, &start);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kSortItems; ++e) {
      if (e < rows && w0 + 32 * e + lane < n) {
        const uint32_t at = cnt[(unsigned)(key[e] >> shift) & 255u] + rank.get(e);
        s_key[at] = key[e];
        s_src[at] = src[e];
      }
    }
    __syncthreads();
  }
  for (int j = tid; j < n; j += kSortThreads) keys[j] = ord.store(s_key[j]);
  for (int q = 0; q < vwords; ++q) {
    uint32_t v[kSortItems];
#pragma unroll
    for (int e = 0; e < kSortItems; ++e) {
      const int j = tid + e * kSortThreads;
      if (j < n) v[e] = vals[(int)s_src[j] * vwords + q];
    }
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kSortItems; ++e) {
      const int j = tid + e * kSortThreads;
      if (j < n) vals[j * vwords + q] = v[e];
    }
  }
}

// ---- single-pass compaction ------------------------------------------------
//
// StreamCompact and Unique in one read of the stencil (or keys), on the
// single-pass driver: a tile's kept elements are counted as it lands, the
// look-back warp finds its offset, and the compute warps write the tile's
// kept elements at their places: the key itself (Unique), the value gathered
// from its array (StreamCompact with an input), or the element's index.
//
// Unique writes in place: a tile's kept keys go below its own start, into
// tiles that have already loaded (their counts are published before this
// tile's offset is known); the only place it shares with a later read is the
// key before the next tile, which it rewrites only when no key before it was
// dropped, that is with the same key.
struct CompactOp {
  int mode;          // 0 stencil int32 != 0; 1 stencil float != 0; 2 key differs from the previous
  int key_kind;      // mode 2: 0 unsigned, 1 signed, 2 float (compared as values)
  const void* test;  // the staged array: stencil or keys
  const uint32_t* values;  // modes 0 / 1: the values to gather (NULL: the index instead)
  int words;               // 32-bit words a value
  void* out;
};

// S: the staged element (uint32_t or unsigned long long).  W: 32-bit words a
// gathered value (StreamCompact with an input: the tile's values are
// prefetched into L2 by one bulk copy when the tile is taken, and a lane
// loads its chunks' W x 16 bytes of values four chunks at a time, before
// their stores), or 0 (Unique's keys, or indices).  UNIQUE: keep the keys that
// differ from the one before; else keep where the stencil is non-zero under
// `mask` (all bits of an int, all but the sign of a float).  The key before a
// tile (Unique) is read by thread 0 when the tile lands, before this tile
// writes anything, and used by thread 0 alone.
//
// A lane keeps its elements' kept bits (the carry) from the sum to the
// output, and four chunks' counts, at most 128 each, are scanned as the bytes
// of one word.  (Testing the elements a second time and scanning each chunk
// took 46 instructions a row of 32, from eight warps: 351 us for 100 M int32
// and their values, 0.92 GB, now 185.)
//
// Values of two words and more leave a chunk (128 elements) at a time through
// shared memory, consecutive lanes storing consecutive words: a lane that stores
// its own elements' words covers a part of as many sectors as it stores words,
// and with sixteen warps in turn few of them meet in L1: 20 M values of three words,
// all kept, 85 M sector writes in L2 and 307 us, now 166; half of them kept, 156
// and 133.  (At 60 M, a twentieth kept, it costs a little: 226 and 236 us; storing
// such chunks from the lanes, behind a test, took 242.)
template <int W>
struct alignas(W == 4 ? 16 : W == 2 ? 8 : 4) Row {
  uint32_t w[W];
};

template <typename S, int W, bool UNIQUE>
struct CompactPass {
  typedef S Staged;
  typedef uint32_t Sum;  // counts: fewer than 2^31 elements
  static constexpr int E = 16 / (int)sizeof(S);
  static constexpr int kTileElems = kSElems, kSChunks = Ring<S>::chunks;
  struct Chunk { S e[E]; };
  struct Carry { unsigned kept; };  // bit c E + e: element e of the lane's chunk c
  static_assert(kSChunks * E <= 32, "a lane's kept bits in one word");
  uint32_t mask;
  int key_kind;
  const S* src;
  const uint32_t* values;
  int vec;  // values 16-byte aligned
  void* out;
  long long n;

  __device__ void on_take(int t) const {
    if (W > 0 && vec)  // the tile's values, into L2 ahead of the gather
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(
                       values + (long long)t * kTileElems * W),
                   "r"((unsigned)(kTileElems * W * 4))
                   : "memory");
  }
  __device__ void on_land(int k, long long b, unsigned long long* aux) const {
    aux[k] = UNIQUE && b > 0 ? (unsigned long long)src[b - 1] : 0ull;
  }
  __device__ bool keep(S x, S prev, bool first) const {
    if (!UNIQUE) return ((uint32_t)x & mask) != 0;
    if (first) return true;
    if (sizeof(S) == 4 && key_kind == 2)
      return __uint_as_float((uint32_t)x) != __uint_as_float((uint32_t)prev);
    return x != prev;
  }
  __device__ Sum thread_sum(S* s_data, int k, long long b, int warp, int lane,
                            const unsigned long long* aux, Carry& carry) const {
    const S* p = lane_chunk0(s_data, warp, lane);
    unsigned kept = 0;
#pragma unroll
    for (int c = 0; c < kSChunks; ++c, p += 32 * E) {
      const Chunk x = *reinterpret_cast<const Chunk*>(p);
      S prev = 0;
      if (UNIQUE && b + (p - s_data) > 0) prev = p > s_data ? p[-1] : (S)aux[k];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        if (keep(x.e[e], prev, b + (p - s_data) + e == 0)) kept |= 1u << (c * E + e);
        prev = x.e[e];
      }
    }
    if (b + kTileElems > n) {  // the ragged tile: the elements past n
      const long long i0 = b + (lane_chunk0(s_data, warp, lane) - s_data);
#pragma unroll
      for (int c = 0; c < kSChunks; ++c)
#pragma unroll
        for (int e = 0; e < E; ++e)
          if (i0 + 32 * c * E + e >= n) kept &= ~(1u << (c * E + e));
    }
    carry.kept = kept;
    return __popc(kept);
  }
  // the W words of each of the lane's E elements of chunk c
  __device__ void load_values(long long wb, int c, int lane, uint4* v) const {
    if constexpr (W > 0) {
      const long long i0 = wb + (32 * c + lane) * E;
      if (vec && i0 + E <= n) {
        const uint4* src4 = reinterpret_cast<const uint4*>(values + i0 * W);
#pragma unroll
        for (int q = 0; q < W; ++q) v[q] = __ldcs(src4 + q);
      } else {
        uint32_t* u = reinterpret_cast<uint32_t*>(v);
#pragma unroll
        for (int e = 0; e < E; ++e)
#pragma unroll
          for (int q = 0; q < W; ++q) u[e * W + q] = i0 + e < n ? values[(i0 + e) * W + q] : 0u;
      }
    }
  }
  __device__ void finish(S* s_data, long long b, Sum run, int warp, int lane, const Carry& carry,
                         bool) const {
    constexpr int kV = W > 0 ? W : 1;
    constexpr int kG = 4;  // chunks whose values are loaded before any of their stores
    const long long wb = b + (lane_chunk0(s_data, warp, 0) - s_data);  // the warp's first element
    const S* p = lane_chunk0(s_data, warp, lane);
    unsigned kept = carry.kept;
#pragma unroll 1
    for (int c0 = 0; c0 < kSChunks; c0 += kG, kept >>= kG * E & 31) {
      uint4 vals[kG][kV];
#pragma unroll
      for (int g = 0; g < kG; ++g) load_values(wb, c0 + g, lane, vals[g]);
      // byte g: the chunk's kept elements before this lane, then in all
      unsigned own = 0;
#pragma unroll
      for (int g = 0; g < kG; ++g)
        own |= __popc((kept >> (g * E)) & ((1u << E) - 1u)) << (8 * g);
      const unsigned incl = warp_inclusive(own, lane), before = incl - own,
                     all = __shfl_sync(kFull, incl, 31);
#pragma unroll
      for (int g = 0; g < kG; ++g) {
        const unsigned count = (all >> (8 * g)) & 0xffu;
        if constexpr (W > 1) {
          // through the warp's part of the staged stencil, which nothing reads again
          Row<W>* const row = reinterpret_cast<Row<W>*>(lane_chunk0(s_data, warp, 0));
          const uint32_t* const words = reinterpret_cast<const uint32_t*>(row);
          const Row<W>* const v = reinterpret_cast<const Row<W>*>(vals[g]);
          unsigned at = (before >> (8 * g)) & 0xffu;
#pragma unroll
          for (int e = 0; e < E; ++e)
            if ((kept >> (g * E + e)) & 1u) row[at++] = v[e];
          __syncwarp();
          uint32_t* const dst = static_cast<uint32_t*>(out) + (unsigned long long)run * W;
#pragma unroll 4
          for (unsigned w = lane; w < count * W; w += 32) dst[w] = words[w];
          __syncwarp();
          run += count;
          continue;
        }
        unsigned long long pos = run + ((before >> (8 * g)) & 0xffu);
        run += count;
        Chunk x;
        if (UNIQUE) x = *reinterpret_cast<const Chunk*>(p + 32 * (c0 + g) * E);
        const long long i0 = wb + (32 * (c0 + g) + lane) * E;
        const uint32_t* u = reinterpret_cast<const uint32_t*>(vals[g]);
#pragma unroll
        for (int e = 0; e < E; ++e)
          if ((kept >> (g * E + e)) & 1u) {
            if constexpr (W > 0) {
              uint32_t* dst = static_cast<uint32_t*>(out) + pos * W;
#pragma unroll
              for (int q = 0; q < W; ++q) dst[q] = u[e * W + q];
            } else if (UNIQUE) {
              static_cast<S*>(out)[pos] = x.e[e];
            } else {
              static_cast<int32_t*>(out)[pos] = (int32_t)(i0 + e);
            }
            ++pos;
          }
      }
    }
  }
  __device__ void store(S*, long long) const {}
};

template <typename S, int W, bool UNIQUE>
__global__ void __launch_bounds__(kSBlock, 1)
    k_compact_single(CompactPass<S, W, UNIQUE> op, long long n, int tiles, ScanCtl* ctl,
                     char* states, int bulk, unsigned polls) {
  single_pass(op, n, tiles, ctl, states, bulk, polls);
}

template <typename S, int W, bool UNIQUE = false>
void compact_single_w(const CompactOp& a, long long n, char* scratch, int num_sms,
                      cudaStream_t s) {
  const CompactPass<S, W, UNIQUE> op{a.mode == 1 ? 0x7fffffffu : ~0u,
                                     a.key_kind,
                                     static_cast<const S*>(a.test),
                                     a.values,
                                     (reinterpret_cast<uintptr_t>(a.values) & 15) == 0,
                                     a.out,
                                     n};
  const int bulk = (reinterpret_cast<uintptr_t>(a.test) & 15) == 0;
  launch_single_pass(k_compact_single<S, W, UNIQUE>, op, n, bulk, scratch, num_sms, s);
}

// Kept elements into op.out, the count to ctl->total on the device.
template <typename S>
void compact_single(const CompactOp& op, long long n, char* scratch, int num_sms, cudaStream_t s) {
  if (op.mode == 2) {
    compact_single_w<S, 0, true>(op, n, scratch, num_sms, s);
    return;
  }
  if constexpr (sizeof(S) == 4) {
    switch (op.values ? op.words : 0) {
      case 1: compact_single_w<S, 1>(op, n, scratch, num_sms, s); break;
      case 2: compact_single_w<S, 2>(op, n, scratch, num_sms, s); break;
      case 3: compact_single_w<S, 3>(op, n, scratch, num_sms, s); break;
      case 4: compact_single_w<S, 4>(op, n, scratch, num_sms, s); break;
      default: compact_single_w<S, 0>(op, n, scratch, num_sms, s); break;
    }
  }
}

// ---- sort driver -----------------------------------------------------------

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// keys and values of the odd passes; 1 KB per kPTile elements for digit counts
// and tile states; the ticket.  (The scratch's size is the callers' to keep: it
// still counts the sums of a scan of 256 counters a tile, of which the ticket
// takes the first word.)
struct SortLayout {
  size_t ktmp, vtmp, hist, ticket, total;
};

SortLayout sort_layout(long long n, int key_bytes, int value_bytes) {
  const long long tiles = ptiles(n);
  const long long hn = 256 * tiles;
  SortLayout L;
  L.ktmp = 0;
  L.vtmp = align256(L.ktmp + (size_t)n * key_bytes);
  L.hist = align256(L.vtmp + (size_t)n * value_bytes);
  L.ticket = align256(L.hist + (size_t)hn * 4);
  L.total = align256(L.ticket + (size_t)sum_slots(hn) * 4);
  return L;
}

template <typename U, int VW>
void launch_sweep(const U* kin, U* kout, const uint32_t* vin, uint32_t* vout, long long n, int shift,
                  const uint32_t* hist, uint32_t* state, unsigned* ticket, KeyOrder<U> ord,
                  unsigned polls, cudaStream_t s) {
  static int opted[64] = {};
  constexpr size_t smem = sweep_smem<U>(VW);
  opt_in_smem((const void*)k_radix_sweep<U, VW>, smem, opted);
  k_radix_sweep<U, VW><<<sort_tiles(n), kSweepThreads, smem, s>>>(kin, kout, vin, vout, n, shift,
                                                                hist, state, ticket, ord, polls);
}

// passes: 8-bit digits to sort, least significant first (an even count, so
// the result ends in keys/vals); plain = the keys are unsigned, ascending and
// need no order mapping; polls: the most polls of a look-back's wait.
//
// Up to kSortTile elements are one launch of one block.  Longer arrays keep
// the tile states, the digit counts and the tickets in the scratch's
// histogram section: 1 KB per 4096 elements, of which the states take 1 KB
// per kSweepTile = 6144; the counts of as many passes as fit beside them
// (all, from 94 K elements) are taken at a time.
template <typename U>
void radix_sort(U* keys, uint32_t* vals, int vwords, long long n, int kind, bool desc,
                char* scratch, int num_sms, cudaStream_t s, int passes = (int)sizeof(U),
                bool plain = false, unsigned polls = kSpinIters) {
  if (n <= kSortTile) {
    static int opted[64] = {};
    const KeyOrder<U> ord{kind, desc, !plain, !plain};
    opt_in_smem((const void*)k_sort_block<U>, block_sort_smem<U>(), opted);
    k_sort_block<U><<<1, kSortThreads, block_sort_smem<U>(), s>>>(keys, vals, vwords, (int)n, passes,
                                                                 ord);
    return;
  }
  const SortLayout L = sort_layout(n, (int)sizeof(U), 4 * vwords);
  U* ktmp = reinterpret_cast<U*>(scratch + L.ktmp);
  uint32_t* vtmp = reinterpret_cast<uint32_t*>(scratch + L.vtmp);
  const int tiles = sort_tiles(n), spare = ptiles(n) - tiles;  // KB beside the states
  const int group = spare < passes ? spare : passes;           // >= 1 for n > kSortTile
  // ... [counts of `group` passes][states][ticket]
  uint32_t* state = reinterpret_cast<uint32_t*>(scratch + L.hist) + 256ll * spare;
  uint32_t* hist = state - 256ll * group;
  unsigned* ticket = reinterpret_cast<unsigned*>(scratch + L.ticket);
  const int bh = resident_blocks(k_radix_hist<U>, kSortThreads, 0, num_sms,
                                 (n + 4 * kSortThreads - 1) / (4 * kSortThreads));
  for (int p = 0; p < passes; ++p) {
    const U* ksrc = (p & 1) ? ktmp : keys;
    U* kdst = (p & 1) ? keys : ktmp;
    const uint32_t* vsrc = (p & 1) ? vtmp : vals;
    uint32_t* vdst = (p & 1) ? vals : vtmp;
    const KeyOrder<U> ord{kind, desc, !plain && p == 0, !plain && p == passes - 1};
    const int at = p % group;
    // the states and the ticket, and before a group of passes its digit counts
    uint32_t* clear = at == 0 ? hist : state;
    cudaMemsetAsync(clear, 0, (size_t)((char*)(ticket + 1) - (char*)clear), s);
    const int counted = passes - p < group ? passes - p : group;
    if (at == 0) k_radix_hist<U><<<bh, kSortThreads, 0, s>>>(ksrc, n, p, counted, hist, ord);
    const uint32_t* h = hist + 256 * at;
    switch (vwords) {
      case 0: launch_sweep<U, 0>(ksrc, kdst, vsrc, vdst, n, 8 * p, h, state, ticket, ord, polls, s); break;
      case 1: launch_sweep<U, 1>(ksrc, kdst, vsrc, vdst, n, 8 * p, h, state, ticket, ord, polls, s); break;
      case 2: launch_sweep<U, 2>(ksrc, kdst, vsrc, vdst, n, 8 * p, h, state, ticket, ord, polls, s); break;
      case 3: launch_sweep<U, 3>(ksrc, kdst, vsrc, vdst, n, 8 * p, h, state, ticket, ord, polls, s); break;
      default: launch_sweep<U, 4>(ksrc, kdst, vsrc, vdst, n, 8 * p, h, state, ticket, ord, polls, s); break;
    }
  }
}

// ---- bounds -------------------------------------------------------------------

template <typename T, bool UPPER>
__global__ void k_bounds(const T* __restrict__ sorted, long long n, const T* values, long long m,
                         int32_t* out) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (long long)gridDim.x * blockDim.x) {
    const T v = values[i];
    long long lo = 0, hi = n;  // first index whose element is >= v (> v for UPPER)
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      const T x = sorted[mid];
      const bool before = UPPER ? !(v < x) : (x < v);
      if (before) lo = mid + 1;
      else hi = mid;
    }
    out[i] = (int32_t)lo;
  }
}

}  // namespace

namespace {

int prim_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms < 1) sms = 1;
  }
  return sms;
}

int bad(const char* msg) {
  set_last_error(msg);
  return DAX_GB300_ERROR_BAD_VALUE;
}

int launched(const char* where) {
  const cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) return DAX_GB300_SUCCESS;
  set_last_error(std::string(where) + ": " + cudaGetErrorString(e));
  return DAX_GB300_ERROR_CUDA;
}

int type_bytes(int t) {
  switch (t) {
    case DAX_GB300_TYPE_I32: case DAX_GB300_TYPE_U32: case DAX_GB300_TYPE_F32: return 4;
    case DAX_GB300_TYPE_I64: case DAX_GB300_TYPE_U64: return 8;
    default: return 0;
  }
}

int type_kind(int t) {
  return (t == DAX_GB300_TYPE_F32) ? 2 : ((t == DAX_GB300_TYPE_I32 || t == DAX_GB300_TYPE_I64) ? 1 : 0);
}

bool size_ok(long long n) { return n >= 0 && n <= 2147483647ll; }

int read_back(void* host, const void* dev, size_t bytes, cudaStream_t s, const char* what) {
  cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess) return DAX_GB300_SUCCESS;
  set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
  return DAX_GB300_ERROR_CUDA;
}

// The element count of a single-pass compaction, or the total of a scan
// (synchronises the stream); a wait that ran out is DAX_GB300_ERROR_TIMEOUT.
int read_count(int64_t* h_count, const char* scratch, cudaStream_t s, const char* what) {
  ScanCtl ctl;
  int st = read_back(&ctl, scratch, sizeof(ctl), s, what);
  if (st) return st;
  if (ctl.error) {
    set_last_error(std::string(what) + ": a wait expired on the device");
    return DAX_GB300_ERROR_TIMEOUT;
  }
  *h_count = (int64_t)ctl.total;
  return DAX_GB300_SUCCESS;
}

size_t scan_bytes(long long n) { return align256((size_t)sum_slots(n) * 8); }

// dax_gb300_scan: the reduce-then-scan sums (floats) or the single-pass
// states (integers), whichever is larger.
size_t public_scan_bytes(long long n) {
  const size_t a = scan_bytes(n), b = align256(single_scan_bytes<int64_t>(n));
  return a > b ? a : b;
}

size_t keep_bytes(long long n) { return align256((size_t)sum_slots(n) * 8); }

}  // namespace
}  // namespace daxgb

namespace daxgb {

void sort_unsigned_bits(void* keys, long long n, bool wide, int bits, void* scratch,
                        cudaStream_t s) {
  if (n < 2) return;
  int passes = (bits + 7) / 8;
  passes += passes & 1;
  const int kind = type_kind(wide ? DAX_GB300_TYPE_U64 : DAX_GB300_TYPE_U32);
  if (wide)
    radix_sort<unsigned long long>(static_cast<unsigned long long*>(keys), nullptr, 0, n, kind,
                                   false, static_cast<char*>(scratch), prim_sms(), s,
                                   passes < 8 ? passes : 8, true);
  else
    radix_sort<uint32_t>(static_cast<uint32_t*>(keys), nullptr, 0, n, kind, false,
                         static_cast<char*>(scratch), prim_sms(), s, passes < 4 ? passes : 4,
                         true);
}

}  // namespace daxgb

using daxgb::align256;

extern "C" {

size_t dax_gb300_scan_scratch_bytes(int64_t n) {
  return daxgb::public_scan_bytes(n < 1 ? 1 : n);
}

int dax_gb300_scan(const void* d_in, void* d_out, int64_t n, int type, int exclusive,
                   void* d_scratch, size_t scratch_bytes, void* h_total, void* stream) {
  using namespace daxgb;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!size_ok(n)) return bad("scan length must be in [0, 2^31 - 1]");
  const int tb = type_bytes(type);
  if (!tb) return bad("unknown element type");
  if (n == 0) {
    if (h_total) memset(h_total, 0, (size_t)tb);
    return DAX_GB300_SUCCESS;
  }
  if (!d_in || !d_out || !d_scratch) return bad("NULL input, output or scratch");
  if (scratch_bytes < public_scan_bytes(n))
    return bad("scratch smaller than dax_gb300_scan_scratch_bytes()");
  const int sms = prim_sms();
  char* sc = static_cast<char*>(d_scratch);
  const bool ex = exclusive != 0;
  switch (type) {
    case DAX_GB300_TYPE_I32: scan_single<int32_t>((const int32_t*)d_in, (int32_t*)d_out, n, ex, sc, sms, s); break;
    case DAX_GB300_TYPE_U32: scan_single<uint32_t>((const uint32_t*)d_in, (uint32_t*)d_out, n, ex, sc, sms, s); break;
    case DAX_GB300_TYPE_F32: scan_t<float>((const float*)d_in, (float*)d_out, n, ex, sc, sms, s); break;
    case DAX_GB300_TYPE_I64: scan_single<int64_t>((const int64_t*)d_in, (int64_t*)d_out, n, ex, sc, sms, s); break;
    default: scan_single<unsigned long long>((const unsigned long long*)d_in, (unsigned long long*)d_out, n, ex, sc, sms, s); break;
  }
  int st = launched("scan kernels");
  if (st || !h_total) return st;
  if (type == DAX_GB300_TYPE_F32)  // the scanned tile sums end with the grand total
    return read_back(h_total, sc + (size_t)ptiles(n) * tb, (size_t)tb, s, "reading the scan total");
  // the single pass: the error word and the total (little-endian, as wide as the element)
  int64_t total = 0;
  st = read_count(&total, sc, s, "reading the scan total");
  if (!st) memcpy(h_total, &total, (size_t)tb);
  return st;
}

int dax_gb300_selfcheck_scan_wait(const int32_t* d_in, int32_t* d_out, int64_t n, uint32_t polls,
                                  int lost, void* d_scratch, size_t scratch_bytes, int32_t* h_total,
                                  void* stream) {
  using namespace daxgb;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!size_ok(n) || n <= kSElems) return bad("the scan must have two tiles or more");
  if (!d_in || !d_out || !d_scratch || !h_total) return bad("NULL argument");
  if (scratch_bytes < public_scan_bytes(n))
    return bad("scratch smaller than dax_gb300_scan_scratch_bytes()");
  scan_single<int32_t>(d_in, d_out, n, false, static_cast<char*>(d_scratch), prim_sms(), s,
                       polls < kSpinIters ? polls : kSpinIters, lost != 0);
  int st = launched("scan kernels");
  int64_t total = 0;
  if (!st) st = read_count(&total, static_cast<char*>(d_scratch), s, "reading the scan total");
  if (!st) *h_total = (int32_t)total;
  return st;
}

size_t dax_gb300_sort_scratch_bytes(int64_t n, int key_type, int value_bytes) {
  using namespace daxgb;
  const int kb = type_bytes(key_type);
  if (!kb || n < 0 || value_bytes < 0 || value_bytes > 16 || (value_bytes & 3)) return 0;
  const long long nn = n < 1 ? 1 : n;
  const SortLayout L = sort_layout(nn, kb, value_bytes);
  return L.total + scan_bytes(256ll * ptiles(nn));
}

int dax_gb300_sort_by_key(void* d_keys, void* d_values, int64_t n, int key_type, int value_bytes,
                          int descending, void* d_scratch, size_t scratch_bytes, void* stream) {
  using namespace daxgb;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!size_ok(n)) return bad("sort length must be in [0, 2^31 - 1]");
  const int kb = type_bytes(key_type);
  if (!kb) return bad("unknown key type");
  if (value_bytes < 0 || value_bytes > 16 || (value_bytes & 3))
    return bad("value size must be 0, 4, 8, 12 or 16 bytes");
  if (n < 2) return DAX_GB300_SUCCESS;
  if (!d_keys || (value_bytes && !d_values) || !d_scratch) return bad("NULL keys, values or scratch");
  if (scratch_bytes < dax_gb300_sort_scratch_bytes(n, key_type, value_bytes))
    return bad("scratch smaller than dax_gb300_sort_scratch_bytes()");
  const int kind = type_kind(key_type);
  char* sc = static_cast<char*>(d_scratch);
  if (kb == 4)
    radix_sort<uint32_t>(static_cast<uint32_t*>(d_keys), static_cast<uint32_t*>(d_values),
                         value_bytes / 4, n, kind, descending != 0, sc, prim_sms(), s);
  else
    radix_sort<unsigned long long>(static_cast<unsigned long long*>(d_keys),
                                   static_cast<uint32_t*>(d_values), value_bytes / 4, n, kind,
                                   descending != 0, sc, prim_sms(), s);
  return launched("sort kernels");
}

int dax_gb300_selfcheck_sort_wait(uint32_t* d_keys, uint32_t* d_values, int64_t n, uint32_t polls,
                                  void* d_scratch, size_t scratch_bytes, void* stream) {
  using namespace daxgb;
  if (!size_ok(n) || n <= kSortTile) return bad("the sort must be of more than one block");
  if (!d_keys || !d_values || !d_scratch) return bad("NULL keys, values or scratch");
  if (scratch_bytes < dax_gb300_sort_scratch_bytes(n, DAX_GB300_TYPE_U32, 4))
    return bad("scratch smaller than dax_gb300_sort_scratch_bytes()");
  radix_sort<uint32_t>(d_keys, d_values, 1, n, 0, false, static_cast<char*>(d_scratch), prim_sms(),
                       static_cast<cudaStream_t>(stream), 4, false,
                       polls < kSpinIters ? polls : kSpinIters);
  return launched("sort kernels");
}

size_t dax_gb300_compact_scratch_bytes(int64_t n, int element_bytes) {
  using namespace daxgb;
  if (n < 0 || element_bytes < 0) return 0;
  const long long nn = n < 1 ? 1 : n;
  return keep_bytes(nn) + align256((size_t)nn * element_bytes);
}

int dax_gb300_unique(void* d_keys, int64_t n, int key_type, void* d_scratch, size_t scratch_bytes,
                     int64_t* h_count, void* stream) {
  using namespace daxgb;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!size_ok(n)) return bad("unique length must be in [0, 2^31 - 1]");
  const int kb = type_bytes(key_type);
  if (!kb) return bad("unknown key type");
  if (n == 0) {
    if (h_count) *h_count = 0;
    return DAX_GB300_SUCCESS;
  }
  if (!d_keys || !d_scratch) return bad("NULL keys or scratch");
  if (scratch_bytes < dax_gb300_compact_scratch_bytes(n, kb))
    return bad("scratch smaller than dax_gb300_compact_scratch_bytes(n, key bytes)");
  // one pass, in place (the kept keys of a tile go below its start)
  char* sc = static_cast<char*>(d_scratch);
  const CompactOp op{2, type_kind(key_type), d_keys, nullptr, 0, d_keys};
  if (kb == 4)
    compact_single<uint32_t>(op, n, sc, prim_sms(), s);
  else
    compact_single<unsigned long long>(op, n, sc, prim_sms(), s);
  int st = launched("unique kernels");
  if (st || !h_count) return st;
  return read_count(h_count, sc, s, "reading the unique count");
}

int dax_gb300_stream_compact(const void* d_input, int value_bytes, const void* d_stencil,
                             int stencil_type, int64_t n, void* d_output, void* d_scratch,
                             size_t scratch_bytes, int64_t* h_count, void* stream) {
  using namespace daxgb;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!size_ok(n)) return bad("compaction length must be in [0, 2^31 - 1]");
  if (stencil_type != DAX_GB300_TYPE_I32 && stencil_type != DAX_GB300_TYPE_F32)
    return bad("stencil must be int32 or float");
  if (d_input && (value_bytes <= 0 || value_bytes > 16 || (value_bytes & 3)))
    return bad("value size must be 4, 8, 12 or 16 bytes");
  if (n == 0) {
    if (h_count) *h_count = 0;
    return DAX_GB300_SUCCESS;
  }
  if (!d_stencil || !d_output || !d_scratch) return bad("NULL stencil, output or scratch");
  if (scratch_bytes < dax_gb300_compact_scratch_bytes(n, 0))
    return bad("scratch smaller than dax_gb300_compact_scratch_bytes(n, 0)");
  char* sc = static_cast<char*>(d_scratch);
  const CompactOp op{stencil_type == DAX_GB300_TYPE_I32 ? 0 : 1, 0, d_stencil,
                     static_cast<const uint32_t*>(d_input), d_input ? value_bytes / 4 : 1,
                     d_output};
  compact_single<uint32_t>(op, n, sc, prim_sms(), s);
  int st = launched("compaction kernels");
  if (st || !h_count) return st;
  return read_count(h_count, sc, s, "reading the compacted count");
}

int dax_gb300_bounds(const void* d_sorted, int64_t n, const void* d_values, int64_t m,
                     int key_type, int upper, int32_t* d_out, void* stream) {
  using namespace daxgb;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!size_ok(n) || !size_ok(m)) return bad("lengths must be in [0, 2^31 - 1]");
  if (!type_bytes(key_type)) return bad("unknown key type");
  if (m == 0) return DAX_GB300_SUCCESS;
  if ((n && !d_sorted) || !d_values || !d_out) return bad("NULL input, values or output");
  const int b = (int)((m + 255) / 256 < prim_sms() * 8 ? (m + 255) / 256 : prim_sms() * 8);
#define DAXGB_BOUNDS(T)                                                                         \
  (upper ? k_bounds<T, true><<<b, 256, 0, s>>>((const T*)d_sorted, n, (const T*)d_values, m, d_out) \
         : k_bounds<T, false><<<b, 256, 0, s>>>((const T*)d_sorted, n, (const T*)d_values, m, d_out))
  switch (key_type) {
    case DAX_GB300_TYPE_I32: DAXGB_BOUNDS(int32_t); break;
    case DAX_GB300_TYPE_U32: DAXGB_BOUNDS(uint32_t); break;
    case DAX_GB300_TYPE_F32: DAXGB_BOUNDS(float); break;
    case DAX_GB300_TYPE_I64: DAXGB_BOUNDS(int64_t); break;
    default: DAXGB_BOUNDS(unsigned long long); break;
  }
#undef DAXGB_BOUNDS
  return launched("bounds kernel");
}

}  // extern "C"
