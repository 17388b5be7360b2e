// The Mandelbulb benchmark's compute pipeline (Benchmarks/Mandlebulb): the
// escape-iteration point field and the per-point normals and colours of the
// extracted surface (the clip-and-count worklet of its cut view is the third
// mode of k_cell_count, classify.cu).  The
// surface itself is the marching-cubes pipeline (extractSurface,
// Mandlebulb.cxx:105-118) or the count-array-driven generate of the cut
// (extractCut, Mandlebulb.cxx:126-157); its GLUT/shader display is replaced
// by the device buffers these kernels write.
//
// Rounding: every add, multiply and divide is spelled out (no fused
// multiply-add) as the reference's float expressions round on the CPU.  The
// transcendental functions of the escape iteration (atan2, pow, sin, tan,
// cos) are CUDA's own; they may differ from the host C library's in the last
// place, so the escape iteration of a point on the fractal's boundary can
// differ between the two.  sqrt and 1/sqrt are correctly rounded on both, so
// normals and colours of the same surface agree bit for bit.
#include "common.cuh"
#include "coolwarm_table.h"
#include "kernels.cuh"

namespace daxgb {

__constant__ unsigned char c_coolwarm[3 * DAX_GB300_COOLWARM_ENTRIES] = DAX_GB300_COOLWARM_RGB;

__device__ __forceinline__ float magsq3(float x, float y, float z) {
  return __fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z));
}

// worklet::Mandlebulb (Benchmarks/Mandlebulb/Worklets.h:65-109): the escape
// iteration of pos -> pos^10 + c (White and Nylander's power, :92-108), 0
// when c itself is outside radius sqrt(2), at most 35.
// One step of it; r2 is the point's squared radius, before and after.
__device__ __forceinline__ void mandelbulb_step(float& x, float& y, float& z, float& r2, float cx,
                                                float cy, float cz) {
  const float t = __fsqrt_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)));
  const float thetaN = __fmul_rn(10.0f, atan2f(t, z));
  const float phiN = __fmul_rn(10.0f, atan2f(y, z));
  const float powR = powf(r2, 5.0f);
  float st, ct;  // sincosf: bit for bit sinf and cosf (checked over every float on GB300)
  sincosf(thetaN, &st, &ct);
  const float px = __fmul_rn(powR, __fmul_rn(st, tanf(phiN)));
  const float py = __fmul_rn(powR, __fmul_rn(st, sinf(phiN)));
  const float pz = __fmul_rn(powR, ct);
  x = __fadd_rn(px, cx);
  y = __fadd_rn(py, cy);
  z = __fadd_rn(pz, cz);
  r2 = magsq3(x, y, z);
}

// Bound by arithmetic: two arctangents, a power, a sine and cosine, a tangent
// and a sine a step, 1 to 34 steps a point.  With a point per lane a warp
// steps until its slowest lane is done, so a lane that is done takes the
// block's next point instead (its tiles of 256 points, strided by the grid,
// in order, from a counter in shared memory), once kRefill lanes wait: the 201^3
// points of [-1, 1]^3 945 us with a point per lane, 757 so; 49^3 41 and 43.  Where
// all points of a warp take the same steps it only costs, a refill about 45
// instructions more than a loop over points: 201^3 points inside the fractal, 34
// steps each, 2030 and 2132, one step each 86 and 98, none (radius above sqrt(2))
// 27 and 36.  (2, 4 and 8 lanes: 783, 761 and 758.  Testing for a refill after
// every step, in the same loop: 787, and 2235 inside.  Stepping the waiting lanes
// too, without a branch: 829.)
constexpr int kRefill = 6;

__global__ void __launch_bounds__(256) k_mandelbulb_field(Grid g, unsigned long long mnx,
                                                          float* __restrict__ out) {
  __shared__ unsigned s_next;
  if (threadIdx.x == 0) s_next = 0;
  __syncthreads();
  const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
  const unsigned P = (unsigned)g.P, tiles = (P + 255u) / 256u;
  // the block's points; the last tile is the last one of its block
  const unsigned mine = (tiles - blockIdx.x + gridDim.x - 1u) / gridDim.x * 256u -
                        ((tiles - 1u) % gridDim.x == blockIdx.x ? tiles * 256u - P : 0u);
  float x = 0, y = 0, z = 0, r2 = 0, cx = 0, cy = 0, cz = 0;
  unsigned p = 0;
  int i = 0;  // the step the lane is at; 0: it has no point
  unsigned idle = kFull;
  bool more = true;
  while (true) {
    if (more) {
      unsigned n = 0;
      if (below == 0u) n = atomicAdd(&s_next, (unsigned)__popc(idle));
      n = __shfl_sync(kFull, n, 0);
      more = n + (unsigned)__popc(idle) < mine;
      n += (unsigned)__popc(idle & below);
      if (i == 0 && n < mine) {
        p = (n >> 8) * (256u * gridDim.x) + 256u * blockIdx.x + (n & 255u);
        const unsigned row = div_by(p, mnx);
        int j, k;
        split_row(g, row, j, k);
        x = cx = coord(g.ox, g.sx, (int)(p - row * (unsigned)g.nx), g.mx);
        y = cy = coord(g.oy, g.sy, j, g.my);
        z = cz = coord(g.oz, g.sz, k, g.mz);
        r2 = magsq3(x, y, z);
        if (r2 > 2.0f) out[p] = 0.0f;
        else i = 1;
      }
      idle = __ballot_sync(kFull, i == 0);
    }
    // steps until kRefill lanes wait or, with no points left, until all do
    const int most = more ? kRefill : 32;
    while (__popc(idle) < most) {
      if (i > 0) {
        mandelbulb_step(x, y, z, r2, cx, cy, cz);
        const bool escaped = r2 > 2.0f;
        if (escaped || i == 34) out[p] = escaped ? (float)i : 35.0f;
        i = escaped || i == 34 ? 0 : i + 1;
      }
      idle = __ballot_sync(kFull, i == 0);
    }
    if (!more && idle == kFull) break;
  }
}

// worklet::ColorsAndNorms (Worklets.h:177-209) on an unmerged triangle
// surface: point v belongs to triangle v / 3; its normal is
// Normal(Cross(b - a, c - a)) = (1 / sqrt(dot(x, x))) * x
// (VectorAnalysis.h:182-201, 227-232; RSqrt is 1 / Sqrt off the GPU), its
// colour the cool-warm entry (int)(257 * clamp(|dot(p, (0.09, 0.09, 0.9))|,
// 0, 0.9999)) (CoolWarmColorMap.h:38-45) with alpha 255.
__device__ __forceinline__ float3 triangle_normal(const float* c) {
  const float ax = __fsub_rn(c[3], c[0]), ay = __fsub_rn(c[4], c[1]), az = __fsub_rn(c[5], c[2]);
  const float bx = __fsub_rn(c[6], c[0]), by = __fsub_rn(c[7], c[1]), bz = __fsub_rn(c[8], c[2]);
  const float xx = __fsub_rn(__fmul_rn(ay, bz), __fmul_rn(az, by));
  const float xy = __fsub_rn(__fmul_rn(az, bx), __fmul_rn(ax, bz));
  const float xz = __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
  const float r = __fdiv_rn(1.0f, __fsqrt_rn(magsq3(xx, xy, xz)));
  return make_float3(__fmul_rn(r, xx), __fmul_rn(r, xy), __fmul_rn(r, xz));
}

__device__ __forceinline__ uchar4 point_color(const float* p, const unsigned char* map) {
  float s = __fadd_rn(__fadd_rn(__fmul_rn(p[0], 0.09f), __fmul_rn(p[1], 0.09f)), __fmul_rn(p[2], 0.9f));
  s = fminf(0.9999f, fmaxf(0.0f, fabsf(s)));
  const int idx = (int)__fmul_rn(257.0f, s);
  return make_uchar4(map[3 * idx + 0], map[3 * idx + 1], map[3 * idx + 2], 255);
}

// Bound by HBM, 28 bytes a point.  A warp takes 32 triangles, 1152 consecutive
// bytes in and out, through shared memory, lane = triangle: every normal is
// computed once and every access of global memory covers 128 bytes.  (Lane =
// point, each computing its triangle's normal from nine strided loads: 44 us
// for 4.6 M points, 35 now.)  nv is a multiple of 3.
__global__ void __launch_bounds__(256) k_colors_and_norms(const float* __restrict__ verts,
                                                          long long nv, float* __restrict__ norms,
                                                          uint8_t* __restrict__ colors) {
  __shared__ unsigned char s_map[3 * DAX_GB300_COOLWARM_ENTRIES];
  __shared__ float s_buf[8][9 * 32];
  __shared__ uchar4 s_color[8][3 * 32];
  for (int t = threadIdx.x; t < 3 * DAX_GB300_COOLWARM_ENTRIES; t += blockDim.x)
    s_map[t] = c_coolwarm[t];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* const buf = s_buf[warp];
  uchar4* const color = s_color[warp];
  const long long T = nv / 3, step = (long long)gridDim.x * 8 * 32;
  for (long long t0 = ((long long)blockIdx.x * 8 + warp) * 32; t0 < T; t0 += step) {
    const int n = (int)min(32ll, T - t0);  // triangles
    const float* in = verts + 9 * t0;
    float* out = norms + 9 * t0;
    uchar4* cout = reinterpret_cast<uchar4*>(colors) + 3 * t0;
#pragma unroll
    for (int e = 0; e < 9; ++e)
      if (32 * e + lane < 9 * n) buf[32 * e + lane] = __ldg(in + 32 * e + lane);
    __syncwarp();
    float c[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) c[e] = buf[9 * lane + e];
    const float3 x = triangle_normal(c);
    if (lane < n) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        color[3 * lane + q] = point_color(c + 3 * q, s_map);
        buf[9 * lane + 3 * q] = x.x;
        buf[9 * lane + 3 * q + 1] = x.y;
        buf[9 * lane + 3 * q + 2] = x.z;
      }
    }
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 9; ++e)
      if (32 * e + lane < 9 * n) out[32 * e + lane] = buf[32 * e + lane];
#pragma unroll
    for (int e = 0; e < 3; ++e)
      if (32 * e + lane < 3 * n) cout[32 * e + lane] = color[32 * e + lane];
    __syncwarp();
  }
}

void launch_mandelbulb_field(const Grid& g, float* out, int num_sms, cudaStream_t s) {
  const int b = resident_blocks(k_mandelbulb_field, 256, 0, num_sms, (g.P + 255) / 256);
  k_mandelbulb_field<<<b, 256, 0, s>>>(g, div_multiplier((unsigned)g.nx), out);
}

void launch_colors_and_norms(const float* verts, long long nv, float* norms, uint8_t* colors,
                             int num_sms, cudaStream_t s) {
  const int b = resident_blocks(k_colors_and_norms, 256, 0, num_sms, (nv / 3 + 255) / 256);
  k_colors_and_norms<<<b, 256, 0, s>>>(verts, nv, norms, colors);
}

}  // namespace daxgb
