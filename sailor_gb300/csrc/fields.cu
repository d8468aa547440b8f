// fields.cu -- trilinear gathers from dense voxel grids at sampled points.
//
// The reference's trilinear aggregation (sampling_kernel.cu:162-327 of
// SAILOR c_lib/VoxelEncoding/src) interpolates per-node corner features; the
// spec extension gathers from a dense per-voxel grid instead: grid
// [B, D, D, D, C] channel-last, voxel (x, y, z) centred at
// bbox_min + (x, y, z) * voxel_size (the fusion grid's convention), corners
// outside the grid contribute zero.  Sample point = ori + z * dir of its ray;
// samples with z < 0 produce 0.
//
// grid_gather_kernel: a warp takes 32 consecutive samples: a lane per sample
// finds its cell and corner weights; with C a multiple of 4, C / 4 lanes then
// share each sample, a float4 of channels a lane, so that corner reads are
// whole 64-byte texels and the output rows are written contiguously (a thread
// per sample wrote its 16 channels 64 bytes apart from its neighbours': the
// L1 data path was 73 % busy).  Sample -> ray -> frame by multiplication (two
// 64-bit divisions a sample were a third of the 1- and 3-channel gathers).
// 12.6 M samples x 16 channels of 256^3: 1.02 -> 0.57 ms; 16.8 M samples x 3
// channels 122 -> 121 us, x 1 90 -> 78 us.
//
// grid_scatter_kernel (the adjoint): 8 lanes per ray walk the ray's samples in
// order, a lane per corner with its C channel sums in registers (four rays a
// warp).  While consecutive samples stay in one trilinear cell their
// contributions w_corner * g_channel accumulate; at a cell change (and at the
// end of the ray) the lane adds its sums into the grid, four channels per
// vector reduction where C is a multiple of 4.  Samples of a ray are
// depth-sorted and cluster in the few hit voxels, so a flush carries many
// samples.  A warp per ray, its lanes over the 8 C slots, took 88 warp
// instructions a sample at C = 16 (staging through shared memory): 12.6 M
// samples 1.16 -> 0.68 ms, at C = 1 0.69 -> 0.34 ms; now bound by the atomics.
//
// Registers (both wait on memory most of the time): 16 channels, gather at 5 /
// 6 / 8 CTAs an SM 0.74 / 0.57 / 0.58 ms, adjoint at 2 / 4 / 5 0.96 / 0.68 / 0.83;
// one and three channels are best without a bound (gather 78 and 121 us against
// 86 and 125 at 6, adjoint 344 against 352 at 4): 0 leaves the choice to the compiler.
//
// mode 1 turns a gathered normalised TSDF t (C == 1) into a density
// sigma = sigmoid(-t * scale / s) / s  (scale = truncation margin in metres,
// s = the density's length scale), so the gather is fused with the field
// transform that feeds compositing.
#include <climits>

#include "ray_core.cuh"

namespace sg {

// Division by a fixed d >= 1, the plain 64-bit quotient where a dividend can
// reach 2^31.
struct FixedDiv {
  FixedDiv31 q;
  uint32_t d;
  int small;  // every dividend is below 2^31
  static FixedDiv of(uint32_t d, long largest) { return FixedDiv{FixedDiv31::of(d), d, largest < (1l << 31) ? 1 : 0}; }
  __device__ __forceinline__ long div(long n) const { return small ? (long)q.div((uint32_t)n) : n / (long)d; }
};

struct GatherParams {
  const float *ori, *dir, *z;
  long R;
  int N, S;
  FixedDiv by_S, by_N;
  const float *grid;
  int D, C;
  const float *vol_bbox, *voxel_size;
  int mode;
  float scale, s;
  float *out;
};

// Geometry of a sample's frame, kept while the frame stays the same.
struct FrameGeom {
  int b = -1;
  float bmin[3], vs, inv_vs;
  __device__ __forceinline__ void load(const float *__restrict__ vol_bbox, const float *__restrict__ voxel_size, int frame) {
    if (frame == b) return;
    b = frame;
#pragma unroll
    for (int a = 0; a < 3; a++) bmin[a] = __ldg(vol_bbox + 6 * b + 2 * a);
    vs = __ldg(voxel_size + b);
    inv_vs = 1.0f / vs;
  }
};

// VEC: grid and output are 16-byte aligned (C a multiple of 4).
template <int C, bool VEC>
__global__ void __launch_bounds__(256, VEC && C >= 8 ? 6 : 0) grid_gather_kernel(GatherParams p) {
  constexpr int L = VEC ? C / 4 : 1;  // lanes of a sample
  const long n = p.R * p.S;
  const int lane = lane_id();
  const long dy = p.D, dx = (long)p.D * p.D;
  FrameGeom g;
  for (long k0 = (((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; k0 < n;
       k0 += ((long)gridDim.x * blockDim.x >> 5) * 32) {
    const long k = k0 + lane;
    const float zz = k < n ? __ldg(p.z + k) : -1.0f;
    unsigned in = 0u;
    long off = 0;  // the lower corner's voxel, frame included
    float f[3] = {0.0f, 0.0f, 0.0f};
    if (zz >= 0.0f) {
      const long r = p.by_S.div(k);
      g.load(p.vol_bbox, p.voxel_size, (int)p.by_N.div(r));
      float pt[3];
      int i0[3];
#pragma unroll
      for (int a = 0; a < 3; a++) pt[a] = __fmaf_rn(__ldg(p.dir + r * 3 + a), zz, __ldg(p.ori + r * 3 + a));
      tap_frac(g.bmin, g.vs, g.inv_vs, pt, i0, f);
      in = corners_inside(i0, p.D);
      off = (((long)g.b * p.D + i0[0]) * p.D + i0[1]) * p.D + i0[2];
      if (in == 0u) f[0] = f[1] = f[2] = 0.0f;  // they may be NaN, and weigh zeros below
    }
    if constexpr (L == 1) {
      float acc[C];
#pragma unroll
      for (int c = 0; c < C; c++) acc[c] = 0.0f;
#pragma unroll
      for (int cr = 0; cr < 8; cr++) {
        if (!((in >> cr) & 1u)) continue;
        const float w = corner_weight(f, cr);
        const float *v = p.grid + (off + ((cr & 4) ? dx : 0) + ((cr & 2) ? dy : 0) + (cr & 1)) * C;
        if constexpr (VEC) {
          const float4 q = __ldg(reinterpret_cast<const float4 *>(v));
          acc[0] = __fmaf_rn(w, q.x, acc[0]);
          acc[1] = __fmaf_rn(w, q.y, acc[1]);
          acc[2] = __fmaf_rn(w, q.z, acc[2]);
          acc[3] = __fmaf_rn(w, q.w, acc[3]);
        } else {
#pragma unroll
          for (int c = 0; c < C; c++) acc[c] = __fmaf_rn(w, __ldg(v + c), acc[c]);
        }
      }
      if (p.mode == 1 && zz >= 0.0f) acc[0] = tsdf_density(acc[0], p.scale / p.s, 1.0f / p.s);
      if (k < n) {
        if constexpr (VEC) {
          *reinterpret_cast<float4 *>(p.out + k * C) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        } else {
#pragma unroll
          for (int c = 0; c < C; c++) p.out[k * C + c] = acc[c];
        }
      }
    } else {
      const int q = lane % L;
#pragma unroll 1
      for (int s0 = 0; s0 < 32; s0 += 32 / L) {
        const int src = s0 + lane / L;
        const unsigned m = __shfl_sync(SG_FULL, in, src);
        const long o = __shfl_sync(SG_FULL, off, src);
        const float fs[3] = {__shfl_sync(SG_FULL, f[0], src), __shfl_sync(SG_FULL, f[1], src),
                             __shfl_sync(SG_FULL, f[2], src)};
        const float4 *v = reinterpret_cast<const float4 *>(p.grid) + o * L + q;
        float4 t[8];
#pragma unroll
        for (int cr = 0; cr < 8; cr++) {
          t[cr] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          if ((m >> cr) & 1u) t[cr] = __ldg(v + (((cr & 4) ? dx : 0) + ((cr & 2) ? dy : 0) + (cr & 1)) * L);
        }
        float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int cr = 0; cr < 8; cr++) {
          const float w = corner_weight(fs, cr);
          acc.x = __fmaf_rn(w, t[cr].x, acc.x);
          acc.y = __fmaf_rn(w, t[cr].y, acc.y);
          acc.z = __fmaf_rn(w, t[cr].z, acc.z);
          acc.w = __fmaf_rn(w, t[cr].w, acc.w);
        }
        if (k0 + src < n) __stcs(reinterpret_cast<float4 *>(p.out + (k0 + src) * C) + q, acc);
      }
    }
  }
}

struct ScatterParams {
  const float *ori, *dir, *z;
  long R;
  int N, S;
  const float *gout;   // [R, S, C]
  const float *grid;   // mode 1: the TSDF grid the forward gathered from
  int D;
  const float *vol_bbox, *voxel_size;
  int mode;
  float scale, s;
  float *ggrid;        // [B, D, D, D, C], accumulated
  int parts, part;     // a ray's samples in so many parts of so many (a multiple of 8)
};

// VEC: gradients and grid are 16-byte aligned (C a multiple of 4).
template <int C, bool VEC>
__device__ __forceinline__ void scatter_flush(const ScatterParams &p, long cell, int cr, unsigned in, float (&acc)[C]) {
  if ((in >> cr) & 1u) {
    float *g = p.ggrid + (cell + ((cr & 4) ? (long)p.D * p.D : 0) + ((cr & 2) ? p.D : 0) + (cr & 1)) * C;
    if constexpr (VEC) {
#pragma unroll
      for (int c = 0; c < C; c += 4)
        if (acc[c] != 0.0f || acc[c + 1] != 0.0f || acc[c + 2] != 0.0f || acc[c + 3] != 0.0f)
          red_add_f32x4(g + c, acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
    } else {
#pragma unroll
      for (int c = 0; c < C; c++)
        if (acc[c] != 0.0f) atomicAdd(g + c, acc[c]);
    }
  }
#pragma unroll
  for (int c = 0; c < C; c++) acc[c] = 0.0f;
}

// PARTS: a ray's samples are walked in p.parts parts of p.part, each by lanes of
// its own: with fewer rays than kScatterFill an SM the eight lanes' chain
// through all samples is what the call takes.  One ray a lane group / in parts,
// 96 samples of 16 channels: 1 ray 33 / 6 us, 500 43 / 10, 4000 45 / 28, 16384 96 / 99;
// of one channel 500 rays 21 / 6, 16384 45 / 38.
constexpr int kScatterFill = 128;

template <int C, bool VEC, bool PARTS>
__global__ void __launch_bounds__(256, C >= 8 ? 4 : 0) grid_scatter_kernel(ScatterParams p) {
  const int cr = lane_id() & 7;  // corner, and sample of a step of 8
  FrameGeom g;
  const long nw = ((long)gridDim.x * blockDim.x) >> 5;
  const long n = PARTS ? p.R * p.parts : p.R;
  for (long r0 = (((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 4; r0 < n; r0 += nw * 4) {
    const long v = r0 + (lane_id() >> 3);
    const bool live = v < n;
    const long r = PARTS ? v / p.parts : v;
    const int first = PARTS ? (int)(v - r * p.parts) * p.part : 0;  // the part's first sample
    float o[3] = {0.0f, 0.0f, 0.0f}, d[3] = {0.0f, 0.0f, 0.0f};
    if (live) {
      g.load(p.vol_bbox, p.voxel_size, (int)(r / p.N));
#pragma unroll
      for (int a = 0; a < 3; a++) {
        o[a] = __ldg(p.ori + r * 3 + a);
        d[a] = __ldg(p.dir + r * 3 + a);
      }
    }
    float acc[C];
#pragma unroll
    for (int c = 0; c < C; c++) acc[c] = 0.0f;
    long cur = 0;        // lower corner's voxel of the current run
    unsigned cur_in = 0u;
    for (int c0 = first; c0 < (PARTS ? first + p.part : p.S); c0 += 8) {
      // a lane per sample: cell, fractions (as the forward tap forms them) and,
      // at one channel, the gradient
      const int i = c0 + cr;
      const float zz = live && i < p.S ? __ldg(p.z + r * p.S + i) : -1.0f;
      unsigned in = 0u;
      long cell = 0;
      float f[3] = {0.0f, 0.0f, 0.0f}, g1 = 0.0f;
      if (zz >= 0.0f) {
        float pt[3];
        int i0[3];
#pragma unroll
        for (int a = 0; a < 3; a++) pt[a] = __fmaf_rn(d[a], zz, o[a]);
        tap_frac(g.bmin, g.vs, g.inv_vs, pt, i0, f);
        in = corners_inside(i0, p.D);
        // with the corners that are inside, this names the cell (an index of -1
        // on an axis wraps into the row before, whose own cells have other corners inside)
        cell = (((long)g.b * p.D + i0[0]) * p.D + i0[1]) * p.D + i0[2];
        if constexpr (C == 1) {
          g1 = __ldg(p.gout + r * p.S + i);
          if (p.mode == 1) {
            // d sigma / d t of sigma = sigmoid(-t scale / s) / s at the gathered t
            float t1[1], wc[8];
#pragma unroll
            for (int c = 0; c < 8; c++) wc[c] = corner_weight(f, c);
            grid_tap_cell<1>(p.grid + (size_t)g.b * p.D * p.D * p.D, p.D, i0, wc, t1);
            const float k = p.scale / p.s;
            const float sg = tsdf_sigmoid(t1[0], k);
            g1 = g1 * (-sg * (1.0f - sg) * (k * (1.0f / p.s)));
          }
        }
      }
      const float *grow = p.gout + ((size_t)(live ? r : 0) * p.S + c0) * C;
#pragma unroll 2
      for (int j = 0; j < 8; j++) {
        const unsigned inj = __shfl_sync(SG_FULL, in, j, 8);
        const long cj = __shfl_sync(SG_FULL, cell, j, 8);
        const float fj[3] = {__shfl_sync(SG_FULL, f[0], j, 8), __shfl_sync(SG_FULL, f[1], j, 8),
                             __shfl_sync(SG_FULL, f[2], j, 8)};
        float gj = 0.0f;
        if constexpr (C == 1) gj = __shfl_sync(SG_FULL, g1, j, 8);
        if (inj == 0u) continue;  // no sample, or no corner of it inside the grid
        if (cj != cur || inj != cur_in) {
          if (cur_in) scatter_flush<C, VEC>(p, cur, cr, cur_in, acc);
          cur = cj;
          cur_in = inj;
        }
        const float w = (((cr & 4) ? fj[0] : 1.0f - fj[0]) * ((cr & 2) ? fj[1] : 1.0f - fj[1])) *
                        ((cr & 1) ? fj[2] : 1.0f - fj[2]);
        if constexpr (C == 1) {
          acc[0] = __fmaf_rn(w, gj, acc[0]);
        } else if constexpr (VEC) {
#pragma unroll
          for (int c = 0; c < C; c += 4) {
            const float4 q = __ldg(reinterpret_cast<const float4 *>(grow + j * C + c));
            acc[c] = __fmaf_rn(w, q.x, acc[c]);
            acc[c + 1] = __fmaf_rn(w, q.y, acc[c + 1]);
            acc[c + 2] = __fmaf_rn(w, q.z, acc[c + 2]);
            acc[c + 3] = __fmaf_rn(w, q.w, acc[c + 3]);
          }
        } else {
#pragma unroll
          for (int c = 0; c < C; c++) acc[c] = __fmaf_rn(w, __ldg(grow + j * C + c), acc[c]);
        }
      }
    }
    if (cur_in) scatter_flush<C, VEC>(p, cur, cr, cur_in, acc);
  }
}

template <bool PARTS>
static void launch_scatter(const ScatterParams &p, int C, sg_stream_t stream) {
  int g = ceil_div(p.R * p.parts * 8, 256);
  if (g > num_sms() * 32) g = num_sms() * 32;
  const bool vec = (((uintptr_t)p.gout) | ((uintptr_t)p.ggrid)) % 16 == 0;
  switch (C) {
    case 1: grid_scatter_kernel<1, false, PARTS><<<g, 256, 0, stream>>>(p); break;
    case 3: grid_scatter_kernel<3, false, PARTS><<<g, 256, 0, stream>>>(p); break;
    case 4:
      if (vec) grid_scatter_kernel<4, true, PARTS><<<g, 256, 0, stream>>>(p);
      else grid_scatter_kernel<4, false, PARTS><<<g, 256, 0, stream>>>(p);
      break;
    case 8:
      if (vec) grid_scatter_kernel<8, true, PARTS><<<g, 256, 0, stream>>>(p);
      else grid_scatter_kernel<8, false, PARTS><<<g, 256, 0, stream>>>(p);
      break;
    default:
      if (vec) grid_scatter_kernel<16, true, PARTS><<<g, 256, 0, stream>>>(p);
      else grid_scatter_kernel<16, false, PARTS><<<g, 256, 0, stream>>>(p);
  }
}

// Zero of the part of a gradient grid [B, Db, Db, Db, C] (the tree's fine
// geometry) that a training pass over the tree's nodes can write: a CTA takes
// BRICKS top bricks, a thread each tests its brick's 26-neighbourhood
// for a node, and all threads clear the bricks found, rate^3 voxels each (rate^2
// z-runs of rate * C floats).  Few bricks are near a node, so a CTA per brick was
// bound by starting CTAs: 4 x 32^3 bricks of 8^3 voxels of 16 channels 182 -> 83
// us, 2 x 16^3 bricks 30 -> 22 us (16).  One brick a CTA where 16 would leave SMs
// without one (8^3 bricks, a quarter of them near nodes: 16 14 us, one 8).  A
// compile-time count: as an argument it took 1.2 to 1.9 times as long.
constexpr int kZeroBricks = 16;

template <int BRICKS>
__global__ void __launch_bounds__(256) zero_near_nodes_kernel(SgTree t, float *grid, int C, int vec4, FixedDiv31 by_brick,
                                                              FixedDiv31 by_run, FixedDiv31 by_rate) {
  __shared__ int2 s_near[BRICKS];
  __shared__ int s_n;
  const int b = blockIdx.y, Dt = t.Dt;
  const int vt = Dt * Dt * Dt;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  const int own = (int)blockIdx.x * BRICKS + (int)threadIdx.x;
  if (threadIdx.x < BRICKS && own < vt) {
    const int Z = own % Dt, xy = own / Dt, Y = xy % Dt, X = xy / Dt;
    const int *node = t.brick_node + (long)b * vt;
    bool near = false;
#pragma unroll
    for (int q = 0; q < 27; q++) {
      const int x = X + q / 9 - 1, y = Y + (q / 3) % 3 - 1, z = Z + q % 3 - 1;
      if (x >= 0 && y >= 0 && z >= 0 && x < Dt && y < Dt && z < Dt) near |= __ldg(node + (x * Dt + y) * Dt + z) >= 0;
    }
    if (near) s_near[atomicAdd(&s_n, 1)] = make_int2(X * t.rate * t.Db + Y * t.rate, Z * t.rate);
  }
  __syncthreads();
  const int r = t.rate, Db = t.Db;
  const int per_run = vec4 ? r * C / 4 : r * C;  // stores per z-run
  float *g = grid + (size_t)b * Db * Db * Db * C;
  const int per_brick = r * r * per_run;
  for (int i = threadIdx.x; i < s_n * per_brick; i += blockDim.x) {
    const int n = (int)by_brick.div((uint32_t)i), j = i - n * per_brick;
    const int xy = (int)by_run.div((uint32_t)j), k = j - xy * per_run, rx = (int)by_rate.div((uint32_t)xy);
    const int2 at = s_near[n];  // first voxel: x * Db + y, z
    const size_t off = ((size_t)(at.x + rx * Db + (xy - rx * r)) * Db + at.y) * C;
    if (vec4) reinterpret_cast<float4 *>(g + off)[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    else g[off + k] = 0.0f;
  }
}

}  // namespace sg

using namespace sg;

extern "C" int sg_grid_gather(const float *ori, const float *dir, const float *z, int B, int N, int S,
                              const float *grid, int D, int C, const float *vol_bbox, const float *voxel_size,
                              int mode, float scale, float s, float *out, sg_stream_t stream) {
  if (!ori || !dir || !z || !grid || !vol_bbox || !voxel_size || !out) return SG_ERR_INVALID_ARG;
  if (B <= 0 || N <= 0 || S <= 0 || D <= 0 || C <= 0 || C > 16) return SG_ERR_INVALID_ARG;
  if (mode == 1 && (C != 1 || s == 0.0f)) return SG_ERR_INVALID_ARG;
  const long samples = (long)B * N * S;
  GatherParams p{ori, dir, z, (long)B * N, N, S, FixedDiv::of(S, samples), FixedDiv::of(N, samples), grid, D, C, vol_bbox, voxel_size, mode, scale, s, out};
  long n = (long)B * N * S;
  int g = ceil_div(n, 256);
  if (g > num_sms() * 64) g = num_sms() * 64;
  const bool vec = (((uintptr_t)grid) | ((uintptr_t)out)) % 16 == 0;
  switch (C) {
    case 1: grid_gather_kernel<1, false><<<g, 256, 0, stream>>>(p); break;
    case 3: grid_gather_kernel<3, false><<<g, 256, 0, stream>>>(p); break;
    case 4:
      if (vec) grid_gather_kernel<4, true><<<g, 256, 0, stream>>>(p);
      else grid_gather_kernel<4, false><<<g, 256, 0, stream>>>(p);
      break;
    case 8:
      if (vec) grid_gather_kernel<8, true><<<g, 256, 0, stream>>>(p);
      else grid_gather_kernel<8, false><<<g, 256, 0, stream>>>(p);
      break;
    case 16:
      if (vec) grid_gather_kernel<16, true><<<g, 256, 0, stream>>>(p);
      else grid_gather_kernel<16, false><<<g, 256, 0, stream>>>(p);
      break;
    default: return SG_ERR_UNSUPPORTED;
  }
  SG_LAUNCH_CHECK();
  return SG_OK;
}

extern "C" int sg_grid_scatter(const float *ori, const float *dir, const float *z, int B, int N, int S,
                               const float *grad_out, const float *grid, int D, int C, const float *vol_bbox,
                               const float *voxel_size, int mode, float scale, float s, float *grad_grid,
                               sg_stream_t stream) {
  if (!ori || !dir || !z || !grad_out || !vol_bbox || !voxel_size || !grad_grid) return SG_ERR_INVALID_ARG;
  if (B <= 0 || N <= 0 || S <= 0 || D <= 0 || C <= 0 || C > 16) return SG_ERR_INVALID_ARG;
  if (mode == 1 && (C != 1 || s == 0.0f || !grid)) return SG_ERR_INVALID_ARG;
  if (mode != 0 && mode != 1) return SG_ERR_INVALID_ARG;
  if (C != 1 && C != 3 && C != 4 && C != 8 && C != 16) return SG_ERR_UNSUPPORTED;
  ScatterParams p{ori, dir, z, (long)B * N, N, S, grad_out, grid, D, vol_bbox, voxel_size, mode, scale, s,
                  grad_grid, 1, 0};
  const long R = (long)B * N, fill = (long)num_sms() * kScatterFill;
  if (R < fill && S > 8) {
    const int steps = (S - 1) / 8 + 1, want = (int)((fill + R - 1) / R);  // steps of 8 samples
    p.part = ((steps - 1) / want + 1) * 8;
    p.parts = (S - 1) / p.part + 1;
  }
  if (p.parts > 1) launch_scatter<true>(p, C, stream);
  else launch_scatter<false>(p, C, stream);
  SG_LAUNCH_CHECK();
  return SG_OK;
}

extern "C" int sg_zero_near_nodes(const SgTree *tree, float *grid, int C, sg_stream_t stream) {
  if (!tree || !tree->brick_node || !grid) return SG_ERR_INVALID_ARG;
  if (tree->B <= 0 || tree->Dt <= 0 || tree->rate <= 0 || tree->Db != tree->Dt * tree->rate || C <= 0)
    return SG_ERR_INVALID_ARG;
  const long vt = (long)tree->Dt * tree->Dt * tree->Dt;
  if (vt > INT_MAX || tree->B > 65535) return SG_ERR_UNSUPPORTED;
  const int vec4 = ((tree->rate * C) % 4 == 0 && ((uintptr_t)grid) % 16 == 0) ? 1 : 0;
  const int per_run = vec4 ? tree->rate * C / 4 : tree->rate * C;
  const FixedDiv31 by_brick = FixedDiv31::of((uint32_t)(tree->rate * tree->rate * per_run)),
                   by_run = FixedDiv31::of((uint32_t)per_run), by_rate = FixedDiv31::of((uint32_t)tree->rate);
  if (vt * tree->B >= (long)num_sms() * kZeroBricks)
    zero_near_nodes_kernel<kZeroBricks><<<dim3((unsigned)ceil_div(vt, kZeroBricks), tree->B), 256, 0, stream>>>(
        *tree, grid, C, vec4, by_brick, by_run, by_rate);
  else
    zero_near_nodes_kernel<1><<<dim3((unsigned)vt, tree->B), 256, 0, stream>>>(*tree, grid, C, vec4, by_brick, by_run,
                                                                               by_rate);
  SG_LAUNCH_CHECK();
  return SG_OK;
}
