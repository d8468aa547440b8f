// render.cu -- fused per-ray render and its adjoint: sampling -> sort -> field
// taps -> compositing, forward and backward in one kernel each.
//
// One warp per ray does, without leaving the SM:
//   the reference's coarse sampling (ray_voxels_sampling_uniform_kernel,
//   sampling_kernel.cu:1070-1177) into shared memory, the per-ray sort
//   (sort_samplings :1308-1329) in registers, per-sample density from the
//   fused TSDF grid and colour from a dense feature grid (trilinear taps and
//   a linear colour head; the stand-in for SRONet's MLP), and density
//   compositing of the sorted samples (volume_rendering_training_forward_
//   kernel, volume_rendering.cu:17-126, with the transmittance carried in
//   strict sample order).
// The forward writes 24 bytes per ray (rgb, depth, weight sum, alpha); the
// sorted depths / node ids only when requested.  With a 3-channel colour
// grid and no head its results equal the unfused chain sg_sample_sorted ->
// sg_grid_gather (x2) -> sg_composite_fwd on the same inputs.
//
// A ray's sorted positions are evaluated in blocks of 32, front to back: the
// density taps of a block, its alphas, the transmittance through it, and
// colour taps for its samples up to the early termination.  The walk stops
// at the block in which the ray ends, so nothing is tapped behind it: of the
// 85 M record slots of the 7.4 M-ray training step 46 M hold samples that
// count, and the taps (latency of scattered 16-byte loads, 3-6 % of HBM)
// are what the kernels are bound by.  What a later pass needs of a position
// (weight, colour, alpha, ...) sits in warp-private shared memory, so the
// block loop stays rolled: one body of code for every sample count (the
// unrolled one stalled on instruction fetch) and 62-80 registers.  Against
// the kernels that evaluated every position first: 2^20 random rays of 96
// samples forward + adjoint 27.2 -> 15.1 ms, 2^20 pixel rays forward (with
// fusion and tree) 4.11 -> 3.71 ms, a 3.9 M-ray training step 11.1 -> 10.1.
//
// The backward saves nothing from the forward: it re-runs the same per-ray
// evaluation (same samples, taps, alpha and transmittance, bit for bit),
// forms the exact adjoint of compositing from in-warp prefix sums, chains
// it through the density transform and the colour head, and scatters the
// per-sample gradients into the TSDF and feature grids: lanes own (corner,
// channel) slots, consecutive samples in one trilinear cell accumulate in
// registers, and each cell change flushes one atomic add per slot.
//
// Launches are persistent grid-stride loops over the rays of all frames and
// target cameras; a segment table (SgRaySegments) gives each ray its frame
// and sample count.
#include <climits>

#include "ray_core.cuh"
#include "scatter.cuh"

// Resident CTAs per SM the register budgets are set for (build-time settings).
// Measured at 3 / 4 / 5 for the forward and the record pass and 2 / 3 / 4 for
// the adjoint, packed taps: 2^20 random rays of 96 samples, forward 1.46 /
// 1.27 / 1.40 ms, adjoint 5.67 / 5.35 / 5.22 ms (at 4 the shared memory of
// 128 positions takes 196 KB of the SM); the record pass and reduction of a
// 4.2 M-ray step 4.13 / 4.01 / 4.05 ms.  Unpacked forward (scalar taps, more
// registers), 2^20 pixel rays of a 512^3 frame with their intersection, at 3 /
// 4 / 5: 1.69 / 1.78 / 1.76 ms.  Unpacked adjoint of 16 channels (at 4 it
// spilled), at 2 / 3 / 4, camera rays over 256^3: 1024 x 48 samples 27 / 31 / 39
// us, 9216 x 96 44 / 58 / 74, 65536 x 64 171 / 159 / 169, 2^18 x 96 772 / 804 / 858;
// training steps by records 2 % slower at 2 and 4 than at 3.
#ifndef SG_RENDER_FWD_MINB
#define SG_RENDER_FWD_MINB(PACKED) ((PACKED) ? 4 : 3)
#endif
#ifndef SG_RENDER_REC_MINB
#define SG_RENDER_REC_MINB(PACKED) ((PACKED) ? 4 : 3)
#endif
#ifndef SG_RENDER_ADJ_MINB
#define SG_RENDER_ADJ_MINB(PACKED) ((PACKED) ? 4 : 3)
#endif
#define SG_RENDER_MINB(MODE, PACKED) ((MODE) == kModeRec ? SG_RENDER_REC_MINB(PACKED) : SG_RENDER_ADJ_MINB(PACKED))

namespace sg {

struct RenderParams {
  SampleParams sp;  // tree, hits, jitter, valid_len, N (rays per frame without segments), W, S (row stride)
  const int *hit_count;
  float rand_const;
  long R;
  int nseg;  // 0: frames of sp.N rays with sp.S samples each
  const int *seg_begin, *seg_frame, *seg_samples;
  const float *ori, *dir;
  const float *tsdf;
  int D;
  float sdf_scale, sdf_s;
  const float *feat;
  int Df;
  const float *fbbox, *fvs;
  const float *head;  // [3, C] or null (C == 3)
  float t_thres;
  float dk, inv_s;    // density constants: sdf_scale / sdf_s, 1 / sdf_s
  bool shared;        // feature grid on the TSDF grid's geometry (one tap cell)
  float *out_rgb, *out_depth, *out_ws, *out_alpha, *out_z;
  int *out_node;
  const float *g_rgb, *g_depth, *g_ws, *g_alpha;
  float *grad_feat, *grad_tsdf, *grad_sigma, *grad_rgb;
  // training step: upstream gradient of loss_scale / 2 * |rgb - target|^2
  const float *target_rgb;
  float loss_scale;
  float *out_loss;
  // gradient records instead of the scatter (deterministic reduction,
  // scatter.cu): the launch's rays are hit_ray[k], k in [*k_begin, *k_end);
  // ray k's records, in sorted position order, go to record slots
  // hit_slot[k], hit_slot[k] + 1, ... (below rec_cap), their count to
  // ray_nrec[k]
  const int *hit_ray, *hit_slot, *k_begin, *k_end;
  int *ray_nrec;
  uint32_t *rec_key;
  GradRecord *rec, *rec_t;
  float *ray_g;  // [k][C]: head^T (colour gradient of ray k)
  long rec_cap;
  RecordKeys keys;
  int cap;  // positions a warp's shared memory holds: 32, 64 or 128
  // packed fields of the voxels near the tree's nodes (pack_fields_kernel),
  // and log2 of the brick edge; null: taps read the grids themselves
  const float4 *packed;
  int rate_shift;
};

__device__ __forceinline__ void ray_frame(const RenderParams &p, long r, int &b, int &S, int &s) {
  if (p.nseg > 0) {
    s = segment_of(p.seg_begin, p.nseg, r);
    b = __ldg(p.seg_frame + s);
    S = min(__ldg(p.seg_samples + s), p.sp.S);
  } else {
    s = 0;
    b = (int)(r / p.sp.N);
    S = p.sp.S;
  }
}

// Warp-private shared memory of the render kernels (dynamic; cap = 32, 64 or
// 128 positions).
//   z    [cap]     samples, then sorted depths
//   f    [32 + 32] transmittance factors of a block and the values before them
//   id, pos [cap]  node ids and sorted positions (forward with out_node)
//   keep [8][cap]  per position, for the adjoint: see Keep
//   cw   [32][9], wg [32]  corner sums and (voxel, corners inside) of a block's
//                  runs (in-kernel scatter)
enum { kKeepW = 0, kKeepR, kKeepG, kKeepB, kKeepS01, kKeepAl, kKeepTb, kKeepDl, kKeepWords };

struct RenderSmem {
  float *z, *f;
  int *id, *pos;
  float *keep;
  float *cw;
  unsigned long long *wg;
  int cap;
  __device__ __forceinline__ float &k(int which, int i) const { return keep[which * cap + i]; }
};

// What a mode of the kernel needs beside the samples.
enum { kModeFwd = 0, kModeBwd = 1, kModeTrain = 2, kModeRec = 3, kModeRecTsdf = 4 };
__host__ __device__ constexpr bool mode_keeps(int mode) {
  return mode == kModeBwd || mode == kModeTrain || mode == kModeRecTsdf;
}
__host__ __device__ constexpr bool mode_scatters(int mode) { return mode == kModeBwd || mode == kModeTrain; }

__host__ __device__ constexpr int render_warp_words(int mode, int cap, bool ids) {
  return cap + 64 + (ids ? 2 * cap : 0) + (mode_keeps(mode) ? kKeepWords * cap : 0) +
         (mode_scatters(mode) ? 32 * 9 + 64 : 0);
}

__device__ __forceinline__ RenderSmem render_smem(float *base, int mode, int cap, bool ids) {
  RenderSmem sm;
  sm.cap = cap;
  float *w = base + (threadIdx.x >> 5) * render_warp_words(mode, cap, ids);
  sm.z = w;
  w += cap;
  sm.f = w;
  w += 64;
  sm.id = sm.pos = nullptr;
  if (ids) {
    sm.id = reinterpret_cast<int *>(w);
    sm.pos = reinterpret_cast<int *>(w + cap);
    w += 2 * cap;
  }
  sm.keep = w;
  if (mode_keeps(mode)) w += kKeepWords * cap;
  sm.cw = w;
  sm.wg = reinterpret_cast<unsigned long long *>(w + 32 * 9);
  return sm;
}

// Geometry of a ray: what the taps of its samples need.
struct RayGeom {
  float o[3], d[3];
  float bmin[3], vs, inv_vs;  // TSDF grid
  int b;
};

__device__ __forceinline__ RayGeom ray_geom(const RenderParams &p, long r, int b) {
  RayGeom g;
  const float *bb = p.sp.t.vol_bbox + 6 * b;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    g.o[a] = __ldg(p.ori + r * 3 + a);
    g.d[a] = __ldg(p.dir + r * 3 + a);
    g.bmin[a] = __ldg(bb + 2 * a);
  }
  g.vs = __ldg(p.sp.t.voxel_size + b);
  g.inv_vs = 1.0f / g.vs;
  g.b = b;
  return g;
}

__device__ __forceinline__ void ray_point(const RayGeom &g, float z, float pt[3]) {
#pragma unroll
  for (int a = 0; a < 3; a++) pt[a] = __fmaf_rn(g.d[a], z, g.o[a]);
}

// Cell and fractions of a sample on the feature grid: the TSDF grid's when
// both lie on one geometry.
__device__ __forceinline__ void feat_cell(const RenderParams &p, const RayGeom &g, float z, int (&i0)[3],
                                          float (&f)[3]) {
  float pt[3];
  ray_point(g, z, pt);
  if (p.shared) {
    tap_frac(g.bmin, g.vs, g.inv_vs, pt, i0, f);
  } else {
    const float *fb = p.fbbox + 6 * g.b;
    const float fmin[3] = {__ldg(fb), __ldg(fb + 2), __ldg(fb + 4)};
    const float fvs = __ldg(p.fvs + g.b);
    tap_frac(fmin, fvs, 1.0f / fvs, pt, i0, f);
  }
}

// Colour of one voxel: the linear head (in shared memory, [3][C]) of its
// features, or its three channels.
template <int C>
__device__ __forceinline__ void voxel_colour(const float *__restrict__ g, bool head, const float *s_head,
                                             float (&rgb)[3]) {
  if constexpr (C % 4 == 0) {
    rgb[0] = rgb[1] = rgb[2] = 0.0f;
#pragma unroll
    for (int c = 0; c < C / 4; c++) {
      const float4 q = __ldg(reinterpret_cast<const float4 *>(g) + c);
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const float4 h = *reinterpret_cast<const float4 *>(s_head + k * C + 4 * c);
        rgb[k] = __fmaf_rn(h.w, q.w, __fmaf_rn(h.z, q.z, __fmaf_rn(h.y, q.y, __fmaf_rn(h.x, q.x, rgb[k]))));
      }
    }
  } else {
    const float v[3] = {__ldg(g), __ldg(g + 1), __ldg(g + 2)};
#pragma unroll
    for (int k = 0; k < 3; k++)
      rgb[k] = head ? __fmaf_rn(s_head[k * C + 2], v[2], __fmaf_rn(s_head[k * C + 1], v[1], s_head[k * C] * v[0])) : v[k];
  }
}

// Colour of a sample: the trilinear tap of the voxels' colours (the head is
// linear, so this is the head of the tapped features), in the arithmetic of
// the packed tap, so that a sample's colour does not depend on where it is
// read from.
template <int C>
__device__ __forceinline__ void colour_tap(const RenderParams &p, const float *s_head, int b, const int (&i0)[3],
                                           const float (&f)[3], float (&rgb)[3]) {
  const float *feat = p.feat + (size_t)b * p.Df * p.Df * p.Df * C;
  rgb[0] = rgb[1] = rgb[2] = 0.0f;
#pragma unroll
  for (int cr = 0; cr < 8; cr++) {
    size_t off;
    if (!corner_inside(i0, cr, p.Df, off)) continue;
    const float w = corner_weight(f, cr);
    float v[3];
    voxel_colour<C>(feat + off * C, p.head != nullptr, s_head, v);
#pragma unroll
    for (int k = 0; k < 3; k++) rgb[k] = __fmaf_rn(w, v[k], rgb[k]);
  }
}

// The head's [3][C] floats into shared memory (the whole CTA).
template <int C>
__device__ __forceinline__ void load_head(const float *__restrict__ head, float *s_head) {
  if (threadIdx.x < 3 * C) s_head[threadIdx.x] = head ? __ldg(head + threadIdx.x) : 0.0f;
  __syncthreads();
}

// Colour and TSDF of a sample from the grids themselves: the packed tap of a
// cell that is not wholly inside the grid or not near a node.
template <int C>
__device__ __noinline__ float4 unpacked_tap(const RenderParams &p, const float *s_head, int b, int x, int y, int z, float fx, float fy,
                                            float fz) {
  const int i0[3] = {x, y, z};
  const float f[3] = {fx, fy, fz};
  float w[8], t1[1], rgb[3];
#pragma unroll
  for (int cr = 0; cr < 8; cr++) w[cr] = corner_weight(f, cr);
  grid_tap_cell<1>(p.tsdf + (size_t)b * p.D * p.D * p.D, p.D, i0, w, t1);
  colour_tap<C>(p, s_head, b, i0, f, rgb);
  return make_float4(rgb[0], rgb[1], rgb[2], t1[0]);
}

// Colour and TSDF of a sample in one trilinear tap of the packed grid.  Every
// corner is packed when the voxel nearest to the sample lies in a node's
// brick (the corners are then within one voxel of the brick); the brick map
// is read beside the corners, and other cells go to the grids themselves.
template <int C>
__device__ __forceinline__ float4 packed_tap(const RenderParams &p, const float *s_head, int b, const int (&i0)[3], const float (&f)[3]) {
  const int D = p.D;
  const unsigned m = (unsigned)(D - 1);
  if ((unsigned)i0[0] < m && (unsigned)i0[1] < m && (unsigned)i0[2] < m) {
    const int Dt = p.sp.t.Dt, sh = p.rate_shift;
    const int X = (i0[0] + (f[0] >= 0.5f)) >> sh, Y = (i0[1] + (f[1] >= 0.5f)) >> sh,
              Z = (i0[2] + (f[2] >= 0.5f)) >> sh;
    const int node = __ldg(p.sp.t.brick_node + (((long)b * Dt + X) * Dt + Y) * Dt + Z);
    const float4 *q = p.packed + (((long)b * D + i0[0]) * D + i0[1]) * D + i0[2];
    const long dx = (long)D * D;
    const float gx = 1.0f - f[0], gy = 1.0f - f[1], gz = 1.0f - f[2];
    const float w[8] = {gx * gy * gz, gx * gy * f[2], gx * f[1] * gz, gx * f[1] * f[2],
                        f[0] * gy * gz, f[0] * gy * f[2], f[0] * f[1] * gz, f[0] * f[1] * f[2]};
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int cr = 0; cr < 8; cr++) {
      const float4 v = __ldg(q + ((cr & 4) ? dx : 0) + ((cr & 2) ? D : 0) + (cr & 1));
      a.x = __fmaf_rn(w[cr], v.x, a.x);
      a.y = __fmaf_rn(w[cr], v.y, a.y);
      a.z = __fmaf_rn(w[cr], v.z, a.z);
      a.w = __fmaf_rn(w[cr], v.w, a.w);
    }
    if (node >= 0) return a;
  }
  return unpacked_tap<C>(p, s_head, b, i0[0], i0[1], i0[2], f[0], f[1], f[2]);
}

// Packed fields: (colour, TSDF) of every voxel in a node's brick or within
// one voxel of one (voxel_colour): a sample then reads 8 x 16 bytes instead
// of 8 x (64 + 4), and no head runs per sample.
// Measured: 5037 nodes of 8^3 bricks with 16 channels (about 0.35 GB read and
// 80 MB written) pack in 82 us, beside the intersection in a training step;
// with it the forward
// of 2^20 random rays of 96 samples takes 1.27 ms where taps of the grids
// took 6.39 ms, their adjoint 5.2 (15.2), and the record pass of a 4.2 M-ray
// step 1.7 (4.5).
// A CTA per top node, in a grid-stride loop over the node list: its rate^3
// voxels and the shell around them, shell voxels of a neighbouring node's
// brick left to that node.  Only bricks with nodes are read (about 5 % of the
// voxels of a fused scene).
template <int C>
__global__ void __launch_bounds__(256) pack_fields_kernel(SgTree t, const float *__restrict__ feat,
                                                          const float *__restrict__ head,
                                                          const float *__restrict__ tsdf, int D,
                                                          float4 *__restrict__ packed) {
  __shared__ __align__(16) float s_head[3 * C];
  __shared__ int s_near[27];
  load_head<C>(head, s_head);
  const int n = __ldg(t.counts), r = t.rate, e = r + 2, Dt = t.Dt;
  const long vt = (long)Dt * Dt * Dt;
  for (int k = blockIdx.x; k < n; k += gridDim.x) {
    const long key = __ldg(t.top_key + k);
    const int b = (int)(key / vt);
    const long l = key - b * vt;
    const int X = (int)(l / ((long)Dt * Dt)), Y = (int)((l / Dt) % Dt), Z = (int)(l % Dt);
    __syncthreads();  // the previous node's readers of s_near are done
    if (threadIdx.x < 27) {
      const int x = X + (int)threadIdx.x / 9 - 1, y = Y + ((int)threadIdx.x / 3) % 3 - 1,
                z = Z + (int)threadIdx.x % 3 - 1;
      s_near[threadIdx.x] = x >= 0 && y >= 0 && z >= 0 && x < Dt && y < Dt && z < Dt &&
                            __ldg(t.brick_node + b * vt + ((long)x * Dt + y) * Dt + z) >= 0;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < e * e * e; i += blockDim.x) {
      const int lx = i / (e * e) - 1, ly = (i / e) % e - 1, lz = i % e - 1;
      const int x = X * r + lx, y = Y * r + ly, z = Z * r + lz;
      if (x < 0 || y < 0 || z < 0 || x >= D || y >= D || z >= D) continue;
      const int nb = (lx < 0 ? 0 : (lx < r ? 9 : 18)) + (ly < 0 ? 0 : (ly < r ? 3 : 6)) + (lz < 0 ? 0 : (lz < r ? 1 : 2));
      if (nb != 13 && s_near[nb]) continue;
      const size_t v = (((size_t)b * D + x) * D + y) * D + z;
      float c[3];
      voxel_colour<C>(feat + v * C, head != nullptr, s_head, c);
      packed[v] = make_float4(c[0], c[1], c[2], __ldg(tsdf + v));
    }
  }
}

// Evaluation of one block of 32 sorted positions of a ray.
struct BlockEval {
  float z, al, tb, dl, s01, w;
  float rgb[3];
  int i0[3];    // cell of a used sample on the feature grid
  float f[3];
  bool used;    // a sample, at or before the early termination
};

// State of a ray's walk over its blocks.
struct RayWalk {
  float T;
  int m0;    // first position that holds a sample (-1: not met yet)
  int end;   // positions at and after it are past the termination
};

// Block e: density taps, alpha, transmittance, and the colour of the samples
// that count -- positions past the early termination are never tapped.
// Returns false when the block holds no sample.
// U: positions per unrolled stretch of the transmittance chain (the record
// pass is the faster for 32, by 0.7 %; forward and adjoint for 8, by 2 to 6 %).
template <int C, bool PACKED, int U = 8>
__device__ __forceinline__ bool eval_block(const RenderParams &p, const RayGeom &g, int S, int e,
                                           const RenderSmem &sm, const float *s_head, RayWalk &wk, BlockEval &v) {
  const int lane = lane_id(), i = e * 32 + lane;
  v.z = i < S ? sm.z[i] : -1.0f;
  const bool valid = v.z >= 0.0f;
  const unsigned vb = __ballot_sync(SG_FULL, valid);
  if (vb == 0u) return false;
  if (wk.m0 < 0) wk.m0 = e * 32 + __ffs(vb) - 1;
  v.al = v.dl = v.s01 = v.w = 0.0f;
  v.rgb[0] = v.rgb[1] = v.rgb[2] = 0.0f;
  if (valid) {
    float pt[3];
    ray_point(g, v.z, pt);
    tap_frac(g.bmin, g.vs, g.inv_vs, pt, v.i0, v.f);
    float t1[1];
    if constexpr (PACKED) {
      const float4 a = packed_tap<C>(p, s_head, g.b, v.i0, v.f);
      v.rgb[0] = a.x;
      v.rgb[1] = a.y;
      v.rgb[2] = a.z;
      t1[0] = a.w;
    } else {
      float wc[8];
#pragma unroll
      for (int cr = 0; cr < 8; cr++) wc[cr] = corner_weight(v.f, cr);
      grid_tap_cell<1>(p.tsdf + (size_t)g.b * p.D * p.D * p.D, p.D, v.i0, wc, t1);
    }
    v.s01 = tsdf_sigmoid(t1[0], p.dk);  // kept for the adjoint
    const float sg = v.s01 * p.inv_s;
    v.dl = depth_step(sm.z, S, i, v.z);
    v.al = 1.0f - expf(-sg * v.dl);
  }
  const int stop = block_transmittance<U>(valid ? 1.0f - v.al : 1.0f, wk.T, p.t_thres, wk.m0 - e * 32, S - e * 32, sm.f,
                                       v.tb);
  if (stop < 32) wk.end = e * 32 + stop + 1;
  v.used = valid && i < wk.end;
  if (v.used) {
    v.w = v.al * v.tb;
    if constexpr (!PACKED) {
      if (!p.shared) feat_cell(p, g, v.z, v.i0, v.f);
      colour_tap<C>(p, s_head, g.b, v.i0, v.f, v.rgb);
    }
  } else if constexpr (PACKED) {
    v.rgb[0] = v.rgb[1] = v.rgb[2] = 0.0f;
  }
  return true;
}

// Samples and sort of ray r; returns the number of samples (sorted depths in
// sm.z, padding first).
template <bool IDS>
__device__ __forceinline__ int sample_and_sort(const RenderParams &p, long r, int b, int S, const RenderSmem &sm) {
  const int nh = p.hit_count ? min(__ldg(p.hit_count + r), p.sp.W) : p.sp.W;
  const int done = warp_sample_ray<IDS>(p.sp, r, b, S, nh, p.rand_const, sm.z, sm.id);
  if (done > 0) warp_sort_samples<4, IDS>(sm.z, sm.pos, S, done);
  return done;
}

extern __shared__ __align__(16) float s_render[];

// The rays of a CTA are eight consecutive ones, and the same a grid apart: warp
// w takes the w-th of each eight, or the warps take them one by one (take_ray), so
// that a ray that misses or ends early leaves its warp free for the next.  One by
// one in the packed forward and in the adjoints: 2^20 random rays, a third of them
// hitting, one by one / fixed, forward 1.19 / 1.27 ms, adjoint 4.30 / 4.94.  Fixed
// in the record pass, whose rays all hit (3.91 / 3.85 with the reduction), and in
// the unpacked forward (pixel rays of a frame, with their intersection, 1.70 /
// 1.68: no gain).
__device__ __forceinline__ long take_ray(int &taken, long first) {
  int i = 0;
  if (lane_id() == 0) i = atomicAdd(&taken, 1);
  i = __shfl_sync(SG_FULL, i, 0);
  return first + ((long)(i >> 3) * gridDim.x + blockIdx.x) * 8 + (i & 7);
}

template <int C, bool IDS, bool PACKED>
__global__ void __launch_bounds__(256, SG_RENDER_FWD_MINB(PACKED)) render_fwd_kernel(RenderParams p) {
  __shared__ __align__(16) float s_head[3 * C];
  load_head<C>(p.head, s_head);
  const RenderSmem sm = render_smem(s_render, kModeFwd, p.cap, IDS);
  const int lane = lane_id();
  const int Smax = p.sp.S;
  // a segment table covers rays [ray_begin[0], total): a sub-table of
  // consecutive segments is a group of targets
  const long r0 = p.nseg > 0 ? (long)__ldg(p.seg_begin) : 0;
  __shared__ int s_taken;
  if (PACKED) {
    if (threadIdx.x == 0) s_taken = 0;
    __syncthreads();
  }
  for (long r = PACKED ? take_ray(s_taken, r0) : r0 + (((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5); r < p.R;
       r = PACKED ? take_ray(s_taken, r0) : r + (((long)gridDim.x * blockDim.x) >> 5)) {
    int b, S, sgm;
    ray_frame(p, r, b, S, sgm);
    const int done = sample_and_sort<IDS>(p, r, b, S, sm);
    if (IDS) {
      for (int i = lane; i < Smax; i += 32) {
        const bool has = done > 0 && i < S;
        p.out_z[(size_t)r * Smax + i] = has ? sm.z[i] : -1.0f;
        p.out_node[(size_t)r * Smax + i] = has ? sm.id[sm.pos[i]] : -1;
      }
    }
    float acc_r = 0.0f, acc_g = 0.0f, acc_b = 0.0f, d = 0.0f, ws = 0.0f, aa = 0.0f;
    if (done > 0) {
      // a ray whose largest depth is < 0 renders 0 (no sample: done == 0)
      const RayGeom g = ray_geom(p, r, b);
      RayWalk wk{1.0f, -1, S};
#pragma unroll 1
      for (int e = (S - done) >> 5; e * 32 < wk.end; e++) {
        BlockEval v;
        if (!eval_block<C, PACKED>(p, g, S, e, sm, s_head, wk, v)) continue;
        if (v.used) {
          acc_r += v.w * v.rgb[0];
          acc_g += v.w * v.rgb[1];
          acc_b += v.w * v.rgb[2];
          d += v.w * v.z;
          ws += v.w;
          aa += v.w * v.al;
        }
      }
      acc_r = warp_sum(acc_r);
      acc_g = warp_sum(acc_g);
      acc_b = warp_sum(acc_b);
      d = warp_sum(d);
      ws = warp_sum(ws);
      aa = warp_sum(aa);
    }
    if (lane == 0) {
      p.out_rgb[r * 3 + 0] = acc_r;
      p.out_rgb[r * 3 + 1] = acc_g;
      p.out_rgb[r * 3 + 2] = acc_b;
      p.out_depth[r] = d;
      p.out_ws[r] = ws;
      p.out_alpha[r] = aa;
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
// Sums over the runs of lanes that share a cell, at each run's first lane:
// 8 corner weights x the compositing weight (A) and x the TSDF gradient (T).
// stop: the first lane behind this one that is not of its run.
template <bool A, bool T>
__device__ __forceinline__ void run_sums(bool has, int stop, const float (&f)[3], float w, float gt, float (&a)[8],
                                         float (&t)[8]) {
  const int lane = lane_id();
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const float cw = corner_weight(f, c);
    if (A) a[c] = has ? cw * w : 0.0f;
    if (T) t[c] = has ? cw * gt : 0.0f;
  }
#pragma unroll 1
  for (int o = 1; __any_sync(SG_FULL, has && lane + o < stop); o <<= 1) {
    const bool in = lane + o < stop;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      if (A) {
        const float x = __shfl_down_sync(SG_FULL, a[c], o);
        if (in) a[c] += x;
      }
      if (T) {
        const float y = __shfl_down_sync(SG_FULL, t[c], o);
        if (in) t[c] += y;
      }
    }
  }
}

// A block's samples added into the grids.  The colour head is linear, so the
// feature gradient of the sample at sorted position i is w_i G with G = head^T
// g_c (g_c: the gradient of the ray's colour, w_i its compositing weight): each
// run of samples in one cell is summed first (run_sums), its first lane leaves
// the 8 sums, the cell's voxel and the corners inside the grid in shared memory,
// and the warp adds run after run.  C == 16: lane l owns corner l / 4, channels
// 4 (l % 4) .. + 3 (one vector reduction), and its corner's TSDF gradient
// (channel group 0).  C == 3: lane l < 24 owns corner l / 3, channel l % 3; lane
// l >= 24 the TSDF gradient of corner l - 24.
//
// keep: the block's 8 x 32 words of the positions' values (all read by now),
// which take the TSDF sums, corner c of lane l at word (l + 4 c) % 32 of row c.
// Sample by sample with a flush at each change of cell, 2^20 random rays of 96
// samples and 16 channels took 5.24 ms, now 4.94 (adjoint; 4.3 with the
// rays shared among a CTA's warps).
template <int C, bool FEAT, bool TSDF>
__device__ __forceinline__ void scatter_block(const RenderParams &p, int b, const RenderSmem &sm, int block, bool used,
                                              const int (&i0)[3], const float (&f)[3], float w, float gt,
                                              const float (&G)[4]) {
  const int lane = lane_id(), D = FEAT ? p.Df : p.D;
  const unsigned in = used ? corners_inside(i0, D) : 0u;
  const unsigned m = __ballot_sync(SG_FULL, in != 0u);
  if (m == 0u) return;
  const int px = __shfl_up_sync(SG_FULL, i0[0], 1), py = __shfl_up_sync(SG_FULL, i0[1], 1),
            pz = __shfl_up_sync(SG_FULL, i0[2], 1);
  const bool head = in != 0u && (lane == 0 || !((m >> (lane - 1)) & 1u) || px != i0[0] || py != i0[1] || pz != i0[2]);
  const unsigned heads = __ballot_sync(SG_FULL, head);
  const unsigned stops = (heads | ~m) & ~((2u << lane) - 1u);
  float a[8], t[8];
  run_sums<FEAT, TSDF>(in != 0u, stops ? __ffs(stops) - 1 : 32, f, w, gt, a, t);
  float *keep = sm.keep + block * 32;
  unsigned long long *cell = sm.wg;
  __syncwarp();
  if (head) {
    // lower corner's voxel (frame included; two's complement) and the corners inside
    const long at = (((long)b * D + i0[0]) * D + i0[1]) * D + i0[2];
    cell[lane] = ((unsigned long long)at << 8) | in;
#pragma unroll
    for (int c = 0; c < 8; c++) {
      if (FEAT) sm.cw[lane * 9 + c] = a[c];
      if (TSDF) keep[c * sm.cap + ((lane + 4 * c) & 31)] = t[c];
    }
  }
  __syncwarp();
  const int cr = C == 16 ? lane >> 2 : (lane < 24 ? lane / 3 : lane - 24);
  const int ch = C == 16 ? 4 * (lane & 3) : lane % 3;
  const long at1 = ((long)(cr >> 2) * D + ((cr >> 1) & 1)) * D + (cr & 1);
  const bool fown = FEAT && (C == 16 || lane < 24), town = TSDF && (C == 16 ? (lane & 3) == 0 : lane >= 24);
  for (unsigned q = heads; q; q &= q - 1) {
    const int j = __ffs(q) - 1;
    const unsigned long long x = cell[j];
    if (!((x >> cr) & 1u)) continue;
    const long v = ((long)x >> 8) + at1;
    if (fown) {
      const float k = sm.cw[j * 9 + cr];
      float *g = p.grad_feat + v * C + ch;
      // terms of 0 are left out; 0 x NaN and 0 x infinity are not 0
      if constexpr (C == 16) {
        const float t0 = k * G[0], t1 = k * G[1], t2 = k * G[2], t3 = k * G[3];
        if (t0 != 0.0f || t1 != 0.0f || t2 != 0.0f || t3 != 0.0f) red_add_f32x4(g, t0, t1, t2, t3);
      } else {
        const float t0 = k * G[0];
        if (t0 != 0.0f) atomicAdd(g, t0);
      }
    }
    if (town) {
      const float k = keep[cr * sm.cap + ((j + 4 * cr) & 31)];
      if (k != 0.0f) atomicAdd(p.grad_tsdf + v, k);
    }
  }
  __syncwarp();
}

// head^T g_c for channel c of the feature grid.
template <int C>
__device__ __forceinline__ float head_grad(const RenderParams &p, int c, const float (&gc)[3]) {
  if (p.head)
    return __fmaf_rn(__ldg(p.head + 2 * C + c), gc[2], __fmaf_rn(__ldg(p.head + C + c), gc[1],
                                                                  __ldg(p.head + c) * gc[0]));
  return c == 0 ? gc[0] : (c == 1 ? gc[1] : (c == 2 ? gc[2] : 0.0f));
}

// Records of a block's samples for the deterministic reduction, one for each
// run of samples of consecutive positions in one cell: the cell (the key) and,
// at the run's first lane, the sums of corner weight x compositing weight (and
// x TSDF gradient) over the run.  The records of a ray are packed, in sorted
// position order, from slot base on (n: those written by the blocks before;
// updated).  A record per sample made 2.1 to 2.3 times as many to write, sort
// and sum.
template <bool TSDF>
__device__ __forceinline__ void emit_records(const RenderParams &p, int b, long base, bool used, const int (&i0)[3],
                                             const float (&f)[3], float w, float gt, int &n) {
  const int lane = lane_id();
  const uint32_t key = used ? record_key(p.keys, b, i0) : p.keys.invalid;
  const bool has = key != p.keys.invalid;
  const unsigned m = __ballot_sync(SG_FULL, has);
  if (m == 0u) return;
  const uint32_t before = __shfl_up_sync(SG_FULL, key, 1);
  const bool head = has && (lane == 0 || before != key);
  const unsigned heads = __ballot_sync(SG_FULL, head);
  const unsigned stops = (heads | ~m) & ~((2u << lane) - 1u);  // lanes behind this one that are not of its run
  const int stop = stops ? __ffs(stops) - 1 : 32;
  float a[8], t[8];
  run_sums<true, TSDF>(has, stop, f, w, gt, a, t);
  const long slot = base + n + __popc(heads & ((1u << lane) - 1u));
  if (head && slot < p.rec_cap) {
    float4 *r = reinterpret_cast<float4 *>(p.rec + slot);
    r[0] = make_float4(a[0], a[1], a[2], a[3]);
    r[1] = make_float4(a[4], a[5], a[6], a[7]);
    if (TSDF) {
      float4 *q = reinterpret_cast<float4 *>(p.rec_t + slot);
      q[0] = make_float4(t[0], t[1], t[2], t[3]);
      q[1] = make_float4(t[4], t[5], t[6], t[7]);
    }
    p.rec_key[slot] = key;
  }
  n += __popc(heads);
}

// MODE kModeBwd: the adjoint for given upstream gradients.  The training
// modes form the upstream gradient in the kernel from the ray's own outputs
// (loss = loss_scale / 2 * |rgb - target|^2 per ray, so d loss / d rgb =
// loss_scale * (rgb - target)); the outputs and per-ray loss are written, and
// nothing is recomputed.  kModeTrain scatters with atomics; in the record
// modes the rays are the compact list of rays with hits and the grid
// gradients leave the kernel as records (emit_records) for the
// deterministic reduction (scatter.cu).  Without the TSDF's gradient
// (kModeRec) a record needs nothing that comes after its sample, so it is
// written as soon as the sample's weight is known and no adjoint runs.
template <int C, int MODE, bool PACKED>
__global__ void __launch_bounds__(256, SG_RENDER_MINB(MODE, PACKED)) render_bwd_kernel(RenderParams p) {
  static_assert(C == 3 || C == 16, "feature grids of 3 or 16 channels");
  constexpr bool REC = MODE == kModeRec || MODE == kModeRecTsdf;
  constexpr bool TRAIN = MODE != kModeBwd;
  __shared__ __align__(16) float s_head[3 * C];
  load_head<C>(p.head, s_head);
  const RenderSmem sm = render_smem(s_render, MODE, p.cap, false);
  const int lane = lane_id();
  const int Smax = p.sp.S;
  // a segment table covers rays [ray_begin[0], total): a sub-table of
  // consecutive segments is a group of targets
  const long it0 = REC ? (long)__ldg(p.k_begin) : (p.nseg > 0 ? (long)__ldg(p.seg_begin) : 0);
  const long it1 = REC ? (long)__ldg(p.k_end) : p.R;
  __shared__ int s_taken;
  if (!REC) {
    if (threadIdx.x == 0) s_taken = 0;
    __syncthreads();
  }
  for (long it = REC ? it0 + (((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) : take_ray(s_taken, it0); it < it1;
       it = REC ? it + (((long)gridDim.x * blockDim.x) >> 5) : take_ray(s_taken, it0)) {
    const long r = REC ? (long)__ldg(p.hit_ray + it) : it;
    int b, S, sgm;
    ray_frame(p, r, b, S, sgm);
    const int done = sample_and_sort<false>(p, r, b, S, sm);
    if (done == 0) {
      if (REC && lane == 0) p.ray_nrec[it] = 0;  // no sample: no record
      if (MODE == kModeBwd && p.grad_sigma) {
        for (int i = lane; i < Smax; i += 32) {
          p.grad_sigma[(size_t)r * Smax + i] = 0.0f;
          for (int k = 0; k < 3; k++) p.grad_rgb[((size_t)r * Smax + i) * 3 + k] = 0.0f;
        }
      }
      if (TRAIN && lane == 0) {
        // no sample: zero outputs, loss of the target alone, no gradient
        float l = 0.0f;
        for (int k = 0; k < 3; k++) {
          const float t = __ldg(p.target_rgb + r * 3 + k);
          p.out_rgb[r * 3 + k] = 0.0f;
          l += t * t;
        }
        p.out_depth[r] = p.out_ws[r] = p.out_alpha[r] = 0.0f;
        if (p.out_loss) p.out_loss[r] = 0.5f * p.loss_scale * l;
      }
      __syncwarp();
      continue;
    }
    const RayGeom g = ray_geom(p, r, b);
    const long base = REC ? (long)__ldg(p.hit_slot + it) : 0;
    int nrec = 0;
    // the ray's blocks, front to back: totals of w*rgb (and, for the general
    // adjoint, w*z, w, w*alpha) in the scans' order
    float cf[3] = {0.0f, 0.0f, 0.0f}, cd = 0.0f, cw = 0.0f, ca = 0.0f;
    RayWalk wk{1.0f, -1, S};
    const int e0 = (S - done) >> 5;
    int e1 = e0;  // blocks [e0, e1) were evaluated
#pragma unroll 1
    for (; e1 * 32 < wk.end; e1++) {
      BlockEval v;
      const bool any = eval_block<C, PACKED, MODE == kModeRec ? 32 : 8>(p, g, S, e1, sm, s_head, wk, v);
      if (mode_keeps(MODE)) {
        const int i = e1 * 32 + lane;
        sm.k(kKeepW, i) = any ? v.w : 0.0f;
        sm.k(kKeepDl, i) = any && v.used ? v.dl : 0.0f;
        if (any) {
          sm.k(kKeepR, i) = v.rgb[0];
          sm.k(kKeepG, i) = v.rgb[1];
          sm.k(kKeepB, i) = v.rgb[2];
          sm.k(kKeepS01, i) = v.s01;
          sm.k(kKeepAl, i) = v.al;
          sm.k(kKeepTb, i) = v.used ? v.tb : 0.0f;
        }
      }
      if (!any) continue;
#pragma unroll
      for (int k = 0; k < 3; k++) cf[k] += warp_sum_scan_order(v.w * v.rgb[k]);
      if (TRAIN) {
        // the loss reads only the colour: depth, weight sum and alpha sum
        // are outputs alone, summed as the forward kernel sums them
        if (v.used) {
          cd += v.w * v.z;
          cw += v.w;
          ca += v.w * v.al;
        }
      } else {
        cd += warp_sum_scan_order(v.w * v.z);
        cw += warp_sum_scan_order(v.w);
        ca += warp_sum_scan_order(v.w * v.al);
      }
      if (MODE == kModeRec) emit_records<false>(p, b, base, v.used, v.i0, v.f, v.w, 0.0f, nrec);
    }
    float gc[3] = {0.0f, 0.0f, 0.0f}, gd = 0.0f, gws = 0.0f, ga = 0.0f;
    if (TRAIN) {
      cd = warp_sum(cd);
      cw = warp_sum(cw);
      ca = warp_sum(ca);
      // forward outputs = the totals; upstream gradient of the per-ray loss
      float l = 0.0f;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const float d = cf[k] - __ldg(p.target_rgb + r * 3 + k);
        gc[k] = p.loss_scale * d;
        l += d * d;
      }
      if (lane == 0) {
        p.out_rgb[r * 3 + 0] = cf[0];
        p.out_rgb[r * 3 + 1] = cf[1];
        p.out_rgb[r * 3 + 2] = cf[2];
        p.out_depth[r] = cd;
        p.out_ws[r] = cw;
        p.out_alpha[r] = ca;
        if (p.out_loss) p.out_loss[r] = 0.5f * p.loss_scale * l;
      }
    } else {
      if (p.g_rgb) {
        gc[0] = __ldg(p.g_rgb + r * 3);
        gc[1] = __ldg(p.g_rgb + r * 3 + 1);
        gc[2] = __ldg(p.g_rgb + r * 3 + 2);
      }
      gd = p.g_depth ? __ldg(p.g_depth + r) : 0.0f;
      gws = p.g_ws ? __ldg(p.g_ws + r) : 0.0f;
      ga = p.g_alpha ? __ldg(p.g_alpha + r) : 0.0f;
    }
    if (REC && lane < C) p.ray_g[it * C + lane] = head_grad<C>(p, lane, gc);
    if constexpr (mode_keeps(MODE)) {
      // exact adjoint per sorted position: d out / d sigma_i = delta_i *
      // (T_{i+1} v_i - sum_{j>i} w_j v_j) (v = rgb, z, 1; 2 alpha T_{i+1} for
      // the alpha sum); d out / d rgb_i = w_i
      float rf[3] = {0.0f, 0.0f, 0.0f}, rd = 0.0f, rw = 0.0f, ra = 0.0f;  // running totals
      const float dsdt_k = -p.dk * p.inv_s;
      float G[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (mode_scatters(MODE) && p.grad_feat) {
        if constexpr (C == 16) {
#pragma unroll
          for (int q = 0; q < 4; q++) G[q] = head_grad<C>(p, 4 * (lane & 3) + q, gc);
        } else {
          if (lane < 24) G[0] = head_grad<C>(p, lane % 3, gc);
        }
      }
#pragma unroll 1
      for (int e = e0; e < e1; e++) {
        const int i = e * 32 + lane;
        const float z = i < S ? sm.z[i] : -1.0f;
        const float w = sm.k(kKeepW, i);
        const bool used = z >= 0.0f && i < wk.end;
        float gsig = 0.0f, s01 = 0.0f;
        if (__any_sync(SG_FULL, used)) {
          const float al = sm.k(kKeepAl, i);
          const float rgb[3] = {sm.k(kKeepR, i), sm.k(kKeepG, i), sm.k(kKeepB, i)};
          const float Ta = sm.k(kKeepTb, i) * (1.0f - al);
          s01 = sm.k(kKeepS01, i);
          float acc = 0.0f;
          if (!TRAIN) {
            const float vd = warp_incl_scan_f(w * z), vw = warp_incl_scan_f(w), va = warp_incl_scan_f(w * al);
            acc = gws * (Ta - (cw - (rw + vw))) + gd * (Ta * z - (cd - (rd + vd))) +
                  ga * (2.0f * al * Ta - (ca - (ra + va)));
            rd += __shfl_sync(SG_FULL, vd, 31);
            rw += __shfl_sync(SG_FULL, vw, 31);
            ra += __shfl_sync(SG_FULL, va, 31);
          }
#pragma unroll
          for (int k = 0; k < 3; k++) {
            const float v = warp_incl_scan_f(w * rgb[k]);
            acc += gc[k] * (Ta * rgb[k] - (cf[k] - (rf[k] + v)));
            rf[k] += __shfl_sync(SG_FULL, v, 31);
          }
          if (used) gsig = sm.k(kKeepDl, i) * acc;
        }
        if (MODE == kModeBwd && p.grad_sigma && i < Smax) {
          p.grad_sigma[(size_t)r * Smax + i] = gsig;
#pragma unroll
          for (int k = 0; k < 3; k++) p.grad_rgb[((size_t)r * Smax + i) * 3 + k] = used ? w * gc[k] : 0.0f;
        }
        const float gt = gsig * (s01 * (1.0f - s01) * dsdt_k);
        if (MODE == kModeRecTsdf) {
          int i0[3] = {0, 0, 0};
          float f[3] = {0.0f, 0.0f, 0.0f};
          if (used) feat_cell(p, g, z, i0, f);
          emit_records<true>(p, b, base, used, i0, f, w, gt, nrec);
        } else if (p.grad_feat || p.grad_tsdf) {
          // scatter into the grids, samples in sorted order
          int i0[3] = {0, 0, 0};
          float f[3] = {0.0f, 0.0f, 0.0f};
          if (used) feat_cell(p, g, z, i0, f);
          if (p.shared) {
            if (p.grad_feat && p.grad_tsdf) scatter_block<C, true, true>(p, b, sm, e, used, i0, f, w, gt, G);
            else if (p.grad_feat) scatter_block<C, true, false>(p, b, sm, e, used, i0, f, w, gt, G);
            else scatter_block<C, false, true>(p, b, sm, e, used, i0, f, w, gt, G);
          } else {
            if (p.grad_feat) scatter_block<C, true, false>(p, b, sm, e, used, i0, f, w, gt, G);
            if (p.grad_tsdf) {
              if (used) {
                float pt[3];
                ray_point(g, z, pt);
                tap_frac(g.bmin, g.vs, g.inv_vs, pt, i0, f);
              }
              scatter_block<C, false, true>(p, b, sm, e, used, i0, f, w, gt, G);
            }
          }
        }
      }
      if (MODE == kModeBwd && p.grad_sigma) {
        // positions of blocks that were not evaluated: no gradient
        for (int i = lane; i < Smax; i += 32) {
          if (i >= e0 * 32 && i < e1 * 32) continue;
          p.grad_sigma[(size_t)r * Smax + i] = 0.0f;
          for (int k = 0; k < 3; k++) p.grad_rgb[((size_t)r * Smax + i) * 3 + k] = 0.0f;
        }
      }
    }
    if (REC && lane == 0) {
      // the ray's records within the slot capacity
      const long room = p.rec_cap - base;
      p.ray_nrec[it] = (int)(room <= 0 ? 0 : (nrec < room ? nrec : room));
    }
    __syncwarp();
  }
}

static int render_grid(long R) {
  long g = (R * 32 + 255) / 256;
  const long cap = (long)num_sms() * tune(SG_TUNE_RENDER_WARPS);
  return (int)(g < cap ? g : cap);
}

// Dynamic shared memory of a kernel (8 warps); above 48 KB it is opted into.
template <typename K>
static int render_smem_bytes(K kernel, int mode, int cap, bool ids, size_t &bytes) {
  bytes = (size_t)8 * render_warp_words(mode, cap, ids) * sizeof(float);
  if (bytes > 48 * 1024 &&
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess)
    return SG_ERR_CUDA;
  return SG_OK;
}

template <int C, int MODE, bool PACKED>
static int launch_bwd(const RenderParams &p, int g, sg_stream_t stream) {
  size_t bytes;
  const int rc = render_smem_bytes(render_bwd_kernel<C, MODE, PACKED>, MODE, p.cap, false, bytes);
  if (rc != SG_OK) return rc;
  render_bwd_kernel<C, MODE, PACKED><<<g, 256, bytes, stream>>>(p);
  return SG_OK;
}

template <int C, bool IDS, bool PACKED>
static int launch_fwd(const RenderParams &p, int g, sg_stream_t stream) {
  size_t bytes;
  const int rc = render_smem_bytes(render_fwd_kernel<C, IDS, PACKED>, kModeFwd, p.cap, IDS, bytes);
  if (rc != SG_OK) return rc;
  render_fwd_kernel<C, IDS, PACKED><<<g, 256, bytes, stream>>>(p);
  return SG_OK;
}

template <int C, bool PACKED>
static int launch_render(const RenderParams &p, int mode, int g, sg_stream_t stream) {
  int rc;
  if (mode == kModeFwd) rc = p.out_z ? launch_fwd<C, true, PACKED>(p, g, stream) : launch_fwd<C, false, PACKED>(p, g, stream);
  else if (mode == kModeBwd) rc = launch_bwd<C, kModeBwd, PACKED>(p, g, stream);
  else if (mode == kModeTrain) rc = launch_bwd<C, kModeTrain, PACKED>(p, g, stream);
  else if (p.grad_tsdf) rc = launch_bwd<C, kModeRecTsdf, PACKED>(p, g, stream);
  else rc = launch_bwd<C, kModeRec, PACKED>(p, g, stream);
  if (rc != SG_OK) return rc;
  SG_LAUNCH_CHECK();
  return SG_OK;
}

// mode: kModeFwd, kModeBwd, kModeTrain, or kModeRec (records; with the TSDF
// gradient when p.grad_tsdf is set)
static int launch_render_c(RenderParams p, int C, int mode, sg_stream_t stream) {
  if (p.R <= 0) return SG_OK;
  const int S = p.sp.S;
  if (S > 128) return SG_ERR_UNSUPPORTED;
  p.cap = S <= 32 ? 32 : (S <= 64 ? 64 : 128);
  const int g = render_grid(p.R);
  if (C == 3) return p.packed ? launch_render<3, true>(p, mode, g, stream) : launch_render<3, false>(p, mode, g, stream);
  if (C == 16)
    return p.packed ? launch_render<16, true>(p, mode, g, stream) : launch_render<16, false>(p, mode, g, stream);
  return SG_ERR_UNSUPPORTED;
}

// log2 of a brick edge that is a power of two, else -1
static int log2_exact(int rate) {
  for (int k = 0; k < 31; k++)
    if (rate == (1 << k)) return k;
  return -1;
}

// Packed fields need one geometry for both grids, bricks of a power of two,
// and the tree's node list and brick map.
static bool packable(const SgTree *tree, const SgRenderArgs *a, const RenderParams &p) {
  return p.shared && log2_exact(tree->rate) >= 0 && tree->Db == a->D && tree->Db == tree->Dt * tree->rate &&
         tree->brick_node && (a->C == 3 || a->C == 16);
}

// packed (may be null) into p, checked
static int use_packed(const SgTree *tree, const SgRenderArgs *a, const float *packed, RenderParams &p) {
  if (!packed) return SG_OK;
  if (((uintptr_t)packed) % 16 != 0) return SG_ERR_INVALID_ARG;
  if (!packable(tree, a, p)) return SG_ERR_UNSUPPORTED;
  p.packed = reinterpret_cast<const float4 *>(packed);
  p.rate_shift = log2_exact(tree->rate);
  return SG_OK;
}

// RenderParams of the batched entry points.
static int segment_params(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *a, RenderParams &p) {
  if (!tree || !seg || !a) return SG_ERR_INVALID_ARG;
  if (seg->count <= 0 || seg->total < 0 || !seg->ray_begin || !seg->frame || !seg->samples)
    return SG_ERR_INVALID_ARG;
  if (!a->hit_idx || !a->hit_t0 || !a->hit_t1 || !a->valid_len || !a->tsdf || !a->feat || !a->feat_bbox ||
      !a->feat_vs)
    return SG_ERR_INVALID_ARG;
  // the render reads ray buffers (for camera segments: sg_segment_rays)
  if (!a->ori || !a->dir) return SG_ERR_INVALID_ARG;
  if (a->W <= 0 || a->S <= 0 || a->D <= 0 || a->Df <= 0 || tree->B <= 0 || a->sdf_s == 0.0f)
    return SG_ERR_INVALID_ARG;
  if (!a->head && a->C != 3) return SG_ERR_INVALID_ARG;
  p = RenderParams{};
  p.sp = SampleParams{*tree, a->hit_idx, a->hit_t0, a->hit_t1, a->rands, a->valid_len, 1, a->W, a->S, 2, 0,
                      nullptr, nullptr, a->rand_seed};
  p.hit_count = a->hit_count;
  p.rand_const = a->rand_const;
  p.R = seg->total;
  p.nseg = seg->count;
  p.seg_begin = seg->ray_begin;
  p.seg_frame = seg->frame;
  p.seg_samples = seg->samples;
  p.ori = a->ori;
  p.dir = a->dir;
  p.tsdf = a->tsdf;
  p.D = a->D;
  p.sdf_scale = a->sdf_scale;
  p.sdf_s = a->sdf_s;
  p.feat = a->feat;
  p.Df = a->Df;
  p.fbbox = a->feat_bbox;
  p.fvs = a->feat_vs;
  p.head = a->head;
  p.t_thres = a->t_thres;
  p.dk = a->sdf_scale / a->sdf_s;
  p.inv_s = 1.0f / a->sdf_s;
  p.shared = a->Df == a->D && a->feat_bbox == tree->vol_bbox && a->feat_vs == tree->voxel_size;
  // float4 loads of the feature rows and of the colour head's rows
  if (a->C == 16 && (((uintptr_t)a->feat) % 16 != 0 || ((uintptr_t)a->head) % 16 != 0)) return SG_ERR_INVALID_ARG;
  return SG_OK;
}

}  // namespace sg

using namespace sg;

extern "C" int sg_render_fused(const SgTree *tree, const int *hit_idx, const float *hit_t0, const float *hit_t1,
                               const int *hit_count, int N, int W, const float *rands, float rand_const,
                               const float *valid_len, int S, int num_levels, int start_level,
                               const float *ori, const float *dir, const float *tsdf, int D, float sdf_scale,
                               float sdf_s, const float *color_grid, int Dc, const float *color_bbox,
                               const float *color_vs, float t_thres, float *out_rgb, float *out_depth,
                               float *out_ws, float *out_alpha, float *out_z, int *out_node,
                               sg_stream_t stream) {
  if (!tree || !hit_idx || !hit_t0 || !hit_t1 || !valid_len || !ori || !dir || !tsdf || !color_grid ||
      !color_bbox || !color_vs || !out_rgb || !out_depth || !out_ws || !out_alpha)
    return SG_ERR_INVALID_ARG;
  if ((out_z == nullptr) != (out_node == nullptr)) return SG_ERR_INVALID_ARG;
  if (N <= 0 || W <= 0 || S <= 0 || D <= 0 || Dc <= 0 || tree->B <= 0 || sdf_s == 0.0f)
    return SG_ERR_INVALID_ARG;
  RenderParams p{};
  p.sp = SampleParams{*tree, hit_idx, hit_t0, hit_t1, rands, valid_len, N, W, S, num_levels, start_level,
                      nullptr, nullptr, 0ull};
  p.hit_count = hit_count;
  p.rand_const = rand_const;
  p.R = (long)tree->B * N;
  p.nseg = 0;
  p.ori = ori;
  p.dir = dir;
  p.tsdf = tsdf;
  p.D = D;
  p.sdf_scale = sdf_scale;
  p.sdf_s = sdf_s;
  p.feat = color_grid;
  p.Df = Dc;
  p.fbbox = color_bbox;
  p.fvs = color_vs;
  p.head = nullptr;
  p.t_thres = t_thres;
  p.dk = sdf_scale / sdf_s;
  p.inv_s = 1.0f / sdf_s;
  p.shared = Dc == D && color_bbox == tree->vol_bbox && color_vs == tree->voxel_size;
  p.out_rgb = out_rgb;
  p.out_depth = out_depth;
  p.out_ws = out_ws;
  p.out_alpha = out_alpha;
  p.out_z = out_z;
  p.out_node = out_node;
  return launch_render_c(p, 3, kModeFwd, stream);
}

extern "C" int sg_pack_fields(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args, float *packed,
                              sg_stream_t stream) {
  RenderParams p;
  int rc = segment_params(tree, seg, args, p);
  if (rc != SG_OK) return rc;
  if (!packed) return SG_ERR_INVALID_ARG;
  rc = use_packed(tree, args, packed, p);
  if (rc != SG_OK) return rc;
  if (!tree->counts || !tree->top_key) return SG_ERR_INVALID_ARG;
  float4 *out = reinterpret_cast<float4 *>(packed);
  const int g = num_sms() * 8;
  if (args->C == 3) pack_fields_kernel<3><<<g, 256, 0, stream>>>(*tree, args->feat, args->head, args->tsdf, args->D, out);
  else pack_fields_kernel<16><<<g, 256, 0, stream>>>(*tree, args->feat, args->head, args->tsdf, args->D, out);
  SG_LAUNCH_CHECK();
  return SG_OK;
}

extern "C" int sg_render_packed_fwd(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                    const float *packed, float *out_rgb, float *out_depth, float *out_ws, float *out_alpha,
                                      float *out_z, int *out_node, sg_stream_t stream) {
  RenderParams p;
  int rc = segment_params(tree, seg, args, p);
  if (rc != SG_OK) return rc;
  if (!out_rgb || !out_depth || !out_ws || !out_alpha || (out_z == nullptr) != (out_node == nullptr))
    return SG_ERR_INVALID_ARG;
  rc = use_packed(tree, args, packed, p);
  if (rc != SG_OK) return rc;
  p.out_rgb = out_rgb;
  p.out_depth = out_depth;
  p.out_ws = out_ws;
  p.out_alpha = out_alpha;
  p.out_z = out_z;
  p.out_node = out_node;
  return launch_render_c(p, args->C, kModeFwd, stream);
}

extern "C" int sg_render_segments_fwd(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                      float *out_rgb, float *out_depth, float *out_ws, float *out_alpha,
                                      float *out_z, int *out_node, sg_stream_t stream) {
  return sg_render_packed_fwd(tree, seg, args, nullptr, out_rgb, out_depth, out_ws, out_alpha, out_z, out_node,
                              stream);
}

extern "C" int sg_render_packed_bwd(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                    const float *packed, const float *g_rgb, const float *g_depth,
                                    const float *g_ws, const float *g_alpha, float *grad_feat, float *grad_tsdf,
                                    float *grad_sigma, float *grad_rgb, sg_stream_t stream) {
  RenderParams p;
  int rc = segment_params(tree, seg, args, p);
  if (rc != SG_OK) return rc;
  if ((grad_sigma == nullptr) != (grad_rgb == nullptr)) return SG_ERR_INVALID_ARG;
  rc = use_packed(tree, args, packed, p);
  if (rc != SG_OK) return rc;
  p.g_rgb = g_rgb;
  p.g_depth = g_depth;
  p.g_ws = g_ws;
  p.g_alpha = g_alpha;
  p.grad_feat = grad_feat;
  p.grad_tsdf = grad_tsdf;
  p.grad_sigma = grad_sigma;
  p.grad_rgb = grad_rgb;
  return launch_render_c(p, args->C, kModeBwd, stream);
}

extern "C" int sg_render_segments_bwd(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                      const float *g_rgb, const float *g_depth, const float *g_ws,
                                      const float *g_alpha, float *grad_feat, float *grad_tsdf,
                                      float *grad_sigma, float *grad_rgb, sg_stream_t stream) {
  return sg_render_packed_bwd(tree, seg, args, nullptr, g_rgb, g_depth, g_ws, g_alpha, grad_feat, grad_tsdf,
                              grad_sigma, grad_rgb, stream);
}

extern "C" int sg_render_packed_train(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                      const float *packed, const float *target_rgb, float loss_scale,
                                      float *out_rgb, float *out_depth, float *out_ws, float *out_alpha,
                                      float *out_loss, float *grad_feat, float *grad_tsdf, sg_stream_t stream) {
  RenderParams p;
  int rc = segment_params(tree, seg, args, p);
  if (rc != SG_OK) return rc;
  if (!target_rgb || !out_rgb || !out_depth || !out_ws || !out_alpha) return SG_ERR_INVALID_ARG;
  rc = use_packed(tree, args, packed, p);
  if (rc != SG_OK) return rc;
  p.target_rgb = target_rgb;
  p.loss_scale = loss_scale;
  p.out_loss = out_loss;
  p.out_rgb = out_rgb;
  p.out_depth = out_depth;
  p.out_ws = out_ws;
  p.out_alpha = out_alpha;
  p.grad_feat = grad_feat;
  p.grad_tsdf = grad_tsdf;
  return launch_render_c(p, args->C, kModeTrain, stream);
}

extern "C" int sg_render_segments_train(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                        const float *target_rgb, float loss_scale, float *out_rgb,
                                        float *out_depth, float *out_ws, float *out_alpha, float *out_loss,
                                        float *grad_feat, float *grad_tsdf, sg_stream_t stream) {
  return sg_render_packed_train(tree, seg, args, nullptr, target_rgb, loss_scale, out_rgb, out_depth, out_ws,
                                out_alpha, out_loss, grad_feat, grad_tsdf, stream);
}

// ---------------------------------------------------------------------------
// training step with the deterministic gradient reduction (scatter.cu)
// ---------------------------------------------------------------------------
extern "C" size_t sg_train_det_workspace_bytes(long long R, int nseg, int C, long long capacity) {
  if (R < 0 || nseg < 0 || C <= 0 || capacity < 0) return 0;
  return det_layout((long)R, nseg, C, (long)(capacity > 0 ? capacity : 1), nullptr, nullptr);
}

extern "C" int sg_render_packed_train_det(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                          const float *packed, int ngroups, const int *groups, const int *group_S,
                                          const float *target_rgb, float loss_scale, float *out_rgb,
                                          float *out_depth, float *out_ws, float *out_alpha, float *out_loss,
                                          float *grad_feat, float *grad_tsdf, void *workspace,
                                          size_t workspace_bytes, long long capacity, SgStatus *status,
                                          sg_stream_t stream) {
  RenderParams p;
  int rc = segment_params(tree, seg, args, p);
  if (rc != SG_OK) return rc;
  if (!target_rgb || !out_rgb || !out_depth || !out_ws || !out_alpha || !grad_feat || !workspace) return SG_ERR_INVALID_ARG;
  if (ngroups <= 0 || !groups || !group_S || groups[0] != 0 || groups[ngroups] != seg->count) return SG_ERR_INVALID_ARG;
  for (int g = 0; g < ngroups; g++)
    if (groups[g + 1] <= groups[g] || group_S[g] <= 0 || group_S[g] > args->S) return SG_ERR_INVALID_ARG;
  if (capacity <= 0 || capacity >= (1ll << 31)) return SG_ERR_INVALID_ARG;
  rc = use_packed(tree, args, packed, p);
  if (rc != SG_OK) return rc;
  if (grad_tsdf && !p.shared) return SG_ERR_UNSUPPORTED;
  if (args->C != 3 && args->C != 16) return SG_ERR_UNSUPPORTED;
  if (!record_keys_fit(tree->B, args->Df)) return SG_ERR_UNSUPPORTED;
  const long R = seg->total;
  if (workspace_bytes < det_layout(R, seg->count, args->C, (long)capacity, nullptr, nullptr))
    return SG_ERR_INVALID_ARG;
  if (((uintptr_t)workspace) % 256 != 0) return SG_ERR_INVALID_ARG;
  if (R == 0) return SG_OK;
  if (!args->hit_count) return SG_ERR_INVALID_ARG;  // the ray scan reads the hit counts
  DetWork w;
  det_layout(R, seg->count, args->C, (long)capacity, (char *)workspace, &w);
  DetTrainOut o{target_rgb, loss_scale, out_rgb, out_depth, out_ws, out_alpha, out_loss};
  rc = launch_det_prepare(w, *seg, args->S, args->hit_count, R, (long)capacity, o, status, stream);
  if (rc != SG_OK) return rc;
  p.target_rgb = target_rgb;
  p.loss_scale = loss_scale;
  p.out_loss = out_loss;
  p.out_rgb = out_rgb;
  p.out_depth = out_depth;
  p.out_ws = out_ws;
  p.out_alpha = out_alpha;
  p.grad_feat = grad_feat;
  p.grad_tsdf = grad_tsdf;
  p.hit_ray = w.hit_ray;
  p.hit_slot = w.hit_slot;
  p.ray_nrec = w.ray_nrec;
  p.rec_key = w.rec_key;
  p.rec = w.rec;
  p.rec_t = w.rec_t;
  p.ray_g = w.ray_g;
  p.rec_cap = (long)capacity;
  p.keys = make_record_keys(tree->B, args->Df);
  for (int g = 0; g < ngroups; g++) {
    RenderParams pg = p;
    pg.sp.S = group_S[g];
    pg.k_begin = w.seg_hit + groups[g];
    pg.k_end = w.seg_hit + groups[g + 1];
    // the group's count of rays with hits is on the device: the grid is the
    // persistent cap, its warps striding over the compact range
    rc = launch_render_c(pg, args->C, kModeRec, stream);
    if (rc != SG_OK) return rc;
  }
  return launch_det_reduce(w, p.keys, *seg, args->S, R, (long)capacity, args->C, grad_feat, grad_tsdf, stream);
}

extern "C" int sg_render_segments_train_det(const SgTree *tree, const SgRaySegments *seg, const SgRenderArgs *args,
                                            int ngroups, const int *groups, const int *group_S,
                                            const float *target_rgb, float loss_scale, float *out_rgb,
                                            float *out_depth, float *out_ws, float *out_alpha, float *out_loss,
                                            float *grad_feat, float *grad_tsdf, void *workspace,
                                            size_t workspace_bytes, long long capacity, SgStatus *status,
                                            sg_stream_t stream) {
  return sg_render_packed_train_det(tree, seg, args, nullptr, ngroups, groups, group_S, target_rgb, loss_scale,
                                    out_rgb, out_depth, out_ws, out_alpha, out_loss, grad_feat, grad_tsdf, workspace,
                                    workspace_bytes, capacity, status, stream);
}
