// project.cu -- projection of sample points into the source views and the
// bilinear gather of per-view 2D feature maps at the projections (the step
// after sampling in SRONet), on sm_103a.
//
// sg_project_sampled_xyz replaces project_xyz (c_lib/VoxelEncoding/src/
// sampling_kernel.cu:55-159) behind MultiLayerOctree::project_sampled_xyz
// (:1333-1381): every (frame, view, ray, sample) is projected, optionally
// with the eight corners of the sample's node; one thread per item, the
// -1 of samples without a node written by the same pass (the reference
// pre-fills the whole output with torch::full first).
//
// sg_project_gather replaces proj_persp (utils_render/utils_render.py:
// 380-414) and the four F.grid_sample calls plus the clamped depth
// difference of BasicRenNet.forward_sample_feature (SRONet/BasicRenNet.py:
// 245-259): one thread per (view image, point) projects the point, writes
// the projection outputs that are asked for, and gathers up to four feature
// maps bilinearly (align_corners=True, zero padding) straight into the
// channel-last [view image, point, C] layout the reference produces with
// permute + contiguous.  Maps are read through strides, so NCHW and
// channels-last tensors both work.  Maps whose channels are contiguous are
// gathered by lane groups, texel rows and output rows in vectors of 16, 8 or
// 4 bytes (gather_rows); maps of up to 4 channels and maps of any other
// layout by a thread per item (gather_map).
//
// sg_channels_last writes a map into channels-last order, for callers that
// gather many points from a map in another layout.
#include <climits>
#include <type_traits>

#include "common.cuh"

namespace sg {

// ---------------------------------------------------------------------------
// project_xyz
// ---------------------------------------------------------------------------
struct ProjSampledParams {
  SgTree t;
  const float *ori, *dir, *z;
  const int *idx;
  const float *K, *RT;
  int B, Nv, N, S;
  float cw, ch;  // ori_w / 2, ori_h / 2
  int corners;
  float *xy, *pz;
};

// (x - c) / c as the reference evaluates it (in double precision, stored as
// float; c = size / 2 is exact): the difference as an exact float pair
// (two_sum), the quotient of its leading part, and one correction from the
// exact remainder of that quotient.  Equal to the reference's value except
// where the exact quotient lies within about 2^-29 ulp of a rounding
// boundary; with c a power of two the difference of two floats is exact
// after scaling and the result is the reference's exactly.
__device__ __forceinline__ float grid_coord(float x, float c) {
  float dh, dl;
  two_sum(x, -c, dh, dl);
  const float q = dh / c;
  const float r = __fmaf_rn(-q, c, dh);  // dh - q c, exact
  return q + (r + dl) / c;
}

// camera point and normalised pixel of world point p in view (K, RT): the
// reference's expressions with the operand order nvcc gives them
// (project_xyz, sampling_kernel.cu:103-116)
__device__ __forceinline__ void project_point(const float *__restrict__ K, const float *__restrict__ P, float px,
                                              float py, float pz, float cw, float ch, float &gx, float &gy,
                                              float &cz) {
  const float cx = __fmaf_rn(P[2], pz, __fmaf_rn(P[0], px, P[1] * py)) + P[3];
  const float cy = __fmaf_rn(P[6], pz, __fmaf_rn(P[4], px, P[5] * py)) + P[7];
  cz = __fmaf_rn(P[10], pz, __fmaf_rn(P[8], px, P[9] * py)) + P[11];
  const float ux = dot3c(K[0], K[1], K[2], cx, cy, cz);
  const float uy = dot3c(K[3], K[4], K[5], cx, cy, cz);
  const float uz = dot3c(K[6], K[7], K[8], cx, cy, cz);
  gx = grid_coord(ux / uz, cw);
  gy = grid_coord(uy / uz, ch);
}

// Centre and edge of node g (a top brick or a fine voxel of the tree), as
// OcTree::calculate_xyz_corners places it (octree.h:109-129); false when g is
// not a node.
__device__ __forceinline__ bool node_centre(const SgTree &t, int g, float c[3], float &vs) {
  int ix, iy, iz, b, size;
  if (g >= t.base_top && g < t.base_top + t.counts[0]) {
    const long key = t.top_key[g - t.base_top];
    const long vt = (long)t.Dt * t.Dt * t.Dt;
    b = (int)(key / vt);
    const long l = key - (long)b * vt;
    ix = (int)(l / ((long)t.Dt * t.Dt)), iy = (int)((l / t.Dt) % t.Dt), iz = (int)(l % t.Dt);
    size = t.Db / t.Dt;
  } else if (g >= t.base_bot && g < t.base_bot + t.counts[1]) {
    const long key = t.bot_key[g - t.base_bot];
    const long vb = (long)t.Db * t.Db * t.Db;
    b = (int)(key / vb);
    const long l = key - (long)b * vb;
    ix = (int)(l / ((long)t.Db * t.Db)), iy = (int)((l / t.Db) % t.Db), iz = (int)(l % t.Db);
    size = 1;
  } else {
    return false;
  }
  const LevelGeom lg = level_geom(t.voxel_size[b], size);
  const float *bb = t.vol_bbox + 6 * b;
  c[0] = node_coord(lg, bb[0], ix);
  c[1] = node_coord(lg, bb[2], iy);
  c[2] = node_coord(lg, bb[4], iz);
  vs = lg.vs;
  return true;
}

__global__ void __launch_bounds__(256) project_sampled_kernel(ProjSampledParams p) {
  const long total = (long)p.B * p.Nv * p.N * p.S;
  const int per = p.corners ? 9 : 1;
  for (long k = (long)blockIdx.x * blockDim.x + threadIdx.x; k < total; k += (long)gridDim.x * blockDim.x) {
    const long rs = k % ((long)p.N * p.S);  // ray * S + sample
    const long bv = k / ((long)p.N * p.S);  // frame * Nv + view
    const int b = (int)(bv / p.Nv);
    const long si = (long)b * p.N * p.S + rs;
    float *xy = p.xy + k * (2 * per);
    float *oz = p.pz + k * per;
    const int id = __ldg(p.idx + si);
    if (id == -1) {  // no node: the reference's -1 fill stays
      for (int i = 0; i < per; i++) {
        xy[2 * i] = -1.0f;
        xy[2 * i + 1] = -1.0f;
        oz[i] = -1.0f;
      }
      continue;
    }
    const long r = rs / p.S;
    const float zs = __ldg(p.z + si);
    const float *o = p.ori + ((long)b * p.N + r) * 3, *d = p.dir + ((long)b * p.N + r) * 3;
    const float px = __fmaf_rn(__ldg(d), zs, __ldg(o));
    const float py = __fmaf_rn(__ldg(d + 1), zs, __ldg(o + 1));
    const float pz = __fmaf_rn(__ldg(d + 2), zs, __ldg(o + 2));
    const float *K = p.K + bv * 9, *P = p.RT + bv * 12;
    float gx, gy, cz;
    project_point(K, P, px, py, pz, p.cw, p.ch, gx, gy, cz);
    xy[0] = gx;
    xy[1] = gy;
    oz[0] = cz;
    if (!p.corners) continue;
    float c[3], vs;
    if (!node_centre(p.t, id, c, vs)) {  // not a node of this tree
      for (int i = 1; i < 9; i++) {
        xy[2 * i] = -1.0f;
        xy[2 * i + 1] = -1.0f;
        oz[i] = -1.0f;
      }
      continue;
    }
    const float h = vs / 2.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float qx = c[0] + ((i & 4) ? h : -h), qy = c[1] + ((i & 2) ? h : -h), qz = c[2] + ((i & 1) ? h : -h);
      project_point(K, P, qx, qy, qz, p.cw, p.ch, gx, gy, cz);
      xy[2 * (i + 1)] = gx;
      xy[2 * (i + 1) + 1] = gy;
      oz[i + 1] = cz;
    }
  }
}

// ---------------------------------------------------------------------------
// proj_persp + grid_sample
// ---------------------------------------------------------------------------
constexpr int kMaxMaps = 4;

struct GatherMap {
  const float *data;
  long sn, sc, sy, sx;  // element strides of [view image, channel, y, x]
  int C, H, W;
  int rows;             // floats per vector of the row gather (4, 2, 1); 0: a thread per item
  float *out;           // [view image, N, C]
};

struct ProjGatherParams {
  const float *gin, *din;  // given grids [BV, N, 2] and depths [BV, N] (gin null: project pts)
  const float *pts;
  long pb, pa, pn;  // element strides of points [batch, axis, point]
  int pt_div;       // point batch = view image / pt_div
  const float *pdep;
  long db, dn;      // p_depths [batch, 1, point] strides (pdep may be null)
  const float *K, *R, *T;
  int BV, N;
  float depth_thres, min_d, max_d, half_res;
  float *ori_pts, *grids, *depth;  // [BV, 3, N], [BV, 2, N], [BV, 1, N]; each may be null
  GatherMap maps[kMaxMaps];
  int n_maps;
  int psdf_map;                    // map holding depth for psdf (-1: none)
  float psdf_clip, psdf_scale;
  float *psdf;                     // [BV, N, 1]
};

// Bilinear footprint of a grid point on an H x W image (F.grid_sample,
// align_corners=True, zero padding): the nw corner (x0, y0), the weights of
// the corners nw, ne, sw, se, and a 4-bit mask of the corners inside the
// image (NaN or far-out coordinates have none).
struct Foot {
  float w[4];
  int x0, y0, mask;
};

__device__ __forceinline__ Foot footprint(int H, int W, float gx, float gy) {
  Foot f;
  const float ix = ((gx + 1.0f) / 2.0f) * (float)(W - 1);
  const float iy = ((gy + 1.0f) / 2.0f) * (float)(H - 1);
  const float x0 = floorf(ix), y0 = floorf(iy);
  const float x1 = x0 + 1.0f, y1 = y0 + 1.0f;
  f.w[0] = (x1 - ix) * (y1 - iy);
  f.w[1] = (ix - x0) * (y1 - iy);
  f.w[2] = (x1 - ix) * (iy - y0);
  f.w[3] = (ix - x0) * (iy - y0);
  const bool xa = x0 >= 0.0f && x0 <= (float)(W - 1), xb = x1 >= 0.0f && x1 <= (float)(W - 1);
  const bool ya = y0 >= 0.0f && y0 <= (float)(H - 1), yb = y1 >= 0.0f && y1 <= (float)(H - 1);
  f.mask = (xa && ya ? 1 : 0) | (xb && ya ? 2 : 0) | (xa && yb ? 4 : 0) | (xb && yb ? 8 : 0);
  f.x0 = f.mask ? (int)x0 : 0;  // in [-1, W - 1] when any corner is inside
  f.y0 = f.mask ? (int)y0 : 0;
  return f;
}

// element offset of corner i (nw, ne, sw, se) of footprint (x0, y0) in image img
__device__ __forceinline__ long corner_off(const GatherMap &m, int img, int x0, int y0, int i) {
  return (long)img * m.sn + (long)(y0 + (i >> 1)) * m.sy + (long)(x0 + (i & 1)) * m.sx;
}

// Per-item gather of NC channels of a map that is not read in lane groups, all
// their loads in flight together; the first channel's value is returned.
// off: element offset of the footprint's first corner in the first channel.
template <int NC, typename Off>
__device__ __forceinline__ float gather_channels(const GatherMap &m, Off off, float *out, const Foot &f) {
  const Off sx = (Off)m.sx, sy = (Off)m.sy, sc = (Off)m.sc;
  float v[NC][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float *at = m.data + (off + ((i & 2) ? sy : 0) + ((i & 1) ? sx : 0));
    const bool in = (f.mask >> i) & 1;
#pragma unroll
    for (int c = 0; c < NC; c++) {
      v[c][i] = 0.0f;
      if (in) v[c][i] = __ldg(at);
      at += sc;
    }
  }
  float a[NC];
#pragma unroll
  for (int c = 0; c < NC; c++) {
    a[c] = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; i++)
      if ((f.mask >> i) & 1) a[c] = __fmaf_rn(v[c][i], f.w[i], a[c]);
    __stcs(out + c, a[c]);
  }
  return a[0];
}

// Per-item gather of a whole map through its channel stride.  Returns channel 0.
template <bool SMALL>
__device__ __forceinline__ float gather_map(const GatherMap &m, int img, long k, const Foot &f) {
  using Off = typename std::conditional<SMALL, int, long>::type;
  float *out = m.out + k * m.C;
  Off off = (Off)img * (Off)m.sn + (Off)f.y0 * (Off)m.sy + (Off)f.x0 * (Off)m.sx;
  if (m.C == 1) return gather_channels<1>(m, off, out, f);
  if (m.C == 3) return gather_channels<3>(m, off, out, f);
  float first = 0.0f;
#pragma unroll 1
  for (int c = 0; c < m.C; c++) {
    const float v = gather_channels<1>(m, off, out + c, f);
    if (c == 0) first = v;
    off += (Off)m.sc;
  }
  return first;
}

// proj_persp for point n of view image img: writes the projection outputs
// that are asked for and returns the grid coordinates and depth.
__device__ __forceinline__ void persp_point(const ProjGatherParams &p, long img, long n, float &gx, float &gy,
                                           float &dep) {
  const long pb = img / p.pt_div;
  const float *pt = p.pts + pb * p.pb + n * p.pn;
  const float x = __ldg(pt), y = __ldg(pt + p.pa), z = __ldg(pt + 2 * p.pa);
  const float *R = p.R + img * 9, *T = p.T + img * 3, *K = p.K + img * 9;
  // pts = R @ points + T
  const float cx = __fmaf_rn(R[2], z, __fmaf_rn(R[1], y, R[0] * x)) + T[0];
  const float cy = __fmaf_rn(R[5], z, __fmaf_rn(R[4], y, R[3] * x)) + T[1];
  const float cz = __fmaf_rn(R[8], z, __fmaf_rn(R[7], y, R[6] * x)) + T[2];
  const bool invalid = cz < p.depth_thres;
  bool invalid_d = false;
  if (p.pdep) {
    const float pd = __ldg(p.pdep + pb * p.db + n * p.dn);
    invalid_d = pd < p.min_d || pd > p.max_d;
  }
  const float dz = invalid ? 1.0f : cz;
  const float qx = cx / dz, qy = cy / dz, qz = cz / dz;
  const float sx = __fmaf_rn(K[2], qz, __fmaf_rn(K[1], qy, K[0] * qx));
  const float sy = __fmaf_rn(K[5], qz, __fmaf_rn(K[4], qy, K[3] * qx));
  gx = (sx - p.half_res) / p.half_res;
  gy = (sy - p.half_res) / p.half_res;
  if (invalid || invalid_d) gx = gy = -2.0f;
  dep = invalid_d ? -2.0f : cz;
  if (p.ori_pts) {
    p.ori_pts[(img * 3 + 0) * p.N + n] = cx;
    p.ori_pts[(img * 3 + 1) * p.N + n] = cy;
    p.ori_pts[(img * 3 + 2) * p.N + n] = cz;
  }
  if (p.grids) {
    p.grids[(img * 2 + 0) * p.N + n] = gx;
    p.grids[(img * 2 + 1) * p.N + n] = gy;
  }
  if (p.depth) p.depth[img * p.N + n] = dep;
}

// Footprints of a warp's 32 items, for the lane groups.
struct WarpFoot {
  float4 w;  // corner weights, 0 for corners outside the image
  int4 a;    // x0, y0, mask, image
};

// V consecutive floats, and their multiply-add by one weight in pairs
// (fma.rn.f32x2: the roundings of two fma.rn.f32).
__device__ __forceinline__ unsigned long long pair_of(float w) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(w));
  return r;
}
__device__ __forceinline__ unsigned long long fma_pair(unsigned long long x, unsigned long long w,
                                                       unsigned long long acc) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(w), "l"(acc));
  return r;
}
template <int V> struct FloatVec;
template <> struct FloatVec<1> {
  using Raw = float;
  using W = float;
  static __device__ __forceinline__ W weight(float w) { return w; }
  static __device__ __forceinline__ Raw zero() { return 0.0f; }
  static __device__ __forceinline__ Raw fma(Raw x, W w, Raw acc) { return __fmaf_rn(x, w, acc); }
};
template <> struct FloatVec<2> {
  using Raw = unsigned long long;
  using W = unsigned long long;
  static __device__ __forceinline__ W weight(float w) { return pair_of(w); }
  static __device__ __forceinline__ Raw zero() { return 0ull; }
  static __device__ __forceinline__ Raw fma(Raw x, W w, Raw acc) { return fma_pair(x, w, acc); }
};
template <> struct FloatVec<4> {
  using Raw = ulonglong2;
  using W = unsigned long long;
  static __device__ __forceinline__ W weight(float w) { return pair_of(w); }
  static __device__ __forceinline__ Raw zero() { return make_ulonglong2(0ull, 0ull); }
  static __device__ __forceinline__ Raw fma(Raw x, W w, Raw acc) {
    return make_ulonglong2(fma_pair(x.x, w, acc.x), fma_pair(x.y, w, acc.y));
  }
};

// Gather of one map with contiguous channels for the 32 items of a warp: lane
// groups of GW (8, or 4 and 2 where a row has no more vectors) take the items,
// kRowItems at a time, lane (group, q) the V-float vectors q, q + GW, ..., so
// each load reads whole vectors of one texel row and each store writes a
// contiguous part of the item's output row.  The items' footprints come from
// the warp's shared array.
//
// Bound by the L1 data path (four texel rows of 128 bytes an item: 82 % busy)
// and by issue, so the loop is kept short: 32-bit offsets where every map allows it (SMALL), two items per
// group with 8 loads in flight a lane, paired multiply-adds, and (WHOLE) no
// test per corner where every footprint of the warp lies wholly inside the
// image or wholly outside it: an item outside reads texel (0, 0)'s corners
// and writes zeros.  33.5 M items of 32 + 32 + 3 + 1 channels: 4.25 -> 3.26 ms
// (of it the projection alone 0.32, a 32-channel map 1.15, the depth map
// 0.17, the colours 0.31).
constexpr int kRowItems = 2;

template <int V, int GW, bool SMALL, bool WHOLE>
__device__ __forceinline__ void gather_rows(const GatherMap &m, long k0, long total, const WarpFoot *sf) {
  using T = FloatVec<V>;
  using Raw = typename T::Raw;
  using Off = typename std::conditional<SMALL, int, long>::type;
  const int lane = lane_id(), grp = lane / GW, q0 = lane % GW;
  constexpr int kGroups = 32 / GW;
  const int C = m.C;
  const int left = total - k0 < 32 ? (int)(total - k0) : 32;  // items past the end are the warp's last ones
  const float *const data = m.data + V * q0;
  float *out = m.out + k0 * C + (grp * C + V * q0);
  const Off sy = (Off)m.sy, sx = (Off)m.sx, sn = (Off)m.sn;
#pragma unroll 1
  for (int r = grp; r < left; r += kGroups * kRowItems, out += kGroups * kRowItems * C) {
    typename T::W w[kRowItems][4];
    int mask[kRowItems];
    const float *at[kRowItems][2];
#pragma unroll
    for (int u = 0; u < kRowItems; u++) {
      const int it = r + kGroups * u;
      const float4 ww = sf[it].w;
      const int4 a = sf[it].a;
      w[u][0] = T::weight(ww.x);
      w[u][1] = T::weight(ww.y);
      w[u][2] = T::weight(ww.z);
      w[u][3] = T::weight(ww.w);
      mask[u] = a.z;
      at[u][0] = data + ((Off)a.w * sn + (Off)a.y * sy + (Off)a.x * sx);
      at[u][1] = at[u][0] + sy;
    }
#pragma unroll 1
    for (int q = V * q0; q < C; q += V * GW) {
      Raw v[kRowItems][4];
#pragma unroll
      for (int u = 0; u < kRowItems; u++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const Raw *const a = reinterpret_cast<const Raw *>(at[u][i >> 1] + ((i & 1) ? sx : 0) + (q - V * q0));
          if constexpr (WHOLE) {
            v[u][i] = __ldg(a);
          } else {
            v[u][i] = T::zero();
            if ((mask[u] >> i) & 1) v[u][i] = __ldg(a);
          }
        }
#pragma unroll
      for (int u = 0; u < kRowItems; u++) {
        Raw acc = T::zero();
#pragma unroll
        for (int i = 0; i < 4; i++) acc = T::fma(v[u][i], w[u][i], acc);
        if (WHOLE && mask[u] == 0) acc = T::zero();
        // streaming: the maps, not the output, should stay in L2
        if (r + kGroups * u < left)
          __stcs(reinterpret_cast<Raw *>(out + kGroups * u * C + (q - V * q0)), acc);
      }
    }
  }
}

template <int V, int GW, bool SMALL>
__device__ __forceinline__ void gather_rows_for(const GatherMap &m, long k0, long total, const WarpFoot *sf, bool whole) {
  if (whole) gather_rows<V, GW, SMALL, true>(m, k0, total, sf);
  else gather_rows<V, GW, SMALL, false>(m, k0, total, sf);
}

// Warp per 32 consecutive (image, point) items: lane = item for the
// projection, the bilinear footprint (once per item; maps of one size share
// it) and the maps gathered item by item; the others in lane groups
// (gather_rows).
template <bool SMALL>
__global__ void __launch_bounds__(256, 4) project_gather_kernel(ProjGatherParams p) {
  __shared__ WarpFoot s_foot[8][32];
  const long total = (long)p.BV * p.N;
  const int lane = lane_id(), w8 = threadIdx.x >> 5;
  const long nwarps = ((long)gridDim.x * blockDim.x) >> 5;
  const bool small = total < (long)INT_MAX;
  for (long k0 = (((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * 32; k0 < total; k0 += nwarps * 32) {
    const long k = k0 + lane;
    const bool live = k < total;
    float gx = -2.0f, gy = -2.0f, dep = 0.0f;
    int img = 0, n = 0;
    if (live) {
      img = small ? (int)k / p.N : (int)(k / p.N);
      n = (int)(k - (long)img * p.N);
      if (p.gin) {
        gx = __ldg(p.gin + 2 * k);
        gy = __ldg(p.gin + 2 * k + 1);
        dep = p.din ? __ldg(p.din + k) : 0.0f;
      } else {
        persp_point(p, img, n, gx, gy, dep);
      }
    }
    int fh = -1, fw = -1;     // size of the map the current footprint is of
    bool staged = false;      // it is in the shared array
    bool whole = false;       // every footprint of the warp is wholly inside the image or wholly outside
    Foot f{};
    for (int mi = 0; mi < p.n_maps; mi++) {
      const GatherMap &m = p.maps[mi];
      if (m.H != fh || m.W != fw) {
        f = footprint(m.H, m.W, gx, gy);
        // past the last item: no corner, and texel (0, 0), which the lane groups
        // read beside their last item's (the footprint of (-2, -2) has a corner
        // in an image of two or three pixels an edge, from texel (-1, -1) on)
        if (!live) f.mask = f.x0 = f.y0 = 0;
        fh = m.H;
        fw = m.W;
        staged = false;
      }
      float first = 0.0f;
      if (m.rows) {
        if (!staged) {
          __syncwarp();  // the previous footprints' readers are done
          s_foot[w8][lane].w = make_float4((f.mask & 1) ? f.w[0] : 0.0f, (f.mask & 2) ? f.w[1] : 0.0f,
                                           (f.mask & 4) ? f.w[2] : 0.0f, (f.mask & 8) ? f.w[3] : 0.0f);
          s_foot[w8][lane].a = make_int4(f.x0, f.y0, f.mask, img);
          __syncwarp();
          staged = true;
          whole = __all_sync(SG_FULL, f.mask == 0 || f.mask == 15) && m.H > 1 && m.W > 1;
        }
        if (m.rows == 4) {
          if (m.C <= 8) gather_rows_for<4, 2, SMALL>(m, k0, total, s_foot[w8], whole);
          else if (m.C <= 16) gather_rows_for<4, 4, SMALL>(m, k0, total, s_foot[w8], whole);
          else gather_rows_for<4, 8, SMALL>(m, k0, total, s_foot[w8], whole);
        } else if (m.rows == 2) {
          gather_rows_for<2, 8, SMALL>(m, k0, total, s_foot[w8], whole);
        } else {
          gather_rows_for<1, 8, SMALL>(m, k0, total, s_foot[w8], whole);
        }
        if (mi == p.psdf_map && live) {  // channel 0 for the depth difference
#pragma unroll
          for (int i = 0; i < 4; i++)
            if ((f.mask >> i) & 1) first = __fmaf_rn(__ldg(m.data + corner_off(m, img, f.x0, f.y0, i)), f.w[i], first);
        }
      } else if (live) {
        first = gather_map<SMALL>(m, img, k, f);
      }
      if (mi == p.psdf_map && live) {
        const float dd = fminf(fmaxf(dep - first, -p.psdf_clip), p.psdf_clip);
        p.psdf[k] = dd * p.psdf_scale;
      }
    }
  }
}

// A map [n, C, H, W] through its strides into [n, H, W, C]: a CTA moves 64
// pixels x 32 channels through shared memory, read along x and written along
// the channels, 128 bytes a warp either way: 4 x 32 x 512^2 floats in 85 us
// cold (3.1 TB/s in and out; latency of the strided reads).
constexpr int kClPix = 64, kClChan = 32;

__global__ void __launch_bounds__(256) channels_last_kernel(const float *__restrict__ src, long sn, long sc, long sy,
                                                            long sx, int C, int H, int W, float *__restrict__ dst) {
  __shared__ float s[kClChan][kClPix + 1];
  const int HW = H * W;
  const int p0 = blockIdx.x * kClPix, c0 = blockIdx.y * kClChan;
  const long n = blockIdx.z;
  const bool lin = sy == (long)W * sx;
#pragma unroll
  for (int i = 0; i < kClPix * kClChan / 256; i++) {
    const int j = i * 256 + threadIdx.x, c = j / kClPix, px = j % kClPix, q = p0 + px;
    if (q < HW && c0 + c < C) {
      const long at = lin ? (long)q * sx : (long)(q / W) * sy + (long)(q % W) * sx;
      s[c][px] = __ldg(src + n * sn + (long)(c0 + c) * sc + at);
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kClPix * kClChan / 256; i++) {
    const int j = i * 256 + threadIdx.x, px = j / kClChan, c = j % kClChan, q = p0 + px;
    if (q < HW && c0 + c < C) dst[(n * HW + q) * C + c0 + c] = s[c][px];
  }
}

}  // namespace sg

using namespace sg;

extern "C" int sg_project_sampled_xyz(const SgTree *tree, const float *ray_ori, const float *ray_dir,
                                      const float *sampled_z, const int *sampled_idx, const float *K,
                                      const float *RT, int B, int num_views, int N, int S, int ori_w, int ori_h,
                                      int record_corners, float *proj_xy, float *proj_z, sg_stream_t stream) {
  if (!ray_ori || !ray_dir || !sampled_z || !sampled_idx || !K || !RT || !proj_xy || !proj_z)
    return SG_ERR_INVALID_ARG;
  if (record_corners && (!tree || !tree->counts || !tree->top_key || !tree->bot_key || !tree->voxel_size ||
                         !tree->vol_bbox || tree->Dt <= 0 || tree->Db != tree->Dt * tree->rate))
    return SG_ERR_INVALID_ARG;
  if (B <= 0 || num_views <= 0 || N < 0 || S <= 0 || ori_w <= 0 || ori_h <= 0) return SG_ERR_INVALID_ARG;
  const long total = (long)B * num_views * N * S;
  if (total == 0) return SG_OK;
  ProjSampledParams p{};
  if (tree) p.t = *tree;
  p.ori = ray_ori;
  p.dir = ray_dir;
  p.z = sampled_z;
  p.idx = sampled_idx;
  p.K = K;
  p.RT = RT;
  p.B = B;
  p.Nv = num_views;
  p.N = N;
  p.S = S;
  p.cw = (float)ori_w * 0.5f;
  p.ch = (float)ori_h * 0.5f;
  p.corners = record_corners ? 1 : 0;
  p.xy = proj_xy;
  p.pz = proj_z;
  long g = (total + 255) / 256;
  if (g > (long)num_sms() * 64) g = (long)num_sms() * 64;
  project_sampled_kernel<<<(int)g, 256, 0, stream>>>(p);
  SG_LAUNCH_CHECK();
  return SG_OK;
}

extern "C" int sg_project_gather(const SgProjGather *a, sg_stream_t stream) {
  if (!a) return SG_ERR_INVALID_ARG;
  if (!a->grids_in) {
    if (!a->points || !a->K || !a->R || !a->T || a->points_div <= 0 || a->n_images % a->points_div != 0 ||
        a->half_res == 0.0f)
      return SG_ERR_INVALID_ARG;
  } else if (a->psdf_map >= 0 && !a->depth_in) {
    return SG_ERR_INVALID_ARG;
  }
  if (a->n_images <= 0 || a->num_points < 0 || a->n_maps < 0 || a->n_maps > kMaxMaps) return SG_ERR_INVALID_ARG;
  if (a->psdf_map >= 0 && (a->psdf_map >= a->n_maps || !a->psdf || a->psdf_clip <= 0.0f)) return SG_ERR_INVALID_ARG;
  ProjGatherParams p{};
  p.gin = a->grids_in;
  p.din = a->depth_in;
  p.pts = a->points;
  p.pb = a->points_stride[0];
  p.pa = a->points_stride[1];
  p.pn = a->points_stride[2];
  p.pt_div = a->points_div;
  p.pdep = a->p_depths;
  p.db = a->p_depths_stride[0];
  p.dn = a->p_depths_stride[1];
  p.K = a->K;
  p.R = a->R;
  p.T = a->T;
  p.BV = a->n_images;
  p.N = a->num_points;
  p.depth_thres = a->depth_thres;
  p.min_d = a->min_d;
  p.max_d = a->max_d;
  p.half_res = a->half_res;
  p.ori_pts = a->ori_pts;
  p.grids = a->grids;
  p.depth = a->depth;
  p.n_maps = a->n_maps;
  bool small = true;
  for (int i = 0; i < a->n_maps; i++) {
    const SgFeatureMap &m = a->maps[i];
    if (!m.data || !m.out || m.C <= 0 || m.H <= 0 || m.W <= 0) return SG_ERR_INVALID_ARG;
    GatherMap &g = p.maps[i];
    g.data = m.data;
    g.sn = m.stride[0];
    g.sc = m.stride[1];
    g.sy = m.stride[2];
    g.sx = m.stride[3];
    g.C = m.C;
    g.H = m.H;
    g.W = m.W;
    g.out = m.out;
    // rows: channels contiguous, more of them than a thread per item reads
    // well (4), vectors as wide as the count, the strides and the addresses allow
    g.rows = 0;
    if (m.stride[1] == 1 && m.C > 4) {
      auto fits = [&](int v) {
        return m.C % v == 0 && m.stride[0] % v == 0 && m.stride[2] % v == 0 && m.stride[3] % v == 0 &&
               ((uintptr_t)m.data) % (4 * v) == 0 && ((uintptr_t)m.out) % (4 * v) == 0;
      };
      g.rows = fits(4) ? 4 : (fits(2) ? 2 : 1);
    }
    // 32-bit offsets hold every step of a map: images, channels (one channel
    // is never stepped over), rows and columns with one beyond the edges
    auto mag = [](long long v) { return (double)(v < 0 ? -v : v); };
    if (mag(m.stride[0]) * a->n_images + (m.C > 1 ? mag(m.stride[1]) * m.C : 0.0) + mag(m.stride[2]) * (m.H + 1.0) +
            mag(m.stride[3]) * (m.W + 1.0) >=
        2147483647.0)
      small = false;
  }
  p.psdf_map = a->psdf_map;
  p.psdf_clip = a->psdf_clip;
  p.psdf_scale = a->psdf_scale;
  p.psdf = a->psdf;
  const long total = (long)a->n_images * a->num_points;
  if (total == 0) return SG_OK;
  if (total > (1L << 40)) return SG_ERR_UNSUPPORTED;
  long g = (total + 255) / 256;
  if (g > (long)num_sms() * 64) g = (long)num_sms() * 64;
  if (small) project_gather_kernel<true><<<(int)g, 256, 0, stream>>>(p);
  else project_gather_kernel<false><<<(int)g, 256, 0, stream>>>(p);
  SG_LAUNCH_CHECK();
  return SG_OK;
}

extern "C" int sg_channels_last(const float *src, const long long *stride, int n, int C, int H, int W, float *dst,
                                sg_stream_t stream) {
  if (n < 0 || C <= 0 || H <= 0 || W <= 0) return SG_ERR_INVALID_ARG;
  if (n == 0) return SG_OK;
  if (!src || !stride || !dst) return SG_ERR_INVALID_ARG;
  const long hw = (long)H * W;
  const long blocks = ((long)C + kClChan - 1) / kClChan;
  constexpr int kMost = 65535;  // images and channel blocks of a grid
  if (hw > INT_MAX - kClPix || blocks > kMost) return SG_ERR_UNSUPPORTED;
  for (int n0 = 0; n0 < n;) {
    const int k = n - n0 < kMost ? n - n0 : kMost;
    const dim3 g((unsigned)((hw + kClPix - 1) / kClPix), (unsigned)blocks, (unsigned)k);
    channels_last_kernel<<<g, 256, 0, stream>>>(src + n0 * stride[0], stride[0], stride[1], stride[2], stride[3], C, H, W,
                                                dst + n0 * hw * C);
    n0 += k;
  }
  SG_LAUNCH_CHECK();
  return SG_OK;
}
