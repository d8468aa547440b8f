// intersect.cu -- ray / two-level tree intersection on sm_103a.
//
// Replaces intersection_kernel.cu (SAILOR c_lib/VoxelEncoding/src):
//   RayVoxelIntersection :36-71, RayVoxelIntersectionNodeListNew :128-284,
//   ray_voxel_traversal :286-439, MultiLayerOctree::voxel_traversal :828-895.
//
// One thread per ray walks the top grid with the reference's Amanatides-Woo
// DDA (same float operations, so the same cells in the same order).  At a
// kept brick the brick's node index comes from the dense brick map and the
// set bits of the brick's fine-occupancy mask give its children in
// ascending order -- the reference's lexicographic children order -- each
// slab-tested with geometry recomputed from its index (the reference copies
// a ~1.1 KB node per test).  The default variant (intersect_kernel) tests in
// the ray's own thread the occupied children the ray can reach; the
// warp-cooperative variant (intersect_warp_kernel, tune knob
// SG_TUNE_ISECT_WARP) tests every occupied child of a hit brick with the
// whole warp, one brick at a time -- the same rows, but measured 17x slower
// (28 against 1.6 ms, the bench's 7.4 M rays), where the reach test leaves ~1/5
// of the children: the tests' second opinion.  Hits
// are appended to the ray's row; the reference's -1 padding of the row tail
// is written by the same warps with bulk copies out of shared memory once
// their rays are done (by a second kernel under the other variant).
//
// With the tree's kept-brick bounds (SgTree.brick_box) the walk stops once
// it has passed them on an axis -- every later cell is empty, so the rows,
// counts and valid lengths are those of the full walk.
//
// Isolated occupied bricks (no occupied neighbour, hence not nodes) are
// treated as empty.  The reference instead looks up node index == the
// brick's local id there, i.e. an unrelated node.
#include <type_traits>

#include "common.cuh"

namespace sg {

struct IsectParams {
  SgTree t;
  const float *ori, *dir;
  int N, W, th_early_stop, opt_num, is_training;
  int *hit_idx;
  float *hit_t0, *hit_t1, *valid_len;
  int *hit_count;
  SgStatus *st;
  long R;                               // rays of the launch
  int nseg;                             // 0: frames of N rays; else ray segments
  const int *seg_begin, *seg_frame;
  const float *cams;                    // segments given as cameras (rays generated here)
  const int *cam_w;
};

// One axis of the ray / cube slab test (slab() in common.cuh, axis by axis): the
// interval [low, high] of the axes before, narrowed by the cell centred at c
// with half edge h; false when it becomes empty.
__device__ __forceinline__ bool slab_axis(float c, float h, float o, float inv, float &low, float &high) {
  float lo = ((c - h) - o) * inv;
  float hi = ((c + h) - o) * inv;
  if (lo > hi) {
    const float t = lo;
    lo = hi;
    hi = t;
  }
  if (hi < low) return false;
  if (lo > high) return false;
  low = (lo > low) ? lo : low;
  high = (hi < high) ? hi : high;
  return !(low > high);
}

// Hits of a ray, appended to its row.
struct HitRow {
  int *idx;
  float *t0, *t1;
  int W, cnt;
  float vlen;
  __device__ __forceinline__ void add(int id, float a, float b, float scale) {
    if (cnt < W) {
      idx[cnt] = id;
      t0[cnt] = a;
      t1[cnt] = b;
    }
    vlen = vlen + (b - a) * scale;
    cnt++;
  }
};

// n <= 16 bits of a brick's mask from bit position at on (rows may cross words
// where the edge is no power of two)
__device__ __forceinline__ uint32_t mask_bits(const uint32_t *__restrict__ mask, int mw, int at, int n) {
  const uint32_t w0 = __ldg(mask + (at >> 5));
  const uint32_t w1 = (at >> 5) + 1 < mw ? __ldg(mask + (at >> 5) + 1) : 0u;
  return __funnelshift_r(w0, w1, at & 31) & ((1u << n) - 1u);
}

// Cells of each x-slab of a brick that a ray can touch.  In voxel units
// relative to the brick the ray is a line; between the (widened) ends of the
// parent interval it covers a box, and between a slab's two x planes, where
// its slopes are of moderate size, a part of that box.  Everything is widened
// by kMargin voxels, in x too: the planes' rounding errors (1e-4 of the slope)
// are far inside what the margin's shift along the slope adds, those of the
// slab test itself are ~1e-6 of a voxel.  Every candidate gets the exact test.
struct ReachedCells {
  float lo[3], hi[3];  // the segment's box
  float y0, dy, z0, dz;  // y, z at x = 0 and slopes over x
  bool slopes;
  int a0, a1;  // slabs reached
  static constexpr float kMargin = 0.02f;

  __device__ __forceinline__ ReachedCells(const float (&u)[3], const float (&du)[3], float p0, float p1, int r) {
    const float tm = 1e-4f * (p1 - p0) + 1e-5f * fabsf(p1) + 1e-6f;
    const float ta = p0 - tm, tb = p1 + tm;
#pragma unroll
    for (int k = 0; k < 3; k++) {
      const float a = u[k] + ta * du[k], b = u[k] + tb * du[k];
      lo[k] = fminf(a, b) - kMargin;
      hi[k] = fmaxf(a, b) + kMargin;
    }
    a0 = max(0, (int)floorf(lo[0]));
    a1 = min(r - 1, (int)floorf(hi[0]));
    const float idu = 1.0f / du[0];
    dy = du[1] * idu;
    dz = du[2] * idu;
    slopes = fabsf(dy) < 1.0e4f && fabsf(dz) < 1.0e4f;  // false for NaN and infinities
    y0 = u[1] - u[0] * dy;
    z0 = u[2] - u[0] * dz;
  }
  // cells [ya, yb] x [za, zb] of slab a; false when there are none
  __device__ __forceinline__ bool slab(int a, int r, int &ya, int &yb, int &za, int &zb) const {
    float yl = lo[1], yh = hi[1], zl = lo[2], zh = hi[2];
    if (slopes) {
      const float n1 = (float)a - kMargin, n2 = (float)a + 1.0f + kMargin;
      const float y1 = y0 + n1 * dy, y2 = y0 + n2 * dy, z1 = z0 + n1 * dz, z2 = z0 + n2 * dz;
      yl = fmaxf(yl, fminf(y1, y2) - kMargin);
      yh = fminf(yh, fmaxf(y1, y2) + kMargin);
      zl = fmaxf(zl, fminf(z1, z2) - kMargin);
      zh = fminf(zh, fmaxf(z1, z2) + kMargin);
    }
    ya = max(0, (int)floorf(yl));
    yb = min(r - 1, (int)floorf(yh));
    za = max(0, (int)floorf(zl));
    zb = min(r - 1, (int)floorf(zh));
    return ya <= yb && za <= zb;
  }
};

// Children of the brick at (bx, by, bz) that the ray hits, in lexicographic
// (x, y, z) order: per x-slab the occupied cells among those the ray can
// reach (one 64-bit mask at 8^3), each given the reference's slab test, an
// axis at a time -- x once per slab -- with the same operations, so the hit
// set and its order equal the reference's full scan over all children.  A hit
// brick has one child hit on average (7.5 bricks and 7 children per ray on the
// 256^3 scenes), so ranks (set bits before a child) are counted at hits alone.
// RATE: the brick edge where it is 2, 4 or 8, else 0.
template <int RATE>
__device__ __forceinline__ void brick_children(const SgTree &t, const float (&o)[3], const float (&d)[3],
                                               const float (&inv)[3], const float (&bmin)[3], const LevelGeom &gb,
                                               int bx, int by, int bz, long brick, int k, float p0, float p1,
                                               HitRow &row) {
  const int r = RATE ? RATE : t.rate;
  const int mw = RATE ? (RATE * RATE * RATE + 31) / 32 : sg_mask_words_dev(r);
  const uint32_t *mask = t.brick_mask + (size_t)brick * mw;
  const int c0[3] = {bx * r, by * r, bz * r};
  const float h = gb.vs / 2.0f, ivs = 1.0f / gb.vs;
  float u[3], du[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    u[a] = (o[a] - (node_coord(gb, bmin[a], c0[a]) - gb.vs * 0.5f)) * ivs;
    du[a] = d[a] * ivs;
  }
  const ReachedCells rc(u, du, p0, p1, r);
  int base = -1, words = 0;  // id of the first child in mask word `words` (-1: not counted yet)
  auto child_id = [&](int bit) {
    if (base < 0) base = t.base_bot + __ldg(t.top_child_base + k);
    while (words < (bit >> 5)) base += __popc(__ldg(mask + words++));
    return base + __popc(__ldg(mask + words) & ((1u << (bit & 31)) - 1u));
  };
#pragma unroll 1
  for (int a = rc.a0; a <= rc.a1; a++) {
    int ya, yb, za, zb;
    if (!rc.slab(a, r, ya, yb, za, zb)) continue;
    const uint32_t zsel = ((2u << zb) - 1u) & ~((1u << za) - 1u);
    if constexpr (RATE != 0) {
      // bits of the slab's candidates
      constexpr int kBits = RATE * RATE;
      unsigned long long cand;
      if constexpr (RATE == 8) {
        const uint2 q = __ldg(reinterpret_cast<const uint2 *>(mask) + a);
        const uint32_t rows = zsel * 0x01010101u;
        cand = ((unsigned long long)(q.y & rows) << 32) | (q.x & rows);
        cand &= (~0ull >> (8 * (7 - yb + ya))) << (8 * ya);
      } else {
        uint32_t w = (__ldg(mask + ((a * kBits) >> 5)) >> ((a * kBits) & 31)) & ((1u << kBits) - 1u);
        w &= zsel * (RATE == 4 ? 0x1111u : 0x5u);
        cand = w & (((1u << (RATE * (yb - ya + 1))) - 1u) << (RATE * ya));
      }
      if (cand == 0ull) continue;
      float lx = 0.0f, hx = 100000.0f;
      if (!slab_axis(node_coord(gb, bmin[0], c0[0] + a), h, o[0], inv[0], lx, hx)) continue;
      do {
        const int bit = __ffsll(cand) - 1;
        cand &= cand - 1ull;
        float l = lx, u1 = hx;
        if (slab_axis(node_coord(gb, bmin[1], c0[1] + bit / RATE), h, o[1], inv[1], l, u1) &&
            slab_axis(node_coord(gb, bmin[2], c0[2] + bit % RATE), h, o[2], inv[2], l, u1) && !(l < 0.0f || u1 < 0.0f))
          row.add(child_id(a * kBits + bit), l, u1, 4.0f);
      } while (cand);
    } else {
      float lx = 0.0f, hx = 100000.0f;
      if (!slab_axis(node_coord(gb, bmin[0], c0[0] + a), h, o[0], inv[0], lx, hx)) continue;
      for (int y = ya; y <= yb; y++) {
        uint32_t zbits = mask_bits(mask, mw, (a * r + y) * r, r) & zsel;
        for (; zbits; zbits &= zbits - 1u) {
          const int z = __ffs(zbits) - 1;
          float l = lx, u1 = hx;
          if (slab_axis(node_coord(gb, bmin[1], c0[1] + y), h, o[1], inv[1], l, u1) &&
              slab_axis(node_coord(gb, bmin[2], c0[2] + z), h, o[2], inv[2], l, u1) && !(l < 0.0f || u1 < 0.0f))
            row.add(child_id((a * r + y) * r + z), l, u1, 4.0f);
        }
      }
    }
  }
}

// -1 padding of a warp's 32 rows: bulk copies out of constant shared memory,
// issued by one lane (the copy engine writes them while other warps walk),
// plain stores up to a row's first 16-byte boundary and behind its last.
constexpr int kFillInts = 1024;  // 4 KB of -1 and 4 KB of -1.0f

__device__ __forceinline__ void bulk_store(void *dst, uint32_t src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void bulk_pad_rows(int *idx, float *t0, float *t1, int rows, int cnt, int W,
                                              const int *fill) {
  const int lane = lane_id();
  const uint32_t fi = (uint32_t)__cvta_generic_to_shared(fill), ff = fi + 4 * kFillInts;
  int a16 = (int)(((uintptr_t)idx >> 2) & 3);  // the row's place in its 16 bytes (the arrays start aligned)
#pragma unroll 1
  for (int i = 0; i < rows; i++) {
    const int c = min(__shfl_sync(SG_FULL, cnt, i), W);
    const int head = min((4 - ((a16 + c) & 3)) & 3, W - c);  // to the first 16-byte boundary
    const int q0 = c + head, n4 = (W - q0) & ~3, end = q0 + n4;
    // lanes 0 .. 3: the head, lanes 4 .. 7: what is left behind the last boundary
    const int q = lane < 4 ? c + lane : end + lane - 4;
    if (lane < head || (lane >= 4 && q < W && lane < 8)) {
      idx[q] = -1;
      t0[q] = -1.0f;
      t1[q] = -1.0f;
    }
    if (lane == 0) {
      for (int p = q0; p < end; p += kFillInts) {
        const uint32_t n = 4 * min(end - p, kFillInts);
        bulk_store(idx + p, fi, n);
        bulk_store(t0 + p, ff, n);
        bulk_store(t1 + p, ff, n);
      }
    }
    idx += W;
    t0 += W;
    t1 += W;
    a16 = (a16 + W) & 3;
  }
  if (lane == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// Pixels of a camera segment in 8 x 4 tiles, a warp each, where its width, its
// height and its place allow it: a tile's rays meet more of the same bricks
// than 32 pixels of a row do.
__device__ __forceinline__ long tiled_pixel(const IsectParams &p, int s, long r) {
  const long begin = __ldg(p.seg_begin + s);
  const long end = s + 1 < p.nseg ? (long)__ldg(p.seg_begin + s + 1) : p.R;
  const int W = __ldg(p.cam_w + s);
  if (begin % 32 != 0 || W % 8 != 0 || (end - begin) % (4 * (long)W) != 0) return r;
  const int tile = (int)((r - begin) >> 5), lane = (int)(r & 31), tx = tile % (W / 8), ty = tile / (W / 8);
  return begin + (long)(ty * 4 + (lane >> 3)) * W + tx * 8 + (lane & 7);
}

// Thread per ray.  The walk and the children are two loops that the warp's
// lanes enter together: every lane walks to its next brick that is a node and
// hit (or to its end), then all of them test that brick's children.  What the
// walk decides (early stop, hit limit) depends on the bricks alone, so it has
// moved on when the children are tested.
//
// The walk keeps the brick's linear index and, per axis, the steps that are
// left until it has passed the frame's kept-brick bounds: past them every
// later cell is empty.  A step is an axis choice, three predicated updates and
// one brick map load, the cells in front of the bounds included (they are -1).
//
// Bound by instruction issue and divergence (10-13 of 32 lanes): per 4.2 M
// pixel rays 1.28 -> 0.81 ms with the rays' generation (1.06 without the pixel
// tiles), 217 K pixel rays 190 -> 117 us, 2^20 random rays 1.73 -> 1.20 ms,
// 16384 rays with padded rows of 1024 116 -> 86 us, 262144 of them 690 -> 551
// us (3.2 GB of rows: 0.48 ms at the measured HBM rate).  Not kept: RATE lanes
// per brick (a slab each; 60 against 91 M warp instructions on random rays, but
// 83 against 70 M on pixel rays: 1.79 ms), and children tested slab by slab and
// row by row under the step-wise walk (1.56 ms).
template <int RATE, bool PAD>
__device__ __forceinline__ void intersect_rays(const IsectParams &p) {
  __shared__ __align__(16) int s_fill[PAD ? 2 * kFillInts : 4];
  if (PAD) {
    for (int i = threadIdx.x; i < 2 * kFillInts; i += blockDim.x)
      s_fill[i] = i < kFillInts ? -1 : __float_as_int(-1.0f);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
  }
  const SgTree &t = p.t;
  const long R = p.R;
  const int lane = lane_id();
  long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int Dt = t.Dt;
  bool walking = false;
  float o[3] = {0.0f, 0.0f, 0.0f}, d[3] = {1.0f, 1.0f, 1.0f}, bmin[3] = {0.0f, 0.0f, 0.0f};
  float tm0 = 0.0f, tm1 = 0.0f, tm2 = 0.0f, td0 = 0.0f, td1 = 0.0f, td2 = 0.0f;
  int rem0 = 0, rem1 = 0, rem2 = 0;     // steps left per axis
  int last0 = 0, last1 = 0, last2 = 0;  // the cell reached with none left
  float vs = 1.0f;
  int b = 0;
  const int *node = t.brick_node;  // of the current cell
  if (r < R) {
    const int sgm = p.nseg > 0 ? segment_of(p.seg_begin, p.nseg, r) : 0;
    if (!PAD && p.cams) r = tiled_pixel(p, sgm, r);
    b = p.nseg > 0 ? __ldg(p.seg_frame + sgm) : (int)(r / p.N);
    const float *bb = t.vol_bbox + 6 * b;
    const float xc = (bb[0] + bb[1]) / 2.0f, yc = (bb[2] + bb[3]) / 2.0f, zc = (bb[4] + bb[5]) / 2.0f;
    vs = t.voxel_size[b];
    const float vs_top = vs * (float)(t.Db / Dt);
#pragma unroll
    for (int a = 0; a < 3; a++) bmin[a] = bb[2 * a];
    segment_ray(p.ori, p.dir, p.cams, p.cam_w, p.seg_begin, sgm, r, o, d);
    float inv[3];
#pragma unroll
    for (int a = 0; a < 3; a++) inv[a] = __fdividef(1.0f, d[a]);
    float T0, T1;
    if (slab(o, inv, xc, yc, zc, vs_top * (float)Dt, T0, T1) && !(T0 < 0.0f || T1 < 0.0f)) {
      int st[3], rem[3], last[3];
      float tm[3], td[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        const float sp = __fmaf_rn(T0, d[a], o[a]);
        const float so = sp - (bb[2 * a] - vs / 2.0f);
        int s = (int)(so / vs_top);
        s = s < 0 ? 0 : s;
        st[a] = s < Dt ? s : Dt - 1;
        const float step = (d[a] >= 0) ? 1.0f : -1.0f;
        const float nb = (step > 0) ? ((float)st[a] + step) * vs_top : (float)st[a] * vs_top;
        tm[a] = (d[a] != 0) ? (nb - so) / d[a] : 9999999.0f;
        td[a] = (d[a] != 0) ? vs_top / d[a] * step : 9999999.0f;
        int lo = 0, hi = Dt - 1;
        if (t.brick_box) {
          lo = __ldg(t.brick_box + 6 * b + a);
          hi = __ldg(t.brick_box + 6 * b + 3 + a);
        }
        last[a] = step > 0 ? hi : lo;
        rem[a] = step > 0 ? hi - st[a] : st[a] - lo;
      }
      tm0 = tm[0], tm1 = tm[1], tm2 = tm[2];
      td0 = td[0], td1 = td[1], td2 = td[2];
      rem0 = rem[0], rem1 = rem[1], rem2 = rem[2];
      last0 = last[0], last1 = last[1], last2 = last[2];
      node += (((long)b * Dt + st[0]) * Dt + st[1]) * Dt + st[2];
      walking = (rem0 | rem1 | rem2) >= 0;
    }
  }
  HitRow row{p.hit_idx + (size_t)r * p.W, p.hit_t0 + (size_t)r * p.W, p.hit_t1 + (size_t)r * p.W, p.W, 0, 0.0f};
  const LevelGeom gt = level_geom(vs, t.Db / Dt), gb = level_geom(vs, 1);
  const bool f0 = d[0] >= 0, f1 = d[1] >= 0, f2 = d[2] >= 0;  // steps forward
  const int dn0 = f0 ? Dt * Dt : -Dt * Dt, dn1 = f1 ? Dt : -Dt, dn2 = f2 ? 1 : -1;
  const bool limits = p.th_early_stop > -1 || p.opt_num > -1;
  bool pre_empty = false, has_valid = false;
  int nsucc = 0, nint = 0;
  while (true) {
    // to the next hit brick
    int k = -1, bx = 0, by = 0, bz = 0;
    float p0 = 0.0f, p1 = 0.0f;
    while (walking && k < 0) {
      k = __ldg(node);
      if (k >= 0) {
        bx = f0 ? last0 - rem0 : last0 + rem0;
        by = f1 ? last1 - rem1 : last1 + rem1;
        bz = f2 ? last2 - rem2 : last2 + rem2;
        const float inv[3] = {__fdividef(1.0f, d[0]), __fdividef(1.0f, d[1]), __fdividef(1.0f, d[2])};
        if (!slab(o, inv, node_coord(gt, bmin[0], bx), node_coord(gt, bmin[1], by), node_coord(gt, bmin[2], bz), gt.vs,
                  p0, p1) ||
            p0 < 0.0f || p1 < 0.0f)
          k = -1;
      }
      if (limits) {
        if (p.th_early_stop > -1) {
          if (k < 0) {
            if (pre_empty && has_valid) nsucc++;
            pre_empty = true;
          } else {
            nsucc = 0;
            pre_empty = false;
            has_valid = true;
          }
          if ((nsucc + 1) >= p.th_early_stop) walking = false;
        }
        if (p.opt_num > -1) {
          if (k >= 0) nint++;
          if (nint >= p.opt_num) walking = false;
        }
      }
      const bool t01 = tm0 < tm1;
      const bool a0 = t01 && tm0 < tm2, a1 = !t01 && tm1 < tm2, a2 = !(a0 || a1);
      node += a0 ? dn0 : (a1 ? dn1 : dn2);
      if (a0) tm0 += td0;
      if (a1) tm1 += td1;
      if (a2) tm2 += td2;
      rem0 -= a0;
      rem1 -= a1;
      rem2 -= a2;
      if ((rem0 | rem1 | rem2) < 0) walking = false;
    }
    if (!__any_sync(SG_FULL, k >= 0)) break;
    if (k >= 0) {
      if (!p.is_training) {
        const float inv[3] = {__fdividef(1.0f, d[0]), __fdividef(1.0f, d[1]), __fdividef(1.0f, d[2])};
        brick_children<RATE>(t, o, d, inv, bmin, gb, bx, by, bz, (((long)b * Dt + bx) * Dt + by) * Dt + bz, k, p0, p1,
                             row);
      }
      row.add(t.base_top + k, p0, p1, 1.0f);
    }
  }
  if (r < R) {
    p.valid_len[r] = row.vlen;
    if (p.hit_count) p.hit_count[r] = row.cnt;
  }
  if (PAD) {
    const size_t at = (size_t)(r - lane) * p.W;
    bulk_pad_rows(p.hit_idx + at, p.hit_t0 + at, p.hit_t1 + at, (int)min(32l, max(0l, R - (r - lane))), row.cnt, p.W, s_fill);
  }
  // warp-aggregated status updates
  int m = row.cnt;
#pragma unroll
  for (int o2 = 16; o2 > 0; o2 >>= 1) m = max(m, __shfl_xor_sync(SG_FULL, m, o2));
  if (lane == 0 && p.st) {
    if (m > 0) atomicMax(&p.st->max_hits, m);
    if (m > p.W) atomicOr(&p.st->flags, SG_FLAG_HIT_OVERFLOW);
  }
  // the fill is read until the bulk copies are done with it
  if (PAD) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// Compact rows, and padded ones.  80 registers against the 64 (and spills) the
// compiler takes by itself: 2^20 random rays 1.20 against 1.24 ms, 217 K pixel
// rays 121 against 139 us; the padded rows' kernel is better off with its own
// choice (80 there spill: 16384 rays 89 against 85 us).
template <int RATE>
__global__ void __maxnreg__(80) intersect_kernel(IsectParams p) {
  intersect_rays<RATE, false>(p);
}
template <int RATE>
__global__ void __launch_bounds__(512) intersect_padded_kernel(IsectParams p) {
  intersect_rays<RATE, true>(p);
}

// Rays from which the walking warps pad their rows themselves: the few warps of
// fewer rays would write them one row after another, where a second kernel has a
// warp a row (64 rows of 1024: 18 us by the walking warps, 12 by two kernels; 200
// rows 20 and 18; 256 and more the walking warps).
constexpr long kPadInWalk = 256;

template <bool PAD>
static void launch_intersect(const IsectParams &p, sg_stream_t stream) {
  const int blk = tune(SG_TUNE_ISECT_BLOCK);
  const int g = ceil_div(p.R, blk);
  auto go = [&](auto rate) {
    constexpr int RATE = decltype(rate)::value;
    if (PAD) intersect_padded_kernel<RATE><<<g, blk, 0, stream>>>(p);
    else intersect_kernel<RATE><<<g, blk, 0, stream>>>(p);
  };
  if (p.t.rate == 8 && ((uintptr_t)p.t.brick_mask) % 8 == 0) go(std::integral_constant<int, 8>());
  else if (p.t.rate == 4) go(std::integral_constant<int, 4>());
  else if (p.t.rate == 2) go(std::integral_constant<int, 2>());
  else go(std::integral_constant<int, 0>());
}

// ---------------------------------------------------------------------------
// Warp-cooperative variant: each lane walks its own ray's DDA (the same
// float operations, hence the same cells), but the children of a hit brick
// are tested by the whole warp: lane l takes children 32 i + l (i over the
// brick's 32-bit mask words), so one warp instruction covers 32 children in
// lexicographic order; a ballot of the hits and a popcount of the lanes
// before give each hit its row position, and the mask bits before a child
// its node rank.  Hit bricks of different lanes in the same DDA step are
// served one after another in lane order, so every ray's row is in the
// reference's order (per brick: children in lexicographic order, then the
// brick).  The valid length is summed hit by hit in row order, as the
// reference sums it.  The DDA state stays in registers (per-axis selects).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) intersect_warp_kernel(IsectParams p) {
  const SgTree &t = p.t;
  const long R = p.R;
  const int lane = lane_id();
  const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = r < R;
  int cnt = 0;
  bool over = false;
  float vlen = 0.0f;
  int b = 0;
  float o[3] = {0.0f, 0.0f, 0.0f}, d[3] = {1.0f, 1.0f, 1.0f}, inv[3] = {1.0f, 1.0f, 1.0f};
  float bmin[3] = {0.0f, 0.0f, 0.0f};
  float vs = 1.0f;
  int st0 = 0, st1 = 0, st2 = 0;
  float tm0 = 0.0f, tm1 = 0.0f, tm2 = 0.0f, td0 = 0.0f, td1 = 0.0f, td2 = 0.0f;
  int sp0 = 1, sp1 = 1, sp2 = 1;
  bool active = false;
  const long vt = (long)t.Dt * t.Dt * t.Dt;
  if (in) {
    const int sgm = p.nseg > 0 ? segment_of(p.seg_begin, p.nseg, r) : 0;
    b = p.nseg > 0 ? __ldg(p.seg_frame + sgm) : (int)(r / p.N);
    const float *bb = t.vol_bbox + 6 * b;
    bmin[0] = bb[0];
    bmin[1] = bb[2];
    bmin[2] = bb[4];
    const float xc = (bb[0] + bb[1]) / 2.0f, yc = (bb[2] + bb[3]) / 2.0f, zc = (bb[4] + bb[5]) / 2.0f;
    vs = t.voxel_size[b];
    const float vs_top = vs * (float)(t.Db / t.Dt);
    const float bst[3] = {bb[0] - vs / 2.0f, bb[2] - vs / 2.0f, bb[4] - vs / 2.0f};
    segment_ray(p.ori, p.dir, p.cams, p.cam_w, p.seg_begin, sgm, r, o, d);
#pragma unroll
    for (int a = 0; a < 3; a++) inv[a] = __fdividef(1.0f, d[a]);
    float T0, T1;
    if (slab(o, inv, xc, yc, zc, vs_top * (float)t.Dt, T0, T1) && !(T0 < 0.0f || T1 < 0.0f)) {
      float so[3];
      int st[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        float spos = __fmaf_rn(T0, d[a], o[a]);
        so[a] = spos - bst[a];
        int s = (int)(so[a] / vs_top);
        s = s < 0 ? 0 : s;
        st[a] = s < t.Dt ? s : t.Dt - 1;
      }
      float step[3], tm[3], td[3];
#pragma unroll
      for (int a = 0; a < 3; a++) {
        step[a] = (d[a] >= 0) ? 1.0f : -1.0f;
        float nb = (step[a] > 0) ? ((float)st[a] + step[a]) * vs_top : (float)st[a] * vs_top;
        tm[a] = (d[a] != 0) ? (nb - so[a]) / d[a] : 9999999.0f;
        td[a] = (d[a] != 0) ? vs_top / d[a] * step[a] : 9999999.0f;
      }
      st0 = st[0], st1 = st[1], st2 = st[2];
      tm0 = tm[0], tm1 = tm[1], tm2 = tm[2];
      td0 = td[0], td1 = td[1], td2 = td[2];
      sp0 = (int)step[0], sp1 = (int)step[1], sp2 = (int)step[2];
      active = true;
    }
  }
  int *oi = p.hit_idx + (size_t)(in ? r : 0) * p.W;
  float *o0 = p.hit_t0 + (size_t)(in ? r : 0) * p.W, *o1 = p.hit_t1 + (size_t)(in ? r : 0) * p.W;
  const int rate = t.rate, r3 = rate * rate * rate;
  const int mw = sg_mask_words_dev(rate);
  bool pre_empty = false, has_valid = false;
  int nsucc = 0, nint = 0;
  const int J = 4 * t.Dt;
  for (int j = 0; j < J; j++) {
    if (!__any_sync(SG_FULL, active)) break;
    // this step's brick of every active lane: a node whose box the ray enters
    bool pend = false;
    int k = -1;
    float p0 = 0.0f, p1 = 0.0f;
    if (active) {
      const long brick = (long)b * vt + ((long)st0 * t.Dt + st1) * t.Dt + st2;
      k = t.brick_node[brick];
      if (k >= 0) {
        const LevelGeom gt = level_geom(vs, t.Db / t.Dt);
        pend = slab(o, inv, node_coord(gt, bmin[0], st0), node_coord(gt, bmin[1], st1), node_coord(gt, bmin[2], st2),
                    gt.vs, p0, p1) &&
               !(p0 < 0.0f || p1 < 0.0f);
      }
    }
    int rid = -1;
    if (!p.is_training) {
      // children of the pending bricks, one brick at a time in lane order
      unsigned pm = __ballot_sync(SG_FULL, pend);
      while (pm) {
        const int L = __ffs(pm) - 1;
        pm &= pm - 1;
        const float oL[3] = {__shfl_sync(SG_FULL, o[0], L), __shfl_sync(SG_FULL, o[1], L),
                             __shfl_sync(SG_FULL, o[2], L)};
        const float iL[3] = {__shfl_sync(SG_FULL, inv[0], L), __shfl_sync(SG_FULL, inv[1], L),
                             __shfl_sync(SG_FULL, inv[2], L)};
        const float bL[3] = {__shfl_sync(SG_FULL, bmin[0], L), __shfl_sync(SG_FULL, bmin[1], L),
                             __shfl_sync(SG_FULL, bmin[2], L)};
        const int sx = __shfl_sync(SG_FULL, st0, L), sy = __shfl_sync(SG_FULL, st1, L),
                  sz = __shfl_sync(SG_FULL, st2, L);
        const int fL = __shfl_sync(SG_FULL, b, L);
        const int kL = __shfl_sync(SG_FULL, k, L);
        const long rL = __shfl_sync(SG_FULL, (long long)(in ? r : 0), L);
        int base = __shfl_sync(SG_FULL, cnt, L);
        float vl = __shfl_sync(SG_FULL, vlen, L);
        const LevelGeom gb = level_geom(__shfl_sync(SG_FULL, vs, L), 1);
        const long brickL = (long)fL * vt + ((long)sx * t.Dt + sy) * t.Dt + sz;
        const uint32_t *mask = t.brick_mask + (size_t)brickL * mw;
        const int cb = t.base_bot + t.top_child_base[kL];
        int *oiL = p.hit_idx + (size_t)rL * p.W;
        float *o0L = p.hit_t0 + (size_t)rL * p.W, *o1L = p.hit_t1 + (size_t)rL * p.W;
        const int x0 = sx * rate, y0 = sy * rate, z0 = sz * rate;
        int rank0 = 0;
        bool ovL = false;
        for (int i = 0; i < mw; i++) {
          const uint32_t word = __ldg(mask + i);
          const int c = 32 * i + lane;
          bool hit = false;
          float c0 = 0.0f, c1 = 0.0f;
          if (c < r3 && ((word >> lane) & 1u)) {
            const int a = c / (rate * rate), y = (c / rate) % rate, z = c % rate;
            hit = slab(oL, iL, node_coord(gb, bL[0], x0 + a), node_coord(gb, bL[1], y0 + y),
                       node_coord(gb, bL[2], z0 + z), gb.vs, c0, c1) &&
                  !(c0 < 0.0f || c1 < 0.0f);
          }
          const unsigned hb = __ballot_sync(SG_FULL, hit);
          if (hit) {
            const int pos = base + __popc(hb & ((1u << lane) - 1u));
            if (pos < p.W) {
              oiL[pos] = cb + rank0 + __popc(word & ((1u << lane) - 1u));
              o0L[pos] = c0;
              o1L[pos] = c1;
            }
          }
          // the ray's valid length, hit by hit in row order
          const float len4 = (c1 - c0) * 4.0f;
          for (unsigned m = hb; m; m &= m - 1) vl = vl + __shfl_sync(SG_FULL, len4, __ffs(m) - 1);
          if (base + __popc(hb) > p.W) ovL = true;
          base += __popc(hb);
          rank0 += __popc(word);
        }
        if (lane == L) {
          cnt = base;
          vlen = vl;
          over = over || ovL;
        }
      }
    }
    if (pend) {
      if (cnt < p.W) {
        oi[cnt] = t.base_top + k;
        o0[cnt] = p0;
        o1[cnt] = p1;
      } else {
        over = true;
      }
      vlen = vlen + (p1 - p0);
      cnt++;
      rid = cnt - 1;
    }
    if (active) {
      if (p.th_early_stop > -1) {
        if (rid == -1) {
          if (pre_empty && has_valid) nsucc++;
          pre_empty = true;
        } else {
          nsucc = 0;
          pre_empty = false;
          has_valid = true;
        }
        if ((nsucc + 1) >= p.th_early_stop) active = false;
      }
      if (p.opt_num > -1) {
        if (rid + 1 > 0) nint++;
        if (nint >= p.opt_num) active = false;
      }
    }
    if (active) {
      int ax;
      if (tm0 < tm1) ax = (tm0 < tm2) ? 0 : 2;
      else ax = (tm1 < tm2) ? 1 : 2;
      if (ax == 0) {
        st0 = (int)((float)st0 + (float)sp0);
        tm0 += td0;
      } else if (ax == 1) {
        st1 = (int)((float)st1 + (float)sp1);
        tm1 += td1;
      } else {
        st2 = (int)((float)st2 + (float)sp2);
        tm2 += td2;
      }
      if (st0 < 0 || st0 >= t.Dt || st1 < 0 || st1 >= t.Dt || st2 < 0 || st2 >= t.Dt) active = false;
    }
  }
  if (in) {
    p.valid_len[r] = vlen;
    if (p.hit_count) p.hit_count[r] = cnt;
  }
  int m = cnt;
#pragma unroll
  for (int o2 = 16; o2 > 0; o2 >>= 1) m = max(m, __shfl_xor_sync(SG_FULL, m, o2));
  const bool anyover = __any_sync(SG_FULL, over);
  if (lane == 0 && p.st) {
    if (m > 0) atomicMax(&p.st->max_hits, m);
    if (anyover) atomicOr(&p.st->flags, SG_FLAG_HIT_OVERFLOW);
  }
}

// -1 padding of row tails [count, W): warp per row
__global__ void pad_rows_kernel(long R, int W, const int *__restrict__ count, int *idx, float *t0,
                                float *t1) {
  const int lane = lane_id();
  for (long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < R;
       r += ((long)gridDim.x * blockDim.x) >> 5) {
    pad_row_tail(idx, t0, t1, (size_t)r * W, min(count[r], W), W, lane);
  }
}

void launch_pad_rows(long R, int W, const int *count, int *idx, float *t0, float *t1, sg_stream_t stream) {
  if (R <= 0 || W <= 0) return;
  int g = ceil_div(R * 32, 256);
  if (g > num_sms() * 64) g = num_sms() * 64;
  pad_rows_kernel<<<g, 256, 0, stream>>>(R, W, count, idx, t0, t1);
}

}  // namespace sg

using namespace sg;

extern "C" int sg_intersect(const SgTree *tree, const float *ori, const float *dir, int N, int W,
                            int th_early_stop, int opt_num, int is_training, int padded, int *hit_idx,
                            float *hit_t0, float *hit_t1, float *valid_len, int *hit_count,
                            SgStatus *status, sg_stream_t stream) {
  if (!tree || !ori || !dir || !hit_idx || !hit_t0 || !hit_t1 || !valid_len) return SG_ERR_INVALID_ARG;
  if (N <= 0 || W <= 0 || tree->B <= 0 || tree->Dt <= 0 || tree->Db != tree->Dt * tree->rate)
    return SG_ERR_INVALID_ARG;
  if (padded && !hit_count) return SG_ERR_INVALID_ARG;
  if (padded && (((uintptr_t)hit_idx) | ((uintptr_t)hit_t0) | ((uintptr_t)hit_t1)) % 16 != 0)
    return SG_ERR_INVALID_ARG;
  long R = (long)tree->B * N;
  IsectParams p{*tree, ori, dir, N, W, th_early_stop, opt_num, is_training,
                hit_idx, hit_t0, hit_t1, valid_len, hit_count, status, R, 0, nullptr, nullptr, nullptr, nullptr};
  if (tune(SG_TUNE_ISECT_WARP)) {
    intersect_warp_kernel<<<ceil_div(R, 256), 256, 0, stream>>>(p);
    if (padded) launch_pad_rows(R, W, hit_count, hit_idx, hit_t0, hit_t1, stream);
  } else if (padded && R >= kPadInWalk) {
    launch_intersect<true>(p, stream);
  } else {
    launch_intersect<false>(p, stream);
    if (padded) launch_pad_rows(R, W, hit_count, hit_idx, hit_t0, hit_t1, stream);
  }
  SG_LAUNCH_CHECK();
  return SG_OK;
}

extern "C" int sg_intersect_segments(const SgTree *tree, const SgRaySegments *seg, const float *ori,
                                     const float *dir, int W, int *hit_idx, float *hit_t0, float *hit_t1,
                                     float *valid_len, int *hit_count, SgStatus *status, sg_stream_t stream) {
  if (!tree || !seg || !hit_idx || !hit_t0 || !hit_t1 || !valid_len || !hit_count) return SG_ERR_INVALID_ARG;
  if ((seg->cameras == nullptr) != (seg->widths == nullptr)) return SG_ERR_INVALID_ARG;
  if (!seg->cameras && (!ori || !dir)) return SG_ERR_INVALID_ARG;
  if (seg->count <= 0 || seg->total < 0 || !seg->ray_begin || !seg->frame) return SG_ERR_INVALID_ARG;
  if (W <= 0 || tree->B <= 0 || tree->Dt <= 0 || tree->Db != tree->Dt * tree->rate) return SG_ERR_INVALID_ARG;
  if (seg->total == 0) return SG_OK;
  IsectParams p{*tree, ori, dir, 1, W, -1, -1, 0, hit_idx, hit_t0, hit_t1, valid_len, hit_count, status,
                (long)seg->total, seg->count, seg->ray_begin, seg->frame, seg->cameras, seg->widths};
  if (tune(SG_TUNE_ISECT_WARP)) {
    intersect_warp_kernel<<<ceil_div((long)seg->total, 256), 256, 0, stream>>>(p);
  } else {
    launch_intersect<false>(p, stream);
  }
  SG_LAUNCH_CHECK();
  return SG_OK;
}
