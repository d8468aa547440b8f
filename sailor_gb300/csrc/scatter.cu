// scatter.cu -- deterministic reduction of the training pass's grid
// gradients: a segmented reduction over the sampled cells, sorted.
//
// The in-kernel scatter of the render backward adds each cell run's
// gradient into the grids with float atomics, so the summation order -- and
// the last bits of the gradient -- change from run to run.  Here the
// training pass (render.cu, record mode) writes one record per run of a ray's
// samples in one trilinear cell instead: the cell as a 32-bit key (frame and
// lower corner, grouped by parity class), and a 32-byte record of the 8
// corners' sums of corner weight x compositing weight (with the TSDF's gradient,
// a second one of its sums); the ray's colour-head factor of the feature
// gradient goes to a per-ray table.
// The pass packs each ray's records at the front of the ray's slots and
// writes their count.  Then
//   1. the records are compacted (slot order kept: a scan over the rays'
//      record counts, a warp per ray moving its keys) and their
//      keys sorted, stably, with the record slots as values (segsort.cu):
//      records of one cell become one run, in slot order (ray order, then
//      sorted sample order -- fixed by the ray layout);
//   2. run heads are flagged and scanned into the list of distinct cells;
//   3. for each of the 8 parity classes in turn, each cell's run is summed in
//      a fixed order into the 8 corners x C channels it touches (four sums of
//      every fourth record, added in pairs: which of the four takes a record
//      depends on its place in the warp's stretch, the four sets and the pairs do
//      not), and the sums are added into the grids.  Cells of one class share no corner, so every
//      grid value gets one addition per class, classes in a fixed order.
// Every grid value is therefore the same sum in the same order on every run:
// the gradients are bit-identical across runs, launch shapes and graph
// replays.
//
// Before the training pass, a scan over the rays (rays with hits, and their
// record slots: S per ray with hits) builds the compact list of rays the
// pass visits; rays without hits get their outputs (0, and the loss of the
// target alone) here.
#include "ray_core.cuh"
#include "scatter.cuh"
#include "segsort.cuh"

namespace sg {

__device__ __forceinline__ long ray_samples(const SgRaySegments &seg, int S_max, long r, int &s) {
  s = segment_of(seg.ray_begin, seg.count, r);
  const int S = __ldg(seg.samples + s);
  return S < S_max ? S : S_max;
}

// per ray: 1 if it has hits
__global__ void det_ray_flags_kernel(const int *__restrict__ hit_count, long R, int *__restrict__ hitb) {
  for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < R; r += (long)gridDim.x * blockDim.x)
    hitb[r] = __ldg(hit_count + r) > 0 ? 1 : 0;
}

// compact ray list and slots (a segment's rays with hits have its sample count
// of slots each); outputs of rays without hits
__global__ void det_ray_emit_kernel(SgRaySegments seg, int S_max, long R, const int *__restrict__ hit_count,
                                    const int *__restrict__ hitb, const int *__restrict__ seg_hit,
                                    const int *__restrict__ seg_slot, int *__restrict__ hit_ray,
                                    int *__restrict__ hit_slot, DetTrainOut o) {
  for (long r = (long)blockIdx.x * blockDim.x + threadIdx.x; r < R; r += (long)gridDim.x * blockDim.x) {
    if (__ldg(hit_count + r) > 0) {
      const int k = hitb[r];
      int s;
      const int S = (int)ray_samples(seg, S_max, r, s);
      hit_ray[k] = (int)r;
      hit_slot[k] = __ldg(seg_slot + s) + (k - __ldg(seg_hit + s)) * S;
    } else if (o.out_rgb) {
      float l = 0.0f;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const float t = __ldg(o.target_rgb + r * 3 + c);
        o.out_rgb[r * 3 + c] = 0.0f;
        l += t * t;
      }
      o.out_depth[r] = o.out_ws[r] = o.out_alpha[r] = 0.0f;
      if (o.out_loss) o.out_loss[r] = 0.5f * o.loss_scale * l;
    }
  }
}

// compact index and slot of each segment's first ray with hits (a scan over the
// segments; one CTA); slots needed, slots used (clamped to the capacity) and
// the capacity flag
__global__ void __launch_bounds__(256) det_seg_kernel(SgRaySegments seg, int S_max, long R, const int *__restrict__ hitb,
                                                      int *__restrict__ cnt, int *__restrict__ seg_hit,
                                                      int *__restrict__ seg_slot, long cap, SgStatus *st) {
  __shared__ int s_warp[17];
  auto first_hit = [&](int s) {
    const long rb = __ldg(seg.ray_begin + s);
    return rb < R ? hitb[rb] : cnt[kDetHits];
  };
  int need = 0;
  for (int s0 = 0; s0 < seg.count; s0 += blockDim.x) {
    const int s = s0 + threadIdx.x;
    int slots = 0, k = 0;
    if (s < seg.count) {
      k = first_hit(s);
      slots = (first_hit(s + 1) - k) * min(__ldg(seg.samples + s), S_max);
    }
    int total;
    const int before = block_excl_scan_256(slots, s_warp, total);
    if (s < seg.count) {
      seg_hit[s] = k;
      seg_slot[s] = need + before;
    }
    need += total;
  }
  if (threadIdx.x == 0) {
    seg_hit[seg.count] = first_hit(seg.count);
    seg_slot[seg.count] = need;
    cnt[kDetSlotsNeeded] = need;
    cnt[kDetSlots] = need < cap ? need : (int)cap;
    if (need > cap && st) {
      atomicOr(&st->flags, SG_FLAG_RECORD_CAPACITY);
    }
  }
}

// the records, compacted in slot order (ray order, then sorted position
// order: each ray's records lead its slots): key and slot, 16 lanes per ray
// (17 records a ray in the mean);
// first = the rays' exclusive record counts
__global__ void det_compact_kernel(const uint32_t *__restrict__ key, const int *__restrict__ cnt,
                                   const int *__restrict__ first, const int *__restrict__ hit_slot,
                                   uint32_t *__restrict__ ckey, uint32_t *__restrict__ cslot) {
  const long n = cnt[kDetHits];
  const int total = cnt[kDetValid];
  const int lane = lane_id() & 15;
  for (long k = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 4; k < n;
       k += ((long)gridDim.x * blockDim.x) >> 4) {
    const int a = __ldg(first + k), e = k + 1 < n ? __ldg(first + k + 1) : total;
    const long base = __ldg(hit_slot + k);
    for (int i = lane; i < e - a; i += 16) {
      ckey[a + i] = __ldg(key + base + i);
      cslot[a + i] = (uint32_t)(base + i);
    }
  }
}

// The distinct cells of the sorted keys, a scan over the heads of their runs
// whose input and output stay in the kernels (as five passes -- flags, their
// scan, the list -- 120 us for 13 M keys, now 66; 26 -> 15 us for 1 M).
// Heads before a thread's four keys j0 .. j0 + 3 of n; head[q]: key j0 + q starts a run.
__device__ __forceinline__ int key_heads(const uint32_t *__restrict__ key, long j0, long n, uint32_t (&k)[4],
                                         uint32_t &prev, bool (&head)[4]) {
  prev = j0 > 0 && j0 < n ? __ldg(key + j0 - 1) : 0u;
  int s = 0;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    k[q] = j0 + q < n ? __ldg(key + j0 + q) : 0u;
    head[q] = j0 + q < n && (j0 + q == 0 || k[q] != (q > 0 ? k[q > 0 ? q - 1 : 0] : prev));
    s += head[q];
  }
  return s;
}

__global__ void __launch_bounds__(256) det_head_sums_kernel(const uint32_t *__restrict__ key, const int *__restrict__ cnt,
                                                            int *__restrict__ sums) {
  __shared__ int s_warp[17];
  const long n = cnt[kDetValid], nb = (n + kScanBlock - 1) / kScanBlock;
  for (long blk = blockIdx.x; blk < nb; blk += gridDim.x) {
    uint32_t k[4], prev;
    bool head[4];
    int total;
    block_excl_scan_256(key_heads(key, blk * kScanBlock + threadIdx.x * 4, n, k, prev, head), s_warp, total);
    if (threadIdx.x == 0) sums[blk] = total;
  }
}

// per cell: key and first sorted position; the end of the last run; the first
// cell of each parity class (bound[8]: the end of the last class); per sorted
// position: the cells that start before it
__global__ void __launch_bounds__(256) det_cells_kernel(const uint32_t *__restrict__ key, const int *__restrict__ sums,
                                                        const int *__restrict__ cnt, uint32_t cls,
                                                        uint32_t *__restrict__ ukey, int *__restrict__ ustart,
                                                        int *__restrict__ heads, int *__restrict__ bound) {
  __shared__ int s_warp[17];
  const long n = cnt[kDetValid], nb = (n + kScanBlock - 1) / kScanBlock;
  const int nu = cnt[kDetCells];
  for (long blk = blockIdx.x; blk < nb; blk += gridDim.x) {
    const long j0 = blk * kScanBlock + threadIdx.x * 4;
    uint32_t k[4], prev;
    bool head[4];
    int total;
    int u = block_excl_scan_256(key_heads(key, j0, n, k, prev, head), s_warp, total) + sums[blk];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const long j = j0 + q;
      if (j >= n) continue;
      heads[j] = u;
      if (head[q]) {
        ukey[u] = k[q];
        ustart[u] = (int)j;
        const int c = (int)(k[q] / cls);
        const uint32_t p = q > 0 ? k[q > 0 ? q - 1 : 0] : prev;
        for (int w = j == 0 ? 0 : (int)(p / cls) + 1; w <= c; w++) bound[w] = u;
        u++;
      }
      if (j + 1 == n) {
        ustart[nu] = (int)n;
        for (int w = (int)(k[q] / cls) + 1; w <= 8; w++) bound[w] = nu;
      }
    }
  }
}

// The one addition a class makes to grid values.  A global float reduction
// takes operands and results below 2^-126 as 0; where the terms are 2^-101 and
// more that cannot show (a subnormal grid value is less than half a unit in
// their last place, and two such values that cancel leave 2^-125 or 0).  Smaller
// terms are added by load and store: no other lane adds to the value in this
// launch.
constexpr float kReduceFrom = 3.9443045e-31f;  // 2^-101
__device__ __forceinline__ void add_once(float *g, float a) {
  if (fabsf(a) >= kReduceFrom) atomicAdd(g, a);
  else if (a != 0.0f) *g += a;
}
__device__ __forceinline__ void add_once4(float *g, const float (&a)[4]) {
  const float lo = fminf(fminf(fabsf(a[0]), fabsf(a[1])), fminf(fabsf(a[2]), fabsf(a[3])));
  if (lo >= kReduceFrom) {
    red_add_f32x4(g, a[0], a[1], a[2], a[3]);
  } else {
    float4 *q = reinterpret_cast<float4 *>(g);
    const float4 v = *q;
    *q = make_float4(v.x + a[0], v.y + a[1], v.z + a[2], v.w + a[3]);
  }
}

// Cells of parity class cls.  A warp takes a stretch of the class's sorted
// records, cut at cell boundaries (the cells that start in the stretch), and
// walks it 16 records at a time: lanes 2 i and 2 i + 1 hold record i's two
// halves (its slot is loaded two steps, the record itself one step ahead), and
// shuffles hand it to the eight lanes that sum it.  Eight lanes sum records i =
// 0, 1, 2, 3 mod 4 each; C == 16: lane = (x corner, four channels), 4 corners x
// 4 channels of sums in registers; C == 3: lane = corner.  At the end of a cell
// the four partial sums meet by exchanging halves, a lane ends with one corner's
// four channels and adds them by a reduction: a voxel gets one addition per
// class, so their order cannot show.
//
// A warp per cell staged up to 32 per-sample records of its run through shared
// memory (12 or fewer of the lanes in use at mean run lengths of 6 to 12),
// after a pass that gathered the records into sorted order, and every CTA began
// with a binary search for the class's cells: 26.7 M samples in 12.7 M runs,
// 2.2 M cells of 4 x 256^3: 1.99 -> 0.89 ms for gather and classes; 2.2 M samples
// in 0.9 M runs, 0.36 M cells: 402 -> 162 us.
template <int C, bool TSDF>
__global__ void __launch_bounds__(256, 3) det_class_kernel(DetReduceParams q, int cls) {
  constexpr int NC = C == 16 ? 4 : 1, NV = C == 16 ? 4 : 3;  // a lane's corners, channels
  if (q.cnt[kDetCells] == 0) return;
  const int lo = q.bound[cls], hi = q.bound[cls + 1];
  if (lo == hi) return;
  const int lane = lane_id(), g = lane >> 3, l8 = lane & 7;
  const int h = l8 >> 2, ch = C == 16 ? 4 * (l8 & 3) : 0;  // x corner, first channel
  // the corner a lane adds at the end of a cell (C == 16), as bit and voxel offset
  const int D = q.keys.D, cr1 = C == 16 ? 4 * h + g : l8;
  const int at1 = ((cr1 >> 2) * D + ((cr1 >> 1) & 1)) * D + (cr1 & 1);
  // (a stretch's position may pass 2^31, no record's does)
  const long P0 = q.ustart[lo], P1 = q.ustart[hi];
  // one stretch a warp, or, where they are long, eight shorter ones a grid
  // apart: they take the warps unequal times (27 M samples 3.85 -> 3.73 ms a pass
  // and reduction; starting more CTAs instead cost 3 us a class on 2 M)
  const long warps = (long)gridDim.x * (blockDim.x >> 5), even = (P1 - P0 + warps - 1) / warps;
  // few records: still four a warp, as a stretch is one chain of loads and sums
  // (steps of 256 / 4096 / 9216 rays with the TSDF, at least 32 / 8 / 4 / 1: 339
  // / 280 / 270 / 261, 402 / 324 / 314 / 310, 414 / 338 / 331 / 329 us; at 65536
  // rays 465 / 420 / 420 / 420)
  const long Q = max(even > 256 ? (even + 7) / 8 : even, 4l);
  long pa = P0 + (((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * Q;
#pragma unroll 1
  for (; pa < P1; pa += warps * Q) {
    int u = __ldg(q.heads + pa);
    const int ub = pa + Q < P1 ? __ldg(q.heads + pa + Q) : hi;
    if (u >= ub) continue;
    uint32_t j = __ldg(q.ustart + u);
    const uint32_t end = __ldg(q.ustart + ub);
    // 32 cells at a time, one a lane: lower corner's voxel, corners inside, end
    int cvox = 0, cin = 0, cend = 0, ci = 0;
    auto load_cells = [&]() {
      if (u + lane < ub) {
        const uint32_t m = __ldg(q.ukey + u + lane) - (uint32_t)cls * q.keys.cls, e = (uint32_t)D + 1;
        cend = __ldg(q.ustart + u + lane + 1);
        const uint32_t xy = q.by_edge.div(m), x = q.by_edge.div(xy), b = q.by_edge.div(x);
        const int i0[3] = {(int)(x - b * e) - 1, (int)(xy - x * e) - 1, (int)(m - xy * e) - 1};
        cvox = (((int)b * D + i0[0]) * D + i0[1]) * D + i0[2];
        cin = (int)corners_inside(i0, D);
      }
      ci = 0;
    };
    load_cells();
    uint32_t ce = __shfl_sync(SG_FULL, cend, 0);
    float acc[NC][NV], acct[TSDF ? NC : 1];
#pragma unroll
    for (int c = 0; c < NC; c++) {
      if (TSDF) acct[c] = 0.0f;
#pragma unroll
      for (int v = 0; v < NV; v++) acc[c][v] = 0.0f;
    }
    const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    auto half = [&](const GradRecord *rec, uint32_t slot) {
      return __ldg(reinterpret_cast<const float4 *>(rec + slot) + (lane & 1));
    };
    const uint32_t i2 = lane >> 1;
    float4 fa = zero4, ft = zero4;
    uint32_t nslot = 0;
    int k = 0, nk = 0;
    if (j + i2 < end) {
      const uint32_t slot = __ldg(q.slot + j + i2);
      fa = half(q.rec, slot);
      if (TSDF) ft = half(q.rec_t, slot);
      k = q.rays.ray(slot);
    }
    if (j + 16 + i2 < end) nslot = __ldg(q.slot + j + 16 + i2);
    for (; j < end; j += 16) {
      float gv[4][NV];  // the rays' G rows
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const float *row = q.ray_g + (size_t)__shfl_sync(SG_FULL, k, 2 * (4 * t + g)) * C + ch;
        if (C == 16) {
          const float4 x = __ldg(reinterpret_cast<const float4 *>(row));
          gv[t][0] = x.x, gv[t][1] = x.y, gv[t][2] = x.z, gv[t][NV - 1] = x.w;
        } else {
#pragma unroll
          for (int v = 0; v < NV; v++) gv[t][v] = __ldg(row + v);
        }
      }
      float4 nfa = zero4, nft = zero4;
      if (j + 16 + i2 < end) {
        nfa = half(q.rec, nslot);
        if (TSDF) nft = half(q.rec_t, nslot);
        nk = q.rays.ray(nslot);
      }
      if (j + 32 + i2 < end) nslot = __ldg(q.slot + j + 32 + i2);
#pragma unroll
      for (int t = 0; t < 4; t++) {
        const int src = 2 * (4 * t + g) + h;
        float a[4] = {__shfl_sync(SG_FULL, fa.x, src), __shfl_sync(SG_FULL, fa.y, src), __shfl_sync(SG_FULL, fa.z, src),
                      __shfl_sync(SG_FULL, fa.w, src)};
        float at[4];
        if (TSDF) {
          at[0] = __shfl_sync(SG_FULL, ft.x, src), at[1] = __shfl_sync(SG_FULL, ft.y, src);
          at[2] = __shfl_sync(SG_FULL, ft.z, src), at[3] = __shfl_sync(SG_FULL, ft.w, src);
        }
        if (C == 3) {  // the lane's own corner
          a[0] = (l8 & 2) ? ((l8 & 1) ? a[3] : a[2]) : ((l8 & 1) ? a[1] : a[0]);
          if (TSDF) at[0] = (l8 & 2) ? ((l8 & 1) ? at[3] : at[2]) : ((l8 & 1) ? at[1] : at[0]);
        }
        const uint32_t r = j + 4 * t + g, past = min(j + 4 * t + 4, end);
        bool open = r < end;  // the lanes' record waits for its cell
        while (true) {
          if (open && r < ce) {
            open = false;
#pragma unroll
            for (int c = 0; c < NC; c++) {
              if (TSDF) acct[c] += at[c];
#pragma unroll
              for (int v = 0; v < NV; v++) acc[c][v] = __fmaf_rn(a[c], gv[t][v], acc[c][v]);
            }
          }
          if (ce > past) break;
          // the end of a cell
          __syncwarp();
          const int at0 = __shfl_sync(SG_FULL, cvox, ci), in = __shfl_sync(SG_FULL, cin, ci);
          const bool add = (in >> cr1) & 1;
          float *gp = q.grad_feat + (long)(at0 + at1) * C + ch;
          if constexpr (C == 16) {
            float s2[2][4], s1[4], t2[2], t1 = 0.0f;
#pragma unroll
            for (int c = 0; c < 2; c++) {
#pragma unroll
              for (int v = 0; v < 4; v++) {
                const float keep = (g & 2) ? acc[2 + c][v] : acc[c][v], send = (g & 2) ? acc[c][v] : acc[2 + c][v];
                s2[c][v] = keep + __shfl_xor_sync(SG_FULL, send, 16);
              }
              if (TSDF) {
                const float keep = (g & 2) ? acct[2 + c] : acct[c], send = (g & 2) ? acct[c] : acct[2 + c];
                t2[c] = keep + __shfl_xor_sync(SG_FULL, send, 16);
              }
            }
#pragma unroll
            for (int v = 0; v < 4; v++)
              s1[v] = ((g & 1) ? s2[1][v] : s2[0][v]) + __shfl_xor_sync(SG_FULL, (g & 1) ? s2[0][v] : s2[1][v], 8);
            if (TSDF) t1 = ((g & 1) ? t2[1] : t2[0]) + __shfl_xor_sync(SG_FULL, (g & 1) ? t2[0] : t2[1], 8);
            if (add) {
              add_once4(gp, s1);
              if (TSDF && (l8 & 3) == 0) add_once(q.grad_tsdf + (long)(at0 + at1), t1);
            }
          } else {
            float v[4] = {acc[0][0], acc[0][1], acc[0][NV - 1], TSDF ? acct[0] : 0.0f};
#pragma unroll
            for (int k = 0; k < (TSDF ? 4 : 3); k++) {
              v[k] += __shfl_xor_sync(SG_FULL, v[k], 16);
              v[k] += __shfl_xor_sync(SG_FULL, v[k], 8);
            }
            if (add) {  // lanes of the four groups: a channel each, the TSDF gradient
              if (g < 3) add_once(gp + g, g == 0 ? v[0] : (g == 1 ? v[1] : v[2]));
              else if (TSDF) add_once(q.grad_tsdf + (long)(at0 + at1), v[3]);
            }
          }
#pragma unroll
          for (int c = 0; c < NC; c++) {
            if (TSDF) acct[c] = 0.0f;
#pragma unroll
            for (int v = 0; v < NV; v++) acc[c][v] = 0.0f;
          }
          if (++u == ub) {
            ce = 0xffffffffu;  // the records are done
            break;
          }
          if (++ci == 32) load_cells();
          ce = __shfl_sync(SG_FULL, cend, ci);
        }
      }
      fa = nfa;
      ft = nft;
      k = nk;
    }
  }
}

// ---------------------------------------------------------------------------
// workspace
// ---------------------------------------------------------------------------
static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

size_t det_layout(long R, int nseg, int C, long cap, char *base, DetWork *w) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char *p = base ? base + off : nullptr;
    off += align256(bytes);
    return p;
  };
  DetWork d{};
  d.cnt = (int *)take(kDetCounters * sizeof(int));
  d.hitb = (int *)take((size_t)R * 4);
  d.hit_ray = (int *)take((size_t)R * 4);
  d.hit_slot = (int *)take((size_t)R * 4);
  d.seg_hit = (int *)take((size_t)(nseg + 1) * 4);
  d.seg_slot = (int *)take((size_t)(nseg + 1) * 4);
  d.ray_nrec = (int *)take((size_t)R * 4);
  d.ray_g = (float *)take((size_t)R * C * 4);
  d.rec_key = (uint32_t *)take((size_t)cap * 4);
  d.rec = (GradRecord *)take((size_t)cap * sizeof(GradRecord));
  d.rec_t = (GradRecord *)take((size_t)cap * sizeof(GradRecord));
  // one more than cap: after the sort, one of the pairs holds the distinct
  // cells' first positions and the end of the last run
  d.ka = (uint32_t *)take((size_t)(cap + 1) * 4);
  d.va = (uint32_t *)take((size_t)(cap + 1) * 4);
  d.kb = (uint32_t *)take((size_t)(cap + 1) * 4);
  d.vb = (uint32_t *)take((size_t)(cap + 1) * 4);
  d.sort_scratch = take(radix_scratch_bytes(cap));
  const size_t sc = scan_scratch_ints(R) > scan_scratch_ints(cap) ? scan_scratch_ints(R) : scan_scratch_ints(cap);
  d.scan_scratch = (int *)take(sc * 4);
  if (w) *w = d;
  return off;
}

static int grid_for(long n, int per_sm = 8) {
  long g = (n + 255) / 256;
  const long cap = (long)num_sms() * per_sm;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}

int launch_det_prepare(const DetWork &w, const SgRaySegments &seg, int S_max, const int *hit_count, long R,
                       long cap, const DetTrainOut &o, SgStatus *status, sg_stream_t stream) {
  det_ray_flags_kernel<<<grid_for(R), 256, 0, stream>>>(hit_count, R, w.hitb);
  launch_excl_scan(w.hitb, R, w.hitb, w.scan_scratch, w.cnt + kDetHits, stream);
  det_seg_kernel<<<1, 256, 0, stream>>>(seg, S_max, R, w.hitb, w.cnt, w.seg_hit, w.seg_slot, cap, status);
  det_ray_emit_kernel<<<grid_for(R), 256, 0, stream>>>(seg, S_max, R, hit_count, w.hitb, w.seg_hit, w.seg_slot,
                                                        w.hit_ray, w.hit_slot, o);
  SG_LAUNCH_CHECK();
  return SG_OK;
}

int launch_det_reduce(const DetWork &w, const RecordKeys &keys, const SgRaySegments &seg, int S_max, long R, long cap,
                      int C, float *grad_feat, float *grad_tsdf, sg_stream_t stream) {
  int key_bits = 1;
  while (key_bits < 32 && ((uint64_t)1 << key_bits) <= (uint64_t)keys.invalid) key_bits++;
  const int g = grid_for(cap, 16);
  // the records, compacted into the b pair (slot order kept): the rays'
  // record counts scanned in place into their first positions
  launch_excl_scan_dev(w.ray_nrec, R, w.cnt + kDetHits, w.ray_nrec, w.scan_scratch, w.cnt + kDetValid, stream);
  det_compact_kernel<<<grid_for(R * 16, 16), 256, 0, stream>>>(w.rec_key, w.cnt, w.ray_nrec, w.hit_slot, w.kb,
                                                                w.vb);
  const int passes = launch_radix_sort(w.kb, w.vb, w.cnt + kDetValid, cap, key_bits, w.ka, w.va, w.kb, w.vb,
                                       w.sort_scratch, stream);
  const uint32_t *skey = (passes & 1) ? w.ka : w.kb;
  const uint32_t *sval = (passes & 1) ? w.va : w.vb;
  // the other pair is free now: the scan over the run heads in one buffer,
  // the distinct cells' first positions in the other
  int *heads = (int *)((passes & 1) ? w.kb : w.ka);
  int *ustart = (int *)((passes & 1) ? w.vb : w.va);
  int *bound = (int *)w.sort_scratch;  // free behind the sort
  det_head_sums_kernel<<<g, 256, 0, stream>>>(skey, w.cnt, w.scan_scratch);
  launch_scan_sums(w.scan_scratch, cap, w.cnt + kDetValid, w.cnt + kDetCells, stream);
  det_cells_kernel<<<g, 256, 0, stream>>>(skey, w.scan_scratch, w.cnt, keys.cls, w.rec_key, ustart, heads, bound);
  DetReduceParams q{keys, FixedDiv31::of((uint32_t)keys.D + 1),
                    SlotRays{w.seg_slot, w.seg_hit, seg.samples, seg.count, S_max},
                    w.cnt, w.rec_key, ustart, heads, bound, sval, w.rec, w.rec_t, w.ray_g, grad_feat, grad_tsdf};
  for (int cls = 0; cls < 8; cls++) {
    const dim3 g(num_sms() * 3), blk(256);
    if (C == 16) {
      if (grad_tsdf) det_class_kernel<16, true><<<g, blk, 0, stream>>>(q, cls);
      else det_class_kernel<16, false><<<g, blk, 0, stream>>>(q, cls);
    } else {
      if (grad_tsdf) det_class_kernel<3, true><<<g, blk, 0, stream>>>(q, cls);
      else det_class_kernel<3, false><<<g, blk, 0, stream>>>(q, cls);
    }
  }
  SG_LAUNCH_CHECK();
  return SG_OK;
}

}  // namespace sg
