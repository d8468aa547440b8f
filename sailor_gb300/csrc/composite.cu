// composite.cu -- volume-rendering compositing and its adjoints on sm_103a.
//
// Replaces volume_rendering.cu (SAILOR c_lib/VoxelEncoding/src):
//   volume_rendering_training_forward_kernel :17-126 (density),
//   volume_rendering_occ_training_forward_kernel :129-240 (occupancy),
//   volume_rendering_occ_kernel :666-745 (pre-sorted occupancy),
//   volume_rendering_training_backward_kernel :244-381 and the occupancy
//   backward :384-522.
//
// One warp per ray.  The sorted positions are taken in blocks of 32, front to
// back: alpha in parallel, transmittance carried in strict sequential order
// through the block (bit-identical to the reference's serial T *= 1 - alpha,
// and so is the early-termination decision T < t_thres), weights; the walk
// stops at the block in which the ray ends, so densities and features behind
// it are not read.  Features are read, and feature gradients written, by row
// groups: the lanes that together hold a sample's row (vectors of 4, 2 or 1
// floats) take 32 / lanes samples at a time, so accesses cover whole rows
// (three channels or fewer: a lane per sample).
//
// The backward recomputes alpha and transmittance from the inputs and the
// per-ray outputs (no per-sample state is saved).  Its feature terms need only
// the scalar s_i = g . f_i of each sample: sum_c g_c (T f_ic - (F_c - P_ic)) =
// T s_i - (g . F - prefix of w s), so one scan takes the place of one per
// channel and no feature is kept.  exact == 0 reproduces the reference's
// gradient formula; exact == 1 is the true derivative of the forward (the
// reference adds g_ws*(1-ws) four extra times and drops the sample that
// triggers early termination).
//
// 131072 rays x 96 samples x 16 channels, rays ending within: forward 0.40 ->
// 0.18 ms, adjoint 1.93 (202 registers, 12 % of the warps) -> 0.33 ms.
#include "ray_core.cuh"

namespace sg {

constexpr int kMaxC = 32;     // forward: FastNerf composites 30 channels (infer_mlp.cu:508-580)
constexpr int kMaxCBwd = 16;  // adjoint (no inference-only caller needs more)

struct CompParams {
  const float *z;
  const int *sort_idx;
  const float *sigma, *feats;
  long R;
  int S, C;
  float t_thres;
  int mode;
  // forward outputs / backward saved outputs
  float *of, *od, *ows, *oa;
  // backward
  const float *g_feat, *g_depth, *g_ws, *g_alpha;
  int exact;
  float *grad_feats, *grad_sigma;
  int lanes;  // lanes of a feature row (row groups)
};

// One block of a ray's sorted positions.
struct CompBlock {
  int s;  // the lane's sample (index in the ray's row), -1: none
  float z, al, dl, tb, w;
  bool used, post;  // counts; and the transmittance after it is >= t_thres
};

struct CompWalk {
  float T;
  int m0, end;  // first position with a sample (-1: not met); positions from end on are past the termination
};

// Depths of the sorted positions into shared memory; false for an invalid ray.
template <bool ONE>
__device__ __forceinline__ bool comp_load(const CompParams &p, size_t rb, float *s_z, int *s_i) {
  const int lane = lane_id(), S = p.S;
  const int last = p.sort_idx ? __ldg(p.sort_idx + rb + S - 1) : S - 1;
  if (__ldg(p.z + rb + last) < 0) return false;
  if (ONE) {
    if (lane < S) s_z[lane] = __ldg(p.z + rb + (p.sort_idx ? __ldg(p.sort_idx + rb + lane) : lane));
  } else {
    for (int i = lane; i < S; i += 32) {
      const int s = p.sort_idx ? __ldg(p.sort_idx + rb + i) : i;
      s_i[i] = s;
      s_z[i] = __ldg(p.z + rb + s);
    }
  }
  __syncwarp();
  return true;
}

template <bool ONE>
__device__ __forceinline__ bool comp_block(const CompParams &p, size_t rb, int e, const float *s_z, const int *s_i, float *s_f,
                                           CompWalk &wk, CompBlock &v) {
  const int lane = lane_id(), i = e * 32 + lane, S = p.S;
  v.z = i < S ? s_z[i] : -1.0f;
  v.s = -1;
  v.al = v.dl = v.w = 0.0f;
  v.used = v.post = false;
  const bool valid = v.z >= 0.0f;
  const unsigned vb = __ballot_sync(SG_FULL, valid);
  if (i < S) v.s = ONE ? (p.sort_idx ? __ldg(p.sort_idx + rb + i) : i) : s_i[i];
  if (vb == 0u) return false;
  if (wk.m0 < 0) wk.m0 = e * 32 + __ffs(vb) - 1;
  if (valid) {
    const float sg = __ldg(p.sigma + rb + v.s);
    if (p.mode == 0) {
      v.dl = depth_step(s_z, S, i, v.z);
      v.al = 1.0f - expf(-sg * v.dl);
    } else {
      v.al = sg;
    }
  }
  const int stop = block_transmittance<32>(valid ? 1.0f - v.al : 1.0f, wk.T, p.t_thres, wk.m0 - e * 32, S - e * 32, s_f, v.tb);
  if (stop < 32) wk.end = e * 32 + stop + 1;
  v.used = valid && i < wk.end;
  v.post = v.used && lane != stop;
  if (v.used) v.w = v.al * v.tb;
  return true;
}

template <int V> struct RowVec;
template <> struct RowVec<1> {
  float v[1];
  __device__ __forceinline__ void load(const float *p) { v[0] = __ldg(p); }
  __device__ __forceinline__ void zero() { v[0] = 0.0f; }
  __device__ __forceinline__ void store(float *p) const { *p = v[0]; }
};
template <> struct RowVec<2> {
  float v[2];
  __device__ __forceinline__ void load(const float *p) {
    const float2 a = __ldg(reinterpret_cast<const float2 *>(p));
    v[0] = a.x, v[1] = a.y;
  }
  __device__ __forceinline__ void zero() { v[0] = v[1] = 0.0f; }
  __device__ __forceinline__ void store(float *p) const { *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]); }
};
template <> struct RowVec<4> {
  float v[4];
  __device__ __forceinline__ void load(const float *p) {
    const float4 a = __ldg(reinterpret_cast<const float4 *>(p));
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
  }
  __device__ __forceinline__ void zero() { v[0] = v[1] = v[2] = v[3] = 0.0f; }
  __device__ __forceinline__ void store(float *p) const {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};

constexpr int kMaxPos = 128;  // sorted positions of a ray
constexpr int kAhead = 4;     // row loads in flight a lane

// V: floats a lane holds of a row (4, 2, 1), p.lanes lanes (a power of two) per
// row; V == 0: a lane per sample, C <= 3.
// OPT, V == 0: at most 32 positions (the loops over blocks go: 16.8 M samples of
// three channels, 32 a ray, 123 -> 98 us).  OPT, V > 0: a block's rows take more
// than kAhead steps; their sums are added in pairs and per block, so that the
// error stays that of a sum over the lanes of a warp.
template <int V, bool OPT>
__global__ void __launch_bounds__(256, 6) composite_fwd_kernel(CompParams p) {
  __shared__ float s_zall[8][kMaxPos];
  __shared__ int s_iall[8][V == 0 && OPT ? 1 : kMaxPos];
  __shared__ __align__(16) float s_fall[8][64];
  const int lane = lane_id();
  float *s_z = s_zall[threadIdx.x >> 5];
  float *s_f = s_fall[threadIdx.x >> 5];
  int *s_i = s_iall[threadIdx.x >> 5];
  const int C = p.C, S = p.S;
  constexpr int N = V ? V : 3;
  constexpr bool ONE = V == 0 && OPT, LONG = V > 0 && OPT;
  const int L = p.lanes, c0 = V ? (lane & (L - 1)) * V : 0;  // the lane's channels
  const bool own = V && c0 < C;
  for (long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < p.R;
       r += ((long)gridDim.x * blockDim.x) >> 5) {
    const size_t rb = (size_t)r * S;
    float acc[N];
#pragma unroll
    for (int c = 0; c < N; c++) acc[c] = 0.0f;
    float d = 0.0f, ws = 0.0f, aa = 0.0f;
    const bool ok = comp_load<ONE>(p, rb, s_z, s_i);
    if (ok) {
      CompWalk wk{1.0f, -1, S};
#pragma unroll 1
      for (int e = 0; ONE ? e < 1 : e * 32 < wk.end; e++) {
        CompBlock v;
        if (!comp_block<ONE>(p, rb, e, s_z, s_i, s_f, wk, v)) continue;
        if (v.used) {
          d += v.w * v.z;
          ws += v.w;
          aa += v.w * v.al;
        }
        if constexpr (V == 0) {
          if (v.used) {
            const float *f = p.feats + (rb + v.s) * C;
#pragma unroll
            for (int c = 0; c < 3; c++)
              if (c < C) acc[c] += v.w * __ldg(f + c);
          }
        } else {
          const unsigned ub = __ballot_sync(SG_FULL, v.used);
          // up to kAhead row loads in flight
          float prev[N], part[N];
#pragma unroll
          for (int c = 0; c < N; c++) part[c] = 0.0f;
          for (int it = 0; it < L; it += kAhead) {
            RowVec<N> f[kAhead];
            float w[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
              const int src = ((it + u) * (32 / L) + lane / L) & 31;
              w[u] = __shfl_sync(SG_FULL, v.w, src);
              const int s = __shfl_sync(SG_FULL, v.s, src);
              const bool on = own && it + u < L && ((ub >> src) & 1u);
              if (on) f[u].load(p.feats + (rb + s) * C + c0);
              else f[u].zero(), w[u] = 0.0f;
            }
            static_assert(kAhead == 4, "two pairs");
#pragma unroll
            for (int c = 0; c < N; c++) {
              const float x = __fmaf_rn(w[0], f[0].v[c], w[1] * f[1].v[c]) + __fmaf_rn(w[2], f[2].v[c], w[3] * f[3].v[c]);
              if (!LONG) acc[c] += x;
              else if (it & kAhead) part[c] += prev[c] + x;
              else prev[c] = x;
            }
          }
          if (LONG) {
#pragma unroll
            for (int c = 0; c < N; c++) acc[c] += part[c];
          }
        }
      }
    }
    if constexpr (V == 0) {
      // totals of 8 values at once: value k ends on lane 4 k
      float v[8] = {d, ws, aa, acc[0], acc[1], acc[2], 0.0f, 0.0f};
      if (ok) warp_sum8(v);
      const int k = lane >> 2;
      if ((lane & 3) == 0 && k < 3 + C) {
        if (k >= 3) p.of[(size_t)r * C + k - 3] = v[0];
        else (k == 0 ? p.od : k == 1 ? p.ows : p.oa)[r] = v[0];
      }
    } else {
      d = warp_sum(d);
      ws = warp_sum(ws);
      aa = warp_sum(aa);
      for (int o = L; o < 32; o <<= 1) {  // over the row groups
#pragma unroll
        for (int c = 0; c < N; c++) acc[c] += __shfl_xor_sync(SG_FULL, acc[c], o);
      }
      if (lane == 0) {
        p.od[r] = d;
        p.ows[r] = ws;
        p.oa[r] = aa;
      }
      if (own && lane < L) {
#pragma unroll
        for (int c = 0; c < N; c++) p.of[(size_t)r * C + c0 + c] = acc[c];
      }
    }
    __syncwarp();
  }
}

// Per position, for the second pass of the adjoint (shared memory).
struct CompKeep {
  float w[kMaxPos], al[kMaxPos], tb[kMaxPos], dl[kMaxPos], s[kMaxPos];
  int idx[kMaxPos];  // sample, with bit 30: counts, bit 31: its gradient is written
};

// CTAs an SM 4 / 5 / 6 (131072 rays x 96): 3 channels 174 / 156 / 158 us, 5 channels
// 334 / 315 / 315, 16 channels 270 / 264 / 283.
template <int V>
__global__ void __launch_bounds__(256, 5) composite_bwd_kernel(CompParams p) {
  extern __shared__ __align__(16) unsigned char s_comp[];
  const int lane = lane_id(), w8 = threadIdx.x >> 5;
  float *s_z = reinterpret_cast<float *>(s_comp) + w8 * (kMaxPos + 64);
  float *s_f = s_z + kMaxPos;
  CompKeep &kp = reinterpret_cast<CompKeep *>(s_comp + 8 * (kMaxPos + 64) * sizeof(float))[w8];
  const int C = p.C, S = p.S;
  constexpr int N = V ? V : 3;
  const int L = p.lanes, c0 = V ? (lane & (L - 1)) * V : 0;
  const bool own = V && c0 < C;
  constexpr int kUse = 1 << 30;
  constexpr int kWrite = (int)0x80000000u;
  for (long r = ((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < p.R;
       r += ((long)gridDim.x * blockDim.x) >> 5) {
    const size_t rb = (size_t)r * S;
    int e1 = 0;  // blocks [0, e1) were evaluated
    float gc[N];
#pragma unroll
    for (int c = 0; c < N; c++) gc[c] = (V ? own : c < C) ? __ldg(p.g_feat + (size_t)r * C + c0 + c) : 0.0f;
    const float gws = __ldg(p.g_ws + r), gd = __ldg(p.g_depth + r), ga = __ldg(p.g_alpha + r);
    const bool ok = comp_load<false>(p, rb, s_z, kp.idx);  // an invalid ray has no gradient (the reference leaves its zero fill)
    // totals over the samples: w s, w z, w, w alpha
    float Fs = 0.0f, Fd = 0.0f, Fw = 0.0f, Fa = 0.0f;
    if (ok) {
      CompWalk wk{1.0f, -1, S};
#pragma unroll 1
      for (; e1 * 32 < wk.end; e1++) {
        CompBlock v;
        const int i = e1 * 32 + lane;
        const bool any = comp_block<false>(p, rb, e1, s_z, kp.idx, s_f, wk, v);
        float sv = 0.0f;  // g . features of the lane's sample
        if (any) {
          if constexpr (V == 0) {
            if (v.used) {
              const float *f = p.feats + (rb + v.s) * C;
#pragma unroll
              for (int c = 0; c < 3; c++)
                if (c < C) sv = __fmaf_rn(gc[c], __ldg(f + c), sv);
            }
          } else {
            const unsigned ub = __ballot_sync(SG_FULL, v.used);
            for (int it = 0; it < L; it += kAhead) {
              RowVec<N> f[kAhead];
#pragma unroll
              for (int u = 0; u < kAhead; u++) {
                const int src = ((it + u) * (32 / L) + lane / L) & 31;
                const int s = __shfl_sync(SG_FULL, v.s, src);
                if (own && it + u < L && ((ub >> src) & 1u)) f[u].load(p.feats + (rb + s) * C + c0);
                else f[u].zero();
              }
#pragma unroll
              for (int u = 0; u < kAhead; u++) {
                if (it + u >= L) break;
                float a = 0.0f;
#pragma unroll
                for (int c = 0; c < N; c++) a = __fmaf_rn(gc[c], f[u].v[c], a);
                for (int o = 1; o < L; o <<= 1) a += __shfl_xor_sync(SG_FULL, a, o);
                // lane src0 + k of the block takes the sum of row group k
                const int src0 = (it + u) * (32 / L);
                const float t = __shfl_sync(SG_FULL, a, ((lane - src0) * L) & 31);
                if (lane >= src0 && lane < src0 + 32 / L) sv = t;
              }
            }
          }
        }
        kp.w[i] = v.w;
        kp.al[i] = v.al;
        kp.tb[i] = any ? v.tb : 0.0f;
        kp.dl[i] = v.dl;
        kp.s[i] = sv;
        kp.idx[i] = v.s < 0 ? -1 : (v.s | (v.used ? kUse : 0) | ((p.exact ? v.used : v.post) ? kWrite : 0));
        if (any) {
          Fs += warp_sum_scan_order(v.w * sv);
          Fd += warp_sum_scan_order(v.w * v.z);
          Fw += warp_sum_scan_order(v.w);
          Fa += warp_sum_scan_order(v.w * v.al);
        }
      }
      if (!p.exact) {  // the reference's formula reads the saved outputs
        Fd = __ldg(p.od + r);
        Fw = __ldg(p.ows + r);
        Fa = __ldg(p.oa + r);
        float a = 0.0f;
        if constexpr (V == 0) {
#pragma unroll
          for (int c = 0; c < 3; c++)
            if (c < C) a = __fmaf_rn(gc[c], __ldg(p.of + (size_t)r * C + c), a);
        } else {
          if (own) {
#pragma unroll
            for (int c = 0; c < N; c++) a = __fmaf_rn(gc[c], __ldg(p.of + (size_t)r * C + c0 + c), a);
          }
          for (int o = 1; o < L; o <<= 1) a += __shfl_xor_sync(SG_FULL, a, o);
        }
        Fs = a;
      }
      __syncwarp();
    }
    float rs = 0.0f, rd = 0.0f, rw = 0.0f, ra = 0.0f;  // running totals
    for (int e = 0; e * 32 < S; e++) {
      const int i = e * 32 + lane;
      float gsig = 0.0f, wv = 0.0f;
      int s = -1;
      if (e < e1) {
        const int id = i < S ? kp.idx[i] : -1;
        s = id == -1 ? -1 : (id & 0x3fffffff);
        const bool use = id != -1 && (id & kUse), wr = id != -1 && (id & kWrite);
        if (__any_sync(SG_FULL, use)) {
          const float w = kp.w[i], al = kp.al[i], sv = kp.s[i], z = i < S ? s_z[i] : 0.0f;
          const float vs = warp_incl_scan_f(w * sv), vd = warp_incl_scan_f(w * z), vw = warp_incl_scan_f(w),
                      va = warp_incl_scan_f(w * al);
          if (wr) {
            const float tb = kp.tb[i], Ta = tb * (1.0f - al);  // transmittance before and after the sample
            // sums over the samples behind this one
            const float ss = Fs - (rs + vs), sd = Fd - (rd + vd), sw = Fw - (rw + vw), sa = Fa - (ra + va);
            if (p.mode == 0) {
              gsig = gws * (Ta - sw) + gd * (Ta * z - sd) + ga * (2.0f * Ta * al - sa) + (Ta * sv - ss);
              if (!p.exact) gsig += 4.0f * (gws * (1.0f - Fw));
              gsig *= kp.dl[i];
            } else if (!p.exact) {
              const float tmp = (1.0f / (1.0f - al + 1e-7f) <= 15.0f) ? 1.0f / (1.0f - al) : 15.0f;
              gsig = (gws * (Ta - sw) + gd * (Ta * z - sd) + ga * (2.0f * Ta * al - sa) + (Ta * sv - ss)) * tmp;
            } else {
              const float om = 1.0f - al, inv = om != 0.0f ? 1.0f / om : 0.0f;
              gsig = gws * (tb - sw * inv) + gd * (tb * z - sd * inv) + ga * (2.0f * al * tb - sa * inv) +
                     (tb * sv - ss * inv);
            }
            wv = w;
          }
          rs += __shfl_sync(SG_FULL, vs, 31);
          rd += __shfl_sync(SG_FULL, vd, 31);
          rw += __shfl_sync(SG_FULL, vw, 31);
          ra += __shfl_sync(SG_FULL, va, 31);
        }
      } else if (i < S) {
        s = ok && p.sort_idx ? __ldg(p.sort_idx + rb + i) : i;
      }
      if (s >= 0) p.grad_sigma[rb + s] = gsig;
      if constexpr (V == 0) {
        if (s >= 0) {
#pragma unroll
          for (int c = 0; c < 3; c++)
            if (c < C) p.grad_feats[(rb + s) * C + c] = gc[c] * wv;
        }
      } else {
        for (int it = 0; it < L; it++) {
          const int src = it * (32 / L) + lane / L;
          const float w = __shfl_sync(SG_FULL, wv, src);
          const int sj = __shfl_sync(SG_FULL, s, src);
          if (own && sj >= 0) {
            RowVec<N> g;
#pragma unroll
            for (int c = 0; c < N; c++) g.v[c] = gc[c] * w;
            g.store(p.grad_feats + (rb + sj) * C + c0);
          }
        }
      }
    }
    __syncwarp();
  }
}

constexpr size_t kBwdSmem = 8 * ((kMaxPos + 64) * sizeof(float) + sizeof(CompKeep));

template <int V>
static int launch_comp(const CompParams &p, bool bwd, sg_stream_t stream) {
  int g = ceil_div(p.R * 32, 256);
  if (g > num_sms() * 64) g = num_sms() * 64;
  if (bwd) composite_bwd_kernel<V><<<g, 256, kBwdSmem, stream>>>(p);
  else if (V == 0 ? p.S <= 32 : p.lanes > kAhead) composite_fwd_kernel<V, true><<<g, 256, 0, stream>>>(p);
  else composite_fwd_kernel<V, false><<<g, 256, 0, stream>>>(p);
  return SG_OK;
}

}  // namespace sg

using namespace sg;

static int comp_dispatch(CompParams p, bool bwd, sg_stream_t stream) {
  if (p.S > kMaxPos) return SG_ERR_UNSUPPORTED;
  // floats a lane takes of a row: as many as the channel count and the
  // addresses allow; up to three channels a lane takes a sample
  const uintptr_t at = (uintptr_t)p.feats | (bwd ? (uintptr_t)p.grad_feats : 0);
  const int v = p.C <= 3 ? 0 : (p.C % 4 == 0 && at % 16 == 0 ? 4 : (p.C % 2 == 0 && at % 8 == 0 ? 2 : 1));
  p.lanes = 1;
  if (v)
    while (p.lanes * v < p.C) p.lanes <<= 1;
  int rc;
  if (v == 4) rc = launch_comp<4>(p, bwd, stream);
  else if (v == 2) rc = launch_comp<2>(p, bwd, stream);
  else if (v == 1) rc = launch_comp<1>(p, bwd, stream);
  else rc = launch_comp<0>(p, bwd, stream);
  if (rc != SG_OK) return rc;
  SG_LAUNCH_CHECK();
  return SG_OK;
}

extern "C" int sg_composite_fwd(const float *z, const int *sort_idx, const float *sigma, const float *feats,
                                int R, int S, int C, float t_thres, int mode, float *out_feat,
                                float *out_depth, float *out_ws, float *out_alpha, sg_stream_t stream) {
  if (!z || !sigma || !feats || !out_feat || !out_depth || !out_ws || !out_alpha) return SG_ERR_INVALID_ARG;
  if (R < 0 || S <= 0 || C <= 0 || C > kMaxC || (mode != 0 && mode != 1)) return SG_ERR_INVALID_ARG;
  if (R == 0) return SG_OK;
  CompParams p{};
  p.z = z;
  p.sort_idx = sort_idx;
  p.sigma = sigma;
  p.feats = feats;
  p.R = R;
  p.S = S;
  p.C = C;
  p.t_thres = t_thres;
  p.mode = mode;
  p.of = out_feat;
  p.od = out_depth;
  p.ows = out_ws;
  p.oa = out_alpha;
  return comp_dispatch(p, false, stream);
}

extern "C" int sg_composite_bwd(const float *g_feat, const float *g_depth, const float *g_ws,
                                const float *g_alpha, const float *o_feat, const float *o_depth,
                                const float *o_ws, const float *o_alpha, const float *z, const int *sort_idx,
                                const float *sigma, const float *feats, int R, int S, int C, float t_thres,
                                int mode, int exact, float *grad_feats, float *grad_sigma,
                                sg_stream_t stream) {
  if (!g_feat || !g_depth || !g_ws || !g_alpha || !z || !sigma || !feats || !grad_feats || !grad_sigma)
    return SG_ERR_INVALID_ARG;
  if (!exact && (!o_feat || !o_depth || !o_ws || !o_alpha)) return SG_ERR_INVALID_ARG;
  if (R < 0 || S <= 0 || C <= 0 || C > kMaxCBwd || (mode != 0 && mode != 1)) return SG_ERR_INVALID_ARG;
  if (R == 0) return SG_OK;
  CompParams p{};
  p.z = z;
  p.sort_idx = sort_idx;
  p.sigma = sigma;
  p.feats = feats;
  p.R = R;
  p.S = S;
  p.C = C;
  p.t_thres = t_thres;
  p.mode = mode;
  p.of = const_cast<float *>(o_feat);
  p.od = const_cast<float *>(o_depth);
  p.ows = const_cast<float *>(o_ws);
  p.oa = const_cast<float *>(o_alpha);
  p.g_feat = g_feat;
  p.g_depth = g_depth;
  p.g_ws = g_ws;
  p.g_alpha = g_alpha;
  p.exact = exact;
  p.grad_feats = grad_feats;
  p.grad_sigma = grad_sigma;
  return comp_dispatch(p, true, stream);
}
