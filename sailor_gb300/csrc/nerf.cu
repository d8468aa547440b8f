// nerf.cu -- FastNerf's occupancy (density) network on the sm_103a tensor
// cores (tcgen05.mma kind::f16, float32 accumulators in tensor memory).
//
// Replaces (SAILOR c_lib/FastNerf/src/infer_mlp.cu):
//   density_feat_kernel  :120-199  per point-view: feature MLP 18->64->64->64->64
//                                  and geometry MLP 18->16->8 (ReLU after each)
//   density_sigma_kernel :202-240  per point: 64->64->64->1, ReLU, ReLU, sigmoid
//   infer_density_mlp    :583-636  the two around a torch.mean over the views
//
// The reference runs one thread per point-view with scalar __hfma chains
// (float16 accumulation rounded at every product).  Here a persistent CTA of
// four warpgroups per SM holds the weights in shared memory once, and each
// warpgroup runs tiles of its own; a tile is 128 rows, P = floor(128 / V)
// points x V views (row v*P + p), so the view mean happens inside the CTA and
// no per-view feature reaches HBM:
//   inputs (z, t_psdf, 16 geometry features) -> float16 rows in shared memory
//   (the next tile's inputs are loaded into registers while the current one
//   runs through the layers);
//   each layer: one thread of the warpgroup issues tcgen05.mma (K-major
//   float16 operands in shared memory) into tensor memory and commits to the
//   warpgroup's mbarrier; the warpgroup then reads its rows back
//   (tcgen05.ld, one row per thread), adds the bias in float32, rounds to
//   float16 and applies ReLU into the next operand tile;
//   after the fourth feature layer the P point rows take the float32 mean of
//   their V view rows (view order, times 1/V, as torch's mean does here), all
//   threads sharing the work, into the sigma layers' operand tile;
//   the sigma layers run once that tile holds the points of up to
//   floor(128 / P) feature tiles (a batch), so they run on full tiles; the
//   last 64->1 layer is a per-row dot product in the epilogue, rounded to
//   float16 before the sigmoid as the reference rounds it.
// Layer outputs are rounded to float16 at the same points as the reference;
// within a layer the products are summed in float32 instead of rounding each
// partial sum to float16, so results differ from the reference by the
// reference's own accumulation error (a few float16 ulps).
//
// Bound by the layers' dependent chain (issue, commit, wait, tensor-memory
// load, epilogue) with four chains an SM to hide it, and by the epilogues'
// instructions.  4.2 M points x 3 views: 1.68 -> 0.93 ms (N = 1000: 31 -> 17
// us), by: sigma layers on batches, the view mean shared by all threads and
// one barrier less per layer 1.25; epilogues as fragments (see epilogue_frag)
// 1.03; descriptors in uniform registers, 32-bit index arithmetic 1.01; a
// fifth warpgroup in the room of the geometry network where its output is
// not wanted 0.93.
//
// Every mbarrier wait has an iteration limit: on expiry the kernel sets
// *error, finishes its batch without waiting again, takes no more, frees its
// tensor memory and returns.
#include <cuda_fp16.h>

#include "common.cuh"
#include "tc05.cuh"

namespace sg {

constexpr int kNerfParamCount = 22521;
constexpr int kSigmaOff = 13696, kGeoOff = 22081;

// Tiles in flight per CTA, one warpgroup each: what shared memory holds beside
// the weights, with and without the geometry network.
template <bool GEO>
constexpr int kNerfTiles = GEO ? 4 : 5;
constexpr uint32_t kNerfTmemCols = 512;  // tile t: features [64 t, 64 t + 64), geometry [320 + 16 t, ...)
constexpr int kGeoCol = 320;
constexpr long kNerfWaitIters = 1L << 24;

// Weights and operand tiles of the geometry network (only where its output
// is wanted: nothing else reads it).
template <bool GEO>
struct NerfGeoSmem {
  alignas(128) uint8_t w1[16 * 32 * 2];  // 18 -> 16, K padded to 32
  alignas(128) uint8_t w2[16 * 16 * 2];  // 16 -> 8, N padded to 16
  alignas(128) uint8_t h[kNerfTiles<GEO>][128 * 16 * 2];  // hidden rows
  alignas(16) float b1[80], b2[8];
};
template <>
struct NerfGeoSmem<false> {};

template <bool GEO>
struct NerfSmem {
  // weights [out][in] in the K-major float16 operand layout
  alignas(128) uint8_t w1[64 * 32 * 2];   // 18 -> 64, K padded to 32
  alignas(128) uint8_t w2[64 * 64 * 2];
  alignas(128) uint8_t w3[64 * 64 * 2];
  alignas(128) uint8_t w4[64 * 64 * 2];
  alignas(128) uint8_t ws1[64 * 64 * 2];
  alignas(128) uint8_t ws2[64 * 64 * 2];
  // per tile: hidden rows (the input rows, K = 32, lie over their first half
  // until the first layer has read them), and the points' view means
  alignas(128) uint8_t h[kNerfTiles<GEO>][128 * 64 * 2];
  alignas(128) uint8_t m[kNerfTiles<GEO>][128 * 64 * 2];
  NerfGeoSmem<GEO> geo;
  alignas(16) float b1[80], b2[80], b3[80], b4[80], bs1[80];  // fragment order
  alignas(16) float bs2[64], ws3[64];
  float bs3;
  alignas(8) uint64_t mbar[kNerfTiles<GEO>];  // one per warpgroup
  int fail[kNerfTiles<GEO>];
  uint32_t tmem_slot;
};

// barrier of one warpgroup (named barrier 1 + t, 128 threads)
__device__ __forceinline__ void wg_sync(int t) {
  asm volatile("bar.sync %0, 128;" ::"r"(t + 1) : "memory");
}

__device__ __forceinline__ float h2f(__half h) { return __half2float(h); }

// W [n_out][n_in] float16 at params + off -> rows n < n_rows, k < K of the
// operand tile (zero padding); 16 bytes at a time where rows are whole vectors
template <int n_in, int n_out, int n_rows, int K>
__device__ __forceinline__ void stage_weights(uint8_t *dst, const __half *params, int off) {
  if (n_in == K && n_out == n_rows && n_in % 8 == 0 && ((uintptr_t)(params + off)) % 16 == 0) {
    for (int i = threadIdx.x; i < n_rows * (K / 8); i += (int)blockDim.x) {
      const int n = i / (K / 8), k8 = i % (K / 8);
      *reinterpret_cast<uint4 *>(dst + tc::kmaj_offset(n, k8 * 8, K)) =
          __ldg(reinterpret_cast<const uint4 *>(params + off) + i);
    }
    return;
  }
  for (int i = threadIdx.x; i < n_rows * K; i += (int)blockDim.x) {
    const int n = i / K, k = i % K;
    const __half v = (n < n_out && k < n_in) ? params[off + n * n_in + k] : __float2half(0.0f);
    *reinterpret_cast<__half *>(dst + tc::kmaj_offset(n, k, K)) = v;
  }
}

__device__ void stage_bias(float *dst, const __half *params, int off, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = h2f(params[off + i]);
}

__device__ __forceinline__ uint32_t pack_half2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);  // one cvt.rn.f16x2.f32
  return *reinterpret_cast<const uint32_t *>(&h);
}

// The reference's relu of a float16 value: max(float(half), 0) back to half
// (NaN -> 0): max.f16x2 returns the operand that is a number.
__device__ __forceinline__ uint32_t relu_half2(uint32_t x) {
  const __half2 h = __hmax2(*reinterpret_cast<const __half2 *>(&x), __half2half2(__ushort_as_half(0)));
  return *reinterpret_cast<const uint32_t *>(&h);
}

// a + b, rounded to float16, ReLU; two values in one word (paired additions:
// add.rn.f32x2 rounds as two add.rn.f32)
__device__ __forceinline__ uint32_t bias_relu_half2(float x, float y, unsigned long long bias) {
  float u, v;
  asm("{\n\t.reg .b64 a, d;\n\tmov.b64 a, {%2, %3};\n\tadd.rn.f32x2 d, a, %4;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(u), "=f"(v)
      : "f"(x), "f"(y), "l"(bias));
  return relu_half2(pack_half2(u, v));
}

// 8 values + bias (shared memory, 16-byte aligned) -> one 16-byte vector
__device__ __forceinline__ uint4 bias_relu8(const float *v, const float *bias) {
  const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(bias);
  const ulonglong2 b1 = *reinterpret_cast<const ulonglong2 *>(bias + 4);
  return make_uint4(bias_relu_half2(v[0], v[1], b0.x), bias_relu_half2(v[2], v[3], b0.y),
                    bias_relu_half2(v[4], v[5], b1.x), bias_relu_half2(v[6], v[7], b1.y));
}

// Biases of a hidden layer, in the fragments' order: the values of columns
// 8 k + 2 c and the next one, k ascending, lie together for each c = 0 .. 3
// (lane % 4), 80 bytes apart so that the four runs meet no common bank.
constexpr int kFragBias = 20;
__device__ __forceinline__ void stage_bias_frag(float *dst, const __half *params, int off, int n) {
  for (int i = threadIdx.x; i < n; i += (int)blockDim.x)
    dst[((i >> 1) & 3) * kFragBias + (i >> 3) * 2 + (i & 1)] = h2f(params[off + i]);
}

// Hidden rows of a warp: 32 rows x 8 KG accumulator columns -> bias, float16,
// ReLU -> its rows of a K-major operand tile with 8 KG columns.  As fragments a
// lane needs the biases of a quarter of the columns, where a row per thread
// needs all of them: the shared-memory reads of 64 biases by every thread
// (64 wavefronts a warp and layer) were what bounded the kernel.
// at: the lane's address in the warp's rows of the tile (frag_base).
template <int KG>
__device__ __forceinline__ void epilogue_frag(uint32_t taddr, const float *bias, uint32_t at) {
  constexpr uint32_t kRow8 = KG * 128;  // bytes of 8 rows
  unsigned long long b[KG];
  const float *bl = bias + (lane_id() & 3) * kFragBias;
#pragma unroll
  for (int k = 0; k < KG; k += 2) {
    const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(bl + 2 * k);
    b[k] = q.x;
    b[k + 1] = q.y;
  }
#pragma unroll
  for (int half = 0; half < 2; half++) {
    float v[4 * KG];
    if constexpr (KG == 8) tc::tmem_ld_frag8(taddr + ((uint32_t)(16 * half) << 16), v);
    else tc::tmem_ld_frag2(taddr + ((uint32_t)(16 * half) << 16), v);
#pragma unroll
    for (int k = 0; k < KG; k += 2)
      tc::stmatrix4(at + 2 * half * kRow8 + k * 128, bias_relu_half2(v[4 * k], v[4 * k + 1], b[k]),
                    bias_relu_half2(v[4 * k + 2], v[4 * k + 3], b[k]),
                    bias_relu_half2(v[4 * k + 4], v[4 * k + 5], b[k + 1]),
                    bias_relu_half2(v[4 * k + 6], v[4 * k + 7], b[k + 1]));
  }
}

// Lane's stmatrix address in rows [32 w, 32 w + 32) of a tile with 8 KG columns
template <int KG>
__device__ __forceinline__ uint32_t frag_base(const uint8_t *tile, int w) {
  const int l = lane_id();
  return tc::smem_addr(tile) + (4 * w + ((l >> 3) & 1)) * (KG * 128) + (l >> 4) * 128 + (l & 7) * 16;
}

struct NerfParams {
  const __half *params;
  const float *z, *tpsdf, *geo;
  int B, N, V;
  float *density, *geo_out;
  int *error;
  int nb;          // feature tiles of a sigma batch
  long n_batches;  // batches of all points
};

// one row's inputs (z, t_psdf, 16 geometry features), loaded ahead
struct NerfRow {
  float x[18];
  long pv;
  bool ok;
};

__device__ __forceinline__ void load_row(const NerfParams &p, long tile, int rv, int rp, int Pt, long n_points,
                                         NerfRow &row) {
  const long g = tile * Pt + rp;
  row.ok = rv < p.V && g < n_points;
  row.pv = 0;
#pragma unroll
  for (int j = 0; j < 18; j++) row.x[j] = 0.0f;
  if (row.ok) {
    // the frame of point g (32-bit division where the points allow it)
    const long b = p.B == 1 ? 0 : (n_points <= 0x7fffffffL ? (long)((uint32_t)g / (uint32_t)p.N) : g / p.N);
    row.pv = (b * p.V + rv) * p.N + (g - b * p.N);
    row.x[0] = __ldg(p.z + row.pv);
    row.x[1] = __ldg(p.tpsdf + row.pv);
    const float4 *gf = reinterpret_cast<const float4 *>(p.geo + row.pv * 16);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float4 f = __ldg(gf + q);
      row.x[2 + 4 * q] = f.x;
      row.x[3 + 4 * q] = f.y;
      row.x[4 + 4 * q] = f.z;
      row.x[5 + 4 * q] = f.w;
    }
  }
}

// issue one M=128 layer: D[tmem + dcol] = A[a] * W^T, K columns in steps of
// 16 (ia, iw: shared-memory addresses of the operands)
template <int K, int N>
__device__ __forceinline__ void issue_layer(uint32_t d, uint32_t ia, uint32_t iw) {
  constexpr uint32_t idesc = tc::idesc_f16_f32(128, N);
  const uint64_t da = tc::smem_desc(ia, 128, K * 16), dw = tc::smem_desc(iw, 128, K * 16);
#pragma unroll
  for (int kk = 0; kk < K / 16; kk++)  // 256 bytes a step, in units of 16 in the address field
    tc::mma_f16(d, da + 16 * kk, dw + 16 * kk, idesc, kk > 0 ? 1u : 0u);
}

template <bool GEO>
__global__ void __launch_bounds__(128 * kNerfTiles<GEO>, 1) nerf_density_kernel(NerfParams p) {
  constexpr int kTiles = kNerfTiles<GEO>;
  extern __shared__ uint8_t smem_raw[];
  NerfSmem<GEO> &sm = *reinterpret_cast<NerfSmem<GEO> *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  const int tid = threadIdx.x;
  // warp and warpgroup through a shuffle, so that the compiler knows them (and
  // the descriptors made of them) to be the same in every lane
  const int warp = __shfl_sync(SG_FULL, tid >> 5, 0);
  const int t = warp >> 2;  // this thread's warpgroup
  const int r = tid & 127;  // its row
  const int V = p.V, Pt = 128 / V, nb = p.nb;
  const long n_points = (long)p.B * p.N;
  const int rv = r / Pt, rp = r % Pt;
  // consecutive batches go to different CTAs, a CTA's to its warpgroups in turn
  const long bstride = (long)gridDim.x * kTiles;
  long batch = blockIdx.x + (long)gridDim.x * t;
  NerfRow cur;      // inputs on their way
  uint32_t xin[9];  // the next tile's inputs, float16 pairs
  bool next_ok = false;
  long next_pv = 0;
  auto take_inputs = [&]() {
#pragma unroll
    for (int j = 0; j < 9; j++) xin[j] = pack_half2(cur.x[2 * j], cur.x[2 * j + 1]);
    next_ok = cur.ok;
    next_pv = cur.pv;
  };
  load_row(p, batch * nb, rv, rp, Pt, n_points, cur);
  const __half *P = p.params;
  // weights and biases, once per CTA
  stage_weights<18, 64, 64, 32>(sm.w1, P, 0);
  stage_weights<64, 64, 64, 64>(sm.w2, P, 1216);
  stage_weights<64, 64, 64, 64>(sm.w3, P, 5376);
  stage_weights<64, 64, 64, 64>(sm.w4, P, 9536);
  stage_weights<64, 64, 64, 64>(sm.ws1, P, kSigmaOff);
  stage_weights<64, 64, 64, 64>(sm.ws2, P, kSigmaOff + 4160);
  if constexpr (GEO) {
    stage_weights<18, 16, 16, 32>(sm.geo.w1, P, kGeoOff);
    stage_weights<16, 8, 16, 16>(sm.geo.w2, P, kGeoOff + 304);
    stage_bias_frag(sm.geo.b1, P, kGeoOff + 288, 16);
    stage_bias(sm.geo.b2, P, kGeoOff + 432, 8);
  }
  stage_bias_frag(sm.b1, P, 1152, 64);
  stage_bias_frag(sm.b2, P, 5312, 64);
  stage_bias_frag(sm.b3, P, 9472, 64);
  stage_bias_frag(sm.b4, P, 13632, 64);
  stage_bias_frag(sm.bs1, P, kSigmaOff + 4096, 64);
  stage_bias(sm.bs2, P, kSigmaOff + 8256, 64);
  stage_bias(sm.ws3, P, kSigmaOff + 8320, 64);
  // the sigma tile's rows past a batch's points stay zero
  for (int i = tid; i < (int)sizeof(sm.m) / 16; i += (int)blockDim.x)
    reinterpret_cast<uint4 *>(sm.m)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) {
    sm.bs3 = h2f(P[kSigmaOff + 8384]);
    for (int q = 0; q < kTiles; q++) {
      tc::mbar_init(tc::smem_addr(&sm.mbar[q]), 1);
      sm.fail[q] = 0;
    }
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tc::smem_addr(&sm.tmem_slot), kNerfTmemCols);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = __shfl_sync(SG_FULL, sm.tmem_slot, 0);
  // warp (tid >> 5) may read tensor-memory lanes 32 * (warp % 4) ..: its rows
  const uint32_t lanes = (uint32_t)(r & ~31) << 16;
  const uint32_t df = 64u * t, dg = kGeoCol + 16u * t;  // columns of the tile's accumulators
  const uint32_t mbar = tc::smem_addr(&sm.mbar[t]);
  uint8_t *hh = sm.h[t], *mm = sm.m[t];
  const uint32_t ih = tc::smem_addr(hh), im = tc::smem_addr(mm);
  const uint32_t fh = frag_base<8>(hh, warp & 3);
  const float inv = 1.0f / (float)V;
  const uint32_t inv_pt = (1u << 20) / Pt + 1;  // i / Pt = (i inv_pt) >> 20 for i < 1024, Pt <= 128
  uint32_t phase = 0;
  bool failed = false;  // a wait of this thread ran out

  // The warpgroups run their tiles independently (own mbarrier, own issuing
  // thread, own named barrier), so one's MMAs overlap the others' epilogues.
  const bool issuing_warp = (warp & 3) == 0;
  auto layer_done = [&]() {
    if (!failed && !tc::mbar_wait(mbar, phase, kNerfWaitIters)) {
      failed = true;
      sm.fail[t] = 1;
    }
    phase ^= 1u;
    __syncwarp();  // the lanes left the wait apart; tensor-memory loads are warp-wide
    tc::fence_after_sync();
  };
  auto operands_ready = [&]() {
    tc::fence_async_smem();
    tc::fence_before_sync();
    wg_sync(t);
  };
  // one layer of hidden rows: D = A W^T, then bias, float16, ReLU into h
  auto hidden_layer = [&](uint32_t a, const uint8_t *w, const float *bias) {
    operands_ready();
    if (issuing_warp && tc::elect_one()) {
      tc::fence_after_sync();
      issue_layer<64, 64>(tmem + df, a, tc::smem_addr(w));
      tc::commit(mbar);
    }
    layer_done();
    epilogue_frag<8>(tmem + lanes + df, bias, fh);
  };

  take_inputs();
  for (; batch < p.n_batches; batch += bstride) {
    const long g0 = batch * nb * Pt;  // the batch's first point
#pragma unroll 1
    for (int s = 0; s < nb; s++) {
      if (g0 + (long)s * Pt >= n_points) break;  // the last batch may hold fewer tiles
      uint4 *const row = reinterpret_cast<uint4 *>(hh + tc::kmaj_offset(r, 0, 32));  // 8-column chunks 128 bytes apart
      row[0] = make_uint4(xin[0], xin[1], xin[2], xin[3]);
      row[8] = make_uint4(xin[4], xin[5], xin[6], xin[7]);
      row[16] = make_uint4(xin[8], 0u, 0u, 0u);
      row[24] = make_uint4(0u, 0u, 0u, 0u);
      const bool row_ok = next_ok;
      const long pv = next_pv;
      // the next tile's inputs: loads in flight while this tile runs
      {
        const long next = s + 1 < nb ? batch * nb + s + 1 : (batch + bstride) * nb;
        load_row(p, next, rv, rp, Pt, n_points, cur);
      }
      operands_ready();
      if (issuing_warp && tc::elect_one()) {
        tc::fence_after_sync();
        issue_layer<32, 64>(tmem + df, ih, tc::smem_addr(sm.w1));
        if constexpr (GEO) issue_layer<32, 16>(tmem + dg, ih, tc::smem_addr(sm.geo.w1));
        tc::commit(mbar);
      }
      layer_done();
      // ---- layer 1 epilogue (features -> h, geometry hidden -> g) -----------
      epilogue_frag<8>(tmem + lanes + df, sm.b1, fh);
      if constexpr (GEO) epilogue_frag<2>(tmem + lanes + dg, sm.geo.b1, frag_base<2>(sm.geo.h[t], warp & 3));
      take_inputs();  // the loads of the first layer's time have arrived
      operands_ready();
      if (issuing_warp && tc::elect_one()) {
        tc::fence_after_sync();
        issue_layer<64, 64>(tmem + df, ih, tc::smem_addr(sm.w2));
        if constexpr (GEO) issue_layer<16, 16>(tmem + dg, tc::smem_addr(sm.geo.h[t]), tc::smem_addr(sm.geo.w2));
        tc::commit(mbar);
      }
      layer_done();
      // ---- layer 2 epilogue; geometry output ----------------------------------
      epilogue_frag<8>(tmem + lanes + df, sm.b2, fh);
      if constexpr (GEO) {
        float v[16];
        tc::tmem_ld16(tmem + lanes + dg, v);
        if (row_ok) {
          const uint4 q = bias_relu8(v, sm.geo.b2);
          const __half2 *hq = reinterpret_cast<const __half2 *>(&q);
          float4 *go = reinterpret_cast<float4 *>(p.geo_out + pv * 8);
          const float2 a = __half22float2(hq[0]), b = __half22float2(hq[1]), c = __half22float2(hq[2]),
                       d = __half22float2(hq[3]);
          go[0] = make_float4(a.x, a.y, b.x, b.y);
          go[1] = make_float4(c.x, c.y, d.x, d.y);
        }
      }
      // ---- layers 3 and 4 -------------------------------------------------------
      hidden_layer(ih, sm.w3, sm.b3);
      hidden_layer(ih, sm.w4, sm.b4);
      wg_sync(t);
      // ---- view mean: sigma row s * Pt + p takes the mean of rows v * Pt + p,
      // 8 channels a thread at a time -------------------------------------------
      for (int i = r; i < Pt * 8; i += 128) {
        const int c8 = (int)(((uint32_t)i * inv_pt) >> 20), q = i - c8 * Pt;  // i / Pt, i < 1024
        float m[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        for (int v0 = 0; v0 < V; v0 += 4) {
          uint4 w[4];  // four views' reads in flight
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (v0 + u < V)
              w[u] = *reinterpret_cast<const uint4 *>(hh + tc::kmaj_offset((v0 + u) * Pt + q, c8 * 8, 64));
#pragma unroll
          for (int u = 0; u < 4; u++) {
            if (v0 + u >= V) break;
            const __half2 *hw = reinterpret_cast<const __half2 *>(&w[u]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
              const float2 f = __half22float2(hw[j]);
              m[2 * j] += f.x;
              m[2 * j + 1] += f.y;
            }
          }
        }
        *reinterpret_cast<uint4 *>(mm + tc::kmaj_offset(s * Pt + q, c8 * 8, 64)) =
            make_uint4(pack_half2(m[0] * inv, m[1] * inv), pack_half2(m[2] * inv, m[3] * inv),
                       pack_half2(m[4] * inv, m[5] * inv), pack_half2(m[6] * inv, m[7] * inv));
      }
      wg_sync(t);  // h is free for the next tile's inputs
    }
    // ---- sigma layers over the batch's points -----------------------------------
    hidden_layer(im, sm.ws1, sm.bs1);
    operands_ready();
    if (issuing_warp && tc::elect_one()) {
      tc::fence_after_sync();
      issue_layer<64, 64>(tmem + df, ih, tc::smem_addr(sm.ws2));
      tc::commit(mbar);
    }
    layer_done();
    {
      float acc = 0.0f;
#pragma unroll
      for (int half = 0; half < 2; half++) {
        float v[32];
        tc::tmem_ld32(tmem + lanes + df + 32 * half, v);
#pragma unroll
        for (int c = 0; c < 4; c++) {
          const uint4 q = bias_relu8(v + 8 * c, sm.bs2 + 32 * half + 8 * c);
          const __half2 *hq = reinterpret_cast<const __half2 *>(&q);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float2 f = __half22float2(hq[j]);
            acc = __fmaf_rn(f.x, sm.ws3[32 * half + 8 * c + 2 * j], acc);
            acc = __fmaf_rn(f.y, sm.ws3[32 * half + 8 * c + 2 * j + 1], acc);
          }
        }
      }
      const long gp = g0 + r;
      if (r < nb * Pt && gp < n_points) {
        const float pre = h2f(__float2half_rn(acc + sm.bs3));
        p.density[gp] = h2f(__float2half_rn(1.0f / (1.0f + expf(-pre))));
      }
    }
    // the next tile's input rows go over h: the sigma MMA has read it
    tc::fence_before_sync();
    wg_sync(t);
    if (*reinterpret_cast<volatile int *>(&sm.fail[t])) break;
  }
  if (failed && p.error) atomicExch(p.error, 1);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, kNerfTmemCols);
  }
}

template <bool GEO>
static int launch_nerf(NerfParams p, long n_tiles, int Pt, sg_stream_t stream) {
  const size_t smem = sizeof(NerfSmem<GEO>) + 128;
  static_assert(sizeof(NerfSmem<GEO>) + 128 <= 227 * 1024, "one CTA per SM");
  // per device and context, so set on every call
  if (cudaFuncSetAttribute(nerf_density_kernel<GEO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
      cudaSuccess)
    return SG_ERR_CUDA;
  // A sigma batch fills its 128 rows (floor(128 / Pt) tiles), unless there are
  // so few tiles that warpgroups would go without one
  const long wgs = (long)num_sms() * kNerfTiles<GEO>;
  const long share = (n_tiles + wgs - 1) / wgs;
  p.nb = (int)(128 / Pt < share ? 128 / Pt : share);
  p.n_batches = (n_tiles + p.nb - 1) / p.nb;
  long grid = num_sms();
  if (grid > p.n_batches) grid = p.n_batches;
  nerf_density_kernel<GEO><<<(int)grid, 128 * kNerfTiles<GEO>, smem, stream>>>(p);
  return SG_OK;
}

}  // namespace sg

using namespace sg;

extern "C" size_t sg_nerf_param_count(void) { return kNerfParamCount; }

extern "C" int sg_nerf_density(const uint16_t *params, const float *points_z, const float *points_tpsdf,
                               const float *feats_geo, int B, int N, int V, float *density, float *geo_feats,
                               int *error, sg_stream_t stream) {
  if (!params || !points_z || !points_tpsdf || !feats_geo || !density) return SG_ERR_INVALID_ARG;
  if (B <= 0 || N <= 0 || V <= 0 || V > 128) return SG_ERR_INVALID_ARG;
  if ((((uintptr_t)feats_geo) % 16) != 0 || (geo_feats && ((uintptr_t)geo_feats) % 16 != 0))
    return SG_ERR_INVALID_ARG;
  const long n_points = (long)B * N;
  const int Pt = 128 / V;
  const long n_tiles = (n_points + Pt - 1) / Pt;
  NerfParams p{reinterpret_cast<const __half *>(params), points_z, points_tpsdf, feats_geo, B, N, V, density,
               geo_feats, error, 1, n_tiles};
  const int rc = geo_feats ? launch_nerf<true>(p, n_tiles, Pt, stream) : launch_nerf<false>(p, n_tiles, Pt, stream);
  if (rc != SG_OK) return rc;
  SG_LAUNCH_CHECK();
  return SG_OK;
}
