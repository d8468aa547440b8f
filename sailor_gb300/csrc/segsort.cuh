// segsort.cuh -- device-wide exclusive scan and stable LSD radix sort
// (segsort.cu) for buffers sized by a host-known capacity whose live count
// sits in device memory.
#pragma once

#include "common.cuh"

namespace sg {

// The scan's parts, for kernels that form its input or use its output in place:
// blocks of kScanBlock elements (256 threads x 4), their sums in sums[block];
// launch_scan_sums turns those of the first min(*n_dev, n) elements into offsets.
constexpr int kScanBlock = 1024;
void launch_scan_sums(int *sums, long n, const int *n_dev, int *total, sg_stream_t stream);

__device__ __forceinline__ int block_excl_scan_256(int v, int *s_warp, int &total) {
  // exclusive scan of one int per thread over a 256-thread block
  const int lane = lane_id(), w = threadIdx.x >> 5;
  const int incl = warp_incl_scan(v);
  if (lane == 31) s_warp[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int x = lane < 8 ? s_warp[lane] : 0;
    const int xi = warp_incl_scan(x);
    if (lane < 8) s_warp[8 + lane] = xi - x;
    if (lane == 7) s_warp[16] = xi;
  }
  __syncthreads();
  const int out = s_warp[8 + w] + incl - v;
  total = s_warp[16];
  __syncthreads();
  return out;
}

// n_dev (may be null): the live count in device memory, at most n
__device__ __forceinline__ long live_count(long n, const int *n_dev) {
  if (!n_dev) return n;
  const long m = *n_dev;
  return m < n ? m : n;
}

// ints of scratch an exclusive scan of n elements needs
size_t scan_scratch_ints(long n);

// Exclusive scan of in[0, n) into out (in place allowed); the sum into
// *total (may be null).  scratch: scan_scratch_ints(n) ints.
void launch_excl_scan(const int *in, long n, int *out, int *scratch, int *total, sg_stream_t stream);

// The same over the first min(*n_dev, n) elements (n_dev in device memory).
void launch_excl_scan_dev(const int *in, long n, const int *n_dev, int *out, int *scratch, int *total,
                          sg_stream_t stream);

// bytes of scratch a radix sort of up to cap items needs
size_t radix_scratch_bytes(long cap);

// Stable sort of (keys_in[i], vals_in[i]) for i < *n_dev (n_dev <= cap;
// vals_in null: the values are i) by the low key_bits bits of the keys, 8
// bits a pass; passes alternate between the (keys_a, vals_a) and (keys_b,
// vals_b) buffers, starting with a (the input may be the b pair).  Returns
// the number of passes: the result is in a when it is odd, in b when even.
int launch_radix_sort(const uint32_t *keys_in, const uint32_t *vals_in, const int *n_dev, long cap, int key_bits,
                      uint32_t *keys_a, uint32_t *vals_a, uint32_t *keys_b, uint32_t *vals_b, void *scratch,
                      sg_stream_t stream);

}  // namespace sg
