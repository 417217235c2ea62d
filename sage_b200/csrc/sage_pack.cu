// Export-side packing: frozen signs / direction indices and trained radii of a spherical
// (SAGE or SPHQuant) linear into the packed buffers the inference kernels read.
//
// Replaces the tensor program of the reference's exporter
// (weight_vq/sphquant/packing.py:32-75): per (row, 128-channel group)
//     minimum = min of the 16 radii, step = fp16((max - min) / levels), minimum = fp16(minimum)
//     code_v  = clamp(round_half_even((radius_v - minimum) / step), 0, levels)    (0 where step == 0)
//     word_v  = sign bits | index << 8 | low (8 - D) bits of code_v << (8 + D)
//     high    = the two high bits of the sixteen codes, two bits per vector
// and the words laid out either in SAGE's tiled form (two codes per 32-bit word,
// [tile][group][16 rows][8 words], rows padded to a multiple of 16 with zero codes and a zero
// grid) or in SPHQuant's row-major int16 form.  Integer work plus a handful of FP32 operations
// that round exactly as the tensor program's do (IEEE division, round-half-even, one rounding
// to FP16), so the packed buffers are identical bit for bit.
//
// One lane per 8-weight vector, half a warp per (row, group): signs, indices and radii are read and codes
// written in the order they lie in memory (one thread per (row, group) read 8 bytes of 32 different
// lines per instruction), the group's minimum, maximum and high word are formed by half-warp
// reductions.  Radii may come as the trained logits: softplus is then one more step of the same pass.
// HBM-bound on the inputs (1 byte of signs and 1 or 1.5 of radius and index per weight in, 0.31 out).
// Measured, 2560 -> 9728 from logits and 64-bit indices: 28.6 us + 18 us of conversion passes -> 27 us.
#include <cooperative_groups.h>

#include "sage_common.cuh"
#include "sage_kernels.h"

namespace sageb200 {
namespace {

constexpr int kPackThreads = 256;

// four sign bytes -> four bits (bit d = byte d negative): one multiply moves bit 7 of each byte to bits
// 24..27 without carries
__device__ __forceinline__ uint32_t sign_bits(uint32_t bytes) {
  return ((((bytes >> 7) & 0x01010101u) * 0x01020408u) >> 24) & 0xfu;
}

template <bool kTiled, bool kLogits, typename Index>
__global__ void __launch_bounds__(kPackThreads) sage_pack_kernel(
    const int8_t *__restrict__ signs, const Index *__restrict__ indices,
    const float *__restrict__ radius, uint32_t *__restrict__ codes, uint32_t *__restrict__ high_out,
    __half *__restrict__ grid_or_scales, __half *__restrict__ mins, int n, int n_padded, int k,
    int dbits) {
  const int groups = k >> 7;
  const long long total = static_cast<long long>(n_padded) * groups;
  const int levels = (1 << (10 - dbits)) - 1;
  const int low_bits = 8 - dbits;
  const int v = threadIdx.x & 15;  // vector of the group
  const unsigned half_mask = 0xffffu << (threadIdx.x & 16);
  for (long long item = (static_cast<long long>(blockIdx.x) * kPackThreads + threadIdx.x) >> 4; item < total;
       item += (static_cast<long long>(gridDim.x) * kPackThreads) >> 4) {
    // (the whole half warp has the same item)
    const int row = total <= 0x7fffffffLL ? static_cast<int>(static_cast<unsigned>(item) / static_cast<unsigned>(groups))
                                          : static_cast<int>(item / groups);
    const int group = static_cast<int>(item - static_cast<long long>(row) * groups);
    uint32_t word = 0, high = 0;
    __half minimum_h = __float2half_rn(0.0f), step_h = __float2half_rn(0.0f);
    if (row < n) {
      const size_t vector = static_cast<size_t>(row) * (k >> 3) + group * 16 + v;
      float value = radius[vector];
      if (kLogits) value = value > 20.0f ? value : log1pf(expf(value));  // softplus with its usual threshold
      const uint32_t index = static_cast<uint32_t>(indices[vector]);
      const uint2 packed_signs = *reinterpret_cast<const uint2 *>(signs + vector * 8);
      float lowest = value, highest = value;
#pragma unroll
      for (int o = 8; o; o >>= 1) {
        lowest = fminf(lowest, __shfl_xor_sync(half_mask, lowest, o));
        highest = fmaxf(highest, __shfl_xor_sync(half_mask, highest, o));
      }
      // the step is rounded to FP16 from the FP32 minimum, then the minimum itself is rounded
      step_h = __float2half_rn(__fdiv_rn(__fsub_rn(highest, lowest), static_cast<float>(levels)));
      minimum_h = __float2half_rn(lowest);
      const float step = __half2float(step_h), minimum = __half2float(minimum_h);
      int code = 0;
      if (step > 0.0f) {
        const float scaled = rintf(__fdiv_rn(__fsub_rn(value, minimum), step));
        code = static_cast<int>(fminf(fmaxf(scaled, 0.0f), static_cast<float>(levels)));
      }
      word = sign_bits(packed_signs.x) | (sign_bits(packed_signs.y) << 4) | (index << 8) |
             (static_cast<uint32_t>(code & ((1 << low_bits) - 1)) << (8 + dbits));
      high = __reduce_or_sync(half_mask, static_cast<uint32_t>(code >> low_bits) << (2 * v));
    }
    // row-major int16 codes [n][k/8] with per-(row, group) words, or the tiled form of the same
    const size_t cell = kTiled ? (static_cast<size_t>(row >> 4) * groups + group) * 16 + (row & 15)
                               : static_cast<size_t>(row) * groups + group;
    reinterpret_cast<uint16_t *>(codes)[cell * 16 + v] = static_cast<uint16_t>(word);
    if (v == 0) {
      high_out[cell] = high;
      if (kTiled) {
        reinterpret_cast<__half2 *>(grid_or_scales)[cell] = __halves2half2(minimum_h, step_h);
      } else {
        grid_or_scales[cell] = step_h;
        mins[cell] = minimum_h;
      }
    }
  }
}

// Direction codebook from angular logits: one thread per entry, every operation rounded on its own as the
// tensor program's are (no contraction), products and sums in its order - the running product of the
// sines as a doubling scan, the sum of squares as a halving tree - so that the halves are the same.
// `planar`: [4][entries][2] (SAGE), otherwise [entries][8] (SPHQuant).
__global__ void codebook_kernel(const float *__restrict__ logits, __half *__restrict__ book, int entries, float scale,
                                float offset, bool planar) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= entries) return;
  float sine[7], cosine[7], x[8];
#pragma unroll
  for (int i = 0; i < 7; ++i) {
    const float sigmoid = __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-logits[e * 7 + i])));
    const float theta = __fadd_rn(offset, __fmul_rn(scale, sigmoid));
    sine[i] = sinf(theta);
    cosine[i] = cosf(theta);
  }
  // inclusive products: pairs, then fours, then the upper half
  sine[1] = __fmul_rn(sine[1], sine[0]);
  sine[3] = __fmul_rn(sine[3], sine[2]);
  sine[5] = __fmul_rn(sine[5], sine[4]);
  sine[2] = __fmul_rn(sine[2], sine[1]);
  sine[3] = __fmul_rn(sine[3], sine[1]);
  sine[6] = __fmul_rn(sine[6], sine[5]);
#pragma unroll
  for (int i = 4; i < 7; ++i) sine[i] = __fmul_rn(sine[i], sine[3]);
  x[0] = cosine[0];
#pragma unroll
  for (int i = 1; i < 7; ++i) x[i] = __fmul_rn(sine[i - 1], cosine[i]);
  x[7] = sine[6];
  float square[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) square[i] = __fmul_rn(x[i], x[i]);
  const float sum = __fadd_rn(__fadd_rn(__fadd_rn(square[0], square[4]), __fadd_rn(square[2], square[6])),
                              __fadd_rn(__fadd_rn(square[1], square[5]), __fadd_rn(square[3], square[7])));
  const float norm = fmaxf(__fsqrt_rn(sum), 1e-12f);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const __half h = __float2half_rn(__fdiv_rn(x[i], norm));
    book[planar ? ((i >> 1) * entries + e) * 2 + (i & 1) : e * 8 + i] = h;
  }
}

// inverse[order[i]] = i.  *verdict: bit 0 where order is not the identity, bit 1 where it is not a permutation (an
// entry out of range, or one that comes twice) - the inverse is then no use, but every entry of it is a channel.
// Bound by latency: three passes over k words.  One cluster, whose barrier orders the passes, so that nothing has to
// be cleared by launches of its own.  Between events, against a memset and a grid that did not look for duplicates:
// 8.2 / 9.2 us at k = 2560, 10.2 / 9.0 at 9728, 12.3 / 9.1 at 25600 (27 there with one CTA).
constexpr int kInvertThreads = 1024, kInvertCtas = 8;
__global__ void __cluster_dims__(kInvertCtas) __launch_bounds__(kInvertThreads)
    invert_permutation_kernel(const long long *__restrict__ order, int *inverse, int *verdict, int k) {
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int first = blockIdx.x * kInvertThreads + threadIdx.x;
  constexpr int kStep = kInvertCtas * kInvertThreads;
  for (int i = first; i < k; i += kStep) inverse[i] = 0;
  if (first == 0) *verdict = 0;
  cluster.sync();
  int found = 0;
  for (int i = first; i < k; i += kStep) {
    const long long at = order[i];
    if (at >= 0 && at < k) inverse[at] = i;
    else found |= 2;
    if (at != i) found |= 1;
  }
  cluster.sync();
  // (k entries in range that all find themselves again are k different ones)
  for (int i = first; i < k; i += kStep) {
    const long long at = order[i];
    if (at >= 0 && at < k && __ldcg(inverse + at) != i) found |= 2;
  }
  const int moved = __syncthreads_or(found & 1), broken = __syncthreads_or(found & 2);
  if (threadIdx.x == 0 && (moved || broken)) atomicOr(verdict, (moved ? 1 : 0) | (broken ? 2 : 0));
}

}  // namespace

cudaError_t launch_codebook(const float *logits, __half *book, int entries, float scale, float offset, bool planar,
                            cudaStream_t stream) {
  codebook_kernel<<<(entries + 31) / 32, 32, 0, stream>>>(logits, book, entries, scale, offset, planar);
  return cudaGetLastError();
}

cudaError_t launch_invert_permutation(const long long *order, int *inverse, int *verdict, int k, cudaStream_t stream) {
  invert_permutation_kernel<<<kInvertCtas, kInvertThreads, 0, stream>>>(order, inverse, verdict, k);
  return cudaGetLastError();
}

cudaError_t launch_pack(const int8_t *signs, const void *indices, int index_bytes, const float *radius, bool logits,
                        uint32_t *codes, uint32_t *high, __half *grid_or_scales, __half *mins, int n, int k, int dbits,
                        bool tiled, cudaStream_t stream, int sm_count) {
  const int n_padded = tiled ? (n + 15) / 16 * 16 : n;
  const long long lanes = static_cast<long long>(n_padded) * (k >> 7) * 16;
  long long blocks = (lanes + kPackThreads - 1) / kPackThreads;
  const long long cap = static_cast<long long>(sm_count) * 32;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  auto launch = [&](auto kernel, auto *index) {
    kernel<<<static_cast<unsigned>(blocks), kPackThreads, 0, stream>>>(signs, index, radius, codes, high, grid_or_scales,
                                                                       mins, n, n_padded, k, dbits);
  };
  const auto *narrow = static_cast<const int32_t *>(indices);
  const auto *wide = static_cast<const long long *>(indices);
  if (index_bytes == 8) {
    if (tiled) logits ? launch(sage_pack_kernel<true, true, long long>, wide) : launch(sage_pack_kernel<true, false, long long>, wide);
    else logits ? launch(sage_pack_kernel<false, true, long long>, wide) : launch(sage_pack_kernel<false, false, long long>, wide);
  } else {
    if (tiled) logits ? launch(sage_pack_kernel<true, true, int32_t>, narrow) : launch(sage_pack_kernel<true, false, int32_t>, narrow);
    else logits ? launch(sage_pack_kernel<false, true, int32_t>, narrow) : launch(sage_pack_kernel<false, false, int32_t>, narrow);
  }
  return cudaGetLastError();
}

}  // namespace sageb200
