// The SwiGLU MLP of routed experts over rows sorted by expert: blocks of at most 16 rows, each belonging to one
// expert whose id is read on the device.
//
// Two launches, gate/up/SwiGLU and down, whatever the number of blocks: a CTA walks a list of items - eight
// 16-row weight tiles of one block, one tile per warp over all of K - and skips the blocks nobody uses.
// (As grouped problems of the decode kernel, 64 to a launch with a staging launch each, a batch of 32 tokens
// of the 30B-A3B layer took eight launches of ~33 us, two CTAs for each of 64 experts and a third of
// them for empty blocks, plus zero fills and a SwiGLU launch.)
//
// Bound: HBM on paper (every live expert's packed bytes once); in practice the decode's instructions, as in the
// decode kernel, whose per-unit arithmetic (compute_unit) this shares.  What an item does:
//   * packed words of a warp's first units are requested before the activations are staged, later ones kInFlight
//     units ahead in registers;
//   * the block's rows come in as [channel][8 rows] (16 bytes per channel), so that one 16-byte read per channel
//     gathers all rows through the expert's permutation, and an 8 x 8 turn in registers gives the operand order;
//   * two CTAs per SM hide each other's staging.
// Gate and up of a tile run one after the other in the same warp (their permutations and codebooks differ), so
// SwiGLU is applied to the accumulators and neither product is stored.
// Measured, 32 tokens x 8 of 128 experts, hidden 2048, intermediate 768, the whole exchange:
// 300 -> 150 us, 97 + 47 of them (under the profiler) in the two launches, whose instructions alone need 66.
#include "../../include/sage_b200.h"
#include "sage_common.cuh"
#include "sage_kernels.h"
#include "sage_skinny_core.cuh"

namespace sageb200 {
namespace {

constexpr int kExpertWarps = 8;
constexpr int kExpertThreads = kExpertWarps * 32;
constexpr int kInFlight = 4;  // units a lane's packed words are requested ahead
// Tiles of an item per warp: two share the staging of a down item (K = 768 is six units a tile).
template <bool kGateUp>
constexpr int kTilesPerWarp = kGateUp ? 1 : 2;

struct ExpertMatrix {
  const uint32_t *codes, *radii, *grid, *book;
  const int32_t *perm;  // null: identity
  long long codes_stride, cell_stride, book_stride;  // from one expert to the next, in 32-bit words
  int entries, dbits;
};

struct ExpertParams {
  ExpertMatrix matrix[2];  // gate and up, or down
  const __half *x;         // [blocks][rows][k]
  __half *y;               // [blocks][rows][n]
  const int *block_experts;
  int blocks, rows, n, k, first_expert, experts;
};

struct UnitWords {
  uint2 code[2];
  uint32_t radius[2], endpoints[2];
};

// Rows 2i and 2i+1 of a channel pair's words: the low or the high halves together.
__device__ __forceinline__ uint32_t low_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410); }
__device__ __forceinline__ uint32_t high_halves(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

// 8 x 8 halves: out[j] = column j of the rows in[0..7] (its own inverse).
__device__ __forceinline__ void turn_8x8(const uint4 (&in)[8], uint4 (&out)[8]) {
  const uint32_t *a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = reinterpret_cast<const uint32_t *>(&in[i]);
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    out[2 * w] = make_uint4(low_halves(a[0][w], a[1][w]), low_halves(a[2][w], a[3][w]), low_halves(a[4][w], a[5][w]),
                            low_halves(a[6][w], a[7][w]));
    out[2 * w + 1] = make_uint4(high_halves(a[0][w], a[1][w]), high_halves(a[2][w], a[3][w]),
                                high_halves(a[4][w], a[5][w]), high_halves(a[6][w], a[7][w]));
  }
}

// Slot of a channel in the [channel][8 rows] buffer, swizzled so that eight lanes eight channels apart hit
// different 16-byte bank groups.
__device__ __forceinline__ int channel_slot(int c) { return c ^ ((c >> 3) & 7); }

__host__ __device__ constexpr int staged_row_bytes(int k) { return 2 * k + 64; }  // rows 64 bytes apart modulo 128

// NB: blocks of eight rows (1 or 2).  kGateUp: two matrices and SwiGLU, otherwise one.
template <int NB, bool kGateUp>
__global__ void __launch_bounds__(kExpertThreads, 2) expert_mlp_kernel(const __grid_constant__ ExpertParams p) {
  extern __shared__ __align__(128) unsigned char shared[];
  pdl_launch_dependents();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int groups = p.k >> 7, tiles = (p.n + 15) / 16, vectors = p.k >> 3;
  constexpr int kTiles = kTilesPerWarp<kGateUp>;
  constexpr int kItemTiles = kExpertWarps * kTiles;
  const int chunks = (tiles + kItemTiles - 1) / kItemTiles;
  // [codebook, 8 copies][rows in original order: NB x [channel][8]][rows as staged]
  int entries = p.matrix[0].entries;
  if (kGateUp) entries = max(entries, p.matrix[1].entries);
  unsigned char *book_shared = shared;
  unsigned char *linear = shared + static_cast<size_t>(entries) * 128;
  unsigned char *staged = linear + static_cast<size_t>(NB) * p.k * 16;
  const int row_bytes = staged_row_bytes(p.k);
  const uint32_t lane_offset = 16u * static_cast<uint32_t>(lane & 7);
  pdl_wait();  // the rows and the experts of the blocks are earlier kernels' output

  for (int item = blockIdx.x; item < p.blocks * chunks; item += gridDim.x) {
    const int block = item / chunks, first_tile = (item - block * chunks) * kItemTiles;
    const int tile = first_tile + warp * kTiles;  // the warp's first tile
    const int expert = __ldg(p.block_experts + block) - p.first_expert;
    __half *y = p.y + static_cast<size_t>(block) * p.rows * p.n;
    if (expert < 0 || expert >= p.experts) {
      if (!kGateUp)  // (a block without an expert of this rank reads as zeros)
        for (int i = tid; i < p.rows * kItemTiles * 16; i += kExpertThreads) {
          const int m = i / (kItemTiles * 16), row = first_tile * 16 + i % (kItemTiles * 16);
          if (row < p.n) y[static_cast<size_t>(m) * p.n + row] = __half(0.0f);
        }
      continue;
    }
    float acc[kGateUp ? 2 : 1][NB][4];
    // lane (g, t): output rows g, g + 8 of the tile, activation rows 2t, 2t + 1 of each block of eight
    auto store = [&](int to) {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int m = nb * 8 + 2 * t + (c & 1), row = to * 16 + g + 8 * (c >> 1);
          __half value = __float2half_rn(acc[0][nb][c]);
          if constexpr (kGateUp)  // rounded as the separate kernels round: gate, up, SiLU, product
            value = __hmul(__float2half_rn(silu_fast(__half2float(value))), __float2half_rn(acc[1][nb][c]));
          if (m < p.rows && to < tiles && row < p.n) y[static_cast<size_t>(m) * p.n + row] = value;
        }
    };
#pragma unroll
    for (int s = 0; s < (kGateUp ? 2 : 1); ++s) {
      const ExpertMatrix &q = p.matrix[s];
      const uint32_t *codes = q.codes + expert * q.codes_stride, *radii = q.radii + expert * q.cell_stride,
                     *grid = q.grid + expert * q.cell_stride;
      // unit u of the warp: group u % groups of its tile u / groups (past the last tile: that one again,
      // nothing is stored)
      int fetch_tile = tile, fetch_group = 0;
      auto fetch = [&]() {
        const size_t cell = (static_cast<size_t>(min(fetch_tile, tiles - 1)) * groups + fetch_group) * 16 + g;
        UnitWords w;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          w.code[h] = ldg_stream_u2(codes + (cell + 8 * h) * 8 + 2 * t);
          w.radius[h] = ldg_stream_u1(radii + cell + 8 * h);
          w.endpoints[h] = ldg_stream_u1(grid + cell + 8 * h);
        }
        if (++fetch_group == groups) fetch_group = 0, ++fetch_tile;
        return w;
      };
      UnitWords ahead[kInFlight];
#pragma unroll
      for (int i = 0; i < kInFlight; ++i) ahead[i] = fetch();
      // the first codebook entry and the first permutation vector of this thread, before the barrier
      const uint32_t *book = q.book + expert * q.book_stride;
      uint4 entry = make_uint4(0u, 0u, 0u, 0u);
      if (tid < q.entries)
        entry = make_uint4(__ldg(book + tid), __ldg(book + q.entries + tid), __ldg(book + 2 * q.entries + tid),
                           __ldg(book + 3 * q.entries + tid));
      const int32_t *perm = q.perm ? q.perm + static_cast<long long>(expert) * p.k : nullptr;
      int held = tid % vectors;  // the vector whose source channels are in lo and hi
      int4 lo, hi;
      auto hold = [&](int v) {
        held = v;
        lo = make_int4(v * 8, v * 8 + 1, v * 8 + 2, v * 8 + 3), hi = make_int4(v * 8 + 4, v * 8 + 5, v * 8 + 6, v * 8 + 7);
        if (perm) {  // (whole int4s: K is a multiple of 128 and the stack is checked to be 16-byte aligned)
          lo = __ldg(reinterpret_cast<const int4 *>(perm) + 2 * v);
          hi = __ldg(reinterpret_cast<const int4 *>(perm) + 2 * v + 1);
        }
      };
      hold(held);

      __syncthreads();  // (everyone is done with the buffers of the matrix before)
      static_assert(kExpertThreads >= 256, "one codebook entry per thread");
      if (tid < q.entries) {
#pragma unroll
        for (int r = 0; r < 8; ++r) reinterpret_cast<uint4 *>(book_shared)[tid * 8 + ((r + lane) & 7)] = entry;
      }
      if (s == 0) {
        const __half *x = p.x + static_cast<size_t>(block) * p.rows * p.k;
        for (int i = tid; i < NB * vectors; i += kExpertThreads) {
          const int plane = NB == 1 ? 0 : i / vectors, v = i - plane * vectors;
          uint4 in[8], out[8];
#pragma unroll
          for (int m = 0; m < 8; ++m) {
            in[m] = make_uint4(0u, 0u, 0u, 0u);
            if (plane * 8 + m < p.rows)
              in[m] = *reinterpret_cast<const uint4 *>(x + static_cast<size_t>(plane * 8 + m) * p.k + v * 8);
          }
          turn_8x8(in, out);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4 *>(linear + (static_cast<size_t>(plane) * p.k + channel_slot(v * 8 + j)) * 16) = out[j];
        }
        __syncthreads();
      }
      for (int i = tid; i < NB * vectors; i += kExpertThreads) {
        const int plane = NB == 1 ? 0 : i / vectors, v = i - plane * vectors;
        uint4 in[8], out[8];
        if (v != held) hold(v);
        const int source[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int j = 0; j < 8; ++j)
          in[j] = *reinterpret_cast<const uint4 *>(linear + (static_cast<size_t>(plane) * p.k + channel_slot(source[j])) * 16);
        turn_8x8(in, out);
        // vector 4t + s of a group lies at [s][t], as the decode arithmetic reads it
        unsigned char *to = staged + (v >> 4) * 256 + ((v & 3) * 4 + ((v & 15) >> 2)) * 16;
#pragma unroll
        for (int m = 0; m < 8; ++m) *reinterpret_cast<uint4 *>(to + static_cast<size_t>(plane * 8 + m) * row_bytes) = out[m];
      }
      __syncthreads();

      FieldConsts f;
      f.index_mask = static_cast<uint32_t>(q.entries - 1) << 7;
      f.hi_shift = 27 - q.dbits;
      f.hi_mask = 3u << f.hi_shift;
      f.lo_mask = ((1u << (8 - q.dbits)) - 1u) << 19;
      f.lo_left = 11 - q.dbits;
      f.lo_right = 5 + q.dbits;
      const unsigned char *x_row[NB];
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        x_row[nb] = staged + static_cast<size_t>(nb * 8 + g) * row_bytes + 16 * t;
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[s][nb][c] = 0.0f;
      }
      int group = 0, done = 0;
      for (int u = 0; u < kTiles * groups; u += kInFlight) {
#pragma unroll
        for (int i = 0; i < kInFlight; ++i) {
          if (u + i >= kTiles * groups) break;
          const UnitWords w = ahead[i];
          ahead[i] = fetch();
          compute_unit<NB, true>(w.code, w.radius, w.endpoints, acc[s], f, book_shared, lane_offset, x_row, t);
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) x_row[nb] += 256;
          if (!kGateUp && ++group == groups) {  // the next tile over the same rows
            store(tile + done);
            ++done;
            group = 0;
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
              x_row[nb] -= 256 * groups;
#pragma unroll
              for (int c = 0; c < 4; ++c) acc[s][nb][c] = 0.0f;
            }
          }
        }
      }
    }
    if (kGateUp) store(tile);
  }
}

size_t shared_bytes(int entries, int rows, int k) {
  const int nb = rows > 8 ? 2 : 1;
  return static_cast<size_t>(entries) * 128 + static_cast<size_t>(nb) * k * 16 + static_cast<size_t>(nb) * 8 * staged_row_bytes(k);
}

template <int NB, bool kGateUp>
cudaError_t launch(const ExpertParams &p, size_t shared, cudaStream_t stream, int sm_count) {
  static bool configured[64] = {};  // per instantiation and device
  int device = 0;
  cudaError_t error = cudaGetDevice(&device);
  if (error != cudaSuccess) return error;
  if (device >= 64 || !configured[device]) {
    error = cudaFuncSetAttribute(expert_mlp_kernel<NB, kGateUp>, cudaFuncAttributeMaxDynamicSharedMemorySize, kExpertSharedLimit);
    if (error != cudaSuccess) return error;
    if (device < 64) configured[device] = true;
  }
  constexpr int kItemTiles = kExpertWarps * kTilesPerWarp<kGateUp>;
  const int chunks = ((p.n + 15) / 16 + kItemTiles - 1) / kItemTiles;
  const long long items = static_cast<long long>(p.blocks) * chunks;
  const int resident = sm_count * (shared + 1024 <= 114 * 1024 ? 2 : 1);
  const unsigned ctas = static_cast<unsigned>(items < resident ? items : resident);
  return launch_dependent(expert_mlp_kernel<NB, kGateUp>, dim3(ctas), dim3(kExpertThreads), shared, stream, p);
}

}  // namespace

bool expert_mlp_fits(int rows, int hidden, int intermediate, int entries) {
  return rows >= 1 && rows <= 16 && shared_bytes(entries, rows, hidden) <= kExpertSharedLimit &&
         shared_bytes(entries, rows, intermediate) <= kExpertSharedLimit;
}

cudaError_t launch_expert_mlp(const ExpertStackView *stacks, const __half *x, __half *act, __half *y,
                              const int *block_experts, int blocks, int rows, cudaStream_t stream, int sm_count) {
  auto matrix = [](const ExpertStackView &v) {
    ExpertMatrix m{};
    m.codes = v.codes;
    m.radii = v.radii;
    m.grid = v.grid;
    m.book = v.book;
    m.perm = v.perm;
    const long long cells = static_cast<long long>((v.n + 15) / 16) * (v.k / 128) * 16;
    m.codes_stride = cells * 8;
    m.cell_stride = cells;
    m.book_stride = 4ll * v.entries;
    m.entries = v.entries;
    m.dbits = direction_bits_of(v.entries);
    return m;
  };
  ExpertParams p{};
  p.matrix[0] = matrix(stacks[0]);
  p.matrix[1] = matrix(stacks[1]);
  p.x = x;
  p.y = act;
  p.block_experts = block_experts;
  p.blocks = blocks;
  p.rows = rows;
  p.n = stacks[0].n;
  p.k = stacks[0].k;
  p.first_expert = stacks[0].first_expert;
  p.experts = stacks[0].experts;
  const int wide = stacks[0].entries > stacks[1].entries ? stacks[0].entries : stacks[1].entries;
  cudaError_t error = rows > 8 ? launch<2, true>(p, shared_bytes(wide, rows, p.k), stream, sm_count)
                               : launch<1, true>(p, shared_bytes(wide, rows, p.k), stream, sm_count);
  if (error != cudaSuccess) return error;
  p.matrix[0] = matrix(stacks[2]);
  p.x = act;
  p.y = y;
  p.n = stacks[2].n;
  p.k = stacks[2].k;
  return rows > 8 ? launch<2, false>(p, shared_bytes(stacks[2].entries, rows, p.k), stream, sm_count)
                  : launch<1, false>(p, shared_bytes(stacks[2].entries, rows, p.k), stream, sm_count);
}

}  // namespace sageb200
