// SAGE packed prefill GEMM for more than 16 activation rows: dequantise weight tiles
// into shared memory, feed tcgen05 FP16 MMAs with FP32 accumulators in tensor memory.
//
// Replaces the reference's sage_gemm_kernel_base / _m64 (csrc/sage/sage_gemm_cuda.cu:35-197,
// 272-445: 32x64 / 64x64 tiles on nvcuda::wmma, every activation tile re-decoding the
// whole weight) and its separate split-K reduce kernel (:199-206).
//
// Orientation ("swap AB"): the MMA's M dimension is 128 OUTPUT rows (eight packed 16-row
// tiles), its N dimension is up to 256 activation rows (tokens), so any token count that
// is a multiple of 16 maps onto one instruction shape without padding waste:
//     D[128 outputs][TN tokens] += Wtile[128][64] . Xq[TN][64]^T      per 64-channel stage
// Both operands are K-major in shared memory with the 128-byte swizzle:
//   A (weights)      written by 16 decode warps with 16-byte stores, bit-exact
//                    w = fp16_rn(float(+-dir) * fmaf(code, step, min))
//                    (reference csrc/sage/sage_gemm_cuda.cu:117-131)
//   B (activations)  one TMA tile load per stage from the activations in quantised
//                    channel order (no cluster multicast)
// One elected thread issues tcgen05.mma (cta_group::1, kind::f16, M=128, N=TN, K=16, four per
// stage) and releases stages with tcgen05.commit; the decode warps then read the
// accumulator with tcgen05.ld and store FP16 outputs.
//
// Every wait is bounded: a wait that exceeds its time limit sets an abort flag in shared
// memory (all later waits return at once), records SAGEB200_ERR_TIMEOUT in the status word
// and the CTA still frees its tensor memory before returning.
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstring>

#include "sage_common.cuh"
#include "sage_kernels.h"
#include "sage_rows.cuh"
#include "sage_tcgen05.cuh"

namespace sageb200 {
namespace {

constexpr int kDecodeWarps = 16;
constexpr int kDecodeThreads = kDecodeWarps * 32;
constexpr int kTmaWarp = kDecodeWarps;
constexpr int kMmaWarp = kDecodeWarps + 1;
constexpr int kGemmThreads = (kDecodeWarps + 2) * 32;
constexpr int kTileRows = 128;             // output rows per CTA = MMA M
constexpr int kDecodeGroups = kDecodeThreads / kTileRows;  // groups of decode warps, each on a stage of its own
constexpr int kStageK = 64;                // channels per stage = one 128-byte swizzle row
constexpr int kAStageBytes = kTileRows * kStageK * 2;
constexpr int kMaxStages = 6;
constexpr int kBookReplicas = 8;           // codebook copies in shared memory: lane % 8 reads its own
constexpr int kBookBytes = 256 * 16 * kBookReplicas;
constexpr int kGemmSharedLimit = 226 * 1024;  // dynamic shared memory the kernel opts into (227 KiB per CTA less its static words)

// One packed linear of a launch.
struct GemmProblem {
  const uint32_t *codes;
  const uint32_t *radii;
  const uint32_t *grid;
  const uint32_t *book;
  const __half *mins;   // SPHQuant only
  const void *bias;     // [n] in the output's type, or null
  void *y;
  int n, tiles;
  int entries, dbits;
  int row_block_begin;  // its first block of 128 output rows in the launch
};

struct GemmParams {
  CUtensorMap x_map[kMaxGemmProblems];  // the problems' activations
  GemmProblem problem[kMaxGemmProblems];
  int count;
  int *status;          // device-visible status word (0 = ok)
  int rows, groups;
  int out_bf16;         // the outputs' type: the FP16 result (of the operator) turned into BF16, or FP16
  int tokens_per_cta;   // TN: multiple of 16, 16..256 (tokens of ONE accumulator)
  int stages;
  int tmem_columns;     // power of two >= max(32, TN); 512 with two accumulators
  int accumulators;     // 1 or 2 token blocks per CTA: one decoded weight stage feeds both
  long long *trace;     // profiling build only: eight clock sums per CTA (null otherwise)
  // output tiles (row blocks x groups of `accumulators` token blocks, row blocks fastest): the first
  // main_tiles have a CTA each, the others k_splits.  CTA z of those runs the 128-channel groups
  // [z * groups_per_split, ...), leaves its FP32 tile in `partial`, and the last CTA of a tile to
  // arrive (counter) adds the splits in index order and writes the FP16 output
  int row_blocks, tiles, main_tiles;
  int k_splits, groups_per_split;
  // packed format: 0 = SAGE (tiled words, planar codebook, (min, step) grid); 1 = SPHQuant
  // (row-major 16-bit codes in `codes`, per-(row, group) high radius word in `radii`, FP16 scales
  // in `grid` and minimums in `mins`, entry-major 64 x 8 codebook, n rows need no padding)
  int format;
  float *partial;       // [k_splits][tiles][accumulators * TN tokens][128 rows]
  unsigned *counters;   // [tiles][8]: one word per part of a tile, zero before and after the launch
};

#ifdef SAGEB200_TRACE
#define GEMM_CLOCK() clock64()
#else
#define GEMM_CLOCK() 0ll
#endif

// Codebook entry by shared address; free to be scheduled early (the codebook never changes, and the
// address depends on packed words that are loaded after it was written).
__device__ __forceinline__ uint4 book_entry(uint32_t address) {
  uint4 v;
  asm("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(address));
  return v;
}

// Two weights: fp16_rn(float(direction) * radius) of each half of `direction`.
__device__ __forceinline__ uint32_t exact_pair(uint32_t direction, float radius) {
  const float2 d = __half22float2(*reinterpret_cast<const __half2 *>(&direction));
  const __half2 w = __floats2half2_rn(d.x * radius, d.y * radius);
  return *reinterpret_cast<const uint32_t *>(&w);
}

// ---------------------------------------------------------------- the kernel

// Dynamic shared memory, 1024-byte aligned by hand:
//   [A stages: stages x 16 KiB][B stages: stages x TN*128][codebook 32 KiB][barriers]
// kPair: the grid is launched in clusters of two CTAs along x (two neighbouring row blocks) that
// run cta_group::2 MMAs.  Both CTAs decode their own 128 rows and load their own half of every
// activation tile; the even CTA (the leader) issues the MMAs and owns the "stage full" barriers:
// its own decode warps arrive there, its TMA thread announces both CTAs' bytes, the odd CTA's
// loads complete on it remotely, and the odd CTA's otherwise idle MMA warp forwards ONE arrival
// per stage once its own decode warps are done.  Stage-free and accumulator-ready arrivals are
// multicast to both CTAs by tcgen05.commit.
template <bool kPair>
__global__ void __launch_bounds__(kGemmThreads, 1)
    sage_gemm_tc_kernel(const __grid_constant__ GemmParams p) {
  extern __shared__ unsigned char raw_shared[];
  __shared__ uint32_t tmem_base_holder;
  __shared__ int abort_flag;
  __shared__ int split_last;

  const uint32_t raw = smem_address(raw_shared);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char *aligned = raw_shared + (base - raw);
  const int tn = p.tokens_per_cta;
  const int accumulators = p.accumulators;
  const int tile_tokens = kPair ? tn / 2 : tn;        // tokens of one accumulator this CTA loads
  const int b_tile_bytes = tile_tokens * kStageK * 2; // one token block's activations of a stage (this CTA's part)
  const uint32_t pair_rank = kPair ? cluster_cta_rank() : 0u;
  const bool leader = pair_rank == 0;
  const int b_stage_bytes = accumulators * b_tile_bytes;
  const uint32_t a_base = base;
  const uint32_t b_base = a_base + p.stages * kAStageBytes;
  const uint32_t book_address = b_base + p.stages * b_stage_bytes;
  uint4 *book_shared = reinterpret_cast<uint4 *>(aligned + (book_address - base));
  const uint32_t bar_base = book_address + kBookBytes;
  // barriers: full[stages], empty[stages], accumulator
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
  const uint32_t accum_bar = bar_base + 8u * (2 * kMaxStages);

  // Programmatic dependent launch: the next kernel of the stream may be scheduled at once; this
  // kernel's set-up, and its decode warps' first stages (packed weights and codebook: data no
  // kernel writes), run while the previous kernel (the gather pre-pass) still works.  Only the
  // activation loads and every global write wait for the previous kernel.
  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (known to be the same in all lanes)
  const int lane = tid & 31;
  // several linears of one input lie side by side along the grid's row blocks
  int problem = 0;
  const int split_tiles = p.tiles - p.main_tiles;
  const bool split = static_cast<int>(blockIdx.x) >= p.main_tiles;
  const int split_cta = static_cast<int>(blockIdx.x) - p.main_tiles;
  const int split_index = split ? split_cta / split_tiles : 0;
  const int split_tile = split ? split_cta - split_index * split_tiles : 0;  // among the split tiles
  const int tile_index = split ? p.main_tiles + split_tile : static_cast<int>(blockIdx.x);
  const int tile_row = tile_index / p.row_blocks, tile_column = tile_index - tile_row * p.row_blocks;
  while (problem + 1 < p.count && tile_column >= p.problem[problem + 1].row_block_begin) ++problem;
  const GemmProblem &q = p.problem[problem];
  const int row_block = tile_column - q.row_block_begin;  // 128 output rows
  const int token_block = tile_row * accumulators;        // first of this CTA's blocks of TN tokens
  const int group_begin = split_index * p.groups_per_split;
  const int group_end = split ? min(p.groups, group_begin + p.groups_per_split) : p.groups;
  const int stage_first = 2 * group_begin;            // first 64-channel stage of this CTA's K range
  const int stages_k = 2 * (group_end - group_begin); // stages this CTA runs

  if (tid == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      // full: the stage's decode warps (one arrival each); + the TMA thread's announcement (and, for
      // a leader, the odd CTA's forwarded arrival)
      mbarrier_init(full_bar(s), kDecodeWarps / kDecodeGroups + (kPair ? (leader ? 2 : 0) : 1));
      mbarrier_init(empty_bar(s), 1);
    }
    mbarrier_init(accum_bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kTmaWarp) {
    if constexpr (kPair) {  // (both CTAs, the same warp, the same holder address)
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_address(&tmem_base_holder)),
                   "r"(static_cast<uint32_t>(p.tmem_columns))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                       smem_address(&tmem_base_holder)),
                   "r"(static_cast<uint32_t>(p.tmem_columns))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  // codebook, interleaved: entry e = 16 bytes (dims 0..7)
  for (int e = tid; e < q.entries; e += kGemmThreads) {
    uint4 entry;
    if (p.format == 1) {
      entry = reinterpret_cast<const uint4 *>(q.book)[e];
    } else {
      entry.x = q.book[e];
      entry.y = q.book[q.entries + e];
      entry.z = q.book[2 * q.entries + e];
      entry.w = q.book[3 * q.entries + e];
    }
    // eight copies, entry-major: lane l reads copy l % 8, so the eight lanes of a quarter warp hit
    // eight different 16-byte bank groups whatever their indices (rotated fill order for the same reason)
#pragma unroll
    for (int r = 0; r < kBookReplicas; ++r) book_shared[e * kBookReplicas + ((r + tid) & (kBookReplicas - 1))] = entry;
  }
  tcgen05_fence_before();
  __syncthreads();
  if constexpr (kPair) cluster_sync_all();  // (no remote arrival before the other CTA's barriers exist)
  tcgen05_fence_after();
  // (only now: a later kernel that takes tensor memory and then waits for this one must not be able to take
  //  the columns that a CTA of this grid still has to get)
  pdl_launch_dependents();
  const uint32_t tmem_base = tmem_base_holder;
  volatile int *abort_ptr = &abort_flag;

  if (warp < kDecodeWarps) {
    // ---------------- weight decode producers: four groups of four warps, group i decodes the stages
    //                  i, i + 4, ...; thread = one output row of the stage, its eight vectors in one
    //                  unrolled run.  A stage's decode is a chain of latencies (free-stage wait,
    //                  codebook load, conversions, store, proxy fence, arrival): with all sixteen
    //                  warps on one stage the chains of successive stages ran one after the other;
    //                  with four stages in the making they overlap, and eight independent vectors
    //                  per thread fill the issue slots.  With the counted MMA and TMA loops below:
    //                  5120 -> 25600 at 2048 rows 448 -> 384 us (1400 TFLOP/s; 1103 cycles a stage,
    //                  1084 of them the tensor pipe's), at 33 rows 113 -> 66 us (bound by the
    //                  decode's own instructions, about 57 issue cycles per vector and scheduler).
    //                  With fewer than four stage buffers only as many groups work: a group that
    //                  finishes stage i knows that the MMAs of stage i - buffers are done, so a wait
    //                  for stage i + groups can only be told from one two rounds earlier (the
    //                  barrier's phase bit) if groups <= buffers.
    const int row = tid & (kTileRows - 1);
    const int groups = min(kDecodeGroups, p.stages);
    const int decode_group = tid / kTileRows < groups ? tid / kTileRows : stages_k;  // (no stage of its own)
    const int out_row = row_block * kTileRows + row;
    const int tile = out_row >> 4;
    // rows past the last packed tile (SAGE) / past n (SPHQuant) decode to zero
    const bool row_valid = p.format == 1 ? out_row < q.n : tile < q.tiles;
    const size_t cell_base = (static_cast<size_t>(row_valid ? tile : 0) * p.groups) * 16 + (out_row & 15);
    const size_t sph_row = static_cast<size_t>(row_valid ? out_row : 0);
    const uint32_t row_offset = static_cast<uint32_t>(row >> 3) * 1024u + static_cast<uint32_t>(row & 7) * 128u;
    const uint32_t book_lane = book_address + static_cast<uint32_t>(lane & (kBookReplicas - 1)) * 16u;
    // bit fields of a code for D direction bits: the codebook offset (entries 128 bytes apart) and the
    // radius code as 1 + code / 16 in an FP32 mantissa, low bits from the code, high two from the row's word
    const uint32_t index_mask = static_cast<uint32_t>(q.entries - 1) << 7;
    const uint32_t hi_shift = 27u - q.dbits, hi_mask = 3u << hi_shift;
    const uint32_t lo_mask = ((1u << (8 - q.dbits)) - 1u) << 19, lo_left = 11u - q.dbits, lo_right = 5u + q.dbits;
    // The thread's packed words of a stage (four code words, the radius word, the grid endpoints) are
    // fetched two of its own stages ahead: they come from cold HBM, and a load issued at the point
    // of use would stall the group for a full memory latency every stage.
    struct StageWords {
      uint4 codes;
      uint32_t radius, endpoints;
    };
    const bool wide_codes = (reinterpret_cast<uintptr_t>(q.codes) & 15) == 0;
    auto fetch_stage = [&](int ks) {
      StageWords g = {make_uint4(0u, 0u, 0u, 0u), 0u, 0u};
      if (row_valid && ks < stages_k) {
        const int group = group_begin + (ks >> 1);
        const size_t cell = p.format == 1 ? sph_row * p.groups + group : cell_base + static_cast<size_t>(group) * 16;
        const uint32_t *codes = q.codes + cell * 8 + 4 * (ks & 1);  // (both formats: 32 bytes per row and group)
        if (wide_codes) {
          g.codes = ldg_stream_u4(codes);
        } else {
          g.codes = make_uint4(ldg_stream_u1(codes), ldg_stream_u1(codes + 1), ldg_stream_u1(codes + 2),
                               ldg_stream_u1(codes + 3));
        }
        g.radius = ldg_stream_u1(q.radii + cell);
        if (p.format == 1) {
          const uint32_t minimum = reinterpret_cast<const unsigned short *>(q.mins)[cell];
          const uint32_t scale = reinterpret_cast<const unsigned short *>(q.grid)[cell];
          g.endpoints = minimum | (scale << 16);  // (min, step) as in the SAGE grid
        } else {
          g.endpoints = ldg_stream_u1(q.grid + cell);
        }
      }
      return g;
    };
    StageWords ahead0 = fetch_stage(decode_group), ahead1 = fetch_stage(decode_group + groups);
    long long waited = 0, worked = 0, fenced = 0, stored = 0;  // (profiling build) clock sums of the phases
    [[maybe_unused]] const long long decode_begin = GEMM_CLOCK();
    bool alive = true;
    int s = decode_group;  // stage buffer of ks, and the phase of its round
    uint32_t phase = 0;
    for (int ks = decode_group; ks < stages_k; ks += groups) {
      const StageWords g = ahead0;
      ahead0 = ahead1;
      ahead1 = fetch_stage(ks + 2 * groups);
      const float2 e = __half22float2(*reinterpret_cast<const __half2 *>(&g.endpoints));
      const uint32_t radius_half = g.radius >> (16 * (ks & 1));
      const uint32_t high[2] = {(radius_half & 0xffu) << hi_shift, (radius_half >> 8) << hi_shift};  // four vectors each
      const uint32_t words[4] = {g.codes.x, g.codes.y, g.codes.z, g.codes.w};
      const long long t0 = GEMM_CLOCK();
      alive = bounded_wait(empty_bar(s), phase ^ 1u, abort_ptr, p.status);
      if (!alive) break;
      const long long t1 = GEMM_CLOCK();
      const uint32_t stage_address = a_base + s * kAStageBytes + row_offset;
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        const uint32_t word = words[v >> 1];
        uint4 out = make_uint4(0u, 0u, 0u, 0u);
        if (row_valid) {
          const uint32_t offset = (v & 1 ? word >> 17 : word >> 1) & index_mask;
          const uint32_t low = (v & 1 ? word >> lo_right : word << lo_left) & lo_mask;
          const uint32_t bits = ((high[v >> 2] >> (2 * (v & 3))) & hi_mask) | low | 0x3f800000u;
          // (the code itself, exactly, and then the reference's one FMA)
          const float radius = fmaf(fmaf(__uint_as_float(bits), 16.0f, -16.0f), e.y, e.x);
          const uint4 dir = book_entry(book_lane + offset);
          const uint32_t signs = (word >> (v & 1 ? 16 : 0)) & 0xffu;
          // sign bits 2q and 2q+1 land on bits 15 and 31 of one product (one multiply and one
          // three-input logic operation per pair of weights; the other product bits are masked)
          out.x = exact_pair(dir.x ^ ((signs * 0x40008000u) & 0x80008000u), radius);
          out.y = exact_pair(dir.y ^ ((signs * 0x10002000u) & 0x80008000u), radius);
          out.z = exact_pair(dir.z ^ ((signs * 0x04000800u) & 0x80008000u), radius);
          out.w = exact_pair(dir.w ^ ((signs * 0x01000200u) & 0x80008000u), radius);
        }
        sts_u4(stage_address + static_cast<uint32_t>(v ^ (row & 7)) * 16u, out);
      }
      const long long t2 = GEMM_CLOCK();
      fence_proxy_async_shared();
      const long long t3 = GEMM_CLOCK();
      __syncwarp();
      if (lane == 0) mbarrier_arrive(full_bar(s));
      s += groups;
      if (s >= p.stages) s -= p.stages, phase ^= 1u;  // (groups <= buffers: at most one wrap)
      waited += t1 - t0;
      worked += GEMM_CLOCK() - t1;
      fenced += t3 - t2;
      stored += t2 - t1;
    }
#ifdef SAGEB200_TRACE
    if (p.trace && (tid == 0 || tid == kDecodeThreads - 1)) {
      long long *record = p.trace + static_cast<size_t>(tile_index) * 16 + (tid == 0 ? 0 : 3);
      record[0] = waited;
      record[1] = worked;
      record[2] = GEMM_CLOCK() - decode_begin;
      if (tid == 0) {
        p.trace[static_cast<size_t>(tile_index) * 16 + 10] = stored;
        p.trace[static_cast<size_t>(tile_index) * 16 + 11] = fenced;
      }
    }
    const long long epilogue_begin = GEMM_CLOCK();
#endif
    // ---------------- epilogue: TMEM -> registers -> FP16 global
    pdl_wait();  // (long since satisfied: the MMAs needed the activations; required before global writes)
    if (alive) alive = bounded_wait(accum_bar, 0, abort_ptr, p.status);
    alive = __all_sync(0xffffffffu, alive);  // tcgen05.ld is warp-collective
    tcgen05_fence_after();
#ifdef SAGEB200_TRACE
    if (p.trace && tid == 0)
      p.trace[static_cast<size_t>(tile_index) * 16 + 12] = GEMM_CLOCK() - epilogue_begin;
#endif
    {
      constexpr int kColumnParts = kDecodeWarps / 4;
      const int quarter = warp & 3;                 // TMEM lanes 32*quarter .. +31
      const int column_part = warp >> 2;            // warps 0-3: first part of the tokens, ...
      const int columns_per_part = (tn / 16 + kColumnParts - 1) / kColumnParts * 16;
      const int column_begin = column_part * columns_per_part;
      const int column_end = min(tn, column_begin + columns_per_part);
      const int out = row_block * kTileRows + quarter * 32 + lane;
      // The accumulator has output rows on lanes and tokens on columns, y is [token][row]: a lane
      // storing its own values writes 2 bytes per instruction (64 bytes per warp), and the store
      // instructions themselves then bound the epilogue.  Each warp therefore turns 16 tokens x 32
      // rows around through 1 KiB of the (now idle) weight stages and stores 16 bytes per lane:
      // eight rows of one token.  Rows beyond n, or an n / y that breaks the 16-byte alignment,
      // take the direct stores.
      const uint32_t turn = a_base + static_cast<uint32_t>(warp) * 1024u;
      const int out_base = row_block * kTileRows + quarter * 32;
      const bool wide = (q.n & 7) == 0 && out_base + 32 <= q.n && (reinterpret_cast<uintptr_t>(q.y) & 15) == 0;
      // (FP16 and BF16 outputs are moved as 16-bit words)
      unsigned short *const y = static_cast<unsigned short *>(q.y);
      const float bias = q.bias && out < q.n ? (p.out_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16 *>(q.bias)[out])
                                                           : __half2float(static_cast<const __half *>(q.bias)[out]))
                                             : 0.0f;
      // the operator's FP16 result, then what the module makes of it: its input's type, and the bias in that type
      auto finish = [&](float v) -> unsigned short {
        const __half h = __float2half_rn(v);
        if (p.out_bf16) {
          __nv_bfloat16 b = __float2bfloat16_rn(__half2float(h));
          if (q.bias) b = __float2bfloat16_rn(__bfloat162float(b) + bias);
          return __bfloat16_as_ushort(b);
        }
        return __half_as_ushort(q.bias ? __float2half_rn(__half2float(h) + bias) : h);
      };
      auto store_chunk = [&](const uint32_t (&r)[16], int a, int c) {
        const int token_base = (token_block + a) * tn + c;
        if (wide) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            asm volatile("st.shared.u16 [%0], %1;" ::"r"(turn + i * 64u + lane * 2u), "h"(finish(__uint_as_float(r[i]))));
          }
          __syncwarp();
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            const int piece = lane + 32 * half;          // token = piece / 4, eight rows = piece % 4
            const int token = token_base + (piece >> 2);
            const uint4 v = lds_u4(turn + static_cast<uint32_t>(piece) * 16u);
            if (token < p.rows)
              *reinterpret_cast<uint4 *>(y + static_cast<size_t>(token) * q.n + out_base + (piece & 3) * 8) = v;
          }
          __syncwarp();
        } else if (out < q.n) {
#pragma unroll
          for (int i = 0; i < 16; ++i) {
            const int token = token_base + i;
            if (token < p.rows)
              y[static_cast<size_t>(token) * q.n + out] = finish(__uint_as_float(r[i]));
          }
        }
      };
      if (!split) {
        if (alive) {
          for (int a = 0; a < accumulators; ++a) {
            for (int c = column_begin; c < column_end; c += 16) {
              uint32_t r[16];
              tmem_load_16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * 256 + c, r);
              tmem_load_wait();
              store_chunk(r, a, c);
            }
          }
        }
      } else {
        // ---- split K: FP32 tile to scratch, in up to three PARTS (runs of 16-token chunks).  Split z
        //      writes the parts in the order z, z+1, ...; whoever completes a part's arrival
        //      counter adds that part's splits in index order and stores it.  CTAs that finish
        //      together are each the last writer of a different part, so the reduction spreads over
        //      the tile's CTAs without anyone waiting (a straggler simply reduces more parts).
        const int tile_id = split_tile;
        const size_t tile_floats = static_cast<size_t>(accumulators) * tn * kTileRows;
        const size_t split_stride = static_cast<size_t>(split_tiles) * tile_floats;
        float *tile_partial = p.partial + static_cast<size_t>(tile_id) * tile_floats;
        float *mine = tile_partial + split_index * split_stride;
        const int chunks_per_accumulator = tn / 16;
        const int chunks = accumulators * chunks_per_accumulator;
        const size_t lane_row = static_cast<size_t>(quarter) * 32 + lane;
        [[maybe_unused]] long long wrote = 0, synced = 0, reduced = 0;
        const int parts = min(p.k_splits, 3);  // (each part costs a fence and two barriers)
        for (int step = 0; step < parts; ++step) {
          const long long e0 = GEMM_CLOCK();
          const int part = (split_index + step) % parts;
          const int chunk_begin = part * chunks / parts, chunk_end = (part + 1) * chunks / parts;
          if (alive) {
            for (int chunk = chunk_begin + column_part; chunk < chunk_end; chunk += kColumnParts) {
              const int a = chunk / chunks_per_accumulator, c = (chunk % chunks_per_accumulator) * 16;
              uint32_t r[16];
              tmem_load_16(tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + a * 256 + c, r);
              tmem_load_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i)
                mine[static_cast<size_t>(a * tn + c + i) * kTileRows + lane_row] = __uint_as_float(r[i]);
            }
          }
          const long long e1 = GEMM_CLOCK();
          __threadfence();
          asm volatile("bar.sync 1, %0;" ::"n"(kDecodeThreads) : "memory");  // (decode warps only, all of them)
          if (tid == 0) {
            unsigned *counter = p.counters + tile_id * 8 + part;
            const bool last = atomicAdd(counter, 1u) == static_cast<unsigned>(p.k_splits - 1);
            if (last) *counter = 0u;  // (zero again for the next launch)
            split_last = last && abort_flag == 0;
          }
          asm volatile("bar.sync 1, %0;" ::"n"(kDecodeThreads) : "memory");
          const long long e2 = GEMM_CLOCK();
          wrote += e1 - e0;
          synced += e2 - e1;
          if (split_last) {
            __threadfence();
            for (int chunk = chunk_begin + column_part; chunk < chunk_end; chunk += kColumnParts) {
              const int a = chunk / chunks_per_accumulator, c = (chunk % chunks_per_accumulator) * 16;
              float sum[16];
#pragma unroll
              for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
              // (index order: the result does not depend on who came last; two splits' loads in
              //  flight at a time, the adds still in index order)
              const float *base = tile_partial + static_cast<size_t>(a * tn + c) * kTileRows + lane_row;
              int z = 0;
              for (; z + 1 < p.k_splits; z += 2) {
                float first[16], second[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) first[i] = __ldcg(base + z * split_stride + static_cast<size_t>(i) * kTileRows);
#pragma unroll
                for (int i = 0; i < 16; ++i) second[i] = __ldcg(base + (z + 1) * split_stride + static_cast<size_t>(i) * kTileRows);
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[i] = (sum[i] + first[i]) + second[i];
              }
              if (z < p.k_splits) {
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[i] += __ldcg(base + z * split_stride + static_cast<size_t>(i) * kTileRows);
              }
              uint32_t r[16];
#pragma unroll
              for (int i = 0; i < 16; ++i) r[i] = __float_as_uint(sum[i]);
              store_chunk(r, a, c);
            }
          }
          reduced += GEMM_CLOCK() - e2;
        }
#ifdef SAGEB200_TRACE
        if (p.trace && tid == 0) {
          long long *record = p.trace + static_cast<size_t>(tile_index) * 16;
          record[13] = wrote;
          record[14] = synced;
          record[15] = reduced;
        }
#endif
      }
    }
#ifdef SAGEB200_TRACE
    if (p.trace && tid == 0)
      p.trace[static_cast<size_t>(tile_index) * 16 + 6] = GEMM_CLOCK() - epilogue_begin;
#endif
  } else if (warp == kTmaWarp) {
    // ---------------- activation tile loads (by one lane)
    {
      pdl_wait();  // the activations are the previous kernel's output
      bool alive = true;
      long long waited = 0;
      int s = 0;
      uint32_t phase = 0;
      for (int ks = 0; ks < stages_k; ++ks) {
        const long long t0 = GEMM_CLOCK();
        alive = __all_sync(0xffffffffu, bounded_wait(empty_bar(s), phase ^ 1u, abort_ptr, p.status));
        if (!alive) break;
        waited += GEMM_CLOCK() - t0;
        if (elect_one()) {
          if constexpr (kPair) {
            // the leader announces both CTAs' bytes; each CTA loads its half of every token block and
            // the copies complete on the leader's barrier
            if (leader) mbarrier_arrive_expect_tx(full_bar(s), static_cast<uint32_t>(2 * b_stage_bytes));
            for (int a = 0; a < accumulators; ++a)
              tma_load_2d_pair(b_base + s * b_stage_bytes + a * b_tile_bytes, &p.x_map[problem], (stage_first + ks) * kStageK,
                               (token_block + a) * tn + static_cast<int>(pair_rank) * tile_tokens, full_bar(s));
          } else {
            mbarrier_arrive_expect_tx(full_bar(s), static_cast<uint32_t>(b_stage_bytes));
            for (int a = 0; a < accumulators; ++a)  // (a block past the last token reads the fill value)
              tma_load_2d(b_base + s * b_stage_bytes + a * b_tile_bytes, &p.x_map[problem], (stage_first + ks) * kStageK,
                          (token_block + a) * tn, full_bar(s));
          }
        }
        __syncwarp();
        if (++s == p.stages) s = 0, phase ^= 1u;
      }
#ifdef SAGEB200_TRACE
      if (p.trace && lane == 0) p.trace[static_cast<size_t>(tile_index) * 16 + 7] = waited;
#endif
    }
  } else {
    // ---------------- MMA issue
    if (kPair && !leader) {
      // ---------------- odd CTA of a pair: forward "my decode warps have filled the stage"
      if (lane == 0) {
        int s = 0;
        uint32_t phase = 0;
        for (int ks = 0; ks < stages_k; ++ks) {
          if (!bounded_wait(full_bar(s), phase, abort_ptr, p.status)) break;
          mbarrier_arrive_leader(full_bar(s));
          if (++s == p.stages) s = 0, phase ^= 1u;
        }
      }
    } else {
      const uint32_t idesc = instruction_descriptor(kPair ? 2 * kTileRows : kTileRows, tn);
      bool alive = true;
      long long waited = 0;
      [[maybe_unused]] const long long mma_begin = GEMM_CLOCK();
      // One lane issues everything here, beside four decode warps on the same scheduler, so each
      // instruction costs a turn: stage index and phase are counted (no division), operand
      // descriptors are 32-bit sums of constants.
      const uint32_t a_low = descriptor_low(a_base), b_low = descriptor_low(b_base);
      const uint32_t b_stage = static_cast<uint32_t>(b_stage_bytes) >> 4, b_tile = static_cast<uint32_t>(b_tile_bytes) >> 4;
      const uint32_t stage_count = static_cast<uint32_t>(p.stages);
      uint32_t s = 0, phase = 0;
      auto issue = [&](uint32_t tmem, uint32_t a, uint32_t b, uint32_t first) {
#pragma unroll
        for (uint32_t j = 0; j < kStageK / 16; ++j) {
          // advancing 16 channels = 32 bytes = 2 units of the descriptor's address field
          if constexpr (kPair) umma_f16_pair(tmem, a + 2 * j, b + 2 * j, idesc, j ? 1u : first);
          else umma_f16(tmem, a + 2 * j, b + 2 * j, idesc, j ? 1u : first);
        }
      };
      for (int ks = 0; ks < stages_k; ++ks) {
        const long long t0 = GEMM_CLOCK();
        alive = __all_sync(0xffffffffu, bounded_wait(full_bar(s), phase, abort_ptr, p.status));
        if (!alive) break;
        waited += GEMM_CLOCK() - t0;
        tcgen05_fence_after();
        const uint32_t a = a_low + s * (kAStageBytes >> 4), b = b_low + s * b_stage;
        if (elect_one()) {
          issue(tmem_base, a, b, ks ? 1u : 0u);
          if (accumulators == 2) issue(tmem_base + 256, a, b + b_tile, ks ? 1u : 0u);
          if constexpr (kPair) umma_commit_pair(empty_bar(s));
          else umma_commit(empty_bar(s));
        }
        __syncwarp();
        if (++s == stage_count) s = 0, phase ^= 1u;
      }
      if (alive && elect_one()) {
        if constexpr (kPair) umma_commit_pair(accum_bar);
        else umma_commit(accum_bar);
      }
      __syncwarp();
#ifdef SAGEB200_TRACE
      if (p.trace && lane == 0) {
        long long *record = p.trace + static_cast<size_t>(tile_index) * 16;
        record[8] = waited;
        record[9] = GEMM_CLOCK() - mma_begin;
      }
#endif
    }
  }

  // Let in-flight TMA copies land before the CTA's shared memory goes away: every issued
  // load targets a full barrier that the MMA thread has waited on unless we aborted; on
  // abort, wait (bounded) for each stage's barrier once more.
  tcgen05_fence_before();
  __syncthreads();
  // (a pair leaves together: the leader's MMAs read the other CTA's shared memory, and both CTAs'
  //  barriers receive remote arrivals until the last commit)
  if constexpr (kPair) cluster_sync_all();
  if (warp == kTmaWarp) {
    if (abort_flag && lane == 0) {
      const unsigned long long begin = global_timer();
      while (global_timer() - begin < 2000000ull) __nanosleep(1000);  // 2 ms grace for copies in flight
    }
    __syncwarp();
    if constexpr (kPair)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                   "r"(static_cast<uint32_t>(p.tmem_columns))
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                   "r"(static_cast<uint32_t>(p.tmem_columns))
                   : "memory");
  }
}

// x_q[m][j] = x[m][perm[j]]  (or a plain copy when perm is null).  One CTA per activation row at a
// time: the row is brought into shared memory with 16-byte (or, for an odd base address, 2-byte)
// loads, the permutation is read eight indices at a time, the gathered values come out of shared
// memory and leave as 16-byte stores - no 2-byte global loads, which cost a sector each.
constexpr int kGatherThreads = 256;
__device__ __forceinline__ uint4 as_halves(uint4 v, const __half *) { return v; }
__device__ __forceinline__ uint4 as_halves(uint4 v, const __nv_bfloat16 *) {
  const __nv_bfloat162 *b = reinterpret_cast<const __nv_bfloat162 *>(&v);
  uint4 out;
  __half2 *h = reinterpret_cast<__half2 *>(&out);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const float2 f = __bfloat1622float2(b[c]);
    h[c] = __floats2half2_rn(f.x, f.y);
  }
  return out;
}
// (T: FP16, or BF16 rounded to FP16 on the way in)
template <typename T>
__global__ void __launch_bounds__(kGatherThreads) sage_gather_kernel(const T *__restrict__ x,
                                                                     const int32_t *__restrict__ perm,
                                                                     __half *__restrict__ xq, int rows, int k) {
  extern __shared__ __align__(16) unsigned char gather_shared[];
  __half *row_shared = reinterpret_cast<__half *>(gather_shared);
  pdl_launch_dependents();  // (the GEMM behind this kernel sets up and decodes its first stages meanwhile)
  pdl_wait();               // the activations are the previous kernel's output
  const int vectors = k >> 3;
  const bool perm_wide = (reinterpret_cast<uintptr_t>(perm) & 15) == 0;
  for (int m = blockIdx.x; m < rows; m += gridDim.x) {
    const T *source = x + static_cast<size_t>(m) * k;
    if ((reinterpret_cast<uintptr_t>(source) & 15) == 0) {
      for (int v = threadIdx.x; v < vectors; v += kGatherThreads)
        reinterpret_cast<uint4 *>(row_shared)[v] = as_halves(reinterpret_cast<const uint4 *>(source)[v], source);
    } else {
      for (int j = threadIdx.x; j < k; j += kGatherThreads) row_shared[j] = __float2half_rn(static_cast<float>(source[j]));
    }
    __syncthreads();
    uint4 *destination = reinterpret_cast<uint4 *>(xq + static_cast<size_t>(m) * k);
    for (int v = threadIdx.x; v < vectors; v += kGatherThreads) {
      if (perm == nullptr) {
        destination[v] = reinterpret_cast<const uint4 *>(row_shared)[v];
        continue;
      }
      int index[8];
      if (perm_wide) {
        *reinterpret_cast<int4 *>(index) = reinterpret_cast<const int4 *>(perm)[2 * v];
        *reinterpret_cast<int4 *>(index + 4) = reinterpret_cast<const int4 *>(perm)[2 * v + 1];
      } else {
#pragma unroll
        for (int d = 0; d < 8; ++d) index[d] = perm[v * 8 + d];
      }
      __align__(16) __half values[8];
#pragma unroll
      for (int d = 0; d < 8; ++d) values[d] = row_shared[index[d]];
      destination[v] = *reinterpret_cast<const uint4 *>(values);
    }
    __syncthreads();
  }
}

// The same for many rows, four at a time (sage_rows.cuh).  Measured at 2048 rows of 9728: 30 -> 16 us.
constexpr int kGatherFourThreads = 512;
constexpr int kGatherFourRows = 512;       // rows from which four at a time still fill the SMs
constexpr int kGatherFourChannels = 25600; // 8 bytes of shared memory each
template <typename T>
__global__ void __launch_bounds__(kGatherFourThreads) sage_gather_four_kernel(const T *__restrict__ x,
                                                                              const int32_t *__restrict__ perm,
                                                                              __half *__restrict__ xq, int rows, int k) {
  extern __shared__ __align__(16) uint2 four_rows[];
  pdl_launch_dependents();
  pdl_wait();
  const int first = blockIdx.x * kRowsAtOnce;
  for (int v = threadIdx.x; v < (k >> 3); v += kGatherFourThreads) {
    uint4 row[kRowsAtOnce];
#pragma unroll
    for (int m = 0; m < kRowsAtOnce; ++m)  // (a row past the last repeats it and is not stored)
      row[m] = as_halves(reinterpret_cast<const uint4 *>(x + static_cast<size_t>(min(first + m, rows - 1)) * k)[v], x);
    put_four_rows(four_rows, v, row);
  }
  __syncthreads();
  write_four_rows(four_rows, perm, xq, first, rows, k, kGatherFourThreads);
}

}  // namespace

namespace {
template <typename Function>
Function driver_function(const char *name) {
  void *symbol = nullptr;
  cudaDriverEntryPointQueryResult query;
  if (cudaGetDriverEntryPoint(name, &symbol, cudaEnableDefault, &query) != cudaSuccess || query != cudaDriverEntryPointSuccess)
    return nullptr;
  return reinterpret_cast<Function>(symbol);
}
}  // namespace

// The driver's call crashes on a thread without a current context.  The runtime binds one at a thread's first launch,
// but the maps are made before the launch, so a thread whose first GPU work this is has none yet: bind it here.
EncodeTiledFn encode_tiled() {
  static const auto encode = driver_function<EncodeTiledFn>("cuTensorMapEncodeTiled");
  static const auto current = driver_function<CUresult (*)(CUcontext *)>("cuCtxGetCurrent");
  if (!encode || !current) return nullptr;
  CUcontext context = nullptr;
  if (current(&context) == CUDA_SUCCESS && context) return encode;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return nullptr;
  return current(&context) == CUDA_SUCCESS && context ? encode : nullptr;
}

namespace {
template <typename T>
cudaError_t launch_gather_of(const T *x, const int32_t *perm, __half *xq, int rows, int k, cudaStream_t stream, int sm_count) {
  const size_t shared = static_cast<size_t>(k) * sizeof(__half);
  if (shared > 200 * 1024) return cudaErrorInvalidValue;  // (K beyond 102400 channels)
  static bool configured[64] = {};
  int device = 0;
  cudaError_t error = cudaGetDevice(&device);
  if (error != cudaSuccess) return error;
  if (device >= 64 || !configured[device]) {
    error = cudaFuncSetAttribute(sage_gather_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (error != cudaSuccess) return error;
    error = cudaFuncSetAttribute(sage_gather_four_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 kGatherFourChannels * sizeof(uint2));
    if (error != cudaSuccess) return error;
    if (device < 64) configured[device] = true;
  }
  if (rows >= kGatherFourRows && k <= kGatherFourChannels && perm != nullptr &&
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(perm)) & 15) == 0)
    return launch_dependent<1>(sage_gather_four_kernel<T>, dim3(static_cast<unsigned>((rows + kRowsAtOnce - 1) / kRowsAtOnce)),
                               dim3(kGatherFourThreads), static_cast<size_t>(k) * sizeof(uint2), stream, x, perm, xq, rows, k);
  int blocks = rows;
  const int cap = (sm_count > 0 ? sm_count : 148) * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return launch_dependent<1>(sage_gather_kernel<T>, dim3(static_cast<unsigned>(blocks)), dim3(kGatherThreads), shared,
                             stream, x, perm, xq, rows, k);
}
}  // namespace

cudaError_t launch_gather(const void *x, bool bf16, const int32_t *perm, __half *xq, int rows, int k, cudaStream_t stream,
                          int sm_count) {
  return bf16 ? launch_gather_of(static_cast<const __nv_bfloat16 *>(x), perm, xq, rows, k, stream, sm_count)
              : launch_gather_of(static_cast<const __half *>(x), perm, xq, rows, k, stream, sm_count);
}

int g_gemm_pairs = 1;  // debug switch (sageb200_debug_gemm_pairs): 0 = never pair CTAs

GemmPlan plan_gemm_tc(int rows, int n, int k, int sm_count, bool allow_split) {
  return plan_gemm_group(rows, &n, 1, k, sm_count, allow_split);
}

GemmPlan plan_gemm_group(int rows, const int *n, int count, int k, int sm_count, bool allow_split) {
  GemmPlan plan{};
  bool paired = g_gemm_pairs != 0;  // CTA pairs need an even number of row blocks in every problem
  for (int i = 0; i < count; ++i) {
    const int blocks = (n[i] + kTileRows - 1) / kTileRows;
    plan.row_blocks += blocks;
    paired = paired && blocks % 2 == 0;
  }
  if (sm_count <= 0) sm_count = 148;
  const int groups = k / 128;
  // Tokens per accumulator (the rows split evenly over some number of token tiles), accumulators per CTA
  // (two token blocks sharing every decoded weight stage) and CTAs per output tile along K.
  // Cost model per 64-channel stage of one CTA, in cycles - the kernel runs at the slowest of
  //   shared-memory traffic / 128 bytes per cycle: the decoded weights written and read again by the
  //     MMA for every accumulator, the codebook reads, the activations written by TMA and read by the
  //     MMA (a pair's CTA: half of them) - 793 measured at 208 tokens where this sum says 800;
  //   the tensor pipe: 135 cycles per 128 x 256 x 16 instruction (1103 measured against 1080);
  //   the decode warps: 630 (measured with the per-role clock sums of the profiling build)
  // times the stages per CTA, plus what every CTA spends before and after its stages (6000 cycles of
  // set-up and pipeline fill and 22 per token of epilogue, measured), times the waves the grid needs;
  // with a K split also the last CTA's pass over all splits' FP32 tiles.  Large grids end up with
  // 256 tokens x 2 (least decode work per output) unless another size fills its last wave better
  // (2560 -> 9728 at 2048 rows: five tiles of 2 x 224 tokens, 380 CTAs in 3 waves, where four of
  // 2 x 256 are 304 CTAs and also 3: 99 -> 93 us; 9728 -> 2560: seven of 2 x 160, 140 CTAs in one
  // wave, for 80: 106 -> 76 us); grids that would leave most SMs idle split K, so the decode work of
  // one weight tile is spread over several SMs.
  // A grid of one to four full waves and a rest leaves the SMs idle for most of the rest's wave: there the tiles
  // of the rest alone are split, so that they are one short wave of many CTAs (gate and up of 2560 -> 9728 at 32 rows,
  // 152 row blocks: 35.5 -> 30.2 us; 5120 -> 25600, 200 row blocks, at 64 rows 67.5 -> 59.8, at 512 rows 117 -> 108).
  // With more waves the rest weighs too little.
  int tn = 0, best_accumulators = 1, best_splits = 1;
  long long best_main = 0;
  double best_cost = 0.0;
  const int split_choices[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16};
  for (int accumulators = 2; accumulators >= 1; --accumulators) {
    const int least = (rows + 256 * accumulators - 1) / (256 * accumulators);
    int last_candidate = 0;
    for (int token_tiles = least; token_tiles < least + 8; ++token_tiles) {
      const int per_accumulator = (rows + token_tiles * accumulators - 1) / (token_tiles * accumulators);
      // (whole 32-token steps where the row blocks pair up: a pair's CTA loads half of a token block)
      const int unit = paired && per_accumulator > 128 ? 32 : 16;
      const int candidate = (per_accumulator + unit - 1) / unit * unit;
      if (candidate == last_candidate || candidate > 256) continue;
      if (accumulators == 2 && candidate < 128) continue;  // (small blocks gain nothing: decode-bound either way)
      last_candidate = candidate;
      const bool pair = paired && candidate % 32 == 0;
      const double b_bytes = accumulators * (pair ? candidate / 2 : candidate) * 128.0;
      double stage = (accumulators * 16384.0 + 32768.0 + 2.0 * b_bytes) / 128.0;
      const double tensor = accumulators * 4.0 * 135.0 * candidate / 256.0;
      if (stage < tensor) stage = tensor;
      if (stage < 630.0) stage = 630.0;
      const double around = 6000.0 + 22.0 * accumulators * candidate;
      const int blocks = (rows + accumulators * candidate - 1) / (accumulators * candidate);
      const long long tiles = static_cast<long long>(plan.row_blocks) * blocks;
      for (int wanted : split_choices) {
        // (a split only where the split grid still fits one wave: it exists to fill idle SMs, and
        //  its FP32 tiles would cost more HBM traffic than they save on a grid of several waves)
        // (... nor where the rest of a grid with a few full waves, split, fits one)
        const long long full_waves = tiles / sm_count;
        const long long whole = full_waves * (paired ? sm_count / 2 * 2 : sm_count);
        const bool rest_only = full_waves >= 1 && full_waves <= 4;
        const long long main = wanted == 1 ? tiles : rest_only ? whole : 0;
        if (wanted > 1 && (!allow_split || wanted * 2 > groups || (tiles - main) * wanted > sm_count || tiles == main)) continue;
        if (wanted > 8 && main == 0) continue;
        const int per_split = (groups + wanted - 1) / wanted;
        const int splits = (groups + per_split - 1) / per_split;  // (no empty split)
        if (splits != wanted) continue;
        const long long waves = wanted == 1 ? (tiles + sm_count - 1) / sm_count : full_waves;
        double cost = (2.0 * groups * stage + around) * static_cast<double>(waves);
        if (splits > 1) {
          const double tile_bytes = accumulators * candidate * 128.0 * 4.0;
          cost += 2.0 * per_split * stage + around + 2000.0;
          // (Two prices for one reduction code, each fitted to the grids that it prices; neither has been measured on the
          //  other's.  One for all would give 2560 -> 1024 at 77 to 512 rows, 9728 -> 2560 at 300 and others another plan.)
          if (rest_only)  // as below, but by the last CTAs of its three parts; and all of it through L2 (~28 bytes per cycle and SM)
            cost += (1.0 + splits / (splits < 3 ? splits : 3.0)) * tile_bytes / 64.0 +
                    2.0 * (tiles - main) * splits * tile_bytes / (28.0 * sm_count);
          else  // tile written once per split, then read back by the last CTA (~64 bytes per cycle)
            cost += (splits + 1.0) * tile_bytes / 64.0;
        }
        if (tn == 0 || cost < best_cost * 0.95) {  // (prefer the earlier, simpler choice on near ties)
          tn = candidate;
          best_accumulators = accumulators;
          best_splits = splits;
          best_main = main;
          best_cost = cost;
        }
      }
    }
  }
  plan.tokens_per_cta = tn;
  plan.token_blocks = (rows + tn - 1) / tn;
  plan.accumulators = best_accumulators;
  // Pairs of CTAs (cta_group::2) whenever the row blocks pair up and each CTA's half of a token
  // block is a whole number of 16-token MMA columns: half the B operand per SM.
  plan.pair = paired && (tn % 32 == 0) ? 1 : 0;
  plan.k_splits = best_splits;
  plan.groups_per_split = (groups + best_splits - 1) / best_splits;
  {
    plan.tiles = plan.row_blocks * ((plan.token_blocks + plan.accumulators - 1) / plan.accumulators);
    plan.main_tiles = static_cast<int>(best_main);
    plan.partial_bytes = static_cast<size_t>(plan.tiles - plan.main_tiles) * best_splits * plan.accumulators * tn * kTileRows * sizeof(float);
  }
  const int stage_bytes = kAStageBytes + plan.accumulators * (plan.pair ? tn / 2 : tn) * kStageK * 2;
  int stages = (kGemmSharedLimit - kBookBytes - 2 * 1024) / stage_bytes;
  if (stages > kMaxStages) stages = kMaxStages;
  if (stages < 2) stages = 2;
  plan.stages = stages;
  int columns = 32;
  while (columns < tn) columns *= 2;
  plan.tmem_columns = plan.accumulators == 2 ? 512 : columns;
  plan.shared_bytes = static_cast<size_t>(stages) * stage_bytes + kBookBytes + (2 * kMaxStages + 1) * 8 + 1024;
  return plan;
}

cudaError_t configure_gemm_tc() {
  cudaError_t error = cudaFuncSetAttribute(sage_gemm_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kGemmSharedLimit);
  if (error != cudaSuccess) return error;
  return cudaFuncSetAttribute(sage_gemm_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              kGemmSharedLimit);
}

cudaError_t launch_gemm_tc(const GemmInput *inputs, int count, int *status, int rows, int k, bool out_bf16,
                           const GemmPlan &plan, cudaStream_t stream, float *partial, unsigned *counters) {
  if (count < 1 || count > kMaxGemmProblems) return cudaErrorInvalidValue;
  if (plan.k_splits > 1 && (!partial || !counters)) return cudaErrorInvalidValue;
  EncodeTiledFn encode = encode_tiled();
  if (!encode) return cudaErrorNotSupported;
  GemmParams p;
  memset(&p, 0, sizeof(p));
  int row_block = 0;
  for (int i = 0; i < count; ++i) {
    const GemmInput &in = inputs[i];
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(k) * 2};
    const cuuint32_t box[2] = {kStageK, static_cast<cuuint32_t>(plan.pair ? plan.tokens_per_cta / 2 : plan.tokens_per_cta)};
    const cuuint32_t element_strides[2] = {1, 1};
    const CUresult encoded = encode(
        &p.x_map[i], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half *>(in.xq), dims, strides, box,
        element_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (encoded != CUDA_SUCCESS) return cudaErrorInvalidValue;
    GemmProblem &q = p.problem[i];
    q.codes = in.codes;
    q.radii = in.radii;
    q.grid = in.grid;
    q.book = in.book;
    q.mins = in.sph_mins;
    q.bias = in.bias;
    q.y = in.y;
    q.n = in.n;
    q.tiles = (in.n + 15) / 16;
    q.entries = in.entries;
    q.dbits = direction_bits_of(in.entries);
    q.row_block_begin = row_block;
    row_block += (in.n + kTileRows - 1) / kTileRows;
  }
  if (row_block != plan.row_blocks) return cudaErrorInvalidValue;  // (a plan for other problems)
  p.count = count;
  p.status = status;
  p.rows = rows;
  p.groups = k / 128;
  p.out_bf16 = out_bf16 ? 1 : 0;
  p.tokens_per_cta = plan.tokens_per_cta;
  p.stages = plan.stages;
  p.tmem_columns = plan.tmem_columns;
  p.accumulators = plan.accumulators;
  p.trace = trace_buffer();
  p.k_splits = plan.k_splits;
  p.groups_per_split = plan.groups_per_split;
  p.partial = partial;
  p.counters = counters;
  p.format = inputs[0].sph_mins ? 1 : 0;
  p.row_blocks = plan.row_blocks;
  p.tiles = plan.tiles;
  p.main_tiles = plan.main_tiles;
  const dim3 blocks(static_cast<unsigned>(plan.main_tiles + (plan.tiles - plan.main_tiles) * plan.k_splits));
  cudaLaunchConfig_t config = {};
  config.gridDim = blocks;
  config.blockDim = dim3(kGemmThreads);
  config.dynamicSmemBytes = plan.shared_bytes;
  config.stream = stream;
  cudaLaunchAttribute attribute[2];
  unsigned attributes = 0;
  if (g_sageb200_pdl & 1) {  // (the same switch as the decode kernels: sageb200_set_pdl)
    attribute[attributes].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[attributes].val.programmaticStreamSerializationAllowed = 1;
    ++attributes;
  }
  if (plan.pair) {
    attribute[attributes].id = cudaLaunchAttributeClusterDimension;
    attribute[attributes].val.clusterDim.x = 2;
    attribute[attributes].val.clusterDim.y = 1;
    attribute[attributes].val.clusterDim.z = 1;
    ++attributes;
  }
  config.attrs = attribute;
  config.numAttrs = attributes;
  return plan.pair ? cudaLaunchKernelEx(&config, sage_gemm_tc_kernel<true>, p)
                   : cudaLaunchKernelEx(&config, sage_gemm_tc_kernel<false>, p);
}

}  // namespace sageb200
