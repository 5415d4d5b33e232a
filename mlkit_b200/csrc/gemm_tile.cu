// Packed matrix product on the 5th-generation tensor cores: y[M, N] = x[M, K] . W^T for more rows than the matvec
// takes, any codec of 2 to 8 bits, fp16 or bf16 activations (sm_100a).
//
// The weight is read as codes; reconstructed 16-bit weights exist in shared memory only.  A tile of the result is 128
// weight rows (the M of tcgen05.mma) x up to 256 activation rows (its N; what shared memory leaves: 256 at 2 bits, 224 for
// 4-bit integer grids, 208 with offsets, 160 at 8 bits, 144 with offsets), fp32 in tensor memory.  A stage of the pipeline
// is a block of 128 K: 32 KB of weights and 256 B per activation row, as two K-major halves in the 128-byte swizzle.
// Roles (23 warps):
//   * warps 0-15 decode, two groups of eight, a block each in turn: a block is a chain of waits, loads and stores, and
//     two of them side by side keep the SM's issue slots busy.  Thread (r, h) of a group owns row r and K half h: 64
//     codes, decoded to one 128-byte row of the stage; their scales it copies ahead itself (cp.async).  Four-bit integer
//     grids: a byte becomes the pair (c0 + min, c1 + min) by PRMT, LOP3 and an exact HFMA2, and one HMUL2 (fp16) or two
//     FMUL and a conversion round it to the weight the reference reconstructs.  Other codecs and offsets: fp32 levels
//     from shared memory;
//   * warps 16-19 are the epilogue: tensor memory to y, or to a partial, while the next tile is multiplied (the
//     accumulators are doubled);
//   * warp 20 feeds the activations (TMA, rows past M read as zero), warp 21 issues the products, warp 22 feeds the
//     codes (TMA into a ring of their own: copied by the decoders, a row of 64 bytes per lane, they took more cycles of
//     the load pipe than the decode takes altogether).
// The work, tiles x blocks of 128 K with a tile's blocks in a row, is one line cut into equal pieces, one per SM: no
// last wave, and a layer of few tiles still fills the GPU.  A piece that ends or begins inside a tile leaves an fp32
// partial, and a second, dependent launch adds the partials of every cut tile in K order on all SMs.
// All hand-offs inside the CTA are mbarriers with bounded waits: on expiry the CTA records a status word and drains.
//
// 4096 -> 14336 in 4 bits, fp16 rows, us (against reconstruct + library GEMM): 17 rows 19.5 (81), 64 rows 23.3 (84), 128
// rows 26.8 (84), 512 rows 67 (109), 1024 rows 120 (146).  Above 200 rows the activations' traffic from L2 and the tensor
// core bound it.  Up to 64 rows neither does, nor the codes' 4.6 us from HBM: an SM has 25 blocks, whose decode takes about
// 450 cycles each (5.7 us in all), so most of the launch pair's time there is its start, its pipeline's and its sums'.
#include <cuda.h>

#include <algorithm>

#include "mkb_common.cuh"

namespace mkb {
namespace {

constexpr int kGroupThreads = 256, kDecodeGroups = 2, kDecodeThreads = kGroupThreads * kDecodeGroups;
constexpr int kTileThreads = kDecodeThreads + 128 + 96;
constexpr int kTileRows = 128;
constexpr int kWeightHalf = kTileRows * 128;       // bytes of weights in half a stage: 128 rows x 64 K
constexpr int kMostStages = 4;
constexpr int kMostCodeSlots = 6, kLeastCodeSlots = 4;
constexpr int kScaleSlots = 3;                     // a decoder's own ring of scales
constexpr int64_t kTileHead = 65536;               // of mkb_gemm's workspace; its last word is the status
constexpr uint32_t kTileSpins = 200000;            // tries of up to 20 us each: a few seconds

enum { DECODE_INT4 = 0, DECODE_TABLE = 1 };

struct TileArgs {
  const __half* scales;
  const __half* zeros;
  const float* lut;
  const uint16_t* bias;
  uint16_t* y;
  float* partials;   // [2 per CTA][columns][128 rows]
  int* status;
  int64_t scale_row_stride;
  int M, N, lut_len, group_shift;
  int word_scales;   // scales and offsets are whole aligned words: they can be copied as such
  int columns, column_tiles, k_blocks, units, per_cta;
  int stages, code_slots, tmem_columns;
  float grid_min;
};

struct TileBarriers {
  uint64_t codes_full[kMostCodeSlots];  // TMA
  uint64_t codes_empty[kMostCodeSlots]; // the eight warps of a group
  uint64_t stage_full[kMostStages];     // the eight warps of the group that decoded the block, and TMA
  uint64_t stage_empty[kMostStages];    // tcgen05.commit
  uint64_t sums_full[2];                // tcgen05.commit
  uint64_t sums_empty[2];               // four epilogue warps
};

__device__ __forceinline__ uint32_t tile_shared(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void tile_barrier(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tile_shared(bar)), "r"(count));
}
__device__ __forceinline__ void tile_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tile_shared(bar)) : "memory");
}
// Bounded wait for the phase of the given parity; false when it gave up (or another role did).
__device__ __forceinline__ bool tile_wait(uint64_t* bar, uint32_t parity, volatile int* failed) {
  uint32_t done = 0;
  for (uint32_t spins = 0; spins < kTileSpins; ++spins) {
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(tile_shared(bar)), "r"(parity), "r"(20000u) : "memory");
    if (done) return true;
    if ((spins & 63) == 63 && *failed) return false;
  }
  *failed = 1;
  return false;
}
// The same for copies in flight after a failure: their stage may also miss decoders, so this one only gives them time.
__device__ __forceinline__ void tile_drain(uint64_t* bar, uint32_t parity) {
  uint32_t done = 0;
  for (int spins = 0; spins < 64 && !done; ++spins)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(done) : "r"(tile_shared(bar)), "r"(parity), "r"(20000u) : "memory");
}
// The warps that issue products and copies run whole: every lane holds the same values, which the compiler keeps in
// uniform registers, where these instructions take their operands from, and one elected lane issues.  (With one lane
// alone in the loop each operand is moved and checked for every instruction: about a hundred cycles a product.)
__device__ __forceinline__ void tile_commit(uint64_t* bar) {
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
               "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(tile_shared(bar)) : "memory");
}
__device__ __forceinline__ void tile_copy4(uint32_t to, const void* from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to), "l"(from) : "memory");
}
// a K-major tile in the 128-byte swizzle: groups of eight rows 1024 bytes apart, descriptor version 1
__device__ __forceinline__ uint64_t tile_descriptor(uint32_t address) {
  return uint64_t((address & 0x3ffffu) >> 4) | (uint64_t(1) << 16) | (uint64_t(1024 >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(2) << 61);
}

template <bool BF16>
__device__ __forceinline__ uint32_t round_pair(float low, float high) {
  if constexpr (BF16) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
    return *reinterpret_cast<const uint32_t*>(&pair);
  } else {
    const __half2 pair = __floats2half2_rn(low, high);
    return *reinterpret_cast<const uint32_t*>(&pair);
  }
}

// codes 2 BYTE and 2 BYTE + 1 of a word as the exact fp16 pair (c0 + min, c1 + min): the byte in both halves under the
// exponent of 1024 is (1024 + c0, 1024 + 16 c1), and `offset` is (min - 1024, min - 64)
template <int BYTE>
__device__ __forceinline__ __half2 centred_pair(uint32_t word, __half2 offset) {
  constexpr uint32_t selector = BYTE == 0 ? 0x1010u : BYTE == 1 ? 0x2121u : BYTE == 2 ? 0x3232u : 0x0303u;
  uint32_t biased;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(biased) : "r"(__byte_perm(word, word, selector)), "r"(0x00f0000fu), "r"(0x64006400u));
  const __half2 one_sixteenth = __halves2half2(__ushort_as_half(0x3c00), __ushort_as_half(0x2c00));   // (1, 1/16)
  return __hfma2(*reinterpret_cast<const __half2*>(&biased), one_sixteenth, offset);
}

template <bool BF16, int DECODE, int BITS>
__global__ void __launch_bounds__(kTileThreads, 1) gemm_tile_kernel(const __grid_constant__ CUtensorMap rows_map,
                                                                    const __grid_constant__ CUtensorMap codes_map, const TileArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (tile_shared(smem_raw) & 1023u)) & 1023u);
  constexpr int WORDS = 2 * BITS;                               // 32-bit words of a thread's 64 codes
  constexpr int PIECE = BITS % 2 == 0 ? 16 : 8, PIECES = 8 * BITS / PIECE;
  constexpr int CODE_SLOT = kTileRows * 16 * BITS;              // a block's codes, rows of 16 BITS bytes, swizzled by TMA
  const int scale_slot = kDecodeThreads * (a.zeros != nullptr ? 16 : 8);   // [2][thread] words with scales, as many with offsets
  const int rows_half = a.columns * 128;
  uint8_t* weight_s = smem;                                     // [stages][2][128 rows][128 B]
  uint8_t* rows_s = weight_s + a.stages * 2 * kWeightHalf;      // [stages][2][columns][128 B]
  uint8_t* code_s = rows_s + a.stages * 2 * rows_half;          // [code slots]
  uint8_t* scale_s = code_s + a.code_slots * CODE_SLOT;         // [kScaleSlots]
  float* level_s = reinterpret_cast<float*>(scale_s + kScaleSlots * scale_slot);
  __shared__ __align__(8) TileBarriers bars;
  __shared__ uint32_t tmem_s;
  __shared__ int failed_s;
  volatile int* failed = &failed_s;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first = int(blockIdx.x) * a.per_cta, end = min(first + a.per_cta, a.units), count = end - first;

  if (warp == 21) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tile_shared(&tmem_s)), "r"(a.tmem_columns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  if (tid == 0) failed_s = 0;
  if (warp == 20) {                // a barrier a lane
    if (lane < kMostCodeSlots) {
      tile_barrier(&bars.codes_full[lane], 1);
      tile_barrier(&bars.codes_empty[lane], kGroupThreads / 32);
    }
    if (lane < kMostStages) {
      tile_barrier(&bars.stage_full[lane], kGroupThreads / 32 + 1);
      tile_barrier(&bars.stage_empty[lane], 1);
    }
    if (lane < 2) {
      tile_barrier(&bars.sums_full[lane], 1);
      tile_barrier(&bars.sums_empty[lane], 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if constexpr (DECODE == DECODE_TABLE) {
    // up to four bits every lane has a copy of the levels of its own (no bank conflicts), above one copy serves all
    constexpr int COPIES = BITS <= 4 ? 32 : 1;
    for (int i = tid; i < (COPIES << BITS); i += kTileThreads) level_s[i] = i / COPIES < a.lut_len ? a.lut[i / COPIES] : 0.f;
  }

  // ---- decoders: a warp owns 16 rows, lane l row l % 16 and K half l / 16 (eight lanes store one chunk of eight rows:
  // no bank conflicts), of the blocks group, group + 2, ... ----
  const int r = ((warp & 7) << 4) + (lane & 15), h = lane >> 4, group = tid / kGroupThreads;
  // The scales are copied two blocks of the group ahead.  Inside a tile their place moves by a constant; a step of two
  // blocks moves the index by an even number, so which half of its word a scale sits in changes with the tile only.
  const uint8_t* scale_from = nullptr;
  const int64_t zero_from = reinterpret_cast<const uint8_t*>(a.zeros) - reinterpret_cast<const uint8_t*>(a.scales);
  const int scale_step = (kDecodeGroups * 256) >> a.group_shift;
  const bool two_scales = a.group_shift == 5;
  int copy_left = 0, copy_block = 0, copy_m0 = 0, copy_rows = 0;
  int copies = tid < kDecodeThreads ? (count - group + kDecodeGroups - 1) / kDecodeGroups : 0;
  const uint32_t scale_base = tile_shared(scale_s) + tid * 4;
  uint32_t copy_slot = 0, odd_scales = 0, odd = 0;   // odd_scales: a bit per slot
  auto enter_tile = [&]() {
    const int64_t n = min(copy_rows + r, a.N - 1);
    const int64_t scale = n * a.scale_row_stride + ((copy_block * 128 + h * 64) >> a.group_shift);
    odd = a.word_scales ? uint32_t(scale & 1) : 0u;
    scale_from = reinterpret_cast<const uint8_t*>(a.scales) + (scale - odd) * 2;
    copy_left = (a.k_blocks - copy_block + kDecodeGroups - 1) / kDecodeGroups;     // blocks of this group left in the tile
  };
  auto copy_scales = [&]() {
    if (copies > 0) {
      --copies;
      const uint32_t to = scale_base + copy_slot * scale_slot;
      if (a.word_scales) {             // the aligned word (or two) around the one or two scales
        tile_copy4(to, scale_from);
        if (two_scales && odd) tile_copy4(to + kDecodeThreads * 4, scale_from + 4);
        if (a.zeros != nullptr) {
          tile_copy4(to + kDecodeThreads * 8, scale_from + zero_from);
          if (two_scales && odd) tile_copy4(to + kDecodeThreads * 12, scale_from + zero_from + 4);
        }
      } else {                         // an odd number of them, or off a word's boundary: one by one, into the word's halves
        auto single = [&](uint32_t into, const uint8_t* from) {
          const uint16_t value = __ldg(reinterpret_cast<const uint16_t*>(from));
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(into), "h"(value) : "memory");
        };
        for (int i = 0; i < (two_scales ? 2 : 1); ++i) {
          single(to + 2 * i, scale_from + 2 * i);
          if (a.zeros != nullptr) single(to + kDecodeThreads * 8 + 2 * i, scale_from + zero_from + 2 * i);
        }
      }
      odd_scales = (odd_scales & ~(1u << copy_slot)) | (odd << copy_slot);
      scale_from += scale_step;
      if (--copy_left == 0) {
        copy_block += (a.k_blocks - copy_block + kDecodeGroups - 1) / kDecodeGroups * kDecodeGroups;
        while (copy_block >= a.k_blocks) {      // a tile of one block leaves the other group's tile out
          copy_block -= a.k_blocks;
          copy_m0 += a.columns;
          if (copy_m0 >= a.M) { copy_m0 = 0; copy_rows += kTileRows; }
        }
        enter_tile();
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    copy_slot = copy_slot + 1 == kScaleSlots ? 0 : copy_slot + 1;
  };
  if (tid < kDecodeThreads) {
    const int tile = (first + group) / a.k_blocks, row_block = tile / a.column_tiles;
    copy_block = first + group - tile * a.k_blocks;
    copy_rows = row_block * kTileRows;
    copy_m0 = (tile - row_block * a.column_tiles) * a.columns;
    enter_tile();
#pragma unroll
    for (int d = 0; d < kScaleSlots - 1; ++d) copy_scales();
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_s;

  if (tid < kDecodeThreads) {
    // ================================ decoders ================================
    const __half2 offset = __floats2half2_rn(a.grid_min - 1024.f, a.grid_min - 64.f);
    // chunk c of the row goes to chunk c ^ (r & 7): an exclusive-or on the address of chunk 0
    const uint32_t row_at = tile_shared(weight_s) + h * kWeightHalf + r * 128 + ((r & 7) << 4);
    int stage = group % a.stages, round = group / a.stages;
    uint32_t code_slot = group, code_round = 0, slot = 0;      // (at least four code slots)
    int i = group;
    for (; i < count; i += kDecodeGroups) {
      if (!tile_wait(&bars.codes_full[code_slot], code_round & 1u, failed)) break;
      uint32_t words[WORDS];
      const uint32_t row_from = tile_shared(code_s) + code_slot * CODE_SLOT + r * (16 * BITS);
#pragma unroll
      for (int p = 0; p < PIECES; ++p) {
        if constexpr (PIECE == 16) {
          // chunk h * PIECES + p of the row, where TMA's swizzle put it
          uint32_t chunk = uint32_t(h * PIECES + p);
          if constexpr (BITS == 2) chunk ^= uint32_t(r >> 2) & 1u;
          if constexpr (BITS == 4) chunk ^= uint32_t(r >> 1) & 3u;
          if constexpr (BITS == 8) chunk ^= uint32_t(r) & 7u;
          asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(words[4 * p]), "=r"(words[4 * p + 1]), "=r"(words[4 * p + 2]), "=r"(words[4 * p + 3])
                       : "r"(row_from + chunk * 16));
        } else {
          asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(words[2 * p]), "=r"(words[2 * p + 1]) : "r"(row_from + h * (8 * BITS) + p * 8));
        }
      }
      asm volatile("cp.async.wait_group %0;" ::"n"(kScaleSlots - 2) : "memory");    // this thread's scales of block i
      // the halves of the copied words that the index's parity names
      auto side = [&](uint32_t at, __half (&out)[2]) {
        const uint32_t from = scale_base + slot * scale_slot + at, first_half = ((odd_scales >> slot) & 1u) * 16u;
        uint32_t low, high;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(low) : "r"(from));
        if (two_scales) {
          asm volatile("ld.shared.u32 %0, [%1];" : "=r"(high) : "r"(from + kDecodeThreads * 4));
          low = __funnelshift_r(low, high, first_half);
          out[0] = __ushort_as_half((unsigned short)(low & 0xffffu));
          out[1] = __ushort_as_half((unsigned short)(low >> 16));
        } else {
          out[0] = out[1] = __ushort_as_half((unsigned short)(low >> first_half));
        }
      };
      __half scales[2], zeros[2] = {__half(), __half()};
      side(0, scales);
      if (a.zeros != nullptr) side(kDecodeThreads * 8, zeros);
      slot = slot + 1 == kScaleSlots ? 0 : slot + 1;
      copy_scales();                   // into the slot read one block ago
      if (round > 0 && !tile_wait(&bars.stage_empty[stage], uint32_t(round - 1) & 1u, failed)) break;
      const uint32_t to = row_at + 2 * stage * kWeightHalf;
#pragma unroll
      for (int c = 0; c < 8; ++c) {    // chunks of eight codes
        uint4 out;
        uint32_t* pairs = &out.x;
        const int which = c >> 2;
        const __half scale = scales[which];
        if constexpr (DECODE == DECODE_INT4) {
          const __half2 p0 = centred_pair<0>(words[c], offset), p1 = centred_pair<1>(words[c], offset);
          const __half2 p2 = centred_pair<2>(words[c], offset), p3 = centred_pair<3>(words[c], offset);
          const __half2 centred[4] = {p0, p1, p2, p3};
          if (!BF16 && a.zeros == nullptr) {
            const __half2 both = __half2half2(scale);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const __half2 w = __hmul2(centred[j], both);
              pairs[j] = *reinterpret_cast<const uint32_t*>(&w);
            }
          } else {                     // a whole number times eleven bits is exact: one rounding by the offset's add, one to 16 bits
            const float s = __half2float(scale), z = __half2float(zeros[which]);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const float2 two = __half22float2(centred[j]);
              pairs[j] = a.zeros == nullptr ? round_pair<BF16>(two.x * s, two.y * s) : round_pair<BF16>(fmaf(two.x, s, z), fmaf(two.y, s, z));
            }
          }
        } else {
          const float s = __half2float(scale), z = __half2float(zeros[which]);
          float w[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int bit = (8 * c + e) * BITS, word = bit >> 5, shift = bit & 31;
            const uint32_t field = shift + BITS <= 32 ? words[word] >> shift : __funnelshift_r(words[word], words[(word + 1) % WORDS], shift);
            const uint32_t code = field & ((1u << BITS) - 1u);
            const float value = BITS <= 4 ? level_s[code * 32 + lane] : level_s[code];
            w[e] = __fmul_rn(value, s);
          }
          if (a.zeros != nullptr) {
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = __fadd_rn(w[e], z);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) pairs[j] = round_pair<BF16>(w[2 * j], w[2 * j + 1]);
        }
        asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(to ^ (uint32_t(c) << 4)), "r"(out.x), "r"(out.y), "r"(out.z), "r"(out.w) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        tile_arrive(&bars.codes_empty[code_slot]);
        tile_arrive(&bars.stage_full[stage]);
      }
      code_slot += kDecodeGroups;
      if (code_slot >= uint32_t(a.code_slots)) { code_slot -= a.code_slots; ++code_round; }
      stage += kDecodeGroups;
      if (stage >= a.stages) { stage -= a.stages; ++round; }
    }
    // A lane whose wait gave up has left the loop alone: it meets the others at the warp barriers of the blocks that it
    // leaves out, or they would stand there while it stands at the CTA's closing barrier.  (Leaving by a vote per block, or
    // staying in the loop without waiting, made 64 rows 1 % slower.)
    for (; i < count; i += kDecodeGroups) __syncwarp();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else if (warp < 20) {
    // ================================ epilogue ================================
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int sub = warp - 16, row = sub * 32 + lane;   // warp 16 + s reads lanes 32 s .. of tensor memory
    int unit = first, buffer = 0, uses = 0;
    while (unit < end) {
      const int tile = unit / a.k_blocks, tile_begin = tile * a.k_blocks, tile_end = tile_begin + a.k_blocks;
      const int stop = min(tile_end, end);
      const bool whole = unit == tile_begin && stop == tile_end;
      const int row_block = tile / a.column_tiles, m0 = (tile - row_block * a.column_tiles) * a.columns;
      const int live = min(a.columns, a.M - m0), n = row_block * kTileRows + row;
      const bool good = tile_wait(&bars.sums_full[buffer], uint32_t(uses) & 1u, failed);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float bias = a.bias == nullptr || n >= a.N ? 0.f
                         : BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.bias)[n])
                                : __half2float(reinterpret_cast<const __half*>(a.bias)[n]);
      // one warp per scheduler does this: no test stands between the stores of sixteen columns, their addresses are
      // immediates (a partial, whose columns past `live` nobody reads) or one addition apart
      float* part = a.partials + ((int64_t(blockIdx.x) * 2 + (unit == tile_begin ? 1 : 0)) * a.columns) * kTileRows + row;
      uint16_t* out = a.y + int64_t(m0) * a.N + n;
      const bool stores = good && n < a.N;
      auto narrow = [&](uint32_t bits) -> uint16_t {
        const float value = __uint_as_float(bits) + bias;
        if constexpr (BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(value));
        else return __half_as_ushort(__float2half_rn(value));
      };
      const uint32_t from = tmem + (uint32_t(sub * 32) << 16) + buffer * (a.tmem_columns >> 1);
      for (int c = 0; c < live; c += 16) {
        uint32_t d[16];
        __syncwarp();
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]),
                       "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
                     : "r"(from + c) : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (!whole) {
#pragma unroll
          for (int j = 0; j < 16; ++j) __stcg(part + j * kTileRows, __uint_as_float(d[j]));
          part += 16 * kTileRows;
        } else if (stores) {
          if (c + 16 <= live) {
#pragma unroll
            for (int j = 0; j < 16; ++j) out[int64_t(j) * a.N] = narrow(d[j]);
          } else {
#pragma unroll
            for (int j = 0; j < 15; ++j)
              if (c + j < live) out[int64_t(j) * a.N] = narrow(d[j]);
          }
          out += int64_t(16) * a.N;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tile_arrive(&bars.sums_empty[buffer]);
      unit = stop;
      buffer ^= 1;
      uses += buffer == 0;
    }
  } else if (warp == 20) {
    // ================================ activations ================================
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint64_t map = reinterpret_cast<uint64_t>(&rows_map);
    const int tile = first / a.k_blocks;
    int m0 = (tile % a.column_tiles) * a.columns, block = first - tile * a.k_blocks, stage = 0, round = 0, sent = 0;
    for (int i = 0; i < count; ++i) {
      if (round > 0 && !__all_sync(0xffffffffu, tile_wait(&bars.stage_empty[stage], uint32_t(round - 1) & 1u, failed))) break;
      const uint32_t bar = tile_shared(&bars.stage_full[stage]), to = tile_shared(rows_s) + 2 * stage * rows_half;
      asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                   "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%4], %5;\n\t"
                   "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t"
                   "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%6], [%1, {%7, %3}], [%4];\n\t}\n"
                   ::"r"(to), "l"(map), "r"(block * 128), "r"(m0), "r"(bar), "r"(2 * rows_half), "r"(to + rows_half), "r"(block * 128 + 64)
                   : "memory");
      __syncwarp();
      ++sent;
      if (++block == a.k_blocks) {
        block = 0;
        m0 += a.columns;
        if (m0 >= a.M) m0 = 0;
      }
      if (++stage == a.stages) { stage = 0; ++round; }
    }
    // no copy is left in flight when the CTA ends, whatever happened to its consumers
    for (int i = max(0, sent - a.stages); *failed && i < sent; ++i)
      tile_drain(&bars.stage_full[i % a.stages], uint32_t(i / a.stages) & 1u);
  } else if (warp == 22) {
    // ================================ codes ================================
    const uint64_t map = reinterpret_cast<uint64_t>(&codes_map);
    const int tile = first / a.k_blocks, row_block = tile / a.column_tiles;
    int block = first - tile * a.k_blocks, m0 = (tile - row_block * a.column_tiles) * a.columns, rows = row_block * kTileRows;
    int slot = 0, round = 0, sent = 0;
    for (int i = 0; i < count; ++i) {
      if (round > 0 && !__all_sync(0xffffffffu, tile_wait(&bars.codes_empty[slot], uint32_t(round - 1) & 1u, failed))) break;
      asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                   "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%4], %5;\n\t"
                   "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}\n"
                   ::"r"(tile_shared(code_s) + slot * CODE_SLOT), "l"(map), "r"(block * (16 * BITS)), "r"(rows),
                     "r"(tile_shared(&bars.codes_full[slot])), "r"(CODE_SLOT) : "memory");
      __syncwarp();
      ++sent;
      if (++block == a.k_blocks) {
        block = 0;
        m0 += a.columns;
        if (m0 >= a.M) { m0 = 0; rows += kTileRows; }
      }
      if (++slot == a.code_slots) { slot = 0; ++round; }
    }
    // no copy is left in flight when the CTA ends
    for (int i = max(0, sent - a.code_slots); i < sent; ++i)
      tile_wait(&bars.codes_full[i % a.code_slots], uint32_t(i / a.code_slots) & 1u, failed);
  } else {
    // ================================ products ================================
    const uint32_t form = (1u << 4) | (BF16 ? (1u << 7) | (1u << 10) : 0u) | (uint32_t(a.columns >> 3) << 17) | (8u << 24);
    int stage = 0, round = 0, buffer = 0, uses = 0, unit = first;
    bool alive = true;
    while (unit < end && alive) {
      const int stop = min((unit / a.k_blocks + 1) * a.k_blocks, end);
      if (uses > 0 && !__all_sync(0xffffffffu, tile_wait(&bars.sums_empty[buffer], uint32_t(uses - 1) & 1u, failed))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sums = tmem + buffer * (a.tmem_columns >> 1);
      for (int i = 0; i < stop - unit; ++i) {
        if (!__all_sync(0xffffffffu, tile_wait(&bars.stage_full[stage], uint32_t(round) & 1u, failed))) { alive = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t weights = tile_descriptor(tile_shared(weight_s) + 2 * stage * kWeightHalf);
        const uint64_t rows = tile_descriptor(tile_shared(rows_s) + 2 * stage * rows_half);
#pragma unroll
        for (int k = 0; k < 8; ++k) {     // 16 K are 32 bytes inside the swizzled row
          asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\telect.sync _|q, 0xffffffff;\n\t"
                       "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                       ::"r"(sums), "l"(weights + (k >> 2) * (kWeightHalf >> 4) + 2 * (k & 3)),
                         "l"(rows + (k >> 2) * (rows_half >> 4) + 2 * (k & 3)), "r"(form), "r"((i | k) ? 1u : 0u) : "memory");
        }
        tile_commit(&bars.stage_empty[stage]);
        if (++stage == a.stages) { stage = 0; ++round; }
      }
      if (!alive) break;
      tile_commit(&bars.sums_full[buffer]);
      unit = stop;
      buffer ^= 1;
      uses += buffer == 0;
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && failed_s) atomicExch(a.status, 1);
  if (warp == 21) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_columns));
}

// Adds the partials of the tiles that are cut.  Block (b, c): the tile with the cut between pieces b and b + 1 (its first
// cut, if it has several), columns 8 c .. 8 c + 7; a thread owns a weight row.
template <bool BF16>
__global__ void __launch_bounds__(kTileRows) gemm_tile_sum_kernel(const TileArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int cut = (int(blockIdx.x) + 1) * a.per_cta, tile = cut / a.k_blocks, tile_begin = tile * a.k_blocks;
  const bool first_cut = cut - a.per_cta <= tile_begin;
  if (cut == tile_begin || !first_cut) return;
  const int row_block = tile / a.column_tiles, m0 = (tile - row_block * a.column_tiles) * a.columns, c0 = int(blockIdx.y) * 8;
  const int live = min(a.columns, a.M - m0), n = row_block * kTileRows + int(threadIdx.x);
  if (c0 >= live) return;
  const int first_cta = tile_begin / a.per_cta, last_cta = (tile_begin + a.k_blocks - 1) / a.per_cta;
  const float bias = a.bias == nullptr || n >= a.N ? 0.f
                     : BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.bias)[n])
                            : __half2float(reinterpret_cast<const __half*>(a.bias)[n]);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  float sum[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sum[j] = 0.f;
#pragma unroll 4
  for (int cta = first_cta; cta <= last_cta; ++cta) {
    const float* part = a.partials + (int64_t(cta) * 2 + (cta * a.per_cta > tile_begin ? 0 : 1)) * a.columns * kTileRows + c0 * kTileRows + threadIdx.x;
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[j] += __ldcg(part + j * kTileRows);   // columns past `live` stay inside the partial
  }
  if (n >= a.N) return;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (c0 + j >= live) break;
    uint16_t* out = a.y + int64_t(m0 + c0 + j) * a.N + n;
    if constexpr (BF16) *reinterpret_cast<__nv_bfloat16*>(out) = __float2bfloat16_rn(sum[j] + bias);
    else *reinterpret_cast<__half*>(out) = __float2half_rn(sum[j] + bias);
  }
}

// ---- host side -----------------------------------------------------------------------------------
struct TilePlan {
  int columns, column_tiles, row_blocks, k_blocks, stages, code_slots, tmem_columns;
  int64_t units;
  int per_cta, ctas;
  size_t smem;
};

// Column tiles of equal width, a multiple of 16 that leaves room for two stages and four slots of codes: 1537 rows are
// seven tiles of 224, not six of 240 and a rest of 97.
TilePlan plan_tiles(int M, int N, int K, int bits, bool table, bool zeros, int sm_count, int max_smem) {
  TilePlan p{};
  const size_t levels = table ? (bits <= 4 ? size_t(128) << bits : size_t(4) << bits) : 0;
  const size_t codes = size_t(kTileRows) * 16 * bits, scales = size_t(kScaleSlots) * kDecodeThreads * (zeros ? 16 : 8);
  const size_t room = size_t(max_smem) - 1024 - 512 - levels - scales;      // alignment, static shared memory
  const int widest = std::min(256, int((room - kLeastCodeSlots * codes) / 2 - 2 * kWeightHalf) / 256 & ~15);
  if (widest < 16) return p;
  p.column_tiles = (M + widest - 1) / widest;
  p.columns = ((M + p.column_tiles - 1) / p.column_tiles + 15) & ~15;
  p.column_tiles = (M + p.columns - 1) / p.columns;
  p.row_blocks = (N + kTileRows - 1) / kTileRows;
  p.k_blocks = K / 128;
  p.units = int64_t(p.row_blocks) * p.column_tiles * p.k_blocks;
  // a piece of two blocks of K at least
  const int64_t most = p.units / 2 < 1 ? 1 : p.units / 2;
  const int64_t ctas = most < sm_count ? most : sm_count;
  p.per_cta = int((p.units + ctas - 1) / ctas);
  p.ctas = int((p.units + p.per_cta - 1) / p.per_cta);
  p.tmem_columns = 32;
  while (p.tmem_columns < 2 * p.columns) p.tmem_columns *= 2;
  const size_t stage = size_t(2) * kWeightHalf + size_t(p.columns) * 256;
  p.stages = int(std::min<size_t>(kMostStages, (room - kLeastCodeSlots * codes) / stage));
  p.code_slots = int(std::min<size_t>(kMostCodeSlots, (room - p.stages * stage) / codes));
  p.smem = 1024 + levels + scales + p.stages * stage + p.code_slots * codes;
  return p;
}

using EncodeMap = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeMap map_encoder() {
  static EncodeMap function = []() -> EncodeMap {
    void* entry = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeMap>(entry);
  }();
  return function;
}

template <bool BF16, int DECODE, int BITS>
int launch_tiles(const TileArgs& a, const TilePlan& p, const CUtensorMap& rows, const CUtensorMap& codes, cudaStream_t stream) {
  auto kernel = gemm_tile_kernel<BF16, DECODE, BITS>;
  static bool configured[64];
  int device = 0;
  cudaGetDevice(&device);
  if (device < 0 || device >= 64 || !configured[device]) {
    const cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, device_info().max_smem_optin - 512);
    if (status != cudaSuccess) return cuda_fail(status, "gemm_tile: shared memory opt-in");
    if (device >= 0 && device < 64) configured[device] = true;
  }
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(unsigned(p.ctas));
  config.blockDim = dim3(kTileThreads);
  config.dynamicSmemBytes = p.smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  cudaError_t launched = cudaLaunchKernelEx(&config, kernel, rows, codes, a);
  if (launched != cudaSuccess) return cuda_fail(launched, "gemm_tile launch");
  if (p.per_cta % p.k_blocks != 0 && p.ctas > 1) {    // some tile is cut
    config.gridDim = dim3(unsigned(p.ctas - 1), unsigned((p.columns + 7) / 8));
    config.blockDim = dim3(kTileRows);
    config.dynamicSmemBytes = 0;
    launched = cudaLaunchKernelEx(&config, gemm_tile_sum_kernel<BF16>, a);
    if (launched != cudaSuccess) return cuda_fail(launched, "gemm_tile sum launch");
  }
  return MKB_OK;
}

template <bool BF16>
int launch_codec(const TileArgs& a, const TilePlan& p, const CUtensorMap& rows, const CUtensorMap& codes, int bits, bool table,
                 cudaStream_t stream) {
  if (!table) return launch_tiles<BF16, DECODE_INT4, 4>(a, p, rows, codes, stream);
  switch (bits) {
    case 2: return launch_tiles<BF16, DECODE_TABLE, 2>(a, p, rows, codes, stream);
    case 3: return launch_tiles<BF16, DECODE_TABLE, 3>(a, p, rows, codes, stream);
    case 4: return launch_tiles<BF16, DECODE_TABLE, 4>(a, p, rows, codes, stream);
    case 5: return launch_tiles<BF16, DECODE_TABLE, 5>(a, p, rows, codes, stream);
    case 6: return launch_tiles<BF16, DECODE_TABLE, 6>(a, p, rows, codes, stream);
    case 7: return launch_tiles<BF16, DECODE_TABLE, 7>(a, p, rows, codes, stream);
    default: return launch_tiles<BF16, DECODE_TABLE, 8>(a, p, rows, codes, stream);
  }
}

bool int4_grid(int bits, int lut_len, int integer_grid, float grid_minimum) {
  return bits == 4 && integer_grid && lut_len == 16 && grid_minimum == float(int(grid_minimum)) && grid_minimum >= -512.f &&
         grid_minimum <= 512.f;
}

int64_t partial_bytes(int M) {
  const int64_t columns = M < 256 ? (M + 15) & ~15 : 256;     // no plan is wider, none has more pieces than SMs
  return int64_t(device_info().sm_count) * 2 * columns * kTileRows * 4;
}

int gemm(const void* x, const uint8_t* packed, const void* scales, const float* lut, const void* zeros, const void* bias, void* y,
         int M, int N, int K, int group, int bits, int lut_len, int x_dtype, int64_t packed_row_stride, int64_t scale_row_stride,
         int integer_grid, float grid_minimum, void* partials, int* status, void* stream) {
  const auto aligned = [](const void* p, uintptr_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; };
  const bool table = !int4_grid(bits, lut_len, integer_grid, grid_minimum);
  const DeviceInfo& info = device_info();
  const TilePlan p = plan_tiles(M, N, K, bits, table, zeros != nullptr, info.sm_count, info.max_smem_optin);
  MKB_REQUIRE(p.stages >= 2 && p.code_slots >= kLeastCodeSlots, MKB_E_UNSUPPORTED, "gemm: no room for the stages");
  MKB_REQUIRE(p.units < (int64_t(1) << 30), MKB_E_UNSUPPORTED, "gemm: %d rows of %d outputs are too many tiles", M, N);
  const EncodeMap encode = map_encoder();
  MKB_REQUIRE(encode != nullptr, MKB_E_CUDA, "gemm: the driver does not offer cuTensorMapEncodeTiled");
  CUtensorMap rows_map, codes_map;
  const cuuint32_t unit[2] = {1, 1};
  const cuuint64_t row_dims[2] = {cuuint64_t(K), cuuint64_t(M)}, row_strides[1] = {cuuint64_t(K) * 2};
  const cuuint32_t row_box[2] = {64, cuuint32_t(p.columns)};
  CUresult encoded = encode(&rows_map, x_dtype == MKB_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                            const_cast<void*>(x), row_dims, row_strides, row_box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  MKB_REQUIRE(encoded == CUDA_SUCCESS, MKB_E_CUDA, "gemm: cuTensorMapEncodeTiled failed with %d", int(encoded));
  const cuuint64_t code_dims[2] = {cuuint64_t(K) / 8 * bits, cuuint64_t(N)}, code_strides[1] = {cuuint64_t(packed_row_stride)};
  const cuuint32_t code_box[2] = {cuuint32_t(16 * bits), cuuint32_t(kTileRows)};
  const CUtensorMapSwizzle swizzle = bits == 2 ? CU_TENSOR_MAP_SWIZZLE_32B : bits == 4 ? CU_TENSOR_MAP_SWIZZLE_64B
                                     : bits == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE;
  encoded = encode(&codes_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<uint8_t*>(packed), code_dims, code_strides, code_box, unit,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  MKB_REQUIRE(encoded == CUDA_SUCCESS, MKB_E_CUDA, "gemm: cuTensorMapEncodeTiled failed with %d", int(encoded));
  TileArgs a{};
  a.scales = static_cast<const __half*>(scales); a.zeros = static_cast<const __half*>(zeros); a.lut = lut;
  a.bias = static_cast<const uint16_t*>(bias); a.y = static_cast<uint16_t*>(y);
  a.status = status;
  a.partials = static_cast<float*>(partials);
  a.scale_row_stride = scale_row_stride;
  a.M = M; a.N = N; a.lut_len = lut_len;
  a.word_scales = aligned(scales, 4) && aligned(zeros, 4) && (int64_t(N) * scale_row_stride) % 2 == 0;
  a.group_shift = group == 128 ? 7 : group == 64 ? 6 : 5;
  a.columns = p.columns; a.column_tiles = p.column_tiles; a.k_blocks = p.k_blocks;
  a.units = int(p.units); a.per_cta = p.per_cta; a.stages = p.stages; a.code_slots = p.code_slots; a.tmem_columns = p.tmem_columns;
  a.grid_min = grid_minimum;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  return x_dtype == MKB_BF16 ? launch_codec<true>(a, p, rows_map, codes_map, bits, table, s)
                             : launch_codec<false>(a, p, rows_map, codes_map, bits, table, s);
}

}  // namespace
}  // namespace mkb

extern "C" int64_t mkb_gemm_tile_partial_bytes(int M) { return M < 1 ? 0 : mkb::partial_bytes(M); }

extern "C" int mkb_gemm_tile(const void* x, const uint8_t* packed, const void* scales, const float* lut, const void* zeros,
                             const void* bias, void* y, int M, int N, int K, int group, int bits, int lut_len, int x_dtype,
                             int scale_dtype, int64_t packed_row_stride, int64_t scale_row_stride, int integer_grid,
                             float grid_minimum, void* partials, int64_t bytes, int* status, void* stream) {
  using namespace mkb;
  MKB_REQUIRE(M >= 1 && N >= 1 && K >= 1 && group >= 1, MKB_E_ARGUMENT, "gemm_tile: bad shape");
  MKB_REQUIRE(x && packed && scales && lut && y && partials && status, MKB_E_ARGUMENT, "gemm_tile: null pointer");
  MKB_REQUIRE(bits >= 2 && bits <= 8 && lut_len >= 1 && lut_len <= (1 << bits), MKB_E_UNSUPPORTED, "gemm_tile: 2 to 8 bits");
  MKB_REQUIRE((x_dtype == MKB_F16 || x_dtype == MKB_BF16) && scale_dtype == MKB_F16 && K % 128 == 0 &&
                  (group == 128 || group == 64 || group == 32),
              MKB_E_UNSUPPORTED, "gemm_tile: needs fp16 or bf16 rows, fp16 scales per 128, 64 or 32 codes and K a multiple of 128");
  MKB_REQUIRE(reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(packed) % 16 == 0 && packed_row_stride % 16 == 0,
              MKB_E_UNSUPPORTED, "gemm_tile: x, packed and its rows start on 16-byte boundaries");
  MKB_REQUIRE(reinterpret_cast<uintptr_t>(partials) % 16 == 0 && bytes >= partial_bytes(M), MKB_E_ARGUMENT,
              "gemm_tile: %lld B for partials, %lld needed", (long long)bytes, (long long)partial_bytes(M));
  return gemm(x, packed, scales, lut, zeros, bias, y, M, N, K, group, bits, lut_len, x_dtype, packed_row_stride, scale_row_stride,
              integer_grid, grid_minimum, partials, status, stream);
}

// ---- the entry point of up to 128 fp16 rows of symmetric INT4 g128: one workspace, a head whose last word is the status
// and the partials ----
extern "C" int64_t mkb_gemm_workspace_bytes(int M, int N, int K) {
  if (M < 1 || M > 128 || N < 1 || K < 128 || K % 128 != 0) return 0;
  return mkb::kTileHead + mkb::partial_bytes(M);
}

extern "C" int mkb_gemm(const void* x, const uint8_t* packed, const void* scales, const float* lut, const void* zeros,
                        const void* bias, void* y, int M, int N, int K, int group, int bits, int lut_len, int x_dtype,
                        int scale_dtype, int64_t packed_row_stride, int64_t scale_row_stride, int integer_grid,
                        float grid_minimum, void* workspace, int64_t workspace_bytes, void* stream) {
  using namespace mkb;
  MKB_REQUIRE(M >= 1 && N >= 1 && K >= 1 && group >= 1, MKB_E_ARGUMENT, "gemm: bad shape");
  MKB_REQUIRE(x && packed && scales && y && workspace, MKB_E_ARGUMENT, "gemm: null pointer");
  MKB_REQUIRE(M <= 128 && bits == 4 && integer_grid && zeros == nullptr && grid_minimum == -8.f && lut_len == 16 && x_dtype == MKB_F16 &&
                  scale_dtype == MKB_F16 && K % 128 == 0 && group == 128 && reinterpret_cast<uintptr_t>(x) % 16 == 0 &&
                  reinterpret_cast<uintptr_t>(packed) % 16 == 0 && packed_row_stride % 16 == 0,
              MKB_E_UNSUPPORTED,
              "gemm: needs 1..128 fp16 rows, symmetric INT4 on the integer grid -8..7 with fp16 scales per 128 codes, "
              "K a multiple of 128 and 16-byte aligned x and packed");
  const int64_t need = mkb_gemm_workspace_bytes(M, N, K);
  MKB_REQUIRE(workspace_bytes >= need, MKB_E_ARGUMENT, "gemm: workspace of %lld B, %lld needed", (long long)workspace_bytes, (long long)need);
  return gemm(x, packed, scales, lut, nullptr, bias, y, M, N, K, group, bits, lut_len, x_dtype, packed_row_stride, scale_row_stride,
              integer_grid, grid_minimum, static_cast<uint8_t*>(workspace) + kTileHead, static_cast<int*>(workspace) + kTileHead / 4 - 1, stream);
}

extern "C" int mkb_gemm_status(const void* workspace, int* status) {
  using namespace mkb;
  MKB_REQUIRE(workspace != nullptr && status != nullptr, MKB_E_ARGUMENT, "gemm_status: null pointer");
  const cudaError_t done = cudaMemcpy(status, static_cast<const int*>(workspace) + kTileHead / 4 - 1, sizeof(int), cudaMemcpyDeviceToHost);
  if (done != cudaSuccess) return cuda_fail(done, "gemm_status");
  return MKB_OK;
}
