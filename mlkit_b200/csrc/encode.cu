// Round-to-nearest encoding of a weight matrix onto a scalar grid with one fp16 scale per row group,
// and packing of the codes into the little-endian bit stream, in one launch (sm_100a).
//
// The arithmetic is the tensor route of the reference, operation for operation, so codes and scales
// are bit-equal to it: per group, scale = max(|w|) clamped from below at 1e-12, times the fp32
// reciprocal of the largest level magnitude, rounded to fp16 (clamped to [2^-24, 65504]); code =
// round-half-even(w / scale) clamped to the grid for integer grids, the nearest level (a tie takes
// the lower one) for codebooks; the division is IEEE binary32.
// Two kernels.
//  * run kernel (groups of 8 to 256 codes, a power of two; rows of whole runs of eight codes): a lane owns eight
//    consecutive weights, which are `bits` whole bytes of the stream.  The weights are read once, as 16-byte
//    loads in their own type, and stay in registers; a group's range is a lane exchange; codes and stream leave as
//    one store each.  Bound by memory: 3.5 bytes per bf16 weight at 4 bits (2 read, 1 + 0.5 written).  The IEEE
//    division per weight and the conversions to integers would cost more than the traffic, so the quotient is formed
//    from the group's reciprocal (three operations, same rounding) and rounded to an integer by an addition.  An offset per group and a
//    flag for infinities and NaNs are formed on the way.
//  * group kernel (every other group): one warp per group, a pass for the range, a pass for the codes (through
//    shared memory), then each lane assembles whole bytes of the stream.
#include <cfloat>

#include "mkb_common.cuh"

namespace mkb {
namespace {

constexpr int kEncodeWarps = 8;
constexpr int kMaxGroup = 1024;

struct EncodeArgs {
  const void* weight;
  const float* levels;
  uint8_t* packed;
  __half* scales;
  uint8_t* codes;
  int64_t rows;
  int width, group, groups, bits, level_count, integer, weight_dtype;
  float low, high, reciprocal;
  // run kernel only
  float* scales32;     // the stored scales widened
  float* offsets32;    // asymmetric: the stored offsets widened
  int* nonfinite;      // set to 1 when a weight is not finite
  int lane_shift;      // log2(group / 8): lanes of a group
  uint32_t row_magic;  // index / (groups << lane_shift) = (umulhi(magic, index) + index) >> shift, for index < 2^31
  int row_shift;
};

__device__ __forceinline__ int nearest_level(float x, const float* levels, int count) {
  // first level >= x (binary search), then the closer of it and the one below; a tie goes below
  int lo = 0, hi = count;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (levels[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  const int above = min(lo, count - 1), below = max(above - 1, 0);
  return fabsf(__fsub_rn(x, levels[below])) <= fabsf(__fsub_rn(x, levels[above])) ? below : above;
}

__global__ void __launch_bounds__(kEncodeWarps * 32) rtn_encode_kernel(const EncodeArgs a) {
  __shared__ uint8_t code_s[kEncodeWarps][kMaxGroup];
  __shared__ float level_s[256];
  for (int i = threadIdx.x; i < a.level_count; i += blockDim.x) level_s[i] = a.levels[i];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t total = a.rows * a.groups;
  for (int64_t item = int64_t(blockIdx.x) * kEncodeWarps + warp; item < total; item += int64_t(gridDim.x) * kEncodeWarps) {
    const int64_t row = item / a.groups;
    const int gi = int(item - row * a.groups);
    const int first = gi * a.group, count = min(a.group, a.width - first);
    const int64_t base = row * a.width + first;
    float biggest = 0.f;
    for (int i = lane; i < count; i += 32) biggest = fmaxf(biggest, fabsf(load_as_float(a.weight, base + i, a.weight_dtype)));
#pragma unroll
    for (int offset = 16; offset; offset >>= 1) biggest = fmaxf(biggest, __shfl_xor_sync(0xffffffffu, biggest, offset));
    float scale = __fmul_rn(fmaxf(biggest, 1e-12f), a.reciprocal);
    const __half stored = __float2half_rn(fminf(fmaxf(scale, 5.9604644775390625e-08f), 65504.f));
    scale = __half2float(stored);
    if (lane == 0) a.scales[row * a.groups + gi] = stored;
    for (int i = lane; i < count; i += 32) {
      const float normalized = __fdiv_rn(load_as_float(a.weight, base + i, a.weight_dtype), scale);
      int code;
      if (a.integer) code = int(fminf(fmaxf(rintf(normalized), a.low), a.high) - a.low);
      else code = nearest_level(normalized, level_s, a.level_count);
      code_s[warp][i] = uint8_t(code);
      if (a.codes != nullptr) a.codes[base + i] = uint8_t(code);
    }
    __syncwarp();
    // the group starts on a byte of the stream (group * bits and width * bits are multiples of 8)
    const int64_t first_byte = (row * int64_t(a.width) + first) * a.bits / 8;
    const int bytes = count * a.bits / 8;
    for (int j = lane; j < bytes; j += 32) {
      uint32_t value = 0;
      const int bit0 = j * 8;
      for (int i = bit0 / a.bits; i * a.bits < bit0 + 8 && i < count; ++i) {
        const int shift = i * a.bits - bit0;  // position of the code's lowest bit relative to the byte
        const uint32_t code = code_s[warp][i];
        value |= shift >= 0 ? code << shift : code >> -shift;
      }
      a.packed[first_byte + j] = uint8_t(value);
    }
    __syncwarp();
  }
}

// ---- run kernel ---------------------------------------------------------------------------------
constexpr int kRunThreads = 256;
constexpr int kRunsPerThread = 2;   // two 16-byte loads in flight per lane
constexpr float kRoundMagic = 12582912.f;           // 1.5 * 2^23: adding it rounds |x| < 2^22 half to even
constexpr uint32_t kRoundMagicBits = 0x4b400000u;   // and leaves the integer in the low bits

// eight weights and the bits of their largest magnitude (a NaN's exceed an infinity's)
__device__ __forceinline__ void load_run8(const void* weight, int64_t at, int dtype, float (&w)[8], uint32_t& largest) {
  if (dtype == MKB_F32) {
    const uint4* source = reinterpret_cast<const uint4*>(static_cast<const float*>(weight) + at);
    const uint4 a = __ldcs(source), b = __ldcs(source + 1);
    const uint32_t bits[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      w[e] = __uint_as_float(bits[e]);
      largest = max(largest, bits[e] & 0x7fffffffu);
    }
    return;
  }
  const uint4 raw = __ldcs(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(weight) + at));
  const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t pair = 0;   // of the magnitudes, both halves of a word at once
#pragma unroll
  for (int i = 0; i < 4; ++i) pair = __vmaxu2(pair, words[i] & 0x7fff7fffu);
  const uint32_t half = max(pair & 0xffffu, pair >> 16);
  if (dtype == MKB_F16) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 two = __half22float2(*reinterpret_cast<const __half2*>(&words[i]));
      w[2 * i] = two.x;
      w[2 * i + 1] = two.y;
    }
    largest = half >= 0x7c00u ? 0x7f800000u : __float_as_uint(__half2float(__ushort_as_half((unsigned short)half)));
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[2 * i] = __uint_as_float(words[i] << 16);
      w[2 * i + 1] = __uint_as_float(words[i] & 0xffff0000u);
    }
    largest = half << 16;
  }
}

// w / scale rounded to fp32, by Markstein's correction of an approximate quotient: the remainder w - q * scale is
// exact, and q plus remainder times reciprocal misses the quotient by 2^-46 of it before its one rounding.  A stored
// scale has eleven significant bits, so no quotient lies within 2^-36 of a point where the rounding would change:
// the result is the IEEE division's.  (Where the remainder underflows the quotient rounds to zero codes anyway.)
__device__ __forceinline__ float quotient(float w, float scale, float inverse) {
  const float q = __fmul_rn(w, inverse);
  return __fmaf_rn(__fmaf_rn(-q, scale, w), inverse, q);
}

template <int BITS, bool INTEGER, bool ASYM>
__global__ void __launch_bounds__(kRunThreads) rtn_encode_runs_kernel(const EncodeArgs a) {
  __shared__ float level_s[256];
  if constexpr (!INTEGER) {
    for (int i = threadIdx.x; i < a.level_count; i += kRunThreads) level_s[i] = a.levels[i];
    __syncthreads();
  }
  const uint32_t lanes_per_group = 1u << a.lane_shift, runs_per_row = uint32_t(a.groups) << a.lane_shift;
  const uint32_t total = uint32_t(a.rows) * runs_per_row;
  const uint32_t first = blockIdx.x * (kRunThreads * kRunsPerThread) + threadIdx.x;
  float w[kRunsPerThread][8];
  uint32_t row[kRunsPerThread], run[kRunsPerThread], largest[kRunsPerThread];
  bool live[kRunsPerThread];
#pragma unroll
  for (int j = 0; j < kRunsPerThread; ++j) {
    const uint32_t index = first + j * kRunThreads;
    row[j] = (__umulhi(a.row_magic, index) + index) >> a.row_shift;   // index / runs_per_row
    run[j] = index - row[j] * runs_per_row;
    live[j] = index < total && run[j] * 8 < uint32_t(a.width);    // the last group of a row may be short
    largest[j] = 0;
    if (live[j]) load_run8(a.weight, int64_t(row[j]) * a.width + run[j] * 8, a.weight_dtype, w[j], largest[j]);
  }
  bool bad = false;
#pragma unroll
  for (int j = 0; j < kRunsPerThread; ++j) {
    bad |= largest[j] >= 0x7f800000u;
    [[maybe_unused]] float low = INFINITY, high = -INFINITY;
    float range;
    if constexpr (ASYM) {
      if (live[j]) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          low = fminf(low, w[j][e]);
          high = fmaxf(high, w[j][e]);
        }
      }
      for (uint32_t offset = lanes_per_group / 2; offset; offset >>= 1) {
        low = fminf(low, __shfl_xor_sync(0xffffffffu, low, offset));
        high = fmaxf(high, __shfl_xor_sync(0xffffffffu, high, offset));
      }
      range = __fsub_rn(high, low);
    } else {
      for (uint32_t offset = lanes_per_group / 2; offset; offset >>= 1)
        largest[j] = max(largest[j], __shfl_xor_sync(0xffffffffu, largest[j], offset));
      range = __uint_as_float(largest[j]);
    }
    const float wide = __fmul_rn(fmaxf(range, 1e-12f), a.reciprocal);
    const __half stored = __float2half_rn(fminf(fmaxf(wide, 5.9604644775390625e-08f), 65504.f));
    const float scale = __half2float(stored);
    float offset = 0.f;
    if constexpr (ASYM) {
      const float exact = __fsub_rn(low, __fmul_rn(a.low, wide));     // from the scale before it is stored
      const float size = __half2float(__float2half_rn(fminf(fmaxf(fabsf(exact), 5.9604644775390625e-08f), 65504.f)));
      offset = exact > 0.f ? size : exact < 0.f ? -size : 0.f;
    }
    if (!live[j]) continue;
    if ((run[j] & (lanes_per_group - 1)) == 0) {
      const int64_t at = int64_t(row[j]) * a.groups + (run[j] >> a.lane_shift);
      if (a.scales != nullptr) a.scales[at] = stored;
      if (a.scales32 != nullptr) a.scales32[at] = scale;
      if constexpr (ASYM) a.offsets32[at] = offset;
    }
    // codes as the low bits of `code` once `base` is taken away (of all of them at once, modulo the word)
    uint32_t code[8];
    constexpr uint32_t base = INTEGER ? kRoundMagicBits : 0u;
    float divisor = scale, moved = offset;
    if constexpr (ASYM) {
      // a narrow group far from zero: its offset ends at fp16's largest value and quotients by a scale of 2^-24 can
      // overflow, which the correction would turn into NaNs.  (Without an offset a scale grows with the weights.)
      if (fmaxf(fabsf(low), fabsf(high)) >= 1e31f) {
#pragma unroll
        for (int e = 0; e < 8; ++e)
          w[j][e] = fminf(fmaxf(__fdiv_rn(__fsub_rn(w[j][e], offset), scale), -FLT_MAX), FLT_MAX);
        divisor = 1.f;
        moved = 0.f;
      }
    }
    const float inverse = __frcp_rn(divisor);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float q = quotient(ASYM ? __fsub_rn(w[j][e], moved) : w[j][e], divisor, inverse);
      if constexpr (INTEGER) code[e] = __float_as_uint(__fadd_rn(fminf(fmaxf(q, a.low), a.high), kRoundMagic));
      else code[e] = uint32_t(nearest_level(q, level_s, a.level_count));
    }
    const uint32_t shift = INTEGER ? base + uint32_t(int(a.low)) : 0u;   // what a code of zero looks like
    const int64_t at = int64_t(row[j]) * a.width + run[j] * 8;
    if (a.codes != nullptr) {
      const uint32_t off = shift * 0x01010101u;
      *reinterpret_cast<uint2*>(a.codes + at) =
          make_uint2(code[0] + (code[1] << 8) + (code[2] << 16) + (code[3] << 24) - off,
                     code[4] + (code[5] << 8) + (code[6] << 16) + (code[7] << 24) - off);
    }
    uint8_t* to = a.packed + at / 8 * BITS;
    if constexpr (BITS <= 4) {
      uint32_t stream = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) stream += (code[e] - shift) << (e * BITS);
      if constexpr (BITS == 4) *reinterpret_cast<uint32_t*>(to) = stream;
      else if constexpr (BITS == 2) *reinterpret_cast<uint16_t*>(to) = uint16_t(stream);
      else {
#pragma unroll
        for (int b = 0; b < BITS; ++b) to[b] = uint8_t(stream >> (8 * b));
      }
    } else {
      uint64_t stream = 0;
#pragma unroll
      for (int e = 0; e < 8; ++e) stream |= uint64_t(code[e] - shift) << (e * BITS);
      if constexpr (BITS == 8) *reinterpret_cast<uint2*>(to) = make_uint2(uint32_t(stream), uint32_t(stream >> 32));
      else if constexpr (BITS == 6) {
#pragma unroll
        for (int b = 0; b < BITS; b += 2) *reinterpret_cast<uint16_t*>(to + b) = uint16_t(stream >> (8 * b));
      } else {
#pragma unroll
        for (int b = 0; b < BITS; ++b) to[b] = uint8_t(stream >> (8 * b));
      }
    }
  }
  if (bad && a.nonfinite != nullptr) *a.nonfinite = 1;
}

template <int BITS>
void launch_runs(const EncodeArgs& a, unsigned blocks, cudaStream_t stream) {
  const bool asym = a.offsets32 != nullptr;
  if (a.integer) {
    if (asym) rtn_encode_runs_kernel<BITS, true, true><<<blocks, kRunThreads, 0, stream>>>(a);
    else rtn_encode_runs_kernel<BITS, true, false><<<blocks, kRunThreads, 0, stream>>>(a);
  } else {
    if (asym) rtn_encode_runs_kernel<BITS, false, true><<<blocks, kRunThreads, 0, stream>>>(a);
    else rtn_encode_runs_kernel<BITS, false, false><<<blocks, kRunThreads, 0, stream>>>(a);
  }
}

// Whether the run kernel covers a layout.
bool runs_cover(const EncodeArgs& a) {
  const auto aligned = [](const void* p, uintptr_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; };
  const int lanes = a.group / 8;
  return a.group % 8 == 0 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && a.width % 8 == 0 && aligned(a.weight, 16) &&
         aligned(a.packed, 8) && (a.codes == nullptr || aligned(a.codes, 8)) &&
         a.rows * a.groups * lanes < (int64_t(1) << 31);
}

int encode(EncodeArgs a, cudaStream_t stream) {
  if (runs_cover(a)) {
    while ((8 << a.lane_shift) < a.group) ++a.lane_shift;
    // the round-up method of dividing by an invariant: 2^shift is the next power of two from the divisor
    const uint32_t divisor = uint32_t(a.groups) << a.lane_shift;
    while ((uint64_t(1) << a.row_shift) < divisor) ++a.row_shift;
    a.row_magic = uint32_t((((uint64_t(1) << a.row_shift) - divisor) << 32) / divisor + 1);
    const int64_t total = a.rows * a.groups * (a.group / 8), per_block = kRunThreads * kRunsPerThread;
    const unsigned blocks = unsigned((total + per_block - 1) / per_block);
    switch (a.bits) {
      case 1: launch_runs<1>(a, blocks, stream); break;
      case 2: launch_runs<2>(a, blocks, stream); break;
      case 3: launch_runs<3>(a, blocks, stream); break;
      case 4: launch_runs<4>(a, blocks, stream); break;
      case 5: launch_runs<5>(a, blocks, stream); break;
      case 6: launch_runs<6>(a, blocks, stream); break;
      case 7: launch_runs<7>(a, blocks, stream); break;
      default: launch_runs<8>(a, blocks, stream); break;
    }
  } else {
    MKB_REQUIRE(a.offsets32 == nullptr && a.scales32 == nullptr && a.nonfinite == nullptr, MKB_E_UNSUPPORTED,
                "rtn_encode: offsets, wide scales and the finite check need groups of 8 to 256 codes (a power of two) and "
                "rows of whole runs of eight");
    const int64_t items = a.rows * a.groups;
    const int64_t wanted = (items + kEncodeWarps - 1) / kEncodeWarps;
    const int blocks = int(wanted < 148 * 16 ? wanted : 148 * 16);
    rtn_encode_kernel<<<blocks, kEncodeWarps * 32, 0, stream>>>(a);
  }
  MKB_LAUNCH_CHECK("rtn_encode launch");
  return MKB_OK;
}

int check_and_fill(EncodeArgs& a, const void* weight, const float* levels, uint8_t* packed, uint8_t* codes, int64_t N, int K,
                   int group, int bits, int level_count, int integer_grid, float grid_low, float grid_high, float reciprocal,
                   int weight_dtype) {
  MKB_REQUIRE(N >= 0 && K >= 1 && group >= 1 && bits >= 1 && bits <= 8, MKB_E_ARGUMENT, "rtn_encode: bad shape");
  MKB_REQUIRE(level_count >= 1 && level_count <= (1 << bits), MKB_E_ARGUMENT,
              "rtn_encode: %d levels do not fit %d-bit codes", level_count, bits);
  MKB_REQUIRE(weight_dtype >= MKB_F16 && weight_dtype <= MKB_F32, MKB_E_ARGUMENT, "rtn_encode: unknown dtype");
  MKB_REQUIRE(grid_high >= grid_low && reciprocal > 0.f, MKB_E_ARGUMENT, "rtn_encode: bad grid range");
  if (N == 0) return MKB_OK;
  MKB_REQUIRE(weight && packed, MKB_E_ARGUMENT, "rtn_encode: null pointer");
  if (group > K) group = K;
  MKB_REQUIRE(group <= kMaxGroup, MKB_E_UNSUPPORTED, "rtn_encode: groups of more than %d codes", kMaxGroup);
  MKB_REQUIRE((int64_t(group) * bits) % 8 == 0 && (int64_t(K) * bits) % 8 == 0, MKB_E_UNSUPPORTED,
              "rtn_encode: a group or a row of %d-bit codes does not end on a byte", bits);
  a.weight = weight; a.levels = levels; a.packed = packed; a.codes = codes;
  a.rows = N; a.width = K; a.group = group; a.groups = (K + group - 1) / group; a.bits = bits;
  a.level_count = level_count; a.integer = integer_grid; a.weight_dtype = weight_dtype;
  a.low = grid_low; a.high = grid_high; a.reciprocal = reciprocal;
  return MKB_OK;
}

}  // namespace
}  // namespace mkb

extern "C" int mkb_rtn_encode(const void* weight, const float* levels, uint8_t* packed, void* scales, uint8_t* codes,
                              int64_t N, int K, int group, int bits, int level_count, int integer_grid,
                              float grid_low, float grid_high, float reciprocal, int weight_dtype, void* stream) {
  using namespace mkb;
  EncodeArgs a{};
  const int status = check_and_fill(a, weight, levels, packed, codes, N, K, group, bits, level_count, integer_grid, grid_low,
                                    grid_high, reciprocal, weight_dtype);
  if (status != MKB_OK || N == 0) return status;
  MKB_REQUIRE(scales != nullptr && levels != nullptr, MKB_E_ARGUMENT, "rtn_encode: null pointer");
  a.scales = static_cast<__half*>(scales);
  return encode(a, static_cast<cudaStream_t>(stream));
}

extern "C" int mkb_rtn_encode_checked(const void* weight, const float* levels, uint8_t* packed, float* scales, float* offsets,
                                      uint8_t* codes, int* nonfinite, int64_t N, int K, int group, int bits,
                                      int level_count, int integer_grid, float grid_low, float grid_high,
                                      float reciprocal, int weight_dtype, void* stream) {
  using namespace mkb;
  EncodeArgs a{};
  const int status = check_and_fill(a, weight, levels, packed, codes, N, K, group, bits, level_count, integer_grid, grid_low,
                                    grid_high, reciprocal, weight_dtype);
  if (status != MKB_OK || N == 0) return status;
  MKB_REQUIRE(scales != nullptr && nonfinite != nullptr && (levels != nullptr || integer_grid), MKB_E_ARGUMENT, "rtn_encode_checked: null pointer");
  a.scales32 = scales; a.offsets32 = offsets; a.nonfinite = nonfinite;
  MKB_REQUIRE(runs_cover(a), MKB_E_UNSUPPORTED,
              "rtn_encode_checked: needs groups of 8 to 256 codes (a power of two), rows of whole runs of eight codes and a "
              "16-byte aligned weight");
  const cudaError_t cleared = cudaMemsetAsync(nonfinite, 0, sizeof(int), static_cast<cudaStream_t>(stream));
  if (cleared != cudaSuccess) return cuda_fail(cleared, "rtn_encode_checked: clearing the flag");
  return encode(a, static_cast<cudaStream_t>(stream));
}
