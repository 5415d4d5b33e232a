// One packed weight row times up to MT activation rows in plain fp32, word by word: the arithmetic of the
// coverage matvec, also what the streaming matvec redoes rows with infinities or NaNs through.
#pragma once

#include "mkb_common.cuh"

namespace mkb {

struct ScalarRow {   // one weight row
  const uint8_t* packed;
  const void* scales;
  const void* zeros;      // offsets or null
  const float* lut;       // `lut_len` levels; a code past the end stands for zero
  int K, group, bits, lut_len, scale_dtype;
};

// Adds the products of the words lane, lane + 32, ... to acc[0..M): w = lut[c] * scale (+ zero), one fp32 rounding
// each, then a fused multiply-add per activation row.  activation(m, k) is element k of activation row m.
template <int MT, typename Activation>
__device__ __forceinline__ void scalar_row_products(const ScalarRow& r, const Activation& activation, int M, int lane,
                                                    float (&acc)[MT]) {
  const int wb = word_bytes(r.bits), wc = word_codes(r.bits);
  const int words = r.K / wc;
  const uint32_t mask = (1u << r.bits) - 1u;
  const bool has_zero = r.zeros != nullptr;
  for (int w = lane; w < words; w += 32) {
    uint64_t word = 0;
    const uint8_t* p = r.packed + int64_t(w) * wb;
    for (int b = 0; b < wb; ++b) word |= uint64_t(__ldg(p + b)) << (8 * b);
    const int k0 = w * wc;
    const float scale = load_as_float(r.scales, k0 / r.group, r.scale_dtype);
    const float zero = has_zero ? load_as_float(r.zeros, k0 / r.group, r.scale_dtype) : 0.f;
    for (int c = 0; c < wc; ++c) {
      const int code = int((word >> (c * r.bits)) & mask);
      const float value = code < r.lut_len ? r.lut[code] : 0.f;
      const float weight = has_zero ? reconstruct(value, scale, zero) : reconstruct(value, scale);
#pragma unroll
      for (int m = 0; m < MT; ++m)
        if (m < M) acc[m] = fmaf(weight, activation(m, k0 + c), acc[m]);
    }
  }
}

}  // namespace mkb
