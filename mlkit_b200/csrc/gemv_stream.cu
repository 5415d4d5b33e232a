// Host side of the streaming matvec: which calls it covers, and the launch.
#include "gemv_stream.cuh"

namespace mkb {
using namespace stream;
namespace {

int dispatch_stream(const StreamArgs& a, const StreamPlan& p, cudaStream_t stream, int* cluster_cap) {
  if (p.mode == MODE_TABLE)
    return p.xt == X_BF16 ? dispatch_table<X_BF16>(a, p, stream, cluster_cap) : dispatch_table<X_F16>(a, p, stream, cluster_cap);
  if (p.bits == 4)
    return p.xt == X_BF16 ? dispatch_raw4<X_BF16>(a, p, stream, cluster_cap) : dispatch_raw4<X_F16>(a, p, stream, cluster_cap);
  return p.xt == X_BF16 ? dispatch_raw<X_BF16>(a, p, stream, cluster_cap) : dispatch_raw<X_F16>(a, p, stream, cluster_cap);
}

// The codec a call maps to: false when the streaming kernel does not cover it.  Four-bit integer grids take the
// masks whatever their group and offsets: two decoder blocks of an 8B shape at two rows, 128 codes per scale and
// offset, take 78 us here and 174 us in the tiled kernel, which folds scale and offset into every weight; with 64
// codes per scale the gather of the table form costs 1.5x the masks.  Offsets with other widths stay there.
bool codec_of(int group, int bits, int lut_len, int x_dtype, const void* zeros, int integer_grid, float grid_minimum, StreamPlan& p) {
  if (lut_len < 1 || lut_len > (1 << bits)) return false;
  p.xt = x_dtype == MKB_BF16 ? X_BF16 : X_F16;
  p.zero = zeros != nullptr;
  const bool ramp = integer_grid && lut_len == (1 << bits) && grid_minimum == float(int(grid_minimum)) &&
                    grid_minimum >= -512.f && grid_minimum <= 512.f;
  if (ramp && ((group == 128 && bits >= 2 && bits <= 8 && (bits == 4 || !p.zero)) ||
               (bits == 4 && (group == 64 || group == 32)))) {
    p.bits = bits; p.mode = MODE_RAW; p.gpt = 128 / group;
    return true;
  }
  if (!p.zero && (bits == 3 || bits == 4) && (group == 64 || group == 128)) {
    p.bits = bits; p.mode = MODE_TABLE; p.gpt = 128 / group;
    return true;
  }
  return false;
}

}  // namespace

int gemv_stream_supported(int M, int N, int K, int group, int bits, int lut_len, int x_dtype, int scale_dtype,
                          const void* x, const uint8_t* packed, const void* scales, int64_t packed_row_stride,
                          int64_t scale_row_stride, const void* zeros, int integer_grid, float grid_minimum) {
  if ((x_dtype != MKB_F16 && x_dtype != MKB_BF16) || scale_dtype != MKB_F16) return 0;
  if (M < 1 || M > 8 || N < 1 || K < 128 || K % 128 != 0) return 0;
  StreamPlan plan{};
  if (!codec_of(group, bits, lut_len, x_dtype, zeros, integer_grid, grid_minimum, plan)) return 0;
  if (reinterpret_cast<uintptr_t>(x) % 16 || reinterpret_cast<uintptr_t>(packed) % 16 || packed_row_stride % 16) return 0;
  // the scales of a row and visit are copied as one aligned piece of 4, 8 or 16 bytes
  const int scales_per_visit = ((K / 128) % 2 == 0 ? 2 : 1) * plan.gpt;
  const uintptr_t side = reinterpret_cast<uintptr_t>(scales) | reinterpret_cast<uintptr_t>(zeros);
  if (scales_per_visit == 1) {
    if (side % 4 || (int64_t(N) * scale_row_stride) % 2) return 0;  // aligned pairs
  } else if (side % (scales_per_visit * 2) || scale_row_stride % scales_per_visit) {
    return 0;
  }
  if (int64_t(N) * packed_row_stride >= (int64_t(1) << 32) || int64_t(N) * scale_row_stride >= (int64_t(1) << 30)) return 0;
  const DeviceInfo& info = device_info();
  return plan_stream(M, N, K, info.sm_count, info.max_smem_optin, 0, plan) ? 1 : 0;
}

// Rotation on load: K = 2^log2 >= 512 and M * K fp32 values of shared memory beside the rings.
int gemv_stream_rotation_supported(int M, int N, int K, int group, int bits, int lut_len, int integer_grid,
                                   float grid_minimum, const void* signs) {
  if (K < kWarpSpan || (K & (K - 1)) != 0 || size_t(M) * K * 4 > kMaxRotationBytes) return 0;
  if (reinterpret_cast<uintptr_t>(signs) % 16) return 0;
  StreamPlan plan{};
  if (!codec_of(group, bits, lut_len, MKB_F16, nullptr, integer_grid, grid_minimum, plan) || plan.gpt > 2) return 0;
  const DeviceInfo& info = device_info();
  return plan_stream(M, N, K, info.sm_count, info.max_smem_optin, 0, plan, size_t(M) * K * 4) ? 1 : 0;
}

namespace {

int launch_any(const void* x, const uint8_t* packed, const void* scales, const float* lut, const void* zeros,
               const void* bias, void* y, int M, int N, int K, int group, int bits, int lut_len, int x_dtype,
               int64_t packed_row_stride, int64_t scale_row_stride, int integer_grid, float grid_minimum, int gated,
               const int8_t* signs, int rotate, int normalize, cudaStream_t stream) {
  const DeviceInfo& info = device_info();
  StreamPlan p{};
  const size_t extra = rotate ? size_t(M) * K * 4 : 0;
  MKB_REQUIRE(codec_of(group, bits, lut_len, x_dtype, zeros, integer_grid, grid_minimum, p) &&
                  plan_stream(M, N, K, info.sm_count, info.max_smem_optin, 0, p, extra),
              MKB_E_UNSUPPORTED, "gemv_stream: no decomposition for N=%d K=%d bits=%d group=%d", N, K, bits, group);
  p.form = rotate ? FORM_ROTATED : gated ? FORM_GATED : FORM_PLAIN;
  MKB_REQUIRE(p.form == FORM_PLAIN || (p.xt == X_F16 && !p.zero && p.gpt <= 2), MKB_E_UNSUPPORTED,
              "gemv_stream: no rotation or gate with this codec");
  StreamArgs a{};
  if (p.slabs > 1) {  // a grid of clusters must be resident as a whole, or it runs in waves
    int cap = 0;
    const int status = dispatch_stream(a, p, stream, &cap);
    if (status != MKB_OK) return status;
    MKB_REQUIRE(cap >= 1, MKB_E_UNSUPPORTED, "gemv_stream: no cluster of %d CTAs fits the GPU", p.slabs);
    if (p.columns > cap)
      MKB_REQUIRE(plan_stream(M, N, K, info.sm_count, info.max_smem_optin, cap, p, extra),
                  MKB_E_UNSUPPORTED, "gemv_stream: no decomposition for N=%d K=%d in %d clusters", N, K, cap);
  }
  a.x = static_cast<const uint16_t*>(x); a.packed = packed; a.scales = static_cast<const __half*>(scales);
  a.zeros = static_cast<const __half*>(zeros); a.group = group; a.bits = bits;
  a.bias = static_cast<const uint16_t*>(bias); a.y = static_cast<uint16_t*>(y); a.lut = lut; a.lut_len = lut_len;
  a.M = M; a.N = N; a.K = K; a.packed_row_stride = packed_row_stride; a.scale_row_stride = scale_row_stride;
  a.row_tiles = (N + 15) / 16; a.k_warps = K / (128 * p.KT); a.KW = p.KW; a.RG = p.RG; a.slabs = p.slabs;
  a.visits = p.visits; a.grid_min = p.mode == MODE_RAW ? grid_minimum : 0.f; a.batch = p.batch; a.early = 1;
  a.kw_inverse = (65536 + p.KW - 1) / p.KW; a.rg_inverse = (65536 + p.RG - 1) / p.RG;
  if (rotate) {
    a.rot_signs = signs;
    while ((1 << a.rot_log2) < K) ++a.rot_log2;
    a.rot_offset = uint32_t(p.smem - extra);
    // the reference forms the scale in fp32: float(torch.tensor(1.0) / torch.tensor(math.sqrt(width)))
    a.rot_scale = normalize ? 1.0f / float(sqrt(double(K))) : 1.0f;
  }
  return dispatch_stream(a, p, stream, nullptr);
}

}  // namespace

int launch_gemv_stream_rotated(const void* x, const uint8_t* packed, const void* scales, const float* lut,
                               const void* bias, void* y, int M, int N, int K, int group, int bits, int lut_len,
                               int64_t packed_row_stride, int64_t scale_row_stride, int integer_grid,
                               float grid_minimum, const int8_t* signs, int normalize, cudaStream_t stream) {
  return launch_any(x, packed, scales, lut, nullptr, bias, y, M, N, K, group, bits, lut_len, MKB_F16, packed_row_stride,
                    scale_row_stride, integer_grid, grid_minimum, 0, signs, 1, normalize, stream);
}

int launch_gemv_stream(const void* x, const uint8_t* packed, const void* scales, const float* lut, const void* zeros,
                       const void* bias, void* y, int M, int N, int K, int group, int bits, int lut_len, int x_dtype,
                       int64_t packed_row_stride, int64_t scale_row_stride, int integer_grid, float grid_minimum,
                       int gated, cudaStream_t stream) {
  return launch_any(x, packed, scales, lut, zeros, bias, y, M, N, K, group, bits, lut_len, x_dtype, packed_row_stride,
                    scale_row_stride, integer_grid, grid_minimum, gated, nullptr, 0, 0, stream);
}

}  // namespace mkb
