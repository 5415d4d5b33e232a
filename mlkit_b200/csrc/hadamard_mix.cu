// The structured transform  y = (B kron H_P)(x * signs)  of many 16-bit rows whose factor basis is a Hadamard matrix,
// all entries +-b (a Paley basis): width = F * P with F <= 48, 128 <= P <= 1024, and F <= 32 at P = 1024 (the row and
// its fp32 values have to fit shared memory: 33 x 1024 would need 235 KB of the 227).
//
// The factor kernel of hadamard.cu gives a row to ceil(F / 4) CTAs, each of which reads the whole row and spends F
// multiply-adds per value: at 4096 rows of 14336 = 28 x 512 it is bound by those and by its two-byte loads (450 us).
// Here a row belongs to one CTA, is read once, and the F-point mix is a tensor-core product: a 16-bit value times +-1
// is exact, so mma.sync forms the same sums in fp32 (the factor b joins the last multiplication, which saves a
// rounding).  At 56 values per thread the butterflies then are the work, about 18 operations per value.
//   * the row arrives by cp.async in shared memory [F][P]; ldmatrix.trans makes the B fragments (K = f, N = p) and
//     the sign flips are exclusive-ors from two to four registers of sign bits;
//   * a warp owns P / 8 consecutive p of every f: stage 0 pairs the two columns of an accumulator, stages 1 and 2
//     are lane exchanges, the next ones pair accumulator tiles, all in ascending stride;
//   * the fp32 values meet in shared memory [F][P + 8] (the pitch keeps the 8-byte stores free of bank conflicts);
//     the last three stages, scale, inverse sign flip, rounding and store follow, eight by four values per step,
//     while the next row is on its way.
// Two CTAs share an SM and hide each other's barriers.  4099 rows of 14336 fp16: 451 -> 70 us (3360 GB/s of the
// 6535 a copy reaches; issue slots bound it), 4099 rows of 6144 = 12 x 512: 128 -> 35 us.
#include <mutex>
#include <set>
#include <utility>

#include "mkb_common.cuh"

namespace mkb {
namespace {

constexpr int kMixWarps = 8;
constexpr int kMixThreads = kMixWarps * 32;

struct MixArgs {
  const uint16_t* x;
  const int8_t* signs;
  const float* basis;   // F x F, entries +-b
  uint16_t* y;
  int64_t M;
  int W, F, P, inverse;
  float scale;          // 1 / sqrt(P), or 1; b joins in the kernel
};

__device__ __forceinline__ void mix_copy16(uint32_t to, const void* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}

template <bool BF16>
__device__ __forceinline__ void mix_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (BF16)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool BF16>
__device__ __forceinline__ uint32_t mix_pair(float low, float high) {
  if constexpr (BF16) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(low, high);
    return *reinterpret_cast<const uint32_t*>(&pair);
  } else {
    const __half2 pair = __floats2half2_rn(low, high);
    return *reinterpret_cast<const uint32_t*>(&pair);
  }
}

// FT: 16-row tiles that hold F (of the output rows and of the contraction alike); NT: 8-column tiles of a warp, P = 64 NT
// where shared memory leaves room for one CTA per SM only, that one gets all the registers
__host__ __device__ constexpr int mix_residents(int ft, int nt) { return (nt == 16 && ft > 1) || (nt == 8 && ft > 2) ? 1 : 2; }
template <int FT, int NT, bool BF16>
__global__ void __launch_bounds__(kMixThreads, mix_residents(FT, NT)) hadamard_mix_kernel(const MixArgs a) {
  extern __shared__ __align__(16) uint8_t smem[];
  constexpr int P = 64 * NT, C = 8 * NT, PITCH = P + 8;
  constexpr int FLAGS = FT * NT * 2;                    // B fragments of a row: one sign bit per half each
  float* z = reinterpret_cast<float*>(smem);            // [F][PITCH]
  uint16_t* x_s = reinterpret_cast<uint16_t*>(z + a.F * PITCH);   // [16 * FT][PITCH]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const uint32_t x_base = uint32_t(__cvta_generic_to_shared(x_s));
  const int chunks = a.W / 8;
  auto fetch = [&](int64_t row) {
    if (row < a.M)
      for (int i = threadIdx.x; i < chunks; i += kMixThreads) {
        const int f = i / (P / 8), c = i % (P / 8);
        mix_copy16(x_base + (f * PITCH + c * 8) * 2, a.x + row * a.W + i * 8);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // the basis and the signs may come from the kernel before, like x
  asm volatile("griddepcontrol.wait;" ::: "memory");
  fetch(blockIdx.x);
  // rows F .. 16 FT of the contraction are zero on both sides
  for (int i = threadIdx.x; i < (16 * FT - a.F) * PITCH; i += kMixThreads) x_s[a.F * PITCH + i] = 0;

  constexpr uint32_t one = BF16 ? 0x3f80u : 0x3c00u, minus = one | 0x8000u;
  uint32_t basis[FT][FT][4];
#pragma unroll
  for (int m = 0; m < FT; ++m)
#pragma unroll
    for (int k = 0; k < FT; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint32_t pair = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int out = 16 * m + g + (i & 1) * 8, in = 16 * k + 2 * t + (i >> 1) * 8 + h;
          if (out < a.F && in < a.F) pair |= (a.basis[a.inverse ? in * a.F + out : out * a.F + in] > 0.f ? one : minus) << (16 * h);
        }
        basis[m][k][i] = pair;
      }
  const float scale = __fmul_rn(a.scale, fabsf(a.basis[0]));
  // fragment (tile j, step k, half i) takes flag n = (j * FT + k) * 2 + i: bits n % 16 (low half) and n % 16 + 16
  uint32_t flips[(FLAGS + 15) / 16];
#pragma unroll
  for (int n = 0; n < (FLAGS + 15) / 16; ++n) flips[n] = 0;
  if (a.signs != nullptr && !a.inverse) {
#pragma unroll
    for (int n = 0; n < FLAGS; ++n) {
      const int i = n & 1, k = (n >> 1) % FT, j = (n >> 1) / FT;
      const int f = 16 * k + 2 * t + 8 * i, p = warp * C + 8 * j + g;
      const uint32_t low = f < a.F && a.signs[f * P + p] < 0, high = f + 1 < a.F && a.signs[(f + 1) * P + p] < 0;
      flips[n / 16] |= (low | high << 16) << (n % 16);
    }
  }

  for (int64_t row = blockIdx.x; row < a.M; row += gridDim.x) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();      // the row has landed; the last one's values have left z
#pragma unroll
    for (int m = 0; m < FT; ++m) {
      float d[NT][4];
#pragma unroll
      for (int j = 0; j < NT; ++j) {
#pragma unroll
        for (int c = 0; c < 4; ++c) d[j][c] = 0.f;
#pragma unroll
        for (int k = 0; k < FT; ++k) {
          uint32_t b0, b1;
          const uint32_t at = x_base + ((16 * k + (lane & 15)) * PITCH + warp * C + 8 * j) * 2;
          asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(b0), "=r"(b1) : "r"(at));
          const int n = (j * FT + k) * 2;
          b0 ^= (flips[n / 16] << (15 - n % 16)) & 0x80008000u;
          b1 ^= (flips[n / 16] << (14 - n % 16)) & 0x80008000u;
          mix_mma<BF16>(d[j], basis[m][k], b0, b1);
        }
      }
      // stages 0, 1, 2: the columns of a tile
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int c = 0; c < 4; c += 2) {
          const float low = d[j][c], high = d[j][c + 1];
          d[j][c] = __fadd_rn(low, high);
          d[j][c + 1] = __fsub_rn(low, high);
        }
#pragma unroll
      for (int s = 1; s <= 2; ++s) {
        const float sign = (t & s) ? -1.f : 1.f;    // the lane with the bit set keeps low - high
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
          for (int c = 0; c < 4; ++c) d[j][c] = __fmaf_rn(d[j][c], sign, __shfl_xor_sync(0xffffffffu, d[j][c], s));
      }
      // the tiles of the warp
#pragma unroll
      for (int span = 1; span < NT; span *= 2)
#pragma unroll
        for (int j = 0; j < NT; ++j)
          if ((j & span) == 0) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float low = d[j][c], high = d[j + span][c];
              d[j][c] = __fadd_rn(low, high);
              d[j + span][c] = __fsub_rn(low, high);
            }
          }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int f = 16 * m + g + 8 * h;
        if (f < a.F) {
#pragma unroll
          for (int j = 0; j < NT; ++j)
            *reinterpret_cast<float2*>(z + f * PITCH + warp * C + 8 * j + 2 * t) = make_float2(d[j][2 * h], d[j][2 * h + 1]);
        }
      }
    }
    __syncthreads();      // z is complete and x_s is free
    fetch(row + gridDim.x);
    for (int task = threadIdx.x; task < a.F * (C / 4); task += kMixThreads) {
      const int f = task / (C / 4), column = task % (C / 4) * 4;
      float4 v[kMixWarps];
#pragma unroll
      for (int s = 0; s < kMixWarps; ++s) v[s] = *reinterpret_cast<const float4*>(z + f * PITCH + s * C + column);
#pragma unroll
      for (int span = 1; span < kMixWarps; span *= 2)
#pragma unroll
        for (int s = 0; s < kMixWarps; ++s)
          if ((s & span) == 0) {
            const float4 low = v[s], high = v[s + span];
            v[s] = make_float4(__fadd_rn(low.x, high.x), __fadd_rn(low.y, high.y), __fadd_rn(low.z, high.z), __fadd_rn(low.w, high.w));
            v[s + span] = make_float4(__fsub_rn(low.x, high.x), __fsub_rn(low.y, high.y), __fsub_rn(low.z, high.z), __fsub_rn(low.w, high.w));
          }
#pragma unroll
      for (int s = 0; s < kMixWarps; ++s) {
        const int at = f * P + s * C + column;
        uint2 out = make_uint2(mix_pair<BF16>(__fmul_rn(v[s].x, scale), __fmul_rn(v[s].y, scale)),
                               mix_pair<BF16>(__fmul_rn(v[s].z, scale), __fmul_rn(v[s].w, scale)));
        if (a.signs != nullptr && a.inverse) {     // the sign byte's top bit flips the rounded value: same bits
          const uint32_t flip = *reinterpret_cast<const uint32_t*>(a.signs + at);
          out.x ^= ((flip & 0x80u) << 8) | ((flip & 0x8000u) << 16);
          out.y ^= ((flip & 0x800000u) >> 8) | (flip & 0x80000000u);
        }
        *reinterpret_cast<uint2*>(a.y + row * a.W + at) = out;
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

int opt_in_shared(const void* kernel, int bytes) {
  static std::mutex lock;
  static std::set<std::pair<const void*, int>> done;
  int device = 0;
  cudaGetDevice(&device);
  std::lock_guard<std::mutex> guard(lock);
  if (done.count({kernel, device})) return MKB_OK;
  const cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (status != cudaSuccess) return cuda_fail(status, "hadamard_mix: shared memory opt-in");
  done.insert({kernel, device});
  return MKB_OK;
}

template <int FT, int NT>
int launch_mix(const MixArgs& a, int dtype, cudaStream_t stream) {
  auto kernel = dtype == MKB_BF16 ? hadamard_mix_kernel<FT, NT, true> : hadamard_mix_kernel<FT, NT, false>;
  constexpr int PITCH = 64 * NT + 8;
  const size_t smem = size_t(a.F) * PITCH * 4 + size_t(16 * FT) * PITCH * 2;
  const DeviceInfo& info = device_info();
  MKB_REQUIRE(smem <= size_t(info.max_smem_optin), MKB_E_UNSUPPORTED, "hadamard_mix: width %d needs %zu B shared memory", a.W, smem);
  // once per instance and device and to the device's limit: factors of one instance need different amounts, and a limit
  // that follows the call could be lowered by another thread before this one launches
  const int opted = opt_in_shared(reinterpret_cast<const void*>(kernel), info.max_smem_optin);
  if (opted != MKB_OK) return opted;
  const int64_t resident = int64_t(info.sm_count) * mix_residents(FT, NT);
  cudaLaunchConfig_t config{};
  config.gridDim = dim3(unsigned(a.M < resident ? a.M : resident));
  config.blockDim = dim3(kMixThreads);
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[1];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = 1;
  config.attrs = attribute;
  config.numAttrs = 1;
  const cudaError_t launched = cudaLaunchKernelEx(&config, kernel, a);
  if (launched != cudaSuccess) return cuda_fail(launched, "hadamard_mix launch");
  return MKB_OK;
}

template <int FT>
int launch_factor(const MixArgs& a, int dtype, cudaStream_t stream) {
  switch (a.P) {
    case 128: return launch_mix<FT, 2>(a, dtype, stream);
    case 256: return launch_mix<FT, 4>(a, dtype, stream);
    case 512: return launch_mix<FT, 8>(a, dtype, stream);
    default:
      if constexpr (FT <= 2) return launch_mix<FT, 16>(a, dtype, stream);
      else MKB_REQUIRE(false, MKB_E_UNSUPPORTED, "hadamard_mix: factors above 32 with 1024 do not fit shared memory");
  }
}

}  // namespace
}  // namespace mkb

extern "C" int mkb_hadamard_mix(const void* x, const int8_t* signs, const float* basis, void* y, int64_t M, int W, int factor,
                                int pow2, int dtype, int inverse, int normalize, void* stream) {
  using namespace mkb;
  MKB_REQUIRE(M >= 0 && W >= 1 && factor >= 1 && pow2 >= 1 && int64_t(factor) * pow2 == W, MKB_E_ARGUMENT, "hadamard_mix: bad shape");
  MKB_REQUIRE((dtype == MKB_F16 || dtype == MKB_BF16) && factor >= 2 && factor <= 48 &&
                  (pow2 == 128 || pow2 == 256 || pow2 == 512 || pow2 == 1024),
              MKB_E_UNSUPPORTED, "hadamard_mix: 16-bit rows, factors of 2 to 48 and powers of two from 128 to 1024 only");
  if (M == 0) return MKB_OK;
  MKB_REQUIRE(x && y && basis, MKB_E_ARGUMENT, "hadamard_mix: null pointer");
  const auto aligned = [](const void* p, uintptr_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; };
  MKB_REQUIRE(aligned(x, 16) && aligned(y, 8) && (signs == nullptr || aligned(signs, 4)), MKB_E_UNSUPPORTED,
              "hadamard_mix: x, y and signs start on 16, 8 and 4 byte boundaries");
  MixArgs a{};
  a.x = static_cast<const uint16_t*>(x); a.signs = signs; a.basis = basis; a.y = static_cast<uint16_t*>(y);
  a.M = M; a.W = W; a.F = factor; a.P = pow2; a.inverse = inverse;
  a.scale = normalize ? 1.0f / float(sqrt(double(pow2))) : 1.0f;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (factor <= 16) return launch_factor<1>(a, dtype, s);
  if (factor <= 32) return launch_factor<2>(a, dtype, s);
  return launch_factor<3>(a, dtype, s);
}
