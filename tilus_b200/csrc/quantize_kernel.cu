// load_and_quantize on the GPU: dense weight[out, in] -> per-group scales + packed weights in
// the b200 layout.
//
// The arithmetic is QuantizedLinear.load_and_quantize of the reference
// (examples/quantization/matmul_a16wx.py:470-528), operation for operation so that the codes
// and scales come out bit-identical to the host path (tilus_b200/quantize.py):
//   scales[g, n] = rn(max(absmax(w[n, group g]) / max_value, 1e-6))             (fp32 division, rounded to
//                                                                                 the activation dtype)
//   q            = clamp(w / float(scales), min_value, max_value)               (fp32 division)
//   integer types: code = rint(q) & mask   (round half to even, as torch.round)
//   float types:   code = the reference's fp32 -> sub-byte encode: round to nearest even at the
//                  target's precision, saturate, flush fp32 subnormals to signed zero
//                  (python/tilus/hidet/ir/primitives/cuda/cast.py:44-100)
// One thread per unit (32 codes of one column, decode.cuh / tilus_b200/packing.py): it reads its 32 weights
// with 16-byte loads, quantizes them, builds the unit's plane words in registers (signed integers in
// offset binary) and stores them at the unit's place.  Scale groups of 32, 64 and 128 rows lie inside the four
// neighbouring lanes of a column, so their absmax is a shuffle and the dense weight is read once; other
// groups get their scales from a pass of their own (quant_scales_kernel, one warp per column and group).
//
// What bounds it: HBM (2 or 4 bytes read and b/8 written per weight), provided the arithmetic stays near ten
// instructions per weight.  The IEEE division of the definition alone is as much, so integer codes come
// from one multiplication by the reciprocal of the scale, and only a unit with a value within the
// multiplication's error of a rounding boundary is computed again with the division: the codes are
// those of the division in every case.  fp16 [28672, 4096] -> int4 g128: 544 us for two scalar passes plus
// the copy into the layer, 94 us in this form (45 us at the copy rate of HBM).
#include "common.cuh"

namespace b200q {

struct QuantParams {
  const void* w;   // [N, K] row-major (row = output feature), leading dimension ldw
  int w_dtype;     // 0 fp16, 1 fp32, 2 bf16
  int ldw;
  uint32_t* bq;    // packed output, K*N*nbits/8 bytes
  unsigned short* scales;  // [K/group, N], 16-bit patterns of the activation dtype
  int act;         // 0 fp16, 1 bf16
  int N, K, G, group;  // G = K / 128
  int kind, ebits, mbits;  // kind: 0 unsigned, 1 two's complement, 2 float
  int vec;                 // every row starts on a 16-byte boundary
  int local;               // groups of 32, 64 or 128 rows: inside the four neighbouring lanes of a column
  float minv, maxv;
};

__device__ __forceinline__ float load_scale(const QuantParams& p, size_t idx) {
  const unsigned short b = p.scales[idx];
  return p.act == 0 ? __half2float(__ushort_as_half(b)) : __uint_as_float((uint32_t)b << 16);
}
// max(absmax / max_value, 1e-6), rounded to the activation dtype; the stored bits
__device__ __forceinline__ unsigned short scale_bits(const QuantParams& p, float amax) {
  const float sc = fmaxf(__fdiv_rn(amax, p.maxv), 1e-6f);
  return p.act == 0 ? __half_as_ushort(__float2half_rn(sc)) : __bfloat16_as_ushort(__float2bfloat16_rn(sc));
}

// E consecutive weights from element idx on, E a multiple of 8, as fp32.  WT: 0 fp16, 1 fp32, 2 bf16;
// p.vec: rows are 16-byte aligned
template <int WT, int E>
__device__ __forceinline__ void load_weights(const QuantParams& p, size_t idx, float (&v)[E]) {
  if (p.vec) {
    constexpr int PER = WT == 1 ? 4 : 8;  // weights per 16 bytes
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(p.w) + idx * (WT == 1 ? 4 : 2));
    uint4 raw[E / PER];
#pragma unroll
    for (int i = 0; i < E / PER; ++i) raw[i] = __ldg(src + i);
#pragma unroll
    for (int i = 0; i < E / PER; ++i) {
      const uint32_t x[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if constexpr (WT == 0) {
          const float2 f = __half22float2(h2_from_bits(x[q]));
          v[i * 8 + 2 * q] = f.x; v[i * 8 + 2 * q + 1] = f.y;
        } else if constexpr (WT == 2) {
          v[i * 8 + 2 * q] = __uint_as_float(x[q] << 16);
          v[i * 8 + 2 * q + 1] = __uint_as_float(x[q] & 0xffff0000u);
        } else {
          v[i * 4 + q] = __uint_as_float(x[q]);
        }
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < E; ++i) {
      if constexpr (WT == 0) v[i] = __half2float(reinterpret_cast<const __half*>(p.w)[idx + i]);
      else if constexpr (WT == 2) v[i] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.w)[idx + i]);
      else v[i] = reinterpret_cast<const float*>(p.w)[idx + i];
    }
  }
}

// scales of groups that are not 32, 64 or 128 rows: one warp per (column, group), 8 weights per lane and step
template <int WT>
__global__ void __launch_bounds__(256) quant_scales_kernel(const QuantParams p) {
  const int lane = threadIdx.x & 31;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int groups = p.K / p.group;
  if (wid >= (long long)p.N * groups) return;
  const int n = (int)(wid / groups), g = (int)(wid % groups);
  const size_t base = (size_t)n * p.ldw + (size_t)g * p.group;
  float m = 0.f;
#pragma unroll 2
  for (int i = lane * 8; i < p.group; i += 256) {  // group is a multiple of 32
    float v[8];
    load_weights<WT, 8>(p, base + i, v);
#pragma unroll
    for (int q = 0; q < 8; ++q) m = fmaxf(m, fabsf(v[q]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) p.scales[(size_t)g * p.N + n] = scale_bits(p, m);
}

// fp32 -> sub-byte float code (sign / e exponent bits / m mantissa bits)
__device__ __forceinline__ uint32_t encode_float_code(float x, int nbits, int e, int m) {
  const uint32_t u = __float_as_uint(x);
  const uint32_t sign = ((u >> 31) & 1u) << (nbits - 1);
  const int exps = (int)((u >> 23) & 0xFFu);
  if (exps == 0) return sign;                                   // zero and fp32 subnormals
  if (exps == 0xFF) return (sign | ((1u << nbits) - 1u)) & ((1u << nbits) - 1u);  // Inf / NaN: all ones
  uint32_t mant = (u & 0x7FFFFFu) | 0x800000u;
  const int shift = 23 - m;
  const uint32_t round_bit = (mant >> (shift - 1)) & 1u;
  const bool sticky = (mant & ((1u << (shift - 1)) - 1u)) != 0u;
  const uint32_t lsb = (mant >> shift) & 1u;
  if (round_bit && (sticky || lsb)) mant += 1u << shift;
  int carry = 0;
  if (mant & 0x01000000u) { mant >>= 1; carry = 1; }
  int exp_value = exps - 127 + carry + (1 << (e - 1)) - 1;
  mant >>= shift;
  if (exp_value >= (1 << e)) return sign | ((1u << (nbits - 1)) - 1u);  // saturate
  if (exp_value <= 0) {
    if (exp_value >= 1 - m) return sign | (mant >> (1 - exp_value));   // subnormal of the target
    return sign;
  }
  return sign | ((uint32_t)exp_value << m) | (mant ^ (1u << m));
}

// code of pair position i (0..31) into the unit's plane words (widths = the set bits of B, widest first)
template <int B, int I, int P = 0>
__device__ __forceinline__ void put_code(uint32_t code, uint32_t (&words)[B]) {
  constexpr int pw = plane_width(B, P), per = 16 / pw, h = I >> 1;
  constexpr int lo = plane_lo(B, P), pos = (h % per) * pw + 16 * (I & 1);
  constexpr uint32_t mask = ((1u << pw) - 1u) << pos;
  uint32_t& w = words[plane_word_base(B, P) + h / per];
  w |= (pos >= lo ? code << (pos >= lo ? pos - lo : 0) : code >> (pos < lo ? lo - pos : 0)) & mask;
  if constexpr (P + 1 < plane_count(B)) put_code<B, I, P + 1>(code, words);
}
template <int B, int I, class F>
__device__ __forceinline__ void put_codes(const F& code_of, uint32_t (&words)[B]) {
  put_code<B, I>(code_of(I), words);
  if constexpr (I + 1 < 32) put_codes<B, I + 1>(code_of, words);
}

template <int WT, int B, bool FLOAT>
__global__ void __launch_bounds__(256) quant_pack_kernel(const QuantParams p) {
  // unit index = ((nt * G + g) * 2 + half) * 32 + lane,  lane = r * 4 + j,  g = 128-row group of K
  const long long unit = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (unit >= (long long)p.N * p.K / 32) return;  // whole warps: N * K / 32 is a multiple of 64
  const int lane = (int)(unit & 31), half = (int)((unit >> 5) & 1);
  const long long grp = unit >> 6;
  const int nt = (int)(grp / p.G), g = (int)(grp - (long long)nt * p.G);
  const int r = lane >> 2, j = lane & 3;
  const int n = nt * 16 + half * 8 + r;
  const int k0 = g * 128 + j * 32;
  float v[32];
  load_weights<WT, 32>(p, (size_t)n * p.ldw + k0, v);
  float s;
  if (p.local) {
    float m = 0.f;
#pragma unroll
    for (int i = 0; i < 32; ++i) m = fmaxf(m, fabsf(v[i]));
    if (p.group >= 64) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    if (p.group == 128) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    const unsigned short sb = scale_bits(p, m);
    if ((k0 % p.group) == 0) p.scales[(size_t)(k0 / p.group) * p.N + n] = sb;
    s = p.act == 0 ? __half2float(__ushort_as_half(sb)) : __uint_as_float((uint32_t)sb << 16);
  } else {
    s = load_scale(p, (size_t)(k0 / p.group) * p.N + n);
  }
  uint32_t words[B];
#pragma unroll
  for (int q = 0; q < B; ++q) words[q] = 0u;
  if constexpr (FLOAT) {
    put_codes<B, 0>([&](int i) {
      const float q = fminf(fmaxf(__fdiv_rn(v[i], s), p.minv), p.maxv);
      return encode_float_code(q, B, p.ebits, p.mbits);
    }, words);
  } else {
    // Offset binary code = rint(clamp(w / s)) + offset.  Estimate: x = w * (1 / s) + offset with two
    // roundings, |x - (w / s + offset)| < 2^(B-22); adding 1.5 * 2^23 rounds it to an integer in the low bits.
    constexpr float MAGIC = 12582912.0f;
    constexpr float EPS = (float)(1 << B) * (1.0f / (1 << 22));
    const float offset = p.kind == 1 ? (float)(1 << (B - 1)) : 0.f;
    const float lo = p.minv + offset, hi = p.maxv + offset;
    const float rs = __fdiv_rn(1.0f, s);
    float worst = s < 1e30f ? 0.f : 1.f;  // beyond that the reciprocal loses bits
    put_codes<B, 0>([&](int i) {
      const float x = fminf(fmaxf(fmaf(v[i], rs, offset), lo), hi);
      const float t = x + MAGIC;
      worst = fmaxf(worst, fabsf(x - (t - MAGIC)));
      return __float_as_uint(t);
    }, words);
    if (worst > 0.5f - EPS) {  // some value sits on a rounding boundary: the definition's own division
#pragma unroll
      for (int q = 0; q < B; ++q) words[q] = 0u;
      put_codes<B, 0>([&](int i) {
        const float q = fminf(fmaxf(__fdiv_rn(v[i], s), p.minv), p.maxv);
        return (uint32_t)((int)rintf(q) + (p.kind == 1 ? (1 << (B - 1)) : 0));
      }, words);
    }
  }
  uint32_t* dst = p.bq + (size_t)unit * B;
  if constexpr (B % 4 == 0) {
#pragma unroll
    for (int q = 0; q < B; q += 4)
      *reinterpret_cast<uint4*>(dst + q) = make_uint4(words[q], words[q + 1], words[q + 2], words[q + 3]);
  } else if constexpr (B % 2 == 0) {
#pragma unroll
    for (int q = 0; q < B; q += 2) *reinterpret_cast<uint2*>(dst + q) = make_uint2(words[q], words[q + 1]);
  } else {
#pragma unroll
    for (int q = 0; q < B; ++q) dst[q] = words[q];
  }
}

template <int WT, int B, bool FLOAT>
static cudaError_t pack_launch(const QuantParams& p, int nbits, cudaStream_t stream) {
  if (nbits == B) {
    const long long units = (long long)p.N * p.K / 32;
    quant_pack_kernel<WT, B, FLOAT><<<(unsigned)((units + 255) / 256), 256, 0, stream>>>(p);
    return cudaGetLastError();
  }
  if constexpr (B < 8) return pack_launch<WT, B + 1, FLOAT>(p, nbits, stream);
  else return cudaErrorInvalidValue;
}
template <int WT>
static cudaError_t quantize_as(const QuantParams& p, int nbits, cudaStream_t stream) {
  if (!p.local) {
    const long long warps = (long long)p.N * (p.K / p.group);
    quant_scales_kernel<WT><<<(unsigned)((warps * 32 + 255) / 256), 256, 0, stream>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return p.kind == 2 ? pack_launch<WT, 3, true>(p, nbits, stream) : pack_launch<WT, 1, false>(p, nbits, stream);
}

cudaError_t quantize_launch(const void* w, int w_dtype, int ldw, void* bq, void* scales, int N, int K, int group,
                            int kind, int nbits, int ebits, int mbits, float minv, float maxv, int act,
                            cudaStream_t stream) {
  QuantParams p;
  p.w = w; p.w_dtype = w_dtype; p.ldw = ldw;
  p.bq = reinterpret_cast<uint32_t*>(bq);
  p.scales = reinterpret_cast<unsigned short*>(scales);
  p.act = act;
  p.N = N; p.K = K; p.G = K / 128; p.group = group;
  p.kind = kind; p.ebits = ebits; p.mbits = mbits;
  p.minv = minv; p.maxv = maxv;
  p.vec = (((uintptr_t)w & 15) == 0 && ldw % (w_dtype == 1 ? 4 : 8) == 0) ? 1 : 0;
  p.local = 128 % group == 0 ? 1 : 0;
  if (w_dtype == 1) return quantize_as<1>(p, nbits, stream);
  if (w_dtype == 2) return quantize_as<2>(p, nbits, stream);
  return quantize_as<0>(p, nbits, stream);
}

}  // namespace b200q
