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
// groups get their scales from a pass of their own (quant_scales_kernel; a warp per column and group, 8 weights per lane, left most of its lanes
// waiting: 14336 x 4096 int4 in groups of 256 85 us, with 32 weights per lane and as many lanes as the group needs 60).
//
// What bounds it: HBM (2 or 4 bytes read and b/8 written per weight), provided the arithmetic stays near four
// instructions per weight.  The IEEE division of the definition alone is ten and the float types' encode thirty, so integer codes come
// from one multiplication by the reciprocal of the scale, and only a unit with a value within the multiplication's error of a rounding
// boundary is computed again from correctly rounded quotients (quotient_f2, three instructions for two weights); float codes come from such
// quotients at once (float_codes).  The codes are those of the division in every case; a scale of 1e30 and more, or a NaN among the weights of a
// float type, takes the definition as it stands.  Signed types (signed_codes) need no clamping where the unit's largest weight
// rounds inside the range, work on two values per instruction and pack 2, 4 and 8 bits in fp32.  [28672, 4096], group 128, us (45 at the copy
// rate of HBM, int4), before the quotients / now: fp16 -> int4 67 / 60, int3 78 / 64, float6 304 / 76, float4 320 / 68; bf16 -> int4 88 / 66,
// int3, whose quotients meet the boundaries more often, 109 / 78.  A ring of cp.async stages, 1024 threads per SM, instead of plain loads: int4
// 63, float6 84 (fp32 weights, 14336 x 4096, 55 instead of 63).  2048 threads leave 32 registers: the 16-bit builds of 5 to 8
// bits spill 32 .. 64 bytes to the stack and are still ahead of 1536 threads with 40 and no spills (28672 x 4096: int5 69 / 71 us, int6 67 / 68,
// int7 71 / 72, int8 60 / 61); float types of two planes and more are not (float6 82 / 76).
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
  int gshift;              // log2(group) if local
  int lshift;              // log2 of the lanes that find a group's scale, if not local
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

// ---- two fp32 values at a time (one instruction on sm_100) ----
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack_f2(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpack_f2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma_f2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// max(|a|, |b|, m) of the numbers among them
__device__ __forceinline__ float max_abs_numbers(float a, float b, float m) {
  float r;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(m));
  return r;
}
// max(|a|, |b|, m), NaN if one of them is
__device__ __forceinline__ float max_abs(float a, float b, float m) {
  float r;
  asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(m));
  return r;
}

// The 32 consecutive weights of a unit as they are in memory: 16-bit pairs, or fp32
template <int WT>
struct UnitWeights {
  uint32_t raw[WT == 1 ? 32 : 16];
  __device__ __forceinline__ void load(const QuantParams& p, size_t idx) {
    if (p.vec) {
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(p.w) + idx * (WT == 1 ? 4 : 2));
#pragma unroll
      for (int i = 0; i < (WT == 1 ? 8 : 4); ++i) {
        const uint4 x = __ldg(src + i);
        raw[4 * i] = x.x; raw[4 * i + 1] = x.y; raw[4 * i + 2] = x.z; raw[4 * i + 3] = x.w;
      }
    } else if constexpr (WT == 1) {
#pragma unroll
      for (int i = 0; i < 32; ++i) raw[i] = __ldg(reinterpret_cast<const uint32_t*>(p.w) + idx + i);
    } else {
      const unsigned short* src = reinterpret_cast<const unsigned short*>(p.w) + idx;
#pragma unroll
      for (int i = 0; i < 16; ++i) raw[i] = (uint32_t)__ldg(src + 2 * i) | ((uint32_t)__ldg(src + 2 * i + 1) << 16);
    }
  }
  __device__ __forceinline__ float2 pair(int i) const {
    if constexpr (WT == 0) return __half22float2(h2_from_bits(raw[i]));
    else if constexpr (WT == 2) return make_float2(__uint_as_float(raw[i] << 16), __uint_as_float(raw[i] & 0xffff0000u));
    else return make_float2(__uint_as_float(raw[2 * i]), __uint_as_float(raw[2 * i + 1]));
  }
  __device__ __forceinline__ float operator[](int i) const { return i & 1 ? pair(i >> 1).y : pair(i >> 1).x; }
  // largest magnitude of the numbers among them
  __device__ __forceinline__ float largest() const {
    if constexpr (WT == 0) {
      __half2 m = __habs2(h2_from_bits(raw[0]));
#pragma unroll
      for (int i = 1; i < 16; ++i) m = __hmax2(m, __habs2(h2_from_bits(raw[i])));
      return fmaxf(fmaxf(__low2float(m), __high2float(m)), 0.f);
    } else if constexpr (WT == 2) {
      __nv_bfloat162 m = __habs2(bf2_from_bits(raw[0]));
#pragma unroll
      for (int i = 1; i < 16; ++i) m = __hmax2(m, __habs2(bf2_from_bits(raw[i])));
      return fmaxf(fmaxf(__low2float(m), __high2float(m)), 0.f);
    } else {
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) m = max_abs_numbers(pair(i).x, pair(i).y, m);
      return m;
    }
  }
};

// scales of groups that are not 32, 64 or 128 rows: p.lanes lanes per (column, group), 32 weights each and step
template <int WT>
__global__ void __launch_bounds__(256) quant_scales_kernel(const QuantParams p) {
  const long long id = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> p.lshift;
  const int lane = threadIdx.x & ((1 << p.lshift) - 1), groups = p.K / p.group;
  float m = 0.f;
  int n = 0, g = 0;
  if (id < (long long)p.N * groups) {
    n = (int)(id / groups), g = (int)(id - (long long)n * groups);
    const size_t base = (size_t)n * p.ldw + (size_t)g * p.group;
    for (int i = lane * 32; i < p.group; i += 32 << p.lshift) {
      UnitWeights<WT> v;
      v.load(p, base + i);
      m = fmaxf(m, v.largest());
    }
  }
  for (int o = 1 << p.lshift >> 1; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0 && id < (long long)p.N * groups) p.scales[(size_t)g * p.N + n] = scale_bits(p, m);
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

// Signed codes of a unit without clamping: the caller has made sure that no value rounds beyond the range.  `v`: the weights,
// taken in pairs (even k, odd k), `rs` the scale's reciprocal.  With C = 1.5 * 2^23, t = v * rs + C rounds the quotient to the
// integer i = t - C, and v * rs - i is how far it was from it; returns the largest of those distances.  Types of one plane (2, 4,
// 8 bits) have the codes of a 16-bit field added up in fp32 as well, even and odd k side by side: sum of i * 2^(B f) + 2^(B - 1)
// in every field, an integer below 2^16.  The others have them OR-ed together from the low mantissa bits.
template <int B, int I = 0>
__device__ __forceinline__ void put_pairs(const uint32_t (&code)[32], uint32_t (&words)[B]);
template <int B, class Weights>
__device__ __forceinline__ float signed_codes(const Weights& v, float rs, uint32_t (&words)[B]) {
  constexpr float C = 12582912.0f;
  const f32x2 rs2 = pack_f2(rs, rs), c2 = pack_f2(C, C), minus = pack_f2(-1.f, -1.f);
  float worst = 0.f;
  if constexpr (B == 2 || B == 4 || B == 8) {
    constexpr int PER = 16 / B;  // pairs per word
    constexpr uint32_t HALVES = (1u << (B - 1)) * (B == 2 ? 0x5555u : B == 4 ? 0x1111u : 0x0101u);
    const f32x2 step = pack_f2((float)(1 << B), (float)(1 << B)), end = pack_f2(C + (float)HALVES, C + (float)HALVES);
#pragma unroll
    for (int w = 0; w < B; ++w) {
      f32x2 sum = 0ull;  // minus the sum: what v * rs needs added is -i
#pragma unroll
      for (int f = PER - 1; f >= 0; --f) {
        const float2 xy = v.pair(w * PER + f);
        const f32x2 x = pack_f2(xy.x, xy.y);
        const f32x2 neg = fma_f2(fma_f2(x, rs2, c2), minus, c2);
        const float2 d = unpack_f2(fma_f2(x, rs2, neg));
        worst = max_abs(d.x, d.y, worst);
        sum = f == PER - 1 ? neg : fma_f2(sum, step, neg);
      }
      const float2 t = unpack_f2(fma_f2(sum, minus, end));
      words[w] = __byte_perm(__float_as_uint(t.x), __float_as_uint(t.y), 0x5410);
    }
  } else {
    const f32x2 off = pack_f2(C + (float)(1 << (B - 1)), C + (float)(1 << (B - 1)));
    uint32_t code[32];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 xy = v.pair(i);
      const f32x2 x = pack_f2(xy.x, xy.y), t = fma_f2(x, rs2, off);
      const float2 d = unpack_f2(fma_f2(x, rs2, fma_f2(t, minus, off)));
      worst = max_abs(d.x, d.y, worst);
      const float2 c = unpack_f2(t);
      code[2 * i] = __float_as_uint(c.x);
      code[2 * i + 1] = __float_as_uint(c.y);
    }
#pragma unroll
    for (int q = 0; q < B; ++q) words[q] = 0u;
    put_pairs<B>(code, words);
  }
  return worst;
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

// both codes of pair I and of those behind it (low bits of `code`) into the plane words, two fields at a time
template <int B, int I, int P = 0>
__device__ __forceinline__ void put_pair(uint32_t both, uint32_t (&words)[B]) {
  constexpr int pw = plane_width(B, P), per = 16 / pw;
  constexpr int lo = plane_lo(B, P), pos = (I % per) * pw;
  constexpr uint32_t mask = (((1u << pw) - 1u) << pos) * 0x00010001u;
  uint32_t& w = words[plane_word_base(B, P) + I / per];
  w |= (pos >= lo ? both << (pos >= lo ? pos - lo : 0) : both >> (pos < lo ? lo - pos : 0)) & mask;
  if constexpr (P + 1 < plane_count(B)) put_pair<B, I, P + 1>(both, words);
}
// put_pair of both_of(i) for every pair i of a unit
template <int B, int I = 0, class F>
__device__ __forceinline__ void put_pairs_of(const F& both_of, uint32_t (&words)[B]) {
  put_pair<B, I>(both_of(I), words);
  if constexpr (I + 1 < 16) put_pairs_of<B, I + 1>(both_of, words);
}
template <int B, int I>
__device__ __forceinline__ void put_pairs(const uint32_t (&code)[32], uint32_t (&words)[B]) {
  put_pair<B, I>(__byte_perm(code[2 * I], code[2 * I + 1], 0x5410), words);
  if constexpr (I + 1 < 16) put_pairs<B, I + 1>(code, words);
}

// x / s for a pair, correctly rounded: q = x * rs with rs = rn(1 / s), then q + rn(x - q * s) * rs (Markstein, IBM J. Res. Dev. 34(1), 1990).
// s is a 16-bit scale, 11 significant bits at most: the remainder is exact (q is off by two units at most, so that it has 13 bits), and
// a quotient by s stays 2^-36 of itself away from the midpoint of two fp32 numbers, where the sum is off by 2^-46 before it is rounded.
// For 1e-6 <= s < 1e30; quotients below 2^-80, whose remainder may underflow, have code 0 either way.
// `q` is the first product: it has the sign of the quotient where that is zero, too.
__device__ __forceinline__ f32x2 quotient_f2(float2 x, f32x2 rs, f32x2 minus_s, f32x2& q) {
  const f32x2 v = pack_f2(x.x, x.y);
  q = fma_f2(v, rs, 0x8000000080000000ull);
  return fma_f2(fma_f2(q, minus_s, v), rs, q);
}

// Codes of a unit of a float type (E exponent bits, M mantissa bits) without clamping; returns the largest quotient, NaN if one is.
// encode_float_code rounds to M + 1 significant bits and then cuts off what the type's subnormals lack: here the first is
// (q + c) - c with c = 1.5 * 2^(23 - M) times q's power of two, the second a product with 2^(bias - 127), after which exponent and
// mantissa stand in fp32's fields as in the code (subnormal where the code is).
template <int B, class Weights>
__device__ __forceinline__ float float_codes(const QuantParams& p, const Weights& v, float s, float rs, uint32_t (&words)[B]) {
  const f32x2 rs2 = pack_f2(rs, rs), ms2 = pack_f2(-s, -s);
  const float c = 1.5f * (float)(1 << (23 - p.mbits)), bias = __uint_as_float(p.ebits == 1 ? 1u << 22 : ((1u << (p.ebits - 1)) - 1u) << 23);
  const f32x2 c2 = pack_f2(c, c), mc2 = pack_f2(-c, -c), b2 = pack_f2(bias, bias);
  const uint32_t mags = ((1u << (B - 1)) - 1u) * 0x00010001u;
  float top = 0.f;
#pragma unroll
  for (int q = 0; q < B; ++q) words[q] = 0u;
  put_pairs_of<B>([&](int i) {
    f32x2 q0;
    const f32x2 q = quotient_f2(v.pair(i), rs2, ms2, q0);
    const float2 qf = unpack_f2(q), sf = unpack_f2(q0);
    top = max_abs(qf.x, qf.y, top);
    const f32x2 e = q & 0x7f8000007f800000ull;
    const float2 r = unpack_f2(fma_f2(fma_f2(e, mc2, fma_f2(e, c2, q)), b2, 0x8000000080000000ull));
    const uint32_t w = __byte_perm(__float_as_uint(r.x), __float_as_uint(r.y), 0x7632);
    const uint32_t signs = __byte_perm(__float_as_uint(sf.x), __float_as_uint(sf.y), 0x7632);
    return ((w >> (7 - p.mbits)) & mags) | ((signs >> (16 - B)) & ((1u << (B - 1)) * 0x00010001u));
  }, words);
  return top;
}

template <int WT, int B, bool FLOAT>
__global__ void __launch_bounds__(256, WT == 1 ? 4 : FLOAT && plane_count(B) > 1 ? 6 : 8) quant_pack_kernel(const QuantParams p) {
  // unit index = ((nt * G + g) * 2 + half) * 32 + lane,  lane = r * 4 + j,  g = 128-row group of K.  A block has four groups,
  // of one 16-column tile where G allows it (a 64-bit division per thread costs as much as a quarter of its weights).
  const int lane = threadIdx.x & 31, half = (threadIdx.x >> 5) & 1;
  const unsigned grp = blockIdx.x * 4 + (threadIdx.x >> 6);
  int nt;
  if ((p.G & 3) == 0) {
    nt = (int)(blockIdx.x / ((unsigned)p.G >> 2));
  } else {
    nt = (int)(grp / (unsigned)p.G);
    if (nt >= p.N >> 4) return;  // whole warps
  }
  const int g = (int)(grp - (unsigned)nt * p.G);
  const long long unit = (long long)grp * 64 + (threadIdx.x & 63);
  const int r = lane >> 2, j = lane & 3;
  const int n = nt * 16 + half * 8 + r;
  const int k0 = g * 128 + j * 32;
  UnitWeights<WT> v;
  v.load(p, (size_t)n * p.ldw + k0);
  const float unit_max = v.largest();
  float s;
  if (p.local) {
    float m = unit_max;
    if (p.group >= 64) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    if (p.group == 128) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    const unsigned short sb = scale_bits(p, m);
    if ((k0 & (p.group - 1)) == 0) p.scales[(size_t)(k0 >> p.gshift) * p.N + n] = sb;
    s = p.act == 0 ? __half2float(__ushort_as_half(sb)) : __uint_as_float((uint32_t)sb << 16);
  } else {
    s = load_scale(p, (size_t)(k0 / p.group) * p.N + n);
  }
  uint32_t words[B];
#pragma unroll
  for (int q = 0; q < B; ++q) words[q] = 0u;
  const float rs = __fdiv_rn(1.0f, s);
  const bool plain = s < 1e30f;
  bool done = false;
  if constexpr (FLOAT) {
    // a largest quotient that rounds to the type's largest number needs no clamping
    if (plain) done = float_codes<B>(p, v, s, rs, words) <= p.maxv + p.maxv * __uint_as_float((124u - p.mbits) << 23);
  } else {
    // Signed types whose largest weight of the unit rounds inside the range: no clamping, see signed_codes.  A unit with a
    // value within the products' error of a rounding boundary, or a NaN, takes the quotients below.
    constexpr float EPS = (float)(1 << B) * (1.0f / (1 << 22)), MAGIC = 12582912.0f;
    if (p.kind == 1 && plain && unit_max * rs <= p.maxv + (0.5f - EPS)) {
      done = signed_codes<B>(v, rs, words) <= 0.5f - EPS;
    } else if (p.kind == 0 && plain) {
      // Unsigned types: code = rint(clamp(w / s)).  Estimate: x = w * (1 / s), |x - w / s| < 2^(B-22); adding 1.5 * 2^23
      // rounds it to an integer in the low bits.
      float worst = 0.f;
      put_codes<B, 0>([&](int i) {
        const float x = fminf(fmaxf(v[i] * rs, p.minv), p.maxv);
        const float t = x + MAGIC;
        worst = fmaxf(worst, fabsf(x - (t - MAGIC)));
        return __float_as_uint(t);
      }, words);
      done = worst <= 0.5f - EPS;
    }
    if (!done && plain) {
      const f32x2 rs2 = pack_f2(rs, rs), ms2 = pack_f2(-s, -s);
      const float off = MAGIC + (p.kind == 1 ? (float)(1 << (B - 1)) : 0.f);
#pragma unroll
      for (int q = 0; q < B; ++q) words[q] = 0u;
      put_pairs_of<B>([&](int i) {
        f32x2 q0;
        const float2 q = unpack_f2(quotient_f2(v.pair(i), rs2, ms2, q0));
        return __byte_perm(__float_as_uint(fminf(fmaxf(q.x, p.minv), p.maxv) + off), __float_as_uint(fminf(fmaxf(q.y, p.minv), p.maxv) + off), 0x5410);
      }, words);
      done = true;
    }
  }
  if (!done) {  // the definition as it stands
#pragma unroll
    for (int q = 0; q < B; ++q) words[q] = 0u;
    put_codes<B, 0>([&](int i) {
      const float q = fminf(fmaxf(__fdiv_rn(v[i], s), p.minv), p.maxv);
      return FLOAT ? encode_float_code(q, B, p.ebits, p.mbits) : (uint32_t)((int)rintf(q) + (p.kind == 1 ? (1 << (B - 1)) : 0));
    }, words);
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
    quant_pack_kernel<WT, B, FLOAT><<<(unsigned)(((long long)(p.N / 16) * p.G + 3) / 4), 256, 0, stream>>>(p);
    return cudaGetLastError();
  }
  if constexpr (B < 8) return pack_launch<WT, B + 1, FLOAT>(p, nbits, stream);
  else return cudaErrorInvalidValue;
}
template <int WT>
static cudaError_t quantize_as(const QuantParams& p, int nbits, cudaStream_t stream) {
  if (!p.local) {
    const long long threads = ((long long)p.N * (p.K / p.group)) << p.lshift;
    quant_scales_kernel<WT><<<(unsigned)((threads + 255) / 256), 256, 0, stream>>>(p);
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
  p.gshift = group == 32 ? 5 : group == 64 ? 6 : 7;
  for (p.lshift = 0; p.lshift < 5 && 32 << p.lshift < group;) ++p.lshift;  // a lane has 32 rows or more, a group up to a warp
  if (w_dtype == 1) return quantize_as<1>(p, nbits, stream);
  if (w_dtype == 2) return quantize_as<2>(p, nbits, stream);
  return quantize_as<0>(p, nbits, stream);
}

}  // namespace b200q
