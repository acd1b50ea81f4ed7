// Decode batches of up to 16 rows with the activations in registers: C[M, N] = A[M, K] x dequant(Bq[K, N]).
//
// What bounds it: HBM, and around a launch 3 us of start, activations and end.  In stream_kernel.cu a warp reads the
// activations of each 128-row group from shared memory, 2 KB for every 1 KB of 4-bit weights: 32 of the 45 cycles that HBM leaves
// an SM per 16 x 128 group went to shared memory, and every CTA staged and converted the activations before its first product.
// Here K is split over the warps of a CTA instead of the column tiles: a warp owns up to four 128-row groups of K and loads
// their activations once, as tensor-core operands (the operand's k order is the packed layout's: lane (r, j) holds 64 contiguous
// bytes of row r per group), and then takes the CTA's column tiles one after the other.  Shared memory carries the weights only,
// and nothing is staged.  us, cold chains, 4 bits, group 128, before (stream or exact kernel) / here: 8 x 4096 x 4096 7.1 / 4.7, 8 x
// 28672 x 4096 19.8 / 13.3, 8 x 4096 x 14336 13.1 / 9.8, 1 x 4096 x 4096 4.6 / 3.6, 1 x 28672 x 4096 13.7 / 12.3; 16 x 4096 x 4096
// 8.2 / 7.1, but 16 x 28672 x 4096 20.3 / 20.6 (two sets of sums per warp: 185 instructions per group, 121 with one).
//
// Weights.  One elected thread of a warp keeps the warp's ring full with TMA bulk copies, as in stream_kernel.cu: slots of one, two or
// four groups of a column tile, about 64 KB per CTA (three slots of 2 KB instead of two: no gain).  All loads of a slot come first, then the
// request for the next one, then the products (loads group by group: 28672 x 4096 14.0 us, 13.6 so).
//
// Products.  mma.sync.m16n8k16, 16 columns of weights against 8 rows of activations: 8 cycles per SM quadrant, so that one
// group costs 16 of the SM's 45 cycles.  An integer code sits in the mantissa of an fp16 subnormal at one of two places (res_target), an
// accumulator each, whose sums are added with the factor between the places: the activations are multiplied as they are (the
// stream kernel multiplies them by 2^-T beforehand, which costs those below 2^(T-14) low bits), for half of the shifts of a single place.
// The zero point: both accumulators start from a quarter of -zero_point * sum(a), and the other half is added behind the group's
// products, so that sums of activations with a mean stay around zero on the way (the sums over a come from eight MMAs per group with a
// constant operand, once per launch).  For 7 and 8 bits that is not enough: their running sums still reach a quarter of (zero point) * sum(a),
// and activations around 3 at 5 to 16 rows left twice as many results off the nearest value as exact_kernel.cu does (0.20 and 0.55 %, there
// 0.09 and 0.30).  8 bits are multiplied as code - zero_point instead, a byte permute and a half subtraction per pair (0.05 .. 0.08 %; us, as a
// subnormal / so: 8 x 4096 x 4096 5.60 / 5.77, 8 x 28672 x 4096 21.0 / 21.1, 16 x 4096 x 2048 5.44 / 5.16); 7 bits, whose codes take six
// instructions per pair already (28672 x 4096 25.7 us, so 29.2), have the zero point taken off by an MMA behind each 16 rows, as in the exact
// kernel (27.2; 0.08 %).  Per group the sums are multiplied by the scale in fp32: no weight is rounded.
//
// Sums.  The 16 warps' parts of a column tile meet in shared memory (four tiles of room, an mbarrier that counts the warps and one
// that frees the room), and one of the warps, in turn, adds them up in order and writes C: results repeat bit for bit.  Where the
// activations of up to 8 rows of A do not fit the registers - more than 8192 rows of K - or where it pays, a cluster of S CTAs
// shares K (9 to 16 rows stop at 4096 rows of K).  The warp that adds up a tile sends the CTA's sum to the CTA that writes the tile (every S-th), which waits for the bytes
// it expects at the end: no CTA reads another's memory, so none has to wait for the others before it leaves.
//
// Every wait is bounded; one that runs out leaves the loops, waits (bounded) for the copies in flight and is reported in the workspace's
// status word.
#include "common.cuh"

#ifndef B200Q_PART
#define B200Q_PART 0
#endif
#ifndef B200Q_NPARTS
#define B200Q_NPARTS 1
#endif

namespace b200q {

// ---- where the codes of a pair sit in the operand's mantissa: two places per width, half of the pairs each ----
// (Places that need the fewest shifts.  Of those 1 and 2 bits take the highest: the tensor core keeps a subnormal's leading zeros, so that a
// code at bit 0 costs the sums ten bits.  Error beyond the rounding of the results, rms of the results, 4096 to 14336 rows of K, 1 to 4 / 5 to 16
// rows: 2 bits at 0 and 2 2.6e-6 / 2.2e-6, at 6 and 8 7e-8 / 1.1e-7; the stream / exact kernel 1.5e-6 / 2.1e-6.  8 bits at 2 instead of 0:
// no difference, 1 % slower.  5 and 6 bits from one and two places up: 0.30 and 0.17 % of the results off the nearest value, from here 0.14 and
// 0.09, for two shifts per unit.  A pair's products carry the factor 2^T, one accumulator per place.)
B200Q_HD constexpr int res_class(int b, int h) {
  return b == 2 ? ~h & 1 : b == 3 || b == 7 ? (h >> 1) & 1 : b == 5 ? (h ^ (h >> 2)) & 1 : h & 1;
}
B200Q_HD constexpr int res_target(int b, int cls) {
  switch (b) {
    case 1: return 8 + cls;
    case 2: return 6 + 2 * cls;
    case 6: return 4 - 2 * cls;
    case 3: case 7: return 1 + 2 * cls;
    case 4: return 4 * cls;
    case 5: return 1 + 4 * cls;
    default: return 0;
  }
}
// the i-th pair of a class, i = 0 .. 7
B200Q_HD constexpr int res_pair(int b, int cls, int i) {
  int n = 0;
  for (int h = 0; h < 16; ++h)
    if (res_class(b, h) == cls && n++ == i) return h;
  return 0;
}
// types whose operand is the value code - zero_point, and those whose zero point has MMAs of its own
B200Q_HD constexpr bool res_by_value(int v) { return !var_is_float(v) && var_bits(v) == 8 && var_bias(v) != 0; }
B200Q_HD constexpr bool res_zero_mma(int v) { return !var_is_float(v) && var_bits(v) == 7 && var_bias(v) != 0; }
template <int VAR, int H>
__device__ __forceinline__ uint32_t res_operand(const uint32_t* w) {
  constexpr int B = var_bits(VAR);
  if constexpr (var_is_float(VAR)) return pair_raw<VAR, H>(w);
  else if constexpr (res_by_value(VAR)) {
    const uint32_t code = __byte_perm(w[H >> 1], 0x64646464u, H & 1 ? 0x4341u : 0x4240u);  // 1024 + code
    return bits_from_h2(__hsub2(h2_from_bits(code), h2_from_bits(dup16(half_bits_of_uint(1024u + var_bias(VAR))))));
  } else {
    constexpr int T = res_target(B, res_class(B, H));
    if constexpr (lin_uniform_inverted(VAR)) return gather_pair<B, H, T>(w, 0u) ^ (0x00010001u << T);
    else return gather_pair<B, H, T>(w, 0u);
  }
}

template <int ACT>
__device__ __forceinline__ unsigned short res_out_bits(float v) {
  if constexpr (ACT == 0) return __half_as_ushort(__float2half_rn(v));
  else return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}
template <int ACT>
__device__ __forceinline__ float res_scale(unsigned short bits) {
  if constexpr (ACT == 0) return __half2float(__ushort_as_half(bits));
  else return __uint_as_float((uint32_t)bits << 16);
}
// two bf16 values as fp16: exact inside fp16's range, larger magnitudes saturate, those below 2^-24 vanish, NaN stays
__device__ __forceinline__ uint32_t res_bf16x2_to_f16x2(uint32_t w) {
  uint32_t h;
  asm("cvt.rn.satfinite.f16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(__uint_as_float(w & 0xffff0000u)), "f"(__uint_as_float(w << 16)));
  return h;
}
// 16 bytes of an activation row, or zeros where there is no row.  In program order, so that all of a warp's loads are in flight at once:
// left to the compiler, some waited for the first conversions (8 x 6144 x 4096 5.55 us, 5.49 so).  Not ld.global.nc: the rows are
// written while this launch is on its SM already, and a non-coherent load may return a line that L1 has had since before.
__device__ __forceinline__ uint4 res_load_row(const uint4* p, bool valid) {
  uint4 v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
               "@p ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n\t}"
               : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w) : "l"(p), "r"((uint32_t)valid));
  return v;
}
// the words of a unit, and one word of every vector load
template <int B>
__device__ __forceinline__ uint32_t res_unit(const unsigned char* ptr, uint32_t (&w)[B]) {
  if constexpr (B % 4 == 0) {
    uint32_t x = 0u;
#pragma unroll
    for (int q = 0; q < B / 4; ++q) {
      const uint4 v = reinterpret_cast<const uint4*>(ptr)[q];
      w[4 * q] = v.x; w[4 * q + 1] = v.y; w[4 * q + 2] = v.z; w[4 * q + 3] = v.w;
      x |= v.x;
    }
    return x;
  } else if constexpr (B % 2 == 0) {
    uint32_t x = 0u;
#pragma unroll
    for (int q = 0; q < B / 2; ++q) {
      const uint2 v = reinterpret_cast<const uint2*>(ptr)[q];
      w[2 * q] = v.x; w[2 * q + 1] = v.y;
      x |= v.x;
    }
    return x;
  } else {
    uint32_t x = 0u;
#pragma unroll
    for (int q = 0; q < B; ++q) { w[q] = reinterpret_cast<const uint32_t*>(ptr)[q]; x |= w[q]; }
    return x;
  }
}

__device__ __forceinline__ unsigned long long f2_pack(float x, float y) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
__device__ __forceinline__ void f2_unpack(unsigned long long v, float& x, float& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long f2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// d = a * b + c with c in registers of its own
__device__ __forceinline__ void mma_m16n8k16_from(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                                  uint32_t b1, float c0, float c1, float c2, float c3) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// Shared memory: barriers of the rings [warp][8] and of the slabs [set][full 4, empty 4]; rings [warp][slot]; scales
// [warp][tile][NG][16]; slabs [set][slot][warp][MT][32 lanes] float4; with a cluster the CTA's sums [tile][MT][32 lanes] float4.
// Columns of `af`, `nb`: rows of A come in sets of eight (MT of them), 128-row groups of K in NG.
template <int VAR, int MT, int NG, int ACT, bool CLUSTER>
__global__ void __launch_bounds__(RES_WARPS * 32, 1) resident_kernel(const ResidentParams p) {
  constexpr int B = var_bits(VAR);
  constexpr bool ZERO_MMA = res_zero_mma(VAR);
  constexpr int BIAS = res_by_value(VAR) || ZERO_MMA ? 0 : lin_uniform_bias(VAR);  // the zero point of the accumulators' start
  constexpr int GI = res_gi(B, NG);
  constexpr int IPT = NG / GI;             // slots per column tile
  constexpr uint32_t GROUP = 256u * B, SLOT = GI * GROUP;
  constexpr int T0 = var_is_float(VAR) ? 0 : res_target(B, 0), T1 = var_is_float(VAR) ? 0 : res_target(B, 1);
  constexpr uint32_t ZP0 = (0x8000u | (uint32_t)(var_bias(VAR) << T0)) * 0x00010001u, ZP1 = (0x8000u | (uint32_t)(var_bias(VAR) << T1)) * 0x00010001u;
  constexpr int FL = res_by_value(VAR) ? 0 : lin_factor_log2(VAR) - T0;
  constexpr float F = (lin_uniform_inverted(VAR) ? -1.0f : 1.0f) * (float)(1u << FL);
  constexpr int NBQ = MT * NG <= 2 ? 4 : 2;  // registers of a zero-point term: as the accumulators have it, or once
  constexpr float R10 = (float)(1 << T1) / (float)(1 << T0), R01 = 1.0f / R10;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t smem_base = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int r = lane >> 2, j = lane & 3;
  const int NST = p.stages, WK = 1 << p.wk_shift, WT = RES_WARPS >> p.wk_shift;
  const int set = warp >> p.wk_shift, wi = warp & (WK - 1);

  int ci = blockIdx.x, chunk = 0;
  if constexpr (CLUSTER) { ci = blockIdx.x / p.S; chunk = blockIdx.x - ci * p.S; }
  const int gc0 = CLUSTER ? p.G * chunk / p.S : 0, gc1 = CLUSTER ? p.G * (chunk + 1) / p.S : p.G;
  const int Gc = gc1 - gc0, base = Gc >> p.wk_shift, rem = Gc & (WK - 1);
  const int n = base + (wi < rem ? 1 : 0), g0 = gc0 + wi * base + min(wi, rem);  // this warp's groups of K
  const int active = min(WK, Gc);                                                 // warps of a set that have any
  const int tile0 = ci * p.T_own, tiles = min(p.T_own, p.NT - tile0);
  const int my = n > 0 && tiles > set ? (tiles - set + WT - 1) >> (4 - p.wk_shift) : 0;  // tiles of this set

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // ---- shared memory ----
  const uint32_t bar0 = smem_base + (uint32_t)warp * 64u;
  const uint32_t full0 = smem_base + 1024u + (uint32_t)set * 64u, empty0 = full0 + 32u;  // [slab slot]
  const uint32_t ring_off = RES_HEADER + (uint32_t)(warp * NST) * SLOT, ring_s = smem_base + ring_off;
  const uint32_t sc_off = RES_HEADER + (uint32_t)(RES_WARPS * NST) * SLOT;
  const int Tw = (p.T_own + WT - 1) >> (4 - p.wk_shift);
  unsigned char* sc_warp = smem_raw + sc_off + (size_t)warp * NG * Tw * 32;
  const uint32_t slab_off = sc_off + (uint32_t)(RES_WARPS * NG * Tw * 32);
  const int D = 1 << p.slab_shift;
  float4* slab = reinterpret_cast<float4*>(smem_raw + slab_off) + (size_t)set * D * WK * MT * 32;
  const uint32_t got_off = slab_off + (uint32_t)(WT * D * WK * MT * 512), got_bar = smem_base + RES_HEADER - 8u;  // cluster: see finish

  // ---- scales of all of the warp's tiles and groups: [tile][group][16]; requested first, as the products wait for them
  // longest (1 x 4096 x 4096, behind the rings' set-up 3.85 us, here 3.63; behind the activations' loads 4.4) ----
  {
    const unsigned char* srow = reinterpret_cast<const unsigned char*>(p.scales) + (size_t)(unsigned)(tile0 + set) * 32u + (lane & 1) * 16;
    const uint32_t row_bytes = (uint32_t)p.N * 2u, dst0 = smem_base + (uint32_t)(sc_warp - smem_raw) + (lane & 1) * 16;
#pragma unroll
    for (int gi = 0; gi < NG; ++gi) {
      if (gi >= n) break;
      const uint32_t row = p.gshift >= 0 ? (uint32_t)(g0 + gi) >> p.gshift : (uint32_t)(g0 + gi) / (uint32_t)p.gdiv;
      const unsigned char* src_row = srow + (size_t)row * row_bytes;
      for (int x = lane >> 1; x < my; x += 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst0 + (uint32_t)((x * NG + gi) * 32)), "l"(src_row + ((uint32_t)x * 32u << (4 - p.wk_shift))) : "memory");
    }
  }

  // ---- weights: the warp's own ring ----
  const int ipt = (n + GI - 1) / GI, n_items = my * ipt;
  const uint32_t last_bytes = (uint32_t)(n - (ipt - 1) * GI) * GROUP;
  const unsigned char* src = reinterpret_cast<const unsigned char*>(p.bq) + ((size_t)(tile0 + set) * p.G + g0) * GROUP;
  const size_t tile_skip = (size_t)WT * p.G * GROUP - (size_t)(ipt - 1) * SLOT;
  int issued = 0, pq = 0;
  auto issue_next = [&](uint32_t bar, uint32_t dst) {
    const bool last = IPT == 1 || pq == ipt - 1;
    const uint32_t bytes = last ? last_bytes : SLOT;
    if (elect_one()) {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
          "r"(bytes), "r"(bar)
          : "memory");
    }
    ++issued;
    if (last) { src += tile_skip; pq = 0; } else { src += SLOT; ++pq; }
  };
  if (lane < NST) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar0 + lane * 8) : "memory");
  if (wi == 0 && lane < 4) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full0 + lane * 8), "r"(active) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + lane * 8) : "memory");
  }
  if (CLUSTER && tid == 0) {
    // what the cluster's CTAs send for the tiles that this one writes (every S-th)
    const uint32_t bytes = (uint32_t)((max(tiles, 0) - chunk + p.S - 1) / p.S * p.S * MT) * 512u;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(got_bar) : "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(got_bar), "r"(bytes) : "memory");
  }
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncwarp();
  if constexpr (CLUSTER) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  for (int s = 0; s < NST && issued < n_items; ++s) issue_next(bar0 + s * 8, ring_s + s * SLOT);

  asm volatile("griddepcontrol.wait;" ::: "memory");

  // ---- activations: operand fragments of the warp's groups, kept for all column tiles ----
  uint32_t af[NG][MT][16];
#pragma unroll
  for (int g = 0; g < NG; ++g)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const bool valid = g < n && mt * 8 + r < p.M;
      const uint4* pa = reinterpret_cast<const uint4*>(reinterpret_cast<const unsigned short*>(p.a) +
                                                       (size_t)(mt * 8 + r) * p.lda + (size_t)(g0 + g) * 128 + j * 32);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 v = res_load_row(pa + q, valid);
        af[g][mt][4 * q] = v.x; af[g][mt][4 * q + 1] = v.y; af[g][mt][4 * q + 2] = v.z; af[g][mt][4 * q + 3] = v.w;
      }
    }
  // a quarter of the zero-point term of every group and row, in the accumulators' unit (row 2j, 2j + 1 of each 8)
  float nb[BIAS != 0 ? NG : 1][BIAS != 0 ? MT : 1][NBQ];
#pragma unroll
  for (int g = 0; g < NG; ++g)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      if constexpr (ACT == 1) {
#pragma unroll
        for (int q = 0; q < 16; ++q) af[g][mt][q] = res_bf16x2_to_f16x2(af[g][mt][q]);
      }
      if constexpr (BIAS != 0) {
        float d[4];
        constexpr uint32_t ONE = 0x3c003c00u;
        mma_m16n8k16_init(d, ONE, ONE, ONE, ONE, af[g][mt][0], af[g][mt][1]);
#pragma unroll
        for (int q = 2; q < 16; q += 2) mma_m16n8k16(d, ONE, ONE, ONE, ONE, af[g][mt][q], af[g][mt][q + 1]);
        constexpr float Q = -0.25f * (float)BIAS / (float)(1u << FL);
#pragma unroll
        for (int q = 0; q < NBQ; ++q) nb[g][mt][q] = d[q] * Q;
      }
    }
  asm volatile("cp.async.wait_all;" ::: "memory");
  if constexpr (CLUSTER) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");  // everybody's barriers are there
  else __syncthreads();

  // ---- column tiles ----
  bool ok = true;
  int next_read = wi;
  auto finish = [&](int ti) {  // adds up the warps' sums of tile ti of this set
    const uint32_t bar = full0 + (uint32_t)(ti & (D - 1)) * 8u;
    // (a warp gives up as a whole: lanes that left alone would miss the others at the next vote)
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar, (uint32_t)(ti >> p.slab_shift) & 1u) ? 1 : 0)) { ok = false; return; }
    const float4* s = slab + (size_t)(ti & (D - 1)) * WK * MT * 32 + lane;
    const int tile = set + ti * WT;
    float4 v[MT];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) v[mt] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int w = 0; w < active; ++w)
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const float4 x = s[(w * MT + mt) * 32];
        v[mt].x += x.x; v[mt].y += x.y; v[mt].z += x.z; v[mt].w += x.w;
      }
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty0 + (uint32_t)(ti & (D - 1)) * 8u) : "memory");
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      v[mt].x *= F; v[mt].y *= F; v[mt].z *= F; v[mt].w *= F;
      if constexpr (CLUSTER) {  // to the CTA that writes the tile: [its tile][CTA][MT][32 lanes]
        const int owner = tile % p.S;
        uint32_t dst, bar;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst)
                     : "r"(smem_base + got_off + (uint32_t)(((tile - owner + chunk) * MT + mt) * 512 + lane * 16)), "r"(owner));
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(bar) : "r"(got_bar), "r"(owner));
        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst), "f"(v[mt].x),
                     "f"(v[mt].y), "f"(v[mt].z), "f"(v[mt].w), "r"(bar)
                     : "memory");
      } else {
        const int m = mt * 8 + 2 * j, col = (tile0 + tile) * 16 + r;
        unsigned short* c = reinterpret_cast<unsigned short*>(p.c) + (size_t)m * p.ldc + col;
        if (m < p.M) { c[0] = res_out_bits<ACT>(v[mt].x); c[8] = res_out_bits<ACT>(v[mt].z); }
        if (m + 1 < p.M) { c[p.ldc] = res_out_bits<ACT>(v[mt].y); c[p.ldc + 8] = res_out_bits<ACT>(v[mt].w); }
      }
    }
  };
  uint32_t slot_off = 0, bar = bar0, parity = 0;
  const unsigned char* ring_g = smem_raw + ring_off;
  const uint32_t w_lane = (uint32_t)(lane * B * 4);
  const unsigned short* sc_lane = reinterpret_cast<const unsigned short*>(sc_warp) + r;
  for (int ti = 0; ti < my && ok; ++ti, sc_lane += NG * 16) {
    unsigned long long acc[MT][2];  // rows 2j, 2j + 1 of columns r and r + 8
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) acc[mt][0] = acc[mt][1] = 0ull;
#pragma unroll
    for (int q = 0; q < IPT; ++q) {
      if (q * GI >= n) break;
      if (!__all_sync(0xffffffffu, mbar_test(bar, parity) ? 1 : 0)) {
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity) ? 1 : 0)) { ok = false; break; }
      }
      const unsigned char* slot = ring_g + slot_off;
      uint32_t loaded = 0u, w0[GI][B], w1[GI][B];
#pragma unroll
      for (int gi = 0; gi < GI; ++gi) {
        loaded |= res_unit<B>(slot + w_lane + gi * GROUP, w0[gi]);
        loaded |= res_unit<B>(slot + w_lane + gi * GROUP + GROUP / 2, w1[gi]);
      }
      __syncwarp();
      if (issued < n_items) issue_next(bar, ring_s + slot_off + (loaded & p.zero));
#pragma unroll
      for (int gi = 0; gi < GI; ++gi) {
        const int g = q * GI + gi;
        if (gi > 0 && g >= n) break;
        const float sf0 = res_scale<ACT>(sc_lane[g * 16]), sf1 = res_scale<ACT>(sc_lane[g * 16 + 8]);
        float d0[MT][4], d1[MT][4];
        unsigned long long z0[MT], z1[MT];
        if constexpr (BIAS != 0) {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            z0[mt] = f2_pack(nb[g][mt][0], nb[g][mt][1]);
            z1[mt] = NBQ == 4 ? f2_pack(nb[g][mt][NBQ - 2], nb[g][mt][NBQ - 1]) : z0[mt];
          }
        }
#define RES_STEP(I)                                                                                                  \
  {                                                                                                                  \
    constexpr int H0 = res_pair(B, 0, 2 * I), H1 = res_pair(B, 0, 2 * I + 1), H2 = res_pair(B, 1, 2 * I),            \
                  H3 = res_pair(B, 1, 2 * I + 1);                                                                    \
    const uint32_t x0 = res_operand<VAR, H0>(w0[gi]), x1 = res_operand<VAR, H0>(w1[gi]), x2 = res_operand<VAR, H1>(w0[gi]),      \
                   x3 = res_operand<VAR, H1>(w1[gi]);                                                                    \
    const uint32_t y0 = res_operand<VAR, H2>(w0[gi]), y1 = res_operand<VAR, H2>(w1[gi]), y2 = res_operand<VAR, H3>(w0[gi]),      \
                   y3 = res_operand<VAR, H3>(w1[gi]);                                                                    \
    _Pragma("unroll") for (int mt = 0; mt < MT; ++mt) {                                                              \
      if constexpr (I > 0) {                                                                                         \
        mma_m16n8k16(d0[mt], x0, x1, x2, x3, af[g][mt][H0], af[g][mt][H1]);                                          \
        mma_m16n8k16(d1[mt], y0, y1, y2, y3, af[g][mt][H2], af[g][mt][H3]);                                          \
      } else if constexpr (BIAS == 0) {                                                                              \
        mma_m16n8k16_init(d0[mt], x0, x1, x2, x3, af[g][mt][H0], af[g][mt][H1]);                                     \
        mma_m16n8k16_init(d1[mt], y0, y1, y2, y3, af[g][mt][H2], af[g][mt][H3]);                                     \
      } else {                                                                                                       \
        float c0, c1, c2, c3, e0, e1, e2, e3;                                                                        \
        f2_unpack(z0[mt], c0, c1); f2_unpack(z1[mt], c2, c3);                                                        \
        mma_m16n8k16_from(d0[mt], x0, x1, x2, x3, af[g][mt][H0], af[g][mt][H1], c0, c1, c2, c3);                     \
        f2_unpack(T1 != T0 ? f2_mul(z0[mt], f2_pack(R10, R10)) : z0[mt], e0, e1);                                    \
        f2_unpack(T1 != T0 ? f2_mul(z1[mt], f2_pack(R10, R10)) : z1[mt], e2, e3);                                    \
        mma_m16n8k16_from(d1[mt], y0, y1, y2, y3, af[g][mt][H2], af[g][mt][H3], e0, e1, e2, e3);                     \
      }                                                                                                              \
      if constexpr (ZERO_MMA) {                                                                                      \
        mma_m16n8k16(d0[mt], ZP0, ZP0, ZP0, ZP0, af[g][mt][H0], af[g][mt][H1]);                                      \
        mma_m16n8k16(d1[mt], ZP1, ZP1, ZP1, ZP1, af[g][mt][H2], af[g][mt][H3]);                                      \
      }                                                                                                              \
    }                                                                                                                \
  }
        RES_STEP(0) RES_STEP(1) RES_STEP(2) RES_STEP(3)
#undef RES_STEP
        const unsigned long long s0 = f2_pack(sf0, sf0), s1 = f2_pack(sf1, sf1), r01 = f2_pack(R01, R01), two = f2_pack(2.f, 2.f);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const unsigned long long lo0 = f2_pack(d0[mt][0], d0[mt][1]), hi0 = f2_pack(d0[mt][2], d0[mt][3]);
          const unsigned long long lo1 = f2_pack(d1[mt][0], d1[mt][1]), hi1 = f2_pack(d1[mt][2], d1[mt][3]);
          unsigned long long lo = T1 != T0 ? f2_fma(lo1, r01, lo0) : f2_add(lo1, lo0);
          unsigned long long hi = T1 != T0 ? f2_fma(hi1, r01, hi0) : f2_add(hi1, hi0);
          if constexpr (BIAS != 0) { lo = f2_fma(z0[mt], two, lo); hi = f2_fma(z1[mt], two, hi); }
          acc[mt][0] = f2_fma(s0, lo, acc[mt][0]);
          acc[mt][1] = f2_fma(s1, hi, acc[mt][1]);
        }
      }
      slot_off += SLOT; bar += 8;
      if (slot_off == (uint32_t)NST * SLOT) { slot_off = 0; bar = bar0; parity ^= 1u; }
    }
    if (!ok) break;
    const int sl = ti & (D - 1);
    if (ti >= D &&
        !__all_sync(0xffffffffu, mbar_wait_bounded(empty0 + (uint32_t)sl * 8u, (uint32_t)((ti >> p.slab_shift) - 1) & 1u) ? 1 : 0)) { ok = false; break; }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
    {
      float4 v;
      f2_unpack(acc[mt][0], v.x, v.y);
      f2_unpack(acc[mt][1], v.z, v.w);
      slab[(sl * WK + wi) * MT * 32 + mt * 32 + lane] = v;
    }
    __syncwarp();
    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(full0 + (uint32_t)sl * 8u) : "memory");
    if (ti > 0 && ti - 1 == next_read) { finish(ti - 1); next_read += active; }
  }
  ok = __all_sync(0xffffffffu, ok ? 1 : 0);
  if (ok && my > 0 && next_read == my - 1) finish(my - 1);
  if (!__all_sync(0xffffffffu, ok ? 1 : 0)) {
    if (lane == 0) {
      atomicExch(p.status, ST_DEVICE_TIMEOUT);
      p.status[1] = 11;  // where: resident kernel
      p.status[2] = blockIdx.x;
      p.status[3] = warp;
    }
    ring_drain(bar0, NST, issued);
  }
  if constexpr (CLUSTER) {
    for (int t = chunk + warp * p.S; t < tiles && ok; t += RES_WARPS * p.S) {
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(got_bar, 0u) ? 1 : 0)) { ok = false; break; }
      const float4* got = reinterpret_cast<const float4*>(smem_raw + got_off) + (t - chunk) * MT * 32 + lane;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int c = 0; c < p.S; ++c) {
          const float4 x = got[(c * MT + mt) * 32];
          v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        const int m = mt * 8 + 2 * j, col = (tile0 + t) * 16 + r;
        unsigned short* c = reinterpret_cast<unsigned short*>(p.c) + (size_t)m * p.ldc + col;
        if (m < p.M) { c[0] = res_out_bits<ACT>(v.x); c[8] = res_out_bits<ACT>(v.z); }
        if (m + 1 < p.M) { c[p.ldc] = res_out_bits<ACT>(v.y); c[p.ldc + 8] = res_out_bits<ACT>(v.w); }
      }
    }
    if (!__all_sync(0xffffffffu, ok ? 1 : 0)) {
      if (lane == 0) { atomicExch(p.status, ST_DEVICE_TIMEOUT); p.status[1] = 11; p.status[2] = blockIdx.x; p.status[3] = warp; }
      // peers may still send their sums: they have left, or are here as well, when this ends
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
}

template <int VAR, int MT, int NG, int ACT, bool CLUSTER>
static cudaError_t launch_one(const ResidentParams& p, int smem_bytes, cudaStream_t stream) {
  auto kern = resident_kernel<VAR, MT, NG, ACT, CLUSTER>;
  static std::atomic<bool> allowed[16];
  const cudaError_t e = allow_smem(kern, allowed);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)p.grid, 1, 1);
  cfg.blockDim = dim3(RES_WARPS * 32, 1, 1);
  cfg.dynamicSmemBytes = (size_t)smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (p.pdl) {  // (without it the requests ahead of griddepcontrol.wait follow the previous kernel, too)
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (CLUSTER) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)p.S;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kern, p);
}

template <int VAR, bool CLUSTER>
static cudaError_t launch_rows8(const ResidentParams& p, int ng, int smem_bytes, cudaStream_t stream) {
  if (ng > 4) return cudaErrorInvalidValue;
  if (p.act == 0)
    return ng <= 2 ? launch_one<VAR, 1, 2, 0, CLUSTER>(p, smem_bytes, stream) : launch_one<VAR, 1, 4, 0, CLUSTER>(p, smem_bytes, stream);
  return ng <= 2 ? launch_one<VAR, 1, 2, 1, CLUSTER>(p, smem_bytes, stream) : launch_one<VAR, 1, 4, 1, CLUSTER>(p, smem_bytes, stream);
}

template <int VAR>
static cudaError_t launch_var(int var, const ResidentParams& p, int mt, int ng, int smem_bytes, cudaStream_t stream) {
  if constexpr (VAR % B200Q_NPARTS == B200Q_PART) {
    if (var == VAR) {
      if (mt == 2) return ng <= 2 && p.act == 0 && p.S == 1 ? launch_one<VAR, 2, 2, 0, false>(p, smem_bytes, stream) : cudaErrorInvalidValue;
      return p.S > 1 ? launch_rows8<VAR, true>(p, ng, smem_bytes, stream) : launch_rows8<VAR, false>(p, ng, smem_bytes, stream);
    }
  }
  if constexpr (VAR + 1 < VAR_COUNT) return launch_var<VAR + 1>(var, p, mt, ng, smem_bytes, stream);
  else return cudaErrorInvalidValue;
}

#define B200Q_CAT2(a, b) a##b
#define B200Q_CAT(a, b) B200Q_CAT2(a, b)
cudaError_t B200Q_CAT(resident_launch_part, B200Q_PART)(int var, const ResidentParams& p, int mt, int ng, int smem_bytes,
                                                         cudaStream_t stream) {
  return launch_var<0>(var, p, mt, ng, smem_bytes, stream);
}

}  // namespace b200q
