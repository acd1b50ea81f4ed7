// C ABI of libb200q (declared in include/b200q.h): argument validation, the static
// shape -> tile table, and kernel dispatch.  No torch types, no allocation.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>

#include <cuda.h>

#include "../../include/b200q.h"
#include "common.cuh"

#ifndef B200Q_NPARTS
#define B200Q_NPARTS 8
#endif

namespace b200q {

#define B200Q_DECL_SPART(i) \
  cudaError_t stream_launch_part##i(int, const StreamParams&, int, int, cudaStream_t);
B200Q_DECL_SPART(0) B200Q_DECL_SPART(1) B200Q_DECL_SPART(2) B200Q_DECL_SPART(3)
B200Q_DECL_SPART(4) B200Q_DECL_SPART(5) B200Q_DECL_SPART(6) B200Q_DECL_SPART(7)
cudaError_t dequant_launch(int var, const DequantParams& p, cudaStream_t stream);
cudaError_t cast_launch(const CastParams& p, int act, bool swiglu, cudaStream_t stream);
cudaError_t host_fetch_launch(const void* src, int lds, void* dst, int M, int K, cudaStream_t stream);
cudaError_t gather_push_launch(const void* src, int lds, int M, int N_loc, int ldc, int* status, const GatherArgs& ga,
                               cudaStream_t stream);
cudaError_t gather_collect_launch(void* dst_local, int ld_local, int M, int ldc, int* status, const GatherArgs& ga,
                                  cudaStream_t stream);
cudaError_t quantize_launch(const void* w, int w_dtype, int ldw, void* bq, void* scales, int N, int K, int group,
                            int kind, int nbits, int ebits, int mbits, float minv, float maxv, int act,
                            cudaStream_t stream);
#define B200Q_DECL_UPART(i) \
  cudaError_t umma_launch_part##i(int, const UmmaParams&, const void*, int, cudaStream_t);
B200Q_DECL_UPART(0) B200Q_DECL_UPART(1) B200Q_DECL_UPART(2) B200Q_DECL_UPART(3)
B200Q_DECL_UPART(4) B200Q_DECL_UPART(5) B200Q_DECL_UPART(6) B200Q_DECL_UPART(7)
#define B200Q_DECL_BPART(i) \
  cudaError_t batch_launch_part##i(int, const BatchParams&, const void*, int, cudaStream_t);
B200Q_DECL_BPART(0) B200Q_DECL_BPART(1) B200Q_DECL_BPART(2) B200Q_DECL_BPART(3)
B200Q_DECL_BPART(4) B200Q_DECL_BPART(5) B200Q_DECL_BPART(6) B200Q_DECL_BPART(7)
#define B200Q_DECL_EPART(i) \
  cudaError_t exact_launch_part##i(int, const BatchParams&, const void*, int, cudaStream_t);
B200Q_DECL_EPART(0) B200Q_DECL_EPART(1) B200Q_DECL_EPART(2) B200Q_DECL_EPART(3)
B200Q_DECL_EPART(4) B200Q_DECL_EPART(5) B200Q_DECL_EPART(6) B200Q_DECL_EPART(7)
#define B200Q_DECL_RPART(i) \
  cudaError_t resident_launch_part##i(int, const ResidentParams&, int, int, int, cudaStream_t);
B200Q_DECL_RPART(0) B200Q_DECL_RPART(1) B200Q_DECL_RPART(2) B200Q_DECL_RPART(3)
B200Q_DECL_RPART(4) B200Q_DECL_RPART(5) B200Q_DECL_RPART(6) B200Q_DECL_RPART(7)
int exact_smem_bytes(int bits, int stages, int M);
int exact_stages(int bits, int max_smem, int M);
int batch_max_clusters(int c);
int batch_smem_bytes(int bits, int stages, int a_stages, int rows, int rpg, int cluster);
void batch_stages(int bits, int max_smem, int rows, int rpg, int cluster, int sets, int* stages, int* a_stages);
int umma_smem_bytes(int tm, int bits, int a_stages, int rpg);
int umma_a_stages(int tm, int bits, int max_smem, int rpg);

static thread_local int g_last_cuda_error = 0;

static cudaError_t stream_launch(int var, const StreamParams& p, int mt, int smem, cudaStream_t s) {
  switch (var % B200Q_NPARTS) {
    case 0: return stream_launch_part0(var, p, mt, smem, s);
    case 1: return stream_launch_part1(var, p, mt, smem, s);
    case 2: return stream_launch_part2(var, p, mt, smem, s);
    case 3: return stream_launch_part3(var, p, mt, smem, s);
    case 4: return stream_launch_part4(var, p, mt, smem, s);
    case 5: return stream_launch_part5(var, p, mt, smem, s);
    case 6: return stream_launch_part6(var, p, mt, smem, s);
    default: return stream_launch_part7(var, p, mt, smem, s);
  }
}

static cudaError_t resident_launch(int var, const ResidentParams& p, int mt, int ng, int smem, cudaStream_t s) {
  switch (var % B200Q_NPARTS) {
    case 0: return resident_launch_part0(var, p, mt, ng, smem, s);
    case 1: return resident_launch_part1(var, p, mt, ng, smem, s);
    case 2: return resident_launch_part2(var, p, mt, ng, smem, s);
    case 3: return resident_launch_part3(var, p, mt, ng, smem, s);
    case 4: return resident_launch_part4(var, p, mt, ng, smem, s);
    case 5: return resident_launch_part5(var, p, mt, ng, smem, s);
    case 6: return resident_launch_part6(var, p, mt, ng, smem, s);
    default: return resident_launch_part7(var, p, mt, ng, smem, s);
  }
}

static cudaError_t batch_launch(int var, const BatchParams& p, const void* tmap, int smem, cudaStream_t s) {
  switch (var % B200Q_NPARTS) {
    case 0: return batch_launch_part0(var, p, tmap, smem, s);
    case 1: return batch_launch_part1(var, p, tmap, smem, s);
    case 2: return batch_launch_part2(var, p, tmap, smem, s);
    case 3: return batch_launch_part3(var, p, tmap, smem, s);
    case 4: return batch_launch_part4(var, p, tmap, smem, s);
    case 5: return batch_launch_part5(var, p, tmap, smem, s);
    case 6: return batch_launch_part6(var, p, tmap, smem, s);
    default: return batch_launch_part7(var, p, tmap, smem, s);
  }
}

static cudaError_t exact_launch(int var, const BatchParams& p, const void* tmap, int smem, cudaStream_t s) {
  switch (var % B200Q_NPARTS) {
    case 0: return exact_launch_part0(var, p, tmap, smem, s);
    case 1: return exact_launch_part1(var, p, tmap, smem, s);
    case 2: return exact_launch_part2(var, p, tmap, smem, s);
    case 3: return exact_launch_part3(var, p, tmap, smem, s);
    case 4: return exact_launch_part4(var, p, tmap, smem, s);
    case 5: return exact_launch_part5(var, p, tmap, smem, s);
    case 6: return exact_launch_part6(var, p, tmap, smem, s);
    default: return exact_launch_part7(var, p, tmap, smem, s);
  }
}

static cudaError_t umma_launch(int var, const UmmaParams& p, const void* tmap, int smem, cudaStream_t s) {
  switch (var % B200Q_NPARTS) {
    case 0: return umma_launch_part0(var, p, tmap, smem, s);
    case 1: return umma_launch_part1(var, p, tmap, smem, s);
    case 2: return umma_launch_part2(var, p, tmap, smem, s);
    case 3: return umma_launch_part3(var, p, tmap, smem, s);
    case 4: return umma_launch_part4(var, p, tmap, smem, s);
    case 5: return umma_launch_part5(var, p, tmap, smem, s);
    case 6: return umma_launch_part6(var, p, tmap, smem, s);
    default: return umma_launch_part7(var, p, tmap, smem, s);
  }
}

// cuTensorMapEncodeTiled through the runtime's driver entry point lookup (no link to libcuda)
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// wtype tag + zero point -> kernel variant (decode.cuh), or -1
static int variant_of(int wtype, int zero_point) {
  const int kind = (wtype >> 16) & 0xff, nbits = (wtype >> 8) & 0xff, e = (wtype >> 4) & 0xf, m = wtype & 0xf;
  if (nbits < 1 || nbits > 8) return -1;
  if (kind == 0) {
    if (zero_point == 0) return (nbits - 1) * 2;
    if (zero_point == (1 << (nbits - 1))) return (nbits - 1) * 2 + 1;
    return -1;
  }
  if (kind == 1) return zero_point == 0 ? (nbits - 1) * 2 + 1 : -1;
  if (kind == 2 && zero_point == 0 && nbits == 1 + e + m) {
    for (int v = 16; v < VAR_COUNT; ++v)
      if (var_float_bits(v) == nbits && var_float_ebits(v) == e) return v;
  }
  return -1;
}

struct DeviceInfo {
  int sm_count = 0;
  int max_smem = 0;
};
static DeviceInfo device_info() {
  static DeviceInfo cache[16];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 16 && cache[dev].sm_count) return cache[dev];
  DeviceInfo d;
  cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&d.max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (d.sm_count <= 0) d.sm_count = 148;
  if (d.max_smem <= 0) d.max_smem = 227 * 1024;
  if (dev >= 0 && dev < 16) cache[dev] = d;
  return d;
}

// shared-memory row pitch (halfs) of an activation chunk of kc columns: 16 bytes of padding
// per 32 columns, and pitch bytes = 64 (mod 128), so that 8 lanes reading 16 bytes each from
// two rows x four 32-column units touch 8 different 16-byte bank groups
static int stream_pitch(int kc) {
  int bytes = kc * 2 + (kc / 32) * 16;
  if (bytes % 128 != 64) bytes += (64 - bytes % 128 + 128) % 128;
  return bytes / 2;
}
// ---- stream kernel (kernel 2) ---------------------------------------------------------------------
// One CTA of 16 warps per SM, or two of 8.
static const int kStreamSmemCap = 113 * 1024;  // half an SM
// Rings beyond this are not worth their room: every CTA fills them before its activations arrive, and what is requested first is
// waited for first (M = 1, 4096 x 14336, 4 bits: rings of 64 / 160 KB, activations staged 2.8 / 4.6 us after the start; the
// linears of a Llama-3-8B block 33.3 / 34.9 us).
static const int kStreamRing = 72 * 1024;
static const int kOneCtaSmem = 116 * 1024;  // more than half an SM
static const int kTwoCtaSmem = 80 * 1024;   // more than a third
static int stream_slot_bytes(int bits) { return stream_gi(bits) * 256 * bits; }
// 8-row activation tiles per launch: 1 or 2 (the kernel's MT)
static int stream_mt(int m_pass) { return m_pass <= 8 ? 1 : 2; }
// most activation rows one launch of the stream kernel takes
static int stream_rows_per_pass(int M) { (void)M; return 16; }
// Whole column tiles a CTA owns: an equal share of all of them where that leaves the last CTA at least one, else what
// divides evenly, the rest being shared item by item (the tiles' sums live in at most 16 KB of shared memory).
static int stream_tiles_owned(int m_pass, int NT, int cpc) {
  const int cap = 32 / stream_mt(m_pass), t = (NT + cpc - 1) / cpc;
  if (t <= cap && (long long)t * (cpc - 1) < NT) return t;
  return NT / cpc < cap ? NT / cpc : cap;
}
// log2 of the warps of a CTA that owns t_own tiles of kc rows, in a launch of `ctas` CTAs.  Launches of more CTAs than SMs: 8, of which two
// share an SM (16 would leave the second one no registers).  At most 16 ring items per CTA: 8, since most of 16 would only be
// started - for one and two rows always, for more rows with at most 8 items and as long as there is not much to stage, which 16 warps
// do faster (16 / 8 warps, us, 4 bits: 4 x 1024 x 1024 3.60 / 3.34, 3 x 2048 x 1024 3.81 / 3.27, 8 x 8192 x 512 4.45 / 3.94; but 4 x
// 2048 x 2048 4.32 / 4.45; 2 bits, four items: 4 x 4096 x 1024 4.45 / 3.60, 4 x 2048 x 2048 4.62 / 4.41, two items: 8 x 1024 x 1024 4.37
// / 4.54; single bits, 14 items: 6 x 16384 x 1024 5.30 / 5.96).
static int stream_warp_shift(int m_pass, int kc, int bits, int t_own, int ctas) {
  if (stream_mt(m_pass) == 1 && ctas > device_info().sm_count) return 3;
  const int KBc = kc / BLOCK_K, items = t_own * KBc * (4 / stream_gi(bits));
  if (t_own < 1 || items > (m_pass <= 2 ? 16 : 8) || m_pass > 8) return 4;
  return m_pass <= 2 || m_pass * KBc <= (items == 3 || items == 4 ? 16 : 12) ? 3 : 4;
}
static int stream_smem(int m_pass, int kc, int bits, int stages, int t_own, int ctas) {
  const int mt = stream_mt(m_pass), warps = 1 << stream_warp_shift(m_pass, kc, bits, t_own, ctas);
  // barriers, rings and scale caches of the warps, own-tile sums, activation chunk (+ 64 zero bytes), group sums as accumulator quads
  return STREAM_HEADER + warps * (stages * stream_slot_bytes(bits) + STREAM_SC_GROUPS * 32) + t_own * 16 * 8 * mt * 4 +
         m_pass * stream_pitch(kc) * 2 + 64 + (kc / 128) * 16 * mt * 4;
}
// What a launch of `ctas` CTAs asks for.  CTAs that fit one per SM must not meet two to an SM while others idle, as they would where the
// previous launch's CTAs leave at different times (128 CTAs of 6144 x 4096 on 88 SMs: 7.2 us, one to an SM 5.4).  Launches of a few KB
// per CTA gain more from starting beside their predecessor (2048 x 2048, 2 bits, 8 KB: 3.1 / 3.8 us; 3 bits, 12 KB: 3.8 / 3.9).
// Likewise three of two (M = 1, 8192 x 1024: 4 bits 3.77 us, 3.51 so; 28672 x 2048, 3 bits, 15.4 / 11.5).
static int stream_launch_smem(int m_pass, int kc, int bits, int stages, int t_own, int ctas) {
  const int smem = stream_smem(m_pass, kc, bits, stages, t_own, ctas), sms = device_info().sm_count;
  const int least = ctas <= sms ? (t_own * (kc / BLOCK_K) * bits > 20 ? kOneCtaSmem : 0) : stream_mt(m_pass) == 1 ? kTwoCtaSmem : 0;
  return smem > least ? smem : least;
}
static int stream_stages_for(int m_pass, int kc, int bits, int t_own, int ctas, int smem) {
  int st = 8;
  while (st > 0 && stream_smem(m_pass, kc, bits, st, t_own, ctas) > smem) --st;
  return st;
}
// The first CTAs of a launch on host buffers fetch the activations, four 16-byte pieces per thread: how many of them that takes
static int stream_fetch_ctas(int M, int N, int K, int bits, const b200q_plan_t& pl) {
  const int kc = K / pl.splits, t_own = stream_tiles_owned(M, N / BLOCK_N, pl.ctas_per_split);
  const int per_cta = (32 << stream_warp_shift(M, kc, bits, t_own, pl.splits * pl.ctas_per_split)) * 4;
  return (M * (K / 8) + per_cta - 1) / per_cta;
}
// CTAs per k chunk: the fewest that finish as soon as one per SM would.  9 to 16 rows: a number near all SMs that divides the column
// tiles, where there is one, since every warp then ends on the end of a tile and hands over its two sets of sums once (host
// calls, 4 bits, us, such a number / the fewest: 9 x 8192 x 8192 23.6 / 29.0, 9 x 32768 x 4096 27.2 / 36.4, 16 x 16384 x 8192 53.9 / 58.9;
// 9 x 28672 x 4096 25.1 / 25.0).
static int stream_ctas_per_chunk(int m_pass, int NT, int s, const DeviceInfo& di) {
  const int full = di.sm_count / s;
  if (full < 1) return 0;
  for (int c = full; m_pass > 8 && c * 5 >= full * 4; --c)
    if (NT % c == 0) return c;
  const int t = (NT + full - 1) / full;
  return (NT + t - 1) / t;
}
// Small layers, few rows: two CTAs of 8 warps per SM, each with its own share of the column tiles, which start, wait and finish beside
// each other.  For rings that one CTA fills for most of its life: column tiles of at most 21 KB, or up to 2048 rows layers of 8 MB in
// all, 8-bit types only the latter; activations of at most 12 KB; not where two equal shares make the fullest SM do an eighth more;
// from three rows on not where one CTA would have 8 warps.  us, one CTA of 16 warps / two of 8: M = 1: 16384 x 1024, 4 bits 5.0 / 4.4, 2
// bits 4.4 / 4.0; 12288 x 2048, 2 bits 5.7 / 5.0; 8192 x 2048, 4 bits 4.9 / 4.5; 12288 x 1536, 5 bits 7.4 / 6.2; 8192 x 1024, 8 bits 4.7
// / 4.4; more rows: 3 x 12288 x 2048, 2 bits 6.4 / 6.0; 6 x 16384 x 1024, 4 bits 6.2 / 5.8; 8 x 16384 x 512 5.2 / 5.0; 4 x 16384 x 1536
// 7.0 / 6.6.  Beyond those lines: 14336 x 4096, 4 bits 9.0 / 9.3; 4096 x 4096 5.1 / 4.9 in a chain of its own, but 0.2 us more among
// the other linears of a block; 16384 x 2048, 8 bits 8.5 / 8.8; 4 x 4096 x 2048, 4 bits 4.7 / 5.0; 5120 x 4096, 3 bits (two tiles on 160
// CTAs) 6.6 / 8.0; 8 x 8192 x 512, single bits (8 warps) 4.3 / 4.5.
static int stream_paired_ctas(int m_pass, int NT, int K, int bits, const DeviceInfo& di) {
  const int tile = 2 * K * bits;  // bytes
  if (m_pass > 8 || m_pass * (K / BLOCK_K) > 12) return 0;
  if (tile > 21 << 10 && K > 2048) return 0;
  if ((bits == 8 || tile > 21 << 10) && (long long)NT * tile > 8 << 20) return 0;
  const int t = (NT + 2 * di.sm_count - 1) / (2 * di.sm_count), ctas = (NT + t - 1) / t;
  const int t1 = (NT + di.sm_count - 1) / di.sm_count, ctas1 = (NT + t1 - 1) / t1;
  if (m_pass > 2 && stream_warp_shift(m_pass, K, bits, t1, ctas1) == 3) return 0;
  return ctas > di.sm_count && 2 * t * 7 <= t1 * 8 ? ctas : 0;
}
static const int kStreamMaxRows = 16;  // what the kernel takes
static const int kStreamPlanRows = 4;  // what the plan gives it at any shape (gather and host-buffer launches: all of the above)
static size_t stream_workspace_bytes(int N) { return WS_HEADER_BYTES + ws_counter_bytes(N) + (size_t)16 * N * sizeof(float); }
// What a number of k chunks costs a launch of 2 to 8 rows, in activations that a CTA stages (82 us per million): those of its chunk, and
// with several chunks 9500 for meeting in the scratch and 0.075 for each sum that goes through it.  Fitted to all divisors
// of K up to 16 forced at 622 shapes (1024 .. 57344 columns, K = 2048 .. 14336, 2, 4 and 8 bits): the choice is behind the best one by 0.7 % on
// average and 14 % at most.  What it replaced - one chunk where it fits, at 7 and 8 rows half of the shared memory - was 7 % behind
// on average, 68 % at most (us, that / now: 4 x 1024 x 14336, 4 bits 11.0 / 6.6, 6 x 3072 x 9216 12.5 / 8.1, 6 x 8192 x 8192 14.6 / 12.3).
static double stream_chunk_cost(int m_pass, int N, int K, int s) {
  return (double)m_pass * K / s + (s > 1 ? 9500.0 + 0.075 * N * m_pass * s : 0.0);
}
// K is cut into S chunks (a divisor of K/512, at most one per SM) so that the activation chunk
// [M, K/S] fits next to the rings; the grid is S * CPC.  2 to 8 rows: the number with the least of what depends on it, see
// stream_chunk_cost.  Otherwise, measured preferences, in this order: all of K in one chunk with two ring slots per warp (the CTAs then write their own tiles without meeting
// anybody in the global scratch); the fewest chunks with three slots and no column tiles left over
// (left-over tiles are shared item-wise through the scratch: the linears of a Llama-3-8B block on 148 CTAs so, one row,
// 41 us, 33 with whole tiles); the fewest chunks with two slots and none left over; then whatever fits.
static int plan_stream(int m_pass, int N, int K, int bits, const DeviceInfo& di, b200q_plan_t* pl) {
  const int KB = K / BLOCK_K, NT = N / BLOCK_N;
  int best_s = 0, best_st = 0, best_c = 0;
  auto consider = [&](int s, int want, bool no_leftover, int smem, int cpc = 0) {
    if (best_s || KB % s) return;
    if (cpc < 1) cpc = stream_ctas_per_chunk(m_pass, NT, s, di);
    if (cpc < 1) return;
    const int t_own = stream_tiles_owned(m_pass, NT, cpc);
    if (no_leftover && cpc * t_own < NT) return;
    const int st = stream_stages_for(m_pass, (KB / s) * 512, bits, t_own, s * cpc, smem);
    if (st < want) return;
    best_s = s; best_st = st; best_c = cpc;
    const int ring = kStreamRing / (stream_slot_bytes(bits) << stream_warp_shift(m_pass, (KB / s) * 512, bits, t_own, s * cpc));
    if (best_st > ring) best_st = ring > want ? ring : want;
  };
  const int s_max = KB < di.sm_count ? KB : di.sm_count;
  const int pairs = stream_paired_ctas(m_pass, NT, K, bits, di);
  if (pairs) consider(1, 2, true, kStreamSmemCap, pairs);
  if (m_pass >= 2 && m_pass <= 8 && !best_s) {
    int cheapest = 0;
    for (int s = 1; s <= s_max; ++s) {
      if (cheapest && stream_chunk_cost(m_pass, N, K, s) >= stream_chunk_cost(m_pass, N, K, cheapest)) continue;
      consider(s, 2, true, di.max_smem);
      if (best_s) cheapest = s;
      best_s = 0;
    }
    if (cheapest) consider(cheapest, 2, true, di.max_smem);
  }
  consider(1, 2, true, kStreamSmemCap);
  consider(1, 2, true, di.max_smem);
  for (int s = 1; s <= s_max; ++s) consider(s, 3, true, di.max_smem);
  for (int s = 1; s <= s_max; ++s) consider(s, 2, true, di.max_smem);
  for (int want = 3; want >= 1; --want)
    for (int s = 1; s <= s_max; ++s) consider(s, want, false, di.max_smem);
  if (!best_s) return ST_UNSUPPORTED;
  pl->kernel = 2;
  pl->m_tiles = stream_mt(m_pass);
  pl->splits = best_s;
  pl->cluster = 1;
  pl->ctas_per_split = best_c;
  const int t_own = stream_tiles_owned(m_pass, NT, best_c), kc = (KB / best_s) * 512;
  pl->warps = 1 << stream_warp_shift(m_pass, kc, bits, t_own, best_s * best_c);
  pl->stages = best_st;
  pl->smem_bytes = stream_smem(m_pass, kc, bits, best_st, t_own, best_s * best_c);
  pl->tile_m = 0;
  pl->pdl = 1;
  return ST_OK;
}

// Shapes every kernel takes: K a multiple of 128 (the packed layout's row group), N a multiple of 16,
// one scale per `group` rows with group = 32, 64 or a multiple of 128 that divides K.  The reference
// asks for K % 16 == 0, N % 16 == 0 and group % block_k == 0 with block_k = 32 as shipped
// (examples/quantization/matmul_a16wx.py:66-71, :207).  for_gemm = false: the dequantize kernel, which
// takes any multiple of 32.
static int check_problem(int M, int N, int K, int wtype, int zero_point, int group, bool for_gemm, int* var) {
  if (M < 1 || N < 1 || K < 1 || group < 1) return ST_INVALID_ARG;
  *var = variant_of(wtype, zero_point);
  if (*var < 0) return ST_UNSUPPORTED;
  if (K % 128 != 0 || N % BLOCK_N != 0) return ST_UNSUPPORTED;
  if (group % 32 != 0 || K % group != 0) return ST_UNSUPPORTED;
  if (for_gemm && group != 32 && group != 64 && group % 128 != 0) return ST_UNSUPPORTED;
  return ST_OK;
}
// the decode kernel works in whole 512-row blocks and applies one scale per 128-row group
static bool stream_takes(int K, int group) { return K % BLOCK_K == 0 && group % 128 == 0; }
static int gshift_of(int group) {  // log2(group / 128) when that is a power of two, else -1
  const int d = group / 128;
  if (d < 1 || (d & (d - 1)) != 0) return -1;
  int s = 0;
  while ((1 << s) < d) ++s;
  return s;
}

// tcgen05 kernel: tile rows, tiles and split-K so that the grid fills the SMs
static int rpg_of(int group) { return group < 128 ? 128 / group : 1; }

static int umma_tail(int tiles, int grid, int kblocks, int uniform_splits, int N, int* splits);
// Uniform split-K of a launch whose tiles leave half of the SMs idle: as many K ranges as still run in one round of the
// persistent CTAs.  (A few items more than SMs double the time: 200 x 5120 x 4096, 4 bits, 40 tiles in 2 / 4 ranges
// 27.1 / 33.8 us; 256 x 5120 x 5120, 8 bits, 34.6 / 42.6.)
static int umma_splits(int ctas, int N, int K, const DeviceInfo& di) {
  const int kblocks = K / 64;
  int splits = 1;
  if (ctas * 2 <= di.sm_count && ctas <= N / BLOCK_N) {
    for (int s = 2; s <= 16; ++s)
      if (kblocks % (2 * s) == 0 && kblocks / s >= 8 && ctas * s <= di.sm_count) splits = s;
  }
  return splits;
}
// Cost of a launch with tiles of tm rows, in rows: rounds of the persistent CTAs (a round cut along K takes its
// fraction and 0.3 of a tile for the sums that meet in L2) times the rows of a tile (the last row tile costs its own
// rows only; a single round lasts as long as its largest tile) and 160 rows' worth for dequantizing the tile's weights.
// Fitted to 256 against 384 rows at 27 shapes, 300 .. 4096 rows, 1264 .. 28672 columns: it picks the faster one at
// 24 of them and loses at most 10 % at the others.  4-bit weights, 256 / 384 rows, us: 300 x 28672 x 4096 131 / 84,
// 640 x 8192 x 4096 55 / 39, 1024 x 4096 x 4096 33 / 39, 2048 x 4096 x 4096 64 / 69, 4096 x 12288 x 4096 361 / 301.
static double umma_cost(int M, int N, int K, int tm, const DeviceInfo& di) {
  const int m_tiles = (M + tm - 1) / tm, tiles = m_tiles * ((N + 127) / 128);
  const int splits = umma_splits(tiles, N, K, di);
  double rounds;
  if (splits > 1 || tiles <= di.sm_count) {
    rounds = splits > 1 ? 1.0 / splits + 0.3 : 1.0;
  } else {
    int tail_splits;
    const int tail = umma_tail(tiles, di.sm_count, K / 64, 1, N, &tail_splits);
    rounds = tail > 0 ? tiles / di.sm_count + 1.0 / tail_splits + 0.3 : (tiles + di.sm_count - 1) / di.sm_count;
  }
  const double rows = rounds <= 1.0 ? (M < tm ? M : tm) : (double)M / m_tiles;
  return rounds * (rows + 160.0);
}
static void plan_umma(int M, int N, int K, int bits, int group, const DeviceInfo& di, int max_tm, b200q_plan_t* pl) {
  int tm = 256;  // (plans start here at 129 rows; smaller tiles only through an edited plan)
  if (M > 256 && max_tm >= 384 && umma_cost(M, N, K, 384, di) < umma_cost(M, N, K, 256, di)) tm = 384;
  const int m_tiles = (M + tm - 1) / tm, n_tiles = (N + 127) / 128;
  const int ctas = m_tiles * n_tiles;
  const int splits = umma_splits(ctas, N, K, di);
  pl->kernel = 1;
  pl->m_tiles = m_tiles;
  pl->splits = splits;
  pl->cluster = 1;
  pl->ctas_per_split = ctas;
  pl->stages = umma_a_stages(tm, bits, di.max_smem, rpg_of(group));
  pl->smem_bytes = umma_smem_bytes(tm, bits, pl->stages, rpg_of(group));
  pl->tile_m = tm;
  pl->warps = 23;
  pl->passes = 1;
  pl->pdl = 0;
}

// small-batch tcgen05 kernel (kernel 3): equal runs of (128-column tile, 128-row group) pairs, one CTA per SM
static const int kBatchMaxRows = 128;
static int batch_rows(int M) { return (M + 15) / 16 * 16; }
// arrival counts and fp32 sums of the column tiles
static size_t batch_count_bytes(int N) { return ((size_t)((N + 127) / 128) * 32 * sizeof(int) + 255) / 256 * 256; }
static size_t batch_scratch_bytes(int M, int N) {
  return batch_count_bytes(N) + (size_t)((N + 127) / 128) * batch_rows(M) * 128 * sizeof(float);
}
// up to 16 rows with one scale per 128-row group at most: weights stay exact, scales go to the sums (exact_kernel.cu)
static bool batch_exact(int M, int group) { return M <= 16 && group % 128 == 0; }
// How the column tiles are shared out, as (CTAs, CTAs per cluster):
//  - equal runs of 128-row groups, one per SM: no SM idles, but the tiles' sums meet in L2;
//  - a cluster of c CTAs per tile: sums meet in distributed shared memory (at most as many tiles as clusters fit);
//  - whole tiles, as many per CTA as one round takes.
// The times are fits to chains of launches on B200 (4-bit weights in fp16, us; 1024 x 4096 .. 4096 x 14336, 16 .. 128 rows, each
// form forced; within 15 % there) and serve every width and both activation types: for 100 x 11008 x 4224, 6 bits in
// bf16, they say 16.1 where a call takes 20.2.  Up to 32 rows of the types that have an SM to themselves (batch_sets) each group of equal runs costs
// more, and of whole tiles on more than half of the SMs: fits to 840 calls of 3, 5, 6 and 8 bits, float6 and float8, 1024 .. 8192 rows of K, 2560 ..
// 18432 columns at 12, 24 and 32 rows, each form forced; the choice is behind the best form by 0.4 % on average, with the 4-bit costs 1.2 (12 x
// 6144 x 4096, float8 in bf16, groups of 64, 11.2 us on equal runs, 9.5 with two CTAs per tile), at most by 24 % (24 x 11008 x 2048 in 8 bits, 10.0 on equal
// runs, whole tiles 8.3), and by up to 5 % behind the form with those costs at 3 of the 840.  Fewer CTAs start and end cheaper because the next launch finds SMs free (17 x 2048 x
// 4096, 4 / 6 CTAs per tile, that is 64 / 96 CTAs, 4.5 / 5.7 us, equal runs 6.0; 64 x 4096 x 4096, 2 / 3 / 4 per tile 8.5 / 8.6 / 8.6).
static int max_clusters(int c) {
  static int cache[16][9];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { (void)cudaGetLastError(); dev = -1; }
  if (dev >= 0 && dev < 16 && cache[dev][c] > 0) return cache[dev][c] - 1;
  static const int typical[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};
  const int n = dev >= 0 ? batch_max_clusters(c) : 0;
  if (n <= 0) return typical[c];
  if (dev < 16) cache[dev][c] = n + 1;
  return n;
}
// Dequantizing sets of a CTA of batch_kernel.cu: three, since two leave a third of the time to latencies (64 x 16384 x 4096,
// 4 bits 15.6 / 14.6 us, 100 x 11008 x 4224, 6 bits in bfloat16 20.3 / 18.7), but beyond 64 rows only where every CTA has one column tile to
// itself and the ring two stages per set: tensor memory then holds a single accumulator next to three sets' slots (128 x 28672 x 4096
// 32.4 / 34.7), and a cluster's ring gets too short (128 x 4096 x 14336 18.7 / 20.7; in 8 bits with scales per 64 rows 119 x 9920 x 4096 19.6 /
// 21.9).  Two for types of which two CTAs share an SM.
static int batch_sets(int var, int rows, int rpg, int cluster, bool one_tile, const DeviceInfo& di) {
  if (rows <= 64) return batch_shares_sm(rows, var) && cluster <= 1 ? 2 : 3;
  int stages, a_stages;
  batch_stages(var_bits(var), di.max_smem, rows, rpg, 1, 3, &stages, &a_stages);
  return cluster == 1 && one_tile && stages >= 6 ? 3 : 2;
}
static void batch_split(int M, int var, int group, int n_tiles, int G, const DeviceInfo& di, int* ctas, int* cluster) {
  long long grid = ((long long)n_tiles * G + 1) / 2;  // at least two groups per CTA
  if (grid > di.sm_count) grid = di.sm_count;
  const bool exact = batch_exact(M, group), shares = !exact && batch_shares_sm(batch_rows(M), var);
  const double groups = (double)n_tiles * G / grid;
  const bool alone = !exact && !shares && M <= 32;
  double best = 6.0 + (M > 24 ? 0.085 * (M - 24) : 0.0) + (alone ? 0.42 : 0.27) * groups + (!exact && groups > 24 ? 0.12 * (groups - 24) : 0.0);
  *ctas = (int)grid;
  *cluster = 1;
  // Kernels whose CTAs share SMs have no clusters: CTAs of cluster launches must not meet two to an SM while others idle, and the
  // two kinds mixed wait for each other's SMs (a Llama-3-8B block at 17 rows 69 us with clusters for its narrow layers, 49 without).
  // The exact kernel's registers allow one CTA per SM.
  for (int c = 1; c <= (shares ? 1 : 8); ++c) {
    const int tiles = c == 1 && !exact ? (n_tiles + di.sm_count - 1) / di.sm_count : 1;  // whole column tiles of a CTA
    const int n = (n_tiles + tiles - 1) / tiles * c;
    if (shares && 2 * n <= di.sm_count) continue;  // (the next launch's CTAs would meet these, 28 x 3200 x 1280 on 25 CTAs 6.2 us for 5.4)
    if ((c > 1 && G < 2 * c) || n > di.sm_count || (c > 1 && n_tiles > max_clusters(c))) continue;
    const int each = tiles * ((G + c - 1) / c);
    double t;
    if (exact) {
      const double start = 0.05 * n - 1.1;
      t = (start > 2.3 ? start : 2.3) + 0.033 * M + 0.29 * each;
    } else {
      const bool overlap = 2 * n <= di.sm_count;  // the next launch finds SMs free
      t = 0.03 * M + (c > 6 ? 0.8 : 0.0);
      if (c == 1) t += (overlap ? 2.0 : 3.5 + (alone ? 0.09 * each : 0.0)) + 0.28 * each + (each > 32 ? 0.08 * (each - 32) : 0.0);
      else t += (overlap ? 2.0 + 0.29 * each : 4.0 + 0.33 * each) + (M > 64 ? 0.05 * (M - 64) / c : 0.0);
    }
    if (t < best) {
      best = t;
      *ctas = n;
      *cluster = c;
    }
  }
}
// Equal runs on so many CTAs are whole column tiles, none of which is shared.
static bool batch_whole_tiles(int n_tiles, int ctas, int cluster, const DeviceInfo& di) {
  const int tiles = (n_tiles + di.sm_count - 1) / di.sm_count;
  return cluster <= 1 && ctas == (n_tiles + tiles - 1) / tiles;
}
static void plan_batch(int M, int N, int K, int var, int group, const DeviceInfo& di, b200q_plan_t* pl) {
  int ctas, cluster;
  const int bits = var_bits(var);
  batch_split(M, var, group, (N + 127) / 128, K / 128, di, &ctas, &cluster);
  pl->kernel = 3;
  const bool exact = batch_exact(M, group);
  const int sets = batch_sets(var, batch_rows(M), rpg_of(group), cluster, ctas == (N + 127) / 128, di);
  pl->m_tiles = 1;
  pl->splits = 1;
  pl->cluster = cluster;
  pl->ctas_per_split = ctas;
  if (exact) {
    pl->stages = exact_stages(bits, di.max_smem, M);
    pl->smem_bytes = exact_smem_bytes(bits, pl->stages, M);
  } else {
    int a_stages;
    batch_stages(bits, di.max_smem, batch_rows(M), rpg_of(group), cluster, sets, &pl->stages, &a_stages);
    pl->smem_bytes = batch_smem_bytes(bits, pl->stages, a_stages, batch_rows(M), rpg_of(group), cluster);
  }
  if (!exact && (cluster > 1 || !batch_shares_sm(batch_rows(M), var)) && pl->smem_bytes < kOneCtaSmem) pl->smem_bytes = kOneCtaSmem;
  pl->tile_m = batch_rows(M);
  pl->warps = exact || sets == 3 ? 20 : 16;
  pl->passes = 1;
  pl->pdl = 1;  // always launched as a programmatic dependent
}

// The persistent CTAs of the transposed tcgen05 kernel take tiles round by round.  When the last round
// would be less than half full, its tiles are cut into `splits` K ranges (whole 128-row groups, at
// least 8 64-row blocks each) so that the round costs a fraction of a tile's time.  Returns the number
// of such tail tiles (0: none).
static int umma_tail(int tiles, int grid, int kblocks, int uniform_splits, int N, int* splits) {
  *splits = 1;
  if (uniform_splits != 1 || tiles <= grid) return 0;
  const int rem = tiles % grid;
  if (rem == 0 || rem * 2 > grid || rem > N / BLOCK_N) return 0;
  int best = 1;
  for (int s = 2; s <= 16; s *= 2)
    if (s * rem <= grid && kblocks % (2 * s) == 0 && kblocks / s >= 8) best = s;
  if (best == 1) return 0;
  *splits = best;
  return rem;
}
// fp32 scratch of the transposed tcgen05 kernel: one [tm][128] slab per tile slot
static size_t umma_partial_bytes(int slots, int tm) { return (size_t)slots * tm * 128 * sizeof(float); }

// The prefill kernel's plan with row tiles of at most max_tm rows.
static void plan_prefill(int M, int N, int K, int var, int group, int max_tm, const DeviceInfo& di, b200q_plan_t* pl) {
  const int bits = var_bits(var);
  // A last row tile of at most 16 rows would cost each column tile the dequantization of its weights once more;
  // those rows go to the decode path in a second launch instead (passes = 2).  Not where the row tiles of the
  // others have room for them (M = 4097 with tiles of 384 rows: 10 and 257 rows more).
  const int tail_rows = M % 256;
  b200q_plan_t tail_plan;
  pl->passes = 0;
  if (M > 256 && tail_rows >= 1 && tail_rows <= kStreamMaxRows && stream_takes(K, group) &&
      plan_stream(tail_rows, N, K, bits, di, &tail_plan) == ST_OK) {
    plan_umma(M - tail_rows, N, K, bits, group, di, max_tm, pl);
    pl->passes = 2;
  }
  if (pl->passes != 2 || pl->tile_m * pl->m_tiles >= M) plan_umma(M, N, K, bits, group, di, max_tm, pl);
  // fp32 slabs per tile slot: every tile of a split-K launch, or the cut tiles of the last round
  const int Mu = pl->passes == 2 ? M - M % 256 : M;
  const int tiles = ((Mu + pl->tile_m - 1) / pl->tile_m) * ((N + 127) / 128);
  const int grid = tiles * pl->splits < di.sm_count ? tiles * pl->splits : di.sm_count;
  int tail_splits;
  const int tail = umma_tail(tiles, grid, K / 64, pl->splits, N, &tail_splits);
  const size_t part = umma_partial_bytes(pl->splits > 1 ? tiles : tail, pl->tile_m);
  size_t need = WS_HEADER_BYTES + ws_counter_bytes(N) + part;
  if (pl->passes == 2) {
    const size_t rows = WS_HEADER_BYTES + ws_counter_bytes(N) + batch_scratch_bytes(M % 256, N);
    if (need < stream_workspace_bytes(N)) need = stream_workspace_bytes(N);
    if (need < rows) need = rows;
  }
  pl->workspace_bytes = need;
}

// What the two rules below were fitted to: the split of an earlier form of the stream kernel (12 warps per CTA and half an SM each, the most
// k chunks and CTAs of at most two per SM, a divisor of the column tiles), and its times.  They have not been fitted again to
// the present form (stream_ctas_per_chunk, stream_paired_ctas), which is faster mostly where that split was a bad one.  Both kernels
// forced now, fp16, 13 widths 1024 .. 28672 x 4 depths 2048 .. 8192: the kernel picked is behind the faster one by 6 / 12 / 7 / 10 / 10
// / 6 % on average at 1 / 2 / 4 / 5 / 6 / 8 rows in 4 bits, by 2 to 3 % in 8 bits.  Nearly all of it is the stream kernel not being
// picked, at worst 1 x 2560 x 2048 in 4 bits, 5.1 us for 3.2, 1 x 3584 x 4096 7.5 for 4.9, 5 x 1024 x 2048 5.7 for 4.4; the other way
// 4 x 2048 x 5120 in 8 bits, 7.2 us for 6.5.  (Speed is not all there is to it: the stream kernel stages fp16 activations times 2^-T, T up to
// 10 - bits, so that those below 2^(T-14) lose low bits there and not in the exact kernel.)
struct PairSplit { int splits, ctas; };
static PairSplit pair_split(int M, int NT, int KB, int bits, const DeviceInfo& di) {
  PairSplit best = {0, 0};
  auto consider = [&](int s, int want, bool whole) {
    const int full = di.sm_count / s;
    if (best.splits || KB % s || full < 1) return;
    int c = 0;
    for (int i = 2 * full; !c && i * 5 >= full * 8; --i) c = NT % i == 0 ? i : 0;
    for (int i = full; !c && i >= 1 && i * 5 >= full * 4; --i) c = NT % i == 0 ? i : 0;
    if (!c) c = full > NT ? NT : full;
    const int own = NT / c < 32 ? NT / c : 32, kc = KB / s * 512;
    if (whole && c * own != NT) return;
    const int fixed = 1024 + 12 * STREAM_SC_GROUPS * 32 + own * 512 + M * stream_pitch(kc) * 2 + 64 + kc / 2;
    int slots = (kStreamSmemCap - fixed) / (12 * stream_slot_bytes(bits));
    if (slots > 8) slots = 8;
    if (slots >= want) best = {s, c};
  };
  const int s_max = KB < di.sm_count ? KB : di.sm_count;
  consider(1, 2, true);
  for (int s = 1; s <= s_max; ++s) consider(s, 3, true);
  for (int s = 1; s <= s_max; ++s) consider(s, 2, true);
  for (int want = 3; want >= 1; --want)
    for (int s = 1; s <= s_max; ++s) consider(s, want, false);
  return best;
}

// Where that split cut K and still had one CTA per SM at most (no divisor of the column tiles near two per SM), its chunks met in the
// scratch like the exact kernel's, at half the warps, and the exact kernel was faster from two rows on, for one row from three
// chunks on (earlier form / exact, us, 4 bits: 7168 x 2048 9.5 / 8.7, 2448 x 11776 13.8 / 11.8, 5120 x 5120 11.3 .. 11.8 / 11.6).  The
// present form does not cut K there: 4 x 7168 x 2048 5.5 / 7.0, 2 x 5120 x 5120 7.2 / 9.2.
static bool stream_outrun(int M, const PairSplit& pl, const DeviceInfo& di) {
  return pl.splits > (M == 1 ? 2 : 1) && pl.splits * pl.ctas <= di.sm_count;
}

// fp16, 5..8 rows: the shapes where the stream kernel's earlier form was the faster one.  What the exact kernel pays is a start and
// an end of 5-6 us and, where equal runs share column tiles, sums in L2; what the stream kernel pays is the staging of the
// activations, once per CTA, and a second pass through the scratch where it cuts K.  Measured, earlier form / exact, us, cold
// chains, 11 types x 17 shapes x 5..8 rows:
//  - two CTAs per SM without cutting K, layers of more than 12 M weights, up to 6 rows (4096 x 4096 at 5 rows: 4 bits 7.2 /
//    7.9, float6 7.3 / 9.2), from 32 M weights up to 8 rows (32768 x 2048 at 8 rows: 4 bits 12.1 / 14.0); at 7 and 8 rows below
//    that the exact kernel (8192 x 2048 at 8 rows, 4 bits 7.2 / 6.2), and between 4 M and 12 M, where its clusters have
//    short ranges, at all (4096 x 2048 at 5 rows, 8 bits 5.8 / 5.1);
//  - two CTAs per SM with K cut in four or more, small layers (4096 x 4096 at 8 rows, 4 bits 7.3 / 7.9; 2048 x 8192 7.2 / 8.4),
//    again not between 4 M and 12 M (2048 x 4096 6.3 / 5.5);
//  - up to 4 M float weights and 6 rows (1024 x 4096 at 5 rows, float8 4.8 / 6.2).
// 8-bit integers, whose bytes the exact kernel takes with the fewest instructions, only from 32 M weights on (8192 x 2048 at 6
// rows 7.7 / 6.5, 8192 x 4096 at 5 rows 10.9 / 11.8).
static bool stream_ahead(int M, int N, int K, int var, const PairSplit& pl, const DeviceInfo& di) {
  const long long million = 1ll << 20, weights = (long long)N * K;
  if (M <= kStreamPlanRows) return true;
  if (M > 8) return false;
  if (pl.splits * pl.ctas > di.sm_count) {
    const bool bytes = var_bits(var) == 8 && !var_is_float(var);
    if (pl.splits == 1) return weights >= 32 * million || (weights > 12 * million && M <= 6 && !bytes);
    if (pl.splits >= 4) return (weights <= 4 * million || (weights > 12 * million && weights <= 20 * million)) && !bytes;
    return false;
  }
  return var_is_float(var) && M <= 6 && weights <= 4 * million;
}

// ---- decode kernel with the activations in registers (resident_kernel.cu) ---------------------------
struct ResidentSplit { int S, T_own, wk_shift, n_max, stages, slab_shift, smem, grid; };
// How S CTAs per cluster share the work: column tiles per cluster, and the warps that share K.  16 of them where that gives each two
// groups of 128 rows or more; for fewer rows of K the warps may form two or four sets that take turns with the column tiles, each with
// the activations of all of K: fewer parts per column tile to add up, more activations to load.  us per launch (4 bits, fits): 0.23
// per group and 0.25 per tile of a warp, 12.5 per MB of activations (1 x 28672 x 2048, 16 / 8 warps 9.3 / 8.0; 8 x 4096 x 2048 3.3 / 3.7;
// four groups per warp are slower than two of twice the warps, 1 x 28672 x 4096 14.9 / 13.4).
static bool resident_split(int M, int N, int K, int bits, int S, const DeviceInfo& di, ResidentSplit* rs) {
  const int G = K / 128, NT = N / BLOCK_N, mt = stream_mt(M), ng_max = mt == 1 ? 4 : 2;
  if (M > 16 || S < 1 || S > 8 || G < S || (S > 1 && mt > 1)) return false;
  int clusters = di.sm_count / S;
  if (S > 1 && max_clusters(S) < clusters) clusters = max_clusters(S);
  if (clusters < 1) return false;
  rs->S = S;
  rs->T_own = (NT + clusters - 1) / clusters;
  rs->grid = S * ((NT + rs->T_own - 1) / rs->T_own);
  const int Gc = (G + S - 1) / S;
  double least = 0.0;
  for (int sh = 4; sh >= 2; --sh) {
    const int n = (Gc + (1 << sh) - 1) >> sh, sets = RES_WARPS >> sh;
    if (n > (sh == 4 ? ng_max : 2)) continue;
    const double cost = ((rs->T_own + sets - 1) / sets) * (0.23 * n + 0.25) + 12.5e-6 * 2.0 * M * Gc * 128 * sets;
    if (least > 0.0 && cost >= least) continue;
    least = cost;
    rs->wk_shift = sh;
    rs->n_max = n;
  }
  if (least <= 0.0) return false;
  const int ng = rs->n_max <= 2 ? 2 : 4, slot = res_gi(bits, ng) * 256 * bits;
  const int sets = RES_WARPS >> rs->wk_shift, Tw = (rs->T_own + sets - 1) / sets;
  rs->slab_shift = Tw <= 1 ? 0 : Tw <= 2 ? 1 : 2;
  const long long fixed = RES_HEADER + (long long)RES_WARPS * ng * Tw * 32 + (RES_WARPS << rs->slab_shift) * mt * 512 +
                          (S > 1 ? (long long)(rs->T_own + S - 1) / S * S * mt * 512 : 0);  // sums that a cluster's CTAs get
  if (fixed > di.max_smem) return false;
  int st = kStreamRing / (RES_WARPS * slot);
  st = st > 8 ? 8 : st < 2 ? 2 : st;
  while (st > 2 && fixed + st * RES_WARPS * slot > di.max_smem) --st;
  rs->stages = st;
  rs->smem = (int)fixed + st * RES_WARPS * slot;
  if (rs->smem > di.max_smem) return false;
  if (rs->smem < kOneCtaSmem) rs->smem = kOneCtaSmem;  // (never two to an SM while others idle, see stream_launch_smem)
  return true;
}
// Where the resident kernel takes a decode call that the table gives to the stream kernel (tile_m 0) or the exact kernel: the CTAs
// per cluster, or 0.  Measured against those, cold chains, 9 widths x 13 depths (1024 .. 14336) x 1, 2, 4 and 8 rows in 4 bits, 5 x 6 in 1, 2, 3,
// 6 and 8 bits; time here over time there:
//  - 5 to 8 rows 0.44 .. 0.97, except 5 to 7 bits on 16384 columns and more beyond 4096 rows of K (1.00 .. 1.03); 2 to 4 rows 0.49 .. 1.0,
//    except where 4096 to 6144 rows of K, in two or three groups per warp, meet many columns (2 x 28672 x 4608 1.16), and 5 to 7 bits beyond
//    8192 rows of K (1.00 .. 1.03);
//  - one row: up to 4096 rows of K 0.68 .. 1.0 (2 bits, 28672 x 2048 1.02); up to 8192 rows of K 0.81 .. 1.0 in 5 bits and more, one CTA
//    per cluster (two: 0.85 .. 1.09), 0.85 .. 0.98 in 1 and 2 bits up to 8192 columns (28672 x 6144 1.04), and in 3 and 4 bits 0.83 .. 1.0 up to
//    6144 columns and, two CTAs per cluster, 0.95 .. 0.99 on wide layers of 7168 rows of K and more (4 bits, 8192 x 4608 1.05, 28672 x 4608
//    1.17); beyond, 0.87 .. 0.95 in 8 bits, 0.72 .. 0.98 in 4 bits (28672 x 14336 1.0), 0.88 .. 1.0 in fewer up to 4096 columns (3 bits,
//    28672 x 14336 1.04, 2 bits 1.08), 1.0 .. 1.1 in 5 to 7 bits;
//  - 9 to 16 rows (fp16 only: the exact kernel takes bfloat16 as it is), whose second set of sums makes the loop 1.5 times longer: up to
//    4096 rows of K in the ranges below 0.55 .. 1.0; beyond 1.0 .. 1.3 (9 and 12 rows, 12288, 14336 and 16384 columns: 3 bits 0.85 .. 0.94, 4
//    and 8 bits 0.87 .. 0.98, float6 0.93 .. 1.02; 9 x 28672 x 4096 1.02; blocks of linears of those widths 0.90 .. 0.99).  The widest layer goes by the
//    depth, since the exact kernel is ahead where a short range of K per CTA fills its SMs: 2, 3, 4 and 8 bits and float6 at 9 to 16 rows, 1024 rows
//    of K 5120 columns 0.69 .. 0.88, 6144 0.98 .. 1.09 (blocks with 4608 x 1024, qkv, 0.93 .. 0.99 to 12 rows, 1.01 .. 1.05 at 16); 1536 to 2048 rows 6144 columns
//    0.79 .. 0.98, 8192 0.89 .. 1.20 (blocks with 4608 x 1536, 5376 x 1792 or 5760 x 1920 0.86 .. 0.99); 2176 rows 8192 and 11008 columns at 9 and 12 rows
//    0.96 .. 1.18, but blocks of hidden size 2176 whose gate_up goes to the exact kernel 1.03 .. 1.10; 2560 rows 0.81 .. 0.96.  Beyond 2048 rows, 13 rows and
//    more: below 3072 columns 0.67 .. 1.03 in chains, blocks with such a layer from 0.93 (2560 x 2560 besides 3840 x 2560) to 1.10 (2176 x 2176
//    besides 6528 x 2176): left to the exact kernel.  Among layers that stay with the exact kernel, whose launches
//    leave SMs to their successors, a launch on all SMs costs those up to 2 us: with 4096 x 4096 here a Llama-3-8B block takes, us, at 9
//    / 13 / 16 rows 47.2 / 49.3 / 51.1 in 4 bits (50.1 / 51.1 / 50.3 without), 54.0 / 54.8 / 57.7 in 8 bits (54.5 / 54.9 / 55.7), 58.1 /
//    60.2 / 61.2 in 3 bits (62.5 / 63.1 / 62.2), 59.8 / 61.6 / 63.4 in float6 (62.9 / 63.5 / 62.8): 8 bits up to 12 rows, 4 bits up to 14.
// S: one CTA per cluster where a warp's activations fit its registers, and where the columns are few or the decoding dear; us, 8 rows,
// 4 bits, S = 1 / 2 / 4: 4096 x 5120 6.3 / 5.9 / 5.9 (6 bits 8.0 / 8.3 / 8.6), 8192 x 8192 11.7 / 10.3 / 10.6, 4096 x 14336 - / 11.1 / 9.8,
// 28672 x 14336 - / 43.8 / 45.2.
static int resident_cluster(int M, int N, int K, int var, int group, int act, bool stream_form, const DeviceInfo& di) {
  if (M > 16 || group % 128 != 0 || (act == B200Q_BF16 && !stream_form)) return 0;
  const int G = K / 128, bits = var_bits(var);
  int S;
  if (M > 8) {
    const int widest = G > 16 ? (M > 12 ? 4096 : bits >= 5 && bits <= 7 ? 11008 : 16384) : G >= 12 ? 6144 : G >= 8 && M <= 12 ? 5120 : 4096;
    if (G > 32 || N > widest || (G > 16 && N < 3072 && M > 12)) return 0;
    if (G > 16 && ((bits == 8 && M > 12) || (bits == 4 && M > 14))) return 0;
    S = 1;
  } else {
    const bool dear = bits >= 5 && bits <= 7;
    if (G <= 32) S = 1;
    else if (M == 1 && G <= 64) S = N < 8192 || bits <= 2 || bits >= 5 ? 1 : 2;
    else if (G <= 40) S = M >= 5 && bits <= 4 ? 2 : 1;
    else if (G <= 64) S = 2;
    else if (M == 1) S = G <= 128 && N >= 8192 && bits <= 4 ? 2 : 4;
    else S = G <= 128 && (N >= 16384 || (G <= 96 && N >= 8192)) ? 2 : 4;
    if (M == 1 && G <= 32) {
      if (bits <= 2 && N > 8192 && G <= 16) return 0;
    } else if (M == 1 && G <= 64) {
      if (bits <= 4 && (bits <= 2 ? N > 8192 : N >= 8192 && G < 56)) return 0;
    } else if (M == 1) {
      if (bits <= 4 ? N > (bits <= 3 ? 4096 : 16384) : dear && stream_form) return 0;
    } else if (M <= 4 && stream_form) {
      if (G > 32 && G < 48 && N >= (M == 2 ? 8192 : 14336)) return 0;
      if (M == 2 && G >= 48 && G < 56 && N >= 16384) return 0;
      if (G > 64 && dear && N >= 6144) return 0;
    } else if (M >= 5 && dear && G > 32 && N >= 16384) {
      return 0;
    }
  }
  ResidentSplit rs;
  return resident_split(M, N, K, bits, S, di, &rs) ? S : 0;
}

static const int kStreamForm = -1;  // in place of an activation type: the stream kernel's plan for any M that it takes

static int make_plan_uncached(int M, int N, int K, int var, int group, int act, b200q_plan_t* pl) {
  const DeviceInfo di = device_info();
  std::memset(pl, 0, sizeof(*pl));
  const int bits = var_bits(var);
  if (act == kStreamForm) {
    if (M > kStreamMaxRows || !stream_takes(K, group)) return ST_UNSUPPORTED;
    const int st = plan_stream(M, N, K, bits, di, pl);
    pl->passes = 1;
    pl->workspace_bytes = stream_workspace_bytes(N);
    return st;
  }
  // Up to 4 rows the mma.sync stream kernel (to 8 rows where stream_ahead says so); above, the tcgen05 kernels, whose
  // cost hardly depends on the rows.  A Llama-3-8B block of linears (4-bit) takes the stream kernel 34.6 / 38.6 / 41.1 /
  // 44.9 / 45.7 us at 1 / 2 / 4 / 6 / 8 rows, the tcgen05 kernel 48.6 / 48.8 / 48.8 / 49.9 / 49.8; at 9 rows the former's
  // second 8-row tile doubles its staging and MMAs.  bfloat16 costs the exact kernel one more half instruction per pair of weights and the stream
  // kernel only a conversion of the activations: at 8 rows the latter is 22 % faster (8192 x 8192, 4-bit, 12.6 / 16.1 us).
  if (M <= 8 && stream_takes(K, group)) {
    const PairSplit pair = pair_split(M, N / BLOCK_N, K / BLOCK_K, bits, di);
    if (pair.splits > 0 && !stream_outrun(M, pair, di) && (act == B200Q_BF16 || stream_ahead(M, N, K, var, pair, di)) &&
        plan_stream(M, N, K, bits, di, pl) == ST_OK) {
      pl->passes = 1;
      pl->workspace_bytes = stream_workspace_bytes(N);  // fp32 scratch [N][8 or 16]
      pl->resident = resident_cluster(M, N, K, var, group, act, true, di);
      return ST_OK;
    }
    std::memset(pl, 0, sizeof(*pl));
  }
  // up to 128 rows the small-batch kernels (weights streamed once); beyond, the prefill kernel
  if (M <= kBatchMaxRows) {
    plan_batch(M, N, K, var, group, di, pl);
    pl->workspace_bytes = WS_HEADER_BYTES + ws_counter_bytes(N) + batch_scratch_bytes(M, N);
    if (batch_exact(M, group)) pl->resident = resident_cluster(M, N, K, var, group, act, false, di);
    if (M <= kStreamMaxRows && stream_takes(K, group)) {  // the decode path's other form, see b200q_plan_t
      pl->kernel = 2;
      pl->m_tiles = stream_mt(M);
      if (pl->workspace_bytes < stream_workspace_bytes(N)) pl->workspace_bytes = stream_workspace_bytes(N);
    }
    return ST_OK;
  }
  plan_prefill(M, N, K, var, group, 384, di, pl);
  return ST_OK;
}

// The table is a pure function of the shape (and of the device's SM count and shared memory, which
// device_info caches for the current device), and a serving loop asks for the same few shapes over
// and over: the latest results are kept per thread.
static int make_plan(int M, int N, int K, int var, int group, int act, b200q_plan_t* pl) {
  struct Entry { int dev, M, N, K, var, group, act, status; b200q_plan_t plan; };
  static thread_local Entry cache[16];
  static thread_local int used = 0, next = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  for (int i = 0; i < used; ++i) {
    const Entry& e = cache[i];
    if (e.M == M && e.N == N && e.K == K && e.var == var && e.group == group && e.act == act && e.dev == dev) {
      *pl = e.plan;
      return e.status;
    }
  }
  const int status = make_plan_uncached(M, N, K, var, group, act, pl);
  Entry& e = cache[next];
  e.dev = dev; e.M = M; e.N = N; e.K = K; e.var = var; e.group = group; e.act = act; e.status = status; e.plan = *pl;
  next = (next + 1) % 16;
  if (used < 16) ++used;
  return status;
}

// The plan for a call that has `scratch` bytes.  Row tiles of 384 come with a K split that 256 rows may do without, or with
// larger slabs (300 x 9472 x 4096): where theirs do not fit, tiles of 256.
static void plan_within(int M, int N, int K, int var, int group, size_t scratch, b200q_plan_t* pl) {
  if (pl->workspace_bytes > (uint64_t)scratch && pl->kernel == 1 && pl->splits > 1 && pl->tile_m > 256)
    plan_prefill(M, N, K, var, group, 256, device_info(), pl);
}

// row tiles per raster group of the transposed tcgen05 kernel: as many as keep one group's
// activation rows (tm x K 16-bit values per tile) within 32 MB, a quarter of L2
static int umma_m_group(int tm, int K, int m_tiles) {
  const long long per_tile = (long long)tm * K * 2;
  long long g = (32ll << 20) / (per_tile > 0 ? per_tile : 1);
  if (g < 1) g = 1;
  if (g > m_tiles) g = m_tiles;
  return (int)g;
}

static int run_umma(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N, int K,
                    int var, int group, int act, void* workspace, size_t ws_bytes, cudaStream_t stream,
                    const b200q_plan_t& pl) {
  // (a small-batch plan edited to this kernel names its rows, a multiple of 16 up to 128: the tile that holds them)
  const bool rows = pl.tile_m >= 16 && pl.tile_m % 16 == 0 && pl.tile_m <= 128;
  const int tm = !rows ? pl.tile_m : pl.tile_m <= 32 ? 32 : pl.tile_m <= 64 ? 64 : 128;
  if (tm != 32 && tm != 64 && tm != 128 && tm != 256 && tm != 384) return ST_INVALID_ARG;
  const int m_tiles = (M + tm - 1) / tm, n_tiles = (N + 127) / 128;
  const int kblocks = K / 64;
  if (pl.splits < 1 || kblocks % (2 * pl.splits) != 0) return ST_INVALID_ARG;  // whole 128-row groups per split
  if (pl.splits > 1 && m_tiles * n_tiles > N / BLOCK_N) return ST_INVALID_ARG;  // counters region
  if ((ldc % 8) != 0 || (((uintptr_t)scales) & 15)) return ST_INVALID_ARG;  // 16-byte stores, bulk-copied scale rows
  const int bits = var_bits(var);
  const int a_stages = umma_a_stages(tm, bits, device_info().max_smem, rpg_of(group));
  const int all_tiles = m_tiles * n_tiles;
  const int grid = pl.splits * all_tiles < device_info().sm_count ? pl.splits * all_tiles : device_info().sm_count;
  int tail_splits = 1;
  int tail_tiles = umma_tail(all_tiles, grid, kblocks, pl.splits, N, &tail_splits);
  size_t need = WS_HEADER_BYTES + ws_counter_bytes(N) + umma_partial_bytes(pl.splits > 1 ? all_tiles : tail_tiles, tm);
  if (tail_tiles > 0 && workspace && ws_bytes < need) {  // a caller with a smaller workspace: whole tiles only
    tail_tiles = 0;
    tail_splits = 1;
    need = WS_HEADER_BYTES + ws_counter_bytes(N);
  }
  if (!workspace || ws_bytes < need || ((uintptr_t)workspace & 255)) return ST_WORKSPACE;
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return ST_CUDA;
  CUtensorMap tmap;
  const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)M};
  const cuuint64_t gstride[1] = {(cuuint64_t)lda * 2};
  const cuuint32_t box[2] = {64u, (cuuint32_t)(tm > 256 ? tm / 2 : tm)};
  const cuuint32_t estr[2] = {1u, 1u};
  CUresult r = enc(&tmap, act == B200Q_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(a), gdim, gstride, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { g_last_cuda_error = (int)r; return ST_CUDA; }
  UmmaParams p;
  p.bq = reinterpret_cast<const uint4*>(bq);
  p.scales = reinterpret_cast<const __half*>(scales);
  p.c = reinterpret_cast<__half*>(c);
  p.status = reinterpret_cast<int*>(workspace);
  p.counters = reinterpret_cast<int*>(reinterpret_cast<char*>(workspace) + WS_HEADER_BYTES);
  p.partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + WS_HEADER_BYTES + ws_counter_bytes(N));
  p.M = M; p.N = N; p.K = K; p.G = K / 128; p.ldc = ldc;
  p.group = group;
  p.rpg = rpg_of(group);
  p.tm = tm; p.m_tiles = m_tiles; p.n_tiles = n_tiles;
  p.splits = pl.splits; p.kblocks_per_split = kblocks / pl.splits;
  p.tail_tiles = tail_tiles; p.tail_splits = tail_tiles > 0 ? tail_splits : 0;
  p.tail_kblocks = tail_tiles > 0 ? kblocks / tail_splits : 0;
  p.a_stages = a_stages;
  p.m_group = umma_m_group(tm, K, m_tiles);
  p.act = act;
  p.grid = grid;
  const int smem = umma_smem_bytes(tm, bits, a_stages, rpg_of(group));
  if (smem > device_info().max_smem) return ST_UNSUPPORTED;
  cudaError_t e = umma_launch(var, p, &tmap, smem, stream);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

// Packed weights as a 3-D tensor of 8-byte elements for one tiled copy per 128-row group of `pieces` 16-column
// pieces: {a group's 256 * bits bytes, groups, pieces}, or for the swizzled widths {128-byte line, lines of
// all groups, pieces} with the 16-byte chunks of a line swizzled by line.
static int encode_weights(EncodeTiledFn enc, CUtensorMap* tmap, const void* bq, int N, int G, int bits, int pieces) {
  const bool swizzled = bits == 2 || bits == 4 || bits == 8;
  const cuuint64_t inner = swizzled ? 16 : 32 * bits, mid = swizzled ? (cuuint64_t)G * 2 * bits : (cuuint64_t)G;
  const cuuint64_t gdim[3] = {inner, mid, (cuuint64_t)(N / BLOCK_N)};
  const cuuint64_t gstride[2] = {inner * 8, inner * 8 * mid};
  const cuuint32_t box[3] = {(cuuint32_t)inner, swizzled ? 2u * bits : 1u, (cuuint32_t)pieces};
  const cuuint32_t estr[3] = {1u, 1u, 1u};
  const CUresult r = enc(tmap, CU_TENSOR_MAP_DATA_TYPE_INT64, 3, const_cast<void*>(bq), gdim, gstride, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, swizzled ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { g_last_cuda_error = (int)r; return ST_CUDA; }
  return ST_OK;
}

static int run_batch(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N, int K,
                     int var, int group, int act, void* workspace, size_t ws_bytes, cudaStream_t stream,
                     const b200q_plan_t& pl) {
  const int bits = var_bits(var);
  if (M > kBatchMaxRows || pl.splits < 1 || pl.ctas_per_split < 1) return ST_INVALID_ARG;
  if ((ldc % 8) != 0 || (((uintptr_t)scales) & 15)) return ST_INVALID_ARG;  // 8-byte stores, bulk-copied scale rows
  const int rows = batch_rows(M), n_tiles = (N + 127) / 128, G = K / 128;
  const size_t fixed = WS_HEADER_BYTES + ws_counter_bytes(N);
  if (!workspace || ws_bytes < fixed || ((uintptr_t)workspace & 255)) return ST_WORKSPACE;
  const bool exact = batch_exact(M, group);
  BatchParams p;
  p.work = n_tiles * G;
  p.unit = 1;
  long long grid = (long long)pl.splits * pl.ctas_per_split;
  if (grid > device_info().sm_count) grid = device_info().sm_count;
  if (grid > p.work) grid = p.work;
  // the plan's clusters, unless the caller has asked for another number of CTAs
  p.cluster = pl.cluster > 1 && pl.cluster <= 8 && grid == (long long)n_tiles * pl.cluster && G >= 2 * pl.cluster ? pl.cluster : 1;
  if (p.cluster > 1) {
    // (distributed shared memory needs no scratch)
  } else if (!exact && batch_whole_tiles(n_tiles, (int)grid, 1, device_info())) {
    p.work = n_tiles;
    p.unit = G;
  } else if (ws_bytes < fixed + batch_scratch_bytes(M, N)) {  // a caller with a smaller workspace: whole tiles need none
    p.work = n_tiles;
    p.unit = G;
    grid = n_tiles < device_info().sm_count ? n_tiles : device_info().sm_count;
  }
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return ST_CUDA;
  CUtensorMap tmaps[2];  // activations; packed weights
  {
    const cuuint64_t gdim[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t gstride[1] = {(cuuint64_t)lda * 2};
    const cuuint32_t box[2] = {64u, (cuuint32_t)rows};
    const cuuint32_t estr[2] = {1u, 1u};
    const CUresult r = enc(&tmaps[0], act == B200Q_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                           const_cast<void*>(a), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { g_last_cuda_error = (int)r; return ST_CUDA; }
  }
  {
    const int r = encode_weights(enc, &tmaps[1], bq, N, G, bits, 8);
    if (r != ST_OK) return r;
  }
  p.scales = reinterpret_cast<const __half*>(scales);
  p.c = reinterpret_cast<__half*>(c);
  p.status = reinterpret_cast<int*>(workspace);
  p.chunk_counters = reinterpret_cast<int*>(reinterpret_cast<char*>(workspace) + fixed);
  p.partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + fixed + batch_count_bytes(N));
  p.M = M; p.N = N; p.K = K; p.G = G; p.ldc = ldc;
  p.group = group;
  p.rpg = rpg_of(group);
  p.rows = rows;
  p.sets = batch_sets(var, rows, p.rpg, p.cluster, grid == n_tiles, device_info());
  batch_stages(bits, device_info().max_smem, rows, p.rpg, p.cluster, p.sets, &p.stages, &p.a_stages);
  if (exact) p.stages = exact_stages(bits, device_info().max_smem, M);
  p.grid = (int)grid;
  p.act = act;
  int smem = exact ? exact_smem_bytes(bits, p.stages, M) : batch_smem_bytes(bits, p.stages, p.a_stages, rows, p.rpg, p.cluster);
  if (!exact && (p.cluster > 1 || !batch_shares_sm(rows, var)) && smem < kOneCtaSmem) smem = kOneCtaSmem;
  if (smem > device_info().max_smem) return ST_UNSUPPORTED;
  cudaError_t e = exact ? exact_launch(var, p, tmaps, smem, stream) : batch_launch(var, p, tmaps, smem, stream);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

// b200q_gather_t of the C ABI -> the kernels' GatherArgs (checked)
static int fill_gather_args(const b200q_gather_t* gather, int M, int N, void* workspace, GatherArgs* ga) {
  std::memset(ga, 0, sizeof(*ga));
  if (gather->world < 1 || gather->world > 8 || gather->rank < 0 || gather->rank >= gather->world) return ST_INVALID_ARG;
  if (gather->mode != B200Q_GATHER_FLAGS && gather->mode != B200Q_GATHER_TAGGED) return ST_INVALID_ARG;
  const bool tagged = gather->mode == B200Q_GATHER_TAGGED;
  if (gather->ldc < gather->col_offset + N || gather->col_offset < 0 || !gather->epoch_local) return ST_INVALID_ARG;
  if ((gather->ldc & 1) || (gather->col_offset & 1)) return ST_INVALID_ARG;  // outputs leave in column pairs
  // dense rows: buffer_elems 16-bit elements between the two buffers; tagged: 64-bit words between the three
  if (gather->buffer_elems < (int64_t)M * gather->ldc / (tagged ? 2 : 1)) return ST_INVALID_ARG;
  if (!tagged && !gather->flags_local) return ST_INVALID_ARG;
  if (gather->a_prev_offset >= 0 && (gather->a_prev_offset & 7)) return ST_INVALID_ARG;
  ga->G = gather->world;
  ga->rank = gather->rank;
  ga->col_off = gather->col_offset;
  ga->mode = gather->mode;
  for (int g = 0; g < gather->world; ++g) {
    if (!gather->out[g] || (!tagged && !gather->flag_slot[g])) return ST_INVALID_ARG;
    ga->out[g] = reinterpret_cast<__half*>(gather->out[g]);
    ga->flag_slot[g] = reinterpret_cast<unsigned*>(gather->flag_slot[g]);
  }
  ga->flags = reinterpret_cast<const unsigned*>(gather->flags_local);
  ga->epoch = reinterpret_cast<unsigned*>(gather->epoch_local);
  ga->buf_elems = gather->buffer_elems;
  ga->a_prev_off = gather->a_prev_offset;
  ga->done = reinterpret_cast<unsigned*>(workspace) + 8;  // word 8 of the status header
  return ST_OK;
}

static int run_stream(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N,
                      int K, int var, int group, int act, void* workspace, size_t ws_bytes, cudaStream_t stream,
                      const b200q_plan_t& pl, const b200q_gather_t* gather = nullptr, const void* a_host = nullptr,
                      int lda_host = 0, bool staging_released = false) {
  // a_host: device-side address of activations in pinned host memory (row stride lda_host); `a` is then
  // the dense [M, K] device staging the kernel's first CTAs fill (see StreamParams)
  const int bits = var_bits(var);
  const int KB = K / BLOCK_K;
  if (!stream_takes(K, group)) return ST_UNSUPPORTED;
  if (pl.splits < 1 || KB % pl.splits != 0 || pl.ctas_per_split < 1) return ST_INVALID_ARG;
  if (pl.stages < 1 || pl.stages > 8) return ST_INVALID_ARG;
  if (((uintptr_t)scales) & 15) return ST_INVALID_ARG;  // scale rows are fetched with 32-byte bulk copies
  const size_t need = stream_workspace_bytes(N);
  if (!workspace || ws_bytes < need || ((uintptr_t)workspace & 255)) return ST_WORKSPACE;
  StreamParams p;
  p.bq = bq;
  p.scales = reinterpret_cast<const __half*>(scales);
  p.status = reinterpret_cast<int*>(workspace);
  p.counters = reinterpret_cast<int*>(reinterpret_cast<char*>(workspace) + WS_HEADER_BYTES);
  p.partial = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + WS_HEADER_BYTES + ws_counter_bytes(N));
  p.N = N; p.K = K; p.lda = lda; p.ldc = ldc; p.KB = KB; p.NT = N / BLOCK_N;
  p.gshift = gshift_of(group);
  // Launches that hand rows over between GPUs release the launch of their successor late: measured on two
  // GPUs, a successor that becomes resident while this launch still waits for its peers costs 0.3 - 0.5 ms
  // per 128-layer step; launches that wait for nobody lose nothing either way.
  p.trig = gather ? 1 : 0;
  p.gdiv = group / 128;
  p.S = pl.splits; p.KBc = KB / pl.splits; p.CPC = pl.ctas_per_split;
  if (p.S * p.CPC > 4 * device_info().sm_count) return ST_INVALID_ARG;
  p.pitch = stream_pitch(p.KBc * 512);
  p.stages = pl.stages;
  p.pdl = pl.pdl;
  p.act = act;
  p.zero = 0u;
  {
    const int ipt = p.KBc * (4 / stream_gi(bits));  // items per column tile inside a k chunk
    p.ipt_shift = -1;
    if ((ipt & (ipt - 1)) == 0)
      for (int sh = 0; sh < 31; ++sh)
        if ((1 << sh) == ipt) p.ipt_shift = sh;
  }
  std::memset(&p.ga, 0, sizeof(p.ga));
  p.a_host = nullptr; p.fetch_flag = nullptr; p.fetch_ctas = 0; p.nowait = 0;
  if (a_host) {
    if (gather || M > stream_rows_per_pass(M)) return ST_INVALID_ARG;
    p.a_host = reinterpret_cast<const __half*>(a_host);
    p.lda = lda_host;
    p.fetch_flag = reinterpret_cast<unsigned*>(workspace) + 16;  // words 16, 17 of the status header
    p.fetch_ctas = stream_fetch_ctas(M, N, K, bits, pl);
    if (p.fetch_ctas > p.S * p.CPC) return ST_INVALID_ARG;
  }
  if (gather) {
    if (M > 16) return ST_INVALID_ARG;
    const int gst = fill_gather_args(gather, M, N, workspace, &p.ga);
    if (gst != ST_OK) return gst;
    p.ldc = gather->ldc;
  }
  const int rows = stream_rows_per_pass(M);
  for (int m0 = 0; m0 < M; m0 += rows) {
    const int mc = (M - m0) < rows ? (M - m0) : rows;
    p.a = reinterpret_cast<const __half*>(a) + (size_t)m0 * lda;  // (a_host: one pass, lda unused)
    p.c = reinterpret_cast<__half*>(c) + (size_t)m0 * ldc;
    p.M = mc;
    p.T_own = stream_tiles_owned(mc, p.NT, p.CPC);
    p.warp_shift = stream_warp_shift(mc, p.KBc * 512, bits, p.T_own, p.S * p.CPC);
    // (staging_released: the previous user of the staging buffer on this stream lets go of it before it
    // releases its successor - only then may this launch write it without waiting)
    p.nowait = (a_host && staging_released && p.S == 1 && p.T_own * p.CPC >= p.NT) ? 1 : 0;  // (the last CTA may own fewer tiles)
    // (rings of a plan edited to more slots than the launch has room for: as many as fit)
    const int fit = stream_stages_for(mc, p.KBc * 512, bits, p.T_own, p.S * p.CPC, device_info().max_smem);
    if (fit < 1) return ST_UNSUPPORTED;
    p.stages = pl.stages < fit ? pl.stages : fit;
    const int smem = stream_launch_smem(mc, p.KBc * 512, bits, p.stages, p.T_own, p.S * p.CPC);
    cudaError_t e = stream_launch(var, p, stream_mt(mc), smem, stream);
    if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  }
  return ST_OK;
}

static int run_resident(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N, int K,
                        int var, int group, int act, void* workspace, size_t ws_bytes, cudaStream_t stream, const b200q_plan_t& pl,
                        const ResidentSplit& rs) {
  // (The workspace and the rows of C that the plan's other form asks for, so that the same calls are refused whichever shapes come here; only the
  // status word is used.  The exact kernel's calls on rows at any distance are the stream kernel's, which K in whole 512-row blocks has.)
  const bool any_rows = (ldc % 8) != 0;
  if (pl.tile_m != 0 && any_rows && !stream_takes(K, group)) return ST_INVALID_ARG;
  const size_t need = pl.tile_m == 0 || any_rows ? stream_workspace_bytes(N) : WS_HEADER_BYTES + ws_counter_bytes(N);
  if (!workspace || ws_bytes < need || ((uintptr_t)workspace & 255)) return ST_WORKSPACE;
  if (((uintptr_t)scales) & 15) return ST_INVALID_ARG;
  ResidentParams p;
  p.a = reinterpret_cast<const __half*>(a);
  p.bq = bq;
  p.scales = reinterpret_cast<const __half*>(scales);
  p.c = reinterpret_cast<__half*>(c);
  p.status = reinterpret_cast<int*>(workspace);
  p.M = M; p.N = N; p.lda = lda; p.ldc = ldc;
  p.G = K / 128; p.NT = N / BLOCK_N;
  p.gshift = gshift_of(group); p.gdiv = group / 128;
  p.S = rs.S; p.T_own = rs.T_own; p.wk_shift = rs.wk_shift;
  p.stages = rs.stages; p.slab_shift = rs.slab_shift; p.grid = rs.grid;
  p.pdl = pl.pdl; p.act = act; p.zero = 0u;
  const cudaError_t e = resident_launch(var, p, stream_mt(M), rs.n_max, rs.smem, stream);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

// the form of the decode path (kernel 2) that exact_kernel.cu runs
static bool plan_is_exact(const b200q_plan_t& pl) { return pl.tile_m == 16 && pl.splits == 1; }

static int run_gemm(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N, int K,
                    int var, int group, int act, void* workspace, size_t ws_bytes, cudaStream_t stream,
                    const b200q_plan_t& pl) {
  if (!a || !bq || !scales || !c) return ST_INVALID_ARG;
  if (((uintptr_t)a | (uintptr_t)bq | (uintptr_t)c) & 15) return ST_INVALID_ARG;
  if (((uintptr_t)scales) & 1) return ST_INVALID_ARG;
  if (lda < K || ldc < N || (lda % 8) != 0) return ST_INVALID_ARG;
  // (a call that the resident kernel does not take - a plan put on more rows, or a tcgen05 plan on bfloat16, whose range fp16 does not
  // have - runs on the plan's other form)
  ResidentSplit rs;
  if (pl.resident > 0 && (pl.kernel == 2 || (pl.kernel == 3 && pl.tile_m == 16)) && group % 128 == 0 && !(act == B200Q_BF16 && (M > 8 || pl.tile_m != 0)) &&
      resident_split(M, N, K, var_bits(var), pl.resident, device_info(), &rs))
    return run_resident(a, lda, bq, scales, c, ldc, M, N, K, var, group, act, workspace, ws_bytes, stream, pl, rs);
  if (pl.kernel == 1 && pl.passes == 2) {
    // the full 256-row tiles on the tcgen05 kernel, the short last tile on the decode kernel
    const int tail = M % 256;
    if (M <= 256 || tail < 1 || tail > kStreamMaxRows) return ST_INVALID_ARG;
    b200q_plan_t tail_plan;
    int st = make_plan(tail, N, K, var, group, act, &tail_plan);
    if (st != ST_OK) return st;
    b200q_plan_t head = pl;
    head.passes = 1;
    st = run_umma(a, lda, bq, scales, c, ldc, M - tail, N, K, var, group, act, workspace, ws_bytes, stream, head);
    if (st != ST_OK) return st;
    const size_t row0 = (size_t)(M - tail);
    return run_gemm(reinterpret_cast<const unsigned short*>(a) + row0 * lda, lda, bq, scales,
                    reinterpret_cast<unsigned short*>(c) + row0 * ldc, ldc, tail, N, K, var, group, act, workspace,
                    ws_bytes, stream, tail_plan);
  }
  if (pl.kernel == 1)
    return run_umma(a, lda, bq, scales, c, ldc, M, N, K, var, group, act, workspace, ws_bytes, stream, pl);
  if (pl.kernel == 2 && plan_is_exact(pl) && (ldc % 8) != 0) {
    // rows of C at any distance: the exact kernel stores four columns at a time, the stream kernel single values
    b200q_plan_t rows;
    const int st = make_plan(M, N, K, var, group, kStreamForm, &rows);
    if (st != ST_OK) return st;
    return run_stream(a, lda, bq, scales, c, ldc, M, N, K, var, group, act, workspace, ws_bytes, stream, rows);
  }
  if (pl.kernel == 2 && plan_is_exact(pl))
    return run_batch(a, lda, bq, scales, c, ldc, M, N, K, var, group, act, workspace, ws_bytes, stream, pl);
  if (pl.kernel == 2 && pl.tile_m != 0 && stream_takes(K, group) && pl.splits > 0 && (K / BLOCK_K) % pl.splits == 0) {
    // a tcgen05 plan edited to more k chunks or to this kernel: the stream kernel's rings and column tiles bound the rest
    b200q_plan_t chunks = pl;
    const int rows = M < stream_rows_per_pass(M) ? M : stream_rows_per_pass(M);
    if (chunks.ctas_per_split > N / BLOCK_N) chunks.ctas_per_split = N / BLOCK_N;
    if (chunks.ctas_per_split > 4 * device_info().sm_count / pl.splits) chunks.ctas_per_split = 4 * device_info().sm_count / pl.splits;
    if (chunks.stages > 8) chunks.stages = 8;
    if (chunks.ctas_per_split > 0) {
      const int t_own = stream_tiles_owned(rows, N / BLOCK_N, chunks.ctas_per_split);
      const int fit = stream_stages_for(rows, K / pl.splits, var_bits(var), t_own, pl.splits * chunks.ctas_per_split, device_info().max_smem);
      if (fit < 1 && plan_stream(rows, N, K, var_bits(var), device_info(), &chunks) != ST_OK) return ST_UNSUPPORTED;
    }
    return run_stream(a, lda, bq, scales, c, ldc, M, N, K, var, group, act, workspace, ws_bytes, stream, chunks);
  }
  if (pl.kernel == 2)
    return run_stream(a, lda, bq, scales, c, ldc, M, N, K, var, group, act, workspace, ws_bytes, stream, pl);
  if (pl.kernel == 3) {
    for (int m0 = 0; m0 < M; m0 += kBatchMaxRows) {  // (more rows only by an edited plan)
      const int st = run_batch(reinterpret_cast<const unsigned short*>(a) + (size_t)m0 * lda, lda, bq, scales,
                               reinterpret_cast<unsigned short*>(c) + (size_t)m0 * ldc, ldc,
                               M - m0 < kBatchMaxRows ? M - m0 : kBatchMaxRows, N, K, var, group, act, workspace, ws_bytes,
                               stream, pl);
      if (st != ST_OK) return st;
    }
    return ST_OK;
  }
  return ST_UNSUPPORTED;
}

static bool act_ok(int act) { return act == B200Q_F16 || act == B200Q_BF16; }

}  // namespace b200q

using namespace b200q;

extern "C" {

int b200q_version(void) { return 100; }
int b200q_layout_version(void) { return 1; }

const char* b200q_status_string(int status) {
  switch (status) {
    case ST_OK: return "ok";
    case ST_INVALID_ARG: return "invalid argument (null or misaligned pointer, bad size or stride)";
    case ST_UNSUPPORTED: return "unsupported weight dtype, zero point, shape or group size";
    case ST_WORKSPACE: return "workspace missing, misaligned or too small";
    case ST_CUDA: return "CUDA runtime error";
    case ST_DEVICE_TIMEOUT: return "a bounded device-side wait timed out";
    default: return "unknown status";
  }
}

int b200q_last_cuda_error(void) { return g_last_cuda_error; }

int b200q_plan(int M, int N, int K, int wtype, int zero_point, int group, b200q_plan_t* plan) {
  return b200q_plan_for(M, N, K, wtype, zero_point, group, B200Q_F16, plan);
}

int b200q_plan_for(int M, int N, int K, int wtype, int zero_point, int group, int act_dtype, b200q_plan_t* plan) {
  if (!plan) return ST_INVALID_ARG;
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  int var;
  int st = check_problem(M, N, K, wtype, zero_point, group, true, &var);
  if (st != ST_OK) return st;
  return make_plan(M, N, K, var, group, act_dtype, plan);
}

size_t b200q_workspace_bytes(int M, int N, int K, int wtype, int zero_point, int group) {
  b200q_plan_t pl;
  if (b200q_plan(M, N, K, wtype, zero_point, group, &pl) != ST_OK) return 0;
  return (size_t)pl.workspace_bytes;
}

int b200q_gemm_planned(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N,
                       int K, int wtype, int zero_point, int group, int act_dtype, void* workspace,
                       size_t workspace_bytes, void* stream, const b200q_plan_t* plan) {
  if (!plan) return ST_INVALID_ARG;
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  int var;
  int st = check_problem(M, N, K, wtype, zero_point, group, true, &var);
  if (st != ST_OK) return st;
  b200q_plan_t pl = *plan;
  if (pl.resident > 0) {  // an edit of any other field names one of the other kernels
    b200q_plan_t own;
    const int rows = M < 16 ? M : 16;
    if (make_plan(rows, N, K, var, group, act_dtype, &own) != ST_OK || own.kernel != pl.kernel || own.tile_m != pl.tile_m ||
        own.splits != pl.splits || own.cluster != pl.cluster || own.ctas_per_split != pl.ctas_per_split || own.stages != pl.stages)
      pl.resident = 0;
  }
  return run_gemm(a, lda, bq, scales, c, ldc, M, N, K, var, group, act_dtype, workspace, workspace_bytes,
                  reinterpret_cast<cudaStream_t>(stream), pl);
}

int b200q_gemm_gather(const void* a, int lda, const void* bq, const void* scales, int M, int N, int K, int wtype,
                      int zero_point, int group, int act_dtype, void* workspace, size_t workspace_bytes, void* stream,
                      const b200q_gather_t* gather) {
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  if (!gather || !bq || !scales) return ST_INVALID_ARG;
  if (M > 16) return ST_UNSUPPORTED;  // the tcgen05 kernel has no fused gather: use b200q_gemm + a collective
  if (gather->a_prev_offset < 0 && (!a || ((uintptr_t)a & 15))) return ST_INVALID_ARG;
  if (gather->a_prev_offset >= 0 && (gather->a_prev_offset % 8) != 0) return ST_INVALID_ARG;
  if (((uintptr_t)bq) & 15) return ST_INVALID_ARG;
  if (lda < K || (lda % 8) != 0) return ST_INVALID_ARG;
  int var;
  int st = check_problem(M, N, K, wtype, zero_point, group, true, &var);
  if (st != ST_OK) return st;
  b200q_plan_t pl;  // the fused gather lives in the stream kernel only
  if (make_plan(M, N, K, var, group, kStreamForm, &pl) != ST_OK) return ST_UNSUPPORTED;
  return run_stream(a, lda, bq, scales, nullptr, gather->ldc, M, N, K, var, group, act_dtype, workspace,
                    workspace_bytes, reinterpret_cast<cudaStream_t>(stream), pl, gather);
}

int b200q_gather_push(const void* shard, int lds, int M, int N_loc, void* workspace, size_t workspace_bytes,
                      void* stream, const b200q_gather_t* gather) {
  if (!shard || !gather || M < 1 || N_loc < 8) return ST_INVALID_ARG;
  if ((N_loc % 8) != 0 || (lds % 8) != 0 || lds < N_loc || (((uintptr_t)shard) & 15)) return ST_INVALID_ARG;
  if ((gather->ldc % 8) != 0 || (gather->col_offset % 8) != 0) return ST_INVALID_ARG;
  if (!workspace || workspace_bytes < WS_HEADER_BYTES || ((uintptr_t)workspace & 255)) return ST_WORKSPACE;
  GatherArgs ga;
  const int st = fill_gather_args(gather, M, N_loc, workspace, &ga);
  if (st != ST_OK) return st;
  cudaError_t e = gather_push_launch(shard, lds, M, N_loc, gather->ldc, reinterpret_cast<int*>(workspace), ga,
                                     reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

int b200q_gather_collect(void* full_local, int ld_local, int M, void* workspace, size_t workspace_bytes, void* stream,
                         const b200q_gather_t* gather) {
  if (!gather || M < 1) return ST_INVALID_ARG;
  if ((gather->ldc % 8) != 0) return ST_INVALID_ARG;
  if (full_local && ((ld_local % 8) != 0 || ld_local < gather->ldc || (((uintptr_t)full_local) & 15))) return ST_INVALID_ARG;
  if (!workspace || workspace_bytes < WS_HEADER_BYTES || ((uintptr_t)workspace & 255)) return ST_WORKSPACE;
  GatherArgs ga;
  const int st = fill_gather_args(gather, M, 0, workspace, &ga);
  if (st != ST_OK) return st;
  cudaError_t e = gather_collect_launch(full_local, ld_local, M, gather->ldc, reinterpret_cast<int*>(workspace), ga,
                                        reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

int b200q_peer_alloc(size_t bytes, void** ptr) {
  if (!ptr || bytes == 0) return ST_INVALID_ARG;
  cudaError_t e = cudaMalloc(ptr, bytes);
  if (e == cudaSuccess) e = cudaMemset(*ptr, 0, bytes);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}
int b200q_peer_export(void* ptr, unsigned char handle[64]) {
  if (!ptr || !handle) return ST_INVALID_ARG;
  static_assert(sizeof(cudaIpcMemHandle_t) == 64, "IPC handle size");
  cudaIpcMemHandle_t h;
  cudaError_t e = cudaIpcGetMemHandle(&h, ptr);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  std::memcpy(handle, &h, 64);
  return ST_OK;
}
int b200q_peer_open(const unsigned char handle[64], void** ptr) {
  if (!ptr || !handle) return ST_INVALID_ARG;
  cudaIpcMemHandle_t h;
  std::memcpy(&h, handle, 64);
  cudaError_t e = cudaIpcOpenMemHandle(ptr, h, cudaIpcMemLazyEnablePeerAccess);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}
int b200q_peer_close(void* ptr) {
  if (!ptr) return ST_INVALID_ARG;
  cudaError_t e = cudaIpcCloseMemHandle(ptr);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}
int b200q_peer_free(void* ptr) {
  if (!ptr) return ST_INVALID_ARG;
  cudaError_t e = cudaFree(ptr);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

int b200q_gemm(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N, int K,
               int wtype, int zero_point, int group, int act_dtype, void* workspace, size_t workspace_bytes,
               void* stream) {
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  int var;
  int st = check_problem(M, N, K, wtype, zero_point, group, true, &var);
  if (st != ST_OK) return st;
  b200q_plan_t pl;
  st = make_plan(M, N, K, var, group, act_dtype, &pl);
  if (st != ST_OK) return st;
  plan_within(M, N, K, var, group, workspace_bytes, &pl);
  return run_gemm(a, lda, bq, scales, c, ldc, M, N, K, var, group, act_dtype, workspace, workspace_bytes,
                  reinterpret_cast<cudaStream_t>(stream), pl);
}

// ---- GEMM on host buffers ------------------------------------------------------------------------
// Activations in (pinned) host memory, result back in host memory, queued on the stream by one
// call.  The activations are copied into a staging buffer the caller owns (every CTA reads all
// of them, which must not cross the host link each time).  The result, which every element of
// is written exactly once, goes straight to the host buffer when that is pinned memory the GPU
// can address (the kernel's stores are the transfer); otherwise through the second staging
// buffer and a copy.
// Who used a staging buffer last on a stream, as far as b200q_gemm_host calls tell: a decode launch that fetches its own
// activations has finished reading the buffer by the time its successor can start; every other kernel reads it
// until it ends.  Threads may share a stream, so the record is the process's.  A captured graph is a record of its own,
// by the order of capture: its first launch follows everything before the graph, and what it captures has not run
// on the stream.
struct StagingUse { cudaStream_t stream; const void* buf; unsigned long long capture; bool released; };
static bool staging_released_by_last_use(cudaStream_t st, const void* buf, bool now_released) {
  static std::mutex mu;
  static StagingUse uses[32];
  static int next = 0;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long capture = 0;
  if (cudaStreamGetCaptureInfo(st, &status, &capture) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;  // (the launch will say what is wrong)
  }
  if (status != cudaStreamCaptureStatusActive) capture = 0;
  std::lock_guard<std::mutex> lock(mu);
  for (StagingUse& u : uses)
    if (u.stream == st && u.buf == buf && u.capture == capture && u.buf != nullptr) {
      const bool was = u.released;
      u.released = now_released;
      return was;
    }
  uses[next] = {st, buf, capture, now_released};
  next = (next + 1) % 32;
  return false;  // unknown history: wait
}

int b200q_gemm_host(const void* a_host, int lda, const void* bq, const void* scales, void* c_host, int ldc, int M,
                    int N, int K, int wtype, int zero_point, int group, int act_dtype, void* a_staging,
                    void* c_staging, void* workspace, size_t workspace_bytes, void* stream) {
  if (!a_host || !c_host || !a_staging || !c_staging) return ST_INVALID_ARG;
  if (M < 1 || N < 1 || K < 1 || lda < K || ldc < N) return ST_INVALID_ARG;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e;
  // Small activation blocks in pinned memory the GPU can address are fetched by a kernel whose PCIe
  // reads lie under the previous GEMM of the stream (fetch_kernel.cu); the rest goes through the copy engine.
  const void* a_mapped = nullptr;
  if ((size_t)M * K * 2 <= (256u << 10) && (K % 8) == 0 && (lda % 8) == 0 && (((uintptr_t)a_staging) & 15) == 0) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, a_host) == cudaSuccess && attr.type == cudaMemoryTypeHost &&
        attr.devicePointer && (((uintptr_t)attr.devicePointer) & 15) == 0)
      a_mapped = attr.devicePointer;
    else
      (void)cudaGetLastError();  // an unregistered host pointer is not an error here
  }
  // Decode batches: the GEMV kernel's own first CTAs fetch the rows (one kernel, no copy operation at
  // all) when the result can also go straight to the host buffer and the launch has CTAs enough for them (a layer of a few
  // column tiles with a long K has not: 4 x 48 x 14336 is three CTAs, its rows take four).
  if (a_mapped && act_ok(act_dtype) && (ldc % 8) == 0 && (size_t)M * N * 2 <= (1u << 20)) {
    int var;
    b200q_plan_t pl;
    cudaPointerAttributes cattr;
    if (check_problem(M, N, K, wtype, zero_point, group, true, &var) == ST_OK &&
        make_plan(M, N, K, var, group, kStreamForm, &pl) == ST_OK &&
        pl.splits * pl.ctas_per_split <= 2 * device_info().sm_count / stream_mt(M) &&
        stream_fetch_ctas(M, N, K, var_bits(var), pl) <= pl.splits * pl.ctas_per_split) {
      if (cudaPointerGetAttributes(&cattr, c_host) == cudaSuccess && cattr.type == cudaMemoryTypeHost &&
          cattr.devicePointer && (((uintptr_t)cattr.devicePointer) & 15) == 0) {
        if (!bq || !scales) return ST_INVALID_ARG;
        if ((((uintptr_t)bq) & 15) || lda < K) return ST_INVALID_ARG;
        const bool released = staging_released_by_last_use(st, a_staging, true);
        return run_stream(a_staging, K, bq, scales, cattr.devicePointer, ldc, M, N, K, var, group, act_dtype, workspace,
                          workspace_bytes, st, pl, nullptr, a_mapped, lda, released);
      }
      (void)cudaGetLastError();
    }
  }
  (void)staging_released_by_last_use(st, a_staging, false);  // what follows reads the buffer until it ends
  if (a_mapped)
    e = host_fetch_launch(a_mapped, lda, a_staging, M, K, st);
  else
    e = lda == K ? cudaMemcpyAsync(a_staging, a_host, (size_t)M * K * 2, cudaMemcpyHostToDevice, st)
                 : cudaMemcpy2DAsync(a_staging, (size_t)K * 2, a_host, (size_t)lda * 2, (size_t)K * 2, M,
                                     cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  // small results into mapped pinned memory: no copy-out operation on the stream
  void* c_direct = nullptr;
  if ((size_t)M * N * 2 <= (1u << 20) && (ldc % 8) == 0) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, c_host) == cudaSuccess && attr.type == cudaMemoryTypeHost &&
        attr.devicePointer && (((uintptr_t)attr.devicePointer) & 15) == 0)
      c_direct = attr.devicePointer;
    else
      (void)cudaGetLastError();  // an unregistered host pointer is not an error here
  }
  if (c_direct)
    return b200q_gemm(a_staging, K, bq, scales, c_direct, ldc, M, N, K, wtype, zero_point, group, act_dtype, workspace,
                      workspace_bytes, stream);
  const int status = b200q_gemm(a_staging, K, bq, scales, c_staging, N, M, N, K, wtype, zero_point, group, act_dtype,
                                workspace, workspace_bytes, stream);
  if (status != ST_OK) return status;
  e = ldc == N ? cudaMemcpyAsync(c_host, c_staging, (size_t)M * N * 2, cudaMemcpyDeviceToHost, st)
               : cudaMemcpy2DAsync(c_host, (size_t)ldc * 2, c_staging, (size_t)N * 2, (size_t)N * 2, M,
                                   cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

// ---- GEMM without a caller-supplied workspace and without any allocation ----------------------
// The split-K scratch (status header, arrival counters, fp32 partial sums) lives in this
// file-scope device array instead of a caller buffer.  Every GPU on which the array's module has
// been loaded holds these bytes until the process exits.  In host code `g_static_ws` is only a
// handle for the symbol, not a device address: the address each device uses is looked up once with
// cudaGetSymbolAddress while that device is current.  Device arrays start zeroed and the kernels
// leave their scratch zeroed, so nothing is cleared here.
#define B200Q_STATIC_WS_BYTES (8u << 20)
static __device__ __align__(256) unsigned char g_static_ws[B200Q_STATIC_WS_BYTES];

static int static_ws_pointer(void** out) {
  static std::mutex mu;
  static void* ptrs[16] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  if (dev < 0 || dev >= 16) return ST_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(mu);
  if (!ptrs[dev]) {
    void* ptr = nullptr;
    e = cudaGetSymbolAddress(&ptr, g_static_ws);  // device `dev` is current
    if (e != cudaSuccess || !ptr) { g_last_cuda_error = (int)e; return ST_CUDA; }
    ptrs[dev] = ptr;
  }
  *out = ptrs[dev];
  return ST_OK;
}

size_t b200q_static_workspace_limit(void) { return (size_t)B200Q_STATIC_WS_BYTES; }

int b200q_static_ws_init(void) {
  void* ws = nullptr;
  return static_ws_pointer(&ws);
}

int b200q_gemm_static_ws(const void* a, int lda, const void* bq, const void* scales, void* c, int ldc, int M, int N,
                         int K, int wtype, int zero_point, int group, int act_dtype, void* stream) {
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  int var;
  int st = check_problem(M, N, K, wtype, zero_point, group, true, &var);
  if (st != ST_OK) return st;
  b200q_plan_t pl;
  st = make_plan(M, N, K, var, group, act_dtype, &pl);
  if (st != ST_OK) return st;
  plan_within(M, N, K, var, group, B200Q_STATIC_WS_BYTES, &pl);
  if (pl.workspace_bytes > (uint64_t)B200Q_STATIC_WS_BYTES) {
    // beyond the built-in scratch - unless all that asks for the room is a K split that the kernel does
    // without when the scratch is too small (small batches; the prefill kernel's last round).  The decode path takes
    // the same problems whichever of its kernels runs: those whose stream scratch fits.
    const bool exact = pl.kernel == 2 && plan_is_exact(pl);
    const uint64_t least = pl.passes == 2 || exact ? stream_workspace_bytes(N) : WS_HEADER_BYTES + ws_counter_bytes(N);
    const bool optional = pl.kernel == 3 || exact || (pl.kernel == 1 && pl.splits == 1);
    if (!(optional && least <= (uint64_t)B200Q_STATIC_WS_BYTES)) return ST_WORKSPACE;
  }
  void* ws = nullptr;
  st = static_ws_pointer(&ws);
  if (st != ST_OK) return st;
  return run_gemm(a, lda, bq, scales, c, ldc, M, N, K, var, group, act_dtype, ws, (size_t)B200Q_STATIC_WS_BYTES,
                  reinterpret_cast<cudaStream_t>(stream), pl);
}

int b200q_dequantize(const void* bq, const void* scales, void* w, int N, int K, int wtype, int zero_point, int group,
                     int act_dtype, void* stream) {
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  int var;
  int st = check_problem(1, N, K, wtype, zero_point, group, false, &var);
  if (st != ST_OK) return st;
  if (!bq || !scales || !w) return ST_INVALID_ARG;
  if (((uintptr_t)bq | (uintptr_t)w) & 15) return ST_INVALID_ARG;
  DequantParams p;
  p.bq = reinterpret_cast<const uint4*>(bq);
  p.scales = reinterpret_cast<const __half*>(scales);
  p.w = reinterpret_cast<__half*>(w);
  p.N = N; p.K = K; p.group = group; p.G = K / 128; p.NT = N / BLOCK_N;
  p.act = act_dtype;
  cudaError_t e = dequant_launch(var, p, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

int b200q_quantize(const void* weight, int weight_dtype, int ldw, void* bq, void* scales, int N, int K, int wtype,
                   int group, int act_dtype, void* stream) {
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  if (!weight || !bq || !scales) return ST_INVALID_ARG;
  if (N < 1 || K < 1 || group < 1 || ldw < K) return ST_INVALID_ARG;
  if (weight_dtype < 0 || weight_dtype > 2) return ST_UNSUPPORTED;
  const int kind = (wtype >> 16) & 0xff, nbits = (wtype >> 8) & 0xff, e = (wtype >> 4) & 0xf, m = wtype & 0xf;
  if (kind > 2 || nbits < 1 || nbits > 8) return ST_UNSUPPORTED;
  if (kind == 2 && (nbits != 1 + e + m || e < 1 || m < 1)) return ST_UNSUPPORTED;
  if (K % 128 != 0 || N % BLOCK_N != 0 || group % 32 != 0 || K % group != 0) return ST_UNSUPPORTED;
  if (((uintptr_t)bq & 15) || ((uintptr_t)scales & 1) || ((uintptr_t)weight & 3)) return ST_INVALID_ARG;
  float minv, maxv;
  if (kind == 0) { minv = 0.f; maxv = (float)((1 << nbits) - 1); }
  else if (kind == 1) { minv = -(float)(1 << (nbits - 1)); maxv = (float)((1 << (nbits - 1)) - 1); }
  else {
    const int bias = (1 << (e - 1)) - 1, top = (1 << e) - 1 - (e == 5 ? 1 : 0);
    maxv = ldexpf(2.0f - ldexpf(1.0f, -m), top - bias);
    minv = -maxv;
  }
  cudaError_t err = quantize_launch(weight, weight_dtype, ldw, bq, scales, N, K, group, kind, nbits, e, m, minv, maxv,
                                    act_dtype, reinterpret_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) { g_last_cuda_error = (int)err; return ST_CUDA; }
  return ST_OK;
}

static int run_cast(const void* x, int ldx, void* out, int ldo, float* out_sf, int tokens, int hidden, int group,
                    int act_dtype, bool swiglu, const int32_t* pos_to_token_topk, const float* topk_weights,
                    const int32_t* pos_to_expert, int use_clamp, float clamp_value, void* stream) {
  if (!act_ok(act_dtype)) return ST_UNSUPPORTED;
  if (!x || !out || !out_sf) return ST_INVALID_ARG;
  if (tokens < 1 || hidden < 1 || group < 1) return ST_INVALID_ARG;
  if (group % 128 != 0 || group > 512 || hidden % group != 0) return ST_UNSUPPORTED;
  if (ldx < (swiglu ? 2 * hidden : hidden) || ldo < hidden || (ldx % 8) != 0 || (ldo % 8) != 0) return ST_INVALID_ARG;
  if ((((uintptr_t)x) & 15) || (((uintptr_t)out) & 7) || (((uintptr_t)out_sf) & 3)) return ST_INVALID_ARG;
  CastParams p;
  p.x = reinterpret_cast<const unsigned short*>(x);
  p.out = reinterpret_cast<unsigned char*>(out);
  p.out_sf = out_sf;
  p.T = tokens; p.H = hidden; p.ldx = ldx; p.ldo = ldo; p.group = group;
  p.pos_to_token_topk = pos_to_token_topk;
  p.topk_weights = topk_weights;
  p.pos_to_expert = pos_to_expert;
  p.clamp = clamp_value;
  p.use_clamp = use_clamp ? 1 : 0;
  cudaError_t e = cast_launch(p, act_dtype, swiglu, reinterpret_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return ST_OK;
}

int b200q_per_token_cast(const void* x, int ldx, void* out, int ldo, float* out_sf, int tokens, int hidden, int group,
                         int act_dtype, void* stream) {
  return run_cast(x, ldx, out, ldo, out_sf, tokens, hidden, group, act_dtype, false, nullptr, nullptr, nullptr, 0, 0.f,
                  stream);
}

int b200q_swiglu_per_token_cast(const void* x, int ldx, void* out, int ldo, float* out_sf, int tokens, int hidden,
                                int group, int act_dtype, const int32_t* pos_to_token_topk, const float* topk_weights,
                                const int32_t* pos_to_expert, int use_clamp, float clamp_value, void* stream) {
  return run_cast(x, ldx, out, ldo, out_sf, tokens, hidden, group, act_dtype, true, pos_to_token_topk, topk_weights,
                  pos_to_expert, use_clamp, clamp_value, stream);
}

int b200q_gemm_swiglu_cast(const void* a, int lda, const void* bq, const void* scales, void* gate_up, int ldg,
                           void* out, int ldo, float* out_sf, int M, int N, int K, int wtype, int zero_point, int group,
                           int act_dtype, int cast_group, int use_clamp, float clamp_value, void* workspace,
                           size_t workspace_bytes, void* stream) {
  if ((N & 1) != 0) return ST_INVALID_ARG;
  const int st = b200q_gemm(a, lda, bq, scales, gate_up, ldg, M, N, K, wtype, zero_point, group, act_dtype, workspace,
                            workspace_bytes, stream);
  if (st != ST_OK) return st;
  return run_cast(gate_up, ldg, out, ldo, out_sf, M, N / 2, cast_group, act_dtype, true, nullptr, nullptr, nullptr,
                  use_clamp, clamp_value, stream);
}

int b200q_device_status(void* workspace, int32_t status[4], void* stream) {
  if (!status) return ST_INVALID_ARG;
  const bool builtin = workspace == nullptr;  // the scratch of b200q_gemm_static_ws
  if (builtin) {
    const int st = static_ws_pointer(&workspace);
    if (st != ST_OK) return st;
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(status, workspace, 16, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && status[0] != 0) {
    // a launch that gave up may have left partial sums and arrival counters behind: the built-in
    // scratch is put back to zero as a whole (its owner cannot do it), a caller's workspace only
    // loses the report (the caller clears the rest, whose size only it knows)
    e = cudaMemsetAsync(workspace, 0, builtin ? (size_t)B200Q_STATIC_WS_BYTES : 16, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  if (e != cudaSuccess) { g_last_cuda_error = (int)e; return ST_CUDA; }
  return status[0] == 0 ? ST_OK : ST_DEVICE_TIMEOUT;
}

}  // extern "C"
